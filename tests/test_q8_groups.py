"""Groups of Q8_0 rows on the int8 tensor cores (experts_prefill.cu), against the oracle: at the edges of
a tile and of the widths at which its tokens are dealt out, with items of one stage, several items a block
and blocks without one."""
import numpy as np
import pytest

from biv_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_embd,ff", [(1, 256, 256), (8, 512, 256), (31, 256, 512), (33, 512, 256), (64, 256, 256),
                                         (65, 512, 256), (127, 256, 256), (129, 256, 2048), (700, 256, 2048)])
def test_a_group_of_every_width(n, n_embd, ff, monkeypatch):
    from biv_b200.moe import Moe
    from test_gpu_parity import run_case
    monkeypatch.setenv("BIVMOE_PREFILL_MIN", "1")
    rng = np.random.default_rng(n)
    layer = W.make_layer(rng, gate_ty=W.Q8_0, down_ty=W.Q8_0, n_embd=n_embd, n_expert=1, k=1, ff=ff, ff_sh=0)
    layer.router[:] = 0
    h = W.rms_normalise(rng.standard_normal((n, n_embd), dtype=np.float32))
    run_case(W.Workload("dense", n, [layer], h), make=lambda l, cap: Moe.dense(l.gate, l.up, l.down, cap))

