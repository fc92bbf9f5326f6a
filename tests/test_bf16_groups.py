"""Groups of BF16 rows on the tensor cores (experts_prefill_bf16.cu), against the oracle: at the edges of a
tile and of the width up to which its tokens are the columns of gate+up, alone and behind whole tiles."""
import numpy as np
import pytest

from biv_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_embd,ff", [(1, 256, 256), (15, 512, 256), (17, 256, 512), (48, 256, 256), (64, 512, 256),
                                         (65, 256, 256), (129, 256, 2048), (192, 512, 256), (321, 256, 4096)])
def test_a_group_of_every_width(n, n_embd, ff, monkeypatch):
    from biv_b200.moe import Moe
    from test_gpu_parity import run_case
    monkeypatch.setenv("BIVMOE_PREFILL_MIN", "1")
    rng = np.random.default_rng(n)
    layer = W.make_layer(rng, gate_ty=W.BF16, down_ty=W.BF16, n_embd=n_embd, n_expert=1, k=1, ff=ff, ff_sh=0)
    layer.router[:] = 0
    h = W.rms_normalise(rng.standard_normal((n, n_embd), dtype=np.float32))
    run_case(W.Workload("dense", n, [layer], h), make=lambda l, cap: Moe.dense(l.gate, l.up, l.down, cap))


def test_a_layers_groups_of_all_widths(monkeypatch):
    from test_gpu_parity import run_case
    monkeypatch.setenv("BIVMOE_PREFILL_MIN", "1")
    rng = np.random.default_rng(3)
    layer = W.make_layer(rng, gate_ty=W.BF16, down_ty=W.BF16, n_embd=256, n_expert=16, k=2, ff=512, ff_sh=256,
                         router_dist="uniform")
    h = W.rms_normalise(rng.standard_normal((610, 256), dtype=np.float32))
    run_case(W.Workload("groups", 610, [layer], h))
