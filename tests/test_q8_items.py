"""The Q8_0 tensor-core kernels by a block's items: the last one's output is made by other warps than the others',
and down products of many short items have a kernel of their own; every row is the same, and the oracle's."""
import numpy as np
import pytest

from biv_b200 import workloads as W

pytestmark = pytest.mark.gpu


# ff 256 and 512 (a stage or two): 700 rows are many items a block for the short items' kernel, 40 rows one or none
# for the other; ff 768: three stages, the other kernel both times.  The shared expert has more rows or fewer than the
# routed ones: a block's last items are empty then, and no item is known to be the last.
@pytest.mark.parametrize("ff,ff_sh", [(256, 0), (512, 512), (256, 768), (768, 256)])
def test_rows_are_the_same_in_small_and_large_passes(ff, ff_sh, monkeypatch):
    import torch
    from biv_b200.moe import Moe
    monkeypatch.setenv("BIVMOE_PREFILL_MIN", "1")
    rng = np.random.default_rng(ff)
    layer = W.make_layer(rng, gate_ty=W.Q8_0, down_ty=W.Q8_0, n_embd=2048, n_expert=24, k=4, ff=ff, ff_sh=ff_sh, router_dist="uniform")
    h = torch.from_numpy(W.rms_normalise(rng.standard_normal((700, 2048), dtype=np.float32))).cuda()
    m = Moe(layer, 700)
    try:
        want = m.moe(h)
        for n in (1, 40, 300):
            assert torch.equal(m.moe(h[:n].contiguous()), want[:n]), n
        m.status()
    finally:
        m.close()


@pytest.mark.parametrize("n,ff,ff_sh", [(700, 256, 512), (90, 512, 256)])
def test_items_against_the_oracle(n, ff, ff_sh, monkeypatch):
    from test_gpu_parity import run_case
    monkeypatch.setenv("BIVMOE_PREFILL_MIN", "1")
    rng = np.random.default_rng(n)
    layer = W.make_layer(rng, gate_ty=W.Q8_0, down_ty=W.Q8_0, n_embd=2048, n_expert=24, k=2, ff=ff, ff_sh=ff_sh, router_dist="uniform")
    h = W.rms_normalise(rng.standard_normal((n, 2048), dtype=np.float32))
    run_case(W.Workload("items", n, [layer], h))
