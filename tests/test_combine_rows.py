"""The combine by the number of its blocks (256 float4 columns of a row each): one kernel while three an SM hold them
all, one while four do, one for more; each adds a row's experts in the same order."""
import numpy as np
import pytest

from biv_b200 import workloads as W

pytestmark = pytest.mark.gpu


# 12 experts a token: the first kernel takes eight at a time.  One block a row (1024 columns) and two, the second ragged
@pytest.mark.parametrize("n_embd,k,ff_sh", [(1024, 12, 256), (1280, 7, 0)])
def test_the_kernels_of_few_and_many_blocks_give_the_same_rows(n_embd, k, ff_sh):
    import torch
    from biv_b200.moe import Moe
    per_row = (n_embd + 1023) // 1024
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    few, some = 3 * sms // per_row, 4 * sms // per_row    # the last row counts of the first two
    n = some + 1
    rng = np.random.default_rng(n_embd)
    layer = W.make_layer(rng, gate_ty=W.Q4_0, down_ty=W.Q4_0, n_embd=n_embd, n_expert=16, k=k, ff=256, ff_sh=ff_sh,
                         router_dist="uniform")
    h = torch.from_numpy(W.rms_normalise(rng.standard_normal((n, n_embd), dtype=np.float32))).cuda()
    m = Moe(layer, n)
    try:
        want = m.moe(h)
        old = torch.randn_like(h)
        sums = m.moe_(h, old.clone(), accumulate=True)
        assert torch.equal(sums, want + old)
        for rows in (few, few + 1, some):
            assert torch.equal(m.moe(h[:rows].contiguous()), want[:rows]), rows
            assert torch.equal(m.moe_(h[:rows].contiguous(), old[:rows].clone(), accumulate=True), sums[:rows]), rows
        m.status()
    finally:
        m.close()


def test_rows_of_some_blocks_against_the_oracle():
    from test_gpu_parity import run_case
    rng = np.random.default_rng(3)
    layer = W.make_layer(rng, gate_ty=W.Q4_0, down_ty=W.Q4_1, n_embd=256, n_expert=16, k=12, ff=256, ff_sh=256,
                         router_dist="uniform")
    h = W.rms_normalise(rng.standard_normal((445, 256), dtype=np.float32))
    run_case(W.Workload("some_blocks", 445, [layer], h))
