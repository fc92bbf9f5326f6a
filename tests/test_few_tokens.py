"""Passes of up to eight tokens: the kernel that routes, quantises and multiplies by gate and up in one
launch, against the oracle and against the kernels of larger passes, bit for bit."""
import numpy as np
import pytest

from biv_b200 import workloads as W

pytestmark = pytest.mark.gpu


# one and eight tokens; with and without a shared expert; one selected expert; 256 experts and more (the
# general kernels); one K-slice, eight (dealt to a block's groups) and nine (too wide for that, or for
# shared memory).  (SwiGLU rows of 512 at most: a re-quantised value off by a step is met about once in
# 10 000 to 100 000, and run_case allows it in 2 % of the pairs; more work items than blocks are below.)
@pytest.mark.parametrize("gate_ty,down_ty,n,kw", [
    (W.Q4_K, W.Q6_K, 1, dict(n_embd=256, n_expert=16, k=4, ff=256, ff_sh=0)),
    (W.Q4_K, W.Q4_K, 8, dict(n_embd=2048, n_expert=64, k=8, ff=512, ff_sh=512)),
    (W.Q5_K, W.Q6_K, 3, dict(n_embd=2048, n_expert=16, k=4, ff=256, ff_sh=512)),
    (W.Q5_K, W.Q5_K, 8, dict(n_embd=2304, n_expert=16, k=1, ff=256, ff_sh=256)),
    (W.Q6_K, W.Q8_0, 7, dict(n_embd=512, n_expert=256, k=6, ff=256, ff_sh=0)),
    (W.Q8_0, W.Q4_0, 8, dict(n_embd=2304, n_expert=16, k=4, ff=256, ff_sh=256)),
    (W.Q4_0, W.Q4_1, 2, dict(n_embd=1280, n_expert=300, k=3, ff=256, ff_sh=256)),
    (W.Q4_1, W.Q4_0, 8, dict(n_embd=768, n_expert=32, k=8, ff=512, ff_sh=256)),
])
def test_a_few_tokens(gate_ty, down_ty, n, kw):
    from test_gpu_parity import run_case
    rng = np.random.default_rng(n)
    layer = W.make_layer(rng, gate_ty=gate_ty, down_ty=down_ty, router_dist="uniform", **kw)
    h = W.rms_normalise(rng.standard_normal((n, layer.n_embd), dtype=np.float32))
    run_case(W.Workload("few", n, [layer], h))


@pytest.mark.parametrize("ty", [W.Q4_K, W.Q5_K, W.Q6_K, W.Q8_0, W.Q4_0, W.Q4_1])
@pytest.mark.parametrize("ff", [256, 3072])
def test_the_same_bits_as_in_a_larger_pass(ty, ff):
    # items that a block's groups share, and more items than blocks; a row with a NaN costs its own output only
    import torch
    from biv_b200.moe import Moe
    rng = np.random.default_rng(ff)
    layer = W.make_layer(rng, gate_ty=ty, n_embd=1024, n_expert=8, k=2, ff=ff, ff_sh=256)
    h = torch.from_numpy(W.rms_normalise(rng.standard_normal((9, 1024), dtype=np.float32))).cuda()
    m = Moe(layer, 9)
    try:
        want = m.moe(h)
        for n in (1, 2, 8):
            for t in (0, 9 - n):
                assert torch.equal(m.moe(h[t:t + n].contiguous()), want[t:t + n]), (n, t)
        h[3, 7] = float("nan")
        got = m.moe(h[:8].contiguous())
        assert torch.isnan(got[3]).all()
        keep = [0, 1, 2, 4, 5, 6, 7]
        assert torch.equal(got[keep], want[keep])
    finally:
        m.close()


# the norm applied by the router and by the quantiser of the few-token kernel, two layers on the residual: one
# token (an item's K-slices dealt to the groups) and eight; a dense layer in a stack is a layer like any other
@pytest.mark.parametrize("gate_ty,down_ty,n,kw", [
    (W.Q4_K, W.Q6_K, 1, dict(n_embd=1024, n_expert=16, k=4, ff=256, ff_sh=256)),
    (W.Q5_K, W.Q5_K, 8, dict(n_embd=512, n_expert=64, k=6, ff=256, ff_sh=256)),
    (W.Q8_0, W.Q8_0, 5, dict(n_embd=1024, n_expert=8, k=2, ff=256, ff_sh=0)),
    (W.Q6_K, W.Q4_K, 3, dict(n_embd=512, n_expert=1, k=1, ff=512, ff_sh=0))])
def test_a_few_tokens_through_a_stack_with_its_norm(gate_ty, down_ty, n, kw):
    import oracle
    import torch
    from helpers import rel_err
    from biv_b200 import capi
    from biv_b200.moe import Moe, MoeStack
    rng = np.random.default_rng(n)
    lays = [W.make_layer(rng, gate_ty=gate_ty, down_ty=down_ty, router_dist="uniform", **kw) for _ in range(2)]
    if kw["n_expert"] == 1:
        for l in lays:
            l.router[:] = 0
    e = kw["n_embd"]
    x0 = rng.standard_normal((n, e), dtype=np.float32)
    norm_w = [(1.0 + 0.1 * rng.standard_normal(e)).astype(np.float32) for _ in lays]
    ref = oracle.moe_stack(lays, norm_w, 1e-6, x0, level=oracle.host_level())
    layers = [Moe.dense(l.gate, l.up, l.down, n) if l.n_expert == 1 else Moe(l, n) for l in lays]
    try:
        for m, nw in zip(layers, norm_w):
            m.set_post_norm(nw, 1e-6)
        x = torch.from_numpy(x0).cuda()
        MoeStack(layers).forward_(x)
        torch.cuda.synchronize()
        assert rel_err(x.cpu().numpy(), ref) < 1e-3
        # the rows the first layer quantised are the normed ones
        h = oracle.rms_norm(oracle.host_level(), x0, norm_w[0], 1e-6)
        for tap, want in zip((capi.TAP_ACT_Q, capi.TAP_ACT_D, capi.TAP_ACT_S), oracle.q8_quantize(h)):
            assert np.array_equal(layers[0].tap(tap).reshape(-1), np.asarray(want).reshape(-1))
        layers[0].status()
    finally:
        for m in layers:
            m.close()
