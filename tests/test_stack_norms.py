"""Stacks in which a layer's combine leaves the rows normed for the next layer, or the norm is a launch of its
own: each against the same layers in stacks of one, where every norm is a launch (bit for bit), and the oracle.
What a norm would have written has to be written by this pass: the rows of an earlier one are NaN."""
import numpy as np
import pytest

from biv_b200 import workloads as W
from helpers import rel_err

pytestmark = pytest.mark.gpu


# Rows too wide for the router kernel that norms what it stages, by the kernels for up to eight rows, by those for
# more, and by the one that norms by itself (256 rows on; a row past 40 KB); the same from 17 rows on of narrower ones.
# More than 2048 columns are several turns of the combine's threads, more than eight experts two of its loop.
@pytest.mark.parametrize("gate_ty,down_ty,n,kw", [
    (W.Q8_0, W.Q8_0, 1, dict(n_embd=4096, n_expert=16, k=4, ff=256, ff_sh=256)),
    (W.Q8_0, W.Q8_0, 8, dict(n_embd=4096, n_expert=16, k=4, ff=256, ff_sh=0)),
    (W.Q4_K, W.Q6_K, 5, dict(n_embd=3328, n_expert=8, k=2, ff=256, ff_sh=256)),
    (W.Q4_0, W.Q4_1, 8, dict(n_embd=5888, n_expert=8, k=2, ff=256, ff_sh=256)),
    (W.Q8_0, W.Q8_0, 9, dict(n_embd=4096, n_expert=16, k=4, ff=256, ff_sh=256)),
    (W.Q8_0, W.Q8_0, 20, dict(n_embd=4096, n_expert=16, k=12, ff=256, ff_sh=256)),
    (W.Q4_K, W.Q4_K, 17, dict(n_embd=2304, n_expert=32, k=9, ff=256, ff_sh=0)),
    (W.Q4_0, W.Q4_0, 2, dict(n_embd=10240, n_expert=4, k=2, ff=256, ff_sh=256)),
    (W.Q4_0, W.Q4_0, 2, dict(n_embd=10496, n_expert=4, k=2, ff=256, ff_sh=256)),
    (W.BF16, W.BF16, 3, dict(n_embd=4096, n_expert=8, k=2, ff=256, ff_sh=256)),
    (W.Q4_0, W.Q4_0, 255, dict(n_embd=512, n_expert=16, k=4, ff=256, ff_sh=256)),
    (W.Q4_0, W.Q4_0, 256, dict(n_embd=512, n_expert=16, k=4, ff=256, ff_sh=256)),
])
@pytest.mark.parametrize("dense", [None, 1])   # a dense layer between the others
def test_every_layer_of_a_stack_gets_normed_rows(gate_ty, down_ty, n, kw, dense):
    import oracle
    import torch
    from biv_b200.moe import Moe, MoeStack
    rng = np.random.default_rng(n)
    e = kw["n_embd"]
    lays = [W.make_layer(rng, gate_ty=gate_ty, down_ty=down_ty, router_dist="uniform",
                         **(kw if l != dense else dict(n_embd=e, n_expert=1, k=1, ff=256, ff_sh=0))) for l in range(3)]
    if dense is not None:
        lays[dense].router[:] = 0
    norm_w = [(1.0 + 0.1 * rng.standard_normal(e)).astype(np.float32) for _ in lays]
    x0 = rng.standard_normal((n, e), dtype=np.float32)
    layers = [Moe.dense(l.gate, l.up, l.down, n) if i == dense else Moe(l, n) for i, l in enumerate(lays)]
    try:
        for m, nw in zip(layers, norm_w):
            m.set_post_norm(nw, 1e-6)

        def one_by_one(x):
            for m in layers:
                MoeStack([m]).forward_(x)
            torch.cuda.synchronize()
            return x

        start = torch.from_numpy(x0).cuda()
        want = one_by_one(start.clone())
        assert torch.isnan(one_by_one(torch.full_like(start, float("nan")))).all()
        x = start.clone()
        MoeStack(layers).forward_(x)
        torch.cuda.synchronize()
        assert torch.equal(x, want)
        # Every layer on the oracle's input to it: a re-quantised value of a SwiGLU row may move by a step, 3e-3 of an
        # expert's output, which the layers behind make more of (two such rows of eight were 3e-3 off, then 1.4e-2).
        ref = x0
        for m, lay, nw in zip(layers, lays, norm_w):
            y = MoeStack([m]).forward_(torch.from_numpy(ref).cuda())
            ref = oracle.moe_stack([lay], [nw], 1e-6, ref, level=oracle.host_level())
            assert rel_err(y.cpu().numpy(), ref) < 1e-2
        # as one graph from the second call on
        stack, st = MoeStack(layers), torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            for _ in range(3):
                one_by_one(x.fill_(float("nan")))
                x.copy_(start)
                stack.forward_(x)
                st.synchronize()
                assert torch.equal(x, want)
        for m in layers:
            m.status()
    finally:
        for m in layers:
            m.close()
