"""Passes of k-quant layers whose groups have some tens of rows: the tcgen05 kernels on f16 records,
against the oracle, at the edges of their tiles and of the widths at which a tile's tokens are dealt out."""
import numpy as np
import pytest

from biv_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gate_ty,down_ty,n", [
    (W.Q4_K, W.Q6_K, 9), (W.Q5_K, W.Q4_K, 16), (W.Q6_K, W.Q5_K, 17), (W.Q4_K, W.Q4_K, 32), (W.Q5_K, W.Q6_K, 33),
    (W.Q6_K, W.Q6_K, 64), (W.Q4_K, W.Q5_K, 65), (W.Q5_K, W.Q5_K, 145)])
def test_a_group_of_every_width(gate_ty, down_ty, n, monkeypatch):
    from biv_b200.moe import Moe
    from test_gpu_parity import run_case
    monkeypatch.setenv("BIVMOE_WIDE_MIN", "1")
    rng = np.random.default_rng(n)
    layer = W.make_layer(rng, gate_ty=gate_ty, down_ty=down_ty, n_embd=512, n_expert=1, k=1, ff=256, ff_sh=0)
    layer.router[:] = 0
    h = W.rms_normalise(rng.standard_normal((n, 512), dtype=np.float32))
    run_case(W.Workload("dense", n, [layer], h), make=lambda l, cap: Moe.dense(l.gate, l.up, l.down, cap))


# Dense layers by the rule, from 128 rows on, whose down product is cut along K: nine slices in two parts, of
# four and five; sixteen in four
@pytest.mark.parametrize("ty,n,n_embd,ff", [(W.Q4_K, 128, 1280, 2304), (W.Q5_K, 145, 1280, 2304), (W.Q6_K, 200, 1280, 2304),
                                            (W.Q4_K, 129, 256, 4096)])
def test_down_product_in_parts_along_k(ty, n, n_embd, ff):
    from test_gpu_parity import check_dense_products
    check_dense_products(ty, n, n_embd, ff)


# rows laid out by position and (from 256 tokens on) by token first; empty and ragged groups; without a
# shared expert; a shared expert of other widths than the routed ones
@pytest.mark.parametrize("gate_ty,down_ty,n,kw", [
    (W.Q4_K, W.Q6_K, 70, dict(n_embd=512, n_expert=16, k=4, ff=256, ff_sh=256)),
    (W.Q5_K, W.Q6_K, 300, dict(n_embd=1024, n_expert=16, k=2, ff=512, ff_sh=0)),
    (W.Q6_K, W.Q4_K, 257, dict(n_embd=256, n_expert=64, k=6, ff=256, ff_sh=512))])
def test_groups_of_a_layer(gate_ty, down_ty, n, kw, monkeypatch):
    from test_gpu_parity import run_case
    monkeypatch.setenv("BIVMOE_WIDE_MIN", "1")
    rng = np.random.default_rng(n)
    layer = W.make_layer(rng, gate_ty=gate_ty, down_ty=down_ty, router_dist="uniform", **kw)
    h = W.rms_normalise(rng.standard_normal((n, layer.n_embd), dtype=np.float32))
    run_case(W.Workload("wide", n, [layer], h))


def test_a_row_with_a_nan_costs_its_own_output():
    import torch
    from biv_b200.moe import Moe
    rng = np.random.default_rng(1)
    layer = W.make_layer(rng, gate_ty=W.Q4_K, down_ty=W.Q6_K, n_embd=512, n_expert=4, k=2, ff=256, ff_sh=256)
    h = torch.from_numpy(W.rms_normalise(rng.standard_normal((200, 512), dtype=np.float32))).cuda()
    m = Moe(layer, 200)          # 100 rows a group: by the rule
    try:
        want = m.moe(h)
        h[11, 5], h[190, 400] = float("nan"), float("-inf")
        got = m.moe(h)
        assert torch.isnan(got[[11, 190]]).all()
        keep = [t for t in range(200) if t not in (11, 190)]
        # (their pairs leave the groups they were in or enter others, which moves no other row's result)
        assert torch.equal(got[keep], want[keep])
    finally:
        m.close()
