"""The router product of many tokens, whose tiles a persistent block works off one after the other: bit for
bit the oracle's, with a last row by itself and without, ragged rows and tokens, one turn and several."""
import numpy as np
import pytest

from biv_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_expert,n,n_embd", [(256, 600, 256), (256, 1365, 512), (100, 1500, 256), (64, 2731, 256),
                                               (128, 2730, 256), (200, 3001, 256), (256, 4097, 256), (95, 6001, 256)])
def test_logits_are_the_oracles(n_expert, n, n_embd):
    import oracle
    import torch
    from biv_b200.moe import Moe
    rng = np.random.default_rng(n)
    layer = W.make_layer(rng, gate_ty=W.Q4_0, down_ty=W.Q4_0, n_embd=n_embd, n_expert=n_expert, k=2, ff=256, ff_sh=256)
    h = W.rms_normalise(rng.standard_normal((n, n_embd), dtype=np.float32))
    m = Moe(layer, n)
    try:
        m.moe(torch.from_numpy(h).cuda())
        logits, gate = m.tap(capi.TAP_LOGITS), m.tap(capi.TAP_SHARED_GATE)
        m.status()
    finally:
        m.close()
    assert logits.shape == (n, n_expert) and gate.shape == (n,)
    pick = np.unique(np.concatenate([np.arange(50), rng.integers(0, n, 100), np.arange(n - 50, n)]))
    rows = np.concatenate([layer.router, layer.sh_gate_inp[None]])
    want = np.array([[oracle.dot_f32(1, w, x) for w in rows] for x in h[pick]], np.float32)
    assert np.array_equal(logits[pick], want[:, :-1])
    assert np.array_equal(gate[pick], want[:, -1])
