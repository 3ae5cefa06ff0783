"""Small-batch router logits at the sizes where their tiles have remainders (tokens, experts)."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntok", [2, 7, 8, 9, 16, 33, 64, 65, 150])
@pytest.mark.parametrize("hidden,n_expert", [(256, 13), (512, 200), (768, 520)])
def test_router_logits_batches(ntok, hidden, n_expert):
    dims = synth.MoeDims(hidden=hidden, n_expert=n_expert, top_k=4, ffn=256, ffn_sh=256)
    layer = synth.moe_layer(ntok, dims)
    x = np.random.default_rng(ntok).normal(0, 1, size=(ntok, hidden)).astype(np.float32)
    m = rc.MoeLayer(layer, max_tokens=ntok)
    _, ids, w, logits = m.forward(x, want_routing=True)
    m.close()
    want = x.astype(np.float64) @ layer.router.astype(np.float64).T
    # summed in double, rounded once
    assert np.all(np.abs(logits - want) <= 2.0 ** -24 * np.abs(want) + 1e-12)
    order = np.argsort(-logits.astype(np.float64), axis=1, kind="stable")[:, :4]
    assert np.array_equal(ids, order)
