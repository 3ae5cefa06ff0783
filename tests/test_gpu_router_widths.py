"""Router logits in every form of their kernel (8 tokens a block or 16, 8 experts or 16, a warp's whole share of a row at once or by steps),
over the row lengths that give a warp 2 to 16 steps of 16 columns, and one beyond: double sums in the same order, so the forms agree bit
for bit, and a logit is its exact sum rounded once."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden", list(range(256, 2049, 256)) + [2304])
def test_forms_agree(hidden):
    dims = synth.MoeDims(hidden=hidden, n_expert=40, top_k=2, ffn=256, ffn_sh=256)
    layer = synth.moe_layer(hidden, dims)
    x = np.random.default_rng(hidden).normal(0, 1, size=(1700, hidden)).astype(np.float32)      # 107 x 5 blocks of 16 x 8: the form of 16 x 16
    m = rc.MoeLayer(layer, max_tokens=1700)
    logits = {n: m.forward(x[:n], want_routing=True)[3] for n in (2, 8, 9, 33, 1700)}
    m.close()
    want = x.astype(np.float64) @ layer.router.astype(np.float64).T
    assert np.all(np.abs(logits[1700] - want) <= 2.0 ** -24 * np.abs(want) + 1e-12)
    for n, got in logits.items():
        assert np.array_equal(got, logits[1700][:n]), n
