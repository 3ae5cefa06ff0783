"""A layer whose experts are wider than its hidden size on the tcgen05 expert kernel: the up rows of a chunk wait in a workspace buffer that has to
hold the wider of the two. Bound: 22-bit digits and truncating accumulators stay below 1e-6 of an expert's output."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


def test_ffn_wider_than_hidden(monkeypatch):
    monkeypatch.setenv("RC_MOE_TC_MIN", "1")
    dims = synth.MoeDims(hidden=512, n_expert=4, top_k=1, ffn=2048, ffn_sh=256)
    layer = synth.moe_layer(5, dims, expert_scale=20.0)
    layer.sh_down[:] = 0
    rng = np.random.default_rng(6)
    x, ids = rng.normal(0, 1, size=(200, 512)).astype(np.float32), rng.integers(0, 4, size=200)
    logits = np.full((200, 4), -10.0, np.float32)
    logits[np.arange(200), ids] = 10.0
    m = rc.MoeLayer(layer, max_tokens=200)
    got = m.forward(x, logits_in=logits)
    m.close()
    for e in range(4):
        deq = lambda t, w, rows, cols: ol.dequant_rows(t, w[e].reshape(rows, -1), cols).astype(np.float64)  # noqa: E731
        xs = x[ids == e].astype(np.float64)
        g, u = xs @ deq(dims.type_gu, layer.gate, 2048, 512).T, xs @ deq(dims.type_gu, layer.up, 2048, 512).T
        want = (g / (1 + np.exp(-g)) * u) @ deq(dims.type_down, layer.down, 512, 2048).T
        assert np.linalg.norm(got[ids == e] - want) / np.linalg.norm(want) <= 2e-6, e
