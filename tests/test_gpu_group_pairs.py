"""Grouping of more pairs than its threads keep in registers (2048 tokens x top-10 are the most), on both expert paths, and sampled rows
of the layer's output against the CPU oracle."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tc_min", ["0", "1"])
@pytest.mark.parametrize("ntok", [308, 2048, 2049, 2500])
def test_many_pairs(ntok, tc_min, monkeypatch):
    monkeypatch.setenv("RC_MOE_TC_MIN", tc_min)
    dims = synth.MoeDims(hidden=256, n_expert=48, top_k=10, ffn=256, ffn_sh=256)
    layer = synth.moe_layer(4, dims)
    rng = np.random.default_rng(ntok)
    x = rng.normal(0, 1, size=(ntok, dims.hidden)).astype(np.float32)
    logits = synth.zipf_routing_logits(3, ntok, dims.n_expert)
    m = rc.MoeLayer(layer, max_tokens=ntok)
    out = m.forward(x, logits_in=logits)
    m.close()
    for t in {0, 1, ntok // 3, 2047 % ntok, ntok - 2, ntok - 1}:
        ref = ol.moe_ffn(layer, x[t], threads=4, logits_in=logits[t])[0]
        # exact operands, activations of 22 bits (chunk kernel) or 24, fp32 sums of 256 products twice: a few 1e-6 of the range
        assert np.max(np.abs(out[t] - ref)) <= 2e-5 * np.max(np.abs(ref)), t
