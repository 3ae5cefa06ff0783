"""IQ3_S (and mixed IQ3_S / IQ2_XXS) experts in the 4-bit layout of the expert kernels, against the CPU oracle: one token,
pair counts around the limits of a work item, a batch, and batches that IQ2_XXS layers would hand to the tcgen05 chunk kernel
(layers with IQ3_S matrices stay on the integer kernels). Bounds: the operands are exact integers, activations are 32-bit fixed
point per 256-column block and everything else is fp32, so a layer output is good to a few 1e-6 of its range; 2e-5 leaves room
for the order of the sums."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


def _check(dims, ntok, seed, one_expert_for_all=False):
    layer = synth.moe_layer(seed, dims)
    x = np.random.default_rng(seed + 1).normal(0, 1, size=(ntok, dims.hidden)).astype(np.float32)
    logits = None
    if one_expert_for_all:                     # every token picks the same experts: work items as full as they get
        logits = np.tile(np.random.default_rng(seed + 2).normal(0, 1, size=(1, dims.n_expert)), (ntok, 1)).astype(np.float32)
    m = rc.MoeLayer(layer, max_tokens=ntok)
    out = m.forward(x, logits_in=logits)
    m.close()
    for t in range(0, ntok, max(1, ntok // 6)):
        ref = ol.moe_ffn(layer, x[t], threads=4, logits_in=None if logits is None else logits[t])[0]
        assert np.max(np.abs(out[t] - ref)) <= 2e-5 * np.max(np.abs(ref)), t


@pytest.mark.parametrize("tg,td", [(synth.IQ3_S, synth.IQ3_S), (synth.IQ3_S, synth.IQ2_XXS), (synth.IQ2_XXS, synth.IQ3_S)])
@pytest.mark.parametrize("ntok", [1, 2, 3, 8, 9, 33])
def test_expert_formats(tg, td, ntok):
    dims = synth.MoeDims(hidden=512, n_expert=16, top_k=4, ffn=256, ffn_sh=256, type_gu=tg, type_down=td)
    _check(dims, ntok, 300 + ntok)
    _check(dims, ntok, 400 + ntok, one_expert_for_all=True)


@pytest.mark.parametrize("hidden,ffn", [(2048, 512), (1024, 1024)])
def test_single_token_full_width(hidden, ffn):
    _check(synth.MoeDims(hidden=hidden, n_expert=24, top_k=10, ffn=ffn, ffn_sh=512, type_gu=synth.IQ3_S, type_down=synth.IQ3_S), 1, 7)


@pytest.mark.parametrize("ntok", [5, 64, 150])
def test_chunk_kernel(ntok, monkeypatch):
    monkeypatch.setenv("RC_MOE_TC_MIN", "1")
    dims = synth.MoeDims(hidden=512, n_expert=8, top_k=4, ffn=256, ffn_sh=256, type_gu=synth.IQ3_S, type_down=synth.IQ3_S)
    _check(dims, ntok, 500 + ntok)
    _check(dims, ntok, 600 + ntok, one_expert_for_all=True)
