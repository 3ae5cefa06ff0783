"""A row with a NaN or an infinity keeps it: the expert kernels work on digits, which cannot hold one, and must not turn such a row
into numbers. The other rows of the batch are untouched."""
import numpy as np
import pytest
import torch

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [synth.IQ3_S, synth.IQ2_XXS])
@pytest.mark.parametrize("ntok", [1, 2, 5, 40])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_nonfinite_row(t, ntok, bad):
    dims = synth.MoeDims(hidden=512, n_expert=16, top_k=4, ffn=256, ffn_sh=256, type_gu=t, type_down=t)
    m = rc.MoeLayer(synth.moe_layer(3, dims), max_tokens=ntok)
    rng = np.random.default_rng(ntok)
    x = rng.normal(0, 1, size=(ntok, dims.hidden)).astype(np.float32)
    logits = rng.normal(0, 1, size=(ntok, dims.n_expert)).astype(np.float32)
    ids = torch.from_numpy(rng.integers(0, dims.n_expert, size=ntok).astype(np.int32)).cuda()

    def pairs(rows):
        xd, o = torch.from_numpy(rows).cuda(), torch.zeros(ntok, dims.hidden, device="cuda")
        m.experts_device(ntok, xd.data_ptr(), ids.data_ptr(), o.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return o.cpu().numpy()

    for f in (pairs, lambda rows: m.forward(rows, logits_in=logits)):
        clean = f(x)
        for r in {0, ntok - 1}:
            y = x.copy()
            y[r, 37] = bad
            got = f(y)
            assert np.isfinite(clean).all() and not np.isfinite(got[r]).any()
            others = np.arange(ntok) != r
            assert np.array_equal(got[others], clean[others])
    m.close()
