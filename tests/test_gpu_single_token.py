"""The single-token matrix-vector kernel at the sizes where its tiling changes form: rows shorter than a warp's slice, ragged
slices, slice counts that do and do not divide the block's warps, a last tile of one row."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,ncols", [(synth.Q6_K, 256), (synth.Q6_K, 768), (synth.Q6_K, 1024), (synth.Q6_K, 2048), (synth.Q6_K, 2304), (synth.Q6_K, 4096), (synth.Q6_K, 6400),
                                     (synth.F16, 64), (synth.F16, 1088), (synth.F16, 4096), (synth.F32, 64), (synth.F32, 960), (synth.F32, 2048), (synth.F32, 3136)])
@pytest.mark.parametrize("nrows", [1, 9, 600, 5001])
def test_single_token_matvec(t, ncols, nrows):
    rng = np.random.default_rng(nrows + ncols)
    if t == synth.Q6_K:
        w = synth.quant_matrix(rng, t, nrows, ncols, 1e-3, 5e-3, (-64, 63))
        deq = ol.dequant_rows(t, w, ncols).astype(np.float64)
    else:
        w = rng.uniform(-1, 1, size=(nrows, ncols)).astype(np.float16 if t == synth.F16 else np.float32)
        deq = w.astype(np.float64)
    x = rng.normal(0, 1, size=(1, ncols)).astype(np.float32)
    got = rc.quant_matvec(t, w, nrows, ncols, x)[0]
    want, mass = deq @ x[0].astype(np.float64), np.abs(deq) @ np.abs(x[0]).astype(np.float64)
    # a weight is within 2 roundings of its exact product with the scales; per run of 16: 8 packed adds, then 2 + 4 adds, a
    # tree of 5 and the final rounding: at most 24 roundings of 2^-24 of sum |w x|; plain rows are summed in double
    assert np.all(np.abs(got - want) <= (24 if t == synth.Q6_K else 1.01) * 2.0 ** -24 * mass)
