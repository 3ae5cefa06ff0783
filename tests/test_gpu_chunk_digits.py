"""Activation digits of the dense chunk GEMM: rows that its threads keep in registers and longer ones, ragged last steps and token groups."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncols", [256, 512, 768, 2048, 2304, 4096])
@pytest.mark.parametrize("ntok", [1, 31, 130])
def test_row_lengths(ncols, ntok):
    rng = np.random.default_rng(ncols + ntok)
    nrows = 96
    rows = synth.quant_matrix(rng, synth.Q6_K, nrows, ncols, 1e-3, 5e-3)
    x = (rng.normal(0, 1, size=(ntok, ncols)) * np.exp(rng.uniform(-6, 6, size=(ntok, 1)))).astype(np.float32)
    got = rc.quant_matmul_tc(synth.Q6_K, rows, nrows, ncols, x).astype(np.float64)
    deq = ol.dequant_rows(synth.Q6_K, rows, ncols).astype(np.float64)
    ref, mag = x.astype(np.float64) @ deq.T, np.abs(x).astype(np.float64) @ np.abs(deq).T
    # a digit of x or w lost would show as 2^-11 of a term; two digits leave 2^-22 each and sums of 256 products in fp32
    assert np.max(np.abs(got - ref) / mag) <= 3e-6
