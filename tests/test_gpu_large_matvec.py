"""One token through a Q6_K matrix of many rows (the LM head's kernel: x as four 8-bit digits per 256 columns, exact sums of 16 columns) against 64-bit sums:
every chunk count of a row, a last tile with few rows, rows of x whose elements differ widely, and one that is not finite. Each sum of 16 columns and each step of the fp32
sums over a row (64 of them, four to a lane and five shuffle steps) rounds by 2^-24, x itself by 2^-31 of its block's largest: relative 2-norm
errors of about 1e-7, where sums of products in fp32 have 1.5e-7 and more. The bound is 2e-7."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu
ROWS = 16384 + 37


@pytest.mark.parametrize("cols", [256, 512, 768, 1024, 1792, 2048])
@pytest.mark.parametrize("kind", ["gauss", "one of 1000", "log-normal", "1e-30"])
def test_error_against_64_bit(cols, kind):
    rng = np.random.default_rng(cols)
    w = synth.quant_matrix(rng, synth.Q6_K, ROWS, cols, 1e-3, 5e-3, (-64, 63))
    x = rng.normal(0, 1, size=cols)
    if kind == "one of 1000":
        x[cols // 2] = 1000.0
    elif kind == "log-normal":
        x = np.exp(2 * rng.normal(0, 1, size=cols)) * np.sign(x)
    elif kind == "1e-30":
        x *= 1e-30
    x = x.astype(np.float32)[None, :]
    got = np.asarray(rc.quant_matvec(synth.Q6_K, w, ROWS, cols, x)).reshape(-1)
    want = ol.dequant_rows(synth.Q6_K, np.asarray(w).reshape(ROWS, -1), cols).astype(np.float64) @ x[0].astype(np.float64)
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 2e-7


def test_a_row_that_is_not_finite():
    rng = np.random.default_rng(1)
    w = synth.quant_matrix(rng, synth.Q6_K, ROWS, 512, 1e-3, 5e-3, (-64, 63))
    for bad in (np.nan, np.inf):
        x = rng.normal(0, 1, size=(1, 512)).astype(np.float32)
        x[0, 300] = bad
        assert not np.isfinite(np.asarray(rc.quant_matvec(synth.Q6_K, w, ROWS, 512, x))).any()


@pytest.mark.parametrize("kind", ["1e-25", "1e-33", "1e-35", "1e4 where the weights vanish", "1e6 where the weights vanish", "one of 256", "1e-37 beside ones"])
@pytest.mark.parametrize("cols", [256, 768, 2048])
def test_rows_that_digits_do_not_hold(cols, kind):
    """Blocks of 256 values with one that stands out, with few that count, or near the least exponents: as right as the products of floats."""
    rng = np.random.default_rng(cols + 1)
    w = np.asarray(synth.quant_matrix(rng, synth.Q6_K, ROWS, cols, 1e-3, 5e-3, (-64, 63))).copy()
    x = rng.normal(0, 1, size=cols)
    if "vanish" in kind:
        w.reshape(ROWS, cols // 256, 210)[:, -1, 192] = 0            # the 8-bit scale of the last block's first 16 columns
        x[cols - 250] = float(kind[:3])
    elif kind == "one of 256":
        x[np.arange(cols) % 256 != 77] = 0.0
    elif "beside" in kind:
        x[-256:] *= 1e-37
        w.reshape(ROWS, cols // 256, 210)[:, :-1, 208:] = 0          # the other blocks' d: what the small block gives is all there is
    else:
        x *= float(kind)
    x = x.astype(np.float32)[None, :]
    got = np.asarray(rc.quant_matvec(synth.Q6_K, w, ROWS, cols, x)).reshape(-1)
    want = ol.dequant_rows(synth.Q6_K, w.reshape(ROWS, -1), cols).astype(np.float64) @ x[0].astype(np.float64)
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 2e-7 + 2.0 ** -150 * ROWS ** 0.5 / np.linalg.norm(want)      # the last: rounding to a subnormal


def test_an_infinity_keeps_its_sign():
    rng = np.random.default_rng(1)
    w = synth.quant_matrix(rng, synth.Q6_K, ROWS, 512, 1e-3, 5e-3, (-64, 63))
    x = rng.normal(0, 1, size=(1, 512)).astype(np.float32)
    x[0, 300] = np.inf
    with np.errstate(invalid="ignore"):
        want = (ol.dequant_rows(synth.Q6_K, np.asarray(w).reshape(ROWS, -1), 512)[:, 300] * np.float32(np.inf))
    assert np.array_equal(np.asarray(rc.quant_matvec(synth.Q6_K, w, ROWS, 512, x)).reshape(-1), want, equal_nan=True)
