"""Host-buffer calls at the sizes where their staging changes form: below and above the single-copy limit (256 KB), several
512 KB pieces with a remainder, more than one round of the 32 MB pinned buffer, matvec batches around the token group of
four, and calls of several threads at once. Values are compared with the CPU oracle (dequantisation bit for bit)."""
import threading

import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


def _rows(seed, t, nrows, ncols):
    return synth.quant_matrix(np.random.default_rng(seed), t, nrows, ncols, 1e-3, 5e-3)


@pytest.mark.parametrize("t", [synth.Q8_0, synth.IQ3_S])
@pytest.mark.parametrize("nrows,ncols", [(1, 256), (32, 2048), (33, 2048), (300, 4096), (2600, 4096)])
def test_dequant_staging_sizes(t, nrows, ncols):
    rows = _rows(nrows + t, t, nrows, ncols)
    got = rc.quant_dequant_rows(t, rows, ncols)
    assert np.array_equal(got.view(np.uint32), ol.dequant_rows(t, rows, ncols).view(np.uint32))


@pytest.mark.parametrize("nrows,ntok", [(8, 4), (1821, 5), (5000, 1)])
def test_matvec_token_groups(nrows, ntok):
    ncols = 2048
    rows = _rows(nrows, synth.Q4_K, nrows, ncols)
    x = np.random.default_rng(ntok).normal(0, 1, size=(ntok, ncols)).astype(np.float32)
    got = rc.quant_matvec(synth.Q4_K, rows, nrows, ncols, x)
    deq = ol.dequant_rows(synth.Q4_K, rows, ncols).astype(np.float64)
    # fp32 sums of 2048 products: 64 sequential adds per lane and a tree of 32, 2^-24 each of sum |w x|
    assert np.all(np.abs(got - x.astype(np.float64) @ deq.T) <= 72 * 2.0 ** -24 * (np.abs(x.astype(np.float64)) @ np.abs(deq).T))


def test_host_calls_from_several_threads():
    shapes = [(64, 256), (700, 2048), (2600, 2048), (5, 4096)]
    rows = [_rows(i, synth.Q6_K, *s) for i, s in enumerate(shapes)]
    want = [ol.dequant_rows(synth.Q6_K, r, s[1]) for r, s in zip(rows, shapes)]
    bad = []

    def work(i):
        for _ in range(5):
            if not np.array_equal(rc.quant_dequant_rows(synth.Q6_K, rows[i], shapes[i][1]), want[i]):
                bad.append(i)

    rc.set_codebooks()
    ts = [threading.Thread(target=work, args=(i % 4,)) for i in range(6)]
    for th in ts:
        th.start()
    for th in ts:
        th.join()
    assert not bad
