"""Stage calls right after a table setter decode with the tables just set (the setters' copies are complete when they return; the
window that a missing wait leaves is microseconds, so the calls are repeated)."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import redcuda, synth

pytestmark = pytest.mark.gpu


def _alternate(set_a, set_b, t):
    rows = synth.quant_matrix(np.random.default_rng(t), t, 8, 2048, 1e-3, 5e-3)
    try:
        want = []
        for s in (set_a, set_b):
            s()
            for _ in range(3):
                got = rc.quant_dequant_rows(t, rows, 2048)
            want.append(got)
        assert not np.array_equal(*want)
        for i in range(60):
            (set_a, set_b)[i & 1]()
            assert np.array_equal(rc.quant_dequant_rows(t, rows, 2048), want[i & 1]), i
    finally:
        rc.set_codebooks()


def test_base_tables():
    g2, g3 = redcuda.default_codebooks()
    _alternate(lambda: rc.set_codebooks(g2, g3), lambda: rc.set_codebooks(g2, np.roll(g3, 7)), synth.IQ3_S)


def test_ext_tables():
    a, b, c = redcuda.default_codebooks_ext()
    _alternate(lambda: redcuda.set_codebooks_ext(a, b, c), lambda: redcuda.set_codebooks_ext(a, b, c[::-1].copy()), synth.IQ4_XS)


def test_xs_tables():
    raw = np.fromfile(redcuda.HERE + "/data/codebooks_iq2xs_iq1m.bin", dtype=np.int8)
    a, b = raw[:4096].copy(), raw[4096:20480].copy()
    _alternate(lambda: redcuda.set_codebooks_xs(a, b), lambda: redcuda.set_codebooks_xs(a, np.roll(b, 8)), synth.IQ1_M)
