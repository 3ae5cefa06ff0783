"""CPU check of csrc/redcuda_q6k_panels.cuh: the steps in which a block of the Q6_K batch kernel stages its panels, against a model of the
staging barrier, and the rule that cuts a launch up."""
import pytest

import q6k_panels_lib as qp


@pytest.fixture(scope="module")
def lib():
    return qp.lib()


CUTS = [(1, 1), (8, 8), (8, 4), (17, 8), (20, 8), (9, 4), (16, 1)]


@pytest.mark.parametrize("row,panel", CUTS)
def test_every_panel_once(lib, row, panel):
    assert lib.check_panels(row, panel, -1, 0, 0) == 0


@pytest.mark.parametrize("waits_late", [1, 2])
@pytest.mark.parametrize("row,panel", CUTS)
def test_a_late_panel_is_the_last(lib, row, panel, waits_late):
    for late in range((row + panel - 1) // panel):
        assert lib.check_panels(row, panel, late, waits_late, 0) == 0


def test_the_model_sees_a_barrier_armed_again(lib):
    assert lib.check_panels(20, 8, 0, 1, 1) & 3 == 3          # armed again, and sent for over copies in flight
    assert lib.check_panels(17, 8, 1, 1, 1) != 0


@pytest.mark.parametrize("pair", [0, 1])
def test_plan(pair):
    for ncols in range(256, 16385, 256):
        for nrows in (16, 256, 512, 2048, 8192):
            for ntok in (3, 7, 8, 9, 33, 64, 75, 127, 512):
                p = qp.plan(pair, nrows, ncols, ntok)
                runs = 2 * ncols // 256                          # runs of 128 columns
                assert 8 % (p["MS"] * p["KS"]) == 0 and runs % p["KS"] == 0
                assert 256 <= p["panel"] <= min(ncols, 4096) and p["panel"] % 256 == 0 and p["smem"] <= 216 * 1024
                assert p["groups"] * 8 >= min(ntok, 8 * (8 // (p["MS"] * p["KS"])))
