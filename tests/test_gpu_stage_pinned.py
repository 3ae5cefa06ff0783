"""Host-buffer calls on arrays that are not ordinary host memory: pinned ones that copies of the default stream are still
filling or still reading, device memory, and more rows than the pinned buffer of a call holds."""
import numpy as np
import pytest
import torch

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu
NROWS, NCOLS = 64, 2048


def _matvec(w, x_ptr, out_ptr, ntok=1):
    lib = rc.lib()
    assert lib.redcuda_quant_matvec(synth.Q6_K, w.ctypes.data, NROWS, NCOLS, x_ptr, ntok, out_ptr) == 1, lib.redcuda_last_error()


@pytest.fixture(scope="module")
def case():
    rng = np.random.default_rng(2)
    w = synth.quant_matrix(rng, synth.Q6_K, NROWS, NCOLS, 1e-3, 5e-3, (-64, 63))
    x = rng.normal(0, 1, size=(1, NCOLS)).astype(np.float32)
    # 256 MB in front of the copy that matters: milliseconds of work for the default stream
    return w, x, rc.quant_matvec(synth.Q6_K, w, NROWS, NCOLS, x), torch.zeros(1 << 26, device="cuda"), torch.zeros(1 << 26).pin_memory()


def test_input_still_being_filled(case):
    w, x, want, big_dev, big_host = case
    src, pinned, out = torch.from_numpy(x).cuda(), torch.zeros(1, NCOLS).pin_memory(), np.empty((1, NROWS), np.float32)
    torch.cuda.synchronize()
    big_host.copy_(big_dev, non_blocking=True)
    pinned.copy_(src, non_blocking=True)
    _matvec(w, pinned.data_ptr(), out.ctypes.data)
    assert np.array_equal(out, want)


def test_output_still_being_read(case):
    w, x, want, big_dev, big_host = case
    pinned, dst = torch.full((1, NROWS), 7.0).pin_memory(), torch.zeros(1, NROWS, device="cuda")
    torch.cuda.synchronize()
    big_dev.copy_(big_host, non_blocking=True)
    dst.copy_(pinned, non_blocking=True)
    _matvec(w, x.ctypes.data, pinned.data_ptr())
    assert np.array_equal(pinned.numpy(), want)
    torch.cuda.synchronize()
    assert torch.all(dst == 7.0)


def test_device_arrays(case):
    w, x, want, _, _ = case
    wd, xd, out = torch.from_numpy(w).cuda(), torch.from_numpy(x).cuda(), torch.zeros(1, NROWS, device="cuda")
    lib = rc.lib()
    assert lib.redcuda_quant_matvec(synth.Q6_K, wd.data_ptr(), NROWS, NCOLS, xd.data_ptr(), 1, out.data_ptr()) == 1, lib.redcuda_last_error()
    assert np.array_equal(out.cpu().numpy(), want)


def test_upload_of_several_rounds():
    nrows, ncols = 9001, 4096                       # 39 MB of Q8_0 rows; the pinned buffer holds 32
    rng = np.random.default_rng(5)
    w = synth.quant_matrix(rng, synth.Q8_0, nrows, ncols, 1e-3, 5e-3)
    x = rng.normal(0, 1, size=(1, ncols)).astype(np.float32)
    got = rc.quant_matvec(synth.Q8_0, w, nrows, ncols, x)[0]
    for r in (0, 1, 4000, 7700, 7711, nrows - 1):   # 32 MB end in row 7710
        one = rc.quant_matvec(synth.Q8_0, w[r:r + 1], 1, ncols, x)[0, 0]
        assert got[r] == one
