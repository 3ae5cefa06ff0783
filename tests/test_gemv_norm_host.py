"""Which single-token GEMVs normalise their input on the way: a launch that cannot is refused, never run on the row as it is, and the rows
that one block writes while the others still read must lie apart from what they read."""
import ctypes as C
import os
import subprocess

import pytest

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import synth

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    rc.lib()
    so = str(tmp_path_factory.mktemp("norm") / "libnorm.so")
    product = rc.redcuda.LIB_PATH
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CUDA_INCLUDE, "-o", so, os.path.join(HERE, "gemv_norm_check.cpp"),
                           product, "-Wl,-rpath," + os.path.dirname(product)])
    L = C.CDLL(so)
    L.norm_ok.argtypes = [C.c_uint32, C.c_uint32] + [C.c_long] * 5
    L.refused.restype = C.c_char_p
    return L


def test_forms(lib):
    assert lib.norm_ok(synth.F32, 2048, 0, 2048, 4096, 6144, 8192) == 1
    assert lib.norm_ok(synth.Q6_K, 2048, 0, -1, 4096, -1, 8192) == 1
    assert lib.norm_ok(synth.Q6_K, 2304, 0, -1, 4096, -1, 8192) == 0          # longer than a block keeps
    assert lib.norm_ok(synth.IQ2_XXS, 2048, 0, -1, 4096, -1, 8192) == 0       # not a type of the single-token kernel
    assert lib.norm_ok(synth.F32, 2048, 1, 2048 + 4, 4096 + 4, -1, 8192) == 0  # unaligned


@pytest.mark.parametrize("at", [0, 4, 2044, 6144, 8188])
def test_written_rows_lie_apart(lib, at):
    """x, the branch and the weights at 0, 2048 and 4096, resid at 6144, normed at 8192: one of the written rows moved onto another"""
    assert lib.norm_ok(synth.F32, 2048, 0, 2048, 4096, 6144, at) == 0
    if at < 6144:
        assert lib.norm_ok(synth.F32, 2048, 0, 2048, 4096, at, 8192) == 0


@pytest.mark.parametrize("t,ntok", [(synth.IQ2_XXS, 1), (synth.Q6_K, 2)])
def test_other_launches_with_a_norm_are_refused(lib, t, ntok):
    assert b"normalised" in lib.refused(t, ntok)
