"""q6k_panels_check.cpp as a library on the host."""
import ctypes as C
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
_lib = None


def lib():
    global _lib
    if _lib is None:
        with tempfile.TemporaryDirectory() as d:
            so = os.path.join(d, "libq6kpanels.so")
            subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", so, os.path.join(HERE, "q6k_panels_check.cpp")])
            _lib = C.CDLL(so)
    return _lib


def plan(pair, nrows, ncols, ntok):
    out = (C.c_uint32 * 5)()
    lib().plan(int(pair), nrows, ncols, ntok, out)
    return dict(zip(("MS", "KS", "groups", "panel", "smem"), out))
