"""CPU check of the host-buffer staging: csrc/redcuda_stage.cu compiled for the host against a fake CUDA runtime (stage_host_check.cpp)."""
import ctypes as C
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def so_path(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    so = str(tmp_path_factory.mktemp("stage") / "libstage.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CUDA_INCLUDE, "-o", so, os.path.join(HERE, "stage_host_check.cpp"),
                           "-x", "c++", os.path.join(HERE, "..", "dwarfstar_red_lite_b200", "csrc", "redcuda_stage.cu"), "-lpthread"])
    return so


@pytest.fixture(scope="module")
def lib(so_path):
    L = C.CDLL(so_path)
    L.check_roundtrip.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t]
    L.check_download_cpu.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
    L.check_download_cpu.restype = C.c_double
    L.check_error.restype = C.c_char_p
    L.check_open_many.argtypes = [C.c_size_t, C.c_int]
    L.check_device_bytes.restype = L.check_pinned_bytes.restype = C.c_size_t
    return L


def _bytes(n, seed=0):
    return np.random.default_rng(seed).integers(0, 256, size=n, dtype=np.uint8), np.empty(n, np.uint8)


@pytest.mark.parametrize("n", [1, 4095, 256 << 10, (256 << 10) + 1, (512 << 10) + 16, (9 << 20) + 7, 32 << 20, (32 << 20) + 16, (70 << 20) + 5])
def test_roundtrip(lib, n):
    """below and above the single-copy limit, several pieces, several rounds of the 32 MB pinned buffer in both directions"""
    a, b = _bytes(n)
    assert lib.check_roundtrip(a.ctypes.data, b.ctypes.data, n) == 1, lib.check_error()


def test_roundtrip_from_several_threads(lib):
    bad = []

    def work(i):
        for k, n in enumerate((3 << 20, 70000, 20 << 20, 900001)):
            a, b = _bytes(n + i, seed=i * 4 + k)
            if lib.check_roundtrip(a.ctypes.data, b.ctypes.data, n + i) != 1:
                bad.append((i, n))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_helpers_sleep_while_the_gpu_works(lib):
    """a download whose bytes are 400 ms away: the copying threads must not spend that time spinning"""
    a, b = _bytes(8 << 20)
    assert lib.check_roundtrip(a.ctypes.data, b.ctypes.data, a.size) == 1         # the threads are started
    t = lib.check_download_cpu(a.ctypes.data, b.ctypes.data, a.size, 400)
    assert 0.0 <= t < 0.2, t                                                       # one thread that spins throughout takes 0.4


def test_idle_memory_is_bounded_and_given_back(lib):
    MB = 1 << 20
    assert lib.check_open_many(200 * MB, 4) == 1
    assert lib.check_device_bytes() <= 256 * MB
    pairs = [_bytes(33 * MB, seed=i) for i in range(4)]
    ts = [threading.Thread(target=lib.check_roundtrip, args=(a.ctypes.data, b.ctypes.data, a.size)) for a, b in pairs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert all(np.array_equal(a, b) for a, b in pairs)
    assert lib.check_device_bytes() <= 256 * MB and lib.check_pinned_bytes() <= 64 * MB
    assert lib.redcuda_trim() == 1
    assert lib.check_device_bytes() == 0 and lib.check_pinned_bytes() == 0
    calls = lib.check_set_device_calls()
    assert lib.redcuda_trim() == 1 and lib.check_set_device_calls() == calls          # nothing kept: no device is touched


def test_a_large_call_keeps_the_warm_areas(lib):
    """a call above the kept size allocates its device area each time, but neither a stream's pinned buffer nor another call's area"""
    MB = 1 << 20
    lib.redcuda_trim()
    small, large = _bytes(3 * MB), _bytes(300 * MB)
    run = lambda p: lib.check_roundtrip(p[0].ctypes.data, p[1].ctypes.data, p[0].size)  # noqa: E731
    assert run(small) == run(large) == run(small) == 1
    dev, pin = lib.check_device_allocs(), lib.check_pinned_allocs()
    assert run(large) == run(small) == run(large) == run(small) == 1
    assert lib.check_device_allocs() == dev + 2 and lib.check_pinned_allocs() == pin


@pytest.mark.parametrize("n", [100, 9 << 20])
def test_without_pinned_memory(lib, n):
    """a host without pinned memory left: the driver copies the pageable arrays itself"""
    a, b = _bytes(n)
    lib.redcuda_trim()
    lib.check_pinned_fails(1)
    try:
        assert lib.check_roundtrip(a.ctypes.data, b.ctypes.data, n) == 1, lib.check_error()
    finally:
        lib.check_pinned_fails(0)
    assert lib.check_roundtrip(a.ctypes.data, b.ctypes.data, n) == 1, lib.check_error()


_FAILING = """
import ctypes as C, sys
import numpy as np
L = C.CDLL(sys.argv[1])
L.check_roundtrip_failing.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
L.check_error.restype = C.c_char_p
a = np.arange(3 << 20, dtype=np.uint8)
b = np.empty_like(a)
seen = set()
for k in range(64):
    L.redcuda_trim()
    ok = L.check_roundtrip_failing(a.ctypes.data, b.ctypes.data, a.size, k)
    if ok == -1:
        break
    assert ok in (0, 1) and (ok == 1 or L.check_error()), k
    seen.add(ok)
    assert L.check_roundtrip_failing(a.ctypes.data, b.ctypes.data, a.size, 1 << 30) == -1
print("runs", k, "errors", 0 in seen)
assert k >= 3 and 0 in seen
"""


def test_a_failing_allocation_ends_a_call_with_an_error(so_path):
    """a process of its own: an exception that left a C entry point would end it"""
    r = subprocess.run([sys.executable, "-c", _FAILING, so_path], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
