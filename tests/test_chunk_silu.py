"""The convolution and SiLU of a chunk's rows (csrc/redcuda_silu.cuh, k_dn_prep_seq) against 64-bit extended sums: the function alone, compiled for the host, to the 2^-50
that it claims; and the kernel, with convolutions of two to four taps, a ragged last group of eight tokens, samples from the state, and arguments from the subnormal
to both sides of the +-80 where the C library's exp takes over."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def helper(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    rc.lib()
    so = str(tmp_path_factory.mktemp("silu") / "libsilu.so")
    product = rc.redcuda.LIB_PATH
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CUDA_INCLUDE, "-o", so, os.path.join(HERE, "silu_check.cpp"),
                           product, "-Wl,-rpath," + os.path.dirname(product)])
    L = C.CDLL(so)
    L.silu_of.argtypes, L.silu_of.restype = [C.c_void_p, C.c_void_p, C.c_long], None
    L.chunk.argtypes = [C.c_void_p, C.c_float, C.c_uint] + [C.c_void_p] * 15
    return L


def _silu(a):
    a = np.asarray(a, np.longdouble)
    with np.errstate(over="ignore"):
        return a / (1 + np.exp(-a))


def test_the_function_is_good_to_two_to_the_minus_50(helper):
    rng = np.random.default_rng(0)
    a = np.concatenate([rng.uniform(-81, 81, 400000), rng.normal(0, 3, 400000), rng.choice([-1, 1], 100000) * np.exp(rng.uniform(-700, 5, 100000)),
                        np.arange(-160, 161) * (np.log(2) / 2), [80.0, -80.0, np.nextafter(80, 0), -np.nextafter(80, 0), 0.0, 5e-324, 700.0, -700.0]])
    got = np.empty_like(a)
    helper.silu_of(a.ctypes.data, got.ctypes.data, a.size)
    want = _silu(a)
    assert np.all(np.abs(got - want) <= 2.0 ** -50 * np.abs(want) + 5e-324)
    for x, y in ((np.inf, np.inf), (np.nan, np.nan), (-800.0, 0.0)):
        helper.silu_of(np.array([x]).ctypes.data, got.ctypes.data, 1)
        assert got[0] == y or (np.isnan(y) and np.isnan(got[0]))


@pytest.mark.gpu
@pytest.mark.parametrize("d_conv", [2, 3, 4])
@pytest.mark.parametrize("S,groups,rank,T", [(32, 2, 4, 1), (64, 1, 2, 7), (128, 2, 4, 21), (256, 1, 2, 8)])
def test_the_kernel_rounds_the_double_sums(helper, S, groups, rank, T, d_conv):
    import torch
    rng = np.random.default_rng(S + T)
    d_inner, channels = rank * S, 2 * S * groups + rank * S
    spread = lambda *shape: (rng.normal(0, 1, shape) * np.exp(rng.uniform(-80, 4.5, shape))).astype(np.float32)  # noqa: E731
    kernel, state, qkv = rng.normal(0, 1, (channels, d_conv)).astype(np.float32), spread(channels, d_conv - 1), spread(T, channels)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()  # noqa: E731
    zeros = lambda *s: torch.zeros(*s, device="cuda")  # noqa: E731
    dims = np.array([d_conv, S, groups, rank, d_inner, channels], np.uint32)
    eps = np.float32(1e-6)
    bufs = [dev(kernel), zeros(rank), zeros(rank), torch.ones(S, device="cuda"), dev(qkv), zeros(T, d_inner), zeros(T, 2 * rank), dev(state), zeros(rank, S, S),
            zeros(T, 2 * groups * S), zeros(T, d_inner), zeros(T, rank), zeros(T, rank), zeros(T, d_inner), zeros(T, d_inner)]
    torch.cuda.synchronize()
    assert helper.chunk(dims.ctypes.data, eps, T, *[b.data_ptr() for b in bufs]) == 1, rc.lib().redcuda_last_error()
    torch.cuda.synchronize()
    qk, v = bufs[9].cpu().numpy(), bufs[10].cpu().numpy()
    rows = np.concatenate([state.T, qkv]).astype(np.longdouble)                    # time, channel
    terms = np.stack([rows[j:j + T] * kernel[:, j].astype(np.longdouble) for j in range(d_conv)])
    y = _silu(terms.sum(0))
    # half a unit of fp32 and the 2^-50; the sum itself is one of doubles, and near its root a SiLU follows it, elsewhere it changes by at most 1.1 times as much
    slack = 1.1 * 2.0 ** -51 * np.abs(terms).sum(0) + 2.0 ** -50 * np.abs(y)
    n_qk = 2 * groups * S
    unit = np.spacing(np.abs(y.astype(np.float32))).astype(np.longdouble)
    assert np.all(np.abs(v - y[:, n_qk:]) <= unit[:, n_qk:] / 2 + slack[:, n_qk:])
    y32 = y[:, :n_qk].astype(np.float32).astype(np.longdouble).reshape(T, 2 * groups, S)
    want = y32 / np.maximum(np.sqrt((y32 * y32).sum(2, keepdims=True)), np.longdouble(eps))
    # y itself may lie a unit off where the sum falls next to half a unit of it
    assert np.all(np.abs(qk.reshape(want.shape) - want) <= 2 * np.spacing(np.abs(want).astype(np.float32)) + slack[:, :n_qk].reshape(want.shape) / np.longdouble(eps) + 2.0 ** -149)
