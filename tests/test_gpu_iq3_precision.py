"""Error of IQ3_S experts (and of mixed IQ3_S / IQ2_XXS ones) against 64-bit sums, for rows whose elements differ widely: fixed-point
activations must be no worse than the fp32 rows that these layers are specified with. Relative 2-norm errors of an expert's output:
fp32 rows and sums 1.3e-7 to 2.1e-7 on every kind of row here, the digits with a scale per 256-column block 0.8e-7 to 1.2e-7; a
24-bit fixed point per row 3.1e-7 on Gaussian rows and up to 5e-4 on the others. The bound is 2e-7."""
import ctypes as C

import numpy as np
import pytest
import torch

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu
BOUND = 2e-7
TYPES = [(synth.IQ3_S, synth.IQ3_S), (synth.IQ3_S, synth.IQ2_XXS), (synth.IQ2_XXS, synth.IQ3_S)]


def _layer(tg, td, hidden, ffn, n_expert, zero_block):
    # top-1 routing: the weight is exactly 1, and with a zero shared expert the layer's output is the expert's
    dims = synth.MoeDims(hidden=hidden, n_expert=n_expert, top_k=1, ffn=ffn, ffn_sh=ffn, type_gu=tg, type_down=td)
    layer = synth.moe_layer(5, dims, expert_scale=20.0)
    layer.sh_down[:] = 0
    if zero_block:                     # the weights of the first 256 columns vanish
        for m in (layer.gate, layer.up):
            m.reshape(-1, hidden // 256, synth.BLOCK_BYTES[tg])[:, 0, 0:2] = 0
    return layer


def _rows(kind, ntok, hidden):
    rng = np.random.default_rng(ntok)
    x = rng.normal(0, 1, size=(ntok, hidden))
    if kind == "one of 1000":
        x[:, 300] = 1000.0
    elif kind == "large where the weights vanish":
        x[:, 17] = 1e4
    elif kind == "log-normal":
        x = np.exp(2 * rng.normal(0, 1, size=(ntok, hidden))) * np.sign(x)
    return x.astype(np.float32), rng


def _exact(layer, x, ids):
    d = layer.dims
    out = np.zeros((x.shape[0], d.hidden))
    for e in np.unique(ids):
        deq = lambda t, m, rows, cols: ol.dequant_rows(t, m[e].reshape(rows, -1), cols).astype(np.float64)  # noqa: E731
        s = ids == e
        xs = x[s].astype(np.float64)
        g, u = xs @ deq(d.type_gu, layer.gate, d.ffn, d.hidden).T, xs @ deq(d.type_gu, layer.up, d.ffn, d.hidden).T
        with np.errstate(over="ignore"):
            act = g / (1 + np.exp(-g)) * u
        out[s] = act @ deq(d.type_down, layer.down, d.hidden, d.ffn).T
    return out


def _rel(got, want):
    return np.linalg.norm(got - want) / np.linalg.norm(want)


@pytest.mark.parametrize("tg,td", TYPES)
@pytest.mark.parametrize("kind", ["gauss", "one of 1000", "large where the weights vanish", "log-normal"])
def test_error_against_64_bit(tg, td, kind):
    layer = _layer(tg, td, 2048, 512, 4, kind == "large where the weights vanish")
    for ntok in (1, 2, 7, 13, 40, 150):                 # one token; items of one to six pairs and their remainders
        x, rng = _rows(kind, ntok, 2048)
        ids = rng.integers(0, 4 if ntok != 13 else 1, size=ntok)
        logits = np.full((ntok, 4), -10.0, np.float32)
        logits[np.arange(ntok), ids] = 10.0
        m = rc.MoeLayer(layer, max_tokens=ntok)
        got = m.forward(x, logits_in=logits)
        m.close()
        assert _rel(got, _exact(layer, x, ids)) <= BOUND, ntok


def test_block_scales_of_every_kind():
    """negative, subnormal, zero and large fp16 block scales in turn"""
    layer = _layer(synth.IQ3_S, synth.IQ3_S, 512, 256, 4, False)
    scales = np.array([-0.01, 6e-8, 0.0, 0.5, 0.02, -3e-5], np.float16).view(np.uint8).reshape(-1, 2)
    for m in (layer.gate, layer.up, layer.down):
        b = m.reshape(-1, synth.BLOCK_BYTES[synth.IQ3_S])
        b[:, 0:2] = scales[np.arange(b.shape[0]) % len(scales)]
    x, rng = _rows("gauss", 9, 512)
    ids = rng.integers(0, 4, size=9)
    logits = np.full((9, 4), -10.0, np.float32)
    logits[np.arange(9), ids] = 10.0
    m = rc.MoeLayer(layer, max_tokens=9)
    got = m.forward(x, logits_in=logits)
    m.close()
    assert _rel(got, _exact(layer, x, ids)) <= BOUND


@pytest.mark.parametrize("hidden,ffn", [(256, 256), (512, 1024), (1024, 512)])
@pytest.mark.parametrize("ntok", [1, 5, 30])
def test_other_widths(hidden, ffn, ntok):
    layer = _layer(synth.IQ3_S, synth.IQ3_S, hidden, ffn, 4, False)
    x, rng = _rows("log-normal", ntok, hidden)
    ids = rng.integers(0, 4, size=ntok)
    logits = np.full((ntok, 4), -10.0, np.float32)
    logits[np.arange(ntok), ids] = 10.0
    m = rc.MoeLayer(layer, max_tokens=ntok)
    got = m.forward(x, logits_in=logits)
    m.close()
    assert _rel(got, _exact(layer, x, ids)) <= BOUND


def test_pieces_and_exchange():
    """experts_device, partial_device and the expert-parallel call of a single rank hand the rows over in different forms."""
    ntok = 21
    layer = _layer(synth.IQ3_S, synth.IQ3_S, 2048, 512, 4, True)
    x, rng = _rows("large where the weights vanish", ntok, 2048)
    ids = rng.integers(0, 4, size=ntok).astype(np.int32)
    want = _exact(layer, x, ids)
    m = rc.MoeLayer(layer, max_tokens=ntok)
    xd, idd, wd, out = torch.from_numpy(x).cuda(), torch.from_numpy(ids).cuda(), torch.ones(ntok, device="cuda"), torch.zeros(ntok, 2048, device="cuda")
    logits = torch.full((ntok, 4), -10.0, device="cuda")
    logits[torch.arange(ntok, device="cuda"), idd.long()] = 10.0
    torch.cuda.synchronize()
    s, lib = torch.cuda.Stream(), rc.lib()
    m.experts_device(ntok, xd.data_ptr(), idd.data_ptr(), out.data_ptr(), s.cuda_stream)
    s.synchronize()
    assert _rel(out.cpu().numpy(), want) <= BOUND
    m.partial_device(ntok, xd.data_ptr(), 2048, idd.data_ptr(), wd.data_ptr(), 1, out.data_ptr(), s.cuda_stream)
    s.synchronize()
    assert _rel(out.cpu().numpy(), want) <= BOUND
    ep = lib.redcuda_ep_create(0, 1, None, ntok, 2048, 1)
    assert ep, lib.redcuda_last_error()
    assert lib.redcuda_ep_layer_forward(C.c_void_p(ep), m.handle, xd.data_ptr(), logits.data_ptr(), out.data_ptr(), s.cuda_stream) == 1, lib.redcuda_last_error()
    s.synchronize()
    assert _rel(out.cpu().numpy(), want) <= BOUND
    lib.redcuda_ep_destroy(ep)
    m.close()
