"""The tcgen05 expert kernel: items at the edges of its 16-column accumulator steps and of its 48 pairs, rows of one to eight blocks, few and many
groups of tiles; and its error against 64-bit sums on rows whose elements differ widely, which must not exceed that of the integer kernels
(3.0e-7 to 3.2e-7 on Gaussian rows, up to 2.7e-6 on the others). Measured 2.8e-7 to 3.8e-7: two fp16 digits are good to 2^-23 of a value,
an accumulator of 64 columns truncates at most eight sums of its size (2^-24 each on average), and 32 such sums are added in fp32."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu
BOUND = 4.5e-7


def _layer(hidden, ffn, n_expert):
    # top-1 routing: the weight is exactly 1, and with a zero shared expert the layer's output is the expert's
    dims = synth.MoeDims(hidden=hidden, n_expert=n_expert, top_k=1, ffn=ffn, ffn_sh=ffn)
    layer = synth.moe_layer(5, dims, expert_scale=20.0)
    layer.sh_down[:] = 0
    return layer


def _run(layer, x, ids, monkeypatch):
    monkeypatch.setenv("RC_MOE_TC_MIN", "1")
    logits = np.full((len(ids), layer.dims.n_expert), -10.0, np.float32)
    logits[np.arange(len(ids)), ids] = 10.0
    m = rc.MoeLayer(layer, max_tokens=len(ids))
    rc.redcuda.profile_enable(True)
    got = m.forward(x, logits_in=logits)
    kernels = rc.redcuda.profile_report()
    rc.redcuda.profile_enable(False)
    m.close()
    assert "moe_gateup_tc" in kernels and "moe_down_tc" in kernels
    return got


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


@pytest.mark.parametrize("hidden,ffn", [(256, 256), (512, 2048), (1024, 256), (2048, 512)])
def test_items_of_every_size(hidden, ffn, monkeypatch):
    counts = [1, 15, 16, 17, 47, 48, 49, 97, 0, 33]
    layer = _layer(hidden, ffn, len(counts))
    ids = np.random.default_rng(3).permutation(np.repeat(np.arange(len(counts)), counts))
    x = np.random.default_rng(4).normal(0, 1, size=(len(ids), hidden)).astype(np.float32)
    got, want = _run(layer, x, ids, monkeypatch), _exact(layer, x, ids)
    for e, c in enumerate(counts):
        if c:
            assert _rel(got[ids == e], want[ids == e]) <= 2 * BOUND, (e, c)       # a single row varies by more than the mean of many


@pytest.mark.parametrize("kind", ["gauss", "one of 1000", "log-normal"])
@pytest.mark.parametrize("hidden,ffn", [(1024, 512), (2048, 512), (2048, 1024)])
def test_error_against_64_bit(kind, hidden, ffn, monkeypatch):
    layer = _layer(hidden, ffn, 4)
    rng = np.random.default_rng(300)
    x = rng.normal(0, 1, size=(300, hidden))
    if kind == "one of 1000":
        x[:, 300] = 1000.0
    elif kind == "log-normal":
        x = np.exp(2 * rng.normal(0, 1, size=x.shape)) * np.sign(x)
    x, ids = x.astype(np.float32), rng.integers(0, 4, size=300)
    assert _rel(_run(layer, x, ids, monkeypatch), _exact(layer, x, ids)) <= BOUND
