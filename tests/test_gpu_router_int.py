"""Router logits of a chunk by integer products: the rounded double-precision sums, within what 40-bit fixed point per row leaves, and in double where that is
not enough. With X, W the largest magnitudes of a row of x and of the router, an element is off by at most 2^-38 of its row's largest, and the products of the lowest digits that are left out
come to less than 2^-42 X W a column; the sum of these is the bound on a logit before it is rounded. Where they lie far below half a unit of fp32
the logits are the rounded sums but for the few that lie that close to half a unit: fewer than one in a hundred here."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


def _logits(layer, x, monkeypatch):
    monkeypatch.setenv("RC_ROUTER_I8_MIN", "1")
    m = rc.MoeLayer(layer, max_tokens=len(x))
    rc.redcuda.profile_enable(True)
    logits = np.array(m.forward(x, want_routing=True)[3])
    assert "moe_router_digits" in rc.redcuda.profile_report()
    rc.redcuda.profile_enable(False)
    m.close()
    return logits


@pytest.mark.parametrize("kind", ["gauss", "one of 1000", "log-normal", "1e-36", "subnormal", "1e30"])
@pytest.mark.parametrize("hidden,n_expert,ntok", [(256, 128, 2), (512, 256, 31), (2048, 128, 33), (1024, 128, 65), (2048, 512, 1200)])
def test_logits_are_the_rounded_sums(kind, hidden, n_expert, ntok, monkeypatch):
    layer = synth.moe_layer(9, synth.MoeDims(hidden=hidden, n_expert=n_expert, top_k=2, ffn=256, ffn_sh=256))
    x = np.random.default_rng(ntok).normal(0, 1, size=(ntok, hidden))
    if kind == "one of 1000":
        x[:, 17] = 1000.0
    elif kind == "log-normal":
        x = np.exp(2 * np.random.default_rng(1).normal(0, 1, size=x.shape)) * np.sign(x)
    elif kind != "gauss":
        x *= 1e-41 if kind == "subnormal" else float(kind)
    x[0, :] = 0.0                                    # a row of zeros among the others
    x = x.astype(np.float32)
    want = (x.astype(np.float64) @ layer.router.reshape(n_expert, hidden).astype(np.float64).T).astype(np.float32)
    got = _logits(layer, x, monkeypatch)
    assert np.array_equal(got[0], want[0])
    w, ax, aw = layer.router.reshape(n_expert, hidden).astype(np.float64), np.abs(x.astype(np.float64)), np.abs(layer.router.reshape(n_expert, hidden).astype(np.float64))
    mx, mw = ax.max(1)[:, None], aw.max(1)[None, :]
    bound = 2.0 ** -38 * (mx * aw.sum(1)[None, :] + mw * ax.sum(1)[:, None]) + 2.0 ** -42 * hidden * mx * mw
    assert np.all(np.abs(got.astype(np.float64) - x.astype(np.float64) @ w.T) <= bound + np.spacing(np.abs(want)) / 2 + 2.0 ** -149)
    assert np.mean(got != want) < 0.01


def test_a_row_that_is_not_finite_is_reported(monkeypatch):
    layer = synth.moe_layer(9, synth.MoeDims(hidden=256, n_expert=128, top_k=2, ffn=256, ffn_sh=256))
    for bad in (np.nan, np.inf):
        x = np.random.default_rng(3).normal(0, 1, size=(40, 256)).astype(np.float32)
        x[7, 100] = bad
        with pytest.raises(rc.redcuda.RedcudaError):
            _logits(layer, x, monkeypatch)
        rc.redcuda.profile_enable(False)


@pytest.mark.parametrize("large", [1e3, 1e5, 1e6, 1e8, 1e20])
@pytest.mark.parametrize("where", ["rows", "router", "both"])
@pytest.mark.parametrize("hidden,n_expert,ntok", [(2048, 512, 41), (256, 128, 70)])
def test_a_large_element_that_meets_a_zero(hidden, n_expert, ntok, where, large, monkeypatch):
    """Beside it the others lose digits, and the sum does not show it: these logits are summed again in double. A logit that is not lacks at most 2^-24 of itself
    before it is rounded, so none is off by more than a unit, and the experts are those of the double sums."""
    layer = synth.moe_layer(9, synth.MoeDims(hidden=hidden, n_expert=n_expert, top_k=4, ffn=256, ffn_sh=256))
    x = np.random.default_rng(ntok).normal(0, 1, size=(ntok, hidden)).astype(np.float32)
    w = layer.router.reshape(n_expert, hidden)
    if where != "router":
        x[1::2, 17], w[:, 17] = large, 0.0
    if where != "rows":
        w[1::2, 200], x[:, 200] = large, 0.0
    exact = x.astype(np.float64) @ w.astype(np.float64).T
    got = _logits(layer, x, monkeypatch)
    assert np.all(np.abs(got.astype(np.float64) - exact) <= np.spacing(np.abs(exact.astype(np.float32))))
    assert np.mean(got != exact.astype(np.float32)) < 0.01
    ids = []
    for least in ("1", "0"):
        monkeypatch.setenv("RC_ROUTER_I8_MIN", least)
        m = rc.MoeLayer(layer, max_tokens=ntok)
        ids.append(np.array(m.forward(x, want_routing=True)[1]))
        m.close()
    assert np.array_equal(ids[0], ids[1])
