"""The lines at which a layer's calls change kernels, as they are by default: on either side of each, the kernels that ran and the result against the CPU oracle."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def layer():
    return synth.moe_layer(11, synth.MoeDims(hidden=256, n_expert=512, top_k=10, ffn=256, ffn_sh=256))


@pytest.fixture(scope="module")
def resident(layer):
    m = rc.MoeLayer(layer, max_tokens=640)
    yield m
    m.close()


@pytest.mark.parametrize("tokens,experts_tc,router_digits", [(449, False, False), (450, True, False), (639, True, False), (640, True, True)])
def test_kernels_beside_a_line(layer, resident, tokens, experts_tc, router_digits, monkeypatch):
    for v in ("RC_MOE_TC_MIN", "RC_ROUTER_I8_MIN", "RC_ROUTER_TC_MIN"):
        monkeypatch.delenv(v, raising=False)
    x = np.random.default_rng(tokens).normal(0, 1, size=(tokens, 256)).astype(np.float32)
    rc.redcuda.profile_enable(True)
    out, ids, _, logits = resident.forward(x, want_routing=True)
    kernels = rc.redcuda.profile_report()
    rc.redcuda.profile_enable(False)
    assert ("moe_gateup_tc" in kernels) == experts_tc and ("moe_down_tc" in kernels) == experts_tc
    assert ("moe_router_digits" in kernels) == router_digits and ("moe_router_exact" in kernels) == router_digits
    exact = x.astype(np.float64) @ layer.router.astype(np.float64).T
    assert np.all(np.abs(logits - exact) <= np.spacing(np.abs(exact.astype(np.float32))))
    for t in (0, tokens // 2, tokens - 1):
        want, want_ids, _, _ = ol.moe_ffn(layer, x[t], threads=4)
        assert np.array_equal(ids[t], want_ids)
        assert np.max(np.abs(out[t] - want)) <= 1e-3 * np.max(np.abs(want))


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_a_row_that_is_not_finite_on_the_tensor_cores(bad, monkeypatch):
    """It stays that, and the other rows of the batch are untouched."""
    import torch
    monkeypatch.delenv("RC_MOE_TC_MIN", raising=False)
    m = rc.MoeLayer(synth.moe_layer(3, synth.MoeDims(hidden=512, n_expert=16, top_k=4, ffn=256, ffn_sh=256)), max_tokens=200)
    rng = np.random.default_rng(0)
    x, logits = rng.normal(0, 1, size=(200, 512)).astype(np.float32), rng.normal(0, 1, size=(200, 16)).astype(np.float32)
    ids = torch.from_numpy(rng.integers(0, 16, size=600).astype(np.int32)).cuda()

    def pairs(rows):                               # 600 pairs of three times the rows
        xd, o = torch.from_numpy(np.tile(rows, (3, 1))).cuda(), torch.zeros(600, 512, device="cuda")
        m.experts_device(600, xd.data_ptr(), ids.data_ptr(), o.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return o.cpu().numpy().reshape(3, 200, 512).transpose(1, 0, 2).reshape(200, -1)

    rc.redcuda.profile_enable(True)
    for f in (pairs, lambda rows: m.forward(rows, logits_in=logits)):
        clean = f(x)
        for r in (0, 199):
            y = x.copy()
            y[r, 37] = bad
            got = f(y)
            assert np.isfinite(clean).all() and not np.isfinite(got[r]).any()
            others = np.arange(200) != r
            assert np.array_equal(got[others], clean[others])
    kernels = rc.redcuda.profile_report()
    rc.redcuda.profile_enable(False)
    assert "moe_gateup_tc" in kernels and "moe_gateup_nib" not in kernels
    m.close()
