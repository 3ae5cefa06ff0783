"""What a layer says that it keeps on the device: the weights, and the router's digits where a call can be long enough to read them."""
import pytest

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


def _bytes(layer, max_tokens):
    m = rc.MoeLayer(layer, max_tokens=max_tokens)
    try:
        return m.resident_bytes()
    finally:
        m.close()


def test_router_digits_are_counted(monkeypatch):
    monkeypatch.delenv("RC_ROUTER_I8_MIN", raising=False)
    layer = synth.moe_layer(1, synth.MoeDims(hidden=256, n_expert=512, top_k=2, ffn=256, ffn_sh=256))
    digits, weights = 5 * 512 * 256, _bytes(layer, 639)
    assert digits <= _bytes(layer, 640) - weights <= digits + 512 * 16 + 256
    monkeypatch.setenv("RC_ROUTER_I8_MIN", "0")                 # never: none are made
    assert _bytes(layer, 640) == weights
    monkeypatch.setenv("RC_ROUTER_I8_MIN", "2")
    assert _bytes(layer, 2) > weights
