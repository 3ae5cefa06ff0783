"""A decoding step with the router logits (opt-in) or the shared expert on the tcgen05 GEMM from the first token on: the first reads the
normalised row, which no kernel before it may be left out to make; the second leaves SiLU(gate) * up to its down projection."""
import numpy as np
import pytest

from dwarfstar_red_lite_b200 import gguf_writer, synth
from dwarfstar_red_lite_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("switch", ["RC_ROUTER_TC_MIN", "RC_SH_TC_MIN"])
def test_step_with_a_tensor_core_form_from_one_token(tmp_path, switch, monkeypatch):
    dims = synth.tiny_model_dims(n_layer=4, type_shared=synth.Q6_K)
    path = str(tmp_path / "tiny.gguf")
    gguf_writer.write_gguf(path, synth.model(61, dims))
    outs, ids = [], []
    for value in (None, "1"):
        if value:
            monkeypatch.setenv(switch, value)
        eng = Engine(path, context=dims.context)
        try:
            eng.step(3)
            outs.append(np.stack([eng.layer_out(l) for l in range(dims.n_layer)]))
            ids.append([eng.router_ids(l).tolist() for l in range(dims.n_layer)])
        finally:
            eng.close()
    # split-fp16 logits carry 1e-6 of sum |w x| (5e-5 of the expert weights); 1e-3 of a layer's range is the parity bound of a step
    assert ids[0] == ids[1]
    assert np.max(np.abs(outs[0] - outs[1])) <= 1e-3 * np.max(np.abs(outs[0]))
