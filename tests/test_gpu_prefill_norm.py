"""The row norms of a chunk at the full width: a warp a row from 148 rows on, a block of 1024 threads below. The same prompt in one chunk
and in chunks that take the other form, against the CPU oracle."""
import os

import numpy as np
import pytest

import oracle_lib as ol
from dwarfstar_red_lite_b200 import gguf_writer, synth
from dwarfstar_red_lite_b200.engine import Engine

pytestmark = pytest.mark.gpu

TOKENS, REL_OUT = 150, 1e-3          # the parity bound of a layer's output


def test_both_forms_of_the_norm(tmp_path, monkeypatch):
    monkeypatch.setenv("RL_KV_F16", "1")
    dims = synth.ModelDims(n_layer=4, vocab=512, n_expert=16, top_k=4, context=TOKENS + 10)
    sm = synth.model(77, dims)
    path = str(tmp_path / "mid.gguf")
    gguf_writer.write_gguf(path, sm)
    prompt = np.random.default_rng(12).integers(0, dims.vocab, TOKENS).astype(np.uint32)
    om = ol.OracleModel(sm, kv_f16=True, context=dims.context)
    for t in prompt:
        ml = om.step(int(t), threads=os.cpu_count() or 1)
    for chunk in (TOKENS, 148, 147, 60):
        eng = Engine(path, context=dims.context, prefill_batch=chunk)
        try:
            gl = eng.prefill(prompt)
            for l in range(dims.n_layer):
                assert np.array_equal(eng.router_ids(l), om.router_ids(l)), (chunk, l)
                a, b = eng.layer_out(l), om.layer_out(l)
                assert np.max(np.abs(a - b)) <= REL_OUT * np.max(np.abs(b)), (chunk, l)
            assert np.max(np.abs(gl - ml)) <= REL_OUT * np.max(np.abs(ml)) + 1e-6, chunk
        finally:
            eng.close()
