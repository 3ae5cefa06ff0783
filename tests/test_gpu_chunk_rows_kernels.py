"""The kernels that take a chunk's rows a warp (norms, attention preparation, DeltaNet preparation and tail): every row length they are built for, convs of
two to four taps, rotations of a part and of the whole head, a ragged last group of tokens, against the CPU oracle (parity bound of a layer's output)."""
import os

import numpy as np
import pytest

import oracle_lib as ol
from dwarfstar_red_lite_b200 import gguf_writer, synth
from dwarfstar_red_lite_b200.engine import Engine

pytestmark = pytest.mark.gpu

TOKENS, REL_OUT = 149, 1e-3
SHAPES = [dict(hidden=1024, n_head=8, head_dim=128, rope_dims=128, d_state=64, n_group=4, dt_rank=8, d_inner=512, d_conv=4),
          dict(hidden=512, n_head=8, head_dim=64, rope_dims=32, d_state=32, n_group=4, dt_rank=8, d_inner=256, d_conv=3),
          dict(hidden=2048, n_head=4, head_dim=256, rope_dims=64, d_state=256, n_group=2, dt_rank=4, d_inner=1024, d_conv=2)]


@pytest.mark.parametrize("shape", SHAPES)
def test_a_chunk_against_the_oracle(shape, tmp_path, monkeypatch):
    monkeypatch.setenv("RL_KV_F16", "0")
    dims = synth.ModelDims(n_layer=4, vocab=256, n_expert=8, top_k=2, ffn=256, ffn_sh=256, context=TOKENS + 10, **shape)
    sm = synth.model(78, dims)
    path = str(tmp_path / "m.gguf")
    gguf_writer.write_gguf(path, sm)
    prompt = np.random.default_rng(12).integers(0, dims.vocab, TOKENS).astype(np.uint32)
    om = ol.OracleModel(sm, kv_f16=False, context=dims.context)
    for t in prompt:
        ml = om.step(int(t), threads=os.cpu_count() or 1)
    eng = Engine(path, context=dims.context, prefill_batch=TOKENS)
    try:
        gl = eng.prefill(prompt)
        for l in range(dims.n_layer):
            assert np.array_equal(eng.router_ids(l), om.router_ids(l)), l
            a, b = eng.layer_out(l), om.layer_out(l)
            assert np.max(np.abs(a - b)) <= REL_OUT * np.max(np.abs(b)), l
        assert np.max(np.abs(gl - ml)) <= REL_OUT * np.max(np.abs(ml)) + 1e-6
    finally:
        eng.close()
