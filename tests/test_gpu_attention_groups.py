"""Decode attention over groups of positions: every head shape it is built for, both cache types, sequence lengths from one
through two slices of 32 and a part of a third, against the CPU oracle."""
import os

import numpy as np
import pytest

import oracle_lib as ol
from dwarfstar_red_lite_b200 import gguf_writer, synth
from dwarfstar_red_lite_b200.engine import Engine

pytestmark = pytest.mark.gpu

REL_OUT = 1e-3      # parity bound of a layer's output


@pytest.mark.parametrize("head_dim,n_head,n_head_kv", [(64, 4, 2), (64, 8, 2), (128, 8, 2), (128, 8, 1), (256, 4, 1), (256, 8, 1)])
@pytest.mark.parametrize("kv_f16", [False, True])
def test_decode_against_the_oracle(head_dim, n_head, n_head_kv, kv_f16, tmp_path, monkeypatch):
    monkeypatch.setenv("RL_KV_F16", "1" if kv_f16 else "0")
    steps = 70
    dims = synth.ModelDims(n_layer=4, vocab=256, hidden=256, n_head=n_head, n_head_kv=n_head_kv, head_dim=head_dim, rope_dims=32, d_state=32, n_group=4, dt_rank=8, d_inner=256,
                           n_expert=8, top_k=2, ffn=256, ffn_sh=256, context=steps + 2)
    sm = synth.model(5, dims)
    path = str(tmp_path / "m.gguf")
    gguf_writer.write_gguf(path, sm)
    om = ol.OracleModel(sm, kv_f16=kv_f16, context=dims.context)
    eng = Engine(path, context=dims.context)
    try:
        for i, t in enumerate(np.random.default_rng(2).integers(0, dims.vocab, steps).astype(np.uint32)):
            want, got = om.step(int(t), threads=os.cpu_count() or 1), eng.step(int(t))
            assert np.max(np.abs(got - want)) <= REL_OUT * np.max(np.abs(want)) + 1e-6, i
    finally:
        eng.close()
