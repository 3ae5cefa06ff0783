"""Decode attention where a warp takes several groups of four positions in turn (the rows of the next one requested ahead, the running maximum carried over, sums rescaled
where it rises): a few tokens of a prompt in eight slices of 100 positions, one token in 64 slices of 63. Every head shape and both cache types against the chunk kernel
(tests/test_gpu_attention_long.py holds that against the CPU oracle), two of them against the oracle itself. The parity bound of a layer's output, 1e-3, would not see a group that is left out: with
one planted in the oracle (positions 340 to 343 of 402) the last layer differs by 6e-4 to 1.2e-3 of its largest value, and of 4001 positions it would be a
tenth of that. Four layers of fp32 sums in two orders differ by 1e-7 to 4e-7; the bound is 5e-6."""
import os

import numpy as np
import pytest

import oracle_lib as ol
from dwarfstar_red_lite_b200 import gguf_writer, synth
from dwarfstar_red_lite_b200.engine import Engine

pytestmark = pytest.mark.gpu

REL_OUT = 5e-6
SHAPES = [(64, 4, 2), (64, 8, 2), (128, 8, 2), (128, 8, 1), (256, 4, 1), (256, 8, 1)]


def _model(tmp_path, shape, context):
    head_dim, n_head, n_head_kv = shape
    dims = synth.ModelDims(n_layer=4, vocab=256, hidden=256, n_head=n_head, n_head_kv=n_head_kv, head_dim=head_dim, rope_dims=32, d_state=32, n_group=4, dt_rank=8, d_inner=256,
                           n_expert=8, top_k=2, ffn=256, ffn_sh=256, context=context)
    sm = synth.model(5, dims)
    path = str(tmp_path / "m.gguf")
    gguf_writer.write_gguf(path, sm)
    return dims, sm, path


def _near(a, b):
    assert np.max(np.abs(a - b)) <= REL_OUT * np.max(np.abs(b))


def _state(eng, dims, logits):
    return [np.array(logits)] + [np.array(eng.layer_out(l)) for l in range(dims.n_layer)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kv_f16", [False, True])
def test_against_the_chunk_kernel(shape, kv_f16, tmp_path, monkeypatch):
    monkeypatch.setenv("RL_KV_F16", "1" if kv_f16 else "0")
    dims, _, path = _model(tmp_path, shape, 4096)
    prompt = np.random.default_rng(3).integers(0, dims.vocab, 4001).astype(np.uint32)
    whole, split = Engine(path, context=4096, prefill_batch=2048), Engine(path, context=4096, prefill_batch=400)
    try:
        for n in (803, 405):                       # the last chunk: three tokens and five, on the kernel under test
            whole.reset(); split.reset()
            want, got = _state(whole, dims, whole.prefill(prompt[:n])), _state(split, dims, split.prefill(prompt[:n]))
            for a, b in zip(got, want):
                _near(a, b)
        whole.reset(); split.reset()
        want = _state(whole, dims, whole.prefill(prompt))
        split.prefill(prompt[:-1])
        for a, b in zip(_state(split, dims, split.step(int(prompt[-1]))), want):
            _near(a, b)
    finally:
        whole.close(); split.close()


@pytest.mark.parametrize("shape,kv_f16", [((64, 8, 2), False), ((256, 8, 1), True)])
def test_against_the_oracle(shape, kv_f16, tmp_path, monkeypatch):
    monkeypatch.setenv("RL_KV_F16", "1" if kv_f16 else "0")
    n = 402
    dims, sm, path = _model(tmp_path, shape, n + 2)
    prompt = np.random.default_rng(4).integers(0, dims.vocab, n).astype(np.uint32)
    om = ol.OracleModel(sm, kv_f16=kv_f16, context=dims.context)
    for t in prompt:
        ml = om.step(int(t), threads=os.cpu_count() or 1)
    eng = Engine(path, context=dims.context, prefill_batch=400)
    try:
        _near(eng.prefill(prompt), ml)
        for l in range(dims.n_layer):
            _near(eng.layer_out(l), om.layer_out(l))
    finally:
        eng.close()
