"""The work a user of the library has it do, case by case, through its public entry points.

Four kinds of case:

  moe     one pass of a batch of tokens through a few distinct resident MoE layers (router, routed experts, shared
          expert): `MoeLayer.forward_device`, or `MoeLayer.forward` with host buffers
  dn      one decode step of every Gated DeltaNet layer of a model for a batch of sequences:
          `redcuda_deltanet_step_noalloc` on device buffers
  engine  one turn of a model through `Engine`: a prompt (chunked prefill), then single-token steps with their logits
  stage   one stage call on host buffers: `quant_matvec`, `quant_matmul_tc`, `quant_dequant_rows`

Every input is synthetic and made from the seed (`synth.py`, `synth_device.py`); shapes are those of the repository's
configurations (hidden 2048, 512 experts, top-10, ffn 512, 16 / 32 DeltaNet heads of 128, vocabulary 151936).
"""
from __future__ import annotations

import ctypes
import math
import os
import tempfile

import numpy as np
import torch

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import gguf_writer, redcuda, synth, synth_device
from dwarfstar_red_lite_b200.engine import Engine

TYPES = {"f16": synth.F16, "q6_k": synth.Q6_K, "iq2_xxs": synth.IQ2_XXS, "iq3_s": synth.IQ3_S, "q8_0": synth.Q8_0, "q2_k": synth.Q2_K, "q4_k": synth.Q4_K,
         "q5_k": synth.Q5_K, "iq3_xxs": synth.IQ3_XXS, "iq2_s": synth.IQ2_S, "iq4_xs": synth.IQ4_XS, "iq2_xs": synth.IQ2_XS, "iq1_m": synth.IQ1_M}
# fp16 block-scale ranges that give weights of a few hundredths, per type
D_RANGE = {"q6_k": (1e-3, 5e-3), "iq2_xxs": (1e-2, 6e-2), "iq3_s": (2e-3, 1.2e-2), "q8_0": (1e-3, 8e-3), "q2_k": (2e-2, 8e-2), "q4_k": (1e-3, 5e-3), "q5_k": (1e-3, 5e-3),
           "iq3_xxs": (2e-3, 1.2e-2), "iq2_s": (1e-2, 6e-2), "iq4_xs": (1e-3, 5e-3), "iq2_xs": (1e-2, 6e-2), "iq1_m": (2e-2, 1e-1)}
VOCAB, CONTEXT, ENGINE_LAYERS = 151936, 4096, 8
DN_LAYERS = 36                                   # DeltaNet layers of the 48-layer model
DN = dict(d_conv=4, d_state=128, n_group=16, dt_rank=32, d_inner=4096, channels=8192, rms_eps=1e-6)


# ---------------------------------------------------------------------------------------------------------------- cases

def _moe(name, tokens, layers, experts="iq2_xxs", routing="computed", resid=False, buffers="device", hidden=2048, n_expert=512, ffn=512):
    c = dict(kind="moe", tokens=tokens, layers=layers, experts=experts, routing=routing, resid=resid, buffers=buffers, hidden=hidden, n_expert=n_expert, ffn=ffn)
    return dict(c, name=name) if name else c


def _engine(name, start, prompt, steps, kv):
    c = dict(kind="engine", start=start, prompt=prompt, steps=steps, kv=kv)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user, one token: the MoE half of 16 layers of a decoding step, router computed, residual added
        _moe("moe token", 1, 16, resid=True),
        # a handful of users decoding together (or a short draft being verified)
        _moe("moe batch of 6", 6, 8),
        # the benchmark's workload: 64 sequences, router logits drawn so that expert popularity is Zipf(1.1)
        _moe("moe batch of 64, skewed", 64, 8, routing="zipf"),
        # the same through the host-buffer call that a C host makes (pinned buffers)
        _moe("moe batch of 64, host buffers", 64, 4, routing="zipf", buffers="host"),
        # a large serving batch or a short prompt chunk
        _moe("moe batch of 300", 300, 4, resid=True),
        # one full prefill chunk (the default chunk of 2048 tokens)
        _moe("moe chunk of 2048", 2048, 2, resid=True),
        # the other expert format of the path, a mid-sized decoding batch
        _moe("moe IQ3_S batch of 24", 24, 4, experts="iq3_s"),
        # eight sequences, one decode step through every DeltaNet layer
        dict(kind="dn", name="deltanet step of 8", batch=8),
        # single-user decoding deep in the context, logits to the host for the sampler; fp16 K/V
        _engine("decode at 3500", 3500, 0, 16, "f16"),
        # a chat turn: an ordinary prompt, then a short answer; fp32 K/V (the default)
        _engine("turn of 93 + 8", 0, 93, 8, "f32"),
        # a long document: two prefill chunks, the second ragged
        _engine("prefill of 3501", 0, 3501, 0, "f16"),
        # the stage call of a tool that holds GGUF rows on the host: one projection for a few tokens
        dict(kind="stage", name="host matvec Q4_K", op="matvec", type="q4_k", rows=8192, cols=2048, tokens=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["moe", "dn", "engine", "stage"], [10, 2, 4, 4])[0]
    if kind == "moe":
        tokens = _log_int(rng, 1, 2048)
        layers = 8 if tokens <= 64 else 4 if tokens <= 512 else 2
        hidden, n_expert, ffn = rng.choices([(2048, 512, 512), (2048, 256, 512), (1024, 128, 512), (2048, 512, 1024)], [7, 1, 1, 1])[0]
        experts = rng.choices(["iq2_xxs", "iq3_s"], [7, 2])[0]
        buffers = rng.choices(["device", "host"], [4, 1])[0]
        return _moe(None, tokens, layers, experts, rng.choice(["computed", "zipf"]), buffers == "device" and rng.random() < 0.5, buffers, hidden, n_expert, ffn)
    if kind == "dn":
        return dict(kind="dn", batch=rng.randint(1, 10))
    if kind == "engine":
        prompt = rng.choice([0, _log_int(rng, 2, 128), _log_int(rng, 129, 3501)])
        steps = rng.randint(0 if prompt else 4, 16)
        return _engine(None, _log_int(rng, 1, 4000 - prompt) if rng.random() < 0.5 else 0, prompt, steps, rng.choice(["f16", "f32"]))
    op = rng.choice(["matvec", "matmul_tc", "dequant"])
    t = rng.choice(["q6_k", "iq2_xxs", "iq3_s"] if op == "matmul_tc" else sorted(TYPES))
    tokens = {"matvec": rng.randint(1, 16), "matmul_tc": _log_int(rng, 8, 512), "dequant": 0}[op]
    return dict(kind="stage", op=op, type=t, rows=_log_int(rng, 32, 8192), cols=256 * _log_int(rng, 1, 16), tokens=tokens)


# -------------------------------------------------------------------------------------------------------------- prepare

def _prepare_moe(c, seed):
    dims = synth.MoeDims(hidden=c["hidden"], n_expert=c["n_expert"], ffn=c["ffn"], type_gu=TYPES[c["experts"]], type_down=TYPES[c["experts"]])
    rc.set_codebooks()
    dev, T, L = torch.device("cuda", 0), c["tokens"], c["layers"]
    layers = []
    for l in range(L):
        tens = synth_device.moe_layer_tensors(seed * 64 + l, dims, dev)
        torch.cuda.synchronize()
        layers.append(rc.MoeLayer(device_tensors=tens, dims=dims, max_tokens=T))
        del tens
    g = torch.Generator(device=dev)
    g.manual_seed(seed + 1)
    x = torch.randn(L, T, dims.hidden, device=dev, generator=g)
    logits = None
    if c["routing"] == "zipf":
        logits = torch.from_numpy(np.stack([synth.zipf_routing_logits(seed * 64 + l, T, dims.n_expert) for l in range(L)])).to(dev)
    s = dict(kind="moe", layers=layers, tokens=T, host=c["buffers"] == "host")
    if s["host"]:
        pin = lambda t: None if t is None else t.cpu().pin_memory().numpy()  # noqa: E731
        return dict(s, x=pin(x), logits=pin(logits), out=pin(torch.zeros_like(x)))
    resid = torch.randn(L, T, dims.hidden, device=dev, generator=g) if c["resid"] else None
    return dict(s, x=x, logits=logits, resid=resid, out=torch.empty_like(x))


def _prepare_dn(c, seed):
    dev, B, L = torch.device("cuda", 0), c["batch"], DN_LAYERS
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    rnd = lambda *shape, scale=1.0: torch.randn(*shape, device=dev, generator=g) * scale  # noqa: E731
    R, S = DN["dt_rank"], DN["d_state"]
    w = dict(conv_kernel=rnd(L, DN["channels"], DN["d_conv"], scale=0.5), dt_bias=rnd(L, R), ssm_a=-torch.exp(rnd(L, R, scale=0.5)), ssm_norm=1.0 + rnd(L, S, scale=0.1))
    params = [redcuda.DeltanetParams(DN["d_conv"], S, DN["n_group"], R, DN["d_inner"], DN["channels"], DN["rms_eps"],
                                     *[ctypes.cast(w[k][l].data_ptr(), redcuda.f32p) for k in ("conv_kernel", "dt_bias", "ssm_a", "ssm_norm")]) for l in range(L)]
    return dict(kind="dn", weights=w, params=params, batch=B, qkv=rnd(L, B, DN["channels"]), z=rnd(L, B, DN["d_inner"]), ba=rnd(L, B, 2 * R),
                conv=rnd(L, B, DN["channels"], DN["d_conv"] - 1), rec=rnd(L, B, R, S, S, scale=0.05), out=torch.empty(L, B, DN["d_inner"], device=dev))


_engines = {}


def _engine_of(kv):
    """The opened model, kept for the life of the process as a server keeps it; an 8-layer model of the full widths (two
    of its layers are attention). The file is written once per machine."""
    if kv not in _engines:
        dims = synth.ModelDims(n_layer=ENGINE_LAYERS, vocab=VOCAB, context=CONTEXT)
        path = os.path.join(tempfile.gettempdir(), "redcuda_cases_%dl_%dv.gguf" % (ENGINE_LAYERS, VOCAB))
        if not os.path.exists(path):
            part = "%s.%d" % (path, os.getpid())
            gguf_writer.write_gguf_streaming(part, 17, dims)
            os.replace(part, path)
        rc.set_codebooks()
        before = os.environ.get("RL_KV_F16")
        os.environ["RL_KV_F16"] = "1" if kv == "f16" else "0"
        try:
            _engines[kv] = Engine(path, context=CONTEXT)
        finally:
            if before is None:
                del os.environ["RL_KV_F16"]
            else:
                os.environ["RL_KV_F16"] = before
    return _engines[kv]


def _prepare_engine(c, seed):
    rng = np.random.default_rng(seed)
    tokens = rng.integers(0, VOCAB, size=c["prompt"] + c["steps"]).astype(np.uint32)
    return dict(kind="engine", engine=_engine_of(c["kv"]), start=c["start"], prompt=tokens[:c["prompt"]], step_tokens=tokens[c["prompt"]:].tolist(),
                logits=np.zeros((c["steps"], VOCAB), np.float32))


def _prepare_stage(c, seed):
    rng = np.random.default_rng(seed)
    t = TYPES[c["type"]]
    if c["type"] == "f16":
        w = rng.uniform(-1, 1, size=(c["rows"], c["cols"])).astype(np.float16)
    else:
        w = synth.quant_matrix(rng, t, c["rows"], c["cols"], *D_RANGE[c["type"]], (-64, 63) if t == synth.Q6_K else None)
    rc.set_codebooks()
    x = rng.normal(0, 1, size=(c["tokens"], c["cols"])).astype(np.float32)
    return dict(kind="stage", op=c["op"], type=t, w=w, rows=c["rows"], cols=c["cols"], x=x)


def prepare(case, seed):
    return {"moe": _prepare_moe, "dn": _prepare_dn, "engine": _prepare_engine, "stage": _prepare_stage}[case["kind"]](case, seed)


# ------------------------------------------------------------------------------------------------------------------ run

def _run_moe(s):
    if s["host"]:
        for l, m in enumerate(s["layers"]):
            m.forward(s["x"][l], logits_in=None if s["logits"] is None else s["logits"][l], out=s["out"][l])
        return s["out"]
    stream = torch.cuda.current_stream().cuda_stream
    for l, m in enumerate(s["layers"]):
        m.forward_device(s["tokens"], s["x"][l].data_ptr(), s["out"][l].data_ptr(), stream, 0 if s["logits"] is None else s["logits"][l].data_ptr(),
                         0 if s["resid"] is None else s["resid"][l].data_ptr())
    return s["out"]


def _run_dn(s):
    lib, stream = rc.lib(), torch.cuda.current_stream().cuda_stream or None
    for l, p in enumerate(s["params"]):
        ok = lib.redcuda_deltanet_step_noalloc(ctypes.byref(p), s["batch"], s["qkv"][l].data_ptr(), s["z"][l].data_ptr(), s["ba"][l].data_ptr(),
                                               s["conv"][l].data_ptr(), s["rec"][l].data_ptr(), s["out"][l].data_ptr(), stream)
        if ok != 1:
            raise RuntimeError(lib.redcuda_last_error().decode())
    return [s["out"], s["conv"], s["rec"]]


def _run_engine(s):
    e, got = s["engine"], []
    e.reset()
    if s["start"]:
        e.set_position(s["start"])
    if s["prompt"].size:
        got.append(e.prefill(s["prompt"]))
    for i, t in enumerate(s["step_tokens"]):
        e.step(t, logits=s["logits"][i])
    return got + [s["logits"]] if s["step_tokens"] else got


def _run_stage(s):
    if s["op"] == "dequant":
        return rc.quant_dequant_rows(s["type"], s["w"], s["cols"])
    f = rc.quant_matvec if s["op"] == "matvec" else rc.quant_matmul_tc
    return f(s["type"], s["w"], s["rows"], s["cols"], s["x"])


def run(state):
    return {"moe": _run_moe, "dn": _run_dn, "engine": _run_engine, "stage": _run_stage}[state["kind"]](state)


# ------------------------------------------------------------------------------------------------------ work, tolerance

def _distinct(T, n_expert, top_k, routing):
    """Expected number of distinct experts that T tokens select."""
    if routing == "computed":
        return n_expert * (1.0 - (1.0 - top_k / n_expert) ** T)
    p = 1.0 / np.arange(1, n_expert + 1) ** 1.1
    # top_k draws without replacement: inclusion probability 1 - exp(-lambda p), lambda such that they add up to top_k
    p, lam = p / p.sum(), float(top_k)
    for _ in range(60):
        lam *= top_k / float((1.0 - np.exp(-lam * p)).sum())
    return float((1.0 - np.exp(-lam * p * T)).sum())


def _moe_layer_work(T, hidden, n_expert, ffn, experts, routing, ffn_sh=512, top_k=10):
    t = TYPES[experts]
    expert = 2 * ffn * synth.row_bytes(t, hidden) + hidden * synth.row_bytes(t, ffn)
    shared = 2 * ffn_sh * synth.row_bytes(synth.Q6_K, hidden) + hidden * synth.row_bytes(synth.Q6_K, ffn_sh)
    router = n_expert * hidden if routing == "computed" else 0
    b = _distinct(T, n_expert, top_k, routing) * expert + shared + 4 * router + 4 * hidden + 8 * T * hidden + (0 if router else 4 * T * n_expert)
    return b, 2.0 * T * (top_k * 3 * hidden * ffn + 3 * hidden * ffn_sh + router)


def _engine_pass_work(positions, kv, logits):
    """A pass of consecutive tokens at `positions` through the 8-layer model: weights read once, K/V read once."""
    d, T = synth.ModelDims(), len(positions)
    q6 = lambda r, c: r * synth.row_bytes(synth.Q6_K, c)  # noqa: E731
    mb, mf = _moe_layer_work(T, d.hidden, d.n_expert, d.ffn, "iq2_xxs", "computed")
    kvb = 2 * d.n_head_kv * d.head_dim * (2 if kv == "f16" else 4)
    b = f = 0.0
    for l in range(ENGINE_LAYERS):
        if d.is_attention(l):
            mats = [(2 * 4096, d.hidden), (512, d.hidden), (512, d.hidden), (d.hidden, 4096)]
            b += kvb * (positions[-1] + 1)
            f += 4.0 * d.n_head * d.head_dim * float(sum(p + 1 for p in positions))
        else:
            mats = [(d.channels, d.hidden), (d.d_inner, d.hidden), (2 * d.dt_rank, d.hidden), (d.hidden, d.d_inner)]
            b += 8.0 * (d.dt_rank * d.d_state ** 2 + 3 * d.channels)
            f += 8.0 * T * d.dt_rank * d.d_state ** 2
        b += sum(q6(*m) for m in mats) + mb
        f += 2.0 * T * sum(r * c for r, c in mats) + mf
    if logits:
        b, f = b + q6(VOCAB, d.hidden) + 4 * VOCAB, f + 2.0 * VOCAB * d.hidden
    return b, f


def work(case):
    c = case
    if c["kind"] == "moe":
        b, f = _moe_layer_work(c["tokens"], c["hidden"], c["n_expert"], c["ffn"], c["experts"], c["routing"])
        b, f = (b + (4 * c["tokens"] * c["hidden"] if c["resid"] else 0)) * c["layers"], f * c["layers"]
    elif c["kind"] == "dn":
        state = DN["dt_rank"] * DN["d_state"] ** 2
        small = 2 * 3 * DN["channels"] + DN["channels"] + 2 * DN["d_inner"] + 2 * DN["dt_rank"]
        b = DN_LAYERS * 4.0 * (c["batch"] * (2 * state + small) + DN["channels"] * DN["d_conv"])
        f = DN_LAYERS * 8.0 * c["batch"] * state
    elif c["kind"] == "engine":
        b = f = 0.0
        at, left = c["start"], c["prompt"]
        while left:
            n = min(left, 2048)
            pb, pf = _engine_pass_work(range(at, at + n), c["kv"], n == left)
            b, f, at, left = b + pb, f + pf, at + n, left - n
        for i in range(c["steps"]):
            pb, pf = _engine_pass_work([at + i], c["kv"], True)
            b, f = b + pb, f + pf
    else:
        wb = c["rows"] * synth.row_bytes(TYPES[c["type"]], c["cols"])
        n = c["rows"] * c["cols"]
        if c["op"] == "dequant":
            b, f = wb + 4.0 * n, float(n)
        else:
            b, f = wb + 4.0 * c["tokens"] * (c["rows"] + c["cols"]), 2.0 * c["tokens"] * n
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    if case["kind"] == "engine":
        # eight layers of 32-bit sums feed the DeltaNet states, the K/V rows and 80 discrete expert choices per token: where
        # two router logits are closer than that noise (one choice in some ten thousand) another expert is as right, and
        # an fp16 K/V row rounds the noise up to half a unit of fp16
        return {"rel": 2e-4}
    if case["kind"] == "stage" and case["op"] == "dequant":
        return "exact"
    return {"rel": 2e-5}                           # 32-bit sums of up to 4096 products, two matrices deep
