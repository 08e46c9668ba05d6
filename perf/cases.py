"""What a user of this framework has it do, as cases that can be timed.

A case is a dict of plain values; `kind` picks the entry point:

  decode    CudaDecoder.Step, a token at a time, the logits in one pinned host buffer
  pairs     CudaDecoder.StepTokens on a token and a draft, then Resolve (speculative decoding)
  product   Context.matmul / matmul_device: one matrix, one to eight tokens
  layer     CudaProjections.apply_device: every product of a DeltaNet layer (and the LM head
            where asked) on the rows of a batch, from one decode row to a whole prompt
  rule      Context.delta_rule_device: the bare Gated DeltaNet update of several sequences
  mixer     CudaMixer.Run: a DeltaNet layer's step, one to four tokens of each sequence
  moe       CudaMoe.MoeFfn: router, top-k and the routed experts of one layer
  attention gufo_cuda_attention_device: gated attention of one token over an fp16 cache

Weights are N(0, 0.02) values packed by this project's quantizers, activations N(0, 1) with a
log-normal scale per channel (some channels of a real residual stream are many times larger
than the rest).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from gufo_npu_b200 import _capi
from gufo_npu_b200 import quantize as Q
from gufo_npu_b200 import synth
from gufo_npu_b200.backend import Context, CudaDecoder, CudaMixer, CudaMoe, CudaProjections, Stage

DEVICE = "cuda:0"
TYPES = {"Q4_K": Q.GGML_Q4_K, "Q5_K": Q.GGML_Q5_K, "Q6_K": Q.GGML_Q6_K, "Q8_0": Q.GGML_Q8_0}
LAYER_STAGES = (Stage.kLinearIn, Stage.kMixerOut, Stage.kFfnIn, Stage.kFfnDown)


def listed():
    return [
        # The headline: single-token decoding of the benchmark's 2B-class dense model.
        {"name": "decode_2b", "kind": "decode", "layers": 24, "hidden": 2048, "ffn": 6144, "vocab": 248320,
         "heads": 8, "kv_heads": 2, "head_dim": 256, "rope_dim": 64, "key_heads": 16, "value_heads": 16, "tokens": 8},
        # The smallest model that is decoded here (the smoke test's): launches and latency only.
        {"name": "decode_small", "kind": "decode", "layers": 4, "hidden": 256, "ffn": 512, "vocab": 512,
         "heads": 2, "kv_heads": 1, "head_dim": 128, "rope_dim": 32, "key_heads": 2, "value_heads": 4, "tokens": 8},
        # Speculative decoding at 4B-class widths (a third of the layers), every logit on the host.
        {"name": "pairs_4b", "kind": "pairs", "layers": 8, "hidden": 2560, "ffn": 9728, "vocab": 248320,
         "heads": 16, "kv_heads": 4, "head_dim": 256, "rope_dim": 64, "key_heads": 16, "value_heads": 32, "tokens": 8},
        # The metric's product: one row of activations, the rows of an FFN gate.
        {"name": "gemv_q4k", "kind": "product", "type": "Q4_K", "rows": 6144, "cols": 2048, "tokens": 1, "host": False},
        # A host decoder that calls Projections::Apply stage by stage; mixed files hold Q5_K rows.
        {"name": "apply_host", "kind": "product", "type": "Q5_K", "rows": 2048, "cols": 2048, "tokens": 1, "host": True},
        # A draft and its alternatives, or four sequences: few rows against 4B-class weights.
        {"name": "layer_4", "kind": "layer", "hidden": 2560, "ffn": 9728, "key_heads": 16, "value_heads": 32,
         "vocab": 0, "tokens": 4},
        # The ragged verify batch: 32 sequences of one to four draft tokens, a layer and the LM head.
        {"name": "verify_79", "kind": "layer", "hidden": 2560, "ffn": 9728, "key_heads": 16, "value_heads": 32,
         "vocab": 248320, "tokens": 79},
        # A prompt's rows through a layer.
        {"name": "prompt_512", "kind": "layer", "hidden": 2560, "ffn": 9728, "key_heads": 16, "value_heads": 32,
         "vocab": 0, "tokens": 512},
        # Eight sequences of sixteen heads: the DeltaNet update by itself.
        {"name": "delta_rule_8", "kind": "rule", "sequences": 8, "key_heads": 16, "value_heads": 16, "head_dim": 128},
        # The mixer step of the verify batch: 32 sequences, one to four tokens each.
        {"name": "mixer_32", "kind": "mixer", "sequences": 32, "hidden": 2560, "key_heads": 16, "value_heads": 32,
         "most": 4},
        # A MoE layer at 35B-A3B-class shapes, four tokens.
        {"name": "moe_4", "kind": "moe", "hidden": 2048, "experts": 256, "used": 8, "expert_ffn": 512, "tokens": 4},
        # Attention with the default cache full: eight query heads on two KV heads.
        {"name": "attention_4096", "kind": "attention", "heads": 8, "kv_heads": 2, "head_dim": 256, "rope_dim": 64,
         "positions": 4096},
    ]


def _log(rng, low, high):
    """A whole number from low to high, even over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _blocks(rng, low, high):
    """The same in whole blocks of 256 values."""
    return 256 * _log(rng, low // 256, high // 256)


def draw(rng):
    kind = rng.choice(["decode", "decode", "pairs", "product", "product", "layer", "layer", "layer", "rule", "mixer",
                       "moe", "attention"])
    heads, kv_heads, head_dim, rope_dim = rng.choice([(2, 1, 128, 32), (8, 2, 256, 64), (16, 4, 256, 64), (4, 4, 64, 64)])
    key_heads, value_heads = rng.choice([(2, 4), (8, 8), (16, 16), (16, 32)])
    if kind in ("decode", "pairs"):
        hidden = _blocks(rng, 256, 2560)
        return {"kind": kind, "layers": rng.randint(4, 12), "hidden": hidden,
                "ffn": min(9728, 256 * max(1, round(hidden * rng.uniform(2.0, 4.0) / 256))),
                "vocab": _log(rng, 512, 152000), "heads": heads, "kv_heads": kv_heads, "head_dim": head_dim,
                "rope_dim": rope_dim, "key_heads": key_heads, "value_heads": value_heads, "tokens": 2 * rng.randint(2, 4)}
    if kind == "product":
        return {"kind": kind, "type": rng.choice(sorted(TYPES)), "rows": _log(rng, 128, 24576),
                "cols": _blocks(rng, 256, 9728), "tokens": rng.choice([1, 1, 2, 3, 4, 5, 8]),
                "host": rng.random() < 0.5}
    if kind == "layer":
        hidden = _blocks(rng, 1024, 2560)
        tokens = _log(rng, 1, 512)
        return {"kind": kind, "hidden": hidden, "ffn": min(9728, 256 * round(hidden * rng.uniform(2.0, 4.0) / 256)),
                "key_heads": key_heads, "value_heads": value_heads,
                # Nobody asks for the logits of a whole prompt.
                "vocab": rng.choice([0, _log(rng, 16384, 248320)]) if tokens <= 128 else 0, "tokens": tokens}
    if kind == "rule":
        return {"kind": kind, "sequences": _log(rng, 1, 48), "key_heads": key_heads, "value_heads": value_heads,
                "head_dim": rng.choice([64, 128, 128])}
    if kind == "mixer":
        return {"kind": kind, "sequences": _log(rng, 1, 48), "hidden": _blocks(rng, 1024, 2560), "key_heads": key_heads,
                "value_heads": value_heads, "most": rng.randint(1, 4)}
    if kind == "moe":
        return {"kind": kind, "hidden": _blocks(rng, 1024, 2560), "experts": rng.choice([64, 128, 256]),
                "used": rng.choice([4, 8]), "expert_ffn": rng.choice([256, 512]), "tokens": _log(rng, 1, 16)}
    return {"kind": "attention", "heads": heads, "kv_heads": kv_heads, "head_dim": head_dim, "rope_dim": rope_dim,
            "positions": _log(rng, 16, 16384)}


# ---- inputs ------------------------------------------------------------------------


class State:
    """What a case's program keeps between passes."""


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _rows(gen, n, width):
    """Activation rows: N(0, 1) with a log-normal scale per channel."""
    scale = torch.exp(0.5 * torch.randn(width, device=DEVICE, generator=gen))
    return torch.randn(n, width, device=DEVICE, generator=gen) * scale


def _packed(gen, name, rows, cols):
    """`rows` x `cols` weights as GGUF bytes on the device."""
    if name in ("Q4_K", "Q6_K"):
        chunks = [torch.randn(min(16384, rows - r), cols, device=DEVICE, generator=gen) * 0.02
                  for r in range(0, rows, 16384)]
        return torch.cat([Q.quantize(TYPES[name], w).reshape(-1) for w in chunks])
    # No quantizer is needed for these: any code bytes are valid beside small fp16 scales.
    per, size = Q.BLOCK_ELEMENTS[TYPES[name]], Q.BLOCK_BYTES[TYPES[name]]
    raw = torch.randint(0, 256, (rows * cols // per, size), device=DEVICE, generator=gen, dtype=torch.uint8)
    for at in ((0, 2) if name == "Q5_K" else (0,)):
        d = (1e-4 * (1.0 + torch.rand(raw.shape[0], device=DEVICE, generator=gen))).half()
        raw[:, at:at + 2] = d.view(torch.uint8).reshape(-1, 2)
    return raw.reshape(-1)


def _model(case, **more):
    return synth.ModelConfig(hidden=case["hidden"], linear_key_heads=case.get("key_heads", 16),
                             linear_value_heads=case.get("value_heads", 16), linear_head_dim=128, **more)


def _layer_model(case):
    return _model(case, layers=1, ffn=case["ffn"], vocab=case["vocab"] or 512)


def _decoder_model(case):
    return _model(case, **{k: case[k] for k in ("layers", "ffn", "vocab", "heads", "kv_heads", "head_dim", "rope_dim")})


def _mixer_counts(case):
    """How many tokens each sequence brings."""
    return [1 + i % case["most"] for i in range(case["sequences"])]


def prepare(case, seed):
    s = State()
    s.kind = case["kind"]
    s.case = case
    gen = _generator(seed)
    s.ctx = Context(0)
    globals()["_prepare_" + ("decode" if s.kind == "pairs" else s.kind)](s, case, gen, seed)
    return s


def _prepare_decode(s, case, gen, seed):
    cfg = _decoder_model(case)
    s.tensors = synth.build_model(cfg, seed=seed, device=DEVICE)
    torch.cuda.synchronize()
    s.projections = CudaProjections(s.ctx, cfg, s.tensors)
    s.decoder = CudaDecoder(s.projections, s.tensors, max_positions=4096)
    s.tokens = np.random.default_rng(seed).integers(0, case["vocab"], case["tokens"]).tolist()
    s.logits = torch.empty(case["vocab"]).pin_memory()


def _prepare_product(s, case, gen, seed):
    rows, cols, tokens = case["rows"], case["cols"], case["tokens"]
    s.raw = _packed(gen, case["type"], rows, cols)
    torch.cuda.synchronize()
    s.parts = [(s.ctx.matrix_from_device(TYPES[case["type"]], s.raw.data_ptr(), rows, cols), 0, rows)]
    x = _rows(gen, tokens, cols)
    if case["host"]:
        s.x = x.cpu().numpy()
    else:
        s.x, s.y = x, torch.empty(tokens, rows, device=DEVICE)
        s.parts_array = Context._parts(s.parts)


def _prepare_layer(s, case, gen, seed):
    cfg = _layer_model(case)
    s.tensors = synth.build_model(cfg, seed=seed, device=DEVICE)
    torch.cuda.synchronize()
    s.projections = CudaProjections(s.ctx, cfg, s.tensors)
    widths = {Stage.kLinearIn: cfg.hidden, Stage.kMixerOut: cfg.value_dim, Stage.kFfnIn: cfg.hidden,
              Stage.kFfnDown: cfg.ffn, Stage.kLmHead: cfg.hidden}
    s.stages = []
    for stage in LAYER_STAGES + ((Stage.kLmHead,) if case["vocab"] else ()):
        out = sum(p[2] for p in s.projections.parts(stage, 0))
        s.stages.append((stage, _rows(gen, case["tokens"], widths[stage]),
                         torch.empty(case["tokens"], out, device=DEVICE)))


def _prepare_rule(s, case, gen, seed):
    n, hk, hv, dk = case["sequences"], case["key_heads"], case["value_heads"], case["head_dim"]
    unit = torch.nn.functional.normalize

    def normal(*shape):
        return torch.randn(*shape, device=DEVICE, generator=gen)
    s.state = normal(n, hv, dk, dk) * 0.1
    s.y = torch.empty(n, hv, dk, device=DEVICE)
    q, k, v = unit(normal(n, hk, dk), dim=-1), unit(normal(n, hk, dk), dim=-1), normal(n, hv, dk)
    decay, beta = torch.exp(-torch.nn.functional.softplus(normal(n, hv))), torch.sigmoid(normal(n, hv))
    s.sequences = [dict(state=s.state[i], q=q[i], k=k[i], v=v[i], decay=decay[i], beta=beta[i], y=s.y[i])
                   for i in range(n)]


def _prepare_mixer(s, case, gen, seed):
    cfg = _model(case, layers=1, ffn=256, vocab=256)
    s.mixer = CudaMixer(s.ctx, cfg, synth.build_model(cfg, seed=seed, device=DEVICE))
    counts = _mixer_counts(case)
    n, rows = len(counts), sum(counts)

    def window():
        return torch.randn(n, cfg.conv_kernel - 1, cfg.conv_channels, device=DEVICE, generator=gen)
    into, h = _rows(gen, rows, cfg.conv_channels + cfg.value_dim + 2 * cfg.linear_value_heads), _rows(gen, rows, cfg.hidden)
    conv_in = window()
    ssm = torch.randn(n, s.mixer.ssm_values(), device=DEVICE, generator=gen) * 0.1
    s.outputs = [ssm, torch.zeros_like(ssm), window(), window(), torch.zeros(rows, cfg.value_dim, device=DEVICE)]
    _, spec, conv_out, conv_saved, y = s.outputs
    s.sequences, at = [], 0
    for i, tokens in enumerate(counts):   # the batch's rows are packed, a sequence's follow one another
        part = slice(at, at + tokens)
        s.sequences.append({"n_tokens": tokens, "in": into[part], "h": h[part], "conv_in": conv_in[i],
                            "conv_out": conv_out[i], "conv_saved": conv_saved[i], "ssm": ssm[i], "ssm_spec": spec[i],
                            "y": y[part]})
        at += tokens


def _prepare_moe(s, case, gen, seed):
    cfg = _model(case, layers=1, vocab=256, experts=case["experts"], experts_used=case["used"],
                 expert_ffn=case["expert_ffn"], shared_expert_ffn=case["expert_ffn"])
    s.tensors = synth.build_model(cfg, seed=seed, device=DEVICE)
    torch.cuda.synchronize()
    s.moe = CudaMoe(CudaProjections(s.ctx, cfg, s.tensors), max_tokens=case["tokens"])
    s.normed = torch.randn(case["tokens"], cfg.hidden, device=DEVICE, generator=gen)
    s.shared = torch.randn(case["tokens"], cfg.hidden, device=DEVICE, generator=gen)
    s.out = torch.empty_like(s.shared)


def _prepare_attention(s, case, gen, seed):
    heads, kv, hd, rope, n = (case[k] for k in ("heads", "kv_heads", "head_dim", "rope_dim", "positions"))
    s.keys = torch.randn(n, kv * hd, device=DEVICE, generator=gen).half()
    s.values = torch.randn(n, kv * hd, device=DEVICE, generator=gen).half()
    s.out = torch.empty(heads * hd, device=DEVICE)
    f32 = dict(dtype=torch.float32, device=DEVICE)
    s.keep = [torch.tensor([n - 1], dtype=torch.int32, device=DEVICE),
              torch.randn(2 * heads * hd + 2 * kv * hd, device=DEVICE, generator=gen),
              1.0 + 0.1 * torch.randn(hd, device=DEVICE, generator=gen),
              1.0 + 0.1 * torch.randn(hd, device=DEVICE, generator=gen),
              (1.0 / 1e7 ** (2.0 * torch.arange(rope // 2, device=DEVICE, dtype=torch.float64) / rope)).float(),
              s.keys, s.values, torch.empty(heads * hd, **f32),
              torch.empty(kv * 32 * (heads // kv) * (hd + 2), **f32), s.out]
    s.args = _capi.AttentionArgs(heads, kv, hd, rope, n, 1e-6, *[t.data_ptr() for t in s.keep])


# ---- one pass ------------------------------------------------------------------------


def run(state):
    return globals()["_run_" + state.kind](state)


def _run_decode(s):
    s.decoder.Reset()
    for token in s.tokens:
        s.decoder.Step(token, s.logits)
    return s.logits   # of the last token: they come from every step's states and cache rows


def _run_pairs(s):
    s.decoder.Reset()
    out = []
    for i in range(0, len(s.tokens), 2):
        out.append(s.decoder.StepTokens(s.tokens[i:i + 2]))
        s.decoder.Resolve(i % 4 == 0)   # every other draft is kept
    return out


def _run_product(s):
    if s.case["host"]:
        return s.ctx.matmul(s.parts, s.x, s.case["tokens"], s.case["rows"])
    s.ctx.matmul_device(s.parts_array, 1, s.x, s.case["tokens"], s.y)
    return s.y


def _run_layer(s):
    tokens = s.case["tokens"]
    for stage, x, y in s.stages:
        s.projections.apply_device(stage, 0, x, tokens, y)
    return [y for _, _, y in s.stages]


def _run_rule(s):
    s.ctx.delta_rule_device(s.sequences, s.case["key_heads"], s.case["value_heads"], s.case["head_dim"])
    return [s.state, s.y]


def _run_mixer(s):
    s.mixer.Run(0, s.sequences)
    return s.outputs


def _run_moe(s):
    s.moe.MoeFfn(0, s.normed, s.shared, s.case["tokens"], s.out)
    return {"out": s.out, "chosen": s.moe.chosen, "weights": s.moe.weights}


def _run_attention(s):
    s.ctx._check(s.ctx.lib.gufo_cuda_attention_device(s.ctx.handle, C.byref(s.args)))
    return [s.out, s.keys, s.values]


# ---- what a pass cannot do without, and how exact it is -------------------------------


def _layer_matrices(cfg, attention):
    """(GGUF type, rows, cols) of a layer's products."""
    p, d = cfg.proj_type, cfg.down_type
    if attention:
        q, kv = cfg.heads * cfg.head_dim, cfg.kv_heads * cfg.head_dim
        mixer = [(p, 2 * q + 2 * kv, cfg.hidden), (p, cfg.hidden, q)]
    else:
        mixer = [(p, cfg.conv_channels + cfg.value_dim, cfg.hidden), (Q.GGML_F32, 2 * cfg.linear_value_heads, cfg.hidden),
                 (p, cfg.hidden, cfg.value_dim)]
    return mixer + [(p, 2 * cfg.ffn, cfg.hidden), (d, cfg.hidden, cfg.ffn)]


def _products(matrices, tokens):
    """Bytes (weights, inputs and outputs once) and operations of products with `tokens` rows."""
    nbytes = sum(rows * Q.row_bytes(t, cols) + 4 * tokens * (rows + cols) for t, rows, cols in matrices)
    return nbytes, sum(2 * tokens * rows * cols for _, rows, cols in matrices)


def work(case):
    kind = case["kind"]
    if kind in ("decode", "pairs"):
        cfg = _decoder_model(case)
        at_once = 2 if kind == "pairs" else 1
        matrices = [(cfg.embed_type, cfg.vocab, cfg.hidden)]
        state = 0
        for il in range(cfg.layers):
            attention = cfg.is_full_attention(il)
            matrices += _layer_matrices(cfg, attention)
            # The DeltaNet state is read and written once a step; the cache of so short a text is nothing.
            state += 0 if attention else 2 * 4 * cfg.value_dim * cfg.linear_head_dim
        nbytes, flops = _products(matrices, at_once)
        steps = case["tokens"] // at_once
        return {"bytes": steps * (nbytes + state), "flops": steps * flops}
    if kind == "product":
        nbytes, flops = _products([(TYPES[case["type"]], case["rows"], case["cols"])], case["tokens"])
        return {"bytes": nbytes, "flops": flops}
    if kind == "layer":
        cfg = _layer_model(case)
        matrices = _layer_matrices(cfg, False) + ([(cfg.embed_type, cfg.vocab, cfg.hidden)] if case["vocab"] else [])
        nbytes, flops = _products(matrices, case["tokens"])
        return {"bytes": nbytes, "flops": flops}
    if kind == "rule":
        hk, hv, dk = case["key_heads"], case["value_heads"], case["head_dim"]
        return {"bytes": case["sequences"] * 4 * (2 * hv * dk * dk + 2 * hk * dk + 2 * hv * dk + 2 * hv),
                "flops": case["sequences"] * 7 * hv * dk * dk}
    if kind == "mixer":
        cfg = _model(case, layers=1, ffn=256, vocab=256)
        counts = _mixer_counts(case)
        ssm, conv = cfg.value_dim * cfg.linear_head_dim, (cfg.conv_kernel - 1) * cfg.conv_channels
        row = cfg.conv_channels + 2 * cfg.value_dim + cfg.hidden
        # One token: the state in and out; more: in, out before the draft, out after it, two windows.
        return {"bytes": 4 * sum(ssm * (2 if n == 1 else 3) + conv * (2 if n == 1 else 3) + n * row for n in counts)
                + 4 * (2 * cfg.linear_value_heads * cfg.hidden + cfg.conv_channels * cfg.conv_kernel),
                "flops": sum(n * (7 * ssm + 4 * cfg.linear_value_heads * cfg.hidden) for n in counts)}
    if kind == "moe":
        hidden, ef, e, n = case["hidden"], case["expert_ffn"], case["experts"], case["tokens"]
        apart = e * (1.0 - (1.0 - case["used"] / e) ** n)   # experts that some token chose, expected
        expert = 2 * ef * Q.row_bytes(Q.GGML_Q4_K, hidden) + hidden * Q.row_bytes(Q.GGML_Q4_K, ef)
        return {"bytes": apart * expert + 4 * (e + 1) * hidden + 4 * n * 3 * hidden,
                "flops": 2 * n * (case["used"] * 3 * ef * hidden + (e + 1) * hidden)}
    heads, kv, hd, n = (case[k] for k in ("heads", "kv_heads", "head_dim", "positions"))
    return {"bytes": 2 * 2 * n * kv * hd + 4 * (3 * heads * hd + 2 * kv * hd), "flops": 4 * n * heads * hd}


def tolerance(case):
    kind = case["kind"]
    if kind in ("decode", "pairs"):
        # fp32 sums through every layer; keys and values rounded to fp16 on the way into the cache.
        return {"rel": 2e-4}
    if kind == "layer" and case["tokens"] > 16:
        # Many rows go through the fp16 tensor cores, weights and activations rounded to 11 bits.
        return {"rel": 1e-3}
    return {"rel": 1e-5}
