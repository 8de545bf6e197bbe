"""Performance cases of the fixed-point operators.

A case is one call (or one decode step) a program built on ``fxpr_vllm`` makes, through the public
operators: what vLLM's plugin hooks call per layer (GEMM, paged attention, RMSNorm), the sampler's
log-softmax, the casts, and an eager decode step of the random-init decoder.  Geometry and value
distributions are those of the repository's benchmark configurations; ``draw`` spreads the same
kinds of calls over the sizes a serving program meets between them.
"""
from __future__ import annotations

import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.abspath("vllm-triton-fixed-point-reductions_b200"))

from fxpr_vllm import _lib as fxp  # noqa: E402
from fxpr_vllm import library_ops as ops  # noqa: E402
from fxpr_vllm.llama_decoder import DecoderConfig, LlamaDecoder, LocalGroup  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}
PAGE = 16
FRAC_BITS = 16


def listed():
    return [
        # Q-format encode and decode of an activation: the casts as stand-alone operators
        dict(name="casts_2048x4096", kind="casts", n=2048 * 4096, dtype="fp32", int_bits=64),
        # residual add + RMSNorm in front of a layer, a batch of 2048 tokens
        dict(name="rms_norm_2048x4096", kind="rms_norm", rows=2048, hidden=4096, dtype="fp32", residual=True),
        # log-probabilities of 256 sampled rows over the whole vocabulary
        dict(name="log_softmax_256x128256", kind="log_softmax", rows=256, cols=128256, dtype="fp32"),
        # a projection for a handful of decoding sequences: the smallest call of a layer
        dict(name="gemm_16x4096x4096", kind="gemm", m=16, n=4096, k=4096, dtype="bf16", int_bits=32, k_tile=0,
             bias=False),
        # gate/up projection of a full decode batch: bound by reading the weights
        dict(name="gemm_64x28672x4096", kind="gemm", m=64, n=28672, k=4096, dtype="bf16", int_bits=64, k_tile=0,
             bias=False),
        # QKV projection with bias of one ragged prefill chunk, fp16
        dict(name="gemm_333x6144x4096_bias", kind="gemm", m=333, n=6144, k=4096, dtype="fp16", int_bits=32,
             k_tile=0, bias=True),
        # the headline GEMM: K-tiles of 64
        dict(name="gemm_4096x4096x4096_kt64", kind="gemm", m=4096, n=4096, k=4096, dtype="bf16", int_bits=64,
             k_tile=64, bias=False),
        # an FFN projection of a long prefill batch at the operators' own K-tile
        dict(name="gemm_8192x14336x4096", kind="gemm", m=8192, n=14336, k=4096, dtype="bf16", int_bits=64,
             k_tile=0, bias=False),
        # decode attention of a few short conversations: latency
        dict(name="decode_attn_5", kind="attention", phase="decode", requests=5, lo=40, hi=700, lens_seed=1,
             q_heads=32, kv_heads=8, head_dim=128, dtype="fp16", int_bits=32, window=0, softcap=0.0),
        # decode attention of a full batch with contexts of 512 to 8192 tokens
        dict(name="decode_attn_64", kind="attention", phase="decode", requests=64, lo=512, hi=8192, lens_seed=3,
             q_heads=32, kv_heads=8, head_dim=128, dtype="bf16", int_bits=64, window=0, softcap=0.0),
        # causal prefill of 16 prompts of 128 to 4096 tokens in one call
        dict(name="prefill_attn_16", kind="attention", phase="prefill", requests=16, lo=128, hi=4096, lens_seed=4,
             q_heads=32, kv_heads=8, head_dim=128, dtype="bf16", int_bits=64, window=0, softcap=0.0),
        # one decode step of a four-layer decoder, launched operator by operator
        dict(name="decoder_step_64", kind="decoder", layers=4, batch=64, context=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_gemm(rng):
    """Rows of any batch, from one sequence to a long prefill; weights of a whole layer, of a
    tensor-parallel shard of one, or of another model's (multiples of 8, ragged against the tiles)."""
    if rng.random() < 0.5:
        n, k = rng.choice([(4096, 4096), (6144, 4096), (28672, 4096), (4096, 14336), (14336, 4096),
                           (768, 4096), (3584, 4096), (4096, 512), (4096, 1792)])
    else:
        n, k = 8 * _log(rng, 32, 1792), 8 * _log(rng, 32, 1024)
    dtype = rng.choice(["bf16", "bf16", "bf16", "bf16", "fp16", "fp16", "fp32"])
    # up to the largest listed product; fp32 (an accuracy check of a model) only with short batches
    top = 8192 * 14336 * 4096 if dtype != "fp32" else 512 * 4096 * 4096
    m = _log(rng, 1, max(1, min(8192 if dtype != "fp32" else 512, top // (n * k))))
    return dict(kind="gemm", m=m, n=n, k=k, dtype=dtype, int_bits=rng.choice([32, 64]),
                k_tile=rng.choice([0, 0, 64]), bias=rng.random() < 0.3)


def _draw_attention(rng):
    phase = rng.choice(["decode", "decode", "prefill", "chunk"])
    q_heads, kv_heads = rng.choice([(32, 8), (32, 8), (16, 4), (8, 2), (4, 1), (32, 32)])
    head_dim = rng.choice([128, 128, 128, 64])
    most = 64 if phase == "decode" else 16
    longest = 8192 if phase == "decode" else 4096
    if kv_heads == 32 or (head_dim == 64 and phase != "decode"):
        most //= 4          # no dearer than the largest listed batch of its phase
    hi = _log(rng, 32, longest)
    return dict(kind="attention", phase=phase, requests=_log(rng, 1, most), lo=max(1, hi // rng.choice([1, 4, 16])),
                hi=hi, lens_seed=rng.randrange(1 << 20), q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim,
                dtype=rng.choice(["bf16", "bf16", "fp16"]), int_bits=rng.choice([32, 64]),
                window=rng.choice([0, 0, 0, 1024]), softcap=rng.choice([0.0, 0.0, 0.0, 50.0]))


def draw(rng):
    kind = rng.choice(["casts", "rms_norm", "log_softmax", "gemm", "gemm", "gemm", "gemm", "attention", "attention",
                       "attention", "decoder"])
    if kind == "gemm":
        return _draw_gemm(rng)
    if kind == "attention":
        return _draw_attention(rng)
    if kind == "casts":
        return dict(kind=kind, n=_log(rng, 1000, 1 << 25), dtype=rng.choice(["fp32", "fp32", "fp16"]),
                    int_bits=rng.choice([16, 32, 64]))
    if kind == "rms_norm":
        hidden = rng.choice([4096, 4096, 8 * _log(rng, 64, 1024), _log(rng, 500, 8192)])
        return dict(kind=kind, rows=_log(rng, 1, 8192), hidden=hidden, dtype=rng.choice(["bf16", "fp16", "fp32"]),
                    residual=rng.random() < 0.7)
    if kind == "log_softmax":
        return dict(kind=kind, rows=_log(rng, 1, 256), cols=rng.choice([128256, 128256, 32000, _log(rng, 1000, 128256)]),
                    dtype=rng.choice(["fp32", "fp32", "bf16"]))
    return dict(kind="decoder", layers=rng.randint(1, 4), batch=_log(rng, 1, 64), context=_log(rng, 16, 1024))


def _lengths(case):
    """(query length, key length) of every request."""
    rng = random.Random(case["lens_seed"])
    keys = [rng.randint(case["lo"], case["hi"]) for _ in range(case["requests"])]
    if case["phase"] == "decode":
        return [(1, s) for s in keys]
    if case["phase"] == "prefill":
        return [(s, s) for s in keys]
    # chunked prefill: some requests decode, the others have a part of their keys cached already
    return [(1 if rng.random() < 0.3 else rng.randint(1, s), s) for s in keys]


def _visible(case):
    """Query-key pairs that causality and the window leave, and the keys some query can see."""
    pairs = seen = 0
    w = case["window"]
    for q, s in _lengths(case):
        first = s - q + 1                       # keys the first query sees without a window
        full = (first + s) * q // 2
        if w:
            lo = max(first, w)
            over = (lo - w + s - w) * (s - lo + 1) // 2 if s >= lo else 0
            pairs += full - over
            seen += s - max(0, first - w)
        else:
            pairs += full
            seen += s
    return pairs, seen


def _prepare_attention(case, g):
    dtype, dev = DTYPES[case["dtype"]], torch.device("cuda")
    lens = _lengths(case)
    pages = [-(-s // PAGE) for _, s in lens]
    kv = torch.randn((sum(pages) + 1, 2, PAGE, case["kv_heads"], case["head_dim"]), generator=g, device=dev, dtype=dtype)
    order = torch.randperm(sum(pages), generator=g, device=dev).to(torch.int32) + 1
    table = torch.zeros((len(lens), max(pages)), dtype=torch.int32, device=dev)
    at = 0
    for i, p in enumerate(pages):
        table[i, :p] = order[at:at + p]
        at += p
    starts = [0]
    for q, _ in lens:
        starts.append(starts[-1] + q)
    q = torch.randn((starts[-1], case["q_heads"], case["head_dim"]), generator=g, device=dev, dtype=dtype)
    return dict(q=q, kv=kv, o=torch.empty_like(q), qsl=torch.tensor(starts, dtype=torch.int32, device=dev),
                lens=torch.tensor([s for _, s in lens], dtype=torch.int32, device=dev), table=table,
                max_q=max(q for q, _ in lens))


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(int(seed))
    kind = case["kind"]
    s = dict(case=case)
    if kind == "attention":
        return dict(s, **_prepare_attention(case, g))
    if kind == "decoder":
        b, length = case["batch"], case["context"]
        model = LlamaDecoder(DecoderConfig(layers=case["layers"]), LocalGroup(1), dev, seed=int(seed), max_seqs=b,
                             max_len=length + 1)
        prompts = torch.randint(0, model.cfg.vocab, (b, length), generator=g, device=dev)
        tokens = model.greedy(model.prefill(prompts))
        return dict(s, model=model, tokens=tokens)
    dtype = DTYPES[case["dtype"]]
    if kind == "casts":
        x = 50.0 * torch.randn(case["n"], generator=g, device=dev)
        return dict(s, x=x.to(dtype), q=torch.round(x * (64.0 if case["int_bits"] == 16 else 65536.0)).to(
            getattr(torch, "int%d" % case["int_bits"])))
    if kind == "rms_norm":
        shape = (case["rows"], case["hidden"])
        return dict(s, x=torch.randn(shape, generator=g, device=dev).to(dtype),
                    r=torch.randn(shape, generator=g, device=dev).to(dtype) if case["residual"] else None,
                    w=(1.0 + 0.1 * torch.randn(case["hidden"], generator=g, device=dev)).to(dtype))
    if kind == "log_softmax":
        return dict(s, x=(2.0 * torch.randn((case["rows"], case["cols"]), generator=g, device=dev)).to(dtype))
    a = torch.randn((case["m"], case["k"]), generator=g, device=dev).to(dtype)
    b = (0.02 * torch.randn((case["k"], case["n"]), generator=g, device=dev)).to(dtype)
    bias = torch.randn(case["n"], generator=g, device=dev).to(dtype) if case["bias"] else None
    return dict(s, a=a, b=b, bias=bias)


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "gemm":
        if c["k_tile"]:
            with fxp.overrides(gemm_k_tile=c["k_tile"]):
                return ops.gemm_fxp(s["a"], s["b"], s["bias"], c["int_bits"], FRAC_BITS)
        return ops.gemm_fxp(s["a"], s["b"], s["bias"], c["int_bits"], FRAC_BITS)
    if kind == "attention":
        ops.unified_attention_fxp(s["q"], s["kv"], s["o"], s["qsl"], s["lens"], s["table"], s["max_q"], None, True,
                                  None, c["int_bits"], FRAC_BITS, c["softcap"], c["window"], 0)
        return s["o"]
    if kind == "decoder":
        model = s["model"]
        logits = model.decode_step(s["tokens"], c["context"])
        return dict(logits=logits, kv=model.shards[0].kv_cache)
    if kind == "rms_norm":
        if s["r"] is None:
            return ops.rms_norm_fxp(s["x"], s["w"], 1e-6)
        # the residual accumulates from pass to pass, as it does from layer to layer
        return ops.rms_norm_fxp_residual(s["x"], s["r"], s["w"], 1e-6), s["r"]
    if kind == "log_softmax":
        return ops.log_softmax_fxp(s["x"], FRAC_BITS)
    frac = 8 if c["int_bits"] == 16 else FRAC_BITS
    return (ops.float_to_fixed(s["x"], c["int_bits"], frac),
            ops.fixed_to_float(s["q"], 16 if c["dtype"] == "fp16" else 32, frac))


def work(case):
    kind = case["kind"]
    if kind == "decoder":
        cfg = DecoderConfig()
        weights = case["layers"] * (cfg.hidden * (cfg.q_heads + 2 * cfg.kv_heads) * cfg.head_dim
                                    + cfg.q_heads * cfg.head_dim * cfg.hidden + 3 * cfg.hidden * cfg.ffn)
        weights += cfg.hidden * cfg.vocab
        keys = case["batch"] * (case["context"] + 1) * case["layers"]
        return {"bytes": 2 * weights + keys * 2 * cfg.kv_heads * cfg.head_dim * 2 + 2 * case["batch"] * cfg.vocab,
                "flops": 2 * case["batch"] * weights + 4 * keys * cfg.q_heads * cfg.head_dim}
    size = SIZE[case["dtype"]]
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": size * (m * k + k * n + m * n + (n if case["bias"] else 0)), "flops": 2 * m * n * k}
    if kind == "attention":
        pairs, seen = _visible(case)
        rows = sum(q for q, _ in _lengths(case)) * case["q_heads"] * case["head_dim"]
        return {"bytes": size * (seen * 2 * case["kv_heads"] * case["head_dim"] + 2 * rows),
                "flops": 4 * pairs * case["q_heads"] * case["head_dim"]}
    if kind == "casts":
        return {"bytes": 2 * case["n"] * (size + case["int_bits"] // 8), "flops": 2 * case["n"]}
    if kind == "rms_norm":
        return {"bytes": size * case["hidden"] * (case["rows"] * (4 if case["residual"] else 2) + 1),
                "flops": 4 * case["rows"] * case["hidden"]}
    return {"bytes": case["rows"] * case["cols"] * (size + 4), "flops": 4 * case["rows"] * case["cols"]}


def tolerance(case):
    """Casts, RMSNorm and log-softmax are defined operation by operation, so their bits are fixed.
    Behind a matrix product only the fp32 sum inside one K-tile (or key tile) may be taken in
    another order; the outputs are rounded to the io type."""
    if case["kind"] in ("casts", "rms_norm", "log_softmax"):
        return "exact"
    if case["kind"] == "decoder":
        return {"rel": 1e-2, "max": 0.1}
    return {"rel": {"bf16": 4e-3, "fp16": 5e-4, "fp32": 1e-5}[case["dtype"]],
            "max": {"bf16": 2e-2, "fp16": 4e-3, "fp32": 1e-3}[case["dtype"]]}
