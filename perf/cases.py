"""Performance cases of the attention path: what a user of the package has it do, with sizes and input makers.

A case is one of three kinds, and every kind goes through `KernelBackend("torch_ext")`:

  decode   one generated token per sequence: (optionally) `rope_kv_append*`, then `flash_attn_decode*`,
           for `layers` layers with caches of their own; the cache is 16-bit, GGML Q8_0 or paged.  With
           `graph` the step is replayed from a CUDA graph, as `apps/generate.py --cuda-graph` does.
  prefill  a prompt, or a chunk of one behind `seq_k - seq_q` keys that are cached already: (optionally)
           `rope_kv_append`, then `flash_attn_causal`
  masked   the dense bool mask entry `flash_attn` on [B, L, H, D] storage seen as [B, H, L, D]: a causal
           mask (`window` 0) or a two-sided sliding window

Run from the repository's root.
"""
import math
import os
import sys

import torch

_PKG = os.path.abspath("minfer-python_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from minfer.const import GGML_QUANT_SIZES, GGMLQuantizationType  # noqa: E402
from minfer.kernels import KernelBackend  # noqa: E402

_KERNS = KernelBackend("torch_ext")
_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
_ROPE_THETA = 500000.0


def _decode(name, batch, heads, kv_heads, head_dim, dtype, cache, len_lo, len_hi, max_len, append=True, style=0,
            page=0, layers=1, graph=False):
    return {"name": name, "kind": "decode", "batch": batch, "heads": heads, "kv_heads": kv_heads, "head_dim": head_dim,
            "dtype": dtype, "cache": cache, "len_lo": len_lo, "len_hi": len_hi, "max_len": max_len, "append": append,
            "style": style, "page": page, "layers": layers, "graph": graph}


def _prefill(name, batch, heads, kv_heads, head_dim, dtype, seq_q, seq_k, append=False, style=0):
    return {"name": name, "kind": "prefill", "batch": batch, "heads": heads, "kv_heads": kv_heads, "head_dim": head_dim,
            "dtype": dtype, "seq_q": seq_q, "seq_k": seq_k, "append": append, "style": style}


def _masked(name, batch, heads, kv_heads, head_dim, dtype, seq, window):
    return {"name": name, "kind": "masked", "batch": batch, "heads": heads, "kv_heads": kv_heads, "head_dim": head_dim,
            "dtype": dtype, "seq": seq, "window": window}


def listed():
    return [
        # one user chatting with an 8B-shaped model, eager: one layer's share of a token, all launch latency
        _decode("decode_chat", 1, 32, 8, 128, "bf16", "plain", 777, 777, 4096),
        # the end-to-end configuration's token step (16 layers, 8 sequences of 512 + 128), replayed from a graph
        _decode("decode_graph_16_layers", 8, 32, 8, 64, "fp16", "plain", 513, 640, 640, layers=16, graph=True),
        # a serving batch of ragged sequences over a padded cache, attention alone: the decode benchmark's shape
        _decode("decode_batch64", 64, 32, 8, 128, "fp16", "plain", 512, 8192, 8192, append=False),
        # a serving step over a paged cache, two-halves rotation, bfloat16
        _decode("decode_paged", 24, 64, 8, 128, "bf16", "paged", 100, 6000, 6016, style=1, page=64),
        # a serving step over a quantised cache
        _decode("decode_q8", 64, 32, 8, 128, "fp16", "q8", 512, 8192, 8192),
        # a short question to an 8B-shaped model: one layer of its prompt
        _prefill("prompt_short", 1, 32, 8, 128, "bf16", 77, 77, append=True),
        # the end-to-end configuration's prompts: one layer
        _prefill("prompt_batch8_d64", 8, 32, 8, 64, "fp16", 512, 512, append=True),
        # chunked prefill: the last 1000 tokens of a 16 k document behind what is cached already
        _prefill("prompt_chunk", 1, 32, 8, 128, "bf16", 1000, 16000, append=True, style=1),
        # the prefill benchmark's shape
        _prefill("prefill_l4096", 4, 32, 8, 128, "fp16", 4096, 4096),
        # long context: the largest call
        _prefill("prefill_l32768", 1, 64, 8, 128, "bf16", 32768, 32768),
        # the dense-mask entry at the benchmark's heads with a sequence that fills no tile: causal mask
        _masked("mask_causal_l1999", 4, 48, 8, 128, "fp16", 1999, 0),
        # the dense-mask entry with a sliding window
        _masked("mask_window_l4096", 4, 48, 8, 128, "fp16", 4096, 256),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


_HEADS = ((32, 8), (32, 8), (64, 8), (48, 8), (24, 8), (16, 16), (8, 1))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "prefill", "prefill", "masked"))
    heads, kv_heads = rng.choice(_HEADS)
    head_dim = rng.choice((64, 128, 128))
    dtype = rng.choice(("fp16", "bf16"))
    style = rng.randrange(2)
    if kind == "decode":
        graph = rng.random() < 0.25
        layers = rng.choice((4, 8, 16)) if graph else 1
        cache = rng.choice(("plain", "plain", "q8", "paged"))
        batch = _log_int(rng, 1, 128)
        # at most 2 GiB of cached keys and values (16-bit) in all layers
        most = (2 << 30) // (batch * kv_heads * head_dim * 4 * layers)
        len_hi = min(_log_int(rng, 48, 16384), max(48, most))
        len_lo = max(1, round(len_hi * rng.choice((0.05, 0.3, 1.0))))
        page = rng.choice((16, 64, 256)) if cache == "paged" else 0
        unit = page or 4
        max_len = -(-round(len_hi * rng.choice((1.0, 1.0, 1.5))) // unit) * unit
        case = _decode("", batch, heads, kv_heads, head_dim, dtype, cache, len_lo, len_hi, max_len, rng.random() < 0.6,
                       style, page, layers, graph)
    elif kind == "prefill":
        seq_k = _log_int(rng, 16, 32768)
        seq_q = seq_k if rng.random() < 0.7 else max(1, round(seq_k * rng.uniform(0.02, 0.5)))
        batch = _log_int(rng, 1, 16)
        # at most 8 TFLOP and 64 k new tokens
        while batch > 1 and (4 * batch * heads * head_dim * _pairs(seq_q, seq_k) > 8e12 or batch * seq_k > 65536):
            batch -= 1
        case = _prefill("", batch, heads, kv_heads, head_dim, dtype, seq_q, seq_k, rng.random() < 0.4, style)
    else:
        seq = _log_int(rng, 32, 8192)
        batch = min(_log_int(rng, 1, 8), max(1, (1 << 28) // (seq * seq)))
        case = _masked("", batch, heads, kv_heads, head_dim, dtype, seq, rng.choice((0, 0, 64, 256, 1000)))
    del case["name"]
    return case


def _pairs(seq_q, seq_k):
    """Visible (query, key) pairs of a causal call."""
    return seq_q * (seq_k - seq_q) + seq_q * (seq_q + 1) // 2


def _visible(case):
    if case["kind"] == "prefill":
        return _pairs(case["seq_q"], case["seq_k"])
    n, w = case["seq"], min(case["window"], case["seq"]) - 1    # |i - j| < window
    return n * (n + 1) // 2 if case["window"] == 0 else n * (2 * w + 1) - w * (w + 1)


def _lengths(case):
    """The batch's cache lengths after this token: evenly spread, so that a case's work does not hang on the seed."""
    n, lo, hi = case["batch"], case["len_lo"], case["len_hi"]
    return [hi] if n == 1 else [lo + (hi - lo) * i // (n - 1) for i in range(n)]


def work(case):
    h, g, d = case["heads"], case["kv_heads"], case["head_dim"]
    b = case["batch"]
    if case["kind"] == "decode":
        total = sum(_lengths(case))
        row = d // 32 * 34 if case["cache"] == "q8" else 2 * d
        per = 2 * g * row * total + 4 * b * h * d            # cached keys and values, q, out
        if case["append"]:
            per += 2 * b * h * d + 4 * b * g * d             # q written back, the new k and v
        return {"bytes": case["layers"] * per, "flops": case["layers"] * 4 * h * d * total}
    flops = 4 * b * h * d * _visible(case)
    if case["kind"] == "masked":
        n = case["seq"]
        return {"bytes": 4 * b * n * d * (h + g) + b * n * n, "flops": flops}
    lq, lk = case["seq_q"], case["seq_k"]
    moved = 4 * b * d * (h * lq + g * lk)                    # q, out, keys, values
    if case["append"]:
        moved += 2 * b * d * (h * lq + 2 * g * lq)           # q written back, the new k and v
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    # the output is a 16-bit value, and the weights take that type as well before they meet the values
    tol = {"rel": 2e-3} if case["dtype"] == "fp16" else {"rel": 1e-2}
    if case.get("cache") == "q8":
        tol["differ"] = 1e-3                                 # quantised keys: a rounding tie may fall either way
    return tol


class _Draws:
    def __init__(self, case, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.dtype = _DTYPES[case["dtype"]]

    def normal(self, *dims, dtype=None):
        return torch.randn(*dims, generator=self.gen, device="cuda", dtype=dtype or self.dtype)

    def permutation(self, n):
        return torch.randperm(n, generator=self.gen, device="cuda")


def _q8_rows(draws, batch, kv_heads, max_len, head_dim):
    """A GGML Q8_0 cache of normal values: blocks of 32 int8 behind one fp16 scale."""
    cache = torch.empty(batch, kv_heads, max_len, head_dim // 32, 34, dtype=torch.uint8, device="cuda")
    for b in range(batch):
        x = draws.normal(kv_heads, max_len, head_dim // 32, 32, dtype=torch.float32)
        d = x.abs().amax(-1, keepdim=True) / 127
        cache[b, ..., :2] = d.half().view(torch.uint8)
        cache[b, ..., 2:] = torch.round(x / d).to(torch.int8).view(torch.uint8)
    return cache.view(batch, kv_heads, max_len, head_dim // 32 * 34)


def _split_qkv(qkv, case):
    """The fused projection's output [B, L, (H + 2 Hkv) D] as q, k, v views [B, L, heads, D]."""
    b, n, _ = qkv.shape
    h, g, d = case["heads"], case["kv_heads"], case["head_dim"]
    return (qkv[..., :h * d].view(b, n, h, d), qkv[..., h * d:(h + g) * d].view(b, n, g, d),
            qkv[..., (h + g) * d:].view(b, n, g, d))


def _prepare_decode(case, seed):
    draws = _Draws(case, seed)
    b, h, g, d = case["batch"], case["heads"], case["kv_heads"], case["head_dim"]
    lens = torch.tensor(_lengths(case), dtype=torch.int32, device="cuda")[draws.permutation(b)].contiguous()
    state = {"case": case, "lens": lens, "start": lens - 1, "layers": []}
    if case["cache"] == "paged":
        per_seq = case["max_len"] // case["page"]
        state["table"] = draws.permutation(b * per_seq).to(torch.int32).view(b, per_seq)
    qkv = draws.normal(case["layers"], b, 1, (h + 2 * g) * d)
    state["out"] = torch.zeros(case["layers"], b, 1, h, d, dtype=draws.dtype, device="cuda")
    for i in range(case["layers"]):
        if case["cache"] == "q8":
            caches = [_q8_rows(draws, b, g, case["max_len"], d) for _ in range(2)]
        elif case["cache"] == "paged":
            caches = [draws.normal(b * per_seq, g, case["page"], d) for _ in range(2)]
        else:
            caches = [draws.normal(b, g, case["max_len"], d) for _ in range(2)]
        state["layers"].append((*_split_qkv(qkv[i], case), *caches, state["out"][i]))
    state["graph"] = None
    if case["graph"]:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _decode_step(state)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            _decode_step(state)
        state["graph"] = graph
    return state


def _decode_step(state):
    case, lens, start = state["case"], state["lens"], state["start"]
    rot, style = case["head_dim"], case["style"]
    for q, k, v, k_cache, v_cache, out in state["layers"]:
        qt, ot = q.transpose(1, 2), out.transpose(1, 2)
        if case["cache"] == "q8":
            if case["append"]:
                _KERNS.rope_kv_append_q8(rot, _ROPE_THETA, style, q, k, v, k_cache, v_cache, start)
            _KERNS.flash_attn_decode_q8(qt, k_cache, v_cache, lens, ot)
        elif case["cache"] == "paged":
            if case["append"]:
                _KERNS.rope_kv_append_paged(rot, _ROPE_THETA, style, q, k, v, k_cache, v_cache, state["table"], start)
            _KERNS.flash_attn_decode_paged(qt, k_cache, v_cache, state["table"], lens, ot)
        else:
            if case["append"]:
                _KERNS.rope_kv_append(rot, _ROPE_THETA, style, q, k, v, k_cache, v_cache, start)
            _KERNS.flash_attn_decode(qt, k_cache, v_cache, lens, ot)


def _prepare_prefill(case, seed):
    draws = _Draws(case, seed)
    b, h, g, d = case["batch"], case["heads"], case["kv_heads"], case["head_dim"]
    lq, lk = case["seq_q"], case["seq_k"]
    state = {"case": case, "k_cache": draws.normal(b, g, lk, d), "v_cache": draws.normal(b, g, lk, d)}
    if case["append"]:
        state["q"], state["k"], state["v"] = _split_qkv(draws.normal(b, lq, (h + 2 * g) * d), case)
        state["start"] = torch.full((b,), lk - lq, dtype=torch.int32, device="cuda")
        state["out"] = torch.zeros(b, lq, h, d, dtype=draws.dtype, device="cuda").transpose(1, 2)
    else:
        state["q"] = draws.normal(b, h, lq, d)
        state["out"] = torch.zeros_like(state["q"])
    return state


def _run_prefill(s):
    case, q = s["case"], s["q"]
    if case["append"]:
        _KERNS.rope_kv_append(case["head_dim"], _ROPE_THETA, case["style"], q, s["k"], s["v"], s["k_cache"],
                              s["v_cache"], s["start"])
        q = q.transpose(1, 2)
    _KERNS.flash_attn_causal(q, s["k_cache"], s["v_cache"], s["out"])


def _prepare_masked(case, seed):
    draws = _Draws(case, seed)
    b, n, h, g, d = case["batch"], case["seq"], case["heads"], case["kv_heads"], case["head_dim"]
    at = torch.arange(n, device="cuda")
    dist = at[None, :] - at[:, None]
    seen = dist <= 0 if case["window"] == 0 else dist.abs() < case["window"]
    return {"case": case,
            "q": draws.normal(b, n, h, d).transpose(1, 2), "k": draws.normal(b, n, g, d).transpose(1, 2),
            "v": draws.normal(b, n, g, d).transpose(1, 2), "mask": seen.expand(b, 1, n, n).contiguous(),
            "out": torch.zeros(b, h, n, d, dtype=draws.dtype, device="cuda"),
            "quant": (GGMLQuantizationType.F16, *GGML_QUANT_SIZES[GGMLQuantizationType.F16])}


def prepare(case, seed):
    return {"decode": _prepare_decode, "prefill": _prepare_prefill, "masked": _prepare_masked}[case["kind"]](case, seed)


def run(state):
    case = state["case"]
    if case["kind"] == "masked":
        _KERNS.flash_attn(*state["quant"], state["q"], state["k"], state["v"], state["mask"], state["out"])
        return state["out"]
    if case["kind"] == "prefill":
        _run_prefill(state)
        return (state["out"], state["q"], state["k_cache"], state["v_cache"]) if case["append"] else state["out"]
    if state["graph"] is not None:
        state["graph"].replay()
    else:
        _decode_step(state)
    if not case["append"]:
        return state["out"]
    # what the step wrote: the outputs, the rotated queries, the caches
    return state["out"], [x for q, _, _, kc, vc, _ in state["layers"] for x in (q, kc, vc)]
