"""The work that users of this library have it do, as cases that can be timed.

Shapes are the library's own: 24 query heads over 4 KV heads of 256, 16 full-attention layers,
prefill in chunks of up to 2048 tokens. Every pass is what an engine calls between two of its
own kernels, through ``hipml_b200.api`` with device tensors that the engine keeps:

* ``decode``      one token through the 16 layers of a single stream: append + attend.
* ``layer_decode`` the same with the attention front end (q|gate split, norm, rope, append)
                  and the output gate, two calls per layer.
* ``batch``       one token for every slot of a multi-slot server, 16 layers.
* ``verify``      a speculative draft's columns checked against one stream, 16 layers.
* ``decode_f32``  the single stream (or a few columns) over the unquantised cache, 16 layers.
* ``chunk``       one layer of a prompt chunk: append its rows, attend over the whole cache.
* ``layer_chunk`` one layer of a prompt chunk with front end, incremental staging and gate.
"""
from __future__ import annotations

import math
import random

import torch

from hipml_b200 import api

HEADS, KV, DIM, LAYERS = 24, 4, 256, 16
QW, W = HEADS * DIM, KV * DIM
SCALE = 1.0 / 16.0
N_ROT, SECTIONS, THETA, EPS = 64, [11, 11, 10, 0], 1.0e7, 1.0e-6
ROW_BYTES = {"q8": 272, "q4": 144}       # one K (or V) row of one KV head
DTYPE_ID = {"q8": 0, "q4": 1}            # decode selector / append dtype
CHUNK_DTYPE_ID = {"f32": 0, "q8": 1, "q4": 2}
HEADROOM = 136                           # cache rows kept past the live ones


def listed():
    return [
        # a chat turn soon after a short prompt: launch latency and the set-up of a kernel count
        {"name": "decode q8 672", "kind": "decode", "dtype": "q8", "depth": 672},
        # the everyday decode step with everything around the attention fused in
        {"name": "layer decode q8 8192", "kind": "layer_decode", "depth": 8192},
        # the small cache format on a document-sized context
        {"name": "decode q4 32768", "kind": "decode", "dtype": "q4", "depth": 32768},
        # the longest context: bound by the stream of cache rows
        {"name": "decode q8 100000", "kind": "decode", "dtype": "q8", "depth": 100000},
        # a server with 8 conversations of unequal length in flight
        {"name": "batch q8 8 slots", "kind": "batch", "dtype": "q8", "slots": 8, "low": 512, "high": 8192,
         "depth_seed": 3},
        # speculative decoding: four columns of one stream in one call
        {"name": "verify q8 4 at 8192", "kind": "verify", "cols": 4, "depth": 8192},
        # the unquantised cache, as far as it is usually taken
        {"name": "decode f32 2048", "kind": "decode_f32", "rows": 1, "depth": 2048},
        # a short prompt over the unquantised cache, one chunk
        {"name": "chunk f32 672", "kind": "chunk", "dtype": "f32", "pos0": 0, "tokens": 672},
        # a few words added to a conversation that has just begun
        {"name": "chunk q4 37 at 29", "kind": "chunk", "dtype": "q4", "pos0": 29, "tokens": 37},
        # the last full chunk of an 8192-token prompt
        {"name": "chunk q8 2048 at 6144", "kind": "chunk", "dtype": "q8", "pos0": 6144, "tokens": 2048},
        # a follow-up question over a longer conversation, with front end and gate
        {"name": "layer chunk q8 301 at 3001", "kind": "layer_chunk", "pos0": 3001, "tokens": 301},
        # a late chunk of a long document, in the engine's key slices
        {"name": "chunk q8 2048 at 30720", "kind": "chunk", "dtype": "q8", "pos0": 30720, "tokens": 2048},
    ]


def _spread(rng: random.Random, low: int, high: int) -> int:
    """A whole number of [low, high], even over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))))


def draw(rng: random.Random):
    kind = rng.choice(["decode", "decode", "layer_decode", "batch", "batch", "verify", "decode_f32", "chunk",
                       "chunk", "chunk", "layer_chunk"])
    if kind == "decode":
        return {"kind": kind, "dtype": rng.choice(["q8", "q8", "q4"]), "depth": _spread(rng, 200, 100000)}
    if kind == "layer_decode":
        return {"kind": kind, "depth": _spread(rng, 200, 60000)}
    if kind == "batch":
        return {"kind": kind, "dtype": rng.choice(["q8", "q8", "q4"]), "slots": rng.randint(2, 16),
                "low": 512, "high": _spread(rng, 1024, 8192), "depth_seed": rng.randrange(1 << 20)}
    if kind == "verify":
        return {"kind": kind, "cols": rng.randint(2, 8), "depth": _spread(rng, 200, 32768)}
    if kind == "decode_f32":
        return {"kind": kind, "rows": rng.choice([1, 1, 1, 2, 4, 8]), "depth": _spread(rng, 100, 8192)}
    if kind == "layer_chunk":
        return {"kind": kind, "pos0": rng.choice([0, _spread(rng, 30, 14000)]), "tokens": _spread(rng, 30, 2048)}
    dtype = rng.choice(["f32", "q8", "q8", "q4"])
    pos0 = rng.choice([0, _spread(rng, 30, 6000 if dtype == "f32" else 30720)])
    return {"kind": kind, "dtype": dtype, "pos0": pos0, "tokens": _spread(rng, 30, 2048)}


def _depths(case):
    r = random.Random(case["depth_seed"])
    return [r.randint(case["low"], case["high"]) for _ in range(case["slots"])]


class _State:
    """What an engine holds for one case: caches, activations, scratch, step words."""

    def __init__(self, case, seed):
        self.case = case
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape):
        return torch.randn(*shape, device="cuda", generator=self.gen)

    def bytes_cache(self, layers, stride, dtype, slots=1):
        """[layers][K, V][slots][KV heads][stride rows] of quantised rows, none live yet."""
        return torch.zeros(layers, 2, slots, KV * stride * ROW_BYTES[dtype], dtype=torch.uint8, device="cuda")

    def fill(self, kc, vc, stride, rows, dtype):
        for start in range(0, rows, 16384):
            n = min(16384, rows - start)
            api.kv_encode_bulk(self.normal(n, W), self.normal(n, W), kc, vc, KV, DIM, stride, start, 0, n,
                               DTYPE_ID[dtype])

    def partials(self, slots, splits):
        self.splits, self.acc_slot, self.ml_slot = splits, HEADS * splits * DIM, HEADS * splits * 2
        self.acc = torch.empty(slots * self.acc_slot, device="cuda")
        self.ml = torch.empty(slots * self.ml_slot, device="cuda")


def _ints(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def prepare(case, seed):
    s = _State(case, seed)
    kind = case["kind"]
    if kind in ("decode", "layer_decode"):
        depth, dtype = case["depth"], case.get("dtype", "q8")
        s.stride = depth + HEADROOM
        s.kv = s.bytes_cache(LAYERS, s.stride, dtype)
        for l in range(LAYERS):
            s.fill(s.kv[l, 0], s.kv[l, 1], s.stride, depth, dtype)
        s.partials(1, api.decode_splits(depth + 1))
        s.step = _ints([depth, depth + 1, 0, 0, depth, depth, depth, depth])
        s.k, s.v = s.normal(LAYERS, W), s.normal(LAYERS, W)
        s.out = torch.empty(LAYERS, QW, device="cuda")
        if kind == "decode":
            s.q = s.normal(LAYERS, QW)
        else:
            s.qg = s.normal(LAYERS, 2 * QW)
            s.q, s.gate = torch.empty(LAYERS, QW, device="cuda"), torch.empty(LAYERS, QW, device="cuda")
            s.q_norm, s.k_norm = 1 + 0.1 * s.normal(LAYERS, DIM), 1 + 0.1 * s.normal(LAYERS, DIM)
            s.pos4 = s.step[4:]
    elif kind == "batch":
        depths, dtype, slots = _depths(case), case["dtype"], case["slots"]
        s.stride = case["high"] + HEADROOM
        s.slot_bytes = KV * s.stride * ROW_BYTES[dtype]
        s.kv = s.bytes_cache(LAYERS, s.stride, dtype, slots)
        for l in range(LAYERS):
            for i, d in enumerate(depths):
                s.fill(s.kv[l, 0, i], s.kv[l, 1, i], s.stride, d, dtype)
        s.partials(slots, api.batch_splits(s.stride, slots))
        s.pos = _ints([[d, d + 1] for d in depths])
        s.q, s.out = s.normal(LAYERS, slots, QW), torch.empty(LAYERS, slots, QW, device="cuda")
        s.k, s.v = s.normal(LAYERS, slots, W), s.normal(LAYERS, slots, W)
    elif kind == "verify":
        depth, cols = case["depth"], case["cols"]
        s.stride = depth + HEADROOM
        s.kv = s.bytes_cache(LAYERS, s.stride, "q8")
        for l in range(LAYERS):
            s.fill(s.kv[l, 0], s.kv[l, 1], s.stride, depth, "q8")
        s.partials(cols, api.decode_splits(depth + cols))
        s.pos = _ints([[depth + c, depth + c + 1] for c in range(cols)])
        s.q, s.out = s.normal(LAYERS, cols, QW), torch.empty(LAYERS, cols, QW, device="cuda")
        s.k, s.v = s.normal(LAYERS, cols, W), s.normal(LAYERS, cols, W)
    elif kind == "decode_f32":
        depth, rows = case["depth"], case["rows"]
        s.n_ctx = depth + HEADROOM
        s.kv = s.normal(LAYERS, 2, s.n_ctx, W)
        s.partials(rows, api.cols_splits(s.n_ctx))
        s.q, s.out = s.normal(LAYERS, rows, QW), torch.empty(LAYERS, rows, QW, device="cuda")
        s.k, s.v = s.normal(LAYERS, rows, W), s.normal(LAYERS, rows, W)
    elif kind == "chunk":
        pos0, tokens, dtype = case["pos0"], case["tokens"], case["dtype"]
        s.stride = pos0 + tokens + HEADROOM
        if dtype == "f32":
            s.kv = s.normal(2, s.stride, W)
        else:
            s.kv = s.bytes_cache(1, s.stride, dtype)[0]
            s.fill(s.kv[0], s.kv[1], s.stride, pos0, dtype)
        s.k, s.v, s.q = s.normal(tokens, W), s.normal(tokens, W), s.normal(tokens, QW)
        s.out = torch.empty(tokens, QW, device="cuda")
        s.splits = api.prefill_splits(pos0)
        s.acc = s.ml = None
        if s.splits >= 2:
            slots = s.splits * ((tokens + 31) // 32 * 32) * HEADS
            s.acc, s.ml = torch.empty(slots * DIM, device="cuda"), torch.empty(slots * 2, device="cuda")
        s.ws = torch.empty(api.attn_chunk_workspace_bytes(KV, DIM, pos0, tokens), dtype=torch.uint8, device="cuda")
    elif kind == "layer_chunk":
        pos0, tokens = case["pos0"], case["tokens"]
        s.stride = pos0 + tokens + HEADROOM
        s.cap = (pos0 + tokens + 127) // 128 * 128
        s.kv = s.bytes_cache(1, s.stride, "q8")[0]
        s.fill(s.kv[0], s.kv[1], s.stride, pos0, "q8")
        s.ws = torch.empty(api.attn_chunk_workspace_bytes(KV, DIM, 0, s.cap), dtype=torch.uint8, device="cuda")
        # the earlier chunks' rows are staged already, as an engine that keeps an image per layer has them
        api.attn_chunk_stage(s.kv[0], s.kv[1], KV, DIM, 1, s.stride, 0, pos0, s.cap, s.ws)
        s.qg, s.k, s.v = s.normal(tokens, 2 * QW), s.normal(tokens, W), s.normal(tokens, W)
        s.q_norm, s.k_norm = 1 + 0.1 * s.normal(DIM), 1 + 0.1 * s.normal(DIM)
        s.q, s.gate = torch.empty(tokens, QW, device="cuda"), torch.empty(tokens, QW, device="cuda")
        s.out = torch.empty(tokens, QW, device="cuda")
    else:
        raise ValueError(f"unknown kind {kind}")
    if kind not in ("chunk", "layer_chunk"):
        # a layer's tensors, as an engine's layer objects hold them
        per_layer = [s.k, s.v, s.q, s.kv[:, 0], s.kv[:, 1], s.out]
        if kind == "layer_decode":
            per_layer += [s.qg, s.gate, s.q_norm, s.k_norm]
        s.layers = [tuple(t[l] for t in per_layer) for l in range(LAYERS)]
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "decode":
        selector = DTYPE_ID[case["dtype"]]
        for k, v, q, kc, vc, out in s.layers:
            api.attn_decode_kv_append(s.step, k, v, q, kc, vc, s.acc, s.ml, out, HEADS, KV, DIM, s.stride, SCALE,
                                      s.splits, selector=selector)
        return {"out": s.out, "cache": s.kv}
    if kind == "layer_decode":
        for k, v, q, kc, vc, out, qg, gate, q_norm, k_norm in s.layers:
            api.attn_front_append_q8(qg, k, v, q, gate, q_norm, k_norm, kc, vc, HEADS, KV, DIM, N_ROT, THETA, EPS,
                                     tokens=1, stride=s.stride, sections=SECTIONS, pos=s.pos4, step=s.step)
            api.attn_decode_kv_gated(s.step, q, kc, vc, s.acc, s.ml, out, gate, HEADS, KV, DIM, s.stride, SCALE,
                                     s.splits)
        return {"out": s.out, "q": s.q, "gate": s.gate, "cache": s.kv}
    if kind == "batch":
        dtype = DTYPE_ID[case["dtype"]]
        for k, v, q, kc, vc, out in s.layers:
            api.attn_decode_batch_append(s.pos, k, v, q, kc, vc, s.acc, s.ml, out, HEADS, KV, DIM, s.stride, SCALE,
                                         s.splits, s.slot_bytes, s.acc_slot, s.ml_slot, QW, case["slots"],
                                         dtype=dtype)
        return {"out": s.out, "cache": s.kv}
    if kind == "verify":
        depth, cols = case["depth"], case["cols"]
        for k, v, q, kc, vc, out in s.layers:
            api.kv_encode_bulk(k, v, kc, vc, KV, DIM, s.stride, depth, 0, cols)
            api.attn_decode_cols(s.pos, q, kc, vc, s.acc, s.ml, out, HEADS, KV, DIM, s.stride, SCALE, s.splits, cols,
                                 s.acc_slot, s.ml_slot, QW)
        return {"out": s.out, "cache": s.kv}
    if kind == "decode_f32":
        depth, rows = case["depth"], case["rows"]
        for k, v, q, kc, vc, out in s.layers:
            api.kv_append_cols_f32(kc, vc, k, v, depth, rows, W)
            api.attn_decode_cols_f32(q, kc, vc, s.acc, s.ml, out, HEADS, KV, DIM, s.n_ctx, depth, rows)
        return {"out": s.out, "cache": s.kv}
    pos0, tokens = case["pos0"], case["tokens"]
    if kind == "chunk":
        if case["dtype"] == "f32":
            api.kv_append_chunk_f32(s.kv[0], s.kv[1], s.k, s.v, pos0, W, tokens)
        else:
            api.kv_encode_bulk(s.k, s.v, s.kv[0], s.kv[1], KV, DIM, s.stride, pos0, 0, tokens,
                               DTYPE_ID[case["dtype"]])
        api.attn_chunk(s.q, s.kv[0], s.kv[1], s.out, HEADS, KV, DIM, pos0, tokens, CHUNK_DTYPE_ID[case["dtype"]],
                       s.stride, s.acc, s.ml, s.splits, 0, s.ws)
        return {"out": s.out, "cache": s.kv}
    api.attn_front_append_q8(s.qg, s.k, s.v, s.q, s.gate, s.q_norm, s.k_norm, s.kv[0], s.kv[1], HEADS, KV, DIM, N_ROT,
                             THETA, EPS, pos0=pos0, tokens=tokens, stride=s.stride)
    api.attn_chunk_stage(s.kv[0], s.kv[1], KV, DIM, 1, s.stride, pos0, pos0 + tokens, s.cap, s.ws)
    api.attn_chunk_staged_gated(s.q, s.out, s.gate, HEADS, KV, DIM, pos0, tokens, s.cap, s.ws)
    return {"out": s.out, "q": s.q, "gate": s.gate, "cache": s.kv}


def work(case):
    """Bytes: every live cache row once per layer and pass, the new rows in and out, the query and
    output rows. Operations: 2 * 2 * 256 for every visible (query head, key) pair."""
    kind = case["kind"]
    if kind in ("chunk", "layer_chunk"):
        pos0, n = case["pos0"], case["tokens"]
        row = W * 4 if case.get("dtype") == "f32" else KV * ROW_BYTES[case.get("dtype", "q8")]
        rows = n * (2 * QW * 4 + 2 * W * 4)
        if kind == "layer_chunk":
            rows += n * 3 * QW * 4      # the joint q|gate rows in, the gate rows out
        pairs = HEADS * (n * pos0 + n * (n + 1) // 2)
        return {"bytes": 2 * row * (pos0 + n) + rows, "flops": 4 * DIM * pairs}
    if kind == "batch":
        live, columns = [d + 1 for d in _depths(case)], case["slots"]
        read, pairs = sum(live), sum(live)
    else:
        columns = case.get("cols", case.get("rows", 1))
        read = case["depth"] + columns
        pairs = columns * case["depth"] + columns * (columns + 1) // 2
    row = W * 4 if kind == "decode_f32" else KV * ROW_BYTES[case.get("dtype", "q8")]
    per_column = 2 * QW * 4 + 2 * W * 4 + (3 * QW * 4 if kind == "layer_decode" else 0)
    return {"bytes": LAYERS * (2 * row * read + columns * per_column), "flops": LAYERS * 4 * DIM * HEADS * pairs}


def tolerance(case):
    """Decode keeps f32 sums over operands split exactly into two 11-bit parts: about 1e-5. Chunk
    attention adds into tensor-core accumulators over thousands of keys: about 3e-5 at the far end
    of a chain. Cache bytes are the same."""
    return {"rel": 5e-5} if case["kind"] in ("chunk", "layer_chunk") else {"rel": 1e-5}
