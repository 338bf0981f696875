"""Performance cases: what programs have this library do, through its public entry points.

A case is one pass of one kind of work, at sizes that decoding and prefill meet:

* ``layer``      one ``Engine.decode_layer`` call: append one token per sequence to one layer's cache and attend
* ``walk``       the layers of a decode step one ``decode_layer`` call after the other, as a model's forward makes them
* ``step``       the layers of a decode step in one ``Engine.decode_step`` call on buffers of all layers
* ``host``       ``Engine.decode_step_host``: the same from pinned host buffers, results back in host memory
* ``launchers``  the reference-compatible launchers (two cache writes and one attention per layer), caller-owned arrays
* ``append``     ``Engine.prefill_append_batch``: prompts of equal length into the cache, layer by layer
* ``prefill``    ``Engine.prefill_layer`` / ``prefill_layer_batch``: cache write and causal attention, layer by layer

``kv_bits`` is 4, 2 or 0 (fp16 cache); head_dim is 128.  Values: K and V ~ N(0, 1) with K channels scaled by exp(N(0, 0.5)),
queries ~ N(0, 1), all fp16; the caches are written by the library's own appends.  A pass does not advance the
positions, so that it can be repeated on the same state.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import triebwerk_b200 as tq
from triebwerk_b200 import ops, synth

D = 128
DECODE_KINDS = ("layer", "walk", "step", "host", "launchers")


def _case(name, kind, bits, layers, heads, kv_heads, seqs, tokens, ragged_from=0, lengths_seed=0):
    """`tokens`: the context of every sequence with the new token (decode kinds) or the prompt's length.  Decode kinds with
    `ragged_from` > 0: contexts uniform in ragged_from .. tokens, drawn from `lengths_seed`."""
    c = dict(kind=kind, bits=bits, layers=layers, heads=heads, kv_heads=kv_heads, seqs=seqs, tokens=tokens, ragged_from=ragged_from,
             lengths_seed=lengths_seed)
    return dict(c, name=name) if name else c


def listed():
    return [
        # four rollouts of one short prompt, one layer: the smallest batched call a rollout loop makes
        _case("layer-4bit-4x612", "layer", 4, 1, 16, 8, 4, 612),
        # a single stream, the layers of a model in turn: latency of a chat or of the last unfinished rollout
        _case("walk-4bit-1x1500", "walk", 4, 28, 16, 8, 1, 1500),
        # an embedder that keeps its own arrays and calls the reference's launchers, 2-bit, a small batch of odd length
        _case("launchers-2bit-8x1023", "launchers", 2, 36, 32, 8, 8, 1023),
        # a full decode step of a rollout batch: 16 prompts x 4 rollouts at context 4096
        _case("step-4bit-64x4096", "step", 4, 28, 16, 8, 64, 4096),
        # the larger model at long context and 2 bits, layer by layer as its forward runs
        _case("walk-2bit-32x8192", "walk", 2, 36, 32, 8, 32, 8192),
        # a continuous batch of very different lengths
        _case("step-4bit-ragged-128", "step", 4, 8, 32, 8, 128, 16384, 128, 0),
        # the same without quantisation (kv_bits = 0), half the batch
        _case("step-fp16-ragged-64", "step", 0, 4, 32, 8, 64, 16384, 128, 1),
        # a head layout with five query heads per KV head (40/8), a small batch
        _case("walk-4bit-40h-8x1777", "walk", 4, 8, 40, 8, 8, 1777),
        # queries, keys and values from host memory, results back: the end-to-end call
        _case("host-4bit-16x2019", "host", 4, 28, 16, 8, 16, 2019),
        # prompts of a rollout batch into the cache
        _case("append-4bit-16x2048", "append", 4, 4, 16, 8, 16, 2048),
        # one prompt of ordinary, odd length through the layers of a model
        _case("prefill-4bit-1x777", "prefill", 4, 28, 16, 8, 1, 777),
        # a long prompt of the larger model into an fp16 cache
        _case("prefill-fp16-1x8192", "prefill", 0, 4, 32, 8, 1, 8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: 1 to 128 sequences, contexts of 64 to 16384 tokens, prompts of 32 to 8192."""
    kind = rng.choice(["layer", "walk", "walk", "step", "step", "host", "launchers", "append", "prefill", "prefill"])
    bits = rng.choice([4, 4, 4, 2, 2, 0])
    heads, kv_heads = rng.choice([(16, 8), (16, 8), (16, 8), (32, 8), (32, 8), (32, 4), (40, 8)])
    layers = 1 if kind == "layer" else rng.choice([4, 8, 28, 36])
    row = _row_bytes(bits, kv_heads)
    if kind in DECODE_KINDS:
        seqs = _log_int(rng, 1, 128 if kind in ("walk", "step") else 32)
        tokens = _log_int(rng, 64, 16384)
        # no drawn case moves more than the largest listed ones (much less where every query head reads the cache itself)
        most = 6e9 if heads // kv_heads in (1, 2, 4, 8) else 5e8
        while seqs * tokens * row * layers > most:
            if layers > 4:
                layers //= 2
            elif tokens > 1024:
                tokens = tokens * 2 // 3
            else:
                seqs = max(1, seqs // 2)
        ragged = tokens >= 256 and seqs > 1 and kind in ("walk", "step") and rng.random() < 0.4
        return _case(None, kind, bits, layers, heads, kv_heads, seqs, tokens, max(1, tokens // 64) if ragged else 0, rng.randrange(1000))
    seqs = _log_int(rng, 1, 16)
    tokens = _log_int(rng, 32, 8192 if kind == "prefill" else 4096)
    most = (2.5e11 if heads // kv_heads in (1, 2, 4, 8) else 2.5e10) if kind == "prefill" else 1e18
    while 2.0 * D * heads * tokens * tokens * seqs * layers > 4 * most or seqs * tokens * layers * kv_heads > 4e6:
        if layers > 1:
            layers //= 2
        elif seqs > 1:
            seqs //= 2
        else:
            tokens = tokens * 2 // 3
    return _case(None, kind, bits, layers, heads, kv_heads, seqs, tokens)


# ---- sizes ---------------------------------------------------------------------------------------------------------------
def _row_bytes(bits, kv_heads):
    """Cache bytes of one token and layer: codes and fp16 norms of K and V, or both as fp16."""
    return 4 * kv_heads * D if bits == 0 else 2 * kv_heads * (D * bits // 8) + 4 * kv_heads


def _lengths(c):
    if not c["ragged_from"]:
        return [c["tokens"]] * c["seqs"]
    return [int(n) for n in np.random.default_rng(c["lengths_seed"]).integers(c["ragged_from"], c["tokens"] + 1, c["seqs"])]


def work(c):
    H, Hkv, NL, G, T = c["heads"], c["kv_heads"], c["layers"], c["seqs"], c["tokens"]
    io = 2 * D * (2 * H + 2 * Hkv)  # fp16 queries in, results out, keys and values in, of one token
    rotations = 0 if c["bits"] == 0 else 2.0 * D * D * (2 * H + 2 * Hkv)  # queries, results, keys, values of one token
    row = _row_bytes(c["bits"], Hkv)
    rot = 0 if c["bits"] == 0 else 2 * D * D
    if c["kind"] in DECODE_KINDS:
        n = sum(_lengths(c))
        return {"bytes": float(NL * (n * row + G * io + rot)), "flops": NL * (4.0 * D * H * n + G * rotations)}
    if c["kind"] == "append":
        return {"bytes": float(NL * (G * T * (4 * Hkv * D + row) + rot)), "flops": NL * G * T * (0.0 if c["bits"] == 0 else 4.0 * D * D * Hkv)}
    return {"bytes": float(NL * (G * T * (io + row) + rot)), "flops": NL * G * (2.0 * D * H * T * (T + 1) + T * rotations)}


def tolerance(c):
    # Codes, norms and fp16 rows in the cache are exact.  Attention results are fp16 (half a unit: 2.4e-4 on average of a
    # value) of sums over fp16 weights and fp16 centroids or rows, accumulated in fp32.
    return "exact" if c["kind"] == "append" else {"rel": 2e-3, "differ": 0.0}


# ---- inputs --------------------------------------------------------------------------------------------------------------
def _fill(eng, c, gen, scales, lengths):
    """Every sequence's first lengths[g] - 1 tokens, in every layer, through the engine's own prompt append."""
    kv_dim = c["kv_heads"] * D
    if not c["ragged_from"]:
        T, block = c["tokens"] - 1, max(1, (1 << 26) // (c["tokens"] * kv_dim))
        for layer in range(c["layers"]):
            for g in range(0, c["seqs"] if T > 0 else 0, block):
                n = min(block, c["seqs"] - g)
                k, v = synth.torch_kv(gen, n * T, kv_dim, scales)
                eng.prefill_append_batch(layer, g, k.view(n, T, kv_dim), v.view(n, T, kv_dim))
        return
    pool_k, pool_v = synth.torch_kv(gen, c["tokens"] + 4096, kv_dim, scales)  # slices of one pool, another one each time
    for layer in range(c["layers"]):
        for g, n in enumerate(lengths):
            if n > 1:
                at = (1237 * layer + 101 * g) % 4096
                eng.prefill_append(layer, g, pool_k[at:at + n - 1], pool_v[at:at + n - 1])


def _engine(c, capacity, capacities=None):
    """An engine over a zeroed arena of the caller's, and all layers' cache bytes as one view of that arena."""
    eng = tq.Engine(capacity, c["bits"], num_layers=c["layers"], num_heads=c["heads"], num_kv_heads=c["kv_heads"], head_dim=D)
    arena = torch.zeros(eng.arena_bytes(c["seqs"], capacity, capacities), dtype=torch.uint8, device="cuda")
    eng.set_arena(arena.data_ptr(), arena.numel(), keep_alive=arena)
    eng.alloc_batch(c["seqs"], capacity, capacities)
    first, last = eng.layer_cache(0), eng.layer_cache(c["layers"] - 1)
    end = [t for t in last if t is not None][-1]
    begin = first[0].data_ptr() - arena.data_ptr()
    size = end.data_ptr() + end.numel() * end.element_size() - first[0].data_ptr()
    return eng, arena[begin:begin + size].view(torch.int64)


def prepare(case, seed):
    c = dict(case)
    NL, G, H, Hkv, bits = c["layers"], c["seqs"], c["heads"], c["kv_heads"], c["bits"]
    q_dim, kv_dim = H * D, Hkv * D
    gen = torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)
    scales = torch.from_numpy(synth.channel_scales(kv_dim, seed)).cuda()
    s = {"kind": c["kind"], "layers": NL, "case": c}
    capacity = -(-c["tokens"] // 256) * 256  # slots as a program reserves them, not cut to the present length
    if c["kind"] in ("append", "prefill"):
        s["eng"], s["cache"] = _engine(c, capacity)
        T = c["tokens"]
        kv = [synth.torch_kv(gen, G * T, kv_dim, scales) for _ in range(NL)]
        shape = (T,) if c["kind"] == "prefill" and G == 1 else (G, T)
        s["k"] = [k.view(*shape, kv_dim) for k, _ in kv]
        s["v"] = [v.view(*shape, kv_dim) for _, v in kv]
        if c["kind"] == "prefill":
            s["q"] = [torch.randn(*shape, q_dim, generator=gen, device="cuda").to(torch.float16) for _ in range(NL)]
            s["out"] = [torch.empty_like(q) for q in s["q"]]
        return s
    lengths = _lengths(c)
    k, v = synth.torch_kv(gen, NL * G, kv_dim, scales)  # the step's new token of every sequence and layer
    k, v = k.view(NL, G, kv_dim), v.view(NL, G, kv_dim)
    q = torch.randn(NL, G, q_dim, generator=gen, device="cuda").to(torch.float16)
    out = torch.empty_like(q)
    if c["kind"] == "launchers":
        vpb = {0: 1, 2: 4, 4: 2}[bits]
        code = torch.float16 if bits == 0 else torch.uint8
        arrays = [torch.zeros(NL, G * capacity, kv_dim // vpb, dtype=code, device="cuda") for _ in range(2)]
        norms = [torch.zeros(NL, G * capacity, Hkv, dtype=torch.float16, device="cuda") for _ in range(2)]
        s["rotation"] = ops.rotation_matrix().cuda()
        s["pos"] = torch.tensor([n - 1 for n in lengths], dtype=torch.int32, device="cuda")
        T = c["tokens"] - 1
        at = torch.arange(T, dtype=torch.int32, device="cuda")
        for layer in range(NL):
            for g in range(G):
                for a, norm, x in zip(arrays, norms, synth.torch_kv(gen, T, kv_dim, scales)):
                    rows = slice(g * capacity, (g + 1) * capacity)
                    if bits == 0:
                        a[layer, rows][:T] = x
                    else:
                        ops.launch_turbo_kv_quantize(a[layer, rows], norm[layer, rows], x, s["rotation"], at, capacity, T, Hkv, D, kv_dim, bits)
        s["arrays"], s["norms"], s["capacity"] = arrays, norms, capacity
        s["ck"], s["cv"] = (list(a.unbind(0)) for a in arrays)
        s["kn"], s["vn"] = (list(n.unbind(0)) for n in norms)
    else:
        s["eng"], s["cache"] = _engine(c, capacity, lengths if c["ragged_from"] else None)
        _fill(s["eng"], c, gen, scales, lengths)
        s["eng"].set_positions([n - 1 for n in lengths])
    if c["kind"] == "host":
        s["q"], s["k"], s["v"] = (t.cpu().pin_memory() for t in (q, k, v))
        s["out"] = torch.empty(q.shape, dtype=torch.float16, pin_memory=True)
    elif c["kind"] == "step":
        s["q"], s["k"], s["v"], s["out"] = q, k, v, out
    else:
        s["q"], s["k"], s["v"], s["outs"] = (list(t.unbind(0)) for t in (q, k, v, out))
        s["out"] = out
    return s


# ---- one pass ------------------------------------------------------------------------------------------------------------
def _run_launchers(s):
    c = s["case"]
    G, H, Hkv, bits, msl = c["seqs"], c["heads"], c["kv_heads"], c["bits"], s["capacity"]
    q_dim, kv_dim, R, pos = H * D, Hkv * D, s["rotation"], s["pos"]
    for l in range(s["layers"]):
        ck, cv, kn, vn = s["ck"][l], s["cv"][l], s["kn"][l], s["vn"][l]
        if bits == 0:
            ops.launch_kv_cache_write_batch(ck, cv, s["k"][l], s["v"][l], pos, msl, G, kv_dim)
            ops.launch_gqa_attention_batch(s["outs"][l], s["q"][l], ck, cv, None, pos, msl, G, H, Hkv, D, q_dim, kv_dim)
        else:
            ops.launch_turbo_kv_quantize_batch(ck, kn, s["k"][l], R, pos, msl, G, Hkv, D, kv_dim, bits)
            ops.launch_turbo_kv_quantize_batch(cv, vn, s["v"][l], R, pos, msl, G, Hkv, D, kv_dim, bits)
            ops.launch_turbo_gqa_attention_batch(s["outs"][l], s["q"][l], ck, cv, kn, vn, R, None, pos, msl, G, H, Hkv, D, q_dim, kv_dim, bits)
    return [s["out"]] + s["arrays"] + (s["norms"] if bits else [])


def run(s):
    kind = s["kind"]
    if kind == "launchers":
        return _run_launchers(s)
    eng, q, k, v = s["eng"], s.get("q"), s["k"], s["v"]
    if kind == "step":
        eng.decode_step(q, k, v, s["out"])
    elif kind == "host":
        eng.decode_step_host(q, k, v, s["out"])
    elif kind == "append":
        for layer in range(s["layers"]):
            eng.prefill_append_batch(layer, 0, k[layer], v[layer])
        return s["cache"]
    elif kind == "prefill":
        one = k[0].dim() == 2
        for layer in range(s["layers"]):
            if one:
                eng.prefill_layer(layer, 0, q[layer], k[layer], v[layer], s["out"][layer])
            else:
                eng.prefill_layer_batch(layer, 0, q[layer], k[layer], v[layer], s["out"][layer])
    else:  # layer, walk
        for layer in range(s["layers"]):
            eng.decode_layer(layer, q[layer], k[layer], v[layer], s["outs"][layer])
    return [s["cache"]] + (s["out"] if isinstance(s["out"], list) else [s["out"]])
