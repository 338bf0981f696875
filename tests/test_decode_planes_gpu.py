"""The streaming decode with one query head per lane (eight KV heads) and its 2-bit scores from bit planes, the cluster form's choice of
CTAs, and the append's per-tile destinations, where they can go wrong: against the oracle and the chain kernel."""
import numpy as np
import pytest
import torch

import triebwerk_b200 as tq
from triebwerk_b200 import ops
from oracle import tqo
from tests import helpers as hp

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("tests.gpu_util")
D, HKV = 128, 8


# one to four query heads per KV head; contexts at the edges of 32-token tiles; queries that fixed point finds hard
@pytest.mark.parametrize("bits,H", [(2, 8), (2, 16), (2, 24), (2, 32), (4, 8), (4, 24)])
def test_streaming_decode_of_eight_kv_heads(bits, H):
    rng = np.random.default_rng(100 * bits + H)
    G, msl, NL, kv_dim = 144, 96, 2, HKV * D
    lengths = [(1, 2, 31, 32, 33, 64, 65, 96)[g % 8] for g in range(G)]
    R = ops.rotation_matrix().numpy()
    eng = tq.Engine(msl, bits, num_layers=NL, num_heads=H, num_kv_heads=HKV, head_dim=D)
    eng.alloc_batch(G, msl)
    eng.reset()
    assert tq.lib().tq_engine_decode_form(eng._h, 0) == 0 and tq.lib().tq_engine_decode_form(eng._h, 1) == 0  # the streaming forms
    k, v = (rng.standard_normal((NL, G, msl, kv_dim), dtype=np.float32).astype(np.float16) for _ in range(2))
    for layer in range(NL):
        eng.prefill_append_batch(layer, 0, gu.dev(k[layer][:, :msl - 1]), gu.dev(v[layer][:, :msl - 1]))
    pos = np.array(lengths, np.int32) - 1
    eng.set_positions(pos)
    q = rng.standard_normal((NL, G, H, D), dtype=np.float32)
    q[:, 1] = 0                                            # no largest coordinate
    q[:, 2] *= 1e-3
    q[:, 3] *= 2  # (fp16 queries and centroids move a score of standard deviation s by 3e-4 s: at 2 a weight by 6e-4, five times that is the bar)
    q[:, 4] = 11 * R[rng.integers(0, D, H)].astype(np.float32)  # rotated: a single coordinate
    q[:, 5] = 6e-8                                         # the smallest fp16 values
    q[:, 6, H // 2, 5] = np.nan                            # one head of one sequence
    q = q.astype(np.float16).reshape(NL, G, H * D)
    kn1 = np.stack([k[:, g, n - 1] for g, n in enumerate(lengths)], 1)
    vn1 = np.stack([v[:, g, n - 1] for g, n in enumerate(lengths)], 1)
    dq, dk, dv = gu.dev(q), gu.dev(kn1), gu.dev(vn1)
    outs = {"layers": gu.host(torch.stack([eng.decode_layer(i, dq[i], dk[i], dv[i]) for i in range(NL)])),
            "step": gu.host(eng.decode_step(dq, dk, dv, torch.empty_like(dq)))}
    assert eng.status() == 0
    for layer in range(NL):
        ck, cv, kn, vn = (gu.host(t) for t in eng.layer_cache(layer))
        ref, _ = tqo.attention_batch(np.nan_to_num(q[layer], nan=0.0), ck, cv, kn, vn, R, pos, msl, H, HKV, D, bits)
        for name, out in outs.items():
            o = out[layer].copy().reshape(G, H, D)
            assert np.isnan(o[6, H // 2]).all(), name
            o[6, H // 2] = ref.reshape(G, H, D)[6, H // 2]
            assert np.isfinite(o).all(), name
            hp.assert_attention_close(o.reshape(G, H * D), ref, H, D, f"{name} {bits} bits, {H} heads, layer {layer}")


# 2-bit queries as fixed point: one rotated coordinate far above the others, at each of a byte's four places, among ordinary ones; and
# beyond fp16, as which the whole-step form holds them: NaN, whatever the codes (bits of 0 and 1 that an infinity leaves in the planes)
def test_queries_with_one_large_coordinate():
    rng = np.random.default_rng(77)
    G, H, msl, NL = 144, 16, 96, 2
    R = ops.rotation_matrix().numpy()
    eng = tq.Engine(msl, 2, num_layers=NL, num_heads=H, num_kv_heads=HKV, head_dim=D)
    eng.alloc_batch(G, msl)
    eng.reset()
    assert tq.lib().tq_engine_decode_form(eng._h, 0) == 0 and tq.lib().tq_engine_decode_form(eng._h, 1) == 0
    k, v = (rng.standard_normal((NL, G, msl, HKV * D), dtype=np.float32).astype(np.float16) for _ in range(2))
    for layer in range(NL):
        eng.prefill_append_batch(layer, 0, gu.dev(k[layer][:, :msl - 1]), gu.dev(v[layer][:, :msl - 1]))
    lengths = np.array([(96, 40, 1, 2)[g // 36] for g in range(G)])
    pos = (lengths - 1).astype(np.int32)
    eng.set_positions(pos)
    Rf, at = R.astype(np.float32), np.arange(G)
    q = rng.standard_normal((NL, G, H, D), dtype=np.float32)
    q[:, :72] += 8 * Rf[at[:72] % D][:, None]
    q[:, 72:] = 65504 * np.where(Rf[at[72:] % D] < 0, -1, 1)[:, None]   # rotated and scaled 7e4 and more
    q = q.astype(np.float16).reshape(NL, G, H * D)
    dq, dk, dv = gu.dev(q), gu.dev(k[:, at, pos]), gu.dev(v[:, at, pos])
    layers = gu.host(torch.stack([eng.decode_layer(i, dq[i], dk[i], dv[i]) for i in range(NL)]))
    step = gu.host(eng.decode_step(dq, dk, dv, torch.empty_like(dq)))
    assert eng.status() == 0
    beyond = np.abs((q[0, :, :D].astype(np.float32) @ Rf.T) * 0.12751743).max(1) > 65520
    assert not beyond[:72].any() and beyond[72:].sum() >= 36
    for layer in range(NL):
        ck, cv, kn, vn = (gu.host(t) for t in eng.layer_cache(layer))
        ref, _ = tqo.attention_batch(q[layer], ck, cv, kn, vn, R, pos, msl, H, HKV, D, 2)
        hp.assert_attention_close(layers[layer, :108], ref[:108], H, D, "layers")  # (one token, or ordinary scores)
        hp.assert_attention_close(step[layer, :72], ref[:72], H, D, "step")
        assert np.isnan(step[layer, beyond]).all()


# the same through one layer's calls with more than 16 query heads: fp32 up to the fixed point, so finite where fp16 is not
@pytest.mark.parametrize("H", [24, 32])
def test_layer_calls_take_queries_beyond_fp16(H):
    rng = np.random.default_rng(H)
    G, msl = 216, 96  # (so many that the batch launcher streams too)
    R = ops.rotation_matrix().numpy()
    eng = tq.Engine(msl, 2, num_layers=1, num_heads=H, num_kv_heads=HKV, head_dim=D)
    eng.alloc_batch(G, msl)
    eng.reset()
    assert tq.lib().tq_engine_decode_form(eng._h, 0) == 0
    k, v = (rng.standard_normal((G, msl, HKV * D), dtype=np.float32).astype(np.float16) for _ in range(2))
    eng.prefill_append_batch(0, 0, gu.dev(k[:, :msl - 1]), gu.dev(v[:, :msl - 1]))
    pos = np.where(np.arange(G) < 108, 95, 0).astype(np.int32)
    eng.set_positions(pos)
    Rf, at = R.astype(np.float32), np.arange(G)
    q = rng.standard_normal((G, H, D), dtype=np.float32)
    q[:108] += 8 * Rf[at[:108] % D][:, None]
    q[108:] = 65504 * np.where(Rf[at[108:] % D] < 0, -1, 1)[:, None]
    assert (np.abs(q[108:, 0] @ Rf.T * 0.12751743).max(1) > 65520).sum() >= 36
    q = q.astype(np.float16).reshape(G, H * D)
    layer = gu.host(eng.decode_layer(0, gu.dev(q), gu.dev(k[at, pos]), gu.dev(v[at, pos])))
    ck, cv, kn, vn = (gu.host(t) for t in eng.layer_cache(0))
    ref, _ = tqo.attention_batch(q, ck, cv, kn, vn, R, pos, msl, H, HKV, D, 2)
    hp.assert_attention_close(layer, ref, H, D, "decode_layer")
    hp.assert_attention_close(gu.gpu_attention_batch(q, ck, cv, kn, vn, R, pos, msl, H, HKV, D, 2), ref, H, D, "batch launcher")
    # one long sequence; one token, with codes that go with the rotated query's signs and the largest norm, has all the weight
    n, j = 40000, 12345
    ck, cv = (rng.integers(0, 256, (n, HKV * D // 4), dtype=np.uint8) for _ in range(2))
    kn, vn = (rng.uniform(0.5, 1.0, (n, HKV)).astype(np.float16) for _ in range(2))
    big = (65504 * np.where(Rf[7] < 0, -1, 1)).astype(np.float16)
    ck[j] = np.tile(hp.pack_codes(np.where(big.astype(np.float32) @ Rf.T > 0, 3, 0), 2), HKV)
    kn[j] = 4.0
    q = np.tile(big, H)
    ref, _ = tqo.attention_batch(q[None], ck, cv, kn, vn, R, np.array([n - 1], np.int32), n, H, HKV, D, 2)
    hp.assert_attention_close(gu.gpu_attention_single(q, ck, cv, kn, vn, R, n - 1, n, H, HKV, D, 2)[None], ref, H, D, "single launcher")
    assert eng.status() == 0


# a slot that 8 CTAs serve with more than one block per warp; the launchers' clusters of one and two CTAs, one per SM
@pytest.mark.parametrize("bits,H,msl,lengths,ctas", [(4, 16, 1536, [1500], 8), (2, 32, 2032, [2032], 8), (2, 32, 1024, [1023] * 8, 2), (4, 16, 512, [300, 512] * 8, 1)])
def test_cluster_sizes_and_the_launchers(bits, H, msl, lengths, ctas):
    rng = np.random.default_rng(bits + H + msl)
    G, kv_dim = len(lengths), HKV * D
    R = ops.rotation_matrix().numpy()
    eng = tq.Engine(msl, bits, num_layers=1, num_heads=H, num_kv_heads=HKV, head_dim=D)
    eng.alloc_batch(G, msl)
    eng.reset()
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert tq.lib().tq_engine_decode_form(eng._h, 0) == ctas
    k, v = (rng.standard_normal((G, msl, kv_dim), dtype=np.float32).astype(np.float16) for _ in range(2))
    eng.prefill_append_batch(0, 0, gu.dev(k), gu.dev(v))
    pos = np.array(lengths, np.int32) - 1
    eng.set_positions(pos)
    q = rng.standard_normal((G, H * D), dtype=np.float32).astype(np.float16)
    at = np.arange(G)
    out = gu.host(eng.decode_layer(0, gu.dev(q), gu.dev(k[at, pos]), gu.dev(v[at, pos])))  # (the token that is there already)
    ck, cv, kn, vn = (gu.host(t) for t in eng.layer_cache(0))
    ref, _ = tqo.attention_batch(q, ck, cv, kn, vn, R, pos, msl, H, HKV, D, bits)
    hp.assert_attention_close(out, ref, H, D, "decode_layer")
    hp.assert_attention_close(gu.gpu_attention_batch(q, ck, cv, kn, vn, R, pos, msl, H, HKV, D, bits), ref, H, D, "launcher")


# tiles of 128 / Hkv tokens that end inside a prompt, on its end, and span two prompts; slots of their own sizes, a first position
@pytest.mark.parametrize("bits,Hkv,n,T,first,caps", [
    (4, 8, 3, 64, 0, None), (4, 8, 5, 79, 0, None), (2, 8, 2, 65, 30, None), (4, 4, 3, 333, 0, None), (2, 4, 4, 130, 7, [160, 140, 192, 137]),
    (4, 8, 2, 128, 0, [128, 150]), (2, 16, 3, 61, 3, None)])
def test_append_destinations(bits, Hkv, n, T, first, caps):
    rng = np.random.default_rng(7 * bits + Hkv + T)
    kv_dim, msl = Hkv * D, first + T
    k, v = (gu.dev(rng.standard_normal((n, T, kv_dim), dtype=np.float32).astype(np.float16)) for _ in range(2))
    caches = []
    for whole in (True, False):
        eng = tq.Engine(msl, bits, num_layers=1, num_heads=Hkv, num_kv_heads=Hkv, head_dim=D)
        eng.alloc_batch(n, max(caps) if caps else msl, caps)
        eng.reset()
        if whole:
            eng.prefill_append_batch(0, 0, k, v, first)
        else:  # pieces below four tiles: the chain kernel
            step = 256 // Hkv
            for g in range(n):
                for t in range(0, T, step):
                    eng.prefill_append(0, g, k[g, t:t + step], v[g, t:t + step], first + t)
        assert eng.status() == 0
        caches.append([gu.host(t) for t in eng.layer_cache(0)])
    for a, b in zip(*caches):
        assert (a.view(np.uint8) == b.view(np.uint8)).all()
