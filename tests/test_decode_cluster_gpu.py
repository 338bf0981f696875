"""The cluster form of the decode step (csrc/tq_decode_cluster.cuh) and the one-vector append where they can go wrong: edges
of 16- and 32-token tiles, clusters of 1 to 16 CTAs with and without a CTA for the new token, more than 8 query heads per KV
head, against the oracle; and the suites that the cluster form serves by default, once more with the streaming forms."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import triebwerk_b200 as tq
from triebwerk_b200 import ops
from oracle import tqo
from tests import helpers as hp

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("tests.gpu_util")
D = 128


# capacity and batch set the cluster size: at most one CTA per SM, a 16-token block per warp
@pytest.mark.parametrize("bits,H,Hkv,msl,lengths,ctas", [
    (4, 16, 8, 64, [1, 16, 17, 33, 64], 1),            # one CTA per cluster, 32-token tiles
    (2, 32, 8, 256, [1, 2, 128, 255], 2),
    (4, 16, 4, 512, [1, 31, 449, 512], 4),             # one of them for the new token
    (2, 8, 1, 2048, [1, 15, 16, 17, 1900], 16),        # 16-token tiles
    (4, 16, 8, 2112, [1801], 16),                      # several tiles per warp
    (4, 16, 4, 1600, [1] * 17 + [17, 700, 1600], 2),   # two on an SM
    (0, 16, 4, 640, [1] * 18 + [639, 640], 2),         # the same, fp16
    (4, 24, 2, 320, [97, 320], 4),                     # 12 query heads per KV head: two clusters share a KV head
    (2, 20, 1, 96, [95], 1),                           # 20: three
    (0, 40, 8, 384, [1, 16, 383], 4),                  # fp16 rows
    (0, 12, 4, 1024, [1000], 8),
])
def test_decode_layer_cluster_form(bits, H, Hkv, msl, lengths, ctas):
    rng = np.random.default_rng(1000 + 7 * bits + H + msl)
    G, kv_dim = len(lengths), Hkv * D
    R = ops.rotation_matrix().numpy()
    eng = tq.Engine(msl, bits, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(G, msl)
    eng.reset()
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert tq.lib().tq_engine_decode_form(eng._h, 0) == ctas
    ks = [rng.standard_normal((n, kv_dim), dtype=np.float32).astype(np.float16) for n in lengths]
    vs = [rng.standard_normal((n, kv_dim), dtype=np.float32).astype(np.float16) for n in lengths]
    ks[0][-1], vs[-1][-1, :D] = 0, 0  # a new token on a quantiser bound everywhere
    for g, n in enumerate(lengths):
        if n > 1:
            eng.prefill_append(0, g, gu.dev(ks[g][:-1]), gu.dev(vs[g][:-1]), 0)
    eng.set_positions([n - 1 for n in lengths])
    q = rng.standard_normal((G, H * D), dtype=np.float32).astype(np.float16)
    k1, v1 = np.stack([k[-1] for k in ks]), np.stack([v[-1] for v in vs])
    out = gu.host(eng.decode_layer(0, gu.dev(q), gu.dev(k1), gu.dev(v1)))
    again = gu.host(eng.decode_layer(0, gu.dev(q), gu.dev(k1), gu.dev(v1)))  # chained: old rows are read early
    assert eng.status() == 0
    assert (out.view(np.uint16) == again.view(np.uint16)).all()
    if bits == 0:
        ck, cv, _, _ = (None if t is None else gu.host(t) for t in eng.layer_cache(0))
        for g, n in enumerate(lengths):
            assert (ck[g * msl + n - 1] == k1[g]).all() and (cv[g * msl + n - 1] == v1[g]).all()
        ref, _ = tqo.fp16_attention_batch(q, ck, cv, np.array(lengths, np.int32) - 1, msl, H, Hkv, D)
        hp.assert_attention_close(out, ref, H, D, f"fp16 {H}/{Hkv}")
        return
    gk, gv, gkn, gvn = (gu.host(t) for t in eng.layer_cache(0))
    for g, n in enumerate(lengths):
        r = g * msl + n - 1
        for got, norms, x in ((gk, gkn, k1), (gv, gvn, v1)):  # the stored bytes are the launcher's (the exact chain everywhere)
            cq, cn = gu.gpu_append_tokens(x[g:g + 1], R, [0], 1, Hkv, D, bits)
            assert (got[r] == cq[0]).all() and (norms[r].view(np.uint16) == cn[0].view(np.uint16)).all()
        sl = slice(g * msl, g * msl + n)
        ref, _ = tqo.attention_single(q[g], gk[sl], gv[sl], gkn[sl], gvn[sl], R, n - 1, n, H, Hkv, D, bits)
        hp.assert_attention_close(out[g][None], ref[None], H, D, f"tq{bits} {H}/{Hkv} seq {g}")


# layouts that only the cluster form serves: through decode_layer, whole steps on device and on host buffers, the launchers
@pytest.mark.parametrize("bits,H,Hkv,msl,lengths", [
    (4, 40, 8, 640, [1, 16, 33, 639]), (2, 20, 1, 96, [95]), (4, 64, 4, 512, [449, 512]), (2, 6, 2, 320, [17, 300, 320]), (2, 40, 8, 64, [64] * 3),
    (0, 40, 8, 384, [1, 16, 383]), (0, 12, 4, 1024, [1000]), (0, 20, 1, 320, [97, 320]),
])
def test_other_layouts_are_off_by_their_rounding_to_fp16_only(bits, H, Hkv, msl, lengths):
    """They used to run with fp32 queries, centroids and weights: the results' distance from the oracle's fp32 ones is that of
    these ones' own rounding to fp16 (3 % for the order of sums and the exponentials)."""
    rng = np.random.default_rng(3000 + bits + H + msl)
    NL, G, kv_dim = 2, len(lengths), Hkv * D
    R = ops.rotation_matrix().numpy()
    eng = tq.Engine(msl, bits, num_layers=NL, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(G, msl)
    pos = [n - 1 for n in lengths]
    for layer in range(NL):
        for g, n in enumerate(pos):
            if n:
                eng.prefill_append(layer, g, *(gu.dev(rng.standard_normal((n, kv_dim), dtype=np.float32).astype(np.float16)) for _ in range(2)))
    eng.set_positions(pos)
    q, k, v = (rng.standard_normal((NL, G, d), dtype=np.float32).astype(np.float16) for d in (H * D, kv_dim, kv_dim))
    dq, dk, dv = gu.dev(q), gu.dev(k), gu.dev(v)
    outs = {"layers": gu.host(torch.stack([eng.decode_layer(i, dq[i], dk[i], dv[i]) for i in range(NL)])),
            "step": gu.host(eng.decode_step(dq, dk, dv, torch.empty_like(dq))),
            "host": eng.decode_step_host(*(t.cpu().pin_memory() for t in (dq, dk, dv)), torch.empty(dq.shape, dtype=torch.float16, pin_memory=True)).numpy()}
    outs["launcher"] = np.empty_like(q)
    ref = np.empty((NL, G, H, D), np.float32)
    for i in range(NL):
        cache = eng.layer_cache(i)
        ck, cv, kn, vn = (None if t is None else gu.host(t) for t in cache)
        o = torch.empty_like(dq[i])
        p = gu.dev(np.array(pos, np.int32))
        if bits == 0:
            ops.launch_gqa_attention_batch(o, dq[i], cache[0], cache[1], None, p, msl, G, H, Hkv, D, H * D, kv_dim)
            ref[i] = tqo.fp16_attention_batch(q[i], ck, cv, np.array(pos, np.int32), msl, H, Hkv, D)[1].reshape(G, H, D)
        else:
            ops.launch_turbo_gqa_attention_batch(o, dq[i], *cache, gu.dev(R), None, p, msl, G, H, Hkv, D, H * D, kv_dim, bits)
            ref[i] = tqo.attention_batch(q[i], ck, cv, kn, vn, R, np.array(pos, np.int32), msl, H, Hkv, D, bits)[1].reshape(G, H, D)
        outs["launcher"][i] = gu.host(o)
    assert eng.status() == 0
    rounding = np.linalg.norm(ref.astype(np.float16).astype(np.float32) - ref)
    for name, out in outs.items():
        err = np.linalg.norm(out.astype(np.float32).reshape(ref.shape) - ref)
        assert err <= 1.03 * rounding, f"{name}: {err / rounding:.2f} times the rounding to fp16"


# The host form's inputs lie where the warps' results go: clusters of 2 to 16 CTAs, with one and several tiles per warp, against the
# same steps on device buffers, which have no such area
@pytest.mark.parametrize("bits,H,Hkv,NL,G,msl,ctas", [
    (0, 16, 8, 2, 4, 256, 2), (0, 32, 8, 2, 2, 512, 4), (0, 16, 8, 1, 2, 1024, 8), (0, 32, 4, 2, 2, 900, 8), (0, 8, 1, 1, 2, 4096, 16),
    (0, 40, 8, 2, 2, 640, 4), (0, 12, 4, 1, 2, 1024, 8), (4, 16, 8, 2, 4, 256, 2), (2, 32, 8, 1, 2, 1024, 8),
    # one CTA each: results leave through shared memory, one to eight heads of a KV head, three clusters to a KV head
    (0, 16, 8, 4, 12, 256, 1), (0, 8, 8, 4, 12, 256, 1), (0, 32, 4, 8, 12, 256, 1), (4, 16, 8, 4, 12, 256, 1), (2, 32, 4, 8, 12, 256, 1), (4, 40, 8, 4, 12, 256, 1),
    (2, 20, 1, 16, 12, 256, 1)])
def test_host_steps_are_those_of_device_buffers(bits, H, Hkv, NL, G, msl, ctas):
    gen = torch.Generator(device="cuda").manual_seed(11 + msl)
    eng = tq.Engine(msl, bits, num_layers=NL, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(G, msl)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert tq.lib().tq_engine_decode_form(eng._h, 1) == ctas
    k, v = (torch.randn(G, msl - 1, Hkv * D, generator=gen, device="cuda").half() for _ in range(2))
    for layer in range(NL):
        eng.prefill_append_batch(layer, 0, k, v)
    eng.set_positions([msl - 1 - 17 * g for g in range(G)])
    for _ in range(20):
        q, k, v = (torch.randn(NL, G, d, generator=gen, device="cuda").half() for d in (H * D, Hkv * D, Hkv * D))
        want = eng.decode_step(q, k, v, torch.empty_like(q))
        got = eng.decode_step_host(*(t.cpu().pin_memory() for t in (q, k, v)), torch.empty(q.shape, dtype=torch.float16, pin_memory=True)).cuda()
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert eng.status() == 0


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("G,Hkv", [(1, 1), (3, 8), (111, 8), (112, 8), (148, 8)])
def test_one_vector_append_vs_oracle(bits, G, Hkv):
    """111 x 8 vectors: the last launch of one CTA per vector on a 148-SM GPU (six per SM); 112 x 8 and 148 x 8 share R in groups."""
    rng = np.random.default_rng(2000 + bits + G)
    R = ops.rotation_matrix().numpy()
    x = rng.standard_normal((G, Hkv * D), dtype=np.float32).astype(np.float16)
    pos = rng.integers(0, 8, G).astype(np.int32)
    got, gn = gu.gpu_append_batch(x, R, pos, 8, Hkv, D, bits)
    want, wn = tqo.alloc_cache(G, 8, Hkv, D, bits)
    tqo.append_batch(want, wn, x, R, pos, 8, Hkv, D, bits)
    # rsqrt.approx against a correctly rounded 1/sqrt: a coordinate on a bound may fall to the other side (test_append_gpu.py)
    assert int((hp.unpack_codes(got, bits) != hp.unpack_codes(want, bits)).sum()) <= 2 + G * Hkv * D // 50000
    assert np.abs(gn.view(np.uint16).astype(np.int32) - wn.view(np.uint16).astype(np.int32)).max() <= 1


@pytest.mark.parametrize("bits,msl", [(4, 288), (4, 320), (2, 64), (2, 96)])
def test_whole_steps_with_and_without_copy_warps(bits, msl):
    """128 sequences, too many for the cluster form: 4-bit slots of 36864 rows in all run without the copy warps on 148 SMs, of
    40960 with them (the line is four tiles per worker: 37888 rows); 2-bit ones of 8192 and 12288 (one tile: 9472)."""
    H, Hkv, NL, G = 16, 8, 2, 128
    rng = np.random.default_rng(3500 + bits + msl)
    R = ops.rotation_matrix().numpy()
    lengths = [int(n) for n in rng.integers(1, min(msl, 288) + 1, G)]
    lengths[:6] = [1, 32, 33, 64, min(msl, 288) - 1, min(msl, 288)]
    eng = tq.Engine(msl, bits, num_layers=NL, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(G, msl)
    pool = gu.dev(rng.standard_normal((2, 512, Hkv * D), dtype=np.float32).astype(np.float16))
    for layer in range(NL):
        for g, n in enumerate(lengths):
            if n > 1:
                at = (37 * g + 11 * layer) % 224
                eng.prefill_append(layer, g, pool[0, at:at + n - 1], pool[1, at:at + n - 1])
    eng.set_positions([n - 1 for n in lengths])
    q, k, v = (gu.dev(rng.standard_normal((NL, G, d), dtype=np.float32).astype(np.float16)) for d in (H * D, Hkv * D, Hkv * D))
    out = gu.host(eng.decode_step(q, k, v, torch.empty_like(q)))
    assert eng.status() == 0
    for layer in range(NL):
        ck, cv, kn, vn = (gu.host(t) for t in eng.layer_cache(layer))
        for g in (0, 1, 2, 3, 4, 5, 64, 127):
            sl = slice(g * msl, g * msl + lengths[g])
            ref, _ = tqo.attention_single(gu.host(q)[layer, g], ck[sl], cv[sl], kn[sl], vn[sl], R, lengths[g] - 1, lengths[g], H, Hkv, D, bits)
            hp.assert_attention_close(out[layer, g][None], ref[None], H, D, f"tq{bits} layer {layer} sequence {g}")


@pytest.mark.parametrize("bits,H,Hkv,NL,G,T", [
    (4, 16, 8, 28, 16, 1000),  # plain and host-buffer steps as one launch, the others as four
    (2, 32, 4, 28, 16, 2000),  # host-buffer steps only
    (4, 16, 8, 4, 64, 64),     # all but the produced ones
    (4, 16, 8, 4, 128, 300),   # none
])
def test_steps_agree_whatever_form_their_inputs_choose(bits, H, Hkv, NL, G, T):
    """Plain, produced (unit norm weights on normed inputs, no rotation), two-phase and host-buffer steps of one batch choose between
    one launch and four by different lines; results agree to the order of sums."""
    gen = torch.Generator(device="cuda").manual_seed(9)
    eng = tq.Engine(T, bits, num_layers=NL, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(G, T)
    k, v = (torch.randn(G, T - 1, Hkv * D, generator=gen, device="cuda").half() for _ in range(2))
    for layer in range(NL):
        eng.prefill_append_batch(layer, 0, k, v)
    eng.set_positions([T - 1] * G)
    q, k, v = (torch.randn(NL, G, d, generator=gen, device="cuda").half() for d in (H * D, Hkv * D, Hkv * D))
    want = eng.decode_step(q, k, v, torch.empty_like(q))
    cache = [t.clone() for t in eng.layer_cache(NL - 1)]
    two, rest = torch.empty_like(q), NL // 2 + 1
    assert eng.step_prepare(q, k, v)
    eng.step_attend_layers(0, rest, two)
    eng.step_attend_layers(rest, NL - rest, two)
    host = eng.decode_step_host(*(t.cpu().pin_memory() for t in (q, k, v)), torch.empty(q.shape, dtype=torch.float16, pin_memory=True)).cuda()
    assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(cache, eng.layer_cache(NL - 1)))
    ones, cos, sin = torch.ones(NL, D, device="cuda").half(), torch.ones(T, 64, device="cuda").half(), torch.zeros(T, 64, device="cuda").half()
    qn, kn = ((t.view(-1, D).float() * torch.rsqrt(t.view(-1, D).float().pow(2).mean(-1, keepdim=True) + 1e-6)).half().view(t.shape) for t in (q, k))
    produced = eng.decode_step_produce(q, k, v, torch.empty_like(q), ones, ones, cos, sin)
    plain = eng.decode_step(qn, kn, v, torch.empty_like(q))
    assert eng.status() == 0
    for name, got, ref in (("two phases", two, want), ("host", host, want), ("produced", produced, plain)):
        hp.assert_attention_close(gu.host(got).reshape(-1, H * D), gu.host(ref).reshape(-1, H * D), H, D, name)


def test_streaming_forms_in_a_child_process():
    """TQ_CLUSTER=0 (read once per process) keeps the streaming kernels for small batches too."""
    if os.environ.get("TQ_CLUSTER") == "0":
        pytest.skip("already the child")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-m", "pytest", "tests/test_attention_gpu.py", "tests/test_fp16_gpu.py", "tests/test_engine_gpu.py",
                        "-q", "-x", "-m", "gpu", "-k", "not child and not prefill", "-p", "no:cacheprovider"],
                       cwd=root, env=dict(os.environ, TQ_CLUSTER="0"), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert " passed" in r.stdout
