"""The tcgen05 prefill attention (csrc/tq_prefill_fa.cuh) where it can go wrong: edges of its 128-row tiles and query blocks, one
and two query blocks per CTA, any number of query heads per KV head, prompts that go through the scratch in groups.  Against the
oracle on the engine's own cache bytes."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import triebwerk_b200 as tq
from oracle import tqo
from tests import helpers as hp

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("tests.gpu_util")
D = 128


@pytest.mark.parametrize("bits,H,Hkv,n,T,msl", [
    # few blocks: one query block per CTA, even and odd tiles in its two slots
    (4, 16, 8, 1, 1, 32), (4, 16, 8, 1, 127, 128), (2, 16, 8, 1, 128, 160), (0, 16, 8, 1, 129, 160), (4, 32, 8, 2, 257, 288),
    (0, 8, 8, 1, 385, 416), (2, 40, 8, 1, 150, 160), (4, 24, 2, 1, 140, 160), (0, 40, 8, 1, 51, 64), (4, 96, 1, 1, 130, 160),
    # many: two query blocks per CTA (8 KV heads x 8 prompts x 3 pairs of blocks), the last pair with one block or none at the end
    (4, 16, 8, 13, 128, 160), (2, 16, 8, 13, 100, 128), (4, 32, 8, 13, 65, 96),  # prompts of one tile: codes converted in place
    (4, 16, 8, 8, 300, 320), (2, 16, 8, 8, 257, 288), (0, 16, 8, 8, 321, 352), (4, 40, 8, 8, 160, 160), (0, 16, 8, 13, 129, 160),
])
def test_prefill_attention_edges(bits, H, Hkv, n, T, msl):
    rng = np.random.default_rng(4000 + 17 * bits + H + T)
    kv_dim = Hkv * D
    R = tq.ops.rotation_matrix().numpy()
    eng = tq.Engine(msl, bits, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(n, msl)
    for t in eng.layer_cache(0):  # rows past the prompts: codes of any kind, norms and fp16 values that are not numbers
        if t is not None:
            t.view(torch.int16).fill_(0x7E00)
    k, v = (rng.standard_normal((n, T, kv_dim), dtype=np.float32).astype(np.float16) for _ in range(2))
    q = rng.standard_normal((n, T, H * D), dtype=np.float32).astype(np.float16)
    got = gu.host(eng.prefill_layer_batch(0, 0, gu.dev(q), gu.dev(k), gu.dev(v)))
    assert eng.status() == 0
    assert np.isfinite(got.astype(np.float32)).all()
    cache = [None if t is None else gu.host(t) for t in eng.layer_cache(0)]
    for i in {0, n // 2, n - 1}:
        sl = slice(i * msl, i * msl + T)
        if bits == 0:
            toks = sorted({0, 1, 24, 25, 63, 64, 127, 128, T // 2, T - 2, T - 1} & set(range(T)))
            ref = np.stack([tqo.fp16_attention_single(q[i, t], k[i], v[i], t, T, H, Hkv, D)[0] for t in toks])
            hp.assert_attention_close(got[i][toks], ref, H, D, f"fp16 {H}/{Hkv} T={T} prompt {i}")
        else:
            ck, cv, kn, vn = (t[sl] for t in cache)
            ref, _ = tqo.prefill_attention(q[i], ck, cv, kn, vn, R, T, H, Hkv, D, bits)
            hp.assert_attention_close(got[i], ref, H, D, f"tq{bits} {H}/{Hkv} T={T} prompt {i}")


@pytest.mark.parametrize("bits,n", [(4, 1), (2, 1), (4, 8)])  # one and two query blocks per CTA
def test_a_norm_that_is_not_finite_reaches_no_earlier_query(bits, n):
    """128 values of 6000 have a norm beyond fp16.  Query token t reads rows 0 .. t: such a V vector at row 70 (KV head 0) and
    such a K vector at row 200 (KV head 1) must not show in the results of the queries before them."""
    H, Hkv, T, msl = 16, 8, 300, 320
    rng = np.random.default_rng(4500 + bits + n)
    R = tq.ops.rotation_matrix().numpy()
    k, v = (rng.standard_normal((n, T, Hkv * D), dtype=np.float32).astype(np.float16) for _ in range(2))
    v[:, 70, :D], k[:, 200, D:2 * D] = 6000, 6000
    q = rng.standard_normal((n, T, H * D), dtype=np.float32).astype(np.float16)
    eng = tq.Engine(msl, bits, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(n, msl)
    got = gu.host(eng.prefill_layer_batch(0, 0, gu.dev(q), gu.dev(k), gu.dev(v)))
    ck, cv, kn, vn = (gu.host(t) for t in eng.layer_cache(0))
    for i in {0, n - 1}:
        at = i * msl
        assert np.isinf(vn[at + 70, 0]) and np.isinf(kn[at + 200, 1])
        for heads, rows in ((slice(0, 2), 70), (slice(2, 4), 200), (slice(4, 16), T)):  # 2 query heads per KV head
            ref, _ = tqo.prefill_attention(q[i, :rows], ck[at:], cv[at:], kn[at:], vn[at:], R, msl, H, Hkv, D, bits)
            sl = slice(heads.start * D, heads.stop * D)
            hp.assert_attention_close(got[i, :rows, sl], ref[:, sl], heads.stop - heads.start, D, f"tq{bits} heads {heads}")


@pytest.mark.parametrize("bits,n", [(4, 1), (2, 1), (4, 8)])  # one and two query blocks per CTA
def test_weights_times_large_norms_stay_finite(bits, n):
    """V norms of about 1e4 and scores that rise by 3.4 powers of two in the second and third tile: a weight of 2^3.4 over a
    reference point of the first tile, times such a norm, is beyond fp16."""
    H, Hkv, T, msl = 16, 8, 300, 320
    rng = np.random.default_rng(4600 + bits + n)
    R = tq.ops.rotation_matrix().numpy()
    u = rng.standard_normal(D).astype(np.float32)
    rise = 3.4 / (float(u @ u) * 1.4426950 / np.sqrt(D))
    k = 0.001 * rng.standard_normal((n, T, Hkv, D)).astype(np.float32)
    k[:, 130], k[:, 260] = rise * u, rise * u
    k = k.reshape(n, T, Hkv * D).astype(np.float16)
    v = (900 * rng.standard_normal((n, T, Hkv * D), dtype=np.float32)).astype(np.float16)
    q = np.broadcast_to(u.astype(np.float16), (n, T, H, D)).reshape(n, T, H * D).copy()
    eng = tq.Engine(msl, bits, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(n, msl)
    got = gu.host(eng.prefill_layer_batch(0, 0, gu.dev(q), gu.dev(k), gu.dev(v))).astype(np.float32)
    ck, cv, kn, vn = (gu.host(t) for t in eng.layer_cache(0))
    for i in {0, n - 1}:
        _, ref = tqo.prefill_attention(q[i], ck[i * msl:], cv[i * msl:], kn[i * msl:], vn[i * msl:], R, msl, H, Hkv, D, bits)
        # fp16 roundings (2^-11 at most) of weights, centroids, queries' share of the scores and results
        err = np.linalg.norm(got[i].reshape(T, H, D) - ref, axis=-1) / np.linalg.norm(ref, axis=-1)
        assert err.max() <= 4 * 2.0 ** -11, f"relative error {err.max():.2e}"


@pytest.mark.parametrize("bits,H,Hkv,n,T,msl", [
    (4, 40, 8, 1, 1, 32), (2, 40, 8, 1, 129, 160), (4, 20, 1, 1, 300, 320), (2, 6, 2, 2, 127, 128), (4, 40, 8, 8, 160, 160),
    (0, 40, 8, 1, 129, 160), (0, 12, 4, 1, 257, 288), (0, 24, 8, 13, 129, 160), (0, 20, 1, 2, 300, 320),
])
def test_other_layouts_are_off_by_their_rounding_to_fp16_only(bits, H, Hkv, n, T, msl):
    """Numbers of query heads per KV head that used to run with fp32 queries, centroids and weights: the results' distance from the
    oracle's fp32 ones is that of these ones' own rounding to fp16 (3 % for the order of sums and the exponentials)."""
    rng = np.random.default_rng(4700 + bits + H + T)
    R = tq.ops.rotation_matrix().numpy()
    eng = tq.Engine(msl, bits, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(n, msl)
    k, v = (rng.standard_normal((n, T, Hkv * D), dtype=np.float32).astype(np.float16) for _ in range(2))
    q = rng.standard_normal((n, T, H * D), dtype=np.float32).astype(np.float16)
    got = gu.host(eng.prefill_layer_batch(0, 0, gu.dev(q), gu.dev(k), gu.dev(v))).astype(np.float32)
    assert eng.status() == 0
    cache = [None if t is None else gu.host(t) for t in eng.layer_cache(0)]
    for i in {0, n - 1}:
        if bits == 0:
            toks = np.unique(np.linspace(0, T - 1, 40).astype(int))
            ref = np.stack([tqo.fp16_attention_single(q[i, t], k[i], v[i], t, T, H, Hkv, D)[1] for t in toks])
        else:
            toks = np.arange(T)
            _, ref = tqo.prefill_attention(q[i], *(t[i * msl:] for t in cache), R, msl, H, Hkv, D, bits)
        ref = ref.reshape(len(toks), H * D)
        err, rounding = np.linalg.norm(got[i, toks] - ref), np.linalg.norm(ref.astype(np.float16).astype(np.float32) - ref)
        assert err <= 1.03 * rounding, f"prompt {i}: {err / rounding:.2f} times the rounding to fp16"


def test_prompts_pass_through_the_scratch_in_groups():
    """40 prompts of 1000 tokens x 4 KV heads: more than the 131072 rows of one KV head that fit the fp16 scratch at a time."""
    H, Hkv, n, T = 8, 4, 40, 1000
    gen = torch.Generator(device="cuda").manual_seed(5)
    k, v = (torch.randn(n, T, Hkv * D, generator=gen, device="cuda").half() for _ in range(2))
    q = torch.randn(n, T, H * D, generator=gen, device="cuda").half()
    eng = tq.Engine(1024, 4, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(n, 1024)
    together = eng.prefill_layer_batch(0, 0, q, k, v)
    for i in (0, 31, 32, 39):
        one = eng.prefill_layer(0, i, q[i], k[i], v[i])
        # (one prompt alone has one query block per CTA, the batch two: another order of summation)
        assert torch.allclose(together[i].float(), one.float(), atol=1e-3, rtol=2e-3)
    assert eng.status() == 0


def test_prompts_on_two_streams_share_the_scratch_in_turn():
    """Prompts of two sequences, layer by layer on a stream each: their fp16 rows go through one scratch, whose second user waits for
    the first one's kernels."""
    H, Hkv, T, NL, msl = 16, 8, 777, 16, 1024
    gen = torch.Generator(device="cuda").manual_seed(8)
    q, k, v = (torch.randn(2, NL, T, d, generator=gen, device="cuda").half() for d in (H * D, Hkv * D, Hkv * D))
    eng = tq.Engine(msl, 4, num_layers=NL, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(2, msl)
    want = torch.stack([torch.stack([eng.prefill_layer(i, s, q[s, i], k[s, i], v[s, i]) for i in range(NL)]) for s in range(2)])
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for delay in range(0, 60000, 3000):  # (cycles by which one stream is late: its conversions meet the other's products)
        got = torch.zeros_like(want)
        torch.cuda.synchronize()
        with torch.cuda.stream(streams[1]):
            torch.cuda._sleep(200000 + delay)
        with torch.cuda.stream(streams[0]):
            torch.cuda._sleep(200000)
        for i in range(NL):
            for s in range(2):
                with torch.cuda.stream(streams[s]):
                    eng.prefill_layer(i, s, q[s, i], k[s, i], v[s, i], got[s, i])
        torch.cuda.synchronize()
        assert eng.status() == 0
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("bits", [4, 2])
def test_long_prompt_passes_through_the_scratch_by_kv_heads(bits):
    """16500 tokens x 8 KV heads do not fit the scratch as a whole: 4 heads, then 4.  The launcher, given those two halves' heads as
    caches of their own, which fit, computes every column in the same order: the same bits; given the prompt as a whole, too."""
    H, Hkv, T, msl = 16, 8, 16500, 16512
    gen = torch.Generator(device="cuda").manual_seed(6)
    k, v = (torch.randn(T, Hkv * D, generator=gen, device="cuda").half() for _ in range(2))
    q = torch.randn(T, H * D, generator=gen, device="cuda").half()
    eng = tq.Engine(msl, bits, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(2, msl)
    got = eng.prefill_layer(0, 1, q, k, v)
    ck, cv, kn, vn = (t[msl:] for t in eng.layer_cache(0))
    want = torch.empty_like(q)
    tq.ops.launch_turbo_gqa_prefill_attention(want, q, ck, cv, kn, vn, tq.ops.rotation_matrix().cuda(), None, T, msl, H, Hkv, D, H * D, Hkv * D, bits)
    assert eng.status() == 0
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    for half in range(2):
        sl = slice(half * Hkv // 2, (half + 1) * Hkv // 2)
        part = [t.view(msl, Hkv, -1)[:, sl].reshape(msl, -1).contiguous() for t in (ck, cv, kn, vn)]
        cols = slice(half * H // 2 * D, (half + 1) * H // 2 * D)
        o = torch.empty(T, H // 2 * D, dtype=torch.float16, device="cuda")
        tq.ops.launch_turbo_gqa_prefill_attention(o, q[:, cols].contiguous(), *part, tq.ops.rotation_matrix().cuda(), None, T, msl, H // 2, Hkv // 2,
                                                  D, H // 2 * D, Hkv // 2 * D, bits)
        assert torch.equal(got[:, cols].contiguous().view(torch.int16), o.view(torch.int16))


def test_a_long_prompt_through_the_launcher_can_be_captured():
    """16500 tokens x 8 KV heads are 135 MB as fp16 rows; the launchers' workspace, 64 MiB after their first call, serves them some KV
    heads at a time and need not grow, which it cannot under capture.  In a child: the workspace is the process's."""
    src = """
import torch, triebwerk_b200 as tq
H, Hkv, D, T, msl = 16, 8, 128, 16500, 16512
R = tq.ops.rotation_matrix().cuda()
ck, cv = (torch.randint(0, 256, (msl, Hkv * 64), dtype=torch.uint8, device='cuda') for _ in range(2))
kn, vn = (torch.rand(msl, Hkv, device='cuda').half() for _ in range(2))
q = torch.randn(T, H * D, device='cuda').half()
out, want = torch.zeros_like(q), torch.zeros_like(q)
run = lambda o, t: tq.ops.launch_turbo_gqa_prefill_attention(o, q, ck, cv, kn, vn, R, None, t, msl, H, Hkv, D, H * D, Hkv * D, 4)
run(want, 100)  # (the first call allocates)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    run(out, T)
g.replay()
run(want, T)
torch.cuda.synchronize()
assert torch.equal(out.view(torch.int16), want.view(torch.int16))
print('captured')
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", src], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]
