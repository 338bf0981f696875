"""Short packed prompts: the append leaves the attention's fp16 rows and norms itself.  The launchers, which make them from the cache in a
launch of their own, have to give the same bits on the same cache."""
import numpy as np
import pytest
import torch

import triebwerk_b200 as tq
from tests import gpu_util as gu
from tests import helpers as hp

pytestmark = pytest.mark.gpu
D = 128


def _draw(rng, *s):
    return torch.from_numpy(rng.standard_normal(s, dtype=np.float32).astype(np.float16)).cuda()


def _launcher(eng, layer, seq, q, msl, H, Hkv, bits):
    ck, cv, kn, vn = (t.view(-1, t.shape[-1])[seq * msl:(seq + 1) * msl].cpu().numpy() for t in eng.layer_cache(layer))
    return gu.gpu_prefill_attention(q.cpu().numpy(), ck, cv, kn, vn, tq.ops.rotation_matrix().numpy(), msl, H, Hkv, D, bits)


@pytest.mark.parametrize("bits,H,Hkv,T", [(4, 16, 8, 129), (4, 16, 8, 143), (4, 32, 8, 256), (2, 16, 8, 257), (4, 16, 8, 777), (2, 32, 4, 400), (4, 4, 2, 333),
                                          (2, 2, 1, 640), (4, 16, 8, 2047)])
def test_rows_made_by_the_append_equal_those_made_from_the_cache(bits, H, Hkv, T):
    rng = np.random.default_rng(T)
    msl = -(-T // 128) * 128 + 128
    eng = tq.Engine(msl, bits, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(2, msl)
    # the scratch holds the norms of a longer prompt, not all of them numbers, behind the one that is looked at
    k, v, q = _draw(rng, msl, Hkv * D), _draw(rng, msl, Hkv * D), _draw(rng, msl, H * D)
    v[T:] = float("inf")
    eng.prefill_layer(0, 1, q, k, v, torch.empty_like(q))
    k, v, q = _draw(rng, T, Hkv * D), _draw(rng, T, Hkv * D), _draw(rng, T, H * D)
    k[5, :D] = 0
    v[7, :D] = 0
    v[T - 1, -D:] *= 800.0  # a V norm past what weights above 1 leave room for
    out = torch.empty_like(q)
    eng.prefill_layer(0, 0, q, k, v, out)
    assert eng.status() == 0
    got, want = out.cpu().numpy(), _launcher(eng, 0, 0, q, msl, H, Hkv, bits)
    assert np.isfinite(got).all()
    assert np.array_equal(got.view(np.uint16), want.view(np.uint16))


@pytest.mark.parametrize("bits,H,Hkv,T", [(4, 16, 8, 4095), (2, 32, 4, 8190)])
def test_rows_of_more_tiles_than_ctas(bits, H, Hkv, T):
    """A CTA of the append has two tiles: the largest V norms of the first, far above or below the second's, are the first's alone."""
    rng = np.random.default_rng(T)
    msl = -(-T // 32) * 32
    eng = tq.Engine(msl, bits, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(1, msl)
    k, v, q = _draw(rng, T, Hkv * D), _draw(rng, T, Hkv * D), _draw(rng, T, H * D)
    v *= torch.exp2(torch.from_numpy(rng.integers(-6, 10, -(-T // 16))).cuda().half().repeat_interleave(16)[:T, None])
    out = torch.empty_like(q)
    want = None
    for _ in range(3):
        eng.prefill_layer(0, 0, q, k, v, out)
        assert eng.status() == 0
        got = out.cpu().numpy()
        if want is None: want = _launcher(eng, 0, 0, q, msl, H, Hkv, bits)
        assert np.isfinite(got).all()
        assert np.array_equal(got.view(np.uint16), want.view(np.uint16))


def test_values_that_are_not_numbers_reach_no_earlier_query():
    bits, H, Hkv, T, msl = 4, 16, 8, 300, 512
    rng = np.random.default_rng(3)
    eng = tq.Engine(msl, bits, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(1, msl)
    k, v, q = _draw(rng, T, Hkv * D), _draw(rng, T, Hkv * D), _draw(rng, T, H * D)
    v[200] = float("inf")
    out = torch.empty_like(q)
    eng.prefill_layer(0, 0, q, k, v, out)
    got, want = out.cpu().numpy(), _launcher(eng, 0, 0, q, msl, H, Hkv, bits)
    assert np.isfinite(got[:200]).all() and not np.isfinite(got[200:]).any()
    assert np.array_equal(got[:200].view(np.uint16), want[:200].view(np.uint16))


@pytest.mark.parametrize("bits,H,Hkv,T,n", [(4, 16, 8, 144, 3), (2, 32, 4, 160, 5), (4, 16, 8, 256, 2)])
def test_several_prompts(bits, H, Hkv, T, n):
    rng = np.random.default_rng(n)
    msl = 288
    eng = tq.Engine(msl, bits, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(n + 1, msl)
    k, v, q = _draw(rng, n, T, Hkv * D), _draw(rng, n, T, Hkv * D), _draw(rng, n, T, H * D)
    out = torch.empty_like(q)
    eng.prefill_layer_batch(0, 1, q, k, v, out)
    assert eng.status() == 0
    for i in range(n):
        hp.assert_attention_close(out[i].cpu().numpy(), _launcher(eng, 0, 1 + i, q[i], msl, H, Hkv, bits), H, D, f"prompt {i}")


@pytest.mark.parametrize("bits,H,Hkv,T,n", [(4, 16, 8, 33, 1), (4, 16, 8, 64, 1), (2, 32, 8, 128, 1), (4, 16, 8, 100, 16), (4, 16, 8, 129, 1), (2, 32, 4, 777, 1),
                                            (4, 40, 8, 300, 1), (4, 16, 8, 2500, 2)])
def test_queries_that_are_the_layer_befores_result(bits, H, Hkv, T, n):
    """The attention reads its queries under the append; they are what the launch before that wrote, or a kernel of another library."""
    NL, msl = 4, -(-T // 32) * 32
    rng = np.random.default_rng(T)
    eng = tq.Engine(msl, bits, num_layers=NL, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(n, msl)
    k, v, q = _draw(rng, NL, n, T, Hkv * D), _draw(rng, NL, n, T, Hkv * D), _draw(rng, n, T, H * D)

    def chain(settle):
        x = q.clone()
        for layer in range(NL):
            out = torch.full_like(x, float("nan"))
            settle()
            eng.prefill_layer_batch(layer, 0, x, k[layer], v[layer], out)
            settle()
            x = out * 4 if layer == 1 else out
            settle()
        return x.cpu().numpy().view(np.uint16)

    want = chain(torch.cuda.synchronize)
    for _ in range(3):
        assert np.array_equal(chain(lambda: None), want)
    assert eng.status() == 0
