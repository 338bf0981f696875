"""Launcher calls that follow each other without a synchronisation, each with another rotation, other positions and queries written just
before: kernels that start under their predecessors must not see the call before's."""
import numpy as np
import pytest
import torch

from oracle import tqo
from triebwerk_b200 import ops

pytestmark = pytest.mark.gpu
D = 128


def _rotations(n, rng):
    return [torch.from_numpy(np.linalg.qr(rng.standard_normal((D, D)))[0].astype(np.float16)).cuda() for _ in range(n)]


@pytest.mark.parametrize("bits,H,Hkv,G,n", [(4, 16, 8, 24, 3000), (2, 32, 8, 40, 2000), (2, 16, 4, 64, 1000), (4, 32, 4, 8, 8000), (2, 32, 8, 300, 64)])
def test_batch_calls_with_other_rotations_and_positions(bits, H, Hkv, G, n):
    rng = np.random.default_rng(bits * H + G)
    calls, kvd = 6, Hkv * D
    ck, cv = (torch.randint(0, 256, (G * n, kvd * bits // 8), dtype=torch.uint8, device="cuda") for _ in range(2))
    kn, vn = (torch.rand(G * n, Hkv, device="cuda").half() * 4 + 8 for _ in range(2))
    rots = _rotations(calls, rng)
    qs = [torch.randn(G, H * D, device="cuda").half() for _ in range(calls)]
    poss = [torch.from_numpy(rng.integers(0, n, G).astype(np.int32)).cuda() for _ in range(calls)]
    R, pos, q = rots[0].clone(), poss[0].clone(), qs[0].clone()  # the same addresses in every call

    def run(settle):
        outs = []
        for i in range(calls):
            R.copy_(rots[i]); pos.copy_(poss[i]); q.copy_(qs[i])
            settle()
            out = torch.full((G, H * D), float("nan"), dtype=torch.float16, device="cuda")
            ops.launch_turbo_gqa_attention_batch(out, q, ck, cv, kn, vn, R, None, pos, n, G, H, Hkv, D, H * D, kvd, bits)
            settle()
            outs.append(out)
        torch.cuda.synchronize()
        return [o.cpu().numpy().view(np.uint16) for o in outs]

    want = run(torch.cuda.synchronize)
    assert all(np.isfinite(w.view(np.float16)).all() for w in want)
    for _ in range(4):
        assert all(np.array_equal(a, b) for a, b in zip(run(lambda: None), want))


@pytest.mark.parametrize("bits,H,Hkv,n", [(2, 32, 8, 40000), (4, 16, 4, 40000), (4, 32, 4, 17000)])
def test_single_calls_with_other_rotations(bits, H, Hkv, n):
    rng = np.random.default_rng(n)
    calls, kvd = 6, Hkv * D
    ck, cv = (torch.randint(0, 256, (n, kvd * bits // 8), dtype=torch.uint8, device="cuda") for _ in range(2))
    kn, vn = (torch.rand(n, Hkv, device="cuda").half() * 4 + 8 for _ in range(2))
    rots = _rotations(calls, rng)
    qs = [torch.randn(H * D, device="cuda").half() for _ in range(calls)]
    R, q = rots[0].clone(), qs[0].clone()

    def run(settle):
        outs = []
        for i in range(calls):
            R.copy_(rots[i]); q.copy_(qs[i])
            settle()
            out = torch.full((H * D,), float("nan"), dtype=torch.float16, device="cuda")
            ops.launch_turbo_gqa_attention(q, ck, cv, kn, vn, R, out, None, n - 1 - 3000 * i, n, H, Hkv, D, bits)
            settle()
            outs.append(out)
        torch.cuda.synchronize()
        return [o.cpu().numpy().view(np.uint16) for o in outs]

    want = run(torch.cuda.synchronize)
    assert all(np.isfinite(w.view(np.float16)).all() for w in want)
    for _ in range(4):
        assert all(np.array_equal(a, b) for a, b in zip(run(lambda: None), want))
    # against 64 bits: the last call
    i = calls - 1
    m = n - 3000 * i
    cent = torch.from_numpy(tqo.tables(bits)[0]).double().cuda()
    sh = torch.arange(0, 8, bits, device="cuda", dtype=torch.uint8)
    un = lambda c, nm: cent[((c[:m].reshape(m, Hkv, -1)[..., None] >> sh) & (2 ** bits - 1)).reshape(m, Hkv, D).long()] * nm[:m].double()[..., None]
    s = torch.einsum("hd,nhd->hn", qs[i].double().view(H, D) @ rots[i].double().T / D ** 0.5, un(ck, kn).repeat_interleave(H // Hkv, 1))
    exact = (torch.einsum("hn,nhd->hd", s.softmax(-1), un(cv, vn).repeat_interleave(H // Hkv, 1)) @ rots[i].double()).flatten()
    got = torch.from_numpy(want[i].view(np.float16).astype(np.float64)).cuda()
    # fp16 centroids, weights and results: 1.4e-4 each of independent roundings, 3 to 5e-4 measured for their sum and the means' cancellation
    assert float((got - exact).norm() / exact.norm()) < 2e-3
