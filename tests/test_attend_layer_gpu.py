"""tq_engine_attend_layer attends with the queries of the last two-launch decode_layer, whatever the layer form rotated since."""
import numpy as np
import pytest
import torch

import triebwerk_b200 as tq
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,H,Hkv,lengths", [(4, 16, 8, [33000, 5]), (2, 32, 8, [33] * 180), (2, 16, 8, [17000] * 3), (4, 12, 4, [20000, 3001, 70, 33])])
def test_attend_layer_after_the_layer_form(bits, H, Hkv, lengths):
    D, G = 128, len(lengths)
    cap = -(-(max(lengths) + 1) // 32) * 32
    rng = np.random.default_rng(9)
    draw = lambda *s: torch.from_numpy(rng.standard_normal(s, dtype=np.float32).astype(np.float16)).cuda()
    eng = tq.Engine(cap, bits, num_layers=2, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(G, cap, [n + 1 for n in lengths])
    eng.reset()  # (the row of the new token is read before it is written)
    assert tq.lib().tq_engine_decode_form(eng._h, 0) == 0  # not the cluster form
    for g, n in enumerate(lengths):
        eng.prefill_append(0, g, draw(n, Hkv * D), draw(n, Hkv * D), 0)
    eng.set_positions(lengths)
    q, other, k, v = draw(G, H * D), draw(G, H * D), draw(G, Hkv * D), draw(G, Hkv * D)
    zeros = gu.host(eng.attend_layer(0, torch.empty_like(q)))  # nothing rotated yet: every score is zero
    eng.decode_layer(0, other, k, v)
    again = gu.host(eng.attend_layer(0, torch.empty_like(q)))  # (the new token is there now: other results, but no scores)
    assert np.isfinite(zeros).all() and np.isfinite(again).all()
    assert np.array_equal(again.reshape(G, Hkv, H // Hkv, D)[:, :, :1].repeat(H // Hkv, 2).reshape(G, -1), again)  # the mean of the values, for every head
    eng.set_fused(False)
    want = gu.host(eng.decode_layer(0, q, k, v))
    assert np.array_equal(gu.host(eng.attend_layer(0, torch.empty_like(q))), want)
    eng.set_fused(True)
    assert not np.array_equal(gu.host(eng.decode_layer(0, other, k, v)), want)
    assert np.array_equal(gu.host(eng.attend_layer(0, torch.empty_like(q))), want)
    assert eng.status() == 0
