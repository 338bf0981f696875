"""One layer in the streaming form (append and query rotation, attention, merge: three launches) against the two-launch form, whose
append and query rotation are fp32 chains and whose merge is the last worker's: the same cache bytes, results up to the order of fp32 sums."""
import numpy as np
import pytest
import torch

import triebwerk_b200 as tq
from tests import gpu_util as gu
from tests import helpers as hp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,H,Hkv,lengths", [
    (4, 16, 8, [1 + (7 * g) % 61 for g in range(300)]),  # more pieces of work than CTAs of the first launch, one tile a sequence and two
    (2, 32, 8, [1 + (11 * g) % 90 for g in range(180)]),
    (4, 16, 8, [33000, 5]),      # a sequence in more parts than one merge round takes
    (2, 16, 8, [17000] * 3),     # fp32 queries for the 2-bit planes
    (4, 12, 4, [20000, 3001, 70, 33]),   # query heads that are no multiple of eight
    (2, 4, 4, [31, 32, 33, 40000]),
    (4, 32, 4, [30000, 63, 64, 65]),
    (4, 16, 8, [33000] + [5] * 25),  # many parts of one sequence, one warp per head
    (2, 32, 8, [9000] * 8), (4, 32, 8, [9000] * 9),  # the last batch that is merged by a CTA per head, and the first that is not
    (4, 16, 8, [3000] * 80),  # more CTAs than SMs in the merge
])
def test_layer_form_equals_two_launch_form(bits, H, Hkv, lengths):
    D, G = 128, len(lengths)
    kv_dim, q_dim = Hkv * D, H * D
    cap = -(-(max(lengths) + 3) // 32) * 32
    caps = [n + 3 for n in lengths]
    rng = np.random.default_rng(5)
    draw = lambda *s: torch.from_numpy(rng.standard_normal(s, dtype=np.float32).astype(np.float16)).cuda()
    engines = []
    for fused in (True, False):
        eng = tq.Engine(cap, bits, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=D)
        eng.alloc_batch(G, cap, caps)
        eng.set_fused(fused)
        engines.append(eng)
    assert tq.lib().tq_engine_decode_form(engines[0]._h, 0) == 0  # not the cluster form
    for g, n in enumerate(lengths):
        k, v = draw(n, kv_dim), draw(n, kv_dim)
        for eng in engines:
            eng.prefill_append(0, g, k, v, 0)
    for step in range(2):
        q, k, v = draw(G, q_dim), draw(G, kv_dim), draw(G, kv_dim)
        if step == 1:  # all zero (every coordinate on a bound), the largest values, values that are not numbers
            k.view(G, Hkv, D)[0, 0] = 0
            v.view(G, Hkv, D)[0, 1] = 65504.0
            k.view(G, Hkv, D)[0, 2, 5] = float("inf")
            v.view(G, Hkv, D)[0, 3, 127] = float("nan")
        outs = []
        for eng in engines:
            eng.set_positions([n + step for n in lengths])
            outs.append(gu.host(eng.decode_layer(0, q, k, v)))
            assert eng.status() == 0
        for x, y, name in zip(engines[0].layer_cache(0), engines[1].layer_cache(0), ("k codes", "v codes", "k norms", "v norms")):
            assert torch.equal(x.view(torch.uint8), y.view(torch.uint8)), f"step {step}: {name} differ"
        rows = slice(1, G) if step == 1 else slice(0, G)
        hp.assert_attention_close(outs[0][rows], outs[1][rows], H, D, f"bits={bits} step {step}")
