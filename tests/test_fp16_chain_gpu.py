"""fp16 layers whose attention starts under the write of the new rows: layers and steps that follow each other without a synchronisation,
each layer's result in place as the next one's queries, give the bits of the same chain with a synchronisation between the calls."""
import numpy as np
import pytest
import torch

import triebwerk_b200 as tq

pytestmark = pytest.mark.gpu
D = 128
EDGES = [1, 2, 15, 16, 17, 31, 63, 64, 65, 300, 511, 512, 513, 1024, 1025, 2048, 2049]  # blocks of 16 tokens, warps' turns of 64, chunks of 512


@pytest.mark.parametrize("H,Hkv,lengths", [
    (8, 8, EDGES * 4), (16, 8, EDGES * 4), (32, 8, EDGES * 4), (64, 8, EDGES * 4 + [9000]), (16, 4, EDGES * 8),
    (16, 8, [n for n in EDGES if n < 510] + [500, 509]),  # one chunk: nothing to merge
    (16, 8, [40000]),
])
def test_chain_of_layers_and_steps(H, Hkv, lengths):
    G, NL, steps = len(lengths), 3, 3
    caps = [n + steps for n in lengths]
    cap = -(-max(caps) // 32) * 32
    if max(lengths) <= 512:
        cap, caps = 512, None
    rng = np.random.default_rng(H + G)
    draw = lambda *s: torch.from_numpy(rng.standard_normal(s, dtype=np.float32).astype(np.float16)).cuda()
    eng = tq.Engine(cap, 0, num_layers=NL, num_heads=H, num_kv_heads=Hkv, head_dim=D)
    eng.alloc_batch(G, cap, caps) if caps else eng.alloc_batch(G, cap)
    eng.reset()
    assert tq.lib().tq_engine_decode_form(eng._h, 0) == 0  # the streaming form
    for layer in range(NL):
        for x in eng.layer_cache(layer)[:2]:
            x.copy_(torch.randn(x.shape, device="cuda").half())
    saved = [[x.clone() for x in eng.layer_cache(layer)[:2]] for layer in range(NL)]
    q0, ks, vs = draw(G, H * D), draw(steps, NL, G, Hkv * D) * 2, draw(steps, NL, G, Hkv * D)
    x, k, v = torch.empty_like(q0), torch.empty_like(ks[0, 0]), torch.empty_like(vs[0, 0])

    def chain(settle):
        for layer in range(NL):
            for a, b in zip(eng.layer_cache(layer)[:2], saved[layer]):
                a.copy_(b)
        x.copy_(q0)
        eng.set_positions([n - 1 for n in lengths])
        outs = []
        for step in range(steps):
            for layer in range(NL):
                k.copy_(ks[step, layer]); v.copy_(vs[step, layer])
                settle()
                eng.decode_layer(layer, x, k, v, x)
                settle()
                outs.append(x.clone())
                x.mul_(8).add_(q0)
                settle()
            eng.advance()
        torch.cuda.synchronize()
        return [o.cpu().numpy().view(np.uint16) for o in outs]

    want = chain(torch.cuda.synchronize)
    assert eng.status() == 0 and all(np.isfinite(w.view(np.float16)).all() for w in want)
    for _ in range(4):
        assert all(np.array_equal(a, b) for a, b in zip(chain(lambda: None), want))
    assert eng.status() == 0
