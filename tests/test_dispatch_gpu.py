"""Which form a layer takes (0: streaming, otherwise the CTAs of a cluster), where the lines lie close: on a GPU of 148 SMs."""
import pytest
import torch

import triebwerk_b200 as tq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,H,Hkv,G,slot,form", [
    # fp16 slots of one chunk: few tiles per warp stay in the cluster form
    (0, 8, 8, 12, 288, 1), (0, 8, 8, 12, 352, 1), (0, 16, 8, 12, 416, 0), (0, 16, 4, 32, 288, 1), (0, 16, 4, 32, 352, 0), (0, 16, 8, 48, 288, 0), (0, 16, 8, 37, 512, 1),
    # 4-bit clusters that would fill the GPU leave the next layer's half of it, unless there is no streaming form and the chains get long; smaller ones only
    # where slots are short
    (4, 32, 4, 2, 4000, 8), (4, 32, 4, 3, 1024, 4), (4, 32, 4, 3, 1056, 8), (4, 32, 4, 3, 6016, 8), (4, 40, 5, 1, 4000, 16), (4, 56, 7, 2, 2048, 8),
    (4, 40, 8, 1, 4000, 8), (4, 40, 8, 2, 1504, 4), (4, 40, 8, 4, 1504, 4), (2, 40, 8, 1, 4000, 16), (4, 24, 2, 2, 4000, 8), (4, 40, 8, 2, 10240, 4), (4, 40, 8, 2, 10272, 8),
    (4, 40, 8, 1, 32000, 8), (4, 24, 2, 4, 16000, 8),
])
def test_form_of_a_layer(bits, H, Hkv, G, slot, form):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("lines of another GPU")
    eng = tq.Engine(slot, bits, num_layers=1, num_heads=H, num_kv_heads=Hkv, head_dim=128)
    eng.alloc_batch(G, slot)
    assert tq.lib().tq_engine_decode_form(eng._h, 0) == form
