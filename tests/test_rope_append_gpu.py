"""Rotary embedding with the KV-page append, in all its forms."""
import pytest
import torch

from onnx_genai_b200 import ops
from onnx_genai_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("hq,hkv,d,rotary,interleaved", [(28, 4, 128, 128, False), (14, 2, 64, 64, False), (3, 1, 128, 64, False), (2, 2, 64, 16, False),
                                                         (4, 2, 64, 24, False), (4, 2, 64, 64, True)])
@pytest.mark.parametrize("t", [1, 37])
def test_rope_kv_append_forms(hq, hkv, d, rotary, interleaved, t):
    """Rotations in 16-byte pieces and one pair at a time: partial rotations, the part of a key that stays, rows that are not cached."""
    g = torch.Generator(device="cuda").manual_seed(t + rotary)
    pages = 4
    qkv = torch.randn(t, (hq + 2 * hkv) * d, device=DEV, generator=g).bfloat16()
    pos = torch.randint(0, 500, (t,), dtype=torch.int32, device=DEV, generator=g)
    slots = torch.randperm(pages * ref.PAGE, device=DEV, generator=g)[:t].to(torch.int32)
    if t > 3:
        slots[3] = -1
    cs = ref.rope_table(512, rotary, 1e6, DEV)
    pool = torch.zeros(pages, hkv, 2, ref.PAGE, d, device=DEV, dtype=torch.bfloat16)
    want, want_pool = qkv.clone(), pool.clone()
    ref.rope_kv_append(want, pos, slots, cs, want_pool, hq, hkv, d, rotary, interleaved)
    ops.rope_kv_append(qkv, pos, slots, cs, pool, hq, hkv, d, rotary, interleaved)
    ops.check_status()
    # one bf16 rounding of a sum of two products each
    assert float((qkv.float() - want.float()).abs().max()) <= 2 ** -7 * float(want.float().abs().max())
    assert float((pool.float() - want_pool.float()).abs().max()) <= 2 ** -7 * float(want_pool.float().abs().max())
