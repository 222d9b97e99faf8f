"""Prompts of few rows that are enough for a tile to take several heads of its KV head (more tiles and heads than SMs): group sizes that do not
divide a tile, both head sizes; and the same tiles by themselves, which keep a head each.  Against the fp32 statement, and against each other."""
import pytest
import torch

from onnx_genai_b200 import ops
from onnx_genai_b200.ops import reference as ref
from test_kernels_gpu import _make_paged, _rel_err

pytestmark = pytest.mark.gpu


def _prefill(q, pool, table, ctx, q_lens, hq, hkv, d, window):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    cu = i32([0] + torch.tensor(q_lens).cumsum(0).tolist())
    ts, tq = ops.prefill_tiles(q_lens)
    out = torch.full((q.shape[0], hq * d), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.paged_prefill(q, out, pool, table, i32(ctx), cu, i32(ts), i32(tq), len(ts), hq, hkv, d, window=window)
    return out, cu, i32(ctx)


@pytest.mark.parametrize("hq,hkv,d", [(3, 1, 128), (9, 1, 128), (9, 1, 64), (14, 2, 64), (16, 16, 64)])
@pytest.mark.parametrize("window", [0, 100])
def test_many_and_few(hq, hkv, d, window):
    q_lens = [1, 8, 9, 16, 17, 32, 33, 64, 65, 80, 131] * (160 // (13 * hq) + 1)
    ctx = [n + 37 * (i % 11) ** 2 for i, n in enumerate(q_lens)]
    assert len(ops.prefill_tiles(q_lens)[0]) * hq > ops.num_sms()
    pool, table = _make_paged(len(ctx), ctx, hkv, d, seed=5)
    q = torch.randn(sum(q_lens), (hq + 2 * hkv) * d, device="cuda", generator=torch.Generator(device="cuda").manual_seed(hq)).bfloat16()
    out, cu, ctx_t = _prefill(q, pool, table, ctx, q_lens, hq, hkv, d, window)
    want = ref.paged_attention(q, pool, table, ctx_t, cu, hq, hkv, d, window=window)
    starts = cu.tolist()
    for s, (a, b) in enumerate(zip(starts, starts[1:])):
        assert _rel_err(out[a:b], want[a:b]) < 2e-2, (s, q_lens[s])
        if s < 11:            # a sequence alone: a head per tile
            alone, _, _ = _prefill(q[a:b].contiguous(), pool, table[s:s + 1].contiguous(), ctx[s:s + 1], q_lens[s:s + 1], hq, hkv, d, window)
            assert torch.equal(alone, out[a:b]), (s, q_lens[s])
    ops.check_status()
