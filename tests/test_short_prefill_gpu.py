"""Prefill tiles that take several heads of a KV head, and clusters that share a tile's keys: against the fp32 statement."""
import pytest
import torch

from onnx_genai_b200 import ops
from onnx_genai_b200.ops import reference as ref
from test_kernels_gpu import _make_paged, _make_paged_fp8, _rel_err

pytestmark = pytest.mark.gpu


def _run(pool, table, scales, q_lens, ctx, hq, hkv, d, window):
    t = sum(q_lens)
    g = torch.Generator(device="cuda").manual_seed(t + hq)
    q = torch.randn(t, (hq + 2 * hkv) * d, device="cuda", generator=g).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    cu, ctx_t = i32([0] + torch.tensor(q_lens).cumsum(0).tolist()), i32(ctx)
    ts, tq = ops.prefill_tiles(q_lens)
    out = torch.full((t, hq * d), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.paged_prefill(q, out, pool, table, ctx_t, cu, i32(ts), i32(tq), len(ts), hq, hkv, d, window=window, kv_scales=scales)
    ops.check_status()
    want = ref.paged_attention(q, pool, table, ctx_t, cu, hq, hkv, d, window=window, kv_scales=scales)
    for a, b in zip(cu[:-1].tolist(), cu[1:].tolist()):        # every sequence on its own: a short one must not hide in the norm
        assert _rel_err(out[a:b], want[a:b]) < 2e-2, (a, b)


Q_LENS = [1, 8, 9, 16, 17, 32, 33, 64, 65, 80, 128 + 3]


@pytest.mark.parametrize("hq,hkv,d", [(28, 4, 128), (14, 2, 64), (3, 1, 128), (16, 1, 64), (9, 1, 128), (4, 4, 64)])
@pytest.mark.parametrize("window", [0, 100])
def test_bf16_pages(hq, hkv, d, window):
    ctx = [n + 37 * i * i for i, n in enumerate(Q_LENS)]
    pool, table = _make_paged(len(ctx), ctx, hkv, d, seed=3)
    _run(pool, table, None, Q_LENS, ctx, hq, hkv, d, window)


@pytest.mark.parametrize("fmt", ["fp8", "int8", "e5m2"])
@pytest.mark.parametrize("hq,hkv", [(28, 4), (3, 1), (16, 1), (4, 4)])
@pytest.mark.parametrize("q_lens", [Q_LENS, [16], [5, 33], [200]])
@pytest.mark.parametrize("window", [0, 100])
def test_one_byte_pages(fmt, hq, hkv, q_lens, window):
    ctx = [n + 211 * i * i + 40 for i, n in enumerate(q_lens)]
    pool, scales, table = _make_paged_fp8(ctx, hkv, 128, fmt=fmt)
    _run(pool, table, scales, q_lens, ctx, hq, hkv, 128, window)
