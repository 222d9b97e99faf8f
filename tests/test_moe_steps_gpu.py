"""The permutation of routes by expert in one CTA and in several launches, the combination of the experts' rows, and 32-bit router logits."""
import pytest
import torch

from onnx_genai_b200.ops import _native
from onnx_genai_b200.ops import moe as moe_ops
from onnx_genai_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,k,experts,e0", [(1, 1, 1, 0), (32, 8, 128, 0), (33, 8, 64, 32), (512, 8, 256, 0), (513, 8, 128, 0), (300, 6, 3, 1)])
def test_permutation(tokens, k, experts, e0):
    g = torch.Generator(device="cuda").manual_seed(tokens + experts)
    total = experts + 2 * e0
    ids = torch.stack([torch.randperm(max(total, k), device="cuda", generator=g)[:k] for _ in range(tokens)]).int().flatten()
    routes = tokens * k
    max_mtiles = (routes + 127) // 128 + experts
    i32 = lambda n: torch.full((n,), -7, dtype=torch.int32, device="cuda")
    counts, offsets, cursor, order, place, tab, meta = (i32(n) for n in (experts, experts + 1, experts, routes, routes, 4 * max_mtiles, 2))
    rc = _native.load().ogb_moe_permute(ids.data_ptr(), counts.data_ptr(), offsets.data_ptr(), cursor.data_ptr(), order.data_ptr(), place.data_ptr(),
                                        tab.data_ptr(), meta.data_ptr(), tokens, k, e0, experts, max_mtiles, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    local = ids.long() - e0
    mine = (local >= 0) & (local < experts)
    want = torch.bincount(local[mine], minlength=experts)
    starts = torch.cat([want.new_zeros(1), want.cumsum(0)])
    assert torch.equal(offsets.long(), starts)
    assert int(meta[1]) == int(mine.sum())
    assert bool((place[~mine] == -1).all())
    n = int(mine.sum())
    assert torch.equal(place[mine].long().sort().values, torch.arange(n, device="cuda"))
    assert torch.equal(order[:n].long()[place[mine].long()], mine.nonzero().flatten())
    assert bool((place[mine] >= starts[local[mine]]).all()) and bool((place[mine] < starts[local[mine] + 1]).all())
    tiles = [[e, r, int(starts[e + 1]), 0] for e in range(experts) for r in range(int(starts[e]), int(starts[e + 1]), 128)]
    assert int(meta[0]) == len(tiles)
    assert tab[: 4 * len(tiles)].view(-1, 4).tolist() == tiles


@pytest.mark.parametrize("t,k,hidden", [(1, 1, 8), (5, 8, 2048), (3, 9, 1032), (2, 32, 1024)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_combination(t, k, hidden, accumulate):
    g = torch.Generator(device="cuda").manual_seed(t + k)
    ys = torch.randn(t * k, hidden, device="cuda", generator=g).bfloat16()
    place = torch.randperm(t * k, device="cuda", generator=g).int().view(t, k)
    place[0, -1] = -1 if k > 1 else place[0, -1]
    w = torch.rand(t, k, device="cuda", generator=g)
    out = torch.randn(t, hidden, device="cuda", generator=g).bfloat16()
    want = (out.double() if accumulate else 0.0) + (ys.double()[place.long().clamp_min(0)] * (w.double() * (place >= 0))[..., None]).sum(1)
    rc = _native.load().ogb_moe_combine(ys.data_ptr(), place.data_ptr(), w.data_ptr(), out.data_ptr(), t, k, hidden, accumulate,
                                        torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert bool(((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all())      # one bf16 rounding of an fp32 sum


def test_experts_take_router_logits_of_both_widths():
    g = torch.Generator(device="cuda").manual_seed(5)
    t, e, k, hidden, inter = 9, 16, 4, 256, 128
    h = torch.randn(t, hidden, device="cuda", generator=g).bfloat16()
    gu = (torch.randn(e, 2 * inter, hidden, device="cuda", generator=g) * 0.05).bfloat16()
    down = (torch.randn(e, hidden, inter, device="cuda", generator=g) * 0.05).bfloat16()
    logits = torch.randn(t, e, device="cuda", generator=g).bfloat16()
    ws = moe_ops.MoEWorkspace(t, k, e, hidden, inter, "cuda")
    outs = [moe_ops.moe_experts(h, x, gu, down, ws, torch.zeros_like(h), k, True, 128).clone() for x in (logits, logits.float())]
    assert torch.equal(*outs)
    ids, w = ref.moe_route(logits, k, True)
    assert torch.equal(ws.topk_ids[: t * k].view(t, k).sort(1).values.cpu(), ids.int().sort(1).values.cpu())
