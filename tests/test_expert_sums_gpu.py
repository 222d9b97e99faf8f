"""Models that choose among experts: scores as wide as on the CPU, and sums over K in the order in which the tile kernel adds, whatever the rows.
A sum in another order is as exact, but it lets experts of near-equal score change places, and one of them is 3 % of a row's logits."""
import numpy as np
import pytest
import torch

from onnx_genai_b200 import ops
from onnx_genai_b200.engine.llm_engine import EngineConfig, LLMEngine
from onnx_genai_b200.models import moe
from onnx_genai_b200.models.config import preset

pytestmark = pytest.mark.gpu
SMS = 148


@pytest.fixture
def whole_tiles():
    """No stream-K: every element of a product is one chain over K, the same for every tile width."""
    old = ops.set_stream_k(False)
    yield
    ops.set_stream_k(old)


class _Model:
    def __init__(self, cfg, rows):
        self.cfg, self.max_tokens, self.device, self.tp, self.rank = cfg, rows, torch.device("cuda"), 1, 0
        self.w = type("W", (), {"swiglu_half": 128})()


def test_scores_that_are_equal_in_bf16():
    """Scores of 1 and 1 + 2^-10 are the same number in bf16, and the lower expert takes the place, as in a tensor-parallel group."""
    cfg = preset("qwen3-30b-a3b", hidden=256)
    e, k, hid, inter, rows = cfg.moe.num_experts, cfg.moe.top_k, cfg.hidden, cfg.moe.expert_intermediate, 3
    router = torch.zeros(e, hid)
    router[:, 0], router[40:, 1] = 1.0, 2.0 ** -10
    h = torch.zeros(rows, hid)
    h[:, :2] = 1.0
    lw = type("L", (), {})()
    lw.router_w = router.bfloat16().cuda()
    lw.expert_gate_up = torch.zeros(e, 2 * inter, hid, dtype=torch.bfloat16, device="cuda")
    lw.expert_down = torch.zeros(e, hid, inter, dtype=torch.bfloat16, device="cuda")
    model = _Model(cfg, rows)
    moe.moe_forward(model, h.bfloat16().cuda(), lw, torch.zeros(rows, hid, dtype=torch.bfloat16, device="cuda"))
    got = model._moe_ws.topk_ids[: rows * k].view(rows, k).sort(1).values
    assert got.tolist() == [list(range(k))] * rows


@pytest.mark.parametrize("m", [1, 17, 128, 200, 256])
@pytest.mark.parametrize("n,k", [(128, 2048), (5120, 2048), (2048, 4096), (20480, 256)])
def test_few_rows_sum_as_many(whole_tiles, m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = (torch.randn(n, k, device="cuda", generator=g) * k ** -0.5).bfloat16()
    x = torch.randn(m, n, device="cuda", generator=g).bfloat16()
    with ops.tile_sums():
        assert torch.equal(ops.gemm(a, w), ops.gemm(a, w, bn=128))
        assert torch.equal(ops.gemm(a, w, residual=x, epilogue="residual"), ops.gemm(a, w, residual=x, epilogue="residual", bn=128))


def test_all_tiles_are_cut_into_ranges():
    """248 tiles of 256 columns on 148 SMs: a range per SM over the iterations of all of them, partials added in the order of the ranges."""
    m, n, k, bn = 128 * 31, 2048, 18944, 256
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = (torch.randn(n, k, device="cuda", generator=g) * k ** -0.5).bfloat16()
    with ops.tile_sums():
        got = ops.gemm(a, w, bn=bn, out_f32=True)
    blocks, tiles = k // 64, (m // 128) * (n // bn)
    base, rem = divmod(tiles * blocks, SMS)
    cuts = sorted({b * base + min(b, rem) for b in range(SMS + 1)})
    old = ops.set_stream_k(False)
    try:
        for t in (0, 1, 30, 31, 124, 147, 148, 200, 247):
            mt, nt = t % (m // 128), t // (m // 128)
            ats = [c - t * blocks for c in cuts if 0 < c - t * blocks < blocks]
            parts = [ops.gemm(a[mt * 128:(mt + 1) * 128, lo * 64:hi * 64].contiguous(), w[nt * bn:(nt + 1) * bn, lo * 64:hi * 64].contiguous(), bn=bn,
                              out_f32=True) for lo, hi in zip([0] + ats, ats + [blocks])]
            want = parts[-1]
            for part in parts[:-1]:
                want = want + part
            assert torch.equal(got[mt * 128:(mt + 1) * 128, nt * bn:(nt + 1) * bn], want)
    finally:
        ops.set_stream_k(old)


@pytest.mark.parametrize("kv", ["bf16", "int8"])
def test_a_models_layers_sum_so(whole_tiles, monkeypatch, kv):
    """Few rows through an expert model, as it is and with the tile kernel asked for by width."""
    cfg = preset("qwen3-30b-a3b", num_layers=2, vocab=4096)
    prompts = [np.random.default_rng(n).integers(0, cfg.vocab, size=n).astype(np.int32) for n in (1, 130)]
    gemm = ops.gemm

    def texts():
        eng = LLMEngine(EngineConfig(model=cfg, num_pages=64, max_seqs=4, max_tokens_per_step=256, max_seq_len=256, kv_dtype=kv), device="cuda:0")
        for p in prompts:
            eng.add_request(p, 6, ignore_eos=True)
        rows = []
        while eng.core.has_work:
            out = eng.step()
            rows.append(eng.model.x[: max(1, len(out.events))].clone())
        eng.check_device_status()
        return rows

    plain = texts()
    # the head stays as it is: the same tokens follow
    monkeypatch.setattr(ops, "gemm", lambda a, w, *args, **kw: gemm(a, w, *args, **({} if w.shape[0] == cfg.vocab else {"bn": 128}), **kw))
    tiles = texts()
    assert len(plain) == len(tiles) > 0
    assert all(torch.equal(a, b) for a, b in zip(plain, tiles))
