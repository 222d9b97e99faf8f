"""Steps whose kernels start early give what steps without it give, bit for bit: eager and replayed, bf16, e4m3 and int8 pages, bf16, int4 (heads of
64; up to four rows and more have kernels of their own) and expert weights."""
import types

import numpy as np
import pytest
import torch

from onnx_genai_b200 import ops
from onnx_genai_b200.engine.llm_engine import EngineConfig, LLMEngine
from onnx_genai_b200.models.config import preset
from onnx_genai_b200.models.decoder import DecoderWeights, LayerWeights

pytestmark = pytest.mark.gpu


def _int4_weights(cfg):
    g = torch.Generator(device="cuda").manual_seed(2)

    def matrix(n, k, bias=None):
        codes = torch.randint(0, 256, (n, k // 32, 16), dtype=torch.uint8, device="cuda", generator=g)
        scales = torch.empty(n, k // 32, device="cuda").uniform_(0.002, 0.0065, generator=g).bfloat16()
        return types.SimpleNamespace(q=codes, scales=scales, zp=None, bias=bias, k=k, block=32)

    draw = lambda *shape: torch.empty(*shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, 0.5, generator=g)
    ones = torch.ones(cfg.hidden, dtype=torch.bfloat16, device="cuda")
    layers = []
    for _ in range(cfg.num_layers):
        quant = {"qkv": [matrix(n, cfg.hidden, draw(n)) for n in (cfg.q_size, cfg.kv_size, cfg.kv_size)], "o": matrix(cfg.hidden, cfg.q_size),
                 "gate": matrix(cfg.intermediate, cfg.hidden), "up": matrix(cfg.intermediate, cfg.hidden), "down": matrix(cfg.hidden, cfg.intermediate)}
        layers.append(LayerWeights(ln1=ones, qkv_w=None, qkv_b=None, o_w=None, ln2=ones, quant=quant))
    embed = draw(cfg.vocab, cfg.hidden)
    return DecoderWeights(embed=embed, layers=layers, final_norm=ones, lm_head=embed, swiglu_half=128)


def _texts(overlap, name, kv, graphs, lengths=(1, 33, 300, 64, 130), int4=False, **over):
    cfg = preset(name, num_layers=3, vocab=4096, **over)
    eng = LLMEngine(EngineConfig(model=cfg, num_pages=512, max_seqs=8, max_tokens_per_step=256, max_seq_len=640, kv_dtype=kv, cuda_graphs=graphs),
                    weights=_int4_weights(cfg) if int4 else None, device="cuda:0")
    eng.model.overlap = overlap and eng.model.overlap
    rng = np.random.default_rng(3)
    prompts = [rng.integers(0, cfg.vocab, size=n).astype(np.int32) for n in lengths]
    ids = [eng.add_request(p, 24, ignore_eos=True) for p in prompts]
    rows = []
    while eng.core.has_work:
        out = eng.step()
        rows.append(eng.model.logits[: len(out.events)].clone())
    for i in ids:
        eng.core.release(i)
    eng.check_device_status()
    return rows


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("name,kv", [("qwen2.5-7b", "bf16"), ("qwen2.5-7b", "fp8"), ("qwen2.5-7b", "int8"), ("qwen3-30b-a3b", "bf16")])
def test_overlapped_steps(name, kv, graphs):
    _compare(name, kv, graphs)


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("lengths", [(1, 33, 300, 64, 130), (77,), (5, 300, 18, 2), (3,)])
def test_overlapped_steps_of_int4_weights(lengths, graphs):
    before = ops.launch_counts["w4a16_gemm"] + ops.launch_counts["w4a16_gemv_fused"]
    _compare("qwen2.5-0.5b", "bf16", graphs, lengths=lengths, int4=True)
    assert ops.launch_counts["w4a16_gemm"] + ops.launch_counts["w4a16_gemv_fused"] > before


def _compare(name, kv, graphs, **how):
    early, plain = _texts(True, name, kv, graphs, **how), _texts(False, name, kv, graphs, **how)
    assert len(early) == len(plain) > 0
    assert all(torch.equal(a, b) for a, b in zip(early, plain))
