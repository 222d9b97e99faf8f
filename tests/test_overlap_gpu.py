"""Steps whose kernels start early give what steps without it give, bit for bit: eager and replayed, every kind of page and weight."""
import numpy as np
import pytest
import torch

from onnx_genai_b200.engine.llm_engine import EngineConfig, LLMEngine
from onnx_genai_b200.models.config import preset

pytestmark = pytest.mark.gpu


def _texts(overlap, name, kv, graphs, **over):
    cfg = preset(name, num_layers=3, vocab=4096, **over)
    eng = LLMEngine(EngineConfig(model=cfg, num_pages=512, max_seqs=8, max_tokens_per_step=256, max_seq_len=640, kv_dtype=kv, cuda_graphs=graphs),
                    device="cuda:0")
    eng.model.overlap = overlap and eng.model.overlap
    rng = np.random.default_rng(3)
    prompts = [rng.integers(0, cfg.vocab, size=n).astype(np.int32) for n in (1, 33, 300, 64, 130)]
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
    for a, b in zip(_texts(True, name, kv, graphs), _texts(False, name, kv, graphs)):
        assert torch.equal(a, b)
