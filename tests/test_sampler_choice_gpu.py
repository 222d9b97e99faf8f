"""Both sides of the line between a cluster and a CTA per row pick the tokens of the scalar sampler, which the same logits in fp32 take."""
import pytest
import torch

from onnx_genai_b200 import ops
from test_sampler_cluster_gpu import _rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["plain", "equal", "near", "tiny", "masked", "nan"])
@pytest.mark.parametrize("rows,vocab", [(32, 1016), (33, 1016), (64, 32768), (65, 32768), (200, 114680), (256, 114688)])
def test_tokens(kind, rows, vocab):
    g = torch.Generator(device="cuda").manual_seed(rows + vocab)
    x = _rows(kind, rows, vocab, g)
    pick = lambda *v: torch.tensor(v, device="cuda")[torch.randint(0, len(v), (rows,), device="cuda", generator=g)]
    for _ in range(2):
        args = (pick(0.0, 0.3, 0.7, 1.0, 5.0, 1e-30), pick(0, 1, 5, 50, 2000, 1 << 30).int(), pick(1.0, 0.9, 0.5, 0.999, 1e-6), pick(0.0, 0.0, 0.05, 1.0),
                torch.rand(rows, device="cuda", generator=g))
        assert torch.equal(ops.sample(x, *args), ops.sample(x.float(), *args))
