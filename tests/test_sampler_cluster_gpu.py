"""The cluster sampler against the one-CTA sampler, which the same logits in fp32 take: equal weights, so equal tokens."""
import pytest
import torch

from onnx_genai_b200 import ops

pytestmark = pytest.mark.gpu


def _rows(kind, rows, vocab, g):
    x = torch.randn(rows, vocab, device="cuda", generator=g) * 2.0
    if kind == "equal":                       # every weight the same: no bucket can be cut
        x.fill_(1.5)
    elif kind == "near":                      # thousands of weights in one bucket
        x = 8.0 + torch.randint(0, 3, (rows, vocab), device="cuda", generator=g).float() * 0.0625
    elif kind == "tiny":                      # thousands of different weights in one bucket
        x = x * 1e-6
        x[:, 3] = 20.0
    elif kind == "masked":                    # all but a few at the type's lowest value, or at -inf
        keep = x[:, ::37].clone()
        x.fill_(torch.finfo(torch.bfloat16).min)
        x[1::2] = float("-inf")
        x[:, ::37] = keep
    elif kind == "nan":
        x[:, 1::3] = float("nan")
        x[0] = float("nan")
        x[1 % rows, 0] = float("inf")
        x[2 % rows] = float("-inf")
    return x.bfloat16()


@pytest.mark.parametrize("kind", ["plain", "equal", "near", "tiny", "masked", "nan"])
@pytest.mark.parametrize("rows,vocab", [(1, 8), (5, 24), (3, 1016), (64, 32000), (2, 152064), (2, 524288), (1, 524296)])
def test_tokens_are_those_of_the_one_cta_kernel(kind, rows, vocab):
    g = torch.Generator(device="cuda").manual_seed(rows + vocab)
    x = _rows(kind, rows, vocab, g)
    pick = lambda *v: torch.tensor(v, device="cuda")[torch.randint(0, len(v), (rows,), device="cuda", generator=g)]
    for _ in range(6):
        args = (pick(0.0, 0.3, 0.7, 1.0, 5.0, 1e-30), pick(0, 1, 5, 50, 2000, 1 << 30).int(), pick(1.0, 0.9, 0.5, 0.999, 1e-6), pick(0.0, 0.0, 0.05, 1.0),
                torch.rand(rows, device="cuda", generator=g))
        assert torch.equal(ops.sample(x, *args), ops.sample(x.float(), *args))
