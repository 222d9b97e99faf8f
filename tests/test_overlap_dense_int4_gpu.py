"""int4 weights that are turned into bf16 in a step whose kernels start early: the first product waits for the kernel that writes them."""
import pytest
import torch

from onnx_genai_b200 import ops
from onnx_genai_b200.ops import quant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [9, 300])
def test_the_first_product_comes_after_its_weight(monkeypatch, m):
    monkeypatch.setattr(quant.QuantLinear, "large_m", "dense")
    g = torch.Generator(device="cuda").manual_seed(m)
    n, k = 1152, 896
    q = torch.randint(0, 256, (n, k // 32, 16), dtype=torch.uint8, device="cuda", generator=g)
    lin = quant.QuantLinear(q, torch.rand(n, k // 32, device="cuda", generator=g).bfloat16() * 0.01, k=k)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    early, gemm = [], quant._gemm

    def product(*args, **kw):
        early.append(ops._scopes.now[1])
        return gemm(*args, **kw)

    monkeypatch.setattr(quant, "_gemm", product)
    with ops.launch_scope(ops.rows_workspace(m, "cuda"), True):
        outs = [lin(x).clone() for _ in range(2)]
    assert early == [False, True]
    want = x.double() @ lin.dense(torch.bfloat16).double().cuda().t()
    for out in outs:
        assert bool(((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + 2e-4 * want.abs().max()).all())
    ops.check_status()
