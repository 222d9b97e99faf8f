"""int4 products with few rows against an fp64 product of the dequantised weights."""
import pytest
import torch

from onnx_genai_b200 import ops
from onnx_genai_b200.ops.quant import QuantLinear

pytestmark = pytest.mark.gpu


def _linear(n, k, g, zp, f32, bias=False):
    kb = k // 32
    q = torch.randint(0, 256, (n, kb, 16), dtype=torch.uint8, device="cuda", generator=g)
    scales = torch.empty(n, kb, device="cuda").uniform_(0.002, 0.0065, generator=g).bfloat16()
    z = torch.randint(0, 256, (n, (kb + 1) // 2), dtype=torch.uint8, device="cuda", generator=g) if zp else None
    b = torch.randn(n, device="cuda", generator=g).bfloat16() if bias else None
    codes = torch.stack([q & 15, q >> 4], -1).reshape(n, kb, 32).double()
    zero = torch.stack([z & 15, z >> 4], -1).reshape(n, -1)[:, :kb].double()[..., None] if zp else 8.0
    # the kernel rounds a weight to bf16 once; as does this
    w = ((codes - zero) * scales.double()[..., None]).float().bfloat16().double().reshape(n, k)
    return QuantLinear(q, scales.float() if f32 else scales, z, b, k), w, b


# bf16 operands, fp32 sums, one bf16 rounding of the result
def _check(got, want):
    err = (got.double() - want).abs()
    assert bool((err <= want.abs() * 2.0 ** -8 + 2e-4 * want.abs().max()).all()), float(err.max())


@pytest.mark.parametrize("m", [9, 16, 64, 65, 200, 256])
@pytest.mark.parametrize("n,k", [(128, 32), (896, 4864), (1152, 896), (160, 96), (1000, 2080)])
@pytest.mark.parametrize("zp,f32", [(False, False), (True, True)])
def test_products(m, n, k, zp, f32):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    lin, w, b = _linear(n, k, g, zp, f32, bias=zp)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    want = x.double() @ w.t() + (b.double() if b is not None else 0.0)
    for _ in range(2):
        _check(lin(x), want)
    ops.check_status()


@pytest.mark.parametrize("m", [5, 64, 129, 160])
@pytest.mark.parametrize("inter,k", [(128, 64), (4864, 896), (200, 352)])
@pytest.mark.parametrize("zp", [False, True])
def test_gated_products(m, inter, k, zp):
    g = torch.Generator(device="cuda").manual_seed(m + inter + k)
    lin, w, _ = _linear(2 * inter, k, g, zp, False)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    out = torch.empty(m, inter, dtype=torch.bfloat16, device="cuda")
    assert lin.gated(x, out)
    gate, up = (x.double() @ w.t()).split(inter, 1)
    _check(out, torch.nn.functional.silu(gate) * up)
    ops.check_status()
