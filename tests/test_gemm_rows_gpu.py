"""Products with few rows against an fp64 product: the edges of the row padding, of the tiles of W, of K and of shared tiles."""
import pytest
import torch

from onnx_genai_b200 import ops

pytestmark = pytest.mark.gpu


# bf16 operands are exact in fp64; an fp32 sum of K products of N(0, 1) and N(0, 0.05) rounds to well under 1e-4 of its size, so one
# bf16 rounding of the result (2^-9 of its size) is what remains
def _check(got, want):
    err = (got.double() - want).abs()
    assert bool((err <= want.abs() * 2.0 ** -8 + 2e-4 * want.abs().max()).all()), float(err.max())


@pytest.mark.parametrize("m", [1, 16, 17, 33, 128, 129, 200, 256])
@pytest.mark.parametrize("n,k", [(128, 64), (136, 72), (3584, 512), (1000, 4160), (520, 8)])
@pytest.mark.parametrize("epilogue,with_bias", [("none", True), ("none", False), ("residual", True), ("residual", False)])
def test_plain_products(m, n, k, epilogue, with_bias):
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n + k)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).bfloat16()
    bias = torch.randn(n, device="cuda", generator=g).bfloat16() if with_bias else None
    res = torch.randn(m, n, device="cuda", generator=g).bfloat16() if epilogue == "residual" else None
    want = a.double() @ w.double().t() + (bias.double() if with_bias else 0.0) + (res.double() if res is not None else 0.0)
    for _ in range(2):          # the second launch finds the counters as the first did
        _check(ops.gemm(a, w, bias=bias, residual=res, epilogue=epilogue), want)
    if res is None:
        assert float((ops.gemm(a, w, bias=bias, out_f32=True).double() - want).abs().max()) < 2e-4 * float(want.abs().max())
    else:                       # in place over the residual
        out = res.clone()
        ops.gemm(a, w, bias=bias, residual=out, epilogue=epilogue, out=out)
        _check(out, want)
    ops.check_status()


@pytest.mark.parametrize("m", [1, 17, 48])
@pytest.mark.parametrize("n,k", [(148 * 128 + 8, 64), (20000, 136), (32000, 448)])
def test_more_tiles_than_sms_in_ranges(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).bfloat16()
    want = a.double() @ w.double().t()
    for _ in range(3):          # the counters of shared tiles wrap
        _check(ops.gemm(a, w), want)
    ops.check_status()


@pytest.mark.parametrize("m,n,k", [(2304, 1280, 18944), (300, 18952, 2048)])
def test_whole_waves_and_a_cut_last_one(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).bfloat16()
    want = a.double() @ w.double().t()
    for _ in range(2):
        _check(ops.gemm(a, w, bn=64), want)
        _check(ops.gemm(a, w), want)
    ops.check_status()


@pytest.mark.parametrize("m", [1, 31, 32, 130])
@pytest.mark.parametrize("inter,k", [(128, 64), (640, 200), (4096, 896)])
def test_gated_products(m, inter, k):
    g = torch.Generator(device="cuda").manual_seed(m + inter)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    gate, up = ((torch.randn(inter, k, device="cuda", generator=g) * 0.05).bfloat16() for _ in range(2))
    x, y = a.double() @ gate.double().t(), a.double() @ up.double().t()
    _check(ops.gemm(a, ops.pack_gate_up(gate, up, 128), epilogue="swiglu", swiglu_half=128), torch.nn.functional.silu(x) * y)
    ops.check_status()


@pytest.mark.parametrize("m,n", [(3, 1536), (256, 1536), (3, 20000)])
def test_a_captured_product_uses_the_scope_of_its_launch(m, n):
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn(m, 2048, device="cuda", generator=g).bfloat16()
    w = (torch.randn(n, 2048, device="cuda", generator=g) * 0.05).bfloat16()
    out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    workspace = ops.rows_workspace(m, "cuda")
    with ops.launch_scope(workspace):
        ops.gemm(a, w, out=out)
        torch.cuda.synchronize()
        first = out.clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ops.gemm(a, w, out=out)
    for _ in range(3):
        out.zero_()
        graph.replay()
        assert torch.equal(out, first)
    ops.check_status()
