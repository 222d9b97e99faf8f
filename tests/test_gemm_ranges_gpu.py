"""Products with few rows over more tiles than SMs, which sum in ranges, at the sizes where they are the faster form: plain and gated (two
accumulators a tile), against an fp64 product; launches that follow one another, eager and replayed, find the counters of shared tiles at zero."""
import pytest
import torch

from onnx_genai_b200 import ops
from onnx_genai_b200.ops import _native

pytestmark = pytest.mark.gpu


# one bf16 rounding of an fp32 sum of products of N(0, 1) and N(0, 0.05)
def _check(got, want):
    err = (got.double() - want).abs()
    assert bool((err <= want.abs() * 2.0 ** -8 + 2e-4 * want.abs().max()).all()), float(err.max())


@pytest.mark.parametrize("m,n,k", [(1, 148 * 128 + 8, 3592), (17, 148 * 128 + 8, 3592), (32, 40000, 1640), (9, 65544, 1032), (48, 65544, 2824), (33, 65544, 2824)])
def test_plain(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).bfloat16()
    bias = torch.randn(n, device="cuda", generator=g).bfloat16()
    assert _native.load().ogb_rows_in_ranges(m, n, k, 0)
    want = a.double() @ w.double().t()
    out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    workspace = ops.rows_workspace(m, "cuda")      # outlives the graph
    with ops.launch_scope(workspace):
        for _ in range(3):
            _check(ops.gemm(a, w, bias=bias, out=out), want + bias.double())
        _check(ops.gemm(a, w, out_f32=True).bfloat16(), want)
        first = ops.gemm(a, w, out=out).clone()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ops.gemm(a, w, out=out)
    for _ in range(3):
        out.zero_()
        graph.replay()
        assert torch.equal(out, first)
    ops.check_status()


@pytest.mark.parametrize("m", [1, 17, 32])
@pytest.mark.parametrize("inter,k", [(149 * 128, 1672), (24576, 2056)])
def test_gated(m, inter, k):
    g = torch.Generator(device="cuda").manual_seed(m + inter)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    gate, up = ((torch.randn(inter, k, device="cuda", generator=g) * 0.05).bfloat16() for _ in range(2))
    assert _native.load().ogb_rows_in_ranges(m, 2 * inter, k, 1)
    x, y = a.double() @ gate.double().t(), a.double() @ up.double().t()
    want, packed = torch.nn.functional.silu(x) * y, ops.pack_gate_up(gate, up, 128)
    for _ in range(3):
        _check(ops.gemm(a, packed, epilogue="swiglu", swiglu_half=128), want)
    ops.check_status()
