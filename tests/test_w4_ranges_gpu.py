"""int4 products with few rows over more tiles than SMs, which sum in ranges: plain and gated (two accumulators a tile), the dequantisers' walk over
tiles that two CTAs share, and counters that later launches find at zero.  Against an fp64 product of the dequantised weights."""
import pytest
import torch

from onnx_genai_b200 import ops
from onnx_genai_b200.ops import _native
from test_w4_rows_gpu import _check, _linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(5, 148 * 128 + 32, 1568), (17, 148 * 128 + 40, 1568), (32, 20000, 1600), (48, 20000, 3104), (33, 148 * 128 + 8, 3072), (8, 33024, 1568)])
@pytest.mark.parametrize("zp,f32", [(False, False), (True, True)])
def test_plain(m, n, k, zp, f32):
    assert _native.load().ogb_rows_in_ranges(m, n, k, 2)
    g = torch.Generator(device="cuda").manual_seed(m + n)
    lin, w, b = _linear(n, k, g, zp, f32, bias=zp)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    want = x.double() @ w.t() + (b.double() if b is not None else 0.0)
    with ops.launch_scope(ops.rows_workspace(m, "cuda")):
        for _ in range(3):
            _check(lin(x), want)
    _check(lin(x), want)                      # a workspace of its own
    ops.check_status()


@pytest.mark.parametrize("m,inter,k", [(5, 148 * 128 + 40, 96), (17, 20000, 320), (32, 19000, 896), (48, 20000, 1568)])
@pytest.mark.parametrize("zp", [False, True])
def test_gated(m, inter, k, zp):
    assert _native.load().ogb_rows_in_ranges(m, 2 * inter, k, 3)
    g = torch.Generator(device="cuda").manual_seed(m + inter)
    lin, w, _ = _linear(2 * inter, k, g, zp, False)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    out = torch.empty(m, inter, dtype=torch.bfloat16, device="cuda")
    gate, up = (x.double() @ w.t()).split(inter, 1)
    want = torch.nn.functional.silu(gate) * up
    with ops.launch_scope(ops.rows_workspace(m, "cuda")):
        for _ in range(3):
            assert lin.gated(x, out)
            _check(out, want)
            out.zero_()
    assert lin.gated(x, out)
    _check(out, want)
    ops.check_status()


def test_sizes_that_are_left_to_the_projection_by_itself():
    g = torch.Generator(device="cuda").manual_seed(3)
    lin, _, _ = _linear(40960, 896, g, False, False)
    x = torch.randn(48, 896, device="cuda", generator=g).bfloat16()
    assert not lin.gated(x, torch.empty(48, 20480, dtype=torch.bfloat16, device="cuda"))
