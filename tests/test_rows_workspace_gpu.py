"""Products that need a workspace, called outside a model's step: it is zeroed in the order of their stream, lives as long as the call, and a
captured graph has its own."""
import pytest
import torch

from onnx_genai_b200 import ops
from onnx_genai_b200.ops import _native

pytestmark = pytest.mark.gpu


def _operands(m, n, k=3592):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).bfloat16()
    assert _native.load().ogb_rows_in_ranges(m, n, k, 0)
    with ops.launch_scope(ops.rows_workspace(m, "cuda")):
        return a, w, ops.gemm(a, w)


def test_streams_of_their_own():
    a, w, want = _operands(17, 20000)

    def streams(count):
        outs = []
        for _ in range(count):
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                outs += [ops.gemm(a, w) for _ in range(3)]
        torch.cuda.synchronize()
        assert all(torch.equal(o, want) for o in outs)
        return torch.cuda.mem_get_info()[0] + torch.cuda.memory_reserved()

    before = streams(2)             # modules are loaded
    # nothing stays behind a stream: its workspace (20 MB) was torch's, and goes back to it
    assert before - streams(6) < 32 << 20
    ops.check_status()


def test_a_graph_beside_the_stream_that_it_was_captured_on():
    a, w, want = _operands(32, 19000)
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(side):
        ops.gemm(a, w)
    side.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        captured = ops.gemm(a, w)
    outs = []
    for _ in range(20):
        with torch.cuda.stream(other):
            graph.replay()
        with torch.cuda.stream(side):
            outs.append(ops.gemm(a, w))
    torch.cuda.synchronize()
    assert torch.equal(captured, want)
    assert all(torch.equal(o, want) for o in outs)
    ops.check_status()
