"""The settings that a step gives the kernels launched by its thread: scopes nest, and threads have their own.  A library that keeps a record
stands in for the kernels."""
import threading

import pytest
import torch

from onnx_genai_b200 import ops
from onnx_genai_b200.ops import _native


class _Library:
    def __init__(self):
        self.calls, self.sums = [], False

    def ogb_launch_scope(self, ws, size, overlap):
        self.calls.append((threading.get_ident(), ws, size, overlap))

    def ogb_tile_sums(self, on):
        old, self.sums = self.sums, bool(on)
        return int(old)


@pytest.fixture
def library(monkeypatch):
    lib = _Library()
    monkeypatch.setattr(_native, "load", lambda: lib)
    return lib


def _last(lib, thread=None):
    return [c[1:] for c in lib.calls if c[0] == (thread or threading.get_ident())][-1]


def test_a_scope_inside_another_gives_it_back(library):
    outer, inner = torch.zeros(64, dtype=torch.uint8), torch.zeros(32, dtype=torch.uint8)
    with ops.launch_scope(outer, True):
        with pytest.raises(RuntimeError):
            with ops.launch_scope(inner):
                assert _last(library) == (inner.data_ptr(), 32, 0)
                raise RuntimeError
        assert _last(library) == (outer.data_ptr(), 64, 1)
    assert _last(library) == (0, 0, 0)


def test_threads_have_scopes_of_their_own(library):
    outer, other = torch.zeros(64, dtype=torch.uint8), torch.zeros(32, dtype=torch.uint8)
    seen = []

    def step():
        with ops.launch_scope(other):
            pass
        seen.append(_last(library))

    with ops.launch_scope(outer, True):
        t = threading.Thread(target=step)
        t.start()
        t.join()
        assert seen == [(0, 0, 0)]
        assert _last(library) == (outer.data_ptr(), 64, 1)


def test_sums_by_tiles_nest(library):
    with ops.tile_sums():
        with ops.tile_sums(False):
            assert not library.sums
        assert library.sums
    assert not library.sums


def test_kernels_in_order_inside_a_scope(library):
    with ops.in_order():
        pass
    assert not library.calls                      # outside a scope nothing starts early
    ws = torch.zeros(64, dtype=torch.uint8)
    with ops.launch_scope(ws, True):
        with ops.in_order():
            assert _last(library) == (ws.data_ptr(), 64, 0)
        assert _last(library) == (ws.data_ptr(), 64, 1)
