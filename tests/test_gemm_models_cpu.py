"""Bounded models of the products' fix-ups: whole waves behind cut tiles, and the counters of tiles shared by ranges."""
import pytest

from onnx_genai_b200.specs import shared_tiles, stream_k


@pytest.mark.parametrize("kw", [dict(ctas=4, slots=1, tiles=9, k_blocks=4, cut=1), dict(ctas=4, slots=2, tiles=7, k_blocks=5, cut=3),
                                dict(ctas=3, slots=1, tiles=8, k_blocks=7, cut=5), dict(ctas=5, slots=2, tiles=7, k_blocks=1, cut=2)])
def test_whole_waves_behind_cut_tiles_never_deadlock(kw):
    assert stream_k.check(**kw).ok


def test_upward_waits_deadlock_with_whole_waves_too():
    r = stream_k.check(ctas=4, slots=1, tiles=7, k_blocks=4, cut=3, guarded=False)
    assert not r.ok and r.kind == "deadlock"


@pytest.mark.parametrize("kw", [dict(ctas=3, tiles=4, k_blocks=2), dict(ctas=3, tiles=5, k_blocks=3), dict(ctas=4, tiles=5, k_blocks=3, launches=1),
                                dict(ctas=2, tiles=4, k_blocks=1)])
def test_shared_tiles_are_stored_once_and_counters_end_at_zero(kw):
    r = shared_tiles.check(**kw)
    assert r.ok, str(r)


def test_an_arrival_ahead_of_its_partial_is_found():
    r = shared_tiles.check(ctas=3, tiles=4, k_blocks=2, launches=1, broken="early")
    assert not r.ok and r.kind == "invariant", str(r)


def test_counters_that_do_not_wrap_are_found():
    r = shared_tiles.check(ctas=3, tiles=4, k_blocks=2, broken="sticky")
    assert not r.ok and r.kind == "deadlock", str(r)
