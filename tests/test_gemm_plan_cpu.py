"""The tile kernel's choice of stream-K, built with the host compiler: tensor-parallel scatter products and the products of expert models divide
their work as they always have, with the constants measured for them."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

KERNELS = Path(__file__).resolve().parent.parent / "csrc" / "kernels"
MAIN = r"""
#include <cstdio>
#include "gemm_plan.h"
int main() {
  int scatter, steady, enabled, tiles, kb, sms;
  while (std::scanf("%d %d %d %d %d %d", &scatter, &steady, &enabled, &tiles, &kb, &sms) == 6) {
    const ogb::SkRule r = ogb::sk_rule(scatter, steady, enabled);
    std::printf("%d %d %.9g\n", ogb::stream_k_applies(tiles, kb, sms, r) ? 1 : 0, r.cut(tiles, sms), ogb::launch_cost(tiles, kb, sms, 1.f, r));
  }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("plan")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(KERNELS), str(d / "main.cpp"), "-o", str(d / "main")], check=True)

    def ask(rows):
        out = subprocess.run([str(d / "main")], input="\n".join(" ".join(map(str, r)) for r in rows), capture_output=True, text=True, check=True).stdout
        return [(bool(int(a)), int(b), float(c)) for a, b, c in (line.split() for line in out.splitlines())]

    return ask


def _ranges_over_all_tiles(fix, tiles, kb, sms):
    """Every tile cut into equal ranges: chosen, and its cost."""
    f = np.float32
    fix, shared = f(fix), f(sms) / f(tiles)
    if shared > f(6):
        fix = fix * shared / f(6)
    waves = -(-tiles // sms)
    cost = f(tiles) / f(sms) + fix / f(kb)
    on = tiles % sms != 0 and tiles * kb >= 2 * sms and cost < f(0.93) * f(waves)
    return bool(on), float(cost if on else f(waves))


SIZES = [(tiles, kb) for tiles in (1, 7, 24, 28, 100, 147, 148, 149, 160, 190, 191, 248, 296, 297, 400, 1000) for kb in (1, 2, 14, 32, 56, 64, 128, 296)]


@pytest.mark.parametrize("scatter,steady,fix", [(1, 0, 13), (1, 1, 13), (0, 1, 40)])
def test_all_tiles_are_cut(plan, scatter, steady, fix):
    for (tiles, kb), (on, cut, cost) in zip(SIZES, plan([(scatter, steady, 1, t, kb, 148) for t, kb in SIZES])):
        want_on, want_cost = _ranges_over_all_tiles(fix, tiles, kb, 148)
        assert (on, cut) == (want_on, tiles), (tiles, kb)
        assert cost == pytest.approx(want_cost, rel=1e-6)


def test_other_products_cut_the_last_wave(plan):
    for (tiles, kb), (on, cut, cost) in zip(SIZES, plan([(0, 0, 1, t, kb, 148) for t, kb in SIZES])):
        assert 0 < cut <= tiles or tiles % 148 == 0
        assert (tiles - cut) % 148 == 0                         # whole waves follow
        assert cut <= 148 + 148 * 2 // 7 + 1
        waves = -(-tiles // 148)
        assert cost <= waves and (on or cost == waves)
    assert not any(on for on, _, _ in plan([(0, 0, 0, t, kb, 148) for t, kb in SIZES]))
