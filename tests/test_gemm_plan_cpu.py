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
  int scatter, steady, enabled, width, tiles, kb, sms;
  long long n;
  while (std::scanf("%d %d %d %d %lld %d %d %d", &scatter, &steady, &enabled, &width, &n, &tiles, &kb, &sms) == 8) {
    const ogb::SkRule r = ogb::sk_rule(scatter, steady, enabled, width, n, kb * 64);
    std::printf("%d %d %.9g\n", ogb::stream_k_applies(tiles, kb, sms, r) ? 1 : 0, r.cut(tiles, kb, sms), ogb::launch_cost(tiles, kb, sms, 1.f, r));
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
@pytest.mark.parametrize("width,n", [(256, 1024), (256, 1 << 24), (128, 1024)])
def test_all_tiles_are_cut(plan, scatter, steady, fix, width, n):
    for (tiles, kb), (on, cut, cost) in zip(SIZES, plan([(scatter, steady, 1, width, n, t, kb, 148) for t, kb in SIZES])):
        want_on, want_cost = _ranges_over_all_tiles(fix, tiles, kb, 148)
        assert (on, cut) == (want_on, tiles), (tiles, kb)
        assert cost == pytest.approx(want_cost, rel=1e-6)


@pytest.mark.parametrize("width,n", [(256, 1024), (256, 1 << 24), (192, 1024)])
def test_other_products_cut_the_last_wave(plan, width, n):
    """Whole waves follow the cut tiles where their main loops are long enough to hide the fix-ups; elsewhere all tiles of full width over a weight
    that stays in L2 are cut, and others are not."""
    cuts = set()
    for (tiles, kb), (on, cut, cost) in zip(SIZES, plan([(0, 0, 1, width, n, t, kb, 148) for t, kb in SIZES])):
        rest = tiles % 148
        last = tiles if tiles <= 148 else rest + 148 if 296 > 7 * rest else rest
        hidden = last == tiles or 25 * (1 + 148 / max(last, 1)) < 0.5 * kb
        all_else = width == 256 and n == 1024
        assert cut == (tiles if not hidden and all_else else last), (tiles, kb)
        waves = -(-tiles // 148)
        assert cost <= waves and (on or cost == waves)
        if cut == tiles:
            assert (on, cost) == pytest.approx(_ranges_over_all_tiles(40, tiles, kb, 148), rel=1e-6)
        elif not hidden:
            assert not on
        cuts.add((on, cut < tiles))
    assert cuts >= {(True, True), (True, False), (False, False)}
    assert not any(on for on, _, _ in plan([(0, 0, 0, width, n, t, kb, 148) for t, kb in SIZES]))


ROWS = r"""
#include <cstdio>
#include "gemm_plan.h"
int main() {
  int m, n, kb, gated, residual, sms;
  while (std::scanf("%d %d %d %d %d %d", &m, &n, &kb, &gated, &residual, &sms) == 6)
    std::printf("%d\n", ogb::rows_applies(m, n, kb, gated, residual, sms) ? 1 : 0);
}
"""


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("rows")
    (d / "main.cpp").write_text(ROWS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(KERNELS), str(d / "main.cpp"), "-o", str(d / "main")], check=True)

    def ask(m, n, k, gated, residual=False):
        out = subprocess.run([str(d / "main")], input=f"{m} {n} {-(-k // 64)} {int(gated)} {int(residual)} 148", capture_output=True, text=True, check=True).stdout
        return out.strip() == "1"

    return ask


# (rows, N, K, gated): where the kernels for few rows took 1.1 to 1.65 times the tile kernel's time, and where they took 0.4 to 0.9 of it
SLOWER = [(256, 7168, 896, False), (256, 16640, 896, False), (256, 9600, 2048, False), (128, 9600, 896, False), (256, 9600, 3584, False), (128, 3584, 896, False),
          (256, 18944, 8192, False), (64, 18944, 896, False), (1, 20000, 576, False), (48, 20000, 896, False), (16, 32000, 896, False), (48, 65536, 2048, False),
          (16, 151936, 576, False), (48, 151936, 896, False), (16, 49152, 896, True), (32, 37888, 2048, True)]
FASTER = [(1, 128, 2048, False), (256, 4608, 3584, False), (256, 3584, 18944, False), (64, 7168, 18944, False), (1, 18944, 3584, False), (16, 9600, 2048, False),
          (1, 152064, 3584, False), (48, 152064, 3584, False), (1, 151936, 896, False), (16, 128256, 2048, False), (32, 9728, 4096, True), (16, 37888, 3584, True),
          (8, 49152, 4096, True)]


@pytest.mark.parametrize("size", SLOWER)
def test_few_rows_are_left_to_the_tile_kernel_where_it_is_faster(rows, size):
    assert not rows(*size)


@pytest.mark.parametrize("size", FASTER)
def test_few_rows_have_their_own_kernel_where_that_is_faster(rows, size):
    assert rows(*size)


def test_sums_with_a_residual_stay_where_they_are_rounded_once(rows):
    assert all(rows(256, n, k, False, True) for n, k in [(128, 64), (3584, 512), (896, 896), (4608, 18944)])


W4 = r"""
#include <cstdio>
#include "gemm_plan.h"
int main() {
  int m, tiles, kb, gated, sms;
  while (std::scanf("%d %d %d %d %d", &m, &tiles, &kb, &gated, &sms) == 5) std::printf("%d\n", ogb::w4_rows_applies(m, tiles, kb, gated, sms) ? 1 : 0);
}
"""


# (rows, rows of W, K, gated, the kernels for few rows): 1.1 to 1.34 times the other kernel's time, or 0.33 to 0.9 of it
@pytest.mark.parametrize("m,n,k,gated,few", [
    (48, 32000, 896, 0, 0), (128, 14336, 2048, 0, 0), (128, 9728, 896, 0, 0), (128, 18944, 4096, 0, 0), (16, 9728, 4096, 0, 0), (8, 11008, 11008, 0, 0),
    (64, 6144, 896, 0, 0), (64, 6144, 2048, 0, 0), (48, 22016, 896, 0, 0), (48, 22016, 2048, 0, 0), (48, 40960, 896, 1, 0), (300, 896, 4864, 0, 0),
    (8, 896, 4864, 0, 1), (256, 4096, 4096, 0, 1), (48, 896, 896, 0, 1), (64, 1152, 896, 0, 1), (256, 6144, 11008, 0, 1), (8, 18944, 4096, 0, 1),
    (32, 22016, 4096, 0, 1), (48, 22016, 4864, 0, 1), (8, 32000, 4096, 0, 1), (64, 9728, 896, 1, 1), (160, 9728, 896, 1, 1), (16, 40960, 896, 1, 1)])
def test_int4_products_of_few_rows(tmp_path_factory, m, n, k, gated, few):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    d = tmp_path_factory.getbasetemp() / "w4"
    if not (d / "main").exists():
        d.mkdir()
        (d / "main.cpp").write_text(W4)
        subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(KERNELS), str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    tiles = -(-n // (2 if gated else 1) // 128)
    out = subprocess.run([str(d / "main")], input=f"{m} {tiles} {-(-k // 64)} {gated} 148", capture_output=True, text=True, check=True).stdout
    assert out.strip() == str(few)
