"""How prompts over one-byte pages share a tile's keys, built with the host compiler."""
import shutil
import subprocess
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parent.parent / "csrc" / "kernels"
MAIN = r"""
#include <cstdio>
#include "attention_plan.h"
int main() {
  int tiles, rows, hkv, group, blocks;
  long long keys;
  while (std::scanf("%d %d %d %d %lld %d", &tiles, &rows, &hkv, &group, &keys, &blocks) == 6) {
    const int s = ogb::prefill_splits(tiles, rows, hkv, group, keys, 148);
    std::printf("%d %d\n", s, ogb::prefill_shares(s, blocks));
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

    def ask(*row):
        out = subprocess.run([str(d / "main")], input=" ".join(map(str, row)), capture_output=True, text=True, check=True).stdout
        return tuple(map(int, out.split()))

    return ask


# tiles, their rows, KV heads, group, keys that no context exceeds, blocks of 64 keys -> cluster, CTAs that share
@pytest.mark.parametrize("sizes,want", [
    ((4, 256, 4, 7, 32768, 2), (1, 1)),          # 112 CTAs of full tiles: 18 -> 123 us in clusters of 8
    ((4, 68, 4, 7, 32768, 2), (2, 1)),           # 17 rows: a tile is two heads
    ((8, 128, 4, 7, 448, 7), (1, 1)),            # too few keys to share
    ((8, 128, 4, 7, 32768, 188), (2, 2)),        # 16 rows against 12000 keys: 1087 -> 327 us
    ((1, 16, 4, 7, 32768, 16), (8, 8)), ((1, 16, 4, 7, 1000, 15), (8, 4)), ((1, 16, 4, 7, 32768, 94), (8, 8)),
    ((1, 16, 4, 7, 32768, 7), (8, 1)), ((1, 16, 4, 7, 32768, 8), (8, 4)),
    ((64, 1024, 8, 4, 32768, 94), (1, 1)),       # the chip is full
    ((3, 3, 1, 1, 32768, 5), (8, 1)), ((1, 1, 1, 1, 32768, 1), (8, 1)),
])
def test_shares(plan, sizes, want):
    assert plan(*sizes) == want


def test_a_share_is_two_blocks_at_least(plan):
    for blocks in (1, 2, 3, 4, 7, 8, 15, 16, 31, 32, 33, 500):
        splits, shares = plan(1, 16, 1, 1, 1 << 20, blocks)
        assert shares <= splits and (shares == 1 or blocks >= 2 * shares)
