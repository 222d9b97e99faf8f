"""What the cluster sampler's search for a threshold rests on, restated on the CPU."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "csrc" / "kernels" / "sampling_cluster.cuh").read_text()


def _constant(name):
    return int(re.search(rf"constexpr int {name} = (\d+)", SOURCE).group(1))


def test_cuts_end():
    """A bucket of ``width`` weights from ``w_min`` on takes [ceil(c width / n), ceil((c + 1) width / n)): the widest after each cut."""
    n = _constant("kClBuckets")
    for width in (1 << 30, (1 << 30) - (1 << 16), (1 << 20) + 1, 1025, 1024, 1023, 2, 1):
        cuts = 0
        while width > 1:
            widest = -(-width // n)
            probe = range(n) if width < 1 << 12 else (0, 1, n // 2, n - 1)
            assert all(-(-(c + 1) * width // n) - -(-c * width // n) <= widest for c in probe)
            width, cuts = widest, cuts + 1
        assert cuts <= _constant("kClMaxCuts")


def test_sums_and_searches_write_words_of_their_own():
    """cl_block_sum ends in reads without a barrier behind them, so what comes next must not write the same words: a search may come next."""
    search = SOURCE[SOURCE.index("auto find = "):]
    search = search[:search.index("\n  };")]
    assert "sh.sums" not in search
    uses = [m.start() for m in re.finditer(r"sh\.sums\[warp\] = ", SOURCE)]
    assert all("__syncthreads();" in SOURCE[at - 120:at] for at in uses)       # the others wait for the reads first


MAIN = r"""
#include <cstdio>
#include "sampling_plan.h"
int main() {
  int rows, vocab;
  while (std::scanf("%d %d", &rows, &vocab) == 2) std::printf("%d\n", ogb::sample_cluster_pays(rows, vocab) ? 1 : 0);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_rows_go_where_they_are_faster(tmp_path):
    """Sizes at which a cluster per row took 1.2 to 5 times the one-CTA sampler's time, and sizes at which it took 0.1 to 0.9 of it."""
    one_cta = [(256, 1024), (148, 4096), (64, 8192), (64, 16384), (148, 24576), (148, 32000), (256, 32000), (256, 50304), (256, 65536), (256, 81920)]
    cluster = [(1, 8), (16, 1024), (32, 8192), (48, 24576), (62, 32000), (74, 50304), (111, 65536), (148, 81920), (256, 128256), (512, 152064), (1, 524288)]
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-I", str(Path(__file__).resolve().parent.parent / "csrc" / "kernels"), str(tmp_path / "main.cpp"), "-o",
                    str(tmp_path / "main")], check=True)
    out = subprocess.run([str(tmp_path / "main")], input="\n".join(f"{r} {v}" for r, v in one_cta + cluster), capture_output=True, text=True, check=True).stdout
    assert out.split() == ["0"] * len(one_cta) + ["1"] * len(cluster)
