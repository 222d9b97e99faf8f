"""What the cluster sampler's search for a threshold rests on, restated on the CPU."""
import re
from pathlib import Path

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
