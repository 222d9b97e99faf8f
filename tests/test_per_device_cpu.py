"""Kernel attributes belong to a device: what one device was prepared for, another still needs.  The record of it, built with the host compiler."""
import shutil
import subprocess
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parent.parent / "csrc" / "kernels"
MAIN = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"
int main() {
  static ogb::OncePerDevice once;
  int done[3] = {0, 0, 0};
  const int order[] = {0, 0, 1, 0, 1, 2};
  for (int d : order)
    if (once(d, [&] { ++done[d]; return 0; }) != 0) return 1;
  if (done[0] != 1 || done[1] != 1 || done[2] != 1) return 2;
  int tries = 0;
  if (once(3, [&] { ++tries; return 7; }) != 7 || once(3, [&] { ++tries; return 0; }) != 0 || once(3, [&] { ++tries; return 7; }) != 0) return 3;
  if (tries != 2) return 4;
  int far = 0;
  for (int i = 0; i < 2; ++i) once(1 << 20, [&] { ++far; return 0; });      // more devices than it keeps: every time
  if (far != 2) return 5;
  static ogb::OncePerDevice shared;
  std::atomic<int> ran{0}, wrong{0};
  std::vector<std::thread> pool;
  for (int i = 0; i < 8; ++i)
    pool.emplace_back([&] {
      for (int d = 0; d < 64; ++d)
        if (shared(d, [&] { ++ran; return 0; }) != 0) ++wrong;
    });
  for (auto& t : pool) t.join();
  return wrong == 0 && ran >= 64 && ran <= 8 * 64 ? 0 : 6;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_each_device_is_prepared(tmp_path):
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(KERNELS), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


@pytest.mark.parametrize("source,launches", [("sampling_cluster.cuh", ["launch_sample_cluster"]), ("gemm_tcgen05.cu", ["launch_rows_one"]),
                                             ("gemm_w4a16.cu", ["launch_w4_rows_one"])])
def test_launches_ask_it(source, launches):
    """The launches whose kernels need more shared memory than a kernel gets by default."""
    text = (KERNELS / source).read_text()
    for name in launches:
        body = text[text.index(f"{name}("):]
        body = body[:body.index("\n}")]
        assert "allow_smem(" in body and "attr_set" not in body
