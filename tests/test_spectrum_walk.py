"""Threads of the spectra's walk (axg_binning.h): they are numbered in 32 bits,
with the grid's stride added to the last, and cover every row."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = r"""
#include <cstdio>
#include "axg_binning.h"
int main() {
  for (int n = 4; n <= 2048; n += 2)
    for (int nx : {n / 2 + 1, n}) {
      for (int rows : {walk_rows(n, nx), walk_rows_single(n, nx)}) {
        const long long t = walk_threads(n, nx, rows);
        std::printf("%d %d %d %lld %d\n", n, nx, rows, t, walk_grid(n, nx, rows));
      }
    }
}
"""


@pytest.fixture(scope="module")
def table(tmp_path_factory):
    cuda = "/usr/local/cuda/include"
    if not os.path.exists(os.path.join(cuda, "cuda.h")):
        pytest.skip("CUDA headers not found")
    d = tmp_path_factory.mktemp("walk")
    (d / "t.cpp").write_text(CODE)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "axion_grav_gb300", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-I", cuda, str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    out = subprocess.run([str(d / "t")], capture_output=True, text=True, check=True).stdout
    return [tuple(map(int, line.split())) for line in out.splitlines()]


def test_threads_count_in_32_bits(table):
    assert len(table) > 4000
    for n, nx, rows, threads, grid in table:
        assert threads == nx * n * -(-n // rows) and rows >= 1
        assert threads + grid * 256 < 2 ** 32
        assert 1 <= grid and (grid * 256 >= threads or grid == 152 * 8)


def test_single_rows_below_the_limit(table):
    # every second entry: walk_rows, then walk_rows_single
    for n, nx, rows, _, _ in table[1::2]:
        assert rows == (1 if nx * n * n <= 2 ** 31 else 2 if nx * n * (n // 2) <= 2 ** 31 else 4)
