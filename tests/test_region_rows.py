"""The CTAs of a cloud-region launch and the memory of their rows
(csrc/region_rows.h), compiled for the host with an allocator that grants a
given number of bytes: within the launch's bound, and with fewer CTAs, down to
one, where memory is short."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "region_rows.h"
int main(int, char **v) {
  const size_t stride = strtoull(v[2], nullptr, 10), free_bytes = strtoull(v[3], nullptr, 10);
  long long grid = socgpu::region_grid(atoll(v[1]), stride);
  printf("%lld ", grid);
  size_t got = 0;
  int asked = 0;
  const bool ok = socgpu::take_rows(grid, stride, [&](size_t b) {
    ++asked;
    if (b > free_bytes) return false;
    got = b;
    return true;
  });
  printf("%d %lld %zu %d\n", ok, grid, got, asked);
}
"""
LIMIT = 1536 << 20


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    d = tmp_path_factory.mktemp("rows")
    (d / "rows.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{ROOT / 'socrates_gb300' / 'csrc'}", str(d / "rows.cpp"), "-o", str(d / "rows")],
                   check=True)

    def call(ctas, stride, free):
        out = subprocess.run([str(d / "rows"), str(ctas), str(stride), str(free)], capture_output=True, text=True, check=True)
        return [int(x) for x in out.stdout.split()]
    return call


@pytest.mark.parametrize("ctas,stride", [(1, 100), (608, 490752), (608, 10243584), (152, 10243584), (3, LIMIT), (5, LIMIT + 1),
                                         (0, 100)])
def test_within_the_bound(rows, ctas, stride):
    bounded, ok, grid, got, asked = rows(ctas, stride, 1 << 40)
    assert ok and grid == bounded == min(ctas, max(1, LIMIT // stride)) and got == grid * stride and asked == 1
    assert got <= LIMIT or grid == 1


@pytest.mark.parametrize("free", [0, 490751, 490752, 40 << 20, 298377215, 298377216])
def test_short_memory(rows, free):
    stride = 490752
    _, ok, grid, got, _ = rows(608, stride, free)
    assert ok == (free >= stride)
    if ok:
        # more than half of what would have fitted
        assert got == grid * stride <= free and 2 * grid >= min(608, free // stride)
