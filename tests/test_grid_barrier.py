"""Arrival count of the one-launch kernels' grid barrier (spoc_barrier.h).

Each of the grid's blocks adds one to a 32-bit word per barrier and waits until
it holds a multiple of the grid size.  A run of 148 blocks passes 2^32 after 3.6
million RK4 steps of one call, and the barrier has to hold there as anywhere."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "spoc_b200" / "csrc"
PROGRAM = """
#include "spoc_barrier.h"
#include <cstdio>
#include <cstdlib>
// counts a block may see at the barriers from `first` on: grid * k + 1 (its own
// arrival) up to grid * (k + 2) - 1 (all others have arrived at the next one)
int main(int, char **v) {
  const unsigned long long grid = strtoull(v[1], 0, 10), first = strtoull(v[2], 0, 10);
  for (unsigned long long k = first; k < first + 64; ++k) {
    const unsigned target = (unsigned)(grid * (k + 1));
    for (unsigned long long c = grid * k + 1; c < grid * (k + 2); ++c)
      if (spoc::barrier_reached((unsigned)c, target) != (c >= grid * (k + 1))) {
        printf("barrier %llu of %llu blocks, count %llu\\n", k, grid, c);
        return 1;
      }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("barrier")
    (d / "barrier.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), str(d / "barrier.cpp"), "-o", str(d / "barrier")],
                   check=True)
    return d / "barrier"


@pytest.mark.parametrize("grid", [1, 2, 7, 148, 296])
@pytest.mark.parametrize("at", [0, 2**31, 2**32, 2**33])
def test_barrier_holds_where_the_count_wraps(program, grid, at):
    first = max(0, at // grid - 32)
    r = subprocess.run([str(program), str(grid), str(first)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
