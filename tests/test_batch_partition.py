"""The batched solver's share-out of problems over blocks, on the host: for
batches that mix large and small lattices no block meets more problems than it
has room for, every set belongs to one block, and every (block, problem) has a
slot of its own for its partial sums."""
import subprocess
from pathlib import Path

import pytest

HEADER = Path(__file__).resolve().parents[1] / "qex_b200" / "csrc" / "batch_part.cuh"

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include <vector>
#include "%s"
using namespace qs;
int main(int argc, char **argv) {  // blocks, then the sets of each problem
  const int blocks = atoi(argv[1]), n = argc - 2;
  std::vector<int> sets, owner;
  for (int j = 0; j < n; j++) sets.push_back(atoi(argv[2 + j]));
  int total = 0, met = 0, bad = 0, at = 0;
  for (int j = 0; j < n; j++) total += sets[j];
  std::set<int> slots;
  for (int b = 0; b < blocks; b++) {
    BPart T;
    fill_part(T, n, [](int) { return false; }, [&](int j) { return sets[j]; }, blocks, b);
    if (T.na != n || T.ntot != total) bad++;
    if (T.s0 < T.s1 && T.s0 != at) bad++;
    if (T.s0 < T.s1) at = T.s1;
    for (int s = T.s0; s < T.s1; s++)
      if (block_of(T, s) != b) bad++;
    for (int q = 0; q < T.np; q++)
      if (!slots.insert(b + T.i0 + q).second) bad++;
    if (T.np > met) met = T.np;
  }
  if (at != total || *slots.rbegin() >= blocks + kMaxBatch) bad++;
  printf("%%d %%d %%d\n", met, kMaxMet, bad);
}
"""


@pytest.fixture(scope="module")
def partition(tmp_path_factory):
    d = tmp_path_factory.mktemp("part")
    (d / "main.cpp").write_text(MAIN % HEADER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-x", "c++", "-o", str(d / "main"), str(d / "main.cpp")], check=True)
    return lambda blocks, sets: [int(v) for v in subprocess.run(
        [str(d / "main"), str(blocks), *map(str, sets)], check=True, capture_output=True, text=True).stdout.split()]


# sets of 32 even sites: 4 of 4^4, 1024 of 16^4, 5184 of 24^4, 16384 of 32^4, ...
@pytest.mark.parametrize("large,n,small", [(16384, 3, 100), (16384, 5, 100), (5184, 8, 100), (5184, 16, 104),
                                           (1024, 60, 68), (40000, 1, 127), (82944, 1, 127), (4, 1, 0), (4, 64, 64),
                                           (23, 1, 1)])
@pytest.mark.parametrize("per_sm", [1, 2])
def test_room_for_every_problem_of_a_chunk(partition, large, n, small, per_sm):
    for sets in ([large] * n + [4] * small, [4] * small + [large] * n):
        met, room, bad = partition(148 * per_sm, sets)
        assert met <= room and bad == 0
