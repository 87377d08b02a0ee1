"""The end of a level in the one-kernel search, which every block evaluates
for itself (csrc/level_rule.h), run for many blocks on the host: they have to
agree whatever the order in which they come out of the barrier."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "graph500-bfs_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "level_rule.h"
using namespace b200bfs;

// The last barrier: block `late` reaches its poll limit just before the last
// arrival, the others go on and the first block has a finished search.
int last_barrier(int late) {
  PersistCtl ctl;
  memset(&ctl, 0, sizeof(ctl));
  for (int b = 0; b < 148; ++b) {
    if (b == late) ctl.error = 1;
    if (b == 0) ctl.done = b == late ? 4 : 1;
  }
  printf("%d\n", published_status(ctl.done, ctl.error));
  return 0;
}

// A bottom-up level of `found` vertices with `entries` entries ends.  Each of
// 148 blocks evaluates the rule; the ones that go back to top-down append
// their share of the frontier at once, before the next block reads.
// Whether a graph of that many rows and entries is searched by the one kernel.
int taken(int option, int64_t rows, int64_t entries) {
  Graph g;
  RunOptions o;
  int2 pair;
  g.csr.nrows = rows;
  g.csr.nedges = entries;
  g.csr.first_pair = &pair;
  o.persistent = option;
  printf("%d\n", use_persistent(g, o) ? 1 : 0);
  return 0;
}

int main(int argc, char** argv) {
  if (argc == 5) return taken(atoi(argv[2]), atoll(argv[3]), atoll(argv[4]));
  if (argc == 2) return last_barrier(atoi(argv[1]));
  const long long R = atoll(argv[1]), found = atoll(argv[2]), entries = atoll(argv[3]);
  const int blocks = 148;
  PersistArgs a;
  memset(&a, 0, sizeof(a));
  a.R = R;
  a.nedges = 32 * R;
  a.t2b = t2b_limit(a.nedges, 10);
  a.b2t = b2t_limit(a.R, 16, 14);
  PersistCounters c;
  memset(&c, 0, sizeof(c));
  c.nq = found;
  LevelState first;
  int differ = 0;
  for (int b = 0; b < blocks; ++b) {
    LevelState s;
    memset(&s, 0, sizeof(s));
    s.level = 5;
    s.visited = R - 2 * found;
    s.prev_nq = 8 * found;
    s.growing = 1;
    level_end(s, a, c);
    if (s.next_forward)
      c.q += (unsigned long long)(found / blocks) << 32 | (unsigned long long)(entries / blocks);
    if (b == 0) first = s;
    differ += s.nq != first.nq || s.visited != first.visited || s.done != first.done ||
              s.next_forward != first.next_forward || s.growing != first.growing ||
              s.cur != first.cur || s.qcur != first.qcur || s.at_set != first.at_set ||
              memcmp(s.at, first.at, sizeof(s.at));
  }
  printf("%d %lld %lld %d\n", differ, first.nq, first.visited, first.next_forward);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("level_rule")
    src = d / "level_rule.cu"
    src.write_text(PROGRAM)
    subprocess.run([NVCC, "-std=c++17", "-I", CSRC, "-o", str(d / "level_rule"), str(src)],
                   check=True)
    return str(d / "level_rule")


# few vertices; just below the switch (R / (14 * 16 * 2) = 2232); at it, where
# the search stays bottom-up
@pytest.mark.parametrize("found,forward", [(148, 1), (1500, 1), (2231, 1), (2232, 0), (9000, 0)])
def test_blocks_agree_after_a_bottom_up_level(program, found, forward):
    r = 1000000
    out = subprocess.run([program, str(r), str(found), str(20 * found)], check=True,
                         capture_output=True, text=True).stdout.split()
    assert [int(x) for x in out] == [0, found, r - found, forward]


@pytest.mark.parametrize("late,status", [(-1, 1), (0, 4), (1, 4), (147, 4)])
def test_a_block_that_gave_up_is_published(program, late, status):
    out = subprocess.run([program, str(late)], check=True, capture_output=True, text=True).stdout
    assert int(out) == status


# a list of all entries has to be expanded without its 32-bit steps wrapping:
# 4 * 32 entries from 2^32 at the nearest
@pytest.mark.parametrize("option,rows,entries,want", [
    (2, 1 << 20, 2**32 - 1, 0), (2, 1 << 20, 2**32 - 128, 0), (2, 1 << 20, 2**32 - 256, 1),
    (1, 1 << 20, 2**32 - 1, 0), (1, 1 << 20, 1 << 25, 1), (1, 3 << 24, 1 << 25, 0),
    (2, 3 << 24, 1 << 25, 1), (0, 1 << 20, 1 << 25, 0)])
def test_graphs_the_one_kernel_takes(program, option, rows, entries, want):
    out = subprocess.run([program, "taken", str(option), str(rows), str(entries)], check=True,
                         capture_output=True, text=True).stdout
    assert int(out) == want
