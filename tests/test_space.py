"""The device memory that a handle keeps, when memory is short: csrc/salsa_space.h with an
allocator of a given budget in place of the device's."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "uclales_salsa_gb300", "csrc")
SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include "salsa_space.h"
// reads: budget, then pairs (blocks wanted, bytes per block); prints the blocks served and the bytes held
int main() {
  size_t budget, used = 0, next = 1;
  std::map<void *, size_t> live;
  salsa::Space s;
  if (std::scanf("%zu", &budget) != 1) return 1;
  long grid, per;
  while (std::scanf("%ld %ld", &grid, &per) == 2) {
    const int g = salsa::lane_blocks(s, (int)grid, (size_t)per,
      [&](size_t b) -> void * {
        if (used + b > budget) return nullptr;
        used += b;
        void *p = (void *)next++;
        live[p] = b;
        return p;
      },
      [&](void *p) { used -= live.at(p); live.erase(p); });
    if (g > 0 && (!s.p || (size_t)g * per > s.bytes || live.count(s.p) == 0 || live[s.p] != s.bytes)) return 2;
    if (live.size() > 1) return 3;
    std::printf("%d %zu\n", g, s.bytes);
  }
}
"""


@pytest.fixture(scope="module")
def prog(tmp_path_factory):
    d = tmp_path_factory.mktemp("space")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    return str(d / "t")


def serve(prog, budget, calls):
    r = subprocess.run([prog], input=" ".join(map(str, [budget] + [x for c in calls for x in c])), text=True,
                       capture_output=True, check=True)
    return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]


@pytest.mark.parametrize("budget,calls,served", [
    (1000, [(10, 100)], [(10, 1000)]),                               # enough
    (10000, [(10, 100), (4, 100), (10, 100)], [(10, 1000)] + [(4, 1000), (10, 1000)]),   # kept for smaller calls
    (760, [(10, 100)], [(5, 500)]),         # neither all nor 8 of 10: half
    (850, [(10, 100)], [(8, 800)]),                                  # three quarters, rounded up
    (499, [(10, 100)], [(0, 0)]),                                    # less than half: the warp form
    (1300, [(6, 100), (10, 100)], [(6, 600), (6, 600)]),             # the old space stays: 6 of 10 is more than half
    (1100, [(2, 100), (10, 100), (2, 100)], [(2, 200), (8, 800), (2, 800)]),   # the old space goes when more is had
    (250, [(2, 100), (10, 100), (2, 100)], [(2, 200), (0, 200), (2, 200)]),    # a refused call leaves the old space
    (1000, [(1, 1000), (1, 1001)], [(1, 1000), (0, 1000)]),
    (1000, [(0, 100), (5, 0)], [(0, 0), (0, 0)]),
])
def test_blocks_served_when_memory_is_short(prog, budget, calls, served):
    assert serve(prog, budget, calls) == served


LISTS = r"""
#include <cstdio>
#include "salsa_space.h"
int main() {
  size_t n, budget;
  while (std::scanf("%zu %zu", &n, &budget) == 2) {
    void *p = nullptr;
    const int k = salsa::order_lists(n, &p, [&](size_t b) -> void * { return b <= budget ? (void *)1 : nullptr; });
    std::printf("%d %d\n", k, p ? 1 : 0);
  }
}
"""


def test_order_lists_when_memory_is_short(tmp_path):
    """One list serves a call whose two do not fit, as before there were two."""
    (tmp_path / "l.cpp").write_text(LISTS)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(tmp_path / "l.cpp"), "-o", str(tmp_path / "l")],
                   check=True)
    r = subprocess.run([str(tmp_path / "l")], input="100 800 100 799 100 400 100 399", text=True, capture_output=True, check=True)
    assert r.stdout.split() == ["2", "1", "1", "1", "1", "1", "0", "0"]
