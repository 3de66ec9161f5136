"""The table of domain groups that the list pass tests (buildDomainGroups), on the host.

A ray whose origin is not finite (a hit point that overflowed) is not turned away by
any box, the unused slots' among them, so every slot has to name a domain that
exists; the exact slab test then turns the domain down."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "spray_gb300" / "csrc"

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "bvh.h"
using namespace spray;

int main(int argc, char** argv) {
  const int n = std::atoi(argv[1]);
  std::vector<float> boxes;
  for (int d = 0; d < n; ++d) {
    const float c[3] = {(float)(d % 5), (float)(d / 5 % 5), (float)(d / 25)};
    for (float x : c) boxes.push_back(x);
    for (float x : c) boxes.push_back(x + (d % 7 == 3 ? -0.5f : 0.9f));  // some inverted
  }
  if (n > 20) boxes[6 * 9] = NAN, boxes[6 * 11 + 4] = INFINITY;
  std::vector<BvhNode4> g;
  int l1 = 0;
  buildDomainGroups(boxes.data(), n, &g, &l1);
  if (l1 != (n + 63) / 64 || (int)g.size() - l1 != (n + 3) / 4) return std::puts("sizes"), 1;
  std::vector<int> seen(n, 0);
  for (size_t k = l1; k < g.size(); ++k)
    for (int c = 0; c < 4; ++c) {
      const int d = g[k].child[c];
      if (d < 0 || d >= n) return std::printf("slot %zu.%d names domain %d of %d\n", k - l1, c, d, n), 1;
      const bool unused = g[k].lox[c] == INFINITY && g[k].hix[c] == -INFINITY && g[k].loy[c] == INFINITY &&
                          g[k].hiy[c] == -INFINITY && g[k].loz[c] == INFINITY && g[k].hiz[c] == -INFINITY;
      if (!unused) ++seen[d];
    }
  for (int d = 0; d < n; ++d)
    if (seen[d] != 1) return std::printf("domain %d in %d slots\n", d, seen[d]), 1;
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("groups")
    (d / "groups.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fopenmp", "-I", str(CSRC), "-o", str(d / "groups"), str(d / "groups.cpp"),
                    str(CSRC / "bvh.cpp")], check=True)
    return d / "groups"


@pytest.mark.parametrize("n", [16, 17, 19, 61, 63, 64, 65, 129, 191, 192])
def test_every_slot_names_a_domain(program, n):
    r = subprocess.run([str(program), str(n)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
