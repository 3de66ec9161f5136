"""The float-pair sums of the shared scalar code against the double-precision
expressions they stand for, bit for bit: on the host, where the same source is
compiled by g++ as in the library."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "spray_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include "spray_math.cuh"
using namespace spray;

static uint32_t bits(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
static float from(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
static long wrong = 0, cases = 0;

static void check(float acc, float w, int spp) {
  const double scale = 1.0 / (double)spp;  // as the view table holds it
  const float hi = (float)scale, lo = (float)(scale - (double)hi);
  const float got = addScaled(acc, w, scale, hi, lo), want = (float)((double)acc + scale * (double)w);
  ++cases;
  if (bits(got) != bits(want) && !(got != got && want != want)) {
    if (wrong++ < 5) std::printf("acc %.9g w %.9g spp %d: %.9g, not %.9g\n", acc, w, spp, got, want);
  }
}

int main(int argc, char** argv) {
  const int sign = std::atoi(argv[1]);
  std::mt19937_64 rng(7 + sign);
  auto uni = [&](double a, double b) { return a + (b - a) * (double)(rng() >> 11) * 0x1p-53; };
  const int spps[] = {1, 2, 3, 5, 6, 7, 11, 16, 33, 100, 4097};
  for (int i = 0; i < 2000000; ++i) {
    const int spp = spps[rng() % 11];
    const float w = (float)((rng() & 1 ? 1 : -1) * std::exp2(uni(-20, 14)));
    const float p = (float)(w / (double)spp);
    float acc;
    if (sign > 0) {  // the same sign, any ratio
      acc = (float)(p * std::exp2(uni(-40, 40)));
    } else if (sign < 0) {  // sums that cancel all but their last few bits, or a ratio's worth
      acc = -from(bits(p) + (uint32_t)(rng() % 9) - 4);
      if (i & 1) acc = (float)(-p * uni(0.25, 4.0));
    } else {  // sums near the middle of two floats, both signs
      const float t = (float)(p * std::exp2(uni(-3, 12)));
      acc = (float)((double)from(bits(t)) + 0.5 * ((double)from(bits(t) + 1) - (double)t) - (double)w / spp);
    }
    check(acc, w, spp);
  }
  const float edge[] = {0.0f, -0.0f, 1.0f, -1.0f, 1e-45f, -1e-38f, 1e-31f, 1e-29f, -1e30f, 1e38f, -3e38f, INFINITY, -INFINITY, NAN};
  for (float acc : edge)
    for (float w : edge)
      for (int spp : spps) check(acc, w, spp);
  // as a light of negative radiance gave it
  check(-567.678589f, 6244.46484f, 11);
  std::printf("%ld of %ld wrong\n", wrong, cases);
  return wrong != 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("pairs")
    (d / "pairs.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-x", "c++", "-I", str(CSRC), "-o", str(d / "pairs"),
                    str(d / "pairs.cpp")], check=True)
    return d / "pairs"


@pytest.mark.parametrize("sign", [1, 0, -1])
def test_scaled_sums_round_as_the_double_expression(program, sign):
    r = subprocess.run([str(program), str(sign)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
