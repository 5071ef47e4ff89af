"""The integer-pipe square root, halving and doubling of the FP64 kernels
(csrc/hyc_div.cuh) against the host's IEEE operations, bit for bit, with the
FP32 reciprocal square root seed exact and two ulps off either way (what the
hardware's approximation may be)."""
import os
import subprocess

import pytest

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hycom-src_gb300", "csrc",
                      "hyc_div.cuh")
SEED = "return (float)(1.0 / sqrt((double)x));"

SRC = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "div.h"
using namespace hyc;
static const uint64_t M = 0xFFFFFFFFFFFFFull, ONE = 0x3FF0000000000000ull;
int main() {
  std::mt19937_64 g(13);
  long bad = 0;
  auto eq = [&](double x, double y, const char *f, double a) {
    if (idiv::bits(x) != idiv::bits(y) && !(x != x && y != y) && bad++ < 5) printf("%s(%a) = %a, want %a\n", f, a, x, y);
  };
  auto chk = [&](double a) {
    eq(sqrt_rn(a), sqrt(a), "sqrt", a);
    eq(half_of(a), 0.5 * a, "half", a);
    eq(twice_of(a), 2.0 * a, "twice", a);
  };
  for (long i = 0; i < 1500000; i++) {
    const uint64_t u = g();
    const double a = idiv::from_bits((u & M) | ONE), s = (double)(u & 4095) * 0x1p-52, r = (double)(u >> 38);
    chk(idiv::from_bits(u));  // any bits
    chk(a);
    chk(2 * a);
    chk(1 + s);
    chk(2 - s);
    chk(2 + 2 * s);
    chk(4 - 2 * s);
    chk(r * r);                   // exact roots and their neighbours
    chk(nextafter(r * r, 1e99));
    chk(nextafter(r * r, 0));
    chk(a * a);
  }
  const double s[] = {0., -0., 1., -3., INFINITY, -INFINITY, NAN, 5e-324, 1e-310, 0x1p-500, 0x1.8p-501, 0x1p500, 1.7e308};
  for (double a : s) chk(a);
  return bad != 0;
}
"""


@pytest.mark.parametrize("ulps", [0, 2, -2])
def test_square_root_equals_ieee(tmp_path, ulps):
    text = open(HEADER).read()
    assert text.count(SEED) == 1
    (tmp_path / "div.h").write_text(text.replace(SEED, f"return u2f(f2u((float)(1.0 / sqrt((double)x))) + ({ulps}));"))
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe, str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
