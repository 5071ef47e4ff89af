"""The integer-pipe division of the FP64 kernels (csrc/hyc_div.cuh) against the
host's IEEE division, bit for bit: the same header built for the host, with
the FP32 reciprocal seed exact and one ulp off either way (what the
hardware's approximate reciprocal may be)."""
import os
import subprocess

import pytest

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hycom-src_gb300", "csrc",
                      "hyc_div.cuh")

SRC = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "div.h"
using namespace hyc;
static const uint64_t M = 0xFFFFFFFFFFFFFull, ONE = 0x3FF0000000000000ull;
int main() {
  std::mt19937_64 g(7);
  long bad = 0;
  auto chk = [&](double a, double b) {
    const double x = div_rn(a, b), y = a / b;
    if (idiv::bits(x) != idiv::bits(y) && !(x != x && y != y) && bad++ < 5) printf("%a / %a = %a, want %a\n", a, b, x, y);
  };
  for (long i = 0; i < 3000000; i++) {
    const uint64_t u = g(), v = g();
    chk(idiv::from_bits(u), idiv::from_bits(v));                                // any bits
    const double a = idiv::from_bits((u & M) | ONE), b = idiv::from_bits((v & M) | ONE);
    chk(a, b);
    chk(a, idiv::from_bits(ONE + (v & 255)));                                   // divisors just above 1
    chk(a, idiv::from_bits(ONE + M - (v & 255)));                               // and just below 2
    chk(-b * (double)(1 + (u >> 40) % 1000), b);                                // exact quotients
    chk(std::fma(b, a, b * 0x1p-53), b);                                        // near a midpoint
    chk(1.0, b);
  }
  const double s[] = {0., -0., 1., -3., INFINITY, -INFINITY, NAN, 5e-324, 1e-310, 0x1p-1022, 0x1p-500, 0x1.8p-501, 0x1p500,
                      0x1.fffffffffffffp499, 1.7e308};
  for (double a : s)
    for (double b : s) chk(a, b);
  return bad != 0;
}
"""


@pytest.mark.parametrize("ulps", [0, 1, -1])
def test_division_equals_ieee(tmp_path, ulps):
    text = open(HEADER).read()
    assert text.count("return 1.0f / x;") == 1
    (tmp_path / "div.h").write_text(text.replace("return 1.0f / x;", f"return u2f(f2u(1.0f / x) + ({ulps}));"))
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe, str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
