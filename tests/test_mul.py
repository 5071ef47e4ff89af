"""The integer-pipe multiplication and the division with a kept reciprocal of
the FP64 kernels (csrc/hyc_div.cuh) against the host's IEEE operations, bit
for bit: the same header built for the host."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hycom-src_gb300", "csrc")

SRC = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "hyc_div.cuh"
using namespace hyc;
static const uint64_t M = 0xFFFFFFFFFFFFFull, ONE = 0x3FF0000000000000ull, S = 1ull << 63;
int main() {
  std::mt19937_64 g(11);
  long bad = 0;
  auto eq = [&](double x, double y, char op, double a, double b) {
    if (idiv::bits(x) != idiv::bits(y) && !(x != x && y != y) && bad++ < 5) printf("%a %c %a = %a, want %a\n", a, op, b, x, y);
  };
  auto chk = [&](double a, double b) {
    eq(mul_rn(a, b), a * b, '*', a, b);
    eq(div_by(a, b, recip_of(b)), a / b, '/', a, b);
  };
  for (long i = 0; i < 2000000; i++) {
    const uint64_t u = g(), v = g();
    chk(idiv::from_bits(u), idiv::from_bits(v));                                            // any bits
    chk(idiv::from_bits((u & (M | S)) | ONE), idiv::from_bits((v & (M | S)) | ONE));
    chk(idiv::from_bits((u & M & ~((1ull << (v >> 58)) - 1)) | ONE),
        idiv::from_bits((v & M & ~((1ull << (u >> 58)) - 1)) | ONE));                       // short significands: ties
    chk(idiv::from_bits(ONE + (u & 1023)), idiv::from_bits(ONE + (v & 1023)));
    chk(idiv::from_bits(ONE + M - (u & 1023)), idiv::from_bits(ONE + M - (v & 1023)));      // products round up to 2^53
    chk((double)(u >> 37) * 33554431.0, (double)((v >> 37) | 1));
  }
  const double s[] = {0., -0., 1., -3., INFINITY, -INFINITY, NAN, 5e-324, 1e-310, 0x1p-1022, 0x1p-500, 0x1.8p-501, 0x1p500,
                      0x1.fffffffffffffp499, 1.7e308};
  for (double a : s)
    for (double b : s) chk(a, b);
  return bad != 0;
}
"""


def test_multiplication_equals_ieee(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", exe, str(tmp_path / "t.cpp")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
