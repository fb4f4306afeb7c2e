"""Integer division, square root and comparisons of the FP64 kernels
(imex_sflow2d_dev_gb300/csrc/sflow_div64.cuh), compiled for the host: the
bits of the FP64 operations and the answers of the FP64 comparisons, on
random bit patterns, mantissas next to rounding boundaries (a quotient times
the divisor, +-2 ulp; divisors of nearly all ones), zeros of both signs,
infinities, NaN, subnormals and the ends of the range; squares +-2 ulp for
the root.  The float estimates that start the iterations are shifted by up
to 2^-22, more than the device's approximations are off."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "imex_sflow2d_dev_gb300", "csrc")

PROG = r'''
#include <cstdio>
#include <cmath>
static int noise = 0;
#define D64_SEED_NOISE noise
#include "sflow_div64.cuh"
using namespace sflow;
static uint64_t s = 88172645463325252ULL;
static uint64_t rn() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double unit() { return 1.0 + (double)(rn() >> 12) * 0x1p-52; }
static long check(double a, double d) {
  const double x = quot64(a, div64(d)), y = a / d;
  long bad = d64_bits(x) != d64_bits(y) && !(x != x && y != y);
  bad += (a < d) != d64_lt(a, d);
  bad += (a > 0) != d64_pos(a);
  bad += (a < 0) != d64_neg(a);
  bad += (a == 0) != d64_zero(a);
  bad += (a > 1.5) != d64_gt_pos(a, 1.5);
  bad += d64_bits(ddiv64(a, d)) != d64_bits(x) && !(x != x);
  const double r = dsqrt64(a), r0 = sqrt(a);
  bad += d64_bits(r) != d64_bits(r0) && !(r != r && r0 != r0);
  const double u = fabs(a), v = fabs(d), m = u > v ? u : v, n = d64_from(d64_absmax(d64_bits(u), d64_bits(v)));
  bad += d64_bits(m) != d64_bits(n) && !(m != m && n != n);
  return bad;
}
int main() {
  const double sp[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, -NAN, 0x1p-1074, -0x1p-1030, 0x1p-1022,
                       0x1.fffffffffffffp1023, 0x1p-430, 0x1p430, 0x1p423, 0x1p-423, 1.5, 3.0, 10.0, 0.1};
  long bad = 0;
  for (double a : sp) for (double d : sp) bad += check(a, d);
  for (long i = 0; i < 2000000; ++i) {
    double a, d;
    noise = (int)(rn() % 1024) - 512;
    switch (i % 7) {
      case 0: a = d64_from((long long)rn()); d = d64_from((long long)rn()); break;
      case 1: a = unit(); d = unit(); break;
      case 2: d = unit(); a = unit() * d; a = d64_from(d64_bits(a) + (long long)(rn() % 5) - 2); break;
      case 3: d = 2.0 - (double)(rn() % 64 + 1) * 0x1p-52; a = unit(); break;
      case 4: d = (double)(rn() % 1000 + 1); a = (double)(rn() % 100000) - 50000.0; break;
      case 5: d = unit(); a = unit(); a = a * a; if (i & 1) a *= 2.0; a = d64_from(d64_bits(a) + (long long)(rn() % 5) - 2); break;
      default: a = sp[rn() % 20]; d = unit(); break;
    }
    bad += check(a, d);
  }
  printf("%ld\n", bad);
}
'''


@pytest.mark.skipif(not shutil.which("g++"), reason="no C++ compiler")
def test_bits_of_the_plain_operations(tmp_path):
    (tmp_path / "t.cpp").write_text(PROG)
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", exe,
                           str(tmp_path / "t.cpp")])
    assert subprocess.check_output([exe]).decode().strip() == "0"
