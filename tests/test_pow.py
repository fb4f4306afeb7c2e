"""x^y of the FP64 kernels (imex_sflow2d_dev_gb300/csrc/sflow_pow.h): its
tables recomputed from exact arithmetic, and the bits of its FP64 and integer
evaluations against those of sfm_pow (sflow_math.h) on the host, over the closures' argument ranges, near
1, at random bit patterns and at the C99 special values.  All of
them round the exact power, so no bit may differ."""
import os
import re
import shutil
import subprocess
from decimal import Decimal, getcontext

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "imex_sflow2d_dev_gb300", "csrc")


def _table(text, name):
    body = re.search(name + r"\[[^\]]*\] = \{(.*?)\};", text, re.S).group(1)
    return [float.fromhex(v.strip()) for v in body.replace("\n", " ").split(",") if v.strip()]


def test_tables_are_the_exact_values_split():
    getcontext().prec = 60
    text = open(os.path.join(CSRC, "sflow_pow.h")).read()
    ln2 = Decimal(2).ln()

    def grid(v, p):
        return Decimal(int((v * 2 ** p).to_integral_value())) / 2 ** p
    t = _table(text, "sfm_pow_log_tab")
    for i in range(128):
        c = Decimal(int((256 / (1 + (Decimal(i) + Decimal("0.5")) / 128)).to_integral_value())) / 256
        hi = grid(-c.ln(), 42)
        assert t[3 * i:3 * i + 3] == [float(c), float(hi), float(-c.ln() - hi)]
    t = _table(text, "sfm_pow_exp_tab")
    for j in range(128):
        v = (ln2 * j / 128).exp()
        assert t[2 * j:2 * j + 2] == [float(v), float(v - Decimal(float(v)))]
    d = {k: float.fromhex(v) for k, v in re.findall(r"#define (SFM_POW_\w+) (-?0x[0-9a-fp.+-]+)", text)}
    assert d["SFM_POW_LN2_HI"] == float(grid(ln2, 42)) and d["SFM_POW_LN2_LO"] == float(ln2 - grid(ln2, 42))
    assert d["SFM_POW_L_HI"] == float(grid(ln2 / 128, 46)) and d["SFM_POW_L_LO"] == float(ln2 / 128 - grid(ln2 / 128, 46))
    assert d["SFM_POW_INV_L"] == float(128 / ln2)


def test_integer_tables_and_coefficients_are_the_rounded_exact_values():
    getcontext().prec = 60
    text = open(os.path.join(CSRC, "sflow_pow.h")).read()
    ln2 = Decimal(2).ln()

    def ints(name):
        body = re.search(name + r"\[[^\]]*\] = \{(.*?)\};", text, re.S).group(1)
        return [int(v.strip().rstrip("L")) for v in body.replace("\n", " ").split(",") if v.strip()]

    def rnd(v):
        return int(v.to_integral_value())
    t, first = ints("sfm_powi_log_tab"), None
    for i in range(128):
        c8 = rnd(256 / (1 + (Decimal(i) + Decimal("0.5")) / 128))
        v = -(Decimal(c8) / 256).ln() / ln2
        if v > Decimal("0.5"):
            first, v = (i if first is None else first), v - 1
        assert t[2 * i:2 * i + 2] == [rnd(v * 2 ** 63), c8]
    assert ints("sfm_powi_exp_tab") == [rnd(((ln2 * j / 128).exp() - 1) * 2 ** 63) for j in range(128)]
    d = {k: int(v) for k, v in re.findall(r"#define SFM_POWI_([JPQ]\d?) \(?(-?\d+)", text)}
    assert d["J"] == first
    f = 1
    for n in range(8):
        assert d[f"P{n}"] == rnd((-1) ** n / ln2 / (n + 1) * Decimal(2) ** (62 - 6 * n))
        f *= n + 1
        if n < 6:
            assert d[f"Q{n}"] == rnd(ln2 ** (n + 1) / f * Decimal(2) ** (62 - 6 * n))


PROG = r'''
#include <stdio.h>
#include "sflow_pow.h"
static uint64_t s = 88172645463325252ULL;
static uint64_t rn(void) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static long differ(double x, double y) {
  const double a = sfm_pow(x, y), b = sfm_pow_quick(x, y), c = sfm_pow_int(x, y);
  return (sfm_bits(a) != sfm_bits(b) || sfm_bits(a) != sfm_bits(c)) && !(a != a && b != b && c != c);
}
int main(void) {
  const double ys[] = {0.687, 4.65, 2.4, 0.5, -1.3, 3.0, 1.0, 17.25, -40.0, 0.0};
  const double sp[] = {0.0, -0.0, 1.0, -1.0, HUGE_VAL, -HUGE_VAL, 0x1p-1074, 0x1p-1022, 0x1.fffffffffffffp1023, -2.5,
                       1.0 / 3.0, 0x1.fffffffffffffp-1, 0x1.0000000000001p0};
  long bad = 0;
  for (long i = 0; i < 2000000; ++i) {
    const uint64_t u = rn();
    const double w = (double)(u >> 11) * 0x1p-53;
    double x, y = ys[rn() % 10];
    switch (i % 4) {
      case 0: x = 1e-6 * pow(1e9, w); break;
      case 1: x = w; break;
      case 2: x = 1.0 + (w - 0.5) * pow(2.0, -(double)(rn() % 50)); break;
      default: x = sfm_from_bits((int64_t)(u & 0x7fffffffffffffffULL)); if (i & 4) y = ((double)(int64_t)rn()) * 0x1p-60;
    }
    bad += differ(x, y);
  }
  for (unsigned i = 0; i < sizeof sp / sizeof sp[0]; ++i)
    for (unsigned j = 0; j < 10; ++j) bad += differ(sp[i], ys[j]);
  for (unsigned i = 0; i < sizeof sp / sizeof sp[0]; ++i)
    for (unsigned j = 0; j < sizeof sp / sizeof sp[0]; ++j) bad += differ(sp[i], sp[j]);
  printf("%ld\n", bad);
  return 0;
}
'''


@pytest.mark.skipif(not shutil.which("gcc"), reason="no C compiler")
def test_quick_power_has_the_bits_of_the_slow_one(tmp_path):
    (tmp_path / "t.c").write_text(PROG)
    exe = str(tmp_path / "t")
    subprocess.check_call(["gcc", "-O2", "-std=gnu11", "-ffp-contract=off", "-I", CSRC, "-o", exe,
                           str(tmp_path / "t.c"), "-lm"])
    assert subprocess.check_output([exe]).decode().strip() == "0"
