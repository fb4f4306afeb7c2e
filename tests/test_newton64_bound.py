"""The FP64 implicit solve (imex_sflow2d_dev_gb300/csrc/sflow_newton64.cuh)
compiled for the host, with friction terms made for the test: the line search
ends after 4096 refused trials also where its step length never falls below
the least step -- an infinite one (the quadratic model's curvature rounds to
zero), one that returns to 1 (the model's minimiser is 1, 2 or 4), a direction
that is not a number -- and the solve as a whole after 100 directions.  A
trial that the halving reaches still ends the search as before."""
import math
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "imex_sflow2d_dev_gb300", "csrc")

# n_solid = 1, q_old = (1, 1, 1, 1, 1), dt = a_diag = 1, Rj = 0: the residual of
# hu is q1 - 1 - nh1(q1), the other components' residuals are 0 throughout, and
# the Jacobian is the identity (org = 1).  nh1(1) = 2 puts the first, unsearched
# step at q1 = 3; the residual there is K = 2^40, so that the second direction
# is capped at 100 n_vars = 500 and the least squares sum falls by far less than
# a tenth.
PROG = r'''
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstdlib>
namespace sflow { constexpr double kEps = DBL_EPSILON; }
#include "sflow_newton64.cuh"
using namespace sflow;
static int which;
static long calls;
static const double K = 0x1p40;
// residual of hu at q1
static double residual(double q1) {
  if (q1 == 1.0) return -2.0;
  if (q1 == 3.0) return K;
  switch (which) {
    case 0: return K + (q1 - 3.0);                               // linear: the curvature rounds to zero
    case 1: return q1 == -497.0 ? K - 250.0 : K;                 // minimiser 1
    case 2: return q1 == -497.0 ? K - 375.0 : K;                 // minimiser 2
    case 3: return q1 == -497.0 ? K - 437.5 : K;                 // minimiser 4
    default: return K;                                           // minimiser 1/2: halved until refused for good
  }
}
struct Closure {
  static void real(const Phys<double>&, double, double, const Div64&, const double* q, FrictPoint& f, double& nh1,
                   double& nh2) {
    if (++calls > 500000) { printf("unbounded\n"); exit(0); }
    nh1 = (q[1] - 1.0) - residual(q[1]);
    nh2 = 0.0;
    f.u = q[1];
  }
  static void imag(const Phys<double>&, double, double, const Div64&, const FrictPoint& f, int col, double, double,
                   double, double, double& im1, double& im2) {
    im1 = im2 = 0.0;
    if (which == 5 && f.u != 1.0 && col == 0) im1 = NAN;
  }
};
int main(int, char** argv) {
  which = atoi(argv[1]);
  Phys<double> P{};
  const double q_old[5] = {1, 1, 1, 1, 1}, R[5] = {0, 0, 0, 0, 0};
  double q[5] = {1, 1, 1, 1, 1};
  const NewtonCtx c{&P, 1.0, 1.0, 0.0, 0.0, q_old, R};
  const int it = solve_rk_step<1, Closure>(c, q);
  printf("%d %ld %g\n", it, calls, q[1]);
}
'''


@pytest.fixture(scope="module")
def solve(tmp_path_factory):
    d = tmp_path_factory.mktemp("newton64")
    (d / "t.cpp").write_text(PROG)
    exe = str(d / "t")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-D__device__=", "-D__noinline__=",
                           "-D__forceinline__=inline", "-w", "-I", CSRC, "-o", exe, str(d / "t.cpp")])

    def run(which):
        out = subprocess.run([exe, str(which)], stdout=subprocess.PIPE, timeout=60, check=True).stdout.decode().split()
        assert out != ["unbounded"]
        return int(out[0]), int(out[1]), float(out[2])

    return run


pytestmark = pytest.mark.skipif(not shutil.which("g++"), reason="no C++ compiler")


def test_infinite_step(solve):
    it, calls, q = solve(0)
    # start, first step, 4096 trials; then the state is not finite
    assert it == 101 and calls == 2 + 4096 and not math.isfinite(q)


@pytest.mark.parametrize("which", [1, 2, 3])
def test_step_that_returns_to_one(solve, which):
    it, calls, _ = solve(which)
    assert it <= 101 and 2 + 4096 <= calls <= 2 + 4096 * 99


def test_direction_not_a_number(solve):
    it, calls, _ = solve(5)
    assert it <= 101 and calls <= 2 + 4096 * 99


def test_halving_still_ends_the_search(solve):
    it, calls, q = solve(4)
    # least step 2^-52 / (500/3) below 2^-59: about 60 trials, back at the old point
    assert it == 2 and calls < 80 and q == 3.0
