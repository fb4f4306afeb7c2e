// sflow_newton64.cuh -- the implicit friction solve of the plain FP64 form:
// the gas-density / temperature closure of c_phys_var
// (constitutive_2d.f90:1154-1322), the friction terms of
// eval_implicit_terms (constitutive_2d.f90:3513-4009, rheology 1 and 6)
// with their complex-step Jacobian (solver_2d.f90:2302-2367), and the
// Newton iteration solve_rk_step / lnsrch / eval_f (solver_2d.f90:1662-2284).
//
// Bound by FP64 instructions (GB300: 2 lanes per clock and SM).  Every value
// that reaches the iterates has the bits of the reference's operation order
// with the complex arithmetic written out (textbook product, Smith's
// quotient, principal square root; R. L. Smith, CACM 5(8), 1962); what is
// left out or shared does not change them:
//  * only the columns hu and hv are perturbed, so q(1), q(4) and the solid
//    masses, and every quantity formed from them alone, stay real;
//  * divisions and square roots run on the integer pipes, and the quotients
//    by one divisor share its reciprocal (sflow_div64.cuh); the real
//    divisors of the two columns equal those of the real evaluation unless a
//    perturbation reaches them (tested on the bits);
//  * the end-of-iteration residual is that of the next iteration's start;
//  * the line search's least step is formed only when a step is refused, its
//    largest step only past 99 n_vars;
//  * comparisons and maxima are integer ones.
// Measured: 8 steps of the 512^2 current with settling (96,000 wet cells, 2.9
// iterations each) 32.8 -> 23.9 ms, 32 steps of a 360 x 180 eroding flood
// 66.3 -> 42.9 ms, both with this solve alone changed.
#pragma once
#include "sflow_div64.cuh"
#include "sflow_types.cuh"

namespace sflow {

struct NewtonCtx {
  const Phys<double>* P;
  double dt, a_diag, Bx, By;
  const double* q_old;
  const double* Rj;
};

struct Cplx {
  double re, im;
};

// a / b by Smith's quotient; v: the divisor b.re with its reciprocal when
// |b.re| >= |b.im|.  known / quot: a numerator real part whose quotient by
// v.d is already at hand.
static __device__ __noinline__ Cplx cdiv_plain(Cplx a, Cplx b) {
  if (!d64_lt(fabs(b.re), fabs(b.im))) {
    const double r = b.im / b.re, den = b.re + b.im * r;
    return Cplx{(a.re + a.im * r) / den, (a.im - a.re * r) / den};
  }
  const double r = b.re / b.im, den = b.re * r + b.im;
  return Cplx{(a.re * r + a.im) / den, (a.im * r - a.re) / den};
}
__device__ __forceinline__ Cplx cdiv(Cplx a, Cplx b, const Div64& v, double known, double quot) {
  if (d64_bits(b.re) == d64_bits(v.d) && !d64_lt(fabs(b.re), fabs(b.im))) {
    const double r = quot64(b.im, v), den = b.re + b.im * r;
    if (d64_bits(den) == d64_bits(v.d)) {
      const double nr = a.re + a.im * r;
      return Cplx{d64_bits(nr) == d64_bits(known) ? quot : quot64(nr, v), quot64(a.im - a.re * r, v)};
    }
  }
  return cdiv_plain(a, b);
}
__device__ __forceinline__ Cplx cmul(Cplx a, Cplx b) {
  return Cplx{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
// principal square root sqrt((|z| + |x|)/2); m2, root, vroot: a real m2 with
// its square root and the root as a divisor
__device__ __forceinline__ Cplx csqrt64(Cplx z, double m2, double root, const Div64& vroot) {
  const double ar = fabs(z.re), ai = fabs(z.im);
  const int er = (d64_hi(ar) >> 20), ei = (d64_hi(ai) >> 20);
  // |im| below 2^-28 |re|: 1 + (im/re)^2 rounds to 1, so |z| = |re|
  if (d64_bits(z.re) == d64_bits(m2) && d64_pos(m2) && ei + 28 < er && er < 0x7fe)
    return Cplx{root, quot64(z.im, vroot) * 0.5};
  if (ar == 0.0 && ai == 0.0) return Cplx{0.0, z.im};
  double m;
  if (ai == 0.0) m = ar;
  else if (ar == 0.0) m = ai;
  else if (ar >= ai) { const double t = ai / ar; m = ar * sqrt(1.0 + t * t); }
  else { const double t = ar / ai; m = ai * sqrt(1.0 + t * t); }
  const double t = sqrt((ar + m) * 0.5);
  if (z.re >= 0.0) return Cplx{t, z.im / (2.0 * t)};
  return Cplx{ai / (2.0 * t), copysign(t, z.im)};
}

// The real closure at one state; what the Jacobian at the same state reads.
struct FrictPoint {
  bool live;              // q(1) > eps
  bool film;              // q(1) <= eps_sing: regularised velocity, T = T_ambient
  bool t_amb;             // T = T_ambient (film, or a non-positive temperature)
  double inv, xc, Rc;     // 1/q(1), carrier mass fraction, carrier gas constant
  Div64 dT;               // q(1) cmix (energy in a gas only)
  double s0;              // film: sqrt2 q(1)
  Div64 den;              // film: sqrt(q(1)^4 + eps_sing^4)
  double dinv;            // sum x_s / rho_s
  Div64 dinvr;            // 1/rho_m
  double rho;             // rho_m
  Div64 drho;             // rho_m
  double nrg, qrg, rg;    // rho_m - rho_a, (rho_m - rho_a)/rho_m, reduced gravity
  double u, v, w, m2, mod;
  Div64 dmod;
  double um, vm;          // u/|v|, v/|v|
};

// nh1, nh2: the friction terms (val(q(1)) > eps and |v| != 0, else 0)
template <int NS>
__device__ __forceinline__ void friction_real(const Phys<double>& P, double Bx, double By, const Div64& dxi,
                                              const double* q, FrictPoint& f, double& nh1, double& nh2) {
  constexpr int ns = NS;
  nh1 = 0.0;
  nh2 = 0.0;
  f.live = P.rheo && d64_gt_pos(q[0], kEps);
  if (!f.live) return;
  f.film = !d64_gt_pos(q[0], P.eps_sing_d);
  f.inv = ddiv64(1.0, q[0]);
  double xs_tot = 0.0, dcp = 0.0, dinv = 0.0;
#pragma unroll
  for (int i = 0; i < ns; ++i) {
    const double xs = q[4 + i] * f.inv;
    xs_tot = xs_tot + xs;
    dcp = dcp + xs * P.sp_heat_s[i];
    dinv = dinv + xs * P.inv_rho_s[i];
  }
  f.xc = 1.0 - xs_tot;
  f.dinv = dinv;
  f.t_amb = f.film;
  double inv_rho_c;
  if (P.gas) {
    const Div64 dxc = div64(f.xc);
    double T;
    if (!f.film) {
      const double cp_c = quot64(f.xc * P.sp_heat_a, dxc);
      const double cmix = dcp + f.xc * cp_c;
      const double e = P.energy ? q[3] - 0.5 * (q[1] * q[1] + q[2] * q[2]) * f.inv : q[3];
      if (P.energy) {
        f.dT = div64(q[0] * cmix);
        T = quot64(e, f.dT);
      } else {
        T = ddiv64(e, q[0] * cmix);
      }
      f.t_amb = T <= 0.0;
    }
    if (f.t_amb) T = P.T_ambient;
    f.Rc = quot64(f.xc * P.sp_gas_const_a, dxc);
    inv_rho_c = f.Rc * T * P.inv_pres;
  } else {
    inv_rho_c = P.inv_rho_l;   // the temperature does not enter
  }
  f.dinvr = div64(dinv + f.xc * inv_rho_c);
  const double rho_m = f.rho = quot64(1.0, f.dinvr);
  if (f.film) {
    double q4 = q[0] * q[0];
    q4 = q4 * q4;
    f.den = div64(dsqrt64(q4 + P.eps_sing4));
    f.s0 = P.sqrt2 * q[0];
    f.u = quot64(f.s0 * q[1], f.den);
    f.v = quot64(f.s0 * q[2], f.den);
  } else {
    f.u = q[1] * f.inv;
    f.v = q[2] * f.inv;
  }
  f.drho = div64(rho_m);
  f.nrg = rho_m - P.rho_a_amb;
  f.qrg = quot64(f.nrg, f.drho);
  f.rg = f.qrg * P.grav;
  f.w = P.slope_corr ? (f.u * Bx + f.v * By) : 0.0;
  f.m2 = f.u * f.u + f.v * f.v + f.w * f.w;
  f.mod = dsqrt64(f.m2);
  if (!d64_zero(f.mod)) {
    f.dmod = div64(f.mod);
    f.um = quot64(f.u, f.dmod);
    f.vm = quot64(f.v, f.dmod);
    if (P.rheo_model == 1) {
      const double turb = quot64(rho_m * f.rg, dxi) * f.m2;
      nh1 = 0.0 - turb * f.um;
      nh2 = 0.0 - turb * f.vm;
    } else if (P.rheo_model == 6) {
      const double hor = sqrt(f.u * f.u + f.v * f.v);
      nh1 = 0.0 - rho_m * (f.u / hor) * P.friction_factor * f.m2;
      nh2 = 0.0 - rho_m * (f.v / hor) * P.friction_factor * f.m2;
    }
  }
}

// imaginary parts of the friction terms at the state of f with hu (col = 0)
// or hv (col = 1) perturbed by i e; one copy of the code for both columns
__device__ __forceinline__ void friction_imag(const Phys<double>& P, double Bx, double By, const Div64& dxi,
                                              const FrictPoint& f, int col, double q1, double q2, double q3, double e,
                                              double& im1, double& im2) {
  im1 = 0.0;
  im2 = 0.0;
  if (!f.live) return;
  const double e1 = col ? 0.0 : e, e2 = col ? e : 0.0;
  // mixture density and reduced gravity: complex through the temperature
  Cplx rho{f.rho, 0.0}, rg{f.rg, 0.0};
  if (P.gas && P.energy && !f.film) {
    const double pr = col ? q2 : q1, ot = col ? q1 : q2;
    const double two = pr * e + e * pr;
    // the perturbed square first or second in the sum: the same sum
    const double s = (pr * pr - e * e) + ot * ot;
    const double nre = q3 - 0.5 * s * f.inv;
    const double nim = 0.0 - 0.5 * two * f.inv;
    const double Tre = quot64(nre, f.dT);
    const bool low = Tre <= 0.0;
    const double Tim = low ? 0.0 : quot64(nim, f.dT);
    const Cplx ir{f.dinv + f.xc * (f.Rc * (low ? P.T_ambient : Tre) * P.inv_pres), f.xc * (f.Rc * Tim * P.inv_pres)};
    rho = cdiv(Cplx{1.0, 0.0}, ir, f.dinvr, 1.0, f.rho);
    const Cplx qr = cdiv(Cplx{rho.re - P.rho_a_amb, rho.im}, rho, f.drho, f.nrg, f.qrg);
    rg = Cplx{qr.re * P.grav, qr.im * P.grav};
  }
  // the velocities: the imaginary part of the perturbed one; a film's real
  // parts are those of the real evaluation (the same products and quotients)
  const Cplx u{f.u, f.film ? quot64(f.s0 * e1, f.den) : e1 * f.inv};
  const Cplx v{f.v, f.film ? quot64(f.s0 * e2, f.den) : e2 * f.inv};
  Cplx w{0.0, 0.0};
  if (P.slope_corr) w = Cplx{f.w, u.im * Bx + v.im * By};
  const Cplx hz{(u.re * u.re - u.im * u.im) + (v.re * v.re - v.im * v.im),
                (u.re * u.im + u.im * u.re) + (v.re * v.im + v.im * v.re)};
  const Cplx m2{hz.re + (w.re * w.re - w.im * w.im), hz.im + (w.re * w.im + w.im * w.re)};
  const Cplx mod = csqrt64(m2, f.m2, f.mod, f.dmod);
  if (d64_zero(mod.re)) return;
  if (P.rheo_model == 1) {
    const Cplx um = cdiv(u, mod, f.dmod, f.u, f.um), vm = cdiv(v, mod, f.dmod, f.v, f.vm);
    const Cplx rr = cmul(rho, rg);
    const Cplx turb = cmul(Cplx{quot64(rr.re, dxi), quot64(rr.im, dxi)}, m2);
    im1 = 0.0 - (turb.re * um.im + turb.im * um.re);
    im2 = 0.0 - (turb.re * vm.im + turb.im * vm.re);
  } else if (P.rheo_model == 6) {
    const Cplx hor = csqrt64(hz, -1.0, 0.0, f.dmod);
    Cplx t = cmul(rho, cdiv_plain(u, hor));
    t = cmul(Cplx{t.re * P.friction_factor, t.im * P.friction_factor}, m2);
    im1 = 0.0 - t.im;
    t = cmul(rho, cdiv_plain(v, hor));
    t = cmul(Cplx{t.re * P.friction_factor, t.im * P.friction_factor}, m2);
    im2 = 0.0 - t.im;
  }
}

// residual of eval_f at q and its half square sum
template <int NS>
__device__ __forceinline__ void newton_residual(const NewtonCtx& c, const double* dtR, const double* q, double nh1,
                                                double nh2, double* f, double& scal_f) {
  constexpr int nv = 4 + NS;
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < nv; ++i) {
    if (i == 1 || i == 2) f[i] = q[i] - c.q_old[i] + c.dt * (c.Rj[i] - c.a_diag * (i == 1 ? nh1 : nh2));
    else f[i] = q[i] - c.q_old[i] + dtR[i];
    s += f[i] * f[i];
  }
  scal_f = 0.5 * s;
}
template <int NS>
__device__ __forceinline__ long long newton_maxf(const double* f) {
  constexpr int nv = 4 + NS;
  long long m = 0;
#pragma unroll
  for (int i = 0; i < nv; ++i) m = d64_absmax(m, d64_bits(f[i]) & kD64Abs);
  return m;
}

// The closure as solve_rk_step reads it (a host test of the iteration passes
// one of its own).
template <int NS>
struct Friction {
  static __device__ __forceinline__ void real(const Phys<double>& P, double Bx, double By, const Div64& dxi,
                                              const double* q, FrictPoint& f, double& nh1, double& nh2) {
    friction_real<NS>(P, Bx, By, dxi, q, f, nh1, nh2);
  }
  static __device__ __forceinline__ void imag(const Phys<double>& P, double Bx, double By, const Div64& dxi,
                                              const FrictPoint& f, int col, double q1, double q2, double q3, double e,
                                              double& im1, double& im2) {
    friction_imag(P, Bx, By, dxi, f, col, q1, q2, q3, e, im1, im2);
  }
};

// solve_rk_step (normalize_q = T, normalize_f = F, opt_search_NL = T;
// implicit set {hu, hv}); returns the iterations used (kMaxNewton + 1 when
// the limit was reached).  The line search's cubic model never chooses its
// step: its minimiser is capped at half the last step and the step kept above
// the same half (solver_2d.f90:2205-2222), so after the first refusal, which
// follows the quadratic model, the step is halved.  The quadratic model's own
// step may be infinite or return to 1, and then no halving reaches the least
// step: after kMaxTrials refusals the last trial is taken, which bounds the
// search.  One loop evaluates the closure for every purpose, so that the code
// holds it once (the kernel's code exceeds the instruction cache).
template <int NS, class F = Friction<NS>>
__device__ __forceinline__ int solve_rk_step(const NewtonCtx& c, double* qj) {
  constexpr int nv = 4 + NS;
  const double STPMX = 100.0, TOLF = 1.0e-10, TOLX = kEps;
  const Phys<double>& P = *c.P;
  double org[nv], rel[nv], f[nv], p[nv], xo[nv], dtR[nv];
  double scal_f = 0.0, scal_old = 0.0, slope = 0.0, alam = 1.0, alamin = -1.0, nh1, nh2;
  FrictPoint fp;
  Div64 dxi{};
  if (P.rheo_model == 1) dxi = div64(P.xi);
  const double h = nv * kEps, one_by_h = 1.0 / h, dta = c.dt * c.a_diag;
#pragma unroll
  for (int i = 0; i < nv; ++i) dtR[i] = c.dt * c.Rj[i];
  enum { START, SCALED, FIRST, TRIAL } phase = START;
  int it = 0, trials = 0;
#pragma unroll 1
  for (;;) {
    F::real(P, c.Bx, c.By, dxi, qj, fp, nh1, nh2);
    if (phase != SCALED) newton_residual<NS>(c, dtR, qj, nh1, nh2, f, scal_f);
    if (phase == START) {
      if (newton_maxf<NS>(f) < d64_bits(TOLF)) return 1;
      if (!isfinite(scal_f)) return kMaxNewton + 1;   // NaN/Inf state: give up at once
      // the Jacobian's state is rel * org, which may differ from qj in the last bit
      bool same = true;
#pragma unroll
      for (int i = 0; i < nv; ++i) {
        org[i] = d64_lt(1.0e-3, fabs(qj[i])) ? fabs(qj[i]) : 1.0e-3;
        rel[i] = ddiv64(qj[i], org[i]);
        const double x = rel[i] * org[i];
        same = same && d64_bits(x) == d64_bits(qj[i]);
        qj[i] = x;
      }
      if (!same) {
        phase = SCALED;
        continue;
      }
    } else if (phase != SCALED) {
      if (phase == TRIAL && (d64_lt(0.9 * scal_old, scal_f) || (d64_bits(scal_f) & kD64Abs) > kD64Inf)) {
        // refused: a shorter step, or stop at the old point (where the step
        // test below holds) when it is below the least step TOLX / max |p|
        if (alamin < 0.0) {
          double mx = 0.0;
#pragma unroll
          for (int i = 0; i < nv; ++i) {
            const double ax = fabs(xo[i]), t = ddiv64(fabs(p[i]), ax > 1.0 ? ax : 1.0);
            if (i == 0 || t > mx) mx = t;
          }
          alamin = ddiv64(TOLX, mx);
        }
        const bool stop = alam < alamin;
        if (stop || ++trials < kMaxTrials) {
          const double quad = (alam == 1.0) ? -slope / (2.0 * (scal_f - scal_old - slope)) : 0.0;
          alam = (quad > 0.5 * alam) ? quad : 0.5 * alam;
#pragma unroll
          for (int i = 0; i < nv; ++i) {
            rel[i] = stop ? xo[i] : xo[i] + alam * p[i];
            qj[i] = rel[i] * org[i];
          }
          if (stop) return it;
          continue;
        }
      }
      if (newton_maxf<NS>(f) < d64_bits(TOLF)) return it;
      // |step| < TOLX max(|rel|, 1) in every component: TOLX is a power of
      // two, so the product is exact and orders as the quotient does (a NaN
      // component is forgotten when a later one is a number, as the maximum
      // forgets it)
      bool small = true, was_nan = false;
#pragma unroll
      for (int i = 0; i < nv; ++i) {
        const double ar = fabs(rel[i]), st = fabs(rel[i] - xo[i]);
        small = (small || was_nan) && d64_lt(st, TOLX * (d64_lt(1.0, ar) ? ar : 1.0));
        was_nan = d64_bits(st) > kD64Inf || (d64_bits(st) == kD64Inf && d64_bits(ar) == kD64Inf);
      }
      if (small) return it;
      // the next iteration's first test
      if (!isfinite(scal_f)) return kMaxNewton + 1;
    }
    // the next direction; qj = rel * org, fp is the closure at qj, f the
    // residual (of the unscaled start state in the first iteration)
    if (++it > kMaxNewton) return kMaxNewton + 1;
    double j1[2], j2[2];
#pragma unroll 1
    for (int col = 0; col < 2; ++col) {
      double a1, a2;
      F::imag(P, c.Bx, c.By, dxi, fp, col, qj[1], qj[2], qj[3], h * (col ? org[2] : org[1]), a1, a2);
      if (col) { j1[1] = a1; j2[1] = a2; }
      else { j1[0] = a1; j2[0] = a2; }
    }
    const double s11 = org[1] - dta * (j1[0] * one_by_h), s12 = 0.0 - dta * (j1[1] * one_by_h);
    const double s21 = 0.0 - dta * (j2[0] * one_by_h), s22 = org[2] - dta * (j2[1] * one_by_h);
    const double inv_det = ddiv64(1.0, s11 * s22 - s21 * s12);
    double nrm = 0.0;
#pragma unroll
    for (int i = 0; i < nv; ++i) {
      // explicit rows: diagonal org, no coupling into the implicit rows
      if (i == 1) p[1] = -((f[1] * s22 - f[2] * s12) * inv_det) + 0.0;
      else if (i == 2) p[2] = -((s11 * f[2] - s21 * f[1]) * inv_det) + 0.0;
      else p[i] = d64_zero(f[i]) ? 0.0 : -ddiv64(f[i], org[i]);
      xo[i] = rel[i];
      nrm += p[i] * p[i];
    }
    scal_old = scal_f;
    phase = (it == 1) ? FIRST : TRIAL;
    if (it > 1) {
      alam = 1.0;
      trials = 0;
      slope = 0.0;
      alamin = -1.0;
      if (!d64_lt(nrm, (99.0 * nv) * (99.0 * nv))) {
        // |p| may pass the largest step, 100 max(|x|, n_vars)
        nrm = sqrt(nrm);
        double nr = 0.0;
#pragma unroll
        for (int i = 0; i < nv; ++i) nr += xo[i] * xo[i];
        const double sn = sqrt(nr), stpmax = STPMX * (sn > double(nv) ? sn : double(nv));
        if (nrm > stpmax) {
#pragma unroll
          for (int i = 0; i < nv; ++i) p[i] = p[i] * stpmax / nrm;
        }
        // a direction so long that TOLX / max |p| is 0 is not tried
        double mx = 0.0;
#pragma unroll
        for (int i = 0; i < nv; ++i) {
          const double ax = fabs(xo[i]), t = fabs(p[i]) / (ax > 1.0 ? ax : 1.0);
          if (i == 0 || t > mx) mx = t;
        }
        alamin = TOLX / mx;
        if (alamin == 0.0) {
#pragma unroll
          for (int i = 0; i < nv; ++i) qj[i] = xo[i] * org[i];
          return it;
        }
      }
      // derivative of the half square sum along p (explicit columns of the
      // matrix: diagonal org)
#pragma unroll
      for (int i = 0; i < nv; ++i)
        slope += ((i == 1) ? f[1] * s11 + f[2] * s21 : (i == 2) ? f[1] * s12 + f[2] * s22 : f[i] * org[i]) * p[i];
    }
#pragma unroll
    for (int i = 0; i < nv; ++i) {
      rel[i] = xo[i] + p[i];
      qj[i] = rel[i] * org[i];
    }
  }
}

}  // namespace sflow
