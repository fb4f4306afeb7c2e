// sflow_flux64.cuh -- the flux kernel of the plain FP64 form: divFlux -
// expl_terms of one explicit stage for the active cells of a part of a tile
// (eval_hyperbolic_terms, solver_2d.f90:2616-2693, and eval_expl_terms), and
// the CFL minimum of timestep (solver_2d.f90:873-1006); what flux_tile does
// for the FP32 form, with the same bits as the reference's operation order.
//
// Bound by FP64 instructions (2 lanes per clock and SM), so the work is laid
// out to have few of them and to spread them over the SMs:
//  * a divided difference (v2 - v1)/(z2 - z1) belongs to a face and is formed
//    once, not by the four cell sides that limit with it; the quotients by
//    one spacing share its reciprocal, and minmod is integer work;
//  * the CFL bound takes one division per block: cfl dx / a falls with a,
//    also when rounded, so the least bound is that of the largest speed;
//  * a block does SH = 4, 2 or 1 rows of a 32 x 8 tile.  Fewer rows repeat
//    more of the halo and the faces between blocks (per cell, 2.28, 2.53 and
//    3.03 faces and 2.3, 3.4 and 5.6 closures of the halo), more rows leave
//    SMs idle on small domains: flux64_rows picks;
//  * 192 threads, 3 blocks per SM (96 registers, with spills): 18 warps cover
//    the latency of the FP64 chains (512^2 current, 2 classes, 224 us; 2 blocks
//    without spills 288; 128 threads, 4 blocks 240).  Shared memory is 59.7,
//    68.4 and 77.1 KB a block with 1, 2 and 3 classes; three of the last do not
//    fit an SM's 228 KB, so runs of 3 classes have 2 blocks and the spills all
//    the same.
// Measured, one kernel of the FP32 layout before -> after: 512^2 current
// (96,000 wet cells) 346 -> 224 us, 200^2 dam break 164 -> 103, 64^2 102 -> 47,
// eroding flood 184 -> 90, FP64 ensemble 328 -> 160 us per step.  (The 512^2
// current with 1 and 3 classes: 189 and 282 us.)
#pragma once
#include "sflow_kernels.cuh"

namespace sflow {

constexpr int kFlux64Threads = 192;
constexpr int kFlux64Rows = 4;          // most rows of a block
constexpr int kFlux64Plane = RX * TileShape<8>::RY;   // stride of a qp plane (recon_side's)
constexpr int kFlux64QX = (TX + 3) * kFlux64Rows;     // divided differences along x: faces -1 .. TX + 1
constexpr int kFlux64QY = TX * (kFlux64Rows + 3);     // along y: faces -1 .. SH + 1
constexpr int kFlux64HX = (TX + 1) * kFlux64Rows, kFlux64HY = TX * (kFlux64Rows + 1);

static inline size_t flux64_smem_bytes(int nv) {
  const size_t np = (size_t)nv + 2;
  const size_t dbl = np * kFlux64Plane + np * (kFlux64QX + kFlux64QY) + (size_t)(nv + 1) * (kFlux64HX + kFlux64HY) +
                     2 * (TX + 3 + kFlux64Rows + 3);
  return (dbl * sizeof(double) + kFlux64Plane + 15) / 16 * 16;
}

// Rows of a tile per block for `tiles` tiles (32 x 8) on `sms` SMs: the most
// that still make two blocks per SM (of the three resident).  200 x 200 dam
// break, 175 tiles: 103 us with 4 rows, 122 with 2; 360 x 180 flood wet in a
// quarter of its 276 tiles: 90 and 72; 64^2 dam break, 16 tiles: 57 us with 2,
// 47 with 1.
static inline int flux64_rows(int64_t tiles, int sms) {
  if (tiles * (8 / 4) >= (int64_t)2 * sms) return 4;
  if (tiles * (8 / 2) >= (int64_t)2 * sms) return 2;
  return 1;
}

// minmod of two slopes by their bits: sign and least magnitude when the
// signs agree, else 0 (the bits of 0.5 (a/|a| + b/|b|) min(|a|, |b|))
__device__ __forceinline__ double minmod64(double a, double b) {
  const long long ba = d64_bits(a), bb = d64_bits(b), ma = ba & kD64Abs, mb = bb & kD64Abs;
  if (ma >= kD64Inf || mb >= kD64Inf) return minmod<double>(a, b);
  const long long m = ma < mb ? ma : mb;
  return ((ba ^ bb) < 0 || m == 0) ? 0.0 : d64_from((ba & ~kD64Abs) | m);
}

// Reconstructed state of one side of a face for an ordinary cell (interior,
// no ring face) from the divided differences behind (qb) and before it (qa);
// v: the cell's physical variables, strides of the planes sv and sq.
template <int NS>
__device__ __forceinline__ void recon64(const double* v, int sv, const double* qb, const double* qa, int sq, double kd,
                                        int plus, double* out) {
#pragma unroll
  for (int i = 0; i < 4 + NS + 2; ++i) {
    const double dq = kd * minmod64(qa[i * sq], qb[i * sq]);
    out[i] = plus ? v[i * sv] + dq : v[i * sv] - dq;
  }
}

// the other cells (domain edge, ring inlet), and every cell of other limiters
// (out of line, through memory: here the state is better off in local memory
// than in the registers of the FP64 arithmetic)
template <int NS, int DIR, int LIM>
__device__ __noinline__ void recon64_other(const KArgs<double>& a, const double* sqp, const uint8_t* sfl, int rx,
                                           int ry, int j, int k, int plus, double* out) {
  recon_side<double, NS, DIR, LIM, 8>(a, sqp, sfl, rx, ry, j, k, plus, out);
}

// face_flux with recon64 for the ordinary cells: qf points at the divided
// differences of this face, step to those of the next face along DIR
template <int NS, int DIR, int LIM, bool FLUX>
__device__ __forceinline__ double face_flux64(const KArgs<double>& a, const double* sqp, const uint8_t* sfl,
                                              const double* qf, int step, int sq, int f, int o, int rxl, int ryl,
                                              int rxh, int ryh, double gcs, double* H) {
  constexpr int nv = 4 + NS, np = nv + 2;
  constexpr int vel = (DIR == 1) ? nv : nv + 1;
  const Grid<double>& g = a.g;
  const int n = (DIR == 1) ? g.nx : g.ny;
  const uint8_t fll = (f > 0) ? sfl[ryl * RX + rxl] : 0;
  const uint8_t flh = (f < n) ? sfl[ryh * RX + rxh] : 0;
  const bool actl = fll & F_ACTIVE, acth = flh & F_ACTIVE;
  const bool radial = a.pr.radial_source;
  const bool src_l = radial && (fll & F_SC_MASK) == 2, src_h = radial && (flh & F_SC_MASK) == 2;
  const bool ring_l = src_l && f - 1 > 0 && f - 1 < n - 1;
  const bool ring_h = src_h && f > 0 && f < n - 1;
  const bool mirror_h = actl && ring_l && ((DIR == 1) ? (fll & F_E) : ((fll & F_N) && !(fll & F_S)));
  const bool mirror_l = !mirror_h && acth && ring_h && ((DIR == 1) ? ((flh & F_W) && !(flh & F_E)) : (flh & F_S));
  const double kd = g.rc * ((DIR == 1) ? g.dx2 : g.dy2);
  double qpl[np], qph[np];
  bool hl = false, hh = false;
  if (f > 0 && actl) {
    if (LIM == 1 && f - 1 > 0 && f < n && !src_l)
      recon64<NS>(sqp + ryl * RX + rxl, kFlux64Plane, qf - step, qf, sq, kd, 1, qpl);
    else
      recon64_other<NS, DIR, LIM>(a, sqp, sfl, rxl, ryl, (DIR == 1) ? f - 1 : o, (DIR == 1) ? o : f - 1, 1, qpl);
    hl = true;
  }
  if (f < n && acth && !mirror_h) {
    if (LIM == 1 && f > 0 && f < n - 1 && !src_h)
      recon64<NS>(sqp + ryh * RX + rxh, kFlux64Plane, qf, qf + step, sq, kd, 0, qph);
    else
      recon64_other<NS, DIR, LIM>(a, sqp, sfl, rxh, ryh, (DIR == 1) ? f : o, (DIR == 1) ? o : f, 0, qph);
    hh = true;
  }
  if (f == 0) {
#pragma unroll
    for (int i = 0; i < np; ++i) qpl[i] = qph[i];
    hl = hh;
  }
  if (f == n) {
#pragma unroll
    for (int i = 0; i < np; ++i) qph[i] = qpl[i];
    hh = hl;
  }
  if (mirror_h) {
#pragma unroll
    for (int i = 0; i < np; ++i) qph[i] = qpl[i];
    qph[vel] = -qph[vel];
    hh = true;
  }
  if (mirror_l) {
#pragma unroll
    for (int i = 0; i < np; ++i) qpl[i] = qph[i];
    qpl[vel] = -qpl[vel];
    hl = true;
  }
  Side<double, NS> L, Hs;
  // one copy of the side closure (instruction cache)
#pragma unroll 1
  for (int s = 0; s < 2; ++s) {
    double t[np];
    Side<double, NS> S;
#pragma unroll
    for (int i = 0; i < np; ++i) t[i] = s ? qph[i] : qpl[i];
    if (s ? hh : hl) side_from_qp<double, NS, DIR, FLUX>(a, t, gcs, S, s ? mirror_h : mirror_l);
    else side_zero(S);
    if (s) Hs = S;
    else L = S;
  }
  if constexpr (!FLUX) return rmax(rmax(rmax(L.vmax, Hs.vmax), 0.0), -rmin(rmin(L.vmin, Hs.vmin), 0.0));
  if (a.pr.scheme == SFLOW_SCHEME_UP) return up_flux<double, NS, DIR>(L, Hs, H);
  return kt_flux<double, NS, DIR>(L, Hs, H);
}

// rows r0 .. r0 + sh - 1 of tile (tx, ty)
template <int NS, int LIM, bool FLUX>
__device__ __forceinline__ void flux_tile64(const KArgs<double>& a, const double* __restrict__ qin,
                                            double* __restrict__ rout, int want_dt, int tx, int ty, int r0, int sh,
                                            unsigned char* smem_raw) {
  constexpr int nv = 4 + NS, np = nv + 2;
  const RunState* st = a.st;
  const Grid<double>& g = a.g;
  const Phys<double>& P = a.pr;
  double* sqp = reinterpret_cast<double*>(smem_raw);   // np planes, rows of RX
  double* sQx = sqp + np * kFlux64Plane;               // np planes, rows of TX + 3
  double* sQy = sQx + np * kFlux64QX;                  // np planes, rows of TX
  double* sHx = sQy + np * kFlux64QY;
  double* sHy = sHx + nv * kFlux64HX;
  double* sAx = sHy + nv * kFlux64HY;
  double* sAy = sAx + kFlux64HX;
  Div64* sdz = reinterpret_cast<Div64*>(sAy + kFlux64HY);   // spacings at the x faces, then the y faces
  uint8_t* sfl = reinterpret_cast<uint8_t*>(sdz + TX + 3 + kFlux64Rows + 3);
  __shared__ unsigned long long s_max[2];
  const int j0 = tx * TX, k0 = ty * 8 + r0;
  const int tid = threadIdx.x;
  const int ryn = sh + 2 * HALO;
  if (k0 >= g.ny) return;   // block-uniform

  __syncthreads();   // shared memory of the previous tile of a persistent block is free
  if (tid < 2) s_max[tid] = 0ull;
  // 1. spacings of the cell centres; physical variables of the rows + halo
  if (LIM == 1 && tid < TX + 3 + sh + 3) {
    const bool x = tid < TX + 3;
    const int m = x ? j0 - 1 + tid : k0 - 1 + (tid - (TX + 3));   // face m between cells m - 1 and m
    sdz[tid] = div64(x ? xcomp(g, m) - xcomp(g, m - 1) : ycomp(g, m) - ycomp(g, m - 1));
  }
  int any_wet = 0, all_wet = 1, any_bsrc = 0;
  for (int idx = tid; idx < RX * ryn; idx += kFlux64Threads) {
    const int rx = idx % RX, ry = idx / RX;
    const int j = j0 + rx - HALO, k = k0 + ry - HALO;
    uint8_t fl = 0;
    double qp[np];
    bool wet = false;
    if (j >= 0 && j < g.nx && k >= 0 && k < g.ny) {
      const int64_t c = cidx(g, j, k);
      fl = a.cflags[c];
      any_bsrc |= (fl & F_BSRC) != 0;
      fl &= F_STATIC;
      if (a.mask[c]) {
        fl |= F_ACTIVE;
        double q[nv];
#pragma unroll
        for (int i = 0; i < nv; ++i) q[i] = qin[i * g.plane + c];
        if (d64_pos(q[0])) {
          qc_to_qp<double, NS>(P, q, qp);
          wet = true;
          fl |= F_WET;
        }
      }
    }
    if (!wet) {
#pragma unroll
      for (int i = 0; i < np; ++i) qp[i] = 0.0;
      qp[3] = P.T_ambient;
    }
#pragma unroll
    for (int i = 0; i < np; ++i) sqp[i * kFlux64Plane + idx] = qp[i];
    sfl[idx] = fl;
    any_wet |= wet;
    all_wet &= wet;
  }
  // dry faces and rows: see flux_tile
  const bool some_wet = __syncthreads_or(any_wet);
  const bool any_bsrc_tile = P.bottom_source ? __syncthreads_or(any_bsrc) != 0 : false;
  const bool inside = j0 - HALO >= 0 && k0 - HALO >= 0 && j0 + TX + HALO <= g.nx && k0 + sh + HALO <= g.ny;
  const bool dry = !some_wet && (g.dry_bc || inside);
  const bool face_checks = !__syncthreads_and(all_wet);

  // 2. divided differences (minmod on every variable): (v2 - v1)/(z2 - z1)
  // between the two cells of a face, for the faces of the cells one beyond
  if (LIM == 1 && !dry) {
    for (int e = tid; e < (TX + 3) * sh; e += kFlux64Threads) {
      const int m = e % (TX + 3), r = e / (TX + 3);   // between region columns m and m + 1
      const Div64 v = sdz[m];
      const int o = (r + HALO) * RX + m;
#pragma unroll
      for (int i = 0; i < np; ++i)
        sQx[i * kFlux64QX + e] = quot64(sqp[i * kFlux64Plane + o + 1] - sqp[i * kFlux64Plane + o], v);
    }
    if (g.ny > 1)
      for (int e = tid; e < TX * (sh + 3); e += kFlux64Threads) {
        const int c = e % TX, m = e / TX;               // between region rows m and m + 1
        const Div64 v = sdz[TX + 3 + m];
        const int o = m * RX + c + HALO;
#pragma unroll
        for (int i = 0; i < np; ++i)
          sQy[i * kFlux64QY + e] = quot64(sqp[i * kFlux64Plane + o + RX] - sqp[i * kFlux64Plane + o], v);
      }
    __syncthreads();
  }

  // 3. faces: the warps take the x faces (f = j0 + fx between cells f - 1 and
  // f) and then the y faces (f = k0 + fy; none in one-row domains) 32 at a
  // time, so that both kinds are in flight together
  const int xch = ((TX + 1) * sh + 31) / 32, ych = g.ny > 1 ? sh + 1 : 0;
  for (int ch = tid / 32; ch < xch + ych && !dry; ch += kFlux64Threads / 32) {
    if (ch < xch) {
      const int fi = ch * 32 + tid % 32;
      if (fi >= (TX + 1) * sh) continue;
      const int fx = fi % (TX + 1), fy = fi / (TX + 1);
      const int f = j0 + fx, k = k0 + fy;
      double H[nv];
      double amax = 0.0;
      const int ry = fy + HALO, rxl = fx - 1 + HALO, rxh = fx + HALO;
      const bool stencil_dry =
          face_checks &&
          !((sfl[ry * RX + rxl - 1] | sfl[ry * RX + rxl] | sfl[ry * RX + rxh] | sfl[ry * RX + rxh + 1]) & F_WET) &&
          (g.dry_bc || (f >= 2 && f + 1 <= g.nx - 1));
      const bool any = (k < g.ny && f <= g.nx) && !stencil_dry &&
                       (((f > 0) && (sfl[ry * RX + rxl] & F_ACTIVE)) || ((f < g.nx) && (sfl[ry * RX + rxh] & F_ACTIVE)));
      if (any) {
        const int64_t cl = cidx(g, f > 0 ? f - 1 : 0, k), ch = cidx(g, f < g.nx ? f : g.nx - 1, k);
        double gcs;
        if (f == 0) gcs = __ldg(a.geo[5] + ch);
        else if (f == g.nx) gcs = __ldg(a.geo[5] + cl);
        else gcs = 0.5 * (__ldg(a.geo[5] + cl) + __ldg(a.geo[5] + ch));
        amax = face_flux64<NS, 1, LIM, FLUX>(a, sqp, sfl, sQx + fy * (TX + 3) + fx + 1, 1, kFlux64QX, f, k, rxl, ry, rxh, ry,
                                       gcs, H);
      } else {
#pragma unroll
        for (int i = 0; i < nv; ++i) H[i] = 0.0;
      }
      if constexpr (FLUX) {
#pragma unroll
        for (int i = 0; i < nv; ++i) sHx[i * kFlux64HX + fi] = H[i];
      }
      sAx[fi] = amax;
    } else {
      const int fi = (ch - xch) * 32 + tid % 32;
      const int fx = fi % TX, fy = fi / TX;
      const int j = j0 + fx, f = k0 + fy;
      double H[nv];
      double amax = 0.0;
      const int rx = fx + HALO, ryl = fy - 1 + HALO, ryh = fy + HALO;
      const bool stencil_dry =
          face_checks &&
          !((sfl[(ryl - 1) * RX + rx] | sfl[ryl * RX + rx] | sfl[ryh * RX + rx] | sfl[(ryh + 1) * RX + rx]) & F_WET) &&
          (g.dry_bc || (f >= 2 && f + 1 <= g.ny - 1));
      const bool any = (j < g.nx && f <= g.ny) && !stencil_dry &&
                       (((f > 0) && (sfl[ryl * RX + rx] & F_ACTIVE)) || ((f < g.ny) && (sfl[ryh * RX + rx] & F_ACTIVE)));
      if (any) {
        const int64_t cl = cidx(g, j, f > 0 ? f - 1 : 0), ch = cidx(g, j, f < g.ny ? f : g.ny - 1);
        double gcs;
        if (f == 0) gcs = __ldg(a.geo[5] + ch);
        else if (f == g.ny) gcs = __ldg(a.geo[5] + cl);
        else gcs = 0.5 * (__ldg(a.geo[5] + cl) + __ldg(a.geo[5] + ch));
        amax = face_flux64<NS, 2, LIM, FLUX>(a, sqp, sfl, sQy + (fy + 1) * TX + fx, TX, kFlux64QY, f, j, rx, ryl, rx, ryh, gcs,
                                       H);
      } else {
#pragma unroll
        for (int i = 0; i < nv; ++i) H[i] = 0.0;
      }
      if constexpr (FLUX) {
#pragma unroll
        for (int i = 0; i < nv; ++i) sHy[i * kFlux64HY + fi] = H[i];
      }
      sAy[fi] = amax;
    }
  }
  __syncthreads();

  // 4. cells: divergence, explicit terms, largest speeds
  unsigned long long mx = 0ull, my = 0ull;
  if (tid < TX * sh) {
    const int cx = tid % TX, cy = tid / TX;
    const int j = j0 + cx, k = k0 + cy;
    const int rx = cx + HALO, ry = cy + HALO;
    const uint8_t fl = sfl[ry * RX + rx];
    const bool active = j < g.nx && k < g.ny && (fl & F_ACTIVE);
    if (want_dt & 2) {   // the row's active cells into the list of k_stage2_list
      const unsigned m = __ballot_sync(0xffffffffu, active);
      unsigned at = 0;
      if (cx == 0 && m) at = atomicAdd(&a.st->list_n, (unsigned)__popc(m));
      at = __shfl_sync(0xffffffffu, at, 0) + (unsigned)__popc(m & ((1u << cx) - 1u));
      if (active) a.cells[at] = (uint32_t)cidx(g, j, k);
    }
    if (active) {
      const int64_t c = cidx(g, j, k);
      if constexpr (FLUX) {
        double qp[np];
#pragma unroll
        for (int i = 0; i < np; ++i) qp[i] = sqp[i * kFlux64Plane + ry * RX + rx];
        double e[nv];
        const Geo<double> geo = load_geo(a, c);
        double ap = 0.0, anx = 0.0, any_ = 0.0, tcoef = 0.0;   // read at ring cells only (arc perimeter > 0)
        if (P.radial_source && (fl & F_SC_MASK) == 2) {
          ap = __ldg(a.arc + c);
          anx = __ldg(a.arc + g.plane + c);
          any_ = __ldg(a.arc + 2 * g.plane + c);
          tcoef = st->src_t_coeff;
        }
        double bf = 0.0, btc = 0.0, bvel = 0.0;   // bottom source cells only
        if (P.bottom_source && any_bsrc_tile && (__ldg(a.cflags + c) & F_BSRC)) {
          bf = __ldg(a.bfrac + c);
          btc = st->bsrc_t_coeff;
          bvel = st->bsrc_vel;
        }
        expl_terms<double, NS>(P, geo, qp, tcoef, ap, anx, any_, bf, btc, bvel, e);
#pragma unroll
        for (int i = 0; i < nv; ++i) {
          double d = 0.0;
          if (!dry) {
            const int x = cy * (TX + 1) + cx;
            d = (sHx[i * kFlux64HX + x + 1] - sHx[i * kFlux64HX + x]) * g.one_by_dx;
            if (g.ny > 1) d = d + (sHy[i * kFlux64HY + tid + TX] - sHy[i * kFlux64HY + tid]) * g.one_by_dy;
          }
          rout[i * g.plane + c] = d - e[i];
        }
      }
      if (want_dt && !dry && owned_row(g, k)) {
        const double xl = sAx[cy * (TX + 1) + cx], xh = sAx[cy * (TX + 1) + cx + 1];
        const double ax = d64_lt(xh, xl) ? xl : xh;
        if (d64_pos(ax)) mx = (unsigned long long)d64_bits(ax);
        if (g.ny > 1) {
          const double yl = sAy[tid], yh = sAy[tid + TX];
          const double ay = d64_lt(yh, yl) ? yl : yh;
          if (d64_pos(ay)) my = (unsigned long long)d64_bits(ay);
        }
      }
    }
  }
  if (want_dt && !dry) {
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long x = __shfl_xor_sync(0xffffffffu, mx, o), y = __shfl_xor_sync(0xffffffffu, my, o);
      mx = x > mx ? x : mx;
      my = y > my ? y : my;
    }
    if ((tid & 31) == 0) {
      atomicMax(&s_max[0], mx);
      atomicMax(&s_max[1], my);
    }
    __syncthreads();
    if (tid < 2 && s_max[tid]) {
      const double bd = ddiv64(g.cfl * (tid ? g.dy : g.dx), d64_from((long long)s_max[tid]));
      if (bd < 1.0e300) atomicMin(&a.st->dtmin_bits, dbits(bd));
    }
  }
}

template <int NS, int LIM, bool FLUX>
__global__ void __launch_bounds__(kFlux64Threads, 3)
    k_flux64(KArgs<double> a, const double* __restrict__ qin, double* __restrict__ rout, int want_dt, int sh) {
  step_kernel_entry();
  const RunState* st = a.st;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // see k_flux
  const int parts = 8 / sh, by = block_row(), ty = by / parts;
  if (ty >= a.g.tiles_y) return;
  const uint8_t ta = a.tile_active[ty * gridDim.x + blockIdx.x];
  const bool go = want_dt ? running(st) : st->run_step != 0;
  if (!go | (ta == 0) | (ta == TILE_DRY_BORDER)) return;
  flux_tile64<NS, LIM, FLUX>(a, qin, rout, want_dt, blockIdx.x, ty, (by % parts) * sh, sh, smem_raw);
}

}  // namespace sflow
