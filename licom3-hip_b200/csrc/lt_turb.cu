// lt_turb.cu - the Canuto 2002 turbulence closure that produces the tracer
// step's vertical mixing (turb_cu with turb_device, interp1d_expabs,
// interp2d_expabs, formld and eplatidepend_fun, readyc.cpp:880-1612, with
// TIDEMIX as the reference is configured).  Compiled with -fmad=false: the
// operation order is the reference's term for term but for the cosine and sine
// of the background's angle; the transcendental functions (atan, acosh, rarely
// sin, cos, log) are CUDA's, so results agree with the reference to a few units
// in the last place, not bit for bit.
//
// One thread per column.  Where the reference first fills per-column work
// arrays (wp1, wp3, wp7, wp8 in [i][j][k] order) and then walks them, this
// kernel makes three passes down and up the column straight from the level
// fields, which a warp reads coalesced (i fastest):
//   1. upward from the deepest interface: the tidal mixing with the
//      reference's bottom-up minimum, and the tidal diagnostics;
//   2. downward: the mixed-layer depth (formld);
//   3. downward: the closure itself, level by level, keeping the few
//      neighbouring levels it looks at in registers, and the diffusivities
//      written as soon as a level is done (level 0 last: the wind-mixing floor
//      applies to it once the column is complete).
//
// Bound by latency: a long chain per level (square roots, atan, acosh,
// quotients, table gathers) at 20 warps per SM, instruction fetch across its
// branches, and idle lanes where neighbours differ in stability.  4.00 -> 2.18
// ms at 720 x 460 x 55 on the global area-depth curve with interleaved tables,
// brackets found without logarithms and the angle's cosine and sine taken from
// its components, which are nearer the exact ones than those of the rounded
// angle (root mean square 0.9e-16 against 6e-11 for the cosine).  Quotients
// that share a divisor are formed from its reciprocal and rounded as divisions
// (ratio).  Four, six or eight blocks per SM instead of five were slower by
// 7, 13 and 6 %.
#include <cmath>
#include <new>
#include <vector>
#include "lt_common.cuh"
#include "lt_domain.h"

struct lt_turb_tab {
  lt::TurbTabDev t;
  void* base = nullptr;
  int dev = 0;
};

namespace lt {
namespace {

constexpr int MT = LT_TURB_MT, MT0 = LT_TURB_MT0, NTH = LT_TURB_NTHETA;
constexpr int N1 = LT_TURB_N1;

// pconst_mod.h:242-247 and canuto_mod.h constants of the configuration
constexpr double kBackTidal = 1.0e-6, kMaxTidal = 1.0e-2, kMixingEf = 0.20, kLocalFrac = 0.33;
constexpr double kEpson2 = 0.288e0, kEplatMin = 7.0e-2, kS2min = 1.0e-14;

__device__ __forceinline__ double sgn(double x, double y) { return y >= 0.0 ? fabs(x) : -fabs(x); }

// Values the reference recomputes at every call from constants, formed once
// per launch on the host.
struct TurbConst {
  double pi4;               // atan(1.0)
  double eplat_den;         // wavelat(f_30, an0)
  double inv_ncc, inv_dth, inv_dri, inv_da;   // reciprocals: ncc (0: divide), deltheta_r, dri, dand2on2
  float log2_gm, per_log2;     // 2-D tables: log2(rib[mt + mt0]), 1/log2(rri)
  float log2_gm1, per_log21;   // zero-shear table
};

// wavelat / eplatidepend_fun (readyc.cpp:880-896)
__device__ __forceinline__ double eplat(const TurbConst& C, double f, double an) {
  const double anum = f * acosh(an / f);
  return anum / C.eplat_den;
}

// a / h with y = 1/h: where the tables allow it (TurbTabDev::plain: entries and
// steps within 1e-100 .. 1e100, entries also zero) the division's bits without
// its code, which this kernel has no room for in the instruction cache (with the
// general form's test and division at thirteen quotients a level 3.54 ms)
template <bool PLAIN>
__device__ __forceinline__ double ratio(double a, double h, double y) {
  return PLAIN ? div_fast(a, h, y) : a / h;
}

// Indices (offset by MT) of the entries that bracket x on an "expabs" grid
// (linear spacing delta up to grid[mt + mt0] = gm, geometric ratio rat beyond),
// lo towards zero, which interp1d_expabs and interp2d_expabs find from a
// quotient or a logarithm and a correction by one (readyc.cpp:922-941,
// 1014-1031).  Here the first guess is a product or a single-precision logarithm
// and the grid itself decides; where x meets an entry, which side of it counts is
// left to the quotient's or logarithm's rounding, so there (rarely) it is formed
// as the reference does: the tables' interpolation and the realizable limit are
// steps at an entry.
struct Bracket {
  int lo, hi;
};
__device__ __noinline__ int met_entry(double ax, const double* __restrict__ g, int s, double gm, double delta,
                                      double rat) {
  const double ti = ax < gm ? ax / delta : (double)MT0 + ((log(ax) - log(gm)) / log(rat));
  int m = max(1, min(MT, (int)ti + 1));
  if (fabs(g[MT + s * m]) < ax) m = min(MT, m + 1);
  else if (m > 1 && fabs(g[MT + s * (m - 1)]) > ax) --m;
  return m;
}
__device__ __forceinline__ Bracket bracket(double x, const double* __restrict__ g, double gm, double delta,
                                           double inv_delta, double rat, float log2_gm, float per_log2) {
  const double ax = fabs(x);
  const int s = x >= 0.0 ? 1 : -1;
  int m;
  if (ax < gm) m = 1 + (int)(ax * inv_delta);
  else m = 1 + MT0 + (int)((__log2f((float)ax) - log2_gm) * per_log2);
  m = max(1, min(MT, m));
  double above = fabs(g[MT + s * m]), below = fabs(g[MT + s * (m - 1)]);
  while (m < MT && above < ax) {
    below = above;
    above = fabs(g[MT + s * ++m]);
  }
  while (m > 1 && below > ax) {
    above = below;
    below = fabs(g[MT + s * (--m - 1)]);
  }
  if (above == ax || below == ax) m = met_entry(ax, g, s, gm, delta, rat);
  return {MT + s * (m - 1), MT + s * m};
}

// interp1d_expabs (readyc.cpp:915-973): false, outputs left as they were, when
// x falls outside the bracketing entries
__device__ __noinline__ bool interp1d(double x, const TurbTabDev& T, const TurbConst& C, double out[4]) {
  const double* x1 = T.and2on2a1;
  if (x > x1[2 * MT]) x = x1[2 * MT];
  else if (x < x1[0]) x = x1[0];
  const double gm = x1[MT + MT0], gmax = x1[2 * MT];
  Bracket b;
  if (fabs(x) >= gm && fabs(x) >= gmax) b.lo = b.hi = x >= 0.0 ? 2 * MT : 0;
  else b = bracket(x, x1, gm, T.dand2on2, C.inv_da, T.rnd2on2, C.log2_gm1, C.per_log21);
  const double x0 = x1[b.lo], xh = x1[b.hi];
  if ((x > 0.0e0 && (x < x0 || x > xh)) || (x < 0.0e0 && (x > x0 || x < xh))) return false;
  const double dta = xh - x0;
  const double dx = x - x0;
  const double* tab[4] = {T.amtaun2a1, T.sma1, T.sha1, T.ssa1};
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const double v = tab[m][b.lo];
    out[m] = v + (b.hi == b.lo ? 0.0e0 : (tab[m][b.hi] - v) / dta) * dx;
  }
  return true;
}

// interp2d_expabs (readyc.cpp:975-1114): ri, rid clipped to the table in
// place; outputs left as they were on the reference's early returns
// (false).  The four tables are interleaved, so a corner of the four is one
// 32-byte sector and two corners of a row are adjacent: the gathers, which
// miss L2 (274 MB of tables), touch 3 sectors per cell instead of 8.
struct Stab {
  double slq2, sm, sh, ss;
};
// 1 / (rib[b.hi] - rib[b.lo]); infinite at an end, where 0 / 0 is the slope
__device__ __forceinline__ double step_inverse(const TurbTabDev& T, Bracket b) {
  if (b.hi == b.lo) return INFINITY;
  const double y = __ldg(T.rstep + min(b.lo, b.hi));
  return b.hi > b.lo ? y : -y;
}
__device__ __forceinline__ Stab quad_at(const TurbTabDev& T, long c) {
  const double2* p = reinterpret_cast<const double2*>(T.quad) + 2 * c;
  const double2 u = __ldg(p), v = __ldg(p + 1);
  return {u.x, u.y, v.x, v.y};
}

template <bool PLAIN>
__device__ __forceinline__ bool interp2d(double& ri, double& rid, const TurbTabDev& T, const TurbConst& C, Stab& out) {
  const double* rib = T.rib;
  const double rmax = T.gmax, rmin = T.rib0, gm = T.gm;
  if (ri > rmax || ri < rmin || rid > rmax || rid < rmin) {
    if (ri > rmax) {
      if (fabs(rid) <= ri) {
        rid = rmax * (rid / ri);
        ri = rmax;
      } else if (rid > ri) {
        ri = rmax * (ri / rid);
        rid = rmax;
      } else if (rid < -ri) {
        ri = rmin * (ri / rid);
        rid = rmin;
      }
    } else if (ri < rmin) {
      if (fabs(rid) <= -ri) {
        rid = rmin * (rid / ri);
        ri = rmin;
      } else if (rid > -ri) {
        ri = rmax * (ri / rid);
        rid = rmax;
      } else if (rid < ri) {
        ri = rmin * (ri / rid);
        rid = rmin;
      }
    } else if (rid > rmax) {
      ri = rmax * (ri / rid);
      rid = rmax;
    } else if (rid < rmin) {
      ri = rmin * (ri / rid);
      rid = rmin;
    }
  }
  const double x_ri = ri, x_rid = rid;
  Bracket d, r;
  if (fabs(x_rid) >= gm && fabs(x_rid) >= rmax) d.lo = d.hi = x_rid >= 0.0 ? 2 * MT : 0;
  else d = bracket(x_rid, rib, gm, T.dri, C.inv_dri, T.rri, C.log2_gm, C.per_log2);
  const double d0 = rib[d.lo], d1 = rib[d.hi];
  if ((x_rid > 0.0e0 && (x_rid < d0 || x_rid > d1)) || (x_rid < 0.0e0 && (x_rid > d0 || x_rid < d1))) return false;
  if (x_ri > fmin(T.rilim[d.lo], T.rilim[d.hi])) {
    out = {0.0e0, 0.0e0, 0.0e0, 0.0e0};
    return true;
  }
  if (fabs(x_ri) >= gm && fabs(x_ri) >= rmax) r.lo = r.hi = x_ri >= 0.0 ? 2 * MT : 0;
  else r = bracket(x_ri, rib, gm, T.dri, C.inv_dri, T.rri, C.log2_gm, C.per_log2);
  const double r0 = rib[r.lo], r1 = rib[r.hi];
  if ((x_ri > 0.0e0 && (x_ri < r0 || x_ri > r1)) || (x_ri < 0.0e0 && (x_ri > r0 || x_ri < r1))) return false;
  const Stab t00 = quad_at(T, (long)N1 * d.lo + r.lo);
  const double drid = x_rid - d0, dri = x_ri - r0;
  if (d.hi == d.lo) {
    // at an end: no slopes, but a NaN in Ri stays one
    const double gone = 0.0e0 * dri, none = 0.0e0 * drid;
    out = {t00.slq2 + gone + none, t00.sm + gone + none, t00.sh + gone + none, t00.ss + gone + none};
  } else {
    const Stab t10 = quad_at(T, (long)N1 * d.hi + r.lo), t01 = quad_at(T, (long)N1 * d.lo + r.hi);
    // one reciprocal per direction, laid out with the grid, serves four
    // quotients, rounded as divisions
    const double dridta = d1 - d0, drita = r1 - r0;
    const double gd = step_inverse(T, d), gr = step_inverse(T, r);
    auto plane = [&](double v00, double v10, double v01) {
      return v00 + ratio<PLAIN>(v01 - v00, drita, gr) * dri + ratio<PLAIN>(v10 - v00, dridta, gd) * drid;
    };
    out.slq2 = plane(t00.slq2, t10.slq2, t01.slq2);
    out.sm = plane(t00.sm, t10.sm, t01.sm);
    out.sh = plane(t00.sh, t10.sh, t01.sh);
    out.ss = plane(t00.ss, t10.ss, t01.ss);
  }
  return true;
}
// the background's second look-up (rare), kept out of the level loop's code
template <bool PLAIN>
__device__ __noinline__ bool interp2d_back(double& ri, double& rid, const TurbTabDev& T, const TurbConst& C, Stab& out) {
  return interp2d<PLAIN>(ri, rid, T, C, out);
}

// One of the background's five tables (back_ra_r, sm_r1, sh_r1, ss_r1, slq2_r1)
// at dth beyond angle it0, with the slope to the next angle
__device__ __forceinline__ double angle(const TurbTabDev& T, int tab, int it0, double dth) {
  const double2 e = __ldg(T.angle + tab * LT_TURB_NB + NTH + it0);
  return e.x + dth * e.y;
}

// The column's interface values (the reference's wp1, wp3, wp8 at level k,
// k < kmt-1): temperature and density interpolated to the interface below
// level k, and its depth in cm
struct Iface {
  const double *T, *pd;
  const double *dz, *hs, *ys, *zz;   // shared memory: dzp, dzp + dzp of the next level, its reciprocal, depth
  long A;
  __device__ double t(int k) const {
    const double a = T[k * A];
    return a - quotient((a - T[(k + 1) * A]) * dz[k], hs[k], ys[k]);
  }
  __device__ double rh_of(int k, double p0, double p1) const {
    return (p0 + quotient((p1 - p0) * dz[k], hs[k], ys[k])) * 1.0e-3;
  }
  __device__ double rh(int k) const { return rh_of(k, pd[k * A], pd[(k + 1) * A]); }
  __device__ double z(int k) const { return zz[k]; }
};

constexpr int kTurbLevels = 256;   // most levels a domain may have

template <bool PLAIN>
__global__ void __launch_bounds__(128, 5)
    k_turb(const __grid_constant__ Arena a, const __grid_constant__ TurbTabDev T, const __grid_constant__ TurbConst C,
           double ncc_f, double fricmx, double wndmix) {
  __shared__ double s_dz[kTurbLevels], s_hs[kTurbLevels], s_ys[kTurbLevels], s_zz[kTurbLevels];
  for (int k = threadIdx.y * blockDim.x + threadIdx.x; k < a.km; k += blockDim.x * blockDim.y) {
    const double dz = a.dzp[k], h = dz + (k + 1 < a.km ? a.dzp[k + 1] : 0.0);
    s_dz[k] = dz;
    s_hs[k] = h;
    s_ys[k] = quotient_reciprocal(h);
    s_zz[k] = -a.zkp[k + 1] * 1.0e+2;
  }
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= a.imt || j >= a.jmt) return;
  const long q = (long)j * a.imt + i;
  const long A = a.A;
  const int km = a.km;
  const int kz = a.kmt[q];
  if (!(i > 0 && i < a.imt - 1 && j > 0 && j < a.jmt - 1 && kz > 0)) {
    // not a column of turb_cu: what the reference's memsets leave
    for (int k = 0; k < km; ++k) {
      a.akmt[k * A + q] = 0.0;
      a.ak_tide[k * A + q] = 0.0;
    }
    a.amld[q] = 0.0;
    return;
  }
  const int n = kz - 1;   // interfaces of the column (iwk)
  const Iface f{a.at[a.cur] + q, a.pdensity + q, s_dz, s_hs, s_ys, s_zz, A};
  const double* __restrict__ rict = a.rict + q;

  // ---- 1. tidal mixing, bottom-up minimum (readyc.cpp:1534-1557); four
  // levels' loads ahead of their stores
  {
    double below = 0.0;
    const double wd = a.wave_dis[q];
    const double* __restrict__ fzt = a.fz_tide + q;
    for (int k = km - 1; k >= n; --k) a.ak_tide[k * A + q] = 0.0;
    double pd1 = n > 0 ? f.pd[n * A] : 0.0;
    for (int k0 = n - 1; k0 >= 0; k0 -= 4) {
      double pd0[4], rc[4], fz[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int k = k0 - c >= 0 ? k0 - c : 0;
        pd0[c] = f.pd[k * A];
        rc[c] = rict[k * A];
        fz[c] = fzt[k * A];
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int k = k0 - c;
        if (k < 0) break;
        const double wp3 = f.rh_of(k, pd0[c], pd1);
        pd1 = pd0[c];
        double v = kBackTidal + kMixingEf * kLocalFrac * wd * fz[c] / (fmax(rc[c], 1.0e-8) * (wp3 * 1000.0));
        if (v > kMaxTidal) v = kMaxTidal;
        if (k <= n - 2) v = fmin(v, below);
        below = v;
        a.ak_tide[k * A + q] = v;
        a.richardson[k * A + q] = rc[c];
        a.fztidal[k * A + q] = fz[c];
        a.wp3_tidal[k * A + q] = wp3;
      }
    }
  }

  // ---- 2. mixed-layer depth (formld, readyc.cpp:902-913)
  double amld;
  if (n > 0) {
    amld = f.z(n - 1);
    const double t0 = f.t(0);
    double tp = t0, zp = f.z(0);
    for (int k = 1; k < n; ++k) {
      const double tk = f.t(k), zk = f.z(k);
      if (fabs(tk - t0) > 0.1) {
        const double tm = t0 - sgn(0.1e0, t0 - tk);
        amld = zk + (zp - zk) * (tm - tk) / (tp - tk + 1.0e-20);
        break;
      }
      tp = tk;
      zp = zk;
    }
  } else {
    amld = 0.0;   // z[0] of an empty column (the work array is zeroed)
  }
  a.amld[q] = amld * 1.0e-2;

  // ---- 3. the closure, level by level (turb_device, readyc.cpp:1116-1454)
  const double coriol = a.fcort[q];
  const double buoytot = a.buoytur[q] * 1.0e+4 + a.buoysol[q] * 1.0e+4;
  const double b1 = T.b1;
  const double al0 = 0.17 * amld;
  double ifbelow = 0.0;
  double an = 0.0;                     // unset in the reference until N^2 >= 0 is met
  Stab st{0.0, 0.0, 0.0, 0.0}, back{0.0, 0.0, 0.0, 0.0};
  double amtaun2 = 0.0;
  double back_ri1 = 0.0, tmp = 0.0;
  double km0 = 0.0, kh0 = 0.0, ks0 = 0.0;   // level 0, written last
  double* akt_t = a.precision == LT_PREC_MIXED ? nullptr : a.akt + q;
  float* akt_t32 = a.precision == LT_PREC_MIXED ? a.akt32 + q : nullptr;
  const long F = a.F;
  auto put = [&](int k, double akm, double akh, double aks) {
    const double tide = a.ak_tide[k * A + q];
    a.akmt[k * A + q] = akm * 1.0e-4 + tide * 5.0;
    const double t_ = quotient(akh * 1.0e-4 + tide, ncc_f, C.inv_ncc);
    const double s_ = quotient(aks * 1.0e-4 + tide, ncc_f, C.inv_ncc);
    if (akt_t) {
      akt_t[k * A] = t_;
      akt_t[F + k * A] = s_;
    } else {
      akt_t32[k * A] = (float)t_;
      akt_t32[F + k * A] = (float)s_;
    }
  };
  // rolling window of interface depths and densities: k-2 .. k+1
  double z_m1 = 0.0, z_0 = n > 0 ? f.z(0) : 0.0, z_p1 = n > 1 ? f.z(1) : 0.0;
  double rh_m2 = 0.0, rh_m1 = 0.0, rh_0 = n > 0 ? f.rh(0) : 0.0, rh_p1 = n > 1 ? f.rh(1) : 0.0;
  int done = 0;   // levels whose diffusivities the closure set
  bool quit = false;
  // the level's inputs are loaded a level ahead
  const double* __restrict__ rit_ = a.rit + q;
  const double* __restrict__ rid_ = a.ricdttms + q;
  const double* __restrict__ s2t_ = a.s2t + q;
  double in_an2 = 0.0, in_ri = 0.0, in_rid = 0.0, in_s2 = 0.0;
  auto fetch = [&](int k) {
    if (k < n) {
      in_an2 = rict[k * A];
      in_ri = rit_[k * A];
      in_rid = rid_[k * A];
      in_s2 = s2t_[k * A];
    }
  };
  fetch(0);
  for (int k = 0; k < n; ++k) {
    const double an2 = in_an2, rik = in_ri, ridk = in_rid;
    double s2 = in_s2;
    fetch(k + 1);
    double ifnofsmall = 0.0;
    if (an2 >= 0.0e0) an = sqrt(an2);
    if (an < fabs(coriol)) ifnofsmall = 1.0;
    double ri1 = rik, rid1 = ridk;
    const int ifpureshear = (an2 < T.rib0 * s2) ? 1 : 0;
    if (ifpureshear == 1) {
      const double and2 = ridk / (rik + 1.0e-25) * an2;
      const double and2on2 = and2 / (an2 + 1.0e-25);
      double v[4];
      if (interp1d(and2on2, T, C, v)) {
        amtaun2 = v[0];
        st.sm = v[1];
        st.sh = v[2];
        st.ss = v[3];
      }
      st.slq2 = (-amtaun2) / ((b1 * b1) * rik + 1.0e-25);
    } else {
      interp2d<PLAIN>(ri1, rid1, T, C, st);
      if (st.slq2 < 0.0e0) { quit = true; break; }
      if (st.slq2 == 0.0e0) ifbelow = 1.0;
    }
    const bool lifupper = ((ifbelow == 0.0 || ifnofsmall == 1.0 || ((ri1 < 0.0e0) && (k <= 1))) && (st.slq2 > 0.0e0));
    double epsy = 0.0e0;
    if (lifupper) epsy = -buoytot / ((1.0e0 / ((b1 * b1) * (st.slq2))) - 0.5e0 * st.sm);
    const bool lifepsy = ((epsy >= 0.0e0) && lifupper);
    const double akz = 0.4 * z_0;
    const double al = akz * al0 / (al0 + akz);
    double al2 = al * al;
    if (ifbelow != 1.0 && !lifepsy) {
      if (ri1 > 0.0e0) {
        const double anlq2 = st.slq2 * ri1;
        if (anlq2 > 0.281e0) {
          al2 *= 0.281e0 / anlq2;
          st.slq2 = 0.281e0 / (ri1 + 1.0e-20);
        }
      }
    }
    // the latitude factor enters through the background (Ri > 0) and, below
    // the mixed part, for Ri >= 0 only
    double epson2 = kEpson2;
    if (!(an2 < 0.0e0) && (!(rik <= 0.0e0) || ri1 >= 0.0e0)) {
      double ep = ifnofsmall == 1.0 ? 0.0e0 : eplat(C, fabs(coriol), an);
      ep = fmax(ep, kEplatMin);
      epson2 = kEpson2 * ep;
    }
    if (rik > 0.0e0) {
      const double rit = (rik + ridk) / 2.0e0;
      const double ric = (rik - ridk) / 2.0e0;
      const double ra_r = sqrt((rit * rit) + (ric * ric));
      double theta_r;
      if (fabs(rit) <= 0.0e0) theta_r = (fabs(ric) <= 0.0e0) ? C.pi4 : 2.0e0 * C.pi4;
      else theta_r = atan(ric / rit);
      if (fabs(theta_r) > 2.0e0 * C.pi4) { quit = true; break; }
      // cos and sin of the angle from its own components: it points along
      // (rit, ric), or against it where rit < 0, and is turned by pi below
      // -pi/4.  Not where the squares in ra_r overflow or lose their bits
      // below the smallest normal number, nor where Ri is small beside Ri_d:
      // there cos + sin is mostly the angle's rounding, which decides whether
      // the column goes on.
      double turn = rit < 0.0e0 ? -1.0 : 1.0;
      if (theta_r < -C.pi4) {
        theta_r += 4.0e0 * C.pi4;
        turn = -turn;
      }
      bool moved = fabs(rit) <= 0.0e0 || !(ra_r > 1.0e-130 && ra_r < 1.0e150 && rik > 1.0e-3 * ra_r);
      const int jt0 = (int)ratio<PLAIN>(theta_r + C.pi4, T.deltheta_r, C.inv_dth);
      int it0 = jt0 - NTH, it1 = it0 + 1;
      double th0 = it0 * T.deltheta_r, th1 = it1 * T.deltheta_r;
      if ((th0 <= T.theta_rcrp) && (theta_r > T.theta_rcrp)) {
        theta_r = th1;
        th0 = th1;
        it0 = it1;
        ++it1;
        th1 += T.deltheta_r;
        moved = true;
      } else if ((th1 >= T.theta_rcrn) && (theta_r < T.theta_rcrn)) {
        theta_r = th0;
        th1 = th0;
        it1 = it0;
        --it0;
        th0 += -T.deltheta_r;
        moved = true;
      }
      if ((it1 > 3 * NTH) || (it0 < -NTH)) { quit = true; break; }
      double dth = theta_r - th0;
      double back_ra_r1 = angle(T, 0, it0, dth);
      int ifrafglt = 0;
      if ((theta_r <= T.theta_rcrp) || (theta_r >= T.theta_rcrn)) {
        if (back_ra_r1 > ra_r) {
          ifrafglt = 1;
          back_ra_r1 = ra_r;
        }
      }
      if (back_ra_r1 < 0.0e0) { quit = true; break; }
      // where the second look-up takes them, from the angle too: small Ri are
      // their own components, and one that meets a table entry would go to a
      // side of it that the angle's rounding decides
      double back_rit1, back_ric1;
      if (moved || ifrafglt == 1) {
        back_rit1 = cos(theta_r) * back_ra_r1;
        back_ric1 = sin(theta_r) * back_ra_r1;
      } else {
        const double scale = turn * back_ra_r1 / ra_r;
        back_rit1 = rit * scale;
        back_ric1 = ric * scale;
      }
      back_ri1 = back_rit1 + back_ric1;
      if (ifrafglt == 1) {
        double back_rid1 = back_rit1 - back_ric1, bri = back_ri1;
        Stab b = back;
        interp2d_back<PLAIN>(bri, back_rid1, T, C, b);
        back_ri1 = bri;
        back = b;
      } else {
        dth = theta_r - it0 * T.deltheta_r;
        back.sm = angle(T, 1, it0, dth);
        back.sh = angle(T, 2, it0, dth);
        back.ss = angle(T, 3, it0, dth);
        back.slq2 = angle(T, 4, it0, dth);
      }
      if (back.slq2 < 0.0e0) { quit = true; break; }
    }
    if (rik <= 0.0e0) back_ri1 = 0.0e0;
    if (ri1 <= 0.0e0) {
      back.sm = 0.0e0;
      back.sh = 0.0e0;
      back.ss = 0.0e0;
    }
    if ((back.sm < 0.0e0) || (back.sh < 0.0e0) || (back.ss < 0.0e0)) { quit = true; break; }
    const double tmp_back = 0.5e0 * b1 * b1 * back_ri1 * back.slq2 * epson2;
    const double v_back = tmp_back * back.sm, t_back = tmp_back * back.sh, s_back = tmp_back * back.ss;
    if ((v_back < 0.0e0) || (t_back < 0.0e0) || (s_back < 0.0e0)) { quit = true; break; }
    if ((rik > 0.0e0) && ((fabs(v_back) <= 0.0e0) || (fabs(t_back) <= 0.0e0) || (fabs(s_back) < 0.0e0))) {
      quit = true;
      break;
    }
    // the mixing scale: the closure's own where the level is not below the
    // mixed part, or is unstable there
    bool shear_scale = ifpureshear != 1;
    if (ifbelow == 1.0) {
      if (ri1 >= 0.0e0) {
        tmp = 0.5e0 * b1 * b1 * ri1 * st.slq2 * epson2;
        shear_scale = false;
      } else if (k >= 2) {
        double delz, delrh, del2rh;
        if (k == n - 1) {
          delz = z_0 - z_m1;
          delrh = rh_0 - rh_m1;
          del2rh = rh_0 - 2.0e0 * rh_m1 + rh_m2;
        } else {
          delz = z_p1 - z_m1;
          delrh = rh_p1 - rh_m1;
          del2rh = rh_p1 - 2.0e0 * rh_0 + rh_m1;
        }
        const double dzrh = delrh / delz;
        const double d2zrh = 4.0e0 * del2rh / (delz * delz);
        const double rdzlndzrh = dzrh / d2zrh;
        const double al0deep = 0.17e0 * fabs(rdzlndzrh);
        const double akz2 = 0.4e0 * z_0;
        const double aldeep = akz2 * al0deep / (al0deep + akz2);
        al2 = aldeep * aldeep;
      }
    }
    if (shear_scale) {
      s2 = fmax(s2, kS2min);
      if (lifepsy && !(ifbelow == 1.0 && k >= 2)) tmp = 0.5e0 * epsy / (s2 + 1.0e-40);
      else tmp = 0.5e0 * b1 * al2 * sqrt(s2 / (st.slq2 + 1.0e-40));
    }
    if (ifpureshear == 1) tmp = 0.5e0 * (b1 * b1) * al2 * sqrt(-an2 / amtaun2);
    const double akm = fmin(tmp * st.sm + v_back, fricmx);
    const double akh = fmin(tmp * st.sh + t_back, fricmx);
    const double aks = fmin(tmp * st.ss + s_back, fricmx);
    if (k == 0) {
      km0 = akm;
      kh0 = akh;
      ks0 = aks;
    } else {
      put(k, akm, akh, aks);
    }
    done = k + 1;
    // slide the window
    z_m1 = z_0;
    z_0 = z_p1;
    z_p1 = (k + 2 < n) ? f.z(k + 2) : 0.0;
    rh_m2 = rh_m1;
    rh_m1 = rh_0;
    rh_0 = rh_p1;
    rh_p1 = (k + 2 < n) ? f.rh(k + 2) : 0.0;
  }
  // the reference returns early on an inconsistent table value: the levels
  // from there on keep their zeroed work arrays and the surface floor is skipped
  if (!quit && n > 0) {
    if (km0 < wndmix) km0 = wndmix;
    if (kh0 < wndmix) kh0 = wndmix;
    if (ks0 < wndmix) ks0 = wndmix;
  }
  put(0, km0, kh0, ks0);
  for (int k = done > 1 ? done : 1; k < n; ++k) put(k, 0.0, 0.0, 0.0);
  for (int k = n > 1 ? n : 1; k < km - 1; ++k) {   // below the column: no tide either
    a.akmt[k * A + q] = 0.0;
    if (akt_t) akt_t[k * A] = akt_t[F + k * A] = 0.0;
    else akt_t32[k * A] = akt_t32[F + k * A] = 0.0f;
  }
  a.akmt[(long)(km - 1) * A + q] = 0.0;
}

// zero, or a magnitude ratio's quick form may divide
__host__ __device__ inline bool plain_entry(double x) {
  const double v = fabs(x);
  return v == 0.0 || (v > 1.0e-100 && v < 1.0e100);
}

// one table into its place among the interleaved four; odd: set where an
// entry is not plain_entry
__global__ void k_interleave(const double* __restrict__ x, double* __restrict__ quad, long n, int* odd) {
  bool plain = true;
  for (long m = (long)blockIdx.x * blockDim.x + threadIdx.x; m < n; m += (long)gridDim.x * blockDim.x) {
    quad[4 * m] = x[m];
    plain = plain && plain_entry(x[m]);
  }
  if (!plain) *odd = 1;
}

}  // namespace

int launch_turb(const Arena& a, const TurbTabDev& T, int ncc, double dfricmx, cudaStream_t s) {
  TurbConst C;
  C.pi4 = std::atan(1.0);
  const double an0 = 5.24e-3, f30 = 4.0 * C.pi4 / 43082.0;
  C.eplat_den = f30 * std::acosh(an0 / f30);
  C.inv_ncc = quotient_reciprocal((double)(float)ncc);
  C.inv_dth = 1.0 / T.deltheta_r;
  C.inv_dri = 1.0 / T.dri;
  C.inv_da = 1.0 / T.dand2on2;
  C.log2_gm = (float)std::log2(T.gm);
  C.per_log2 = (float)(1.0 / std::log2(T.rri));
  C.log2_gm1 = (float)std::log2(T.gm1);
  C.per_log21 = (float)(1.0 / std::log2(T.rnd2on2));
  // warps of 8 x 4 columns: depths and stability alike, so fewer idle lanes
  // (720 x 460 x 55 deep: rows of 32 were 11 % slower)
  dim3 b(8, 16), g((a.imt + 7) / 8, (a.jmt + 15) / 16);
  (T.plain ? k_turb<true> : k_turb<false>)<<<g, b, 0, s>>>(a, T, C, (double)(float)ncc, dfricmx * 1.0e+4,
                                                           a.p.dwndmix * 1.0e+4);
  LT_LAUNCHED();
  return LT_OK;
}

}  // namespace lt

using namespace lt;

extern "C" {

int lt_turb_tables_create(const lt_turb_tables* h, lt_turb_tab** out) {
  if (!h || !out || !h->rib || !h->irimax || !h->slq2b || !h->smb || !h->shb || !h->ssb || !h->and2on2a1 ||
      !h->amtaun2a1 || !h->sma1 || !h->sha1 || !h->ssa1 || !h->back_ra_r || !h->sm_r1 || !h->sh_r1 || !h->ss_r1 ||
      !h->slq2_r1) {
    set_error("lt_turb_tables_create: a table pointer is missing");
    return LT_E_INVALID;
  }
  if (!(h->dri > 0.0) || !(h->rri > 1.0) || !(h->dand2on2 > 0.0) || !(h->rnd2on2 > 1.0) || !(h->deltheta_r > 0.0)) {
    set_error("lt_turb_tables_create: grid steps must be positive and ratios above 1");
    return LT_E_INVALID;
  }
  for (int m = 0; m < N1; ++m)
    if (h->irimax[m] < -MT || h->irimax[m] > MT) {
      set_error("lt_turb_tables_create: irimax[%d] = %d outside -%d..%d", m, h->irimax[m], MT, MT);
      return LT_E_INVALID;
    }
  const size_t n1 = N1, n2 = (size_t)N1 * N1, nb = LT_TURB_NB;
  struct Item { const void* src; size_t bytes; const void** dst; };
  lt_turb_tab* t = new (std::nothrow) lt_turb_tab;
  if (!t) return LT_E_OOM;
  TurbTabDev& T = t->t;
  const int* odd = nullptr;        // set while the 2-D tables are interleaved
  std::vector<double> rilim(n1);   // the realizable limit of Ri itself
  for (int m = 0; m < N1; ++m) rilim[m] = h->rib[MT + h->irimax[m]];
  std::vector<double> rstep(n1, 0.0);
  for (size_t m = 0; m + 1 < n1; ++m) rstep[m] = 1.0 / (h->rib[m + 1] - h->rib[m]);
  std::vector<double2> angle(5 * nb);
  const double* angles[] = {h->back_ra_r, h->sm_r1, h->sh_r1, h->ss_r1, h->slq2_r1};
  for (size_t t = 0; t < 5; ++t)
    for (size_t m = 0; m < nb; ++m)
      angle[t * nb + m] = {angles[t][m], m + 1 < nb ? (angles[t][m + 1] - angles[t][m]) / h->deltheta_r : 0.0};
  const Item items[] = {
      {nullptr, 4 * n2 * 8, (const void**)&T.quad}, {nullptr, sizeof(int), (const void**)&odd},
      {h->rib, n1 * 8, (const void**)&T.rib},         {rstep.data(), n1 * 8, (const void**)&T.rstep},
      {rilim.data(), n1 * 8, (const void**)&T.rilim},
      {h->and2on2a1, n1 * 8, (const void**)&T.and2on2a1}, {h->amtaun2a1, n1 * 8, (const void**)&T.amtaun2a1},
      {h->sma1, n1 * 8, (const void**)&T.sma1},       {h->sha1, n1 * 8, (const void**)&T.sha1},
      {h->ssa1, n1 * 8, (const void**)&T.ssa1},       {angle.data(), 5 * nb * 16, (const void**)&T.angle}};
  size_t total = 0;
  for (const Item& it : items) total += (it.bytes + 255) / 256 * 256;
  char* base = nullptr;
  double* one = nullptr;   // one 2-D table on its way into the interleaved four
  cudaError_t e = cudaMalloc(&base, total);
  if (e == cudaSuccess && (e = cudaMalloc(&one, n2 * 8)) != cudaSuccess) cudaFree(base);
  if (e != cudaSuccess) {
    delete t;
    set_error("lt_turb_tables_create: cudaMalloc(%zu) failed: %s", total + n2 * 8, cudaGetErrorString(e));
    return LT_E_OOM;
  }
  size_t off = 0;
  for (const Item& it : items) {
    *it.dst = base + off;
    if (it.src && e == cudaSuccess) e = cudaMemcpy(base + off, it.src, it.bytes, cudaMemcpyHostToDevice);
    off += (it.bytes + 255) / 256 * 256;
  }
  if (e == cudaSuccess) e = cudaMemset(const_cast<int*>(odd), 0, sizeof(int));
  const double* tabs[4] = {h->slq2b, h->smb, h->shb, h->ssb};
  for (int m = 0; m < 4 && e == cudaSuccess; ++m) {
    e = cudaMemcpy(one, tabs[m], n2 * 8, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) break;
    k_interleave<<<1184, 256>>>(one, const_cast<double*>(T.quad) + m, (long)n2, const_cast<int*>(odd));
    lt::count_launches(1);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
  }
  cudaFree(one);
  int any_odd = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&any_odd, odd, sizeof(int), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    cudaFree(base);
    delete t;
    return cuda_fail(e, "lt_turb_tables_create");
  }
  bool plain = !any_odd && plain_entry(h->deltheta_r);
  for (size_t m = 0; m < n1 && plain; ++m)
    plain = plain_entry(h->rib[m]) && (m == 0 || (h->rib[m] != h->rib[m - 1] && plain_entry(h->rib[m] - h->rib[m - 1])));
  T.plain = plain ? 1 : 0;
  T.rib0 = h->rib[0];
  T.gm = h->rib[MT + MT0];
  T.gmax = h->rib[2 * MT];
  T.gm1 = h->and2on2a1[MT + MT0];
  T.rri = h->rri;
  T.rnd2on2 = h->rnd2on2;
  T.dri = h->dri;
  T.deltheta_r = h->deltheta_r;
  T.b1 = h->b1;
  T.theta_rcrp = h->theta_rcrp;
  T.theta_rcrn = h->theta_rcrn;
  T.dand2on2 = h->dand2on2;
  t->base = base;
  cudaGetDevice(&t->dev);
  *out = t;
  return LT_OK;
}

int lt_turb_tables_destroy(lt_turb_tab* t) {
  if (!t) return LT_E_INVALID;
  cudaFree(t->base);
  delete t;
  return LT_OK;
}

int lt_turb(lt_domain* d, const lt_turb_tab* t, const lt_turb_params* p) {
  if (!d || !t || !p || p->ncc < 1) {
    set_error("lt_turb: invalid arguments");
    return LT_E_INVALID;
  }
  int rc = ensure_turb(d);
  if (rc) return rc;
  return launch_turb(d->a, t->t, p->ncc, p->dfricmx, d->stream);
}

}  // extern "C"
