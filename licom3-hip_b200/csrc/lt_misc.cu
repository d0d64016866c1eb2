// lt_misc.cu - convective adjustment, sea-ice adjustment, mask derivation,
// global sums, numeric scan and the device side of the synthetic-domain
// upload.  Compiled with -fmad=false (operation order kept as written).
#include <cstring>
#include <vector>
#include "lt_common.cuh"
#include "lt_halo.cuh"
#include "lt_tracer_tma.cuh"
#include "lt_synth.h"
#include "../../include/licom_synth.h"

const lt::Domain* lt_synth_domain(const lt_synth* s);

namespace lt {
namespace {

// The convadj coefficients of every level in shared memory: cc [9][km], to, so
// [km], dzp [km].
struct ConvTab {
  const double *cc, *to, *so, *dz;
  int km;
  // density departure of the convadj polynomial at coefficient level l
  // (convadj.cpp:57-77) of water (t, s)
  __device__ double rho(double t_, double s_, int l) const {
    const double t = t_ - to[l], s = s_ - so[l];
    return (cc[l] + (cc[3 * km + l] + cc[6 * km + l] * s) * s +
            (cc[2 * km + l] + cc[7 * km + l] * s + cc[5 * km + l] * t) * t) * t +
           (cc[1 * km + l] + (cc[4 * km + l] + cc[8 * km + l] * s) * s) * s;
  }
};

// convadj_cu (convadj.cpp:29-288) without its last step: one thread per
// column; finds the shallowest statically unstable interface, mixes T and S
// thickness-weighted over the unstable stretch and grows it up and down while
// unstable, then continues below.
//
// The reference keeps every interface's two densities in arrays; each is a
// function of one level's water that is still unmixed when it is used, so
// here they are formed where they are needed (the same bits) and a column
// holds two levels in registers instead of 2 x km doubles in local memory,
// whose traffic was more than the fields' own.  The search loads four levels
// ahead of their use.  The step over every cell that follows is a kernel of
// its own, level by level (k_convadj_tend).  720 x 460 x 55 deep: 164 us and
// 256 us (6.9 TB/s) against 904 us as one kernel with the arrays.
constexpr int kConvAhead = 4;
constexpr int kConvLevels = 128;   // most levels taken
__global__ void __launch_bounds__(kColX * kColY) k_convadj(const __grid_constant__ Arena a, int row0) {
  extern __shared__ double s_conv[];
  const int km = a.km;
  for (int m = threadIdx.x; m < 12 * km; m += kColX * kColY)
    s_conv[m] = m < 9 * km ? a.cc[m] : m < 10 * km ? a.to[m - 9 * km] : m < 11 * km ? a.so[m - 10 * km] : a.dzp[m - 11 * km];
  __syncthreads();
  const ConvTab C{s_conv, s_conv + 9 * km, s_conv + 10 * km, s_conv + 11 * km, km};
  const int i = blockIdx.x * kColX + threadIdx.x % kColX;
  const int j = (row0 + blockIdx.y) * kColY + threadIdx.x / kColX;
  if (i >= a.imt || j >= a.jmt) return;
  const long A = a.A, F = a.F;
  const long q = (long)j * a.imt + i;
  double* __restrict__ at = a.at[a.cur] + q;
  const double* dzp = C.dz;
  auto T = [&](int l) -> double& { return at[(long)l * A]; };
  auto S = [&](int l) -> double& { return at[F + (long)l * A]; };
  // densities across the interface below level l at the coefficients of level l+1
  auto lower = [&](int l) { return C.rho(T(l), S(l), l + 1); };
  auto upper = [&](int l) { return C.rho(T(l), S(l), l); };
  const int kcon = a.kmt[q];
  int lcon = 0;   // 1-based: the level above the shallowest unstable interface
  if (kcon > 1) {
    double t0 = T(0), s0 = S(0);
    for (int l0 = 0; l0 < kcon - 1 && lcon == 0; l0 += kConvAhead) {
      double t[kConvAhead], s[kConvAhead];
#pragma unroll
      for (int c = 0; c < kConvAhead; ++c) {
        const int l = min(l0 + c + 1, kcon - 1);
        t[c] = T(l);
        s[c] = S(l);
      }
#pragma unroll
      for (int c = 0; c < kConvAhead; ++c) {
        const int l = l0 + c;
        if (l < kcon - 1) {
          if (lcon == 0 && C.rho(t0, s0, l + 1) > C.rho(t[c], s[c], l + 1)) lcon = l + 1;
          t0 = t[c];
          s0 = s[c];
        }
      }
    }
  }
  if (lcon != 0) {
    for (;;) {
      int lcona = lcon, lconb = lcon + 1;
      double dztsum = dzp[lcona - 1] + dzp[lconb - 1];
      double trasum[2];
      for (int n = 0; n < 2; ++n) {
        double* X = at + n * F;
        trasum[n] = X[(long)(lcona - 1) * A] * dzp[lcona - 1] + X[(long)(lconb - 1) * A] * dzp[lconb - 1];
        const double tramix = trasum[n] / dztsum;
        X[(long)(lcona - 1) * A] = tramix;
        X[(long)(lconb - 1) * A] = tramix;
      }
      for (;;) {
        if (lconb != kcon) {
          if (lower(lconb - 1) > upper(lconb)) {
            lconb = lconb + 1;
            dztsum = dztsum + dzp[lconb - 1];
            for (int n = 0; n < 2; ++n) {
              double* X = at + n * F;
              trasum[n] = trasum[n] + X[(long)(lconb - 1) * A] * dzp[lconb - 1];
              const double tramix = trasum[n] / dztsum;
              for (int lm = lcona - 1; lm < lconb; ++lm) X[(long)lm * A] = tramix;
            }
            continue;
          }
        }
        if (lcona > 1) {
          if (lower(lcona - 2) > upper(lcona - 1)) {
            lcona = lcona - 1;
            dztsum = dztsum + dzp[lcona - 1];
            for (int n = 0; n < 2; ++n) {
              double* X = at + n * F;
              trasum[n] = trasum[n] + X[(long)(lcona - 1) * A] * dzp[lcona - 1];
              const double tramix = trasum[n] / dztsum;
              for (int lm = lcona; lm <= lconb; ++lm) X[(long)(lm - 1) * A] = tramix;
            }
            continue;
          }
        }
        break;
      }
      if (lconb == kcon) break;
      lcon = lconb;
      bool done = false;
      for (;;) {
        lcon = lcon + 1;
        if (lcon == kcon) { done = true; break; }
        if (lower(lcon - 1) <= upper(lcon)) continue;
        break;
      }
      if (done) break;
    }
  }
}

// The tendency diagnostics and atb = at of every cell (convadj.cpp:258-276),
// level by level (blockIdx.z: tracer and level): 48 B per cell and tracer.
__global__ void __launch_bounds__(256) k_convadj_tend(const __grid_constant__ Arena a, double dts, double inv_dts) {
  const long A = a.A;
  const int k = blockIdx.y, n = blockIdx.z;
  const double* __restrict__ at = a.at[a.cur] + n * a.F + k * A;
  double* __restrict__ atb = a.atb[a.cur] + n * a.FB + (k + 1) * A;
  double* __restrict__ tend = a.tend + n * a.F + k * A;
  double* __restrict__ conv = a.dt_conv + n * a.F + k * A;
  const long q0 = (long)blockIdx.x * (4 * 256) + threadIdx.x;
  double x[4], b[4], d[4];
  int kz[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const long q = q0 + c * 256;
    if (q < A) {
      x[c] = at[q];
      b[c] = atb[q];
      d[c] = tend[q];
      kz[c] = a.kmt[q];
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const long q = q0 + c * 256;
    if (q < A) {
      const double dt = quotient(x[c] - b[c], dts, inv_dts) * (k < kz[c] ? 1.0 : 0.0);
      __stcs(conv + q, dt);
      tend[q] = d[c] + dt;
      atb[q] = x[c];
    }
  }
}

// ---------------------------------------------------------------- icesnow
// icesnow_cu (icesnow.cpp:15-68): one thread per point of the domain, halo
// included, i fastest across a warp.  Surface freezing of ocean columns into
// QICE with the brine term on S, melting of QICE where the surface is above
// the freezing point, then T raised to tbice at every level (land included).
// Operation order is the reference's, so the results are bit-identical; the
// FRC_CORE reset of QICE is folded in (0 + x == x exactly).  HBM-bound: T is
// read at every level and written only where it changes.
__global__ void k_icesnow(Arena a, double tbice, double cp, double latice, int reset) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= a.imt || j >= a.jmt) return;
  const long q = (long)j * a.imt + i;
  const long A = a.A;
  double* T = a.at[a.cur] + q;
  double* S = T + a.F;
  const double sal_ocn = 34.7e0, sal_ice = 4.0e0;
  double qi = reset ? 0.0 : a.qice[q];
  double t0 = T[0];
  if (t0 < tbice && a.kmt[q] > 0) {
    const double tdiff = tbice - t0;
    qi += tdiff * a.dzp[0] / a.dzp[0];
    S[0] += tdiff * (sal_ocn - sal_ice) * cp / latice * 0.001e0;
    t0 = tbice;
    T[0] = t0;
  }
  if (qi > 0.0 && t0 > tbice) {
    const double tdiff = fmin(t0 - tbice, qi);
    qi -= tdiff;
    t0 -= tdiff;
    T[0] = t0;
    S[0] -= tdiff * (sal_ocn - sal_ice) * cp / latice * 0.001e0;
  }
  if (t0 < tbice) T[0] = tbice;
  a.qice[q] = qi;
  // the levels below in groups of 8: all loads of a group issued before any
  // store, so that a warp keeps 8 rows in flight
  for (int k0 = 1; k0 < a.km; k0 += 8) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = (k0 + u < a.km) ? T[(k0 + u) * A] : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (k0 + u < a.km && v[u] < tbice) T[(k0 + u) * A] = tbice;
  }
}

// ---------------------------------------------------------------- masks
// boundary.F90:24-52, grid.F90:1343-1346, grid.F90:2030-2051
__global__ void k_masks(Arena a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int imt = a.imt, jmt = a.jmt;
  if (i >= imt || j >= jmt) return;
  const long q = (long)j * imt + i;
  const int* kmt = a.kmt;
  int ku = 0;
  if (j < jmt - 1 && i >= 1) ku = min(min(kmt[q - 1], kmt[q]), min(kmt[q + imt - 1], kmt[q + imt]));
  a.kmu[q] = ku;
  a.kmtn[q] = j > 0 ? kmt[q - imt] : 0;
  a.kmts[q] = j < jmt - 1 ? kmt[q + imt] : 0;
  a.kmte[q] = i < imt - 1 ? kmt[q + 1] : 0;
  a.kmtw[q] = i > 0 ? kmt[q - 1] : 0;
}

// KMU ghost fill, SW-corner location (no averaging, top physical row kept)
__global__ void k_kmu_halo(Arena a) {
  const int imt = a.imt, jmt = a.jmt, nx = imt - 4;
  int* f = a.kmu;
  // ghost rows from the fold first read only physical rows 2,3; E-W copies
  // touch only ghost columns of physical rows - disjoint, so one pass is safe
  for (long m = threadIdx.x; m < (long)imt * jmt; m += blockDim.x) {
    const int j = (int)(m / imt), i = (int)(m % imt);
    if (j >= 2 && j < jmt - 2 && a.ew_cyclic) {
      if (i < 2) f[m] = f[(long)j * imt + nx + i];
      else if (i >= imt - 2) f[m] = f[(long)j * imt + i - nx];
    }
  }
  __syncthreads();
  if (!a.tripole) return;
  for (int i = threadIdx.x; i < imt; i += blockDim.x) {
    int g = halo_iglobal(i, nx, a.ew_cyclic);
    int isrc = nx - g + 1;
    if (isrc == 0) isrc = nx;
    if (isrc > nx) isrc = isrc - nx;  // g == 0 on a closed side maps to nx+1; keep it in range
    f[i] = f[3L * imt + isrc + 1];          // row 0 <- physical row 3
    f[imt + i] = f[2L * imt + isrc + 1];    // row 1 <- physical row 2
  }
}

__global__ void k_inv_depth(Arena a) {
  const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= a.A) return;
  double s = 0.0;
  for (int k = 0; k < a.km; ++k) s = s + (k < a.kmt[q] ? 1.0 : 0.0) * a.dzp[k];
  a.ohbt[q] = s > 0.0 ? 1.0 / s : 0.0;
  s = 0.0;
  for (int k = 0; k < a.km; ++k) s = s + (k < a.kmu[q] ? 1.0 : 0.0) * a.dzp[k];
  a.ohbu[q] = s > 0.0 ? 1.0 / s : 0.0;
  if (q < a.km) a.odzp[q] = 1.0 / a.dzp[q];
}

// ------------------------------------------------------------- reductions
constexpr int RB2 = 1024;
__global__ void k_content_first(const double* at, const double* tarea, const double* dzp, const int* kmt,
                                 int nx, int ny, int imt, long A, long n, double* part) {
  __shared__ double s[2 * RB2];
  const long base = (long)blockIdx.x * 2 * RB2;
  auto term = [&](long m) -> double {
    if (m >= n) return 0.0;
    const long per = (long)nx * ny;
    const int k = (int)(m / per);
    const long r = m % per;
    const int j = 2 + (int)(r / nx), i = 2 + (int)(r % nx);
    const long q = (long)j * imt + i;
    return (k < kmt[q]) ? tarea[q] * dzp[k] * at[(long)k * A + q] : 0.0;
  };
  const int t = threadIdx.x;
  s[t] = term(base + t);
  s[t + RB2] = term(base + t + RB2);
  for (int stride = RB2; stride > 0; stride >>= 1) {
    __syncthreads();
    if (t < stride) s[t] = s[t] + s[t + stride];
  }
  if (t == 0) part[blockIdx.x] = s[0];
}

__global__ void k_count_bad(const double* x, long n, int* count) {
  long m = (long)blockIdx.x * blockDim.x + threadIdx.x;
  int bad = 0;
  for (; m < n; m += (long)gridDim.x * blockDim.x) bad += !isfinite(x[m]);
  if (bad) atomicAdd(count, bad);
}

// ------------------------------------------------------- synthetic upload
__global__ void k_synth_state(CellTables t, double* at, double* atb, double* restore) {
  const long m = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long A = (long)t.imt * t.jmt, F = A * t.km;
  if (m >= F) return;
  const int k = (int)(m / A);
  const long r = m % A;
  const int j = (int)(r / t.imt), i = (int)(r % t.imt);
  const double T = cell_T(t, k, j, i), S = cell_S(t, k, j, i);
  at[m] = T;
  at[F + m] = S;
  if (restore) { restore[m] = T; restore[F + m] = S; }
  (void)atb;
}

__global__ void k_synth_vel(CellTables t, double ncc1, double* utf, double* vtf, double* utl, double* vtl,
                            double* akt) {
  const long m = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long A = (long)t.imt * t.jmt, F = A * t.km;
  if (m >= F) return;
  const int k = (int)(m / A);
  const long r = m % A;
  const int j = (int)(r / t.imt), i = (int)(r % t.imt);
  const double u = cell_U(t, k, j, i), v = cell_V(t, k, j, i);
  utl[m] = u; vtl[m] = v;
  utf[m] = ncc1 * u; vtf[m] = ncc1 * v;
  akt[m] = cell_akt(t, 0, k, j, i);
  akt[F + m] = cell_akt(t, 1, k, j, i);
}

}  // namespace

int launch_convadj(const Arena& a, cudaStream_t s) {
  if (a.km > kConvLevels) { set_error("convadj: km > %d", kConvLevels); return LT_E_INVALID; }
  if (int rc = for_column_rows(a, [&](int r, int rows) {
        k_convadj<<<dim3((a.imt + kColX - 1) / kColX, rows), kColX * kColY, 12 * a.km * sizeof(double), s>>>(a, r);
        LT_LAUNCHED();
        return (int)LT_OK;
      }))
    return rc;
  k_convadj_tend<<<dim3((unsigned)((a.A + 1023) / 1024), a.km, 2), 256, 0, s>>>(a, a.p.dts, quotient_reciprocal(a.p.dts));
  LT_LAUNCHED();
  return LT_OK;
}

int launch_icesnow(const Arena& a, const lt_icesnow_params& p, cudaStream_t s) {
  dim3 b(32, 8), g((a.imt + 31) / 32, (a.jmt + 7) / 8);
  k_icesnow<<<g, b, 0, s>>>(a, p.tbice, p.cp, p.latice, p.reset_qice != 0);
  LT_LAUNCHED();
  return LT_OK;
}

int launch_derive_masks(const Arena& a, cudaStream_t s) {
  dim3 b(32, 8), g((a.imt + 31) / 32, (a.jmt + 7) / 8);
  k_masks<<<g, b, 0, s>>>(a);
  LT_LAUNCHED();
  k_kmu_halo<<<1, 1024, 0, s>>>(a);
  LT_LAUNCHED();
  k_inv_depth<<<(unsigned)((a.A + 255) / 256), 256, 0, s>>>(a);
  LT_LAUNCHED();
  return LT_OK;
}

int launch_tracer_content(const Arena& a, cudaStream_t s) {
  const long n = (long)a.nx * a.ny * a.km;
  for (int tr = 0; tr < 2; ++tr) {
    long nb = (n + 2 * RB2 - 1) / (2 * RB2);
    k_content_first<<<(unsigned)nb, RB2, 0, s>>>(a.at[a.cur] + tr * a.F, a.tarea, a.dzp, a.kmt, a.nx, a.ny, a.imt,
                                                  a.A, n, a.red_part);
    LT_LAUNCHED();
    int rc = launch_tree_sum(a.red_part, nb, a.red_part + nb, a.scalars + 1 + tr, s);
    if (rc) return rc;
  }
  return LT_OK;
}

int launch_check_numeric(const Arena& a, cudaStream_t s) {
  LT_CUDA_OK(cudaMemsetAsync(a.status, 0, sizeof(int), s));
  k_count_bad<<<1184, 256, 0, s>>>(a.at[a.cur], 2 * a.F, a.status);
  LT_LAUNCHED();
  return LT_OK;
}

}  // namespace lt

using namespace lt;

extern "C" int lt_synth_upload(const lt_synth* syn, lt_domain* dom);

namespace {
template <class T>
int up(cudaStream_t s, T** dst, const std::vector<T>& v, std::vector<void*>& owned) {
  void* p = nullptr;
  if (cudaMalloc(&p, v.size() * sizeof(T)) != cudaSuccess) return LT_E_OOM;
  owned.push_back(p);
  cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s);
  *dst = static_cast<T*>(p);
  return LT_OK;
}
}  // namespace

extern "C" int lt_get_field_device(lt_domain* d, int f, void* dst, size_t nbytes);
extern "C" int lt_set_field_device(lt_domain* d, int f, const void* src, size_t nbytes);

// Device-generated 3-D inputs, host-built 2-D/1-D inputs.
extern "C" int lt_synth_upload(const lt_synth* syn, lt_domain* dom) {
  const Domain* d = lt_synth_domain(syn);
  if (!d || !dom) return LT_E_INVALID;
  lt_grid g;
  lt_synth_grid(syn, &g);
  // 2-D / 1-D from the host builder
  const int two_d[] = {LT_F_H0F, LT_F_H0L, LT_F_SWV, LT_F_NSWV, LT_F_SST, LT_F_SSS, LT_F_FRESH, LT_F_SEAICE,
                       LT_F_TAREA, LT_F_TAREA_R, LT_F_HTW, LT_F_HTS, LT_F_HUN, LT_F_HUE, LT_F_DXU, LT_F_DYU,
                       LT_F_AHF, LT_F_DTN, LT_F_DTS, LT_F_DTE, LT_F_DTW, LT_F_OHBT, LT_F_OHBU, LT_F_AU0,
                       LT_F_AUS, LT_F_AUW, LT_F_AUSW, LT_F_KMT, LT_F_KMU, LT_F_KMTN, LT_F_KMTS, LT_F_KMTE,
                       LT_F_KMTW, LT_F_DZP, LT_F_ODZP, LT_F_ODZT, LT_F_PEN, LT_F_TO, LT_F_SO, LT_F_C};
  for (int f : two_d) {
    const size_t nb = field_bytes(f, d->imt, d->jmt, d->km);
    std::vector<char> buf(nb);
    int rc = lt_synth_field(syn, f, buf.data(), nb);
    if (!rc) rc = lt_set_field(dom, f, buf.data(), nb);
    if (rc) return rc;
  }
  // tables for the device expansion
  cudaStream_t s = nullptr;
  std::vector<void*> owned;
  CellTables t = d->tables();
  int rc = LT_OK;
  double *tprof, *ssurf, *psi, *uprof, *rdyu, *rdxu, *akt_tab;
  int *kmt, *dmin;
  rc |= up(s, &tprof, d->tprof, owned);
  rc |= up(s, &ssurf, d->ssurf, owned);
  rc |= up(s, &psi, d->psi, owned);
  rc |= up(s, &uprof, d->uprof, owned);
  rc |= up(s, &rdyu, d->rdyu, owned);
  rc |= up(s, &rdxu, d->rdxu, owned);
  rc |= up(s, &akt_tab, d->akt_tab, owned);
  rc |= up(s, &kmt, d->kmt, owned);
  rc |= up(s, &dmin, d->dmin, owned);
  if (rc) { for (void* p : owned) cudaFree(p); return LT_E_OOM; }
  t.tprof = tprof; t.ssurf = ssurf; t.psi = psi; t.uprof = uprof; t.rdyu = rdyu; t.rdxu = rdxu;
  t.akt_tab = akt_tab; t.kmt = kmt; t.dmin = dmin;
  const long A = (long)d->imt * d->jmt, F = A * d->km, FB = A * (d->km + 1);
  double *at = nullptr, *atb = nullptr, *vel = nullptr;
  if (cudaMalloc(&at, 2 * F * sizeof(double)) != cudaSuccess || cudaMalloc(&atb, 2 * FB * sizeof(double)) != cudaSuccess) {
    for (void* p : owned) cudaFree(p);
    if (at) cudaFree(at);
    return LT_E_OOM;
  }
  const unsigned nb = (unsigned)((F + 255) / 256);
  k_synth_state<<<nb, 256, 0, s>>>(t, at, atb, nullptr);
  launch_halo_r8(at, 2 * d->km, d->imt, d->jmt, d->cfg.ew_cyclic, d->cfg.tripole, s);
  for (int n = 0; n < 2; ++n) {
    cudaMemsetAsync(atb + n * FB, 0, A * sizeof(double), s);
    cudaMemcpyAsync(atb + n * FB + A, at + n * F, F * sizeof(double), cudaMemcpyDeviceToDevice, s);
  }
  cudaStreamSynchronize(s);
  rc = lt_set_field_device(dom, LT_F_AT, at, 2 * F * sizeof(double));
  if (!rc) rc = lt_set_field_device(dom, LT_F_ATB, atb, 2 * FB * sizeof(double));
  cudaFree(atb);
  if (!rc) {
    if (cudaMalloc(&vel, 6 * F * sizeof(double)) != cudaSuccess) rc = LT_E_OOM;
  }
  if (!rc) {
    k_synth_vel<<<nb, 256, 0, s>>>(t, (double)(d->cfg.ncc + 1), vel, vel + F, vel + 2 * F, vel + 3 * F, vel + 4 * F);
    cudaStreamSynchronize(s);
    rc = lt_set_field_device(dom, LT_F_UTF, vel, F * sizeof(double));
    if (!rc) rc = lt_set_field_device(dom, LT_F_VTF, vel + F, F * sizeof(double));
    if (!rc) rc = lt_set_field_device(dom, LT_F_UTL, vel + 2 * F, F * sizeof(double));
    if (!rc) rc = lt_set_field_device(dom, LT_F_VTL, vel + 3 * F, F * sizeof(double));
    if (!rc) rc = lt_set_field_device(dom, LT_F_AKT, vel + 4 * F, 2 * F * sizeof(double));
    cudaFree(vel);
  }
  cudaFree(at);
  for (void* p : owned) cudaFree(p);
  if (cudaGetLastError() != cudaSuccess && !rc) rc = LT_E_CUDA;
  return rc;
}
