// lt_column_fp64.cu - the FP64 tspas step of both tracers as four passes
// over the columns, each expression in the reference's operation order
// (advection_tracer_2/3 with tracer_del4_1/2, tracer_5..9 and invtrit;
// tracer.cpp:291-978, 1238-1699).  Compiled with -fmad=false.
//
//   k_laplace64   the first Laplacian of atb (on a small grid in k_limit64's launch)
//   k_limit64     per cell and tracer: the predictor, its masked extrema and
//                 the limiter flag (one bit)
//   k_explicit64  per wet cell and tracer: limited fluxes, second
//                 Laplacian, shortwave, explicit vertical mixing, surface
//                 terms; leaves the explicitly updated value in the new state
//   k_thomas      (lt_thomas.cuh) per column and tracer: the implicit half of
//                 the vertical mixing, the new state, dry levels copied (with
//                 diagnostics also their zeros)
//
// Why passes.  Only the implicit sweep runs up and down a column; the rest is a
// stencil that is free in every direction and limited by instruction issue and
// the FP64 pipe, not by memory (about 240 FP64 operations per cell and tracer).
// As one fused march per tile the whole step was a serial chain of levels with
// two block barriers each, at 16 warps per SM, with a third of the predictors
// computed twice on tile halos.  Split, every cell's predictor is formed once,
// a small grid spreads its levels over the SMs and a level has one barrier;
// the price is the flags and the Laplacian going through memory (16 B per cell
// and pass).  The Laplacian lives in the new previous state atb[cur^1] and the
// explicit value in at[cur^1] until the last pass replaces them, so the passes
// need a bit per cell and tracer of storage.
//
// One step of the fused kernel against these passes, 720 x 460 x 55 on the
// global area-depth curve: 2.66 ms against 0.13 (Laplacian, 3.4 TB/s) + 0.43
// (limiter: issue slots 49 % busy, FP64 pipe 35 %) + 0.60 (explicit: 52 %, 35 %)
// + 0.37 (implicit, 3.8 TB/s); 36 x 40 x 55: 270 us against 50.
#include <cstdio>
#include "lt_common.cuh"
#include "lt_thomas.cuh"

namespace lt {
namespace {

constexpr int CX = kColX, CY = kColY, CT = CX * CY;   // a block's columns, one thread each (both tracers)
// A warp takes a patch of PX x PY columns rather than a row of 32: the depths
// of neighbouring columns are alike, so fewer of its lanes idle in the levels
// below some columns' bottoms (lanes active per instruction on a realistic
// depth map: 22.1 of 32 for a row).
constexpr int PX = 8, PY = 4;
// Row of a box with a halo, columns x0-2 .. x0+CX+5: a pitch of 16 banks more
// than a multiple of 32 keeps a patch's rows on different banks.
constexpr int HW = CX + 8;
constexpr int HB = ((CY + 2) * HW * 8 + 127) / 128 * 16; // doubles of such a box, to a 128-byte boundary
constexpr int kColCtas = 512 / CT;                      // blocks per SM: 16 warps of 128 registers
// Most levels of one block, whose level constants sit in shared memory; more
// levels are cut into equal chunks, each of which reads the levels above and
// below it again (1440 x 920 x 55 in two chunks: 5.29 ms of column passes, in
// one 5.19).
constexpr int kChunkMax = 56;

// ------------------------------------------------------------ level pipeline
// One level of a block's columns in shared memory: T and S with a one-point
// halo, the face transports and w; k_explicit64 adds the previous state and
// the mixing of the columns and the first Laplacian with its halo.
struct LimitSlot {
  alignas(128) double at[2][HB];         // rows y0-1 .. y0+CY
  alignas(128) double uw[CY * HW];       // rows y0 .. , columns x0 .. x0+CX+7
  alignas(128) double vs[(CY + 1) * CX]; // rows y0-1 .. y0+CY-1
  alignas(128) double ws[CY * CX];
};
struct ExplicitSlot : LimitSlot {
  alignas(128) double d2[2][HB];
  alignas(128) double atb[2][CY * CX];
  alignas(128) double akt[2][CY * CX];
};
constexpr uint32_t kLimitBytes = 8u * (2 * (CY + 2) * HW + CY * HW + (CY + 1) * CX + CY * CX);
constexpr uint32_t kExplicitBytes = kLimitBytes + 8u * (2 * (CY + 2) * HW + 4 * CY * CX);

template <class Slot, int D>
struct ColumnSmem {
  Slot slot[D];
  // level-free data: per face {h, 1/h} (x faces west of columns x0 .. x0+CX,
  // y faces south of rows y0-1 .. y0+CY-1), per column tarea_r and the
  // biharmonic coefficients {dtn, dts, dte, dtw}
  double2 fx[CY * (CX + 1)], fy[(CY + 1) * CX];
  double2 ns[CT], ew[CT];
  double tr[CT];
  double odzp[kChunkMax], odzt[kChunkMax + 1], pen[kChunkMax + 1];   // of level k at k-k0; pen: level k-1
  uint64_t bar[D];
  int wmax[CT / 32];
};
constexpr int kLimitDepth = 4, kExplicitDepth = 3;
using LimitSmem = ColumnSmem<LimitSlot, kLimitDepth>;
using ExplicitSmem = ColumnSmem<ExplicitSlot, kExplicitDepth>;

// Level L into a slot: TMA boxes issued by one thread, or per-thread asynchronous copies of the same boxes (zeros
// outside the domain, as TMA fills them).
__device__ __forceinline__ void copy_box(double* dst, const double* lvl, const Arena& a, int w, int rows, int bx,
                                         int by) {
  for (int m = threadIdx.x; m < w * rows; m += CT) {
    const int gj = by + m / w, gi = bx + m % w;
    const bool in = gj >= 0 && gj < a.jmt && gi >= 0 && gi < a.imt;
    cp_async8z(dst + m, lvl + (in ? (long)gj * a.imt + gi : 0), in);
  }
}

template <bool EXPLICIT, class Slot>
__device__ __forceinline__ void fill_slot(Slot& sl, uint64_t* bar, const Arena& a, const ColumnMaps& m, bool tma, int L,
                                          int x0, int y0) {
  const int km = a.km;
  if (tma) {
    if (threadIdx.x != 0) return;
    mbar_expect_tx(bar, EXPLICIT ? kExplicitBytes : kLimitBytes);
    tma_load_3d(sl.at[0], &m.at[a.cur], x0 - 2, y0 - 1, L, bar);
    tma_load_3d(sl.at[1], &m.at[a.cur], x0 - 2, y0 - 1, km + L, bar);
    tma_load_3d(sl.uw, &m.uw, x0, y0, L, bar);
    tma_load_3d(sl.vs, &m.vs, x0, y0 - 1, L, bar);
    tma_load_3d(sl.ws, &m.ws, x0, y0, L, bar);
    if constexpr (EXPLICIT) {
      tma_load_3d(sl.d2[0], &m.atb[a.cur ^ 1], x0 - 2, y0 - 1, L + 1, bar);
      tma_load_3d(sl.d2[1], &m.atb[a.cur ^ 1], x0 - 2, y0 - 1, km + 1 + L + 1, bar);
      tma_load_3d(sl.atb[0], &m.atb_own[a.cur], x0, y0, L + 1, bar);
      tma_load_3d(sl.atb[1], &m.atb_own[a.cur], x0, y0, km + 1 + L + 1, bar);
      tma_load_3d(sl.akt[0], &m.akt, x0, y0, L, bar);
      tma_load_3d(sl.akt[1], &m.akt, x0, y0, km + L, bar);
    }
    return;
  }
  const long A = a.A, l = (long)L * A;
  copy_box(sl.at[0], a.at[a.cur] + l, a, HW, CY + 2, x0 - 2, y0 - 1);
  copy_box(sl.at[1], a.at[a.cur] + a.F + l, a, HW, CY + 2, x0 - 2, y0 - 1);
  copy_box(sl.uw, a.uwf + l, a, HW, CY, x0, y0);
  copy_box(sl.vs, a.vsf + l, a, CX, CY + 1, x0, y0 - 1);
  copy_box(sl.ws, a.ws + l, a, CX, CY, x0, y0);
  if constexpr (EXPLICIT) {
    for (int n = 0; n < 2; ++n) {
      copy_box(sl.d2[n], a.atb[a.cur ^ 1] + n * a.FB + l + A, a, HW, CY + 2, x0 - 2, y0 - 1);
      copy_box(sl.atb[n], a.atb[a.cur] + n * a.FB + l + A, a, CX, CY, x0, y0);
      copy_box(sl.akt[n], a.akt + n * a.F + l, a, CX, CY, x0, y0);
    }
  }
  cp_async_mbar_arrive(bar);
}

// The first D levels of the block's march on their way.
template <bool EXPLICIT, int D, class Smem>
__device__ __forceinline__ void start_levels(Smem& S, const Arena& a, const ColumnMaps& maps, bool tma, int x0, int y0,
                                             int k0, int kend) {
  const int kdata = min(kend + 1, a.km);
  for (int L = k0; L < k0 + D && L < kdata; ++L)
    fill_slot<EXPLICIT>(S.slot[L - k0], &S.bar[L - k0], a, maps, tma, L, x0, y0);
}

// The block's march over its levels k0 .. kend-1 (top down): the slot of level
// k+1 has arrived when body(k, slot(k), slot(k+1)) runs, the one of level k-1
// is refilled D-1 levels ahead.  One barrier per level.  kdata: levels below
// kend read (kend itself for the level below the last, where there is one).
template <bool EXPLICIT, int D, class Smem, class Body>
__device__ __forceinline__ void march(Smem& S, const Arena& a, const ColumnMaps& maps, bool tma, int x0, int y0, int k0,
                                      int kend, Body body) {
  const int kdata = min(kend + 1, a.km);
  auto slot_of = [&](int L) { return (L - k0) % D; };
  auto fill = [&](int L) {
    const int s = slot_of(L);
    fill_slot<EXPLICIT>(S.slot[s], &S.bar[s], a, maps, tma, L, x0, y0);
  };
  for (int k = k0 - 1; k < kend; ++k) {
    // wait for level k+1 (k0 first)
    const int L = k + 1;
    bool ok = true;
    if (L < kdata) ok = mbar_wait(&S.bar[slot_of(L)], (uint32_t)(((L - k0) / D) & 1), a.wait_limit);
    if (__syncthreads_or(!ok)) {
      // a wait ran out: record it, let the copies still in flight land
      // (bounded) and leave together
      if (threadIdx.x == 0) {
        atomicExch(a.status + 1, 1);
        const int filled = max(k0 + D, k - 1 + D);   // one past the last level filled so far
        for (int l = L; l < kdata && l < filled; ++l)
          mbar_wait(&S.bar[slot_of(l)], (uint32_t)(((l - k0) / D) & 1));
      }
      __syncthreads();
      return;
    }
    if (k < k0) continue;
    // every thread is done with level k-1: its slot takes level k-1+D
    if (k > k0 && k - 1 + D < kdata) fill(k - 1 + D);
    body(k, S.slot[slot_of(k)], S.slot[slot_of(k + 1 < kdata ? k + 1 : k)]);
  }
}

template <class Smem>
__device__ __forceinline__ int block_max(Smem& S, int v) {
  v = __reduce_max_sync(0xffffffffu, v);
  if (threadIdx.x % 32 == 0) S.wmax[threadIdx.x / 32] = v;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < CT / 32; ++w) v = max(v, S.wmax[w]);
  return v;
}

// The block's level barriers (before a __syncthreads).
template <int D, class Smem>
__device__ __forceinline__ void init_bars(Smem& S, bool tma) {
  if (threadIdx.x == 0) {
    // arrivals per level: the issuing thread's (TMA), or one per copying thread
    for (int s = 0; s < D; ++s) mbar_init(&S.bar[s], tma ? 1 : CT);
    mbar_fence_init();
  }
}

// The block's level-free data, loaded while its first levels are on their way.
template <class Smem>
__device__ __forceinline__ void load_block(Smem& S, const Arena& a, int x0, int y0, int k0, int kc) {
  const int tid = threadIdx.x, imt = a.imt, jmt = a.jmt, km = a.km;
  for (int m = tid; m < CY * (CX + 1) + (CY + 1) * CX; m += CT) {
    const bool x = m < CY * (CX + 1);
    const int f = x ? m : m - CY * (CX + 1);
    const int gj = x ? y0 + f / (CX + 1) : y0 - 1 + f / CX, gi = x0 + (x ? f % (CX + 1) : f % CX);
    const bool in = gj >= 0 && gj < jmt && gi < imt;
    const long q = in ? (long)gj * imt + gi : 0;
    const double h = !in ? 0.0 : x ? a.htw[q] * a.hun[q] : a.hts[q] * a.hue[q];
    (x ? S.fx : S.fy)[f] = make_double2(h, 1.0 / h);
  }
  for (int m = tid; m < CT; m += CT) {
    const int gj = y0 + m / CX, gi = x0 + m % CX;
    if (gj >= jmt || gi >= imt) continue;
    const long q = (long)gj * imt + gi;
    S.tr[m] = a.tarea_r[q];
    S.ns[m] = make_double2(a.dtn[q], a.dts[q]);
    S.ew[m] = make_double2(a.dte[q], a.dtw[q]);
  }
  for (int c = tid; c <= kc; c += CT) {
    const int k = k0 + c;
    if (c < kc && k < km) S.odzp[c] = a.odzp[k];
    S.odzt[c] = k < km ? a.odzt[k] : 0.0;
    S.pen[c] = k >= 1 && k <= km ? a.pen[k - 1] : 0.0;
  }
  __syncthreads();
}

// ----------------------------------------------------------------- divisions
// The face divisions: lt_common.cuh's quotient, four of them sharing one test
// of their dividends' magnitudes.

// One column's faces and metric in the block's level-free data.
struct Faces {
  const double2 *e, *w, *s, *n;
  double tr, tr2;       // tarea_r, 2*tarea_r (the reference's *2.0*tarea_r; not its *tarea_r*2.0, rounded before it doubles)
  bool fast;
};

template <class Smem>
__device__ __forceinline__ Faces column_faces(const Smem& S, int tx, int ty) {
  Faces f;
  f.w = S.fx + ty * (CX + 1) + tx;
  f.e = f.w + 1;
  f.n = S.fy + ty * CX + tx;
  f.s = f.n + CX;
  f.fast = div_admits(f.e->x) && div_admits(f.w->x) && div_admits(f.s->x) && div_admits(f.n->x);
  f.tr = S.tr[ty * CX + tx];
  f.tr2 = 2.0 * f.tr;
  return f;
}

// Horizontal and vertical transports of one cell and the factors of the
// vertical terms both tracers share.
struct Flow {
  double ue, uw, vs, vn, wk, w1;
  double A, B, C1, C2;   // 0.5*odzp*w(k), 0.5*odzp*w(k+1), their Lax-Wendroff factors (upper one negated)
};

__device__ __forceinline__ void vertical_factors(Flow& f, double odzp, double odzt, double odzt1) {
  const double hz = 0.5 * odzp;
  f.A = hz * f.wk;
  f.B = hz * f.w1;
  f.C1 = -f.A * f.wk * odzt;
  f.C2 = f.B * f.w1 * odzt1;
}

// s + x*2.0: doubling is exact, so the fused sum is rounded as the separate one
// (where 2x overflows it is not, and the sum is at the end of the range)
__device__ __forceinline__ double plus_twice(double s, double x) { return __fma_rn(2.0, x, s); }

// unlimited (Lax-Wendroff) parts of the horizontal face fluxes
struct Lw {
  double e, w, s, n;
};
__device__ __forceinline__ Lw lax_wendroff(const Faces& g, const Flow& f, double dts, double de, double dw, double ds,
                                           double dn) {
  const double ae = -dts * de * g.tr2 * f.ue * f.ue, aw = dts * dw * g.tr2 * f.uw * f.uw;
  const double as = -dts * ds * g.tr2 * f.vs * f.vs, an = dts * dn * g.tr2 * f.vn * f.vn;
  Lw r{div_fast(ae, g.e->x, g.e->y), div_fast(aw, g.w->x, g.w->y), div_fast(as, g.s->x, g.s->y), div_fast(an, g.n->x, g.n->y)};
  const unsigned key = max(max(div_key(ae), div_key(aw)), max(div_key(as), div_key(an)));
  if (key >= kDivSpan || !g.fast) {
    // out of range: a zero (land faces) is right as it is
    auto bad = [](double x) { return div_key(x) >= kDivSpan && x != 0.0; };
    if (!g.fast || bad(ae) || bad(aw) || bad(as) || bad(an)) {
      r.e = ae / g.e->x;
      r.w = aw / g.w->x;
      r.s = as / g.s->x;
      r.n = an / g.n->x;
    }
  }
  return r;
}

// ------------------------------------------------------------ limiter flags
// Levels of a column whose flags anything reads: without diagnostics those
// with a wet cell here or across one of the faces (the flag of a dry cell
// below its own column's bottom meets the column only through w = 0).
struct Kmt5 {
  int c, n, s, e, w;
  __device__ int deepest() const { return max(max(max(n, s), max(e, w)), c); }
};
__device__ __forceinline__ Kmt5 load_kmt5(const Arena& a, long q) {
  return {a.kmt[q], a.kmt[q - a.imt], a.kmt[q + a.imt], a.kmt[q + 1], a.kmt[q - 1]};
}

// ---------------------------------------------------------- first Laplacian
// tracer_del4_1 at the wet cells of levels k0 .. k1-1 of one column: ahf *
// (masked Laplacian of atb), left in the new previous state (level k at atb's
// level k+1).  Memory bound: neighbours come through L1.
__device__ __forceinline__ void laplace_column(const Arena& a, int i, int j, int k0, int k1) {
  if (!(i >= 1 && i < a.imt - 1 && j >= 1 && j < a.jmt - 1)) return;
  const int imt = a.imt;
  const long A = a.A, FB = a.FB;
  const long q = (long)j * imt + i;
  const Kmt5 kq = load_kmt5(a, q);
  k1 = min(k1, kq.c);
  if (k0 >= k1) return;
  const double dtn = a.dtn[q], dts = a.dts[q], dte = a.dte[q], dtw = a.dtw[q], ahf = a.ahf[q];
  const double* __restrict__ atb = a.atb[a.cur];
  double* __restrict__ d2 = a.atb[a.cur ^ 1];
  // two levels' loads together, whatever the masks say
  constexpr int AH = 2;
  for (int kb = k0; kb < k1; kb += AH) {
    double x[AH][2][5];   // here, north, south, east, west
#pragma unroll
    for (int d = 0; d < AH; ++d)
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const double* p = atb + n * FB + (long)(min(kb + d, k1 - 1) + 1) * A + q;
        x[d][n][0] = p[0];
        x[d][n][1] = p[-imt];
        x[d][n][2] = p[imt];
        x[d][n][3] = p[1];
        x[d][n][4] = p[-1];
      }
#pragma unroll
    for (int d = 0; d < AH; ++d) {
      const int k = kb + d;
      if (k >= k1) break;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        double h = 0.0, cc = 0.0;
        auto term = [&](bool there, double v, double cf) {
          if (there) {
            h += cf * v;
            cc -= cf;
          }
        };
        term(k < kq.n, x[d][n][1], dtn);
        term(k < kq.s, x[d][n][2], dts);
        term(k < kq.e, x[d][n][3], dte);
        term(k < kq.w, x[d][n][4], dtw);
        d2[n * FB + (long)(k + 1) * A + q] = ahf * (cc * x[d][n][0] + h);
      }
    }
  }
}

constexpr int kLaplaceLevels = 8;
__global__ void __launch_bounds__(128) k_laplace64(const __grid_constant__ Arena a, int row0) {
  chain_grid();
  const int k0 = blockIdx.z * kLaplaceLevels;
  laplace_column(a, blockIdx.x * CX + threadIdx.x, (row0 + blockIdx.y) * CY + threadIdx.y, k0, k0 + kLaplaceLevels);
}

// The thread's column in the block: warp w is the patch (w % (CX/PX), w / (CX/PX)).
struct Column {
  int tx, ty;
  __device__ Column() {
    const int w = threadIdx.x / 32, l = threadIdx.x % 32;
    tx = w % (CX / PX) * PX + l % PX;
    ty = w / (CX / PX) * PY + l / PX;
  }
};
// Flag words [tracer][level][patch row][patch column], bit l: the patch's lane l.
__device__ __forceinline__ int patches_x() { return gridDim.x * (CX / PX); }
__device__ __forceinline__ int patches_y(const Arena& a) { return (a.jmt + CY - 1) / CY * (CY / PY); }

// Bound by issue and FP64 latency at 16 warps per SM.  Both tracers in one
// thread: transports, masks, metric terms and the level's bookkeeping are 60 %
// of a level's instructions (with a tracer per thread and 24 warps per SM it
// took 557 us instead of 432, 720 x 460 x 55 deep).
template <bool DIAG>
__global__ void __launch_bounds__(CT, kColCtas) k_limit64(const __grid_constant__ Arena a, const __grid_constant__ ColumnMaps maps,
                                                          int kc, int nch, int tma, int row0) {
  chain_grid();
  extern __shared__ __align__(128) unsigned char smem_col[];
  LimitSmem& S = *reinterpret_cast<LimitSmem*>(smem_col);
  const Column col;
  const int tx = col.tx, ty = col.ty;
  const int x0 = blockIdx.x * CX, y0 = (row0 + blockIdx.y) * CY, i = x0 + tx, j = y0 + ty;
  const int km = a.km;
  if ((int)blockIdx.z >= nch) {   // the Laplacian's blocks
    const int k = ((int)blockIdx.z - nch) * kc;
    laplace_column(a, i, j, k, min(k + kc, km));
    return;
  }
  const bool ring = i >= 1 && i < a.imt - 1 && j >= 1 && j < a.jmt - 1;
  const long q = (long)j * a.imt + i;
  const int k0 = blockIdx.z * kc;
  Kmt5 kq{0, 0, 0, 0, 0};
  int k1 = k0;   // end of this thread's levels
  if (ring) {
    kq = load_kmt5(a, q);
    k1 = min(k0 + kc, DIAG ? flow_end(a, q, kq.c) : kq.deepest());
  }
  init_bars<kLimitDepth>(S, tma != 0);
  const int kend = block_max(S, k1);
  if (k0 >= kend) return;
  start_levels<false, kLimitDepth>(S, a, maps, tma != 0, x0, y0, k0, kend);
  load_block(S, a, x0, y0, k0, kc);
  const double dts = a.p.dts;
  const Faces g = column_faces(S, tx, ty);
  double up[2] = {0.0, 0.0}, cc[2] = {0.0, 0.0};   // levels k-1 and k
  if (k0 < k1 && k0 > 0)
    for (int n = 0; n < 2; ++n) up[n] = a.at[a.cur][n * a.F + (long)(k0 - 1) * a.A + q];
  const int r = (ty + 1) * HW + tx + 2, ru = ty * HW + tx, rv = ty * CX + tx;
  const long level = (long)patches_x() * patches_y(a);
  unsigned* words = a.flags + k0 * level + (long)(j / PY) * patches_x() + i / PX;
  march<false, kLimitDepth>(S, a, maps, tma != 0, x0, y0, k0, kend, [&](int k, const LimitSlot& L, const LimitSlot& D) {
    bool flag[2] = {false, false};
    if (k < k1) {
      const bool last = k == km - 1;
      Flow f;
      f.ue = L.uw[ru + 1];
      f.uw = L.uw[ru];
      f.vs = L.vs[rv + CX];
      f.vn = L.vs[rv];
      f.wk = L.ws[rv];
      f.w1 = last ? 0.0 : D.ws[rv];
      // a dry cell whose faces carry no transport: either form of its face
      // fluxes is the same zero, so its flag stays 0
      const bool wet = k < kq.c;
      bool skip = false;
      if (!wet) skip = f.ue == 0.0 && f.uw == 0.0 && f.vs == 0.0 && f.vn == 0.0;
      if (k == k0)
        for (int n = 0; n < 2; ++n) cc[n] = L.at[n][r];
      double lo[2];
      for (int n = 0; n < 2; ++n) lo[n] = last ? 0.0 : D.at[n][r];
      if (!skip) {
        const double odzp = S.odzp[k - k0];
        vertical_factors(f, odzp, S.odzt[k - k0], S.odzt[k - k0 + 1]);
        const double du = f.ue - f.uw, dv = f.vs - f.vn;
        const bool wn = k < kq.n, wso = k < kq.s, ww = k < kq.w, we = k < kq.e;
        const bool wu = k > 0 && k - 1 < kq.c, wl = k + 1 < kq.c;
        const bool land = !(wn && wso && ww && we && (wl || last));   // beside or below a wet cell
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const double* at = L.at[n] + r;
          const double c = cc[n], e = at[1], w = at[-1], s = at[HW], nn = at[-HW];
          const double x0v = (e + c) * f.ue * g.tr - (c + w) * f.uw * g.tr;
          const double y0v = ((s + c) * f.vs - (c + nn) * f.vn) * g.tr;
          const Lw lw = lax_wendroff(g, f, dts, e - c, c - w, s - c, c - nn);
          const double cx = -c * du * g.tr;
          const double cy = -c * dv * g.tr;
          double za, zb1, zb2, zc;
          if (k == 0) {
            za = -f.B * (lo[n] + c);
            zb1 = 0.0;
            zb2 = f.C2 * (c - lo[n]) * dts;
            zc = odzp * c * f.w1;
          } else if (last) {
            za = f.A * (c + up[n]);
            zb1 = f.C1 * (up[n] - c) * dts;
            zb2 = 0.0;
            zc = -odzp * c * f.wk;
          } else {
            za = f.A * (c + up[n]) - f.B * (c + lo[n]);
            zb1 = f.C1 * (up[n] - c) * dts;
            zb2 = f.C2 * (c - lo[n]) * dts;
            zc = -odzp * c * (f.wk - f.w1);
          }
          const double xx = -plus_twice(x0v + lw.e + lw.w, cx);
          const double yy = -plus_twice(y0v + lw.s + lw.n, cy);
          const double zz = -(zb1 + zb2 + za + zc);
          const double a00 = c + (xx + yy + zz) * dts;
          // a00 > max or a00 < min over the cell and its wet neighbours,
          // without forming the extrema: beyond a wet cell's own value in one
          // direction, and not short of any wet neighbour in it.  Comparing
          // with both signs flipped turns "below" into "above".  Land counts
          // as -1e10 for the maximum and +1e10 for the minimum, either -1e10
          // when turned; a dry cell's own value too, so it is asked in both
          // directions.
          auto beyond = [&](int flip) {
            auto turned = [&](double t) { return __hiloint2double(__double2hiint(t) ^ flip, __double2loint(t)); };
            const double x = turned(a00);
            bool out = x > (wet ? turned(c) : -1.0e10);
            auto seen = [&](bool there, double t) { out = out && !(there && x <= turned(t)); };
            seen(wn, nn);
            seen(wso, s);
            seen(ww, w);
            seen(we, e);
            seen(wu, up[n]);
            seen(wl, lo[n]);
            return out && !(land && x <= -1.0e10);
          };
          const int below = (int)0x80000000;
          flag[n] = beyond(a00 < c ? below : 0);
          if (!wet) flag[n] = flag[n] || beyond(a00 < c ? 0 : below);
        }
      }
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        up[n] = cc[n];
        cc[n] = lo[n];
      }
    }
    const unsigned w0 = __ballot_sync(0xffffffffu, flag[0]), w1 = __ballot_sync(0xffffffffu, flag[1]);
    if (threadIdx.x % 32 == 0) {
      words[0] = w0;
      words[km * level] = w1;
    }
    words += level;
  });
}

// ----------------------------------------------------------- explicit update
// Without diagnostics the wet inner cells; with them every ring cell (ax, ay,
// az) and every inner cell (dz, penetrate, the value) above the block's
// dry_from.  Bound as
// k_limit64: 605 us at 720 x 460 x 55 deep (1216 with neighbours loaded through
// L1 instead of level slots).
// ROW0: a launch over part of the rows (the offset costs this kernel, at its limit
// of registers, 1 %).
template <bool DIAG, bool ROW0>
__global__ void __launch_bounds__(CT, kColCtas) k_explicit64(const __grid_constant__ Arena a,
                                                      const __grid_constant__ ColumnMaps maps, int kc, int tma, int row0) {
  chain_grid();
  extern __shared__ __align__(128) unsigned char smem_col[];
  ExplicitSmem& S = *reinterpret_cast<ExplicitSmem*>(smem_col);
  const Column col;
  const int tx = col.tx, ty = col.ty, lane = threadIdx.x % 32;
  const int x0 = blockIdx.x * CX, y0 = (ROW0 ? row0 + blockIdx.y : blockIdx.y) * CY, i = x0 + tx, j = y0 + ty;
  const int imt = a.imt, jmt = a.jmt, km = a.km;
  const long A = a.A, F = a.F;
  const bool inner = i >= 2 && i < imt - 2 && j >= 2 && j < jmt - 2;
  const bool ring = i >= 1 && i < imt - 1 && j >= 1 && j < jmt - 1;
  const long q = (long)j * imt + i;
  const int k0 = blockIdx.z * kc;
  Kmt5 kq{0, 0, 0, 0, 0};
  int k1 = k0;
  if (DIAG ? ring : inner) {
    kq = load_kmt5(a, q);
    k1 = min(k0 + kc, DIAG ? flow_end(a, q, kq.c) : kq.c);
  }
  const int kz = kq.c;
  init_bars<kExplicitDepth>(S, tma != 0);
  const int kend = block_max(S, k1);
  if (k0 >= kend) return;
  if (DIAG && ring) k1 = kend;   // the block's columns alike: the last pass takes them from there
  start_levels<true, kExplicitDepth>(S, a, maps, tma != 0, x0, y0, k0, kend);
  load_block(S, a, x0, y0, k0, kc);
  const lt_params& p = a.p;
  const double dts = p.dts;
  const Faces g = column_faces(S, tx, ty);
  double swv = 0.0;
  double up[2] = {0.0, 0.0}, cc[2] = {0.0, 0.0};                         // at of levels k-1, k
  double bc[2] = {0.0, 0.0}, mix[2] = {0.0, 0.0};                        // atb of level k; mixing flux from above it
  if (k0 < k1) {
    swv = inner ? a.swv[q] : 0.0;
    if (k0 > 0)
      for (int n = 0; n < 2; ++n) {
        const long c = (long)(k0 - 1) * A + q;
        const double* atb = a.atb[a.cur] + n * a.FB + c + A;   // level k0-1
        up[n] = a.at[a.cur][n * F + c];
        mix[n] = a.akt[n * F + c] * (atb[0] - atb[A]) * a.odzt[k0] * (k0 < kz ? 1.0 : 0.0);
      }
  }
  // Flag words of the warp's patch at levels k-1, k, k+1; those of level k+1's
  // neighbour patches (west, east, north, south) and of level k+2 are loaded a
  // level ahead, one per lane: lanes 0-4 tracer 0's, lanes 8-12 tracer 1's.
  const int npx = patches_x(), npy = ROW0 ? patches_y(a) : gridDim.y * (CY / PY), px = i / PX, py = j / PY, what = lane % 8;
  const long level = (long)npx * npy;
  const unsigned* words = a.flags + (lane < 8 ? 0L : km * level) + k0 * level + (long)py * npx + px;
  const bool word_in = lane < 16 && (what == 0 || (what == 1 && px > 0) || (what == 2 && px + 1 < npx) ||
                                     (what == 3 && py > 0) || (what == 4 && py + 1 < npy));
  const long word_at = what == 0 ? level : what == 1 ? -1 : what == 2 ? 1 : what == 3 ? -(long)npx : (long)npx;
  auto load_words = [&](int k) {
    return word_in && k < kend && (what > 0 || k + 1 < km) ? words[(k - k0) * level + word_at] : 0u;
  };
  const unsigned me = 1u << lane;
  unsigned next = load_words(k0), wu[2], wc[2];
  {
    const unsigned own = lane == 0 || lane == 8 ? words[0] : 0u;
    const unsigned above = (lane == 0 || lane == 8) && k0 > 0 ? words[-level] : 0u;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      wc[n] = __shfl_sync(0xffffffffu, own, 8 * n);
      wu[n] = __shfl_sync(0xffffffffu, above, 8 * n);
    }
  }
  const int r = (ty + 1) * HW + tx + 2, ru = ty * HW + tx, rv = ty * CX + tx;
  double* __restrict__ out = a.at[a.cur ^ 1];
  long c0 = (long)k0 * A + q;
  march<true, kExplicitDepth>(S, a, maps, tma != 0, x0, y0, k0, kend,
                              [&](int k, const ExplicitSlot& L, const ExplicitSlot& D) {
    // the faces that are limited: where either cell's predictor leaves its bounds
    unsigned le[2], lw[2], ln[2], ls[2], lu[2], ld[2];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const unsigned below = __shfl_sync(0xffffffffu, next, 8 * n);
      const unsigned ww = __shfl_sync(0xffffffffu, next, 8 * n + 1), we = __shfl_sync(0xffffffffu, next, 8 * n + 2);
      const unsigned wn = __shfl_sync(0xffffffffu, next, 8 * n + 3), wsn = __shfl_sync(0xffffffffu, next, 8 * n + 4);
      const unsigned w = wc[n];
      static_assert(PX == 8 && PY == 4, "patch shifts");
      le[n] = w | ((w >> 1) & 0x7f7f7f7fu) | ((we << 7) & 0x80808080u);
      lw[n] = w | ((w << 1) & 0xfefefefeu) | ((ww >> 7) & 0x01010101u);
      ln[n] = w | (w << 8) | (wn >> 24);
      ls[n] = w | (w >> 8) | (wsn << 24);
      lu[n] = w | wu[n];
      ld[n] = w | below;
      wu[n] = w;
      wc[n] = below;
      if (DIAG && !(k == 0 || k == km - 1)) {
        // at the rim, between the top and bottom level, such a face keeps its form
        if (!(i <= imt - 3)) le[n] = 0u;
        if (!(i >= 2)) lw[n] = 0u;
        if (!(j <= jmt - 3)) ls[n] = 0u;
        if (!(j >= 2)) ln[n] = 0u;
      }
    }
    next = load_words(k + 1);
    if (k >= k1) return;
    const bool last = k == km - 1;
    const int kl = k - k0;
    Flow f;
    f.ue = L.uw[ru + 1];
    f.uw = L.uw[ru];
    f.vs = L.vs[rv + CX];
    f.vn = L.vs[rv];
    f.wk = L.ws[rv];
    f.w1 = last ? 0.0 : D.ws[rv];
    if (k == k0)
      for (int n = 0; n < 2; ++n) {
        cc[n] = L.at[n][r];
        bc[n] = L.atb[n][rv];
      }
    const double odzp = S.odzp[kl], odzt = S.odzt[kl], odzt1 = S.odzt[kl + 1];
    vertical_factors(f, odzp, odzt, odzt1);
    const double du = f.ue - f.uw, dv = f.vs - f.vn;
    const double vit_k = !DIAG || k < kz ? 1.0 : 0.0, vit_kp1 = k + 1 < kz ? 1.0 : 0.0;
    const bool dry = DIAG && k >= kz;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const double* at = L.at[n] + r;
      const double c = cc[n], e = at[1], w = at[-1], s = at[HW], nn = at[-HW];
      const double lo = last ? 0.0 : D.at[n][r];
      const long cg = n * F + c0;
      double adv;
      {
        const double de = e - c, dw = c - w, ds = s - c, dn = c - nn;
        Lw xy = lax_wendroff(g, f, dts, de, dw, ds, dn);
        if (le[n] & me) xy.e = -de * fabs(f.ue) * g.tr;
        if (lw[n] & me) xy.w = dw * fabs(f.uw) * g.tr;
        if (ls[n] & me) xy.s = -ds * fabs(f.vs) * g.tr;
        if (ln[n] & me) xy.n = dn * fabs(f.vn) * g.tr;
        double za, zb1 = 0.0, zb2 = 0.0, zc;
        // the upwind forms -0.5*|w|*odzp*d and 0.5*|w|*odzp*d, the factor 0.5 exact
        if (k > 0) zb1 = (lu[n] & me) ? -fabs(f.A) * (up[n] - c) : f.C1 * (up[n] - c) * dts;
        if (!last) zb2 = (ld[n] & me) ? fabs(f.B) * (c - lo) : f.C2 * (c - lo) * dts;
        if (k == 0) {
          za = -f.B * (lo + c);
          zc = odzp * c * f.w1;
        } else if (last) {
          za = f.A * (c + up[n]);
          zc = -odzp * c * f.wk;
        } else {
          za = f.A * (c + up[n]) - f.B * (c + lo);
          zc = -odzp * c * (f.wk - f.w1);
        }
        const double cx = -c * du * g.tr;
        const double cy = -c * dv * g.tr;
        const double x0v = (e + c) * f.ue * g.tr - (c + w) * f.uw * g.tr;
        const double y0v = ((s + c) * f.vs - (c + nn) * f.vn) * g.tr;
        const double xx = -plus_twice(x0v + xy.e + xy.w, cx);
        const double yy = -plus_twice(y0v + xy.s + xy.n, cy);
        const double zz = -(za + zb1 + zb2 + zc);
        adv = xx + yy + zz;
        if (DIAG) {
          a.ax[cg] = xx;
          a.ay[cg] = yy;
          a.az[cg] = zz;
        }
      }
      if (!DIAG || inner) {
        double tf = adv * vit_k;
        if (!dry) {
          const double* d = L.d2[n] + r;
          const double2 ns = S.ns[rv], ew = S.ew[rv];
          double h = 0.0, c5 = 0.0;
          if (k < kq.n) { h += ns.x * d[-HW]; c5 -= ns.x; }
          if (k < kq.s) { h += ns.y * d[HW]; c5 -= ns.y; }
          if (k < kq.e) { h += ew.x * d[1]; c5 -= ew.x; }
          if (k < kq.w) { h += ew.y * d[-1]; c5 -= ew.y; }
          tf += p.ah * (c5 * d[0] + h);
        }
        // shortwave, T only (tracer.cpp:1430-1474)
        if (n == 0) {
          if (k == 0) {
            const double w1 = swv * S.pen[kl + 1] * (1 < kz ? 1.0 : 0.0);
            tf = tf - odzp * w1;
            if (DIAG) a.penetrate[c0] = -w1 * odzp;
          } else if (last) {
            const double w2 = swv * S.pen[kl] * vit_k;
            tf = tf + odzp * w2;
            if (DIAG) a.penetrate[c0] = w2 * odzp;
          } else {
            const double w1 = swv * S.pen[kl] * vit_k;
            const double w2 = swv * S.pen[kl + 1] * vit_kp1;
            tf = tf + (w1 - w2) * odzp;
            if (DIAG) a.penetrate[c0] = (w1 - w2) * odzp;
          }
        }
        // explicit half of the vertical mixing (tracer.cpp:1476-1543)
        // (the flux through a face is one expression in both of its cells)
        const double bl = last ? 0.0 : D.atb[n][rv];
        const double w1 = mix[n], w2 = last ? 0.0 : L.akt[n][rv] * (bc[n] - bl) * odzt1 * vit_kp1;
        if (k == 0) {
          tf = tf - odzp * w2 * 0.5;
          if (DIAG) a.dzd[cg] = -odzp * w2 * 0.5;
        } else if (last) {
          tf = tf + odzp * w1 * (1.0 - 0.5);
          if (DIAG) a.dzd[cg] = odzp * w1 * 0.5;
        } else {
          tf = tf + odzp * (w1 - w2) * 0.5;
          if (DIAG) a.dzd[cg] = odzp * (w1 - w2) * 0.5;
        }
        mix[n] = w2;
        if (dry) {
          // below the bottom every term is masked: the value stays
          out[cg] = c;
        } else {
          if (k == 0) {
            const double stf = a.stf_n[n * A + q];
            if (n == 1) {
              tf = tf + stf * (1.0 - 0.5) * odzp;
              tf = tf + a.scalars[0] * vit_k;
            } else {
              tf = tf + stf * odzp * 0.5;
            }
          }
          if (p.simple_assm && k < p.ktv) tf = tf + vit_k * (a.restore_at[cg] - bc[n]) * assm_rate(k);
          if (p.boundary_restore == 1 && k >= 1) {
            const double lamda = 1.0 / (15.0 * 86400.0);
            tf = tf + vit_k * (a.restore[cg] - bc[n]) * lamda;
          }
          out[cg] = c + dts * tf;
        }
        bc[n] = bl;
      }
      up[n] = c;
      cc[n] = lo;
    }
    c0 += A;
  });
}

}  // namespace

// Levels per block: a thread keeps the levels above and below in registers,
// so long chunks read each level once; short ones give a small grid enough
// blocks (eight rounds of the resident ones) to fill the GPU evenly although
// most of a shallow grid's levels are dry (360 x 218 x 30: 181 us of column
// passes; with four rounds 191).
static int chunk_levels(long column_blocks, int km) {
  const long want = 148L * kColCtas * 8;
  long chunks = (want + column_blocks - 1) / column_blocks;
  const long most = (km + 3) / 4, least = (km + kChunkMax - 1) / kChunkMax;
  chunks = chunks > most ? most : chunks < least ? least : chunks;
  return (int)((km + chunks - 1) / chunks);
}

// Raises the column kernels' shared-memory limit on the current device (not
// inside a stream capture).
int prepare_column_fp64() {
  if (int rc = prepare_thomas()) return rc;
  const void* lim[] = {(const void*)k_limit64<false>, (const void*)k_limit64<true>};
  const void* ex[] = {(const void*)k_explicit64<false, false>, (const void*)k_explicit64<true, false>,
                      (const void*)k_explicit64<false, true>, (const void*)k_explicit64<true, true>};
  for (const void* k : lim)
    LT_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LimitSmem)));
  for (const void* k : ex)
    LT_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ExplicitSmem)));
  return LT_OK;
}

int launch_column_fp64(const Arena& a, const ColumnMaps& maps, bool tma, cudaStream_t s) {
  if (int rc = launch_assm_dt_restore(a, s)) return rc;
  const unsigned gx = (a.imt + CX - 1) / CX, gy = (a.jmt + CY - 1) / CY;
  const int kc = chunk_levels((long)gx * gy, a.km);
  const int nch = (a.km + kc - 1) / kc;
  const int t = tma ? 1 : 0;
  // The first Laplacian: on a small grid in the limiter's launch, whose blocks
  // leave the GPU partly idle (36 x 40 x 55: a launch of 14 us less per step);
  // on a large one in a kernel of its own, at three times the occupancy.
  const bool together = (long)gx * gy * nch < 148L * kColCtas * 4;
  if (!together) {
    if (int rc = for_column_rows(a, [&](int r, int rows) {
          return launch_chained(k_laplace64, dim3(gx, rows, (a.km + kLaplaceLevels - 1) / kLaplaceLevels), dim3(CX, CY), 0, s,
                                a, r);
        }))
      return rc;
  }
  if (int rc = for_column_rows(a, [&](int r, int rows) {
        return launch_chained(a.diagnostics ? k_limit64<true> : k_limit64<false>,
                              dim3(gx, rows, together ? 2 * nch : nch), dim3(CT), sizeof(LimitSmem), s, a, maps, kc, nch, t, r);
      }))
    return rc;
  if (int rc = for_column_rows(a, [&](int r, int rows) {
        const bool part = rows < (int)gy;
        return launch_chained(a.diagnostics ? (part ? k_explicit64<true, true> : k_explicit64<true, false>)
                                            : (part ? k_explicit64<false, true> : k_explicit64<false, false>),
                              dim3(gx, rows, nch), dim3(CT), sizeof(ExplicitSmem), s, a, maps, kc, t, r);
      }))
    return rc;
  return a.diagnostics ? launch_thomas<true>(a, maps, tma, s) : launch_thomas<false>(a, maps, tma, s);
}

}  // namespace lt
