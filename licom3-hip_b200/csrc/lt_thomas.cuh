// lt_thomas.cuh - the last pass over the columns of the FP64 tspas step: the
// implicit half of the vertical mixing (invtrit, tracer.cpp:923-978), the new
// state, and the dry levels.
//
// The pass finds the explicitly updated values in the new state at[cur^1].
// One thread per column and tracer eliminates from the bottom level up and
// substitutes from the top down; the elimination coefficients take the place
// of the values they came from (f in at[cur^1], e in atb[cur^1]), written
// with an L2 evict-last policy and read back evict-first, so that they stay
// on chip: 16 B per level and column in flight.  The level data arrive in
// stages of kThLevels levels through a ring of shared-memory slots, so a
// warp's chain of divisions never waits for memory: by TMA boxes, or by
// per-thread asynchronous copies where the row pitch does not allow boxes.
// Every wait is bounded.
//
// Bound by the chain of divisions per level and by L2: 374 us at 720 x 460 x 55
// on the global area-depth curve, 1.43 GB of DRAM traffic (3.8 TB/s).  Two
// stages and five blocks per SM: more blocks (six: 1.73 ms at 1440 x 920 x 55)
// or more stages (three: 1.54 ms) push the coefficients out of L2 or leave
// fewer blocks, against 1.34 ms.
#pragma once
#include "lt_common.cuh"
#include "lt_tracer_tma.cuh"

namespace lt {

constexpr int kThX = kThomasX, kThY = kThomasY, kThT = kThX * kThY;
constexpr int kThLevels = kThomasLevels;
static_assert(kThX == kColX && kThY == kColY, "the passes share their blocks");
constexpr int kThStages = 2;

struct ThomasSmem {
  struct alignas(128) Slot {
    alignas(128) double d8[kThLevels * kThT];   // levels l0 .. l0+kThLevels-1 of the explicit values
    alignas(128) double akt[kThLevels * kThT];      // levels l0-1 .. of the mixing coefficient
  } slot[kThStages];
  uint64_t bar[kThStages];
  int wmax[kThT / 32];
};

// With diagnostics a column's levels from here down are below its bottom and
// carry no transport through its four faces or w (kflow of its own column
// covers its west and south faces and w, that of its east and north neighbours
// the other two).  They need no flags: a zero transport gives the same signed
// zero in the upwind and the Lax-Wendroff form of a flux.  The passes leave the
// levels below the deepest such column of a block of 32 x 4 (dry_from) to
// dry_levels.
__device__ __forceinline__ int flow_end(const Arena& a, long q, int kmt) {
  if (!a.kflow) return a.km;
  return max(max(kmt, a.kflow[q]), max(a.kflow[q + 1], a.kflow[q - a.imt]));
}
// The block's dry_from: one past the deepest flow_end of its ring cells (this
// thread's at q).  wmax: a word per warp.
__device__ __forceinline__ int dry_from(const Arena& a, bool ring, long q, int* wmax) {
  if (!a.kflow) return a.km;
  int v = __reduce_max_sync(0xffffffffu, ring ? flow_end(a, q, a.kmt[q]) : 0);
  __syncthreads();   // wmax is free
  if (threadIdx.x % 32 == 0) wmax[threadIdx.x / 32] = v;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kThT / 32; ++w) v = max(v, wmax[w]);
  return v;
}

// Columns of one block: x0.., y0.., tracer n.  DIAG: with the diagnostics of
// tracer_9 (tend, dt_diff) and the pre-fold values of the top row.
template <bool DIAG>
__device__ __forceinline__ void thomas_block(const Arena& a, const ColumnMaps& maps, bool tma, int x0, int y0, int n) {
  extern __shared__ __align__(128) unsigned char smem_th[];
  ThomasSmem& S = *reinterpret_cast<ThomasSmem*>(smem_th);
  const int tid = threadIdx.x, tx = tid % kThX, ty = tid / kThX;
  const int i = x0 + tx, j = y0 + ty;
  const int imt = a.imt, jmt = a.jmt, km = a.km;
  const long A = a.A;
  const bool inner = i >= 2 && i < imt - 2 && j >= 2 && j < jmt - 2;
  const long q = inner ? (long)j * imt + i : 0;
  const int kz = inner ? a.kmt[q] : 0;
  const int top = __reduce_max_sync(0xffffffffu, kz);
  if (tid % 32 == 0) S.wmax[tid / 32] = top;
  if (tid == 0) {
    for (int s = 0; s < kThStages; ++s) mbar_init(&S.bar[s], kThT);   // one arrival per thread and stage
    mbar_fence_init();
  }
  __syncthreads();
  int kmax = 0;
#pragma unroll
  for (int w = 0; w < kThT / 32; ++w) kmax = max(kmax, S.wmax[w]);

  int kout = kz;   // levels of this column the pass writes
  if (DIAG) {
    const bool ring = i >= 1 && i < imt - 1 && j >= 1 && j < jmt - 1;
    kout = dry_from(a, ring, (long)j * imt + i, S.wmax);
  }

  double* __restrict__ at_out = a.at[a.cur ^ 1] + n * a.F;
  double* __restrict__ atb_out = a.atb[a.cur ^ 1] + n * a.FB;
  const double* __restrict__ at_in = a.at[a.cur] + n * a.F;
  const double* __restrict__ akt = a.akt + n * a.F;
  // stage t holds levels l0(t) .. l0(t)+kThLevels-1, l0(t) = (stages-1-t)*kThLevels
  const int stages = (kmax + kThLevels - 1) / kThLevels;
  auto issue = [&](int t) {
    const int l0 = (stages - 1 - t) * kThLevels, r = t % kThStages;
    ThomasSmem::Slot& sl = S.slot[r];
    if (tma) {
      if (tid == 0) {
        mbar_expect_tx(&S.bar[r], (uint32_t)(kThLevels * kThT * 2 * sizeof(double)));
        // boxes of both tracers' levels: beyond a tracer's last level the box
        // reads its neighbour's levels or zeros, which no column uses
        tma_load_3d(sl.d8, &maps.th_at[a.cur ^ 1], x0, y0, n * km + l0, &S.bar[r]);
        tma_load_3d(sl.akt, &maps.th_akt, x0, y0, n * km + l0 - 1, &S.bar[r]);
      } else {
        mbar_arrive(&S.bar[r]);
      }
    } else {
#pragma unroll
      for (int c = 0; c < kThLevels; ++c) {
        const int k = l0 + c;
        const bool in = inner && k < kz;
        cp_async8z(&sl.d8[c * kThT + tid], at_out + (in ? (long)k * A + q : 0), in);
        const bool ia = in && k >= 1;
        cp_async8z(&sl.akt[c * kThT + tid], akt + (ia ? (long)(k - 1) * A + q : 0), ia);
      }
      cp_async_mbar_arrive(&S.bar[r]);
    }
  };
  for (int t = 0; t < kThStages && t < stages; ++t) issue(t);

  const double dts = a.p.dts;
  const double* __restrict__ odzp = a.odzp;
  const double* __restrict__ odzt = a.odzt;
  double e = 0.0, f = 0.0;                                       // of the level below
  double ak = 0.0;                                               // akt of level k
  const uint64_t keep = l2_evict_last();
  for (int t = 0; t < stages; ++t) {
    const int l0 = (stages - 1 - t) * kThLevels, r = t % kThStages;
    const bool ok = mbar_wait(&S.bar[r], (uint32_t)((t / kThStages) & 1), a.wait_limit);
    if (__syncthreads_or(!ok)) {
      // a wait ran out: record it, let the copies still in flight land
      // (bounded) and leave together
      if (tid == 0) {
        atomicExch(a.status + 1, 1);
        for (int u = t; u < stages && u < t + kThStages; ++u)
          mbar_wait(&S.bar[u % kThStages], (uint32_t)((u / kThStages) & 1));
      }
      __syncthreads();
      return;
    }
    const ThomasSmem::Slot& sl = S.slot[r];
#pragma unroll
    for (int c = kThLevels - 1; c >= 0; --c) {
      const int k = l0 + c;
      if (k >= kz) continue;
      const double d8 = sl.d8[c * kThT + tid], au = sl.akt[c * kThT + tid];
      double a8, c8, b8;
      if (k >= 1) a8 = au * odzt[k] * odzp[k] * dts * 0.5;
      else a8 = odzp[0] * dts * 0.5;
      if (k == kz - 1) {
        c8 = odzp[kz - 1] * dts * 0.5;
        b8 = 1.0 + a8;
      } else {
        c8 = ak * odzt[k + 1] * odzp[k] * dts * 0.5;
        b8 = k >= 1 ? 1.0 + a8 + c8 : 1.0 + c8;
      }
      const double g0 = 1.0 / (b8 - c8 * e);
      e = a8 * g0;
      f = (d8 + c8 * f) * g0;
      ak = au;
      st_l2(at_out + (long)k * A + q, f, keep);
      st_l2(atb_out + (long)(k + 1) * A + q, e, keep);
      if (DIAG) a.dt_diff[n * a.F + (long)k * A + q] = d8;
    }
    __syncthreads();   // the slot is read
    if (t + kThStages < stages) issue(t + kThStages);
  }
  if (!inner) return;

  // substitution, top down: the coefficients of SUB levels are loaded while
  // the SUB levels above are substituted
  const double stf = a.stf_n[n * A + q];
  constexpr int SUB = 8;
  const uint64_t once = l2_evict_first();
  double x = 0.0;
  const int kend = kout;
  double ev[SUB], fv[SUB];
  auto load = [&](int k0) {
#pragma unroll
    for (int c = 0; c < SUB; ++c) {
      const int k = k0 + c;
      ev[c] = k < kz ? ld_l2(atb_out + (long)(k + 1) * A + q, once) : 0.0;
      fv[c] = k < kend ? ld_l2(at_out + (long)k * A + q, once) : 0.0;
    }
  };
  load(0);
  for (int k0 = 0; k0 < kend; k0 += SUB) {
    double ec[SUB], fc[SUB];
#pragma unroll
    for (int c = 0; c < SUB; ++c) {
      ec[c] = ev[c];
      fc[c] = fv[c];
    }
    load(k0 + SUB);
#pragma unroll
    for (int c = 0; c < SUB; ++c) {
      const int k = k0 + c;
      if (k >= kend) break;
      double v = fc[c];
      if (k < kz) v = x = ec[c] * (k == 0 ? stf : x) + fc[c];
      if (DIAG) {
        const long cg = n * a.F + (long)k * A + q;
        const double vit = k < kz ? 1.0 : 0.0;
        const double d8 = k < kz ? a.dt_diff[cg] : v;
        a.tend[cg] = (v - at_in[(long)k * A + q]) / dts * vit;
        if (k == 0) a.dt_diff[cg] = (v - d8) / dts * vit - stf * 0.5 * odzp[0];
        else a.dt_diff[cg] = (v - d8) / dts * vit;
        if (j == 2 && a.tripole) a.fold_save[((long)(n * km + k)) * imt + i] = d8;
      }
      __stcs(at_out + (long)k * A + q, v);
      __stcs(atb_out + (long)(k + 1) * A + q, v);
    }
  }
}

// The dry levels of a block's columns keep their values (with diagnostics the
// sweep and dry_levels write them): eight levels' loads ahead of their stores.
__device__ __forceinline__ void copy_dry(const Arena& a, int x0, int y0, int n) {
  const int i = x0 + threadIdx.x % kThX, j = y0 + threadIdx.x / kThX;
  if (!(i >= 2 && i < a.imt - 2 && j >= 2 && j < a.jmt - 2)) return;
  const long A = a.A, q = (long)j * a.imt + i;
  const int km = a.km;
  const double* __restrict__ src = a.at[a.cur] + n * a.F + q;
  double* __restrict__ at_out = a.at[a.cur ^ 1] + n * a.F + q;
  double* __restrict__ atb_out = a.atb[a.cur ^ 1] + n * a.FB + A + q;
  for (int k0 = a.kmt[q]; k0 < km; k0 += 8) {
    double v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = k0 + c < km ? __ldcs(src + (long)(k0 + c) * A) : 0.0;
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (k0 + c < km) {
        __stcs(at_out + (long)(k0 + c) * A, v[c]);
        __stcs(atb_out + (long)(k0 + c) * A, v[c]);
      }
  }
}

// The levels of a block of columns from dry_from down (every ring cell below
// its bottom, no transport): the diagnostics of advection_tracer_3 (the upwind
// form of each flux), of tracer_5 (penetrate, dz) and of tracer_9 (tend,
// dt_diff, with the value kept: every term is masked) and the new state.
// All signed zeros and copies: bound by memory, so a block takes a chunk of
// levels of both tracers, whose transports it reads once, and nothing is written
// twice.  With such levels in all three passes instead (each read them, the last
// one wrote the explicit pass's value again) a step with diagnostics took 45.1 ms
// at 3600 x 2302 x 55 on the linear depth map and 53.6 on the global area-depth
// curve, with these blocks 33.0 and 49.7; 360 x 218 x 30: 495 and 549 us, now 405
// and 542.  As a launch of its own 31.4 and 49.9 ms, but 419 and 567 us; in the
// explicit pass's launch 40.1 and 51.9 ms.
constexpr int kDryLevels = 16;
__device__ __forceinline__ void dry_levels(const Arena& a, int x0, int y0, int chunk, int* wmax) {
  const int i = x0 + threadIdx.x % kThX, j = y0 + threadIdx.x / kThX;
  const int imt = a.imt, jmt = a.jmt, km = a.km;
  const bool ring = i >= 1 && i < imt - 1 && j >= 1 && j < jmt - 1;
  const bool inner = i >= 2 && i < imt - 2 && j >= 2 && j < jmt - 2;
  const long A = a.A, F = a.F, FB = a.FB;
  const long q = (long)j * imt + i;
  const int from = dry_from(a, ring, q, wmax);
  int k = max(from, chunk * kDryLevels);
  const int kend = min(km, (chunk + 1) * kDryLevels);
  if (!ring || k >= kend) return;
  const double* __restrict__ at_in = a.at[a.cur] + q;
  const double* __restrict__ atb_in = a.atb[a.cur] + A + q;   // level 0
  const double* __restrict__ akt = a.akt + q;
  const double* __restrict__ uwf = a.uwf + q;
  const double* __restrict__ vsf = a.vsf + q;
  const double* __restrict__ ws = a.ws + q;
  double* __restrict__ at_out = a.at[a.cur ^ 1] + q;
  double* __restrict__ atb_out = a.atb[a.cur ^ 1] + A + q;
  const double tr = a.tarea_r[q], swv = inner ? a.swv[q] : 0.0;
  const double inv = 1.0 / a.p.dts, none = 0.0;   // none: the mask below the bottom
  long c = (long)k * A;
  double wk = ws[c];
  double up[2], x[2], bx[2], mix[2];   // at of levels k-1 and k; atb of level k; mixing flux from above
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    x[n] = at_in[n * F + c];
    up[n] = k > 0 ? at_in[n * F + c - A] : 0.0;
    bx[n] = inner ? atb_in[n * FB + c] : 0.0;
    mix[n] = inner && k > 0 ? akt[n * F + c - A] * (atb_in[n * FB + c - A] - bx[n]) * a.odzt[k] * none : 0.0;
  }
  for (; k < kend; ++k, c += A) {
    const bool last = k == km - 1;
    const double odzp = a.odzp[k];
    const double ue = uwf[c + 1], uw = uwf[c], vs = vsf[c], vn = vsf[c - imt];
    const double w1 = last ? 0.0 : ws[c + A];
    double lo[2], e[2], w[2], s[2], nn[2], bl[2], ak[2];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const double* p = at_in + n * F + c;
      e[n] = p[1];
      w[n] = p[-1];
      s[n] = p[imt];
      nn[n] = p[-imt];
      lo[n] = last ? 0.0 : p[A];
      bl[n] = inner && !last ? atb_in[n * FB + c + A] : 0.0;
      ak[n] = inner && !last ? akt[n * F + c] : 0.0;
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const double v = x[n];
      const long cg = n * F + c + q;
      const double xe = -(e[n] - v) * fabs(ue) * tr, xw = (v - w[n]) * fabs(uw) * tr;
      const double ys = -(s[n] - v) * fabs(vs) * tr, yn = (v - nn[n]) * fabs(vn) * tr;
      const double x0v = (e[n] + v) * ue * tr - (v + w[n]) * uw * tr;
      const double y0v = ((s[n] + v) * vs - (v + nn[n]) * vn) * tr;
      const double cx = -v * (ue - uw) * tr * 2.0, cy = -v * (vs - vn) * tr * 2.0;
      double za, zb1 = 0.0, zb2 = 0.0, zc;
      if (k > 0) zb1 = -0.5 * fabs(wk) * odzp * (up[n] - v);
      if (!last) zb2 = 0.5 * fabs(w1) * odzp * (v - lo[n]);
      if (k == 0) {
        za = -0.5 * odzp * w1 * (lo[n] + v);
        zc = odzp * v * w1;
      } else if (last) {
        za = 0.5 * odzp * wk * (v + up[n]);
        zc = -odzp * v * wk;
      } else {
        za = 0.5 * odzp * wk * (v + up[n]) - 0.5 * odzp * w1 * (v + lo[n]);
        zc = -odzp * v * (wk - w1);
      }
      __stcs(a.ax + cg, -(x0v + xe + xw + cx));
      __stcs(a.ay + cg, -(y0v + ys + yn + cy));
      __stcs(a.az + cg, -(za + zb1 + zb2 + zc));
      up[n] = v;
      x[n] = lo[n];
      if (!inner) continue;
      if (n == 0) {
        double pen;
        if (k == 0) pen = -(swv * a.pen[0] * none) * odzp;
        else if (last) pen = swv * a.pen[km - 2] * none * odzp;
        else pen = (swv * a.pen[k - 1] * none - swv * a.pen[k] * none) * odzp;
        __stcs(a.penetrate + c + q, pen);
      }
      const double below = last ? 0.0 : ak[n] * (bx[n] - bl[n]) * a.odzt[k + 1] * none;
      double dz;
      if (k == 0) dz = -odzp * below * 0.5;
      else if (last) dz = odzp * mix[n] * 0.5;
      else dz = odzp * (mix[n] - below) * 0.5;
      __stcs(a.dzd + cg, dz);
      mix[n] = below;
      bx[n] = bl[n];
      const double kept = (v - v) * inv * none;   // no change
      __stcs(a.tend + cg, kept);
      __stcs(a.dt_diff + cg, k == 0 ? kept - a.stf_n[n * A + q] * 0.5 * odzp : kept);
      if (j == 2 && a.tripole) a.fold_save[((long)(n * km + k)) * imt + i] = v;
      __stcs(at_out + n * F + c, v);
      __stcs(atb_out + n * FB + c, v);
    }
    wk = w1;
  }
}

template <bool DIAG>
__global__ void __launch_bounds__(kThT) k_thomas(const __grid_constant__ Arena a, const __grid_constant__ ColumnMaps maps,
                                                 int tma, int parts, int row0) {
  chain_grid();
  // blockIdx.x: the column of tiles and the block's part (the sweep of either
  // tracer, then the dry levels: of either tracer, with diagnostics a chunk of
  // levels of both): the copying blocks only move memory, the sweeping ones
  // mostly wait for their chains of divisions, so the two kinds run side by side
  if (!DIAG) parts = 4;
  const int part = blockIdx.x % parts, x0 = blockIdx.x / parts * kThX, y0 = (row0 + blockIdx.y) * kThY;
  if (part < 2) {
    thomas_block<DIAG>(a, maps, tma != 0, x0, y0, part);
  } else if (DIAG) {
    extern __shared__ __align__(128) unsigned char smem_th[];
    dry_levels(a, x0, y0, part - 2, reinterpret_cast<ThomasSmem*>(smem_th)->wmax);
  } else {
    copy_dry(a, x0, y0, part - 2);
  }
}

// shared-memory size of the pass on the current device (not inside a capture)
inline int prepare_thomas() {
  const int sm = (int)sizeof(ThomasSmem);
  LT_CUDA_OK(cudaFuncSetAttribute(k_thomas<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
  LT_CUDA_OK(cudaFuncSetAttribute(k_thomas<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
  return LT_OK;
}

template <bool DIAG>
int launch_thomas(const Arena& a, const ColumnMaps& maps, bool tma, cudaStream_t s) {
  const size_t sm = sizeof(ThomasSmem);
  const int parts = !DIAG ? 4 : a.kflow ? 2 + (a.km + kDryLevels - 1) / kDryLevels : 2;
  return for_column_rows(a, [&](int r, int rows) {
    return launch_chained(k_thomas<DIAG>, dim3((a.imt + kThX - 1) / kThX * parts, rows), dim3(kThT), sm, s, a, maps,
                          tma ? 1 : 0, parts, r);
  });
}

}  // namespace lt
