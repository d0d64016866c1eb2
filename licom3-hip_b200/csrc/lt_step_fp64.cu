// lt_step_fp64.cu - the plain FP64 tracer step (the drop-in form).
//
// Compiled with -fmad=false: every floating-point expression keeps the
// operation order of the reference kernels it replaces (cited per kernel), so
// results match the FP64 CPU oracle bit for bit.
//
// Launch sequence of one step (replacing tracer.cpp:1701-1903):
//   k_surface       SSH mean (h0f*onbc, stf), surface fluxes of
//                   both tracers, net, the surface mixing floor (tracer_1_0, tracer_5/6 surface parts)
//   k_cont_march64  (small grids: k_cont_levels64, k_cont_columns64) uk/vk,
//                   divergence, w by upward integration, face
//                   transports, scaled utf/vtf                  (tracer_1, upwell_2..4, advection_tracer_1_0)
//   k_sss_norm      deterministic SSS-normalisation sum         (tracer.cpp:1849-1868)
//   k_laplace64, k_limit64, k_explicit64, k_thomas (lt_column_fp64.cu;
//                   k_tracer64 for the centred and flux schemes), both
//                   tracers: tspas predictor/limiter, biharmonic
//                   diffusion, shortwave, explicit and implicit
//                   vertical diffusion, surface terms, update   (advection_tracer_2/3, tracer_del4_1/2,
//                                                                tracer_5..9, invtrit)
//   k_halo_state_parts  ghost fill + fold of the new state and
//                   of net                                      (pop_haloupdate_tracer1/2, tracer_9 for ghosts)
// A step whose forcing is still being copied in starts with k_ssh and the
// continuity, then k_surface_fluxes, the two halves of k_surface.  With
// diagnostics net's ghost cells are a launch before the columns (k_halo_r8) and
// each tracer's state halo one after them (k_halo_state).
#include <cstdio>
#include "lt_common.cuh"
#include "lt_halo.cuh"
#include "lt_tracer_tma.cuh"

namespace lt {

namespace {

__device__ __forceinline__ long q2(int j, int i, int imt) { return (long)j * imt + i; }

// ------------------------------------------------------------------ surface
// One thread per column.  tracer_1_0 (tracer.cpp:1081-1093): h0f*onbc and the
// SSH mean stf; tracer_del4_2's surface floor on akt(T) (tracer.cpp:1315-1317);
// salt flux of tracer_5 (tracer.cpp:1480-1520) and heat flux of tracer_6
// (tracer.cpp:1545-1565) from the previous time level; net (both tracers).
// The SSH part (h0f_out, stf_ssh), which the continuity needs, and the flux
// part, which needs the surface forcing, are separate so that a step can
// run the continuity while its forcing is being copied in.
__device__ __forceinline__ double ssh_col(const Arena& a, long q) {
  const lt_params& p = a.p;
  const double h0 = a.h0f[q] * p.onbc;
  a.h0f_out[q] = h0;
  const double ssh = 0.5 * h0 + 0.5 * a.h0l[q];
  a.stf_ssh[q] = ssh;
  return ssh;
}

__device__ __forceinline__ void flux_col(const Arena& a, int i, int j, long q, double ssh) {
  const lt_params& p = a.p;
  if (q == 0) a.status[kTicket] = 0;   // the column kernel's work items start over
  if (i >= 1 && i < a.imt - 1 && j >= 1 && j < a.jmt - 1) {
    if (a.akt) {
      if (a.akt[q] < p.dwndmix) a.akt[q] = p.dwndmix;
    } else if (a.akt32[q] < (float)p.dwndmix) {
      a.akt32[q] = (float)p.dwndmix;
    }
  }
  double sT = ssh, sS = ssh;
  if (a.kmt[q] > 0) {
    const double* atb = a.atb[a.cur];
    const double odzp0 = a.odzp[0];
    const double s_top = atb[a.FB + a.A + q];
    sS = a.fresh[q] * 34.7 * p.od0 / 1000.0 + p.gamma * (a.sss[q] - s_top) * a.seaice[q] / odzp0 +
         p.gamma * 30.0 / 365.0 / 4.0 * 50.0 * (a.sss[q] - s_top) / odzp0 * (1.0 - a.seaice[q]);
    a.net[a.A + q] = sS * odzp0;
    const double t_top = atb[a.A + q];
    sT = ((a.swv[q] + a.nswv[q]) * p.od0cp + a.seaice[q] * p.gamma * (a.sst[q] - t_top) / odzp0);
    a.net[q] = sT * odzp0;
  }
  a.stf_n[q] = sT;
  a.stf_n[a.A + q] = sS;
}

__device__ __forceinline__ void surface_col(const Arena& a, int i, int j) {
  if (i >= a.imt || j >= a.jmt) return;
  const long q = q2(j, i, a.imt);
  flux_col(a, i, j, q, ssh_col(a, q));
}

// The nudging term of every inner cell of the levels k < ktv, written to
// dt_restore as tracer_7 writes it (land and below-bottom cells included:
// their vit of 0 makes it a signed zero).  It reads only the step's inputs
// (restore_at, the previous time level atb, kmt), so it runs beside the
// column kernel, which adds the same term to the wet cells' tendencies.
// Grid: x over the cells of a level, y the level, z the tracer.
__global__ void k_assm_dt_restore(Arena a) {
  const int k = blockIdx.y, n = blockIdx.z;
  const int imt = a.imt, jmt = a.jmt;
  const long A = a.A, F = a.F, FB = a.FB;
  const double rate = assm_rate(k);
  const double* atb = a.atb[a.cur] + n * FB + (long)(k + 1) * A;
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < A; q += (long)gridDim.x * blockDim.x) {
    const int j = (int)(q / imt), i = (int)(q % imt);
    if (j < 2 || j >= jmt - 2 || i < 2 || i >= imt - 2) continue;
    const double vit = k < a.kmt[q] ? 1.0 : 0.0;
    const long c = n * F + (long)k * A + q;
    a.dt_restore[c] = vit * (a.restore_at[c] - atb[q]) * rate;
  }
}

__global__ void k_ssh(Arena a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= a.imt || j >= a.jmt) return;
  ssh_col(a, q2(j, i, a.imt));
}

__global__ void k_surface_fluxes(Arena a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= a.imt || j >= a.jmt) return;
  const long q = q2(j, i, a.imt);
  flux_col(a, i, j, q, a.stf_ssh[q]);
}

// both, where the forcing is already there
__global__ void k_surface(const __grid_constant__ Arena a) {
  chain_grid();
  surface_col(a, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.y * blockDim.y + threadIdx.y);
}

// every member's columns in one launch: blockIdx.z is the member
__global__ void k_surface_batch(const MemberDesc* __restrict__ mem) {
  surface_col(mem[blockIdx.z].a, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.y * blockDim.y + threadIdx.y);
}

// --------------------------------------------------------- deterministic sum
// Fixed binary tree: blocks of 2048 consecutive terms, pairs (t, t+stride) for
// stride = 1024..1, zero padding; repeated on the block sums until one value.
constexpr int RB = 1024;

template <class Term>
__device__ __forceinline__ void tree_block(const Term& term, long n, double* part, long blk) {
  __shared__ double s[2 * RB];
  const long base = blk * 2 * RB;
  const int t = threadIdx.x;
  s[t] = (base + t < n) ? term(base + t) : 0.0;
  s[t + RB] = (base + t + RB < n) ? term(base + t + RB) : 0.0;
  for (int stride = RB; stride > 0; stride >>= 1) {
    __syncthreads();
    if (t < stride) s[t] = s[t] + s[t + stride];
  }
  if (t == 0) part[blk] = s[0];
}

template <class Term>
__global__ void k_tree_first(Term term, long n, double* part) {
  tree_block(term, n, part, blockIdx.x);
}

struct ArrayTerm {
  const double* x;
  __device__ double operator()(long m) const { return x[m]; }
};

// SSS-norm term of interior column m (row-major over j=2..jmt-3, i=2..imt-3):
// tarea*net(S)*vit(k=0) (tracer.cpp:1522-1525)
struct SssTerm {
  const double* tarea;
  const double* net_s;
  const int* kmt;
  int nx, imt;
  __device__ double operator()(long m) const {
    const int j = 2 + (int)(m / nx), i = 2 + (int)(m % nx);
    const long q = (long)j * imt + i;
    return tarea[q] * net_s[q] * (kmt[q] > 0 ? 1.0 : 0.0);
  }
};

// The whole sum and fw_norm2 in one launch: the last block to finish its part
// (counted in a.status[kSssDone], which it clears again) takes the tree's
// further passes over the block sums, which are few: the same fixed tree, so
// the same bits, without a launch per pass, a copy of the result and a launch
// to finish it (about 12 us of a small grid's step).
struct PartTerm {   // block sums of other blocks of this launch: past L1
  const double* x;
  __device__ double operator()(long m) const { return __ldcg(x + m); }
};
__global__ void k_sss_norm(const __grid_constant__ Arena a) {
  chain_grid();
  long n = (long)a.nx * a.ny, nb = gridDim.x;
  tree_block(SssTerm{a.tarea, a.net + a.A, a.kmt, a.nx, a.imt}, n, a.red_part, blockIdx.x);
  __shared__ int last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(a.status + kSssDone, 1) == (int)nb - 1;
  }
  __syncthreads();
  if (!last) return;
  double* cur = a.red_part;
  while (nb > 1) {
    __threadfence();
    double* nxt = cur + nb;
    n = nb;
    nb = (n + 2 * RB - 1) / (2 * RB);
    for (long blk = 0; blk < nb; ++blk) {
      tree_block(PartTerm{cur}, n, nxt, blk);
      __syncthreads();   // the block's sums and its shared array are free again
    }
    cur = nxt;
  }
  if (threadIdx.x == 0) {
    const double sum = *cur;
    a.scalars[4] = sum;
    a.scalars[0] = -sum / a.p.area_t;
    a.status[kSssDone] = 0;
  }
}

// The same tree for every member of a batch, pass by pass: pass 0 sums the
// member's SSS terms into its red_part, pass p > 0 the block sums of pass
// p-1; blockIdx.y is the member, blocks beyond a member's count at this pass
// (or members whose tree ended) leave at once.
__device__ __forceinline__ long tree_blocks(long n) {
  const long nb = (n + 2 * RB - 1) / (2 * RB);
  return nb < 1 ? 1 : nb;
}

__global__ void k_sss_tree_batch(const MemberDesc* __restrict__ mem, int pass) {
  const Arena& a = mem[blockIdx.y].a;
  long n = (long)a.nx * a.ny, nb = tree_blocks(n), off = 0;
  for (int q = 0; q < pass; ++q) {
    if (nb <= 1) return;
    off += nb;
    n = nb;
    nb = tree_blocks(n);
  }
  if ((long)blockIdx.x >= nb) return;
  if (pass == 0) tree_block(SssTerm{a.tarea, a.net + a.A, a.kmt, a.nx, a.imt}, n, a.red_part, blockIdx.x);
  else tree_block(ArrayTerm{a.red_part + off - n}, n, a.red_part + off, blockIdx.x);
}

// the member's total (the last pass's single block sum) and fw_norm2
__global__ void k_finish_sss_batch(const MemberDesc* __restrict__ mem, int nmem) {
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  if (z >= nmem) return;
  const Arena& a = mem[z].a;
  long nb = tree_blocks((long)a.nx * a.ny), off = 0;
  while (nb > 1) { off += nb; nb = tree_blocks(nb); }
  const double sum = a.red_part[off];
  a.scalars[4] = sum;
  a.scalars[0] = -sum / a.p.area_t;
}

template <class Term>
int tree_sum(Term term, long n, double* part, double* out, cudaStream_t s) {
  long nb = (n + 2 * RB - 1) / (2 * RB);
  if (nb < 1) nb = 1;
  k_tree_first<<<(unsigned)nb, RB, 0, s>>>(term, n, part);
  LT_LAUNCHED();
  double* cur = part;
  double* nxt = part + nb;
  while (nb > 1) {
    const long nb2 = (nb + 2 * RB - 1) / (2 * RB);
    k_tree_first<<<(unsigned)nb2, RB, 0, s>>>(ArrayTerm{cur}, nb, nxt);
    LT_LAUNCHED();
    cur = nxt;
    nxt = nxt + nb2;
    nb = nb2;
  }
  LT_CUDA_OK(cudaMemcpyAsync(out, cur, sizeof(double), cudaMemcpyDeviceToDevice, s));
  return LT_OK;
}

// ------------------------------------------------------------------ halo
// In-place ghost fill of nz levels (e.g. net), one block per level.
__device__ __forceinline__ void halo_r8_level(double* lvl, int imt, int jmt, int ew_cyclic, int tripole) {
  extern __shared__ double top[];
  for (int i = threadIdx.x; i < imt; i += blockDim.x) top[i] = lvl[2L * imt + i];
  __syncthreads();
  HaloCells hc{imt, jmt, tripole};
  const long nc = hc.count();
  for (long m = threadIdx.x; m < nc; m += blockDim.x) {
    int j, i;
    hc.cell(m, j, i);
    double v;
    if (halo_cell_value(lvl, top, j, i, imt, jmt, ew_cyclic, tripole, v)) lvl[(long)j * imt + i] = v;
  }
}

// A level's ghost cells spread over kHaloParts blocks (one block per level
// left most SMs idle: 55 blocks per tracer, each thread walking ~120 cells
// in turn).  With the fold, part 0 takes rows 0..2 (the only cells that read
// the staged top row, and the only ones that rewrite it; rows 0 and 1 read
// interior columns of rows 3 and 4, which no part rewrites) and the other
// parts share the rest; without it the parts share all cells.
constexpr int kHaloParts = 8;
__device__ __forceinline__ bool halo_part(long nc, int imt, int tripole, int part, long& m0, long& m1) {
  long base = 0, parts = kHaloParts;
  if (tripole) {
    if (part == 0) { m0 = 0; m1 = 3L * imt; return true; }
    base = 3L * imt;
    parts = kHaloParts - 1;
    part -= 1;
  }
  const long per = (nc - base + parts - 1) / parts;
  m0 = base + part * per;
  m1 = m0 + per < nc ? m0 + per : nc;
  return m0 < m1;
}

// part blockIdx.x of one level
__device__ __forceinline__ void halo_r8_part(double* lvl, int imt, int jmt, int ew_cyclic, int tripole) {
  HaloCells hc{imt, jmt, tripole};
  long m0, m1;
  if (!halo_part(hc.count(), imt, tripole, blockIdx.x, m0, m1)) return;
  extern __shared__ double top[];
  const bool fold = tripole && blockIdx.x == 0;
  if (fold) {
    for (int i = threadIdx.x; i < imt; i += blockDim.x) top[i] = lvl[2L * imt + i];
    __syncthreads();
  }
  for (long m = m0 + threadIdx.x; m < m1; m += blockDim.x) {
    int j, i;
    hc.cell(m, j, i);
    double v;
    if (halo_cell_value(lvl, top, j, i, imt, jmt, ew_cyclic, tripole, v)) lvl[(long)j * imt + i] = v;
  }
}

// part blockIdx.x of level blockIdx.y
__global__ void k_halo_r8(double* f, int imt, int jmt, int ew_cyclic, int tripole) {
  halo_r8_part(f + (long)blockIdx.y * imt * jmt, imt, jmt, ew_cyclic, tripole);
}

// net (both tracers) of every member: blockIdx.x the level, blockIdx.y the member
__global__ void k_halo_net_batch(const MemberDesc* __restrict__ mem) {
  const Arena& a = mem[blockIdx.y].a;
  halo_r8_level(a.net + (long)blockIdx.x * a.A, a.imt, a.jmt, a.ew_cyclic, a.tripole);
}

// ------------------------------------------------------------- continuity
constexpr int kCont64TileY = 8;   // tile height of the FP64 continuity march (4: slower)

// Continuity as one level march per 32 x BY tile (tracer_1, upwell_2,
// operators_div, advection_tracer_1_0 and upwell_3/4 with the same
// expressions in the same order).  The U-point velocities of the tile and a
// one-point halo north and east go through a three-level staging ring filled
// by per-thread asynchronous copies, so three levels are in flight while one
// is computed; each thread converts the points it copied itself (mean
// velocities wkd, wkb and the free-surface scaled uk, vk, whose level-free
// factor it keeps in registers) into a double-buffered level, read by all
// after the step's one barrier.  Each thread's first copy is its own cell's
// point, so the scaled utf, vtf it writes come from its own staged copies
// (a global re-read of them per level cost 9.00 -> 7.67 ms per 0.1-degree
// step).  The column divergence W accumulates in level order during the
// march; w is integrated upward afterwards from the wka the march wrote.
template <int BY>
__global__ void __launch_bounds__(32 * BY) k_cont_march64(const __grid_constant__ Arena a) {
  chain_grid();
  constexpr int BX = 32, UX = BX + 1, UY = BY + 1, UN = UX * UY, NT = BX * BY;
  constexpr int NPT = (UN + NT - 1) / NT, NST = 3;
  __shared__ double s_st[NST][4][UN];   // staged utf, utl, vtf, vtl of three levels
  __shared__ double s_wkd[2][UN], s_wkb[2][UN], s_uk[2][UN], s_vk[2][UN];
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * BX + tx;
  const int x0 = blockIdx.x * BX, y0 = blockIdx.y * BY;
  const int imt = a.imt, jmt = a.jmt, km = a.km;
  const long A = a.A;
  const lt_params& p = a.p;
  static_assert(NPT == 2 && UN - NT == UX + BY, "own point plus one of the row above or the column east");
  // region point of this thread's copy pt: its own cell's U point first (so
  // that the own point's raw velocities are this thread's own copies, read
  // without a barrier), then one point of the row above the tile (threads
  // 0 .. UX-1) or of the column east of it (threads UX .. UX+BY-1)
  auto point_of = [&](int pt) {
    if (pt == 0) return (ty + 1) * UX + tx;
    return tid < UX ? tid : (tid - UX + 1) * UX + BX;
  };
  const bool has_extra = tid < UX + BY;
  long rq[NPT];
  bool rin[NPT], rok[NPT];
  double rfac[NPT];
#pragma unroll
  for (int pt = 0; pt < NPT; ++pt) {
    const int m = point_of(pt);
    const int uj = y0 - 1 + m / UX, ui = x0 + m % UX;
    rin[pt] = (pt == 0 || has_extra) && uj >= 0 && uj < jmt && ui < imt;
    rq[pt] = rin[pt] ? q2(uj, ui, imt) : 0;
    rok[pt] = rin[pt] && uj < jmt - 1 && ui >= 1;
    rfac[pt] = 0.0;
    if (rok[pt]) {
      const long q = rq[pt];
      const double work = a.au0[q] * a.stf_ssh[q] + a.aus[q] * a.stf_ssh[q + imt] +
                          a.auw[q] * a.stf_ssh[q - 1] + a.ausw[q] * a.stf_ssh[q + imt - 1];
      rfac[pt] = 1.0 + work * a.ohbu[q];
    }
  }
  auto issue = [&](int L) {
    if (L < km) {
      const long lvl = (long)L * A;
#pragma unroll
      for (int pt = 0; pt < NPT; ++pt) {
        if (!rin[pt]) continue;
        const int m = point_of(pt);
        const long c = lvl + rq[pt];
        double(*st)[UN] = s_st[L % NST];
        cp_async8(&st[0][m], a.utf + c);
        cp_async8(&st[1][m], a.utl + c);
        cp_async8(&st[2][m], a.vtf + c);
        cp_async8(&st[3][m], a.vtl + c);
      }
    }
    cp_async_commit();
  };
  // the points this thread copied, level L, into buffer b; the own point's
  // raw utf, vtf of level L into own_utf, own_vtf
  double own_utf = 0.0, own_vtf = 0.0;
  auto park = [&](int L, int b) {
    const double(*st)[UN] = s_st[L % NST];
#pragma unroll
    for (int pt = 0; pt < NPT; ++pt) {
      if (pt > 0 && !has_extra) continue;
      const int m = point_of(pt);
      if (pt == 0) {
        own_utf = rin[0] ? st[0][m] : 0.0;
        own_vtf = rin[0] ? st[2][m] : 0.0;
      }
      double wkd = 0.0, wkb = 0.0, uk = 0.0, vk = 0.0;
      if (rin[pt]) {
        wkd = 0.5 * (st[0][m] * p.oncc) + 0.5 * st[1][m];
        wkb = 0.5 * (st[2][m] * p.oncc) + 0.5 * st[3][m];
        if (rok[pt]) {
          uk = rfac[pt] * wkd;
          vk = rfac[pt] * wkb;
        }
      }
      s_wkd[b][m] = wkd; s_wkb[b][m] = wkb; s_uk[b][m] = uk; s_vk[b][m] = vk;
    }
  };
  issue(0);
  issue(1);
  issue(2);
  cp_async_wait<2>();
  park(0, 0);
  const int i = x0 + tx, j = y0 + ty;
  const bool own = i < imt && j < jmt;
  const bool col = own && j >= 1 && j < jmt - 1 && i >= 1 && i < imt - 1;
  const long qo = own ? q2(j, i, imt) : 0;
  const int kz = own ? a.kmt[qo] : 0;
  const double htw_o = own ? a.htw[qo] : 0.0, hts_o = own ? a.hts[qo] : 0.0;
  const double htw_e = (own && i < imt - 1) ? a.htw[qo + 1] : 0.0;
  const double hts_n = (own && j >= 1) ? a.hts[qo - imt] : 0.0;
  // flux scheme: each U-point mean weighted by its own dyu (west face) or
  // dxu (south face) before the face mean (advection_tracer_1_0, Str 1)
  const bool flux = p.adv_tracer == LT_ADV_FLUX;
  const double dyu_o = (flux && own) ? a.dyu[qo] : 0.0, dyu_n = (flux && own && j >= 1) ? a.dyu[qo - imt] : 0.0;
  const double dxu_o = (flux && own) ? a.dxu[qo] : 0.0, dxu_e = (flux && own && i < imt - 1) ? a.dxu[qo + 1] : 0.0;
  const double trr = own ? a.tarea_r[qo] : 0.0;
  const int m0 = (ty + 1) * UX + tx, mn = ty * UX + tx;
  double W = 0.0;
  int kf = 0;   // one past the deepest level with a nonzero west or south face transport or w here
  double dzp_k = a.dzp[0];
  for (int k = 0; k < km; ++k) {
    const int b = k & 1;
    const double dzp_c = dzp_k;
    if (k + 1 < km) dzp_k = a.dzp[k + 1];
    // level k parked by every thread; buffer b^1 and the staging slot of
    // level k are no longer read
    __syncthreads();
    issue(k + 3);
    if (own) {
      const double* wd = s_wkd[b];
      const double* wb = s_wkb[b];
      const double* uk = s_uk[b];
      const double* vk = s_vk[b];
      const long c = (long)k * A + qo;
      __stcs(a.utf_out + c, own_utf * p.oncc);
      __stcs(a.vtf_out + c, own_vtf * p.oncc);
      // the faces outside these ranges stay zero
      double uwv = 0.0, vsv = 0.0;
      if (flux) {
        if (j >= 1 && j < jmt - 1) __stcs(a.uwf + c, uwv = (wd[mn] * dyu_n + wd[m0] * dyu_o) * 0.25);
        if (i >= 1 && i < imt - 1) __stcs(a.vsf + c, vsv = (wb[m0] * dxu_o + wb[m0 + 1] * dxu_e) * 0.25);
      } else {
        if (j >= 1 && j < jmt - 1) __stcs(a.uwf + c, uwv = (wd[mn] + wd[m0]) * htw_o * 0.25);
        if (i >= 1 && i < imt - 1) __stcs(a.vsf + c, vsv = (wb[m0] + wb[m0 + 1]) * hts_o * 0.25);
      }
      if (uwv != 0.0 || vsv != 0.0) kf = k + 1;
      double wka = 0.0;
      if (j >= 1 && i < imt - 1 && k <= kz - 1) {
        const double east = (uk[m0 + 1] + uk[mn + 1]) * htw_e;
        const double west = (uk[m0] + uk[mn]) * htw_o;
        const double south = (vk[m0 + 1] + vk[m0]) * hts_o;
        const double north = (vk[mn + 1] + vk[mn]) * hts_n;
        wka = 0.5 * (east - west + south - north) * trr;
      }
      st_l2(a.wka + c, wka, l2_evict_last());
      if (col) W = W - dzp_c * wka * (k < kz ? 1.0 : 0.0);
    }
    if (k + 1 < km) {
      cp_async_wait<2>();   // this thread's copies of level k+1 have landed
      park(k + 1, b ^ 1);
    }
  }
  cp_async_wait<0>();
  if (!col) {
    if (a.kflow && own) a.kflow[qo] = kf;
    return;
  }
  const double ohbt = a.ohbt[qo];
  const double fac = 1.0 / (1.0 + a.stf_ssh[qo] * ohbt);
  double wsp = a.ws[qo];
  // upward integration; the wka of CH levels are loaded together ahead of
  // their stores (one round trip per CH levels).  The march wrote wka with
  // an L2 evict-last policy (the tile's levels stay in L2 until read here,
  // then leave it); the outputs go out as streaming stores.
  constexpr int CH = 8;
  for (int k0 = 1; k0 < km; k0 += CH) {
    double wk[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) wk[c] = k0 + c < km ? ld_l2(a.wka + (long)(k0 + c - 1) * A + qo, l2_evict_first()) : 0.0;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int k = k0 + c;
      if (k >= km) break;
      const double raw = (k < kz ? 1.0 : 0.0) * (wsp + a.dzp[k - 1] * (W * ohbt + wk[c]));
      const double wv = raw * fac;
      __stcs(a.ws + (long)k * A + qo, wv);
      if (wv != 0.0) kf = max(kf, k + 1);
      wsp = raw;
    }
  }
  if (a.kflow) a.kflow[qo] = kf;
}

// The same continuity for grids whose tiles do not fill the GPU, where the
// march is a chain of km levels on a few SMs: first every level at once
// (k_cont_levels64: face transports, scaled velocities, divergence; the
// neighbours' velocities come through L1), then the two sums of each column
// (k_cont_columns64).  Same expressions in the same order.
// 36 x 40 x 55: 21 us of a step, with the march (and the SSH mean's launch) 59.
constexpr int kContChunk = 4;   // levels per thread of k_cont_levels64
__global__ void __launch_bounds__(256) k_cont_levels64(const __grid_constant__ Arena a) {
  chain_grid();
  const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y;
  const int imt = a.imt, jmt = a.jmt;
  if (i >= imt || j >= jmt) return;
  const long A = a.A, q = q2(j, i, imt);
  const lt_params& p = a.p;
  const bool north = j >= 1, east = i < imt - 1;
  // the free-surface factor at a U point where uk, vk are formed (elsewhere
  // they are zero)
  auto formed = [&](int uj, int ui) { return uj >= 0 && uj < jmt - 1 && ui >= 1 && ui < imt; };
  auto factor = [&](int uj, int ui) {
    if (!formed(uj, ui)) return 0.0;
    const long c = q2(uj, ui, imt);
    const double work = a.au0[c] * a.stf_ssh[c] + a.aus[c] * a.stf_ssh[c + imt] + a.auw[c] * a.stf_ssh[c - 1] +
                        a.ausw[c] * a.stf_ssh[c + imt - 1];
    return 1.0 + work * a.ohbu[c];
  };
  const bool u0 = formed(j, i), un = formed(j - 1, i), u1 = formed(j, i + 1), un1 = formed(j - 1, i + 1);
  const bool div = north && east;
  const int kz = a.kmt[q];
  const double f0 = factor(j, i), fn = factor(j - 1, i), f1 = factor(j, i + 1), fn1 = factor(j - 1, i + 1);
  const double htw_o = a.htw[q], hts_o = a.hts[q];
  const double htw_e = east ? a.htw[q + 1] : 0.0, hts_n = north ? a.hts[q - imt] : 0.0;
  const bool flux = p.adv_tracer == LT_ADV_FLUX;
  const double dyu_o = flux ? a.dyu[q] : 0.0, dyu_n = flux && north ? a.dyu[q - imt] : 0.0;
  const double dxu_o = flux ? a.dxu[q] : 0.0, dxu_e = flux && east ? a.dxu[q + 1] : 0.0;
  const double trr = a.tarea_r[q];
  const double* __restrict__ utf = a.utf;
  const double* __restrict__ utl = a.utl;
  const double* __restrict__ vtf = a.vtf;
  const double* __restrict__ vtl = a.vtl;
  const int k0 = blockIdx.z * kContChunk;
#pragma unroll
  for (int d = 0; d < kContChunk; ++d) {
    const int k = k0 + d;
    if (k >= a.km) break;
    const long c = (long)k * A + q;
    // mean velocities of the four U points: here, north, east, north-east
    // (zero outside the domain)
    double wd[4], wb[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const bool in = (!(m & 1) || north) && (!(m & 2) || east);
      const long u = c - (m & 1 ? imt : 0) + (m & 2 ? 1 : 0);
      wd[m] = in ? 0.5 * (utf[u] * p.oncc) + 0.5 * utl[u] : 0.0;
      wb[m] = in ? 0.5 * (vtf[u] * p.oncc) + 0.5 * vtl[u] : 0.0;
    }
    a.utf_out[c] = utf[c] * p.oncc;
    a.vtf_out[c] = vtf[c] * p.oncc;
    if (flux) {
      if (j >= 1 && j < jmt - 1) a.uwf[c] = (wd[1] * dyu_n + wd[0] * dyu_o) * 0.25;
      if (i >= 1 && i < imt - 1) a.vsf[c] = (wb[0] * dxu_o + wb[2] * dxu_e) * 0.25;
    } else {
      if (j >= 1 && j < jmt - 1) a.uwf[c] = (wd[1] + wd[0]) * htw_o * 0.25;
      if (i >= 1 && i < imt - 1) a.vsf[c] = (wb[0] + wb[2]) * hts_o * 0.25;
    }
    double wka = 0.0;
    if (div && k <= kz - 1) {
      const double uk0 = u0 ? f0 * wd[0] : 0.0, ukn = un ? fn * wd[1] : 0.0;
      const double uk1 = u1 ? f1 * wd[2] : 0.0, ukn1 = un1 ? fn1 * wd[3] : 0.0;
      const double vk0 = u0 ? f0 * wb[0] : 0.0, vkn = un ? fn * wb[1] : 0.0;
      const double vk1 = u1 ? f1 * wb[2] : 0.0, vkn1 = un1 ? fn1 * wb[3] : 0.0;
      const double e = (uk1 + ukn1) * htw_e;
      const double w = (uk0 + ukn) * htw_o;
      const double s = (vk1 + vk0) * hts_o;
      const double n = (vkn1 + vkn) * hts_n;
      wka = 0.5 * (e - w + s - n) * trr;
    }
    a.wka[c] = wka;
  }
}

__global__ void __launch_bounds__(128) k_cont_columns64(const __grid_constant__ Arena a) {
  chain_grid();
  const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 4 + threadIdx.y;
  const int imt = a.imt, km = a.km;
  if (!(j >= 1 && j < a.jmt - 1 && i >= 1 && i < imt - 1)) return;
  const long A = a.A, q = q2(j, i, imt);
  const int kz = a.kmt[q];
  const double* __restrict__ wka = a.wka + q;
  const double* __restrict__ dzp = a.dzp;
  constexpr int CH = 8;
  double W = 0.0;
  for (int k0 = 0; k0 < km; k0 += CH) {
    double w[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) w[c] = k0 + c < km ? wka[(long)(k0 + c) * A] : 0.0;
#pragma unroll
    for (int c = 0; c < CH; ++c)
      if (k0 + c < km) W = W - dzp[k0 + c] * w[c] * (k0 + c < kz ? 1.0 : 0.0);
  }
  const double ohbt = a.ohbt[q];
  const double fac = 1.0 / (1.0 + a.stf_ssh[q] * ohbt);
  double wsp = a.ws[q];
  double* __restrict__ ws = a.ws + q;
  for (int k0 = 1; k0 < km; k0 += CH) {
    double w[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) w[c] = k0 + c < km ? wka[(long)(k0 + c - 1) * A] : 0.0;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int k = k0 + c;
      if (k >= km) break;
      const double raw = (k < kz ? 1.0 : 0.0) * (wsp + dzp[k - 1] * (W * ohbt + w[c]));
      ws[(long)k * A] = raw * fac;
      wsp = raw;
    }
  }
}

// ------------------------------------------- plain-load march (centred, flux)
// The column march of the centred and flux advection schemes (no predictor
// or limiter), with each level's region loaded by plain loads.
// Shared-memory regions of a TX x TY column tile:
//   H2: rows y0-2..y0+TY+1, cols x0-2..x0+TX+1   (RY x RX)   tracer, atb, kmt
//   H1: rows y0-1..y0+TY,   cols x0-1..x0+TX     (QY x QX)   w, d2tk
constexpr int RX = TX + 4, RY = TY + 4, QX = TX + 2, QY = TY + 2;
constexpr int UWN = QY * RX;          // u_wface: H1 rows, cols x0-2..x0+TX+1
constexpr int VSN = (QY + 1) * QX;    // v_sface: rows y0-2..y0+TY, H1 cols

struct TSmem {
  double at[4][RY * RX];
  double ws[3][QY * QX];
  double uw[2][UWN], vs[2][VSN];
  double atb[RY * RX];
  double d2[QY * QX];
  double tr[QY * QX];
  double dtn[QY * QX], dts[QY * QX], dte[QY * QX], dtw[QY * QX], ahf[QY * QX];
  int kmt[RY * RX];
};

__device__ __forceinline__ int slot4(int k) { return k & 3; }
__device__ __forceinline__ int slot3(int k) { return k % 3; }

// load one level of a [km][jmt][imt] field over region rows r0.., cols c0..
// (ny x nxr), zero outside the domain
__device__ __forceinline__ void load_region(double* dst, const double* lvl, int r0, int c0, int nyr, int nxr,
                                            int imt, int jmt) {
  for (int m = threadIdx.x; m < nyr * nxr; m += TTHREADS) {
    const int gj = r0 + m / nxr, gi = c0 + m % nxr;
    dst[m] = (gj >= 0 && gj < jmt && gi >= 0 && gi < imt) ? lvl[(long)gj * imt + gi] : 0.0;
  }
}

// first masked Laplacian of atb at level kk on H1 (tracer_del4_1, tracer.cpp:1238-1293)
__device__ void del4_first(TSmem& S, const Arena& a, int kk, int x0, int y0) {
  for (int m = threadIdx.x; m < QY * QX; m += TTHREADS) {
    const int hj = m / QX, hi = m % QX;
    const int gj = y0 - 1 + hj, gi = x0 - 1 + hi;
    if (!(gi >= 1 && gi < a.imt - 1 && gj >= 1 && gj < a.jmt - 1)) { S.d2[m] = 0.0; continue; }
    const int r = (hj + 1) * RX + (hi + 1);
    double h = 0.0, cc = 0.0;
    if (kk <= S.kmt[r] - 1) {
      if (kk <= S.kmt[r - RX] - 1) { h += S.dtn[m] * S.atb[r - RX]; cc -= S.dtn[m]; }
      if (kk <= S.kmt[r + RX] - 1) { h += S.dts[m] * S.atb[r + RX]; cc -= S.dts[m]; }
      if (kk <= S.kmt[r + 1] - 1) { h += S.dte[m] * S.atb[r + 1]; cc -= S.dte[m]; }
      if (kk <= S.kmt[r - 1] - 1) { h += S.dtw[m] * S.atb[r - 1]; cc -= S.dtw[m]; }
    }
    S.d2[m] = S.ahf[m] * (cc * S.atb[r] + h);
  }
}

// advection_tracer_1 for the centred (Str 0) and flux (Str 1) schemes at one
// inner cell of level k (tracer.cpp:120-289), from the tile's level slots.
// The centred form accumulates ax, ay, az with weight 1/nss, once per level
// (the reference repeats its top- and bottom-level statements in every
// level thread of its launch, so there those two levels' accumulations race).
template <int ADV, bool DIAG>
__device__ __forceinline__ double simple_adv(const TSmem& S, const Arena& a, int k, int n, long cg, int rc, int hc,
                                             int uc, int vc, const double* at_c, const double* at_u,
                                             const double* at_d) {
  const int km = a.km;
  const double* odzp = a.odzp;
  const double tr = S.tr[hc];
  const double c = at_c[rc], e = at_c[rc + 1], w = at_c[rc - 1], s = at_c[rc + RX], nn = at_c[rc - RX];
  const double* uw = S.uw[k & 1];
  const double* vs = S.vs[k & 1];
  const double ue = uw[uc + 1], uwc = uw[uc], vsc = vs[vc], vn = vs[vc - QX];
  const double wk = S.ws[slot3(k)][hc];
  const double w1 = k < km - 1 ? S.ws[slot3(k + 1)][hc] : 0.0;
  if (ADV == LT_ADV_CENTERED) {
    const double h = (-uwc * (c - w) - ue * (e - c) - vsc * (s - c) - vn * (c - nn)) * tr;
    double z;
    if (k == 0) z = 0.5 * odzp[0] * (w1 * (c - at_d[rc]));
    else if (k == km - 1) z = 0.5 * odzp[km - 1] * (wk * (at_u[rc] - c));
    else z = 0.5 * odzp[k] * (wk * (at_u[rc] - c) + w1 * (c - at_d[rc]));
    if (DIAG) {
      const long q = (long)n * a.F + cg;
      const double nss = (double)a.p.nss;
      a.ax[q] = a.ax[q] + (-uwc * (c - w) - ue * (e - c)) * tr / nss;
      a.ay[q] = a.ay[q] + (-vsc * (s - c) - vn * (c - nn)) * tr / nss;
      a.az[q] = a.az[q] - z / nss;
    }
    return h - z;
  } else {
    const double h = (-uwc * (c + w) + ue * (e + c) - vn * (c + nn) + vsc * (s + c)) * tr;
    const double z1 = k == 0 ? 0.0 : wk * (at_u[rc] + c) * 0.5;
    const double z2 = k == km - 1 ? 0.0 : w1 * (c + at_d[rc]) * 0.5;
    return h - odzp[k] * (z2 - z1);
  }
}

template <bool DIAG, int ADV>
__global__ void __launch_bounds__(TTHREADS) k_tracer64(Arena a, int ntx, long ntiles) {
  static_assert(ADV == LT_ADV_CENTERED || ADV == LT_ADV_FLUX, "the tspas scheme runs in lt_column_fp64.cu");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TSmem& S = *reinterpret_cast<TSmem*>(smem_raw);
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int imt = a.imt, jmt = a.jmt, km = a.km;
  const long A = a.A, F = a.F, FB = a.FB;
  const lt_params& p = a.p;
  const double dts = p.dts;
  const double aidif = 0.5;
  const double* __restrict__ odzp = a.odzp;
  const double* __restrict__ odzt = a.odzt;
  const int NV = a.nv_scratch;
  double* scr = a.col_scratch + (long)blockIdx.x * km * NV * TTHREADS;

  for (long w = blockIdx.x; w < 2 * ntiles; w += gridDim.x) {
    const long tile = w >> 1;
    const int n = (int)(w & 1);
    const int x0 = (int)(tile % ntx) * TX, y0 = (int)(tile / ntx) * TY;
    const int i = x0 + tx, j = y0 + ty;
    const double* at_in = a.at[a.cur] + n * F;
    const double* atb_in = a.atb[a.cur] + n * FB;
    double* at_out = a.at[a.cur ^ 1] + n * F;
    double* atb_out = a.atb[a.cur ^ 1] + n * FB;
    const double* akt = a.akt + n * F;

    __syncthreads();  // previous tile finished with shared memory
    // ---- per-tile 2-D statics
    for (int m = tid; m < RY * RX; m += TTHREADS) {
      const int gj = y0 - 2 + m / RX, gi = x0 - 2 + m % RX;
      S.kmt[m] = (gj >= 0 && gj < jmt && gi >= 0 && gi < imt) ? a.kmt[q2(gj, gi, imt)] : 0;
    }
    for (int m = tid; m < QY * QX; m += TTHREADS) {
      const int gj = y0 - 1 + m / QX, gi = x0 - 1 + m % QX;
      const bool in = (gj >= 0 && gj < jmt && gi >= 0 && gi < imt);
      const long q = in ? q2(gj, gi, imt) : 0;
      S.tr[m] = in ? a.tarea_r[q] : 0.0;
      S.dtn[m] = in ? a.dtn[q] : 0.0;
      S.dts[m] = in ? a.dts[q] : 0.0;
      S.dte[m] = in ? a.dte[q] : 0.0;
      S.dtw[m] = in ? a.dtw[q] : 0.0;
      S.ahf[m] = in ? a.ahf[q] : 0.0;
    }
    // ---- prologue: levels km-1 and km-2 of the tracer, w and faces at km-1
    load_region(S.at[slot4(km - 1)], at_in + (long)(km - 1) * A, y0 - 2, x0 - 2, RY, RX, imt, jmt);
    load_region(S.at[slot4(km - 2)], at_in + (long)(km - 2) * A, y0 - 2, x0 - 2, RY, RX, imt, jmt);
    load_region(S.ws[slot3(km - 1)], a.ws + (long)(km - 1) * A, y0 - 1, x0 - 1, QY, QX, imt, jmt);
    load_region(S.uw[(km - 1) & 1], a.uwf + (long)(km - 1) * A, y0 - 1, x0 - 2, QY, RX, imt, jmt);
    load_region(S.vs[(km - 1) & 1], a.vsf + (long)(km - 1) * A, y0 - 2, x0 - 1, QY + 1, QX, imt, jmt);

    const bool own = (i < imt && j < jmt);
    const bool inner = own && i >= 2 && i < imt - 2 && j >= 2 && j < jmt - 2;
    const long qo = own ? q2(j, i, imt) : 0;
    const int kz = own ? a.kmt[qo] : 0;
    const int rc = (ty + 2) * RX + (tx + 2);     // own cell in H2
    const int hc = (ty + 1) * QX + (tx + 1);     // own cell in H1
    const int uc = (ty + 1) * RX + (tx + 2);     // own column in uw
    const int vc = (ty + 2) * QX + (tx + 1);     // own row in vs
    const double swv = (inner && n == 0) ? a.swv[qo] : 0.0;
    const double stf = own ? a.stf_n[n * A + qo] : 0.0;
    double atb_kp1 = 0.0;                                       // tracer level k+1 of atb
    double atb_k = own ? atb_in[(long)km * A + qo] : 0.0;       // level km-1
    double wkc_k = 0.0;
    double e_prev = 0.0, f_prev = 0.0;

    for (int k = km - 1; k >= 0; --k) {
      // ---- phase A: loads for this level
      __syncthreads();
      if (k >= 2) load_region(S.at[slot4(k - 2)], at_in + (long)(k - 2) * A, y0 - 2, x0 - 2, RY, RX, imt, jmt);
      if (k >= 1) {
        load_region(S.ws[slot3(k - 1)], a.ws + (long)(k - 1) * A, y0 - 1, x0 - 1, QY, QX, imt, jmt);
        load_region(S.uw[(k - 1) & 1], a.uwf + (long)(k - 1) * A, y0 - 1, x0 - 2, QY, RX, imt, jmt);
        load_region(S.vs[(k - 1) & 1], a.vsf + (long)(k - 1) * A, y0 - 2, x0 - 1, QY + 1, QX, imt, jmt);
      }
      load_region(S.atb, atb_in + (long)(k + 1) * A, y0 - 2, x0 - 2, RY, RX, imt, jmt);
      const double atb_km1 = (own && k >= 1) ? atb_in[(long)k * A + qo] : 0.0;  // tracer level k-1
      const double wkc_km1 = (own && k >= 1) ? akt[(long)(k - 1) * A + qo] : 0.0;
      if (k == km - 1) wkc_k = 0.0;
      __syncthreads();
      // ---- phase B: first Laplacian at this level
      del4_first(S, a, k, x0, y0);
      __syncthreads();
      // ---- phase C: own column
      if (inner) {
        const double* at_c = S.at[slot4(k)];
        const double* at_u = k > 0 ? S.at[slot4(k - 1)] : nullptr;
        const double* at_d = k < km - 1 ? S.at[slot4(k + 1)] : nullptr;
        const long cg = (long)k * A + qo;
        const double adv = simple_adv<ADV, DIAG>(S, a, k, n, cg, rc, hc, uc, vc, at_c, at_u, at_d);
        if (inner) {
          const double vit_k = k < kz ? 1.0 : 0.0;
          const double vit_kp1 = (k + 1 < kz) ? 1.0 : 0.0;
          double tf = adv * vit_k;
          // second Laplacian (tracer_del4_2)
          {
            const int r = rc;
            double h = 0.0, cc = 0.0;
            if (k <= S.kmt[r] - 1) {
              if (k <= S.kmt[r - RX] - 1) { h += S.dtn[hc] * S.d2[hc - QX]; cc -= S.dtn[hc]; }
              if (k <= S.kmt[r + RX] - 1) { h += S.dts[hc] * S.d2[hc + QX]; cc -= S.dts[hc]; }
              if (k <= S.kmt[r + 1] - 1) { h += S.dte[hc] * S.d2[hc + 1]; cc -= S.dte[hc]; }
              if (k <= S.kmt[r - 1] - 1) { h += S.dtw[hc] * S.d2[hc - 1]; cc -= S.dtw[hc]; }
            }
            tf += p.ah * (cc * S.d2[hc] + h);
          }
          // shortwave penetration, temperature only (tracer_5)
          if (n == 0) {
            if (k >= 1 && k < km - 1) {
              const double w1 = swv * a.pen[k - 1] * vit_k;
              const double w2 = swv * a.pen[k] * vit_kp1;
              tf = tf + (w1 - w2) * odzp[k];
              if (DIAG) a.penetrate[cg] = (w1 - w2) * odzp[k];
            } else if (k == 0) {
              const double w1 = swv * a.pen[0] * ((1 < kz) ? 1.0 : 0.0);
              tf = tf - odzp[0] * w1;
              if (DIAG) a.penetrate[cg] = -w1 * odzp[0];
            } else {
              const double w2 = swv * a.pen[km - 2] * vit_k;
              tf = tf + odzp[km - 1] * w2;
              if (DIAG) a.penetrate[cg] = w2 * odzp[km - 1];
            }
          }
          // explicit half of the vertical diffusion (tracer_5)
          if (k >= 1 && k < km - 1) {
            const double w1 = wkc_km1 * (atb_km1 - atb_k) * odzt[k] * vit_k;
            const double w2 = wkc_k * (atb_k - atb_kp1) * odzt[k + 1] * vit_kp1;
            tf = tf + odzp[k] * (w1 - w2) * 0.5;
            if (DIAG) a.dzd[n * F + cg] = odzp[k] * (w1 - w2) * 0.5;
          } else if (k == 0) {
            const double w1 = wkc_k * (atb_k - atb_kp1) * odzt[1] * vit_kp1;
            tf = tf - odzp[0] * w1 * 0.5;
            if (DIAG) a.dzd[n * F + cg] = -odzp[0] * w1 * 0.5;
          } else {
            const double w2 = wkc_km1 * (atb_km1 - atb_k) * odzt[km - 1] * vit_k;
            tf = tf + odzp[km - 1] * w2 * (1.0 - aidif);
            if (DIAG) a.dzd[n * F + cg] = odzp[km - 1] * w2 * 0.5;
          }
          // surface fluxes (tracer_5 salt, tracer_6 SSS norm / heat)
          if (k == 0) {
            if (n == 1) {
              if (kz > 0) tf = tf + stf * (1.0 - aidif) * odzp[0];
              tf = tf + a.scalars[0] * vit_k;
            } else if (kz > 0) {
              tf = tf + stf * odzp[0] * 0.5;
            }
          }
          // nudging (tracer_7, simple_assm), then restoring (boundary_restore == 1)
          if (p.simple_assm && k < p.ktv) tf = tf + vit_k * (a.restore_at[n * F + cg] - atb_k) * assm_rate(k);
          if (p.boundary_restore == 1 && k >= 1) {
            const double lamda = 1.0 / (15.0 * 86400.0);
            tf = tf + vit_k * (a.restore[n * F + cg] - atb_k) * lamda;
          }
          // explicit update (tracer_8) and one elimination step of the
          // implicit sweep (invtrit, tracer.cpp:923-978)
          const double d8 = at_c[rc] + dts * tf;
          double ev = 0.0, fv = d8;
          if (k < kz) {
            double a8, c8, b8;
            if (k >= 1) a8 = wkc_km1 * odzt[k] * odzp[k] * dts * 0.5;
            else a8 = odzp[0] * dts * 0.5;
            if (k == kz - 1) {
              c8 = odzp[kz - 1] * dts * 0.5;
              b8 = 1.0 + a8;
            } else if (k >= 1) {
              c8 = wkc_k * odzt[k + 1] * odzp[k] * dts * 0.5;
              b8 = 1.0 + a8 + c8;
            } else {
              c8 = wkc_k * odzt[k + 1] * odzp[k] * dts * 0.5;
              b8 = 1.0 + c8;
            }
            if (k == kz - 1) { e_prev = 0.0; f_prev = 0.0; }
            const double g0 = 1.0 / (b8 - c8 * e_prev);
            ev = a8 * g0;
            fv = (d8 + c8 * f_prev) * g0;
            e_prev = ev;
            f_prev = fv;
          }
          double* sl = scr + (long)k * NV * TTHREADS;
          sl[tid] = ev;
          sl[TTHREADS + tid] = fv;
          if (DIAG) sl[2 * TTHREADS + tid] = d8;
        }
      }
      atb_kp1 = atb_k;
      atb_k = atb_km1;
      wkc_k = wkc_km1;
    }
    // ---- substitution, top down, and the new state of the inner cells
    if (inner) {
      double x = 0.0;
      const double stf_c = stf;
      for (int k = 0; k < km; ++k) {
        const double* sl = scr + (long)k * NV * TTHREADS;
        const double ev = sl[tid], fv = sl[TTHREADS + tid];
        const long cg = (long)k * A + qo;
        double v;
        if (k < kz) {
          const double vit_k = 1.0;
          v = (k == 0) ? (ev * stf_c + fv) * vit_k : (ev * x + fv) * vit_k;
          x = v;
        } else {
          v = fv;
        }
        if (DIAG) {
          const double d8 = sl[2 * TTHREADS + tid];
          const double vit_k = k < kz ? 1.0 : 0.0;
          const double at_old = at_in[cg];
          a.tend[n * F + cg] = (v - at_old) / dts * vit_k;
          if (k == 0) a.dt_diff[n * F + cg] = (v - d8) / dts * vit_k - stf_c * 0.5 * odzp[0];
          else a.dt_diff[n * F + cg] = (v - d8) / dts * vit_k;
          if (j == 2 && a.tripole) a.fold_save[((long)(n * km + k)) * imt + i] = d8;
        }
        at_out[cg] = v;
        atb_out[(long)(k + 1) * A + qo] = v;
      }
    }
  }
}

// ------------------------------------------------------------- state halo
// One block per (level, tracer): ghost cells of the new state take the halo
// values (pop_haloupdate_tracer2 then tracer_9 for every point); cells the
// halo does not reach take the vtl input, which is what the reference's
// scratch use of vtl leaves there (tracer.cpp:1629-1653, 1895).
// Launched once per tracer (temperature first), so the salinity pass can read
// the temperature's final ghost values, which is what vtl holds in the
// reference between the two passes.
template <bool DIAG>
__device__ __forceinline__ void halo_state_level(const Arena& a, int n, int k) {
  extern __shared__ double top[];
  const int imt = a.imt, jmt = a.jmt;
  const long A = a.A, F = a.F, FB = a.FB;
  double* lvl = a.at[a.cur ^ 1] + n * F + (long)k * A;
  double* lvlb = a.atb[a.cur ^ 1] + n * FB + (long)(k + 1) * A;
  const double* old = a.at[a.cur] + n * F + (long)k * A;
  const double* vin = a.vtl ? a.vtl + (long)k * A : nullptr;
  const float* vin32 = a.vtl32 ? a.vtl32 + (long)k * A : nullptr;
  const double* tnew = a.at[a.cur ^ 1] + (long)k * A;  // temperature after its halo (n == 1 only)
  for (int i = threadIdx.x; i < imt; i += blockDim.x) top[i] = lvl[2L * imt + i];
  __syncthreads();
  HaloCells hc{imt, jmt, a.tripole};
  const long nc = hc.count();
  const double dts = a.p.dts;
  for (long m = threadIdx.x; m < nc; m += blockDim.x) {
    int j, i;
    hc.cell(m, j, i);
    const long q = (long)j * imt + i;
    double v;
    const bool filled = halo_cell_value(lvl, top, j, i, imt, jmt, a.ew_cyclic, a.tripole, v);
    if (!filled) v = vin ? vin[q] : (double)vin32[q];
    if (DIAG) {
      const double vit = k < a.kmt[q] ? 1.0 : 0.0;
      const bool inner = (i >= 2 && i < imt - 2 && j >= 2 && j < jmt - 2);
      double ori;
      if (inner) ori = a.fold_save[((long)(n * a.km + k)) * imt + i];
      else if (n == 0 || !filled) ori = vin ? vin[q] : (double)vin32[q];
      else ori = tnew[q];
      a.tend[n * F + (long)k * A + q] = (v - old[q]) / dts * vit;
      if (k == 0)
        a.dt_diff[n * F + q] = (v - ori) / dts * vit - a.stf_n[n * A + q] * 0.5 * a.odzp[0];
      else
        a.dt_diff[n * F + (long)k * A + q] = (v - ori) / dts * vit;
    }
    lvl[q] = v;
    lvlb[q] = v;
  }
}

template <bool DIAG>
__global__ void k_halo_state(Arena a, int n) {
  halo_state_level<DIAG>(a, n, blockIdx.x);
}

// Without diagnostics the two tracers' ghost fills are independent: one
// launch, part blockIdx.x (as k_halo_r8) of level blockIdx.y of tracer
// blockIdx.z, the same values as halo_state_level<false>; blockIdx.z 2 is the
// surface flux net (both tracers), whose ghost cells nothing reads within the
// step.
__global__ void k_halo_state_parts(const __grid_constant__ Arena a) {
  chain_grid();
  const int n = blockIdx.z, k = blockIdx.y;
  const int imt = a.imt, jmt = a.jmt;
  if (n == 2) {
    if (k < 2) halo_r8_part(a.net + (long)k * a.A, imt, jmt, a.ew_cyclic, a.tripole);
    return;
  }
  HaloCells hc{imt, jmt, a.tripole};
  long m0, m1;
  if (!halo_part(hc.count(), imt, a.tripole, blockIdx.x, m0, m1)) return;
  const long A = a.A, F = a.F, FB = a.FB;
  double* lvl = a.at[a.cur ^ 1] + n * F + (long)k * A;
  double* lvlb = a.atb[a.cur ^ 1] + n * FB + (long)(k + 1) * A;
  const double* vin = a.vtl ? a.vtl + (long)k * A : nullptr;
  const float* vin32 = a.vtl32 ? a.vtl32 + (long)k * A : nullptr;
  extern __shared__ double top[];
  if (a.tripole && blockIdx.x == 0) {
    for (int i = threadIdx.x; i < imt; i += blockDim.x) top[i] = lvl[2L * imt + i];
    __syncthreads();
  }
  for (long m = m0 + threadIdx.x; m < m1; m += blockDim.x) {
    int j, i;
    hc.cell(m, j, i);
    const long q = (long)j * imt + i;
    double v;
    if (!halo_cell_value(lvl, top, j, i, imt, jmt, a.ew_cyclic, a.tripole, v)) v = vin ? vin[q] : (double)vin32[q];
    lvl[q] = v;
    lvlb[q] = v;
  }
}

// tracer n of every member: blockIdx.x the level, blockIdx.y the member
__global__ void k_halo_state_batch(const MemberDesc* __restrict__ mem, int n) {
  const Arena& a = mem[blockIdx.y].a;
  if ((int)blockIdx.x >= a.km) return;
  if (a.diagnostics) halo_state_level<true>(a, n, blockIdx.x);
  else halo_state_level<false>(a, n, blockIdx.x);
}

__global__ void k_vtl_clobber(Arena a) {
  // tracer_ leaves vtl holding S with its halo (tracer.cpp:1891-1893)
  const long m = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= a.F) return;
  a.vtl[m] = a.at[a.cur][a.F + m];
}

}  // namespace

// ---------------------------------------------------------------- launchers
int launch_assm_dt_restore(const Arena& a, cudaStream_t s) {
  const int levels = a.p.ktv < a.km ? a.p.ktv : a.km;
  if (!a.p.simple_assm || levels <= 0) return LT_OK;
  const int bx = (int)((a.A + 255) / 256 < 64 ? (a.A + 255) / 256 : 64);
  k_assm_dt_restore<<<dim3(bx, levels, 2), 256, 0, s>>>(a);
  LT_LAUNCHED();
  return LT_OK;
}

int launch_ssh(const Arena& a, cudaStream_t s) {
  dim3 b(32, 8), g((a.imt + 31) / 32, (a.jmt + 7) / 8);
  k_ssh<<<g, b, 0, s>>>(a);
  LT_LAUNCHED();
  return LT_OK;
}

int launch_surface(const Arena& a, cudaStream_t s) {
  dim3 b(32, 8), g((a.imt + 31) / 32, (a.jmt + 7) / 8);
  return launch_chained(k_surface, g, b, 0, s, a);
}

int launch_surface_fluxes(const Arena& a, cudaStream_t s) {
  dim3 b(32, 8), g((a.imt + 31) / 32, (a.jmt + 7) / 8);
  k_surface_fluxes<<<g, b, 0, s>>>(a);
  LT_LAUNCHED();
  return LT_OK;
}

size_t tree_sum_part_elems(long n) {
  size_t tot = 0;
  long nb = (n + 2 * RB - 1) / (2 * RB);
  if (nb < 1) nb = 1;
  tot += nb;
  while (nb > 1) { nb = (nb + 2 * RB - 1) / (2 * RB); tot += nb; }
  return tot + 4;
}

int launch_interior_sum_sss(const Arena& a, cudaStream_t s) {
  const long n = (long)a.nx * a.ny, nb = (n + 2 * RB - 1) / (2 * RB);
  return launch_chained(k_sss_norm, dim3((unsigned)nb), dim3(RB), 0, s, a);
}

int launch_tree_sum(const double* x, long n, double* part, double* out, cudaStream_t s) {
  return tree_sum(ArrayTerm{x}, n, part, out, s);
}

int launch_halo_r8(double* f, int nz, int imt, int jmt, int ew_cyclic, int tripole, cudaStream_t s) {
  k_halo_r8<<<dim3(kHaloParts, nz), 256, imt * sizeof(double), s>>>(f, imt, jmt, ew_cyclic, tripole);
  LT_LAUNCHED();
  return LT_OK;
}

int launch_continuity_fp64(const Arena& a, cudaStream_t s) {
  constexpr int BY = kCont64TileY;
  static_assert(BY == 8, "continuity_tiles");
  dim3 b(32, BY), g((a.imt + 31) / 32, (a.jmt + BY - 1) / BY);
  if (continuity_by_levels(continuity_tiles(a))) {
    if (int rc = launch_chained(k_cont_levels64, dim3(g.x, g.y, (a.km + kContChunk - 1) / kContChunk), b, 0, s, a)) return rc;
    return launch_chained(k_cont_columns64, dim3(g.x, (a.jmt + 3) / 4), dim3(32, 4), 0, s, a);
  }
  return launch_chained(k_cont_march64<BY>, g, b, 0, s, a);
}

int launch_tracer_fp64(const Arena& a, cudaStream_t s, int slots) {
  const int ntx = (a.imt + TX - 1) / TX;
  const long ntiles = (long)ntx * ((a.jmt + TY - 1) / TY);
  const size_t sm = sizeof(TSmem);
  // [scheme - 1][diagnostics]: the centred and flux schemes (lt_adv_scheme order)
  using Kern = void (*)(Arena, int, long);
  static const Kern kern[2][2] = {
      {k_tracer64<false, LT_ADV_CENTERED>, k_tracer64<true, LT_ADV_CENTERED>},
      {k_tracer64<false, LT_ADV_FLUX>, k_tracer64<true, LT_ADV_FLUX>}};
  static bool attr = false;
  if (!attr) {
    for (auto& row : kern)
      for (Kern k : row) LT_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    attr = true;
  }
  const int adv = a.p.adv_tracer;
  if (adv != LT_ADV_CENTERED && adv != LT_ADV_FLUX) return LT_E_INVALID;
  if (int rc = launch_assm_dt_restore(a, s)) return rc;
  kern[adv - 1][a.diagnostics ? 1 : 0]<<<slots, TTHREADS, sm, s>>>(a, ntx, ntiles);
  LT_LAUNCHED();
  return LT_OK;
}

int launch_halo_state(const Arena& a, cudaStream_t s) {
  if (!a.diagnostics) {
    return launch_chained(k_halo_state_parts, dim3(kHaloParts, a.km, 3), dim3(256), a.imt * sizeof(double), s, a);
  }
  // with diagnostics, salinity's dt_diff reads temperature's new ghost values
  for (int n = 0; n < 2; ++n) {
    k_halo_state<true><<<a.km, 256, a.imt * sizeof(double), s>>>(a, n);
    LT_LAUNCHED();
  }
  return LT_OK;
}

// The small kernels of a batch step over every member at once (member
// descriptors in device memory; the largest member's sizes set the grids).
int launch_small_batch_pre(const MemberDesc* mem, int nmem, int max_imt, int max_jmt, long max_cols,
                           cudaStream_t s) {
  {
    dim3 b(32, 8), g((max_imt + 31) / 32, (max_jmt + 7) / 8, nmem);
    k_surface_batch<<<g, b, 0, s>>>(mem);
    LT_LAUNCHED();
  }
  long nb = (max_cols + 2 * RB - 1) / (2 * RB);
  if (nb < 1) nb = 1;
  for (int pass = 0;; ++pass) {
    k_sss_tree_batch<<<dim3((unsigned)nb, nmem), RB, 0, s>>>(mem, pass);
    LT_LAUNCHED();
    if (nb <= 1) break;
    nb = (nb + 2 * RB - 1) / (2 * RB);
  }
  k_finish_sss_batch<<<(nmem + 127) / 128, 128, 0, s>>>(mem, nmem);
  LT_LAUNCHED();
  k_halo_net_batch<<<dim3(2, nmem), 256, max_imt * sizeof(double), s>>>(mem);
  LT_LAUNCHED();
  return LT_OK;
}

int launch_halo_state_batch(const MemberDesc* mem, int nmem, int max_imt, int km_max, cudaStream_t s) {
  for (int n = 0; n < 2; ++n) {
    k_halo_state_batch<<<dim3(km_max, nmem), 256, max_imt * sizeof(double), s>>>(mem, n);
    LT_LAUNCHED();
  }
  return LT_OK;
}

int launch_vtl_clobber(const Arena& a, cudaStream_t s) {
  const long nb = (a.F + 255) / 256;
  k_vtl_clobber<<<(unsigned)nb, 256, 0, s>>>(a);
  LT_LAUNCHED();
  return LT_OK;
}

}  // namespace lt
