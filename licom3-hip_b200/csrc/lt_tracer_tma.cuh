// lt_tracer_tma.cuh - what the TMA-fed kernels of the step share: the tensor
// maps of a domain's level boxes, the batch member descriptor and the launchers
// that take either.
//
// The mixed column kernel (k_tracer_mixed) marches a tile of columns from the
// bottom level up: the data of one level arrive as 3-D TMA boxes (no multicast)
// into one of three shared-memory level slots guarded by mbarriers, issued one
// step ahead of their first use.  At step k a CTA computes the tspas predictor
// and masked extrema at level k-1 on the tile plus a 1-cell halo and the first
// Laplacian of the biharmonic operator at level k (tracer.cpp:291-547,
// 1238-1293), then per column the limited flux divergence at level k, the
// second Laplacian, shortwave, the explicit half of the vertical diffusion,
// surface fluxes, the explicit update and one elimination step of the implicit
// tridiagonal sweep, which runs upward with the march (tracer.cpp:549-921,
// 1295-1699, 923-978).  A final downward pass substitutes through the sweep and
// writes the new state of the inner cells; ghost cells and the fold are done by
// the halo kernel afterwards.  The FP64 form splits the same work into passes
// (lt_column_fp64.cu).
#pragma once
#include "lt_common.cuh"
#include "lt_tma.cuh"

namespace lt {

constexpr int SW = 40;      // row width of loaded boxes: columns x0-4 .. x0+35
constexpr int HQX = TX + 2;   // a row of the tile plus a 1-cell halo

// Mixed precision: the column kernel's boxes and those of the continuity march
// (vel: utf, vtf, utl, vtl).
struct TracerMaps {
  CUtensorMap at[2], atb[2], ws, uw, vs, akt;
  CUtensorMap vel[4];
};
// The FP64 tspas passes: the limiter's and the explicit pass's boxes (atb_own:
// the previous state of a block's own columns) and the implicit pass's (th_*).
struct ColumnMaps {
  CUtensorMap at[2], atb[2], atb_own[2], ws, uw, vs, akt;
  CUtensorMap th_at[2], th_akt;
};

// One member of a batched launch, in device memory.  The tensor maps come
// first: a map read from global memory must be 64-byte aligned.
struct alignas(64) MemberDesc {
  TracerMaps maps;
  Arena a;
  long item0;    // first work item (a tile, both tracers) of this member in the batch list
  long ntiles;   // column tiles of this member
  int ntx;       // tiles along i
  int tma;       // 1: level boxes by TMA; 0: by per-thread copies (row pitch TMA cannot take)
};

// Launches over blocks of 32 x 4 columns: launch(first block row, block rows),
// again where the rows are more than a grid's y dimension takes (262140 rows).
template <class Launch>
int for_column_rows(const Arena& a, Launch launch) {
  constexpr int most = 65535;
  const int rows = (a.jmt + kColY - 1) / kColY;
  for (int r = 0; r < rows; r += most)
    if (int rc = launch(r, rows - r < most ? rows - r : most)) return rc;
  return LT_OK;
}

// The FP64 tspas passes over the columns (lt_column_fp64.cu); tma: their level
// data by TMA boxes (else per-thread copies)
int launch_column_fp64(const Arena& a, const ColumnMaps& maps, bool tma, cudaStream_t s);
// sets its kernels' shared-memory size on the current device
int prepare_column_fp64();
// Batched forms (mixed precision): nmem members, total work items, one
// persistent column launch of `grid` CTAs with per-CTA scratch of km_max
// levels; continuity over every member's tiles with tiles of 32 x cby columns
// (the TMA-fed march at its own tile height).
int launch_tracer_mixed_batch(const MemberDesc* mem, int nmem, long total, double* scratch, int km_max, int grid,
                              cudaStream_t s);
int launch_continuity_mixed_batch(const MemberDesc* mem, int nmem, int max_imt, int max_jmt, int km_max, int cby,
                                  cudaStream_t s);
// The small kernels of a batch step for every member in one launch each:
// surface fluxes, the SSS-norm tree (one launch per tree pass; max_cols is
// the largest member's nx * ny) and its finish, the net halo; and the state
// halo (two launches, temperature first).
int launch_small_batch_pre(const MemberDesc* mem, int nmem, int max_imt, int max_jmt, long max_cols,
                           cudaStream_t s);
int launch_halo_state_batch(const MemberDesc* mem, int nmem, int max_imt, int km_max, cudaStream_t s);
// sets the batched column kernel's shared-memory size on the current device
int prepare_tracer_mixed_batch();
// The mixed column kernel; tma: its level boxes by TMA (else per-thread copies)
int launch_tracer_tma_mixed(const Arena& a, const TracerMaps& maps, bool tma, cudaStream_t s, int grid);
// The mixed continuity: TMA-fed when the domain has its maps (tma), else
// plain loads.
int launch_continuity_mixed(const Arena& a, const TracerMaps& maps, bool tma, cudaStream_t s);
// Build the tensor maps of a mixed or FP64 domain; false if the layout does not
// allow TMA (row pitch not a multiple of 16 bytes for some field).
bool build_tracer_maps(const Arena& a, TracerMaps* maps);
bool build_column_maps(const Arena& a, ColumnMaps* maps);

// Records a timed-out wait and drains this CTA's outstanding loads (bounded).
template <class SM>
__device__ __forceinline__ void tma_bail(SM& S, const Arena& a, uint32_t par, uint32_t outstanding) {
  constexpr int ns = sizeof(S.bar) / sizeof(S.bar[0]);
  if (threadIdx.x == 0) {
    atomicExch(a.status + 1, 1);
    for (int s = 0; s < ns; ++s)
      if (outstanding & (1u << s)) mbar_wait(&S.bar[s], (par >> s) & 1u);
  }
  __syncthreads();
}

}  // namespace lt
