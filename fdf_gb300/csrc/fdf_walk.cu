// fdf_walk.cu -- fused advect + walking-search locate, one thread per particle.
//
// Restates, per particle, UpdateParticlePosition (ParticleMotion.c:19-29) and
// LocateParticleOrFindMigrationTarget_TEST (walkingsearch.c:1094-1242) with
// EvaluateParticlePosition (:811-859), DeterminePointPosition (:407-462),
// UpdateCellIndicesBasedOnDistancesTEST (:882-959) and UpdateParticleWeights
// (ParticleSwarm.c:1010-1047).  The per-cell plane table holds every
// particle-independent value of ComputeSignedDistanceToPlane, computed with the
// reference's own operation order, so each FP64 signed distance here is the
// reference's bit for bit: d = (fc - p) . n, then |d| < thr -> 0.
//
// The walk's steps take their face classes from the FP32 plane table with a rigorous
// error bound and fall back to the FP64 distance of a face only where the bound cannot
// decide (fdf_walk.cuh), so the path of cells is the FP64 walk's; the concluding cell's
// six distances are computed in FP64 as the reference computes them, for the weights.
// Positions, velocities and weights are the reference's bit for bit; what goes is the
// FP64 work of every evaluation before the last.
//
// The stuck-cell tie-breaker (walkingsearch.c:1149-1185) cannot fire on one
// rank: an evaluation either concludes (position >= 0) or reports some d < 0,
// and UpdateCellIndices then changes at least one index, so the same cell is
// never visited twice in a row.  It is therefore not restated here.
//
// Cycle cut-off.  The next cell of the walk is a function of (cell, position)
// only, so once the walk returns to a cell it has already evaluated without
// concluding, it repeats that cycle until MAX_TRAVERSAL and the particle is
// LOST.  This happens for points in the thin gap between a cell's FRONT plane
// and the next cell's BACK plane on curved grids (the two planes are built from
// different corner vertices, walkingsearch.c:303-325).  The walk here detects
// the revisit (Brent's method: compare with the cell saved at step 2^m) and
// concludes LOST at once; the outcome, cell (-1,-1,-1), and the unchanged
// weights are the reference's, and the evaluation count reported for parity is
// the reference's (MAX_TRAVERSAL).
#include "fdf_internal.cuh"
#include "fdf_exact.cuh"
#include "fdf_counters.cuh"
#include "fdf_walk.cuh"

namespace {

using fdfx::add;
using fdfx::sub;
using fdfx::mul;

// The pair a walk in FP64 positions takes for a coordinate: (hi, lo) within 2^-48 |v| of v; a nonzero
// |v| below 2^-120 (where the split's error is absolute) gives a NaN pair, whose faces all take the
// FP64 route.
__device__ __forceinline__ float2 walk_pair(double v) {
  const unsigned long long mag = fdfx::ubits(v) & fdfx::ABS_MASK;
  if (mag < (903ull << 52) && mag != 0ull) return make_float2(__int_as_float(0x7fc00000), 0.f);
  return fdfx::split_rn(v);
}

// UpdateParticleWeights (ParticleSwarm.c:1010-1047) from the concluding cell's FP64 distances (INT: exact_face).
template <bool INT>
__device__ __forceinline__ void exact_weights(const double *__restrict__ row, double x, double y, double z, double &a1,
                                              double &a2, double &a3) {
  double d[6];
#pragma unroll
  for (int f = 0; f < 6; ++f) d[f] = exact_face<INT>(row, f, x, y, z);
  const unsigned long long tol_bits = fdfx::ubits(FDF_INTERP_DIST_TOL);
#pragma unroll
  for (int f = 0; f < 6; ++f)
    if (fdfx::le_pos(d[f], tol_bits)) d[f] = FDF_INTERP_DIST_TOL;
  a1 = fdfx::div_rn(d[F_LEFT], add(d[F_LEFT], d[F_RIGHT]));
  a2 = fdfx::div_rn(d[F_BOTTOM], add(d[F_BOTTOM], d[F_TOP]));
  a3 = fdfx::div_rn(d[F_BACK], add(d[F_FRONT], d[F_BACK]));
}

// The step's walk.  Bound by the FP64 pipe in a large swarm (advection, the weights of the concluding
// cell: 36 of 54 operations are its six distances) and by the walk's dependent row loads in a small one.
// INT: two of each distance's three products on the integer pipe, at 1152 resident threads; per step
// in a 64 x 64 x 1024 grid 249 -> 240 us at 2M particles, 467 -> 415 at 4M, and 1848 -> 1707 at 16M in
// 96 x 96 x 1536 (one product 1830, three 1778, two at 1024 threads 1718, at 1280 1741).  The products'
// extra instructions lengthen each warp's chain, which a small swarm waits for: 83 -> 90 us at 500k,
// 139 -> 143 at 1M.  So INT is false below WALK_INT_MIN slots, about ten waves of resident threads.
constexpr int WALK_INT_MIN = 3 << 19;

template <bool INT>
__global__ void __launch_bounds__(FDF_PLAIN_THREADS, FDF_PLAIN_MIN_BLOCKS + (INT ? 1 : 0))
    k_locate(SwarmBuf b, GridDims g, const float *__restrict__ table, const double *__restrict__ planes, double dt,
               int advect, int reset_first, const double *__restrict__ bbox, int drop_removed, DevCounters *cnt,
               unsigned int *__restrict__ keys, unsigned int *__restrict__ rank, unsigned int *__restrict__ count,
               unsigned int sentinel) {
  const int n = cnt->n_sorted;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s == 0) {
    cnt->n_start = n;
    if (advect) atomicAdd(&cnt->psteps_total, (unsigned long long)n);
  }
  LocCounts m;
  unsigned int hkey = 0xffffffffu;
  if (s < n) {
    double x = b.x[s], y = b.y[s], z = b.z[s];
    if (advect) {
      x = add(x, mul(b.u[s], dt));
      y = add(y, mul(b.v[s], dt));
      z = add(z, mul(b.w[s], dt));
      b.x[s] = x; b.y[s] = y; b.z[s] = z;
    }
    unsigned char st = b.status[s];
    if (reset_first && st == ST_ACTIVE_AND_LOCATED) st = ST_NEEDS_LOCATION;
    int cell = b.cell[s];
    bool lost = false;
    if (st != ST_ACTIVE_AND_LOCATED) {
      Walk32 w;
      w.i = 0; w.j = 0; w.k = 0;   // InitializeTraversalParameters: previous cell, else (0,0,0)
      if (cell >= 0 && (long long)cell < g.Nc) cell_ijk(g, (unsigned int)cell, w.i, w.j, w.k);
      walk_ref32<true, false, false, true>(table, planes, g, walk_pair(x), walk_pair(y), walk_pair(z),
                                            FDF_MAX_TRAVERSAL, w, cnt, x, y, z);
      if (w.degenerate) m.err |= ERRBIT_DEGENERATE;
      m.evals += (unsigned int)(w.cycle ? FDF_MAX_TRAVERSAL : w.steps);
      m.done += w.evaluated();
      if (w.lost || !w.concluded) {
        lost = true;
        cell = -1;
        st = ST_LOST;
      } else {
        cell = (int)(((long long)w.k * g.JM + w.j) * g.IM + w.i);
        double a1, a2, a3;
        exact_weights<INT>(planes + (long long)cell * FDF_ROW, x, y, z, a1, a2, a3);
        b.a1[s] = a1; b.a2[s] = a2; b.a3[s] = a3;
        st = ST_ACTIVE_AND_LOCATED;
      }
      b.cell[s] = cell;
      b.status[s] = st;
    } else {
      lost = (cell < 0);
    }
    unsigned int key = lost ? sentinel : (unsigned int)cell;
    if (lost) m.lost_total += 1;
    if (drop_removed) {   // CheckAndRemoveLostParticles, then CheckAndRemoveOutOfBoundsParticles
      if (lost) {
        m.lost += 1;
      } else {
        // IsParticleInBox, the six comparisons on the integer pipe
        const bool inside = fdfx::in_range(x, bbox[0], bbox[3]) && fdfx::in_range(y, bbox[1], bbox[4]) &&
                            fdfx::in_range(z, bbox[2], bbox[5]);
        if (!inside) { m.oob += 1; key = sentinel; }
      }
    }
    keys[s] = key;
    if (key < sentinel) hkey = key;
    else if (!drop_removed) hkey = sentinel;   // the initial setup keeps LOST particles, at the end
  }
  const unsigned int r = warp_histogram_rank(hkey, count);
  if (rank && hkey != 0xffffffffu) rank[s] = r;
  block_flush_counts(m, cnt);
}

// The walk and the weights of points that are not the swarm (fdf_LocatePoints), in the callers' layout:
// no swarm buffers, sort keys or histogram.  cell_in == cell_out is allowed (null: from cell (0,0,0)).
__global__ void __launch_bounds__(FDF_PLAIN_THREADS, FDF_PLAIN_MIN_BLOCKS)
    k_locate_points(const double *__restrict__ pos, const long long *cell_in, int n, GridDims g,
                    const float *__restrict__ table, const double *__restrict__ planes, DevCounters *cnt,
                    long long *cell_out, double *__restrict__ weight, long long *__restrict__ status) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const double x = pos[3 * (size_t)p], y = pos[3 * (size_t)p + 1], z = pos[3 * (size_t)p + 2];
  Walk32 w;
  w.i = 0; w.j = 0; w.k = 0;
  if (cell_in) {
    const long long i = cell_in[3 * (size_t)p], j = cell_in[3 * (size_t)p + 1], k = cell_in[3 * (size_t)p + 2];
    if (i >= 0 && i < g.IM && j >= 0 && j < g.JM && k >= 0 && k < g.KM) { w.i = (int)i; w.j = (int)j; w.k = (int)k; }
  }
  walk_ref32<true, false, false, true>(table, planes, g, walk_pair(x), walk_pair(y), walk_pair(z), FDF_MAX_TRAVERSAL, w,
                                      cnt, x, y, z);
  if (w.degenerate) atomicOr(&cnt->err, (unsigned int)ERRBIT_DEGENERATE);
  const bool lost = w.lost || !w.concluded;
  double a1 = 0.0, a2 = 0.0, a3 = 0.0;
  if (!lost) {
    const long long cell = ((long long)w.k * g.JM + w.j) * g.IM + w.i;
    exact_weights<false>(planes + cell * FDF_ROW, x, y, z, a1, a2, a3);
  }
  cell_out[3 * (size_t)p] = lost ? -1 : w.i;
  cell_out[3 * (size_t)p + 1] = lost ? -1 : w.j;
  cell_out[3 * (size_t)p + 2] = lost ? -1 : w.k;
  weight[3 * (size_t)p] = a1; weight[3 * (size_t)p + 1] = a2; weight[3 * (size_t)p + 2] = a3;
  status[p] = lost ? ST_LOST : ST_ACTIVE_AND_LOCATED;
}

}  // namespace

void launch_locate_points(const double *pos, const long long *cell_in, int n, GridDims g, const float *table,
                          const double *planes, DevCounters *cnt, long long *cell_out, double *weight, long long *status,
                          cudaStream_t s) {
  constexpr int th = FDF_PLAIN_THREADS;
  k_locate_points<<<(unsigned int)((n + th - 1) / th), th, 0, s>>>(pos, cell_in, n, g, table, planes, cnt, cell_out,
                                                                 weight, status);
}

void launch_locate(const SwarmBuf &b, int n_cap, GridDims g, const float *table, const double *planes, double dt,
                   int advect, const double *bbox, int drop_removed, DevCounters *cnt, unsigned int *keys,
                   unsigned int *rank, unsigned int *count, unsigned int sentinel, cudaStream_t s) {
  // advect and drop_removed are both set by the fused step, which also resets statuses first
  constexpr int th = FDF_PLAIN_THREADS;
  const unsigned int blocks = n_cap > 0 ? (unsigned int)((n_cap + th - 1) / th) : 1u;
  auto *kern = n_cap >= WALK_INT_MIN ? k_locate<true> : k_locate<false>;
  kern<<<blocks, th, 0, s>>>(b, g, table, planes, dt, advect, drop_removed, bbox, drop_removed, cnt, keys, rank, count,
                             sentinel);
}
