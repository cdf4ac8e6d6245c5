// fdf_fp32.cu -- the precision form: interpolation, advection and deposition in FP32,
// cell location decided exactly as the FP64 reference walk decides it.
//
// Positions.  The form holds each coordinate as a float pair (hi, lo) with |lo| <=
// ulp(hi)/2; the form's position is the exact sum hi + lo (a double).  Advection adds
// the FP32 displacement fl32(u * dt) by double-float addition (FP32 operations only).
// Uploads split the caller's FP64 position (an error of at most 2^-48 |p|); downloads
// return hi + lo exactly.
//
// Walk.  Every face class the walk needs is decided exactly as the FP64 reference decides it
// (fdf_walk.cuh: the FP32 plane table with a rigorous error bound, FP64 where it cannot
// decide), so the cells, statuses and walk paths are the reference's for the form's own
// positions.
#include "fdf_internal.cuh"
#include "fdf_exact.cuh"
#include "fdf_counters.cuh"
#include "fdf_walk.cuh"

namespace {

using fdfx::add;
using fdfx::mul;
using fdfx::sub;

// One 128-B FP32 row per cell (the layout and the error bound are in fdf_walk.cuh): the first
// vertex c0 as a float pair, the two margins, then per face n32 = fl32(n) and
// e32 = fl32(n . (fc - c0)).
__global__ void k_build_table32(const double *__restrict__ planes, const double *__restrict__ coor, GridDims g,
                                float *__restrict__ table) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= g.Nc) return;
  int i, j, k;
  cell_ijk(g, (unsigned int)c, i, j, k);
  const double *v0 = coor + 3 * (((long long)k * (g.JM + 1) + j) * (long long)(g.IM + 1) + i);
  const double *row = planes + c * FDF_ROW;
  float *t = table + c * FDF_ROW32;
  const unsigned int sw = row32_swizzle((unsigned int)c);
  float *h0 = t + 4 * sw, *h1 = t + 4 * (1u ^ sw);
  double c0[3], size = 0.0;
  for (int q = 0; q < 3; ++q) {
    const float h = __double2float_rn(v0[q]);
    const float l = __double2float_rn(sub(v0[q], (double)h));
    h0[q] = h;
    h1[q] = l;
    c0[q] = add((double)h, (double)l);   // exact: the pair's value
    size = add(size, fabs((double)h));
  }
  double sigma = 0.0;   // max over faces of sum_i |fc_i - c0_i| |n_i|
  bool wide = false;    // a value the FP32 bound does not cover: every face goes to FP64
  for (int f = 0; f < 6; ++f) {
    const double *p = row + 6 * f;
    const double dx = sub(p[0], c0[0]), dy = sub(p[1], c0[1]), dz = sub(p[2], c0[2]);
    const double e = add(add(mul(dx, p[3]), mul(dy, p[4])), mul(dz, p[5]));
    const double sg = add(add(mul(fabs(dx), fabs(p[3])), mul(fabs(dy), fabs(p[4]))), mul(fabs(dz), fabs(p[5])));
    sigma = sg > sigma ? sg : sigma;
    wide = wide || !(fabs(e) <= 0x1p100) || !(sg <= 0x1p100);
    float *o = t + 4 * ((2u + f) ^ sw);
    o[0] = __double2float_rn(p[3]);
    o[1] = __double2float_rn(p[4]);
    o[2] = __double2float_rn(p[5]);
    o[3] = __double2float_rn(e);
  }
  // The faces' own margin: thr rounded up with a little headroom (thr32 (1 - 2^-24)^2 >= thr), and
  // the FP64 roundings of e and of the reference's own distance, 32 eps sigma (rounded up)
  h1[3] = fabsf(__fadd_rn(__double2float_ru(mul(row[36], 1.0 + 0x1p-22)), __double2float_ru(mul(sigma, 0x1p-48))));
  // The cell's: the same with headroom for its own roundings, and the row's part of 40 u sum_i ex_i
  const double slack = add(mul(sigma, 0x1p-48), mul(size, 40.0 * 0x1p-48));
  const float base = __double2float_ru(mul(add(row[36], slack), 1.0 + 0x1p-19));
  if (fdfx::ubits(row[37]) != 0ULL) {   // a degenerate cell
    h1[3] = -1.0f;
    wide = true;
  }
  h0[3] = wide ? __int_as_float(0x7f800000) : base;
}

// (hi, lo) float pair held in a double slot of the swarm arrays
__device__ __forceinline__ float2 ld_pair(const double *a, int s) {
  return *reinterpret_cast<const float2 *>(a + s);
}
__device__ __forceinline__ void st_pair(double *a, int s, float2 v) { *reinterpret_cast<float2 *>(a + s) = v; }

// (hi, lo) + v for a float v (double-float addition, FP32 operations only).
__device__ __forceinline__ float2 pair_add(float2 p, float v) {
  const float sh = __fadd_rn(p.x, v);
  const float bv = __fsub_rn(sh, p.x);
  const float e = __fadd_rn(__fsub_rn(p.x, __fsub_rn(sh, bv)), __fsub_rn(v, bv));   // exact error of p.x + v
  const float t = __fadd_rn(p.y, e);
  const float h = __fadd_rn(sh, t);
  return make_float2(h, __fsub_rn(t, __fsub_rn(h, sh)));
}


// Writes the located (or LOST) particle: weights (UpdateParticleWeights in FP32: clamp
// d <= 1e-14, then the three ratios), cell and status.
__device__ __forceinline__ void store_located32(const SwarmBuf &b, int s, int cell, bool lost, float (&dv)[6]) {
  if (lost) {
    b.cell[s] = -1;
    b.status[s] = ST_LOST;
    return;
  }
#pragma unroll
  for (int f = 0; f < 6; ++f)
    if (!(dv[f] > 1e-14f)) dv[f] = (dv[f] != dv[f]) ? dv[f] : 1e-14f;
  b.a1f[s] = __fdiv_rn(dv[F_LEFT], __fadd_rn(dv[F_LEFT], dv[F_RIGHT]));
  b.a2f[s] = __fdiv_rn(dv[F_BOTTOM], __fadd_rn(dv[F_BOTTOM], dv[F_TOP]));
  b.a3f[s] = __fdiv_rn(dv[F_BACK], __fadd_rn(dv[F_FRONT], dv[F_BACK]));
  b.cell[s] = cell;
  b.status[s] = ST_ACTIVE_AND_LOCATED;
}

// Sort key of a particle whose location is final, with IsParticleInBox on the form's
// position: decided in FP32 when the hi parts are clear of the box faces by more than the
// lo parts and rounding can move them (fbox = the box shrunk accordingly), exactly in
// FP64 otherwise.
__device__ __forceinline__ unsigned int settle_key32(bool lost, int cell, float2 px, float2 py, float2 pz,
                                                     int drop_removed, const double *__restrict__ bbox,
                                                     const float *__restrict__ fbox, unsigned int sentinel,
                                                     unsigned int &my_lost, unsigned int &my_oob,
                                                     unsigned int &my_lost_total) {
  unsigned int key = lost ? sentinel : (unsigned int)cell;
  if (lost) my_lost_total += 1;
  if (drop_removed) {
    if (lost) {
      my_lost += 1;
    } else {
      const float4 fb0 = *reinterpret_cast<const float4 *>(fbox), fb1 = *reinterpret_cast<const float4 *>(fbox + 4);
      const bool surely_in = px.x > fb0.x && px.x < fb1.x && py.x > fb0.y && py.x < fb1.y && pz.x > fb0.z &&
                             pz.x < fb1.z;
      bool inside = surely_in;
      if (!surely_in) {
        const double x = pair_value(px), y = pair_value(py), z = pair_value(pz);
        inside = x >= bbox[0] && x <= bbox[3] && y >= bbox[1] && y <= bbox[4] && z >= bbox[2] && z <= bbox[5];
      }
      if (!inside) { my_oob += 1; key = sentinel; }
    }
  }
  return key;
}

// Advect + locate, one thread per particle.
//   FAR: the walks may start far from the particles (walk_ref32): without the advection and, in the learned form,
//        where particles may have no previous cell.
//   FIRST == false: the reference walk from the previous cell (or cell (0,0,0)).
//   FIRST == true:  the reference's first evaluation, in the previous cell; a particle that it
//                   does not conclude and that lies at least far_cells past that cell is
//                   marked in `pending` (per warp of slots: a bit mask [W] and its count
//                   [W + 1], W = ceil(n_cap / 32)) with its cell field set to P1, the
//                   walk's second cell, and finished by k_locate32_path (its key and
//                   histogram entry are written there); a nearer one continues the reference
//                   walk here.
//   DENSE: more slots than cells.  A warp's rows then mostly come from L1 and L2 and two more blocks an SM
//          (56 registers, a few spilled) hide more of the walk than the spills cost: per step 64M particles
//          in 14M cells 2.29 -> 2.20 ms, the learned form's first pass 2.32 -> 2.17, 16M in 4.2M cells
//          0.518 -> 0.493; 6M in 14M cells 0.285 against 0.290 (four more: 2.47, 2.19, 0.554, 0.333).
template <bool FIRST, bool FAR, bool DENSE>
__global__ void __launch_bounds__(FDF_LOC_THREADS, FDF_LOC_MIN_BLOCKS + (DENSE ? 128 / FDF_LOC_THREADS : 0)) k_locate32(SwarmBuf b, GridDims g, const float *__restrict__ table,
                                                  const double *__restrict__ planes, float dt32, int advect,
                                                  int reset_first, const double *__restrict__ bbox,
                                                  const float *__restrict__ fbox, int drop_removed,
                                                  DevCounters *cnt, unsigned int *__restrict__ keys,
                                                  unsigned int *__restrict__ rank,
                                                  unsigned int *__restrict__ count, unsigned int sentinel,
                                                  unsigned int *__restrict__ pending, int n_cap, float far_cells) {
  const int n = cnt->n_sorted;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s == 0) {
    cnt->n_start = n;
    if (advect) atomicAdd(&cnt->psteps_total, (unsigned long long)n);
  }
  LocCounts m;
  unsigned int hkey = 0xffffffffu;
  bool wait = false;
  if (s < n) {
    float2 px = ld_pair(b.x, s), py = ld_pair(b.y, s), pz = ld_pair(b.z, s);
    if (advect) {   // FP32 displacement added to the (hi, lo) position
      px = pair_add(px, __fmul_rn(b.uf[s], dt32));
      py = pair_add(py, __fmul_rn(b.vf[s], dt32));
      pz = pair_add(pz, __fmul_rn(b.wf[s], dt32));
      st_pair(b.x, s, px); st_pair(b.y, s, py); st_pair(b.z, s, pz);
    }
    unsigned char st = b.status[s];
    if (reset_first && st == ST_ACTIVE_AND_LOCATED) st = ST_NEEDS_LOCATION;
    int cell = b.cell[s];
    bool lost = false;
    if (st != ST_ACTIVE_AND_LOCATED) {
      Walk32 w;
      w.i = 0; w.j = 0; w.k = 0;
      if (cell >= 0 && (long long)cell < g.Nc) cell_ijk(g, (unsigned int)cell, w.i, w.j, w.k);
      // LOST before, so from cell (0,0,0): as the setup walks.  One such particle holds its whole launch
      // (a 1536-cell walk 2.50 -> 1.47 ms, 512 cells 0.77 -> 0.48, in the first step after a setup).
      if (!FIRST && !FAR && cell < 0)
        walk_ref32<false, false, false, true>(table, planes, g, px, py, pz, FDF_MAX_TRAVERSAL, w, cnt);
      else
        walk_ref32<false, false, FIRST, FAR>(table, planes, g, px, py, pz, FDF_MAX_TRAVERSAL, w, cnt, 0.0, 0.0, 0.0,
                                             nullptr, far_cells);
      if (w.degenerate) m.err |= ERRBIT_DEGENERATE;
      m.done += w.evaluated();
      m.evals += FIRST ? w.evaluated() : (unsigned int)(w.cycle ? FDF_MAX_TRAVERSAL : w.steps);
      wait = FIRST && w.wait;
      const int at = (int)(((long long)w.k * g.JM + w.j) * g.IM + w.i);
      if (wait) {
        b.cell[s] = at;   // P1, where the walk continues
      } else {
        lost = w.lost || !w.concluded;
        store_located32(b, s, at, lost, w.dv);
        cell = lost ? -1 : at;
      }
    } else {
      lost = (cell < 0);
    }
    if (!wait) {
      const unsigned int key =
          settle_key32(lost, cell, px, py, pz, drop_removed, bbox, fbox, sentinel, m.lost, m.oob, m.lost_total);
      keys[s] = key;
      if (key < sentinel) hkey = key;
      else if (!drop_removed) hkey = sentinel;
    }
  }
  if (FIRST) {   // the warp's pending slots as a bit mask and its count (scanned, then compacted)
    const unsigned int mask = __ballot_sync(0xffffffffu, s < n_cap && wait);
    const int W = (n_cap + 31) >> 5, w = s >> 5;
    if ((threadIdx.x & 31) == 0 && w < W) {
      pending[w] = mask;
      pending[W + w] = (unsigned int)__popc(mask);
      if (w == 0) pending[2 * W] = 0u;
    }
  }
  const unsigned int r = warp_histogram_rank(hkey, count);
  if (hkey != 0xffffffffu) rank[s] = r;
  block_flush_counts(m, cnt);
}

// pf = the warps' masks [W], then the exclusive scan of their counts [W + 1]: warp w's pending
// slots go to list[scan[w]...] in ascending order, which keeps the slot (cell) order.
__global__ void k_compact_pending(const unsigned int *__restrict__ pf, int n_cap, unsigned int *__restrict__ list,
                                  DevCounters *cnt) {
  const int W = (n_cap + 31) >> 5;
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w == 0) cnt->pending = pf[2 * W];
  if (w < W) {
    unsigned int m = pf[w], o = pf[W + w];
    while (m) {
      list[o++] = (unsigned int)(32 * w + __ffs((int)m) - 1);
      m &= m - 1u;
    }
  }
}

// The pending particles of the learned form (the list from k_locate32<true>; b.cell[s] holds P1,
// the reference walk's second cell): the reference walk from P1, exactly as the FP32 form walks
// it, with the plane-table rows of the path the network predicts -- P1 stepping one index per
// axis toward the guessed cell -- prefetched into L1 ahead of the walk (`lookahead` cells after
// P1).  Whatever the guess, the cells, weights and statuses are the reference walk's; a good
// guess turns the walk's dependent row loads into L1 hits.  Grid-stride over the list with a
// warp-uniform trip count; path_hits counts the evaluations whose row was prefetched.
__device__ __forceinline__ void prefetch_row_l1(const float *row) {   // a row is one 128-B line
  asm volatile("prefetch.global.L1 [%0];" ::"l"(row));
}

// FAR: in a run that may hold particles without a previous cell (walk_ref32): one of them, whose walk crosses
// the grid, holds the whole launch.  First step after a setup that kept 3,000 LOST of 100,000 (1024 cells along
// k): 2.13 ms without, 1.08 with; elsewhere the registers of those evaluations cost more (64M particles, 527
// against 534 us).
template <bool FAR>
__global__ void __launch_bounds__(FDF_GUESS_THREADS, FDF_GUESS_MIN_BLOCKS) k_locate32_path(SwarmBuf b, GridDims g, const float *__restrict__ table,
                                                        const double *__restrict__ planes,
                                                        const double *__restrict__ bbox,
                                                        const float *__restrict__ fbox, int drop_removed,
                                                        DevCounters *cnt, unsigned int *__restrict__ keys,
                                                        unsigned int *__restrict__ rank,
                                                        unsigned int *__restrict__ count, unsigned int sentinel,
                                                        const unsigned int *__restrict__ pending,
                                                        const int *__restrict__ guess, int lookahead) {
  const unsigned int npend = (unsigned int)cnt->pending;   // at most FDF_MAX_PARTICLES = 2^29
  const unsigned int stride = gridDim.x * blockDim.x;
  const unsigned int lane = threadIdx.x & 31;
  unsigned int pev = 0, hits = 0;
  LocCounts m;
  for (unsigned int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < npend; base += stride) {
    const unsigned int t = base + lane;
    unsigned int hkey = 0xffffffffu;
    int s = 0;
    if (t < npend) {
      s = (int)pending[t];
      const float2 px = ld_pair(b.x, s), py = ld_pair(b.y, s), pz = ld_pair(b.z, s);
      Walk32 w;
      cell_ijk(g, (unsigned int)b.cell[s], w.i, w.j, w.k);
      int gi, gj, gk;
      cell_ijk(g, (unsigned int)guess[t], gi, gj, gk);
      // P1 and the guess lie in the grid, so does every cell of the path between them
      for (int q = 1; q <= lookahead; ++q) {
        const int ci = path_index(w.i, gi, q), cj = path_index(w.j, gj, q), ck = path_index(w.k, gk, q);
        prefetch_row_l1(table + (size_t)(((unsigned int)ck * g.JM + cj) * g.IM + ci) * FDF_ROW32);
        if (ci == gi && cj == gj && ck == gk) break;   // the predicted path has reached the guess
      }
      Path32 path{w.i, w.j, w.k, gi, gj, gk, 0u};
      walk_ref32<false, true, false, FAR>(table, planes, g, px, py, pz, FDF_MAX_TRAVERSAL - 1, w, cnt, 0.0, 0.0, 0.0,
                                          &path);
      hits += path.hits;
      if (w.degenerate) m.err |= ERRBIT_DEGENERATE;
      pev += w.evaluated();
      const bool lost = w.lost || !w.concluded;
      const int at = (int)(((long long)w.k * g.JM + w.j) * g.IM + w.i);
      store_located32(b, s, at, lost, w.dv);
      const int cell = lost ? -1 : at;
      const unsigned int key =
          settle_key32(lost, cell, px, py, pz, drop_removed, bbox, fbox, sentinel, m.lost, m.oob, m.lost_total);
      keys[s] = key;
      if (key < sentinel) hkey = key;
      else if (!drop_removed) hkey = sentinel;
    }
    const unsigned int r = warp_histogram_rank(hkey, count);
    if (hkey != 0xffffffffu) rank[s] = r;
  }
  m.done = m.evals = pev;
  block_flush_counts(m, cnt);
  block_add_u64(hits, &cnt->guess_taken_total);
  block_add_u64(pev, &cnt->guess_evals_total);
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&cnt->guess_asked_total, (unsigned long long)npend);
}

// UpdateAllParticlePositions in the precision form: fl32(v dt) added to the (hi, lo) position,
// as the fused step does it.
__global__ void k_advect32(SwarmBuf b, float dt32, DevCounters *cnt) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s == 0) atomicAdd(&cnt->psteps_total, (unsigned long long)cnt->n_sorted);   // particles advanced
  if (s >= cnt->n_sorted) return;
  st_pair(b.x, s, pair_add(ld_pair(b.x, s), __fmul_rn(b.uf[s], dt32)));
  st_pair(b.y, s, pair_add(ld_pair(b.y, s), __fmul_rn(b.vf[s], dt32)));
  st_pair(b.z, s, pair_add(ld_pair(b.z, s), __fmul_rn(b.wf[s], dt32)));
}

// Sort keys of the particles held (a re-sort by cell), dropping the LOST ones
// (CheckAndRemoveLostParticles, ParticleMotion.c:532-625) and/or the ones outside the
// bounding box (CheckAndRemoveOutOfBoundsParticles, :283-383; the FP32 form decides as the
// step does).  Kept particles without a cell go to the LOST bucket at the end; the removed
// ones get key all ones and no slot.
template <bool F32>
__global__ void __launch_bounds__(256) k_resort_keys(SwarmBuf b, GridDims g, int remove_lost, int remove_oob,
                                                    const double *__restrict__ bbox, const float *__restrict__ fbox,
                                                    DevCounters *cnt, unsigned int *__restrict__ keys,
                                                    unsigned int *__restrict__ rank, unsigned int *__restrict__ count,
                                                    unsigned int sentinel) {
  const int n = cnt->n_sorted;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  LocCounts m;
  unsigned int hkey = 0xffffffffu;
  if (s < n) {
    const int cell = b.cell[s];
    unsigned int key = (cell >= 0 && (long long)cell < g.Nc) ? (unsigned int)cell : sentinel;
    if (remove_lost && b.status[s] == ST_LOST) {
      m.lost += 1;
      key = 0xffffffffu;
    } else if (remove_oob) {
      bool inside;
      if (F32) {
        const float2 px = ld_pair(b.x, s), py = ld_pair(b.y, s), pz = ld_pair(b.z, s);
        unsigned int l0 = 0, o1 = 0, l2 = 0;
        inside = settle_key32(false, 0, px, py, pz, 1, bbox, fbox, sentinel, l0, o1, l2) != sentinel;
      } else {
        const double x = b.x[s], y = b.y[s], z = b.z[s];
        inside = x >= bbox[0] && x <= bbox[3] && y >= bbox[1] && y <= bbox[4] && z >= bbox[2] && z <= bbox[5];
      }
      if (!inside) {
        m.oob += 1;
        key = 0xffffffffu;
      }
    }
    keys[s] = key;
    hkey = key;
  }
  const unsigned int r = warp_histogram_rank(hkey, count);
  if (hkey != 0xffffffffu) rank[s] = r;
  block_flush_counts(m, cnt);
}

// Corner field in FP32: mean of the valid adjacent cells.  A thread carries NK nodes up the k
// direction and keeps each layer's four cells for the next node: 12 loads a node instead of 24, and the
// neighbours' indices and bounds once a column.  (One node per thread was bound by issue: 296
// instructions a node, 73 % of the issue slots.  14M cells beside the sort: 182 us then, 108 now; columns
// of 8 nodes 104, of 2 125, but a small grid then has too few threads.)
template <int NK>
__global__ void __launch_bounds__(256) k_center_to_corner32(const float *__restrict__ ucat, GridDims g,
                                                           float *__restrict__ corner) {
  const unsigned int layer = (unsigned int)(g.IM + 1) * (unsigned int)(g.JM + 1);
  const unsigned int across_blocks = (layer + 255u) / 256u, up = blockIdx.x / across_blocks;
  const unsigned int q = (blockIdx.x - up * across_blocks) * 256u + threadIdx.x;
  if (q >= layer) return;
  const unsigned int j = g.fMX.div(q), i = q - j * (unsigned int)(g.IM + 1);
  const unsigned int IM = g.IM, JM = g.JM, KM = g.KM, k0 = up * NK;
  // the column's four cells of a layer, in (dj, di) order
  const bool in[4] = {j > 0 && i > 0, j > 0 && i < IM, j < JM && i > 0, j < JM && i < IM};
  const unsigned int at[4] = {(j - 1) * IM + i - 1, (j - 1) * IM + i, j * IM + i - 1, j * IM + i};
  const int across = (in[0] ? 1 : 0) + (in[1] ? 1 : 0) + (in[2] ? 1 : 0) + (in[3] ? 1 : 0);
  float lo[3][4], hi[3][4];   // the layers below and above the node
  auto load = [&](unsigned int kc, float (&v)[3][4]) {
    const unsigned int base = kc * (IM * JM);
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int e = 0; e < 4; ++e) v[d][e] = kc < KM && in[e] ? __ldg(ucat + d * g.Nc + (base + at[e])) : 0.f;
  };
  load(k0 - 1u, lo);   // k0 = 0: no such layer
#pragma unroll
  for (int m = 0; m < NK; ++m) {
    const unsigned int k = k0 + m;
    if (k > KM) return;
    load(k, hi);
    const int cells = ((k > 0 ? 1 : 0) + (k < KM ? 1 : 0)) * across;
    const float r = cells == 8 ? 0.125f : cells == 4 ? 0.25f : cells == 2 ? 0.5f : cells == 1 ? 1.0f : 0.0f;
    const unsigned int node = k * layer + q;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      // the sum of the valid cells in order, from zero; a cell that is not there adds zero to it (a sum
      // that is -0 by then is +0 after the first addition either way)
      float t = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) t += lo[d][e];
#pragma unroll
      for (int e = 0; e < 4; ++e) t += hi[d][e];
      corner[d * g.Nn + node] = t * r;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int e = 0; e < 4; ++e) lo[d][e] = hi[d][e];
  }
}

// What the gather takes of a particle, as one aligned 64-byte record: positions, pid | weights, P | cell.
__global__ void __launch_bounds__(256) k_pack32(SwarmBuf b, const DevCounters *cnt, uint4 *__restrict__ rec) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= cnt->n_sorted) return;
  const ulonglong2 xy = make_ulonglong2(fdfx::ubits(b.x[p]), fdfx::ubits(b.y[p]));
  const ulonglong2 zp = make_ulonglong2(fdfx::ubits(b.z[p]), (unsigned long long)b.pid[p]);
  uint4 *r = rec + 4 * (size_t)p;
  *reinterpret_cast<ulonglong2 *>(r) = xy;
  *reinterpret_cast<ulonglong2 *>(r + 1) = zp;
  r[2] = make_uint4(__float_as_uint(b.a1f[p]), __float_as_uint(b.a2f[p]), __float_as_uint(b.a3f[p]),
                    __float_as_uint(b.Pf[p]));
  r[3] = make_uint4((unsigned int)b.cell[p], 0u, 0u, 0u);
}

// REC: the particles come from k_pack32's records (mode GATHER_INTERP).
template <bool REC>
__global__ void __launch_bounds__(256) k_gather_interp32(SwarmBuf src, SwarmBuf dst, GridDims g,
                                                         const float *__restrict__ corner,
                                                         const unsigned int *__restrict__ perm,
                                                         const unsigned int *__restrict__ cell_start,
                                                         DevCounters *cnt, int mode, const uint4 *__restrict__ rec) {
  const int n = (int)cell_start[g.Nc + 1];
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s == 0) {
    cnt->n = (int)cell_start[g.Nc];
    cnt->n_sorted = n;
  }
  if (s >= n) return;
  const unsigned int p = perm ? perm[s] : (unsigned int)s;
  int cell;
  float a1, a2, a3;
  unsigned char st = 0;
  if (REC) {
    const uint4 *r = rec + 4 * (size_t)p;
    const ulonglong2 xy = *reinterpret_cast<const ulonglong2 *>(r), zp = *reinterpret_cast<const ulonglong2 *>(r + 1);
    const uint4 wp = r[2];
    cell = (int)r[3].x;
    a1 = __uint_as_float(wp.x); a2 = __uint_as_float(wp.y); a3 = __uint_as_float(wp.z);
    dst.x[s] = __longlong_as_double((long long)xy.x); dst.y[s] = __longlong_as_double((long long)xy.y); dst.z[s] = __longlong_as_double((long long)zp.x);
    dst.Pf[s] = __uint_as_float(wp.w);
    dst.pid[s] = (long long)zp.y;
  } else {
    cell = src.cell[p];
    a1 = src.a1f[p]; a2 = src.a2f[p]; a3 = src.a3f[p];
    st = src.status[p];
    dst.x[s] = src.x[p]; dst.y[s] = src.y[p]; dst.z[s] = src.z[p];
    dst.Pf[s] = src.Pf[p];
    dst.pid[s] = src.pid[p];
  }
  dst.a1f[s] = a1; dst.a2f[s] = a2; dst.a3f[s] = a3;
  if (!REC && mode == GATHER_COPY) {
    dst.uf[s] = src.uf[p]; dst.vf[s] = src.vf[p]; dst.wf[s] = src.wf[p];
    dst.cell[s] = cell;
    dst.status[s] = st;
    return;
  }
  float ux = 0.f, uy = 0.f, uz = 0.f;
  if (cell < 0) {
    dst.cell[s] = -1;
    dst.status[s] = REC || mode == GATHER_INTERP ? (unsigned char)ST_LOST : st;
  } else {
    dst.cell[s] = cell;
    dst.status[s] = REC || mode == GATHER_INTERP ? (unsigned char)ST_ACTIVE_AND_LOCATED : st;
    int i, j, k;
    cell_ijk(g, (unsigned int)cell, i, j, k);
    a1 = fminf(fmaxf(a1, 0.f), 1.f);   // NaN -> 0 as PetscMax(0, PetscMin(1, NaN))
    a2 = fminf(fmaxf(a2, 0.f), 1.f);
    a3 = fminf(fmaxf(a3, 0.f), 1.f);
    const float oa1 = 1.f - a1, oa2 = 1.f - a2, oa3 = 1.f - a3;
    const float p00 = oa1 * oa2, p10 = a1 * oa2, p01 = oa1 * a2, p11 = a1 * a2;
    const float w[8] = {p00 * oa3, p10 * oa3, p01 * oa3, p11 * oa3, p00 * a3, p10 * a3, p01 * a3, p11 * a3};
    const long long mx = g.IM + 1, my = g.JM + 1;
    const long long q0 = ((long long)k * my + j) * mx + i;
    const long long off[8] = {0, 1, mx, mx + 1, mx * my, mx * my + 1, mx * my + mx, mx * my + mx + 1};
    float sw = 0.f, ax = 0.f, ay = 0.f, az = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const long long q = q0 + off[c];
      ax = fmaf(w[c], __ldg(corner + q), ax);
      ay = fmaf(w[c], __ldg(corner + g.Nn + q), ay);
      az = fmaf(w[c], __ldg(corner + 2 * g.Nn + q), az);
      sw += w[c];
    }
    if (sw > 1.0e-14f) { ux = ax / sw; uy = ay / sw; uz = az / sw; }
  }
  dst.uf[s] = ux; dst.vf[s] = uy; dst.wf[s] = uz;
}

// Neumaier-compensated running sum.
struct KSum {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float v) {
    float t = s + v;
    if (fabsf(s) >= fabsf(v)) c += (s - t) + v; else c += (v - t) + s;
    s = t;
  }
  __device__ __forceinline__ float value() const { return s + c; }
};

// Resident 256-thread blocks per SM the volume and the momentum deposits are compiled for.  The
// per-node chains wait on their loads, so 2048 resident threads (32 registers, a few spilled)
// beat the 48-register default for the volume deposit (64-bit indices: 0.617 -> 0.532 ms per
// 64M-particle step; 0.558 at 5 blocks, 0.550 at 6); 1024 (64 registers) beat 768 (80) for the momentum deposit:
// 2.95 -> 2.88 ms per 128M-particle step.
#ifndef FDF_DEP32_MIN_BLOCKS
#define FDF_DEP32_MIN_BLOCKS 8
#endif
#ifndef FDF_DEPM32_MIN_BLOCKS
#define FDF_DEPM32_MIN_BLOCKS 4
#endif
// CH: particles of a segment whose loads are issued before their in-order adds (the own cell's half of
// that).  Where the particles are fewer than the cells most segments hold none or one, and the chunk's
// idle entries only take issue slots, which bound this kernel: 6M particles in 14M cells 218 us with 4,
// 232 with 8; above, the loads' latency counts, 64M particles 477 us with 8, 495 with 4.  (Every index
// is 32 bits: with 64-bit ones a node took 550 instructions, 268 and 521 us.)
template <bool MOM, int CH>
__global__ void __launch_bounds__(256, MOM ? FDF_DEPM32_MIN_BLOCKS : FDF_DEP32_MIN_BLOCKS)
    k_deposit32(SwarmBuf b, GridDims g, const unsigned int *__restrict__ cs, float third, float *__restrict__ count,
                float *__restrict__ avg, float *__restrict__ fi, float *__restrict__ fj, float *__restrict__ fk,
                float *__restrict__ mi, float *__restrict__ mj, float *__restrict__ mk) {
  const unsigned int q = blockIdx.x * blockDim.x + threadIdx.x;   // below 2^31, as every index here
  if (q >= (unsigned int)g.Nn) return;
  const unsigned int IM = g.IM, JM = g.JM, KM = g.KM;
  unsigned int i, j, k;
  {
    int ii, jj, kk;
    node_ijk(g, q, ii, jj, kk);
    i = ii; j = jj; k = kk;
  }
  const unsigned int row = k * JM + j, c = row * IM + i;   // the cell's row and id, were (i, j, k) a cell
  const bool face_i = j < JM && k < KM, face_j = i < IM && k < KM, face_k = i < IM && j < JM;
  const bool is_cell = face_i && i < IM;
  unsigned int s0 = 0u, s1 = 0u;
  if (face_i) s0 = s1 = __ldg(cs + c);   // (i = IM: where the row's last cell ends)
  if (is_cell) s1 = __ldg(cs + c + 1u);
  // per face the lower cell's segment first, then this cell's; the three lower segments run
  // first and this cell's segment then feeds the P sum and the three upper parts in one pass
  // (every accumulator receives its values in the same order as face by face)
  KSum acc[3], mm[3][3];
  auto lower = [&](int f, const float *__restrict__ wgt, unsigned int l0, unsigned int l1) {
    for (unsigned int s = l0; s < l1; s += CH) {
      float a[CH], u[CH], v[CH], w[CH];
#pragma unroll
      for (int e = 0; e < CH; ++e) {
        const bool in = s + e < l1;
        a[e] = in ? __ldg(wgt + s + e) : 0.f;
        if (MOM) {
          u[e] = in ? __ldg(b.uf + s + e) : 0.f;
          v[e] = in ? __ldg(b.vf + s + e) : 0.f;
          w[e] = in ? __ldg(b.wf + s + e) : 0.f;
        }
      }
#pragma unroll
      for (int e = 0; e < CH; ++e) {
        if (s + e >= l1) break;
        const float fr = a[e] * third;
        acc[f].add(fr);
        if (MOM) { mm[f][0].add(fr * u[e]); mm[f][1].add(fr * v[e]); mm[f][2].add(fr * w[e]); }
      }
    }
  };
  if (face_i && i > 0) lower(0, b.a1f, __ldg(cs + c - 1u), s0);
  if (face_j && j > 0) lower(1, b.a2f, __ldg(cs + c - IM), __ldg(cs + c - IM + 1u));
  if (face_k && k > 0) lower(2, b.a3f, __ldg(cs + c - IM * JM), __ldg(cs + c - IM * JM + 1u));
  KSum sum;
  constexpr int OCH = MOM ? CH : (CH + 1) / 2;
  for (unsigned int s = s0; s < s1; s += OCH) {
    float P[OCH], w[OCH][3], u[OCH], v[OCH], ww[OCH];
#pragma unroll
    for (int e = 0; e < OCH; ++e) {
      const bool in = s + e < s1;
      P[e] = in ? __ldg(b.Pf + s + e) : 0.f;
      w[e][0] = in ? __ldg(b.a1f + s + e) : 0.f;
      w[e][1] = in ? __ldg(b.a2f + s + e) : 0.f;
      w[e][2] = in ? __ldg(b.a3f + s + e) : 0.f;
      if (MOM) {
        u[e] = in ? __ldg(b.uf + s + e) : 0.f;
        v[e] = in ? __ldg(b.vf + s + e) : 0.f;
        ww[e] = in ? __ldg(b.wf + s + e) : 0.f;
      }
    }
#pragma unroll
    for (int e = 0; e < OCH; ++e) {
      if (s + e >= s1) break;
      sum.add(P[e]);
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        const float fr = (1.f - w[e][f]) * third;
        acc[f].add(fr);
        if (MOM) { mm[f][0].add(fr * u[e]); mm[f][1].add(fr * v[e]); mm[f][2].add(fr * ww[e]); }
      }
    }
  }
  {
    const unsigned int nc = s1 - s0;
    count[q] = (float)nc;
    avg[q] = nc > 0 ? sum.value() / (float)nc : 0.f;
  }
  auto store = [&](int f, float *vol, float *mom, long long nf, unsigned int at) {
    vol[at] = acc[f].value();
    if (MOM) { mom[at] = mm[f][0].value(); mom[nf + at] = mm[f][1].value(); mom[2 * nf + at] = mm[f][2].value(); }
  };
  // (row (IM + 1) + i, (k (JM + 1) + j) IM + i, c)
  if (face_i) store(0, fi, mi, MOM ? (IM + 1LL) * JM * KM : 0, c + row);
  if (face_j) store(1, fj, mj, MOM ? IM * (JM + 1LL) * KM : 0, c + k * IM);
  if (face_k) store(2, fk, mk, MOM ? (long long)IM * JM * (KM + 1LL) : 0, c);
}

__global__ void k_from_aos32(const double *__restrict__ pos, const double *__restrict__ vel,
                             const double *__restrict__ wgt, const double *__restrict__ P,
                             const long long *__restrict__ cell3, const long long *__restrict__ pid,
                             const long long *__restrict__ status, int n, GridDims g, SwarmBuf b) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  for (int q = 0; q < 3; ++q) {
    const double v = pos[3 * p + q];
    const float h = __double2float_rn(v);
    const float l = __double2float_rn(__dsub_rn(v, (double)h));
    st_pair(q == 0 ? b.x : q == 1 ? b.y : b.z, p, make_float2(h, l));
  }
  b.uf[p] = (float)vel[3 * p]; b.vf[p] = (float)vel[3 * p + 1]; b.wf[p] = (float)vel[3 * p + 2];
  b.a1f[p] = (float)wgt[3 * p]; b.a2f[p] = (float)wgt[3 * p + 1]; b.a3f[p] = (float)wgt[3 * p + 2];
  b.Pf[p] = (float)P[p];
  b.pid[p] = pid[p];
  const long long i = cell3[3 * p], j = cell3[3 * p + 1], k = cell3[3 * p + 2];
  int c = -1;
  if (i >= 0 && i < g.IM && j >= 0 && j < g.JM && k >= 0 && k < g.KM) c = (int)((k * g.JM + j) * g.IM + i);
  b.cell[p] = c;
  const long long st = status[p];
  b.status[p] = (unsigned char)((st >= 0 && st <= ST_UNINITIALIZED) ? st : ST_UNINITIALIZED);
}

__global__ void k_to_aos32(SwarmBuf b, int n, GridDims g, double *__restrict__ pos, double *__restrict__ vel,
                           double *__restrict__ wgt, double *__restrict__ P, long long *__restrict__ cell3,
                           long long *__restrict__ pid, long long *__restrict__ status) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  pos[3 * p] = pair_value(ld_pair(b.x, p));
  pos[3 * p + 1] = pair_value(ld_pair(b.y, p));
  pos[3 * p + 2] = pair_value(ld_pair(b.z, p));
  vel[3 * p] = b.uf[p]; vel[3 * p + 1] = b.vf[p]; vel[3 * p + 2] = b.wf[p];
  wgt[3 * p] = b.a1f[p]; wgt[3 * p + 1] = b.a2f[p]; wgt[3 * p + 2] = b.a3f[p];
  P[p] = b.Pf[p];
  pid[p] = b.pid[p];
  const int c = b.cell[p];
  if (c >= 0) {
    int i, j, k;
    cell_ijk(g, (unsigned int)c, i, j, k);
    cell3[3 * p] = i; cell3[3 * p + 1] = j; cell3[3 * p + 2] = k;
  } else {
    cell3[3 * p] = -1; cell3[3 * p + 1] = -1; cell3[3 * p + 2] = -1;
  }
  status[p] = b.status[p];
}

// Layout conversion straight from / to the caller's page-locked DMSwarm arrays over the host
// link.  A block stages 256 particles' AoS records (15 x 8 B each: position, velocity, weights,
// P, cell triple, PID, status) in shared memory, moving each field's contiguous range with
// coalesced 16-byte accesses -- the access pattern that reaches the link's copy rate -- and each
// thread converts its own particle to or from the device SoA buffers as the per-particle
// kernels above do.  The arrays must be 16-byte aligned.
constexpr int XF_TILE = 256;
// field f: doubles per particle, and the field's offset in the shared tile (in doubles)
__host__ __device__ constexpr int xf_bs(int f) { return (f < 3 || f == 4) ? 3 : 1; }
__host__ __device__ constexpr int xf_off(int f) { return XF_TILE * (f <= 3 ? 3 * f : f == 4 ? 10 : f == 5 ? 13 : 14); }

struct HostSwarm {
  const double *f[7];   // position, velocity, weight, P, cell (int64), pid (int64), status (int64)
};

__device__ __forceinline__ void tile_in(double *dst, const double *__restrict__ src, int count) {
  const double2 *s2 = reinterpret_cast<const double2 *>(src);
  double2 *d2 = reinterpret_cast<double2 *>(dst);
  for (int q = threadIdx.x; q < count / 2; q += XF_TILE) d2[q] = s2[q];
  if ((count & 1) && threadIdx.x == 0) dst[count - 1] = src[count - 1];
}
__device__ __forceinline__ void tile_out(double *__restrict__ dst, const double *src, int count) {
  const double2 *s2 = reinterpret_cast<const double2 *>(src);
  double2 *d2 = reinterpret_cast<double2 *>(dst);
  for (int q = threadIdx.x; q < count / 2; q += XF_TILE) d2[q] = s2[q];
  if ((count & 1) && threadIdx.x == 0) dst[count - 1] = src[count - 1];
}

template <bool F32>
__global__ void __launch_bounds__(XF_TILE) k_from_host(HostSwarm h, int n, GridDims g, SwarmBuf b) {
  __shared__ __align__(16) double sm[15 * XF_TILE];
  const int p0 = blockIdx.x * XF_TILE, m = min(XF_TILE, n - p0);
#pragma unroll
  for (int f = 0; f < 7; ++f) tile_in(sm + xf_off(f), h.f[f] + (long long)xf_bs(f) * p0, xf_bs(f) * m);
  __syncthreads();
  const int t = threadIdx.x;
  if (t >= m) return;
  const int p = p0 + t;
  const double *pos = sm + xf_off(0) + 3 * t, *vel = sm + xf_off(1) + 3 * t, *wgt = sm + xf_off(2) + 3 * t;
  const long long *c3 = reinterpret_cast<const long long *>(sm + xf_off(4)) + 3 * t;
  if (F32) {
    st_pair(b.x, p, fdfx::split_rn(pos[0])); st_pair(b.y, p, fdfx::split_rn(pos[1])); st_pair(b.z, p, fdfx::split_rn(pos[2]));
    b.uf[p] = fdfx::d2f_rn(vel[0]); b.vf[p] = fdfx::d2f_rn(vel[1]); b.wf[p] = fdfx::d2f_rn(vel[2]);
    b.a1f[p] = fdfx::d2f_rn(wgt[0]); b.a2f[p] = fdfx::d2f_rn(wgt[1]); b.a3f[p] = fdfx::d2f_rn(wgt[2]);
    b.Pf[p] = fdfx::d2f_rn(sm[xf_off(3) + t]);
  } else {
    b.x[p] = pos[0]; b.y[p] = pos[1]; b.z[p] = pos[2];
    b.u[p] = vel[0]; b.v[p] = vel[1]; b.w[p] = vel[2];
    b.a1[p] = wgt[0]; b.a2[p] = wgt[1]; b.a3[p] = wgt[2];
    b.P[p] = sm[xf_off(3) + t];
  }
  b.pid[p] = reinterpret_cast<const long long *>(sm + xf_off(5))[t];
  const long long i = c3[0], j = c3[1], k = c3[2];
  int c = -1;
  if (i >= 0 && i < g.IM && j >= 0 && j < g.JM && k >= 0 && k < g.KM) c = (int)((k * g.JM + j) * g.IM + i);
  b.cell[p] = c;
  const long long st = reinterpret_cast<const long long *>(sm + xf_off(6))[t];
  b.status[p] = (unsigned char)((st >= 0 && st <= ST_UNINITIALIZED) ? st : ST_UNINITIALIZED);
}

template <bool F32>
__global__ void __launch_bounds__(XF_TILE) k_to_host(SwarmBuf b, int n, GridDims g, HostSwarm h) {
  __shared__ __align__(16) double sm[15 * XF_TILE];
  const int p0 = blockIdx.x * XF_TILE, m = min(XF_TILE, n - p0);
  const int t = threadIdx.x;
  if (t < m) {
    const int p = p0 + t;
    double *pos = sm + xf_off(0) + 3 * t, *vel = sm + xf_off(1) + 3 * t, *wgt = sm + xf_off(2) + 3 * t;
    if (F32) {
      pos[0] = pair_value(ld_pair(b.x, p)); pos[1] = pair_value(ld_pair(b.y, p)); pos[2] = pair_value(ld_pair(b.z, p));
      vel[0] = b.uf[p]; vel[1] = b.vf[p]; vel[2] = b.wf[p];
      wgt[0] = b.a1f[p]; wgt[1] = b.a2f[p]; wgt[2] = b.a3f[p];
      sm[xf_off(3) + t] = b.Pf[p];
    } else {
      pos[0] = b.x[p]; pos[1] = b.y[p]; pos[2] = b.z[p];
      vel[0] = b.u[p]; vel[1] = b.v[p]; vel[2] = b.w[p];
      wgt[0] = b.a1[p]; wgt[1] = b.a2[p]; wgt[2] = b.a3[p];
      sm[xf_off(3) + t] = b.P[p];
    }
    long long *c3 = reinterpret_cast<long long *>(sm + xf_off(4)) + 3 * t;
    const int c = b.cell[p];
    if (c >= 0) {
      int i, j, k;
      cell_ijk(g, (unsigned int)c, i, j, k);
      c3[0] = i; c3[1] = j; c3[2] = k;
    } else {
      c3[0] = -1; c3[1] = -1; c3[2] = -1;
    }
    reinterpret_cast<long long *>(sm + xf_off(5))[t] = b.pid[p];
    reinterpret_cast<long long *>(sm + xf_off(6))[t] = b.status[p];
  }
  __syncthreads();
#pragma unroll
  for (int f = 0; f < 7; ++f)
    tile_out(const_cast<double *>(h.f[f]) + (long long)xf_bs(f) * p0, sm + xf_off(f), xf_bs(f) * m);
}

__global__ void k_f32_to_f64(const float *__restrict__ in, double *__restrict__ out, long long n) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q < n) out[q] = (double)in[q];
}

inline unsigned int blocks_for(long long n, int th) { return (unsigned int)(n > 0 ? (n + th - 1) / th : 1); }

}  // namespace

void launch_build_table32(const double *planes, const double *coor, GridDims g, float *table, cudaStream_t s) {
  k_build_table32<<<blocks_for(g.Nc, 128), 128, 0, s>>>(planes, coor, g, table);
}

void launch_locate32(const SwarmBuf &b, int n_cap, GridDims g, const float *table, const double *planes, double dt,
                     int advect, const double *bbox, const float *fbox, int drop_removed, DevCounters *cnt,
                     unsigned int *keys, unsigned int *rank, unsigned int *count, unsigned int sentinel,
                     unsigned int *pending, float far_cells, bool from_nowhere, cudaStream_t s) {
  constexpr int th = FDF_LOC_THREADS;
  auto go = [&](auto kernel, unsigned int *pend, float far) {
    kernel<<<blocks_for(n_cap, th), th, 0, s>>>(b, g, table, planes, (float)dt, advect, drop_removed, bbox, fbox,
                                                drop_removed, cnt, keys, rank, count, sentinel, pend, n_cap, far);
  };
  // without the advection the particles come from anywhere (the initial setup's corner start)
  const bool dense = n_cap > g.Nc;
  if (pending && !from_nowhere && dense) go(k_locate32<true, false, true>, pending, far_cells);
  else if (pending && !from_nowhere) go(k_locate32<true, false, false>, pending, far_cells);
  else if (pending) go(k_locate32<true, true, false>, pending, far_cells);
  else if (advect && dense) go(k_locate32<false, false, true>, nullptr, 0.f);
  else if (advect) go(k_locate32<false, false, false>, nullptr, 0.f);
  else go(k_locate32<false, true, false>, nullptr, 0.f);
}

void launch_compact_pending(const unsigned int *scan, int n_cap, unsigned int *list, DevCounters *cnt,
                            cudaStream_t s) {
  k_compact_pending<<<blocks_for((n_cap + 31) / 32, 256), 256, 0, s>>>(scan, n_cap, list, cnt);
}

void launch_locate32_path(const SwarmBuf &b, int n_cap, GridDims g, const float *table, const double *planes,
                          const double *bbox, const float *fbox, int drop_removed, DevCounters *cnt,
                          unsigned int *keys, unsigned int *rank, unsigned int *count, unsigned int sentinel,
                          const unsigned int *pending, const int *guess, int num_sms, bool from_nowhere,
                          cudaStream_t s) {
  // grid-stride kernel: one wave of resident blocks, so that no SM runs a partial last wave
  static int resident = 0, res_device = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (res_device != dev) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, k_locate32_path<false>, FDF_GUESS_THREADS, 0);
    res_device = dev;   // (the same launch bounds: the same for <true>)
  }
  const long long need = ((long long)n_cap + FDF_GUESS_THREADS - 1) / FDF_GUESS_THREADS;
  long long blocks = (long long)num_sms * (resident > 0 ? resident : 1);
  if (blocks > need) blocks = need;
  auto *kernel = from_nowhere ? k_locate32_path<true> : k_locate32_path<false>;
  kernel<<<(unsigned)(blocks < 1 ? 1 : blocks), FDF_GUESS_THREADS, 0, s>>>(
      b, g, table, planes, bbox, fbox, drop_removed, cnt, keys, rank, count, sentinel, pending, guess,
      FDF_PATH_LOOKAHEAD);
}

void launch_center_to_corner32(const float *ucat, GridDims g, float *corner, cudaStream_t s) {
  constexpr int NK = 4;
  const unsigned int layer = (unsigned int)(g.IM + 1) * (unsigned int)(g.JM + 1);
  const unsigned int blocks = blocks_for(layer, 256) * (unsigned int)((g.KM + NK) / NK);   // KM + 1 layers of nodes
  k_center_to_corner32<NK><<<blocks, 256, 0, s>>>(ucat, g, corner);
}

void launch_advect32(const SwarmBuf &b, int n_cap, double dt, DevCounters *cnt, cudaStream_t s) {
  k_advect32<<<blocks_for(n_cap, 256), 256, 0, s>>>(b, (float)dt, cnt);
}

void launch_resort_keys(const SwarmBuf &b, int n_cap, GridDims g, int f32, int remove_lost, int remove_oob,
                        const double *bbox, const float *fbox, DevCounters *cnt, unsigned int *keys,
                        unsigned int *rank, unsigned int *count, unsigned int sentinel, cudaStream_t s) {
  if (f32)
    k_resort_keys<true><<<blocks_for(n_cap, 256), 256, 0, s>>>(b, g, remove_lost, remove_oob, bbox, fbox, cnt, keys,
                                                               rank, count, sentinel);
  else
    k_resort_keys<false><<<blocks_for(n_cap, 256), 256, 0, s>>>(b, g, remove_lost, remove_oob, bbox, fbox, cnt, keys,
                                                                rank, count, sentinel);
}

void launch_gather_interp32(const SwarmBuf &src, const SwarmBuf &dst, int n_cap, GridDims g, const float *corner,
                            const unsigned int *perm, const unsigned int *cell_start, DevCounters *cnt,
                            cudaStream_t s, int mode) {
  k_gather_interp32<false><<<blocks_for(n_cap, 256), 256, 0, s>>>(src, dst, g, corner, perm, cell_start, cnt, mode,
                                                                  nullptr);
}

void launch_gather_interp32_packed(const SwarmBuf &src, const SwarmBuf &dst, int n_cap, GridDims g, const float *corner,
                                   const unsigned int *perm, const unsigned int *cell_start, DevCounters *cnt, void *rec,
                                   cudaStream_t s) {
  uint4 *r = static_cast<uint4 *>(rec);
  k_pack32<<<blocks_for(n_cap, 256), 256, 0, s>>>(src, cnt, r);
  k_gather_interp32<true><<<blocks_for(n_cap, 256), 256, 0, s>>>(src, dst, g, corner, perm, cell_start, cnt,
                                                                 GATHER_INTERP, r);
}

void launch_deposit32(const SwarmBuf &b, int n_cap, GridDims g, const unsigned int *cell_start, double volume, float *count,
                      float *avg, float *fi, float *fj, float *fk, float *mi, float *mj, float *mk, cudaStream_t s) {
  constexpr int th = 256;
  const unsigned int blocks = blocks_for(g.Nn, th);
  const float third = (float)(volume / 3.0);
  if (mi)
    k_deposit32<true, 4><<<blocks, th, 0, s>>>(b, g, cell_start, third, count, avg, fi, fj, fk, mi, mj, mk);
  else if (n_cap <= g.Nc)
    k_deposit32<false, 4><<<blocks, th, 0, s>>>(b, g, cell_start, third, count, avg, fi, fj, fk, nullptr, nullptr, nullptr);
  else
    k_deposit32<false, 8><<<blocks, th, 0, s>>>(b, g, cell_start, third, count, avg, fi, fj, fk, nullptr, nullptr, nullptr);
}

void launch_swarm_from_aos32(const double *pos, const double *vel, const double *wgt, const double *P,
                             const long long *cell3, const long long *pid, const long long *status, int n, GridDims g,
                             const SwarmBuf &b, cudaStream_t s) {
  if (n <= 0) return;
  k_from_aos32<<<blocks_for(n, 256), 256, 0, s>>>(pos, vel, wgt, P, cell3, pid, status, n, g, b);
}

void launch_swarm_to_aos32(const SwarmBuf &b, int n, GridDims g, double *pos, double *vel, double *wgt, double *P,
                           long long *cell3, long long *pid, long long *status, cudaStream_t s) {
  if (n <= 0) return;
  k_to_aos32<<<blocks_for(n, 256), 256, 0, s>>>(b, n, g, pos, vel, wgt, P, cell3, pid, status);
}

void launch_swarm_from_host(const void *const f[7], int n, GridDims g, const SwarmBuf &b, bool f32, cudaStream_t s) {
  if (n <= 0) return;
  HostSwarm h;
  for (int q = 0; q < 7; ++q) h.f[q] = static_cast<const double *>(f[q]);
  const unsigned blocks = (unsigned)((n + XF_TILE - 1) / XF_TILE);
  if (f32) k_from_host<true><<<blocks, XF_TILE, 0, s>>>(h, n, g, b);
  else k_from_host<false><<<blocks, XF_TILE, 0, s>>>(h, n, g, b);
}

void launch_swarm_to_host(const SwarmBuf &b, int n, GridDims g, void *const f[7], bool f32, cudaStream_t s) {
  if (n <= 0) return;
  HostSwarm h;
  for (int q = 0; q < 7; ++q) h.f[q] = static_cast<const double *>(f[q]);
  const unsigned blocks = (unsigned)((n + XF_TILE - 1) / XF_TILE);
  if (f32) k_to_host<true><<<blocks, XF_TILE, 0, s>>>(b, n, g, h);
  else k_to_host<false><<<blocks, XF_TILE, 0, s>>>(b, n, g, h);
}

void launch_f32_to_f64(const float *in, double *out, long long n, cudaStream_t s) {
  k_f32_to_f64<<<blocks_for(n, 256), 256, 0, s>>>(in, out, n);
}
