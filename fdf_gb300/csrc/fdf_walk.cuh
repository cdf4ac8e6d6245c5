// fdf_walk.cuh -- the walking search's cell evaluation with exact decisions from the FP32
// plane table, shared by the plain FP64 walk (fdf_walk.cu) and the precision forms
// (fdf_fp32.cu).  EvaluateParticlePosition / DeterminePointPosition (walkingsearch.c:407-462,
// 811-859) and the index update of UpdateCellIndicesBasedOnDistancesTEST (:882-959).
//
// Each face class the walk needs -- d < 0, d == 0 (|d| < thr), d > 0 -- is decided from an
// FP32 signed distance when that is provably the FP64 class for the position, and from the
// exact FP64 distance (the FP64 plane table, the reference's arithmetic) otherwise.
//
// FP32 distance.  With c0 = c0h + c0l the cell's first vertex as a float pair (exact),
// P = p - c0, E = n . (fc - c0) and d = (fc - p) . n = E - n . P, the row holds n32 = fl32(n)
// and e32 = fl32(E64) (E64: E in FP64), and the kernel computes
//     pr_i = fl32(fl32(ph_i - c0h_i) + fl32(pl_i - c0l_i)),  d32 = e32 - (n32 . pr)
// (the dot product as an FMA chain, then one subtraction).  With B_i = |P_i|,
// ex_i = u (|ph_i| + |c0h_i|), u = 2^-24, eps = 2^-53 and A_i = |fc_i - c0_i|, the roundings
// are bounded by
//     |pr_i - P_i| <= 2u B_i + 2u ex_i                     (the pair subtraction)
//     |e32 - E| <= u |E| + 6 eps sum_i A_i |n_i|            (E64, then fl32)
//     dot product 3u, n32 u, the final subtraction u |d|, the reference's own d64 within
//     5 eps sum_i (A_i + B_i) |n_i| of d,
// which add up to
//     |d32 - d64| <= u S (1 + 12u) + 23 eps sigma,   S = 2 |e32| + 7 sum_i |n32_i| (|pr_i| + ex_i)
// with sigma = max over faces of sum_i A_i |n_i|.  A face's own margin is
//     M_f = fl32(4u S32 + base_f),   base_f = fl32(thr32 + slack) (in the row), slack >= 32 eps sigma,
// thr32 >= thr (1 + 2^-22) (both rounded up; S32: S in FP32, within 8u of S), and
//     d32 > M_f -> d64 >= thr (positive);  d32 < -M_f -> d64 <= -thr (negative).
// Most evaluations need no face's own margin, because one for the whole cell is passed by all six
// distances: the normals are unit vectors, so |n32_i| <= 1 + 2u and |e32| <= (1 + 2u) |d32| +
// (1 + 6u) A with A = sum_i (|pr_i| + ex_i); hence |d32| <= M_f implies |d32| (1 - 8.1u) <= 36.1u A +
// base_f, which the cell's margin
//     M = fl32(40 u sum_i |pr_i| + X + base),   X = fl32(40 u^2 sum_i |ph_i|) (once per particle),
//     base >= (thr + 32 eps sigma + 40 u^2 sum_i |c0h_i|) (1 + 2^-19)        (in the row)
// exceeds: the smallest |d32| above M settles the six classes as the M_f would.  (It takes 10
// instructions where the six M_f take 60 of an evaluation's 150.)  Otherwise each face below M is
// decided by its M_f, and what M_f leaves open (including NaN) by the exact FP64 distance of that
// face.  A row whose values leave [-2^100, 2^100] has base = inf, which sends every face to its M_f.
// The cells, statuses and walk paths are therefore the reference's for the position.
// Fallbacks are counted.  The hot loop issues no FP64 instruction.
//
// Positions.  The precision forms hold each coordinate as a float pair (hi, lo) whose exact
// sum is the position.  The plain form walks its FP64 position x through its split
// (hi = fl32(x), lo = fl32(x - hi), within 2^-48 |x| <= u ex of x): that offset adds at most
// u sum_i |n_i| ex_i to the error, well inside the 7 sum_i |n32_i| ex_i of S, and the undecided
// faces are computed from x itself (EXACT), so every class is x's own.
//
// Per-cell FP32 row (128 B, one cache line, 8 chunks of 16 B): c0h (3 x f32), base (f32),
// c0l (3 x f32), base_f (f32, negative for a degenerate cell, whose base is inf), then per face LEFT..BACK: n32 (3 x f32), e32.
// Chunk q lies at position q ^ row32_swizzle(cell).  A warp's lanes read the same chunk of
// different rows; unswizzled these all fall on the same L1 banks and one 16-B load took 14
// wavefronts (L1's data pipe 84 % busy); swizzled they spread over the banks and it takes 5.
// The FP32 form's walk of 64M particles on 96x96x1536 cells at CFL 4: 3.19 ms unswizzled, with the
// per-face margins, calls for the exact distances and shuffled counter sums; 2.71 ms swizzled,
// with one REDUX per counter and no spill in the loop; 2.32 ms with one margin per cell.
#pragma once
#include "fdf_internal.cuh"
#include "fdf_exact.cuh"

namespace {

using fdfx::add;
using fdfx::mul;
using fdfx::sub;

__device__ __forceinline__ double pair_value(float2 p) { return __dadd_rn((double)p.x, (double)p.y); }

// Exact FP64 signed distance of face f (the plain path's arithmetic), thresholded.  INT: two of its three
// products on the integer pipe (the same bits).
template <bool INT = false>
__device__ __forceinline__ double exact_face(const double *__restrict__ row64, int f, double x, double y, double z) {
  const double2 *r = reinterpret_cast<const double2 *>(row64);
  double2 p0 = __ldg(r + 3 * f), p1 = __ldg(r + 3 * f + 1), p2 = __ldg(r + 3 * f + 2);
  double2 tf = __ldg(r + 18);
  const double tx = INT ? fdfx::mul_int(sub(p0.x, x), p1.y) : mul(sub(p0.x, x), p1.y);
  const double ty = INT ? fdfx::mul_int(sub(p0.y, y), p2.x) : mul(sub(p0.y, y), p2.x);
  double dd = add(add(tx, ty), mul(sub(p1.x, z), p2.y));
  if (fdfx::abs_lt_bits(dd, fdfx::ubits(tf.x), fdfx::is_nan(tf.x))) dd = 0.0;
  return dd;
}

// The reference walk from (i, j, k): its state, and where it ended.  dv: the distances of the last
// cell evaluated, whose classes are the FP64 distances' (dv < 0 exactly for the negative faces).
struct Walk32 {
  int i, j, k, steps;
  unsigned int saved;   // the cell of the last step 2^m - 1 (the cycle detection's)
  bool concluded, lost, cycle, degenerate;
  bool wait;            // FIRST: left its first cell far behind, the walk stops at the second
  float dv[6];
  // evaluations made: the step that ends a walk as lost (outside, a cycle, a degenerate cell) makes none
  __device__ __forceinline__ unsigned int evaluated() const { return (unsigned int)steps - (lost ? 1u : 0u); }
};

// The cell a walk from (i0, j0, k0) toward (ti, tj, tk) reaches after q steps if every step moves
// each index one closer (the reference's steps move each index by at most one).
__device__ __forceinline__ int path_index(int a0, int t, int q) { return a0 + max(-q, min(q, t - a0)); }

// The predicted path of the learned form's walk from P1, and the evaluations after the first whose
// cell is the one the path reaches after as many steps (the rows fetched ahead).
struct Path32 {
  int i0, j0, k0, ti, tj, tk;
  unsigned int hits;
  __device__ __forceinline__ void count(int i, int j, int k, int steps) {
    const int q = steps - 1;
    if (q > 0) hits += (i == path_index(i0, ti, q) && j == path_index(j0, tj, q) && k == path_index(k0, tk, q)) ? 1u : 0u;
  }
};

// X of the margin: the particle's part of 40 u sum_i ex_i.
__device__ __forceinline__ float walk_margin(float2 px, float2 py, float2 pz) {
  return __fmul_rn(__fadd_rn(__fadd_rn(fabsf(px.x), fabsf(py.x)), fabsf(pz.x)), 40.0f * 0x1p-48f);
}

// The row of cell cur: 128-byte aligned, so one XOR on this address reaches chunk q.
__device__ __forceinline__ size_t row32_address(const float *table, unsigned int cur) {
  return reinterpret_cast<size_t>(table + (size_t)cur * FDF_ROW32) ^ (row32_swizzle(cur) << 4);
}
__device__ __forceinline__ float4 row32_chunk(size_t row, unsigned int q) {
  return __ldg(reinterpret_cast<const float4 *>(row ^ (q << 4)));
}

// The same chunk loaded anew (the compiler does not see that it was loaded before).
__device__ __forceinline__ float4 row32_again(size_t row, unsigned int q) {
  float4 v;
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(row ^ (q << 4)));
  return v;
}

// pr and the six distances d32 of the header comment.
__device__ __forceinline__ void row32_distances(size_t row, float4 h0, float4 h1, float2 px, float2 py, float2 pz,
                                                float (&pr)[3], float (&dv)[6]) {
  float4 fr[6];   // per face: n32 (x, y, z), e32 (w); six 16-B loads
#pragma unroll
  for (int q = 0; q < 6; ++q) fr[q] = row32_chunk(row, 2 + q);
  pr[0] = __fadd_rn(__fsub_rn(px.x, h0.x), __fsub_rn(px.y, h1.x));
  pr[1] = __fadd_rn(__fsub_rn(py.x, h0.y), __fsub_rn(py.y, h1.y));
  pr[2] = __fadd_rn(__fsub_rn(pz.x, h0.z), __fsub_rn(pz.y, h1.z));
#pragma unroll
  for (int f = 0; f < 6; ++f)
    dv[f] = __fsub_rn(fr[f].w, __fmaf_rn(fr[f].z, pr[2], __fmaf_rn(fr[f].y, pr[1], __fmul_rn(fr[f].x, pr[0]))));
}

// Below zero when a face is negative (NaN distances are in no class).
__device__ __forceinline__ float walk_low(const Walk32 &w) {
  return fminf(fminf(fminf(w.dv[0], w.dv[1]), fminf(w.dv[2], w.dv[3])), fminf(w.dv[4], w.dv[5]));
}

// UpdateCellIndicesBasedOnDistancesTEST (walkingsearch.c:882-959).
__device__ __forceinline__ void walk_advance(Walk32 &w) {
  if (w.dv[F_FRONT] < 0.f) w.k += 1; else if (w.dv[F_BACK] < 0.f) w.k -= 1;
  if (w.dv[F_LEFT] < 0.f) w.i -= 1; else if (w.dv[F_RIGHT] < 0.f) w.i += 1;
  if (w.dv[F_BOTTOM] < 0.f) w.j -= 1; else if (w.dv[F_TOP] < 0.f) w.j += 1;
}

// The walk's next cell: its id in cur, or the end of the walk (false) outside the grid or at a cell
// met before (Brent's cycle detection: a revisited cell repeats forever, which the reference
// ends as LOST after MAX_TRAVERSAL evaluations).
template <bool FIRST>
__device__ __forceinline__ bool walk_enter(Walk32 &w, int IM, int JM, int KM, unsigned int &cur) {
  ++w.steps;
  if ((unsigned int)w.i >= (unsigned int)IM || (unsigned int)w.j >= (unsigned int)JM ||
      (unsigned int)w.k >= (unsigned int)KM) {
    w.lost = true;
    return false;
  }
  cur = ((unsigned int)w.k * JM + w.j) * IM + w.i;
  if (cur == w.saved) {
    w.cycle = true;
    w.lost = true;
    return false;
  }
  const int t = w.steps - (FIRST ? 1 : 0);   // FIRST: counted from the second cell
  if ((t & (t + 1)) == 0) w.saved = cur;
  return true;
}

// How far past the previous cell a particle is, in cells, from the first evaluation's
// distances: for each index direction with a negative face, -d_neg / (d_lower + d_upper)
// (the two planes' distances add up to the cell's width there).  Only steers which exact path
// the learned form takes, so it may be approximate; a degenerate width gives +inf.
__device__ __forceinline__ float beyond_cells(const float (&dv)[6]) {
  float far = 0.f;
  const int lo[3] = {F_LEFT, F_BOTTOM, F_BACK}, hi[3] = {F_RIGHT, F_TOP, F_FRONT};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float dl = dv[lo[a]], dh = dv[hi[a]], width = dl + dh;
    const float neg = dl < 0.f ? -dl : (dh < 0.f ? -dh : 0.f);
    if (neg > 0.f) far = fmaxf(far, width > 0.f ? __fdividef(neg, width) : INFINITY);
  }
  return far;
}

// The learned form's question after the first evaluation: does the particle lie at least far_cells
// past its cell?  (A next cell outside the grid ends the walk instead, as the reference's loop test.)
__device__ __forceinline__ bool walk_asks(Walk32 &w, int IM, int JM, int KM, float far_cells) {
  w.wait = (unsigned int)w.i < (unsigned int)IM && (unsigned int)w.j < (unsigned int)JM &&
           (unsigned int)w.k < (unsigned int)KM && far_cells <= beyond_cells(w.dv);
  return w.wait;
}

// The evaluation of a cell that the cell's margin leaves open (about 2e-5 of the evaluations of a
// step; one in a thousand of a walk from far away): w.dv from the faces' own margins and, where
// these decide nothing, the exact FP64 distances.  Returns whether a face is within its threshold.
template <bool EXACT>
__device__ __forceinline__ bool eval_hard32(const double *__restrict__ planes, size_t row, unsigned int cur, float2 px,
                                            float2 py, float2 pz, double xe, double ye, double ze, Walk32 &w,
                                            DevCounters *cnt) {
  const float4 h0 = row32_again(row, 0), h1 = row32_again(row, 1);
  if ((__float_as_uint(h1.w) >> 31) != 0u) {
    w.degenerate = true;
    return false;
  }
  const float prx = __fadd_rn(__fsub_rn(px.x, h0.x), __fsub_rn(px.y, h1.x));
  const float pry = __fadd_rn(__fsub_rn(py.x, h0.y), __fsub_rn(py.y, h1.y));
  const float prz = __fadd_rn(__fsub_rn(pz.x, h0.z), __fsub_rn(pz.y, h1.z));
  const float ax = __fmaf_rn(__fadd_rn(fabsf(px.x), fabsf(h0.x)), 0x1p-24f, fabsf(prx));
  const float ay = __fmaf_rn(__fadd_rn(fabsf(py.x), fabsf(h0.y)), 0x1p-24f, fabsf(pry));
  const float az = __fmaf_rn(__fadd_rn(fabsf(pz.x), fabsf(h0.z)), 0x1p-24f, fabsf(prz));
  unsigned int undecided = 0u;
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const float4 n = row32_again(row, 2u + f);
    const float S = __fmaf_rn(7.0f, __fmaf_rn(fabsf(n.z), az, __fmaf_rn(fabsf(n.y), ay, __fmul_rn(fabsf(n.x), ax))),
                              __fadd_rn(fabsf(n.w), fabsf(n.w)));
    if (!(fabsf(w.dv[f]) > __fmaf_rn(S, 4.0f * 0x1p-24f, h1.w))) undecided |= 1u << f;
  }
  bool zero = false;
#pragma unroll 1
  while (undecided) {   // a loop the compiler cannot if-convert: FP64 only for the faces left
    const int f = __ffs((int)undecided) - 1;
    undecided &= undecided - 1u;
    const double *row64 = planes + (size_t)cur * FDF_ROW;
    const double d64 = EXACT ? exact_face(row64, f, xe, ye, ze)
                             : exact_face(row64, f, pair_value(px), pair_value(py), pair_value(pz));
    zero = zero || fdfx::eq0(d64);
    float df = __double2float_rn(d64);
    if (fdfx::lt0(d64) && !(df < 0.f)) df = -1e-30f;   // a negative distance below the float range
    atomicAdd(&cnt->stripes[blockIdx.x & (FDF_CNT_STRIPES - 1)][CNT_FB], 1ull);
#pragma unroll
    for (int q = 0; q < 6; ++q)
      if (q == f) w.dv[q] = df;
  }
  return zero;
}

// The walk on from a cell that the cell's margin leaves open, to its end: w stands at that cell,
// entered, with its FP32 distances.
template <bool EXACT, bool FIRST>
__device__ __forceinline__ void walk_hard32(const float *__restrict__ table, const double *__restrict__ planes,
                                            const GridDims &g, float2 px, float2 py, float2 pz, int limit, double xe,
                                            double ye, double ze, Walk32 &w, DevCounters *cnt, Path32 *path,
                                            float far_cells) {
  unsigned int cur = ((unsigned int)w.k * g.JM + w.j) * g.IM + w.i;
#pragma unroll 1
  for (;;) {
    const size_t row = row32_address(table, cur);
    const bool zero = eval_hard32<EXACT>(planes, row, cur, px, py, pz, xe, ye, ze, w, cnt);
    if (w.degenerate) {
      w.lost = true;
      return;
    }
    if (!(walk_low(w) < 0.f) || zero) {
      w.concluded = true;
      return;
    }
    walk_advance(w);
    if (FIRST && w.steps == 1 && walk_asks(w, g.IM, g.JM, g.KM, far_cells)) return;
    if (w.steps >= limit || !walk_enter<FIRST>(w, g.IM, g.JM, g.KM, cur)) return;
    if (path) path->count(w.i, w.j, w.k, w.steps);
    float pr[3];
    const size_t next = row32_address(table, cur);
    row32_distances(next, row32_again(next, 0), row32_again(next, 1), px, py, pz, pr, w.dv);
  }
}

// The reference walk from (w.i, w.j, w.k) for at most `limit` evaluations.
// EXACT: the position is the FP64 (xe, ye, ze) and the pairs are its split (hi = fl32(x),
// lo = fl32(x - hi), within 2^-48 |x| of it, which the margins cover); the faces the
// FP32 bounds cannot decide are then computed from the FP64 position itself.
// FIRST: the learned form's first pass; a particle that asks (walk_asks) stops at its second cell.
// FAR: where walks may start far away (no previous cell), the cells that the cell's margin leaves
// open are evaluated in the loop: the margin grows with the distance, one particle in a thousand
// stays within it of a face along its whole walk, and after the loop it would double its warp's
// time (ten steps of 10,000 particles with a 280-cell walk before: 1.79 against 1.52 ms).  In a step, whose walks are short,
// those evaluations wait until the loop has ended, to the walk's end, which keeps their registers out
// of it (64M particles: 2.32 against 2.47 ms).
template <bool EXACT = false, bool TRACK = false, bool FIRST = false, bool FAR = false>
__device__ __forceinline__ void walk_ref32(const float *__restrict__ table, const double *__restrict__ planes,
                                           const GridDims &g, float2 px, float2 py, float2 pz, int limit, Walk32 &w,
                                           DevCounters *cnt, double xe = 0.0, double ye = 0.0, double ze = 0.0,
                                           Path32 *path = nullptr, float far_cells = 0.f) {
  const float X = walk_margin(px, py, pz);
  w.saved = 0xffffffffu;
  w.steps = 0;
  w.concluded = false; w.lost = false; w.cycle = false; w.degenerate = false; w.wait = false;
  bool hard = false;
  while (w.steps < limit) {
    unsigned int cur;
    if (!walk_enter<FIRST>(w, g.IM, g.JM, g.KM, cur)) break;
    if (TRACK) path->count(w.i, w.j, w.k, w.steps);
    const size_t row = row32_address(table, cur);
    const float4 h0 = row32_chunk(row, 0), h1 = row32_chunk(row, 1);
    float pr[3];
    row32_distances(row, h0, h1, px, py, pz, pr, w.dv);
    const float M = __fmaf_rn(__fadd_rn(__fadd_rn(fabsf(pr[0]), fabsf(pr[1])), fabsf(pr[2])), 40.0f * 0x1p-24f,
                              __fadd_rn(h0.w, X));
    const float(&d)[6] = w.dv;
    const float least = fminf(fminf(fminf(fabsf(d[0]), fabsf(d[1])), fminf(fabsf(d[2]), fabsf(d[3]))),
                              fminf(fabsf(d[4]), fabsf(d[5])));
    bool zero = false;
    // a NaN among the distances comes with M = inf or NaN (from the position or the row), so that
    // the minimum, which passes over NaN, cannot let it through
    if (!(least > M)) {
      if (!FAR) {
        hard = true;
        break;
      }
      zero = eval_hard32<EXACT>(planes, row, cur, px, py, pz, xe, ye, ze, w, cnt);
      if (w.degenerate) {
        w.lost = true;
        break;
      }
    }
    if (!(walk_low(w) < 0.f) || zero) {
      w.concluded = true;
      break;
    }
    walk_advance(w);
    if (FIRST && w.steps == 1 && walk_asks(w, g.IM, g.JM, g.KM, far_cells)) break;
  }
  if (!FAR && hard)
    walk_hard32<EXACT, FIRST>(table, planes, g, px, py, pz, limit, xe, ye, ze, w, cnt, TRACK ? path : nullptr,
                              far_cells);
}

}  // namespace
