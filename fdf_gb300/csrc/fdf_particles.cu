// fdf_particles.cu -- grid-to-particle interpolation fused with the sorted
// gather, the deterministic particle-to-grid deposits, and the DMSwarm AoS <->
// device SoA marshalling.
#include "fdf_internal.cuh"
#include "fdf_exact.cuh"
#include "fdf_corner.cuh"

#include <algorithm>

namespace {

using fdfx::add;
using fdfx::sub;
using fdfx::mul;

// ComputeTrilinearWeights (interpolation.c:839-864) and TrilinearInterpolation_Vector (:957-1042): the
// velocity from the eight corner values value(c, x, y, z), c in bit order (i, j, k).
template <bool INT, typename Value>
__device__ __forceinline__ void trilinear(double a1, double a2, double a3, Value value, double &ux, double &uy,
                                          double &uz) {
  a1 = fdfx::clamp01(a1);
  a2 = fdfx::clamp01(a2);
  a3 = fdfx::clamp01(a3);
  const double oa1 = sub(1.0, a1), oa2 = sub(1.0, a2), oa3 = sub(1.0, a3);
  // w[c] = (x*y)*z as the reference evaluates it; the four (x*y) pair products are shared
  // The 36 products run on the integer pipe (fdfx::mul_int, the same bits as the FP64
  // multiply) and the sums on the FP64 pipe, so both pipes work at once.  Moving products back to
  // the FP64 pipe (3 to 12 of them) is no faster: 4.64 to 5.28 against 4.66 ms for 64M particles.  (Few
  // particles: INT false, k_gather_interp.)
  auto wmul = [](double x, double y) { return INT ? fdfx::mul_int(x, y) : mul(x, y); };
  const double p00 = wmul(oa1, oa2), p10 = wmul(a1, oa2), p01 = wmul(oa1, a2), p11 = wmul(a1, a2);
  double w[8];
  w[0] = wmul(p00, oa3); w[1] = wmul(p10, oa3); w[2] = wmul(p01, oa3); w[3] = wmul(p11, oa3);
  w[4] = wmul(p00, a3);  w[5] = wmul(p10, a3);  w[6] = wmul(p01, a3);  w[7] = wmul(p11, a3);
  // accumulators start at 0.0: the first "0.0 + t" is t except that -0.0 becomes +0.0
  double ax, ay, az, sw;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    double vx, vy, vz;
    value(c, vx, vy, vz);
    const double tx = wmul(w[c], vx), ty = wmul(w[c], vy), tz = wmul(w[c], vz);
    ax = c ? add(ax, tx) : fdfx::add0(tx);
    ay = c ? add(ay, ty) : fdfx::add0(ty);
    az = c ? add(az, tz) : fdfx::add0(tz);
    sw = c ? add(sw, w[c]) : fdfx::add0(w[c]);
  }
  // sumW > 1e-14 (false for NaN); x / 1.0 == x exactly, so the common sumW == 1 skips the divides
  if (!fdfx::is_nan(sw) && !fdfx::le_pos(sw, fdfx::ubits(1.0e-14))) {
    if (fdfx::ubits(sw) == 0x3ff0000000000000ULL) {
      ux = ax; uy = ay; uz = az;
    } else {
      const fdfx::Divisor dsw = fdfx::make_divisor(sw);
      ux = fdfx::div_by(ax, dsw); uy = fdfx::div_by(ay, dsw); uz = fdfx::div_by(az, dsw);
    }
  }
}

// What the gather takes of a particle, as one 16-byte aligned 80-byte record: position, weights, P, pid, cell.
__global__ void __launch_bounds__(256) k_pack(SwarmBuf b, const DevCounters *cnt, ulonglong2 *__restrict__ rec) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= cnt->n_sorted) return;
  ulonglong2 *r = rec + 5 * (size_t)p;
  r[0] = make_ulonglong2(fdfx::ubits(b.x[p]), fdfx::ubits(b.y[p]));
  r[1] = make_ulonglong2(fdfx::ubits(b.z[p]), fdfx::ubits(b.a1[p]));
  r[2] = make_ulonglong2(fdfx::ubits(b.a2[p]), fdfx::ubits(b.a3[p]));
  r[3] = make_ulonglong2(fdfx::ubits(b.P[p]), (unsigned long long)b.pid[p]);
  r[4] = make_ulonglong2((unsigned long long)(long long)b.cell[p], 0ull);
}

// Sorted slot s takes the particle from slot perm[s] of the previous order, then
// interpolates ucat to it: ComputeTrilinearWeights (interpolation.c:839-864) and
// TrilinearInterpolation_Vector (:957-1042) from the node-averaged field, with
// the stencil guard of InterpolateEulerFieldToSwarm (:1356-1372).
// 2048 resident threads: the products' integer chains and the sums' FP64 chains wait on one another,
// so resident warps beat the spills of 32 registers (64M particles 4.66 ms; 4.94 at 1536 threads, 5.0 at
// 1280, 5.5 at the compiler's choice of 48 registers).
// REC: the particles come from k_pack's records (mode GATHER_INTERP).
// FEW: up to GATHER_FEW particles, about two and a half warps per scheduler, each warp's own chain is the time,
// and the FP64 pipe's products and 128 registers make it shorter: 10k particles 11.0 -> 6.2 us, 30k 14.0 -> 12.2;
// 100k 20.9 against 23, 1M 93 against 125, so not above.
constexpr int GATHER_FEW = 3 << 14;
template <bool REC, bool FEW>
__global__ void __launch_bounds__(FEW ? 64 : 256, 8) k_gather_interp(SwarmBuf src, SwarmBuf dst, GridDims g,
                                                       const double *__restrict__ corner,
                                                       const unsigned int *__restrict__ perm,
                                                       const unsigned int *__restrict__ cell_start,
                                                       DevCounters *cnt, int mode, const ulonglong2 *__restrict__ rec) {
  const int n = (int)cell_start[g.Nc + 1];
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s == 0) {   // the new sizes, read by the next step
    cnt->n = (int)cell_start[g.Nc];
    cnt->n_sorted = n;
  }
  if (s >= n) return;
  const unsigned int p = perm ? perm[s] : (unsigned int)s;
  int cell;
  double a1, a2, a3;
  unsigned char st = 0;
  if (REC) {
    const ulonglong2 *r = rec + 5 * (size_t)p;
    const ulonglong2 xy = r[0], za = r[1], ab = r[2], Pp = r[3];
    cell = (int)r[4].x;
    a1 = __longlong_as_double((long long)za.y); a2 = __longlong_as_double((long long)ab.x); a3 = __longlong_as_double((long long)ab.y);
    dst.x[s] = __longlong_as_double((long long)xy.x); dst.y[s] = __longlong_as_double((long long)xy.y); dst.z[s] = __longlong_as_double((long long)za.x);
    dst.P[s] = __longlong_as_double((long long)Pp.x);
    dst.pid[s] = (long long)Pp.y;
  } else {
    cell = src.cell[p];
    a1 = src.a1[p]; a2 = src.a2[p]; a3 = src.a3[p];
    st = src.status[p];
    dst.x[s] = src.x[p]; dst.y[s] = src.y[p]; dst.z[s] = src.z[p];
    dst.P[s] = src.P[p];
    dst.pid[s] = src.pid[p];
  }
  dst.a1[s] = a1; dst.a2[s] = a2; dst.a3[s] = a3;
  if (!REC && mode == GATHER_COPY) {
    dst.u[s] = src.u[p]; dst.v[s] = src.v[p]; dst.w[s] = src.w[p];
    dst.cell[s] = cell;
    dst.status[s] = st;
    return;
  }
  double ux = 0.0, uy = 0.0, uz = 0.0;
  if (cell < 0) {
    dst.cell[s] = -1;
    dst.status[s] = REC || mode == GATHER_INTERP ? (unsigned char)ST_LOST : st;
  } else {
    dst.cell[s] = cell;
    dst.status[s] = REC || mode == GATHER_INTERP ? (unsigned char)ST_ACTIVE_AND_LOCATED : st;
    int i, j, k;
    cell_ijk(g, (unsigned int)cell, i, j, k);
    const long long mx = g.IM + 1, my = g.JM + 1;
    const double *at = corner + (((long long)k * my + j) * mx + i);
    trilinear<!FEW>(a1, a2, a3, [&](int c, double &vx, double &vy, double &vz) {
      const long long off = (c & 1) + ((c & 2) ? mx : 0) + ((c & 4) ? mx * my : 0);
      vx = __ldg(at + off); vy = __ldg(at + g.Nn + off); vz = __ldg(at + 2 * g.Nn + off);
    }, ux, uy, uz);
  }
  dst.u[s] = ux; dst.v[s] = uy; dst.w[s] = uz;
}

// InterpolateEulerFieldToSwarm for particles the caller holds (fdf_InterpolatePoints), in the callers'
// layout.  DIRECT: each point averages its eight corners from ucat itself, node by node as the corner
// field's kernel does, instead of reading the whole corner field made for it.
template <bool DIRECT>
__global__ void __launch_bounds__(128) k_interp_points(const long long *__restrict__ cell,
                                                      const double *__restrict__ weight, int n, GridDims g,
                                                      const double *__restrict__ field, double *__restrict__ vel) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const long long i = cell[3 * (size_t)p], j = cell[3 * (size_t)p + 1], k = cell[3 * (size_t)p + 2];
  double ux = 0.0, uy = 0.0, uz = 0.0;
  if (i >= 0 && i < g.IM && j >= 0 && j < g.JM && k >= 0 && k < g.KM) {
    const long long mx = g.IM + 1, my = g.JM + 1;
    trilinear<true>(weight[3 * (size_t)p], weight[3 * (size_t)p + 1], weight[3 * (size_t)p + 2],
              [&](int c, double &vx, double &vy, double &vz) {
                const int ni = (int)i + (c & 1), nj = (int)j + ((c >> 1) & 1), nk = (int)k + (c >> 2);
                if (DIRECT) {
                  fdfx::corner_value<0>(field, g, ni, nj, nk, vx, vy, vz);
                } else {
                  const double *at = field + (((long long)nk * my + nj) * mx + ni);
                  vx = __ldg(at); vy = __ldg(at + g.Nn); vz = __ldg(at + 2 * g.Nn);
                }
              },
              ux, uy, uz);
  }
  vel[3 * (size_t)p] = ux; vel[3 * (size_t)p + 1] = uy; vel[3 * (size_t)p + 2] = uz;
}

// One thread per grid node (i<=IM, j<=JM, k<=KM).  The node-sized outputs are the
// reference's ParticleCount and P average (interpolation.c:2063-2116): cell (i,j,k)
// sits at node slot (i,j,k).  The thread also owns the three faces whose lower
// corner is this node: i-face (i,j,k) between cells i-1 and i, and likewise j, k.
// A face sums its lower cell's particles (weight a) and then its upper cell's
// (weight 1-a), each in sorted order: a fixed order, so the sum is deterministic.
// The momentum variant adds the same split of V * velocity (SoA [3][faces]), each component
// summed in the same order.
//
// Bound by FP64 adds: a warp-wide FP64 instruction holds its unit for 64 cycles with one active lane
// as with 32, and the chains of a warp's 32 nodes (a face's lower cell, then its upper cell) differ
// in length.  So the chains contain the reference's adds and nothing else:
//   * the products (a * V/3 below the face, (1 - a) * V/3 above it, and their products with the
//     velocity) are made beforehand on the integer pipe (mul_int), lanes striding over the warp's
//     particles, into shared memory.  The lower-cell and own cells of consecutive nodes are
//     consecutive cells, so a face's entries are two contiguous particle ranges per warp;
//   * a face's two segments are one chain: a warp runs as long as its longest chain, and the longest
//     sum of two lengths is shorter than the sum of the two longest;
//   * a chain's first add, to 0.0, is a sign test (add0): most chains of a sparse grid need no more.
// A warp whose ranges exceed CAP entries makes the products in its chains.  Every sum takes the
// same values in the same order either way.
// Per step, with products on the FP64 pipe and lower and upper loops apart -> now: 64M particles in 14M
// cells 4.16 -> 2.20 ms, 16M 1.59 -> 0.82, 1M in 4M cells 0.25 -> 0.12, 32M in 1.2M cells 1.64 -> 1.09; with the
// momentum, 16M in 4.2M cells, 4.08 -> 1.79 ms.
// Entries of a warp's two ranges kept in shared memory: 4.5 particles per cell and a bit (64 cells);
// more would take the L1 cache and the resident blocks from the others.
constexpr int DEP_WARPS = 8, DEP_CAP = 320;

// STAGED: the products made beforehand in shared memory (volume only: with the momentum's four values
// per entry that costs more resident warps than it saves, 2.1 to 3.0 ms against 1.8 per 16M-particle
// step at 3.8 per cell).  Resident blocks: the chains wait on one another's adds, so 2048 threads
// (32 registers, a few spilled) beat 1024 for the volume (64M particles 2.20 against 2.58 ms);
// the momentum's take 64 registers.
template <bool MOM, bool STAGED>
__global__ void __launch_bounds__(DEP_WARPS * 32, MOM ? 4 : 8) k_deposit(SwarmBuf b, GridDims g,
                                                                           const unsigned int *__restrict__ cs,
                                                                           double third, double *__restrict__ count,
                                                                           double *__restrict__ avg,
                                                                           double *__restrict__ fi,
                                                                           double *__restrict__ fj,
                                                                           double *__restrict__ fk,
                                                                           double *__restrict__ mi,
                                                                           double *__restrict__ mj,
                                                                           double *__restrict__ mk) {
  constexpr int V = MOM ? 4 : 1;
  __shared__ double stage[DEP_WARPS][STAGED ? DEP_CAP : 1];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long q = (blockIdx.x * (long long)DEP_WARPS + wid) * 32 + lane;
  if (q - lane >= g.Nn) return;   // the whole warp is past the last node
  const bool node = q < g.Nn;
  const int IM = g.IM, JM = g.JM, KM = g.KM;
  int i = 0, j = 0, k = 0;
  if (node) node_ijk(g, (unsigned int)q, i, j, k);
  const long long c = ((long long)k * JM + j) * IM + i;
  const bool is_cell = node && i < IM && j < JM && k < KM;
  // a role's cell and particles [s0, s1), and the warp's particles [r0, r0 + n) of that role
  struct Role {
    unsigned int s0, s1, r0, n;
  };
  auto role = [&](bool has, long long cell) {
    const unsigned int NONE = 0xffffffffu;
    const unsigned int rc = has ? (unsigned int)cell : NONE;
    const unsigned int lo = __reduce_min_sync(0xffffffffu, rc), hi = __reduce_max_sync(0xffffffffu, has ? rc : 0u);
    Role r{0u, 0u, 0u, 0u};
    if (lo != NONE) {
      r.r0 = __ldg(cs + lo);
      r.n = __ldg(cs + hi + 1) - r.r0;
    }
    r.s0 = has ? __ldg(cs + rc) : r.r0;
    r.s1 = has ? __ldg(cs + rc + 1) : r.r0;
    return r;
  };
  const Role own = role(is_cell, c);
  // AccumulateParticleField + CalculateParticleCountPerCell + NormalizeGridVectorByCount
  double sum = 0.0;
  if (STAGED && own.n <= (unsigned int)DEP_CAP) {
    for (unsigned int e = lane; e < own.n; e += 32) stage[wid][e] = __ldg(b.P + own.r0 + e);
    __syncwarp();
    if (own.s1 > own.s0) sum = fdfx::add0(stage[wid][own.s0 - own.r0]);
    for (unsigned int s = own.s0 + 1; s < own.s1; ++s) sum = add(sum, stage[wid][s - own.r0]);
    __syncwarp();
  } else if (own.s1 > own.s0) {
    sum = fdfx::add0(__ldg(b.P + own.s0));
    double next = own.s0 + 1 < own.s1 ? __ldg(b.P + own.s0 + 1) : 0.0;
    for (unsigned int s = own.s0 + 1; s < own.s1; ++s) {
      const double P = next;
      if (s + 1 < own.s1) next = __ldg(b.P + s + 1);
      sum = add(sum, P);
    }
  }
  if (node) {
    const unsigned int ncell = own.s1 - own.s0;   // count += 1.0 per particle is exact in FP64
    count[q] = fdfx::u32_to_double(ncell);
    avg[q] = ncell > 0 ? fdfx::div_count(sum, ncell) : 0.0;
  }
  // one face: its lower cell's particles (none on the first face of a direction), then its upper's
  auto face = [&](bool has, bool below, long long lower_cell, const double *__restrict__ wgt,
                  double *__restrict__ vol, double *__restrict__ mom, long long nf, long long fidx) {
    const Role low = role(has && below, lower_cell);
    const unsigned int nl = low.s1 - low.s0, T = has ? nl + (own.s1 - own.s0) : 0u;
    double acc[V];
#pragma unroll
    for (int m = 0; m < V; ++m) acc[m] = 0.0;
    if (STAGED && low.n + own.n <= (unsigned int)DEP_CAP) {
      const bool few = low.n + own.n <= 32u;   // one pass: the FP64 pipe's subtraction is done sooner
      for (unsigned int e = lane; e < low.n + own.n; e += 32) {
        const bool upper = e >= low.n;
        double a = __ldg(wgt + (upper ? own.r0 + (e - low.n) : low.r0 + e));
        if (upper) a = few ? sub(1.0, a) : fdfx::one_minus(a);
        stage[wid][e] = fdfx::mul_int(a, third);
      }
      __syncwarp();
      const unsigned int at_low = low.s0 - low.r0, at_own = low.n + (own.s0 - own.r0) - nl;
      if (T > 0u) acc[0] = fdfx::add0(stage[wid][nl > 0u ? at_low : at_own]);
      for (unsigned int t = 1; t < T; ++t) acc[0] = add(acc[0], stage[wid][t + (t < nl ? at_low : at_own)]);
      __syncwarp();
    } else if (T > 0u) {
      // the chain's particles, the next one's values loading while this one's are added
      double a, u[3];
      auto load = [&](unsigned int t) {
        const unsigned int s = t < nl ? low.s0 + t : own.s0 + (t - nl);
        a = __ldg(wgt + s);
        if (MOM) { u[0] = __ldg(b.u + s); u[1] = __ldg(b.v + s); u[2] = __ldg(b.w + s); }
      };
      load(0u);
      for (unsigned int t = 0; t < T; ++t) {
        double x[V];
        const double wa = a, wu[3] = {u[0], u[1], u[2]};
        if (t + 1 < T) load(t + 1);
        x[0] = fdfx::mul_int(t < nl ? wa : fdfx::one_minus(wa), third);
#pragma unroll
        for (int m = 1; m < V; ++m) x[m] = fdfx::mul_int(x[0], wu[m - 1]);
#pragma unroll
        for (int m = 0; m < V; ++m) acc[m] = t == 0u ? fdfx::add0(x[m]) : add(acc[m], x[m]);
      }
    }
    if (has) {
      vol[fidx] = acc[0];
      if (MOM) { mom[fidx] = acc[V - 3]; mom[nf + fidx] = acc[V - 2]; mom[2 * nf + fidx] = acc[V - 1]; }
    }
  };
  const long long nfi = (IM + 1LL) * JM * KM, nfj = IM * (JM + 1LL) * KM, nfk = (long long)IM * JM * (KM + 1LL);
  // i-face (i,j,k), i in [0, IM]; j-face, j in [0, JM]; k-face, k in [0, KM]
  face(node && j < JM && k < KM, i > 0, c - 1, b.a1, fi, mi, nfi, ((long long)k * JM + j) * (IM + 1) + i);
  face(node && i < IM && k < KM, j > 0, c - IM, b.a2, fj, mj, nfj, ((long long)k * (JM + 1) + j) * IM + i);
  face(node && i < IM && j < JM, k > 0, c - (long long)IM * JM, b.a3, fk, mk, nfk, c);
}

// The same sums with a node's four chains -- the cell's P and its three faces -- in four blocks (blockIdx.y),
// for grids whose nodes do not fill the chip: one thread then waits for one chain instead of four in a
// row, with four particles' loads and products under way before their adds.  Products on the integer
// pipe for the volume, on the FP64 pipe for the momentum, whose 24 a particle would lengthen the chain.
// 18k nodes (20 x 20 x 40 cells), 60 particles per cell: 73 us against 166 in one chain after another, with the
// momentum 213 against 325; 71k nodes, 30 per cell 105 against 123; 274k nodes, 18 per cell 195 against 227.
template <bool MOM>
__global__ void __launch_bounds__(DEP_WARPS * 32, MOM ? 4 : 8) k_deposit_apart(SwarmBuf b, GridDims g,
                                                                              const unsigned int *__restrict__ cs,
                                                                              double third, double *__restrict__ count,
                                                                              double *__restrict__ avg,
                                                                              double *__restrict__ fi,
                                                                              double *__restrict__ fj,
                                                                              double *__restrict__ fk,
                                                                              double *__restrict__ mi,
                                                                              double *__restrict__ mj,
                                                                              double *__restrict__ mk) {
  constexpr int V = MOM ? 4 : 1, CH = 4;
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= g.Nn) return;
  const int IM = g.IM, JM = g.JM, KM = g.KM, f = blockIdx.y;   // f: the face's direction, 3 the cell
  int i, j, k;
  node_ijk(g, (unsigned int)q, i, j, k);
  const long long c = ((long long)k * JM + j) * IM + i;
  unsigned int s0 = 0u, s1 = 0u;
  if (i < IM && j < JM && k < KM) { s0 = __ldg(cs + c); s1 = __ldg(cs + c + 1); }
  if (f == 3) {
    double sum = 0.0;
    for (unsigned int s = s0; s < s1; s += CH) {
      double P[CH];
#pragma unroll
      for (int e = 0; e < CH; ++e) P[e] = s + e < s1 ? __ldg(b.P + s + e) : 0.0;
#pragma unroll
      for (int e = 0; e < CH; ++e)
        if (s + e < s1) sum = add(sum, P[e]);
    }
    const unsigned int ncell = s1 - s0;
    count[q] = fdfx::u32_to_double(ncell);
    avg[q] = ncell > 0 ? fdfx::div_count(sum, ncell) : 0.0;
    return;
  }
  if ((f != 0 && i >= IM) || (f != 1 && j >= JM) || (f != 2 && k >= KM)) return;   // no such face
  const long long lower = c - (f == 0 ? 1LL : f == 1 ? (long long)IM : (long long)IM * JM);
  unsigned int l0 = 0u, l1 = 0u;
  if ((f == 0 ? i : f == 1 ? j : k) > 0) { l0 = __ldg(cs + lower); l1 = __ldg(cs + lower + 1); }
  const double *__restrict__ wgt = f == 0 ? b.a1 : f == 1 ? b.a2 : b.a3;
  const unsigned int nl = l1 - l0, T = nl + (s1 - s0);
  auto product = [](double x, double y) { return MOM ? mul(x, y) : fdfx::mul_int(x, y); };
  double acc[V];
#pragma unroll
  for (int m = 0; m < V; ++m) acc[m] = 0.0;
  for (unsigned int t = 0; t < T; t += CH) {
    double x[CH][V];
#pragma unroll
    for (int e = 0; e < CH; ++e) {
      const unsigned int s = t + e < nl ? l0 + (t + e) : s0 + (t + e - nl);
      const bool in = t + e < T;
      const double a = in ? __ldg(wgt + s) : 0.0;
      x[e][0] = product(t + e < nl ? a : sub(1.0, a), third);
      if (MOM) {
        x[e][V - 3] = product(x[e][0], in ? __ldg(b.u + s) : 0.0);
        x[e][V - 2] = product(x[e][0], in ? __ldg(b.v + s) : 0.0);
        x[e][V - 1] = product(x[e][0], in ? __ldg(b.w + s) : 0.0);
      }
    }
#pragma unroll
    for (int e = 0; e < CH; ++e)
      if (t + e < T) {
#pragma unroll
        for (int m = 0; m < V; ++m) acc[m] = add(acc[m], x[e][m]);
      }
  }
  const long long at = f == 0 ? ((long long)k * JM + j) * (IM + 1) + i : f == 1 ? ((long long)k * (JM + 1) + j) * IM + i : c;
  (f == 0 ? fi : f == 1 ? fj : fk)[at] = acc[0];
  if (MOM) {
    const long long nf = f == 0 ? (IM + 1LL) * JM * KM : f == 1 ? IM * (JM + 1LL) * KM : (long long)IM * JM * (KM + 1LL);
    double *mom = f == 0 ? mi : f == 1 ? mj : mk;
    mom[at] = acc[V - 3]; mom[nf + at] = acc[V - 2]; mom[2 * nf + at] = acc[V - 1];
  }
}

// Slot t of dst takes slot a + t of src for t < b - a, and slot c + (t - (b - a)) after that: the
// held particles of a k-slab ([a, b) in the cell-sorted order) followed by those without a cell
// ([c, n)); every field of both forms moves.
__global__ void k_move_kept(SwarmBuf src, SwarmBuf dst, int a, int b, int c, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = (b - a) + (n - c);
  if (t >= m) return;
  const int p = t < b - a ? a + t : c + (t - (b - a));
  dst.x[t] = src.x[p]; dst.y[t] = src.y[p]; dst.z[t] = src.z[p];
  dst.u[t] = src.u[p]; dst.v[t] = src.v[p]; dst.w[t] = src.w[p];
  dst.a1[t] = src.a1[p]; dst.a2[t] = src.a2[p]; dst.a3[t] = src.a3[p];
  dst.P[t] = src.P[p];
  dst.uf[t] = src.uf[p]; dst.vf[t] = src.vf[p]; dst.wf[t] = src.wf[p];
  dst.a1f[t] = src.a1f[p]; dst.a2f[t] = src.a2f[p]; dst.a3f[t] = src.a3f[p];
  dst.Pf[t] = src.Pf[p];
  dst.pid[t] = src.pid[p];
  dst.cell[t] = src.cell[p];
  dst.status[t] = src.status[p];
}

// The k-faces of layer k (between cells k - 1 and k) summed again from seed values: seed[j][i]
// stands for the lower cell's part of the sum (0.0 + its particles' a V/3 in (cell, PID) order,
// made where the lower cell's particles are held), and the held particles of cell (i, j, k) add
// their (1 - a) V/3 (and its products with the velocity) after it, in sorted order -- the
// single-rank sum, operation for operation.  Momentum seeds are [j][i][3].
__global__ void k_deposit_k_layer(SwarmBuf b, GridDims g, const unsigned int *__restrict__ cs, int k, double third,
                                  const double *__restrict__ seed, const double *__restrict__ seed_mom,
                                  double *__restrict__ fk, double *__restrict__ mk) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;   // (j, i) of the layer
  const long long L = (long long)g.IM * g.JM;
  if (q >= L) return;
  const long long f = (long long)k * L + q;
  double acc = seed[q];
  double m0 = 0.0, m1 = 0.0, m2 = 0.0;
  if (mk) { m0 = seed_mom[3 * q]; m1 = seed_mom[3 * q + 1]; m2 = seed_mom[3 * q + 2]; }
  if (k < g.KM) {
    const unsigned int s0 = __ldg(cs + f), s1 = __ldg(cs + f + 1);
    for (unsigned int s = s0; s < s1; ++s) {
      const double x = mul(sub(1.0, __ldg(b.a3 + s)), third);
      acc = add(acc, x);
      if (mk) {
        m0 = add(m0, mul(x, __ldg(b.u + s)));
        m1 = add(m1, mul(x, __ldg(b.v + s)));
        m2 = add(m2, mul(x, __ldg(b.w + s)));
      }
    }
  }
  fk[f] = acc;
  if (mk) {
    const long long nfk = L * (g.KM + 1LL);
    mk[f] = m0; mk[nfk + f] = m1; mk[2 * nfk + f] = m2;
  }
}

__global__ void k_from_aos(const double *__restrict__ pos, const double *__restrict__ vel,
                           const double *__restrict__ wgt, const double *__restrict__ P,
                           const long long *__restrict__ cell3, const long long *__restrict__ pid,
                           const long long *__restrict__ status, int n, GridDims g, SwarmBuf b) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  b.x[p] = pos[3 * p]; b.y[p] = pos[3 * p + 1]; b.z[p] = pos[3 * p + 2];
  b.u[p] = vel[3 * p]; b.v[p] = vel[3 * p + 1]; b.w[p] = vel[3 * p + 2];
  b.a1[p] = wgt[3 * p]; b.a2[p] = wgt[3 * p + 1]; b.a3[p] = wgt[3 * p + 2];
  b.P[p] = P[p];
  b.pid[p] = pid[p];
  long long i = cell3[3 * p], j = cell3[3 * p + 1], k = cell3[3 * p + 2];
  int c = -1;
  if (i >= 0 && i < g.IM && j >= 0 && j < g.JM && k >= 0 && k < g.KM) c = (int)((k * g.JM + j) * g.IM + i);
  b.cell[p] = c;
  long long st = status[p];
  b.status[p] = (unsigned char)((st >= 0 && st <= ST_UNINITIALIZED) ? st : ST_UNINITIALIZED);
}

__global__ void k_to_aos(SwarmBuf b, int n, GridDims g, double *__restrict__ pos, double *__restrict__ vel,
                         double *__restrict__ wgt, double *__restrict__ P, long long *__restrict__ cell3,
                         long long *__restrict__ pid, long long *__restrict__ status) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  pos[3 * p] = b.x[p]; pos[3 * p + 1] = b.y[p]; pos[3 * p + 2] = b.z[p];
  vel[3 * p] = b.u[p]; vel[3 * p + 1] = b.v[p]; vel[3 * p + 2] = b.w[p];
  wgt[3 * p] = b.a1[p]; wgt[3 * p + 1] = b.a2[p]; wgt[3 * p + 2] = b.a3[p];
  P[p] = b.P[p];
  pid[p] = b.pid[p];
  int c = b.cell[p];
  if (c >= 0) {
    int i, j, k;
    cell_ijk(g, (unsigned int)c, i, j, k);
    cell3[3 * p] = i; cell3[3 * p + 1] = j; cell3[3 * p + 2] = k;
  } else {
    cell3[3 * p] = -1; cell3[3 * p + 1] = -1; cell3[3 * p + 2] = -1;
  }
  status[p] = b.status[p];
}

// ResetAllParticleStatuses (ParticleMotion.c:2149-2176): ACTIVE_AND_LOCATED -> NEEDS_LOCATION.
__global__ void k_reset_status(unsigned char *__restrict__ status, const DevCounters *cnt) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < cnt->n_sorted && status[s] == ST_ACTIVE_AND_LOCATED) status[s] = ST_NEEDS_LOCATION;
}

// UpdateAllParticlePositions (ParticleMotion.c:38-95): x += v dt per component, as the fused
// step does it.
__global__ void k_advect(SwarmBuf b, double dt, DevCounters *cnt) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s == 0) atomicAdd(&cnt->psteps_total, (unsigned long long)cnt->n_sorted);   // particles advanced
  if (s >= cnt->n_sorted) return;
  b.x[s] = add(b.x[s], mul(b.u[s], dt));
  b.y[s] = add(b.y[s], mul(b.v[s], dt));
  b.z[s] = add(b.z[s], mul(b.w[s], dt));
}

}  // namespace

void launch_reset_status(const SwarmBuf &b, int n_cap, const DevCounters *cnt, cudaStream_t s) {
  k_reset_status<<<(n_cap + 255) / 256 > 0 ? (n_cap + 255) / 256 : 1, 256, 0, s>>>(b.status, cnt);
}

void launch_advect(const SwarmBuf &b, int n_cap, double dt, DevCounters *cnt, cudaStream_t s) {
  k_advect<<<(n_cap + 255) / 256 > 0 ? (n_cap + 255) / 256 : 1, 256, 0, s>>>(b, dt, cnt);
}

void launch_gather_interp(const SwarmBuf &src, const SwarmBuf &dst, int n_cap, GridDims g, const double *corner,
                          const unsigned int *perm, const unsigned int *cell_start, DevCounters *cnt,
                          cudaStream_t s, int mode) {
  int th = 256;
  int blocks = (n_cap + th - 1) / th;
  if (blocks == 0) blocks = 1;
  if (n_cap <= GATHER_FEW)
    k_gather_interp<false, true><<<std::max((n_cap + 63) / 64, 1), 64, 0, s>>>(src, dst, g, corner, perm, cell_start, cnt,
                                                                              mode, nullptr);
  else
    k_gather_interp<false, false><<<blocks, th, 0, s>>>(src, dst, g, corner, perm, cell_start, cnt, mode, nullptr);
}

void launch_gather_interp_packed(const SwarmBuf &src, const SwarmBuf &dst, int n_cap, GridDims g, const double *corner,
                                 const unsigned int *perm, const unsigned int *cell_start, DevCounters *cnt, void *rec,
                                 cudaStream_t s) {
  const unsigned int blocks = n_cap > 0 ? (unsigned int)((n_cap + 255) / 256) : 1u;
  ulonglong2 *r = static_cast<ulonglong2 *>(rec);
  k_pack<<<blocks, 256, 0, s>>>(src, cnt, r);
  k_gather_interp<true, false><<<blocks, 256, 0, s>>>(src, dst, g, corner, perm, cell_start, cnt, GATHER_INTERP, r);
}

void launch_deposit(const SwarmBuf &b, int n_cap, GridDims g, const unsigned int *cell_start, double volume, double *count,
                    double *avg, double *fi, double *fj, double *fk, double *mi, double *mj, double *mk,
                    cudaStream_t s) {
  const double third = volume / 3.0;
  constexpr int th = DEP_WARPS * 32;
  const unsigned int blocks = (unsigned int)((g.Nn + th - 1) / th);
  // Above five particles per cell most warps' ranges exceed DEP_CAP, and the staging's shared memory
  // only takes from the L1 cache (27 per cell, 32M particles: 1.25 ms staged, 1.09 without; 4.5 per
  // cell, 64M: 2.20 staged, 2.85 without).  The capacity stands for the count, which only the device knows.
  const bool dense = n_cap > 5 * g.Nc;
  // The chains apart: with 18k nodes faster at every density (one and 4.9 per cell: 16.4 and 22.0 us against
  // 20.8 and 35.3 staged, momentum 22.6 and 38.1 against 30.7 and 57.6), with 71k nodes staged (23.1 and 29.7
  // at one and three per cell against 22.3 and 30.1) or with the momentum (36.2 and 97 at one and eight against
  // 38.1 and 119) no longer.  Without the staging up to half a million nodes: 274k nodes 111 against 127 us at
  // eight per cell, 195 against 229 at 18; 545k nodes 207 against 207, 365 against 376; 1.2M 437 against 417.
  const bool apart = g.Nn <= (1 << 15) || (!mi && dense && g.Nn <= (1 << 19));
  const dim3 four(blocks, 4);
  if (apart && mi) k_deposit_apart<true><<<four, th, 0, s>>>(b, g, cell_start, third, count, avg, fi, fj, fk, mi, mj, mk);
  else if (apart) k_deposit_apart<false><<<four, th, 0, s>>>(b, g, cell_start, third, count, avg, fi, fj, fk, mi, mj, mk);
  else if (mi) k_deposit<true, false><<<blocks, th, 0, s>>>(b, g, cell_start, third, count, avg, fi, fj, fk, mi, mj, mk);
  else if (!dense)
    k_deposit<false, true><<<blocks, th, 0, s>>>(b, g, cell_start, third, count, avg, fi, fj, fk, mi, mj, mk);
  else k_deposit<false, false><<<blocks, th, 0, s>>>(b, g, cell_start, third, count, avg, fi, fj, fk, mi, mj, mk);
}

void launch_interp_points(const long long *cell, const double *weight, int n, GridDims g, const double *field, bool direct,
                          double *vel, cudaStream_t s) {
  const unsigned int blocks = (unsigned int)((n + 127) / 128);
  if (direct) k_interp_points<true><<<blocks, 128, 0, s>>>(cell, weight, n, g, field, vel);
  else k_interp_points<false><<<blocks, 128, 0, s>>>(cell, weight, n, g, field, vel);
}

void launch_move_kept(const SwarmBuf &src, const SwarmBuf &dst, int a, int b, int c, int n, cudaStream_t s) {
  const int m = (b - a) + (n - c);
  if (m <= 0) return;
  k_move_kept<<<(m + 255) / 256, 256, 0, s>>>(src, dst, a, b, c, n);
}

void launch_deposit_k_layer(const SwarmBuf &b, GridDims g, const unsigned int *cell_start, int k, double volume,
                            const double *seed, const double *seed_mom, double *fk, double *mk, cudaStream_t s) {
  const long long L = (long long)g.IM * g.JM;
  k_deposit_k_layer<<<(unsigned)((L + 255) / 256), 256, 0, s>>>(b, g, cell_start, k, volume / 3.0, seed, seed_mom, fk,
                                                                 mk);
}

void launch_swarm_from_aos(const double *pos, const double *vel, const double *wgt, const double *P,
                           const long long *cell3, const long long *pid, const long long *status, int n, GridDims g,
                           const SwarmBuf &b, cudaStream_t s) {
  if (n <= 0) return;
  k_from_aos<<<(n + 255) / 256, 256, 0, s>>>(pos, vel, wgt, P, cell3, pid, status, n, g, b);
}

void launch_swarm_to_aos(const SwarmBuf &b, int n, GridDims g, double *pos, double *vel, double *wgt, double *P,
                         long long *cell3, long long *pid, long long *status, cudaStream_t s) {
  if (n <= 0) return;
  k_to_aos<<<(n + 255) / 256, 256, 0, s>>>(b, n, g, pos, vel, wgt, P, cell3, pid, status);
}
