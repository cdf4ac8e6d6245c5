// fdf_grid.cu -- grid-side kernels: per-cell face-plane table and center->corner
// averaging of ucat.
//
// All FP64 arithmetic on the parity path uses the _rn intrinsics, which the
// compiler never contracts into an FMA, so every value is rounded exactly as the
// reference (compiled without FMA) rounds it.
#include "fdf_internal.cuh"
#include "fdf_exact.cuh"
#include "fdf_corner.cuh"
#include "fdf_counters.cuh"
#include <cfloat>

namespace {

struct V3 { double x, y, z; };

using fdfx::add;
using fdfx::sub;
using fdfx::mul;

__device__ __forceinline__ V3 node(const double *coor, GridDims g, long long i, long long j, long long k) {
  const double *q = coor + 3 * ((k * (g.JM + 1) + j) * (long long)(g.IM + 1) + i);
  return V3{q[0], q[1], q[2]};
}

// One face of ComputeSignedDistanceToPlane (walkingsearch.c:102-227) with every
// particle-independent quantity evaluated: face centroid and oriented unit normal.
__device__ __forceinline__ bool face_plane(V3 v1, V3 v2, V3 v3, V3 v4, V3 cc, double *row) {
  double e1x = sub(v2.x, v1.x), e1y = sub(v2.y, v1.y), e1z = sub(v2.z, v1.z);
  double e2x = sub(v4.x, v1.x), e2y = sub(v4.y, v1.y), e2z = sub(v4.z, v1.z);
  double nxi = sub(mul(e1y, e2z), mul(e1z, e2y));
  double nyi = sub(mul(e1z, e2x), mul(e1x, e2z));
  double nzi = sub(mul(e1x, e2y), mul(e1y, e2x));
  double mag = __dsqrt_rn(add(add(mul(nxi, nxi), mul(nyi, nyi)), mul(nzi, nzi)));
  bool degenerate = mag < 1.0e-12;
  double fcx = mul(0.25, add(add(add(v1.x, v2.x), v3.x), v4.x));
  double fcy = mul(0.25, add(add(add(v1.y, v2.y), v3.y), v4.y));
  double fcz = mul(0.25, add(add(add(v1.z, v2.z), v3.z), v4.z));
  double tx = sub(cc.x, fcx), ty = sub(cc.y, fcy), tz = sub(cc.z, fcz);
  double dot = add(add(mul(nxi, tx), mul(nyi, ty)), mul(nzi, tz));
  double nx = nxi, ny = nyi, nz = nzi;
  if (dot > 1.0e-9) { nx = -nxi; ny = -nyi; nz = -nzi; }
  row[0] = fcx; row[1] = fcy; row[2] = fcz;
  row[3] = __ddiv_rn(nx, mag); row[4] = __ddiv_rn(ny, mag); row[5] = __ddiv_rn(nz, mag);
  return degenerate;
}

__global__ void k_build_planes(const double *__restrict__ coor, GridDims g, double *__restrict__ planes,
                               unsigned int *any_degenerate) {
  long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= g.Nc) return;
  int i, j, k;
  cell_ijk(g, (unsigned int)c, i, j, k);
  // walkingsearch.c:521-549 vertex numbering
  V3 v[8];
  v[0] = node(coor, g, i, j, k);         v[1] = node(coor, g, i + 1, j, k);
  v[2] = node(coor, g, i + 1, j + 1, k); v[3] = node(coor, g, i, j + 1, k);
  v[4] = node(coor, g, i, j + 1, k + 1); v[5] = node(coor, g, i + 1, j + 1, k + 1);
  v[6] = node(coor, g, i + 1, j, k + 1); v[7] = node(coor, g, i, j, k + 1);
  // GetCellCharacteristicSize, walkingsearch.c:25-59
  const int e[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                        {6, 7}, {7, 4}, {0, 7}, {1, 6}, {2, 5}, {3, 4}};
  double total = 0.0;
#pragma unroll
  for (int q = 0; q < 12; ++q) {
    V3 A = v[e[q][0]], B = v[e[q][1]];
    double dx = sub(B.x, A.x), dy = sub(B.y, A.y), dz = sub(B.z, A.z);
    total = add(total, __dsqrt_rn(add(add(mul(dx, dx), mul(dy, dy)), mul(dz, dz))));
  }
  double h = __ddiv_rn(total, 12.0);
  double thr = mul(FDF_DISTANCE_THRESHOLD, h);
  // cell centroid, walkingsearch.c:286-296
  V3 cc{0.0, 0.0, 0.0};
#pragma unroll
  for (int q = 0; q < 8; ++q) { cc.x = add(cc.x, v[q].x); cc.y = add(cc.y, v[q].y); cc.z = add(cc.z, v[q].z); }
  cc.x = __ddiv_rn(cc.x, 8.0); cc.y = __ddiv_rn(cc.y, 8.0); cc.z = __ddiv_rn(cc.z, 8.0);
  double *row = planes + c * FDF_ROW;
  bool degen = false;
  // face vertex lists, walkingsearch.c:303-378
  degen |= face_plane(v[0], v[3], v[2], v[1], cc, row + 6 * F_BACK);
  degen |= face_plane(v[4], v[7], v[6], v[5], cc, row + 6 * F_FRONT);
  degen |= face_plane(v[0], v[1], v[6], v[7], cc, row + 6 * F_BOTTOM);
  degen |= face_plane(v[3], v[4], v[5], v[2], cc, row + 6 * F_TOP);
  degen |= face_plane(v[0], v[7], v[4], v[3], cc, row + 6 * F_LEFT);
  degen |= face_plane(v[1], v[2], v[5], v[6], cc, row + 6 * F_RIGHT);
  row[36] = thr;
  row[37] = degen ? 1.0 : 0.0;
  if (degen) *any_degenerate = 1u;
}

// The corner field (fdf_corner.cuh), one thread per node.  With cell_start non-null, nodes none of
// whose adjacent cells holds a particle are skipped: the corner field is an intermediate of the
// interpolation and only those nodes are ever read.
// Bound by FP64 adds, 21 a node: of each component's seven two go to the integer pipe (mask 0x88: the
// fourth and the eighth cell's), which then takes as long.  Per step 178 -> 132 us for 4.2M cells with 1M
// particles, 628 -> 465 us for 14M with 16M (one component zero); with four to ten of the 21 there
// 138/491, 137/448, 147/459, 157/489 us.  The lanes of a row's ends take the same path as the others, the
// occupancy test reads a row's two cells at once and every index has 32 bits: with the former per-cell
// branches six integer additions gained nothing (175 us).
// AOS: the output is [Nn][3] instead of [3][Nn] (for the host).
template <bool AOS>
__global__ void k_center_to_corner(const double *__restrict__ ucat, GridDims g, double *__restrict__ corner,
                                   const unsigned int *__restrict__ cell_start, unsigned long long *nodes_done) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const bool work = q < g.Nn;
  int i = 0, j = 0, k = 0;
  if (work) node_ijk(g, (unsigned int)q, i, j, k);
  if (cell_start) {
    // count the nodes this step computes (for the roofline bytes); the cells of a row are neighbours in
    // cell_start, so a row's are empty where nothing starts between the first and the one after the last
    bool need = false;
    if (work) {
      const unsigned int i0 = max(i - 1, 0), i1 = min(i, g.IM - 1) + 1;
      const unsigned int j0 = max(j - 1, 0), j1 = min(j, g.JM - 1), k0 = max(k - 1, 0), k1 = min(k, g.KM - 1);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const unsigned int row = (((e & 2) ? k1 : k0) * g.JM + ((e & 1) ? j1 : j0)) * g.IM;
        need |= __ldg(cell_start + row + i1) > __ldg(cell_start + row + i0);
      }
    }
    if (nodes_done) block_add_u64(need ? 1ull : 0ull, nodes_done);
    if (!need) return;
  }
  if (!work) return;
  double ox, oy, oz;
  fdfx::corner_value<0x88>(ucat, g, i, j, k, ox, oy, oz);
  if (AOS) {
    corner[3 * q] = ox; corner[3 * q + 1] = oy; corner[3 * q + 2] = oz;
  } else {
    corner[q] = ox; corner[g.Nn + q] = oy; corner[2 * g.Nn + q] = oz;
  }
}

// Vector fields between the callers' layout (three components together) and the device's (one array
// per component): one thread per entry, 9 us for 0.9M cells, so that only the copies over the host
// link count.  (In loops on the host they took 33 of the 37 ms of reading 12.6M faces' momentum,
// and an exchange step of 2M particles, with 0.9M cells' ucat in, 5.5 ms against 3.9 now.)
__global__ void k_ucat_in(const double *__restrict__ aos, GridDims g, int mx, int my, double *__restrict__ ucat,
                          float *__restrict__ ucat32) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= g.Nc) return;
  int i, j, k;
  cell_ijk(g, (unsigned int)c, i, j, k);
  const double *v = aos + 3 * (((long long)k * my + j) * mx + i);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    ucat[d * g.Nc + c] = v[d];
    ucat32[d * g.Nc + c] = fdfx::d2f_rn(v[d]);
  }
}

// node_sized: the reference's node-sized layout, whose entries past the cells are zero.
__global__ void k_ucat_out(const double *__restrict__ ucat, GridDims g, int node_sized, double *__restrict__ aos) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= (node_sized ? g.Nn : g.Nc)) return;
  long long c = q;
  bool cell = true;
  if (node_sized) {
    int i, j, k;
    node_ijk(g, (unsigned int)q, i, j, k);
    cell = i < g.IM && j < g.JM && k < g.KM;
    c = ((long long)k * g.JM + j) * g.IM + i;
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) aos[3 * q + d] = cell ? ucat[d * g.Nc + c] : 0.0;
}

template <typename T>
__global__ void k_vec3_out(const T *__restrict__ soa, long long n, double *__restrict__ aos) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= n) return;
#pragma unroll
  for (int d = 0; d < 3; ++d) aos[3 * q + d] = (double)soa[d * n + q];
}

inline unsigned int blocks_for(long long n) { return (unsigned int)((n + 255) / 256); }

}  // namespace

void launch_ucat_in(const double *aos, GridDims g, int node_sized, double *ucat, float *ucat32, cudaStream_t s) {
  k_ucat_in<<<blocks_for(g.Nc), 256, 0, s>>>(aos, g, g.IM + (node_sized ? 1 : 0), g.JM + (node_sized ? 1 : 0), ucat,
                                             ucat32);
}

void launch_ucat_out(const double *ucat, GridDims g, int node_sized, double *aos, cudaStream_t s) {
  k_ucat_out<<<blocks_for(node_sized ? g.Nn : g.Nc), 256, 0, s>>>(ucat, g, node_sized, aos);
}

void launch_vec3_out(const double *soa, long long n, double *aos, cudaStream_t s) {
  k_vec3_out<<<blocks_for(n), 256, 0, s>>>(soa, n, aos);
}

void launch_vec3_out(const float *soa, long long n, double *aos, cudaStream_t s) {
  k_vec3_out<<<blocks_for(n), 256, 0, s>>>(soa, n, aos);
}

void launch_build_planes(const double *coor, GridDims g, double *planes, unsigned int *any_degenerate, cudaStream_t s) {
  int th = 128;
  long long blocks = (g.Nc + th - 1) / th;
  k_build_planes<<<(unsigned)blocks, th, 0, s>>>(coor, g, planes, any_degenerate);
}

void launch_center_to_corner(const double *ucat, GridDims g, double *corner, const unsigned int *cell_start,
                             unsigned long long *nodes_done, cudaStream_t s) {
  k_center_to_corner<false><<<blocks_for(g.Nn), 256, 0, s>>>(ucat, g, corner, cell_start, nodes_done);
}

void launch_center_to_corner_aos(const double *ucat, GridDims g, double *corner, cudaStream_t s) {
  k_center_to_corner<true><<<blocks_for(g.Nn), 256, 0, s>>>(ucat, g, corner, nullptr, nullptr);
}
