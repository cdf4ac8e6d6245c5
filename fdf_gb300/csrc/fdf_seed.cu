// fdf_seed.cu -- on-device volumetric particle seeding for large synthetic workloads.
//
// Restates, on the GPU, the harness generator of fdf_gb300/workloads.py
// (volumetric_particles): the reference's volumetric initialisation
// (ParticleSwarm.c:229-312) -- a random cell, random logical coordinates in [0,1)
// clamped to 1 - 1e-7 -- mapped to physical space by the trilinear blend of
// Metric.c:48-62, with the same counter-based splitmix64 streams and the same FP64
// operation order (no FMA), so the particles are bit-identical to the host's.
#include "fdf_internal.cuh"
#include "fdf_exact.cuh"

namespace {

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

// uniform01(seed, stream)[idx] of workloads.py: the top 53 bits of the stream's word, times 2^-53.
// Exact, so INT puts it together from the bits.
template <bool INT>
__device__ __forceinline__ double uniform01(unsigned long long seed, unsigned long long stream,
                                            unsigned long long idx) {
  const unsigned long long base =
      mix64(seed * 0xD1B54A32D192ED03ULL + stream * 0xA24BAED4963EE407ULL + 0x632BE59BD9B4E019ULL);
  const unsigned long long k = mix64(base + (idx + 1ULL) * 0x9E3779B97F4A7C15ULL) >> 11;
  if (!INT) return __dmul_rn((double)k, 0x1p-53);
  if (k == 0ull) return 0.0;
  const int lz = __clzll((long long)k);   // 11 .. 63
  return __longlong_as_double((long long)(((unsigned long long)(1032 - lz) << 52) + (k << (lz - 11))));
}

// (long long)x for 0 <= x < 2^31.
__device__ __forceinline__ int truncate(double x) {
  const unsigned long long u = fdfx::ubits(x);
  const int e = (int)(u >> 52) - 1023;
  return e < 0 ? 0 : (int)(((u & 0x000fffffffffffffull) | 0x0010000000000000ull) >> (52 - e));
}

// Bound by FP64 when written with it (118 FP64 instructions per particle, 12.0 ms for 64M of them in
// 14M cells): the conversions, the clamps and the 39 products run on the integer pipe, with the same
// bits, and 24 subtractions and additions are left: 9.5 ms, by the random gathers of eight nodes.
// INT false: up to SEED_FEW particles each warp's own chain is the time, and the FP64 pipe makes it shorter (the
// whole call, 10,000 particles 22.5 us against 24.9, 30,000 22.6 against 25.6; 60,000 28.8 against 26.7).
constexpr long long SEED_FEW = 3 << 14;
template <bool INT>
__global__ void k_seed(const double *__restrict__ coor, GridDims g, double dIM, double dJM, double dKM, long long n,
                       unsigned long long seed, long long pid_base, int hint, int form32, double P0, float P0f,
                       SwarmBuf b) {
  const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (p >= n) return;
  const unsigned long long idx = (unsigned long long)p;
  auto mul = [](double a, double c) { return INT ? fdfx::mul_int(a, c) : fdfx::mul(a, c); };
  auto below = [](double v, int cells) { return min(INT ? truncate(v) : (int)v, cells - 1); };
  const double r[3] = {uniform01<INT>(seed, 0, idx), uniform01<INT>(seed, 1, idx), uniform01<INT>(seed, 2, idx)};
  const int ci = below(mul(r[0], dIM), g.IM), cj = below(mul(r[1], dJM), g.JM), ck = below(mul(r[2], dKM), g.KM);
  const double lim = 1.0 - 1.0e-7;
  double t[3][2];   // the two weights of each direction: 1 - xi, xi
#pragma unroll
  for (int d = 0; d < 3; ++d) {   // np.maximum(np.minimum(u, lim), 0.0) on [0,1) values, ordered as their bits are
    const unsigned long long u = min(fdfx::ubits(uniform01<INT>(seed, 3 + d, idx)), fdfx::ubits(lim));
    t[d][1] = __longlong_as_double((long long)u);
    t[d][0] = fdfx::sub(1.0, t[d][1]);
  }
  double x = 0.0, y = 0.0, z = 0.0;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const double N = mul(mul(t[0][c & 1], t[1][(c >> 1) & 1]), t[2][c >> 2]);
    const long long ii = ci + (c & 1), jj = cj + ((c >> 1) & 1), kk = ck + (c >> 2);
    const double *V = coor + 3 * ((kk * (g.JM + 1) + jj) * (long long)(g.IM + 1) + ii);
    const double vx = mul(N, V[0]), vy = mul(N, V[1]), vz = mul(N, V[2]);
    x = c ? fdfx::add(x, vx) : fdfx::add0(vx);
    y = c ? fdfx::add(y, vy) : fdfx::add0(vy);
    z = c ? fdfx::add(z, vz) : fdfx::add0(vz);
  }
  if (form32) {
    const double v[3] = {x, y, z};
    double *dst[3] = {b.x, b.y, b.z};
    for (int q = 0; q < 3; ++q) *reinterpret_cast<float2 *>(dst[q] + p) = fdfx::split_rn(v[q]);
    b.uf[p] = 0.f; b.vf[p] = 0.f; b.wf[p] = 0.f;
    b.a1f[p] = 0.f; b.a2f[p] = 0.f; b.a3f[p] = 0.f;
    b.Pf[p] = P0f;
  } else {
    b.x[p] = x; b.y[p] = y; b.z[p] = z;
    b.u[p] = 0.0; b.v[p] = 0.0; b.w[p] = 0.0;
    b.a1[p] = 0.0; b.a2[p] = 0.0; b.a3[p] = 0.0;
    b.P[p] = P0;
  }
  b.pid[p] = pid_base + p;
  b.cell[p] = hint ? (int)(((long long)ck * g.JM + cj) * g.IM + ci) : -1;
  b.status[p] = ST_UNINITIALIZED;
}

}  // namespace

void launch_seed(const double *coor, GridDims g, long long n, unsigned long long seed, long long pid_base, int hint,
                 int form32, double P0, const SwarmBuf &b, cudaStream_t s) {
  if (n <= 0) return;
  auto *kernel = n <= SEED_FEW ? k_seed<false> : k_seed<true>;
  kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(coor, g, (double)g.IM, (double)g.JM, (double)g.KM, n, seed,
                                                    pid_base, hint, form32, P0, (float)P0, b);
}
