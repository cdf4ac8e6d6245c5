// fdf_corner.cuh -- one node of the corner field: InterpolateFieldFromCenterToCorner_Vector_Petsc
// (interpolation.c:598-679).  A node averages its valid adjacent cells in (dk, dj, di) order.  The
// count is a product of per-direction counts of 1 or 2, i.e. 1, 2, 4 or 8, so sum/count is exactly
// sum*(1/count): both are the correctly rounded value of the same real.  The running sum starts at
// 0.0; "0.0 + first" is the first value except that a -0.0 becomes +0.0 (add0).
#pragma once
#include "fdf_internal.cuh"
#include "fdf_exact.cuh"

namespace fdfx {

__device__ __forceinline__ void corner_value(const double *__restrict__ ucat, const GridDims &g, int i, int j, int k,
                                             double &ox, double &oy, double &oz) {
  const double *ux = ucat, *uy = ucat + g.Nc, *uz = ucat + 2 * g.Nc;
  double sx = 0.0, sy = 0.0, sz = 0.0;
  int count = 0;
#pragma unroll
  for (int dk = -1; dk <= 0; ++dk) {
    const long long ck = k + dk;
    if (ck < 0 || ck >= g.KM) continue;
#pragma unroll
    for (int dj = -1; dj <= 0; ++dj) {
      const long long cj = j + dj;
      if (cj < 0 || cj >= g.JM) continue;
#pragma unroll
      for (int di = -1; di <= 0; ++di) {
        const long long ci = i + di;
        if (ci < 0 || ci >= g.IM) continue;
        const long long c = (ck * g.JM + cj) * g.IM + ci;
        const double vx = __ldg(ux + c), vy = __ldg(uy + c), vz = __ldg(uz + c);
        if (count == 0) {
          sx = add0(vx); sy = add0(vy); sz = add0(vz);
        } else {
          sx = add(sx, vx); sy = add(sy, vy); sz = add(sz, vz);
        }
        ++count;
      }
    }
  }
  ox = 0.0; oy = 0.0; oz = 0.0;
  if (count > 0) {
    const int sh = count == 1 ? 0 : count == 2 ? 1 : count == 4 ? 2 : 3;   // sum * 0.5^sh, exact
    ox = scale_down(sx, sh); oy = scale_down(sy, sh); oz = scale_down(sz, sh);
  }
}

}  // namespace fdfx
