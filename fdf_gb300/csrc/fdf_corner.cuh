// fdf_corner.cuh -- one node of the corner field: InterpolateFieldFromCenterToCorner_Vector_Petsc
// (interpolation.c:598-679).  A node averages its valid adjacent cells in (dk, dj, di) order.  The
// count is a product of per-direction counts of 1 or 2, i.e. 1, 2, 4 or 8, so sum/count is exactly
// sum*(1/count): both are the correctly rounded value of the same real.  The running sum starts at
// 0.0; "0.0 + first" is the first value except that a -0.0 becomes +0.0 (add0).  It is never -0.0 after
// that, so a cell that is not there can add +0.0: the lanes of a row's ends take the others' path.
#pragma once
#include "fdf_internal.cuh"
#include "fdf_exact.cuh"

namespace fdfx {

// INT: bit e puts the addition of the e-th cell to each component on the integer pipe (the same bits).
template <int INT>
__device__ __forceinline__ void corner_value(const double *__restrict__ ucat, const GridDims &g, int i, int j, int k,
                                             double &ox, double &oy, double &oz) {
  const unsigned int IM = g.IM, JM = g.JM;
  const bool i_lo = i > 0, i_hi = i < g.IM, j_lo = j > 0, j_hi = j < g.JM, k_lo = k > 0, k_hi = k < g.KM;
  double sx = 0.0, sy = 0.0, sz = 0.0;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const bool row_in = ((r & 2) ? k_hi : k_lo) && ((r & 1) ? j_hi : j_lo);
    // the row's two cells; the first one's index wraps for i = 0, where it is not read
    const unsigned int c1 = ((unsigned int)(k - 1 + (r >> 1)) * JM + (unsigned int)(j - 1 + (r & 1))) * IM + (unsigned int)i;
#pragma unroll
    for (int di = 0; di < 2; ++di) {
      const int e = 2 * r + di;
      const bool in = row_in && (di ? i_hi : i_lo);
      const double *u = ucat + (di ? c1 : c1 - 1u);
      const double vx = in ? __ldg(u) : 0.0, vy = in ? __ldg(u + g.Nc) : 0.0, vz = in ? __ldg(u + 2 * g.Nc) : 0.0;
      if (e == 0) {
        sx = add0(vx); sy = add0(vy); sz = add0(vz);
      } else {
        sx = (INT >> e & 1) ? add_int(sx, vx) : add(sx, vx);
        sy = (INT >> e & 1) ? add_int(sy, vy) : add(sy, vy);
        sz = (INT >> e & 1) ? add_int(sz, vz) : add(sz, vz);
      }
    }
  }
  const int sh = (int)(i_lo && i_hi) + (int)(j_lo && j_hi) + (int)(k_lo && k_hi);   // sum * 0.5^sh, exact
  ox = scale_down(sx, sh); oy = scale_down(sy, sh); oz = scale_down(sz, sh);
}

}  // namespace fdfx
