// Shared by the column-pass kernels (lh_column.cu, lh_column_tile.cu): the RK
// coefficients and the rows of the Helmholtz matrices.
#pragma once

#include "lh_kernels.cuh"

namespace lh {

struct RK {
    double a, b, g, c, d;
};

__device__ __forceinline__ RK rk_coeffs(int kRK)
{
    // start.f90:439-453
    RK r;
    if (kRK == 1) {
        r.a = 4.0 / 15.0; r.b = 4.0 / 15.0; r.g = 8.0 / 15.0; r.c = 0.0; r.d = 8.0 / 15.0;
    } else if (kRK == 2) {
        r.a = 1.0 / 15.0; r.b = 1.0 / 15.0; r.g = 5.0 / 12.0; r.c = -17.0 / 60.0; r.d = 2.0 / 15.0;
    } else {
        r.a = 1.0 / 6.0; r.b = 1.0 / 6.0; r.g = 3.0 / 4.0; r.c = -5.0 / 12.0; r.d = 1.0 / 3.0;
    }
    return r;
}

__device__ __forceinline__ double2 cscale(double s, double2 a) { return make_double2(s * a.x, s * a.y); }

// Helmholtz rows of one grid (solveU's LU_build, tridLU_3D.f90:163-221):
// row 0 [0, 1, w0], rows 1..n [-beta d1, 1 - beta (d2 + k2), -beta d3],
// row n+1 [wt, 1, 0].  With beta times a power of two, and that as one, the
// interior rows come out times it, the same bits otherwise.
struct HRow {
    double a1, a2, a3;
};
__device__ __forceinline__ HRow helm_row(int j, int n, const double *d, double beta, double k2x, double k2z,
                                         double w0, double wt, double one = 1.0)
{
    if (j == 0) return HRow{0.0, 1.0, w0 * 1.0};
    if (j == n + 1) return HRow{wt, 1.0, 0.0};
    return HRow{-beta * d[3 * j], one - beta * (d[3 * j + 1] + k2x + k2z), -beta * d[3 * j + 2]};
}

}  // namespace lh
