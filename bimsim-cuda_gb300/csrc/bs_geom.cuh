// bs_geom.cuh -- per-(pixel, sphere) geometry shared by the near-field kernels.
#pragma once

#include "bs_math.cuh"

namespace bs {

// Geometry that feeds a discrete decision (inside/outside a sphere, d == 0,
// d < 1e-6) is rounded operation by operation in the order of the host
// restatement, with no fused multiply-add, so the GPU and the double
// precision reference agree on every boundary pixel.
__device__ __forceinline__ void pixel_pos(const Scene& sc, int iu, int iv, double p[3]) {
    // quad::operator()(u, v) = (A + X u) + Y v with u = iu / R (nfScalarUf.cu:66-71); quot gives the correctly
    // rounded quotient, as invR = 1 / R is and R's significand is not all ones
    const double u = quot((double)iu, (double)sc.R, sc.invR), v = quot((double)iv, (double)sc.R, sc.invR);
#pragma unroll
    for (int c = 0; c < 3; c++) p[c] = __dadd_rn(__dadd_rn(sc.A[c], __dmul_rn(sc.X[c], u)), __dmul_rn(sc.Y[c], v));
}

// |p - c| as sqrt((x*x + y*y) + z*z), each operation rounded separately
__device__ __forceinline__ double dist_exact(const double p[3], const double c[3], double r[3]) {
    r[0] = __dsub_rn(p[0], c[0]);
    r[1] = __dsub_rn(p[1], c[1]);
    r[2] = __dsub_rn(p[2], c[2]);
    double s = __dadd_rn(__dadd_rn(__dmul_rn(r[0], r[0]), __dmul_rn(r[1], r[1])), __dmul_rn(r[2], r[2]));
    return __dsqrt_rn(s);
}

// Table of one (pixel, sphere) pair.
struct TableSel {
    int64_t off;
    int rows;
    double x;  // fractional row index
};

__device__ __forceinline__ TableSel select_table(const Sphere& S, double d) {
    TableSel t;
    if (d < S.a) {  // internal field, ai = (d - dmin)/(a - dmin) (aR - 1)  (nfScalarUpLut.cu:54)
        t.off = S.uip_off;
        t.rows = S.aR;
        t.x = ((d - S.dmin) / (S.a - S.dmin)) * (S.aR - 1);
    } else {        // scattered field, di = (d - r0)/(dmax - r0) (dR - 1)  (nfScalarUpLut.cu:53)
        t.off = S.usp_off;
        t.rows = S.dR;
        t.x = ((d - S.r0) / (S.dmax - S.r0)) * (S.dR - 1);
    }
    // unnormalised texture coordinates with clamp addressing = clamped index
    t.x = fmin(fmax(t.x, 0.0), (double)(t.rows - 1));
    return t;
}

// select_table with the per-sphere scales (rows - 1) / (range) of the host in
// place of the division: the index may differ in its last bit, which moves a
// sample across a row boundary only where the bilinear value is continuous.
__device__ __forceinline__ TableSel select_table_scaled(const Sphere& S, double d) {
    TableSel t;
    if (d < S.a) {
        t.off = S.uip_off;
        t.rows = S.aR;
        t.x = (d - S.dmin) * S.xs_uip;
    } else {
        t.off = S.usp_off;
        t.rows = S.dR;
        t.x = (d - S.r0) * S.xs_usp;
    }
    t.x = fmin(fmax(t.x, 0.0), (double)(t.rows - 1));
    return t;
}

}  // namespace bs
