// bs_math.cuh -- device arithmetic: complex numbers, the reference's
// Legendre recurrence (rts/math/legendre.h) and
// double-precision spherical Bessel functions for the Mie coefficients and
// the lookup tables.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

#include "bs_internal.h"

namespace bs {

template <class T>
struct cpx {
    T re, im;
};
using zd = cpx<double>;

template <class T>
__host__ __device__ __forceinline__ cpx<T> mk(T r, T i) {
    cpx<T> z;
    z.re = r;
    z.im = i;
    return z;
}
template <class T>
__host__ __device__ __forceinline__ cpx<T> operator+(cpx<T> a, cpx<T> b) { return mk(a.re + b.re, a.im + b.im); }
template <class T>
__host__ __device__ __forceinline__ cpx<T> operator-(cpx<T> a, cpx<T> b) { return mk(a.re - b.re, a.im - b.im); }
template <class T>
__host__ __device__ __forceinline__ cpx<T> operator*(cpx<T> a, cpx<T> b) {
    return mk(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re);
}
template <class T>
__host__ __device__ __forceinline__ cpx<T> operator*(cpx<T> a, T s) { return mk(a.re * s, a.im * s); }
template <class T>
__host__ __device__ __forceinline__ cpx<T> operator*(T s, cpx<T> a) { return mk(a.re * s, a.im * s); }
template <class T>
__host__ __device__ __forceinline__ cpx<T> operator/(cpx<T> a, cpx<T> b) {
    // Smith's algorithm: scale by the larger component of b to avoid overflow
    if (fabs(b.re) >= fabs(b.im)) {
        T r = b.im / b.re, den = b.re + b.im * r;
        return mk((a.re + a.im * r) / den, (a.im - a.re * r) / den);
    }
    T r = b.re / b.im, den = b.re * r + b.im;
    return mk((a.re * r + a.im) / den, (a.im * r - a.re) / den);
}

__device__ __forceinline__ double zabs(zd a) { return hypot(a.re, a.im); }

// sin, cos of a complex argument (rts/math/complex.h:379-395)
__device__ __forceinline__ zd zsin(zd z) { return mk(sin(z.re) * cosh(z.im), cos(z.re) * sinh(z.im)); }
__device__ __forceinline__ zd zcos(zd z) { return mk(cos(z.re) * cosh(z.im), -(sin(z.re) * sinh(z.im))); }

// i^l
__device__ __forceinline__ zd ipow(int l) {
    switch (l & 3) {
        case 0: return mk(1.0, 0.0);
        case 1: return mk(0.0, 1.0);
        case 2: return mk(-1.0, 0.0);
        default: return mk(0.0, -1.0);
    }
}

// ---------------------------------------------------------------------------
// The reference's three-term recurrence
// ---------------------------------------------------------------------------
// P_n from P_{n-1}, P_{n-2} (rts/math/legendre.h:17-25)
__device__ __forceinline__ void legendre_step(int n, double x, double& P0, double& P1) {
    double Pn = ((2 * n - 1) * x * P1 - (n - 1) * P0) / n;
    P0 = P1;
    P1 = Pn;
}

// ---------------------------------------------------------------------------
// Accurate spherical Bessel functions, double precision.
//   j_l: upward from j_0, j_1 while l < x, otherwise Miller's downward
//        recurrence from a start order well above max(l, x), normalised to
//        j_0 = sin z / z (or j_1 when |j_1| > |j_0|);
//   y_l: upward from y_0, y_1 (stable).
// The reference scales J_{l+1/2} with sqrt(PI/(2x)), PI = 3.14159
// (bessjy.cpp:719-723), so every value carries the factor sqrt(3.14159/pi).
// Its Zhang & Jin routines stop at the order where J falls below 1e-200 (the
// MSTA1 estimate) and leave higher entries unset; those entries are zero here.
// ---------------------------------------------------------------------------
// Start order of Miller's recurrence for the orders up to N of an argument of modulus ax and imaginary part im.
// What the start leaves in order l is of relative size exp(-2 eta), eta = M acosh(M / m) - sqrt(M^2 - m^2) from
// m = max(N, ax) on (Debye's expansion), below 2^-60 for M = m + 6 + 8 m^(1/3): 57 steps where m + 16 +
// sqrt(60 (m + 1)) took 80 at m = 25.  Far from the real axis, where j_0 is large beside the start value, the longer
// run keeps the scale in range.
__device__ __forceinline__ int miller_start(int N, double ax, double im = 0.0) {
    const double m = fmax((double)N, ax);
    if (fabs(im) > 20.0) return (int)(m + 16.0 + sqrt(60.0 * (m + 1.0)));
    return (int)m + 7 + (int)(8.f * cbrtf((float)m));
}

// |v| above 2^830 (7e249), from the high word: a comparison off the FP64 pipe
__device__ __forceinline__ bool beyond_2_830(double v) { return (__double2hiint(v) & 0x7fffffff) >= 0x73d00000; }

__device__ __forceinline__ double digits_at(int n, double x) {
    return 0.5 * log10(6.28 * n) - n * log10(1.36 * x / n);
}

// Order where J_n(x) ~ 10^-mp, by secant iteration on digits_at: routine MSTA1 of
// S. Zhang and J. Jin, Computation of Special Functions (Wiley, 1996), which the
// reference's bessjy.cpp:268-290 also follows (its constants 6.28, 1.36, 1.1).
__device__ inline int order_cutoff(double x, int mp) {
    double a = fabs(x);
    int lo = (int)(1.1 * a) + 1, hi = lo + 5;
    double flo = digits_at(lo, a) - mp, fhi = digits_at(hi, a) - mp;
    int nn = hi;
    for (int it = 0; it < 20; it++) {
        nn = (int)(hi - (hi - lo) / (1.0 - flo / fhi));
        double f = digits_at(nn, a) - mp;
        if (abs(nn - hi) < 1) break;
        lo = hi;
        flo = fhi;
        hi = nn;
        fhi = f;
    }
    return nn;
}

// min(N, order_cutoff) without the iteration where J_N(x) is above 1e-190 by the same estimate
// (which rises with the order), as it nearly always is.
__device__ inline int orders_kept(int N, double x) {
    const float a = (float)fabs(x), n = (float)N;
    const float digits = 0.5f * log10f(6.28f * n) - n * log10f(1.36f * a / n);
    if (digits < 190.f) return N;
    const int m = order_cutoff(x, 200);
    return m < N ? m : N;
}

// a / b by multiplication with inv = 1 / b and one correction with the exact remainder
// (Markstein, IBM J. Res. Dev. 34, 1990): the quotient's own rounding, at two instructions more
// than a product.
__device__ __forceinline__ double quot(double a, double b, double inv) {
    const double q = a * inv;
    return fma(fma(-q, b, a), inv, q);
}

// j[l], y[l] for l = 0..N (stride `st` between orders) of a real x > 0.  The recurrences' factors
// (2l + 1) / x come from one reciprocal, which leaves one fused multiply-add per order in the
// serial chain (a division per order before: 4096 x 50 table rows 0.40 ms).
__device__ inline void sph_real(int N, double x, double* j, double* y, int st) {
    const double cs = sqrt(PI_BES / TRUE_PI);
    if (x < 1e-15) {
        double sc = sqrt(PI_BES / (x * 2.0));
        for (int l = 0; l <= N; l++) {
            j[l * st] = 0.0 * sc;
            y[l * st] = -1e308 * sc;
        }
        return;
    }
    int Nv = N;
    if (N >= 2 && N > (int)(0.9 * x)) Nv = orders_kept(N, x);
    const double inv = 1.0 / x;
    double s, c;
    sincos(x, &s, &c);
    double j0 = s / x, j1 = s / (x * x) - c / x;
    if (Nv < x) {
        j[0] = j0;
        if (Nv >= 1) j[st] = j1;
        double a = j0, b = j1;
        for (int l = 2; l <= Nv; l++) {
            double t = fma(quot(2 * l - 1, x, inv), b, -a);
            a = b;
            b = t;
            j[l * st] = t;
        }
    } else {
        int M = miller_start(Nv, x);
        double fp = 0.0, fc = 1e-300;
        if (M <= Nv) j[M * st] = fc;
        for (int l = M; l >= 1; l--) {
            double fm = fma(quot(2 * l + 1, x, inv), fc, -fp);
            fp = fc;
            fc = fm;
            if (l - 1 <= Nv) j[(l - 1) * st] = fm;
            if (beyond_2_830(fc)) {
                for (int q = l - 1; q <= Nv; q++) j[q * st] *= 1e-250;
                fc *= 1e-250;
                fp *= 1e-250;
            }
        }
        double sc = (fabs(j0) >= fabs(j1)) ? j0 / j[0] : j1 / j[st];
        for (int l = 0; l <= Nv; l++) j[l * st] *= sc;
    }
    double ya = -c / x, yb = -c / (x * x) - s / x;
    y[0] = ya;
    if (Nv >= 1) y[st] = yb;
    for (int l = 2; l <= Nv; l++) {
        double t = fma(quot(2 * l - 1, x, inv), yb, -ya);
        ya = yb;
        yb = t;
        y[l * st] = t;
    }
    for (int l = 0; l <= N; l++) {
        if (l > Nv) {
            j[l * st] = 0.0;
            y[l * st] = 0.0;
        } else {
            j[l * st] *= cs;
            y[l * st] *= cs;
        }
    }
}

// j[l], l = 0..N, of a complex argument.
__device__ inline void sph_complex(int N, zd z, zd* j) {
    const double cs = sqrt(PI_BES / TRUE_PI);
    double az = zabs(z);
    int Nv = N;
    if (N >= 2 && N > (int)(0.25 * az)) Nv = orders_kept(N, az);
    const zd inv = mk(1.0, 0.0) / z;
    zd s = zsin(z), c = zcos(z);
    zd j0 = s / z, j1 = s / (z * z) - c / z;
    int M = miller_start(N, az, z.im);
    zd fp = mk(0.0, 0.0), fc = mk(1e-300, 0.0);
    if (M <= N) j[M] = fc;
    for (int l = M; l >= 1; l--) {
        const zd w = (double)(2 * l + 1) * inv;
        const zd fm = mk(fma(w.re, fc.re, fma(-w.im, fc.im, -fp.re)), fma(w.re, fc.im, fma(w.im, fc.re, -fp.im)));
        fp = fc;
        fc = fm;
        if (l - 1 <= N) j[l - 1] = fm;
        if (beyond_2_830(fc.re) || beyond_2_830(fc.im)) {
            for (int q = l - 1; q <= N; q++) j[q] = j[q] * 1e-250;
            fc = fc * 1e-250;
            fp = fp * 1e-250;
        }
    }
    zd sc = (zabs(j0) >= zabs(j1)) ? j0 / j[0] : j1 / j[1 <= N ? 1 : 0];
    for (int l = 0; l <= N; l++) j[l] = j[l] * sc;
    for (int l = 0; l <= N; l++) j[l] = l > Nv ? mk(0.0, 0.0) : j[l] * cs;
}

}  // namespace bs
