// bs_nearfield.cu -- near-field kernels: incident field Uf, Mie coefficients,
// per-sphere lookup tables, and the scattered field Us summed over spheres
// and Monte Carlo plane waves, with the Uf + Us assembly of nfSumUf.cu fused
// into the epilogue.
#include <cuda_runtime.h>

#include <cmath>

#include "bs_geom.cuh"
#include "bs_kernels.h"
#include "bs_math.cuh"
#include "bs_mie.cuh"

namespace bs {

// ---------------------------------------------------------------------------
// Incident field (double precision; stored as T)
// ---------------------------------------------------------------------------
// gpuScalarUf, nfScalarUf.cu:46-175: Debye-focused field as a Legendre series over l = 0..m,
//   2 pi A sum_l i^l w_l j_l(k d) P_l(cos),
// with w_l = (P_{l+1} - P_{l-1})(cos a) - (P_{l+1} - P_{l-1})(cos b) of the condenser aperture the same for
// every pixel.  The kernel is bound by the FP64 pipe, so the host's UfOrder carries all that depends on the order
// alone: P_l runs in monic form (u_l = x u_{l-1} - beta_l u_{l-2}, two instructions), its scale, w_l and
// the sign of i^l in one weight; even orders sum into the real part, odd ones into the imaginary part.
// 3072^2 pixels, 11 orders, table mode: 6.0 -> 2.4 ms; direct mode at 1280^2: 1.43 -> 0.72 ms, and 0.57 ms with the
// clamps, the order's factors and four of the five divisions off the pipe as well.
struct UfLegendre {  // u_l(x), l = 0, 1, 2, ... in turn
    double u2 = 0, u1 = 1;
    __device__ __forceinline__ double next(int l, double x, double beta) {
        if (l == 0) return 1.0;
        const double u = fma(x, u1, -beta * u2);
        u2 = u1;
        u1 = u;
        return u;
    }
};

// The "convergence" clamp of the upward j_l (spherical_bessel.h:102-119: once l > x, a value outside [0.0145, 0.4] is
// replaced by zero) off the FP64 pipe: the high words of CONV_MIN and CONV_MAX decide, but where they are equal.
__device__ __forceinline__ double clamp_j(double j, bool beyond) {
    constexpr int LO = 0x3f8db22d, HI = 0x3fd99999;
    const int h = __double2hiint(j);
    return beyond && (h <= LO || h >= HI) && (h < LO || h > HI || j < CONV_MIN || j > CONV_MAX) ? 0.0 : j;
}

// The clamped upward j_l recurrence, one reciprocal for all quotients and orders.
__device__ zd uf_direct(const Scene& sc, const UfOrder* __restrict__ w, const double p[3]) {
    double r[3];
    double d = dist_exact(p, sc.focus, r);
    if (d < EPS_FLOAT) return mk(sc.amp * 2 * PI_REF * (sc.cos_a - sc.cos_b), 0.0);
    const double cth = quot(sc.kdir[0] * r[0] + sc.kdir[1] * r[1] + sc.kdir[2] * r[2], d, 1.0 / d);
    const double kd = sc.kmag * d, inv = 1.0 / kd;
    double s, c;
    sincos(kd, &s, &c);
    double j0 = quot(s, kd, inv), j1 = quot(j0, kd, inv) - quot(c, kd, inv);
    const int lclamp = kd < (double)MAX_ORDER ? (int)kd : MAX_ORDER;  // l > kd exactly for l > lclamp
    zd sum = mk(j0 * w[0].w, 0.0);
    if (sc.m == 0) return sum;
    double u2 = 1.0, u1 = cth;  // u_{l-1} and u_l, see UfLegendre
    sum.im = j1 * u1 * w[1].w;
    auto step = [&](int l) {  // j_l u_l
        const double jl = clamp_j(fma(quot(w[l].odd, kd, inv), j1, -j0), l > lclamp);
        j0 = j1;
        j1 = jl;
        const double u = fma(cth, u1, -w[l].beta * u2);
        u2 = u1;
        u1 = u;
        return jl * u;
    };
    for (int l = 2; l <= sc.m; l += 2) {
        sum.re = fma(step(l), w[l].w, sum.re);
        if (l + 1 > sc.m) break;
        sum.im = fma(step(l + 1), w[l + 1].w, sum.im);
    }
    return sum;
}

// gpuScalarUfLut, nfScalarUfLut.cu:11-123: j_l(k d) read from the table with
// linear filtering along d (texture y) and exact order (texture x = l + 0.5).
__device__ zd uf_lut(const Scene& sc, const double* __restrict__ tab, const UfOrder* __restrict__ w,
                     const double p[3]) {
    double r[3];
    double d = dist_exact(p, sc.focus, r);
    if (d == 0) return mk(sc.amp * 2 * PI_REF * (sc.cos_a - sc.cos_b), 0.0);
    const double cth = (sc.kdir[0] * r[0] + sc.kdir[1] * r[1] + sc.kdir[2] * r[2]) / d;
    const int L = sc.m + 1;
    double y = (d - sc.uf_dmin) * sc.uf_scale;
    y = fmin(fmax(y, 0.0), (double)(sc.uf_dR - 1));
    const int i0 = (int)y;
    const double be = y - i0;
    const int i1 = min(i0 + 1, sc.uf_dR - 1);
    const double* t0 = tab + (size_t)i0 * L;
    const double* t1 = tab + (size_t)i1 * L;
    UfLegendre P;
    zd sum = mk(0.0, 0.0);
    for (int l = 0; l <= sc.m; l += 2) {
        double a = t0[l];
        sum.re = fma(fma(be, t1[l] - a, a) * P.next(l, cth, w[l].beta), w[l].w, sum.re);
        if (l + 1 > sc.m) break;
        a = t0[l + 1];
        sum.im = fma(fma(be, t1[l + 1] - a, a) * P.next(l + 1, cth, w[l + 1].beta), w[l + 1].w, sum.im);
    }
    return sum;
}

template <class T>
__global__ void uf_kernel(Scene sc, const double* __restrict__ tab, const UfOrder* __restrict__ w,
                          cpx<T>* __restrict__ Uf) {
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= sc.R * sc.R) return;
    double p[3];
    pixel_pos(sc, idx % sc.R, idx / sc.R, p);
    zd v;
    if (!sc.scalar && sc.lut_uf) {
        v = mk(0.0, 0.0);  // nfVectorUfLut.cu:7-10 is empty
    } else if (sc.plane_wave) {
        // gpuScalarUfp, nfScalarUf.cu:9-44
        double kr = sc.kmag * (sc.kdir[0] * (p[0] - sc.focus[0]) + sc.kdir[1] * (p[1] - sc.focus[1]) +
                               sc.kdir[2] * (p[2] - sc.focus[2]));
        double s, c;
        sincos(kr, &s, &c);
        v = mk(c * sc.amp, s * sc.amp);
    } else if (sc.lut_uf) {
        v = uf_lut(sc, tab, w, p);
    } else {
        v = uf_direct(sc, w, p);
    }
    Uf[idx] = mk((T)v.re, (T)v.im);
}

// nearfieldStruct::calcBesselLut (nearfield.cpp:222-283): j_l(k d) for
// d in [dmin, dmax], NaN/Inf replaced by 0 (1 for l = 0 at k d = 0).
__global__ void uf_table_kernel(Scene sc, double* __restrict__ tab, double* __restrict__ scratch) {
    int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= sc.uf_dR) return;
    int L = sc.m + 1;
    double dr = (sc.uf_dmax - sc.uf_dmin) / (sc.uf_dR - 1);
    double d = id * dr + sc.uf_dmin;
    double kd = sc.kmag * d;
    double* j = tab + (size_t)id * L;
    double* y = scratch + (size_t)id * L;
    sph_real(sc.m, kd, j, y, 1);
    for (int l = 0; l < L; l++) {
        double v = j[l];
        if (isnan(v) || isinf(v)) j[l] = (kd == 0 && l == 0) ? 1.0 : 0.0;
    }
}

// ---------------------------------------------------------------------------
// Mie coefficients (sphere::calcCoeff, sphere.cpp:21-97), one block per sphere
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(MIE_NT) mie_kernel(const Sphere* __restrict__ sph, double k, zd* __restrict__ A,
                                                     zd* __restrict__ B) {
    __shared__ MieShared sm;
    const Sphere& S = sph[blockIdx.x];
    mie_block(sm, S.Nl, S.a, mk(S.n_re, S.n_im), k, A + S.coef_off, B + S.coef_off);
}

// Per-row order coefficients of the spheres [s0, s0 + n) in one launch:
//   rows [0, dR):  C_l(r) = B_l (j_l + i y_l)(k r),  r in [r0, dmax]  (sphere.cpp:154-203)
//   rows [dR, dR+aR): D_l(r) = A_l j_l(k n r),       r in [0, a]      (sphere.cpp:99-152)
// Thread g takes global row g; starts[i] / starts[n + 1 + i] are sphere i's first global row and its first
// coefficient in tab (rows of Nl + 1 coefficients; starts[n], the total row count, bounds the grid).  The scratch
// holds 2 (Nl + 1) doubles per row: every order up to MAX_ORDER fits, whatever the sphere.  With `bias` (mixed path)
// every coefficient is stored as SplitCoef instead, and bias[g] is a power of two of at least twice the sum of the
// row's coefficients, see lut_build_mixed_kernel.
// Bound by the FP64 instructions on one thread's chain: 1600 rows of 25 orders 77 us, 205 000 rows of 21 orders 230 us.
// Four warps sharing 32 rows through shared memory took 44 and 213 us, but orders above 434 did not fit it, and in
// some blocks with rows of two spheres two of the warps formed a wrong scale, for no reason that the source shows (run
// on the CPU with its barriers it has no race and no dependence on what the memory held before).  Here a
// thread reads only what it has written itself.
__global__ void __launch_bounds__(128) coef_rows_batch_kernel(const Sphere* __restrict__ sph, int s0, int n,
                                                              const long long* __restrict__ starts, double k,
                                                              const zd* __restrict__ A, const zd* __restrict__ B,
                                                              zd* __restrict__ tab, double* __restrict__ scratch,
                                                              float* __restrict__ bias) {
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= starts[n]) return;
    int lo = 0, hi = n - 1;  // last sphere whose first row is <= g
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (starts[mid] <= g) lo = mid;
        else hi = mid - 1;
    }
    const Sphere& S = sph[s0 + lo];
    const int row = (int)(g - starts[lo]), L = S.Nl + 1;
    const long long c0 = starts[n + 1 + lo] + (long long)row * L;
    zd* out = tab + c0;
    double* sj = scratch + 2 * c0;
    const zd* a = (row < S.dR ? B : A) + S.coef_off;
    if (row < S.dR) {
        const double dr = (S.dmax - S.r0) / (S.dR - 1);
        sph_real(S.Nl, k * (row * dr + S.r0), sj, sj + L, 1);
    } else if (row > S.dR) {  // the centre, row dR, has the order 0 alone
        const double da = S.a / (S.aR - 1);
        sph_complex(S.Nl, (mk(S.n_re, S.n_im) * k) * ((row - S.dR) * da), reinterpret_cast<zd*>(sj));
    }
    float sum = 0.f;
    for (int l = 0; l < L; l++) {
        zd c;
        if (row < S.dR) c = a[l] * mk(sj[l], sj[L + l]);
        else if (row > S.dR) c = a[l] * mk(sj[2 * l], sj[2 * l + 1]);
        else c = a[l] * mk(l == 0 ? 1.0 : 0.0, 0.0);
        if (bias) {  // {hr, hi, lr, li} of SplitCoef, in the bits of two doubles
            const float hr = (float)c.re, hi = (float)c.im;
            const float lr = (float)(c.re - (double)hr), li = (float)(c.im - (double)hi);
            sum += fmaxf(fabsf(hr), fabsf(hi));
            c = mk(__hiloint2double(__float_as_int(hi), __float_as_int(hr)),
                   __hiloint2double(__float_as_int(li), __float_as_int(lr)));
        }
        out[l] = c;
    }
    if (bias) bias[g] = scalbnf(1.f, ilogbf(fmaxf(sum, 1e-30f)) + 2);
}

// P_l(cos theta_t), theta_t = t * dtheta (sphere.cu:16-21).  The reference's step
// (PI) / (thetaR - 1) divides the float literal PI by an int: a single-precision
// quotient in every build, kept here.
__global__ void legendre_table_kernel(int thetaR, int Lmax, double* __restrict__ P) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= thetaR) return;
    double dtheta = (double)__fdiv_rn(3.14159f, (float)(thetaR - 1));
    double x = cos(dtheta * t);
    double* row = P + (size_t)t * Lmax;
    double P0 = 1, P1 = x;
    row[0] = P0;
    if (Lmax > 1) row[1] = P1;
    for (int l = 2; l < Lmax; l++) {
        legendre_step(l, x, P0, P1);
        row[l] = P1;
    }
}

// The mixed path's copy of that table, order-major: P_l of angle t at P[l * stride + t] as the
// nearest float and the rest.
__global__ void legendre_split_kernel(int thetaR, int Lmax, int stride, float2* __restrict__ P) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= thetaR) return;
    double dtheta = (double)__fdiv_rn(3.14159f, (float)(thetaR - 1));
    double x = cos(dtheta * t);
    double P0 = 1, P1 = x;
    for (int l = 0; l < Lmax; l++) {
        if (l > 1) legendre_step(l, x, P0, P1);
        const double v = l == 0 ? 1.0 : P1;
        const float h = (float)v;
        P[(size_t)l * stride + t] = make_float2(h, (float)(v - (double)h));
    }
}

// ---------------------------------------------------------------------------
// LUT build: T(r, t) = sum_l coef_l(r) P_l(cos theta_t) (gpuScalarUsp /
// gpuScalarUip, sphere.cu:4-99), then stored as bilinear patches
//     {T00, T10 - T00, T01 - T00, T11 - T10 - T01 + T00}
// at (r, t), with r+1 and t+1 clamped, so that one 32-byte (float) or 64-byte
// (double) load gives a whole bilinear cell.
// ---------------------------------------------------------------------------
// Bound by the FP64 pipe (2 multiply-adds per entry and order).  A tile of 15 x 31 cells sums 16 x 32 entries, two
// for each thread: a tenth of the work is its neighbours' again (8 x 32 cells: a quarter, the last pass of 41 of 256
// threads taking the time of two full warps).  One launch for the tables of a batch: 8 spheres with 576 x 1000 entries
// of 17 orders 0.42 ms in 16 launches of that tile, 0.30 ms in 2 now.
constexpr int LB_TR = 15, LB_TT = 31;

__global__ void __launch_bounds__(256) lut_build_kernel(const LutBuildJob* __restrict__ jobs, const zd* __restrict__ tab,
                                                        const double* __restrict__ P, int Pstride,
                                                        Patch<double>* __restrict__ out) {
    __shared__ zd sv[LB_TR + 1][LB_TT + 1];
    const LutBuildJob& job = jobs[blockIdx.z];
    const int rows = job.rows, L = job.L, thetaR = job.thetaR;
    const int r0 = blockIdx.y * LB_TR, t0 = blockIdx.x * LB_TT;
    if (r0 >= rows || t0 >= thetaR) return;
    tab += job.tab_off;
    out += job.lin_off;
    for (int e = threadIdx.x; e < (LB_TR + 1) * (LB_TT + 1); e += 256) {
        const int i = e / (LB_TT + 1), j = e % (LB_TT + 1);
        const int r = min(r0 + i, rows - 1), t = min(t0 + j, thetaR - 1);
        const zd* c = tab + (size_t)r * L;
        const double* pl = P + (size_t)t * Pstride;
        zd acc = mk(0.0, 0.0);
        for (int l = 0; l < L; l++) acc = acc + c[l] * pl[l];
        sv[i][j] = acc;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < LB_TR * LB_TT; e += 256) {
        const int i = e / LB_TT, j = e % LB_TT, r = r0 + i, t = t0 + j;
        if (r >= rows || t >= thetaR) continue;
        const zd a = sv[i][j], b = sv[i + 1][j], c = sv[i][j + 1], d = sv[i + 1][j + 1];
        Patch<double> pt;
        pt.v[0] = a.re;
        pt.v[1] = a.im;
        pt.v[2] = b.re - a.re;
        pt.v[3] = b.im - a.im;
        pt.v[4] = c.re - a.re;
        pt.v[5] = c.im - a.im;
        pt.v[6] = d.re - b.re - c.re + a.re;
        pt.v[7] = d.im - b.im - c.im + a.im;
        out[(size_t)r * thetaR + t] = pt;
    }
}

// The tables of the plain mixed kernel: the same sums, rounded to float2 in linear rows with the last column repeated.
// A thread per entry, 8 rows x 32 angles per block.
__global__ void __launch_bounds__(256) lut_build_plain_kernel(const LutBuildJob* __restrict__ jobs,
                                                              const zd* __restrict__ tab, const double* __restrict__ P,
                                                              int Pstride, float2* __restrict__ lin) {
    const LutBuildJob& j = jobs[blockIdx.z];
    const int r = blockIdx.y * 8 + (threadIdx.x >> 5), t = blockIdx.x * 32 + (threadIdx.x & 31);
    if (r >= j.rows || t >= j.thetaR) return;
    const zd* c = tab + j.tab_off + (size_t)min(r, j.last) * j.L;
    const double* pl = P + (size_t)t * Pstride;
    zd acc = mk(0.0, 0.0);
    for (int l = 0; l < j.L; l++) acc = acc + c[l] * pl[l];
    const float2 v = make_float2((float)acc.re, (float)acc.im);
    float2* row = lin + j.lin_off + (size_t)r * j.lin_stride;
    row[t] = v;
    if (t == j.thetaR - 1) row[j.thetaR] = v;  // clamped neighbour of the last column
}

// Per (sphere, wave): (subA / nk) exp(i k k_w . (p_s - f)) (nfScalarUpLut.cu:71,84,90)
template <class T>
__global__ void phase_kernel(Scene sc, const Sphere* __restrict__ sph, const double* __restrict__ waves,
                             cpx<T>* __restrict__ ph, float4* __restrict__ kw4) {
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < sc.nk && kw4) {
        kw4[idx] = make_float4((float)waves[3 * idx], (float)waves[3 * idx + 1], (float)waves[3 * idx + 2], 0.f);
    }
    if (idx >= sc.ns * sc.nk) return;
    int s = idx / sc.nk, w = idx % sc.nk;
    const double* k = waves + 3 * w;
    double c0 = sph[s].p[0] - sc.focus[0], c1 = sph[s].p[1] - sc.focus[1], c2 = sph[s].p[2] - sc.focus[2];
    double arg = sc.kmag * (k[0] * c0 + k[1] * c1 + k[2] * c2);
    double sn, cs;
    sincos(arg, &sn, &cs);
    ph[idx] = mk((T)(sc.wave_amp * cs), (T)(sc.wave_amp * sn));
}

// ---------------------------------------------------------------------------
// Scattered field from the LUTs (gpuScalarUpLut, nfScalarUpLut.cu:11-97),
// all spheres of [s0, s1) in one launch, then Uf added where the pixel is
// outside every sphere (nfSumUf.cu:6-49).
// ---------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// Plain double precision, one pixel per thread.  Bound by the FP64 pipe, on which the library's acos took
// half of about 60 instructions per lookup.  Here a single-precision arc cosine (on the idle FP32 pipe)
// picks the nearest of ACOS_NODES equal steps of [0, pi], and the rest is the inverse series of
// cos(theta_j + e) = c: with x = (cos theta_j - c) / sin theta_j and kappa = cot theta_j,
//   e = x - kappa/2 x^2 + (3 kappa^2 + 1)/6 x^3 - kappa (5 kappa^2 + 3)/8 x^4
//         + (35 kappa^4 + 30 kappa^2 + 3)/40 x^5 - ...
// whose next term is below 2e-17 for |x| <= pi/30000 and |kappa| <= 6; closer to the poles (9.5 degrees)
// acos itself is called.  The nodes hold the coefficients in columns and powers of cos theta_j - c, so that the
// column costs five instructions, and conversions, which share the pipe, are left out: the float cosine is
// put together from c's high word, and a table gives the column's number as a double.  20 instructions per
// lookup.  8 spheres, 288^2 pixels, 200 directions: 12.8 ms with acos, 6.57 ms with 2048 nodes of six terms
// (nine instructions), 5.54 ms with these nodes, 4.94 ms without the conversions.  The nodes' 0.8 MB are
// read by neighbouring pixels at neighbouring angles.  Blocks of 64 pixels: at 128 the last wave of that slice is a
// quarter full.
// ---------------------------------------------------------------------------
__global__ void acos_node_kernel(int thetaR, double tsc, AcosNode* __restrict__ nodes) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    double* cols = reinterpret_cast<double*>(nodes + ACOS_NODES + 1);
    for (int i = j; i < thetaR; i += gridDim.x * blockDim.x) cols[i] = i;
    if (j > ACOS_NODES) return;
    AcosNode n;
    double sn;
    sincospi((double)j / ACOS_NODES, &sn, &n.c);
    const bool pole = j == 0 || j == ACOS_NODES;
    const double k = pole ? 0.0 : n.c / sn, k2 = k * k, is = pole ? 0.0 : 1.0 / sn, is2 = is * is;
    n.t = j * (TRUE_PI / ACOS_NODES) * tsc;
    n.d1 = tsc * is;
    n.d2 = -0.5 * k * tsc * is2;
    n.d3 = (3.0 * k2 + 1.0) / 6.0 * tsc * (is2 * is);
    n.d4 = -k * (5.0 * k2 + 3.0) / 8.0 * tsc * (is2 * is2);
    nodes[j] = n;
}

constexpr int F64_BLOCK = 64;
__global__ void __launch_bounds__(F64_BLOCK) us_lut_f64_kernel(Scene sc, const Sphere* __restrict__ sph, int s0, int s1,
                                                          int accumulate, int finalize,
                                                          const double* __restrict__ waves,
                                                          const AcosNode* __restrict__ nodes,
                                                          const zd* __restrict__ ph, const Patch<double>* __restrict__ lut,
                                                          const zd* __restrict__ Uf, zd* __restrict__ U) {
    constexpr int POLE = 864;  // nodes within 9.5 degrees of a pole
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= sc.R * sc.R) return;
    double p[3];
    pixel_pos(sc, idx % sc.R, idx / sc.R, p);
    zd total = accumulate ? U[idx] : mk(0.0, 0.0);
    for (int s = s0; s < s1; s++) {
        const Sphere& S = sph[s];
        double r[3];
        double d = dist_exact(p, S.p, r);
        TableSel ts = select_table(S, d);
        int ir = (int)floor(ts.x);
        double al = ts.x - ir;
        const Patch<double>* row = lut + ts.off + (size_t)ir * S.thetaR;
        double rn[3] = {0, 0, 0}, cb = 1.0;  // d == 0: cos(theta) := 1
        if (d != 0) {
            rn[0] = r[0] / d;
            rn[1] = r[1] / d;
            rn[2] = r[2] / d;
            cb = 0.0;
        }
        const double tmax = S.thetaR - 1, tsc = tmax * (1.0 / PI_REF);
        const double* cols = reinterpret_cast<const double*>(nodes + ACOS_NODES + 1);
        zd sum = mk(0.0, 0.0);
        const zd* phs = ph + (size_t)s * sc.nk;
#pragma unroll 4
        for (int w = 0; w < sc.nk; w++) {
            const double* k = waves + 3 * w;
            const double c = fma(k[0], rn[0], fma(k[1], rn[1], fma(k[2], rn[2], cb)));
            const int hc = __double2hiint(c), mag = min(hc & 0x7fffffff, 0x47e00000) - 0x38000000;
            const float cf = __int_as_float((hc & 0x80000000) | max(mag, 0) << 3);  // c, its high word's 20 bits
            const int j = __float2int_rn(acosf(fminf(fmaxf(cf, -1.f), 1.f)) * (float)(ACOS_NODES / TRUE_PI));
            double t;
            if (j > POLE && j < ACOS_NODES - POLE) {
                const AcosNode n = nodes[j];
                const double y = n.c - c;
                t = fma(fma(fma(fma(n.d4, y, n.d3), y, n.d2), y, n.d1), y, n.t);
            } else {
                t = fmin(acos(fmin(fmax(c, -1.0), 1.0)) * tsc, tmax);
            }
            const double u = __dadd_rd(t, 6755399441055744.0);  // 1.5 2^52: the sum's low word is floor(t)
            const double be = t - cols[__double2loint(u)];
            const Patch<double>& q = row[__double2loint(u)];
            const double vr = fma(be, fma(al, q.v[6], q.v[4]), fma(al, q.v[2], q.v[0]));
            const double vi = fma(be, fma(al, q.v[7], q.v[5]), fma(al, q.v[3], q.v[1]));
            const zd pw = phs[w];
            sum = mk(fma(pw.re, vr, fma(-pw.im, vi, sum.re)), fma(pw.re, vi, fma(pw.im, vr, sum.im)));
        }
        total = total + sum;
    }
    if (finalize) {
        bool outside = true;
        for (int s = 0; s < sc.ns; s++) {
            const Sphere& S = sph[s];
            double r[3];
            if (dist_exact(p, S.p, r) < S.a) outside = false;
        }
        if (outside) total = total + Uf[idx];
    }
    U[idx] = total;
}

// Mixed path: the sums of lut_build_kernel for the tables of a sphere batch in one launch, stored as
// float2 in linear rows with the last column repeated (a lookup's right neighbour needs no clamp).
//
// The sums were bound by the FP64 pipe (2 DFMA per entry and order at 1/64 of the single-precision
// rate).  Here coefficients and Legendre values are split into two floats each, and a sum is kept as
// H + lo: H starts at the row's bias, a power of two of at least twice the sum of |coefficients|, so
// that H + c p rounds to a multiple of ulp(bias), its change (H' - H) is exact, and what the rounding
// left of the product, c p - (H' - H), comes from one fused multiply-add; lo collects those rests and
// the cross terms.  H - bias is exact, so the result carries about 46 bits relative to the bias and
// its float is the double-precision sum's but next to a rounding boundary (6 of 100 000 entries differ in
// the last bit; the tables' error against double precision is 2.6e-8 either way).  Six packed
// instructions per (entry, order).  GB300, 50 spheres x 4096 x 1024: 12.4 -> 2.2 ms with the
// coefficient rows; 120 spheres 25.6 -> 4.3 ms.
// A block makes 32 rows x 128 angles, a thread 4 rows x 4 angles (angles one warp apart: coalesced
// rows), with LBM_L orders of both factors in shared memory at a time.
constexpr int LBM_R = 32, LBM_T = 128, LBM_L = 16;

__device__ __forceinline__ unsigned long long pk2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ unsigned long long pk_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long pk_add(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long pk_sub(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__global__ void __launch_bounds__(256, 2) lut_build_mixed_kernel(const LutBuildJob* __restrict__ jobs,
                                                                 const SplitCoef* __restrict__ tab,
                                                                 const float* __restrict__ bias,
                                                                 const float2* __restrict__ P, int Pstride,
                                                                 float2* __restrict__ lin) {
    __shared__ SplitCoef sc[LBM_L][LBM_R];
    __shared__ float2 sp[LBM_L][LBM_T];
    const LutBuildJob& j = jobs[blockIdx.z];
    const int r0 = blockIdx.y * LBM_R, t0 = blockIdx.x * LBM_T;
    if (r0 >= j.rows || t0 >= j.thetaR) return;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, L = j.L, thetaR = j.thetaR, last = j.last;
    const SplitCoef* c = tab + j.tab_off;
    unsigned long long H[4][4], lo[4][4];
    float b[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        b[i] = bias[j.row_off + min(r0 + ty + 8 * i, last)];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            H[i][k] = pk2(b[i], b[i]);
            lo[i][k] = 0ull;
        }
    }
    for (int l0 = 0; l0 < L; l0 += LBM_L) {
        const int nl = min(LBM_L, L - l0);
        __syncthreads();
        for (int e = threadIdx.x; e < LBM_R * LBM_L; e += 256) {
            const int l = e % LBM_L, r = e / LBM_L;
            if (l < nl) sc[l][r] = c[(size_t)min(r0 + r, last) * L + l0 + l];
        }
        for (int e = threadIdx.x; e < LBM_T * nl; e += 256) {
            const int t = e % LBM_T, l = e / LBM_T;
            sp[l][t] = P[(size_t)(l0 + l) * Pstride + min(t0 + t, thetaR - 1)];
        }
        __syncthreads();
        for (int l = 0; l < nl; l++) {
            unsigned long long ph[4], pl[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float2 p = sp[l][tx + 32 * k];
                ph[k] = pk2(p.x, p.x);
                pl[k] = pk2(p.y, p.y);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const SplitCoef q = sc[l][ty + 8 * i];
                const unsigned long long ch = pk2(q.hr, q.hi), cl = pk2(q.lr, q.li);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const unsigned long long h = pk_fma(ch, ph[k], H[i][k]);
                    const unsigned long long rest = pk_fma(ch, ph[k], pk_sub(H[i][k], h));
                    H[i][k] = h;
                    lo[i][k] = pk_fma(cl, ph[k], pk_fma(ch, pl[k], pk_add(lo[i][k], rest)));
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = r0 + ty + 8 * i;
        if (r >= j.rows) continue;
        float2* row = lin + j.lin_off + (size_t)r * j.lin_stride;
        const unsigned long long bb = pk2(b[i], b[i]);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int t = t0 + tx + 32 * k;
            if (t >= thetaR) continue;
            const unsigned long long v = pk_add(pk_sub(H[i][k], bb), lo[i][k]);
            *reinterpret_cast<unsigned long long*>(row + t) = v;
            if (t == thetaR - 1) *reinterpret_cast<unsigned long long*>(row + thetaR) = v;
        }
    }
}

// ---------------------------------------------------------------------------
// Direct scattered field through the addition theorem of spherical harmonics.
// The per-pixel sum over waves, sum_w pw_w sum_l c_l P_l(k_w . r^), is
// sum_l c_l Q_l(r^) with Q_l(r^) = sum_w pw_w P_l(k_w . r^).  With the Schmidt
// semi-normalised associated Legendre functions S_l^m (S_l^m = sqrt(e_m (l-m)!
// / (l+m)!) P_l^m, e_0 = 1, e_m = 2), P_l(cos g) = sum_{m<=l} S_l^m(cos t1)
// S_l^m(cos t2) cos(m (f1 - f2)), so
//   Q_l(r^) = sum_m S_l^m(r_z) (cos(m f_r) C_lm + sin(m f_r) S_lm),
//   (C_lm, S_lm) = sum_w pw_w S_l^m(k_wz) (cos, sin)(m f_w)   per sphere,
// with f the azimuth about the harmonics' axis.  A (pixel, sphere) pair then costs L (L + 1) / 2
// terms instead of nk L, and the result is the same sum up to rounding.
//
// The axis is the slice's normal (ShFrame): a pixel's cosine is then h / d with the sphere's distance h
// from the plane, the same for all pixels, and where the plane goes through the sphere's centre (h = 0)
// every S_l^m is a constant, zero for odd l - m, that goes into the coefficients.
// FP64 instructions per term (the kernel's bound): the three-term recurrence of the S_l^m in monic form
// (u_l = x u_{l-1} - beta_l u_{l-2}, scale in the coefficients) 2, its cosine and sine part 2, the sum
// Q_l 4 -- 8 where summing c_l S_l^m (...) took 13 -- and 4 on half of the terms where h = 0.
// Tables are in (m, l) order: index(m, l) = m L - m (m - 1) / 2 + (l - m).
// The tables' kernels are bound by the FP64 instructions on one warp's chain (64 cycles each), so they run a warp
// per m, a thread per (wave, m) and a thread per index and sixteenth of the waves: 25 orders, 400 directions, one
// sphere 6 + 9 + 23 us, where a thread per m, per wave and per index took 64 + 128 + 103 us.
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ int sh_index(int L, int m, int l) { return m * L - m * (m - 1) / 2 + (l - m); }

// Per (m, l): a, b of S_l^m = a x S_{l-1}^m - b S_{l-2}^m for l >= m + 2 (a = (2l - 1) / sqrt(l^2 - m^2),
// b = sqrt((l-1)^2 - m^2) / sqrt(l^2 - m^2)), a = sqrt(2m + 1) for l = m + 1, and for l = m the diagonal
// factor S_m^m = a sin(t) S_{m-1}^{m-1} (a = 1 for m = 1, sqrt((2m - 1) / (2m)) above); the monic form
// S_l^m = kappa u_l, beta = b kappa_{l-2} / kappa_l; and zero = S_l^m at x = 0.
// A warp per m, a lane per l: roots and quotients side by side, the products over l (kappa, zero) as scans.
__global__ void __launch_bounds__(32) sh_recur_kernel(int L, ShRec* __restrict__ rec) {
    const int m = blockIdx.x, lane = threadIdx.x;
    const unsigned all = 0xffffffffu;
    double diag = 1;  // S_m^m at sin t = 1
    for (int i = 2 + lane; i <= m; i += 32) diag *= sqrt((2.0 * i - 1.0) / (2.0 * i));
    for (int d = 16; d >= 1; d >>= 1) diag *= __shfl_xor_sync(all, diag, d);
    const double m2 = (double)m * m;
    double kap0 = 1, z_even = diag, z_odd = 0;  // kappa of the order before the 32, and zero at the last even, odd l - m
    double a_before = 1;
    for (int l0 = m; l0 < L; l0 += 32) {
        const int l = l0 + lane, q = l - m;
        const double den = sqrt((double)l * l - m2);
        const double a = q == 0 ? 1.0 : (2.0 * l - 1.0) / den;
        const double b = q < 2 ? 0.0 : sqrt((double)(l - 1) * (l - 1) - m2) / den;
        double a1 = __shfl_up_sync(all, a, 1);
        if (lane == 0) a1 = a_before;
        double kap = a, z = q < 2 ? 1.0 : -b;
        for (int d = 1; d < 32; d <<= 1) {
            const double k2 = __shfl_up_sync(all, kap, d), z2 = __shfl_up_sync(all, z, 2 * d);
            if (lane >= d) kap *= k2;
            if (lane >= 2 * d) z *= z2;
        }
        kap *= kap0;
        z *= q & 1 ? z_odd : z_even;
        if (l < L) {
            ShRec r;
            r.a = q == 0 ? (m < 2 ? 1.0 : sqrt((2.0 * m - 1.0) / (2.0 * m))) : a;
            r.b = b;
            r.beta = q < 2 ? 0.0 : b / (a * a1);
            r.kappa = kap;
            r.zero = z;
            rec[sh_index(L, m, l)] = r;
        }
        kap0 = __shfl_sync(all, kap, 31);
        a_before = __shfl_sync(all, a, 31);
        z_even = __shfl_sync(all, z, 30);
        z_odd = 0;
    }
}

__device__ __forceinline__ double dot3(const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

// Per wave: tab[w][index(m, l)] = S_l^m(k_n) (cos, sin)(m f_k), k_n the component along the normal: a thread per
// (wave, m), from S_m^m (cos, sin)(m f) = S_m^m(0) (k_x + i k_y)^m.  The ns last values of m: the phases
// pw[s][w] as phase_kernel's, in double precision.
__global__ void __launch_bounds__(32) sh_wave_kernel(Scene sc, ShFrame fr, const Sphere* __restrict__ sph, int L,
                                                     const double* __restrict__ waves, const ShRec* __restrict__ rec,
                                                     double2* __restrict__ tab, zd* __restrict__ pw) {
    const int m = blockIdx.x % (L + sc.ns), w = blockIdx.x / (L + sc.ns) * 32 + threadIdx.x;
    if (w >= sc.nk) return;
    const double* k = waves + 3 * w;
    if (m >= L) {
        const Sphere& S = sph[m - L];
        const double arg =
            sc.kmag * (k[0] * (S.p[0] - sc.focus[0]) + k[1] * (S.p[1] - sc.focus[1]) + k[2] * (S.p[2] - sc.focus[2]));
        double sn, cs;
        sincos(arg, &sn, &cs);
        pw[(size_t)(m - L) * sc.nk + w] = mk(sc.wave_amp * cs, sc.wave_amp * sn);
        return;
    }
    const double kz = dot3(k, fr.e3);
    zd b = mk(dot3(k, fr.e1), dot3(k, fr.e2)), e = mk(1.0, 0.0);
    for (int i = m; i; i >>= 1) {
        if (i & 1) e = mk(e.re * b.re - e.im * b.im, e.re * b.im + e.im * b.re);
        b = mk(b.re * b.re - b.im * b.im, 2.0 * b.re * b.im);
    }
    const ShRec* r = rec + sh_index(L, m, m);
    e = e * r[0].zero;
    double2* out = tab + (size_t)w * (L * (L + 1) / 2) + sh_index(L, m, m);
    double p2 = 0, p1 = 1;
    out[0] = make_double2(e.re, e.im);
#pragma unroll 4
    for (int q = 1; q < L - m; q++) {  // b is 0 for q = 1
        const double v = fma(r[q].a * kz, p1, -r[q].b * p2);
        p2 = p1;
        p1 = v;
        out[q] = make_double2(v * e.re, v * e.im);
    }
}

// Whether the slice's plane goes through the sphere's centre, to rounding.
__device__ __forceinline__ bool sh_in_plane(const Scene& sc, const ShFrame& fr, const Sphere& S, double& h) {
    const double r[3] = {sc.A[0] - S.p[0], sc.A[1] - S.p[1], sc.A[2] - S.p[2]};
    h = dot3(r, fr.e3);
    return fabs(h) <= 4e-16 * (fabs(r[0]) + fabs(r[1]) + fabs(r[2]));
}

// Per sphere s and table index: coef[s][0][index] = (C, S) = B_l scale sum_w pw[s][w] tab[w][index], with the scale
// kappa, or S_l^m(0) for a sphere centred in the plane; coef[s][1] with A_l for the pixels inside the sphere.
// A block takes 8 indices, thread t every 16th wave of index t mod 8.
constexpr int SC_I = 8, SC_W = 16;
__global__ void __launch_bounds__(SC_I* SC_W) sh_coef_kernel(Scene sc, ShFrame fr, const Sphere* __restrict__ sph, int L,
                                                             const ShRec* __restrict__ rec,
                                                             const double2* __restrict__ tab,
                                                             const zd* __restrict__ pw, const zd* __restrict__ A,
                                                             const zd* __restrict__ B, zd* __restrict__ coef) {
    __shared__ zd s_c[SC_W][SC_I], s_s[SC_W][SC_I];
    const int s = blockIdx.y, nlm = L * (L + 1) / 2;
    const int ti = threadIdx.x % SC_I, tw = threadIdx.x / SC_I, i = blockIdx.x * SC_I + ti;
    zd ac = mk(0.0, 0.0), as = mk(0.0, 0.0);
    if (i < nlm) {
        const zd* p = pw + (size_t)s * sc.nk;
#pragma unroll 4
        for (int w = tw; w < sc.nk; w += SC_W) {
            const double2 v = tab[(size_t)w * nlm + i];
            const zd f = p[w];
            ac = mk(fma(f.re, v.x, ac.re), fma(f.im, v.x, ac.im));
            as = mk(fma(f.re, v.y, as.re), fma(f.im, v.y, as.im));
        }
    }
    s_c[tw][ti] = ac;
    s_s[tw][ti] = as;
    __syncthreads();
    if (tw != 0 || i >= nlm) return;
    for (int q = 1; q < SC_W; q++) {
        ac = ac + s_c[q][ti];
        as = as + s_s[q][ti];
    }
    double h;
    const double scale = sh_in_plane(sc, fr, sph[s], h) ? rec[i].zero : rec[i].kappa;
    int m = 0, k = i;  // i = index(m, l)
    while (k >= L - m) k -= L - m++;
    const int l = m + k;
    const bool have = l <= sph[s].Nl;
    const zd b = have ? B[sph[s].coef_off + l] : mk(0.0, 0.0), a = have ? A[sph[s].coef_off + l] : b;
    zd* o = coef + (size_t)4 * s * nlm + 2 * i;
    o[0] = (ac * scale) * b;
    o[1] = (as * scale) * b;
    o[2 * nlm] = (ac * scale) * a;
    o[2 * nlm + 1] = (as * scale) * a;
}

// The radial functions of one (pixel, sphere) pair, order after order:
//   outside (d > a):  j_l + i y_l (k d)   with the reference clamps (spherical_bessel.h:102-141)
//   inside  (d <= a): j_l(k n d)          (1 for l = 0 and else 0 when Re(k n d) < 1e-6)
// (--recursive; nfScalarUs.cu:17-95, 201-245, 333-491); their factors B_l and A_l are in the coefficients.
// They depend on (pixel, sphere) only; the reference re-runs them for every wave (nfScalarUs.cu:69-93).
// One reciprocal serves all orders, and outside the clamps compare high words, off the FP64 pipe: ten
// FP64 instructions per order with the sum over l, where twenty-one took 4.72 ms of a 1280^2 slice with one sphere
// (3.63 ms now).
struct ShRadial {
    bool inside, centre;
    int xi;  // outside: l > x when l > xi
    double x, inv, odd;
    zd z, zinv;
    zd p0, p1;  // outside: (j, y) of the last two orders; inside: j

    __device__ __forceinline__ void start(const Scene& sc, const Sphere& S, double d) {
        inside = d <= S.a;
        centre = false;
        if (inside) {
            z = mk(sc.kmag * d * S.n_re, sc.kmag * d * S.n_im);
            centre = z.re < EPS_FLOAT;
            if (centre) return;
            zinv = mk(1.0, 0.0) / z;
            const zd j0 = zsin(z) / z;
            p0 = j0;
            p1 = j0 / z - zcos(z) / z;
        } else {
            x = sc.kmag * d;
            xi = x < (double)MAX_ORDER ? (int)x : MAX_ORDER;
            inv = 1.0 / x;
            odd = 1.0;
            double sn, cs;
            sincos(x, &sn, &cs);
            const double s1 = quot(sn, x, inv), c1 = quot(cs, x, inv);
            p0 = mk(s1, -c1);
            p1 = mk(quot(s1, x, inv) - c1, quot(-c1, x, inv) - s1);
        }
    }
    // The function of order l = 0, 1, 2, ... in turn
    __device__ __forceinline__ zd next(int l) {
        if (inside) {
            if (centre) return mk(l == 0 ? 1.0 : 0.0, 0.0);
            if (l < 2) return l == 0 ? p0 : p1;
            const zd w = (2.0 * l - 1.0) * zinv;
            zd b = mk(fma(w.re, p1.re, fma(-w.im, p1.im, -p0.re)), fma(w.re, p1.im, fma(w.im, p1.re, -p0.im)));
            if (l > z.re && (b.re < CONV_MIN || b.re > CONV_MAX)) b = mk(0.0, 0.0);
            p0 = p1;
            p1 = b;
            return b;
        }
        if (l < 2) return l == 0 ? p0 : p1;
        odd += 2.0;
        const double w = quot(odd, x, inv);
        const bool beyond = l > xi;
        const double j = clamp_j(fma(w, p1.re, -p0.re), beyond);
        double y = fma(w, p1.im, -p0.im);
        constexpr unsigned FLOOR = 0xc6c8a6e3u;  // Y_FLOOR's high word
        const int hy = __double2hiint(y);
        if ((beyond && hy > 0) || ((unsigned)hy >= FLOOR && ((unsigned)hy > FLOOR || y < Y_FLOOR))) {
            y = 0;
            p1.im = 0;
        }
        p0 = p1;
        p1 = mk(j, y);
        return p1;
    }
};

// Per pixel: U = sum_s sum_l c_l(r) Q_l(r^) (+ Uf outside every sphere).  All in double precision, stored as T.
constexpr int SH_BLOCK = 64;
template <class T>
__global__ void __launch_bounds__(SH_BLOCK) us_sh_kernel(Scene sc, ShFrame fr, const Sphere* __restrict__ sph, int L,
                                                         const ShRec* __restrict__ rec, const zd* __restrict__ coef,
                                                         const cpx<T>* __restrict__ Uf, cpx<T>* __restrict__ U) {
    extern __shared__ unsigned char smem_raw[];
    zd* col = reinterpret_cast<zd*>(smem_raw) + threadIdx.x;  // the thread's L values, SH_BLOCK apart
    const int nlm = L * (L + 1) / 2;
    int idx = blockIdx.x * SH_BLOCK + threadIdx.x;
    const bool valid = idx < sc.R * sc.R;
    if (!valid) idx = sc.R * sc.R - 1;
    double p[3];
    pixel_pos(sc, idx % sc.R, idx / sc.R, p);
    zd tot = mk(0.0, 0.0), cmp = mk(0.0, 0.0);
    bool outside = true;
    for (int s = 0; s < sc.ns; s++) {
        const Sphere& S = sph[s];
        double r[3], h;
        const double d = dist_exact(p, S.p, r);
        if (d < S.a) outside = false;
        const int Ls = S.Nl + 1;
        const bool in_plane = sh_in_plane(sc, fr, S, h);
        const double r1 = dot3(r, fr.e1), r2 = dot3(r, fr.e2), rho = sqrt(r1 * r1 + r2 * r2);
        const double irho = 1.0 / rho;
        const double cf = rho > 0 ? quot(r1, rho, irho) : 1.0, sf = rho > 0 ? quot(r2, rho, irho) : 0.0;
        ShRadial rad;
        rad.start(sc, S, d);
        const zd* cs_ = coef + ((size_t)2 * s + (rad.inside ? 1 : 0)) * nlm * 2;
        zd acc = mk(0.0, 0.0);
        auto add = [&](zd f, zd q) {
            acc = mk(fma(f.re, q.re, fma(-f.im, q.im, acc.re)), fma(f.re, q.im, fma(f.im, q.re, acc.im)));
        };
        if (in_plane) {
            double cm = 1, sm = 0;
            for (int m = 0; m < Ls; m++) {  // cos(m f), sin(m f)
                col[m * SH_BLOCK] = mk(cm, sm);
                const double c2 = cm * cf - sm * sf;
                sm = sm * cf + cm * sf;
                cm = c2;
            }
            for (int l = 0; l < Ls; l++) {
                zd q = mk(0.0, 0.0);
#pragma unroll 4
                for (int m = l & 1; m <= l; m += 2) {
                    const int k = sh_index(L, m, l);
                    const zd C = cs_[2 * k], Sn = cs_[2 * k + 1], e = col[m * SH_BLOCK];
                    q = mk(fma(e.re, C.re, fma(e.im, Sn.re, q.re)), fma(e.re, C.im, fma(e.im, Sn.im, q.im)));
                }
                add(rad.next(l), q);
            }
        } else {
            const double x = d != 0 ? h / d : 0.0, st = d != 0 ? rho / d : 0.0;
            for (int l = 0; l < Ls; l++) col[l * SH_BLOCK] = mk(0.0, 0.0);
            double cm = 1, sm = 0, smm = 1;
            for (int m = 0; m < Ls; m++) {
                if (m > 0) {
                    smm *= rec[sh_index(L, m, m)].a * st;
                    const double c2 = cm * cf - sm * sf;
                    sm = sm * cf + cm * sf;
                    cm = c2;
                }
                const double c = smm * cm, sn = smm * sm;
                double u2 = 0, u1 = 1;
                const int k0 = sh_index(L, m, m);
#pragma unroll 4
                for (int l = m; l < Ls; l++) {
                    const int k = k0 + l - m;
                    if (l > m) {  // beta is 0 for l = m + 1
                        const double u = fma(x, u1, -rec[k].beta * u2);
                        u2 = u1;
                        u1 = u;
                    }
                    const zd C = cs_[2 * k], Sn = cs_[2 * k + 1];
                    const double wc = c * u1, ws = sn * u1;
                    zd& q = col[l * SH_BLOCK];
                    q = mk(fma(wc, C.re, fma(ws, Sn.re, q.re)), fma(wc, C.im, fma(ws, Sn.im, q.im)));
                }
            }
            for (int l = 0; l < Ls; l++) add(rad.next(l), col[l * SH_BLOCK]);
        }
        // Kahan over spheres
        const zd y = acc - cmp;
        const zd t = tot + y;
        cmp = (t - tot) - y;
        tot = t;
    }
    if (!valid) return;
    if (outside) tot = tot + (mk((double)Uf[idx].re, (double)Uf[idx].im) - cmp);
    U[idx] = mk((T)tot.re, (T)tot.im);
}

// Vector stub of the reference: no scattered field, U = Uf outside every sphere.
template <class T>
__global__ void sum_only_kernel(Scene sc, const Sphere* __restrict__ sph, const cpx<T>* __restrict__ Uf,
                                cpx<T>* __restrict__ U) {
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= sc.R * sc.R) return;
    double p[3];
    pixel_pos(sc, idx % sc.R, idx / sc.R, p);
    bool outside = true;
    for (int s = 0; s < sc.ns; s++) {
        const Sphere& S = sph[s];
        double r[3];
        if (dist_exact(p, S.p, r) < S.a) outside = false;
    }
    U[idx] = outside ? Uf[idx] : mk((T)0, (T)0);
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
static inline unsigned blocks_for(long long n, int b) { return (unsigned)((n + b - 1) / b); }

template <class T>
void launch_uf(const Scene& sc, const double* tab, const UfOrder* w, cpx<T>* Uf, cudaStream_t st) {
    long long n = (long long)sc.R * sc.R;
    uf_kernel<T><<<blocks_for(n, 128), 128, 0, st>>>(sc, tab, w, Uf);
}

void launch_uf_table(const Scene& sc, double* tab, double* scratch, cudaStream_t st) {
    uf_table_kernel<<<blocks_for(sc.uf_dR, 128), 128, 0, st>>>(sc, tab, scratch);
}

void launch_mie(const Sphere* sph, int ns, double k, zd* A, zd* B, cudaStream_t st) {
    mie_kernel<<<ns, MIE_NT, 0, st>>>(sph, k, A, B);
}

void launch_coef_rows_batch(const Sphere* sph, int s0, int n, const long long* starts, long long total_rows, double k,
                            const zd* A, const zd* B, zd* tab, double* scratch, float* bias, cudaStream_t st) {
    coef_rows_batch_kernel<<<blocks_for(total_rows, 128), 128, 0, st>>>(sph, s0, n, starts, k, A, B, tab, scratch, bias);
}

void launch_legendre_split(int thetaR, int Lmax, int stride, float2* P, cudaStream_t st) {
    legendre_split_kernel<<<blocks_for(thetaR, 64), 64, 0, st>>>(thetaR, Lmax, stride, P);
}

void launch_legendre_table(int thetaR, int Lmax, double* P, cudaStream_t st) {
    legendre_table_kernel<<<blocks_for(thetaR, 128), 128, 0, st>>>(thetaR, Lmax, P);
}

void launch_lut_build(const LutBuildJob* jobs, int njobs, int max_rows, int max_theta, const zd* tab, const double* P,
                      int Pstride, Patch<double>* out, cudaStream_t st) {
    dim3 grid(blocks_for(max_theta, LB_TT), blocks_for(max_rows, LB_TR), (unsigned)njobs);
    lut_build_kernel<<<grid, 256, 0, st>>>(jobs, tab, P, Pstride, out);
}

void launch_lut_build_plain(const LutBuildJob* jobs, int njobs, int max_rows, int max_theta, const zd* tab,
                            const double* P, int Pstride, float2* lin, cudaStream_t st) {
    dim3 grid(blocks_for(max_theta, 32), blocks_for(max_rows, 8), (unsigned)njobs);
    lut_build_plain_kernel<<<grid, 256, 0, st>>>(jobs, tab, P, Pstride, lin);
}

template <class T>
void launch_phase(const Scene& sc, const Sphere* sph, const double* waves, cpx<T>* ph, float4* kw4, cudaStream_t st) {
    long long n = std::max<long long>((long long)sc.ns * sc.nk, sc.nk);
    phase_kernel<T><<<blocks_for(n, 128), 128, 0, st>>>(sc, sph, waves, ph, kw4);
}

void launch_acos_nodes(int thetaR, AcosNode* nodes, cudaStream_t st) {
    acos_node_kernel<<<blocks_for(ACOS_NODES + 1, 64), 64, 0, st>>>(thetaR, (thetaR - 1) * (1.0 / PI_REF), nodes);
}

void launch_us_lut_f64(const Scene& sc, const Sphere* sph, int s0, int s1, int accumulate, int finalize,
                       const double* waves, const AcosNode* nodes, const zd* ph, const Patch<double>* lut, const zd* Uf,
                       zd* U, cudaStream_t st) {
    long long n = (long long)sc.R * sc.R;
    us_lut_f64_kernel<<<blocks_for(n, F64_BLOCK), F64_BLOCK, 0, st>>>(sc, sph, s0, s1, accumulate, finalize, waves, nodes, ph, lut,
                                                           Uf, U);
}

void launch_lut_build_mixed(const LutBuildJob* jobs, int njobs, int max_rows, int max_theta, const zd* tab,
                            const float* bias, const float2* P, int Pstride, float2* lin, cudaStream_t st) {
    if (njobs < 1 || max_rows < 1) return;
    dim3 grid(blocks_for(max_theta, LBM_T), blocks_for(max_rows, LBM_R), (unsigned)njobs);
    lut_build_mixed_kernel<<<grid, 256, 0, st>>>(jobs, reinterpret_cast<const SplitCoef*>(tab), bias, P, Pstride, lin);
}

// Orthonormal frame of the slice: the u axis and the normal; of a slice that is a line, the line
// and an axis across it (of a point, the coordinate axes).
static ShFrame sh_frame(const Scene& sc) {
    auto len = [](const double* a) { return std::sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]); };
    auto cross = [](const double* a, const double* b, double* c) {
        for (int i = 0; i < 3; i++) c[i] = a[(i + 1) % 3] * b[(i + 2) % 3] - a[(i + 2) % 3] * b[(i + 1) % 3];
    };
    ShFrame f{{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
    const double* X = len(sc.X) > 0 ? sc.X : sc.Y;
    const double lx = len(X);
    if (!(lx > 0)) return f;
    for (int i = 0; i < 3; i++) f.e1[i] = X[i] / lx;
    cross(sc.X, sc.Y, f.e3);
    if (!(len(f.e3) > 1e-14 * lx * lx)) {
        int k = 0;  // the coordinate axis farthest from the line
        for (int i = 1; i < 3; i++)
            if (std::fabs(f.e1[i]) < std::fabs(f.e1[k])) k = i;
        const double a[3] = {double(k == 0), double(k == 1), double(k == 2)};
        cross(f.e1, a, f.e3);
    }
    const double ln = len(f.e3);
    for (int i = 0; i < 3; i++) f.e3[i] /= ln;
    cross(f.e3, f.e1, f.e2);
    return f;
}

void launch_sh_tables(const Scene& sc, const Sphere* sph, int L, const double* waves, ShRec* rec, double2* tab,
                      const zd* A, const zd* B, zd* coef, cudaStream_t st) {
    const ShFrame fr = sh_frame(sc);
    const int nlm = L * (L + 1) / 2;
    zd* pw = reinterpret_cast<zd*>(tab + (size_t)sc.nk * nlm);
    sh_recur_kernel<<<L, 32, 0, st>>>(L, rec);
    sh_wave_kernel<<<blocks_for(sc.nk, 32) * (unsigned)(L + sc.ns), 32, 0, st>>>(sc, fr, sph, L, waves, rec, tab, pw);
    sh_coef_kernel<<<dim3(blocks_for(nlm, SC_I), sc.ns), SC_I * SC_W, 0, st>>>(sc, fr, sph, L, rec, tab, pw, A, B, coef);
}

template <class T>
void launch_us_sh(const Scene& sc, const Sphere* sph, int L, const ShRec* rec, const zd* coef, const cpx<T>* Uf, cpx<T>* U, cudaStream_t st) {
    const size_t smem = (size_t)L * SH_BLOCK * sizeof(zd);
    // the kernel's attribute is one for all threads of the process: the largest size on every call, so that another
    // context cannot lower it before this launch
    cudaFuncSetAttribute(us_sh_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_OPTIN);
    const long long n = (long long)sc.R * sc.R;
    us_sh_kernel<T><<<blocks_for(n, SH_BLOCK), SH_BLOCK, smem, st>>>(sc, sh_frame(sc), sph, L, rec, coef, Uf, U);
}

template <class T>
void launch_sum_only(const Scene& sc, const Sphere* sph, const cpx<T>* Uf, cpx<T>* U, cudaStream_t st) {
    long long n = (long long)sc.R * sc.R;
    sum_only_kernel<T><<<blocks_for(n, 128), 128, 0, st>>>(sc, sph, Uf, U);
}

// ---------------------------------------------------------------------------
// Near-field rotation (gpuInterpolateU / gpuInterpolateUf, nfInterpolate.cu:13-58):
// dst(iu, iv) = src sampled at the pixel rotated by an angle about the slice
// centre, bilinear, zero outside the slice (border addressing).  The centre is
// (int)(R/2) for U and R/2 for Uf, as in the reference; coordinates are formed
// in single precision like the reference's (cosine and sine of the angle come
// from the host rounded to float; every operation is rounded on its own, no
// fused multiply-add), the weights are exact.
// ---------------------------------------------------------------------------
template <class T>
__global__ void rotate_fields_kernel(int R, float c, float s, const cpx<T>* __restrict__ src,
                                     cpx<T>* __restrict__ dst) {
    const int iu = blockIdx.x * blockDim.x + threadIdx.x, iv = blockIdx.y;
    const int b = blockIdx.z;  // 0: U, 1: Uf
    if (iu >= R) return;
    const float uc = b == 0 ? (float)(int)(R / 2.0) : (float)(R / 2.0);
    const float du = __fsub_rn((float)iu, uc), dv = __fsub_rn((float)iv, uc);
    const float nx = __fsub_rn(__fadd_rn(uc, __fmul_rn(du, c)), __fmul_rn(dv, s));
    const float ny = __fadd_rn(__fadd_rn(uc, __fmul_rn(du, s)), __fmul_rn(dv, c));
    const cpx<T>* f = src + (size_t)b * R * R;
    const float fx = floorf(nx), fy = floorf(ny);
    const int i0 = (int)fx, j0 = (int)fy;
    const T a = (T)(nx - fx), e = (T)(ny - fy);
    auto at = [&](int i, int j) -> cpx<T> {
        return (i >= 0 && i < R && j >= 0 && j < R) ? f[(size_t)j * R + i] : mk((T)0, (T)0);
    };
    const cpx<T> v00 = at(i0, j0), v01 = at(i0 + 1, j0), v10 = at(i0, j0 + 1), v11 = at(i0 + 1, j0 + 1);
    const T w00 = (1 - a) * (1 - e), w01 = a * (1 - e), w10 = (1 - a) * e, w11 = a * e;
    dst[(size_t)b * R * R + (size_t)iv * R + iu] =
        mk(w00 * v00.re + w01 * v01.re + w10 * v10.re + w11 * v11.re,
           w00 * v00.im + w01 * v01.im + w10 * v10.im + w11 * v11.im);
}

template <class T>
void launch_rotate_fields(int R, float c, float s, const cpx<T>* src, cpx<T>* dst, cudaStream_t st) {
    dim3 grid(blocks_for(R, 128), R, 2);
    rotate_fields_kernel<T><<<grid, 128, 0, st>>>(R, c, s, src, dst);
}

// Loads every kernel of this file (cudaFuncGetAttributes), see preload_kernels.
template <class T>
static void preload_nearfield_t() {
    cudaFuncAttributes a;
    cudaFuncGetAttributes(&a, uf_kernel<T>);
    cudaFuncGetAttributes(&a, phase_kernel<T>);
    cudaFuncGetAttributes(&a, us_sh_kernel<T>);
    cudaFuncGetAttributes(&a, sum_only_kernel<T>);
    cudaFuncGetAttributes(&a, rotate_fields_kernel<T>);
}
void preload_nearfield_kernels() {
    preload_nearfield_t<float>();
    preload_nearfield_t<double>();
    cudaFuncAttributes a;
    cudaFuncGetAttributes(&a, uf_table_kernel);
    cudaFuncGetAttributes(&a, mie_kernel);
    cudaFuncGetAttributes(&a, coef_rows_batch_kernel);
    cudaFuncGetAttributes(&a, legendre_table_kernel);
    cudaFuncGetAttributes(&a, legendre_split_kernel);
    cudaFuncGetAttributes(&a, acos_node_kernel);
    cudaFuncGetAttributes(&a, us_lut_f64_kernel);
    cudaFuncGetAttributes(&a, lut_build_kernel);
    cudaFuncGetAttributes(&a, lut_build_mixed_kernel);
    cudaFuncGetAttributes(&a, lut_build_plain_kernel);
    cudaFuncGetAttributes(&a, sh_recur_kernel);
    cudaFuncGetAttributes(&a, sh_wave_kernel);
    cudaFuncGetAttributes(&a, sh_coef_kernel);
}

#define BS_INST(T)                                                                                              \
    template void launch_rotate_fields<T>(int, float, float, const cpx<T>*, cpx<T>*, cudaStream_t);             \
    template void launch_uf<T>(const Scene&, const double*, const UfOrder*, cpx<T>*, cudaStream_t);             \
    template void launch_phase<T>(const Scene&, const Sphere*, const double*, cpx<T>*, float4*, cudaStream_t);  \
    template void launch_us_sh<T>(const Scene&, const Sphere*, int, const ShRec*,         \
                                  const zd*, const cpx<T>*, cpx<T>*, cudaStream_t);                           \
    template void launch_sum_only<T>(const Scene&, const Sphere*, const cpx<T>*, cpx<T>*, cudaStream_t);
BS_INST(float)
BS_INST(double)

}  // namespace bs
