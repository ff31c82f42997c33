// bs_mie.cuh -- Mie coefficients of one sphere by one thread block (sphere::calcCoeff,
// sphere.cpp:21-97), shared by the context path and the allocation-free entry point.
#pragma once

#include "bs_math.cuh"

namespace bs {

// What bounds it is latency: a sphere's coefficients need three recurrences of 50 to 700 steps (j of
// k a and of k n a downwards, y of k a upwards), each a serial chain.  One thread per sphere ran them
// one after the other with a complex division and a hypot per step: 0.45 ms for two spheres, 1.1 ms
// for 200.  Here the step factors (2l + 1) / z are divided out beforehand by all threads, each chain
// runs on a warp of its own at one or two fused multiply-adds per step, the trigonometric start
// values and the order cut-offs on two more warps, and everything per order (derivatives,
// coefficients) in parallel.  All in shared memory.  A warp's FP64 instruction takes 64 cycles of its
// quarter of the SM's pipe whatever its lanes do, so a chain's time is its count of them: the parts of the
// complex recurrence run on two lanes, and the rescaling tests look at high words (one sphere of 24
// orders: 59 us with both parts on one lane and comparisons in FP64, 38 us now).
constexpr int MIE_NT = 160;
constexpr int MIE_N = MAX_ORDER + 1;  // orders 0 .. MAX_ORDER
constexpr int MIE_W = 768;            // step factors kept; beyond (large |n| k a) they are divided per step

struct MieShared {
    double w1[MIE_W];
    zd w2[MIE_W];
    double j[MIE_N], y[MIE_N];
    zd jn[MIE_N];
    short sj[MIE_N], sn[MIE_N];  // rescalings done when j[l], jn[l] were stored
    int tj, tn;                  // and in all
    double j0, j1;
    zd n0, n1;                   // j_0, j_1 of k n a
    int Nj, Nn;                  // orders kept
};

// 1e-250^d
__device__ __forceinline__ double mie_scale(int d) { return d == 0 ? 1.0 : (d == 1 ? 1e-250 : 0.0); }

// A_l, B_l for l = 0 .. N (N <= MAX_ORDER); called by all MIE_NT threads of a block.
__device__ inline void mie_block(MieShared& sm, int N, double a, zd n, double k, zd* __restrict__ A, zd* __restrict__ B) {
    const int tid = threadIdx.x;
    const double ka = k * a, cs = sqrt(PI_BES / TRUE_PI);
    const zd kna = (n * k) * a;
    const double az = fabs(ka), anz = zabs(kna);
    const int M1 = miller_start(N, az), M2 = miller_start(N, anz, kna.im);
    for (int l = tid; l < min(max(M1, M2) + 1, MIE_W); l += MIE_NT) {
        sm.w1[l] = (2.0 * l + 1.0) / ka;
        sm.w2[l] = mk(2.0 * l + 1.0, 0.0) / kna;
    }
    __syncthreads();
    if (tid == 0) {  // j of k a, Miller's downward recurrence
        double fp = 0.0, fc = 1e-300;
        int s = 0;
#pragma unroll 4
        for (int l = M1; l >= 1; l--) {
            const double fm = fma(l < MIE_W ? sm.w1[l] : (2.0 * l + 1.0) / ka, fc, -fp);
            fp = fc;
            fc = fm;
            if (l - 1 <= N) {
                sm.j[l - 1] = fm;
                sm.sj[l - 1] = (short)s;
            }
            if (beyond_2_830(fc)) {
                fc *= 1e-250;
                fp *= 1e-250;
                s++;
            }
        }
        sm.tj = s;
    } else if (tid == 32 || tid == 33) {  // j of k n a, one part on each lane
        const int im = tid & 1;
        double fp = 0.0, fc = im ? 0.0 : 1e-300;
        int s = 0;
#pragma unroll 4
        for (int l = M2; l >= 1; l--) {
            const zd w = l < MIE_W ? sm.w2[l] : mk(2.0 * l + 1.0, 0.0) / kna;
            const double other = __shfl_xor_sync(3u, fc, 1);
            const double fm = fma(w.re, fc, fma(im ? w.im : -w.im, other, -fp));
            fp = fc;
            fc = fm;
            if (l - 1 <= N) {
                reinterpret_cast<double*>(&sm.jn[l - 1])[im] = fm;
                sm.sn[l - 1] = (short)s;
            }
            if (__any_sync(3u, beyond_2_830(fc))) {
                fc *= 1e-250;
                fp *= 1e-250;
                s++;
            }
        }
        sm.tn = s;
    } else if (tid == 64) {  // y of k a upwards, with the reference's y_0 slip above 12 (cbessjy.cpp:541)
        double sn, c;
        sincos(ka, &sn, &c);
        const double j0 = sn / ka;
        sm.j0 = j0;
        sm.j1 = sn / (ka * ka) - c / ka;
        double ya = -c / ka, yb = -c / (ka * ka) - sn / ka;
        if (az > 12.0) ya += j0;
        sm.y[0] = ya;
        if (N >= 1) sm.y[1] = yb;
#pragma unroll 4
        for (int l = 2; l <= N; l++) {
            const double t = fma(sm.w1[l - 1], yb, -ya);
            ya = yb;
            yb = t;
            sm.y[l] = t;
        }
    } else if (tid == 96) {
        const zd s = zsin(kna), c = zcos(kna);
        sm.n0 = s / kna;
        sm.n1 = s / (kna * kna) - c / kna;
    } else if (tid == 128 || tid == 129) {
        const double z = tid == 128 ? az : anz;
        const int Nv = N >= 2 && N > (int)(0.25 * z) ? min(N, orders_kept(N, z)) : N;
        if (tid == 128) sm.Nj = Nv;
        else sm.Nn = Nv;
    }
    __syncthreads();
    const int i1 = N >= 1 ? 1 : 0;
    const double sj = fabs(sm.j0) >= fabs(sm.j1) ? sm.j0 / (sm.j[0] * mie_scale(sm.tj - sm.sj[0]))
                                                  : sm.j1 / (sm.j[i1] * mie_scale(sm.tj - sm.sj[i1]));
    const zd sn = zabs(sm.n0) >= zabs(sm.n1) ? sm.n0 / (sm.jn[0] * mie_scale(sm.tn - sm.sn[0]))
                                             : sm.n1 / (sm.jn[i1] * mie_scale(sm.tn - sm.sn[i1]));
    const int Nj = sm.Nj, Nn = sm.Nn;
    __syncthreads();
    for (int l = tid; l <= N; l += MIE_NT) {
        sm.j[l] = l > Nj ? 0.0 : sm.j[l] * mie_scale(sm.tj - sm.sj[l]) * sj * cs;
        sm.y[l] = l > Nj ? 0.0 : sm.y[l] * cs;
        sm.jn[l] = l > Nn ? mk(0.0, 0.0) : (sm.jn[l] * mie_scale(sm.tn - sm.sn[l])) * sn * cs;
    }
    __syncthreads();
    for (int l = tid; l <= N; l += MIE_NT) {
        // j_0' = -j_1, j_l' = j_{l-1} - (l+1)/z j_l (cbessjy.cpp:590-593 and 726-733)
        const double j = sm.j[l], y = sm.y[l], p1 = l + 1.0;
        const zd jn = sm.jn[l];
        double jp, yp;
        zd jnp;
        if (l > 0) {
            jp = sm.j[l - 1] - p1 * j / ka;
            yp = sm.y[l - 1] - p1 * y / ka;
            jnp = sm.jn[l - 1] - (p1 * jn) / kna;
        } else if (N >= 1) {
            jp = -sm.j[1];
            yp = -sm.y[1];
            jnp = zd{0, 0} - sm.jn[1];
        } else {
            const double c = cos(ka), s = sin(ka);
            jp = -sm.j1 * cs;
            yp = (c / (ka * ka) + s / ka) * cs;
            jnp = zd{0, 0} - sm.n1 * cs;
        }
        const zd h = mk(j, y), hp = mk(jp, yp);  // j + i y and its derivative
        const zd an = j * hp - jp * h;
        const zd bn = jn * hp - (h * jnp) * n;
        const zd cn = (j * jnp) * n - jn * jp;
        const zd f = mk(2.0 * l + 1.0, 0.0) * ipow(l);
        A[l] = f * (an / bn);
        B[l] = f * (cn / bn);
    }
}

}  // namespace bs
