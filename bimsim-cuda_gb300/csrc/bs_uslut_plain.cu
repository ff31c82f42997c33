// bs_uslut_plain.cu -- mixed-precision scattered field of slices with few spheres or few directions
// (lut_plain, lut_few): one thread per pixel, the directions in their chunks' order.
#include <cuda_runtime.h>

#include "bs_kernels.h"
#include "bs_lut.cuh"

namespace bs {

// Per-(pixel, sphere) geometry in double, per-wave work in float, per-chunk partial sums combined with Kahan
// compensation.  The absorbance of a slice with few spheres is the small difference of two float images, so that
// its last four digits hang on the order in which a pixel's terms are summed: this kernel keeps that order, where
// the sorted kernel of bs_uslut.cu sums over its lanes (lut_plain has the figures).
//
// A block owns a 16 x 16 pixel tile, one or two pixels per thread.  The waves arrive
// grouped by direction into compact chunks of `chunk` waves (64, 32 or 16) and
// are processed chunk by chunk; the host gives each chunk a bounding cone
// (axis c_k, half-angle beta_k).  For a
// tile whose pixels all lie outside the sphere and see it within an angle
// gamma of the tile-centre direction r_c, every lookup angle of a chunk lies
// in angle(c_k, r_c) +- (beta_k + gamma) (triangle inequality on the sphere of
// directions).  The table values of the tile's rows times that angular window
// (float2, at most lut_plain_entries(chunk) of them) are copied to shared memory once per
// chunk and the bilinear cells are read from there.  Chunks whose window does
// not fit, and tiles touching or containing the sphere, read the cells from the
// table itself.  Both interpolate with the same single-precision
// formula, so they give the same bits; edge cells clamp like the reference's
// texture fetch.
constexpr int UP_TILE = 256;  // 16 x 16 pixel tile
// Pixels per thread of the staged kernel: with 64-wave chunks two (128 threads at 128 registers, 4 blocks per SM;
// 730 ms against 755 ms for one on a 3072^2 slice of 50 spheres and 1000 directions), with 16- and 32-wave chunks,
// whose barriers and window copies weigh more, one on 8 warps (307 against 366 ms with 16-wave chunks on a 1536^2
// slice).
constexpr int UP_TWO_PIXEL_MIN_CHUNK = 64;
constexpr int UP_SMEM = lut_plain_entries(16) * (int)sizeof(float2);  // the larger of the windows

// Fractional LUT angle index t = acos(c) tsc for c in [-1, 1] (c is clamped),
// tsc = (thetaR - 1) / PI_REF, tscpi = tsc * pi.  acos(x) = sqrt(1 - x) g(x)
// on [0, 1] with g analytic there (the square-root factorisation of acos at
// x = 1, as in Abramowitz & Stegun 4.4.45-46), and acos(-x) = pi - acos(x).
// g is our own degree-7 least-squares fit on 4000 Chebyshev nodes of [0, 1],
// weighted for absolute error; evaluated in single precision the angle is
// within 3.5e-7 rad of acos over [-1, 1] (about 1e-4 of one table column at
// thetaR = 1024).
__device__ __forceinline__ float theta_index(float c, float tsc, float tscpi) {
    const float ax = fminf(fabsf(c), 1.f);
    float s;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(s) : "f"(1.f - ax));
    float g = -1.411853940e-03f;
    g = fmaf(g, ax, 7.149144541e-03f);
    g = fmaf(g, ax, -1.768672466e-02f);
    g = fmaf(g, ax, 3.125903755e-02f);
    g = fmaf(g, ax, -5.028845742e-02f);
    g = fmaf(g, ax, 8.899561316e-02f);
    g = fmaf(g, ax, -2.145996839e-01f);
    g = fmaf(g, ax, 1.570796371e+00f);
    const float v = (s * tsc) * g;
    return c < 0.f ? tscpi - v : v;
}

// 8-byte global -> shared copy that does not go through registers (cp.async)
__device__ __forceinline__ void copy_async8(float2* dst, const float2* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ void copy_async16(float4* dst, const float4* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

// theta_index of two pixels with the polynomial and the final products in packed
// f32x2 instructions; every lane rounds as the scalar instruction, so t0, t1 are
// theta_index(c0, ...), theta_index(c1, ...) bit for bit.
__device__ __forceinline__ void theta_index2(float c0, float c1, float tsc, float tscpi, float& t0, float& t1) {
    const float ax0 = fminf(fabsf(c0), 1.f), ax1 = fminf(fabsf(c1), 1.f);
    float s0, s1;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(s0) : "f"(1.f - ax0));
    asm("sqrt.approx.f32 %0, %1;" : "=f"(s1) : "f"(1.f - ax1));
    const f32x2 ax = f2_pack(ax0, ax1);
    f32x2 g = f2_splat(-1.411853940e-03f);
    g = f2_fma(g, ax, f2_splat(7.149144541e-03f));
    g = f2_fma(g, ax, f2_splat(-1.768672466e-02f));
    g = f2_fma(g, ax, f2_splat(3.125903755e-02f));
    g = f2_fma(g, ax, f2_splat(-5.028845742e-02f));
    g = f2_fma(g, ax, f2_splat(8.899561316e-02f));
    g = f2_fma(g, ax, f2_splat(-2.145996839e-01f));
    g = f2_fma(g, ax, f2_splat(1.570796371e+00f));
    const float2 v = f2_unpack(f2_mul(f2_mul(f2_pack(s0, s1), f2_splat(tsc)), g));
    t0 = c0 < 0.f ? tscpi - v.x : v.x;
    t1 = c1 < 0.f ? tscpi - v.y : v.y;
}

__device__ __forceinline__ void copy_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Block-uniform values of one (tile, sphere) pair, kept in shared memory so
// that they are re-read per chunk instead of holding registers through the
// wave loops.
struct TileSphere {
    float cx, cy, cz;  // unit direction from the sphere to the tile centre
    float gam;         // angular radius of the tile seen from the sphere, plus margin
    float tsc, tscpi;
    int rlo, nrows;    // staged table rows [rlo, rlo + nrows); nrows = 0: cells from the table only
    int thetaR, lin_stride;
    long long off;     // first entry of the table in the linear pool
};

// Window of a wave chunk with bounding cone `cone` for the block's (tile, sphere):
// first column and width, width 0 when the block does not stage this sphere or
// the window does not fit.  Columns go up to thetaR: the linear rows carry a
// copy of the last column there.
__device__ __forceinline__ int2 chunk_plan(const float4 cone, const TileSphere& ts, int stage_cap) {
    if (ts.nrows == 0) return make_int2(0, 0);
    const float tsc = ts.tsc, gam = ts.gam;
    const float thc = acosf(fminf(fmaxf(cone.x * ts.cx + cone.y * ts.cy + cone.z * ts.cz, -1.f), 1.f));
    const int t_lo = max(0, (int)floorf((thc - cone.w - gam) * tsc) - 1);
    const int t_hi = min(ts.thetaR, (int)floorf((thc + cone.w + gam) * tsc) + 2);
    int W = t_hi - t_lo + 1;
    if (W < 2 || ts.nrows * lut_plain_stride(W) > stage_cap) W = 0;
    return make_int2(t_lo, W);
}

// STAGE = false: no dynamic shared memory and 6 blocks per SM.  PPT pixels per thread: the tile's eight 4 x 8 warp
// blocks are spread over 8 / PPT warps, and each wave's direction and phase (shared-memory broadcasts) are read
// once for the thread's PPT pixels.  Every pixel's arithmetic is the same for any PPT.
template <bool STAGE, int PPT>
__global__ void __launch_bounds__(UP_TILE / PPT, STAGE ? (PPT == 1 ? 3 : 4) : 6)
    us_lut_plain_kernel(Scene sc, const Sphere* __restrict__ sph, int s0, int s1, int accumulate, int finalize,
                        const float4* __restrict__ kw4, const float4* __restrict__ cones,
                        const cpx<float>* __restrict__ ph, const float2* __restrict__ lin,
                        const cpx<float>* __restrict__ Uf, cpx<float>* __restrict__ U,
                        unsigned long long* __restrict__ counters, float2* __restrict__ kcmp, int chunk,
                        int counted_chunk, int stage_cap) {
    constexpr int NT = UP_TILE / PPT, NWARP = NT / 32;
    static_assert(NT >= WAVE_CHUNK_MAX && NT % 32 == 0, "one thread per wave of a chunk");
    extern __shared__ float2 s_stage[];
    __shared__ float4 s_k[WAVE_CHUNK_MAX];
    __shared__ float2 s_p[WAVE_CHUNK_MAX];
    __shared__ int s_red[4][NWARP];
    __shared__ TileSphere s_ts;
    __shared__ int2 s_plan;  // staged window of the next chunk: first column, width (0: cells from the table)
    __shared__ double s_pa[3][16], s_pb[3][16];  // pixel position = s_pa[.][column] + s_pb[.][row]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the tile is covered by eight 4 x 8 pixel blocks (half-warps 4 x 4): the compact footprint of
    // one load instruction has the fewest shared-memory bank conflicts (8 x 4 blocks: 1 % slower,
    // 16 x 2: 22 %).  Pixel j of a thread lies in block warp + NWARP j.
    const int tiles_u = (sc.R + 15) / 16;
    const int tu = (blockIdx.x % tiles_u) * 16, tv = (blockIdx.x / tiles_u) * 16;
    int iu[PPT], iv[PPT], lu[PPT], lv[PPT];
    bool valid[PPT];
#pragma unroll
    for (int j = 0; j < PPT; j++) {
        const int blk = warp + NWARP * j;
        iu[j] = tu + (lane & 3) + 4 * (blk & 3);
        iv[j] = tv + (lane >> 2) + 8 * (blk >> 2);
        valid[j] = iu[j] < sc.R && iv[j] < sc.R;
        lu[j] = min(iu[j], sc.R - 1) - tu;
        lv[j] = min(iv[j], sc.R - 1) - tv;
    }
    // pixel_pos computes (A + X u) + Y v: the terms of the tile's 16 columns and 16 rows, once
    if (threadIdx.x < 32) {
        const int k = threadIdx.x & 15;
        const double t = __ddiv_rn((double)min((threadIdx.x < 16 ? tu : tv) + k, sc.R - 1), (double)sc.R);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            if (threadIdx.x < 16) s_pa[c][k] = __dadd_rn(sc.A[c], __dmul_rn(sc.X[c], t));
            else s_pb[c][k] = __dmul_rn(sc.Y[c], t);
        }
    }
    __syncthreads();
    float tot_r[PPT], tot_i[PPT], cmp_r[PPT], cmp_i[PPT];  // Kahan sums over chunk partials
#pragma unroll
    for (int j = 0; j < PPT; j++) {
        tot_r[j] = tot_i[j] = cmp_r[j] = cmp_i[j] = 0.f;
        if (accumulate && valid[j]) {
            tot_r[j] = U[iv[j] * sc.R + iu[j]].re;
            tot_i[j] = U[iv[j] * sc.R + iu[j]].im;
            if (kcmp) {  // the Kahan compensation the previous sphere chunk left: the sum goes on as in one launch
                cmp_r[j] = kcmp[iv[j] * sc.R + iu[j]].x;
                cmp_i[j] = kcmp[iv[j] * sc.R + iu[j]].y;
            }
        }
    }
    const int nchunks = (sc.nk + chunk - 1) / chunk;
    unsigned staged_chunks = 0;
    for (int s = s0; s < s1; s++) {
        const Sphere& S = sph[s];
        float rx[PPT], ry[PPT], rz[PPT], cb[PPT], al[PPT];
        int ir[PPT];
        unsigned cell[PPT];   // entry of the lower row's first column, from the sphere's first table
        int next[PPT];        // entries to the row above it
        bool far[PPT];  // outside the sphere, d > 0
#pragma unroll
        for (int j = 0; j < PPT; j++) {
            double p[3], r[3];
#pragma unroll
            for (int c = 0; c < 3; c++) p[c] = __dadd_rn(s_pa[c][lu[j]], s_pb[c][lv[j]]);
            const double d = dist_exact(p, S.p, r);
            const TableSel ts = select_table_scaled(S, d);
            ir[j] = (int)floor(ts.x);
            al[j] = (float)(ts.x - ir[j]);
            cell[j] = (unsigned)(ts.off - S.usp_off) + (unsigned)ir[j] * (unsigned)S.lin_stride;
            next[j] = ir[j] + 1 < ts.rows ? S.lin_stride : 0;
            rx[j] = ry[j] = rz[j] = 0.f;
            cb[j] = 1.f;  // d == 0: cos(theta) := 1
            if (d != 0) {
                const float inv = 1.f / (float)d;
                rx[j] = (float)r[0] * inv;
                ry[j] = (float)r[1] * inv;
                rz[j] = (float)r[2] * inv;
                cb[j] = 0.f;
            }
            far[j] = d >= S.a && d != 0;
        }
        // every pixel of a staged tile lies outside the sphere: its table is Usp (dR rows)
        const int rows = S.dR;
        // ---- tile bounds: table rows and angular radius gamma ----
        int rlo = 0, rhi = 0, ok = 0;
        if (!STAGE) {
            __syncthreads();  // s_ts is reused for every sphere
            if (threadIdx.x == 0) {
                s_ts.tsc = S.tsc;
                s_ts.tscpi = (float)((S.thetaR - 1) / PI_REF * TRUE_PI);
                s_ts.nrows = 0;
            }
        } else {
            // tile centre in single precision (bounds only, covered by the margins)
            const float u = ((float)tu + 7.5f) / (float)sc.R, v = ((float)tv + 7.5f) / (float)sc.R;
            float cx = (float)sc.A[0] + (float)sc.X[0] * u + (float)sc.Y[0] * v - (float)S.p[0];
            float cy = (float)sc.A[1] + (float)sc.X[1] * u + (float)sc.Y[1] * v - (float)S.p[1];
            float cz = (float)sc.A[2] + (float)sc.X[2] * u + (float)sc.Y[2] * v - (float)S.p[2];
            const float cl = sqrtf(cx * cx + cy * cy + cz * cz);
            bool far_ok = cl > 0.f;
            float gam = 0.f;
            if (cl > 0.f) {
                cx /= cl;
                cy /= cl;
                cz /= cl;
            }
            rlo = INT_MAX;
            rhi = INT_MIN;
#pragma unroll
            for (int j = 0; j < PPT; j++) {
                if (!valid[j]) continue;
                far_ok = far_ok && far[j];
                if (cl > 0.f)
                    gam = fmaxf(gam, acosf(fminf(fmaxf(rx[j] * cx + ry[j] * cy + rz[j] * cz, -1.f), 1.f)));
                rlo = min(rlo, ir[j]);
                rhi = max(rhi, ir[j]);
            }
            rlo = __reduce_min_sync(0xffffffffu, rlo);
            rhi = __reduce_max_sync(0xffffffffu, rhi);
            int gbits = (int)__reduce_max_sync(0xffffffffu, (unsigned)__float_as_int(gam));
            ok = __all_sync(0xffffffffu, far_ok);
            __syncthreads();  // s_red and s_ts are reused for every sphere
            if (lane == 0) {
                s_red[0][warp] = rlo;
                s_red[1][warp] = rhi;
                s_red[2][warp] = gbits;
                s_red[3][warp] = ok;
            }
            __syncthreads();
#pragma unroll
            for (int w = 0; w < NWARP; w++) {
                rlo = min(rlo, s_red[0][w]);
                rhi = max(rhi, s_red[1][w]);
                gbits = max(gbits, s_red[2][w]);
                ok = ok && s_red[3][w];
            }
            if (threadIdx.x == 0) {
                s_ts.cx = cx;
                s_ts.cy = cy;
                s_ts.cz = cz;
                s_ts.gam = __int_as_float(gbits) + LUT_PLAIN_MARGIN;
                s_ts.tsc = S.tsc;
                s_ts.tscpi = (float)((S.thetaR - 1) / PI_REF * TRUE_PI);
                // staged rows: [rlo, rhi + 1] clamped to the table
                s_ts.rlo = rlo;
                s_ts.nrows = ok ? min(rhi + 1, rows - 1) - rlo + 1 : 0;
                s_ts.thetaR = S.thetaR;
                s_ts.lin_stride = S.lin_stride;
                s_ts.off = S.usp_off;
                s_plan = chunk_plan(cones[0], s_ts, stage_cap);
            }
        }
        // local rows of each pixel in the staged block (clamped, so always in bounds)
        const int nrows_b = ok ? min(rhi + 1, rows - 1) - rlo + 1 : 1;
        int lr0[PPT], drow0[PPT];
#pragma unroll
        for (int j = 0; j < PPT; j++) {
            lr0[j] = min(max(ir[j] - rlo, 0), max(nrows_b, 1) - 1);
            drow0[j] = min(max(min(ir[j] + 1, rows - 1) - rlo, 0), max(nrows_b, 1) - 1) - lr0[j];
        }
        for (int ch = 0; ch < nchunks; ch++) {
            const int w0 = ch * chunk;
            const int nw = min(chunk, sc.nk - w0);
            __syncthreads();  // the previous chunk's readers are done; s_ts is written
            const int nrows = s_ts.nrows;
            // window of this chunk: planned by thread 0 (before the first chunk, or while the
            // previous chunk was summed)
            const int2 pl = STAGE ? s_plan : make_int2(0, 0);
            const int t_lo = pl.x, W = pl.y, Ws = lut_plain_stride(W);
            const bool staged = STAGE && W > 0;
            if (threadIdx.x < nw) {
                copy_async16(&s_k[threadIdx.x], kw4 + w0 + threadIdx.x);
                copy_async8(&s_p[threadIdx.x], reinterpret_cast<const float2*>(ph + (size_t)s * sc.nk + w0) + threadIdx.x);
            }
            if (STAGE && staged) {
                // asynchronous copies, one table row per warp at a time, all in flight together
                const float2* table = lin + s_ts.off + (size_t)s_ts.rlo * s_ts.lin_stride + t_lo;
                const int ls = s_ts.lin_stride;
                for (int rr = warp; rr < nrows; rr += NWARP) {
                    const float2* src = table + (size_t)rr * ls;
                    float2* dst = s_stage + rr * Ws;
                    for (int tt = lane; tt < W; tt += 32) copy_async8(dst + tt, src + tt);
                }
            }
            copy_async_wait_all();
            __syncthreads();
            if (STAGE && threadIdx.x == 0 && ch + 1 < nchunks) s_plan = chunk_plan(cones[ch + 1], s_ts, stage_cap);
            // t < thetaR - 1 + 1e-3 (PI_REF < pi): the rows repeat the last column, so t past thetaR - 1 reads
            // it, as a clamp would
            const float tsc = s_ts.tsc, tscpi = s_ts.tscpi;
            // the chunk's sum of pw v as sum(pw.x v) and sum(pw.y v), each a (re, im) pair:
            // Re = x.re - y.im, Im = x.im + y.re
            float2 sx[PPT], sy[PPT];
            if (STAGE && staged) {
                staged_chunks++;
                const unsigned lt_max = (unsigned)(W - 2);
                const float2* row0[PPT];
                int drow[PPT];
                f32x2 alp[PPT], ax[PPT], ay[PPT];
#pragma unroll
                for (int j = 0; j < PPT; j++) {
                    row0[j] = s_stage + lr0[j] * Ws;
                    drow[j] = drow0[j] * Ws;
                    alp[j] = f2_splat(al[j]);
                    ax[j] = ay[j] = 0ull;
                }
                // one lookup of pixel j at angle index t, wave weight (pwx, pwy)
                auto lookup = [&](int j, float t, f32x2 pwx, f32x2 pwy) {
                    const float tf = floorf(t);
                    const float be = t - tf;
                    // in the window by construction; the unsigned clamp only keeps a bad bound in bounds
                    const unsigned lt = min((unsigned)((int)tf - t_lo), lt_max);
                    const f32x2* q = reinterpret_cast<const f32x2*>(row0[j] + lt);
                    const f32x2 e00 = q[0], e01 = q[1], e10 = q[drow[j]], e11 = q[drow[j] + 1];
                    const f32x2 bep = f2_splat(be);
                    const f32x2 a0 = f2_fma(bep, f2_sub(e01, e00), e00);
                    const f32x2 a1 = f2_fma(bep, f2_sub(e11, e10), e10);
                    const f32x2 v = f2_fma(alp[j], f2_sub(a1, a0), a0);
                    ax[j] = f2_fma(pwx, v, ax[j]);
                    ay[j] = f2_fma(pwy, v, ay[j]);
                };
                // cb = 0 here: every d > 0.  The angle indices of two lookups at a time (the thread's
                // two pixels, or one pixel's two consecutive waves) in packed instructions; the lookups
                // and their sums run in wave order, so the bits are those of one at a time.
                // 32 lookups per thread per unrolled step (3072^2 pixels, 50 spheres, 1000 directions: 697 ms; 8:
                // 721 ms, 16: 700 ms, 64: 792 ms)
                if (PPT == 2) {
#pragma unroll 16
                    for (int w = 0; w < nw; w++) {
                        const float4 kk = s_k[w];
                        const float2 pw = s_p[w];
                        const f32x2 pwx = f2_splat(pw.x), pwy = f2_splat(pw.y);
                        float t0, t1;
                        theta_index2(fmaf(kk.x, rx[0], fmaf(kk.y, ry[0], kk.z * rz[0])),
                                     fmaf(kk.x, rx[PPT - 1], fmaf(kk.y, ry[PPT - 1], kk.z * rz[PPT - 1])), tsc,
                                     tscpi, t0, t1);
                        lookup(0, t0, pwx, pwy);
                        lookup(PPT - 1, t1, pwx, pwy);
                    }
                } else {
                    int w = 0;
#pragma unroll 16
                    for (; w + 1 < nw; w += 2) {
                        const float4 k0 = s_k[w], k1 = s_k[w + 1];
                        const float2 p0 = s_p[w], p1 = s_p[w + 1];
                        float t0, t1;
                        theta_index2(fmaf(k0.x, rx[0], fmaf(k0.y, ry[0], k0.z * rz[0])),
                                     fmaf(k1.x, rx[0], fmaf(k1.y, ry[0], k1.z * rz[0])), tsc, tscpi, t0, t1);
                        lookup(0, t0, f2_splat(p0.x), f2_splat(p0.y));
                        lookup(0, t1, f2_splat(p1.x), f2_splat(p1.y));
                    }
                    if (w < nw) {
                        const float4 kk = s_k[w];
                        const float2 pw = s_p[w];
                        lookup(0, theta_index(fmaf(kk.x, rx[0], fmaf(kk.y, ry[0], kk.z * rz[0])), tsc, tscpi),
                               f2_splat(pw.x), f2_splat(pw.y));
                    }
                }
#pragma unroll
                for (int j = 0; j < PPT; j++) {
                    sx[j] = f2_unpack(ax[j]);
                    sy[j] = f2_unpack(ay[j]);
                }
            } else {
                const float2* tab = lin + S.usp_off;
                const int last = S.thetaR - 1;
                f32x2 alp[PPT], ax[PPT], ay[PPT];
#pragma unroll
                for (int j = 0; j < PPT; j++) {
                    alp[j] = f2_splat(al[j]);
                    ax[j] = ay[j] = 0ull;
                }
#pragma unroll 4
                for (int w = 0; w < nw; w++) {
                    const float4 kk = s_k[w];
                    const float2 pw = s_p[w];
#pragma unroll
                    for (int j = 0; j < PPT; j++) {
                        const float c = fmaf(kk.x, rx[j], fmaf(kk.y, ry[j], fmaf(kk.z, rz[j], cb[j])));
                        const float t = theta_index(c, tsc, tscpi);
                        const float tf = floorf(t);
                        const f32x2 bep = f2_splat(t - tf);
                        const int n = min(max((int)tf, 0), last);
                        const f32x2* q = reinterpret_cast<const f32x2*>(tab + (size_t)(cell[j] + (unsigned)n));
                        const f32x2 e00 = __ldg(q), e01 = __ldg(q + 1), e10 = __ldg(q + next[j]), e11 = __ldg(q + next[j] + 1);
                        const f32x2 a0 = f2_fma(bep, f2_sub(e01, e00), e00);
                        const f32x2 a1 = f2_fma(bep, f2_sub(e11, e10), e10);
                        const f32x2 v = f2_fma(alp[j], f2_sub(a1, a0), a0);
                        ax[j] = f2_fma(f2_splat(pw.x), v, ax[j]);
                        ay[j] = f2_fma(f2_splat(pw.y), v, ay[j]);
                    }
                }
#pragma unroll
                for (int j = 0; j < PPT; j++) {
                    sx[j] = f2_unpack(ax[j]);
                    sy[j] = f2_unpack(ay[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < PPT; j++) {
                const float ar = sx[j].x - sy[j].y, ai = sx[j].y + sy[j].x;
                // Kahan: add the chunk partial to the running total
                const float yr = ar - cmp_r[j], yi = ai - cmp_i[j];
                const float tr = tot_r[j] + yr, ti = tot_i[j] + yi;
                cmp_r[j] = (tr - tot_r[j]) - yr;
                cmp_i[j] = (ti - tot_i[j]) - yi;
                tot_r[j] = tr;
                tot_i[j] = ti;
            }
        }
    }
    if (threadIdx.x == 0 && counters) {
        atomicAdd(counters, (unsigned long long)staged_chunks);
        atomicAdd(counters + 1, (unsigned long long)(s1 - s0) * ((sc.nk + counted_chunk - 1) / counted_chunk));
    }
#pragma unroll
    for (int j = 0; j < PPT; j++) {
        if (!valid[j]) continue;
        const int idx = iv[j] * sc.R + iu[j];
        if (finalize) {
            double p[3];
#pragma unroll
            for (int c = 0; c < 3; c++) p[c] = __dadd_rn(s_pa[c][lu[j]], s_pb[c][lv[j]]);
            if (outside_all(sc, sph, p)) {
                tot_r[j] += Uf[idx].re - cmp_r[j];
                tot_i[j] += Uf[idx].im - cmp_i[j];
            }
        } else if (kcmp) {
            kcmp[idx] = make_float2(cmp_r[j], cmp_i[j]);
        }
        U[idx] = mk(tot_r[j], tot_i[j]);
    }
}

void launch_us_lut_plain(const Scene& sc, const Sphere* sph, int s0, int s1, int accumulate, int finalize,
                         const float4* kw4, const float4* cones, const cpx<float>* ph, const float2* lin,
                         const cpx<float>* Uf, cpx<float>* U, unsigned long long* counters, float2* kcmp, bool stage,
                         int chunk, int counted_chunk, cudaStream_t st) {
    const unsigned tiles = (sc.R + 15) / 16;
    const bool two = chunk >= UP_TWO_PIXEL_MIN_CHUNK;
    const int cap = stage ? lut_plain_entries(chunk) : 0, smem = cap * (int)sizeof(float2);
    auto kernel = !stage ? us_lut_plain_kernel<false, 1> : two ? us_lut_plain_kernel<true, 2> : us_lut_plain_kernel<true, 1>;
    // per device, cheap and the same value on every call; a failure shows up as the launch error
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, UP_SMEM);
    kernel<<<tiles * tiles, stage && two ? UP_TILE / 2 : UP_TILE, smem, st>>>(sc, sph, s0, s1, accumulate, finalize, kw4,
                                                                            cones, ph, lin, Uf, U, counters, kcmp, chunk,
                                                                            counted_chunk, cap);
}

// Loads every kernel of this file (cudaFuncGetAttributes), see preload_nearfield_kernels.
void preload_uslut_plain_kernels() {
    cudaFuncAttributes a;
    cudaFuncGetAttributes(&a, us_lut_plain_kernel<false, 1>);
    cudaFuncGetAttributes(&a, us_lut_plain_kernel<true, 1>);
    cudaFuncGetAttributes(&a, us_lut_plain_kernel<true, 2>);
}

}  // namespace bs
