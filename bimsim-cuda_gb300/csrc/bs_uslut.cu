// bs_uslut.cu -- mixed-precision scattered field from the sphere tables
// (gpuScalarUpLut, nfScalarUpLut.cu:11-97), all spheres of [s0, s1) in one
// launch, with Uf added where the pixel is outside every sphere
// (nfSumUf.cu:6-49): per-(pixel, sphere) geometry in double, per-wave work in
// single precision, per-sphere sums combined with Kahan compensation.
#include <cuda_runtime.h>

#include "bs_kernels.h"
#include "bs_lut.cuh"

namespace bs {

// Fractional table columns of two directions: t = acos(c) tsc - t0, with c clamped to
// [-1, 1] and hb = (pi / 2) tsc - t0.  acos(x) = sqrt(1 - x) g(x) on [0, 1] with g analytic
// there (the square-root factorisation of acos at x = 1, as in Abramowitz & Stegun
// 4.4.45-46); g is our own degree-7 least-squares fit on 4000 Chebyshev nodes of [0, 1],
// weighted for absolute error.  w = pi/2 - acos|c| takes the sign of c, so that
// acos(c) = pi/2 - w for both signs; within 1.6e-7 rad of acos over [-1, 1].
__device__ __forceinline__ f32x2 theta_column2(f32x2 c, f32x2 ntsc, f32x2 hb) {
    const float2 cc = f2_unpack(c);
    const float ax0 = fminf(fabsf(cc.x), 1.f), ax1 = fminf(fabsf(cc.y), 1.f);
    const f32x2 ax = f2_pack(ax0, ax1);
    const float2 om = f2_unpack(f2_sub(f2_splat(1.f), ax));
    float s0, s1;  // 1 - |c| is 0 or at least 2^-24: flushing subnormals changes nothing
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(s0) : "f"(om.x));
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(s1) : "f"(om.y));
    f32x2 g = f2_splat(1.411853940e-03f);  // -g
    g = f2_fma(g, ax, f2_splat(-7.149144541e-03f));
    g = f2_fma(g, ax, f2_splat(1.768672466e-02f));
    g = f2_fma(g, ax, f2_splat(-3.125903755e-02f));
    g = f2_fma(g, ax, f2_splat(5.028845742e-02f));
    g = f2_fma(g, ax, f2_splat(-8.899561316e-02f));
    g = f2_fma(g, ax, f2_splat(2.145996839e-01f));
    g = f2_fma(g, ax, f2_splat(-1.570796371e+00f));
    const float2 w = f2_unpack(f2_fma(f2_pack(s0, s1), g, f2_splat(1.570796371e+00f)));
    return f2_fma(f2_pack(copysignf(w.x, cc.x), copysignf(w.y, cc.y)), ntsc, hb);
}

// hb of the columns from t_lo on.  From column 0 on it is at least the largest w in columns, rounded up:
// a direction through the pixel (c = 1) then has column 0 or a little above, where the rounding of hb
// and tsc alone could leave it below 0 and outside the table or the window.
__device__ __forceinline__ float column_base(float hp_hi, float hp_lo, float tsc, int t_lo) {
    const float hb = (hp_hi - (float)t_lo) + hp_lo;
    return t_lo == 0 ? fmaxf(hb, __fmul_ru(1.570796371f, tsc)) : hb;
}

// ---------------------------------------------------------------------------
// The sorted kernel (where neither lut_plain nor lut_few applies)
//
// A block owns a 16 x 16 pixel tile, each of its 8 warps two rows of 16 pixels.  Per sphere:
//  * the block sorts the directions by their angle to the tile centre's direction (as seen
//    from the sphere; up to SW_WAVES at a time), so that 32 consecutive directions, one per
//    lane, fall into neighbouring table columns for every pixel of the tile: a warp's load
//    touches a few contiguous words instead of 32 scattered ones;
//  * a warp takes bands of consecutive groups of 32 directions whose columns fit a window (64
//    columns of 16 pixels, or more columns of fewer pixels at a time, see plan_bands), blends
//    each pixel's two table rows over that window (the radial weight is the same for every
//    direction) and keeps the blended row in shared memory: a lookup then reads two values
//    instead of four.  Groups whose window does not fit read the table itself;
//  * a lane walks its direction over the row's 16 pixels.  The column t along the row is
//    smooth, so far from the poles it is a polynomial through 4 or 6 Chebyshev points of the
//    row instead of 16 arc cosines (row_mode below), and evaluating it for the pixels +-s
//    shares its even and odd parts.
// Sums run over the lane's directions in sorted order, then over the lanes in a fixed tree, then
// over spheres with Kahan compensation: the same for the staged and the unstaged kernel, whose
// results are therefore identical.
// ---------------------------------------------------------------------------
constexpr int SW_BATCH = 4;      // pixels whose table rows a lane loads together
constexpr int SW_NT = 256;       // threads per block
constexpr int SW_WAVES = 1024;   // directions sorted at a time
constexpr int SW_W = 64;         // columns of a pixel's window
constexpr int SW_GROUPS = SW_WAVES / 32;
constexpr float SW_HALF = 7.5f;  // half a row, pixels

template <int N>
struct Int {  // a compile-time argument of the kernel's lambdas
    static constexpr int value = N;
};

struct PixRow {
    unsigned off;  // first entry of the pixel's lower table row, from the sphere's first table
    float al;      // radial weight of the next row
};

constexpr int SW_BUCKETS = 128;

struct SwShared {
    float2 win[8][16 * SW_W];  // blended rows of the warp's 16 pixels
    float4 k[SW_WAVES];        // ordered directions
    float2 p[SW_WAVES];        // and their phases for the current sphere
    unsigned hist[8][SW_BUCKETS];
    unsigned wsum[4];
    float2 gb[SW_GROUPS];      // smallest and largest column of each group at the tile centre
    int4 band[SW_GROUPS];      // the band that starts at a group, see plan_bands
    float2 acc[8][2][32];      // Kahan sum and compensation of the warps' rows
    float rdist[8][2];         // 1 / distance of the rows' centres from the sphere
    float3 X, Y;               // the slice's axes in single precision (bounds and node directions)
    float iR, half;            // 1 / R; half a row, um
    PixRow px[8][32];
    float4 dir[8][2][16];      // pixel directions, pixels i and 15 - i together: {x, x', y, y'}, {z, z', cb, cb'}
    float4 node[8][2][10];     // directions of the row's 2 + 3 node pairs, same layout
    double pa[3][16], pb[3][16];  // pixel position = pa[.][column] + pb[.][row]
};

constexpr int SW_SMEM = (int)sizeof(SwShared);

// +-cos of the Chebyshev angles of 4 and of 6 points
__constant__ float c_nodes[10] = {0.923879533f, -0.923879533f, 0.382683432f, -0.382683432f, 0.965925826f,
                                  -0.965925826f, 0.707106781f, -0.707106781f, 0.258819045f, -0.258819045f};

// Points a row's column polynomial needs: 4, 6, or 0 for an arc cosine per pixel.  With
// rho = (distance of the row's centre from the sphere) x (smallest sine of the angle between
// the row's directions and the group's waves) and q = (half row length) / rho, the error of the
// interpolated angle is below 0.0318 q^4 rad (4 points) and 0.0056 q^6 rad (6 points): the
// largest over 4e4 random geometries per decade of q.  Both limits keep it under 6e-8 rad,
// half of what single precision leaves of the arc cosine itself.
__device__ __forceinline__ int row_mode(float q) { return q <= 0.037f ? 4 : (q <= 0.148f ? 6 : 0); }
// In windows of 8 pixels (shape 2) the polynomial is made twice, of 4 (shape 3) four times: 4 points still cost
// less than 8 arc cosines, 6 do not, and nothing less than 4.
__device__ __forceinline__ int band_mode(float q, int shape) {
    const int mode = row_mode(q);
    return shape < 2 || (shape == 2 && mode == 4) ? mode : 0;
}

// Order the nkb directions kw[0 .. nkb) by their angle to `ctr` and write them, with their
// phases, to sm.k and sm.p: a stable counting sort over SW_BUCKETS equal steps of the cosine
// between chi (the largest expected) and chi - SW_BUCKETS / scale, about three table columns each.
// The last group is filled up with copies of the last direction of weight zero.
__device__ __forceinline__ void order_waves(SwShared& sm, const float4* __restrict__ kw,
                                            const cpx<float>* __restrict__ ph, int nkb, float3 ctr, float chi,
                                            float scale) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float4 kv[SW_WAVES / SW_NT];
    int slot[SW_WAVES / SW_NT];  // bucket, and rank within (warp, bucket)
#pragma unroll
    for (int i = 0; i < SW_BUCKETS / 32; i++) sm.hist[warp][lane + 32 * i] = 0;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < SW_WAVES / SW_NT; i++) {
        const int e = i * SW_NT + tid;
        if (i * SW_NT >= nkb) break;
        const bool valid = e < nkb;
        kv[i] = kw[valid ? e : nkb - 1];
        const float c = fmaf(kv[i].x, ctr.x, fmaf(kv[i].y, ctr.y, kv[i].z * ctr.z));
        const int b = valid ? min(max((int)((chi - c) * scale), 0), SW_BUCKETS - 1) : SW_BUCKETS;
        const unsigned m = __match_any_sync(0xffffffffu, b);
        const int rank = __popc(m & ((1u << lane) - 1u));
        unsigned base = 0;
        if (valid && rank == 0) {
            base = sm.hist[warp][b];
            sm.hist[warp][b] = base + __popc(m);
        }
        base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
        slot[i] = b | (int)(base + rank) << 8;
        __syncwarp();
    }
    __syncthreads();  // counts done; and the readers of the previous k and p
    unsigned cnt[8], sum = 0, incl = 0;
    if (tid < SW_BUCKETS) {
#pragma unroll
        for (int w = 0; w < 8; w++) sum += cnt[w] = sm.hist[w][tid];
        incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += o;
        }
        if (lane == 31) sm.wsum[warp] = incl;
    }
    __syncthreads();
    if (tid < SW_BUCKETS) {
        unsigned o = incl - sum;
#pragma unroll
        for (int w = 0; w < 3; w++) o += w < warp ? sm.wsum[w] : 0;
#pragma unroll
        for (int w = 0; w < 8; w++) {
            sm.hist[w][tid] = o;
            o += cnt[w];
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < SW_WAVES / SW_NT; i++) {
        const int e = i * SW_NT + tid;
        if (e < nkb) {
            const unsigned pos = sm.hist[warp][slot[i] & 255] + ((unsigned)slot[i] >> 8);
            sm.k[pos] = kv[i];
            sm.p[pos] = make_float2(ph[e].re, ph[e].im);
        }
    }
    __syncthreads();
    if (nkb & 31) {
        if (tid < 32 - (nkb & 31)) {
            sm.k[nkb + tid] = sm.k[nkb - 1];
            sm.p[nkb + tid] = make_float2(0.f, 0.f);
        }
        __syncthreads();
    }
}

// Warp 0: lane g finds the band that starts at group g, the groups [g, nx) whose columns, seen from
// anywhere in the tile, fit one window: band[g] = {first column, nx | shape << 8 | columns << 16,
// (half row length) / (smallest sine of the angles between the band's directions and the tile's
// pixels), 0}.  The window holds 16 pixels x 64 columns, half the row's pixels x 128 or a quarter x 256
// (shapes 1, 2, 3): wider ones take in more groups per blended row, but a row's polynomials are made
// again for each part.  The shape of least cost per (pixel, group) is taken, in instructions and their
// shared-memory share: 24 per 64 columns blended, and the row's polynomial (3.5 or 5.5 a pixel each time it is made)
// or arc cosine (11); none (shape 0: a band of one group, cells from the table) where all are above 34.
// Measured with 16 x 64 alone, with all three and polynomials of 6 points in all, and now: 768^2 pixels of 0.39 um,
// 120 spheres, 1000 directions 144, 120 and 115 ms; 906^2 of 0.13 um, NA 0.9 18.7, 17.0 and 16.0 ms; 3072^2 of 0.1 um
// (narrow windows throughout) the same.
// Returns the number of chunks of `chunk` directions (64, 32 or 16) in the bands with a window (lane 0;
// chunk 0: none).
__device__ __forceinline__ unsigned plan_bands(SwShared& sm, int G, int nkb, int thetaR, float tsc, float gam, float rdist,
                                               int chunk) {
    const int lane = threadIdx.x & 31;
    const float gcol = gam * tsc;
    int info = 0;
    if (lane < G) {
        const int t_lo = max(0, (int)floorf(sm.gb[lane].x - gcol) - 1) & ~1;
        float best = 34.f, bq = 0.f;
        info = (lane + 1);
        float lo = sm.gb[lane].x, hi = sm.gb[lane].y;
        auto quotient = [&]() {  // (half row length) / (smallest sine)
            const float rt = 1.f / tsc, th0 = lo * rt - gam, th1 = hi * rt + gam;
            const float sn = th0 > 0.f && th1 < (float)TRUE_PI ? fminf(__sinf(th0), __sinf(th1)) : 0.f;
            return sm.half / fmaxf(sn, 1e-30f);
        };
        bq = quotient();
        int nx = lane, t_hi = t_lo;
        for (int s = 0; s < 3; s++) {  // the groups that fit a wider window continue those of the narrower
            while (nx < G) {
                const float2 b = sm.gb[nx];
                const int th = min(thetaR, (int)floorf(b.y + gcol) + 2);
                if (th - t_lo > (SW_W << s) - 1 || max(0, (int)floorf(b.x - gcol) - 1) < t_lo) break;
                t_hi = max(t_hi, th);
                lo = fminf(lo, b.x);
                hi = fmaxf(hi, b.y);
                nx++;
            }
            if (nx == lane) continue;
            const float q = quotient();
            const int mode = band_mode(q * rdist, s + 1);
            const float cost = 24.f * (1 << s) / (nx - lane) + (mode == 4 ? 3.5f * (1 << s) : mode == 6 ? 5.5f : 11.f);
            if (cost < best) {
                best = cost;
                bq = q;
                info = nx | (s + 1) << 8 | (t_hi - t_lo) << 16;
            }
            if (nx == G) break;
        }
        sm.band[lane] = make_int4(t_lo, info, __float_as_int(bq), 0);
    }
    unsigned mask = 0;  // groups in bands that fit
    for (int g = 0; g < G;) {
        const int i = __shfl_sync(0xffffffffu, info, g), nx = i & 255;
        if (i & 0x300) mask |= (nx < 32 ? (1u << nx) - 1u : 0xffffffffu) & ~((1u << g) - 1u);
        g = nx;
    }
    const unsigned last = mask >> (G - 1) & 1u;
    if (chunk == 64) return __popc(mask & (mask >> 1) & 0x55555555u) + (G & 1 ? last : 0u);
    if (chunk == 32) return __popc(mask);
    return chunk == 16 ? 2 * __popc(mask) - (((nkb - 1) & 31) < 16 ? last : 0u) : 0u;
}

template <bool STAGE>
__global__ void __launch_bounds__(SW_NT, 2)
    us_lut_sorted_kernel(Scene sc, const Sphere* __restrict__ sph, int s0, int s1, int accumulate, int finalize,
                         const float4* __restrict__ kw4, const cpx<float>* __restrict__ ph,
                         const float2* __restrict__ lin, const cpx<float>* __restrict__ Uf, cpx<float>* __restrict__ U,
                         unsigned long long* __restrict__ counters, float2* __restrict__ kcmp,
                         float* __restrict__ part, int chunk, float4 cone, float margin) {
    extern __shared__ __align__(1024) unsigned char sw_smem[];
    SwShared& sm = *reinterpret_cast<SwShared*>(sw_smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_u = (sc.R + 15) / 16;
    const int tu = (blockIdx.x % tiles_u) * 16, tv = (blockIdx.x / tiles_u) * 16;
    // blockIdx.y: the block's share of all the spheres (lut_splits), with sums of its own
    const int share = blockIdx.y, shares = gridDim.y;
    const int sb = max(s0, (int)((long long)sc.ns * share / shares));
    const int se = min(s1, (int)((long long)sc.ns * (share + 1) / shares));
    const size_t plane = 2 * (size_t)sc.R * sc.R;
    float* sum = part ? part + 2 * share * plane : reinterpret_cast<float*>(U);
    float* comp = part ? sum + plane : reinterpret_cast<float*>(kcmp);
    // pixel_pos computes (A + X u) + Y v: the terms of the tile's 16 columns and 16 rows, once
    if (threadIdx.x < 32) {
        const int k = threadIdx.x & 15;
        const double t = __ddiv_rn((double)min((threadIdx.x < 16 ? tu : tv) + k, sc.R - 1), (double)sc.R);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            if (threadIdx.x < 16) sm.pa[c][k] = __dadd_rn(sc.A[c], __dmul_rn(sc.X[c], t));
            else sm.pb[c][k] = __dmul_rn(sc.Y[c], t);
        }
    }
    __syncthreads();
    // lane L ends up with component L & 1 of pixel L >> 1 of each of the warp's rows
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int opx = tu + (lane >> 1), iv = tv + 2 * warp + r;
        float2 a = make_float2(0.f, 0.f);
        if (accumulate && opx < sc.R && iv < sc.R) {
            const size_t o = 2 * ((size_t)iv * sc.R + opx) + (lane & 1);
            a.x = sum[o];
            if (comp) a.y = comp[o];
        }
        sm.acc[warp][r][lane] = a;
    }
    if (threadIdx.x == 0) {
        sm.X = make_float3((float)sc.X[0], (float)sc.X[1], (float)sc.X[2]);
        sm.Y = make_float3((float)sc.Y[0], (float)sc.Y[1], (float)sc.Y[2]);
        sm.iR = 1.f / (float)sc.R;
        sm.half = SW_HALF * sm.iR * sqrtf(sm.X.x * sm.X.x + sm.X.y * sm.X.y + sm.X.z * sm.X.z);
    }
    unsigned staged_units = 0;
    const unsigned win0 = (unsigned)(warp * sizeof(sm.win[0]));
    __syncthreads();
    for (int s = sb; s < se; s++) {
        const Sphere& S = sph[s];
        // ---- the warp's pixels: lanes 0-15 the first row, 16-31 the second ----
        {
            const int j = lane & 15, r = lane >> 4, lv = 2 * warp + (lane >> 4), lu = lane & 15;
            double p[3], rr[3];
#pragma unroll
            for (int c = 0; c < 3; c++) p[c] = __dadd_rn(sm.pa[c][lu], sm.pb[c][lv]);
            const double d = dist_exact(p, S.p, rr);
            const TableSel ts = select_table_scaled(S, d);
            // rows ir and ir + 1 (every table has two rows or more)
            const int ir = min((int)ts.x, max(ts.rows, 2) - 2);
            PixRow q;
            q.off = (unsigned)(ts.off - S.usp_off) + (unsigned)ir * (unsigned)S.lin_stride;
            q.al = (float)(ts.x - ir);
            const float rx = (float)rr[0], ry = (float)rr[1], rz = (float)rr[2];
            const float inv = d != 0 ? 1.f / (float)d : 0.f;
            __syncwarp();  // the previous sphere's readers of this warp's pixel data are done
            sm.px[warp][lane] = q;
            float* dv = reinterpret_cast<float*>(sm.dir[warp][r]);
            const int pi = j < 8 ? j : 15 - j, sl = j < 8 ? 0 : 1;
            dv[8 * pi + sl] = rx * inv;
            dv[8 * pi + 2 + sl] = ry * inv;
            dv[8 * pi + 4 + sl] = rz * inv;
            dv[8 * pi + 6 + sl] = d != 0 ? 0.f : 1.f;  // d == 0: cos(theta) := 1
            // row centres from each row's first pixel (never clamped in x), and the node directions
            const float3 X = sm.X;
            const float hx = SW_HALF * sm.iR;
            const float3 cen = make_float3(__shfl_sync(0xffffffffu, rx, lane & 16) + X.x * hx,
                                           __shfl_sync(0xffffffffu, ry, lane & 16) + X.y * hx,
                                           __shfl_sync(0xffffffffu, rz, lane & 16) + X.z * hx);
            if (j == 0) sm.rdist[warp][r] = 1.f / sqrtf(cen.x * cen.x + cen.y * cen.y + cen.z * cen.z);
            if (j < 10) {
                const float w = c_nodes[j] * hx;
                const float vx = fmaf(X.x, w, cen.x), vy = fmaf(X.y, w, cen.y), vz = fmaf(X.z, w, cen.z);
                const float l2 = vx * vx + vy * vy + vz * vz;
                const float ni = l2 > 0.f ? 1.f / sqrtf(l2) : 0.f;
                float* nv = reinterpret_cast<float*>(sm.node[warp][r]) + 8 * (j >> 1) + (j & 1);
                nv[0] = vx * ni;
                nv[2] = vy * ni;
                nv[4] = vz * ni;
            }
        }
        const float tsc = S.tsc, hp_hi = S.hp_hi, hp_lo = S.hp_lo;
        const int thetaR = S.thetaR, row_len = S.lin_stride;
        const float2* tab = lin + S.usp_off;
        for (int w0 = 0; w0 < sc.nk; w0 += SW_WAVES) {
            const int nkb = min(SW_WAVES, sc.nk - w0), G = (nkb + 31) >> 5;
            const cpx<float>* phs = ph + (size_t)s * sc.nk + w0;
            // ---- the tile seen from the sphere: centre direction, angular radius gamma ----
            float3 ctr;
            float gam, tile_rdist = 0.f;  // 1 / distance of the tile's centre
            {
                // from the sphere's centre: differences of absolute positions in single precision would lose the
                // angles of a slice far from the origin
                const float3 A = make_float3(S.rel[0], S.rel[1], S.rel[2]), X = sm.X, Y = sm.Y;
                const float iR = sm.iR;
                auto at = [&](float u, float v) {
                    return make_float3(fmaf(X.x, u * iR, fmaf(Y.x, v * iR, A.x)), fmaf(X.y, u * iR, fmaf(Y.y, v * iR, A.y)),
                                       fmaf(X.z, u * iR, fmaf(Y.z, v * iR, A.z)));
                };
                ctr = at((float)tu + 7.5f, (float)tv + 7.5f);
                const float cl2 = ctr.x * ctr.x + ctr.y * ctr.y + ctr.z * ctr.z;
                gam = (float)TRUE_PI;
                if (cl2 > 0.f) {
                    const float ci = 1.f / sqrtf(cl2);
                    tile_rdist = ci;
                    ctr = make_float3(ctr.x * ci, ctr.y * ci, ctr.z * ci);
                    const float3 q = at((float)((lane & 1) ? min(tu + 15, sc.R - 1) : tu),
                                        (float)((lane & 2) ? min(tv + 15, sc.R - 1) : tv));
                    // the largest angle of a rectangle seen from outside lies at a corner; one that
                    // surrounds the sphere's centre has a corner at 90 degrees or more.  The angle from
                    // the chord between the unit vectors: 2 asin(chord / 2), at most chord + 0.06 chord^3
                    // up to a chord of 1.3 (79 degrees)
                    const float qi = 1.f / sqrtf(q.x * q.x + q.y * q.y + q.z * q.z);
                    const float ex = fmaf(q.x, qi, -ctr.x), ey = fmaf(q.y, qi, -ctr.y), ez = fmaf(q.z, qi, -ctr.z);
                    const float ch = sqrtf(ex * ex + ey * ey + ez * ez);
                    const float a = ch <= 1.3f ? fmaf(ch * ch, 0.06f * ch, ch) + margin : (float)TRUE_PI;
                    gam = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(a)));
                } else {
                    ctr = make_float3(0.f, 0.f, 1.f);
                }
                if (cone.w >= 3.f) gam = (float)TRUE_PI;  // directions that are not unit vectors: no angle bounds
            }
            // range of the cosines the directions' cone allows (only the order depends on it)
            float chi, bscale;
            {
                const float al = acosf(fminf(fmaxf(cone.x * ctr.x + cone.y * ctr.y + cone.z * ctr.z, -1.f), 1.f));
                chi = __cosf(fmaxf(al - cone.w, 0.f));
                bscale = SW_BUCKETS / fmaxf(chi - __cosf(fminf(al + cone.w, (float)TRUE_PI)), 1e-6f);
            }
            order_waves(sm, kw4 + w0, phs, nkb, ctr, chi, bscale);
            for (int g = warp; g < G; g += 8) {
                const float4 k = sm.k[32 * g + lane];
                const float c = fmaf(k.x, ctr.x, fmaf(k.y, ctr.y, k.z * ctr.z)) + 4.f;  // positive: ordered as bits
                const float lo = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(c))) - 4.f;
                const float hi = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(c))) - 4.f;
                const float2 t = f2_unpack(theta_column2(f2_pack(hi, lo), f2_splat(-tsc), f2_splat(hp_hi)));
                if (lane == 0) sm.gb[g] = t;
            }
            __syncthreads();
            if (warp == 0) staged_units += plan_bands(sm, G, nkb, thetaR, tsc, gam, tile_rdist, STAGE ? chunk : 0);
            __syncthreads();
#pragma unroll 1
            for (int r = 0; r < 2; r++) {
                if (tv + 2 * warp + r >= sc.R) break;
                const PixRow* px = &sm.px[warp][16 * r];
                float ar[16], ai[16];
#pragma unroll
                for (int j = 0; j < 16; j++) ar[j] = ai[j] = 0.f;
                int g0 = 0;
                while (g0 < G) {
                    const int4 band = sm.band[g0];
                    const int t_lo = band.x, g1 = band.y & 255, shape = band.y >> 8 & 3, width = band.y >> 16;
                    const int mode = band_mode(__int_as_float(band.z) * sm.rdist[warp][r], shape);
                    // the blended rows of part h of the row: pixels i and 15 - i, i in [8 h / parts, 8 (h + 1) / parts)
                    auto stage = [&](auto sh, int h) {
                        constexpr int S = decltype(sh)::value, NP = 16 >> S, W = SW_W << S;
                        __syncwarp();  // readers of the previous window are done
#pragma unroll 1
                        for (int c = 2 * lane; c <= width; c += 64) {
                            if (t_lo + c + 2 > row_len) break;
                            const float2* src = tab + t_lo + c;
                            float2* dst = &sm.win[warp][c];
#pragma unroll 1
                            for (int e0 = 0; e0 < NP; e0 += SW_BATCH) {
                                ulonglong2 a[SW_BATCH], b[SW_BATCH];
                                float al_[SW_BATCH];
#pragma unroll
                                for (int q = 0; q < SW_BATCH; q++) {
                                    const int sl = e0 + q, i = h * (NP / 2) + (sl >> 1);
                                    const PixRow pr = px[sl & 1 ? 15 - i : i];
                                    a[q] = __ldg(reinterpret_cast<const ulonglong2*>(src + pr.off));
                                    b[q] = __ldg(reinterpret_cast<const ulonglong2*>(src + pr.off + row_len));
                                    al_[q] = pr.al;
                                }
#pragma unroll
                                for (int q = 0; q < SW_BATCH; q++) {
                                    const f32x2 al = f2_splat(al_[q]);
                                    ulonglong2 v;
                                    v.x = f2_fma(al, f2_sub(b[q].x, a[q].x), a[q].x);
                                    v.y = f2_fma(al, f2_sub(b[q].y, a[q].y), a[q].y);
                                    *reinterpret_cast<ulonglong2*>(dst + (e0 + q) * W) = v;
                                }
                            }
                        }
                        __syncwarp();
                    };
                    const f32x2 ntsc = f2_splat(-tsc), hb = f2_splat(column_base(hp_hi, hp_lo, tsc, t_lo));
                    // polynomial coefficients of a direction's column along the row (x = +-(7.5 - i) / 7.5)
                    auto node = [&](float4 k, int n) {
                        const float4 xy = sm.node[warp][r][2 * n];
                        const float2 z = *reinterpret_cast<const float2*>(&sm.node[warp][r][2 * n + 1]);
                        return f2_unpack(theta_column2(
                            f2_fma(f2_splat(k.x), f2_pack(xy.x, xy.y),
                                   f2_fma(f2_splat(k.y), f2_pack(xy.z, xy.w), f2_fma(f2_splat(k.z), f2_pack(z.x, z.y), 0ull))),
                            ntsc, hb));
                    };
                    auto coefs = [&](auto nc, float4 k, float (&a)[6]) {
                        if constexpr (decltype(nc)::value == 4) {
                            const float2 u = node(k, 0), v = node(k, 1);
                            const float e0 = 0.5f * (u.x + u.y), e1 = 0.5f * (v.x + v.y);
                            const float o0 = (u.x - u.y) * 0.541196100f, o1 = (v.x - v.y) * 1.306562965f;
                            a[2] = (e0 - e1) * 1.414213562f, a[0] = fmaf(a[2], -0.146446609f, e1);
                            a[3] = (o0 - o1) * 1.414213562f, a[1] = fmaf(a[3], -0.146446609f, o1);
                        } else if constexpr (decltype(nc)::value == 6) {
                            const float2 u = node(k, 2), v = node(k, 3), w = node(k, 4);
                            const float y0 = 0.933012702f, y1 = 0.5f, y2 = 0.066987298f;
                            auto poly = [&](float f0, float f1, float f2, float& c0_, float& c2_, float& c4_) {
                                const float b1 = (f1 - f2) * (1.f / (y1 - y2));
                                c4_ = ((f0 - f1) * (1.f / (y0 - y1)) - b1) * (1.f / (y0 - y2));
                                c2_ = fmaf(c4_, -(y1 + y2), b1);
                                c0_ = fmaf(b1, -y2, fmaf(c4_, y1 * y2, f2));
                            };
                            poly(0.5f * (u.x + u.y), 0.5f * (v.x + v.y), 0.5f * (w.x + w.y), a[0], a[2], a[4]);
                            poly((u.x - u.y) * 0.517638090f, (v.x - v.y) * 0.707106781f, (w.x - w.y) * 1.931851653f, a[1],
                                 a[3], a[5]);
                        }
                    };
                    auto column = [&](auto nc, const float (&a)[6], float4 k, int i) {
                        const float x = (SW_HALF - i) / SW_HALF;
                        float ev = 0.f, od = 0.f;
                        if constexpr (decltype(nc)::value == 4) {
                            ev = fmaf(a[2], x * x, a[0]), od = fmaf(a[3], x * x, a[1]);
                        } else if constexpr (decltype(nc)::value == 6) {
                            ev = fmaf(fmaf(a[4], x * x, a[2]), x * x, a[0]);
                            od = fmaf(fmaf(a[5], x * x, a[3]), x * x, a[1]);
                        } else {  // an arc cosine per pixel
                            const float4 xy = sm.dir[warp][r][2 * i], zc = sm.dir[warp][r][2 * i + 1];
                            return f2_unpack(theta_column2(
                                f2_fma(f2_splat(k.x), f2_pack(xy.x, xy.y),
                                       f2_fma(f2_splat(k.y), f2_pack(xy.z, xy.w),
                                              f2_fma(f2_splat(k.z), f2_pack(zc.x, zc.y), f2_pack(zc.z, zc.w)))),
                                ntsc, hb));
                        }
                        return make_float2(fmaf(-x, od, ev), fmaf(x, od, ev));
                    };
                    auto add = [&](float2 pw, int j, float2 a, float2 c, float be) {
                        const float vr = fmaf(be, c.x - a.x, a.x), vi = fmaf(be, c.y - a.y, a.y);
                        ar[j] = fmaf(-pw.y, vi, fmaf(pw.x, vr, ar[j]));
                        ai[j] = fmaf(pw.y, vr, fmaf(pw.x, vi, ai[j]));
                    };
                    auto look = [&](auto sh, float2 pw, int i, float2 tt) {  // pixels i and 15 - i from the window
                        constexpr int S = decltype(sh)::value, NP = 16 >> S, W = SW_W << S;
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const int j = h ? 15 - i : i;
                            const float tj = h ? tt.y : tt.x;
                            // adding 1.5 2^23, rounded down, leaves floor(t); adding 1.5 2^20 leaves 8 floor(t) in
                            // the low bits but the last three.  Inside the window by construction; the mask
                            // keeps any column in it
                            const float be = tj - (__fadd_rd(tj, 12582912.f) - 12582912.f);
                            const unsigned o = (__float_as_uint(__fadd_rd(tj, 1572864.f)) & (8u * (W - 1))) | win0;
                            const float2* e = reinterpret_cast<const float2*>(
                                reinterpret_cast<const char*>(&sm.win[0][0]) + o + 8 * W * (2 * (i % (NP / 2)) + h));
                            add(pw, j, e[0], e[1], be);
                        }
                    };
                    auto part = [&](auto nc, auto sh, auto hh) {
                        constexpr int NI = 8 >> decltype(sh)::value, I0 = decltype(hh)::value * NI;
                        stage(sh, decltype(hh)::value);
#pragma unroll 1
                        for (int g = g0; g < g1; g++) {
                            // keeps the row's node and pixel directions in shared memory: held in registers over
                            // this loop they spill the sums (24.6 against 22.6 ms, 3072^2 pixels x 2 spheres)
                            asm volatile("" ::: "memory");
                            float a[6];
                            const float2 pa = sm.p[32 * g + lane];
                            const float4 k = sm.k[32 * g + lane];
                            coefs(nc, k, a);
#pragma unroll
                            for (int i = 0; i < NI; i++) look(sh, pa, I0 + i, column(nc, a, k, I0 + i));
                        }
                    };
                    auto rows = [&](auto nc, auto sh) {
                        constexpr int S = decltype(sh)::value;
                        part(nc, sh, Int<0>{});
                        if constexpr (S > 0) part(nc, sh, Int<1>{});
                        if constexpr (S > 1) {
                            part(nc, sh, Int<2>{});
                            part(nc, sh, Int<3>{});
                        }
                    };
                    auto by_mode = [&](auto sh) {
                        constexpr int S = decltype(sh)::value;
                        if constexpr (S < 2)
                            if (mode == 4) {
                                rows(Int<4>{}, sh);
                                return;
                            }
                        if constexpr (S == 0)
                            if (mode == 6) {
                                rows(Int<6>{}, sh);
                                return;
                            }
                        rows(Int<0>{}, sh);
                    };
                    if (STAGE && shape == 1) {
                        by_mode(Int<0>{});
                    } else if (STAGE && shape == 2) {
                        by_mode(Int<1>{});
                    } else if (STAGE && shape == 3) {
                        by_mode(Int<2>{});
                    } else {
#pragma unroll 1
                        for (int g = g0; g < g1; g++) {
                            const float4 k = sm.k[32 * g + lane];
                            const float2 pw = sm.p[32 * g + lane];
                            float a[6];
                            if (mode == 4) coefs(Int<4>{}, k, a);
                            if (mode == 6) coefs(Int<6>{}, k, a);
#pragma unroll
                            for (int i = 0; i < 8; i++) {
                                const float2 t = mode == 4 ? column(Int<4>{}, a, k, i)
                                                           : mode == 6 ? column(Int<6>{}, a, k, i) : column(Int<0>{}, a, k, i);
#pragma unroll
                                for (int h = 0; h < 2; h++) {
                                    const int j = h ? 15 - i : i;
                                    const float tj = h ? t.y : t.x, tf = floorf(tj);
                                    const int n = min(max(t_lo + (int)tf, 0), thetaR - 1);
                                    const PixRow q = px[j];
                                    const f32x2* e = reinterpret_cast<const f32x2*>(tab + (size_t)(q.off + (unsigned)n));
                                    const f32x2 al = f2_splat(q.al);
                                    const f32x2 e00 = e[0], e01 = e[1], e10 = e[row_len], e11 = e[row_len + 1];
                                    add(pw, j, f2_unpack(f2_fma(al, f2_sub(e10, e00), e00)),
                                        f2_unpack(f2_fma(al, f2_sub(e11, e01), e01)), tj - tf);
                                }
                            }
                        }
                    }
                    g0 = g1;
                }
                // ---- the lanes' sums: 16 pixels x (re, im) reduced over 32 lanes, value L to lane L ----
                float v[32];
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    v[2 * j] = ar[j];
                    v[2 * j + 1] = ai[j];
                }
#pragma unroll
                for (int m = 16; m >= 1; m >>= 1) {
                    const bool up = lane & m;
#pragma unroll
                    for (int i = 0; i < m; i++) {
                        const float send = up ? v[i] : v[i + m], keep = up ? v[i + m] : v[i];
                        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
                    }
                }
                                // Kahan: add the sphere's sum to the running total
                const float2 a = sm.acc[warp][r][lane];
                const float y = v[0] - a.y, t = a.x + y;
                sm.acc[warp][r][lane] = make_float2(t, (t - a.x) - y);
            }
        }
    }
    if (threadIdx.x == 0 && counters) {
        atomicAdd(counters, (unsigned long long)staged_units);
        atomicAdd(counters + 1, (unsigned long long)max(se - sb, 0) * ((sc.nk + chunk - 1) / chunk));
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int lv = 2 * warp + r, lu = (lane >> 1), opx = tu + lu, iv = tv + lv;
        if (opx >= sc.R || iv >= sc.R) continue;
        float2 a = sm.acc[warp][r][lane];
        const size_t o = 2 * ((size_t)iv * sc.R + opx) + (lane & 1);
        if (finalize && !part) {
            double p[3];
#pragma unroll
            for (int c = 0; c < 3; c++) p[c] = __dadd_rn(sm.pa[c][lu], sm.pb[c][lv]);
            if (outside_all(sc, sph, p)) a.x += reinterpret_cast<const float*>(Uf)[o] - a.y;
        } else if (comp) {
            comp[o] = a.y;
        }
        sum[o] = a.x;
    }
}

// The shares' sums added in order (Kahan), and Uf where the pixel is outside every sphere.
__global__ void __launch_bounds__(128) us_lut_join_kernel(Scene sc, const Sphere* __restrict__ sph, int shares,
                                                          const float* __restrict__ part,
                                                          const cpx<float>* __restrict__ Uf, cpx<float>* __restrict__ U) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= sc.R * sc.R) return;
    const size_t plane = (size_t)sc.R * sc.R;
    const float2* v = reinterpret_cast<const float2*>(part) + idx;
    float2 tot = make_float2(0.f, 0.f), cmp = tot;
    auto add = [&](float2 a) {
        const float yr = a.x - cmp.x, yi = a.y - cmp.y, tr = tot.x + yr, ti = tot.y + yi;
        cmp = make_float2((tr - tot.x) - yr, (ti - tot.y) - yi);
        tot = make_float2(tr, ti);
    };
    for (int q = 0; q < shares; q++, v += 2 * plane) {
        add(v[0]);
        add(make_float2(-v[plane].x, -v[plane].y));
    }
    double p[3];
    pixel_pos(sc, idx % sc.R, idx / sc.R, p);
    if (outside_all(sc, sph, p)) {
        tot.x += Uf[idx].re - cmp.x;
        tot.y += Uf[idx].im - cmp.y;
    }
    U[idx] = mk(tot.x, tot.y);
}

// The spheres of a slice are shared out over blocks: a small grid leaves SMs with one block of 8 warps or none,
// the tiles' work differs and two blocks at a time leave a long tail on grids of a few rounds, and blocks that
// work on the same few spheres find their tables (34 MB each at 4096 x 1024) in L2.  About 128 blocks per SM;
// from 64 tiles per SM on the sums' memory (16 bytes a pixel and share) is not worth it, see lut_ranges.  A
// sphere's share depends on the slice alone, so that chunked tables give the bits of one launch.  Scattered
// field in one share, 4 blocks per SM and 128: 192^2 pixels, 12 spheres, 400 directions 1.16, 0.70 and 0.59 ms;
// 384^2, 50, 200: 7.2, 7.2 and 6.0 ms; 768^2, 120, 1000: 115, 115 and 102 ms.
int lut_splits(int R, int ns, int nk) {
    const long long tiles = (long long)((R + 15) / 16) * ((R + 15) / 16);
    if (lut_plain(ns) || lut_few(ns, nk) || tiles >= 64 * GB300_SMS) return 1;
    return (int)std::max(1LL, std::min({(long long)ns, 16LL, (128 * GB300_SMS + tiles - 1) / tiles}));
}

// Launches the spheres of a chunk are spread over where lut_splits gives one share: each with about twice the L2
// cache's size of tables, up to 8.  3072^2 pixels, 50 spheres with 34 MB each: 576 ms in one launch, 563 in 6.
int lut_ranges(int R, int ns, int nk, size_t table_bytes) {
    if (lut_plain(ns) || lut_few(ns, nk) || lut_splits(R, ns, nk) > 1) return 1;
    return (int)std::max<size_t>(1, std::min<size_t>(std::min(ns, 8), table_bytes >> 28));
}

void launch_us_lut_mixed(const Scene& sc, const Sphere* sph, int s0, int s1, int accumulate, int finalize,
                         const float4* kw4, const cpx<float>* ph, const float2* lin, const cpx<float>* Uf,
                         cpx<float>* U, unsigned long long* counters, float2* kcmp, float* part, bool stage, int chunk,
                         float4 cone, float margin, cudaStream_t st) {
    const unsigned tiles = (sc.R + 15) / 16;
    const int shares = part ? lut_splits(sc.R, sc.ns, sc.nk) : 1;
    // per device and cheap; a failure shows up as the launch error
    auto kernel = stage ? us_lut_sorted_kernel<true> : us_lut_sorted_kernel<false>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SW_SMEM);
    kernel<<<dim3(tiles * tiles, shares), SW_NT, SW_SMEM, st>>>(sc, sph, s0, s1, accumulate, finalize, kw4, ph,
                                                                         lin, Uf, U, counters, kcmp, part, chunk, cone, margin);
    if (part && finalize)
        us_lut_join_kernel<<<(sc.R * sc.R + 127) / 128, 128, 0, st>>>(sc, sph, shares, part, Uf, U);
}

// Loads every kernel of this file (cudaFuncGetAttributes), see preload_nearfield_kernels.
void preload_uslut_kernels() {
    cudaFuncAttributes a;
    cudaFuncGetAttributes(&a, us_lut_sorted_kernel<true>);
    cudaFuncGetAttributes(&a, us_lut_sorted_kernel<false>);
    cudaFuncGetAttributes(&a, us_lut_join_kernel);
}

}  // namespace bs
