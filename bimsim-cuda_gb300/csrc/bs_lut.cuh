// bs_lut.cuh -- what the mixed-precision lookup-table kernels share.
#pragma once

#include "bs_geom.cuh"

namespace bs {

// Two single-precision lanes in one 64-bit register pair (low lane first), worked
// on by packed f32x2 instructions; each lane rounds exactly like the scalar one.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2_pack(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f32x2 f2_splat(float a) { return f2_pack(a, a); }
__device__ __forceinline__ float2 f2_unpack(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 f2_sub(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Whether a pixel lies outside every sphere (nfSumUf.cu:35).
__device__ __forceinline__ bool outside_all(const Scene& sc, const Sphere* __restrict__ sph, const double p[3]) {
    for (int s = 0; s < sc.ns; s++) {
        const Sphere& S = sph[s];
        // clearly outside in single precision (0.1 % margin on d^2), else the exact test
        const float dx = (float)(p[0] - S.p[0]), dy = (float)(p[1] - S.p[1]), dz = (float)(p[2] - S.p[2]);
        const float af = (float)S.a;
        if (dx * dx + dy * dy + dz * dz > 1.001f * af * af) continue;
        double r[3];
        if (dist_exact(p, S.p, r) < S.a) return false;
    }
    return true;
}

}  // namespace bs
