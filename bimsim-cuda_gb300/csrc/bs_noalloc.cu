// bs_noalloc.cu -- Mie coefficients for callers that cannot allocate device
// memory.
//
// bs_mie_noalloc computes the same coefficients as the context path
// (sphere::calcCoeff of the reference) but takes every buffer from the caller
// and allocates nothing: its Bessel work space is the blocks' shared memory.
// Callers that cannot call cudaMalloc include code running inside CUDA stream
// capture (where an allocation would end the capture), real-time or serving
// loops that reserve all memory up front, and frameworks whose memory belongs
// to their own pool allocator and must not be fragmented by a library.
#include <cuda_runtime.h>

#include "bimsim_gb300.h"
#include "bs_mie.cuh"

namespace bs {

void set_last_error(const char* msg);

namespace {

constexpr int NOALLOC_MAX_SPHERES = 256;
constexpr int NOALLOC_MAX_ORDER = 127;

// The sphere's own order count Nl = ceil(ka + 4 (ka)^(1/3) + 2) in single
// precision, in the order of sphere::calcNl (sphere.h:71-74) and of the host's
// calc_nl, with lambda = 2 PI / k rounded to float.  powf on the GPU may differ
// from the host's by an ulp, which changes Nl only when the sum lies within a
// few ulps of an integer.
__device__ int noalloc_calc_nl(double a_in, double k) {
    const float lam = (float)(2.0 * (double)3.14159f / k);
    const float pif = 3.14159f;
    float ka = __fmul_rn(2.0f, pif);
    ka = __fmul_rn(ka, (float)a_in);
    ka = __fdiv_rn(ka, lam);
    const float third = (float)(1.0 / 3.0);
    float v = __fmul_rn(4.0f, powf(ka, third));
    v = __fadd_rn(ka, v);
    v = __fadd_rn(v, 2.0f);
    return (int)ceilf(v);
}

__global__ void __launch_bounds__(MIE_NT) mie_noalloc_kernel(const double* __restrict__ sph, int nl_cap, double k,
                                                             zd* __restrict__ A, zd* __restrict__ B) {
    __shared__ MieShared sm;
    const int s = blockIdx.x;
    const double a = sph[3 * s], n_re = sph[3 * s + 1], n_im = sph[3 * s + 2];
    // Orders above the sphere's own Nl are not part of its series (the context
    // path never computes them); they are returned as zeros.  Evaluating them
    // would divide underflowed Bessel values (0/0, 0 * inf) for small spheres.
    const int nl = max(0, min(nl_cap, noalloc_calc_nl(a, k)));
    zd* As = A + (size_t)s * (nl_cap + 1);
    zd* Bs = B + (size_t)s * (nl_cap + 1);
    for (int l = nl + 1 + threadIdx.x; l <= nl_cap; l += MIE_NT) As[l] = Bs[l] = mk(0.0, 0.0);
    mie_block(sm, nl, a, mk(n_re, n_im), k, As, Bs);
}

}  // namespace
}  // namespace bs

extern "C" bs_status bs_mie_noalloc(const double* spheres, int32_t ns, int32_t nl, double k, double* A, double* B,
                                    void* stream) {
    using namespace bs;
    if (ns < 0 || ns > NOALLOC_MAX_SPHERES) {
        set_last_error("bs_mie_noalloc: sphere count outside 0..256 (the call takes 256 spheres)");
        return BS_ERR_ARG;
    }
    if (nl < 0 || nl > NOALLOC_MAX_ORDER) {
        set_last_error("bs_mie_noalloc: order outside 0..127 (the call takes 128 orders)");
        return BS_ERR_ARG;
    }
    if (!(k > 0)) {
        set_last_error("bs_mie_noalloc: wavenumber must be > 0");
        return BS_ERR_ARG;
    }
    if (ns > 0 && (!spheres || !A || !B)) {
        set_last_error("bs_mie_noalloc: null buffer");
        return BS_ERR_ARG;
    }
    if (ns == 0) return BS_OK;
    mie_noalloc_kernel<<<ns, MIE_NT, 0, (cudaStream_t)stream>>>(spheres, nl, k, (zd*)A, (zd*)B);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_last_error(cudaGetErrorString(e));
        return BS_ERR_CUDA;
    }
    return BS_OK;
}
