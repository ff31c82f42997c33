// bs_kernels.h -- launchers of the CUDA kernels (bs_nearfield.cu, bs_detector.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "bs_internal.h"

namespace bs {

// Mixed LUT kernels: angle margins (radians) of the sorted and of the plain kernel's window bounds.
constexpr float LUT_STAGE_MARGIN = 5e-4f;
constexpr float LUT_PLAIN_MARGIN = 2e-3f;
constexpr int GB300_SMS = 152;
constexpr int SMEM_OPTIN = 227 * 1024;  // most shared memory of a block
constexpr int LUT_TILE = 16;
constexpr int LUT_WINDOW = 256;  // table columns of the widest staged window
constexpr int WAVE_CHUNK_MAX = 64;
// Slices whose mixed scattered field the plain kernel sums (bs_uslut_plain.cu), from tables summed in double
// precision, with the directions' order and chunks.  The absorbance of a slice with little contrast is a small
// difference of two float images, and hangs on the order of the sums: with the sorted kernel's, over lanes, it moves
// by more than 2e-5 in 17 of 782 drawn slices, all of at most 4 spheres (699 slices of more than 8: by 1.6e-5 at
// most).  768^2 pixels, one sphere, 400 directions: 1.08 ms sorted, 1.73 ms plain.
constexpr int LUT_PLAIN_SPHERES = 8;
inline bool lut_plain(int ns) { return ns <= LUT_PLAIN_SPHERES; }
// More spheres with few directions: the plain kernel too, without windows and from the sorted kernel's tables.  Two
// groups of 32 directions do not pay for the sorted kernel's ordering and blending; scattered field plain and sorted,
// 20 spheres, 1536^2 pixels, 33 and 64 directions: 6.5 and 18.3, 11.1 and 16.8 ms; 768^2: 1.8 and 4.5, 3.0 and
// 4.3 ms; 192^2: 0.25 and 0.35, 0.38 and 0.34 ms.  Each direction more adds 1/64 of the plain figure, 32 more less
// than a sixth of the sorted one.
constexpr int LUT_FEW_WAVES = 64;
inline bool lut_few(int ns, int nk) { return !lut_plain(ns) && nk <= LUT_FEW_WAVES; }
// Float2 values of the plain kernel's staged windows: 51 KB with 64-wave chunks (4 blocks per SM), 72 KB (3) with
// smaller ones.
__host__ __device__ constexpr int lut_plain_entries(int chunk) { return chunk >= 64 ? 6400 : 9000; }
// Shared-memory row stride of such a window W entries wide: odd, so that lanes reading the same column of different
// rows fall in different banks.
__host__ __device__ constexpr int lut_plain_stride(int W) { return W | 1; }

template <class T>
struct cpx;
using zd = cpx<double>;

// Load every kernel of the library into the current device's context now: with
// CUDA's default lazy loading a kernel is loaded at its first launch, and a load
// while other streams' kernels run waits for them (a served request that was the
// first to use a kernel waited for the long slices on the other workers' streams:
// p50 8.3 s against 1.9 s with every kernel loaded up front).
void preload_nearfield_kernels();
void preload_uslut_kernels();
void preload_uslut_plain_kernels();
void preload_detector_kernels();

// One bilinear LUT cell at (r, t): {T00, T10 - T00, T01 - T00, T11 - T10 - T01 + T00}
// as (re, im) pairs, so that T(r + a, t + b) = (v0 + a v1) + b (v2 + a v3).
template <class T>
struct alignas(8 * sizeof(T)) Patch {
    T v[8];
};

// ---- near field ----
template <class T>
void launch_uf(const Scene& sc, const double* tab, const UfOrder* w, cpx<T>* Uf, cudaStream_t st);
void launch_uf_table(const Scene& sc, double* tab, double* scratch, cudaStream_t st);
void launch_mie(const Sphere* sph, int ns, double k, zd* A, zd* B, cudaStream_t st);
// spheres [s0, s0 + n) in one launch; starts (device): first global row of each
// sphere (n + 1 values, the last = total_rows) then first coefficient (n values);
// scratch: 2 doubles per coefficient; bias (device, one float per row) selects the mixed path's split coefficients
struct SplitCoef {
    float hr, hi, lr, li;  // a complex coefficient: nearest floats and the rests; the size of a zd
};
void launch_coef_rows_batch(const Sphere* sph, int s0, int n, const long long* starts, long long total_rows, double k,
                            const zd* A, const zd* B, zd* tab, double* scratch, float* bias, cudaStream_t st);
// Legendre values of the mixed path: P[l * stride + t] = {nearest float, rest}
void launch_legendre_split(int thetaR, int Lmax, int stride, float2* P, cudaStream_t st);
void launch_legendre_table(int thetaR, int Lmax, double* P, cudaStream_t st);
template <class T>
void launch_phase(const Scene& sc, const Sphere* sph, const double* waves, cpx<T>* ph, float4* kw4, cudaStream_t st);
// Nodes of the double-precision arc cosine at j pi / ACOS_NODES: the cosine c, the angle t in columns of a table of
// thetaR angles, and d1 .. d4 of the column t + d1 y + d2 y^2 + d3 y^3 + d4 y^4 at the cosine c - y
// (us_lut_f64_kernel); ACOS_NODES + 1 of them, then the numbers 0 .. thetaR - 1 as doubles.
constexpr int ACOS_NODES = 16384;
struct alignas(16) AcosNode {
    double c, t, d1, d2, d3, d4;
};
void launch_acos_nodes(int thetaR, AcosNode* nodes, cudaStream_t st);
void launch_us_lut_f64(const Scene& sc, const Sphere* sph, int s0, int s1, int accumulate, int finalize,
                       const double* waves, const AcosNode* nodes, const zd* ph, const Patch<double>* lut, const zd* Uf,
                       zd* U, cudaStream_t st);
// mixed path.  lin: linear float2 tables (Sphere::usp_off / uip_off in float2 units, rows
// of Sphere::lin_stride entries, even and 16-byte aligned);
// counters[0..1] receive the staged and total (tile, sphere, chunk of `chunk` waves) counts
// (may be null); kcmp (R x R, or null with a single sphere chunk) carries each pixel's Kahan
// compensation from one sphere chunk's launch to the next, so that chunked
// tables give the bits of one launch over all spheres;
// stage = false reads every cell from the tables; cone: axis and half-angle of a cone that holds
// every direction (half-angle pi: directions that are not unit vectors); margin: added to the tiles' angular radii
void launch_us_lut_mixed(const Scene& sc, const Sphere* sph, int s0, int s1, int accumulate, int finalize,
                         const float4* kw4, const cpx<float>* ph, const float2* lin, const cpx<float>* Uf,
                         cpx<float>* U, unsigned long long* counters, float2* kcmp, float* part, bool stage, int chunk,
                         float4 cone, float margin, cudaStream_t st);
// the same field by the plain kernel (lut_plain, lut_few): the waves in chunks of `chunk`, one bounding cone {axis,
// half-angle} per chunk (read with `stage` only); counters in chunks of counted_chunk waves
void launch_us_lut_plain(const Scene& sc, const Sphere* sph, int s0, int s1, int accumulate, int finalize,
                         const float4* kw4, const float4* cones, const cpx<float>* ph, const float2* lin,
                         const cpx<float>* Uf, cpx<float>* U, unsigned long long* counters, float2* kcmp, bool stage,
                         int chunk, int counted_chunk, cudaStream_t st);
// Shares of the spheres that launch_us_lut_mixed runs side by side; above 1, `part` (else null) holds
// 4 floats per pixel and share.
int lut_splits(int R, int ns, int nk);
// Launches of launch_us_lut_mixed, over parts of the spheres, for spheres with `table_bytes` of tables in all.
int lut_ranges(int R, int ns, int nk, size_t table_bytes);
// One table of the mixed path's table build: the rows of one sphere's Usp or Uip with their
// coefficient rows at tab + tab_off and biases at bias + row_off, written to the linear rows at
// lin + lin_off.
struct LutBuildJob {
    long long tab_off, lin_off, row_off;
    int rows, L, thetaR, lin_stride;
    int last;  // rows above this one repeat it (a Uip of one row is stored twice)
};
// the tables of `jobs` (device array of njobs <= 65535 entries, at most max_rows rows and max_theta
// angles each) in one launch; tab holds SplitCoef entries
void launch_lut_build_mixed(const LutBuildJob* jobs, int njobs, int max_rows, int max_theta, const zd* tab,
                            const float* bias, const float2* P, int Pstride, float2* lin, cudaStream_t st);

// the same in double precision, rounded, for the plain kernel's tables; tab holds zd entries
void launch_lut_build_plain(const LutBuildJob* jobs, int njobs, int max_rows, int max_theta, const zd* tab,
                            const double* P, int Pstride, float2* lin, cudaStream_t st);
// the same in double precision, as bilinear patches at out + lin_off
void launch_lut_build(const LutBuildJob* jobs, int njobs, int max_rows, int max_theta, const zd* tab, const double* P,
                      int Pstride, Patch<double>* out, cudaStream_t st);

// Direct scattered field through the addition theorem of spherical harmonics:
// recurrence factors rec (L(L+1)/2), per-wave tables tab (nk x L(L+1)/2, then the ns x nk
// phases), per-sphere
// coefficients coef (ns x {outside, inside} x L(L+1)/2 x 2 complex, with the Mie
// coefficients B, A), then the per-pixel sum.
struct ShRec {
    double a, b, beta, kappa, zero;
};
struct ShFrame {
    double e1[3], e2[3], e3[3];  // the harmonics' axes: e3 the slice's normal
};
void launch_sh_tables(const Scene& sc, const Sphere* sph, int L, const double* waves, ShRec* rec, double2* tab,
                      const zd* A, const zd* B, zd* coef, cudaStream_t st);
template <class T>
void launch_us_sh(const Scene& sc, const Sphere* sph, int L, const ShRec* rec, const zd* coef, const cpx<T>* Uf, cpx<T>* U, cudaStream_t st);
template <class T>
void launch_sum_only(const Scene& sc, const Sphere* sph, const cpx<T>* Uf, cpx<T>* U, cudaStream_t st);
// U and Uf (src: U then Uf, R x R each) rotated about the slice centre into dst;
// c, s: cosine and sine of the angle
template <class T>
void launch_rotate_fields(int R, float c, float s, const cpx<T>* src, cpx<T>* dst, cudaStream_t st);

// ---- detector ----
// twiddles: out[i * ld_i + j * ld_j] = exp(sign 2 pi i ((off_i + i) * freq[j] mod R) / R)
template <class T>
void launch_twiddle(int ni, int nj, const int* freq, int off_i, int R, int sign, int ld_i, int ld_j, cpx<T>* out,
                    cudaStream_t st);

// C[b] (M x N) = A[b] (M x K) * B[b] (K x N), complex, row-major, batch over
// blockIdx.z with element strides sA, sB, sC (0 = shared operand).
// epi 0: store; epi 1: multiply by mask[m*N + n]; epi 2: store |scale * c|^2
// into the real array I[b] (M x N, batch stride sC); epi 3: store scale * c.
// GEMMs with fewer output tiles than SMs split K over more blocks and add the
// parts in a fixed order (deterministic) when `scratch` holds
// cgemm_scratch_elems(M, N, K, batch) elements; else one block per tile.
template <class T>
size_t cgemm_scratch_elems(int M, int N, int K, int batch);
template <class T>
void launch_cgemm(int M, int N, int K, int batch, const cpx<T>* A, int lda, long long sA, const cpx<T>* B, int ldb,
                  long long sB, cpx<T>* C, int ldc, long long sC, int epi, const float* mask, T scale, T* I,
                  cpx<T>* scratch, size_t scratch_elems, cudaStream_t st);

// Double-precision forward transform of the rows x_0 .. x_{R-1} of a batch of M x R arrays, the bins 0 .. npos - 1
// and R - nneg .. R - 1 (stored in that order): bin j of row m to C[b sC + m row_stride + j bin_stride], times
// mask[m row_stride + j bin_stride] unless mask is null.  nh = max(npos, nneg + 1); tab of launch_fold_table holds
// ldt >= nh columns; scratch fold_scratch_elems.
struct FoldDft {
    int M, R, npos, nneg, nh, lda, ldt, row_stride, bin_stride;
    long long sA, sC;
};
void launch_fold_table(int R, int nh, zd* tab, cudaStream_t st);
size_t fold_scratch_elems(const FoldDft& f, int batch);
void launch_fold_dft(const FoldDft& f, int batch, const zd* A, const zd* tab, zd* C, const float* mask, zd* scratch,
                     cudaStream_t st);

// D[b][iv][iu] (+)= sum over the ss x ss block of I[b] / ss^2 (fieldslice.cu:71-108);
// accumulate adds to D (the detector sums point sources)
template <class T>
void launch_bin(int res, int ss, int batch, int accumulate, const T* I, T* D, cudaStream_t st);

// Ring point sources on the detector (microscope.cu:37-250): dst[b] += src[b]
// rotated by (c, s) about ((int)(res/2), (int)(res/2)), b = 0, 1; line[b][r] +=
// the tree sum of src[b] at radius r, angles with (cos, sin) cs[k], k < points
// (points <= 1023); D[b] = line[b] interpolated at each pixel's radius.
template <class T>
void launch_rotate_add_images(int res, float c, float s, const T* src, T* dst, cudaStream_t st);
template <class T>
void launch_ring_line(int res, int points, int L, const float2* cs, const T* img, T* line, cudaStream_t st);
template <class T>
void launch_line_image(int res, int L, const T* line, T* D, cudaStream_t st);

// Real part of the reference's FFT Hilbert transform of chi2 (N samples zero-padded
// to M) at the first N points, chi1; g is scratch of M doubles.
void launch_kk(int N, int M, const double* chi2, double* g, double* chi1, cudaStream_t st);

// x[i] *= a[i], i < n (complex)
template <class T>
void launch_cmul(int n, const cpx<T>* a, cpx<T>* x, cudaStream_t st);

// image kinds 2, 3: -log10(D/Di), D/Di (microscope.cu:722-775); 0, 1: copies
template <class T>
void launch_image(int n, int kind, const T* D, const T* Di, T* out, cudaStream_t st);

}  // namespace bs
