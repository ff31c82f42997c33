// bs_api.cu -- the C ABI of include/bimsim_gb300.h: context, device memory,
// the per-slice stage pipeline, and result readback.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <memory>
#include <string>
#include <type_traits>
#include <vector>

#include "bimsim_gb300.h"
#include "bs_internal.h"
#include "bs_kernels.h"
#include "bs_math.cuh"

using namespace bs;

namespace {

thread_local std::string g_err;

bs_status fail(bs_status st, const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    std::vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_err = buf;
    return st;
}

#define CK(x)                                                                                               \
    do {                                                                                                    \
        cudaError_t e_ = (x);                                                                               \
        if (e_ != cudaSuccess)                                                                              \
            return fail(e_ == cudaErrorMemoryAllocation ? BS_ERR_NOMEM : BS_ERR_CUDA, "%s failed: %s (%s:%d)", \
                        #x, cudaGetErrorString(e_), __FILE__, __LINE__);                                    \
    } while (0)

#define LAUNCHED(ctx)                                                                                   \
    do {                                                                                                \
        (ctx)->launches++;                                                                              \
        cudaError_t e_ = cudaGetLastError();                                                            \
        if (e_ != cudaSuccess)                                                                          \
            return fail(BS_ERR_CUDA, "kernel launch failed: %s (%s:%d)", cudaGetErrorString(e_), __FILE__, \
                        __LINE__);                                                                      \
    } while (0)

// A context's device buffer.  Allocation and release are stream-ordered on
// the owning context's stream (cudaMallocAsync / cudaFreeAsync): cudaFree
// would wait for every stream of the device, so a context growing a buffer
// would stall behind a long slice running on another context of the server.
struct DevBuf {
    void* p = nullptr;
    size_t n = 0;
    const cudaStream_t* st = nullptr;  // the owning context's stream (set by bs_create)
    cudaError_t ensure(size_t bytes) {
        if (bytes == 0) bytes = 256;
        if (bytes <= n) return cudaSuccess;
        release();
        cudaError_t e = st ? cudaMallocAsync(&p, bytes, *st) : cudaMalloc(&p, bytes);
        if (e == cudaSuccess) n = bytes;
        else p = nullptr;
        return e;
    }
    void release() {
        if (p) {
            if (st) cudaFreeAsync(p, *st);
            else cudaFree(p);
        }
        p = nullptr;
        n = 0;
    }
    template <class X>
    X* as() const {
        return reinterpret_cast<X*>(p);
    }
};

bool valid_params(const bs_params* p, std::string& why) {
    if (!(p->lambda > 0)) { why = "lambda must be > 0"; return false; }
    if (p->resolution <= 0) { why = "resolution must be > 0"; return false; }
    if (p->padding < 0) { why = "padding must be >= 0"; return false; }
    if (p->supersample < 1) { why = "supersample must be >= 1"; return false; }
    if (p->field_order < 0 || p->field_order > MAX_ORDER) { why = "field order out of range"; return false; }
    if (p->condenser[0] < 0 || p->condenser[1] > 1 || p->condenser[0] > p->condenser[1]) {
        why = "condenser NA must satisfy 0 <= NA_in <= NA_out <= 1"; return false;
    }
    long long R = (long long)p->resolution * p->supersample * (2LL * p->padding + 1);
    if (R > 65536) { why = "near-field resolution above 65536"; return false; }
    if (p->us_lut_r == 1 || p->us_lut_theta == 1 || p->uf_lut_r == 1 || p->us_lut_r < 0 || p->us_lut_theta < 0 ||
        p->uf_lut_r < 0) {
        why = "LUT sizes must be 0 (reference default) or >= 2"; return false;
    }
    return true;
}

}  // namespace

struct bs_ctx {
    bs_params prm{};
    std::vector<bs_sphere> spheres;
    std::vector<double> waves;
    bool waves_set = false;
    int device = 0;
    cudaStream_t st = nullptr;
    cudaEvent_t ev[6] = {};
    // The incident field and the transforms' tables, which the scattered field does not need, run beside the
    // Mie coefficients and lookup tables on a second stream (SideWork, made by the first run).
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr, uf_ev[2] = {};
    size_t budget = 0;  // LUT bytes allowed; 0 = automatic

    // derived per simulate
    Scene sc{};
    std::vector<Sphere> hs;
    int res = 0, ss = 1, crop = 0, off = 0, R = 0, Lmax = 1;
    int prec = -1;
    bool have = false;

    DevBuf d_sph, d_waves, d_kw4, d_ph, d_A, d_B, d_tab, d_tabscr, d_legP, d_lut, d_uft, d_uftscr;
    DevBuf d_cnt;           // staged / total counters of the mixed LUT kernels
    DevBuf d_cones;         // bounding cones of the plain mixed LUT kernel's wave chunks
    DevBuf d_far;           // far fields Ud, Ufd on request (bs_get_far_field)
    DevBuf d_starts;        // row / coefficient offsets of a coefficient batch
    DevBuf d_lbjobs, d_lbjobs2;  // Usp and Uip tables of a coefficient batch for the LUT builds
    DevBuf d_kcmp;               // Kahan compensation of the mixed LUT sums between sphere chunks
    DevBuf d_part;               // mixed LUT sums of the spheres' shares (lut_splits)
    DevBuf d_fsave;         // U, Uf of a ring's first source (bs_simulate_ring_interp)
    DevBuf d_dacc;          // detector sum of bs_simulate_ring_detector
    DevBuf d_line, d_ringcs;  // radial lines and ring (cos, sin) of bs_simulate_ring_line
    int det_Nv = 0;         // passband rows of the last detector run (0: no far field)
    DevBuf d_fields;  // [2][R*R] U then Uf
    DevBuf d_su, d_sv, d_mask, d_wx, d_wy, d_wix, d_wiy, d_f1, d_f2, d_g1, d_I, d_D, d_img;
    int legP_theta = 0, legP_L = 0;
    bool legP_split = false;  // d_legP holds the mixed path's order-major split values
    DevBuf d_bias;            // mixed path: bias of every coefficient row
    DevBuf d_acos;            // FP64 path: nodes of the arc cosine for acos_theta angles
    int acos_theta = 0;
    int tab_s0 = 0, tab_s1 = 0;  // spheres whose tables the last run left in d_lut
    int64_t launches = 0;
    int64_t interactions = 0;
    bs_stats stats{};
    // table reuse between runs (bs_set_lut_reuse)
    bool reuse = false;
    int stream_prio = 0;  // bs_set_stream_priority (0: the default priority)
    int lut_staging = 0;  // bs_set_lut_staging: 0, 1 staged kernel, 2 unstaged kernel
    int lut_chunk = 0;    // bs_set_lut_wave_chunk: 0 default, else waves per counted chunk
    bool bp_on = false;   // bs_set_backpropagation
    double bp_d = 0;
    DevBuf d_bp;          // back-propagation phase on the passband grid
    DevBuf d_shrec, d_shtab, d_shcoef;  // direct method: harmonic recurrences, per-wave and per-sphere tables
    DevBuf d_gscr;        // split-K parts of the detector GEMMs
    DevBuf d_ufw;         // condenser aperture factor per order of the incident field
    bool lut_valid = false;
    std::vector<double> lut_key;
};

// Every linear device buffer of a context.
static std::vector<DevBuf*> ctx_bufs(bs_ctx* c) {
    return {&c->d_sph, &c->d_waves, &c->d_kw4, &c->d_ph, &c->d_A, &c->d_B, &c->d_tab, &c->d_tabscr,
            &c->d_bias, &c->d_acos, &c->d_legP, &c->d_lut, &c->d_uft, &c->d_uftscr, &c->d_fields, &c->d_su,
            &c->d_sv, &c->d_mask, &c->d_wx, &c->d_wy, &c->d_wix, &c->d_wiy, &c->d_f1, &c->d_f2,
            &c->d_g1, &c->d_I, &c->d_D, &c->d_img, &c->d_cnt, &c->d_cones, &c->d_far,
            &c->d_starts, &c->d_lbjobs, &c->d_lbjobs2, &c->d_kcmp, &c->d_part, &c->d_fsave, &c->d_dacc, &c->d_line, &c->d_ringcs, &c->d_bp, &c->d_shrec, &c->d_shtab, &c->d_shcoef, &c->d_gscr, &c->d_ufw};
}

static void release_all(bs_ctx* c) {
    for (DevBuf* b : ctx_bufs(c)) b->release();
    c->legP_theta = c->legP_L = c->acos_theta = 0;
    c->lut_valid = false;
    c->have = false;
}

static size_t elem_r(int prec) { return prec == BS_PREC_FP64 ? sizeof(double) : sizeof(float); }

extern "C" {

const char* bs_version(void) { return "bimsim-gb300 0.1 (sm_103a)"; }

const char* bs_last_error(void) { return g_err.c_str(); }

}  // extern "C"

// Lets other translation units of the library report through bs_last_error().
namespace bs {
void set_last_error(const char* msg) { g_err = msg; }
}  // namespace bs

extern "C" {

// Every kernel loaded on the context's device before its first run (once per
// device and process; see preload_nearfield_kernels).
static void preload_kernels(int device) {
    static std::mutex mu;
    static std::vector<int> done;
    std::lock_guard<std::mutex> lock(mu);
    if (std::find(done.begin(), done.end(), device) != done.end()) return;
    preload_nearfield_kernels();
    preload_uslut_kernels();
    preload_uslut_plain_kernels();
    preload_detector_kernels();
    cudaGetLastError();  // a kernel this device cannot load reports at its launch instead
    done.push_back(device);
}

static void free_streams(bs_ctx* c) {
    for (cudaEvent_t e : c->ev)
        if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : {c->uf_ev[0], c->uf_ev[1], c->fork, c->join})
        if (e) cudaEventDestroy(e);
    if (c->side) cudaStreamDestroy(c->side);
    if (c->st) cudaStreamDestroy(c->st);
}

bs_status bs_create(const bs_params* params, bs_ctx** out) {
    if (!params || !out) return fail(BS_ERR_ARG, "bs_create: null argument");
    std::string why;
    if (!valid_params(params, why)) return fail(BS_ERR_ARG, "bs_create: %s", why.c_str());
    bs_ctx* c = new bs_ctx();
    c->prm = *params;
    cudaError_t e = cudaGetDevice(&c->device);
    if (e == cudaSuccess) preload_kernels(c->device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking);
    for (int i = 0; i < 6 && e == cudaSuccess; i++) e = cudaEventCreate(&c->ev[i]);
    for (DevBuf* b : ctx_bufs(c)) b->st = &c->st;
    if (e != cudaSuccess) {
        free_streams(c);
        delete c;
        return fail(BS_ERR_CUDA, "bs_create: %s", cudaGetErrorString(e));
    }
    *out = c;
    return BS_OK;
}

bs_status bs_destroy(bs_ctx* c) {
    if (!c) return BS_OK;
    if (c->st) cudaStreamSynchronize(c->st);
    release_all(c);
    if (c->st) cudaStreamSynchronize(c->st);  // the stream-ordered frees
    free_streams(c);
    delete c;
    return BS_OK;
}

bs_status bs_set_params(bs_ctx* c, const bs_params* params) {
    if (!c || !params) return fail(BS_ERR_ARG, "bs_set_params: null argument");
    std::string why;
    if (!valid_params(params, why)) return fail(BS_ERR_ARG, "bs_set_params: %s", why.c_str());
    c->prm = *params;
    c->have = false;
    return BS_OK;
}

bs_status bs_set_spheres(bs_ctx* c, const bs_sphere* s, int32_t n) {
    if (!c || n < 0 || (n > 0 && !s)) return fail(BS_ERR_ARG, "bs_set_spheres: bad arguments");
    for (int i = 0; i < n; i++)
        if (!(s[i].a > 0) || !std::isfinite(s[i].x) || !std::isfinite(s[i].y) || !std::isfinite(s[i].z))
            return fail(BS_ERR_ARG, "bs_set_spheres: sphere %d has a non-positive radius or bad centre", i + 1);
    c->spheres.assign(s, s + n);
    c->have = false;
    return BS_OK;
}

bs_status bs_set_waves(bs_ctx* c, const double* dirs, int32_t nk) {
    if (!c || nk < 1 || !dirs) return fail(BS_ERR_ARG, "bs_set_waves: need at least one direction");
    c->waves.assign(dirs, dirs + 3 * (size_t)nk);
    c->waves_set = true;
    c->have = false;
    return BS_OK;
}

bs_status bs_sample_waves_compat(bs_ctx* c, int32_t nk) {
    if (!c || nk < 1) return fail(BS_ERR_ARG, "bs_sample_waves_compat: nk must be >= 1");
    c->waves.resize(3 * (size_t)nk);
    mc_sample_compat(nk, c->prm.k_dir, c->prm.condenser[0], c->prm.condenser[1], c->waves.data());
    c->waves_set = true;
    c->have = false;
    return BS_OK;
}

bs_status bs_set_lut_budget(bs_ctx* c, size_t bytes) {
    if (!c) return fail(BS_ERR_ARG, "bs_set_lut_budget: null context");
    c->budget = bytes;
    return BS_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Derivation of the slice and sphere parameters (arguments.h:340-438,
// microscope.cu:700-718, sphere.cpp:222-240, nfScalarUpLut.cu:365-379)
// ---------------------------------------------------------------------------
static bs_status derive(bs_ctx* c) {
    const bs_params& p = c->prm;
    Quad det = quad_from(p.plane_min, p.plane_max, p.plane_normal);
    Quad nf = quad_scale(det, (double)(2 * p.padding + 1));
    c->res = p.resolution;
    c->ss = p.supersample;
    c->crop = c->res * c->ss;
    c->off = p.padding * c->crop;
    c->R = c->crop * (2 * p.padding + 1);
    Scene& sc = c->sc;
    sc = Scene{};
    const V3* v[3] = {&nf.A, &nf.X, &nf.Y};
    double* d[3] = {sc.A, sc.X, sc.Y};
    for (int i = 0; i < 3; i++) {
        d[i][0] = v[i]->x;
        d[i][1] = v[i]->y;
        d[i][2] = v[i]->z;
    }
    for (int i = 0; i < 3; i++) {
        sc.focus[i] = p.focus[i];
        sc.kdir[i] = p.k_dir[i];
    }
    sc.kmag = 2 * PI_REF / p.lambda;
    sc.amp = p.amplitude;
    sc.cos_a = std::cos(std::asin(p.condenser[0]));
    sc.cos_b = std::cos(std::asin(p.condenser[1]));
    sc.R = c->R;
    sc.m = p.field_order;
    sc.plane_wave = p.plane_wave;
    sc.lut_uf = p.lut_uf;
    sc.lut_us = p.lut_us;
    sc.scalar = p.scalar;
    if (p.plane_wave) {
        sc.nk = 1;
        sc.wave_amp = p.amplitude;
    } else {
        if (!c->waves_set)
            return fail(BS_ERR_STATE, "bs_simulate: no plane-wave directions (call bs_set_waves or bs_sample_waves_compat)");
        sc.nk = (int)(c->waves.size() / 3);
        double sub = 2 * PI_REF * p.amplitude * ((1 - sc.cos_b) - (1 - sc.cos_a));
        // the Monte Carlo weight is the reference's single-precision quotient 1.0f/nk
        // (nfScalarUs.cu:457, nfScalarUpLut.cu:83,89), kept in every precision
        sc.wave_amp = (double)(1.0f / (float)sc.nk) * sub;
    }
    V3 f{p.focus[0], p.focus[1], p.focus[2]};
    sc.uf_dmin = quad_dist(nf, f);
    sc.uf_dmax = quad_dist_max(nf, f);
    sc.uf_dR = p.uf_lut_r > 0 ? p.uf_lut_r : 2 * c->R;
    sc.uf_scale = (sc.uf_dR - 1) / (sc.uf_dmax - sc.uf_dmin);
    sc.invR = 1.0 / c->R;
    sc.ns = (int)c->spheres.size();
    c->hs.resize(sc.ns);
    double diag = v3_len(V3{nf.X.x + nf.Y.x, nf.X.y + nf.Y.y, nf.X.z + nf.Y.z});
    int coef = 0;
    c->Lmax = std::max(2, sc.m + 1);
    for (int i = 0; i < sc.ns; i++) {
        const bs_sphere& in = c->spheres[i];
        Sphere& S = c->hs[i];
        S = Sphere{};
        S.p[0] = in.x;
        S.p[1] = in.y;
        S.p[2] = in.z;
        S.a = in.a;
        S.n_re = in.n_re;
        S.n_im = in.n_im;
        S.Nl = calc_nl(in.a, p.lambda);
        if (S.Nl < 1 || S.Nl > MAX_ORDER) return fail(BS_ERR_ARG, "sphere %d: order %d out of range", i + 1, S.Nl);
        V3 ctr{in.x, in.y, in.z};
        S.dmin = quad_dist(nf, ctr);
        S.dmax = quad_dist_max(nf, ctr);
        double a_inter = (S.dmin < in.a) ? std::sqrt(in.a - S.dmin) : 0.0;  // sphere.cpp:231-233 (sic)
        S.aR = (int)(1 + 2.0 * c->R * a_inter / diag);
        S.dR = p.us_lut_r > 0 ? p.us_lut_r : 2 * c->R;
        S.thetaR = p.us_lut_theta > 0 ? p.us_lut_theta : 1000;
        S.r0 = std::max(in.a, S.dmin);
        S.xs_usp = (S.dR - 1) / (S.dmax - S.r0);
        S.xs_uip = (S.aR - 1) / (S.a - S.dmin);
        const double tsc = (S.thetaR - 1) / PI_REF, hp = 0.5 * TRUE_PI * tsc;
        S.tsc = (float)tsc;
        S.hp_hi = (float)hp;
        S.hp_lo = (float)(hp - (double)S.hp_hi);
        for (int k = 0; k < 3; k++) S.rel[k] = (float)(sc.A[k] - S.p[k]);
        S.coef_off = coef;
        coef += S.Nl + 1;
        c->Lmax = std::max(c->Lmax, S.Nl + 1);
    }
    return BS_OK;
}

// ---------------------------------------------------------------------------
// The band-limited detector (microscope.cu:495-526, 608-662)
// ---------------------------------------------------------------------------
// Frequency of FFT bin i as the reference's bandpass kernel assigns it (note
// -(R-1-i) rather than -(R-i) on the negative side).
static double bin_freq(int i, int R, double step) { return (i <= R / 2) ? i * step : -(double)(R - 1 - i) * step; }

// applyBackpropagation's factor -exp(i kz d) at spectrum bin (iu, iv) of an R x R near field, in the
// reference kernel's own arithmetic (microscope.cu:423-488): the momentum-space width Kx, its step
// dkx, kx, k and kz are single-precision variables, du, dv and lambda double, and the phase kz d a
// single-precision product; zero where kx^2 + ky^2 >= k^2, compared in single precision.
static void backprop_factor(int iu, int iv, int R, double du, double dv, double lambda, float d, double* re,
                            double* im) {
    const float two_pi = 2.0f * (float)PI_REF;  // 2*PI, PI = 3.14159f
    const float dkx = (float)((double)(two_pi * (float)R) * du) / (float)R;
    const float dky = (float)((double)(two_pi * (float)R) * dv) / (float)R;
    const float kx = (float)(iu <= R / 2 ? (double)iu * (double)dkx : -(double)(R - 1 - iu) * (double)dkx);
    const float ky = (float)(iv <= R / 2 ? (double)iv * (double)dky : -(double)(R - 1 - iv) * (double)dky);
    const float k = (float)((double)two_pi / lambda);
    const float kx_sq = kx * kx, ky_sq = ky * ky, k_sq = k * k;
    if (!(kx_sq + ky_sq < k_sq)) {
        *re = *im = 0.0;
        return;
    }
    const float kk = k * k, q = kk - kx_sq;
    const float kz = std::sqrt(q - ky_sq);
    const double ph = (double)(kz * d);
    *re = -std::cos(ph);
    *im = -std::sin(ph);
}

// Bins along u and v inside the objective's outer NA (the only ones the
// band-pass keeps), with the frequency steps.
static void passbands(const bs_ctx* c, std::vector<int>& su, std::vector<int>& sv, double& du, double& dv) {
    const int R = c->R;
    du = 1.0 / std::sqrt(c->sc.X[0] * c->sc.X[0] + c->sc.X[1] * c->sc.X[1] + c->sc.X[2] * c->sc.X[2]);
    dv = 1.0 / std::sqrt(c->sc.Y[0] * c->sc.Y[0] + c->sc.Y[1] * c->sc.Y[1] + c->sc.Y[2] * c->sc.Y[2]);
    const double hi = c->prm.objective[1] / c->prm.lambda;
    su.clear();
    sv.clear();
    for (int i = 0; i < R; i++) {
        if (std::fabs(bin_freq(i, R, du)) <= hi) su.push_back(i);
        if (std::fabs(bin_freq(i, R, dv)) <= hi) sv.push_back(i);
    }
}

// The folded forward transforms: fields [R][R] along x to f1 [Nu][R], f1 along y to f2 [Nv][Nu].  A passband is
// the bins 0 .. npos - 1 and R - nneg .. R - 1 (bin_freq is monotonic on both sides).
static FoldDft fold_dft(int R, const std::vector<int>& bins) {
    FoldDft f{};
    f.R = f.lda = R;
    while (f.npos < (int)bins.size() && bins[f.npos] <= R / 2) f.npos++;
    f.nneg = (int)bins.size() - f.npos;
    f.nh = std::max(f.npos, f.nneg + 1);
    return f;
}
static FoldDft fold_x(int R, const std::vector<int>& su, const std::vector<int>& sv) {
    FoldDft f = fold_dft(R, su);
    f.M = R;
    f.ldt = std::max(f.nh, fold_dft(R, sv).nh);
    f.row_stride = 1;
    f.bin_stride = R;
    f.sA = (long long)R * R;
    f.sC = (long long)su.size() * R;
    return f;
}
static FoldDft fold_y(int R, const std::vector<int>& su, const std::vector<int>& sv) {
    FoldDft f = fold_dft(R, sv);
    f.M = (int)su.size();
    f.ldt = std::max(f.nh, fold_dft(R, su).nh);
    f.row_stride = 1;
    f.bin_stride = (int)su.size();
    f.sA = (long long)su.size() * R;
    f.sC = (long long)su.size() * sv.size();
    return f;
}

// Elements of the split-K scratch of a slice's transforms
template <class T>
static size_t detector_scratch_elems(const FoldDft& fx, const FoldDft& fy, int Nu, int Nv, int C) {
    const int R = fx.R;
    const size_t fwd = sizeof(T) == 8 ? std::max(fold_scratch_elems(fx, 2), fold_scratch_elems(fy, 2))
                                      : std::max(cgemm_scratch_elems<T>(R, Nu, R, 2), cgemm_scratch_elems<T>(Nv, Nu, R, 2));
    return std::max(fwd, std::max(cgemm_scratch_elems<T>(Nv, C, Nu, 2), cgemm_scratch_elems<T>(C, C, Nv, 2)));
}

// The detector's device buffers and small host tables (passbands, mask), before the streams part.
template <class T>
static bs_status detector_buffers(bs_ctx* c) {
    const bs_params& p = c->prm;
    const int R = c->R;
    double du, dv;
    std::vector<int> su, sv;
    passbands(c, su, sv, du, dv);
    double lo = p.objective[0] / p.lambda, hi = p.objective[1] / p.lambda;
    auto freq = [R](int i, double step) { return bin_freq(i, R, step); };
    const int Nu = (int)su.size(), Nv = (int)sv.size(), C = c->crop, res = c->res;
    c->det_Nv = (Nu == 0) ? 0 : Nv;
    CK(c->d_D.ensure(2 * (size_t)res * res * sizeof(T)));
    if (Nu == 0 || Nv == 0) return BS_OK;
    std::vector<float> mask((size_t)Nv * Nu);
    for (int j = 0; j < Nv; j++)
        for (int k = 0; k < Nu; k++) {
            double u = freq(su[k], du), v = freq(sv[j], dv);
            double fm = std::sqrt(u * u + v * v);
            mask[(size_t)j * Nu + k] = (fm < lo || fm > hi) ? 0.f : 1.f;
        }
    size_t ce = sizeof(cpx<T>);
    CK(c->d_su.ensure(Nu * sizeof(int)));
    CK(c->d_sv.ensure(Nv * sizeof(int)));
    CK(c->d_mask.ensure(mask.size() * sizeof(float)));
    const FoldDft fx = fold_x(R, su, sv), fy = fold_y(R, su, sv);
    if (sizeof(T) == 8) {
        CK(c->d_wx.ensure((size_t)(R / 2 + 1) * fx.ldt * ce));
    } else {
        CK(c->d_wx.ensure((size_t)R * Nu * ce));
        CK(c->d_wy.ensure((size_t)Nv * R * ce));
    }
    CK(c->d_wix.ensure((size_t)Nu * C * ce));
    CK(c->d_wiy.ensure((size_t)C * Nv * ce));
    CK(c->d_f1.ensure(2 * (size_t)R * Nu * ce));
    CK(c->d_f2.ensure(2 * (size_t)Nv * Nu * ce));
    CK(c->d_g1.ensure(2 * (size_t)Nv * C * ce));
    CK(c->d_I.ensure(2 * (size_t)C * C * sizeof(T)));
    // split-K scratch for the GEMMs with few output tiles
    CK(c->d_gscr.ensure(std::max<size_t>(detector_scratch_elems<T>(fx, fy, Nu, Nv, C), 1) * ce));
    CK(cudaMemcpyAsync(c->d_su.p, su.data(), Nu * sizeof(int), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(c->d_sv.p, sv.data(), Nv * sizeof(int), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(c->d_mask.p, mask.data(), mask.size() * sizeof(float), cudaMemcpyHostToDevice, c->st));
    return BS_OK;
}

// The transforms' tables, on the stream st.
template <class T>
static bs_status detector_tables(bs_ctx* c, cudaStream_t st) {
    const int R = c->R, C = c->crop;
    double du, dv;
    std::vector<int> su, sv;
    passbands(c, su, sv, du, dv);
    const int Nu = (int)su.size(), Nv = (int)sv.size();
    if (Nu == 0 || Nv == 0) return BS_OK;
    const int *fu = c->d_su.as<int>(), *fv = c->d_sv.as<int>();
    // forward x: Wx[x][k] = e^{-2 pi i x su_k / R}; forward y: Wy[j][y] = e^{-2 pi i y sv_j / R}
    if constexpr (sizeof(T) == 8) {
        launch_fold_table(R, fold_x(R, su, sv).ldt, c->d_wx.as<zd>(), st);
        LAUNCHED(c);
    } else {
        launch_twiddle<T>(R, Nu, fu, 0, R, -1, Nu, 1, c->d_wx.as<cpx<T>>(), st);
        LAUNCHED(c);
        launch_twiddle<T>(R, Nv, fv, 0, R, -1, 1, R, c->d_wy.as<cpx<T>>(), st);
        LAUNCHED(c);
    }
    // inverse on the crop only: Wix[k][x] = e^{+2 pi i (off+x) su_k / R}, Wiy[y][j] likewise
    launch_twiddle<T>(C, Nu, fu, c->off, R, +1, 1, C, c->d_wix.as<cpx<T>>(), st);
    LAUNCHED(c);
    launch_twiddle<T>(C, Nv, fv, c->off, R, +1, Nv, 1, c->d_wiy.as<cpx<T>>(), st);
    LAUNCHED(c);
    return BS_OK;
}

// The detector images of the fields in d_fields, with the buffers and tables of the slice's near field.
template <class T>
static bs_status run_detector(bs_ctx* c, bool accumulate) {
    const bs_params& p = c->prm;
    const int R = c->R;
    double du, dv;
    std::vector<int> su, sv;
    passbands(c, su, sv, du, dv);
    const int Nu = (int)su.size(), Nv = (int)sv.size(), C = c->crop, res = c->res;
    if (Nu == 0 || Nv == 0) {
        if (!accumulate) CK(cudaMemsetAsync(c->d_D.p, 0, 2 * (size_t)res * res * sizeof(T), c->st));
        return BS_OK;
    }
    constexpr bool fp64 = sizeof(T) == 8;
    const FoldDft fx = fold_x(R, su, sv), fy = fold_y(R, su, sv);
    cpx<T>* wx = c->d_wx.as<cpx<T>>();
    cpx<T>* wy = c->d_wy.as<cpx<T>>();
    cpx<T>* wix = c->d_wix.as<cpx<T>>();
    cpx<T>* wiy = c->d_wiy.as<cpx<T>>();
    const cpx<T>* fields = c->d_fields.as<cpx<T>>();
    cpx<T>* f1 = c->d_f1.as<cpx<T>>();
    cpx<T>* f2 = c->d_f2.as<cpx<T>>();
    cpx<T>* g1 = c->d_g1.as<cpx<T>>();
    T* I = c->d_I.as<T>();
    long long RR = (long long)R * R;
    const size_t scr = detector_scratch_elems<T>(fx, fy, Nu, Nv, C);
    cpx<T>* gs = c->d_gscr.as<cpx<T>>();
    if constexpr (fp64) {  // f1 transposed: [Nu][R]
        launch_fold_dft(fx, 2, fields, wx, f1, nullptr, gs, c->st);
        LAUNCHED(c);
        launch_fold_dft(fy, 2, f1, wx, f2, c->d_mask.as<float>(), gs, c->st);
        LAUNCHED(c);
    } else {
        launch_cgemm<T>(R, Nu, R, 2, fields, R, RR, wx, Nu, 0, f1, Nu, (long long)R * Nu, 0, nullptr, (T)1, nullptr, gs,
                        scr, c->st);
        LAUNCHED(c);
        launch_cgemm<T>(Nv, Nu, R, 2, wy, R, 0, f1, Nu, (long long)R * Nu, f2, Nu, (long long)Nv * Nu, 1,
                        c->d_mask.as<float>(), (T)1, nullptr, gs, scr, c->st);
        LAUNCHED(c);
    }
    if (c->bp_on) {
        // applyBackpropagation (microscope.cu:423-488, 592-605) on U only: -exp(i kz d) with
        // kz = sqrt(k^2 - kx^2 - ky^2), k = 2 PI / lambda, kx = 2 PI u; zero where kx^2 + ky^2 >= k^2
        std::vector<cpx<T>> bp((size_t)Nv * Nu);
        for (int j = 0; j < Nv; j++)
            for (int kk = 0; kk < Nu; kk++) {
                double re, im;
                backprop_factor(su[kk], sv[j], R, du, dv, p.lambda, (float)c->bp_d, &re, &im);
                bp[(size_t)j * Nu + kk] = mk((T)re, (T)im);
            }
        CK(c->d_bp.ensure(bp.size() * sizeof(cpx<T>)));
        CK(cudaMemcpyAsync(c->d_bp.p, bp.data(), bp.size() * sizeof(cpx<T>), cudaMemcpyHostToDevice, c->st));
        launch_cmul<T>(Nv * Nu, c->d_bp.as<cpx<T>>(), f2, c->st);  // batch 0: U
        LAUNCHED(c);
        CK(cudaStreamSynchronize(c->st));  // bp is a host vector of this scope
    }
    launch_cgemm<T>(Nv, C, Nu, 2, f2, Nu, (long long)Nv * Nu, wix, C, 0, g1, C, (long long)Nv * C, 0, nullptr, (T)1,
                    nullptr, gs, scr, c->st);
    LAUNCHED(c);
    T scale = (T)(1.0 / ((double)R * (double)R));
    launch_cgemm<T>(C, C, Nv, 2, wiy, Nv, 0, g1, C, (long long)Nv * C, nullptr, C, (long long)C * C, 2, nullptr,
                    scale, I, gs, scr, c->st);
    LAUNCHED(c);
    launch_bin<T>(res, c->ss, 2, accumulate ? 1 : 0, I, c->d_D.as<T>(), c->st);
    LAUNCHED(c);
    return BS_OK;
}

// Place each sphere's Usp and Uip patches in the LUT pool; spheres whose
// tables together exceed the budget go to later chunks (each chunk is built
// and applied before the next one overwrites the pool).  FP64: one
// Patch<double> per entry.  Mixed: one float2 per entry in linear rows of
// thetaR + 1 entries (the last column repeated, rounded up to an even count
// for 16-byte rows; a Uip of one row is stored twice).
static bs_status plan_tables(std::vector<Sphere>& hs, bool mixed, size_t budget, std::vector<int>& chunk_start,
                             size_t& pool) {
    const size_t patch = mixed ? sizeof(float2) : sizeof(Patch<double>);
    const int ns = (int)hs.size();
    chunk_start.clear();
    size_t acc = 0;
    pool = 0;
    for (int i = 0; i < ns; i++) {
        Sphere& S = hs[i];
        S.lin_stride = mixed ? ((S.thetaR + 2) & ~1) : S.thetaR;
        // mixed: two rows or more per table, so that a lookup's row pair needs no clamp
        size_t need = (size_t)(S.dR + (mixed ? std::max(S.aR, 2) : S.aR)) * S.lin_stride * patch;
        if (need > budget)
            return fail(BS_ERR_NOMEM, "LUT of sphere %d needs %zu bytes, over the budget of %zu", i + 1, need, budget);
        if (i == 0 || acc + need > budget) {
            chunk_start.push_back(i);
            acc = 0;
        }
        S.usp_off = (int64_t)(acc / patch);
        S.uip_off = S.usp_off + (int64_t)S.dR * S.lin_stride;
        acc += need;
        pool = std::max(pool, acc);
    }
    chunk_start.push_back(ns);
    return BS_OK;
}

// Spheres whose coefficient rows are computed in one launch: consecutive
// spheres of a table chunk, at most COEF_BATCH_ROWS rows together (a single
// larger sphere forms its own batch).  starts: first global row of each sphere
// and the total, then the first coefficient of each sphere.
constexpr long long COEF_BATCH_ROWS = 1 << 19;

struct CoefBatch {
    int b0, b1;
    long long rows, coefs;
    std::vector<long long> starts;
};

static std::vector<CoefBatch> coef_batches(const std::vector<Sphere>& hs, const std::vector<int>& chunk_start) {
    std::vector<CoefBatch> out;
    for (size_t ci = 0; ci + 1 < chunk_start.size(); ci++) {
        int b0 = chunk_start[ci];
        const int s1 = chunk_start[ci + 1];
        while (b0 < s1) {
            CoefBatch b{b0, b0, 0, 0, {}};
            std::vector<long long> cs;
            while (b.b1 < s1) {
                const Sphere& S = hs[b.b1];
                const long long r = S.dR + S.aR;
                if (b.b1 > b0 && b.rows + r > COEF_BATCH_ROWS) break;
                b.starts.push_back(b.rows);
                cs.push_back(b.coefs);
                b.rows += r;
                b.coefs += r * (S.Nl + 1);
                b.b1++;
            }
            b.starts.push_back(b.rows);
            b.starts.insert(b.starts.end(), cs.begin(), cs.end());
            out.push_back(std::move(b));
            b0 = out.back().b1;
        }
    }
    return out;
}

static bs_status plan_luts(bs_ctx* c, bool mixed, std::vector<int>& chunk_start, size_t& pool) {
    size_t budget = c->budget;
    if (!budget) {
        size_t free_b = 0, total_b = 0;
        CK(cudaMemGetInfo(&free_b, &total_b));
        budget = (size_t)(0.80 * (double)(free_b + c->d_lut.n));
    }
    return plan_tables(c->hs, mixed, budget, chunk_start, pool);
}

// Order plane waves in compact groups of `chunk`: their projections on the
// plane perpendicular to the mean direction are split recursively at a
// multiple of `chunk` along the wider axis (a median split when the count
// allows), so every group but one holds `chunk` waves and the one short
// group goes last.  The sum over waves does not depend on the order (up to
// rounding); compact groups have narrow bounding cones, so each tile's table
// window per group stays small enough for shared memory (3072^2 pixels, 50
// spheres, 1000 directions: 98-99.7 % of windows fit, against 60-86 % for
// chunks cut from a Hilbert curve order, which can straddle the curve's jumps).
static void group_split(std::vector<size_t>& idx, size_t lo, size_t hi, const std::vector<double>& px,
                        const std::vector<double>& py, size_t chunk, std::vector<std::pair<size_t, size_t>>& groups) {
    const size_t n = hi - lo;
    if (n <= chunk) {
        groups.push_back({lo, hi});
        return;
    }
    double x0 = px[idx[lo]], x1 = x0, y0 = py[idx[lo]], y1 = y0;
    for (size_t i = lo; i < hi; i++) {
        x0 = std::min(x0, px[idx[i]]);
        x1 = std::max(x1, px[idx[i]]);
        y0 = std::min(y0, py[idx[i]]);
        y1 = std::max(y1, py[idx[i]]);
    }
    const std::vector<double>& key = (x1 - x0 >= y1 - y0) ? px : py;
    std::stable_sort(idx.begin() + lo, idx.begin() + hi, [&key](size_t a, size_t b) { return key[a] < key[b]; });
    const size_t half = (size_t)std::llround((double)n / (2.0 * (double)chunk));
    const size_t k = chunk * std::max<size_t>(1, half);
    group_split(idx, lo, lo + k, px, py, chunk, groups);
    group_split(idx, lo + k, hi, px, py, chunk, groups);
}

static void sort_waves(std::vector<double>& w, int chunk) {
    size_t nk = w.size() / 3;
    if (nk < 3) return;
    double m[3] = {0, 0, 0};
    for (size_t i = 0; i < nk; i++)
        for (int c = 0; c < 3; c++) m[c] += w[3 * i + c];
    double ml = std::sqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
    if (!(ml > 0)) return;
    for (int c = 0; c < 3; c++) m[c] /= ml;
    double a[3] = {1, 0, 0};
    if (std::fabs(m[0]) > 0.9) a[0] = 0, a[1] = 1;
    double e1[3] = {a[1] * m[2] - a[2] * m[1], a[2] * m[0] - a[0] * m[2], a[0] * m[1] - a[1] * m[0]};
    double l1 = std::sqrt(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]);
    for (int c = 0; c < 3; c++) e1[c] /= l1;
    double e2[3] = {m[1] * e1[2] - m[2] * e1[1], m[2] * e1[0] - m[0] * e1[2], m[0] * e1[1] - m[1] * e1[0]};
    std::vector<double> px(nk), py(nk);
    std::vector<size_t> idx(nk);
    for (size_t i = 0; i < nk; i++) {
        const double* k = &w[3 * i];
        px[i] = k[0] * e1[0] + k[1] * e1[1] + k[2] * e1[2];
        py[i] = k[0] * e2[0] + k[1] * e2[1] + k[2] * e2[2];
        idx[i] = i;
    }
    std::vector<std::pair<size_t, size_t>> groups;
    group_split(idx, 0, nk, px, py, (size_t)chunk, groups);
    std::stable_partition(groups.begin(), groups.end(),
                          [chunk](const std::pair<size_t, size_t>& g) { return g.second - g.first == (size_t)chunk; });
    std::vector<double> out;
    out.reserve(w.size());
    for (const auto& g : groups)
        for (size_t i = g.first; i < g.second; i++)
            for (int c = 0; c < 3; c++) out.push_back(w[3 * idx[i] + c]);
    w.swap(out);
}

// Bounding cone (unit axis, half-angle in radians, at most 2.9) of all directions; half-angle pi
// if one of them is not a unit vector, which turns the mixed LUT kernel's angle bounds off.  A length of
// 1 + e, e <= 1e-6, moves an angle by up to acos(1 / (1 + e)) < sqrt(2 e) at the poles: added to `margin`.
static float4 wave_cone(const std::vector<double>& w, float& margin) {
    double m[3] = {0, 0, 0}, off = 0;
    for (size_t i = 0; i < w.size(); i += 3) {
        const double l = std::sqrt(w[i] * w[i] + w[i + 1] * w[i + 1] + w[i + 2] * w[i + 2]);
        if (!(std::fabs(l - 1.0) <= 1e-6)) return make_float4(0.f, 0.f, 1.f, (float)TRUE_PI);
        off = std::max(off, std::fabs(l - 1.0));
        for (int k = 0; k < 3; k++) m[k] += w[i + k];
    }
    margin += (float)std::sqrt(2 * off);
    const double ml = std::sqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
    if (!(ml > 1e-3)) return make_float4(0.f, 0.f, 1.f, 2.9f);
    double c = 1;
    for (size_t i = 0; i < w.size(); i += 3) c = std::min(c, (w[i] * m[0] + w[i + 1] * m[1] + w[i + 2] * m[2]) / ml);
    return make_float4((float)(m[0] / ml), (float)(m[1] / ml), (float)(m[2] / ml),
                       (float)std::min(2.9, std::acos(std::max(-1.0, c))));
}

// Predicted fraction of the sorted mixed LUT kernel's (tile, sphere, chunk) units whose columns fit
// its window, from the kernel's own bounds on a sample of tiles and spheres: the tile's angular
// radius seen from the sphere (its corners) and an even share of the angles between the
// sampled directions and the tile centre's direction for each group of 32.
static double predict_staged_fraction(const bs_ctx* c, const std::vector<double>& w) {
    const Scene& sc = c->sc;
    const int R = sc.R, tiles = (R + LUT_TILE - 1) / LUT_TILE, ns = sc.ns;
    const int nk = (int)(w.size() / 3), groups = (std::min(nk, 1024) + 31) / 32;
    const int ts = std::max(1, tiles / 8), ss = std::max(1, ns / 4), ws = std::max(1, nk / 48);
    long long staged = 0, total = 0;
    for (int ty = 0; ty < tiles; ty += ts)
        for (int tx = 0; tx < tiles; tx += ts)
            for (int si = 0; si < ns; si += ss) {
                const Sphere& S = c->hs[si];
                auto at = [&](double u, double v, double* q) {
                    double l = 0;
                    for (int k = 0; k < 3; k++) {
                        q[k] = sc.A[k] + sc.X[k] * (u / R) + sc.Y[k] * (v / R) - S.p[k];
                        l += q[k] * q[k];
                    }
                    l = std::sqrt(l);
                    for (int k = 0; k < 3 && l > 0; k++) q[k] /= l;
                };
                const double u0 = tx * LUT_TILE, v0 = ty * LUT_TILE, e = LUT_TILE - 1;
                double ctr[3], q[3], cmin = 1;
                at(u0 + 7.5, v0 + 7.5, ctr);
                for (int k = 0; k < 4; k++) {
                    at((k & 1) ? std::min(u0 + e, R - 1.0) : u0, (k & 2) ? std::min(v0 + e, R - 1.0) : v0, q);
                    cmin = std::min(cmin, q[0] * ctr[0] + q[1] * ctr[1] + q[2] * ctr[2]);
                }
                const double gam = std::acos(std::max(-1.0, cmin)) + LUT_STAGE_MARGIN, tsc = (S.thetaR - 1) / PI_REF;
                double lo = 1, hi = -1;
                for (int i = 0; i < nk; i += ws) {
                    const double d = w[3 * i] * ctr[0] + w[3 * i + 1] * ctr[1] + w[3 * i + 2] * ctr[2];
                    lo = std::min(lo, d);
                    hi = std::max(hi, d);
                }
                const double range = std::acos(std::max(-1.0, std::min(1.0, lo))) - std::acos(std::max(-1.0, std::min(1.0, hi)));
                total++;
                if (gam <= 1.4 && (range / groups + 2 * gam) * tsc + 4.5 <= LUT_WINDOW) staged++;
            }
    return total ? (double)staged / (double)total : 0.0;
}

// Bounding cone (unit axis, half-angle in radians) of every `chunk`
// consecutive waves, with a small margin for single-precision rounding.  A
// chunk holding a direction that is not a unit vector gets half-angle pi,
// which turns the angular window off for it.
static std::vector<float4> wave_cones(const std::vector<double>& w, int chunk) {
    size_t nk = w.size() / 3;
    size_t nch = (nk + chunk - 1) / chunk;
    std::vector<float4> out(nch);
    for (size_t ch = 0; ch < nch; ch++) {
        size_t a = ch * chunk, b = std::min(nk, a + chunk);
        double m[3] = {0, 0, 0};
        bool unit = true;
        for (size_t i = a; i < b; i++) {
            const double* k = &w[3 * i];
            double kl = std::sqrt(k[0] * k[0] + k[1] * k[1] + k[2] * k[2]);
            if (!(std::fabs(kl - 1.0) <= 1e-6)) unit = false;
            for (int c = 0; c < 3; c++) m[c] += k[c];
        }
        double ml = std::sqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
        double beta = 0;
        if (ml > 1e-3 && unit) {
            for (int c = 0; c < 3; c++) m[c] /= ml;
            for (size_t i = a; i < b; i++) {
                const double* k = &w[3 * i];
                double cth = k[0] * m[0] + k[1] * m[1] + k[2] * m[2];
                beta = std::max(beta, std::acos(std::min(1.0, std::max(-1.0, cth))));
            }
        } else {
            m[0] = 0, m[1] = 0, m[2] = 1;
            beta = TRUE_PI;
        }
        out[ch] = make_float4((float)m[0], (float)m[1], (float)m[2], (float)(beta + 1e-4));
    }
    return out;
}

// Predicted fraction of (tile, sphere, wave chunk) units whose table window the plain mixed LUT kernel can hold in
// shared memory, from the kernel's own bounds evaluated on a sample of tiles, spheres and chunks: the tile's
// distance range (nearest point of the tile rectangle, farthest corner) gives the rows, the corners' angles from
// the tile-centre direction give gamma.  Below staged_min_fraction the kernel without windows is faster: reads
// that do not fit one run with the L1 that the staged kernel's shared memory leaves.
static double staged_min_fraction(int chunk) { return chunk >= WAVE_CHUNK_MAX ? 0.3 : 0.7; }
static double plain_staged_fraction(const bs_ctx* c, const std::vector<float4>& cones, int s0, int s1, int chunk) {
    const int cap = lut_plain_entries(chunk);
    const Scene& sc = c->sc;
    const int R = sc.R, tiles = (R + LUT_TILE - 1) / LUT_TILE;
    const int ts = std::max(1, tiles / 16), ss = std::max(1, (s1 - s0) / 32);
    const int cs = std::max(1, (int)cones.size() / 16);
    auto pos = [&](double u, double v, double* q) {
        for (int k = 0; k < 3; k++) q[k] = sc.A[k] + sc.X[k] * (u / R) + sc.Y[k] * (v / R);
    };
    const double X2 = sc.X[0] * sc.X[0] + sc.X[1] * sc.X[1] + sc.X[2] * sc.X[2];
    const double Y2 = sc.Y[0] * sc.Y[0] + sc.Y[1] * sc.Y[1] + sc.Y[2] * sc.Y[2];
    long long staged = 0, total = 0;
    for (int ty = 0; ty < tiles; ty += ts)
        for (int tx = 0; tx < tiles; tx += ts) {
            const double u0 = tx * LUT_TILE, v0 = ty * LUT_TILE;
            const double u1 = std::min(u0 + LUT_TILE - 1, (double)R - 1), v1 = std::min(v0 + LUT_TILE - 1, (double)R - 1);
            for (int si = s0; si < s1; si += ss) {
                const Sphere& S = c->hs[si];
                double e[3];
                for (int k = 0; k < 3; k++) e[k] = S.p[k] - sc.A[k];
                // nearest point of the tile rectangle (X and Y span the plane at right angles)
                const double un = std::min(std::max((e[0] * sc.X[0] + e[1] * sc.X[1] + e[2] * sc.X[2]) / X2 * R, u0), u1);
                const double vn = std::min(std::max((e[0] * sc.Y[0] + e[1] * sc.Y[1] + e[2] * sc.Y[2]) / Y2 * R, v0), v1);
                double q[3], ctr[3];
                pos(un, vn, q);
                const double dmin = std::sqrt((q[0] - S.p[0]) * (q[0] - S.p[0]) + (q[1] - S.p[1]) * (q[1] - S.p[1]) +
                                              (q[2] - S.p[2]) * (q[2] - S.p[2]));
                const int nch = (int)((cones.size() + cs - 1) / cs);
                total += nch;
                if (!(dmin >= S.a) || dmin == 0) continue;
                pos(u0 + 7.5, v0 + 7.5, ctr);
                double cl = 0;
                for (int k = 0; k < 3; k++) {
                    ctr[k] -= S.p[k];
                    cl += ctr[k] * ctr[k];
                }
                cl = std::sqrt(cl);
                double dmax = 0, gam = 0;
                const double cu[4] = {u0, u1, u0, u1}, cv[4] = {v0, v0, v1, v1};
                for (int k = 0; k < 4; k++) {
                    pos(cu[k], cv[k], q);
                    double r[3] = {q[0] - S.p[0], q[1] - S.p[1], q[2] - S.p[2]};
                    const double d = std::sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
                    dmax = std::max(dmax, d);
                    const double cosg = (r[0] * ctr[0] + r[1] * ctr[1] + r[2] * ctr[2]) / (d * cl);
                    gam = std::max(gam, std::acos(std::min(1.0, std::max(-1.0, cosg))));
                }
                gam += LUT_PLAIN_MARGIN;
                auto row = [&](double d) {
                    double x = (d - S.r0) / (S.dmax - S.r0) * (S.dR - 1);
                    return (int)std::floor(std::min(std::max(x, 0.0), (double)(S.dR - 1)));
                };
                const int rlo = row(dmin), nrows = std::min(row(dmax) + 1, S.dR - 1) - rlo + 1;
                const double tsc = (S.thetaR - 1) / PI_REF;
                for (size_t ch = 0; ch < cones.size(); ch += cs) {
                    const float4 k = cones[ch];
                    const double thc =
                        std::acos(std::min(1.0, std::max(-1.0, (k.x * ctr[0] + k.y * ctr[1] + k.z * ctr[2]) / cl)));
                    const int t_lo = std::max(0, (int)std::floor((thc - k.w - gam) * tsc) - 1);
                    const int t_hi = std::min(S.thetaR, (int)std::floor((thc + k.w + gam) * tsc) + 2);
                    const int W = t_hi - t_lo + 1;
                    if (W >= 2 && (long long)nrows * lut_plain_stride(W) <= cap) staged++;
                }
            }
        }
    return total ? (double)staged / (double)total : 0.0;
}

// Waves per chunk of the plain mixed LUT kernel, with the matching wave order and cones: the largest of 64, 32 and
// 16 whose predicted staged fraction reaches 0.8, else the one with the largest fraction if that reaches its
// staged_min_fraction, else the largest fraction among those that reach theirs, else 64.  Smaller chunks have
// narrower cones, so more windows fit, but each chunk pays a window copy, two barriers and a Kahan step.  The
// chunk and the order of the waves in it decide the last bits of the sums, so bs_set_lut_staging has no say here;
// bs_set_lut_wave_chunk fixes the chunk instead.
struct ChunkPlan {
    int chunk = WAVE_CHUNK_MAX;
    std::vector<double> w;
    std::vector<float4> cones;
    double predicted = 0;
};

static ChunkPlan chunk_plan(const bs_ctx* c, const std::vector<double>& waves, int chunk) {
    ChunkPlan cp;
    cp.chunk = chunk;
    cp.w = waves;
    if (!c->prm.plane_wave) sort_waves(cp.w, chunk);
    cp.cones = wave_cones(cp.w, chunk);
    cp.predicted = plain_staged_fraction(c, cp.cones, 0, c->sc.ns, chunk);
    return cp;
}

static ChunkPlan choose_chunk(const bs_ctx* c, const std::vector<double>& waves) {
    if (c->lut_chunk) return chunk_plan(c, waves, c->lut_chunk);
    ChunkPlan first = chunk_plan(c, waves, WAVE_CHUNK_MAX), best = first, viable;
    if (c->prm.plane_wave) return first;
    viable.predicted = best.predicted >= staged_min_fraction(best.chunk) ? best.predicted : -1;
    if (viable.predicted >= 0) viable = best;  // the best that the staged kernel would run to advantage
    for (int cand = WAVE_CHUNK_MAX / 2; cand >= WAVE_CHUNK_MAX / 4 && best.predicted < 0.8; cand /= 2) {
        ChunkPlan cp = chunk_plan(c, waves, cand);
        if (cp.predicted >= staged_min_fraction(cand) && cp.predicted > viable.predicted) viable = cp;
        if (cp.predicted > best.predicted || cp.predicted >= 0.8) best = std::move(cp);
    }
    if (best.predicted >= staged_min_fraction(best.chunk)) return best;
    return viable.predicted >= 0 ? viable : first;
}

// ---------------------------------------------------------------------------
// The near field
// ---------------------------------------------------------------------------
// Work on the context's second stream, from what was on the first at the fork on.  The first waits for it at
// join(), or when a failed run leaves the scope.
struct SideWork {
    bs_ctx* c;
    bool open = false;
    cudaError_t fork() {
        cudaError_t e = cudaSuccess;
        for (cudaEvent_t* v : {&c->uf_ev[0], &c->uf_ev[1]})
            if (e == cudaSuccess && !*v) e = cudaEventCreate(v);
        if (!c->side) e = cudaStreamCreateWithPriority(&c->side, cudaStreamNonBlocking, c->stream_prio);
        for (cudaEvent_t* v : {&c->fork, &c->join})
            if (e == cudaSuccess && !*v) e = cudaEventCreateWithFlags(v, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventRecord(c->fork, c->st);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(c->side, c->fork, 0);
        open = e == cudaSuccess;
        return e;
    }
    cudaError_t join() {
        open = false;
        cudaError_t e = cudaEventRecord(c->join, c->side);
        return e == cudaSuccess ? cudaStreamWaitEvent(c->st, c->join, 0) : e;
    }
    ~SideWork() {
        if (open) join();
    }
};

template <class T>
static bs_status run_nearfield(bs_ctx* c) {
    Scene& sc = c->sc;
    const bs_params& p = c->prm;
    const int R = c->R, ns = sc.ns, nk = sc.nk;
    const bool fp64 = std::is_same<T, double>::value;
    CK(c->d_fields.ensure(2 * (size_t)R * R * sizeof(cpx<T>)));
    cpx<T>* U = c->d_fields.as<cpx<T>>();
    cpx<T>* Uf = U + (size_t)R * R;
    // upload spheres and waves
    CK(c->d_sph.ensure(std::max(1, ns) * sizeof(Sphere)));
    std::vector<double> w(c->waves);
    int chunk = c->lut_chunk ? c->lut_chunk : WAVE_CHUNK_MAX;
    const bool mixed_lut = !fp64 && p.scalar && p.lut_us && ns > 0;
    const bool plain = mixed_lut && lut_plain(ns), few = mixed_lut && lut_few(ns, nk);
    const bool split = mixed_lut && !plain;  // tables of the split single-precision build
    float4 cone = make_float4(0.f, 0.f, 1.f, (float)TRUE_PI);
    float margin = LUT_STAGE_MARGIN;
    std::vector<float4> cones;
    double predicted = 0;
    if (p.plane_wave) w.assign(p.k_dir, p.k_dir + 3);
    if (plain) {
        ChunkPlan cp = choose_chunk(c, w);
        chunk = cp.chunk;
        w.swap(cp.w);
        cones.swap(cp.cones);
        predicted = cp.predicted;
    } else if (split) {
        cone = wave_cone(w, margin);  // ordered per tile on the device
    } else if (!p.plane_wave) {
        sort_waves(w, WAVE_CHUNK_MAX);
    }
    const bool unit = cone.w < 3.f;  // the sorted LUT kernel's angle bounds hold
    // waves per counted chunk; without windows the chunks are counted in 64s
    const int counted_chunk = !c->lut_chunk && c->lut_staging == 2 ? WAVE_CHUNK_MAX : chunk;
    c->stats.lut_wave_chunk = counted_chunk;
    CK(c->d_waves.ensure(w.size() * sizeof(double)));
    CK(cudaMemcpyAsync(c->d_waves.p, w.data(), w.size() * sizeof(double), cudaMemcpyHostToDevice, c->st));

    // ---- what the second stream needs ----
    cudaEventRecord(c->ev[0], c->st);
    const bool uf_table = p.lut_uf && !p.plane_wave && p.scalar;
    if (uf_table) {
        CK(c->d_uft.ensure((size_t)sc.uf_dR * (sc.m + 1) * sizeof(double)));
        CK(c->d_uftscr.ensure((size_t)sc.uf_dR * (sc.m + 1) * sizeof(double)));
    }
    std::vector<UfOrder> ufw(sc.m + 1);
    {
        // condenser aperture factor of each order, the same for every pixel (nfScalarUf.cu:46-175)
        double kap = 1, kap2 = 1;  // P_l = kappa_l u_l, kappa_l = (2l - 1) / l kappa_{l-1}
        double a0 = 1, a1 = sc.cos_a, a2 = 1, b0 = 1, b1 = sc.cos_b, b2 = 1;
        auto step = [](int n, double x, double& q0, double& q1) {  // rts/math/legendre.h:17-25
            const double qn = ((2 * n - 1) * x * q1 - (n - 1) * q0) / n;
            q0 = q1;
            q1 = qn;
        };
        for (int l = 0; l <= sc.m; l++) {
            if (l > 0) {
                a2 = a0;
                step(l + 1, sc.cos_a, a0, a1);
                b2 = b0;
                step(l + 1, sc.cos_b, b0, b1);
            }
            ufw[l].odd = 2.0 * l - 1.0;
            ufw[l].beta = 0;
            if (l > 0) {
                const double k1 = kap;
                kap *= (2.0 * l - 1.0) / l;
                if (l > 1) ufw[l].beta = (l - 1.0) / l * kap2 / kap;
                kap2 = k1;
            }
            ufw[l].w = (l & 2 ? -1.0 : 1.0) * kap * (l == 0 ? a1 - b1 : a1 - a2 - b1 + b2) * (2.0 * PI_REF * sc.amp);
        }
        CK(c->d_ufw.ensure(ufw.size() * sizeof(UfOrder)));
        CK(cudaMemcpyAsync(c->d_ufw.p, ufw.data(), ufw.size() * sizeof(UfOrder), cudaMemcpyHostToDevice, c->st));
    }
    bs_status det = detector_buffers<T>(c);
    if (det != BS_OK) return det;
    SideWork side{c};
    CK(side.fork());
    cudaEventRecord(c->ev[1], c->st);

    // ---- LUT placement (before the sphere table goes to the device) ----
    std::vector<int> chunk_start;
    std::vector<CoefBatch> batches;
    size_t pool = 0;
    if (p.scalar && p.lut_us && ns > 0) {
        bs_status pst = plan_luts(c, !fp64, chunk_start, pool);
        if (pst != BS_OK) return pst;
        batches = coef_batches(c->hs, chunk_start);
    }

    // ---- Mie coefficients ----
    int ncoef = 0;
    for (auto& S : c->hs) ncoef += S.Nl + 1;
    const bool scatter = p.scalar && ns > 0;
    if (scatter) {
        CK(c->d_A.ensure(ncoef * sizeof(zd)));
        CK(c->d_B.ensure(ncoef * sizeof(zd)));
        CK(cudaMemcpyAsync(c->d_sph.p, c->hs.data(), ns * sizeof(Sphere), cudaMemcpyHostToDevice, c->st));
        launch_mie(c->d_sph.as<Sphere>(), ns, sc.kmag, c->d_A.as<zd>(), c->d_B.as<zd>(), c->st);
        LAUNCHED(c);
        if (p.lut_us) {  // the LUT kernels' phases and float directions (the direct method forms its own)
            CK(c->d_ph.ensure((size_t)ns * nk * sizeof(cpx<T>)));
            CK(c->d_kw4.ensure((size_t)nk * sizeof(float4)));
            launch_phase<T>(sc, c->d_sph.as<Sphere>(), c->d_waves.as<double>(), c->d_ph.as<cpx<T>>(),
                            c->d_kw4.as<float4>(), c->st);
            LAUNCHED(c);
        }
    } else if (ns > 0) {
        CK(cudaMemcpyAsync(c->d_sph.p, c->hs.data(), ns * sizeof(Sphere), cudaMemcpyHostToDevice, c->st));
    }
    cudaEventRecord(c->ev[2], c->st);

    // ---- incident field and the transforms' tables, beside the Mie coefficients and lookup tables ----
    cudaEventRecord(c->uf_ev[0], c->side);
    if (uf_table) {
        launch_uf_table(sc, c->d_uft.as<double>(), c->d_uftscr.as<double>(), c->side);
        LAUNCHED(c);
    }
    launch_uf<T>(sc, c->d_uft.as<double>(), c->d_ufw.as<UfOrder>(), Uf, c->side);
    LAUNCHED(c);
    cudaEventRecord(c->uf_ev[1], c->side);
    det = detector_tables<T>(c, c->side);
    if (det != BS_OK) return det;
    c->interactions = 0;

    if (!p.scalar) {
        CK(side.join());
        launch_sum_only<T>(sc, c->d_sph.as<Sphere>(), Uf, U, c->st);
        LAUNCHED(c);
        cudaEventRecord(c->ev[3], c->st);
    } else if (!p.lut_us) {
        cudaEventRecord(c->ev[3], c->st);
        if (ns == 0) {
            CK(side.join());
            CK(cudaMemcpyAsync(U, Uf, (size_t)R * R * sizeof(cpx<T>), cudaMemcpyDeviceToDevice, c->st));
        } else {
            // the addition theorem turns the per-wave Legendre sums into per-sphere coefficients
            const int L = c->Lmax, nlm = L * (L + 1) / 2;
            CK(c->d_shrec.ensure((size_t)nlm * sizeof(ShRec)));
            CK(c->d_shtab.ensure((size_t)nk * (nlm + ns) * sizeof(double2)));
            CK(c->d_shcoef.ensure((size_t)ns * nlm * 4 * sizeof(zd)));
            launch_sh_tables(sc, c->d_sph.as<Sphere>(), L, c->d_waves.as<double>(), c->d_shrec.as<ShRec>(),
                             c->d_shtab.as<double2>(), c->d_A.as<zd>(), c->d_B.as<zd>(), c->d_shcoef.as<zd>(), c->st);
            c->launches += 3;
            CK(side.join());
            launch_us_sh<T>(sc, c->d_sph.as<Sphere>(), L, c->d_shrec.as<ShRec>(), c->d_shcoef.as<zd>(), Uf, U, c->st);
            LAUNCHED(c);
        }
        c->interactions = (long long)R * R * ns * nk;
    } else {
        int thetaR = ns > 0 ? c->hs[0].thetaR : 1000;
        if (ns > 0) {
            CK(c->d_lut.ensure(pool));
            long long maxcoef = 0, maxstarts = 0, maxrow = 0;
            for (const CoefBatch& b : batches) {
                maxcoef = std::max(maxcoef, b.coefs);
                maxrow = std::max(maxrow, b.rows);
                maxstarts = std::max(maxstarts, (long long)b.starts.size());
            }
            CK(c->d_tab.ensure((size_t)maxcoef * sizeof(zd)));
            CK(c->d_tabscr.ensure((size_t)maxcoef * 2 * sizeof(double)));
            CK(c->d_starts.ensure((size_t)maxstarts * sizeof(long long)));
            if (split) CK(c->d_bias.ensure((size_t)maxrow * sizeof(float)));
            if (fp64 && c->acos_theta != thetaR) {
                CK(c->d_acos.ensure((ACOS_NODES + 1) * sizeof(AcosNode) + thetaR * sizeof(double)));
                launch_acos_nodes(thetaR, c->d_acos.as<AcosNode>(), c->st);
                LAUNCHED(c);
                c->acos_theta = thetaR;
            }
            if (c->legP_theta != thetaR || c->legP_L < c->Lmax || c->legP_split != split) {
                CK(c->d_legP.ensure((size_t)thetaR * c->Lmax * sizeof(double)));
                if (!split) launch_legendre_table(thetaR, c->Lmax, c->d_legP.as<double>(), c->st);
                else launch_legendre_split(thetaR, c->Lmax, thetaR, c->d_legP.as<float2>(), c->st);
                LAUNCHED(c);
                c->legP_split = split;
                c->legP_theta = thetaR;
                c->legP_L = c->Lmax;
            }
        }
        const int nchunks = (int)chunk_start.size() - 1;
        const int shares = fp64 || ns == 0 ? 1 : lut_splits(R, ns, nk);
        if (shares > 1) CK(c->d_part.ensure((size_t)shares * 4 * R * R * sizeof(float)));
        const int ranges = fp64 || ns == 0 ? 1 : lut_ranges(R, ns, nk, pool);
        const bool carry = shares == 1 && (nchunks > 1 || ranges > 1);
        if (!fp64 && carry) CK(c->d_kcmp.ensure((size_t)R * R * sizeof(float2)));
        bool use_stage = false;
        // tables of the previous run still in the pool?
        std::vector<double> key;
        if (c->reuse && nchunks == 1) {
            key = {fp64 ? 1.0 : plain ? 2.0 : 0.0, sc.kmag, (double)c->Lmax, (double)ns};
            for (const Sphere& S : c->hs) {
                const double v[] = {S.p[0], S.p[1], S.p[2], S.a, S.n_re, S.n_im, S.dmin, S.dmax, S.r0,
                                    (double)S.Nl, (double)S.aR, (double)S.dR, (double)S.thetaR,
                                    (double)S.lin_stride, (double)S.usp_off, (double)S.uip_off};
                key.insert(key.end(), v, v + sizeof(v) / sizeof(v[0]));
            }
        }
        const bool reuse_now = !key.empty() && c->lut_valid && key == c->lut_key;
        c->lut_valid = false;  // set again below once this run's tables are complete
        c->stats.lut_tables_built = reuse_now ? 0 : ns;
        if (!fp64 && ns > 0) {
            // tables of the mixed path stay within the GPU's 2D gather extent (thetaR wide, rows + 1 high)
            int maxw = 0, maxh = 0;
            CK(cudaDeviceGetAttribute(&maxw, cudaDevAttrMaxTexture2DGatherWidth, c->device));
            CK(cudaDeviceGetAttribute(&maxh, cudaDevAttrMaxTexture2DGatherHeight, c->device));
            for (const Sphere& S : c->hs)
                if (S.thetaR > maxw || std::max(S.dR, S.aR) + 1 > maxh)
                    return fail(BS_ERR_UNSUPPORTED,
                                "mixed precision: a %d x %d lookup table exceeds the %d x %d texture limit of this GPU "
                                "(use BS_PREC_FP64 or fewer table samples)",
                                std::max(S.dR, S.aR), S.thetaR, maxh - 1, maxw);
            if (plain) {
                use_stage = c->lut_staging == 1 || (c->lut_staging == 0 && predicted >= staged_min_fraction(chunk));
                CK(c->d_cones.ensure(cones.size() * sizeof(float4)));
                CK(cudaMemcpyAsync(c->d_cones.p, cones.data(), cones.size() * sizeof(float4), cudaMemcpyHostToDevice,
                                   c->st));
            } else if (!few) {
                predicted = unit ? predict_staged_fraction(c, w) : 0.0;
                use_stage = unit && c->lut_staging != 2;
            }
            c->stats.lut_staged_predicted = predicted;
            CK(c->d_cnt.ensure(2 * sizeof(unsigned long long)));
            CK(cudaMemsetAsync(c->d_cnt.p, 0, 2 * sizeof(unsigned long long), c->st));
        }
        bool first_build = true;
        for (int ci = 0; ci < std::max(1, nchunks); ci++) {
            int s0 = ns > 0 ? chunk_start[ci] : 0, s1 = ns > 0 ? chunk_start[ci + 1] : 0;
            for (const CoefBatch& b : batches) {
                if (reuse_now || b.b0 < s0 || b.b1 > s1) continue;
                CK(cudaMemcpyAsync(c->d_starts.p, b.starts.data(), b.starts.size() * sizeof(long long),
                                   cudaMemcpyHostToDevice, c->st));
                launch_coef_rows_batch(c->d_sph.as<Sphere>(), b.b0, b.b1 - b.b0, c->d_starts.as<long long>(), b.rows,
                                       sc.kmag, c->d_A.as<zd>(), c->d_B.as<zd>(), c->d_tab.as<zd>(),
                                       c->d_tabscr.as<double>(), split ? c->d_bias.as<float>() : nullptr, c->st);
                LAUNCHED(c);
                // the tables of every sphere of the batch in two launches (the dR-row Usp tables,
                // then the shorter Uip tables)
                for (int t = 0; t < 2; t++) {
                    std::vector<LutBuildJob> jobs;
                    int max_rows = 0, max_theta = 1;
                    for (int i = b.b0; i < b.b1; i++) {
                        const Sphere& S = c->hs[i];
                        const int L = S.Nl + 1;
                        LutBuildJob j{};
                        j.tab_off = b.starts[(size_t)(b.b1 - b.b0) + 1 + (i - b.b0)] + (t ? (long long)S.dR * L : 0);
                        j.lin_off = t ? S.uip_off : S.usp_off;
                        j.row_off = b.starts[i - b.b0] + (t ? S.dR : 0);
                        j.rows = t ? (fp64 ? S.aR : std::max(S.aR, 2)) : S.dR;
                        j.last = (t ? S.aR : S.dR) - 1;
                        j.L = L;
                        j.thetaR = S.thetaR;
                        j.lin_stride = S.lin_stride;
                        max_rows = std::max(max_rows, j.rows);
                        max_theta = std::max(max_theta, S.thetaR);
                        jobs.push_back(j);
                    }
                    if (jobs.empty()) continue;
                    DevBuf& jb = t ? c->d_lbjobs2 : c->d_lbjobs;
                    CK(jb.ensure(jobs.size() * sizeof(LutBuildJob)));
                    CK(cudaMemcpyAsync(jb.p, jobs.data(), jobs.size() * sizeof(LutBuildJob), cudaMemcpyHostToDevice,
                                       c->st));
                    for (size_t j0 = 0; j0 < jobs.size(); j0 += 65535) {  // the grid's z extent
                        const int nj = (int)std::min<size_t>(65535, jobs.size() - j0);
                        if (fp64)
                            launch_lut_build(jb.as<LutBuildJob>() + j0, nj, max_rows, max_theta, c->d_tab.as<zd>(),
                                             c->d_legP.as<double>(), c->legP_L, c->d_lut.as<Patch<double>>(), c->st);
                        else if (plain)
                            launch_lut_build_plain(jb.as<LutBuildJob>() + j0, nj, max_rows, max_theta,
                                                   c->d_tab.as<zd>(), c->d_legP.as<double>(), c->legP_L,
                                                   c->d_lut.as<float2>(), c->st);
                        else
                            launch_lut_build_mixed(jb.as<LutBuildJob>() + j0, nj, max_rows, max_theta,
                                                   c->d_tab.as<zd>(), c->d_bias.as<float>(), c->d_legP.as<float2>(),
                                                   thetaR, c->d_lut.as<float2>(), c->st);
                        LAUNCHED(c);
                    }
                }
            }
            if (first_build) {
                cudaEventRecord(c->ev[3], c->st);
                first_build = false;
                CK(side.join());
            }
            int finalize = (ci == std::max(1, nchunks) - 1);
            if (fp64) {
                launch_us_lut_f64(sc, c->d_sph.as<Sphere>(), s0, s1, ci > 0, finalize, c->d_waves.as<double>(),
                                  c->d_acos.as<AcosNode>(), c->d_ph.as<zd>(), c->d_lut.as<Patch<double>>(),
                                  (const zd*)Uf, (zd*)U, c->st);
            } else if (plain || few) {
                launch_us_lut_plain(sc, c->d_sph.as<Sphere>(), s0, s1, ci > 0, finalize, c->d_kw4.as<float4>(),
                                    c->d_cones.as<float4>(), c->d_ph.as<cpx<float>>(), c->d_lut.as<float2>(),
                                    (const cpx<float>*)Uf, (cpx<float>*)U, c->d_cnt.as<unsigned long long>(),
                                    carry ? c->d_kcmp.as<float2>() : nullptr, use_stage, chunk, counted_chunk, c->st);
            } else {
                for (int q = 0; q < ranges; q++) {
                    const int r0 = s0 + (int)((long long)(s1 - s0) * q / ranges);
                    const int r1 = s0 + (int)((long long)(s1 - s0) * (q + 1) / ranges);
                    const int last = q == ranges - 1;
                    launch_us_lut_mixed(sc, c->d_sph.as<Sphere>(), r0, r1, ci > 0 || q > 0, finalize && last,
                                        c->d_kw4.as<float4>(), c->d_ph.as<cpx<float>>(), c->d_lut.as<float2>(),
                                        (const cpx<float>*)Uf, (cpx<float>*)U,
                                        ns > 0 ? c->d_cnt.as<unsigned long long>() : nullptr,
                                        carry ? c->d_kcmp.as<float2>() : nullptr,
                                        shares > 1 ? c->d_part.as<float>() : nullptr, use_stage, chunk, cone, margin,
                                        c->st);
                    if (!last) LAUNCHED(c);
                }
                if (shares > 1 && finalize) c->launches++;
            }
            LAUNCHED(c);
            c->tab_s0 = s0;
            c->tab_s1 = s1;
        }
        if (!key.empty()) {
            c->lut_key.swap(key);
            c->lut_valid = true;
        }
        c->interactions = (long long)R * R * ns * nk;
    }
    cudaEventRecord(c->ev[4], c->st);
    return BS_OK;
}

// Device bytes the buffers of run_nearfield and run_detector reach for the
// derived scene of `c` (each DevBuf at least 256 bytes).  0 if the tables do not
// fit lut_budget.
static size_t estimate_bytes(bs_ctx* c, bool fp64, size_t lut_budget) {
    const bs_params& p = c->prm;
    const Scene& sc = c->sc;
    const size_t R = c->R, ns = sc.ns, nk = sc.nk, C = c->crop, res = c->res;
    const size_t cT = fp64 ? sizeof(cpx<double>) : sizeof(cpx<float>), rT = fp64 ? sizeof(double) : sizeof(float);
    auto B = [](size_t n) { return std::max<size_t>(n, 256); };
    size_t b = 0;
    b += B(2 * R * R * cT);                                   // U, Uf
    b += B(std::max<size_t>(1, ns) * sizeof(Sphere));
    b += B((p.plane_wave ? 1 : nk) * 3 * sizeof(double));     // directions
    if (p.lut_uf && !p.plane_wave && p.scalar) b += 2 * B((size_t)sc.uf_dR * (sc.m + 1) * sizeof(double));
    b += B((size_t)(sc.m + 1) * sizeof(UfOrder));              // incident-field order weights
    if (p.scalar && ns > 0) {
        size_t ncoef = 0;
        for (const Sphere& S : c->hs) ncoef += S.Nl + 1;
        b += 2 * B(ncoef * sizeof(zd));
        if (p.lut_us) b += B(ns * nk * cT) + B(nk * sizeof(float4));  // phases, float directions
        if (!p.lut_us) {  // direct method: harmonic recurrences, per-wave and per-sphere tables
            const size_t nlm = (size_t)c->Lmax * (c->Lmax + 1) / 2;
            b += B(nlm * sizeof(ShRec)) + B(nk * (nlm + ns) * sizeof(double2)) + B(ns * nlm * 4 * sizeof(zd));
        }
    }
    if (p.scalar && p.lut_us && ns > 0) {
        std::vector<Sphere> hs = c->hs;
        std::vector<int> cs;
        size_t pool = 0;
        if (plan_tables(hs, !fp64, lut_budget ? lut_budget : SIZE_MAX / 4, cs, pool) != BS_OK)
            return 0;
        const size_t thetaR = hs[0].thetaR;
        long long maxcoef = 0, maxstarts = 0, maxrow = 0;
        for (const CoefBatch& cb : coef_batches(hs, cs)) {
            maxcoef = std::max(maxcoef, cb.coefs);
            maxrow = std::max(maxrow, cb.rows);
            maxstarts = std::max(maxstarts, (long long)cb.starts.size());
        }
        b += 2 * B(ns * sizeof(LutBuildJob)) + B(pool) + 2 * B((size_t)maxcoef * sizeof(zd)) +
             B((size_t)maxstarts * sizeof(long long));
        b += B(thetaR * (size_t)c->Lmax * sizeof(double));    // Legendre table
        if (fp64) b += B((ACOS_NODES + 1) * sizeof(AcosNode) + c->hs[0].thetaR * sizeof(double));
        if (!fp64) {
            if (lut_plain((int)ns)) b += B((nk + 15) / 16 * sizeof(float4));  // cones
            else b += B((size_t)maxrow * sizeof(float));                      // biases
            const int shares = lut_splits((int)R, (int)ns, (int)nk);
            if (shares > 1) b += B((size_t)shares * 4 * R * R * sizeof(float));
            else if (cs.size() > 2 || lut_ranges((int)R, (int)ns, (int)nk, pool) > 1)
                b += B(R * R * sizeof(float2));  // Kahan carry between chunks
            b += B(2 * sizeof(unsigned long long));
        }
    }
    std::vector<int> su, sv;
    double du, dv;
    passbands(c, su, sv, du, dv);
    const size_t Nu = su.size(), Nv = sv.size();
    b += B(2 * res * res * rT);                               // D, Di
    if (Nu && Nv) {
        b += B(Nu * sizeof(int)) + B(Nv * sizeof(int)) + B(Nv * Nu * sizeof(float));
        const FoldDft fx = fold_x((int)R, su, sv), fy = fold_y((int)R, su, sv);
        b += fp64 ? B((R / 2 + 1) * fx.ldt * cT) : B(R * Nu * cT) + B(Nv * R * cT);
        b += B(Nu * C * cT) + B(C * Nv * cT);
        b += B(2 * R * Nu * cT) + B(2 * Nv * Nu * cT) + B(2 * Nv * C * cT) + B(2 * C * C * rT);
        const size_t scr = fp64 ? detector_scratch_elems<double>(fx, fy, (int)Nu, (int)Nv, (int)C)
                                : detector_scratch_elems<float>(fx, fy, (int)Nu, (int)Nv, (int)C);
        b += B(std::max<size_t>(scr, 1) * cT);  // split-K parts
    }
    b += B(res * res * rT);                                   // image staging
    return b;
}

extern "C" {

bs_status bs_set_backpropagation(bs_ctx* c, int32_t enable, double d) {
    if (!c || !std::isfinite(d)) return fail(BS_ERR_ARG, "bs_set_backpropagation: bad arguments");
    c->bp_on = enable != 0;
    c->bp_d = d;
    return BS_OK;
}

bs_status bs_set_lut_wave_chunk(bs_ctx* c, int32_t chunk) {
    if (!c || (chunk != 0 && chunk != 16 && chunk != 32 && chunk != 64))
        return fail(BS_ERR_ARG, "bs_set_lut_wave_chunk: chunk must be 0, 16, 32 or 64");
    c->lut_chunk = chunk;
    return BS_OK;
}

bs_status bs_set_lut_staging(bs_ctx* c, int32_t mode) {
    if (!c || mode < 0 || mode > 2) return fail(BS_ERR_ARG, "bs_set_lut_staging: mode must be 0, 1 or 2");
    c->lut_staging = mode;
    return BS_OK;
}

bs_status bs_set_stream_priority(bs_ctx* c, int32_t priority) {
    if (!c) return fail(BS_ERR_ARG, "bs_set_stream_priority: null context");
    int least = 0, greatest = 0;
    cudaError_t e = cudaDeviceGetStreamPriorityRange(&least, &greatest);
    if (e != cudaSuccess) return fail(BS_ERR_CUDA, "bs_set_stream_priority: %s", cudaGetErrorString(e));
    const int prio = std::min(least, std::max(greatest, (int)priority));
    if (prio == c->stream_prio) return BS_OK;
    // the context's work so far finishes on the old stream; later work goes to the new one
    e = cudaStreamSynchronize(c->st);
    cudaStream_t st = nullptr;
    if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&st, cudaStreamNonBlocking, prio);
    if (e != cudaSuccess) return fail(BS_ERR_CUDA, "bs_set_stream_priority: %s", cudaGetErrorString(e));
    cudaStreamDestroy(c->st);
    c->st = st;
    if (c->side) cudaStreamDestroy(c->side);  // made anew by the next run
    c->side = nullptr;
    c->stream_prio = prio;
    return BS_OK;
}

bs_status bs_set_lut_reuse(bs_ctx* c, int32_t enable) {
    if (!c) return fail(BS_ERR_ARG, "bs_set_lut_reuse: null context");
    c->reuse = enable != 0;
    if (!c->reuse) c->lut_valid = false;
    return BS_OK;
}

bs_status bs_release_buffers(bs_ctx* c) {
    if (!c) return fail(BS_ERR_ARG, "bs_release_buffers: null context");
    CK(cudaStreamSynchronize(c->st));
    release_all(c);
    return BS_OK;
}

bs_status bs_estimate_bytes(const bs_params* params, const bs_sphere* spheres, int32_t ns, int32_t nk,
                            bs_precision prec, uint64_t lut_budget, uint64_t* bytes) {
    if (!params || !bytes || ns < 0 || nk < 0 || (ns > 0 && !spheres))
        return fail(BS_ERR_ARG, "bs_estimate_bytes: bad arguments");
    if (prec != BS_PREC_FP64 && prec != BS_PREC_MIXED) return fail(BS_ERR_ARG, "bs_estimate_bytes: unknown precision");
    std::string why;
    if (!valid_params(params, why)) return fail(BS_ERR_ARG, "bs_estimate_bytes: %s", why.c_str());
    std::unique_ptr<bs_ctx> c(new bs_ctx());  // host state only: no stream, no device memory
    c->prm = *params;
    c->spheres.assign(spheres, spheres + ns);
    c->waves.assign(3 * (size_t)std::max(nk, 1), 0.0);
    c->waves_set = true;
    bs_status st = derive(c.get());
    if (st != BS_OK) return st;
    size_t b = estimate_bytes(c.get(), prec == BS_PREC_FP64, (size_t)lut_budget);
    if (!b) return fail(BS_ERR_NOMEM, "bs_estimate_bytes: a sphere's tables exceed the LUT budget of %llu bytes",
                        (unsigned long long)lut_budget);
    *bytes = b;
    return BS_OK;
}

}  // extern "C"

// One slice; with accumulate the detector images add to those of the previous
// slice on this context (same precision and detector size).
static bs_status simulate_impl(bs_ctx* c, bs_precision prec, bool accumulate) {
    c->have = false;
    bs_status st = derive(c);
    if (st != BS_OK) return st;
    c->prec = prec;
    c->stats.lut_tables_built = 0;
    c->stats.lut_staged_predicted = 0;
    int64_t l0 = c->launches;
    st = (prec == BS_PREC_FP64) ? run_nearfield<double>(c) : run_nearfield<float>(c);
    if (st != BS_OK) return st;
    st = (prec == BS_PREC_FP64) ? run_detector<double>(c, accumulate) : run_detector<float>(c, accumulate);
    if (st != BS_OK) return st;
    cudaEventRecord(c->ev[5], c->st);
    const bool counted = prec == BS_PREC_MIXED && c->prm.scalar && c->prm.lut_us && !c->hs.empty();
    CK(cudaStreamSynchronize(c->st));
    CK(cudaGetLastError());
    float t[5] = {0, 0, 0, 0, 0};
    for (int i = 0; i < 5; i++) cudaEventElapsedTime(&t[i], c->ev[i], c->ev[i + 1]);
    cudaEventElapsedTime(&t[0], c->uf_ev[0], c->uf_ev[1]);  // beside the next two
    c->stats.ms_uf = t[0];
    c->stats.ms_mie = t[1];
    c->stats.ms_lut = t[2];
    c->stats.ms_us = t[3];
    c->stats.ms_detector = t[4];
    float tot = 0;
    cudaEventElapsedTime(&tot, c->ev[0], c->ev[5]);
    c->stats.ms_total = tot;
    c->stats.kernel_launches = c->launches - l0;
    c->stats.us_interactions = c->interactions;
    c->stats.lut_chunks_staged = c->stats.lut_chunks_total = 0;
    if (counted) {  // after the wait: a copy to pageable memory that waits itself holds up other threads' calls
        unsigned long long cnt[2] = {0, 0};
        CK(cudaMemcpy(cnt, c->d_cnt.p, sizeof(cnt), cudaMemcpyDeviceToHost));
        c->stats.lut_chunks_staged = (int64_t)cnt[0];
        c->stats.lut_chunks_total = (int64_t)cnt[1];
    }
    c->have = true;
    return BS_OK;
}

extern "C" {

bs_status bs_simulate(bs_ctx* c, bs_precision prec) {
    if (!c) return fail(BS_ERR_ARG, "bs_simulate: null context");
    if (prec != BS_PREC_FP64 && prec != BS_PREC_MIXED) return fail(BS_ERR_ARG, "bs_simulate: unknown precision");
    return simulate_impl(c, prec, false);
}

bs_status bs_simulate_sources(bs_ctx* c, const double* sources, int32_t n, bs_precision prec) {
    if (!c || !sources || n < 1) return fail(BS_ERR_ARG, "bs_simulate_sources: need at least one source");
    if (prec != BS_PREC_FP64 && prec != BS_PREC_MIXED)
        return fail(BS_ERR_ARG, "bs_simulate_sources: unknown precision");
    for (int32_t i = 0; i < n; i++)
        for (int k = 0; k < 4; k++)
            if (!std::isfinite(sources[4 * i + k]))
                return fail(BS_ERR_ARG, "bs_simulate_sources: source %d is not finite", i + 1);
    const bs_params saved = c->prm;
    const bool saved_reuse = c->reuse;
    c->reuse = true;  // the sphere tables do not depend on the focus or the amplitude
    bs_stats sum{};
    bs_status st = BS_OK;
    for (int32_t i = 0; i < n && st == BS_OK; i++) {
        for (int k = 0; k < 3; k++) c->prm.focus[k] = sources[4 * i + k];
        c->prm.amplitude = sources[4 * i + 3];
        st = simulate_impl(c, prec, i > 0);
        if (st != BS_OK) break;
        const bs_stats& s = c->stats;
        sum.ms_total += s.ms_total;
        sum.ms_uf += s.ms_uf;
        sum.ms_mie += s.ms_mie;
        sum.ms_lut += s.ms_lut;
        sum.ms_us += s.ms_us;
        sum.ms_detector += s.ms_detector;
        sum.kernel_launches += s.kernel_launches;
        sum.us_interactions += s.us_interactions;
        sum.lut_chunks_staged += s.lut_chunks_staged;
        sum.lut_chunks_total += s.lut_chunks_total;
        sum.lut_tables_built += s.lut_tables_built;
        sum.lut_staged_predicted = s.lut_staged_predicted;
        sum.lut_wave_chunk = s.lut_wave_chunk;
    }
    c->reuse = saved_reuse;
    if (!saved_reuse) c->lut_valid = false;
    const bool have = c->have;
    c->prm = saved;
    c->have = have && st == BS_OK;  // images stay valid: they do not depend on prm after the run
    if (st == BS_OK) c->stats = sum;
    return st;
}

}  // extern "C"

template <class T>
static bs_status far_field(bs_ctx* c, int which, double* host) {
    const int C = c->crop, Nv = c->det_Nv;
    const size_t n = (size_t)C * C;
    if (Nv == 0) {  // nothing passes the objective: the far field is zero
        std::fill(host, host + 2 * n, 0.0);
        return BS_OK;
    }
    CK(c->d_far.ensure(n * sizeof(cpx<T>)));
    const T scale = (T)(1.0 / ((double)c->R * (double)c->R));
    const cpx<T>* g1 = c->d_g1.as<cpx<T>>() + (size_t)which * Nv * C;
    launch_cgemm<T>(C, C, Nv, 1, c->d_wiy.as<cpx<T>>(), Nv, 0, g1, C, 0, c->d_far.as<cpx<T>>(), C, 0, 3, nullptr,
                    scale, nullptr, c->d_gscr.as<cpx<T>>(), c->d_gscr.n / sizeof(cpx<T>), c->st);
    LAUNCHED(c);
    std::vector<cpx<T>> t(n);
    CK(cudaMemcpyAsync(t.data(), c->d_far.p, n * sizeof(cpx<T>), cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
    for (size_t i = 0; i < n; i++) {
        host[2 * i] = (double)t[i].re;
        host[2 * i + 1] = (double)t[i].im;
    }
    return BS_OK;
}

extern "C" {

bs_status bs_get_far_field(bs_ctx* c, bs_field_kind kind, double* host, size_t count) {
    if (!c || !host) return fail(BS_ERR_ARG, "bs_get_far_field: null argument");
    if (!c->have) return fail(BS_ERR_STATE, "bs_get_far_field: no simulation result");
    if (kind != BS_FIELD_TOTAL && kind != BS_FIELD_INCIDENT) return fail(BS_ERR_ARG, "bs_get_far_field: unknown field");
    if (count < (size_t)c->crop * c->crop)
        return fail(BS_ERR_ARG, "bs_get_far_field: need %zu complex values", (size_t)c->crop * c->crop);
    const int which = kind == BS_FIELD_TOTAL ? 0 : 1;
    return c->prec == BS_PREC_FP64 ? far_field<double>(c, which, host) : far_field<float>(c, which, host);
}

bs_status bs_material_eval(const char* path, const double* lambdas, int32_t n, double* out) {
    if (!path || n < 0 || (n > 0 && (!lambdas || !out))) return fail(BS_ERR_ARG, "bs_material_eval: bad arguments");
    std::ifstream f(path);
    if (!f) return fail(BS_ERR_IO, "Material Error -- file not found: %s", path);
    std::string text((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
    std::vector<float> lam, re, im;
    std::string err;
    if (!material_load(text, lam, re, im, err)) return fail(BS_ERR_IO, "%s: %s", path, err.c_str());
    for (int32_t i = 0; i < n; i++) {
        float r, k;
        material_eval(lam, re, im, (float)lambdas[i], r, k);
        out[2 * i] = r;
        out[2 * i + 1] = k;
    }
    return BS_OK;
}

bs_status bs_material_kk(const char* path, double n0, int32_t n_samples, int32_t pf, double* lambdas, double* n_out) {
    if (!path || !lambdas || !n_out || n_samples < 0 || pf < 1 || !(n0 > 0))
        return fail(BS_ERR_ARG, "bs_material_kk: bad arguments");
    std::ifstream f(path);
    if (!f) return fail(BS_ERR_IO, "Material Error -- file not found: %s", path);
    std::string text((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
    // rts::material<double>: the instantiation whose arrays match FFTW's double transforms
    std::vector<double> lam, re, im;
    std::string err;
    if (!material_load(text, lam, re, im, err)) return fail(BS_ERR_IO, "%s: %s", path, err.c_str());
    const int N = n_samples ? n_samples : (int)lam.size();
    if (N < 2 || N > BS_KK_MAX_SAMPLES)
        return fail(BS_ERR_ARG, "bs_material_kk: %d samples (2 to %d)", N, BS_KK_MAX_SAMPLES);
    if (pf > 16) return fail(BS_ERR_ARG, "bs_material_kk: padding factor %d above 16", pf);
    const int M = N * pf;
    // resample kappa at evenly spaced wavenumbers, from the shortest wavelength up (material.h:294-316)
    const double nu_min = 10000.0 / lam.back(), nu_max = 10000.0 / lam.front();
    const double dnu = (nu_max - nu_min) / (N - 1);
    std::vector<double> chi2(N), kap(N);
    for (int i = 0; i < N; i++) {
        const double l = 10000.0 / (nu_max - i * dnu);
        double nr, ni;
        material_eval(lam, re, im, l, nr, ni);
        kap[i] = ni;
        const float k = (float)(2 * (float)PI_REF / l);      // float k, alpha as in the reference
        const float alpha = (float)(ni * (double)(2 * k));
        chi2[i] = -(double)alpha * (n0 / (double)k);
        lambdas[i] = l;
    }
    double *d_chi2 = nullptr, *d_g = nullptr, *d_chi1 = nullptr;
    cudaStream_t st = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&d_chi2, N * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&d_g, (size_t)M * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&d_chi1, N * sizeof(double));
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_chi2, chi2.data(), N * sizeof(double), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        launch_kk(N, M, d_chi2, d_g, d_chi1, st);
        e = cudaGetLastError();
    }
    std::vector<double> chi1(N);
    if (e == cudaSuccess) e = cudaMemcpyAsync(chi1.data(), d_chi1, N * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d_chi2);
    cudaFree(d_g);
    cudaFree(d_chi1);
    if (st) cudaStreamDestroy(st);
    if (e != cudaSuccess) return fail(BS_ERR_CUDA, "bs_material_kk: %s", cudaGetErrorString(e));
    for (int i = 0; i < N; i++) {
        n_out[2 * i] = chi1[i] / (2 * n0) + n0;
        n_out[2 * i + 1] = kap[i];
    }
    return BS_OK;
}

}  // extern "C"

// Ring point sources (--interpolate 1, 2, 3; microscope.cu:1004-1253).  Ring
// r = 1, 2, ... has radius r um; its sources sit at the angles of
// generatePointSources (microscope.cu:1298-1325): t_0 = 2 pi / points in float,
// each next one the float sum of the previous and that step; cosines and sines
// are double values rounded to float (the reference used float ones).
static std::vector<float> ring_angles(int points) {
    const float step = 2 * (float)PI_REF / (float)points;
    std::vector<float> t(points);
    float th = step;
    for (int i = 0; i < points; i++) {
        t[i] = th;
        th += step;
    }
    return t;
}

static void stats_add(bs_stats& sum, const bs_stats& s) {
    sum.ms_total += s.ms_total;
    sum.ms_uf += s.ms_uf;
    sum.ms_mie += s.ms_mie;
    sum.ms_lut += s.ms_lut;
    sum.ms_us += s.ms_us;
    sum.ms_detector += s.ms_detector;
    sum.kernel_launches += s.kernel_launches;
    sum.us_interactions += s.us_interactions;
    sum.lut_chunks_staged += s.lut_chunks_staged;
    sum.lut_chunks_total += s.lut_chunks_total;
    sum.lut_tables_built += s.lut_tables_built;
    sum.lut_staged_predicted = s.lut_staged_predicted;
    sum.lut_wave_chunk = s.lut_wave_chunk;
}

// One source of a ring driver at (x, y, z) with amplitude a; its stats are
// added to sum.  The sphere tables are built by the first source and reused.
static bs_status ring_source(bs_ctx* c, bs_precision prec, const double* xyz, double a, bool accumulate,
                             bs_stats& sum) {
    if (xyz)
        for (int k = 0; k < 3; k++) c->prm.focus[k] = xyz[k];
    c->prm.amplitude = a;
    bs_status st = simulate_impl(c, prec, accumulate);
    if (st == BS_OK) stats_add(sum, c->stats);
    return st;
}

// The detector images of the near field in d_fields rotated by each angle,
// added to the detector (nearfieldStruct::Interpolate + SimulateImaging,
// microscope.cu:834-846); d_fields itself is kept in d_fsave and overwritten.
template <class T>
static bs_status field_rotations(bs_ctx* c, const std::vector<float>& angles) {
    const size_t n = 2 * (size_t)c->R * c->R;
    CK(c->d_fsave.ensure(n * sizeof(cpx<T>)));
    CK(cudaMemcpyAsync(c->d_fsave.p, c->d_fields.p, n * sizeof(cpx<T>), cudaMemcpyDeviceToDevice, c->st));
    for (float a : angles) {
        launch_rotate_fields<T>(c->R, (float)std::cos((double)a), (float)std::sin((double)a), c->d_fsave.as<cpx<T>>(),
                                c->d_fields.as<cpx<T>>(), c->st);
        LAUNCHED(c);
        bs_status st = run_detector<T>(c, true);
        if (st != BS_OK) return st;
    }
    CK(cudaStreamSynchronize(c->st));
    CK(cudaGetLastError());
    return BS_OK;
}

// Mode 1 (InterpAtDetector, microscope.cu:312-321): the sum so far is in
// d_dacc, the ring's first source alone in d_D; both are added to d_dacc, then
// that image rotated by each angle.
template <class T>
static bs_status image_rotations(bs_ctx* c, const std::vector<float>& angles) {
    const T* one = c->d_D.as<T>();
    T* acc = c->d_dacc.as<T>();
    launch_rotate_add_images<T>(c->res, 1.f, 0.f, one, acc, c->st);  // angle 0: the image itself
    LAUNCHED(c);
    for (float a : angles) {
        launch_rotate_add_images<T>(c->res, (float)std::cos((double)a), (float)std::sin((double)a), one, acc, c->st);
        LAUNCHED(c);
    }
    CK(cudaStreamSynchronize(c->st));
    CK(cudaGetLastError());
    return BS_OK;
}

// Mode 2 (InterpLineForAllPointSources, microscope.cu:336-354): the current
// source's D and Di feed their radial lines.
template <class T>
static bs_status line_samples(bs_ctx* c, int points, int L) {
    launch_ring_line<T>(c->res, points, L, c->d_ringcs.as<float2>(), c->d_D.as<T>(), c->d_line.as<T>(), c->st);
    LAUNCHED(c);
    CK(cudaGetLastError());
    return BS_OK;
}

// Shared frame of the ring drivers: tables reused across the sources, the
// context's focus, amplitude and reuse setting restored afterwards.
template <class F>
static bs_status ring_driver(bs_ctx* c, bs_precision prec, int32_t points, int32_t rings, const char* name, F&& body) {
    if (!c || points < 1 || rings < 1) return fail(BS_ERR_ARG, "%s: points and rings must be >= 1", name);
    if (prec != BS_PREC_FP64 && prec != BS_PREC_MIXED) return fail(BS_ERR_ARG, "%s: unknown precision", name);
    const bs_params saved = c->prm;
    const bool saved_reuse = c->reuse;
    c->reuse = true;  // the sphere tables do not depend on the focus or the amplitude
    bs_stats sum{};
    bs_status st = body(sum);
    c->prm = saved;
    c->reuse = saved_reuse;
    if (!saved_reuse) c->lut_valid = false;
    if (st != BS_OK) {
        c->have = false;
        return st;
    }
    c->stats = sum;
    c->have = true;
    return BS_OK;
}

static void ring_focus(float t0, int ring, double* xyz) {
    xyz[0] = (float)std::cos((double)t0) * (float)ring;
    xyz[1] = (float)std::sin((double)t0) * (float)ring;
    xyz[2] = 0;
}

extern "C" {

bs_status bs_simulate_ring_interp(bs_ctx* c, int32_t points, int32_t rings, bs_precision prec) {
    return ring_driver(c, prec, points, rings, "bs_simulate_ring_interp", [&](bs_stats& sum) {
        // the source at the context's own focus (SimulateExtendedSourceWithInterpolation, microscope.cu:1189-1253)
        bs_status st = ring_source(c, prec, nullptr, c->prm.amplitude, false, sum);
        const std::vector<float> th = ring_angles(points);
        const std::vector<float> rest(th.begin() + 1, th.end());
        for (int ring = 1; ring < rings && st == BS_OK; ring++) {
            double f[3];
            ring_focus(th[0], ring, f);
            // only a ring's first source is simulated; source i's near field is that one rotated by its angle
            st = ring_source(c, prec, f, 1.0, true, sum);
            if (st == BS_OK && !rest.empty())
                st = prec == BS_PREC_FP64 ? field_rotations<double>(c, rest) : field_rotations<float>(c, rest);
        }
        return st;
    });
}

bs_status bs_simulate_ring_detector(bs_ctx* c, int32_t points, int32_t rings, bs_precision prec) {
    return ring_driver(c, prec, points, rings, "bs_simulate_ring_detector", [&](bs_stats& sum) {
        // SimulateExtendedSourceInterpAtDetector (microscope.cu:1004-1093)
        bs_status st = ring_source(c, prec, nullptr, c->prm.amplitude, false, sum);
        if (st != BS_OK) return st;
        const size_t bytes = 2 * (size_t)c->res * c->res * elem_r(prec);
        CK(c->d_dacc.ensure(bytes));
        CK(cudaMemcpyAsync(c->d_dacc.p, c->d_D.p, bytes, cudaMemcpyDeviceToDevice, c->st));
        const std::vector<float> th = ring_angles(points);
        const std::vector<float> rest(th.begin() + 1, th.end());
        for (int ring = 1; ring < rings && st == BS_OK; ring++) {
            double f[3];
            ring_focus(th[0], ring, f);
            st = ring_source(c, prec, f, 1.0, false, sum);  // d_D: this source alone (saveDetectorForOnePs)
            if (st == BS_OK)
                st = prec == BS_PREC_FP64 ? image_rotations<double>(c, rest) : image_rotations<float>(c, rest);
        }
        if (st != BS_OK) return st;
        CK(cudaMemcpyAsync(c->d_D.p, c->d_dacc.p, bytes, cudaMemcpyDeviceToDevice, c->st));
        CK(cudaStreamSynchronize(c->st));
        return BS_OK;
    });
}

bs_status bs_simulate_ring_line(bs_ctx* c, int32_t points, int32_t rings, bs_precision prec) {
    if (points > BS_RING_LINE_MAX_POINTS)
        return fail(BS_ERR_ARG, "bs_simulate_ring_line: at most %d points per ring (one thread block per ring)",
                    BS_RING_LINE_MAX_POINTS);
    return ring_driver(c, prec, points, rings, "bs_simulate_ring_line", [&](bs_stats& sum) {
        // SimulateExtendedSourceInterpLineAtDetector (microscope.cu:1097-1183): the context's focus, then
        // (j, 0, 0) for j = 1 .. rings-1, all with amplitude 1; every source's image feeds the radial lines
        // of `rings` entries, which then replace the detector images.
        const size_t er = elem_r(prec), L = (size_t)rings;
        CK(c->d_line.ensure(2 * L * er));
        CK(cudaMemsetAsync(c->d_line.p, 0, 2 * L * er, c->st));
        std::vector<float2> cs(points);
        for (int k = 0; k < points; k++) {
            const float t = (float)((2.0 * PI_REF / points) * (k + 1));
            cs[k] = make_float2((float)std::cos((double)t), (float)std::sin((double)t));
        }
        CK(c->d_ringcs.ensure(cs.size() * sizeof(float2)));
        CK(cudaMemcpyAsync(c->d_ringcs.p, cs.data(), cs.size() * sizeof(float2), cudaMemcpyHostToDevice, c->st));
        bs_status st = BS_OK;
        for (int j = 0; j < rings && st == BS_OK; j++) {
            const double f[3] = {(double)j, 0, 0};
            st = ring_source(c, prec, j == 0 ? nullptr : f, 1.0, false, sum);
            if (st == BS_OK) st = prec == BS_PREC_FP64 ? line_samples<double>(c, points, rings)
                                                       : line_samples<float>(c, points, rings);
        }
        if (st != BS_OK) return st;
        if (prec == BS_PREC_FP64)
            launch_line_image<double>(c->res, rings, c->d_line.as<double>(), c->d_D.as<double>(), c->st);
        else
            launch_line_image<float>(c->res, rings, c->d_line.as<float>(), c->d_D.as<float>(), c->st);
        LAUNCHED(c);
        CK(cudaStreamSynchronize(c->st));
        CK(cudaGetLastError());
        return BS_OK;
    });
}

bs_status bs_plane_point(const bs_params* params, double u, double v, double* xyz) {
    if (!params || !xyz) return fail(BS_ERR_ARG, "bs_plane_point: null argument");
    Quad q = quad_from(params->plane_min, params->plane_max, params->plane_normal);
    xyz[0] = q.A.x + q.X.x * u + q.Y.x * v;
    xyz[1] = q.A.y + q.X.y * u + q.Y.y * v;
    xyz[2] = q.A.z + q.X.z * u + q.Y.z * v;
    return BS_OK;
}

extern "C++" {

// An image into the caller's res x res values of type H; the detector images themselves need no kernel, and
// values of the run's own type no staging.
template <class T, class H>
static bs_status image_values(bs_ctx* c, bs_image_kind kind, H* host) {
    const size_t n = (size_t)c->res * c->res;
    const T* img = c->d_D.as<T>() + (kind == BS_IMG_INCIDENT ? n : 0);
    if (kind > BS_IMG_INCIDENT) {
        CK(c->d_img.ensure(n * sizeof(T)));
        launch_image<T>((int)n, kind, img, img + n, c->d_img.as<T>(), c->st);
        LAUNCHED(c);
        img = c->d_img.as<T>();
    }
    std::vector<T> tmp(sizeof(T) > sizeof(H) ? n : 0);
    // floats for a double buffer go to its upper half and are widened from the front
    T* to = sizeof(T) > sizeof(H) ? tmp.data() : reinterpret_cast<T*>(host) + (sizeof(H) / sizeof(T) - 1) * n;
    CK(cudaMemcpyAsync(to, img, n * sizeof(T), cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
    if (sizeof(T) != sizeof(H))
        for (size_t k = 0; k < n; k++) {
            T v;
            std::memcpy(&v, to + k, sizeof(T));
            const H h = (H)v;
            std::memcpy(host + k, &h, sizeof(H));
        }
    return BS_OK;
}

template <class H>
static bs_status image_to_host(bs_ctx* c, bs_image_kind kind, H* host) {
    if (!c->have) return fail(BS_ERR_STATE, "no simulation result (call bs_simulate first)");
    if (kind < BS_IMG_INTENSITY || kind > BS_IMG_TRANSMITTANCE) return fail(BS_ERR_ARG, "unknown image kind");
    return c->prec == BS_PREC_FP64 ? image_values<double>(c, kind, host) : image_values<float>(c, kind, host);
}

}  // extern "C++"

bs_status bs_get_image(bs_ctx* c, bs_image_kind kind, float* host, size_t count) {
    if (!host) return fail(BS_ERR_ARG, "bs_get_image: null buffer");
    if (c && count < (size_t)c->res * c->res) return fail(BS_ERR_ARG, "bs_get_image: buffer holds %zu of %d values", count, c->res * c->res);
    if (!c) return fail(BS_ERR_ARG, "null context");
    return image_to_host(c, kind, host);
}

bs_status bs_get_image_f64(bs_ctx* c, bs_image_kind kind, double* host, size_t count) {
    if (!host) return fail(BS_ERR_ARG, "bs_get_image_f64: null buffer");
    if (c && count < (size_t)c->res * c->res) return fail(BS_ERR_ARG, "bs_get_image_f64: buffer too small");
    if (!c) return fail(BS_ERR_ARG, "null context");
    return image_to_host(c, kind, host);
}

bs_status bs_get_field(bs_ctx* c, bs_field_kind kind, double* host, size_t count) {
    if (!c || !host) return fail(BS_ERR_ARG, "bs_get_field: null argument");
    if (!c->have) return fail(BS_ERR_STATE, "bs_get_field: no simulation result");
    size_t n = (size_t)c->R * c->R;
    if (count < n) return fail(BS_ERR_ARG, "bs_get_field: buffer holds %zu of %zu complex values", count, n);
    size_t off = (kind == BS_FIELD_INCIDENT) ? n : 0;
    if (c->prec == BS_PREC_FP64) {
        CK(cudaMemcpy(host, c->d_fields.as<zd>() + off, n * sizeof(zd), cudaMemcpyDeviceToHost));
    } else {
        std::vector<cpx<float>> tmp(n);
        CK(cudaMemcpy(tmp.data(), c->d_fields.as<cpx<float>>() + off, n * sizeof(cpx<float>), cudaMemcpyDeviceToHost));
        for (size_t i = 0; i < n; i++) {
            host[2 * i] = tmp[i].re;
            host[2 * i + 1] = tmp[i].im;
        }
    }
    return BS_OK;
}

bs_status bs_write_envi(bs_ctx* c, bs_image_kind kind, const char* path, int32_t append, double band_value) {
    if (!path) return fail(BS_ERR_ARG, "bs_write_envi: null path");
    if (!c) return fail(BS_ERR_ARG, "null context");
    std::vector<float> f((size_t)c->res * c->res);
    bs_status st = image_to_host(c, kind, f.data());
    if (st != BS_OK) return st;
    char err[512] = {0};
    if (envi_add_band(path, f.data(), c->res, c->res, band_value, append, err, sizeof(err)) != 0)
        return fail(BS_ERR_IO, "%s", err);
    return BS_OK;
}

bs_status bs_envi_add_band(const char* path, const float* band, int32_t samples, int32_t lines, double band_value,
                           int32_t append) {
    if (!path || !band || samples < 1 || lines < 1) return fail(BS_ERR_ARG, "bs_envi_add_band: bad argument");
    char err[512] = {0};
    if (envi_add_band(path, band, samples, lines, band_value, append, err, sizeof(err)) != 0)
        return fail(BS_ERR_IO, "%s", err);
    return BS_OK;
}

bs_status bs_sweep(bs_ctx* c, const double* lambdas, int32_t nl, const double* n_table, bs_precision prec,
                   bs_image_kind kind, float* images, const char* envi_path, int32_t band_as_nu) {
    if (!c || !lambdas || nl < 1) return fail(BS_ERR_ARG, "bs_sweep: need at least one wavelength");
    const size_t ns = c->spheres.size();
    if (ns > 0 && !n_table) return fail(BS_ERR_ARG, "bs_sweep: need the refractive-index table");
    for (int32_t l = 0; l < nl; l++)
        if (!(lambdas[l] > 0)) return fail(BS_ERR_ARG, "bs_sweep: wavelength %d is not positive", l + 1);
    const bs_params saved_p = c->prm;
    const std::vector<bs_sphere> saved_s = c->spheres;
    const size_t npix = (size_t)c->prm.resolution * c->prm.resolution;
    bs_status st = BS_OK;
    for (int32_t l = 0; l < nl && st == BS_OK; l++) {
        c->prm.lambda = lambdas[l];
        for (size_t i = 0; i < ns; i++) {
            c->spheres[i].n_re = n_table[2 * ((size_t)l * ns + i)];
            c->spheres[i].n_im = n_table[2 * ((size_t)l * ns + i) + 1];
        }
        st = bs_simulate(c, prec);
        if (st == BS_OK && images) st = bs_get_image(c, kind, images + (size_t)l * npix, npix);
        if (st == BS_OK && envi_path)
            st = bs_write_envi(c, kind, envi_path, l > 0, band_as_nu ? 1e4 / lambdas[l] : lambdas[l]);
    }
    c->prm = saved_p;
    c->spheres = saved_s;
    c->have = false;
    return st;
}

bs_status bs_get_info(bs_ctx* c, bs_info* out) {
    if (!c || !out) return fail(BS_ERR_ARG, "bs_get_info: null argument");
    const bs_params& p = c->prm;
    int R = p.resolution * p.supersample * (2 * p.padding + 1);
    out->nf_res = R;
    out->det_res = p.resolution;
    out->n_spheres = (int)c->spheres.size();
    out->n_waves = p.plane_wave ? 1 : (int)(c->waves.size() / 3);
    out->uf_lut_r = p.uf_lut_r > 0 ? p.uf_lut_r : 2 * R;
    out->us_lut_theta = p.us_lut_theta > 0 ? p.us_lut_theta : 1000;
    int64_t tot = 0;
    for (const DevBuf* b : ctx_bufs(c)) tot += (int64_t)b->n;
    out->device_bytes = tot;
    return BS_OK;
}

bs_status bs_get_stats(bs_ctx* c, bs_stats* out) {
    if (!c || !out) return fail(BS_ERR_ARG, "bs_get_stats: null argument");
    *out = c->stats;
    return BS_OK;
}

bs_status bs_get_mie(bs_ctx* c, int32_t sphere, double* A, double* B, int32_t count) {
    if (!c || !A || !B) return fail(BS_ERR_ARG, "bs_get_mie: null argument");
    if (!c->have || sphere < 0 || sphere >= (int)c->hs.size() || !c->prm.scalar)
        return fail(BS_ERR_STATE, "bs_get_mie: no coefficients for sphere %d", sphere);
    const Sphere& S = c->hs[sphere];
    if (count < S.Nl + 1) return fail(BS_ERR_ARG, "bs_get_mie: need %d orders", S.Nl + 1);
    CK(cudaMemcpy(A, c->d_A.as<zd>() + S.coef_off, (S.Nl + 1) * sizeof(zd), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(B, c->d_B.as<zd>() + S.coef_off, (S.Nl + 1) * sizeof(zd), cudaMemcpyDeviceToHost));
    return BS_OK;
}

bs_status bs_get_lut(bs_ctx* c, int32_t sphere, int32_t which, double* host, size_t count) {
    if (!c || !host) return fail(BS_ERR_ARG, "bs_get_lut: null argument");
    if (!c->have || !c->prm.lut_us || !c->prm.scalar || sphere < 0 || sphere >= (int)c->hs.size())
        return fail(BS_ERR_STATE, "bs_get_lut: no table for sphere %d", sphere);
    const Sphere& S = c->hs[sphere];
    size_t rows = which == 0 ? S.dR : S.aR;
    size_t n = rows * S.thetaR;
    if (count < n) return fail(BS_ERR_ARG, "bs_get_lut: need %zu complex values", n);
    int64_t off = which == 0 ? S.usp_off : S.uip_off;
    if (c->prec == BS_PREC_FP64) {
        std::vector<Patch<double>> t(n);
        CK(cudaMemcpy(t.data(), c->d_lut.as<Patch<double>>() + off, n * sizeof(Patch<double>), cudaMemcpyDeviceToHost));
        for (size_t i = 0; i < n; i++) {
            host[2 * i] = t[i].v[0];
            host[2 * i + 1] = t[i].v[1];
        }
    } else {
        if (sphere < c->tab_s0 || sphere >= c->tab_s1)
            return fail(BS_ERR_STATE, "bs_get_lut: table of sphere %d not resident", sphere);
        std::vector<float2> t(n);
        CK(cudaMemcpy2D(t.data(), S.thetaR * sizeof(float2), c->d_lut.as<float2>() + off, S.lin_stride * sizeof(float2),
                        S.thetaR * sizeof(float2), rows, cudaMemcpyDeviceToHost));
        for (size_t i = 0; i < n; i++) {
            host[2 * i] = t[i].x;
            host[2 * i + 1] = t[i].y;
        }
    }
    return BS_OK;
}

}  // extern "C"
