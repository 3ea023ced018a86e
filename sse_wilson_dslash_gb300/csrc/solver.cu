// Even-odd preconditioned Wilson solver on one GPU.
//
//   M = 1 - kappa^2 D_eo D_oe   on checkerboard 0 (even sites), D = the
//   Dslash of this library (D_oe: even source -> odd target, cb = 0;
//   D_eo: odd source -> even target, cb = 1); M^+ is the same with isign = -1.
//
// CG on the normal equations A x = c, A = M^+ M, c = M^+ b.
//   inner_prec 64: all-FP64 CG.
//   inner_prec 32: FP32 CG (FP32 fields, FP32 arithmetic, per-block sums in
//                  FP64) inside FP64 defect correction: the residual
//                  r = b - M x, the solution update and all global norms stay
//                  in FP64 on the GPU; the inner right-hand side M^+ r is
//                  formed in FP32 (two FP64 Dslash applications per cycle
//                  instead of four).  The normal-equation solve keeps
//                  r = c - A x in FP64.
//   inner_prec 16 / 17: the same with the CG's direction p and the operator's
//                  intermediates (M p, D_oe p) stored as half with a
//                  per-site norm (16) or bfloat16 (17), FP16 links, FP32
//                  arithmetic; the CG's solution and residual stay FP32.
// The reference library provides only D; a caller such as Chroma builds M and
// its solvers around it (tests/dslashm_w.cc states D the same way).  Scalars
// of the iteration (rr, pAp, alpha, beta) live in device memory and are
// computed by the kernels themselves; the host reads rr only to test
// convergence.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <vector>

#include "dslash_gen.cuh"

namespace gbds {
namespace {

using Scalars = CgScalars;

constexpr int kThreads = 128;

inline int blocks(const Geom &g) { return (g.Vh + kThreads - 1) / kThreads; }

template <typename T> using SV = typename VecOf<T>::S;  // float4 / double2
template <typename T> constexpr int nvec() { return sizeof(T) == 4 ? 6 : 12; }

__device__ __forceinline__ float4 axpy_v(float a, float4 x, float4 y) {
    return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}
__device__ __forceinline__ double2 axpy_v(double a, double2 x, double2 y) {
    return make_double2(fma(a, x.x, y.x), fma(a, x.y, y.y));
}
__device__ __forceinline__ float norm_v(float4 v) { return v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w; }
__device__ __forceinline__ double norm_v(double2 v) { return v.x * v.x + v.y * v.y; }

// x += alpha p;  p = r + beta p  (r -= alpha A p is M^+'s second launch's, the
// update epilogue of the Dslash kernels)
template <typename T>
__global__ void __launch_bounds__(kThreads) cg_xpay(const SV<T> *__restrict__ r, SV<T> *x, SV<T> *p, const Scalars *sc,
                                                   int Vh, int stride) {
    pdl_allow_next();
    pdl_wait_prev();
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
    const T a = (T)sc->alpha, b = (T)sc->beta;
#pragma unroll
    for (int k = 0; k < nvec<T>(); k++) {
        const size_t i = (size_t)k * stride + h;
        const SV<T> pv = p[i];
        x[i] = axpy_v(a, pv, x[i]);
        p[i] = axpy_v(b, pv, r[i]);
    }
}

// r = c - v; partial |r|^2  (FP64 defect residual)
__global__ void __launch_bounds__(kThreads) xmy_norm(const double2 *__restrict__ c, const double2 *__restrict__ v,
                                                    double2 *r, int Vh, int stride, double *partials) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    double nrm = 0;
    if (h < Vh) {
#pragma unroll
        for (int k = 0; k < 12; k++) {
            const size_t i = (size_t)k * stride + h;
            const double2 d = make_double2(c[i].x - v[i].x, c[i].y - v[i].y);
            r[i] = d;
            nrm += norm_v(d);
        }
    }
    block_sum_to<double>(partials, nrm);
}

// r = c - v for v in double-float (the outer residual's M x); partial |r|^2
__global__ void __launch_bounds__(kThreads) xmy_norm_df(const double2 *__restrict__ c, const float4 *__restrict__ v,
                                                       double2 *r, int Vh, int stride, double *partials) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    double nrm = 0;
    if (h < Vh) {
#pragma unroll
        for (int k = 0; k < 12; k++) {
            const size_t i = (size_t)k * stride + h;
            const double2 m = df_to_double2(v[i]);
            const double2 d = make_double2(c[i].x - m.x, c[i].y - m.y);
            r[i] = d;
            nrm += norm_v(d);
        }
    }
    block_sum_to<double>(partials, nrm);
}

// partial |v|^2, and optionally dst = v
template <typename T>
__global__ void __launch_bounds__(kThreads) norm_copy(const SV<T> *__restrict__ v, SV<T> *dst, SV<T> *dst2, int Vh,
                                                     int stride, double *partials) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    T nrm = 0;
    if (h < Vh) {
#pragma unroll
        for (int k = 0; k < nvec<T>(); k++) {
            const size_t i = (size_t)k * stride + h;
            const SV<T> a = v[i];
            if (dst) dst[i] = a;
            if (dst2) dst2[i] = a;
            nrm += norm_v(a);
        }
    }
    block_sum_to<T>(partials, nrm);
}

template <typename T>
__global__ void __launch_bounds__(kThreads) zero_field(SV<T> *v, int Vh, int stride) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
    const SV<T> z = {};
#pragma unroll
    for (int k = 0; k < nvec<T>(); k++) v[(size_t)k * stride + h] = z;
}

// r32 = r64 / sqrt(outer_rr);  p32 = r32
__global__ void __launch_bounds__(kThreads) demote_residual(const double2 *__restrict__ r64, float4 *r32, float4 *p32,
                                                           const Scalars *sc, int Vh, int stride) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
    const double s = 1.0 / sqrt(sc->outer_rr);
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const double2 a = r64[(size_t)(2 * k) * stride + h], b = r64[(size_t)(2 * k + 1) * stride + h];
        const float4 f = make_float4((float)(a.x * s), (float)(a.y * s), (float)(b.x * s), (float)(b.y * s));
        r32[(size_t)k * stride + h] = f;
        p32[(size_t)k * stride + h] = f;
    }
}

// x64 += sqrt(outer_rr) * e32
__global__ void __launch_bounds__(kThreads) promote_update(const float4 *__restrict__ e32, double2 *x64,
                                                          const Scalars *sc, int Vh, int stride) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
    const double s = sqrt(sc->outer_rr);
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const float4 e = e32[(size_t)k * stride + h];
        double2 &a = x64[(size_t)(2 * k) * stride + h];
        double2 &b = x64[(size_t)(2 * k + 1) * stride + h];
        a.x = fma(s, (double)e.x, a.x);
        a.y = fma(s, (double)e.y, a.y);
        b.x = fma(s, (double)e.z, b.x);
        b.y = fma(s, (double)e.w, b.y);
    }
}

// r32 = inv * r64
__global__ void __launch_bounds__(kThreads) demote_scaled(const double2 *__restrict__ r64, double inv, float4 *r32,
                                                         int Vh, int stride) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const double2 a = r64[(size_t)(2 * k) * stride + h], b = r64[(size_t)(2 * k + 1) * stride + h];
        r32[(size_t)k * stride + h] =
            make_float4((float)(a.x * inv), (float)(a.y * inv), (float)(b.x * inv), (float)(b.y * inv));
    }
}

// r32 = a * v;  p32 = r32
__global__ void __launch_bounds__(kThreads) scale_copy(const float4 *__restrict__ v, float a, float4 *r32, float4 *p32,
                                                      int Vh, int stride) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const float4 x = v[(size_t)k * stride + h];
        const float4 y = make_float4(a * x.x, a * x.y, a * x.z, a * x.w);
        r32[(size_t)k * stride + h] = y;
        p32[(size_t)k * stride + h] = y;
    }
}

// x64 += s * e32
__global__ void __launch_bounds__(kThreads) promote_scaled(const float4 *__restrict__ e32, double s, double2 *x64, int Vh,
                                                          int stride) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const float4 e = e32[(size_t)k * stride + h];
        double2 &a = x64[(size_t)(2 * k) * stride + h];
        double2 &b = x64[(size_t)(2 * k + 1) * stride + h];
        a.x = fma(s, (double)e.x, a.x);
        a.y = fma(s, (double)e.y, a.y);
        b.x = fma(s, (double)e.z, b.x);
        b.y = fma(s, (double)e.w, b.y);
    }
}

// --- 16-bit direction vectors (Sio formats), FP32 solution and residual ---

// float4 component k of a spinor holds complexes 2k and 2k+1
__device__ __forceinline__ float4 pair(const cx<float> (&s)[4][3], int k) {
    const cx<float> a = s[(2 * k) / 3][(2 * k) % 3], b = s[(2 * k + 1) / 3][(2 * k + 1) % 3];
    return make_float4(a.r, a.i, b.r, b.i);
}

// x += alpha p;  p = r + beta p   (p 16-bit)
template <int FMT>
__global__ void __launch_bounds__(kThreads) cg_xpay_h(const float4 *__restrict__ r, float4 *x, char *p, const Scalars *sc,
                                                     int Vh, int stride) {
    pdl_allow_next();
    pdl_wait_prev();
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
    const float a = (float)sc->alpha, b = (float)sc->beta;
    cx<float> ps[4][3];
    Sio<FMT>::load(p, stride, h, ps);
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const size_t i = (size_t)k * stride + h;
        const float4 rv = r[i];
        x[i] = axpy_v(a, pair(ps, k), x[i]);
        cx<float> &u = ps[(2 * k) / 3][(2 * k) % 3];
        cx<float> &v = ps[(2 * k + 1) / 3][(2 * k + 1) % 3];
        u = {fmaf(b, u.r, rv.x), fmaf(b, u.i, rv.y)};
        v = {fmaf(b, v.r, rv.z), fmaf(b, v.i, rv.w)};
    }
    Sio<FMT>::store(p, stride, h, ps);
}

// r32 = r64 / sqrt(outer_rr);  p = r32 (16-bit)
template <int FMT>
__global__ void __launch_bounds__(kThreads) demote_residual_h(const double2 *__restrict__ r64, float4 *r32, char *p,
                                                             const Scalars *sc, int Vh, int stride) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
    const double s = 1.0 / sqrt(sc->outer_rr);
    cx<float> ps[4][3];
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const double2 a = r64[(size_t)(2 * k) * stride + h], b = r64[(size_t)(2 * k + 1) * stride + h];
        const float4 f = make_float4((float)(a.x * s), (float)(a.y * s), (float)(b.x * s), (float)(b.y * s));
        r32[(size_t)k * stride + h] = f;
        ps[(2 * k) / 3][(2 * k) % 3] = {f.x, f.y};
        ps[(2 * k + 1) / 3][(2 * k + 1) % 3] = {f.z, f.w};
    }
    Sio<FMT>::store(p, stride, h, ps);
}

// r32 = a * v;  p = r32 (16-bit)
template <int FMT>
__global__ void __launch_bounds__(kThreads) scale_copy_h(const float4 *__restrict__ v, float a, float4 *r32, char *p,
                                                        int Vh, int stride) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
    cx<float> ps[4][3];
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const float4 x = v[(size_t)k * stride + h];
        const float4 f = make_float4(a * x.x, a * x.y, a * x.z, a * x.w);
        r32[(size_t)k * stride + h] = f;
        ps[(2 * k) / 3][(2 * k) % 3] = {f.x, f.y};
        ps[(2 * k + 1) / 3][(2 * k + 1) % 3] = {f.z, f.w};
    }
    Sio<FMT>::store(p, stride, h, ps);
}

// Deterministic sum of the block partials (fixed order), then the scalar step.
__global__ void __launch_bounds__(1024) finish(const double *partials, int n, Scalars *sc, int mode) {
    pdl_allow_next();
    pdl_wait_prev();
    __shared__ double buf[1024];
    double t = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) t += partials[i];
    buf[threadIdx.x] = t;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) buf[threadIdx.x] += buf[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    sum_step(sc, mode, buf[0]);
}

__global__ void f64_to_f32(const double *__restrict__ a, float *b, size_t n) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

}  // namespace
}  // namespace gbds

using namespace gbds;

// kCheck iterations of an inner CG less their first part, recorded once per
// solver (every buffer is the solver's own) and launched as one CUDA graph: a
// small lattice's iteration is bound by the host's seven launches of about 3 us
// each.  us an iteration, launched one by one / as a graph: 8^3x16 35.3 / 32.8, 16^3x32
// 64.8 / 62.5, 24^3x48 202.6 / 201.2; 16 rhs on 16^3x32 38.0 / 37.5 ms a solve.
constexpr int kCheck = 4;  // iterations between convergence tests
struct IterGraph {
    cudaGraphExec_t exec = nullptr;
    int launches = 0;
};

struct gbds_solver_s {
    Geom g;
    gbds_solver_params prm;
    void *gauge64 = nullptr;  // FP64, recon 18
    void *gauge32 = nullptr;  // FP32, inner recon
    // mixed solves with outer_double_float: the outer residual's operator in
    // double-float (dfloat.cuh) on the FP32 pipes: the links, and the
    // solution converted for it
    void *gauge_df = nullptr, *xdf = nullptr;
    // FP64 fields (checkerboard 0 except t64: checkerboard 1)
    void *b64 = nullptr, *c64 = nullptr, *x64 = nullptr, *r64 = nullptr, *p64 = nullptr, *Ap64 = nullptr,
         *Mp64 = nullptr, *t64 = nullptr;
    // FP32 inner fields
    void *e32 = nullptr, *r32 = nullptr, *p32 = nullptr, *Mp32 = nullptr, *t32 = nullptr;
    // 16-bit inner fields and FP16 links (inner_prec 16 / 17)
    void *p16 = nullptr, *Mp16 = nullptr, *t16 = nullptr, *gauge16 = nullptr;
    int fmt16 = 0;
    double *partials = nullptr;
    Scalars *sc = nullptr;    // device
    Scalars *hsc = nullptr;   // pinned host copy
    cudaEvent_t read = nullptr;  // the copy of a convergence test has arrived
    IterGraph steps;             // the inner CG's
    unsigned *ticket = nullptr;  // 0 between launches (SumHere)
    bool have_gauge = false;
};

namespace {

// Dslash launches through the precision-specific entry points (the kernels are
// instantiated once, in dslash_f32.cu / dslash_f64.cu).
template <typename T>
cudaError_t dslash(const Geom &g, int recon, const void *gauge, const void *psi, void *res, int isign, int cb,
                   cudaStream_t st) {
    if constexpr (sizeof(T) == 4) {
        int block, variant;
        f32_tuning(g, recon, &block, &variant);
        return launch_dslash_f32(g, recon, gauge, psi, res, isign, cb, block, variant, st);
    } else return launch_dslash_f64(g, recon, gauge, psi, res, isign, cb, st);
}

template <typename T>
cudaError_t dslash_xpay(const Geom &g, int recon, const void *gauge, const void *psi, const void *x, T coef, void *res,
                        double *partials, int isign, int cb, cudaStream_t st, const SumHere &here) {
    if constexpr (sizeof(T) == 4)
        return launch_dslash_xpay_f32(g, recon, gauge, psi, x, coef, res, partials, isign, cb, st, here);
    else return launch_dslash_xpay_f64(g, gauge, psi, x, coef, res, partials, isign, cb, st);
}

// n: the partials to add up (0: one per 128-site block); to: the scalars (default:
// the solver's)
cudaError_t finish_on(gbds_solver s, int mode, cudaStream_t st, int n = 0, Scalars *to = nullptr) {
    launch_pdl(finish, dim3(1), 1024, st, (const double *)s->partials, n ? n : blocks(s->g), to ? to : s->sc, mode);
    count_launch();
    return cudaGetLastError();
}

// out_e = in_e - kappa^2 D_eo(isign) D_oe(isign) in_e  (partials: |out|^2)
template <typename T>
cudaError_t apply_M(gbds_solver s, const void *gauge, int recon, const void *in, void *tmp, void *out, int isign,
                    double *partials, cudaStream_t st, const SumHere &here = {}) {
    const Geom &g = s->g;
    const double k2 = s->prm.kappa * s->prm.kappa;
    cudaError_t e = dslash<T>(g, recon, gauge, in, tmp, isign, 0, st);
    if (e != cudaSuccess) return e;
    return dslash_xpay<T>(g, recon, gauge, tmp, in, (T)(-k2), out, partials, isign, 1, st, here);
}

// r -= alpha M^+ in, |r|^2 in the partials: M^+'s second launch updates r in
// place of storing M^+ in
template <typename T>
cudaError_t apply_Mdag_update(gbds_solver s, const void *gauge, int recon, const void *in, void *tmp, void *r,
                              cudaStream_t st, const SumHere &here) {
    const Geom &g = s->g;
    const double k2 = s->prm.kappa * s->prm.kappa;
    cudaError_t e = dslash<T>(g, recon, gauge, in, tmp, -1, 0, st);
    if (e != cudaSuccess) return e;
    if constexpr (sizeof(T) == 4)
        return launch_dslash_cg_update_f32(g, recon, gauge, tmp, in, (float)(-k2), &s->sc->alpha, r, s->partials, -1, 1, st,
                                           here);
    else return launch_dslash_cg_update_f64(g, gauge, tmp, in, -k2, &s->sc->alpha, r, s->partials, -1, 1, st);
}

// The outer residual's operator in double-float (outer_double_float): out
// (double-float, in the storage of an FP64 field) = M in for the FP64 field
// `in`, which is converted into xdf first.  About 48 significant bits: the
// residual b - M x is exact to ~1e-14 |b|, far below the tolerances the
// defect correction reaches, at a fraction of the FP64 operator's time (GB300
// issues FP64 at 1/64 of the FP32 rate).  By default the FP64 operator forms
// the residual.
constexpr int kDfVariant = 0;  // the colour-split kernel (dslash_df.cu)

cudaError_t apply_M_df(gbds_solver s, const void *in64, void *out_df, int isign, cudaStream_t st) {
    const Geom &g = s->g;
    const double k2 = s->prm.kappa * s->prm.kappa;
    cudaError_t e = launch_f64_to_df(in64, s->xdf, spinor_bytes(g, 64) / 16, st);
    if (e == cudaSuccess) e = launch_dslash_df(g, 18, s->gauge_df, s->xdf, s->t64, isign, 0, 128, kDfVariant, st);
    if (e != cudaSuccess) return e;
    return launch_dslash_xpay_df(g, s->gauge_df, s->t64, s->xdf, -k2, out_df, isign, 1, st);
}

// Fields within FP32's exponent range (the double-float operator's): |b|^2
// well inside it, else the FP64 operator forms the residual.
bool df_range(double b2) { return b2 > 1e-50 && b2 < 1e50; }

// r = b - M x (FP64 fields), partial |r|^2 in s->partials
cudaError_t outer_residual(gbds_solver s, const void *b64, const void *x64, void *r64, bool df, cudaStream_t st) {
    const Geom &g = s->g;
    const int nb = blocks(g);
    cudaError_t e;
    if (df && s->gauge_df) {
        e = apply_M_df(s, x64, s->Mp64, +1, st);
        if (e != cudaSuccess) return e;
        xmy_norm_df<<<nb, kThreads, 0, st>>>(static_cast<const double2 *>(b64), static_cast<const float4 *>(s->Mp64),
                                             static_cast<double2 *>(r64), g.Vh, g.stride, s->partials);
    } else {
        e = apply_M<double>(s, s->gauge64, 18, x64, s->t64, s->Mp64, +1, nullptr, st);
        if (e != cudaSuccess) return e;
        xmy_norm<<<nb, kThreads, 0, st>>>(static_cast<const double2 *>(b64), static_cast<const double2 *>(s->Mp64),
                                          static_cast<double2 *>(r64), g.Vh, g.stride, s->partials);
    }
    count_launch();
    return cudaGetLastError();
}

// A low-precision inner solve whose residual has not dropped below 0.9 of its
// best value for 96 iterations has reached the accuracy its storage allows:
// the defect correction takes over from there.
bool stagnated(double rr, int k, double &best, int &best_k) {
    if (rr < 0.81 * best) {
        best = rr;
        best_k = k;
        return false;
    }
    return k - best_k >= 96;
}

cudaError_t read_scalars(gbds_solver s, cudaStream_t st) {
    cudaError_t e = cudaMemcpyAsync(s->hsc, s->sc, sizeof(Scalars), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e;
}

// A counter that is 0 for every stream, without the default stream: a caller may be
// capturing a stream that synchronises with it, or have work on it to wait for.
cudaError_t new_ticket(unsigned **ticket) {
    cudaStream_t st = nullptr;
    cudaError_t e = cudaMalloc(ticket, sizeof(unsigned));
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMemsetAsync(*ticket, 0, sizeof(unsigned), st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (st) cudaStreamDestroy(st);
    return e;
}

// Record body(stream), which makes `launches` counted launches.  Where it cannot
// be recorded, the graph stays empty and the iterations are launched one by one.
template <typename BODY>
void record(IterGraph &g, int launches, const BODY &body) {
    cudaStream_t cs = nullptr;
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        const cudaError_t le = body(cs);
        e = cudaStreamEndCapture(cs, &graph);
        if (le != cudaSuccess) e = le;
        else count_launch(-launches);  // recorded, not launched
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&g.exec, graph, 0);
    if (e != cudaSuccess) {
        g.exec = nullptr;
        (void)cudaGetLastError();
    }
    if (graph) cudaGraphDestroy(graph);
    if (cs) cudaStreamDestroy(cs);
    g.launches = launches;
}

cudaError_t launch(const IterGraph &g, cudaStream_t st) {
    count_launch(g.launches);
    return cudaGraphLaunch(g.exec, st);
}

// The convergence test reads rr back every few iterations.  So that the GPU does
// not idle while the host waits for it, the next iteration's first part (M p and
// alpha, which write neither x nor r nor p) is enqueued behind the copy: unused
// if the solve has converged.  On large lattices the unused part would cost more
// than the wait (24^3x48: 100 us against 15), so there it follows the test.
bool look_ahead(const Geom &g) { return blocks(g) <= 912; }

// CG on A = M^+ M with x = 0, r = p = rhs, sc->rr = |rhs|^2 prepared.  first():
// M p and alpha; second(): r -= alpha A p, beta, x += alpha p, p = r + beta p;
// steps (where recorded): second() and kCheck - 1 whole iterations.  Stops when
// rr <= target_rr, after max_iter iterations, or (inner solves) when it stagnates.
template <typename FIRST, typename SECOND>
cudaError_t cg_loop(gbds_solver s, const FIRST &first, const SECOND &second, const IterGraph *steps, bool inner,
                    double target_rr, int max_iter, int *iters, cudaStream_t st) {
    const int check_every = inner ? kCheck : 1;
    cudaError_t e = cudaSuccess;
    int k = 0;
    double best = 1e300;
    int best_k = 0;
    bool ahead = false;  // first() of iteration k is already enqueued
    while (k < max_iter) {
        if (!ahead) e = first(st);
        ahead = false;
        if (e != cudaSuccess) break;
        if (steps && steps->exec && k % kCheck == 0 && k + kCheck <= max_iter) {
            e = launch(*steps, st);
            k += kCheck;
        } else {
            e = second(st);
            k++;
        }
        if (e != cudaSuccess) break;
        if (k % check_every == 0 || k == max_iter) {
            e = cudaMemcpyAsync(s->hsc, s->sc, sizeof(Scalars), cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaEventRecord(s->read, st);
            if (e == cudaSuccess && k < max_iter && look_ahead(s->g)) {
                e = first(st);
                ahead = true;
            }
            if (e == cudaSuccess) e = cudaEventSynchronize(s->read);
            if (e != cudaSuccess) break;
            if (!(s->hsc->rr > target_rr)) break;  // converged (or NaN: stop)
            if (inner && stagnated(s->hsc->rr, k, best, best_k)) break;
        }
    }
    *iters = k;
    return e;
}

// The fields of one CG.
struct CgFields {
    const void *gauge;
    int recon;
    void *x, *r, *p, *Mp, *t;
};

CgFields inner_fields(gbds_solver s) {
    return {s->gauge32, s->prm.inner_recon, s->e32, s->r32, s->p32, s->Mp32, s->t32};
}

// Whether the inner CG's operator launches finish their sums themselves (small
// lattices), without a launch of their own.
bool sums_here(gbds_solver s) { return s->prm.inner_prec == 32 && f32_sums_here(s->g, s->prm.inner_recon); }

template <typename T>
SumHere sum_here_to(gbds_solver s, int mode) {
    SumHere h;
    if (sizeof(T) == 4 && sums_here(s)) h = {s->ticket, s->sc, mode};
    return h;
}

template <typename T>
cudaError_t cg_first(gbds_solver s, const CgFields &f, cudaStream_t st) {
    const SumHere here = sum_here_to<T>(s, kAlpha);
    cudaError_t e = apply_M<T>(s, f.gauge, f.recon, f.p, f.t, f.Mp, +1, s->partials, st, here);
    if (e != cudaSuccess || here.ticket) return e;
    return finish_on(s, kAlpha, st, sizeof(T) == 4 ? f32_partials(s->g, f.recon) : 0);
}

template <typename T>
cudaError_t cg_second(gbds_solver s, const CgFields &f, cudaStream_t st) {
    const Geom &g = s->g;
    const SumHere here = sum_here_to<T>(s, kBeta);
    cudaError_t e = apply_Mdag_update<T>(s, f.gauge, f.recon, f.Mp, f.t, f.r, st, here);
    if (e == cudaSuccess && !here.ticket)
        e = finish_on(s, kBeta, st, sizeof(T) == 4 ? f32_partials(g, f.recon) : 0);
    if (e != cudaSuccess) return e;
    launch_pdl(cg_xpay<T>, dim3(blocks(g)), kThreads, st, static_cast<const SV<T> *>(f.r), static_cast<SV<T> *>(f.x),
               static_cast<SV<T> *>(f.p), (const Scalars *)s->sc, g.Vh, g.stride);
    count_launch();
    return cudaGetLastError();
}

template <typename T>
cudaError_t cg(gbds_solver s, const CgFields &f, double target_rr, int max_iter, int *iters, cudaStream_t st) {
    constexpr bool inner = sizeof(T) == 4;
    return cg_loop(
        s, [&](cudaStream_t t) { return cg_first<T>(s, f, t); }, [&](cudaStream_t t) { return cg_second<T>(s, f, t); },
        inner ? &s->steps : nullptr, inner, target_rr, max_iter, iters, st);
}

// second() and kCheck - 1 whole iterations, recorded
template <typename FIRST, typename SECOND>
void record_steps(gbds_solver s, const FIRST &first, const SECOND &second) {
    const int n1 = sums_here(s) ? 2 : 3, n2 = sums_here(s) ? 3 : 4;  // launches of first(), second()
    record(s->steps, kCheck * n2 + (kCheck - 1) * n1, [&](cudaStream_t cs) {
        cudaError_t e = second(cs);
        for (int i = 1; i < kCheck && e == cudaSuccess; i++) {
            e = first(cs);
            if (e == cudaSuccess) e = second(cs);
        }
        return e;
    });
}

// The 16-bit operator: out = in - kappa^2 D_eo D_oe in, FP16 links.
cudaError_t apply_M_h(gbds_solver s, const void *in, void *tmp, void *out, int isign, double *partials, cudaStream_t st) {
    const Geom &g = s->g;
    const float k2 = (float)(s->prm.kappa * s->prm.kappa);
    cudaError_t e = launch_gen_h16(s->fmt16, g, s->prm.inner_recon, s->gauge16, in, tmp, isign, 0, nullptr, 0.f, nullptr, st);
    if (e != cudaSuccess) return e;
    return launch_gen_h16(s->fmt16, g, s->prm.inner_recon, s->gauge16, tmp, out, isign, 1, in, -k2, partials, st);
}

cudaError_t apply_Mdag_update_h(gbds_solver s, const void *in, void *tmp, void *r, cudaStream_t st) {
    const Geom &g = s->g;
    const float k2 = (float)(s->prm.kappa * s->prm.kappa);
    cudaError_t e = launch_gen_h16(s->fmt16, g, s->prm.inner_recon, s->gauge16, in, tmp, -1, 0, nullptr, 0.f, nullptr, st);
    if (e != cudaSuccess) return e;
    return launch_gen_h16(s->fmt16, g, s->prm.inner_recon, s->gauge16, tmp, nullptr, -1, 1, in, -k2, s->partials, st, r,
                          &s->sc->alpha);
}

template <int FMT>
cudaError_t cg_first_h(gbds_solver s, cudaStream_t st) {
    cudaError_t e = apply_M_h(s, s->p16, s->t16, s->Mp16, +1, s->partials, st);
    return e == cudaSuccess ? finish_on(s, kAlpha, st) : e;
}

template <int FMT>
cudaError_t cg_second_h(gbds_solver s, cudaStream_t st) {
    const Geom &g = s->g;
    cudaError_t e = apply_Mdag_update_h(s, s->Mp16, s->t16, s->r32, st);
    if (e == cudaSuccess) e = finish_on(s, kBeta, st);
    if (e != cudaSuccess) return e;
    launch_pdl(cg_xpay_h<FMT>, dim3(blocks(g)), kThreads, st, static_cast<const float4 *>(s->r32),
               static_cast<float4 *>(s->e32), static_cast<char *>(s->p16), (const Scalars *)s->sc, g.Vh, g.stride);
    count_launch();
    return cudaGetLastError();
}

template <int FMT>
cudaError_t cg_h(gbds_solver s, double target_rr, int max_iter, int *iters, cudaStream_t st) {
    return cg_loop(
        s, [&](cudaStream_t t) { return cg_first_h<FMT>(s, t); }, [&](cudaStream_t t) { return cg_second_h<FMT>(s, t); },
        &s->steps, true, target_rr, max_iter, iters, st);
}

// Record the inner CG's steps (inner_prec 32, 16 or 17).
void record_inner(gbds_solver s) {
    if (s->prm.inner_prec == 32) {
        const CgFields f = inner_fields(s);
        return record_steps(
            s, [&](cudaStream_t t) { return cg_first<float>(s, f, t); },
            [&](cudaStream_t t) { return cg_second<float>(s, f, t); });
    }
    if (s->fmt16 == kFmtF16N)
        return record_steps(
            s, [&](cudaStream_t t) { return cg_first_h<kFmtF16N>(s, t); },
            [&](cudaStream_t t) { return cg_second_h<kFmtF16N>(s, t); });
    return record_steps(
        s, [&](cudaStream_t t) { return cg_first_h<kFmtBF16>(s, t); },
        [&](cudaStream_t t) { return cg_second_h<kFmtBF16>(s, t); });
}

template <typename T>
cudaError_t norm_into(gbds_solver s, const void *v, void *dst, void *dst2, int mode, cudaStream_t st,
                      Scalars *to = nullptr) {
    norm_copy<T><<<blocks(s->g), kThreads, 0, st>>>(static_cast<const SV<T> *>(v), static_cast<SV<T> *>(dst),
                                                     static_cast<SV<T> *>(dst2), s->g.Vh, s->g.stride, s->partials);
    count_launch();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? finish_on(s, mode, st, 0, to) : e;
}

template <typename T>
cudaError_t zero(gbds_solver s, void *v, cudaStream_t st) {
    zero_field<T><<<blocks(s->g), kThreads, 0, st>>>(static_cast<SV<T> *>(v), s->g.Vh, s->g.stride);
    count_launch();
    return cudaGetLastError();
}

void release(gbds_solver s) {
    void *bufs[] = {s->gauge64, s->gauge32, s->gauge_df, s->xdf, s->b64, s->c64, s->x64, s->r64, s->p64, s->Ap64,
                    s->Mp64, s->t64,
                    s->e32, s->r32, s->p32, s->Mp32, s->t32, s->p16, s->Mp16, s->t16, s->gauge16,
                    s->partials, s->sc, s->ticket};
    for (void *b : bufs)
        if (b) cudaFree(b);
    if (s->hsc) cudaFreeHost(s->hsc);
    if (s->read) cudaEventDestroy(s->read);
    if (s->steps.exec) cudaGraphExecDestroy(s->steps.exec);
}

}  // namespace

// single: solves on its own (else the batched solver's FP64 side)
static int create_solver(gbds_solver *out, const int dims[4], const gbds_solver_params *p, bool single) {
    if (!out || !p) return set_error(GBDS_ERROR_INVALID_VALUE, "NULL argument");
    *out = nullptr;
    if (p->inner_prec != 64 && p->inner_prec != 32 && p->inner_prec != 16 && p->inner_prec != 17)
        return set_error(GBDS_ERROR_INVALID_VALUE, "inner_prec must be 64, 32, 16 or 17");
    if (p->inner_recon != 18 && p->inner_recon != 12) return set_error(GBDS_ERROR_INVALID_VALUE, "inner_recon must be 18 or 12");
    if (!(p->tol > 0) || p->max_iter <= 0 || !(p->kappa > 0))
        return set_error(GBDS_ERROR_INVALID_VALUE, "tol, max_iter and kappa must be positive");
    Geom g;
    int rc = make_geom(dims, 4, &g);
    if (rc != GBDS_SUCCESS) return rc;
    gbds_solver s = new (std::nothrow) gbds_solver_s;
    if (!s) return set_error(GBDS_ERROR_OUT_OF_MEMORY, "host allocation failed");
    s->g = g;
    s->prm = *p;
    if (!(s->prm.inner_tol > 0 && s->prm.inner_tol < 1)) s->prm.inner_tol = 1e-5;
    const size_t f64 = spinor_bytes(g, 64), f32 = spinor_bytes(g, 32);
    cudaError_t e = cudaSuccess;
    void **d64[] = {&s->b64, &s->c64, &s->x64, &s->r64, &s->p64, &s->Ap64, &s->Mp64, &s->t64};
    for (void **b : d64)
        if (e == cudaSuccess) e = cudaMalloc(b, f64);
    if (p->inner_prec == 32) {
        void **d32[] = {&s->e32, &s->r32, &s->p32, &s->Mp32, &s->t32};
        for (void **b : d32)
            if (e == cudaSuccess) e = cudaMalloc(b, f32);
        if (e == cudaSuccess) e = cudaMalloc(&s->gauge32, gauge_bytes(g, 32, p->inner_recon));
    } else if (p->inner_prec == 16 || p->inner_prec == 17) {
        s->fmt16 = p->inner_prec == 16 ? kFmtF16N : kFmtBF16;
        const size_t f16 = (size_t)gen_spinor_bytes(s->fmt16) * g.stride;
        void **d32[] = {&s->e32, &s->r32, &s->Mp32, &s->t32};
        for (void **b : d32)
            if (e == cudaSuccess) e = cudaMalloc(b, f32);
        void **d16[] = {&s->p16, &s->Mp16, &s->t16};
        for (void **b : d16)
            if (e == cudaSuccess) e = cudaMalloc(b, f16);
        if (e == cudaSuccess) e = cudaMalloc(&s->gauge32, gauge_bytes(g, 32, p->inner_recon));
        if (e == cudaSuccess) e = cudaMalloc(&s->gauge16, gauge_bytes(g, 32, p->inner_recon) / 2);
    }
    if (e == cudaSuccess) e = cudaMalloc(&s->gauge64, gauge_bytes(g, 64, 18));
    const bool df = p->inner_prec != 64 && p->outer_double_float;
    if (e == cudaSuccess && df) e = cudaMalloc(&s->gauge_df, gauge_bytes(g, 64, 18));
    if (e == cudaSuccess && df) e = cudaMalloc(&s->xdf, f64);
    const int parts = std::max(blocks(g), f32_partials(g, p->inner_recon));
    if (e == cudaSuccess) e = cudaMalloc(&s->partials, sizeof(double) * (size_t)parts);
    if (e == cudaSuccess) e = cudaMalloc(&s->sc, sizeof(Scalars));
    if (e == cudaSuccess) e = new_ticket(&s->ticket);
    if (e == cudaSuccess) e = cudaMallocHost(&s->hsc, sizeof(Scalars));
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s->read, cudaEventDisableTiming);
    if (e == cudaSuccess && p->inner_prec != 64 && single) record_inner(s);
    if (e != cudaSuccess) {
        release(s);
        delete s;
        return cuda_error(e, "gbds_solver_create");
    }
    *out = s;
    return GBDS_SUCCESS;
}

extern "C" int gbds_solver_create(gbds_solver *out, const int dims[4], const gbds_solver_params *p) {
    return create_solver(out, dims, p, true);
}

extern "C" int gbds_solver_destroy(gbds_solver s) {
    if (!s) return GBDS_SUCCESS;
    cudaDeviceSynchronize();
    release(s);
    delete s;
    return GBDS_SUCCESS;
}

extern "C" int gbds_solver_set_gauge(gbds_solver s, const double *u_packed, void *stream) {
    if (!s) return set_error(GBDS_ERROR_NOT_INITIALIZED, "solver is NULL");
    if (!u_packed || (reinterpret_cast<uintptr_t>(u_packed) & 15u))
        return set_error(GBDS_ERROR_INVALID_VALUE, "u_packed must be a 16-byte aligned device pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = launch_pack_gauge(s->g, 64, 18, u_packed, nullptr, s->gauge64, st);
    if (e == cudaSuccess && s->gauge_df) e = launch_f64_to_df(s->gauge64, s->gauge_df, gauge_bytes(s->g, 64, 18) / 16, st);
    if (e == cudaSuccess && s->prm.inner_prec != 64) {
        const size_t n = (size_t)s->g.V * 72;
        float *tmp = nullptr;
        e = cudaMallocAsync(reinterpret_cast<void **>(&tmp), n * sizeof(float), st);
        if (e == cudaSuccess) {
            f64_to_f32<<<1024, 256, 0, st>>>(u_packed, tmp, n);
            count_launch();
            e = cudaGetLastError();
            if (e == cudaSuccess) e = launch_pack_gauge(s->g, 32, s->prm.inner_recon, tmp, nullptr, s->gauge32, st);
            if (e == cudaSuccess && s->gauge16)
                e = convert_links_f16(s->gauge32, s->gauge16, gauge_bytes(s->g, 32, s->prm.inner_recon) / 4, st);
            cudaFreeAsync(tmp, st);
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_error(e, "gbds_solver_set_gauge");
    s->have_gauge = true;
    return GBDS_SUCCESS;
}

extern "C" int gbds_solver_apply(gbds_solver s, const double *x_packed, double *y_packed, int dagger, void *stream) {
    if (!s) return set_error(GBDS_ERROR_NOT_INITIALIZED, "solver is NULL");
    if (!s->have_gauge) return set_error(GBDS_ERROR_NOT_INITIALIZED, "gbds_solver_set_gauge has not been called");
    if (!x_packed || !y_packed) return set_error(GBDS_ERROR_INVALID_VALUE, "NULL field pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = launch_pack_spinor(s->g, 64, x_packed, nullptr, 0, 0, s->b64, st);
    if (e == cudaSuccess) e = apply_M<double>(s, s->gauge64, 18, s->b64, s->t64, s->Mp64, dagger ? -1 : 1, nullptr, st);
    if (e == cudaSuccess) e = launch_unpack_spinor(s->g, 64, s->Mp64, nullptr, 0, 0, y_packed, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? GBDS_SUCCESS : cuda_error(e, "gbds_solver_apply");
}

static int solve_impl(gbds_solver s, const double *b_packed, double *x_packed, gbds_solver_stats *stats, void *stream,
                      bool normal);

extern "C" int gbds_solver_solve(gbds_solver s, const double *b_packed, double *x_packed, gbds_solver_stats *stats,
                                 void *stream) {
    return solve_impl(s, b_packed, x_packed, stats, stream, false);
}

extern "C" int gbds_solver_solve_normal(gbds_solver s, const double *c_packed, double *x_packed, gbds_solver_stats *stats,
                                        void *stream) {
    return solve_impl(s, c_packed, x_packed, stats, stream, true);
}

// Mixed-precision solve of M x = b by defect correction on the true
// residual: each cycle forms r = b - M x in FP64 (two FP64 Dslash
// applications, or the double-float operator with outer_double_float), then
// c = M^+ r in FP32 (the normal-equation right-hand side
// for the inner CG and, through |c|, the stopping test |M^+ (b - M x)| <=
// tol |M^+ b|: the cancellation is in the FP64 subtraction, so |c| carries
// FP32 relative accuracy of its own size), then the inner CG on M^+ M and
// x += |c| e in FP64.
static int solve_mixed(gbds_solver s, const double *b_packed, double *x_packed, gbds_solver_stats *stats,
                       cudaStream_t st, std::chrono::steady_clock::time_point t0) {
    const Geom &g = s->g;
    const int nb = blocks(g);
    const double tol2 = s->prm.tol * s->prm.tol;
    const bool half = s->prm.inner_prec != 32;
    gbds_solver_stats out = {};
    cudaError_t e = launch_pack_spinor(g, 64, b_packed, nullptr, 0, 0, s->b64, st);
    if (e == cudaSuccess) e = norm_into<double>(s, s->b64, s->r64, nullptr, kOuterRR, st);  // r = b
    if (e == cudaSuccess) e = zero<double>(s, s->x64, st);
    if (e == cudaSuccess) e = read_scalars(s, st);
    if (e != cudaSuccess) return cuda_error(e, "gbds_solver_solve");
    const double b2 = s->hsc->outer_rr;
    double r2 = b2;   // |b - M x|^2, FP64
    double c2 = 0;    // |M^+ b|^2
    double n2 = 0;    // |M^+ (b - M x)|^2
    int total = 0;
    bool stop = false;
    while (b2 > 0) {
        // c = M^+ (r / |r|) in FP32 and |c|^2
        demote_scaled<<<nb, kThreads, 0, st>>>(static_cast<const double2 *>(s->r64), 1.0 / std::sqrt(r2),
                                               static_cast<float4 *>(s->r32), g.Vh, g.stride);
        count_launch();
        e = cudaGetLastError();
        if (e == cudaSuccess)
            e = apply_M<float>(s, s->gauge32, s->prm.inner_recon, s->r32, s->t32, s->Mp32, -1, s->partials, st);
        if (e == cudaSuccess) e = finish_on(s, kNorm, st, f32_partials(g, s->prm.inner_recon));
        if (e == cudaSuccess) e = read_scalars(s, st);
        if (e != cudaSuccess) break;
        const double s2 = s->hsc->norm;
        n2 = r2 * s2;
        if (out.cycles == 0) c2 = n2;
        if (stop || !(n2 > tol2 * c2) || total >= s->prm.max_iter || !(s2 > 0)) break;
        // inner CG on A e = c / |c|, from e = 0
        const float inv = (float)(1.0 / std::sqrt(s2));
        if (!half)
            scale_copy<<<nb, kThreads, 0, st>>>(static_cast<const float4 *>(s->Mp32), inv, static_cast<float4 *>(s->r32),
                                                static_cast<float4 *>(s->p32), g.Vh, g.stride);
        else if (s->fmt16 == kFmtF16N)
            scale_copy_h<kFmtF16N><<<nb, kThreads, 0, st>>>(static_cast<const float4 *>(s->Mp32), inv,
                                                            static_cast<float4 *>(s->r32), static_cast<char *>(s->p16),
                                                            g.Vh, g.stride);
        else
            scale_copy_h<kFmtBF16><<<nb, kThreads, 0, st>>>(static_cast<const float4 *>(s->Mp32), inv,
                                                            static_cast<float4 *>(s->r32), static_cast<char *>(s->p16),
                                                            g.Vh, g.stride);
        count_launch();
        e = cudaGetLastError();
        if (e == cudaSuccess) e = zero<float>(s, s->e32, st);
        if (e == cudaSuccess) e = norm_into<float>(s, s->r32, nullptr, nullptr, kSetRR, st);
        if (e != cudaSuccess) break;
        double delta = s->prm.inner_tol;
        const double need = 0.5 * s->prm.tol * std::sqrt(c2 / n2);
        if (need > delta) delta = need;
        int it = 0;
        if (!half)
            e = cg<float>(s, inner_fields(s), delta * delta, s->prm.max_iter - total, &it, st);
        else if (s->fmt16 == kFmtF16N)
            e = cg_h<kFmtF16N>(s, delta * delta, s->prm.max_iter - total, &it, st);
        else
            e = cg_h<kFmtBF16>(s, delta * delta, s->prm.max_iter - total, &it, st);
        total += it;
        out.cycles++;
        if (e != cudaSuccess) break;
        // x += |c| e (the correction A^-1 M^+ r);  r = b - M x on FP64 fields
        // (the FP64 operator, or the double-float one with outer_double_float)
        promote_scaled<<<nb, kThreads, 0, st>>>(static_cast<const float4 *>(s->e32), std::sqrt(n2),
                                                static_cast<double2 *>(s->x64), g.Vh, g.stride);
        count_launch();
        e = cudaGetLastError();
        if (e == cudaSuccess) e = outer_residual(s, s->b64, s->x64, s->r64, df_range(b2), st);
        if (e == cudaSuccess) e = finish_on(s, kOuterRR, st);
        if (e == cudaSuccess) e = read_scalars(s, st);
        if (e != cudaSuccess) break;
        const double prev = r2;
        r2 = s->hsc->outer_rr;
        if (!(r2 < prev) || !(r2 > 0)) stop = true;  // no progress (or NaN, or exact): measure once more, then stop
    }
    if (e == cudaSuccess) e = launch_unpack_spinor(g, 64, s->x64, nullptr, 0, 0, x_packed, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_error(e, "gbds_solver_solve");
    out.iterations = total;
    out.residual = c2 > 0 ? std::sqrt(n2 / c2) : 0.0;
    out.true_residual = b2 > 0 ? std::sqrt(r2 / b2) : 0.0;
    out.converged = out.residual <= s->prm.tol ? 1 : 0;
    out.seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (stats) *stats = out;
    return GBDS_SUCCESS;
}

static int solve_impl(gbds_solver s, const double *b_packed, double *x_packed, gbds_solver_stats *stats, void *stream,
                      bool normal) {
    if (!s) return set_error(GBDS_ERROR_NOT_INITIALIZED, "solver is NULL");
    if (!s->have_gauge) return set_error(GBDS_ERROR_NOT_INITIALIZED, "gbds_solver_set_gauge has not been called");
    if (!b_packed || !x_packed) return set_error(GBDS_ERROR_INVALID_VALUE, "NULL field pointer");
    if ((reinterpret_cast<uintptr_t>(b_packed) | reinterpret_cast<uintptr_t>(x_packed)) & 15u)
        return set_error(GBDS_ERROR_INVALID_VALUE, "fields must be 16-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const auto t0 = std::chrono::steady_clock::now();
    if (!normal && s->prm.inner_prec != 64) return solve_mixed(s, b_packed, x_packed, stats, st, t0);
    gbds_solver_stats out = {};
    const Geom &g = s->g;
    const double tol2 = s->prm.tol * s->prm.tol;
    // b, c = M^+ b, |c|^2
    cudaError_t e = launch_pack_spinor(g, 64, b_packed, nullptr, 0, 0, normal ? s->c64 : s->b64, st);
    if (e == cudaSuccess) {
        if (normal) e = norm_into<double>(s, s->c64, nullptr, nullptr, kOuterRR, st);
        else e = apply_M<double>(s, s->gauge64, 18, s->b64, s->t64, s->c64, -1, s->partials, st);
    }
    if (e == cudaSuccess && !normal) e = finish_on(s, kOuterRR, st);
    if (e == cudaSuccess) e = zero<double>(s, s->x64, st);
    if (e == cudaSuccess) e = read_scalars(s, st);
    if (e != cudaSuccess) return cuda_error(e, "gbds_solver_solve");
    const double c2 = s->hsc->outer_rr;
    double outer_rr = c2;
    int total = 0;
    bool have_residual = false;  // r64 = c - A x and Mp64 = M x are current
    if (c2 > 0) {
        if (s->prm.inner_prec == 64) {
            // all-FP64 CG: r = p = c
            e = norm_into<double>(s, s->c64, s->r64, s->p64, kSetRR, st);
            int it = 0;
            if (e == cudaSuccess)
                e = cg<double>(s, {s->gauge64, 18, s->x64, s->r64, s->p64, s->Mp64, s->t64}, tol2 * c2, s->prm.max_iter, &it, st);
            total = it;
            out.cycles = 1;
        } else {
            // FP64 defect correction around FP32 CG; r64 starts as c.
            e = norm_into<double>(s, s->c64, s->r64, nullptr, kOuterRR, st);
            const bool half = s->prm.inner_prec != 32;
            while (e == cudaSuccess && outer_rr > tol2 * c2 && total < s->prm.max_iter) {
                const int nb = blocks(g);
                if (!half) {
                    demote_residual<<<nb, kThreads, 0, st>>>(static_cast<const double2 *>(s->r64),
                                                             static_cast<float4 *>(s->r32), static_cast<float4 *>(s->p32),
                                                             s->sc, g.Vh, g.stride);
                } else if (s->fmt16 == kFmtF16N) {
                    demote_residual_h<kFmtF16N><<<nb, kThreads, 0, st>>>(static_cast<const double2 *>(s->r64),
                                                                         static_cast<float4 *>(s->r32),
                                                                         static_cast<char *>(s->p16), s->sc, g.Vh, g.stride);
                } else {
                    demote_residual_h<kFmtBF16><<<nb, kThreads, 0, st>>>(static_cast<const double2 *>(s->r64),
                                                                         static_cast<float4 *>(s->r32),
                                                                         static_cast<char *>(s->p16), s->sc, g.Vh, g.stride);
                }
                count_launch();
                e = cudaGetLastError();
                if (e == cudaSuccess) e = zero<float>(s, s->e32, st);
                if (e == cudaSuccess) e = norm_into<float>(s, s->r32, nullptr, nullptr, kSetRR, st);
                if (e != cudaSuccess) break;
                // inner target: the requested reduction, but no further than the outer goal needs
                double delta = s->prm.inner_tol;
                const double need = 0.5 * s->prm.tol * std::sqrt(c2 / outer_rr);
                if (need > delta) delta = need;
                int it = 0;
                if (!half)
                    e = cg<float>(s, inner_fields(s), delta * delta, s->prm.max_iter - total, &it, st);
                else if (s->fmt16 == kFmtF16N)
                    e = cg_h<kFmtF16N>(s, delta * delta, s->prm.max_iter - total, &it, st);
                else
                    e = cg_h<kFmtBF16>(s, delta * delta, s->prm.max_iter - total, &it, st);
                total += it;
                out.cycles++;
                if (e != cudaSuccess) break;
                promote_update<<<nb, kThreads, 0, st>>>(static_cast<const float4 *>(s->e32), static_cast<double2 *>(s->x64),
                                                        s->sc, g.Vh, g.stride);
                count_launch();
                e = cudaGetLastError();
                // true residual r = c - A x in FP64
                if (e == cudaSuccess) e = apply_M<double>(s, s->gauge64, 18, s->x64, s->t64, s->Mp64, +1, nullptr, st);
                if (e == cudaSuccess) e = apply_M<double>(s, s->gauge64, 18, s->Mp64, s->t64, s->Ap64, -1, nullptr, st);
                if (e == cudaSuccess) {
                    xmy_norm<<<nb, kThreads, 0, st>>>(static_cast<const double2 *>(s->c64), static_cast<const double2 *>(s->Ap64),
                                                      static_cast<double2 *>(s->r64), g.Vh, g.stride, s->partials);
                    count_launch();
                    e = cudaGetLastError();
                }
                if (e == cudaSuccess) e = finish_on(s, kOuterRR, st);
                if (e == cudaSuccess) e = read_scalars(s, st);
                if (e != cudaSuccess) break;
                have_residual = true;
                const double prev = outer_rr;
                outer_rr = s->hsc->outer_rr;
                if (!(outer_rr < prev)) break;  // no progress (or NaN): stop
            }
        }
    }
    if (e != cudaSuccess) return cuda_error(e, "gbds_solver_solve");
    // FP64 checks: |c - A x| / |c| and |b - M x| / |b|.  The defect-correction
    // loop leaves both r = c - A x (norm in outer_rr) and M x (in Mp64) from
    // its last cycle; the FP64 CG's recursive residual is not the true one, so
    // there they are computed here.
    const int nb = blocks(g);
    double final_rr = outer_rr;
    if (!have_residual) {
        e = apply_M<double>(s, s->gauge64, 18, s->x64, s->t64, s->Mp64, +1, nullptr, st);
        if (e == cudaSuccess) e = apply_M<double>(s, s->gauge64, 18, s->Mp64, s->t64, s->Ap64, -1, nullptr, st);
        if (e == cudaSuccess) {
            xmy_norm<<<nb, kThreads, 0, st>>>(static_cast<const double2 *>(s->c64), static_cast<const double2 *>(s->Ap64),
                                              static_cast<double2 *>(s->r64), g.Vh, g.stride, s->partials);
            count_launch();
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = finish_on(s, kOuterRR, st);
        if (e == cudaSuccess) e = read_scalars(s, st);
        final_rr = s->hsc->outer_rr;
    }
    if (!normal) {
        if (e == cudaSuccess) {
            xmy_norm<<<nb, kThreads, 0, st>>>(static_cast<const double2 *>(s->b64), static_cast<const double2 *>(s->Mp64),
                                              static_cast<double2 *>(s->p64), g.Vh, g.stride, s->partials);
            count_launch();
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = finish_on(s, kNorm, st);
        if (e == cudaSuccess) e = norm_into<double>(s, s->b64, nullptr, nullptr, kOuterRR, st);
        if (e == cudaSuccess) e = read_scalars(s, st);
    } else {
        s->hsc->norm = final_rr;
        s->hsc->outer_rr = c2;
    }
    if (e == cudaSuccess) e = launch_unpack_spinor(g, 64, s->x64, nullptr, 0, 0, x_packed, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_error(e, "gbds_solver_solve");
    out.iterations = total;
    out.residual = c2 > 0 ? std::sqrt(final_rr / c2) : 0.0;
    out.true_residual = s->hsc->outer_rr > 0 ? std::sqrt(s->hsc->norm / s->hsc->outer_rr) : 0.0;
    out.converged = out.residual <= s->prm.tol ? 1 : 0;
    out.seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (stats) *stats = out;
    return GBDS_SUCCESS;
}

// ---------------------------------------------------------------------------
// Batched solve: nrhs independent systems M x_k = b_k on one gauge field.
// The inner FP32 CGs of all right-hand sides advance in lockstep on the
// multi-RHS operator (rhs fastest in memory: every link load serves all of
// them), each with its own scalars and its own stopping point; a converged
// right-hand side is masked out of the vector updates.  The FP64 defect
// correction (residual, solution update, norms) is done per right-hand side
// with the FP64 operator.
// ---------------------------------------------------------------------------

namespace gbds {
namespace {

using BScalars = RhsCgScalars;  // rr, pAp, alpha, beta, active (dslash_gen.cuh)

enum BFinish { kBAlpha = 0, kBBeta = 1, kBSetRR = 2 };

// r -= alpha_r Ap;  per-rhs partial |r|^2  (active rhs only; the matching
// x += alpha_r p happens in bcg_xpay, which reads p anyway)
template <int NRHS>
__global__ void __launch_bounds__(128) bcg_update(float4 *r, const float4 *__restrict__ Ap, const BScalars *sc, long long n,
                                                 size_t cs, double *partials) {
    pdl_allow_next();
    pdl_wait_prev();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int q = (int)(t % NRHS);
    float nrm = 0.f;
    if (t < n && sc[q].active) {
        const float a = (float)sc[q].alpha;
#pragma unroll
        for (int k = 0; k < 6; k++) {
            const size_t i = (size_t)k * cs + (size_t)t;
            const float4 rn = axpy_v(-a, Ap[i], r[i]);
            r[i] = rn;
            nrm += norm_v(rn);
        }
    }
    block_sum_rhs<NRHS>(partials, nrm);
}

// x += alpha_r p;  p = r + beta_r p  (active rhs only)
template <int NRHS>
__global__ void __launch_bounds__(128) bcg_xpay(float4 *x, const float4 *__restrict__ r, float4 *p, const BScalars *sc,
                                               long long n, size_t cs, int reverse) {
    pdl_allow_next();
    pdl_wait_prev();
    const unsigned block = reverse ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
    const long long t = (long long)block * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int q = (int)(t % NRHS);
    if (!sc[q].active) return;
    const float a = (float)sc[q].alpha, b = (float)sc[q].beta;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const size_t i = (size_t)k * cs + (size_t)t;
        const float4 pv = p[i];
        x[i] = axpy_v(a, pv, x[i]);
        p[i] = axpy_v(b, pv, r[i]);
    }
}

// per-rhs partial |v|^2
template <int NRHS>
__global__ void __launch_bounds__(128) bnorm(const float4 *__restrict__ v, long long n, size_t cs, double *partials) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float nrm = 0.f;
    if (t < n) {
#pragma unroll
        for (int k = 0; k < 6; k++) nrm += norm_v(v[(size_t)k * cs + (size_t)t]);
    }
    block_sum_rhs<NRHS>(partials, nrm);
}

// Per-rhs sums of the (block, rhs) partials, in a fixed order: block j of the
// grid sums rows [j * kBRows, (j + 1) * kBRows) of every rhs (thread t takes
// rhs t % nrhs: coalesced reads), and the last block to finish sums the
// blocks' and takes the scalar step.  Latency-bound: with 16 rhs on 16^3x32
// (8192 rows, 1 MB) blocks of 1024 rows and a second launch that added them
// serially took 14.4 + 4.0 us; this takes 6 us less, and the solve there 38.0
// instead of 39.1 ms.  (Finishing the sums inside the producing kernels gains
// nothing: the fence before the ticket waits for the block's result stores.)
constexpr int kBRows = 64;
__global__ void __launch_bounds__(256) bfinish(const double *partials, int nrows, int nrhs, double *partials2,
                                               unsigned *ticket, BScalars *sc, int mode) {
    pdl_allow_next();
    pdl_wait_prev();
    __shared__ double buf[256];
    __shared__ bool last;
    const int q = threadIdx.x % nrhs, lanes = 256 / nrhs;  // nrhs divides 256
    // the sum over rows [row0, row1) of p, for rhs threadIdx.x < nrhs
    auto sum_rows = [&](const double *p, int row0, int row1) {
        double t = 0;
        for (int i = row0 + threadIdx.x / nrhs; i < row1; i += lanes) t += __ldcg(p + (size_t)i * nrhs + q);
        buf[threadIdx.x] = t;
        __syncthreads();
        for (int k = 128; k >= nrhs; k >>= 1) {  // nrhs is a power of two
            if (threadIdx.x < k) buf[threadIdx.x] += buf[threadIdx.x + k];
            __syncthreads();
        }
        return buf[q];
    };
    const int row0 = blockIdx.x * kBRows;
    const double part = sum_rows(partials, row0, min(row0 + kBRows, nrows));
    if (threadIdx.x < nrhs) {
        partials2[(size_t)blockIdx.x * nrhs + threadIdx.x] = part;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;  // back to 0 for the next launch
    __syncthreads();
    if (!last) return;
    __threadfence();
    const double sum = sum_rows(partials2, 0, gridDim.x);
    if (threadIdx.x >= nrhs) return;
    BScalars &c = sc[threadIdx.x];
    switch (mode) {
    case kBAlpha:
        if (c.active) {
            c.pAp = sum;
            c.alpha = sum > 0 ? c.rr / sum : 0.0;
        }
        break;
    case kBBeta:
        if (c.active) {
            c.beta = c.rr > 0 ? sum / c.rr : 0.0;
            c.rr = sum;
        }
        break;
    default: c.rr = sum; break;
    }
}

// r = p = scale_q * v (scale in sc[q].beta; zero for inactive rhs)
template <int NRHS>
__global__ void __launch_bounds__(128) bscale_copy(const float4 *__restrict__ v, const BScalars *sc, float4 *r, float4 *p,
                                                  long long n, size_t cs) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int q = (int)(t % NRHS);
    const float a = sc[q].active ? (float)sc[q].beta : 0.f;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const size_t i = (size_t)k * cs + (size_t)t;
        const float4 x = v[i];
        const float4 y = make_float4(a * x.x, a * x.y, a * x.z, a * x.w);
        r[i] = y;
        p[i] = y;
    }
}

// The per-rhs FP64 fields of all rhs and a scale for each, in the kernel
// parameters (512 bytes).
struct RhsFields {
    double2 *v[32];
    double s[32];
};

// All columns of the multi-RHS inner fields in one launch.  A CTA of 256
// threads takes 32 sites: lane = site (coalesced reads of the per-rhs FP64
// fields), warp w the rhs w, w + 8, ...
constexpr int kBXSites = 32;

// r = p = s_q r64_q (s_q = 1 / |r64_q|), or 0 where s_q = 0; each component
// passes through a [site][rhs] tile in shared memory, so that the
// interleaved (site, rhs) stores are contiguous too
__global__ void __launch_bounds__(256) bdemote_all(const RhsFields f, float4 *r, float4 *p, int Vh, int stride,
                                                  int nrhs, size_t cs) {
    __shared__ float4 tile[kBXSites][33];  // padded: lanes of one rhs hit different banks
    const int base = blockIdx.x * kBXSites;
    const int h = base + (threadIdx.x & 31);
    const int n = min(kBXSites, Vh - base) * nrhs;  // (site, rhs) entries of this CTA
#pragma unroll 1
    for (int k = 0; k < 6; k++) {
        // the inner fields are FP32 spin pairs: float4 k holds complex
        // elements e0 and e0 + 3 (spins 0/1 or 2/3 of colour k % 3) as (e0.r,
        // e1.r, e0.i, e1.i)
        const int e0 = (k < 3 ? 0 : 6) + k % 3;
        if (h < Vh) {
            for (int q = threadIdx.x >> 5; q < nrhs; q += 8) {
                const double inv = f.s[q];
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (inv != 0.0) {
                    const double2 *r64 = f.v[q];
                    const double2 a = r64[(size_t)e0 * stride + h], b = r64[(size_t)(e0 + 3) * stride + h];
                    v = make_float4((float)(a.x * inv), (float)(b.x * inv), (float)(a.y * inv), (float)(b.y * inv));
                }
                tile[threadIdx.x & 31][q] = v;
            }
        }
        __syncthreads();
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            const float4 v = tile[j / nrhs][j % nrhs];
            const size_t i = (size_t)k * cs + (size_t)base * nrhs + j;
            r[i] = v;
            p[i] = v;
        }
        __syncthreads();
    }
}

// x64_q += s_q * column q of e for the rhs with s_q != 0
__global__ void __launch_bounds__(256) bpromote_all(const float4 *__restrict__ e, const RhsFields f, int Vh, int stride,
                                                   int nrhs, size_t cs) {
    const int h = blockIdx.x * kBXSites + (threadIdx.x & 31);
    if (h >= Vh) return;
    for (int q = threadIdx.x >> 5; q < nrhs; q += 8) {
        const double s = f.s[q];
        if (s == 0.0) continue;
        double2 *x64 = f.v[q];
#pragma unroll
        for (int k = 0; k < 6; k++) {
            const int e0 = (k < 3 ? 0 : 6) + k % 3;  // the pair layout, as in bdemote_all
            const float4 v = e[(size_t)k * cs + (size_t)h * nrhs + q];
            double2 &a = x64[(size_t)e0 * stride + h];
            double2 &b = x64[(size_t)(e0 + 3) * stride + h];
            a.x = fma(s, (double)v.x, a.x);
            a.y = fma(s, (double)v.z, a.y);
            b.x = fma(s, (double)v.y, b.x);
            b.y = fma(s, (double)v.w, b.y);
        }
    }
}

}  // namespace
}  // namespace gbds

struct gbds_bsolver_s {
    gbds_solver s1 = nullptr;  // FP64 gauge, FP64 operator temporaries, FP32 links, reductions
    Geom gm{};                 // s1's geometry with the multi-RHS kernels' site order
    int nrhs = 0;
    std::vector<void *> b64, x64, r64;  // per rhs, FP64, checkerboard 0
    void *e = nullptr, *r = nullptr, *p = nullptr, *Ap = nullptr, *Mp = nullptr, *t = nullptr;  // multi-RHS FP32
    double *bpartials = nullptr, *bpartials2 = nullptr;
    unsigned *ticket = nullptr;  // 0 between launches of bfinish
    IterGraph steps;             // kCheck iterations of the inner CG
    BScalars *bsc = nullptr, *hbsc = nullptr;
    Scalars *osc = nullptr, *hosc = nullptr;  // per rhs: the FP64 residuals' norms
};

namespace {

long long bcount(gbds_bsolver b) { return (long long)b->s1->g.Vh * b->nrhs; }
int bblocks(gbds_bsolver b) { return (int)((bcount(b) + 127) / 128); }
size_t bcs(gbds_bsolver b) { return (size_t)b->s1->g.stride * b->nrhs; }

#define GBDS_BN(NR, CALL) \
    switch (NR) {         \
    case 2: CALL(2); break; \
    case 4: CALL(4); break; \
    case 8: CALL(8); break; \
    case 16: CALL(16); break; \
    default: CALL(32); break; \
    }

int bblocks2(gbds_bsolver b) { return (bblocks(b) + kBRows - 1) / kBRows; }

cudaError_t bfinish_on(gbds_bsolver b, int mode, cudaStream_t st) {
    launch_pdl(bfinish, dim3(bblocks2(b)), 256, st, b->bpartials, bblocks(b), b->nrhs, b->bpartials2, b->ticket, b->bsc,
               mode);
    count_launch();
    return cudaGetLastError();
}

// the multi-RHS kernel of the launches without an epilogue (FP32 spin pairs,
// 24^3x48: 8 rhs 0.167 ms with variant 2 against 0.197 with 3 and 0.194 plain,
// 16 rhs 0.278 with 3 against 0.297 with 2)
int packed_variant(gbds_bsolver b) { return b->nrhs >= 16 ? 3 : b->nrhs == 8 ? 2 : 0; }

// out = in - kappa^2 D_eo D_oe in for all rhs (partials: per-rhs |out|^2)
// flip: the direction of the first of the two launches (the second's is the other)
cudaError_t apply_Mb(gbds_bsolver b, const void *in, void *out, int isign, double *partials, cudaStream_t st,
                     bool flip = false) {
    gbds_solver s = b->s1;
    const float k2 = (float)(s->prm.kappa * s->prm.kappa);
    // inner fields in FP32 spin pairs: the fully packed FP32x2 kernel from 8
    // rhs on (measured faster there), from 16 on with two rhs a thread where
    // there is no epilogue
    const int v = b->nrhs >= 8 ? 2 : 0;
    cudaError_t e = launch_gen_f32p(b->gm, s->prm.inner_recon, b->nrhs, s->gauge32, in, b->t, isign, 0, nullptr, 0.f,
                                    nullptr, st, packed_variant(b), flip);
    if (e != cudaSuccess) return e;
    return launch_gen_f32p(b->gm, s->prm.inner_recon, b->nrhs, s->gauge32, b->t, out, isign, 1, in, -k2, partials, st, v,
                           !flip);
}

// The fully packed operator (8, 16, 32 rhs) fuses the CG's r -= alpha Ap into
// M^+'s second launch: Ap is never stored.
bool fused_update(gbds_bsolver b) { return b->nrhs >= 8; }

// r -= alpha_r M^+ in for all active rhs, per-rhs |r|^2 partials
cudaError_t apply_Mb_dagger_update(gbds_bsolver b, const void *in, cudaStream_t st, bool flip) {
    gbds_solver s = b->s1;
    const float k2 = (float)(s->prm.kappa * s->prm.kappa);
    cudaError_t e =
        launch_gen_f32p(b->gm, s->prm.inner_recon, b->nrhs, s->gauge32, in, b->t, -1, 0, nullptr, 0.f, nullptr, st,
                        packed_variant(b), flip);
    if (e != cudaSuccess) return e;
    return launch_gen_f32p_cg_update(b->gm, s->prm.inner_recon, b->nrhs, s->gauge32, b->t, -1, 1, in, -k2, b->bsc, b->r,
                                     b->bpartials, st, !flip);
}

// the FP64 norms of all rhs in one read (a read after each rhs left the GPU idle
// for about 15 us: 16 rhs on 16^3x32 37.2 -> 36.1 ms a solve, 8 rhs on 8^3x16
// 5.20 -> 4.89)
cudaError_t read_norms(gbds_bsolver b, cudaStream_t st) {
    cudaError_t e = cudaMemcpyAsync(b->hosc, b->osc, sizeof(Scalars) * b->nrhs, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e;
}

cudaError_t read_bscalars(gbds_bsolver b, cudaStream_t st) {
    cudaError_t e = cudaMemcpyAsync(b->hbsc, b->bsc, sizeof(BScalars) * b->nrhs, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e;
}

// One iteration of the lockstep CG (7 launches, 8 without the fused update).
// flip alternates: an iteration's five passes over the fields alternate too.
cudaError_t bcg_iteration(gbds_bsolver b, cudaStream_t st, bool flip) {
    const long long n = bcount(b);
    const int nb = bblocks(b);
    const size_t cs = bcs(b);
    const int nr = b->nrhs;
    cudaError_t e = apply_Mb(b, b->p, b->Mp, +1, b->bpartials, st, flip);
    if (e == cudaSuccess) e = bfinish_on(b, kBAlpha, st);
    if (e == cudaSuccess && fused_update(b)) {
        e = apply_Mb_dagger_update(b, b->Mp, st, flip);
    } else if (e == cudaSuccess) {
        e = apply_Mb(b, b->Mp, b->Ap, -1, nullptr, st, flip);
        if (e != cudaSuccess) return e;
#define GBDS_UPD(NR)                                                                                      \
    launch_pdl(bcg_update<NR>, dim3(nb), 128, st, static_cast<float4 *>(b->r), static_cast<const float4 *>(b->Ap), \
               (const BScalars *)b->bsc, n, cs, b->bpartials)
        GBDS_BN(nr, GBDS_UPD)
#undef GBDS_UPD
        count_launch();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = bfinish_on(b, kBBeta, st);
    if (e != cudaSuccess) return e;
#define GBDS_XP(NR)                                                                                         \
    launch_pdl(bcg_xpay<NR>, dim3(nb), 128, st, static_cast<float4 *>(b->e), static_cast<const float4 *>(b->r), \
               static_cast<float4 *>(b->p), (const BScalars *)b->bsc, n, cs, (int)flip)
    GBDS_BN(nr, GBDS_XP)
#undef GBDS_XP
    count_launch();
    return cudaGetLastError();
}

// Lockstep CG on the active right-hand sides (x = e = 0, r = p = residual,
// rr set); each stops at rr <= target[q] or when it stagnates.
cudaError_t bcg(gbds_bsolver b, const std::vector<double> &target, int max_iter, std::vector<int> &iters,
                cudaStream_t st) {
    const int nr = b->nrhs;
    std::vector<double> best(nr, 1e300);
    std::vector<int> best_k(nr, 0);
    cudaError_t e = read_bscalars(b, st);
    int k = 0;
    while (e == cudaSuccess && k < max_iter) {
        bool any = false;
        for (int q = 0; q < nr; q++) any |= b->hbsc[q].active != 0;
        if (!any) break;
        int done = 1;
        if (b->steps.exec && k % kCheck == 0 && k + kCheck <= max_iter) {
            e = launch(b->steps, st);
            done = kCheck;
        } else {
            e = bcg_iteration(b, st, k & 1);
        }
        if (e != cudaSuccess) break;
        k += done;
        for (int q = 0; q < nr; q++)
            if (b->hbsc[q].active) iters[q] += done;
        if (k % kCheck == 0 || k == max_iter) {
            e = read_bscalars(b, st);
            if (e != cudaSuccess) break;
            bool changed = false;
            for (int q = 0; q < nr; q++) {
                BScalars &c = b->hbsc[q];
                if (!c.active) continue;
                if (!(c.rr > target[q]) || stagnated(c.rr, k, best[q], best_k[q])) {
                    c.active = 0;  // converged, stagnated or NaN
                    changed = true;
                }
            }
            if (changed) {
                e = cudaMemcpyAsync(b->bsc, b->hbsc, sizeof(BScalars) * nr, cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            }
        }
    }
    return e;
}

void brelease(gbds_bsolver b) {
    for (auto *v : {&b->b64, &b->x64, &b->r64})
        for (void *p : *v)
            if (p) cudaFree(p);
    void *bufs[] = {b->e, b->r, b->p, b->Ap, b->Mp, b->t, b->bpartials, b->bpartials2, b->ticket, b->bsc, b->osc};
    for (void *p : bufs)
        if (p) cudaFree(p);
    if (b->hbsc) cudaFreeHost(b->hbsc);
    if (b->hosc) cudaFreeHost(b->hosc);
    if (b->steps.exec) cudaGraphExecDestroy(b->steps.exec);
    if (b->s1) gbds_solver_destroy(b->s1);
}

}  // namespace

extern "C" int gbds_bsolver_create(gbds_bsolver *out, const int dims[4], int nrhs, const gbds_solver_params *p) {
    if (!out || !p) return set_error(GBDS_ERROR_INVALID_VALUE, "NULL argument");
    *out = nullptr;
    if (nrhs != 2 && nrhs != 4 && nrhs != 8 && nrhs != 16 && nrhs != 32)
        return set_error(GBDS_ERROR_INVALID_VALUE, "nrhs must be 2, 4, 8, 16 or 32");
    if (p->inner_prec != 32) return set_error(GBDS_ERROR_UNSUPPORTED, "the batched solver runs an FP32 inner CG (inner_prec 32)");
    gbds_bsolver b = new (std::nothrow) gbds_bsolver_s;
    if (!b) return set_error(GBDS_ERROR_OUT_OF_MEMORY, "host allocation failed");
    b->nrhs = nrhs;
    int rc = create_solver(&b->s1, dims, p, false);
    if (rc != GBDS_SUCCESS) {
        delete b;
        return rc;
    }
    const Geom &g = b->s1->g;
    b->gm = g;
    b->gm.zblock = gen_zblock(g, nrhs, GBDS_SPINOR_F32_PAIRS, p->inner_recon);
    const size_t f64 = spinor_bytes(g, 64), f32m = spinor_bytes(g, 32) * nrhs;
    cudaError_t e = cudaSuccess;
    for (auto *v : {&b->b64, &b->x64, &b->r64}) {
        v->assign(nrhs, nullptr);
        for (int q = 0; q < nrhs && e == cudaSuccess; q++) e = cudaMalloc(&(*v)[q], f64);
    }
    void **bufs[] = {&b->e, &b->r, &b->p, &b->Mp, &b->t};
    for (void **x : bufs)
        if (e == cudaSuccess) e = cudaMalloc(x, f32m);
    if (e == cudaSuccess && !fused_update(b)) e = cudaMalloc(&b->Ap, f32m);  // else never stored
    if (e == cudaSuccess) e = cudaMalloc(&b->bpartials, sizeof(double) * (size_t)bblocks(b) * nrhs);
    if (e == cudaSuccess) e = cudaMalloc(&b->bpartials2, sizeof(double) * (size_t)bblocks2(b) * nrhs);
    if (e == cudaSuccess) e = new_ticket(&b->ticket);
    if (e == cudaSuccess) e = cudaMalloc(&b->bsc, sizeof(BScalars) * nrhs);
    if (e == cudaSuccess) e = cudaMallocHost(&b->hbsc, sizeof(BScalars) * nrhs);
    if (e == cudaSuccess) e = cudaMalloc(&b->osc, sizeof(Scalars) * nrhs);
    if (e == cudaSuccess) e = cudaMallocHost(&b->hosc, sizeof(Scalars) * nrhs);
    if (e == cudaSuccess)
        record(b->steps, kCheck * (fused_update(b) ? 7 : 8), [&](cudaStream_t cs) {
            cudaError_t le = cudaSuccess;
            for (int i = 0; i < kCheck && le == cudaSuccess; i++) le = bcg_iteration(b, cs, i & 1);
            return le;
        });
    if (e != cudaSuccess) {
        brelease(b);
        delete b;
        return cuda_error(e, "gbds_bsolver_create");
    }
    *out = b;
    return GBDS_SUCCESS;
}

extern "C" int gbds_bsolver_destroy(gbds_bsolver b) {
    if (!b) return GBDS_SUCCESS;
    cudaDeviceSynchronize();
    brelease(b);
    delete b;
    return GBDS_SUCCESS;
}

extern "C" int gbds_bsolver_set_gauge(gbds_bsolver b, const double *u_packed, void *stream) {
    if (!b) return set_error(GBDS_ERROR_NOT_INITIALIZED, "solver is NULL");
    return gbds_solver_set_gauge(b->s1, u_packed, stream);
}

extern "C" int gbds_bsolver_solve(gbds_bsolver b, const double *b_packed, double *x_packed, gbds_solver_stats *stats,
                                  void *stream) {
    if (!b) return set_error(GBDS_ERROR_NOT_INITIALIZED, "solver is NULL");
    gbds_solver s = b->s1;
    if (!s->have_gauge) return set_error(GBDS_ERROR_NOT_INITIALIZED, "gbds_bsolver_set_gauge has not been called");
    if (!b_packed || !x_packed) return set_error(GBDS_ERROR_INVALID_VALUE, "NULL field pointer");
    if ((reinterpret_cast<uintptr_t>(b_packed) | reinterpret_cast<uintptr_t>(x_packed)) & 15u)
        return set_error(GBDS_ERROR_INVALID_VALUE, "fields must be 16-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const auto t0 = std::chrono::steady_clock::now();
    const Geom &g = s->g;
    const int nr = b->nrhs;
    const long long n = bcount(b);
    const size_t cs = bcs(b);
    const double tol2 = s->prm.tol * s->prm.tol;
    const size_t vlen = (size_t)g.V * 24;  // doubles per packed right-hand side
    // per rhs: |b|^2, |b - M x|^2 (FP64), |M^+ b|^2, |M^+ (b - M x)|^2
    std::vector<double> b2(nr, 0.0), r2(nr, 0.0), c2(nr, 0.0), n2(nr, 0.0);
    std::vector<int> iters(nr, 0), cycles(nr, 0);
    std::vector<char> live(nr, 0);  // still being solved
    std::vector<char> last(nr, 0);  // no progress in the last cycle: measure once more, then stop
    cudaError_t e = cudaSuccess;
    for (int q = 0; q < nr && e == cudaSuccess; q++) {
        e = launch_pack_spinor(g, 64, b_packed + q * vlen, nullptr, 0, 0, b->b64[q], st);
        if (e == cudaSuccess) e = norm_into<double>(s, b->b64[q], b->r64[q], nullptr, kOuterRR, st, b->osc + q);  // r = b
        if (e == cudaSuccess) e = zero<double>(s, b->x64[q], st);
    }
    if (e == cudaSuccess) e = read_norms(b, st);
    for (int q = 0; q < nr && e == cudaSuccess; q++) {
        b2[q] = r2[q] = b->hosc[q].outer_rr;
        live[q] = b2[q] > 0;
    }
    int total = 0;
    bool first = true;
    while (e == cudaSuccess) {
        // c_q = M^+ (r_q / |r_q|) in FP32 for all right-hand sides at once, and |c_q|^2
        {
            RhsFields f{};
            for (int q = 0; q < nr; q++) {
                f.v[q] = static_cast<double2 *>(b->r64[q]);
                f.s[q] = live[q] ? 1.0 / std::sqrt(r2[q]) : 0.0;
            }
            bdemote_all<<<(g.Vh + kBXSites - 1) / kBXSites, 256, 0, st>>>(
                f, static_cast<float4 *>(b->r), static_cast<float4 *>(b->p), g.Vh, g.stride, nr, cs);
            count_launch();
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = apply_Mb(b, b->r, b->Mp, -1, b->bpartials, st);
        for (int q = 0; q < nr; q++) b->hbsc[q] = BScalars{};
        if (e == cudaSuccess) e = cudaMemcpyAsync(b->bsc, b->hbsc, sizeof(BScalars) * nr, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = bfinish_on(b, kBSetRR, st);
        if (e == cudaSuccess) e = read_bscalars(b, st);
        if (e != cudaSuccess) break;
        std::vector<double> target(nr, 0.0);
        bool any = false;
        for (int q = 0; q < nr; q++) {
            const double s2 = b->hbsc[q].rr;
            BScalars &c = b->hbsc[q];
            c = BScalars{};
            if (!live[q]) continue;
            n2[q] = r2[q] * s2;
            if (first) c2[q] = n2[q];
            if (last[q] || !(n2[q] > tol2 * c2[q]) || total >= s->prm.max_iter || !(s2 > 0)) {
                live[q] = 0;  // converged, stalled, or nothing left to solve
                continue;
            }
            double delta = s->prm.inner_tol;
            const double need = 0.5 * s->prm.tol * std::sqrt(c2[q] / n2[q]);
            if (need > delta) delta = need;
            target[q] = delta * delta;
            c.active = 1;
            c.beta = 1.0 / std::sqrt(s2);  // scale of the inner right-hand side
            any = true;
        }
        first = false;
        if (!any) break;
        // inner CG on A e_q = c_q / |c_q| from e = 0
        e = cudaMemcpyAsync(b->bsc, b->hbsc, sizeof(BScalars) * nr, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) {
#define GBDS_SC(NR)                                                                                                  \
    bscale_copy<NR><<<bblocks(b), 128, 0, st>>>(static_cast<const float4 *>(b->Mp), b->bsc, static_cast<float4 *>(b->r), \
                                                static_cast<float4 *>(b->p), n, cs)
            GBDS_BN(nr, GBDS_SC)
#undef GBDS_SC
            count_launch();
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemsetAsync(b->e, 0, spinor_bytes(g, 32) * nr, st);
        if (e == cudaSuccess) {
#define GBDS_NRM(NR) bnorm<NR><<<bblocks(b), 128, 0, st>>>(static_cast<const float4 *>(b->r), n, cs, b->bpartials)
            GBDS_BN(nr, GBDS_NRM)
#undef GBDS_NRM
            count_launch();
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = bfinish_on(b, kBSetRR, st);
        std::vector<int> it(nr, 0);
        if (e == cudaSuccess) e = bcg(b, target, s->prm.max_iter - total, it, st);
        if (e != cudaSuccess) break;
        int most = 0;
        for (int q = 0; q < nr; q++) {
            if (target[q] == 0.0) continue;
            iters[q] += it[q];
            cycles[q]++;
            most = std::max(most, it[q]);
        }
        total += most;
        // x_q += |c_q| e_q (all rhs in one launch);  r_q = b_q - M x_q in FP64
        {
            RhsFields f{};
            for (int q = 0; q < nr; q++) {
                f.v[q] = static_cast<double2 *>(b->x64[q]);
                f.s[q] = target[q] == 0.0 ? 0.0 : std::sqrt(n2[q]);
            }
            bpromote_all<<<(g.Vh + kBXSites - 1) / kBXSites, 256, 0, st>>>(static_cast<const float4 *>(b->e), f, g.Vh,
                                                                           g.stride, nr, cs);
            count_launch();
            e = cudaGetLastError();
        }
        for (int q = 0; q < nr && e == cudaSuccess; q++) {
            if (target[q] == 0.0) continue;
            e = outer_residual(s, b->b64[q], b->x64[q], b->r64[q], df_range(b2[q]), st);
            if (e == cudaSuccess) e = finish_on(s, kOuterRR, st, 0, b->osc + q);
        }
        if (e == cudaSuccess) e = read_norms(b, st);
        for (int q = 0; q < nr && e == cudaSuccess; q++) {
            if (target[q] == 0.0) continue;
            const double prev = r2[q];
            r2[q] = b->hosc[q].outer_rr;
            if (!(r2[q] < prev) || !(r2[q] > 0)) last[q] = 1;  // no progress (or NaN, or exact)
        }
    }
    for (int q = 0; q < nr && e == cudaSuccess; q++)
        e = launch_unpack_spinor(g, 64, b->x64[q], nullptr, 0, 0, x_packed + q * vlen, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_error(e, "gbds_bsolver_solve");
    const double secs = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (stats) {
        for (int q = 0; q < nr; q++) {
            gbds_solver_stats &o = stats[q];
            o.iterations = iters[q];
            o.cycles = cycles[q];
            o.residual = c2[q] > 0 ? std::sqrt(n2[q] / c2[q]) : 0.0;
            o.true_residual = b2[q] > 0 ? std::sqrt(r2[q] / b2[q]) : 0.0;
            o.converged = o.residual <= s->prm.tol ? 1 : 0;
            o.seconds = secs;
        }
    }
    return GBDS_SUCCESS;
}
