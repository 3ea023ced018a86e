// The FP64 Dslash on the integer pipes (block fixed point, fixpoint.cuh).
//
// GB300 issues 2 FP64 operations a clock and SM.  The operator needs 816 a
// site, so in FP64 arithmetic it ran at 0.16 of the HBM roofline with the FP64
// pipe 92 % busy (24^3x48 0.493 ms, 32^3x64 1.477 ms).  32 x 32 -> 64-bit
// integer multiply-adds issue at about 22 a clock and SM, and three of them
// make one multiply-add of two 59-bit fixed-point numbers, with exact sums.
// Here only the projection (96 additions a site) and the final conversion
// (48) stay in FP64; the colour multiply and the accumulation run on
// integers: 24^3x48 0.175 ms, 32^3x64 0.533 ms (12-real links 0.301, 0.950).
// Bound by integer issue (ALU 56 %, IMAD pipe 49 %, FP64 pipe 45 % busy, 464
// instructions a hop and thread).
//
// Error against 64 bits (random SU(3), N(0,1) spinors): 1.45e-16 of the
// result's norm, where the FP64 kernel had 1.96e-16 (it rounds each of the 6
// multiply-adds and 16 additions that form a component; here the projection
// and the result are rounded).
//
// A CTA of three warps takes 32 consecutive sites and warp c computes colour
// c of their outputs, as in the double-float kernel (dslash_df.cu): it loads
// colour c of the neighbour's four spins, projects them, converts the four
// reals against their largest exponent and passes them to the other warps
// through shared memory (one barrier a hop, two buffers); each warp converts
// row c of U (forward) or column c (backward) to the exponent that puts
// every product on the common scale of its sums.  So each number is converted
// once, except that the 12-real links' rebuilt row is formed where it is
// used.  80 registers (7 CTAs per SM; 6 and 8 measured 0.187 and 0.184 ms;
// prefetching the next hop's spinors 0.189 ms).
//
// The scale of the sums follows the largest product so far (spinor exponent
// + link exponent); when it grows, the sums are shifted.  An output is within
// a few units of 2^-54 of the largest product of its colour, before its own
// rounding.  Operands beyond the exponents the integers cover (2^177 and up,
// infinities, NaN, or every product below 2^-646) take the plain FP64 path
// at the end of the kernel, site by site.
#include "dslash_kernel.cuh"
#include "fixpoint.cuh"

namespace gbds {

namespace {

constexpr int kFxSites = 32;  // sites of a group of three warps
constexpr uint32_t kFxTop = 1200, kFxLeast = 1400;  // biased operand and (two operands') product exponents

template <int GROUPS>
struct FxShared {
    int4 h[GROUPS][2][2][3][kFxSites];   // [buffer][spin half][colour][site]: n, g of re, im
    uint32_t e[GROUPS][2][3][kFxSites];  // biased scale exponent of the colour's four reals
};

__device__ __forceinline__ double2 ld_link(const double2 *p, uint64_t pol) {
    double2 v;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
        : "=d"(v.x), "=d"(v.y)
        : "l"(p), "l"(pol));
    return v;
}

__device__ __forceinline__ uint32_t hi_word(double v) { return (uint32_t)__double2hiint(v); }
__device__ __forceinline__ fix2 to_fix(double v, uint32_t t) {
    return fix_convert(hi_word(v), (uint32_t)__double2loint(v), t);
}

// conj(a x b)_j of one colour j: a_k b_l - a_l b_k, conjugated
__device__ __forceinline__ double2 cross_conj(double2 ak, double2 bl, double2 al, double2 bk) {
    return make_double2(fma(ak.x, bl.x, -ak.y * bl.y) - fma(al.x, bk.x, -al.y * bk.y),
                        -(fma(ak.x, bl.y, ak.y * bl.x) - fma(al.x, bk.y, al.y * bk.x)));
}

// Row c (DAG: column c) of the link; component i of a link block at i * stride.
template <int RECON, bool DAG, typename LOAD>
__device__ __forceinline__ void link_row(const LOAD &ld, int c, double2 (&u)[3]) {
    if constexpr (RECON == 18) {
#pragma unroll
        for (int j = 0; j < 3; j++) u[j] = ld(DAG ? j * 3 + c : c * 3 + j);
    } else if constexpr (DAG) {
        const int k = c == 2 ? 0 : c + 1, l = c == 0 ? 2 : c - 1;
        u[0] = ld(c);
        u[1] = ld(3 + c);
        u[2] = cross_conj(ld(k), ld(3 + l), ld(l), ld(3 + k));
    } else if (c < 2) {
#pragma unroll
        for (int j = 0; j < 3; j++) u[j] = ld(c * 3 + j);
    } else {
        double2 r[6];
#pragma unroll
        for (int j = 0; j < 6; j++) r[j] = ld(j);
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const int k = (j + 1) % 3, l = (j + 2) % 3;
            u[j] = cross_conj(r[k], r[3 + l], r[l], r[3 + k]);
        }
    }
}

// the barrier of the three warps of group grp
template <int GROUPS>
__device__ __forceinline__ void fx_sync(int grp) {
    if constexpr (GROUPS == 1) __syncthreads();
    else asm volatile("bar.sync %0, 96;" ::"r"(grp + 1) : "memory");
}

// acc += code * w for one complex, code 0: +1, 1: -1, 2: +i, 3: -i
template <int CODE>
__device__ __forceinline__ void fx_acc(int64_t (&acc)[2], const int64_t (&w)[2]) {
    if constexpr (CODE == 0) { acc[0] += w[0]; acc[1] += w[1]; }
    else if constexpr (CODE == 1) { acc[0] -= w[0]; acc[1] -= w[1]; }
    else if constexpr (CODE == 2) { acc[0] -= w[1]; acc[1] += w[0]; }
    else { acc[0] += w[1]; acc[1] -= w[0]; }
}

// What a thread (colour c of one site) keeps over its hops.
struct FxSum {
    int64_t acc[4][2];  // the four output spins, in units of 2^(e - 2 * 1023 - kFixUnit)
    uint32_t e;         // the two operands' biased exponents at the scale of the sums
    uint32_t top;       // the largest biased exponent of any operand
    uint32_t any;       // the spinor exponents, or-ed: 0 when every source is 0 (or subnormal)
};

// The thread's place: colour c, lane, group grp; act: it has a site.
struct FxThread {
    int c, lane, grp;
    bool act;
    uint64_t pol;
};

template <int MU, int SIGMA, bool DAG, int ND, int RECON, int GROUPS>
__device__ __forceinline__ void fx_hop(const DslashArgs<double> &a, const FxThread &th, int nbr, int hl, int lp,
                                       FxShared<GROUPS> &sm, FxSum &S) {
    using P = Proj<MU>;
    constexpr int f = SIGMA > 0 ? 0 : 1, buf = DAG ? 1 : 0;
    const int stride = a.g.stride, c = th.c, lane = th.lane, grp = th.grp;
    double2 ud[3];
    if (th.act) {
        const double2 *U = reinterpret_cast<const double2 *>(a.gauge + (size_t)(lp * ND + MU) * a.link_block_bytes) + hl;
        link_row<RECON, DAG>([&](int i) { return ld_link(U + (size_t)i * stride, th.pol); }, c, ud);
        cx<double> s[4];
#pragma unroll
        for (int sp = 0; sp < 4; sp++) {
            const double2 q = __ldg(a.psi + (size_t)(sp * 3 + c) * stride + nbr);
            s[sp] = {q.x, q.y};
        }
        const cx<double> h0 = cadd(s[0], mulc<P::a0 ^ f>(s[P::j0])), h1 = cadd(s[1], mulc<P::a1 ^ f>(s[P::j1]));
        const double v[4] = {h0.r, h0.i, h1.r, h1.i};
        uint32_t ex[4], e = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            ex[i] = fix_exponent(hi_word(v[i]));
            e = max(e, ex[i]);
        }
        fix2 q[4];
#pragma unroll
        for (int i = 0; i < 4; i++) q[i] = to_fix(v[i], e + 3 - ex[i]);
        sm.h[grp][buf][0][c][lane] = make_int4(q[0].n, q[0].g, q[1].n, q[1].g);
        sm.h[grp][buf][1][c][lane] = make_int4(q[2].n, q[2].g, q[3].n, q[3].g);
        sm.e[grp][buf][c][lane] = e;
    }
    fx_sync<GROUPS>(grp);
    if (!th.act) return;
    uint32_t ex[3][2], eh[3], et = 0;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        ex[j][0] = fix_exponent(hi_word(ud[j].x));
        ex[j][1] = fix_exponent(hi_word(ud[j].y));
        eh[j] = sm.e[grp][buf][j][lane];
        const uint32_t eu = max(ex[j][0], ex[j][1]);
        S.top = max(S.top, max(eu, eh[j]));
        S.any |= eh[j];
        et = max(et, eu + eh[j]);
    }
    if (et > S.e) {
        const uint32_t d = et - S.e;
#pragma unroll
        for (int sp = 0; sp < 4; sp++)
#pragma unroll
            for (int p = 0; p < 2; p++) S.acc[sp][p] = fix_sar(S.acc[sp][p], d);
        S.e = et;
    }
    // W: the products' high parts; X: their cross parts, in units of 2^-32
    // (the constant rounds them to nearest)
    int64_t W[2][2], X[2][2];
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
        for (int p = 0; p < 2; p++) {
            W[k][p] = 0;
            X[k][p] = 1ll << 31;
        }
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const uint32_t t0 = S.e - eh[j] + 3;
        const fix2 ur = to_fix(ud[j].x, t0 - ex[j][0]), ui = to_fix(ud[j].y, t0 - ex[j][1]);
        const fix2 um = {-ui.n, ~ui.g};
        // re += ur hr - ui hi, im += ur hi + ui hr (U^+: ui changes sign)
        const fix2 a1 = DAG ? ui : um, a2 = DAG ? um : ui;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int4 q = sm.h[grp][buf][k][j][lane];
            fix_mad(W[k][0], ur.n, q.x); fix_mad(X[k][0], ur.n, q.y); fix_mad(X[k][0], ur.g, q.x);
            fix_mad(W[k][0], a1.n, q.z); fix_mad(X[k][0], a1.n, q.w); fix_mad(X[k][0], a1.g, q.z);
            fix_mad(W[k][1], ur.n, q.z); fix_mad(X[k][1], ur.n, q.w); fix_mad(X[k][1], ur.g, q.z);
            fix_mad(W[k][1], a2.n, q.x); fix_mad(X[k][1], a2.n, q.y); fix_mad(X[k][1], a2.g, q.x);
        }
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
#pragma unroll
        for (int p = 0; p < 2; p++) W[k][p] += X[k][p] >> 32;
        fx_acc<0>(S.acc[k], W[k]);
    }
    fx_acc<P::b2 ^ f>(S.acc[2], W[P::k2]);
    fx_acc<P::b3 ^ f>(S.acc[3], W[P::k3]);
}

// Colour c of one hop in plain FP64.
template <int MU, int SIGMA, bool DAG, int ND, int RECON>
__device__ __forceinline__ void fx_plain_hop(const DslashArgs<double> &a, int c, int nbr, int hl, int lp,
                                             cx<double> (&acc)[4]) {
    using P = Proj<MU>;
    constexpr int f = SIGMA > 0 ? 0 : 1;
    const int stride = a.g.stride;
    const double2 *U = reinterpret_cast<const double2 *>(a.gauge + (size_t)(lp * ND + MU) * a.link_block_bytes) + hl;
    double2 u[3];
    link_row<RECON, DAG>([&](int i) { return __ldg(U + (size_t)i * stride); }, c, u);
    cx<double> w[2] = {};
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const cx<double> m = {u[j].x, DAG ? -u[j].y : u[j].y};
        cx<double> s[4];
#pragma unroll
        for (int sp = 0; sp < 4; sp++) {
            const double2 q = __ldg(a.psi + (size_t)(sp * 3 + j) * stride + nbr);
            s[sp] = {q.x, q.y};
        }
        const cx<double> hs[2] = {cadd(s[0], mulc<P::a0 ^ f>(s[P::j0])), cadd(s[1], mulc<P::a1 ^ f>(s[P::j1]))};
#pragma unroll
        for (int k = 0; k < 2; k++) {
            w[k].r = fma(-m.i, hs[k].i, fma(m.r, hs[k].r, w[k].r));
            w[k].i = fma(m.i, hs[k].r, fma(m.r, hs[k].i, w[k].i));
        }
    }
    acc[0] = cadd(acc[0], w[0]);
    acc[1] = cadd(acc[1], w[1]);
    acc[2] = cadd(acc[2], mulc<P::b2 ^ f>(w[P::k2]));
    acc[3] = cadd(acc[3], mulc<P::b3 ^ f>(w[P::k3]));
}

// whether every real of the site's source spinors is +-0
template <int ND>
__device__ __forceinline__ bool fx_sources_zero(const DslashArgs<double> &a, const Nbr &n) {
    unsigned long long bits = 0;
#pragma unroll
    for (int mu = 0; mu < ND; mu++)
#pragma unroll 1
        for (int i = 0; i < 12; i++) {
            const double2 *p = a.psi + (size_t)i * a.g.stride;
            const double2 f = __ldg(p + n.f[mu]), b = __ldg(p + n.b[mu]);
            bits |= __double_as_longlong(f.x) | __double_as_longlong(f.y) | __double_as_longlong(b.x) |
                    __double_as_longlong(b.y);
        }
    return (bits << 1) == 0;
}

template <int ND, int RECON, int ISIGN, int MU, int GROUPS>
__device__ __forceinline__ void fx_dir(const DslashArgs<double> &a, const FxThread &th, int h, const Nbr &n,
                                       FxShared<GROUPS> &sm, FxSum &S) {
    fx_hop<MU, ISIGN, false, ND, RECON>(a, th, n.f[MU], h, a.pt, sm, S);
    fx_hop<MU, -ISIGN, true, ND, RECON>(a, th, n.b[MU], n.b[MU], 1 - a.pt, sm, S);
}

template <int ND, int RECON, int ISIGN, int MU>
__device__ __forceinline__ void fx_plain_dir(const DslashArgs<double> &a, int c, int h, const Nbr &n, cx<double> (&acc)[4]) {
    fx_plain_hop<MU, ISIGN, false, ND, RECON>(a, c, n.f[MU], h, a.pt, acc);
    fx_plain_hop<MU, -ISIGN, true, ND, RECON>(a, c, n.b[MU], n.b[MU], 1 - a.pt, acc);
}

// res = Dslash psi, or (EPI 1) x + coef Dslash psi with partials[block] = the
// block's sum of |res|^2 where partials != nullptr, or (EPI 2) the CG's update
// r -= alpha (x + coef Dslash psi) in place of the store, with |r|^2.  GROUPS groups of three
// warps a CTA: 1, or 4 where partials of 128-site blocks are wanted.
template <int ND, int RECON, int ISIGN, int EPI, int GROUPS>
__global__ void __launch_bounds__(96 * GROUPS, GROUPS == 1 ? 7 : 2)
    dslash_fx_kernel(const DslashArgs<double> a, const double2 *__restrict__ x, double coef, const CgUpdate<double> upd,
                     double *partials) {
    __shared__ FxShared<GROUPS> sm;
    if (gridDim.x > 152 * (GROUPS == 1 ? 7 : 2)) pdl_allow_next();
    const int warp = threadIdx.x >> 5;
    FxThread th;
    th.lane = threadIdx.x & 31;
    th.grp = GROUPS == 1 ? 0 : warp / 3;
    th.c = GROUPS == 1 ? warp : warp % 3;
    const int h = a.first + (blockIdx.x * GROUPS + th.grp) * kFxSites + th.lane;
    th.act = h < a.end;
    Nbr n;
    if (th.act) neighbours<ND>(a.g, h, a.pt, n);
    th.pol = l2_evict_first_policy();
    pdl_wait_prev();
    FxSum S;
#pragma unroll
    for (int s = 0; s < 4; s++) S.acc[s][0] = S.acc[s][1] = 0;
    S.e = S.top = S.any = 0;
    fx_dir<ND, RECON, ISIGN, 0>(a, th, h, n, sm, S);
    fx_dir<ND, RECON, ISIGN, 1>(a, th, h, n, sm, S);
    fx_dir<ND, RECON, ISIGN, 2>(a, th, h, n, sm, S);
    if constexpr (ND == 4) fx_dir<ND, RECON, ISIGN, 3>(a, th, h, n, sm, S);
    double nrm = 0;
    if (th.act) {
        cx<double> r[4] = {};
        if (S.top <= kFxTop && S.e >= kFxLeast) {
            const double sc = __hiloint2double((int)((S.e - (2046 + kFixUnit - 1023)) << 20), 0);
#pragma unroll
            for (int sp = 0; sp < 4; sp++) r[sp] = {(double)S.acc[sp][0] * sc, (double)S.acc[sp][1] * sc};
        } else if (S.any != 0 || S.top >= 2047 || !fx_sources_zero<ND>(a, n)) {
            fx_plain_dir<ND, RECON, ISIGN, 0>(a, th.c, h, n, r);
            fx_plain_dir<ND, RECON, ISIGN, 1>(a, th.c, h, n, r);
            fx_plain_dir<ND, RECON, ISIGN, 2>(a, th.c, h, n, r);
            if constexpr (ND == 4) fx_plain_dir<ND, RECON, ISIGN, 3>(a, th.c, h, n, r);
        }
#pragma unroll
        for (int sp = 0; sp < 4; sp++) {
            const size_t i = (size_t)(sp * 3 + th.c) * a.g.stride + h;
            if constexpr (EPI) {
                const double2 xv = __ldg(x + i);
                r[sp] = {fma(coef, r[sp].r, xv.x), fma(coef, r[sp].i, xv.y)};
                if constexpr (EPI == 2) {
                    const double al = -*upd.alpha;
                    const double2 ro = upd.r[i];
                    r[sp] = {fma(al, r[sp].r, ro.x), fma(al, r[sp].i, ro.y)};
                }
                nrm = fma(r[sp].r, r[sp].r, nrm);
                nrm = fma(r[sp].i, r[sp].i, nrm);
            }
            if constexpr (EPI == 2) upd.r[i] = make_double2(r[sp].r, r[sp].i);
            else __stcs(a.res + i, make_double2(r[sp].r, r[sp].i));
        }
    }
    if constexpr (EPI) {
        if (partials) block_sum_to<double>(partials, nrm);
    }
}

DslashArgs<double> f64_args(const Geom &g, int recon, const void *gauge, const void *psi, void *res, int cb,
                            const SiteRange &range = {}) {
    DslashArgs<double> a;
    a.g = g;
    a.psi = static_cast<const double2 *>(psi);
    a.res = static_cast<double2 *>(res);
    a.gauge = static_cast<const char *>(gauge);
    a.link_block_bytes = (size_t)Field<double>::link_vecs(recon) * g.stride * 16;
    a.pt = 1 - cb;
    a.first = range.first;
    a.end = range.end(g);
    return a;
}

template <int ND, int RECON, int EPI, int GROUPS>
cudaError_t launch_fx(const DslashArgs<double> &a, int isign, const double2 *x, double coef, double *partials,
                      cudaStream_t st, const CgUpdate<double> &upd = {}) {
    const dim3 grid((a.end - a.first + kFxSites * GROUPS - 1) / (kFxSites * GROUPS));
    const int threads = 96 * GROUPS;
    if (isign > 0) launch_pdl(dslash_fx_kernel<ND, RECON, 1, EPI, GROUPS>, grid, threads, st, a, x, coef, upd, partials);
    else launch_pdl(dslash_fx_kernel<ND, RECON, -1, EPI, GROUPS>, grid, threads, st, a, x, coef, upd, partials);
    count_launch();
    return cudaGetLastError();
}

}  // namespace

// FP64 has one kernel and launch shape: block and variant are accepted and
// make no difference.
cudaError_t launch_dslash_f64(const Geom &g, int recon, const void *gauge, const void *psi, void *res, int isign, int cb,
                              cudaStream_t stream, const SiteRange &range) {
    const DslashArgs<double> a = f64_args(g, recon, gauge, psi, res, cb, range);
    if (g.nd == 4)
        return recon == 18 ? launch_fx<4, 18, 0, 1>(a, isign, nullptr, 0.0, nullptr, stream)
                           : launch_fx<4, 12, 0, 1>(a, isign, nullptr, 0.0, nullptr, stream);
    return recon == 18 ? launch_fx<3, 18, 0, 1>(a, isign, nullptr, 0.0, nullptr, stream)
                       : launch_fx<3, 12, 0, 1>(a, isign, nullptr, 0.0, nullptr, stream);
}

// 4D, 18-real links (the solvers' FP64 links)
cudaError_t launch_dslash_xpay_f64(const Geom &g, const void *gauge, const void *psi, const void *x, double coef,
                                   void *res, double *partials, int isign, int cb, cudaStream_t stream) {
    const DslashArgs<double> a = f64_args(g, 18, gauge, psi, res, cb);
    const double2 *xv = static_cast<const double2 *>(x);
    return partials ? launch_fx<4, 18, 1, 4>(a, isign, xv, coef, partials, stream)
                    : launch_fx<4, 18, 1, 1>(a, isign, xv, coef, nullptr, stream);
}

cudaError_t launch_dslash_cg_update_f64(const Geom &g, const void *gauge, const void *psi, const void *x, double coef,
                                        const double *alpha, void *r, double *partials, int isign, int cb,
                                        cudaStream_t stream) {
    return launch_fx<4, 18, 2, 4>(f64_args(g, 18, gauge, psi, nullptr, cb), isign, static_cast<const double2 *>(x), coef,
                                  partials, stream, {static_cast<double2 *>(r), alpha});
}

}  // namespace gbds
