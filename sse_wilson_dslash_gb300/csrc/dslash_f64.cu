// The FP64 Dslash on the integer pipes (block fixed point, fixpoint.cuh).
//
// GB300 issues 2 FP64 operations a clock and SM.  The operator needs 816 a
// site, so in FP64 arithmetic it ran at 0.16 of the HBM roofline with the FP64
// pipe 92 % busy (24^3x48 0.493 ms, 32^3x64 1.477 ms).  32 x 32 -> 64-bit
// integer multiply-adds issue at about 22 a clock and SM, and three of them
// make one multiply-add of two 59-bit fixed-point numbers, with exact sums.
// Here only the projection (96 additions a site) and the final conversion
// (48) stay in FP64; the colour multiply and the accumulation run on
// integers: 24^3x48 0.179 ms, 32^3x64 0.552 ms (24^3x48 with 12-real links 0.299).
// Bound by integer issue (ALU 57 %, IMAD pipe 49 %, FP64 pipe 44 % busy, 465
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
// + link exponent); when it grows, the sums are shifted.  So their error, a few
// units of 2^-54 of the largest product of the colour, is absolute, and an output
// whose own terms are all small beside it (a small spin, the smaller of the real
// and imaginary part) would keep fewer bits than in FP64 arithmetic.  The moduli
// of the hops' sums are therefore added up for each output (12 instructions a
// hop, 24^3x48 174.7 -> 179.3 us), and the outputs that stay below half of the scale
// (fix_resolved), with operands beyond the exponents the integers cover all of them
// (2^177 and up, infinities, NaN, or every product below 2^-646), are formed in FP64
// at the end of the kernel, site by site, from the half spinors that they take.
// us at 24^3x48, against the kernel in FP64 arithmetic's 493 whatever the field:
// random fields 179, unit links 184, one spin 2^-3 of the others 290, 2^-20 491; a
// source of one spin 258, of one spin and colour 293, zero 234.
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
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"  // see ld_once
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

// acc += code * w for one complex, code 0: +1, 1: -1, 2: +i, 3: -i; m: the
// moduli's high words of w, added up in seen
template <int CODE>
__device__ __forceinline__ void fx_acc(int64_t (&acc)[2], uint32_t (&seen)[2], const int64_t (&w)[2], const uint32_t (&m)[2]) {
    if constexpr (CODE == 0) { acc[0] += w[0]; acc[1] += w[1]; }
    else if constexpr (CODE == 1) { acc[0] -= w[0]; acc[1] -= w[1]; }
    else if constexpr (CODE == 2) { acc[0] -= w[1]; acc[1] += w[0]; }
    else { acc[0] += w[1]; acc[1] -= w[0]; }
    seen[0] += m[CODE >> 1];
    seen[1] += m[1 - (CODE >> 1)];
}

// What a thread (colour c of one site) keeps over its hops.
struct FxSum {
    int64_t acc[4][2];    // the four output spins, in units of 2^(e - 2 * 1023 - kFixUnit)
    uint32_t seen[4][2];  // the hops' moduli (fix_resolved)
    uint32_t e;           // the two operands' biased exponents at the scale of the sums
    uint32_t top;         // the largest biased exponent of any operand
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
        et = max(et, eu + eh[j]);
    }
    if (et > S.e) {
        const uint32_t d = et - S.e;
#pragma unroll
        for (int sp = 0; sp < 4; sp++)
#pragma unroll
            for (int p = 0; p < 2; p++) {
                S.acc[sp][p] = fix_sar(S.acc[sp][p], d);
                S.seen[sp][p] = fix_shr(S.seen[sp][p], d);
            }
        S.e = et;
    }
    int64_t W[2][2], X[2][2];
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
        for (int p = 0; p < 2; p++) {
            W[k][p] = 0;
            X[k][p] = kFixHalf;
        }
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const uint32_t t0 = S.e - eh[j] + 3;
        const fix2 ur = to_fix(ud[j].x, t0 - ex[j][0]), ui = to_fix(ud[j].y, t0 - ex[j][1]);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int4 q = sm.h[grp][buf][k][j][lane];
            fix_cmad<DAG>(W[k], X[k], ur, ui, {q.x, q.y}, {q.z, q.w});
        }
    }
    uint32_t m[2][2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
#pragma unroll
        for (int p = 0; p < 2; p++) {
            W[k][p] += X[k][p] >> 32;
            m[k][p] = fix_modulus_hi(W[k][p]);
        }
        fx_acc<0>(S.acc[k], S.seen[k], W[k], m[k]);
    }
    fx_acc<P::b2 ^ f>(S.acc[2], S.seen[2], W[P::k2], m[P::k2]);
    fx_acc<P::b3 ^ f>(S.acc[3], S.seen[3], W[P::k3], m[P::k3]);
}

// Whether the real or the imaginary part is other than +-0.
__device__ __forceinline__ bool nonzero(double2 v) {
    return ((hi_word(v.x) | hi_word(v.y)) << 1 | (uint32_t)__double2loint(v.x) | (uint32_t)__double2loint(v.y)) != 0;
}

// Proj's coefficients of half spinor k by direction, two bits each; a lower
// spin's is the conjugate of the one that the half spinor took that spin with.
template <int K>
constexpr uint32_t proj_codes() {
    return K == 0 ? Proj<0>::a0 | Proj<1>::a0 << 2 | Proj<2>::a0 << 4 | Proj<3>::a0 << 6
                  : Proj<0>::a1 | Proj<1>::a1 << 2 | Proj<2>::a1 << 4 | Proj<3>::a1 << 6;
}

// v with its sign bit changed by s (0 or 2^31)
__device__ __forceinline__ double turn_sign(double v, uint32_t s) {
    return __hiloint2double((int)(hi_word(v) ^ s), __double2loint(v));
}

// Half spinor K of one hop in FP64, colour c: w = (row c of U or U^+) h, added to
// output spin K and to the lower spin of the pair where they are in `open`.  special: an operand is
// infinite or NaN; else products with a factor 0 are left out (diluted sources,
// sites without neighbours).
template <int K, int RECON>
__device__ __forceinline__ void fx_plain_half(const DslashArgs<double> &a, int c, int nbr, const double2 *U, bool dag, int mu,
                                              int flip, uint32_t open, bool special, cx<double> (&p)[4]) {
    const bool third = (mu < 2) == (K == 0);  // the lower spin is spin 3
    const double2 *own = a.psi + (size_t)(K * 3) * a.g.stride + nbr, *low = a.psi + (size_t)(third ? 9 : 6) * a.g.stride + nbr;
    double2 q[3], t[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        q[j] = __ldg(own + (size_t)j * a.g.stride);
        t[j] = __ldg(low + (size_t)j * a.g.stride);
    }
    bool used[3];
#pragma unroll
    for (int j = 0; j < 3; j++) used[j] = special || nonzero(q[j]) || nonzero(t[j]);
    if (!(used[0] || used[1] || used[2])) return;
    const auto ld = [&](int i) { return __ldg(U + (size_t)i * a.g.stride); };
    double2 u[3];
    if (dag) link_row<RECON, true>(ld, c, u);
    else link_row<RECON, false>(ld, c, u);
    const uint32_t code = (proj_codes<K>() >> (2 * mu) & 3) ^ flip;
    const bool turned = code & 2;  // +-i
    const uint32_t sx = (code ^ code >> 1) << 31, sy = code << 31;  // set for codes 1 and 2, 1 and 3
    cx<double> w = {};
#pragma unroll
    for (int j = 0; j < 3; j++) {
        if (!used[j] || !(special || nonzero(u[j]))) continue;
        const double hr = q[j].x + turn_sign(turned ? t[j].y : t[j].x, sx);
        const double hi = q[j].y + turn_sign(turned ? t[j].x : t[j].y, sy);
        const double mr = u[j].x, mi = dag ? -u[j].y : u[j].y;
        w.r = fma(-mi, hi, fma(mr, hr, w.r));
        w.i = fma(mi, hr, fma(mr, hi, w.i));
    }
    if (open & 3u << (2 * K)) p[K] = cadd(p[K], w);
    if (!(open & (third ? 0xc0 : 0x30))) return;
    // conj(code) w
    const cx<double> l = turned ? cx<double>{turn_sign(w.i, ~sx & 1u << 31), turn_sign(w.r, ~sy & 1u << 31)}
                                : cx<double>{turn_sign(w.r, sx), turn_sign(w.i, sy)};
    if (third) p[3] = cadd(p[3], l);
    else p[2] = cadd(p[2], l);
}

// The outputs of colour c of which a part is marked in `open` (bit 2 s + part of
// spin s), in FP64, from the half spinors that they take.
template <int ND, int RECON, int ISIGN>
__device__ __forceinline__ void fx_plain(const DslashArgs<double> &a, int c, int h, const Nbr &n, uint32_t open, bool special,
                                         cx<double> (&p)[4]) {
#pragma unroll 1
    for (int hop = 0; hop < 2 * ND; hop++) {
        const int mu = hop >> 1;
        const bool bwd = hop & 1;
        // directions 0 and 1 pair spins 0, 3 and 1, 2; directions 2 and 3 spins 0, 2 and 1, 3
        const uint32_t half0 = mu < 2 ? 0xc3 : 0x33;
        const int f = mu == 0 ? n.f[0] : mu == 1 ? n.f[1] : mu == 2 ? n.f[2] : n.f[3];
        const int b = mu == 0 ? n.b[0] : mu == 1 ? n.b[1] : mu == 2 ? n.b[2] : n.b[3];
        const int nbr = bwd ? b : f, lp = bwd ? 1 - a.pt : a.pt;
        const double2 *U =
            reinterpret_cast<const double2 *>(a.gauge + (size_t)(lp * ND + mu) * a.link_block_bytes) + (bwd ? b : h);
        const int flip = bwd == (ISIGN > 0) ? 1 : 0;
        if (open & half0) fx_plain_half<0, RECON>(a, c, nbr, U, bwd, mu, flip, open, special, p);
        if (open & ~half0) fx_plain_half<1, RECON>(a, c, nbr, U, bwd, mu, flip, open, special, p);
    }
}

template <int ND, int RECON, int ISIGN, int MU, int GROUPS>
__device__ __forceinline__ void fx_dir(const DslashArgs<double> &a, const FxThread &th, int h, const Nbr &n,
                                       FxShared<GROUPS> &sm, FxSum &S) {
    fx_hop<MU, ISIGN, false, ND, RECON>(a, th, n.f[MU], h, a.pt, sm, S);
    fx_hop<MU, -ISIGN, true, ND, RECON>(a, th, n.b[MU], n.b[MU], 1 - a.pt, sm, S);
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
    for (int s = 0; s < 4; s++) {
        S.acc[s][0] = S.acc[s][1] = 0;
        S.seen[s][0] = S.seen[s][1] = 0;
    }
    S.e = S.top = 0;
    fx_dir<ND, RECON, ISIGN, 0>(a, th, h, n, sm, S);
    fx_dir<ND, RECON, ISIGN, 1>(a, th, h, n, sm, S);
    fx_dir<ND, RECON, ISIGN, 2>(a, th, h, n, sm, S);
    if constexpr (ND == 4) fx_dir<ND, RECON, ISIGN, 3>(a, th, h, n, sm, S);
    double nrm = 0;
    if (th.act) {
        cx<double> r[4] = {};
        uint32_t open = 0xff;  // outputs that the sums do not resolve: in FP64
        if (S.top <= kFxTop && S.e >= kFxLeast) {
            open = 0;
            const double sc = __hiloint2double((int)((S.e - (2046 + kFixUnit - 1023)) << 20), 0);
#pragma unroll
            for (int sp = 0; sp < 4; sp++) {
                r[sp] = {(double)S.acc[sp][0] * sc, (double)S.acc[sp][1] * sc};
                open |= fix_resolved(S.seen[sp][0]) ? 0 : 1u << (2 * sp);
                open |= fix_resolved(S.seen[sp][1]) ? 0 : 2u << (2 * sp);
            }
        }
        if (open) {
            cx<double> p[4] = {};
            fx_plain<ND, RECON, ISIGN>(a, th.c, h, n, open, S.top >= 2047, p);
#pragma unroll
            for (int sp = 0; sp < 4; sp++) {
                if (open >> (2 * sp) & 1) r[sp].r = p[sp].r;
                if (open >> (2 * sp) & 2) r[sp].i = p[sp].i;
            }
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
