// FP32 instantiations of the fused Dslash kernel (4D/3D x recon 18/12 x isign).
#include "dslash_kernel.cuh"

namespace gbds {
namespace {

template <int ND, int RECON, int EPI = 0>
cudaError_t launch_split(const DslashArgs<float> &a, int isign, cudaStream_t st, const float4 *x = nullptr, float coef = 0.f,
                         const CgUpdate<float> &upd = {}, double *partials = nullptr, const SumHere &here = {}) {
    const dim3 grid((a.g.Vh + kSplitSites - 1) / kSplitSites);
    if (isign > 0) launch_pdl(dslash_split_kernel<ND, RECON, 1, EPI>, grid, 128, st, a, x, coef, upd, partials, here);
    else launch_pdl(dslash_split_kernel<ND, RECON, -1, EPI>, grid, 128, st, a, x, coef, upd, partials, here);
    count_launch();
    return cudaGetLastError();
}

DslashArgs<float> f32_args(const Geom &g, int recon, const void *gauge, const void *psi, void *res, int cb,
                           const SiteRange &range = {}) {
    DslashArgs<float> a;
    a.g = g;
    a.psi = static_cast<const float4 *>(psi);
    a.res = static_cast<float4 *>(res);
    a.gauge = static_cast<const char *>(gauge);
    a.link_block_bytes = (size_t)recon * 4 * g.stride;
    a.pt = 1 - cb;
    a.first = range.first;
    a.end = range.end(g);
    return a;
}

// Part of a lattice, registers capped for 6 CTAs per SM.
template <int ND, int RECON>
cudaError_t launch_range(const DslashArgs<float> &a, int isign, cudaStream_t st) {
    const dim3 grid((a.end - a.first + 127) / 128);
    if (isign > 0) launch_pdl(dslash_kernel<float, ND, RECON, 1, 6, true>, grid, 128, st, a);
    else launch_pdl(dslash_kernel<float, ND, RECON, -1, 6, true>, grid, 128, st, a);
    count_launch();
    return cudaGetLastError();
}

// Four warps a site: the variant after the register caps.
constexpr int kSplitVariant = Variants<float>::n;

}  // namespace

// Block and variant for a lattice, by how many waves its CTAs make on 152 SMs
// (n CTAs of 128 sites; resident: uncapped registers 456, capped for 6 or 7 CTAs
// per SM 912 or 1064, four warps a site 228).  A wave lasts as long as a
// thread's chain of hops, shorter with more registers (more loads in flight)
// and with the chain split, and a last wave that is nearly empty costs a whole
// one.  us a launch in a chain (18 / 12 reals):
//               4 warps a site   uncapped       cap 6          cap 7
//   n = 16       1.7 /  1.7       2.3 /  2.3     3.4 /  3.2     4.5 /  3.4
//   n = 162      3.6 /  3.3       4.3 /  4.5     6.3 /  5.8     8.0 /  5.7
//   n = 256      6.4 /  5.6       4.8 /  5.0     8.5 /  7.8    10.9 /  8.2
//   n = 512     10.1 /  9.2       9.8 /  9.0    10.1 /  9.2    12.7 /  9.3
//   n = 945     17.1 / 15.3      18.3 / 14.4    18.9 / 15.3    16.8 / 12.0
//   n = 1296    23.3 / 21.3      24.5 / 18.2    23.1 / 19.2    29.1 / 20.1
//   n = 2592    44.2 / 39.7      45.7 / 35.1    40.8 / 33.3    48.6 / 34.3
//   n = 4116    68.1 / 61.0      70.5 / 54.3    64.4 / 52.2    70.2 / 50.3
//   n = 8192     131 /  117       135 /  102     123 /  98.1    135 /  95.1
// The cap of 7 makes the 18-real kernel spill, so there it only pays where it
// saves the second of two waves.
void f32_tuning(const Geom &g, int recon, int *block, int *variant) {
    const int n = (g.Vh + 127) / 128;
    constexpr int kUncapped = 0, kCap6 = 1, kCap7 = 2;
    auto waves = [&](int resident) { return (n + resident - 1) / resident; };
    *block = 128;
    if (n <= 228) *variant = kSplitVariant;
    else if (n <= 512) *variant = kUncapped;
    else if (recon == 18) *variant = waves(912) == 2 && waves(1064) == 1 ? kCap7 : kCap6;
    else if (n <= 1064) *variant = kCap7;
    else if (n <= 4 * 456) *variant = kUncapped;
    else *variant = waves(1064) < waves(912) ? kCap7 : kCap6;
    if (*variant == kUncapped) *block = 64;
}

cudaError_t launch_dslash_f32(const Geom &g, int recon, const void *gauge, const void *psi, void *res,
                              int isign, int cb, int block, int variant, cudaStream_t stream, const SiteRange &range) {
    if (range.count >= 0) {
        const DslashArgs<float> a = f32_args(g, recon, gauge, psi, res, cb, range);
        if (g.nd == 4) return recon == 18 ? launch_range<4, 18>(a, isign, stream) : launch_range<4, 12>(a, isign, stream);
        return recon == 18 ? launch_range<3, 18>(a, isign, stream) : launch_range<3, 12>(a, isign, stream);
    }
    if (variant == kSplitVariant) {
        const DslashArgs<float> a = f32_args(g, recon, gauge, psi, res, cb);
        if (g.nd == 4) return recon == 18 ? launch_split<4, 18>(a, isign, stream) : launch_split<4, 12>(a, isign, stream);
        return recon == 18 ? launch_split<3, 18>(a, isign, stream) : launch_split<3, 12>(a, isign, stream);
    }
    return launch_dslash_t<float>(g, recon, gauge, psi, res, isign, cb, block, variant, stream);
}
int dslash_variants(int prec) { return prec == 32 ? Variants<float>::n + 1 : 3; }
// The launches with an epilogue take four warps a site or uncapped registers where
// f32_tuning does (there 64-thread blocks; here 128, a partial each), else registers
// capped for 6 CTAs per SM.  Uncapped with 12-real links and 1065 to 1824 CTAs, us an
// iteration of the FP32-inner solve, against the cap: 20^3x36 (1125) 104 / 108, 24^4
// (1296) 110 / 115, 16^2x32x44 (1408) 124 / 125, 24^3x32 (1728) 141 / 141.
namespace {

template <bool UPD>
cudaError_t launch_epilogue(const Geom &g, int recon, const void *gauge, const void *psi, const void *x, float coef, void *res,
                            double *partials, int isign, int cb, cudaStream_t st, const SumHere &here,
                            const CgUpdate<float> &upd = {}) {
    int block, variant;
    f32_tuning(g, recon, &block, &variant);
    constexpr int EPI = UPD ? 2 : 1;
    if (variant == kSplitVariant) {
        const DslashArgs<float> a = f32_args(g, recon, gauge, psi, res, cb);
        const float4 *xv = static_cast<const float4 *>(x);
        return recon == 18 ? launch_split<4, 18, EPI>(a, isign, st, xv, coef, upd, partials, here)
                           : launch_split<4, 12, EPI>(a, isign, st, xv, coef, upd, partials, here);
    }
    if (variant == 0)
        return launch_dslash_xpay_t<float, UPD, 0, 0>(g, recon, gauge, psi, x, coef, res, partials, isign, cb, st, upd,
                                                      here);
    return launch_dslash_xpay_t<float, UPD>(g, recon, gauge, psi, x, coef, res, partials, isign, cb, st, upd);
}

}  // namespace

int f32_partials(const Geom &g, int recon) {
    int block, variant;
    f32_tuning(g, recon, &block, &variant);
    return variant == kSplitVariant ? (g.Vh + kSplitSites - 1) / kSplitSites : xpay_blocks(g);
}

bool f32_sums_here(const Geom &g, int recon) {
    int block, variant;
    f32_tuning(g, recon, &block, &variant);
    return variant == kSplitVariant || (variant == 0 && xpay_blocks(g) <= 512);
}

cudaError_t launch_dslash_xpay_f32(const Geom &g, int recon, const void *gauge, const void *psi, const void *x,
                                   float coef, void *res, double *partials, int isign, int cb, cudaStream_t stream,
                                   const SumHere &here) {
    return launch_epilogue<false>(g, recon, gauge, psi, x, coef, res, partials, isign, cb, stream, here);
}
cudaError_t launch_dslash_cg_update_f32(const Geom &g, int recon, const void *gauge, const void *psi, const void *x,
                                        float coef, const double *alpha, void *r, double *partials, int isign, int cb,
                                        cudaStream_t stream, const SumHere &here) {
    return launch_epilogue<true>(g, recon, gauge, psi, x, coef, nullptr, partials, isign, cb, stream, here,
                                 {static_cast<float4 *>(r), alpha});
}
}  // namespace gbds
