// Block fixed point: a double as the signed integer pair (n, g),
//   v 2^(27 - e) = n + g 2^-32,   |n| <= 2^28, g the fraction in [-1/2, 1/2),
// against a scale exponent e with |v| < 2^(e + 1): 59 bits below the scale
// where a double's mantissa has 53.  A product of two such numbers is
// n n' + (n g' + g n') 2^-32 in 64-bit integers; only g g' 2^-64 (a quarter of
// a unit at most) is dropped, and sums of products are exact.
//
// Plain integer code for host and device: the conversion is tested on the
// host, the FP64 Dslash (dslash_f64.cu) uses it on the device.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define GBDS_FIX_FN __host__ __device__ __forceinline__
#else
#define GBDS_FIX_FN inline
#endif

namespace gbds {

struct fix2 {
    int32_t n, g;
};

constexpr int kFixUnit = 54;  // a product's unit is 2^(e + e' - 54)

// arithmetic shift right; t above 63 leaves the sign
GBDS_FIX_FN int64_t fix_sar(int64_t v, uint32_t t) {
#ifdef __CUDA_ARCH__
    int64_t r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(t));
    return r;
#else
    return v >> (t > 63 ? 63 : t);
#endif
}

// biased exponent of the double with high word hi
GBDS_FIX_FN uint32_t fix_exponent(uint32_t hi) { return (hi << 1) >> 21; }

// (n, g) of the double (hi, lo) for t = 3 + e - its exponent >= 3.  The
// mantissa with its hidden bit at bit 62, in one's complement when negative
// (one part in 2^62), shifted to the scale and rounded to nearest.  From
// t = 63 on the result is (0, 0) or (0, -1): zeros and what lies below the
// scale's reach vanish.
GBDS_FIX_FN fix2 fix_convert(uint32_t hi, uint32_t lo, uint32_t t) {
    const uint32_t sg = (uint32_t)((int32_t)hi >> 31);
    const uint32_t m = (hi & 0xfffffu) | 0x100000u;
    const uint32_t w1 = ((m << 10) | (lo >> 22)) ^ sg, w0 = (lo << 10) ^ sg;
    const int64_t y = fix_sar((int64_t)(((uint64_t)w1 << 32) | w0), t);
    const uint32_t g = (uint32_t)y;
    return {(int32_t)((uint32_t)(y >> 32) + (g >> 31)), (int32_t)g};
}

// logical shift right; t above 31 gives 0
GBDS_FIX_FN uint32_t fix_shr(uint32_t v, uint32_t t) {
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm("shr.u32 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(t));
    return r;
#else
    return t > 31 ? 0 : v >> t;
#endif
}

// acc += a b, 32 x 32 -> 64 bits
GBDS_FIX_FN void fix_mad(int64_t &acc, int32_t a, int32_t b) {
#ifdef __CUDA_ARCH__
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc) : "r"(a), "r"(b));
#else
    acc += (int64_t)a * b;
#endif
}

// One complex multiply-add (W, X) += u h (DAG: conj(u) h): W the products'
// high parts, X their cross parts in units of 2^-32.
template <bool DAG>
GBDS_FIX_FN void fix_cmad(int64_t (&W)[2], int64_t (&X)[2], fix2 ur, fix2 ui, fix2 hr, fix2 hi) {
    const fix2 um = {-ui.n, ~ui.g};
    // re += ur hr - ui hi, im += ur hi + ui hr (U^+: ui changes sign)
    const fix2 a1 = DAG ? ui : um, a2 = DAG ? um : ui;
    fix_mad(W[0], ur.n, hr.n); fix_mad(X[0], ur.n, hr.g); fix_mad(X[0], ur.g, hr.n);
    fix_mad(W[0], a1.n, hi.n); fix_mad(X[0], a1.n, hi.g); fix_mad(X[0], a1.g, hi.n);
    fix_mad(W[1], ur.n, hi.n); fix_mad(X[1], ur.n, hi.g); fix_mad(X[1], ur.g, hi.n);
    fix_mad(W[1], a2.n, hr.n); fix_mad(X[1], a2.n, hr.g); fix_mad(X[1], a2.g, hr.n);
}
constexpr int64_t kFixHalf = 1ll << 31;  // X starts here: its sum is rounded to nearest

// The sums' error is absolute, a few units: 0.5 for each rounded X, 1/4 (a
// product's g g') and 1/8 (the operands' last bits) at most for each product, rms
// 1 over the 48 products of an output.  But an output's own terms may all be
// small against the scale, which other spins' or the other part's products set,
// and FP64 arithmetic would round to those terms.  So the moduli of the hops'
// partial sums are added up for each output (`seen`, in 2^32 units; no partial sum
// exceeds its terms' moduli), and an output counts as resolved if they reach
// 2^53 units, half of 2^(e + e').  Simulated, rms error over the output's rms in
// FP64 / here: 1.46e-16 / 0.72e-16; with one spin 2^-3 of the others 1.44e-16 /
// 1.15e-16, at 2^-7, where no output of that spin is resolved any more, 1.47e-16 /
// 1.1e-15.  A thread of random fields has an unresolved output once in 4 million
// (a line at 2^54: 6e-5; by the largest partial sum instead of the moduli's sum
// 6e-5 at 2^52).
GBDS_FIX_FN uint32_t fix_modulus_hi(int64_t w) {
    const int32_t hi = (int32_t)(w >> 32);
#ifdef __CUDA_ARCH__
    return (uint32_t)abs(hi);
#else
    return (uint32_t)(hi < 0 ? -hi : hi);
#endif
}
GBDS_FIX_FN bool fix_resolved(uint32_t seen) { return seen >> 21 != 0; }

}  // namespace gbds
