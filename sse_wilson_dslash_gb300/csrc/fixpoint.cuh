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

// acc += a b, 32 x 32 -> 64 bits
GBDS_FIX_FN void fix_mad(int64_t &acc, int32_t a, int32_t b) {
#ifdef __CUDA_ARCH__
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc) : "r"(a), "r"(b));
#else
    acc += (int64_t)a * b;
#endif
}

}  // namespace gbds
