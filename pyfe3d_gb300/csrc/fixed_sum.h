// Sums of doubles in fixed point relative to the largest term, with integer
// operations only (host and device): the terms are split into limbs, whoever
// holds the terms adds the limbs (on the device the warp's integer reductions),
// and the total is rounded once.
//
// Units are 2^-62 of the power of two at or below the largest term.  A term
// loses less than one unit, towards zero, and terms within 2^10 of the largest
// lose nothing, so n <= FS_TERMS terms are summed to half a unit in the result's
// last place and n 2^-62 of the largest term, whatever their order.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define FS_FN __host__ __device__ __forceinline__
#else
#define FS_FN inline
#endif

namespace fe3d {

constexpr int FS_TERMS = 256;  // terms at most: limbs of 21 bits, 32-bit sums
// biased exponents of the largest term for which no sum of FS_TERMS terms leaves
// the normal range: it is below 2^9 times the power of two at or below that term
constexpr int FS_EMIN = 128, FS_EMAX = 0x7fe - 9;

FS_FN bool fixed_range(int emax) { return (unsigned)(emax - FS_EMIN) <= (unsigned)(FS_EMAX - FS_EMIN); }

struct FixedLimbs {
    uint32_t lo, mid;  // 21 bits each
    int32_t hi;        // signed
};

// m 2^-d, d >= 0; 0 from d = 64 on (the instruction's own rule).
FS_FN uint64_t fixed_shift(uint64_t m, int d) {
#ifdef __CUDA_ARCH__
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(d));
    return r;
#else
    return d < 64 ? m >> d : 0;
#endif
}

// Adds the term with the bits b to f; emax: the largest term's biased exponent,
// in fixed_range (a zero or denormal term then moves out entirely).
FS_FN void fixed_add(FixedLimbs &f, int64_t b, int emax) {
    int64_t m = (int64_t)fixed_shift((uint64_t)((b & 0xfffffffffffffll) | (1ll << 52)) << 10,
                                     emax - ((int)(b >> 52) & 0x7ff));
    if (b < 0) m = -m;
    f.lo += (uint32_t)m & 0x1fffffu;
    f.mid += (uint32_t)(m >> 21) & 0x1fffffu;
    f.hi += (int32_t)(m >> 42);
}

// The bits of the sum of the limbs f, to nearest, ties to even.
FS_FN int64_t fixed_round(const FixedLimbs &f, int emax) {
    const int64_t T = ((int64_t)f.hi << 21) + f.mid + (f.lo >> 21);  // below 2^50
    uint32_t l = f.lo & 0x1fffffu;
    // |total| = t 2^21 + l
    const bool neg = T < 0;
    const uint64_t t = neg ? (uint64_t)(-T) - (l != 0) : (uint64_t)T;
    if (neg) l = (0x200000u - l) & 0x1fffffu;
    // the leading 64 bits of it, what is cut off kept as the last one
    const int s = (t >> 43) != 0 ? 7 : 0;
    const uint64_t a = t << (21 - s) | l >> s | ((l & ((1u << s) - 1u)) != 0);
    if (a == 0) return 0;
#ifdef __CUDA_ARCH__
    const int lz = __clzll((long long)a);
#else
    const int lz = __builtin_clzll(a);
#endif
    uint64_t m = a << lz;                // leading one at bit 63
    const int e = emax - 62 + s + 63 - lz;  // its biased exponent
    const uint64_t r = m & 0x7ffull;
    m >>= 11;
    if (r > 0x400ull || (r == 0x400ull && (m & 1))) m++;  // a carry moves into the exponent
    return (int64_t)((((uint64_t)(e - 1) << 52) + m) | (neg ? 1ull << 63 : 0ull));
}

}  // namespace fe3d
