// a / b for the scalars of the resident PCG iteration (team_pcg.cu), where the
// division with its comparison takes 830 cycles of a chain that every block waits
// for.  Newton's iteration for the reciprocal and one correction of the quotient by
// its residual (P. W. Markstein, Computation of elementary functions on the IBM RISC
// System/6000 processor, IBM J. Res. Dev. 34, 1990).
#pragma once
#include <cuda_runtime.h>

namespace fe3d {

__device__ __forceinline__ int exponent_of(double v) { return (int)((unsigned)__double2hiint(v) >> 20 & 0x7ffu); }
__device__ __forceinline__ bool bits_zero(double v) { return (__double_as_longlong(v) << 1) == 0; }

// Divisors away from the ends of the range; the others (0, denormals,
// infinities and NaN among them) are left to the division.
__device__ __forceinline__ bool quotient_range(double b) { return exponent_of(b) > 64 && exponent_of(b) < 1984; }

// a / b, 0 where b is 0.
__device__ __noinline__ double plain_quotient(double a, double b) { return b != 0. ? a / b : 0.; }

// a / b from a reciprocal y of b (quotient_range) with the relative error d: q = a y
// is off by d, its residual a - q b is known to 53 bits, and the corrected quotient
// is off by d^2 and half a unit in its last place, as long as it and the residual
// are normal numbers (|a| from 2^-900 on).  Infinite where a y is.
__device__ __forceinline__ double quotient_by(double a, double b, double y) {
    const double q = a * y, c = fma(fma(-q, b, a), y, q);
    return exponent_of(c) < 0x7ff ? c : q;
}

// a / b, 0 where b is 0: the hardware's approximate reciprocal (d below 2^-19) and
// one Newton step (d below 2^-37), half a unit and 2^-20 units in the last place.
__device__ __forceinline__ double quotient(double a, double b) {
    if (!quotient_range(b)) return plain_quotient(a, b);
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return quotient_by(a, b, fma(fma(-b, y, 1.), y, y));
}

}  // namespace fe3d
