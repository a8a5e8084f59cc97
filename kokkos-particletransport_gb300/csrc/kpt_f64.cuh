// FP64 comparisons, tests and conversions on the integer pipes, and divisions
// by known divisors, for the FP64 kernels: on GB300 one FP64 warp instruction
// (a compare or a conversion too) takes 64 cycles of its SM sub-partition, an
// integer one one or two.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace kpt {
namespace {

__device__ __forceinline__ long long f64_bits(double v) { return __double_as_longlong(v); }

// Monotonic key of a double (signed order of the keys = order of the values;
// -0 sorts just below +0, NaN beyond the infinities).
__host__ __device__ __forceinline__ long long f64_key(long long bits) {
    return bits ^ ((bits >> 63) & 0x7fffffffffffffffll);
}

__device__ __forceinline__ bool f64_finite(double v) {
    return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000;
}

// a < b for b > 0 finite and a not NaN (a negative double is a negative
// integer, non-negative doubles order like their bit patterns)
__device__ __forceinline__ bool f64_below(double a, double b) {
    return f64_bits(a) < f64_bits(b);
}

__device__ __forceinline__ bool f64_positive(double v) {  // v > 0, v not NaN
    return f64_bits(v) > 0;
}

__device__ __forceinline__ bool f64_zero(double v) { return (f64_bits(v) << 1) == 0; }

__device__ __forceinline__ bool f64_nan(double v) {
    return (f64_bits(v) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}

__device__ __forceinline__ bool f64_negative(double v) {  // v < 0, v not NaN
    return f64_bits(v) < 0 && !f64_zero(v);
}

// clamp_mu for a bound m > 0
__device__ __forceinline__ double f64_clamp(double v, double m) {
    return !f64_nan(v) && (f64_bits(v) & 0x7fffffffffffffffll) > f64_bits(m)
               ? (f64_bits(v) < 0 ? -m : m)
               : v;
}

// |v| in [2^-400, 2^400] (0 excluded)
__device__ __forceinline__ bool f64_moderate(double v) {
    const unsigned e = (static_cast<unsigned>(__double2hiint(v)) >> 20) & 0x7ffu;
    return e - (1023u - 400u) <= 800u;
}

// The double of an integer 0 <= k < 2^31.
__device__ __forceinline__ double f64_of_int(int k) {
    const int lz = __clz(k);
    const unsigned m = lz >= 31 ? 0u : static_cast<unsigned>(k) << (lz + 1);  // leading 1 dropped
    const unsigned hi = (static_cast<unsigned>(1023 + 31 - lz) << 20) | (m >> 12);
    return k == 0 ? 0.0 : __hiloint2double(static_cast<int>(hi), static_cast<int>(m << 20));
}

// floor(v) of -1 <= v < 2^31 from the bits of its significand; false for any
// other v.
__device__ __forceinline__ bool f64_floor(double v, int& out) {
    const int hi = __double2hiint(v);
    if (hi < 0) {
        out = f64_zero(v) ? 0 : -1;
        return f64_key(f64_bits(v)) >= f64_key(f64_bits(-1.0));
    }
    const int e = (hi >> 20) - 1023;
    const unsigned long long m =
        (static_cast<unsigned long long>(f64_bits(v)) & 0x000fffffffffffffull) |
        0x0010000000000000ull;
    out = e < 0 ? 0 : static_cast<int>(m >> (52 - (e > 30 ? 30 : e)));
    return e <= 30;
}

// u in [0, 1) with 53 random bits, as u01_f64: n 2^-53 for the 53-bit n,
// exact, so the conversion and the scaling are a normalisation.
__device__ __forceinline__ double u01_f64_int(uint32_t lo, uint32_t hi) {
    const unsigned long long n =
        ((static_cast<unsigned long long>(hi) << 32) | lo) >> 11;
    const int lz = __clzll(static_cast<long long>(n));  // >= 11
    const unsigned long long m = (n << (lz - 11)) & 0x000fffffffffffffull;
    const unsigned long long e = static_cast<unsigned long long>(1022 - (lz - 11));
    return n == 0 ? 0.0 : __longlong_as_double(static_cast<long long>((e << 52) | m));
}

// a / b for a divisor whose rounded reciprocal r = RN(1/b) is at hand:
// q = RN(a r), one exact remainder, one correction (Markstein's theorem: the
// result is the correctly rounded quotient).  Operands near the ends of the
// exponent range, where the remainder may not be exact, divide.
__device__ __forceinline__ double div_known(double a, double b, double r) {
    if (f64_moderate(a) && f64_moderate(b)) {
        const double q = __dmul_rn(a, r);
        return __fma_rn(__fma_rn(-q, b, a), r, q);
    }
    return f64_zero(a) && f64_moderate(b) ? __dmul_rn(a, r) : __ddiv_rn(a, b);
}

}  // namespace
}  // namespace kpt
