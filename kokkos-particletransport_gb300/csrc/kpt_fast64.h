/* FP64 reciprocal, roots, logarithm and sine/cosine for the library solver's
 * FP64 step, built around the cost of FP64 on GB300: one FP64 warp instruction
 * takes 64 cycles of its SM sub-partition, an FP32 seed or an integer
 * operation one or two.
 *
 * Reciprocal and roots start from the FP32 hardware approximations (relative
 * error below 2^-21 with the operand's truncation to FP32) and take one
 * higher-order Newton-Householder step in FP64: with e the residual of the
 * seed, 1/x = r (1 + e + e^2), x^(-1/2) = y (1 + e/2 + 3 e^2/8), x^(1/3) =
 * y (1 + e/3 + 2 e^2/9), each cut below 2^-60.  The logarithm is the atanh
 * series ln m = 2 s (1 + z/3 + z^2/5 + ...), s = (m - 1)/(m + 1), z = s^2, on
 * m in [sqrt(1/2), sqrt 2) (Taylor terms to z^9; the rest below 2^-55); sine
 * and cosine of 2 pi u are their Taylor polynomials on the quarter turn around
 * the nearest multiple of 1/4, which the fixed-point draw gives exactly.
 *
 * Errors: at most 1.5 ulp each (2 ulp for the logarithm; sine and cosine 0.75
 * ulp of 1), tested against extended precision on the host and, with the
 * hardware's seeds, on the device; measured there 0.50 (rcp, cbrt), 0.75
 * (sqrt), 0.99 (rsqrt) and 0.87 (log).  The divisions and roots they stand for
 * were correctly rounded, several to a quantity, with the wraps and divisions of
 * a coordinate between them; the state after the steps is no further from its
 * exact value than with those (300 000 particles, 40 steps: 4.6e-16 with either;
 * nine other sizes of 1 000 to 450 000 particles, 4 to 55 steps: 3e-16 to 2e-15,
 * 2e-15 to 1e-13).  FP64 instructions: 3 (rcp), 5 (sqrt, rsqrt), 9 (cbrt), 23
 * (log), 20 (sine and cosine) against 6, 9, 14, 18, 33 and 27 for CUDA's
 * functions.
 *
 * Operands outside [2^-100, 2^100] go through the C library's functions.
 * Host builds (the tests) seed with FP32 divisions and roots instead.
 */
#ifndef KPT_FAST64_H
#define KPT_FAST64_H

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define KPT_F64_FN __host__ __device__ static __forceinline__
#else
#define KPT_F64_FN static inline
#endif

KPT_F64_FN uint64_t kpt_f64_to_bits(double v) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t u;
    memcpy(&u, &v, sizeof(u));
    return u;
#endif
}

KPT_F64_FN double kpt_f64_from_bits(uint64_t u) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double v;
    memcpy(&v, &u, sizeof(v));
    return v;
#endif
}

/* 2^-100 <= v < 2^100 (v positive) */
KPT_F64_FN int kpt_f64_seedable(double v) {
    const uint32_t e = (uint32_t)(kpt_f64_to_bits(v) >> 52); /* sign included: negative is huge */
    return e - (1023u - 100u) < 200u;
}

/* the FP32 value below a seedable v, from its bits */
KPT_F64_FN float kpt_f64_seed(double v) {
    const uint64_t u = kpt_f64_to_bits(v);
    const uint32_t f = (uint32_t)((u - ((uint64_t)896 << 52)) >> 29);
#if defined(__CUDA_ARCH__)
    return __uint_as_float(f);
#else
    float r;
    memcpy(&r, &f, sizeof(r));
    return r;
#endif
}

/* a positive normal float as a double, from its bits */
KPT_F64_FN double kpt_f64_widen(float f) {
#if defined(__CUDA_ARCH__)
    const uint32_t u = __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, sizeof(u));
#endif
    return kpt_f64_from_bits(((uint64_t)u << 29) + ((uint64_t)896 << 52));
}

KPT_F64_FN float kpt_seed_rcp(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / x;
#endif
}

KPT_F64_FN float kpt_seed_rsqrt(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / sqrtf(x);
#endif
}

KPT_F64_FN float kpt_seed_cbrt(float x) {
#if defined(__CUDA_ARCH__)
    float l, r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(l * (1.0f / 3.0f)));
    return r;
#else
    return cbrtf(x);
#endif
}

/* 1 / x for x > 0 (other x: the division) */
KPT_F64_FN double kpt_rcp(double x) {
    if (!kpt_f64_seedable(x)) return 1.0 / x;
    const double r = kpt_f64_widen(kpt_seed_rcp(kpt_f64_seed(x)));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

/* x^(-1/2) for x > 0 */
KPT_F64_FN double kpt_rsqrt(double x) {
    if (!kpt_f64_seedable(x)) return 1.0 / sqrt(x);
    const double y = kpt_f64_widen(kpt_seed_rsqrt(kpt_f64_seed(x)));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y, e * fma(e, 0.375, 0.5), y);
}

/* x^(1/2) */
KPT_F64_FN double kpt_sqrt(double x) {
    if (!kpt_f64_seedable(x)) return sqrt(x);
    const double y = kpt_f64_widen(kpt_seed_rsqrt(kpt_f64_seed(x)));
    const double t = x * y;
    const double e = fma(-t, y, 1.0);
    return fma(t, e * fma(e, 0.375, 0.5), t);
}

/* x^(1/3).  x = m 2^(3k) with m in [1, 8): the seed's logarithm stays below 3,
 * where FP32 holds it to 2^-22; of 2^100 it would keep 2^-18. */
KPT_F64_FN double kpt_cbrt(double x) {
    if (!kpt_f64_seedable(x)) return cbrt(x);
    const uint64_t bits = kpt_f64_to_bits(x);
    const int k = ((int)(bits >> 52) - (1023 - 102)) / 3 - 34; /* floor(exponent / 3) */
    const double m = kpt_f64_from_bits(bits - ((uint64_t)(int64_t)(3 * k) << 52));
    const float mf = kpt_f64_seed(m);
    const double y = kpt_f64_widen(kpt_seed_cbrt(mf));
    const double d = fma(-(y * y), y, m); /* y y exact: y has 24 bits */
    const double r0 = kpt_f64_widen(kpt_seed_rcp(mf));
    const double r = fma(r0, fma(-m, r0, 1.0), r0);
    const double e = d * r;
    const double root = fma(y, e * fma(e, 2.0 / 9.0, 1.0 / 3.0), y);
    return kpt_f64_from_bits(kpt_f64_to_bits(root) + ((uint64_t)(int64_t)k << 52));
}

/* ln u for a normal u in (0, 1] */
KPT_F64_FN double kpt_log(double u) {
    const uint64_t bits = kpt_f64_to_bits(u);
    int e = (int)(bits >> 52) - 1023;
    uint64_t mb = (bits & 0x000fffffffffffffULL) | 0x3ff0000000000000ULL;
    if (mb > 0x3ff6a09e667f3bcdULL) { /* sqrt 2 */
        mb -= 0x0010000000000000ULL;
        e += 1;
    }
    const double m = kpt_f64_from_bits(mb);
    const double f = m - 1.0; /* exact */
    const double s = f * kpt_rcp(2.0 + f);
    const double z = s * s;
    double p = 0x1.af286bca1af28p-4;        /* 2/19 */
    p = fma(p, z, 0x1.e1e1e1e1e1e1ep-4);    /* 2/17 */
    p = fma(p, z, 0x1.1111111111111p-3);    /* 2/15 */
    p = fma(p, z, 0x1.3b13b13b13b14p-3);    /* 2/13 */
    p = fma(p, z, 0x1.745d1745d1746p-3);    /* 2/11 */
    p = fma(p, z, 0x1.c71c71c71c71cp-3);    /* 2/9 */
    p = fma(p, z, 0x1.2492492492492p-2);    /* 2/7 */
    p = fma(p, z, 0x1.999999999999ap-2);    /* 2/5 */
    p = fma(p, z, 0x1.5555555555555p-1);    /* 2/3 */
    /* ln(1 + f) = f - (f^2/2 - s (f^2/2 + z P(z))): the leading term is exact,
     * so the rounding of s only touches the small ones (fdlibm's arrangement) */
    const double h = 0.5 * f * f;
    const double w = fma(z, p, h);
    if (e == 0) return f - fma(-s, w, h);
    const int a = e < 0 ? -e : e; /* 1 .. 1022 */
#if defined(__CUDA_ARCH__)
    const int lz = __clz(a);
#else
    const int lz = __builtin_clz((unsigned)a);
#endif
    const double ed = kpt_f64_from_bits(((uint64_t)(e < 0 ? 1u : 0u) << 63) |
                                        ((uint64_t)(1023 + 31 - lz) << 52) |
                                        (((uint64_t)((uint32_t)a << lz) << 21) &
                                         0x000fffffffffffffULL));
    /* ln 2 = head (42 bits, e head exact) + tail */
    const double tail = fma(s, w, ed * 0x1.ef35793c76730p-45);
    return fma(ed, 0x1.62e42fefa3800p-1, f - (h - tail));
}

/* sin and cos of 2 pi n 2^-53 for a 53-bit draw n */
KPT_F64_FN void kpt_sincos_turn(uint64_t n, double* sine, double* cosine) {
    const uint64_t quarter = (n + ((uint64_t)1 << 50)) >> 51; /* nearest multiple of 1/4 */
    const int64_t rest = (int64_t)(n - (quarter << 51));      /* |rest| <= 2^50 */
    const uint64_t mag = (uint64_t)(rest < 0 ? -rest : rest);
    double f = 0.0; /* rest 2^-53, exact */
    if (mag != 0) {
#if defined(__CUDA_ARCH__)
        const int lz = __clzll((long long)mag);
#else
        const int lz = __builtin_clzll(mag);
#endif
        f = kpt_f64_from_bits(((uint64_t)(rest < 0 ? 1u : 0u) << 63) |
                              ((uint64_t)(1023 + 63 - lz - 53) << 52) |
                              ((mag << (lz - 11)) & 0x000fffffffffffffULL));
    }
    const double t = f * f;
    double s = 0x1.aaec32af93359p-4;
    s = fma(s, t, -0x1.6fadb9f155744p-1);
    s = fma(s, t, 0x1.e8f434d018d63p+1);
    s = fma(s, t, -0x1.e3074fde8871fp+3);
    s = fma(s, t, 0x1.50783487ee782p+5);
    s = fma(s, t, -0x1.32d2cce62bd86p+6);
    s = fma(s, t, 0x1.466bc6775aae2p+6);
    s = fma(s, t, -0x1.4abbce625be53p+5);
    s = fma(f * t, s, 0x1.921fb54442d18p+2 * f);
    double c = 0x1.20c62c2f2d7f5p-2;
    c = fma(c, t, -0x1.b6e24f44b128fp+0);
    c = fma(c, t, 0x1.f9d38a3763cc3p+2);
    c = fma(c, t, -0x1.a6d1f2a204a8cp+4);
    c = fma(c, t, 0x1.e1f506891babbp+5);
    c = fma(c, t, -0x1.55d3c7e3cbffap+6);
    c = fma(c, t, 0x1.03c1f081b5ac4p+6);
    c = fma(c, t, -0x1.3bd3cc9be45dep+4);
    c = fma(c, t, 1.0);
    const double a = (quarter & 1u) ? c : s;
    const double b = (quarter & 1u) ? s : c;
    const uint64_t sign = (uint64_t)1 << 63;
    *sine = kpt_f64_from_bits(kpt_f64_to_bits(a) ^ ((quarter & 2u) ? sign : 0));
    *cosine = kpt_f64_from_bits(kpt_f64_to_bits(b) ^ (((quarter + 1u) & 2u) ? sign : 0));
}

#endif /* KPT_FAST64_H */
