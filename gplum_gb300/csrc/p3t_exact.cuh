// Correctly rounded FP64 square root, reciprocal and quotient in integer
// arithmetic, for the kernels that the FP64 pipe bounds.
//
// An FP64 instruction of a warp takes 64 cycles on this GPU whatever its
// active lanes, and an SM takes one per 19 cycles from all its warps together;
// the library's sqrt and division cost about ten and six of them (measured in a
// dependent chain: 611 and 367 cycles).  The integer pipe issues an
// instruction per cycle and sub-partition, so the same roundings from 32 x 32
// bit products leave the FP64 pipe to the sums and products that need it.
//
// Method: Newton's iteration in fixed point from the FP32 approximation (whose
// relative error is below 2^-20.5), twice, which leaves the root or reciprocal
// within 2^-59; then the 53-bit floor U and the midpoint U + 1/2: the result is
// U + 1 exactly when the operand is not below the midpoint's square (product).
// That remainder is below 2^63 in the units of its last place, so 64-bit
// wrap-around arithmetic gives its sign exactly.  A midpoint is never the
// exact result: its square (product) has more significant bits than the operand.
// So the results are the IEEE round-to-nearest ones, bit for bit
// (tests/test_exact_arith.py); zeros, subnormals, infinities, NaN, negative
// roots and results near the range's ends take the library's operation.
#pragma once
#include <cstdint>
#include <cstring>

#include <cmath>

#ifdef __CUDACC__
#define P3T_HD __host__ __device__ __forceinline__
#else
#define P3T_HD static inline
#endif

namespace p3t {

P3T_HD uint64_t ex_bits(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}
P3T_HD double ex_double(uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
// bits of the FP32 approximations of 1 / sqrt(m) and 1 / m, m given as bits
P3T_HD uint32_t ex_rsqrt32(uint32_t m) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(m)));
    return __float_as_uint(y);
#else
    float f;
    std::memcpy(&f, &m, 4);
    f = (float)(1.0 / std::sqrt((double)f));
    std::memcpy(&m, &f, 4);
    return m;
#endif
}
P3T_HD uint32_t ex_rcp32(uint32_t m) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(m)));
    return __float_as_uint(y);
#else
    float f;
    std::memcpy(&f, &m, 4);
    f = (float)(1.0 / (double)f);
    std::memcpy(&m, &f, 4);
    return m;
#endif
}
// an approximation of a value in (1/2, 1] as a 32-bit fraction (it may be a
// last place outside)
P3T_HD uint32_t ex_frac32(uint32_t y) {
    const int32_t t = (int32_t)(y - 0x3f000000u);
    return 0x80000000u + ((uint32_t)(t < 0x7fffff ? t : 0x7fffff) << 8);
}

constexpr uint64_t EX_ONE = 1ULL << 52;

// the operands outside the integer forms' range: one copy of the library's operations
#ifdef __CUDACC__
static __device__ __noinline__ double ex_library(double a, double b, int op) { return op ? a / b : sqrt(a); }
#endif
P3T_HD double ex_outside(double a, double b, int op) {
#ifdef __CUDA_ARCH__
    return ex_library(a, b, op);
#else
    return op ? a / b : std::sqrt(a);
#endif
}

// RN(sqrt(x)); `seed`: the FP32 approximation of 1 / sqrt(m) (see sqrt_rn)
P3T_HD uint64_t ex_sqrt_core(uint64_t X, uint32_t seed, uint32_t e) {
    // X: m in [1, 4) with 62 fraction bits, x = m 4^k
    const uint32_t Y = ex_frac32(seed);
    const int32_t Ys = (int32_t)(Y >> 1);
    const uint32_t s0 = (uint32_t)(((X >> 32) * (uint64_t)Y) >> 32);                 // 30 fraction bits
    const int64_t d0 = (int64_t)((X >> 2) - (uint64_t)s0 * s0);                       // m - s0^2, 60 bits
    const uint64_t s1 = ((uint64_t)s0 << 16) + (uint64_t)(((int64_t)(int32_t)(d0 >> 12) * Ys) >> 34);  // 46 bits
    const int64_t d1 = (int64_t)((X << 30) - s1 * s1);                                // m - s1^2, 92 bits
    const uint64_t s2 = (s1 << 16) + (uint64_t)(((int64_t)(int32_t)(d1 >> 24) * Ys) >> 38);  // 62 bits
    const uint64_t U = s2 >> 10, mid = 2 * U + 1;
    const int64_t r = (int64_t)((X << 44) - mid * mid);                               // m - mid^2, 106 bits
    return ((uint64_t)(((e + 1023u) >> 1) - 1u) << 52) + U + (uint64_t)(r >= 0);
}
P3T_HD double sqrt_rn(double x) {
    const uint64_t b = ex_bits(x);
    const uint32_t hi = (uint32_t)(b >> 32);
    if (hi - 0x00100000u >= 0x7fe00000u) return ex_outside(x, 0., 0);
    const uint32_t e = hi >> 20, odd = (e & 1u) ^ 1u;
    const uint64_t X = ((b & (EX_ONE - 1)) | EX_ONE) << (10 + odd);
    const uint32_t m32 = ((127u + odd) << 23) | ((uint32_t)(b >> 29) & 0x7fffffu);
    return ex_double(ex_sqrt_core(X, ex_rsqrt32(m32), e));
}

// 1 / m to 2^-60 with 63 fraction bits: m in [1, 2) as the integer F with 52
P3T_HD uint64_t ex_rcp63(uint64_t F, uint32_t seed) {
    const uint32_t Y = ex_frac32(seed);
    const int32_t Ys = (int32_t)(Y >> 1);
    const uint64_t M = F << 11;
    const uint64_t p = (M >> 32) * (uint64_t)Y + (((M & 0xffffffffULL) * (uint64_t)Y) >> 32);
    const int64_t e0 = (int64_t)((1ULL << 63) - p);                                   // 1 - m y0, 63 bits
    const uint64_t y1 = ((uint64_t)Y << 16) + (uint64_t)(((int64_t)(int32_t)(e0 >> 12) * Ys) >> 34);  // 48 bits
    const int64_t e1 = (int64_t)(0 - F * y1);                                         // 1 - m y1, 100 bits
    return (y1 << 15) + (uint64_t)(((int64_t)(int32_t)(e1 >> 29) * Ys) >> 39);
}
P3T_HD uint64_t ex_rcp_core(uint64_t b, uint32_t seed) {
    const uint64_t F = (b & (EX_ONE - 1)) | EX_ONE;
    const uint32_t e = (uint32_t)(b >> 52) & 0x7ffu;
    const uint64_t U = ex_rcp63(F, seed) >> 10, mid = 2 * U + 1;
    const int64_t r = (int64_t)(0 - F * mid);                                         // 1 - m mid, 106 bits
    return ((b >> 63) << 63) + ((uint64_t)(2044u - e) << 52) + U + (uint64_t)(r >= 0);
}
// RN(1 / x)
P3T_HD double rcp_rn(double x) {
    const uint64_t b = ex_bits(x);
    const uint32_t hi = (uint32_t)(b >> 32) & 0x7fffffffu;
    if (hi - 0x00100000u >= 0x7fb00000u) return ex_outside(1., x, 1);  // biased exponents 1..2043
    const uint32_t m32 = 0x3f800000u | ((uint32_t)(b >> 29) & 0x7fffffu);
    return ex_double(ex_rcp_core(b, ex_rcp32(m32)));
}

P3T_HD uint64_t ex_mulhi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
P3T_HD uint64_t ex_div_core(uint64_t ba, uint64_t bb, uint32_t seed) {
    const uint64_t A = (ba & (EX_ONE - 1)) | EX_ONE, F = (bb & (EX_ONE - 1)) | EX_ONE;
    const uint32_t ea = (uint32_t)(ba >> 52) & 0x7ffu, eb = (uint32_t)(bb >> 52) & 0x7ffu;
    // q = a / b in (1/2, 2): doubled where a < b, so that it lies in [1, 2)
    const uint32_t lt = A < F;
    const uint64_t N = A << lt;
    const uint64_t q = ex_mulhi(N << 10, ex_rcp63(F, seed));                          // 61 fraction bits
    const uint64_t U = q >> 9, mid = 2 * U + 1;
    const int64_t r = (int64_t)((N << 53) - F * mid);                                 // a - b mid, 105 bits
    return ((ba ^ bb) & (1ULL << 63)) + ((uint64_t)(ea - eb + 1022u - lt) << 52) + U + (uint64_t)(r >= 0);
}
// RN(a / b)
P3T_HD double div_rn(double a, double b) {
    const uint64_t ba = ex_bits(a), bb = ex_bits(b);
    const uint32_t ha = (uint32_t)(ba >> 52) & 0x7ffu, hb = (uint32_t)(bb >> 52) & 0x7ffu;
    if (ha - 1u >= 2046u || hb - 1u >= 2046u || ha - hb + 1020u >= 2040u) return ex_outside(a, b, 1);
    const uint32_t m32 = 0x3f800000u | ((uint32_t)(bb >> 29) & 0x7fffffu);
    return ex_double(ex_div_core(ba, bb, ex_rcp32(m32)));
}

}  // namespace p3t
