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

// Powers of 1 / sqrt(x) with one rounding each, within 0.6 units of the last
// place (a root, a quotient and products round once apiece).  One cubic step
// from the FP32 approximation y0: y = y0 (1 + e/2 + 3 e^2/8), e = 1 - m y0^2,
// |e| < 2^-20, leaves 5/16 e^3 < 2^-61; the products keep 62 fraction bits.
struct InvRoots {
    double y1, y3, y4, y5;
};
// m in [1, 4) as X with 62 fraction bits -> 1 / sqrt(m) with 63
P3T_HD uint64_t ex_rsqrt63(uint64_t X, uint32_t seed) {
    const uint64_t Y0 = ex_frac32(seed);
    const int64_t e = (int64_t)((1ULL << 62) - ex_mulhi(X, Y0 * Y0));
    const int64_t eh = (int64_t)(int32_t)(e >> 12);
    const int64_t c = (e >> 1) + ((eh * eh * 3) >> 41);
    const int64_t d = (int64_t)(c >> 32) * (int64_t)Y0 + (int64_t)(((uint64_t)(uint32_t)c * Y0) >> 32);
    return ((Y0 << 30) + (uint64_t)d) << 1;
}
P3T_HD uint32_t ex_clz_high(uint64_t v) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__clz((int)(v >> 32));
#else
    return (uint32_t)__builtin_clzll(v);
#endif
}
// v 2^(s - 62), rounded once; v in [2^57, 2^62]
P3T_HD double ex_pack62(uint64_t v, int32_t s) {
    const uint32_t n = ex_clz_high(v);
    v <<= n;
    return ex_double(((uint64_t)(uint32_t)(1023 - (int32_t)n + s) << 52) + (v >> 11) + ((v >> 10) & 1));
}
// operands outside 2^-380 .. 2^380, zero, infinite or NaN: the library's operations
#ifdef __CUDACC__
static __device__ __noinline__ InvRoots ex_inv_roots_library(double x) {
    const double y = 1.0 / sqrt(x), y2 = y * y;
    return InvRoots{y, y2 * y, y2 * y2, y2 * (y2 * y)};
}
#endif
P3T_HD bool ex_inv_roots_range(double x) { return (uint32_t)(ex_bits(x) >> 52) - 643u < 760u; }
// WITH_HIGH: y4 and y5 as well
template <bool WITH_HIGH>
P3T_HD InvRoots inv_roots_in(double x) {
    const uint64_t b = ex_bits(x);
    const uint32_t e = (uint32_t)(b >> 52), odd = (e & 1u) ^ 1u;
    const uint64_t X = ((b & (EX_ONE - 1)) | EX_ONE) << (10 + odd);
    const uint32_t m32 = ((127u + odd) << 23) | ((uint32_t)(b >> 29) & 0x7fffffu);
    const int32_t k = ((int32_t)(e - odd) - 1023) >> 1;
    const uint64_t Y = ex_rsqrt63(X, ex_rsqrt32(m32));
    const uint64_t y2 = ex_mulhi(Y, Y), y3 = ex_mulhi(y2 << 1, Y);  // 62 fraction bits
    InvRoots r;
    r.y1 = ex_pack62(Y >> 1, -k);
    r.y3 = ex_pack62(y3, -3 * k);
    if (WITH_HIGH) {
        r.y4 = ex_pack62(ex_mulhi(y2 << 1, y2 << 1), -4 * k);
        r.y5 = ex_pack62(ex_mulhi(y2 << 1, y3 << 1), -5 * k);
    } else {
        r.y4 = r.y5 = 0.;
    }
    return r;
}

}  // namespace p3t
