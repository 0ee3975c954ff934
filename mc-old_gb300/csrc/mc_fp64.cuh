// mc_fp64.cuh -- FP64 arithmetic of the history kernels, with as few FP64
// instructions as the result's bits allow.
//
// Measured on GB300 (one kernel per operation, cycles an SM spends per warp
// instruction, whatever the number of active lanes): FP64 add, multiply, FMA
// and compare 19, division 141, square root 143, conversion from or to a
// 64-bit integer 16; an integer instruction is issued four a cycle.  So
// uniforms are assembled from their bits, comparisons are made on bit
// patterns, quantities a comparison alone needs are bounded in FP32, and
// divisors known in advance come with their reciprocal.  Every function here
// returns the bits of the operation sequence it names.
#pragma once

#include "mc_fp64tables.h"
#include "mc_math.cuh"

namespace mc {

// a < b.  Nonnegative finite doubles (and +inf) order as their bit patterns;
// anything else takes the FP64 compare.
__device__ __forceinline__ bool dlt(double a, double b)
{
    const uint32_t ha = (uint32_t)__double2hiint(a), hb = (uint32_t)__double2hiint(b);
    if (max(ha, hb) < 0x7FF00000u) return dbits(a) < dbits(b);
    return a < b;
}

__device__ __forceinline__ bool is_zero(double a) { return (dbits(a) << 1) == 0; }

// The 52 random bits of a draw; u01 of them is (2 v + 1) 2^-53
// (((double)v + 0.5) * 2^-52: both steps are exact).
__device__ __forceinline__ double u01_bits(uint64_t v)
{
    const uint64_t n = 2 * v + 1;
    const int lz = __clzll((long long)n);           // 11..63
    return dfrom(((uint64_t)(1032 - lz) << 52) + (n << (lz - 11)));
}

// 2.0 * u - 1.0 = (2 v + 1 - 2^52) 2^-52, exact as well
__device__ __forceinline__ double mu_bits(uint64_t v)
{
    const long long s = (long long)(2 * v + 1) - (1ll << 52);
    const uint64_t m = (uint64_t)(s < 0 ? -s : s);  // odd
    const int lz = __clzll((long long)m);
    return dfrom((((uint64_t)(1033 - lz) << 52) + (m << (lz - 11))) | (s < 0 ? 0x8000000000000000ull : 0ull));
}

// The FP32 value of a double, its significand cut to 24 bits (relative error
// below 2^-23); 0 below FP32's normal range and +-inf above it.
__device__ __forceinline__ float f32_of(double x)
{
    const uint32_t h = (uint32_t)__double2hiint(x), l = (uint32_t)__double2loint(x);
    const uint32_t a = h & 0x7FFFFFFFu;
    const uint32_t f = __funnelshift_l(l, a - 0x38000000u, 3);
    return __uint_as_float((a < 0x38100000u ? 0u : (a >= 0x47F00000u ? 0x7F800000u : f)) | (h & 0x80000000u));
}

// -log(u) in FP32, relative error below 2e-6 (measured: 4e-7)
static __device__ __noinline__ float neglog_bits(uint64_t v)
{
    if (v >> 51) {                                   // u >= 1/2: from 1 - u = (2 (2^52 - 1 - v) + 1) 2^-53
        return -log1pf(-f32_of(u01_bits(((1ull << 52) - 1) - v)));
    }
    return -__logf(f32_of(u01_bits(v)));
}

static __device__ __noinline__ double fdiv(double a, double b) { return a / b; }
static __device__ __noinline__ double fsqrt(double x) { return dsqrt(x); }

// a / d with 1/d given as hi + lo, for d in recip64's range.  q0 is within a
// unit in the last place of a / d (hi + lo has 2^-104 relative error), so the
// remainder a - d q0 is exact and q0 + r hi rounds to RN(a / d) (Markstein,
// IBM J. Res. Dev. 34, 1990, theorem on the final division step).  Where the
// remainder could be subnormal, or a is 0, not finite or far out of range,
// the plain division is made.
__device__ __forceinline__ double div_by(double a, double d, const Recip64 &r)
{
    const uint32_t e = (uint32_t)(__double2hiint(a) & 0x7FF00000);
    if (r.hi == 0.0 || e < (1023u - 300u) << 20 || e > (1023u + 300u) << 20) return fdiv(a, d);
    const double q = __fma_rn(a, r.hi, __dmul_rn(a, r.lo));
    return __fma_rn(__fma_rn(-d, q, a), r.hi, q);
}

// k ln2 in plog's two parts, for k = -kLnMin .. 1: a product of two uniforms
// is at least 2^-106
constexpr int kLnMin = 108;
struct LnTable {
    struct { double hi, lo; } k[kLnMin + 2];
};
constexpr LnTable make_ln_table()
{
    LnTable t{};
    for (int i = 0; i < kLnMin + 2; ++i) {
        t.k[i].hi = (double)(i - kLnMin) * kLn2Hi;
        t.k[i].lo = (double)(i - kLnMin) * kLn2Lo;
    }
    return t;
}

// plog for 2^-kLnMin <= x < 1 (mc_math.cuh), same bits
__device__ __forceinline__ double plog_unit(double x, const LnTable &T)
{
    const uint64_t b = dbits(x);
    int k = (int)(b >> 52) - 1023;
    uint64_t mb = (b & 0x000FFFFFFFFFFFFFull) | 0x3FF0000000000000ull;
    if (mb > 0x3FF6A09E667F3BCDull) { mb -= 0x0010000000000000ull; k += 1; }   // m > kSqrt2
    const double f = dfrom(mb) - 1.0;
    const double s = fdiv(f, 2.0 + f);
    const double z = s * s;
    double p = 0x1.642c8590b2164p-5;
    p = 0x1.8618618618618p-5 + z * p;
    p = 0x1.af286bca1af28p-5 + z * p;
    p = 0x1.e1e1e1e1e1e1ep-5 + z * p;
    p = 0x1.1111111111111p-4 + z * p;
    p = 0x1.3b13b13b13b14p-4 + z * p;
    p = 0x1.745d1745d1746p-4 + z * p;
    p = 0x1.c71c71c71c71cp-4 + z * p;
    p = 0x1.2492492492492p-3 + z * p;
    p = 0x1.999999999999ap-3 + z * p;
    p = 0x1.5555555555555p-2 + z * p;
    const double two_s = is_zero(s) ? s : dfrom(dbits(s) + 0x0010000000000000ull);   // 2.0 * s
    const double r = two_s + two_s * (z * p);
    return T.k[k + kLnMin].hi + (r + T.k[k + kLnMin].lo);
}

// preduce of x = 2 pi u (or pi/2 u): the quadrant follows from u's bits
// (round-half-up of x 2/pi is (v + 2^49) >> 50, and v >> 51: sampled, and at
// the limits, in tests/fp64_check.cu), and the products n kPio2_i are constants.
__device__ __forceinline__ double reduce_quadrant(double x, int n)
{
    if (n == 0) return x;
    const double p1 = n == 1 ? kPio2_1 : (n == 2 ? 2.0 * kPio2_1 : (n == 3 ? 3.0 * kPio2_1 : 4.0 * kPio2_1));
    const double p2 = n == 1 ? kPio2_2 : (n == 2 ? 2.0 * kPio2_2 : (n == 3 ? 3.0 * kPio2_2 : 4.0 * kPio2_2));
    const double p3 = n == 1 ? kPio2_3 : (n == 2 ? 2.0 * kPio2_3 : (n == 3 ? 3.0 * kPio2_3 : 4.0 * kPio2_3));
    return ((x - p1) - p2) - p3;
}

__device__ __forceinline__ double flip(double x, bool neg) { return dfrom(dbits(x) ^ (neg ? 0x8000000000000000ull : 0ull)); }

// psin and pcos of x = 2 pi u (mc_math.cuh), both from one reduction
__device__ __forceinline__ void psincos_azi(double x, uint64_t v, double &sn, double &cs)
{
    const int n = (int)((v + (1ull << 49)) >> 50);
    const double r = reduce_quadrant(x, n);
    const double s = psin_poly(r), c = pcos_poly(r);
    const int q = n & 3;
    sn = flip((q & 1) ? c : s, q & 2);
    cs = flip((q & 1) ? s : c, q == 1 || q == 2);
}

// pcos of x = pi/2 u: one polynomial with the quadrant's coefficients, as the
// lanes of a warp are in both
__device__ __forceinline__ double pcos_quarter(double x, uint64_t v)
{
    const bool one = (v >> 51) != 0;
    const double r = one ? ((x - kPio2_1) - kPio2_2) - kPio2_3 : x;
    const double z = r * r;
    double p = one ? 0x1.952c77030ad4ap-49 : -0x1.6827863b97d97p-53;
    p = (one ? -0x1.ae7f3e733b81fp-41 : 0x1.ae7f3e733b81fp-45) + z * p;
    p = (one ? 0x1.6124613a86d09p-33 : -0x1.93974a8c07c9dp-37) + z * p;
    p = (one ? -0x1.ae64567f544e4p-26 : 0x1.1eed8eff8d898p-29) + z * p;
    p = (one ? 0x1.71de3a556c734p-19 : -0x1.27e4fb7789f5cp-22) + z * p;
    p = (one ? -0x1.a01a01a01a01ap-13 : 0x1.a01a01a01a01ap-16) + z * p;
    p = (one ? 0x1.1111111111111p-7 : -0x1.6c16c16c16c17p-10) + z * p;
    p = (one ? -0x1.5555555555555p-3 : 0x1.5555555555555p-5) + z * p;
    // quadrant 1: -(r + r (z p)); quadrant 0: 1 - (z/2 - (z z) p)
    const double a = one ? z : z * z;
    const double zp = a * p;
    const double y = (one ? r : 0.5 * z) + (one ? r * zp : -zp);
    return one ? -y : 1.0 - y;
}

}  // namespace mc
