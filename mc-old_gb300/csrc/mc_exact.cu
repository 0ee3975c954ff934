// mc_exact.cu -- exact per-bin tally sums of the FP64 modes, for merging
// disjoint history ranges (several GPUs, several processes) bit for bit.
//
// The reference folds each history's tally into a running FP64 sum
// (Estimator.cpp:339-346): sum += h, squared += h * h.  FP64 replay keeps that
// order, so one run over [0, n) equals the reference bit for bit; but the
// sum of two runs over [0, a) and [a, n) rounds differently from the single
// run, because FP64 addition is not associative.  So beside the running sums
// the FP64 modes accumulate every bin's sum of history totals and sum of
// their (FP64-rounded) squares exactly, as an integer multiple of 2^-1074
// (every double is one).  Integer addition is associative: exact sums of
// disjoint ranges added in any order, then rounded once to the nearest
// double, give what one run over the union gives, bit for bit.
//
// Representation of one exact value: kExactLimbs signed 64-bit limbs,
// value = sum_j limb[j] * 2^(32 j - 1074).  A double's 53-bit significand
// at its binary position lands in three consecutive limbs as 32-bit digits
// (carry-save: a limb absorbs 2^31 such adds before it could overflow), and
// normalising propagates the carries so that limbs 0..kExactLimbs-2 hold
// digits in [0, 2^32) and the last limb holds the signed rest -- one
// representation per value, which is what mc_exact_sums_read returns.
#include <cmath>
#include <cstring>

#include "mc_device.h"
#include "mc_engine.h"

namespace mc {

namespace {

__device__ __forceinline__ void exact_normalize(long long *acc)
{
    for (int j = 0; j < kExactLimbs - 1; ++j) {
        const long long carry = acc[j] >> 32;     // arithmetic: floor division by 2^32
        acc[j] -= carry * 4294967296ll;
        acc[j + 1] += carry;
    }
}

typedef unsigned __int128 u128;

// +-mag 2^(p - 1074) into a bin's limbs as signed 32-bit digits, with 64-bit
// integer atomics (exact, in any order)
__device__ __forceinline__ void exact_add(unsigned long long *limbs, u128 mag, int p, bool neg)
{
    const int j = p >> 5, sh = p & 31;
    const unsigned long long top = sh ? (unsigned long long)(mag >> (128 - sh)) : 0ull;
    mag <<= sh;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const unsigned long long d = i < 4 ? (unsigned long long)(mag >> (32 * i)) & 0xFFFFFFFFull : top;
        if (d) atomicAdd(limbs + j + i, neg ? 0ull - d : d);   // two's complement: signed add
    }
}

constexpr int kExactThreads = 256;
constexpr int kExactValues = 16;   // histories per thread
constexpr uint32_t kExactSlice = (uint32_t)kExactThreads * kExactValues;
// binades below a slice's largest value that its 128-bit accumulators cover:
// 53 + 48 bits and 12 for the 2^12 values of a slice, and the sign
constexpr int kExactWindow = 48;

// Block (bin, slice of histories): the exact sums of the slice's nonzero
// history totals and of their FP64 squares.  Almost every tally keeps its
// histories' totals within a few binades, so each thread adds its values'
// significands as integers in a 128-bit window under the slice's largest
// exponent, the block adds those, and one thread adds the result's digits to
// the bin's limbs; a value below the window goes to the limbs by itself.
// kTree adds the slice's FP64 sums to sum / sq too (plain mode), from the
// same loads.
//
// Bound and measure (GB300): one read of the columns (0.5 GB for 2,000,000
// histories x 31 bins: 75 us at the measured copy rate).  Before, one thread
// per (bin, slice) walked 68 limbs in local memory and a second kernel made
// the tree sums: 3.37 ms together there; now 0.16 ms.
template <bool kTree>
__global__ void __launch_bounds__(kExactThreads) k_fold_exact(const double *__restrict__ hist, uint32_t n, uint64_t ld,
                                                              long long *ex, double *sum, double *sq)
{
    __shared__ int s_max[2];
    __shared__ unsigned long long s_acc[2][kExactThreads / 32][2];
    __shared__ double s_tree[2][kExactThreads / 32];
    const long long bin = blockIdx.x;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint64_t h0 = (uint64_t)blockIdx.y * kExactSlice;
    const double *col = hist + (uint64_t)bin * ld;
    double v[kExactValues];
    bool any = false;
#pragma unroll
    for (int i = 0; i < kExactValues / 2; ++i) {
        const uint64_t h = h0 + 2 * ((uint64_t)i * kExactThreads + t);
        const double2 x = h < n ? *reinterpret_cast<const double2 *>(col + h) : double2{0.0, 0.0};   // zero from n on
        v[2 * i] = x.x;
        v[2 * i + 1] = x.y;
        any = any || ((__double_as_longlong(x.x) | __double_as_longlong(x.y)) << 1) != 0;
    }
    if (t < 2) s_max[t] = -1;
    if (!__syncthreads_or(any)) return;
    if constexpr (kTree) {
        double s = 0.0, q = 0.0;
#pragma unroll
        for (int i = 0; i < kExactValues; ++i)
            if ((__double_as_longlong(v[i]) << 1) != 0) {
                s += v[i];
                q += v[i] * v[i];
            }
        if (__any_sync(0xffffffffu, any))
            for (int o = 16; o > 0; o >>= 1) {
                s += __shfl_down_sync(0xffffffffu, s, o);
                q += __shfl_down_sync(0xffffffffu, q, o);
            }
        if (lane == 0) { s_tree[0][warp] = s; s_tree[1][warp] = q; }
        __syncthreads();
        if (t < 2) {
            double r = 0.0;
            for (int w = 0; w < kExactThreads / 32; ++w) r += s_tree[t][w];
            if (r != 0.0) atomicAdd((t ? sq : sum) + bin, r);
        }
    }
    unsigned long long *limbs = reinterpret_cast<unsigned long long *>(ex + (size_t)bin * 2 * kExactLimbs);
#pragma unroll 1
    for (int which = 0; which < 2; ++which, limbs += kExactLimbs) {
        // largest exponent of the slice; a square below the smallest subnormal
        // adds nothing, and a non-finite value (an overflowed square) has no
        // exact value and is left out
        int pmax = -1;
#pragma unroll
        for (int i = 0; i < kExactValues; ++i) {
            if (which && (__double_as_longlong(v[i]) << 1) != 0) v[i] = v[i] * v[i];
            const unsigned long long b = (unsigned long long)__double_as_longlong(v[i]);
            const int e = (int)((b >> 52) & 0x7FF);
            if (e == 0x7FF) { if (which) v[i] = 0.0; continue; }
            if ((b << 1) != 0) pmax = max(pmax, e ? e - 1 : 0);   // value = m 2^(p - 1074)
        }
        pmax = __reduce_max_sync(0xffffffffu, pmax);
        if (lane == 0 && pmax >= 0) atomicMax(&s_max[which], pmax);
        __syncthreads();
        if (s_max[which] < 0) continue;
        const int base = max(s_max[which] - kExactWindow, 0);
        u128 acc = 0;
#pragma unroll
        for (int i = 0; i < kExactValues; ++i) {
            const unsigned long long b = (unsigned long long)__double_as_longlong(v[i]);
            const int e = (int)((b >> 52) & 0x7FF);
            if ((b << 1) == 0 || e == 0x7FF) continue;
            const unsigned long long m = (b & ((1ull << 52) - 1)) | (e ? 1ull << 52 : 0ull);
            const int p = e ? e - 1 : 0;
            if (p < base) { exact_add(limbs, m, p, b >> 63); continue; }
            const u128 x = (u128)m << (p - base);
            acc = (b >> 63) ? acc - x : acc + x;
        }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long lo = __shfl_down_sync(0xffffffffu, (unsigned long long)acc, o);
            const unsigned long long hi = __shfl_down_sync(0xffffffffu, (unsigned long long)(acc >> 64), o);
            acc += ((u128)hi << 64) | lo;
        }
        if (lane == 0) {
            s_acc[which][warp][0] = (unsigned long long)acc;
            s_acc[which][warp][1] = (unsigned long long)(acc >> 64);
        }
        __syncthreads();
        if (t == 0) {
            acc = 0;
            for (int w = 0; w < kExactThreads / 32; ++w) acc += ((u128)s_acc[which][w][1] << 64) | s_acc[which][w][0];
            const bool neg = (long long)(acc >> 64) < 0;
            exact_add(limbs, neg ? (u128)0 - acc : acc, base, neg);
        }
    }
}

__global__ void k_exact_normalize(long long *ex, long long count)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    long long a[kExactLimbs];
    long long *p = ex + (size_t)i * kExactLimbs;
    for (int j = 0; j < kExactLimbs; ++j) a[j] = p[j];
    exact_normalize(a);
    for (int j = 0; j < kExactLimbs; ++j) p[j] = a[j];
}

}  // namespace

cudaError_t launch_fold_exact(const double *hist, uint32_t n, uint64_t ld, long long nb, long long *ex, double *sum,
                              double *sq, cudaStream_t st)
{
    if (nb <= 0 || n == 0) return cudaSuccess;
    const dim3 grid((unsigned)nb, (n + kExactSlice - 1) / kExactSlice);
    if (sum) k_fold_exact<true><<<grid, kExactThreads, 0, st>>>(hist, n, ld, ex, sum, sq);
    else k_fold_exact<false><<<grid, kExactThreads, 0, st>>>(hist, n, ld, ex, nullptr, nullptr);
    return cudaGetLastError();
}

cudaError_t launch_exact_normalize(long long *ex, long long nb, cudaStream_t st)
{
    if (nb <= 0) return cudaSuccess;
    const long long count = 2 * nb;
    k_exact_normalize<<<(unsigned)((count + 127) / 128), 128, 0, st>>>(ex, count);
    return cudaGetLastError();
}

// Nearest double (ties to even) of one exact value: the limbs are
// normalised on a copy, the sign taken from the top, the magnitude's top 64
// bits rounded to 53 with the lower bits as a sticky bit.  Every value is a
// multiple of 2^-1074, so a magnitude below 2^-1022 is exactly a subnormal.
double exact_round(const int64_t *limbs)
{
    long long a[kExactLimbs];
    std::memcpy(a, limbs, sizeof(a));
    for (int j = 0; j < kExactLimbs - 1; ++j) {
        const long long carry = a[j] >> 32;
        a[j] -= carry * 4294967296ll;
        a[j + 1] += carry;
    }
    const bool neg = a[kExactLimbs - 1] < 0;
    if (neg) {   // magnitude: negate the whole number, then normalise again
        for (int j = 0; j < kExactLimbs; ++j) a[j] = -a[j];
        for (int j = 0; j < kExactLimbs - 1; ++j) {
            const long long carry = a[j] >> 32;
            a[j] -= carry * 4294967296ll;
            a[j + 1] += carry;
        }
    }
    // digits d[0..K-1] in [0, 2^32) except possibly the top one (>= 0)
    int top = kExactLimbs - 1;
    while (top >= 0 && a[top] == 0) --top;
    if (top < 0) return 0.0;
    // the top limb may exceed 32 bits only for magnitudes far above DBL_MAX
    if (top == kExactLimbs - 1 && (unsigned long long)a[top] >= (1ull << 32)) return neg ? -HUGE_VAL : HUGE_VAL;
    const int lz = __builtin_clzll((unsigned long long)a[top]);
    const int msb = 32 * top + (63 - lz);          // bit index of the leading one
    if (msb < 53) {                                 // below 2^-1021: exact (a multiple of 2^-1074, < 2^53 units)
        unsigned long long v = 0;
        for (int j = top; j >= 0; --j) v = (v << 32) | (unsigned long long)a[j];
        const double r = std::ldexp((double)v, -1074);
        return neg ? -r : r;
    }
    // the 64 bits below and including the leading one, and whether anything
    // below them is nonzero
    unsigned long long hi = 0;
    bool sticky = false;
    for (int bit = msb, k = 0; k < 64; ++k, --bit) {
        unsigned long long b = 0;
        if (bit >= 0) b = ((unsigned long long)a[bit >> 5] >> (bit & 31)) & 1ull;
        hi = (hi << 1) | b;
    }
    for (int bit = msb - 64; bit >= 0 && !sticky; --bit)
        if (((unsigned long long)a[bit >> 5] >> (bit & 31)) & 1ull) sticky = true;
    unsigned long long mant = hi >> 11;             // 53 bits
    const unsigned long long rest = hi & 0x7FFull;  // 11 bits below
    const bool up = rest > 0x400ull || (rest == 0x400ull && (sticky || (mant & 1ull)));
    int e = msb - 52 - 1074;                        // value = mant * 2^e
    if (up) {
        ++mant;
        if (mant == (1ull << 53)) { mant >>= 1; ++e; }
    }
    if (e > 1023 - 52) return neg ? -HUGE_VAL : HUGE_VAL;
    const double r = std::ldexp((double)mant, e);
    return neg ? -r : r;
}

}  // namespace mc
