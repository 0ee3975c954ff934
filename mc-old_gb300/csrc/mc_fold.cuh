// mc_fold.cuh -- the ordered history fold of FP64 replay, many histories at once.
//
// Estimator::end_history (Estimator.cpp:339-346) adds one history after the
// other to a running FP64 sum, and replay must give that sum's bits.  Taken
// literally it is one serial chain per bin: every addition waits for the one
// before it (64 cycles on this chip, and the load in front of it), while all
// but one thread per bin idle.  It is not serial arithmetic, though.  While
// the running sum s keeps its binade, s = k u with u its unit in the last
// place and 2^52 <= |k| < 2^53, and adding v rounds v / u to the nearest
// integer independently of s, except that a tie goes to the side that leaves
// k even.  So in a fixed binade one addition is the map
//     k -> k + inc[k & 1]
// given by two integers (equal unless v is a tie), and such maps compose
// associatively: (f then g)[p] = f[p] + g[(p + f[p]) & 1].  A block scans
// them over kFoldThreads x kFoldValues histories at a time in integer
// arithmetic.  Where the sum could leave its binade (about once per doubling
// of a sum of positive terms), or where it is zero, subnormal or not finite,
// the values are added one by one in FP64 (one thread's, or a longer run of
// them where a signed sum keeps wandering about zero), and the scan goes on
// behind them.  Every result bit is the serial chain's.
//
// Bound and measure (GB300): the latency of the steps of the densest column
// (barriers, shuffles, 64-bit shifts) and of its loads, three blocks of which
// are in flight.  500,000 histories x 19 bins: 61.5 ms as one serial chain per
// bin, 0.72 ms here; 50,000 x 931 derivative columns, signed and mostly zero:
// 7.75 -> 0.44 ms, where the slowest column adds 6,700 values serially; 3,001 x
// 180: 0.47 -> 0.04 ms.  (One block in flight, and squares multiplied in the
// serial chain, whose every instruction takes the pipe 64 cycles: 0.87, 0.84
// and 0.12 ms.)
#pragma once

#include <cstdint>

#include "mc_math.cuh"

namespace mc {

constexpr int kFoldThreads = 256;
constexpr int kFoldValues = 8;    // consecutive histories per thread and step
constexpr int kFoldAhead = 3;     // blocks of histories whose loads are in flight
// Where a step fails, the values of this many threads are added serially: two
// at first, more when steps fail one after the other (a sum that starts from
// zero, or a signed one that wanders about it).
__host__ __device__ constexpr int fold_run(int streak) { return streak < 3 ? 2 : (streak < 12 ? 16 : 64); }

// inc[0], inc[1]: what the histories so far add to k if it starts even / odd
struct FoldMap {
    long long a0, a1;
};

__device__ __forceinline__ FoldMap fold_then(const FoldMap &f, const FoldMap &g)
{
    FoldMap r;
    r.a0 = f.a0 + ((f.a0 & 1) ? g.a1 : g.a0);
    r.a1 = f.a1 + ((f.a1 & 1) ? g.a0 : g.a1);
    return r;
}

// A thread's map where some terms are ties (rare: the plain sum of rounded
// terms serves otherwise).  es, sb: exponent field and bits of the sum.
__device__ __noinline__ FoldMap fold_map(const double (&v)[kFoldValues], int es, uint64_t sb)
{
    FoldMap f{0, 0};
    for (int j = 0; j < kFoldValues; ++j) {
        const uint64_t b = dbits(v[j]);
        if ((b << 1) == 0) continue;
        const int ev = (int)((b >> 52) & 0x7FF);
        const uint64_t m = (b & 0x000FFFFFFFFFFFFFull) | (ev ? 0x0010000000000000ull : 0ull);
        const int sh = es - max(ev, 1);
        if (sh < 0 || sh > 63) continue;
        const uint64_t rem = sh > 0 ? m << (64 - sh) : 0ull;
        const uint64_t q = m >> sh;
        uint64_t u0 = rem >> 63, u1 = u0;
        if (rem == 0x8000000000000000ull) {             // to even
            u0 = (uint64_t)(f.a0 + (long long)q) & 1u;
            u1 = (uint64_t)(f.a1 + (long long)q + 1) & 1u;
        }
        const bool neg = (b ^ sb) >> 63;
        f.a0 += neg ? -(long long)(q + u0) : (long long)(q + u0);
        f.a1 += neg ? -(long long)(q + u1) : (long long)(q + u1);
    }
    return f;
}

// One chain: block (bin, which), which = 0 the sum of the column's values,
// 1 the sum of their squares.  hist is [bins][ld], ld even and at least n, zero
// from n on.  Adding zero changes nothing, and most histories score few bins,
// so the column's nonzero values go through a ring in shared memory and every
// step scans kStep of them.
__global__ void __launch_bounds__(kFoldThreads) k_fold_ordered(const double *__restrict__ hist, uint32_t n,
                                                               uint64_t ld, double *__restrict__ sum,
                                                               double *__restrict__ sq)
{
    constexpr uint32_t kStep = (uint32_t)kFoldThreads * kFoldValues, kRing = 2 * kStep;
    constexpr int kWarps = kFoldThreads / 32;
    __shared__ double s_ring[kRing + kRing / 8];   // 9 doubles for 8: a thread's values miss its neighbours' banks
    __shared__ FoldMap s_warp[kWarps];
    __shared__ int s_count[kWarps];
    __shared__ double s_run;      // the running sum before the current step
    __shared__ int s_fail;        // first thread whose values need the serial chain
    __shared__ FoldMap s_total;
    const long long bin = blockIdx.x;
    const bool squares = blockIdx.y != 0;
    double *dst = (squares ? sq : sum) + bin;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const double *col = hist + (uint64_t)bin * ld;
    auto slot = [&](uint32_t i) -> double & {
        i &= kRing - 1;
        return s_ring[i + (i >> 3)];
    };
    // the column's next values, kFoldAhead blocks of kStep histories ahead
    double nxt[kFoldAhead][kFoldValues];
    auto fetch = [&](double (&to)[kFoldValues], uint64_t at) {
        const uint64_t h = at + (uint64_t)t * kFoldValues;
        const double2 *p = reinterpret_cast<const double2 *>(col + h);
#pragma unroll
        for (int j = 0; j < kFoldValues / 2; ++j) {
            const double2 x = h + 2 * j < n ? p[j] : double2{0.0, 0.0};   // zero from n to its pair's end
            to[2 * j] = x.x;
            to[2 * j + 1] = x.y;
        }
    };
    if (t == 0) s_run = *dst;
    uint64_t pos = 0;
    uint32_t head = 0, count = 0;   // the ring's first value and how many it holds
    // one block of histories: its nonzero values (or their squares) go behind
    // the ring's last, and the buffer is filled again
    auto place = [&](double (&buf)[kFoldValues]) {
        double w[kFoldValues];
        int nz = 0;
#pragma unroll
        for (int j = 0; j < kFoldValues; ++j) {
            w[j] = buf[j];
            nz += (dbits(w[j]) << 1) != 0 ? 1 : 0;
        }
        fetch(buf, pos + (uint64_t)kFoldAhead * kStep);
        pos += kStep;
        if (!__syncthreads_or(nz)) return;
        int at = nz;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int p = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o) at += p;
        }
        if (lane == 31) s_count[warp] = at;
        at -= nz;
        __syncthreads();
        int total = 0;
#pragma unroll
        for (int i = 0; i < kWarps; ++i) {
            if (i < warp) at += s_count[i];
            total += s_count[i];
        }
        uint32_t i = head + count + (uint32_t)at;
#pragma unroll
        for (int j = 0; j < kFoldValues; ++j)
            if ((dbits(w[j]) << 1) != 0) slot(i++) = squares ? w[j] * w[j] : w[j];
        count += (uint32_t)total;
        __syncthreads();
    };
    int turn = 0, streak = 0;
#pragma unroll
    for (int a = 0; a < kFoldAhead; ++a) fetch(nxt[a], (uint64_t)a * kStep);
    for (;;) {
        while (count < kStep && pos < n) {
#pragma unroll
            for (int a = 0; a < kFoldAhead; ++a)
                if (turn == a) place(nxt[a]);
            turn = turn + 1 == kFoldAhead ? 0 : turn + 1;
        }
        if (count == 0) break;
        const uint32_t have = min(count, kStep);
        double v[kFoldValues];
        bool any = false;
#pragma unroll
        for (int j = 0; j < kFoldValues; ++j) {
            const uint32_t i = (uint32_t)t * kFoldValues + j;
            v[j] = i < have ? slot(head + i) : 0.0;
            any = any || i < have;
        }
        const uint64_t sb = dbits(s_run);
        const int es = (int)((sb >> 52) & 0x7FF);
        const bool scannable = es > 0 && es < 0x7FF;
        const long long k = (long long)((sb & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull);
        // this thread's map, and a bound on how far k moves within it: without
        // ties both entries are the sum of the rounded terms
        long long move = 0;
        unsigned long long reach = 0;
        bool bad = false, tie = false;
        if (any) {
#pragma unroll
            for (int j = 0; j < kFoldValues; ++j) {
                const uint64_t b = dbits(v[j]);
                const int ev = (int)((b >> 52) & 0x7FF);
                const uint64_t m = (b & 0x000FFFFFFFFFFFFFull) | (ev ? 0x0010000000000000ull : 0ull);
                const int sh = es - max(ev, 1);         // v / u = m 2^-sh
                bad = bad || ((b << 1) != 0 && (ev == 0x7FF || sh < 0));
                const uint64_t rem = (sh > 0 && sh < 64) ? m << (64 - sh) : 0ull;   // the bits below the unit
                const uint64_t q = ((sh >= 0 && sh < 64) ? m >> sh : 0ull) + (rem >> 63);
                tie = tie || rem == 0x8000000000000000ull;
                reach += q + 1;
                move += ((b ^ sb) >> 63) ? -(long long)q : (long long)q;
            }
            bad = bad || !scannable;
        }
        // k before this thread's histories (k0), and the block's total
        long long k0;
        if (!__syncthreads_or(tie)) {
            long long inc = move;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const long long p = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += p;
            }
            if (lane == 31) s_warp[warp].a0 = inc;
            if (t == 0) s_fail = kFoldThreads;
            __syncthreads();
            long long w = 0, total = 0;
#pragma unroll
            for (int i = 0; i < kFoldThreads / 32; ++i) {
                const long long x = s_warp[i].a0;
                if (i < warp) w += x;
                total += x;
            }
            k0 = k + w + inc - move;
            if (t == 0) s_total = FoldMap{total, total};
        } else {
            FoldMap inc = any && !bad ? fold_map(v, es, sb) : FoldMap{0, 0};
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                FoldMap p;
                p.a0 = __shfl_up_sync(0xffffffffu, inc.a0, o);
                p.a1 = __shfl_up_sync(0xffffffffu, inc.a1, o);
                if (lane >= o) inc = fold_then(p, inc);
            }
            FoldMap before;
            before.a0 = __shfl_up_sync(0xffffffffu, inc.a0, 1);
            before.a1 = __shfl_up_sync(0xffffffffu, inc.a1, 1);
            if (lane == 0) before = FoldMap{0, 0};
            if (lane == 31) s_warp[warp] = inc;
            if (t == 0) s_fail = kFoldThreads;
            __syncthreads();
            FoldMap w{0, 0};
            for (int i = 0; i < warp; ++i) w = fold_then(w, s_warp[i]);
            if (warp == kFoldThreads / 32 - 1 && lane == 0) s_total = fold_then(w, s_warp[warp]);
            before = fold_then(w, before);
            k0 = k + ((k & 1) ? before.a1 : before.a0);
        }
        // k stays in the binade through this thread's histories if it cannot
        // reach either end.  (Threads behind the first failing one may see
        // wrapped values; they are taken again.)
        if (any && (bad || k0 <= (1ll << 52) || k0 >= (1ll << 53) || reach >= (1ull << 53) ||
                    (unsigned long long)(k0 - (1ll << 52)) <= reach || (unsigned long long)((1ll << 53) - k0) <= reach))
            atomicMin(&s_fail, t);
        __syncthreads();
        const int fail = s_fail;
        const uint64_t keep = sb & 0xFFF0000000000000ull;   // sign and exponent of the running sum
        uint32_t taken = have;
        if (fail == kFoldThreads) {
            if (t == 0) {
                const long long kn = k + ((k & 1) ? s_total.a1 : s_total.a0);
                s_run = scannable ? dfrom(keep | ((uint64_t)kn & 0x000FFFFFFFFFFFFFull)) : s_run;
            }
            streak = 0;
        } else {
            const uint32_t first = (uint32_t)fail * kFoldValues;
            taken = min(have, first + (uint32_t)fold_run(++streak) * kFoldValues);
            if (t == fail) {
                double s = scannable ? dfrom(keep | ((uint64_t)k0 & 0x000FFFFFFFFFFFFFull)) : s_run;
#pragma unroll 8
                for (uint32_t i = first; i < taken; ++i) s += slot(head + i);
                s_run = s;
            }
        }
        head += taken;
        count -= taken;
        __syncthreads();
    }
    if (t == 0) *dst = s_run;
}

}  // namespace mc
