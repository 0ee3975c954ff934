// mc_history_kernels.cuh -- FP64 history-based transport (replay and plain modes).
//
// One thread walks one history at a time, with the arithmetic and the draws
// of Simulator::start and Simulator::random_walk on the CPU
// (src/simulator/handler.cpp:11-48, general.cpp:13-211): the particle and its
// split copies come from a per-thread LIFO stack, and every tally contribution
// is added to the history's own entry of a per-history bin array, in the
// reference's order.  mc_fold.cuh and mc_exact.cu fold the entries
// (Estimator::end_history, Estimator.cpp:339-346).
//
// Replay mode uses the portable elementary functions of mc_math.cuh and is
// built with -fmad=false (mc_history.cu), so every history's event sequence
// and every tally bin equal the CPU oracle's bit for bit.  Plain mode swaps in
// CUDA's native FP64 log/sin/cos, contracts products and sums into FMAs
// (mc_history_plain.cu) and folds with a parallel tree: the plain
// double-precision GPU history path.
//
// What bounds it is the FP64 pipe: 19 SM cycles per warp instruction, however
// few lanes are active (mc_fp64.cuh).  Hence:
//   * One flat loop instead of a walk per history: a lane whose particle died
//     takes its next one while the others go on (nested loops ran with 11 of
//     32 lanes active: a warp waited for its longest walk).
//   * Steps chosen per warp: an advance (decide between collision and
//     crossing, almost without FP64), else the crossings or the collisions
//     that wait, once enough lanes do.
//   * What only decides something is bounded in FP32 first, and in FP64 where
//     the bounds cannot tell: whether the particle reaches a surface before
//     its collision, the sign of a surface's equation in the cell search, the
//     branch and the rejection test of a free-gas candidate.  The decision is
//     always the FP64 one; only values that enter the history's state are
//     computed in FP64: one logarithm of an accepted candidate, not three of
//     each rejected one.
//   * Cross sections are looked up once per energy and material, all three
//     of them with shared quotients, through the tables of mc_fp64tables.h.
//
// Measured (GB300, transport kernel): 50,000 shield histories in replay 74.0 ->
// 11.8 ms, 200,000 in plain mode 150 -> 31.3 ms, 2,000,000 deep-slab histories
// in plain mode 31.0 -> 3.4 ms; FP64 pipe busy 67 to 77 % of active cycles, the
// rest instruction fetch and the latency of integer and FP32 chains.
//
// Fission is out of scope: collision() skips the implicit-fission block of
// general.cpp:135-151 and Sigma_f is zero.  A capture-only user nuclide has
// sigma_t = sigma_a = sigma_c, sigma_s = 0 (the reference leaves sigma_t
// unset and crashes).
#pragma once

#include <cfloat>

#include "mc_device.h"
#include "mc_fp64.cuh"
#include "mc_math.cuh"

namespace mc {

namespace {

constexpr double kPi = 0x1.921fb54442d18p+1;
constexpr double kPi2 = 2.0 * kPi;
constexpr double kPiHalf = 0.5 * kPi;
constexpr double kPiSqrt = 0x1.c5bf891b4ef6ap+0;
constexpr double kEpsF = (double)FLT_EPSILON;
constexpr double kMaxF = (double)FLT_MAX;
constexpr double kMaxFLess = 0.9 * kMaxF;
constexpr int kMaxFilt = 8;
constexpr int kMaxIl = 64;
constexpr int kMaxParams = kMaxLrParams;
constexpr float kInfF = __builtin_huge_valf();
constexpr int kBlock = 128;

enum { C_FLIGHTS = 0, C_COLL, C_CROSS, C_TALLY, C_PART, C_SPLIT, C_XS, C_FREEGAS, C_NUC };

__device__ const LnTable d_ln = make_ln_table();

// The kernel's loop runs a warp through all of its code once per event, and
// instruction fetch was its second limit (10 of 20 cycles per issue with
// everything inlined).  What is called from several places is out of line: a
// call costs a few cycles against the 64 of one FP64 instruction.
__device__ __noinline__ U4 philox_block(uint32_t b, uint32_t event, uint32_t id, uint32_t hist_lo, uint32_t k0, uint32_t k1)
{
    return philox(b, event, id, hist_lo, k0, k1);
}
__device__ __noinline__ double log_replay(double x) { return plog_unit(x, d_ln); }
__device__ __noinline__ double log_plain(double x) { return ::log(x); }

// a particle on the split stack
struct PartD {
    double x, y, z, u, v, w;
    double E, E_old, speed, wgt, t, t_old;
    int cell, cell_old, surf_old, g;
    unsigned id;
    int alive;
};

template <bool R> struct Fn;
template <> struct Fn<true> {
    static __device__ __forceinline__ double log(double x) { return log_replay(x); }
    static __device__ __forceinline__ void sincos(double x, uint64_t v, double &s, double &c) { psincos_azi(x, v, s, c); }
    static __device__ __forceinline__ double cos_quarter(double x, uint64_t v) { return pcos_quarter(x, v); }
};
template <> struct Fn<false> {
    static __device__ __forceinline__ double log(double x) { return log_plain(x); }
    static __device__ __forceinline__ void sincos(double x, uint64_t, double &s, double &c) { ::sincos(x, &s, &c); }
    static __device__ __forceinline__ double cos_quarter(double x, uint64_t) { return ::cos(x); }
};

// The draws of one particle and event: draw d is the words (0,1) or (2,3) of
// block d / 2 of its Philox stream (mc_math.cuh, Stream), as 52 bits.
struct Draws {
    uint32_t k0, k1, hist_lo, id, event, draw;
    U4 blk;
    __device__ __forceinline__ void init(uint64_t seed, uint64_t history)
    {
        k0 = (uint32_t)seed;
        k1 = (uint32_t)(seed >> 32) ^ (uint32_t)(history >> 32);
        hist_lo = (uint32_t)history;
        id = 0; event = 0; draw = 0;
    }
    __device__ __forceinline__ void start(uint32_t ev) { event = ev; draw = 0; }
    __device__ __forceinline__ uint64_t next()
    {
        uint32_t lo = blk.z, hi = blk.w;
        if (!(draw & 1u)) {
            blk = philox_block(draw >> 1, event, id, hist_lo, k0, k1);
            lo = blk.x;
            hi = blk.y;
        }
        ++draw;
        return (((uint64_t)hi << 32) | lo) >> 12;
    }
    __device__ __forceinline__ uint64_t first() const { return (((uint64_t)blk.y << 32) | blk.x) >> 12; }
};

// A lane's particle and history.
struct Lane {
    double x, y, z, u, v, w, E, speed, wgt, t, t_old;
    int cell, surf_old, g;
    // macroscopic cross sections of material xm at the particle's energy
    // (xm < -1: none yet), and the grid place they came from
    double xT, xS, xC;
    double xS0;            // the first nuclide's part of xS (continuous energy)
    int xm, gid, gi;
    double q1, q2;
    Draws rng;
    double *hist;          // the history's place in the first column
    unsigned long long digest;
    int sp, status;
    uint32_t cnt[kNumCounters];
    // likelihood-ratio state of the derivative kernels: S[k] = d ln(weight x
    // path probability) / d param_k for the materials in `visited` (the
    // others' are zero); split copies keep theirs in lr_stack
    uint32_t visited;
};

// What a kernel carries: continuous-energy problems, multigroup ones, and
// multigroup ones with derivatives.
enum { F_CE = 0, F_MG = 1, F_LR = 2 };

struct Ctx {
    const DevTables &T;
    const HistoryArgs &A;
    PartD *stack;
    double *lr_stack;
    double *S;
    int depth, K, Kc;
};

__device__ __forceinline__ void dig(Lane &P, unsigned long long v) { P.digest = (P.digest ^ v) * 0x100000001B3ULL; }

// Algorithm.cpp:46-64
__device__ __forceinline__ int bsearch_d(double x, const double *vec, int n)
{
    int left = 0, right = n - 1;
#pragma unroll 1
    while (left <= right) {
        const int mid = (left + right) / 2;
        if (dlt(vec[mid], x)) left = mid + 1;
        else right = mid - 1;
    }
    return right;
}

// Algorithm.cpp:16-38
__device__ __forceinline__ double geometry_quad(double a, double b, double c)
{
    const double D = b * b - 4.0 * a * c;
    if (D <= 0.0) return kMaxF;
    const double sqrtD = fsqrt(D);
    const double ai = fdiv(0.5, a);
    double r1 = ai * (-1.0 * b - sqrtD);
    double r2 = ai * (-1.0 * b + sqrtD);
    if (r1 < 0) r1 = kMaxF;
    if (r2 < 0) r2 = kMaxF;
    return fmin(r1, r2);
}

// Geometry.cpp:29-69
__device__ __noinline__ double surface_eval(const DevTables &T, int s, double px, double py, double pz)
{
    const double *k = T.surf_coef + 8 * s;
    switch (T.surf_type[s]) {
    case 0: return px - k[0];
    case 1: return py - k[0];
    case 2: return pz - k[0];
    case 3: return k[0] * px + k[1] * py + k[2] * pz - k[3];
    case 4: {
        const double xt = px - k[0], yt = py - k[1], zt = pz - k[2];
        return xt * xt + yt * yt + zt * zt - k[4];
    }
    case 5: {
        const double yt = py - k[0], zt = pz - k[1];
        return yt * yt + zt * zt - k[3];
    }
    case 6: {
        const double xt = px - k[0], zt = py - k[1];
        return xt * xt + zt * zt - k[3];
    }
    default: {
        const double xt = px - k[0], yt = py - k[1];
        return xt * xt + yt * yt - k[3];
    }
    }
}

__device__ __forceinline__ double axis_distance(double loc, double pos, double dir)
{
    if (dlt(kEpsF, fabs(dir))) {
        const double num = loc - pos;
        // a quotient of unlike signs, or of zero, is not > 0
        if (is_zero(num) || ((dbits(num) ^ dbits(dir)) >> 63)) return kMaxF;
        const double dist = fdiv(num, dir);
        if (dist > 0.0) return dist;
        return kMaxF;
    }
    return kMaxF;
}

// Geometry.cpp:76-188
__device__ __noinline__ double surface_distance(const DevTables &T, int s, const double px, const double py, const double pz,
                                                const double u, const double v, const double w)
{
    const double *k = T.surf_coef + 8 * s;
    switch (T.surf_type[s]) {
    case 0: return axis_distance(k[0], px, u);
    case 1: return axis_distance(k[0], py, v);
    case 2: return axis_distance(k[0], pz, w);
    case 3: {
        const double denom = k[0] * u + k[1] * v + k[2] * w;
        if (dlt(kEpsF, fabs(denom))) {
            const double dist = fdiv(k[3] - k[0] * px - k[1] * py - k[2] * pz, denom);
            if (dist > 0.0) return dist;
            return kMaxF;
        }
        return kMaxF;
    }
    case 4: {
        const double b = 2.0 * ((px - k[0]) * u + (py - k[1]) * v + (pz - k[2]) * w);
        return geometry_quad(1.0, b, surface_eval(T, s, px, py, pz));
    }
    case 5: {
        const double a = 1.0 - u * u;
        const double b = 2.0 * ((py - k[0]) * v + (pz - k[1]) * w);
        return geometry_quad(a, b, surface_eval(T, s, px, py, pz));
    }
    case 6: {
        const double a = 1.0 - v * v;
        const double b = 2.0 * ((px - k[0]) * u + (pz - k[1]) * w);
        return geometry_quad(a, b, surface_eval(T, s, px, py, pz));
    }
    default: {
        const double a = 1.0 - w * w;
        const double b = 2.0 * ((px - k[0]) * u + (py - k[1]) * v);
        return geometry_quad(a, b, surface_eval(T, s, px, py, pz));
    }
    }
}

// FP32 bounds lo <= d <= hi of surface_distance's value d, kMaxF taken as
// infinite.  A quadric whose equation a t^2 + 2 h t + c has no root up to the
// distance `reach` gets lo = infinity (nothing nearer than `reach` is all its
// caller asks); a nearer one, and a general plane, the FP64 value.
// Error terms: f32_of cuts at 2^-23, FP32 operations round at 2^-24 and the
// approximate division at 2 ulp; the margins are above the sum of these
// by a factor of 5 and more.
__device__ __noinline__ float2 distance_bounds(const DevTables &T, int s, double px, double py, double pz, double du, double dv,
                                               double dw, float reach)
{
    const double *k = T.surf_coef + 8 * s;
    const int type = T.surf_type[s];
    if (type <= 2) {
        const double pos = type == 0 ? px : (type == 1 ? py : pz);
        const double dir = type == 0 ? du : (type == 1 ? dv : dw);
        const double num = k[0] - pos;
        if (!dlt(kEpsF, fabs(dir)) || is_zero(num) || ((dbits(num) ^ dbits(dir)) >> 63)) return float2{kInfF, kInfF};
        const float f = __fdividef(fabsf(f32_of(num)), fabsf(f32_of(dir)));
        return float2{f * (1.f - 4e-6f), fmaxf(f * (1.f + 4e-6f), 1e-30f)};
    }
    if (type >= 4) {
        const float x = f32_of(px), y = f32_of(py), z = f32_of(pz), u = f32_of(du), v = f32_of(dv), w = f32_of(dw);
        const float k0 = f32_of(k[0]), k1 = f32_of(k[1]);
        float d0, d1, d2 = 0.f, e0, e1, e2 = 0.f, r2, kk = k0 * k0 + k1 * k1, a = 1.f;
        if (type == 4) {
            const float k2 = f32_of(k[2]);
            d0 = x - k0; d1 = y - k1; d2 = z - k2;
            e0 = u; e1 = v; e2 = w;
            r2 = f32_of(k[4]);
            kk += k2 * k2;
        } else {
            // the reference evaluates cylinder_y's equation at (x, y) and its
            // direction term at (x, z): leave that one to FP64
            d0 = (type == 5 ? y : x) - k0;
            d1 = (type == 5 ? z : y) - k1;
            e0 = type == 5 ? v : u;
            e1 = type == 5 ? w : v;
            const float n = type == 5 ? u : w;
            a = fabsf(1.f - n * n);
            r2 = f32_of(k[3]);
        }
        const float q = d0 * d0 + d1 * d1 + d2 * d2;
        const float h = d0 * e0 + d1 * e1 + d2 * e2;
        const float ha = fabsf(d0 * e0) + fabsf(d1 * e1) + fabsf(d2 * e2);
        // |h| with what cutting x, k and the direction can move it
        const float hm = fabsf(h) + 4e-6f * (ha + (fabsf(k0) + fabsf(k1) + fabsf(d0) + fabsf(d1) + fabsf(d2)) *
                                                      (fabsf(e0) + fabsf(e1) + fabsf(e2)) + sqrtf(kk));
        const float c = fabsf(q - r2) - 4e-6f * (q + fabsf(r2) + kk);
        // (the FP64 root's own error, 2^-49 |h| / a, is far below what the
        // margin in c moves a root by, unless the flight runs along the axis)
        if (type != 6 && a > 1e-5f && ((a + 1e-6f) * reach + 2.f * hm) * reach * 1.0001f < c)
            return float2{kInfF, kInfF};   // (not taken where anything overflowed)
    }
    const double d = surface_distance(T, s, px, py, pz, du, dv, dw);
    const float f = f32_of(d);
    if (f >= FLT_MAX * 0.999f) return float2{kInfF, kInfF};
    return float2{f * (1.f - 1e-6f), fmaxf(f * (1.f + 1e-6f), 1e-30f)};
}

// whether surface_eval(...) * sense < 0 (general.cpp:13-24): the sign of the
// equation, bounded in FP32 where that can tell
__device__ __forceinline__ bool outside(const DevTables &T, int s, int sense, double px, double py, double pz)
{
    if (sense == 0) return false;
    const double *k = T.surf_coef + 8 * s;
    const int type = T.surf_type[s];
    float c = 0.f, err = kInfF;
    if (type <= 2) {
        const float p = f32_of(type == 0 ? px : (type == 1 ? py : pz)), k0 = f32_of(k[0]);
        c = p - k0;
        err = 1e-6f * (fabsf(p) + fabsf(k0));
    } else if (type >= 4) {
        const float x = f32_of(px), y = f32_of(py), z = f32_of(pz), k0 = f32_of(k[0]), k1 = f32_of(k[1]);
        const float k2 = type == 4 ? f32_of(k[2]) : 0.f;
        const float d0 = (type == 5 ? y : x) - k0, d1 = (type == 5 ? z : y) - k1, d2 = type == 4 ? z - k2 : 0.f;
        const float r2 = f32_of(k[type == 4 ? 4 : 3]);
        const float q = d0 * d0 + d1 * d1 + d2 * d2;
        c = q - r2;
        err = 4e-6f * (q + fabsf(r2) + k0 * k0 + k1 * k1 + k2 * k2);
    }
    if (fabsf(c) > err + 1e-30f) return (c < 0.f) == (sense > 0);   // false where anything is not finite
    return surface_eval(T, s, px, py, pz) * sense < 0;
}

// Geometry.cpp:195-222
__device__ __forceinline__ void surface_reflect(const DevTables &T, int s, double &u, double &v, double &w)
{
    const double *k = T.surf_coef + 8 * s;
    switch (T.surf_type[s]) {
    case 0: u = -u; break;
    case 1: v = -v; break;
    case 2: w = -w; break;
    case 3: {
        const double K = k[0] * u + k[1] * v + k[2] * w;
        const double qx = u - k[4] * K, qy = v - k[5] * K, qz = w - k[6] * K;
        u = qx; v = qy; w = qz;
        break;
    }
    default: break;
    }
}

// Particle.cpp:42-56, 66-81 (the time is kept only where a time filter reads it)
__device__ __forceinline__ void p_move(const DevTables &T, Lane &P, double d)
{
    P.x += P.u * d;
    P.y += P.v * d;
    P.z += P.w * d;
    if (T.any_time) {
        P.t_old = P.t;
        P.t += fdiv(d, P.speed);
    }
}

enum { XS_T = 0, XS_S, XS_C };

// The place of E on a nuclide's grid (Nuclide.cpp:18-24): the last point
// below E, -1 if none.
__device__ __forceinline__ int grid_place(const DevTables &T, const Grid64 &g, double E)
{
    const XsRow64 *row = T.xs_row + g.row;
    int lo = 0, hi = g.len;                 // how many points lie below E
    const uint64_t e = dbits(E);
    if (g.fast && e < 0x7FF0000000000000ull) {
        const uint64_t key = e >> g.shift;
        if (key < g.key0) return -1;
        if (key - g.key0 >= (uint64_t)g.n_bkt) return g.len - 1;
        const int *b = T.xs_bkt + g.bkt + (int)(key - g.key0);
        lo = b[0];
        hi = b[1];
#pragma unroll 1
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (dbits(row[mid].E) < e) lo = mid + 1;
            else hi = mid;
        }
        return lo - 1;
    }
    int left = 0, right = g.len - 1;        // Algorithm.cpp:46-64, on whatever the table holds
#pragma unroll 1
    while (left <= right) {
        const int mid = (left + right) / 2;
        if (row[mid].E < E) left = mid + 1;
        else right = mid - 1;
    }
    return right;
}

// The place of E on a grid and the two quotients of Algorithm.cpp:103-105.
struct Place {
    double q1, q2;
    int i;
};

__device__ __noinline__ Place grid_quotients(const DevTables &T, int gid, double E)
{
    const Grid64 &g = T.xs_grid[gid];
    Place p{0.0, 0.0, grid_place(T, g, E)};
    if (p.i < 0 || p.i == g.len - 1) return p;
    const XsRow64 *row = T.xs_row + g.row + p.i;
    const double x1 = row[0].E, x2 = row[1].E;
    const double d = x2 - x1;               // x1 - x2 is its negative, exactly
    const Recip64 r = g.fast ? T.xs_inv[g.inv + p.i] : Recip64{0.0, 0.0};
    p.q1 = -div_by(E - x2, d, r);
    p.q2 = div_by(E - x1, d, r);
    return p;
}

// The lane's place on grid gid, kept until its energy changes.
__device__ __forceinline__ void locate(const DevTables &T, Lane &P, int gid)
{
    if (P.gid == gid) return;
    const Place p = grid_quotients(T, gid, P.E);
    P.gid = gid;
    P.gi = p.i;
    P.q1 = p.q1;
    P.q2 = p.q2;
}

// sigma_s of nuclide n at the lane's energy (XSec.cpp:9-40)
__device__ __forceinline__ double nuclide_scatter(const DevTables &T, Lane &P, const Nuc64 &N)
{
    if (N.kind == 1) return 0.0;
    locate(T, P, N.grid);
    const XsRow64 *row = T.xs_row + N.row;
    if (P.gi == N.len - 1) return row[N.len - 1].S;
    if (P.gi == -1) return row[0].S;
    return P.q1 * row[P.gi].S + P.q2 * row[P.gi + 1].S;
}

// Sigma_t, Sigma_s, Sigma_c of material m at the lane's energy or group
// (Material.cpp:18-57; absorption == capture: sigma_f = 0), once per energy
// and material
template <int F>
__device__ __forceinline__ void material_xs(const DevTables &T, Lane &P, int m)
{
    if (P.xm == m) return;
    P.xm = m;
    if constexpr (F != F_CE) {
        const Mg64 &r = T.mg[m * T.mg_groups + P.g];
        P.xT = r.T;
        P.xS = r.S;
        P.xC = r.C;
        return;
    }
    double sT = 0.0, sS = 0.0, sC = 0.0;
#pragma unroll 1
    for (int i = T.mat_off[m]; i < T.mat_off[m + 1]; ++i) {
        const Nuc64 &N = T.nuc[T.mat_nuc[i]];
        const double dens = T.mat_dens[i];
        if (N.kind == 1) {
            sT += N.constant * dens;
            sS += 0.0 * dens;
            sC += N.constant * dens;
            if (i == T.mat_off[m]) P.xS0 = sS;
            continue;
        }
        locate(T, P, N.grid);
        const XsRow64 *row = T.xs_row + N.row;
        double t, s, c;
        if (P.gi == N.len - 1 || P.gi == -1) {
            const XsRow64 &e = row[P.gi == -1 ? 0 : N.len - 1];
            t = e.T; s = e.S; c = e.C;
        } else {
            const XsRow64 r0 = row[P.gi], r1 = row[P.gi + 1];
            t = P.q1 * r0.T + P.q2 * r1.T;
            s = P.q1 * r0.S + P.q2 * r1.S;
            c = P.q1 * r0.C + P.q2 * r1.C;
        }
        sT += t * dens;
        sS += s * dens;
        sC += c * dens;
        if (i == T.mat_off[m]) P.xS0 = sS;
    }
    P.xT = sT;
    P.xS = sS;
    P.xC = sC;
}

// Algorithm.cpp:67-101
struct Dir {
    double x, y, z;
};

template <bool R>
__device__ __noinline__ Dir scatter_direction(uint64_t v, double dx, double dy, double dz, double mu0)
{
    double sin_azi, cos_azi;
    Fn<R>::sincos(kPi2 * u01_bits(v), v, sin_azi, cos_azi);
    const double Ac = fsqrt(1.0 - mu0 * mu0);
    // the two forms differ in the roles of y and z alone
    const bool pole = dz == 1.0;
    const double a = pole ? dy : dz, b = pole ? dz : dy;
    const double B = fsqrt(1.0 - a * a);
    const double Cc = fdiv(Ac, B);
    Dir o;
    o.x = dx * mu0 + (dx * a * cos_azi - b * sin_azi) * Cc;
    const double ob = b * mu0 + (b * a * cos_azi + dx * sin_azi) * Cc;
    const double oa = a * mu0 - cos_azi * Ac * B;
    o.y = pole ? oa : ob;
    o.z = pole ? ob : oa;
    return o;
}

struct Il { int bin; double l; };

// Filter::idx_l (Estimator.cpp:133-246); -1 when more than cap pairs needed
__device__ int filter_idx_l(const DevTables &T, int f, const Lane &p, double l, Il *out, int cap)
{
    const double *grid = T.filt_grid + T.filt_grid_off[f];
    const int glen = T.filt_grid_len[f];
    const int nbin = glen - 1;
    if (cap < 1) return -1;
    switch (T.filt_kind[f]) {
    case 0: {
        const int b = bsearch_d((double)p.surf_old, grid, glen) + 1;
        if (b < 0 || b >= T.filt_size[f]) return 0;
        out[0].bin = b; out[0].l = l; return 1;
    }
    case 1: {
        const int b = bsearch_d((double)p.cell, grid, glen) + 1;
        if (b < 0 || b >= T.filt_size[f]) return 0;
        out[0].bin = b; out[0].l = l; return 1;
    }
    case 2: {
        const int b = bsearch_d(p.E, grid, glen);
        if (b < 0 || b >= nbin) return 0;
        out[0].bin = b; out[0].l = l; return 1;
    }
    case 4:
        out[0].bin = p.g; out[0].l = l; return 1;
    default: {
        const int loc1 = bsearch_d(p.t_old, grid, glen);
        const int loc2 = bsearch_d(p.t, grid, glen);
        if (loc1 == loc2) {
            if (loc1 >= 0 && loc1 < nbin) { out[0].bin = loc1; out[0].l = l; return 1; }
            return 0;
        }
        const int num_bin = loc2 - loc1 - 1;
        const int need = (loc1 >= 0) + (num_bin > 0 ? num_bin : 0) + (loc2 < nbin);
        if (need > cap) return -1;
        int n = 0;
        if (loc1 >= 0) { out[n].bin = loc1; out[n].l = (grid[loc1 + 1] - p.t_old) * p.speed; ++n; }
#pragma unroll 1
        for (int i = 1; i <= num_bin; ++i) {
            out[n].bin = loc1 + i; out[n].l = (grid[loc1 + i + 1] - grid[loc1 + i]) * p.speed; ++n;
        }
        if (loc2 < nbin) { out[n].bin = loc2; out[n].l = (p.t - grid[loc2]) * p.speed; ++n; }
        return n;
    }
    }
}

// Score::score (Estimator.cpp:17-124); the cross sections are the lane's
// (score_xs brought them up to date)
__device__ __forceinline__ double score_value(const DevTables &T, Lane &P, int sc, int m, double l)
{
    const int kernel = T.score_kernel[sc], kind = T.score_kind[sc];
    const double k = kernel == 0 ? P.wgt * l : (kernel == 1 ? fdiv(P.wgt, m >= 0 ? P.xT : 0.0) : P.wgt);
    P.cnt[C_XS] += m >= 0 ? (kernel == 1 ? 1u : 0u) + (kind != 0 ? 1u : 0u) : 0u;
    if (kind == 0) return k;
    return (m >= 0 ? (kind == 2 ? P.xS : (kind == 4 ? P.xT : P.xC)) : 0.0) * k;
}

// d(score)/d(Sigma_s), d(score)/d(Sigma_a) of the cell's material when the
// score itself holds a cross section (Estimator.cpp:29, 60-124); 1-group
__device__ __forceinline__ void direct_terms(const DevTables &T, int sc, int m, const Lane &P, double v, double &ds, double &da)
{
    ds = 0.0;
    da = 0.0;
    if (m < 0) return;
    const Mg64 &r = T.mg[m * T.mg_groups + P.g];
    const double st = r.T, ss = r.S, sa = r.C;
    const int kind = T.score_kind[sc];
    if (kind == 2 && ss != 0.0) ds += v / ss;
    if ((kind == 1 || kind == 3) && sa != 0.0) da += v / sa;
    if (kind == 4) { ds += v / st; da += v / st; }
    if (T.score_kernel[sc] == 1) { ds -= v / st; da -= v / st; }
}

// one contribution to a bin, and to its derivative columns
template <int F>
__device__ __forceinline__ void tally(const Ctx &C, Lane &P, int sc, int m, long long bin, double v)
{
    P.hist[(size_t)bin * C.A.hist_ld] += v;
    P.cnt[C_TALLY]++;
    if constexpr (F == F_LR) {
        // d(contribution)/d(param_k) = v S_k + direct dependence; a material
        // the history never met has S = 0 and adds nothing
        const size_t ld = C.A.hist_ld;
        double *dh = P.hist + ((size_t)C.T.n_bins + (size_t)bin * C.Kc) * ld;
        double ds, da;
        direct_terms(C.T, sc, m, P, v, ds, da);
        const uint32_t all = C.K >= 64 ? 0xFFFFFFFFu : (1u << (C.K / 2)) - 1u;
        uint32_t todo = fabs(v) <= DBL_MAX ? P.visited | (m >= 0 ? 1u << m : 0u) : all;
#pragma unroll 1
        while (todo) {
            const int mm = __ffs(todo) - 1;
            todo &= todo - 1;
            const bool met = (P.visited >> mm) & 1u;
            double d_s = v * (met ? C.S[2 * mm] : 0.0), d_a = v * (met ? C.S[2 * mm + 1] : 0.0);
            if (mm == m) { d_s += ds; d_a += da; }
            dh[(size_t)(2 * mm) * ld] += d_s;
            dh[(size_t)(2 * mm + 1) * ld] += d_a;
            // rho d/drho = Sigma_s d/dSigma_s + Sigma_a d/dSigma_a, per history
            if (C.Kc > C.K) {
                const Mg64 &r = C.T.mg[mm * C.T.mg_groups];
                dh[(size_t)(C.K + mm) * ld] += r.S * d_s + r.C * d_a;
            }
        }
    }
}

// Estimator::score (Estimator.cpp:298-336) in full: a time filter may split
// one flight over several bins
template <int F>
__device__ __noinline__ void estimator_score_general(const Ctx &C, Lane &P, int e, double l_in)
{
    const DevTables &T = C.T;
    const int m = T.cell_mat[P.cell];
    const int f0 = T.est_filt_off[e], nf = T.est_filt_off[e + 1] - f0;
    const int s0 = T.est_score_off[e], ns = T.est_score_off[e + 1] - s0;
    const double *fac = T.est_factor + T.est_factor_off[e];
    const long long base = T.est_bin_off[e];
    Il il[kMaxIl];
    int off[kMaxFilt + 1], nil[kMaxFilt], idx[kMaxFilt];
    off[0] = 0;
#pragma unroll 1
    for (int i = 0; i < nf; ++i) {
        const int n = filter_idx_l(T, f0 + i, P, l_in, il + off[i], kMaxIl - off[i]);
        if (n < 0) { P.status = DS_OVERFLOW; return; }
        if (n == 0) return;
        nil[i] = n;
        off[i + 1] = off[i] + n;
        idx[i] = 0;
    }
#pragma unroll 1
    for (int guard = 0; guard <= off[nf]; ++guard) {   // each pass advances one filter
        double l = kMaxF;
#pragma unroll 1
        for (int i = 0; i < nf; ++i) {
            const double x = il[off[i] + idx[i]].l;
            l = (x < l) ? x : l;
        }
        int idx1 = 0;
#pragma unroll 1
        for (int i = 0; i < nf; ++i) idx1 += (int)(il[off[i] + idx[i]].bin * fac[i + 1]);
#pragma unroll 1
        for (int s = 0; s < ns; ++s) {
            tally<F>(C, P, s0 + s, m, base + idx1, score_value(T, P, s0 + s, m, l));
            idx1 += (int)fac[0];
        }
#pragma unroll 1
        for (int i = 0; i < nf; ++i) {
            Il &cur = il[off[i] + idx[i]];
            cur.l -= l;
            if (cur.l < kEpsF) {
                if (idx[i] == nil[i] - 1) return;
                idx[i]++;
            }
        }
        if (nf == 0) return;
    }
}

// Estimator::score.  Without a time filter every filter gives one bin or
// none and the whole length, so the combination loop is one pass; `pre` is
// the index part of the cell or surface filter the attachment fixes.
template <int F>
__device__ __forceinline__ void estimator_score(const Ctx &C, Lane &P, int e, double l_in, int pre)
{
    const DevTables &T = C.T;
    if (!(fabs(l_in) <= DBL_MAX)) {   // non-finite track: the combination loop would never advance
        P.status = DS_NAN;
        return;
    }
    const int m = T.cell_mat[P.cell];
    const int s0 = T.est_score_off[e], s1 = T.est_score_off[e + 1];
    if (m >= 0) {
        bool need = false;
#pragma unroll 1
        for (int s = s0; s < s1; ++s) need = need || T.score_kernel[s] == 1 || T.score_kind[s] != 0;
        if (need) material_xs<F>(T, P, m);
    }
    if (T.est_time[e] || dlt(kMaxF, l_in)) {
        Lane q = P;                    // a copy: the lane itself stays in registers
        estimator_score_general<F>(C, q, e, l_in);
        P.status = q.status;
        P.cnt[C_TALLY] = q.cnt[C_TALLY];
        P.cnt[C_XS] = q.cnt[C_XS];
        return;
    }
    if (pre < 0) return;
    int idx1 = pre;
    const int f0 = T.est_filt_off[e], nf = T.est_filt_off[e + 1] - f0;
    const int *fac = T.est_ifac + T.est_factor_off[e];
#pragma unroll 1
    for (int i = 1; i < nf; ++i) {     // the attachment's own filter comes first
        const int f = f0 + i;
        int b = P.g;
        if (T.filt_kind[f] == 2) {
            const int glen = T.filt_grid_len[f];
            b = bsearch_d(P.E, T.filt_grid + T.filt_grid_off[f], glen);
            if (b < 0 || b >= glen - 1) return;
        }
        idx1 += b * fac[i + 1];
    }
    const long long base = T.est_bin_off[e];
#pragma unroll 1
    for (int s = s0; s < s1; ++s) {
        tally<F>(C, P, s, m, base + idx1, score_value(T, P, s, m, l_in));
        idx1 += fac[0];
    }
}

// population_control.cpp:9-15
__device__ __forceinline__ bool weight_roulette(const DevTables &T, Lane &P)
{
    if (dlt(P.wgt, T.wr)) {
        if (dlt(u01_bits(P.rng.next()), fdiv(P.wgt, T.ws))) { P.wgt = T.ws; return true; }
        P.wgt = 0.0;
        return false;
    }
    return true;
}

// population_control.cpp:21-49
template <int F>
__device__ __forceinline__ bool cell_importance(const Ctx &C, Lane &P, double Iold, double Inew)
{
    const DevTables &T = C.T;
    const double rat = fdiv(Inew, Iold);
    if (rat < 1.0) {
        if (u01_bits(P.rng.next()) < rat) { P.wgt = fdiv(P.wgt, rat); return true; }
        P.wgt = 0.0;
        return false;
    }
    const int n = (int)floor(rat + u01_bits(P.rng.next()));
    P.wgt = fdiv(P.wgt, (double)n);
#pragma unroll 1
    for (int i = 0; i < n - 1; ++i) {
        if (P.sp >= C.depth) { P.status = DS_OVERFLOW; return true; }
        PartD q;
        q.x = P.x; q.y = P.y; q.z = P.z; q.u = P.u; q.v = P.v; q.w = P.w;
        q.E = P.E; q.E_old = 0.0; q.speed = P.speed; q.wgt = P.wgt; q.t = P.t; q.t_old = P.t_old;
        q.cell = P.cell; q.cell_old = -1; q.surf_old = P.surf_old; q.g = P.g;
        q.id = child_id(P.rng.id, P.rng.event, (uint32_t)(i + 1));
        q.alive = 1;
        if constexpr (F == F_LR)
#pragma unroll 1
            for (int k = 0; k < C.K; ++k)
                C.lr_stack[(size_t)P.sp * C.K + k] = ((P.visited >> (k / 2)) & 1u) ? C.S[k] : 0.0;
        C.stack[P.sp++] = q;
        P.cnt[C_SPLIT]++;
    }
    (void)T;
    return true;
}

// general.cpp:26-34 (search_cell with test_point)
__device__ __noinline__ int search_cell(const DevTables &T, double px, double py, double pz)
{
#pragma unroll 1
    for (int c = 0; c < T.n_cell; ++c) {
        bool in = true;
#pragma unroll 1
        for (int i = T.cell_surf_off[c]; i < T.cell_surf_off[c + 1] && in; ++i)
            in = !outside(T, T.cell_surf[i], T.cell_sense[i], px, py, pz);
        if (in) return c;
    }
    return -1;
}

// general.cpp:73-83
template <int F>
__device__ __forceinline__ void move_particle(const Ctx &C, Lane &P, int m, double l)
{
    const DevTables &T = C.T;
    p_move(T, P, l);
    P.cnt[C_FLIGHTS]++;
    if (F == F_CE && m >= 0) P.cnt[C_NUC] += (uint32_t)(T.mat_off[m + 1] - T.mat_off[m]);
    if constexpr (F == F_LR) {
        // the flight's probability carries exp(-Sigma_t l): d/dSigma_s = d/dSigma_a = -l
        if (m >= 0) {
            if (!((P.visited >> m) & 1u)) { P.visited |= 1u << m; C.S[2 * m] = 0.0; C.S[2 * m + 1] = 0.0; }
            C.S[2 * m] -= l;
            C.S[2 * m + 1] -= l;
        }
    }
}

// general.cpp:89-101: the boundary condition or the next cell; false if the
// particle died
__device__ __forceinline__ bool surface_hit(const DevTables &T, Lane &P, int s)
{
    P.cnt[C_CROSS]++;
    P.surf_old = s;
    const int bc = T.surf_bc[s];
    if (bc == -1) {
        P.wgt = 0.0;
        return false;
    }
    if (bc != 0) surface_reflect(T, s, P.u, P.v, P.w);
    p_move(T, P, kEpsF);
    if (bc == 0) {
        const int c = search_cell(T, P.x, P.y, P.z);
        if (c < 0) { P.status = DS_LOST; P.wgt = 0.0; return false; }
        P.cell = c;
    }
    return true;
}

// A free-gas candidate as the reference computes it (Reaction.cpp:47-72): the
// target speed of its draws, and the acceptance probability.  For the rare
// candidate whose FP32 bounds cannot tell.
template <bool R>
__device__ __noinline__ bool candidate_accepted(bool w2, uint64_t v1, uint64_t v2, uint64_t v3, uint64_t vm, uint64_t va,
                                                double beta, double speed)
{
    double x;
    if (w2) {
        x = fsqrt(-Fn<R>::log(u01_bits(v1) * u01_bits(v2)));
    } else {
        const double c = Fn<R>::cos_quarter(kPiHalf * u01_bits(v1), v1);
        x = fsqrt(-Fn<R>::log(u01_bits(v2)) - Fn<R>::log(u01_bits(v3)) * c * c);
    }
    const double V = fdiv(x, beta), mu = mu_bits(vm);
    const double acc = fdiv(fsqrt(speed * speed + V * V - 2.0 * speed * V * mu), speed + V);
    return !(u01_bits(va) > acc);
}

// The branch of a candidate, u < 2 / (2 + sqrt(pi) y), in FP32: 1 or 0, -1
// within 1e-5 of the limit (which is good to 1e-6).
__device__ __forceinline__ int branch_test(uint64_t vb, float y32)
{
    const float p = __fdividef(2.f, 2.f + 1.7724539f * y32), u = f32_of(u01_bits(vb));
    return fabsf(u - p) > 1e-5f * p ? (u < p ? 1 : 0) : -1;
}

// The acceptance test of a candidate (Reaction.cpp:63-72) in FP32: 1 accept,
// 0 reject, -1 too close.  u > sqrt(s^2 + V^2 - 2 s V mu) / (s + V) depends on
// V / s = x / y alone; squared, with r the smaller of x / y and y / x, it
// compares u^2 (1 + r)^2 with 1 + r^2 - 2 r mu.  x is good to 2e-6 plus 1e-6
// absolute (the cosine), the rest to 1e-6.
__device__ __noinline__ int candidate_test(bool w2, uint64_t v1, uint64_t v2, uint64_t v3, uint64_t vm, uint64_t va,
                                              float y32)
{
    float q;                       // x^2
    if (w2) {
        q = neglog_bits(v1) + neglog_bits(v2);
    } else {
        const float c = __cosf(1.5707963f * f32_of(u01_bits(v1)));
        q = neglog_bits(v2) + neglog_bits(v3) * (c * c);
    }
    const float x32 = sqrtf(q);
    const float top = fmaxf(x32, y32), r = __fdividef(fminf(x32, y32), top);
    const float ua = f32_of(u01_bits(va));
    const float lhs = ua * ua * (1.f + r) * (1.f + r), rhs = 1.f + r * r - 2.f * r * f32_of(mu_bits(vm));
    return fabsf(lhs - rhs) > 6e-5f + __fdividef(3e-5f, top) ? (lhs < rhs ? 1 : 0) : -1;
}

// Free-gas elastic scatter (Reaction.cpp:27-118) in three parts, so that a
// warp's lanes go through each of them together: the lab cosine's draw, the
// target's candidates (one per call), and the outgoing velocity.
struct FreeGas {
    uint64_t vmu0;             // draw of the centre-of-mass cosine
    uint64_t v1, v2, v3, vm;   // draws of the accepted candidate
    float y32;
    int nuc, tried;
    bool w2;
};

__device__ __forceinline__ void free_gas_begin(const DevTables &T, Lane &P, FreeGas &g)
{
    g.vmu0 = P.rng.next();
    g.y32 = f32_of(T.nuc[g.nuc].beta * P.speed);
    g.tried = 0;
}

// true when the candidate is accepted (or the limit of candidates is reached)
template <bool R>
__device__ __forceinline__ bool free_gas_candidate(const DevTables &T, Lane &P, FreeGas &g)
{
    P.cnt[C_FREEGAS]++;
    if (++g.tried > (1 << 20) + 1) { P.status = DS_TIMEOUT; return true; }   // acceptance is >= ~1/2
    const double beta = T.nuc[g.nuc].beta;
    const uint64_t vb = P.rng.next();
    int is = branch_test(vb, g.y32);
    if (is < 0) is = u01_bits(vb) < fdiv(2.0, 2.0 + kPiSqrt * (beta * P.speed));
    g.w2 = is != 0;
    g.v1 = P.rng.next();
    g.v2 = P.rng.next();
    if (!g.w2) g.v3 = P.rng.next();
    g.vm = P.rng.next();
    const uint64_t va = P.rng.next();
    is = candidate_test(g.w2, g.v1, g.v2, g.v3, g.vm, va, g.y32);
    if (is < 0) is = candidate_accepted<R>(g.w2, g.v1, g.v2, g.v3, g.vm, va, beta, P.speed);
    return is != 0;
}

template <bool R>
__device__ __forceinline__ void free_gas_finish(const DevTables &T, Lane &P, const FreeGas &g)
{
    const Nuc64 &N = T.nuc[g.nuc];
    const double A = N.A;
    // the accepted candidate in FP64
    double q = -Fn<R>::log(g.w2 ? u01_bits(g.v1) * u01_bits(g.v2) : u01_bits(g.v2));
    if (!g.w2) {
        const double cos_val = Fn<R>::cos_quarter(kPiHalf * u01_bits(g.v1), g.v1);
        q = q - Fn<R>::log(u01_bits(g.v3)) * cos_val * cos_val;
    }
    const double V_tilda = div_by(fsqrt(q), N.beta, N.inv_beta);
    const Dir nd = scatter_direction<R>(P.rng.next(), P.u, P.v, P.w, mu_bits(g.vm));
    const double Vx = nd.x * V_tilda, Vy = nd.y * V_tilda, Vz = nd.z * V_tilda;
    double vx = P.speed * P.u, vy = P.speed * P.v, vz = P.speed * P.w;
    const double ux = div_by(vx + A * Vx, N.onepA, N.inv_onepA);
    const double uy = div_by(vy + A * Vy, N.onepA, N.inv_onepA);
    const double uz = div_by(vz + A * Vz, N.onepA, N.inv_onepA);
    double cx = vx - ux, cy = vy - uy, cz = vz - uz;
    const double speed_c = fsqrt(cx * cx + cy * cy + cz * cz);
    const Dir n = scatter_direction<R>(P.rng.next(), fdiv(cx, speed_c), fdiv(cy, speed_c), fdiv(cz, speed_c),
                                       mu_bits(g.vmu0));
    cx = speed_c * n.x; cy = speed_c * n.y; cz = speed_c * n.z;
    vx = cx + ux; vy = cy + uy; vz = cz + uz;
    // Particle::setSpeed (Particle.cpp:49-56)
    P.speed = fsqrt(vx * vx + vy * vy + vz * vz);
    P.E = 5.2270376e-13 * P.speed * P.speed;
    P.u = fdiv(vx, P.speed); P.v = fdiv(vy, P.speed); P.w = fdiv(vz, P.speed);
    P.xm = -2;
    P.gid = -1;
}

// general.cpp:121-163 without implicit fission, up to the scatter: what is
// left to do after it
enum { COL_DEAD = 0, COL_DONE, COL_FREE_GAS, COL_ISOTROPIC };

template <int F>
__device__ __forceinline__ int collision_begin(const Ctx &C, Lane &P, int m, FreeGas &g)
{
    const DevTables &T = C.T;
    if (m < 0) { P.wgt = 0.0; return COL_DEAD; }
    P.cnt[C_XS] += 4;
    if constexpr (F != F_CE) {
        const int G = T.mg_groups;
        const Mg64 &r = T.mg[m * G + P.g];
        if constexpr (F == F_LR) {
            // collision density Sigma_t times implicit-capture factor Sigma_s/Sigma_t
            // = Sigma_s: d/dSigma_s = 1/Sigma_s, d/dSigma_a = 0 (1 group)
            C.S[2 * m] += 1.0 / r.S;
        }
        P.wgt = div_by(P.wgt * r.TmC, r.T, r.inv_T);
        // first group whose cumulative row sum exceeds u
        const double *cum = T.mg_cum + ((size_t)m * G + P.g) * G;
        const double u = r.S * u01_bits(P.rng.next());
        int lo = 0, hi = G;
#pragma unroll 1
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (dlt(u, cum[mid])) hi = mid;
            else lo = mid + 1;
        }
        if (lo >= G) return COL_DONE;
        if (P.g != lo) { P.g = lo; P.xm = -2; }
        return COL_ISOTROPIC;
    }
    // the advance left the cross sections of this cell at this energy
    const double implicit = P.xC + 0.0;
    P.wgt = fdiv(P.wgt * (P.xT - implicit), P.xT);
    // Material::nuclide_scatter (Material.cpp:106-115): the sum over all
    // nuclides is Sigma_s itself, and the lookup left its first term (with two
    // nuclides none is looked up again: 200,000 plain shields 31.3 -> 30.8 ms)
    const double u = P.xS * u01_bits(P.rng.next());
    double s = P.xS0;
    g.nuc = -1;
    const int first = T.mat_off[m], last = T.mat_off[m + 1] - 1;
#pragma unroll 1
    for (int i = first; i <= last && g.nuc < 0; ++i) {
        if (i == last) s = P.xS;
        else if (i != first) s = s + nuclide_scatter(T, P, T.nuc[T.mat_nuc[i]]) * T.mat_dens[i];
        if (dlt(u, s)) g.nuc = T.mat_nuc[i];
    }
    if (g.nuc < 0) return COL_DONE;
    free_gas_begin(T, P, g);
    return COL_FREE_GAS;
}

template <int F>
__device__ __forceinline__ void digest_event(Lane &P, unsigned long long type)
{
    dig(P, type | ((unsigned long long)(unsigned)P.cell << 8));
    dig(P, dbits(P.x)); dig(P, dbits(P.y)); dig(P, dbits(P.z));
    dig(P, dbits(P.u)); dig(P, dbits(P.v)); dig(P, dbits(P.w));
    dig(P, F != F_CE ? (unsigned long long)P.g : dbits(P.E));
    dig(P, dbits(P.wgt));
}

// population_control.cpp:55-84, after every random walk (handler.cpp:27), on
// the thread's bank.  The first tooth is the one draw, from the stream of the
// particle that just walked at event kCombEvent.  A particle passes at most
// one tooth (the reference's `if`), and tooth j is filled from a bank entry
// i >= j, so the bank is compacted in place; the teeth left over hold the
// bank's first particle with its own weight (bank_tmp(teeth, Pbank[0])).
// The copies get ids child_id(walker, kCombEvent, j + 1).
constexpr uint32_t kCombEvent = 0xFFFFFFFFu;

__device__ __noinline__ void particle_comb(const Ctx &C, Lane &P, uint32_t walker)
{
    const DevTables &T = C.T;
    if (P.sp < T.comb_bank_max) return;
    const int teeth = T.comb_teeth;
    if (teeth > C.depth) { P.status = DS_OVERFLOW; return; }
    double W = 0.0;
#pragma unroll 1
    for (int i = 0; i < P.sp; ++i) W += C.stack[i].wgt;
    const double w_avg = W / (double)teeth;
    P.rng.id = walker;
    P.rng.start(kCombEvent);
    double tooth = u01_bits(P.rng.next()) * w_avg;
    const PartD first = C.stack[0];
    double sum = 0.0;
    int j = 0;
#pragma unroll 1
    for (int i = 0; i < P.sp; ++i) {
        sum += C.stack[i].wgt;
        if (sum > tooth && j < teeth) {   // j < teeth: rounding cannot add a tooth
            PartD q = C.stack[i];
            q.wgt = w_avg;
            C.stack[j++] = q;
            tooth += w_avg;
        }
    }
#pragma unroll 1
    for (int k = j; k < teeth; ++k) C.stack[k] = first;
    P.sp = teeth;
#pragma unroll 1
    for (int k = 0; k < teeth; ++k) C.stack[k].id = child_id(walker, kCombEvent, (uint32_t)(k + 1));
}

// Source.cpp:20-24, 42-45 and Distribution.cpp:30-33, 78-96: the source point
// and the sampled direction and energy
struct SrcDraw64 {
    double u, v, w, E, speed;
    int s;
};

template <bool R>
__device__ __forceinline__ SrcDraw64 draw_source(const DevTables &T, Draws &rng)
{
    SrcDraw64 o;
    const double xi = u01_bits(rng.next());
    int s = bsearch_d(xi, T.src_cdf, T.n_src + 1);
    s = s < 0 ? 0 : (s >= T.n_src ? T.n_src - 1 : s);
    o.s = s;
    const double *ep = T.src_e_par + 2 * s;
    // the compiled reference samples the energy before the direction
    o.E = (T.src_e_kind[s] == 1) ? ep[0] + u01_bits(rng.next()) * ep[1] : ep[0];
    const double *dp = T.src_dir_par + 9 * s;
    const int dk = T.src_dir_kind[s];
    if (dk == 0) {
        o.u = dp[0]; o.v = dp[1]; o.w = dp[2];
    } else if (dk == 1 || dk == 3) {
        const uint64_t vm = rng.next();
        const double mu = (dk == 1) ? mu_bits(vm) : u01_bits(vm);
        const uint64_t va = rng.next();
        const double c = fsqrt(1.0 - mu * mu);
        double sn, cs;
        Fn<R>::sincos(kPi2 * u01_bits(va), va, sn, cs);
        o.v = cs * c;
        o.w = sn * c;
        o.u = mu;
    } else {
        double d[3];
#pragma unroll
        for (int k = 2; k >= 0; --k) {   // z component first, as compiled
            const double *q = dp + 3 * k;
            d[k] = ((int)q[0] == 1) ? q[1] + u01_bits(rng.next()) * q[2] : q[1];
        }
        o.u = d[0]; o.v = d[1]; o.w = d[2];
    }
    // Particle::setEnergy (Particle.cpp:42-47)
    o.speed = 13831.5926439 * fsqrt(o.E) * 100.0;
    return o;
}

__device__ __forceinline__ void place_source(const DevTables &T, const SrcDraw64 &o, Lane &P)
{
    P.x = T.src_pos[3 * o.s]; P.y = T.src_pos[3 * o.s + 1]; P.z = T.src_pos[3 * o.s + 2];
    P.u = o.u; P.v = o.v; P.w = o.w;
    P.t = 0.0; P.t_old = 0.0; P.wgt = 1.0;
    P.cell = T.src_cell[o.s];
    P.surf_old = -1;
    P.E = o.E;
    P.speed = o.speed;
    P.g = T.src_group[o.s];
}

// Multigroup histories last a few events, and a source costs some 70 FP64
// instructions: a warp draws 32 of them together into a ring in shared memory
// and its idle lanes read one each (2,000,000 deep-slab histories: 4.89 -> 4.15
// ms).  While histories run out
// a warp draws only what it needs.
struct SrcSlot64 {
    SrcDraw64 o;
    unsigned hl;               // history of the chunk
};
constexpr int kRing = 64;
struct SrcRing64 {
    SrcSlot64 slot[kRing];
    unsigned last, pos;        // histories handed out when this warp last took some; next slot to read
    int left;
};

template <bool R>
__device__ __noinline__ void ring_draw(const DevTables &T, const HistoryArgs &A, unsigned hl, SrcSlot64 &slot)
{
    Draws rng;
    rng.init(A.seed, A.first + hl);
    slot.o = draw_source<R>(T, rng);
    slot.hl = hl;
}

// makes `want` sources available if the histories last; all lanes
template <bool R>
__device__ __forceinline__ void ring_fill(const DevTables &T, const HistoryArgs &A, SrcRing64 &Q, int want)
{
    const int lane = threadIdx.x & 31, left = Q.left;
    if (left >= want) return;
    const unsigned pos = Q.pos;
    const bool far = (uint64_t)Q.last + 4ull * gridDim.x * kBlock < A.n;
    const int take = far ? 32 : want - left;
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(A.next, (unsigned)take);
    base = __shfl_sync(0xffffffffu, base, 0);
    const int got = base >= A.n ? 0 : (int)min((unsigned)take, A.n - base);
    if (lane < got) ring_draw<R>(T, A, base + lane, Q.slot[(pos + left + lane) % kRing]);
    __syncwarp();
    if (lane == 0) {
        Q.last = base;
        Q.left = left + got;
    }
    __syncwarp();
}

// The advance (general.cpp:40-83, 177-200): collision or crossing?  The
// exponential distance and the surface distances are bounded in FP32, and
// computed in FP64 where the bounds overlap.  Returns the surface the particle
// crosses, -1 for a collision, -2 on an error; the flight's length is computed
// by the step that makes it.
template <bool R, int F>
__device__ __forceinline__ int next_surface(const DevTables &T, Lane &P, int m)
{
    float clo = 0.9f * FLT_MAX, chi = clo;
    if (m >= 0) {
        const uint64_t v0 = P.rng.next();
        P.cnt[C_XS]++;
        material_xs<F>(T, P, m);
        const float c = __fdividef(neglog_bits(v0), f32_of(P.xT));
        clo = c * (1.f - 1e-5f);
        chi = c * (1.f + 1e-5f);
    }
    const bool sane = chi < 1e30f;      // also false for NaN: everything in FP64 then
    const int i0 = T.cell_surf_off[P.cell], i1 = T.cell_surf_off[P.cell + 1];
    int S = -1;
    if (sane) {
        float minhi = kInfF, near_lo = kInfF, other_lo = kInfF;   // the surface with the least hi, and the least lo of the rest
#pragma unroll 1
        for (int i = i0; i < i1; ++i) {
            const int s = T.cell_surf[i];
            const float2 b = distance_bounds(T, s, P.x, P.y, P.z, P.u, P.v, P.w, chi);
            if (b.y < minhi) {
                other_lo = fminf(other_lo, near_lo);
                minhi = b.y;
                near_lo = b.x;
                S = s;
            } else {
                other_lo = fminf(other_lo, b.x);
            }
        }
        if (chi < fminf(near_lo, other_lo)) return -1;
        if (minhi < clo && minhi < other_lo) return S;
    }
    // the reference's own order and comparisons
    double dist = kMaxF;
    S = -1;
#pragma unroll 1
    for (int i = i0; i < i1; ++i) {
        const int s = T.cell_surf[i];
        const double d = surface_distance(T, s, P.x, P.y, P.z, P.u, P.v, P.w);
        if (d < dist) { dist = d; S = s; }
    }
    const double dcol = (m >= 0) ? fdiv(-Fn<R>::log(u01_bits(P.rng.first())), P.xT) : kMaxFLess;
    if (!(dcol > dist)) return -1;
    if (S < 0) { P.status = DS_LOST; return -2; }
    return S;
}

// What a particle does next.
enum { AT_FLIGHT = 0, AT_COLLISION, AT_SURFACE };

// When to make the crossings that wait.  A crossing step costs the warp X FP64
// instructions for however many lanes, a collision step C; with a crossings
// arriving per collision step, waiting for k of them costs a X / k for the
// steps and (k - 1) / 64 C for the lanes that wait meanwhile, least at
// k^2 = 64 a X / C; a is counted, and 64 X / C about 20 for multigroup
// collisions and 8 for continuous energy.  Measured at a half / once / twice
// that: 16-layer slab 3.25 / 3.31 / 3.56 ms, deep slab 3.66 / 3.64 / 3.75 ms,
// 100,000 duct histories 14.9 / 15.2 / 15.6 ms (crossings with every advance:
// 3.63, 4.15 and 15.1 ms).  A warp that was given few lanes is bound by its
// longest history and waits for none.
template <int F> constexpr uint32_t kCrossCost = F == F_CE ? 4u : 12u;

// idle lanes that take new histories together, while others have work (deep
// slab 4.17 / 4.16 / 4.19 / 4.15 ms at 1 / 2 / 4 / 8 from a ring, 16-layer slab
// 3.89 / 3.79 / 3.64 / 3.64; shield 33.3 / 33.3 / 33.8 ms at 2 / 4 / 8)
constexpr int kRefillLanes = 4, kRefillRinged = 8;

// CTAs per SM: registers allow 3 for continuous energy (168 a thread; at 128
// the spills cost more than a fourth CTA gives while histories run out: 13.8
// against 12.1 ms on 50,000 shields) and 4 for the multigroup flavours (deep
// slab 6.0 / 5.1 / 4.9 ms at 2 / 3 / 4).
constexpr int ctas_per_sm(int flavour) { return flavour == F_CE ? 3 : 4; }

template <bool R, int F>
__global__ void __launch_bounds__(kBlock, ctas_per_sm(F)) k_history_fp64(const __grid_constant__ DevTables T,
                                                            const __grid_constant__ HistoryArgs A)
{
    const size_t tid = (size_t)blockIdx.x * kBlock + threadIdx.x;
    const int lane = threadIdx.x & 31;
    constexpr bool L = F == F_LR;
    double S[L ? kMaxParams : 1];
    const int K = L ? A.n_params : 0;
    const Ctx C{T, A, reinterpret_cast<PartD *>(A.stack) + tid * A.stack_depth,
                L ? A.lr_stack + tid * A.stack_depth * (size_t)A.n_params : nullptr, S, (int)A.stack_depth, K,
                L ? (A.n_cols > A.n_params ? A.n_cols : A.n_params) : 0};
    Lane P;
    P.status = DS_OK;
    P.sp = 0;
    P.xm = -2;
    P.gid = -1;
    P.gi = 0;
    P.visited = 0;
    for (int i = 0; i < kNumCounters; ++i) P.cnt[i] = 0;
    constexpr bool kRinged = F != F_CE;
    __shared__ SrcRing64 s_ring[kRinged ? kBlock / 32 : 1];
    SrcRing64 &Q = s_ring[kRinged ? threadIdx.x / 32 : 0];
    if (kRinged && lane == 0) { Q.last = 0; Q.pos = 0; Q.left = 0; }
    __syncwarp();
    const bool digests = A.digest != nullptr;
    bool have = false, open = false, exhausted = lane >= A.lanes;
    int stage = AT_FLIGHT, sx = -1;        // what the particle does next; the surface it will cross
    uint32_t n_cross = 0, n_collide = 1;   // the warp's crossings and collision steps of late
    const uint32_t cross_cost = A.lanes == 32 ? kCrossCost<F> : 0u;
    uint32_t walks = 0;
    unsigned hl = 0;
    for (;;) {
        // the next particle: the history's own split copies first (LIFO), then
        // a new history
        if (!have && open) {
            if constexpr (F != F_LR)              // the derivative kernels refuse combed problems on the host
                if (T.comb_teeth > 0 && P.status == DS_OK) {
                    Lane q = P;
                    particle_comb(C, q, P.rng.id);
                    P.sp = q.sp;
                    P.status = q.status;
                }
            if (P.sp > 0 && P.status == DS_OK) {
                --P.sp;
                const PartD q = C.stack[P.sp];
                P.x = q.x; P.y = q.y; P.z = q.z; P.u = q.u; P.v = q.v; P.w = q.w;
                P.E = q.E; P.speed = q.speed; P.wgt = q.wgt; P.t = q.t; P.t_old = q.t_old;
                P.cell = q.cell; P.surf_old = q.surf_old; P.g = q.g;
                P.xm = -2;
                P.gid = -1;
                if constexpr (F == F_LR) {
                    P.visited = 0;
#pragma unroll 1
                    for (int k = 0; k < K; ++k) {
                        S[k] = C.lr_stack[(size_t)P.sp * K + k];
                        if (!is_zero(S[k])) P.visited |= 1u << (k / 2);
                    }
                }
                if (++walks > (1u << 24)) P.status = DS_TIMEOUT;   // bounded history
                have = P.status == DS_OK;
                P.rng.id = q.id;
                P.rng.start(0);
                P.cnt[C_PART]++;
                if (digests) dig(P, 0xA5A5A5A5ULL ^ q.id);
            }
            if (!have) {                   // the history is over, or failed
                if (digests) A.digest[hl] = P.digest;
                open = false;
                if (P.status != DS_OK) {
                    atomicCAS(A.status, 0, P.status);
                    exhausted = true;
                }
            }
        }
        const unsigned idle = __ballot_sync(0xffffffffu, !have && !exhausted);
        const unsigned adv = __ballot_sync(0xffffffffu, have && stage == AT_FLIGHT);
        const unsigned col = __ballot_sync(0xffffffffu, have && stage == AT_COLLISION);
        const unsigned crs = __ballot_sync(0xffffffffu, have && stage == AT_SURFACE);
        if ((idle | adv | col | crs) == 0u) break;
        if (idle && (__popc(idle) >= (kRinged ? kRefillRinged : kRefillLanes) || (adv | col | crs) == 0u)) {
            const bool need = (idle >> lane) & 1u;
            const int r = __popc(idle & ((1u << lane) - 1u)), want = __popc(idle);
            SrcDraw64 o;
            bool got = false;
            if constexpr (kRinged) {
                ring_fill<R>(T, A, Q, want);
                const int left = Q.left;
                const unsigned pos = Q.pos;
                got = need && r < left;
                if (got) {
                    const SrcSlot64 &q = Q.slot[(pos + r) % kRing];
                    o = q.o;
                    hl = q.hl;
                    P.rng.init(A.seed, A.first + hl);
                }
                __syncwarp();
                if (lane == 0) {
                    Q.pos = (pos + min(want, left)) % kRing;
                    Q.left = left - min(want, left);
                }
                __syncwarp();
            } else {
                unsigned base = 0;
                const int leader = __ffs(idle) - 1;
                if (lane == leader) base = atomicAdd(A.next, (unsigned)want);
                base = __shfl_sync(0xffffffffu, base, leader);
                got = need && base + (unsigned)r < A.n;
                if (got) {
                    hl = base + (unsigned)r;
                    P.rng.init(A.seed, A.first + hl);
                    o = draw_source<R>(T, P.rng);
                }
            }
            if (got) {
                place_source(T, o, P);
                P.hist = A.hist + hl;
                P.digest = 0xCBF29CE484222325ULL;
                P.sp = 0;
                P.visited = 0;
                P.xm = -2;
                P.gid = -1;
                P.rng.start(0);
                P.cnt[C_PART]++;
                if (digests) dig(P, 0xA5A5A5A5ULL);
                walks = 1;
                have = open = true;
                stage = AT_FLIGHT;
            } else if (need) {
                exhausted = true;
            }
            continue;
        }
        // one step of the warp: an advance, else a crossing or a collision
        if (adv) {
            if (have && stage == AT_FLIGHT) {
                P.rng.start(P.rng.event + 1);
                sx = -2;
                if (P.rng.event > A.max_events) P.status = DS_TIMEOUT;   // bounded walk
                else sx = next_surface<R, F>(T, P, T.cell_mat[P.cell]);
                stage = sx == -1 ? AT_COLLISION : AT_SURFACE;
                if (P.status != DS_OK) have = false;
            }
            __syncwarp();
            continue;
        }
        const int nx = __popc(crs);
        const bool colliding = nx == 0 || (col != 0u && (uint32_t)(nx * nx) * n_collide < cross_cost * n_cross);
        if (colliding) ++n_collide;
        else n_cross += (uint32_t)nx;
        if (n_collide > 1024u || n_cross > 16384u) {
            n_collide = (n_collide + 1u) / 2u;
            n_cross /= 2u;
        }
        const bool moves = have && stage == (colliding ? AT_COLLISION : AT_SURFACE);
        const int m = moves ? T.cell_mat[P.cell] : -1, cell_old = P.cell, s = sx;
        double dist = kMaxFLess;
        if (moves) {
            stage = AT_FLIGHT;
            if (!colliding) {
                dist = surface_distance(T, s, P.x, P.y, P.z, P.u, P.v, P.w);
            } else if (m >= 0) {
                const double L0 = -Fn<R>::log(u01_bits(P.rng.first()));
                if constexpr (F != F_CE) dist = div_by(L0, P.xT, T.mg[m * T.mg_groups + P.g].inv_T);
                else dist = fdiv(L0, P.xT);
            }
        }
        __syncwarp();
        if (moves) move_particle<F>(C, P, m, dist);
        // the scores of the flight, then those of the crossing or collision
        bool alive = moves;
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            int i0 = 0, i1 = 0;
            const int *list = T.cell_tl, *pre = T.cell_tl_pre;
            if (moves && pass == 0) {
                i0 = T.cell_tl_off[P.cell];
                i1 = T.cell_tl_off[P.cell + 1];
            } else if (moves && colliding) {
                P.cnt[C_COLL]++;
                list = T.cell_c;
                pre = T.cell_c_pre;
                if (m >= 0) {
                    i0 = T.cell_c_off[P.cell];
                    i1 = T.cell_c_off[P.cell + 1];
                }
            } else if (moves) {
                alive = surface_hit(T, P, s);
                list = T.surf_est;
                pre = T.surf_est_pre;
                if (P.status != DS_LOST) {
                    i0 = T.surf_est_off[s];
                    i1 = T.surf_est_off[s + 1];
                }
            }
#pragma unroll 1
            for (int i = i0; i < i1; ++i) estimator_score<F>(C, P, list[i], pass ? 0.0 : dist, pre[i]);
            __syncwarp();
        }
        if (!colliding) {
            if (alive) {
                const double Iold = T.cell_imp[cell_old], Inew = T.cell_imp[P.cell];
                if (Inew != Iold) alive = cell_importance<F>(C, P, Iold, Inew);
            }
        } else {
            int cst = COL_DEAD;
            FreeGas g;
            if (moves) cst = collision_begin<F>(C, P, m, g);
            __syncwarp();
            if constexpr (F == F_CE) {
                bool pend = cst == COL_FREE_GAS;
#pragma unroll 1
                while (__any_sync(0xffffffffu, pend)) {
                    if (pend) pend = !free_gas_candidate<R>(T, P, g);
                    __syncwarp();
                }
                if (cst == COL_FREE_GAS && P.status == DS_OK) free_gas_finish<R>(T, P, g);
            } else if (cst == COL_ISOTROPIC) {
                const double mu = mu_bits(P.rng.next());
                const Dir n = scatter_direction<R>(P.rng.next(), P.u, P.v, P.w, mu);
                P.u = n.x; P.v = n.y; P.w = n.z;
            }
            alive = cst != COL_DEAD;
        }
        __syncwarp();
        if (moves) {
            have = alive && weight_roulette(T, P);
            if (digests) digest_event<F>(P, colliding ? 2 : 1);
        }
        if (P.status != DS_OK) have = false;
        // one step adds at most 2^20 + a few to a counter
        uint32_t big = 0;
        for (int i = 0; i < kNumCounters; ++i) big |= P.cnt[i];
        if (big >= (1u << 30))
            for (int i = 0; i < kNumCounters; ++i) {
                atomicAdd(A.counters + i, (unsigned long long)P.cnt[i]);
                P.cnt[i] = 0;
            }
    }
    for (int i = 0; i < kNumCounters; ++i) {
        unsigned long long v = P.cnt[i];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0 && v) atomicAdd(A.counters + i, v);
    }
}

}  // namespace
}  // namespace mc
