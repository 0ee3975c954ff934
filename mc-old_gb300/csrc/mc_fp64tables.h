// mc_fp64tables.h -- tables of the FP64 history kernels, derived from Tables.
//
// On this GPU an FP64 instruction occupies its SM for 19 cycles per warp
// whatever the number of active lanes (a division takes 141, a square root
// 143), so everything that depends only on the input is worked out here, with
// the same IEEE operations the reference uses at run time:
//
//   * pointwise cross sections as one 32-byte row {E, sigma_s, sigma_c,
//     sigma_t} per grid point, and each distinct energy grid once, with a
//     bucket index over the bit patterns of E (positive doubles order as
//     integers) that leaves the search a few integer comparisons;
//   * divisors that the tables fix (a grid interval, a nuclide's beta and
//     1 + A, a group's Sigma_t) with their reciprocal as a pair hi + lo, so
//     that the kernels divide with four operations (div_by, mc_fp64.cuh);
//   * multigroup rows with Sigma_t - Sigma_c, and the running maximum of the
//     cumulative scatter row (the first group whose cumulative sum exceeds u
//     is the first whose running maximum does), for a search by bisection;
//   * the part of the flattened tally index that the cell or surface filter
//     of an attachment fixes.
#pragma once

#include <cstdint>
#include <vector>

#include "mc_problem.h"

namespace mc {

struct alignas(32) XsRow64 {
    double E, S, C, T;
};

// 1/d as hi + lo; hi = 0: divide by d itself (out of div_by's range)
struct Recip64 {
    double hi, lo;
};

struct alignas(16) Nuc64 {
    double A, beta, onepA, constant;     // beta = sqrt(c A) (Reaction.cpp:39), 1 + A
    Recip64 inv_beta, inv_onepA;
    int64_t row;                         // first of its rows
    int32_t kind, len, grid, pad;
};

struct alignas(16) Grid64 {
    uint64_t key0;                       // bits(first point) >> shift
    int64_t row, inv;                    // a row range holding the grid; its intervals' reciprocals
    int32_t shift, n_bkt, bkt, len;      // bkt: first of n_bkt + 1 counts of points below a bucket
    int32_t fast, pad0, pad1, pad2;      // 0: not sorted, not positive or out of range
};

struct alignas(16) Mg64 {
    double T, S, C, TmC;
    Recip64 inv_T;
    double pad0, pad1;
};

struct Fp64Tables {
    std::vector<XsRow64> row;
    std::vector<Recip64> inv;
    std::vector<int32_t> bkt;
    std::vector<Nuc64> nuc;
    std::vector<Grid64> grid;
    std::vector<Mg64> mg;                // [n_mat][G]
    std::vector<double> mg_cum;          // [n_mat][G][G]
    std::vector<int32_t> tl_pre, c_pre, s_pre;   // per attachment: index part, -1 = outside the filter
    std::vector<int32_t> est_ifac, est_time;     // integer factors; whether the estimator has a time filter
    int32_t any_time = 0;
};

Recip64 recip64(double d);

// The multigroup rows of n_mat x G values (the reader's, or a derivative
// run's parameters).
void build_mg64(int n_mat, int G, const double *total, const double *scatter, const double *scat_tot,
                const double *capture, std::vector<Mg64> &mg, std::vector<double> &cum);

void build_fp64_tables(const Tables &t, Fp64Tables &f);

}  // namespace mc
