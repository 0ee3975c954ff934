// mc_evtables.h -- FP32 tables of the mixed-precision event engine.
//
// Built on the host from Tables (mc_problem.h):
//  * geometry in FP32, plus per-(surface, side) neighbour lists: the cells
//    that list a surface with a given sense, in input order, which is where a
//    particle crossing that surface can land;
//  * continuous-energy data as per-material macroscopic tables on the union
//    of the material's nuclide energy grids.  Each nuclide's cross section is
//    linear between its own grid points, so between consecutive union points
//    every nuclide -- and their density-weighted sum -- is linear: one
//    interpolation of Sigma_t / Sigma_s / Sigma_c replaces the reference's
//    per-nuclide loop (Material.cpp:18-57) with the same values up to
//    rounding.  N_k sigma_s,k per nuclide on the same grid serves the
//    scatter-nuclide choice (Material.cpp:106-115).  A log-spaced bucket
//    table maps log2(E) to a grid index, so no binary search is needed;
//  * multigroup data in FP32 with cumulative scatter rows;
//  * what an event reads about its cell, each of the cell's surfaces, each
//    attached estimator and its material as records of one or two 16-byte
//    vectors, instead of a value at a time from parallel arrays: fewer loads
//    and address computations, and fewer of them one after the other.
#pragma once

#include <stdint.h>
#include <vector_types.h>   // float4, int4, int2 (plain structs; host code builds the rows)

#include <vector>

#include "mc_problem.h"

namespace mc {

// Attachment records, one per score of an attached estimator.  The low bits of
// a code: the estimator takes the general path (one record for all its
// scores), or besides the cell or surface filter that the attachment fixes it
// has no filter, an energy filter or a group filter, whose index is added to
// the bin as it is.  ATT_KERNEL: what the score multiplies (Kernel), ATT_KIND:
// the cross section it multiplies by (ScoreKind).
enum AttCode : int {
    ATT_GENERAL = 0, ATT_PLAIN, ATT_ENERGY, ATT_GROUP, ATT_CODES = 15,
    ATT_KERNEL = 16,   // x Kernel (2 bits)
    ATT_KIND = 64,     // x ScoreKind (3 bits)
};

struct EvTables {
    // records (see above)
    const int4 *cell_rec;             // [n_cell][2]: {material, first surface record, how many, first track-length
                                      // record}, {how many, first collision record, how many, 0}
    const float4 *surf_rec;           // [cell's surfaces][2]: {surface, type, sense, k0}, {k1, k2, k3, k4}
    const int4 *tl_rec, *c_rec, *s_rec;   // per attached score: {bin or, in general, index part (-1: outside the
                                      // filter), code, estimator or energy grid offset, grid length}
    const int2 *surf_est_rec;         // per surface: first crossing record, how many
    const int4 *mat_rec;              // [n_mat][2], continuous energy: {grid offset, length, bucket offset, buckets},
                                      // {log2 E0, buckets per unit log2, first nuclide, how many}
    // geometry
    int n_surf, n_cell;
    const int *surf_type, *surf_bc;
    const float *surf_coef;           // 8 per surface
    const float *cell_imp;
    const int *cell_mat;
    const int *nb_off, *nb_cell;      // CSR over 2*n_surf lists: index 2*s + (sense > 0)
    // estimators
    int n_est;
    long long n_bins;
    const int *est_score_off, *score_kind, *score_kernel;
    const int *est_filt_off, *filt_kind, *filt_size, *filt_grid_len;
    const int *filt_grid_off;
    const float *filt_grid;
    const int *est_factor;            // nfilt+1 per estimator (integers)
    const int *est_factor_off;
    const int *est_bin_off;
    int has_time;                     // a time filter exists (track time)
    int general;                      // an attached estimator takes the general path (ATT_GENERAL)
    // continuous-energy materials
    int n_mat;
    // union grid and macroscopic tables, one 16-byte row per grid point:
    // {Sigma_t, Sigma_s, Sigma_c, E}, so that the two rows bracketing E
    // (one 32-byte load) give the bracket check and all three values
    const float4 *xrow;
    const int2 *mnuc_rec;             // per nuclide of a material: {offset of its table in nucS less the material's
                                      // grid offset, mass A (float bits)}
    const float *nucS;                // N_k sigma_s,k tables
    const int *bkt;                   // grid index of the last point <= bucket start
    // multigroup
    int G;
    const float *mg_total, *mg_scat_tot, *mg_capture;   // [n_mat][G]
    const float *mg_cdf;              // [n_mat][G][G] cumulative scatter rows
    // sources
    int n_src;
    const float *src_pos, *src_dir_par, *src_e_par, *src_cdf;
    const int *src_cell, *src_dir_kind, *src_e_kind, *src_group;
    float wr, ws;
    int comb_bank_max, comb_teeth;    // particle comb (0 teeth: off)
};

// Host-side storage behind EvTables (one packed device allocation).
struct EvHost {
    std::vector<char> blob;                     // packed arrays
    std::vector<std::pair<const void **, size_t>> fix;
    EvTables view{};
    size_t mg_bytes = 0;                        // bytes of the MG tables
};

// Builds the FP32 tables; false + err if the problem cannot run in this mode.
bool build_event_tables(const Tables &t, EvHost &h, std::string &err);

}  // namespace mc
