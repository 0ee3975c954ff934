// mc_fp64tables.cpp -- builds the FP64 kernels' tables (see mc_fp64tables.h).
#include "mc_fp64tables.h"

#include <cmath>
#include <cstring>

namespace mc {

namespace {

uint64_t bits_of(double x)
{
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
}

// Algorithm.cpp:46-64
int bsearch_host(double x, const double *vec, int n)
{
    int left = 0, right = n - 1;
    while (left <= right) {
        const int mid = (left + right) / 2;
        if (vec[mid] < x) left = mid + 1;
        else right = mid - 1;
    }
    return right;
}

// div_by's range: away from overflow and underflow by more than the products
// and remainders it forms
bool in_range(double d) { return d >= 0x1p-200 && d <= 0x1p200; }

void build_grid(const double *E, int len, Fp64Tables &f, Grid64 &g)
{
    g.len = len;
    g.fast = 1;
    for (int i = 0; i < len; ++i)
        if (!in_range(E[i]) || (i > 0 && !(E[i] > E[i - 1] && in_range(E[i] - E[i - 1])))) g.fast = 0;
    g.inv = (int64_t)f.inv.size();
    g.bkt = (int32_t)f.bkt.size();
    if (!g.fast) return;
    for (int i = 0; i + 1 < len; ++i) f.inv.push_back(recip64(E[i + 1] - E[i]));
    // about one point per bucket, at most two buckets per point
    const uint64_t lo = bits_of(E[0]), hi = bits_of(E[len - 1]);
    int shift = 52;
    while (shift > 0 && (hi >> (shift - 1)) - (lo >> (shift - 1)) + 1 <= 2 * (uint64_t)len) --shift;
    g.shift = shift;
    g.key0 = lo >> shift;
    g.n_bkt = (int32_t)((hi >> shift) - g.key0 + 1);
    int below = 0;
    for (int k = 0; k <= g.n_bkt; ++k) {
        while (below < len && (bits_of(E[below]) >> shift) - g.key0 < (uint64_t)k) ++below;
        f.bkt.push_back(below);
    }
}

}  // namespace

Recip64 recip64(double d)
{
    if (!in_range(d)) return {0.0, 0.0};
    const double hi = 1.0 / d;
    return {hi, std::fma(-d, hi, 1.0) * hi};
}

void build_mg64(int n_mat, int G, const double *total, const double *scatter, const double *scat_tot,
                const double *capture, std::vector<Mg64> &mg, std::vector<double> &cum)
{
    mg.assign((size_t)n_mat * G, Mg64{});
    cum.assign((size_t)n_mat * G * G, 0.0);
    for (size_t i = 0; i < mg.size(); ++i) {
        Mg64 &m = mg[i];
        m.T = total[i];
        m.S = scat_tot[i];
        m.C = capture[i];
        m.TmC = total[i] - (capture[i] + 0.0);
        m.inv_T = recip64(total[i]);
        double s = 0.0, top = 0.0;
        for (int g = 0; g < G; ++g) {
            s += scatter[i * G + g];
            top = (g == 0 || s > top) ? s : top;
            cum[i * G + g] = top;
        }
    }
}

void build_fp64_tables(const Tables &t, Fp64Tables &f)
{
    f = Fp64Tables();
    f.row.resize(t.xs_E.size());
    for (size_t i = 0; i < t.xs_E.size(); ++i) f.row[i] = {t.xs_E[i], t.xs_S[i], t.xs_C[i], t.xs_T[i]};
    for (int n = 0; n < t.n_nuc(); ++n) {
        Nuc64 u{};
        u.A = t.nuc_A[n];
        u.beta = std::sqrt(2.0659834e-11 * u.A);
        u.onepA = 1.0 + u.A;
        u.constant = t.nuc_const[n];
        u.inv_beta = recip64(u.beta);
        u.inv_onepA = recip64(u.onepA);
        u.row = t.nuc_off[n];
        u.kind = t.nuc_kind[n];
        u.len = t.nuc_len[n];
        u.grid = -1;
        if (u.kind == N_TABLE) {
            const double *E = &t.xs_E[(size_t)u.row];
            for (int k = 0; k < (int)f.grid.size() && u.grid < 0; ++k)   // nuclides often share a grid
                if (f.grid[k].len == u.len && std::memcmp(E, &t.xs_E[(size_t)f.grid[k].row], 8 * (size_t)u.len) == 0)
                    u.grid = k;
            if (u.grid < 0) {
                Grid64 g{};
                g.row = u.row;
                build_grid(E, u.len, f, g);
                u.grid = (int32_t)f.grid.size();
                f.grid.push_back(g);
            }
        }
        f.nuc.push_back(u);
    }
    if (t.mg_groups > 0)
        build_mg64(t.n_mat(), t.mg_groups, t.mg_total.data(), t.mg_scatter.data(), t.mg_scat_tot.data(),
                   t.mg_capture.data(), f.mg, f.mg_cum);

    for (double x : t.est_factor) f.est_ifac.push_back((int32_t)x);
    f.est_time.assign(t.n_est(), 0);
    for (int e = 0; e < t.n_est(); ++e)
        for (int i = t.est_filt_off[e]; i < t.est_filt_off[e + 1]; ++i)
            if (t.filt_kind[i] == F_TIME) f.est_time[e] = f.any_time = 1;
    // Filter::idx_l of the filter the attachment fixes (Estimator.cpp:133-170)
    auto fixed = [&](int e, int kind, int id) -> int32_t {
        int32_t idx = 0;
        for (int i = t.est_filt_off[e]; i < t.est_filt_off[e + 1]; ++i) {
            if (t.filt_kind[i] != kind) continue;
            const int b = bsearch_host((double)id, &t.filt_grid[(size_t)t.filt_grid_off[i]], t.filt_grid_len[i]) + 1;
            if (b < 0 || b >= t.filt_size[i]) return -1;
            idx += (int32_t)(b * t.est_factor[(size_t)t.est_factor_off[e] + (i - t.est_filt_off[e]) + 1]);
        }
        return idx;
    };
    f.tl_pre.resize(t.cell_tl.size());
    f.c_pre.resize(t.cell_c.size());
    f.s_pre.resize(t.surf_est.size());
    for (int c = 0; c < t.n_cell(); ++c) {
        for (int i = t.cell_tl_off[c]; i < t.cell_tl_off[c + 1]; ++i) f.tl_pre[i] = fixed(t.cell_tl[i], F_CELL, c);
        for (int i = t.cell_c_off[c]; i < t.cell_c_off[c + 1]; ++i) f.c_pre[i] = fixed(t.cell_c[i], F_CELL, c);
    }
    for (int s = 0; s < t.n_surf(); ++s)
        for (int i = t.surf_est_off[s]; i < t.surf_est_off[s + 1]; ++i) f.s_pre[i] = fixed(t.surf_est[i], F_SURFACE, s);
}

}  // namespace mc
