// mc_engine.cpp -- device tables, tally accumulation and the FP64 history
// engine driver (see mc_engine.h).
#include "mc_engine.h"

#include <algorithm>
#include <cstring>

namespace mc {

std::string cuda_msg(cudaError_t e, const char *what)
{
    cudaGetLastError();   // reported here: a later launch's check must not find it again
    return std::string(what) + ": " + cudaGetErrorString(e);
}

mc_status status_from_device(int ds)
{
    switch (ds) {
    case DS_OK: return MC_OK;
    case DS_OVERFLOW: return MC_ERR_OVERFLOW;
    case DS_LOST: return MC_ERR_LOST;
    case DS_TIMEOUT: return MC_ERR_TIMEOUT;
    case DS_NAN: return MC_ERR_NAN;
    default: return MC_ERR_CUDA;
    }
}

const char *device_status_text(int ds)
{
    switch (ds) {
    case DS_LOST: return "a particle was lost (no cell contains it)";
    case DS_OVERFLOW: return "split stack or filter buffer overflow";
    case DS_TIMEOUT:
        return "a particle exceeded the event limit, a history its particle limit, or the free-gas loop its "
               "candidate limit";
    case DS_NAN: return "a non-finite track length, energy or weight";
    default: return "device error status";
    }
}

bool devbuf_reserve(DevBuf &buf, size_t bytes)
{
    if (bytes <= buf.bytes && buf.ptr) return true;
    if (buf.ptr) cudaFree(buf.ptr);
    buf.ptr = nullptr;
    buf.bytes = 0;
    if (bytes == 0) bytes = 256;
    if (cudaMalloc(&buf.ptr, bytes) != cudaSuccess) {
        cudaGetLastError();
        buf.ptr = nullptr;
        return false;
    }
    buf.bytes = bytes;
    return true;
}

void devbuf_free(DevBuf &buf)
{
    if (buf.ptr) cudaFree(buf.ptr);
    buf.ptr = nullptr;
    buf.bytes = 0;
}

namespace {

// Packs host vectors into one staging buffer (256-byte aligned sections) and
// records where each lands so the device pointers can be patched in.
struct Packer {
    std::vector<char> buf;
    std::vector<std::pair<const void **, size_t>> fix;

    template <class T>
    void add(const std::vector<T> &v, const T **slot)
    {
        size_t off = (buf.size() + 255) & ~(size_t)255;
        buf.resize(off + std::max<size_t>(v.size() * sizeof(T), 8), 0);
        if (!v.empty()) std::memcpy(buf.data() + off, v.data(), v.size() * sizeof(T));
        fix.emplace_back(reinterpret_cast<const void **>(slot), off);
    }
};

}  // namespace

// Saved states are keyed by a fingerprint of the problem: FNV-1a over the
// reader's tables in this order, each at the next multiple of 256 bytes.  The
// order and padding are part of the file format.
uint64_t table_fingerprint(const Tables &t)
{
    uint64_t h = 0xCBF29CE484222325ULL;
    size_t at = 0;
    auto zeros = [&](size_t n) {
        at += n;
        while (n--) h *= 0x100000001B3ULL;
    };
    auto add = [&](const auto &v) {
        zeros((256 - at % 256) % 256);
        const unsigned char *b = reinterpret_cast<const unsigned char *>(v.data());
        const size_t bytes = v.size() * sizeof(v[0]);
        for (size_t i = 0; i < bytes; ++i) h = (h ^ b[i]) * 0x100000001B3ULL;
        at += bytes;
        if (bytes < 8) zeros(8 - bytes);      // (an empty table takes eight)
    };
    add(t.surf_type); add(t.surf_bc); add(t.surf_coef); add(t.cell_imp); add(t.cell_mat);
    add(t.cell_surf_off); add(t.cell_surf); add(t.cell_sense); add(t.cell_tl_off); add(t.cell_tl);
    add(t.cell_c_off); add(t.cell_c); add(t.surf_est_off); add(t.surf_est); add(t.mat_off); add(t.mat_nuc);
    add(t.mat_dens); add(t.nuc_kind); add(t.nuc_len); add(t.nuc_A); add(t.nuc_const); add(t.nuc_off);
    add(t.xs_E); add(t.xs_S); add(t.xs_C); add(t.xs_T); add(t.mg_total); add(t.mg_scatter);
    add(t.mg_scat_tot); add(t.mg_capture); add(t.est_score_off); add(t.score_kind); add(t.score_kernel);
    add(t.est_filt_off); add(t.filt_kind); add(t.filt_size); add(t.filt_grid_len); add(t.filt_grid_off);
    add(t.filt_grid); add(t.est_factor); add(t.est_factor_off); add(t.est_bin_off); add(t.src_pos);
    add(t.src_dir_par); add(t.src_e_par); add(t.src_cdf); add(t.src_cell); add(t.src_dir_kind);
    add(t.src_e_kind); add(t.src_group);
    return h;
}

mc_status device_problem_init(const Tables &t, DeviceProblem &d, std::string &err)
{
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        err = "no CUDA device available (the library has no CPU fallback)";
        return MC_ERR_CUDA;
    }
    cudaGetDevice(&d.device);
    cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, d.device);
    if ((e = cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking)) != cudaSuccess) {
        err = cuda_msg(e, "cudaStreamCreate");
        return MC_ERR_CUDA;
    }
    for (auto &ev : d.ev) cudaEventCreate(&ev);
    cudaEventCreate(&d.ev_end);

    DevTables &T = d.dt;
    T.n_surf = t.n_surf(); T.n_cell = t.n_cell(); T.n_mat = t.n_mat(); T.n_nuc = t.n_nuc();
    T.mg_groups = t.mg_groups; T.n_est = t.n_est(); T.n_src = t.n_src();
    T.n_bins = t.n_bins();
    T.wr = t.wr; T.ws = t.ws;
    T.comb_bank_max = t.comb_bank_max; T.comb_teeth = t.comb_teeth;
    Fp64Tables F;
    build_fp64_tables(t, F);
    T.any_time = F.any_time;
    Packer P;
    P.add(t.surf_type, &T.surf_type); P.add(t.surf_bc, &T.surf_bc); P.add(t.surf_coef, &T.surf_coef);
    P.add(t.cell_imp, &T.cell_imp); P.add(t.cell_mat, &T.cell_mat); P.add(t.cell_surf_off, &T.cell_surf_off);
    P.add(t.cell_surf, &T.cell_surf); P.add(t.cell_sense, &T.cell_sense);
    P.add(t.cell_tl_off, &T.cell_tl_off); P.add(t.cell_tl, &T.cell_tl);
    P.add(t.cell_c_off, &T.cell_c_off); P.add(t.cell_c, &T.cell_c);
    P.add(t.surf_est_off, &T.surf_est_off); P.add(t.surf_est, &T.surf_est);
    P.add(F.tl_pre, &T.cell_tl_pre); P.add(F.c_pre, &T.cell_c_pre); P.add(F.s_pre, &T.surf_est_pre);
    P.add(t.mat_off, &T.mat_off); P.add(t.mat_nuc, &T.mat_nuc); P.add(t.mat_dens, &T.mat_dens);
    P.add(F.nuc, &T.nuc); P.add(F.grid, &T.xs_grid); P.add(F.row, &T.xs_row); P.add(F.inv, &T.xs_inv);
    P.add(F.bkt, &T.xs_bkt); P.add(F.mg, &T.mg); P.add(F.mg_cum, &T.mg_cum);
    P.add(t.est_score_off, &T.est_score_off); P.add(t.score_kind, &T.score_kind);
    P.add(t.score_kernel, &T.score_kernel); P.add(t.est_filt_off, &T.est_filt_off);
    P.add(t.filt_kind, &T.filt_kind); P.add(t.filt_size, &T.filt_size); P.add(t.filt_grid_len, &T.filt_grid_len);
    std::vector<long long> fgo(t.filt_grid_off.begin(), t.filt_grid_off.end());
    P.add(fgo, &T.filt_grid_off);
    P.add(t.filt_grid, &T.filt_grid); P.add(t.est_factor, &T.est_factor); P.add(F.est_ifac, &T.est_ifac);
    P.add(F.est_time, &T.est_time);
    P.add(t.est_factor_off, &T.est_factor_off);
    std::vector<long long> ebo(t.est_bin_off.begin(), t.est_bin_off.end());
    P.add(ebo, &T.est_bin_off);
    P.add(t.src_pos, &T.src_pos); P.add(t.src_dir_par, &T.src_dir_par); P.add(t.src_e_par, &T.src_e_par);
    P.add(t.src_cdf, &T.src_cdf); P.add(t.src_cell, &T.src_cell); P.add(t.src_dir_kind, &T.src_dir_kind);
    P.add(t.src_e_kind, &T.src_e_kind); P.add(t.src_group, &T.src_group);

    d.blob_bytes = P.buf.size();
    if ((e = cudaMalloc(&d.blob, d.blob_bytes)) != cudaSuccess) { err = cuda_msg(e, "cudaMalloc(tables)"); return MC_ERR_NOMEM; }
    const size_t nb = (size_t)std::max<int64_t>(t.n_bins(), 1);
    const size_t stage = (d.blob_bytes + 255) & ~(size_t)255;
    if ((e = cudaHostAlloc(&d.h_blob, stage + kCtlBytes + 2 * nb * sizeof(double), cudaHostAllocDefault)) != cudaSuccess) {
        err = cuda_msg(e, "cudaHostAlloc(tables)");
        return MC_ERR_NOMEM;
    }
    d.h_stage = static_cast<char *>(d.h_blob) + stage;
    std::memcpy(d.h_blob, P.buf.data(), d.blob_bytes);
    for (auto &f : P.fix) *f.first = static_cast<const char *>(d.blob) + f.second;
    mc_status us = upload_tables(d, err);
    if (us != MC_OK) return us;

    d.tally_bytes = nb * (2 * sizeof(double) + 2 * kExactLimbs * sizeof(long long));
    if ((e = cudaMalloc(&d.tallies, d.tally_bytes)) != cudaSuccess) {
        err = cuda_msg(e, "cudaMalloc(tallies)");
        return MC_ERR_NOMEM;
    }
    d.d_sum = static_cast<double *>(d.tallies);
    d.d_sq = d.d_sum + nb;
    d.d_exact = reinterpret_cast<long long *>(d.d_sq + nb);
    d.ready = true;
    return reset_tallies(d, err);
}

void device_problem_free(DeviceProblem &d)
{
    if (d.stream) cudaStreamSynchronize(d.stream);
    event_state_free(d.ev_state);
    d.ev_state = nullptr;
    bank_state_free(d.bank_state);
    d.bank_state = nullptr;
    lr_scratch_free(d.lr);
    d.lr = nullptr;
    devbuf_free(d.hist); devbuf_free(d.stack); devbuf_free(d.digest); devbuf_free(d.misc);
    if (d.blob) cudaFree(d.blob);
    if (d.h_blob) cudaFreeHost(d.h_blob);
    if (d.tallies) cudaFree(d.tallies);
    for (auto &ev : d.ev) if (ev) cudaEventDestroy(ev);
    if (d.ev_end) cudaEventDestroy(d.ev_end);
    if (d.stream) cudaStreamDestroy(d.stream);
    d = DeviceProblem();
}

mc_status upload_tables(DeviceProblem &d, std::string &err)
{
    cudaError_t e;
    if ((e = cudaMemcpyAsync(d.blob, d.h_blob, d.blob_bytes, cudaMemcpyHostToDevice, d.stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(d.stream)) != cudaSuccess) {
        err = cuda_msg(e, "upload tables");
        return MC_ERR_CUDA;
    }
    return MC_OK;
}

cudaError_t upload_tables_async(DeviceProblem &d, cudaStream_t st)
{
    return cudaMemcpyAsync(d.blob, d.h_blob, d.blob_bytes, cudaMemcpyHostToDevice, st);
}

cudaError_t reset_tallies_async(DeviceProblem &d, cudaStream_t st)
{
    if (!d.tallies) return cudaErrorInvalidValue;   // the problem was not loaded (no bytes to clear would be no error)
    const cudaError_t e = cudaMemsetAsync(d.tallies, 0, d.tally_bytes, st);
    if (e != cudaSuccess) return e;
    tallies_were_reset(d);
    return cudaSuccess;
}

void tallies_were_reset(DeviceProblem &d)
{
    d.exact_valid = true;
    d.histories = 0;
    d.ntrack = 0;
}

mc_status reset_tallies(DeviceProblem &d, std::string &err)
{
    cudaError_t e = reset_tallies_async(d, d.stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(d.stream);
    if (e != cudaSuccess) {
        err = cuda_msg(e, "reset tallies");
        return MC_ERR_CUDA;
    }
    return MC_OK;
}

mc_status read_bins(const DeviceProblem &d, size_t from, size_t count, double *out, std::string &err)
{
    if (count == 0) return MC_OK;
    if (!d.tallies) { err = "read tallies: problem was not loaded"; return MC_ERR_CUDA; }
    const size_t pitch = (size_t)((const char *)d.d_sq - (const char *)d.d_sum), width = count * sizeof(double);
    std::lock_guard<std::mutex> lk(*d.stage_mu);
    cudaError_t e;
    if ((e = cudaMemcpy2DAsync(d.h_stage + kCtlBytes, width, d.d_sum + from, pitch, width, 2, cudaMemcpyDeviceToHost,
                               d.stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(d.stream)) != cudaSuccess) {
        err = cuda_msg(e, "read tallies");
        return MC_ERR_CUDA;
    }
    std::memcpy(out, d.h_stage + kCtlBytes, 2 * width);
    return MC_OK;
}

mc_status read_sums(const DeviceProblem &d, std::vector<double> &sum, std::vector<double> &sq, std::string &err)
{
    const size_t nb = (size_t)std::max<long long>(d.dt.n_bins, 1);
    std::vector<double> both(2 * nb);
    const mc_status st = read_bins(d, 0, nb, both.data(), err);
    if (st != MC_OK) return st;
    sum.assign(both.begin(), both.begin() + nb);
    sq.assign(both.begin() + nb, both.end());
    return MC_OK;
}

mc_status run_histories(const Tables &t, DeviceProblem &d, uint64_t first, uint64_t n, uint64_t seed,
                        mc_mode mode, const mc_tune *tune, std::string &err)
{
    std::memset(&d.last, 0, sizeof(d.last));
    if (n == 0) return MC_OK;
    if (mode == MC_MIXED_EVENT) return run_event(t, d, first, n, seed, tune, err);
    return run_fp64(t, d, first, n, seed, mode == MC_FP64_REPLAY, tune, err);
}

mc_status run_fp64(const Tables &t, DeviceProblem &d, uint64_t first, uint64_t n, uint64_t seed, bool replay,
                   const mc_tune *tune, std::string &err)
{
    const int block = (tune && tune->block) ? (int)tune->block : 128;
    if (block != 128) { err = "FP64 history kernels are built for 128-thread blocks"; return MC_ERR_ARG; }
    uint32_t depth = (tune && tune->stack_depth) ? tune->stack_depth : 32;
    // a combed bank holds `teeth` particles plus the split copies of one walk
    if (t.comb_teeth > 0 && !(tune && tune->stack_depth)) depth = std::max<uint32_t>(depth, (uint32_t)t.comb_teeth + 32);
    const bool want_digest = tune && tune->record_digests;
    const long long nb = std::max<long long>(d.dt.n_bins, 1);
    const uint64_t chunk = hist_chunk((uint64_t)nb, n, tune ? tune->chunk : 0);
    HistoryShape shape = history_fp64_shape(chunk, t.mg_groups > 0);
    if (tune && tune->grid_blocks) shape = {(int)tune->grid_blocks, 32};
    const int grid = shape.grid;
    const uint64_t threads = (uint64_t)grid * block;
    const uint64_t ld = hist_rows(chunk);
    if (!devbuf_reserve(d.hist, (size_t)ld * nb * sizeof(double)) ||
        !devbuf_reserve(d.stack, (size_t)threads * depth * fp64_particle_bytes()) ||
        !devbuf_reserve(d.misc, kCtlBytes) ||
        (want_digest && !devbuf_reserve(d.digest, (size_t)chunk * sizeof(uint64_t)))) {
        err = "cannot allocate FP64 scratch";
        return MC_ERR_NOMEM;
    }
    char *misc = static_cast<char *>(d.misc.ptr);
    unsigned long long *d_cnt = reinterpret_cast<unsigned long long *>(misc + kCtlCounters);
    int *d_status = reinterpret_cast<int *>(misc + kCtlStatus);
    unsigned int *d_next = reinterpret_cast<unsigned int *>(misc + kCtlNext);
    cudaError_t e;
    if ((e = cudaMemsetAsync(misc, 0, kCtlBytes, d.stream)) != cudaSuccess) {
        err = cuda_msg(e, "memset");
        return MC_ERR_CUDA;
    }
    if (want_digest) d.digests.assign(n, 0);
    else d.digests.clear();

    float t_transport = 0.f, t_fold = 0.f;
    uint32_t launches = 0;
    uint64_t unnormalized = 0;   // histories added to the exact sums since their carries were propagated
    // the exact sums stay valid only if this run completes
    const bool exact_was_valid = d.exact_valid;
    d.exact_valid = false;
    cudaEventRecord(d.ev[0], d.stream);
    for (uint64_t c0 = 0; c0 < n; c0 += chunk) {
        const uint32_t cn = (uint32_t)std::min<uint64_t>(chunk, n - c0);
        HistoryArgs A;
        A.first = first + c0;
        A.n = cn;
        A.seed = seed;
        A.hist = static_cast<double *>(d.hist.ptr);
        A.hist_ld = ld;
        A.stack = d.stack.ptr;
        A.stack_depth = depth;
        if (tune && tune->max_events) A.max_events = tune->max_events;
        A.counters = d_cnt;
        A.digest = want_digest ? static_cast<unsigned long long *>(d.digest.ptr) : nullptr;
        A.status = d_status;
        A.next = d_next;
        A.lanes = shape.lanes;
        if (c0 > 0 && (e = cudaMemsetAsync(d_next, 0, sizeof(unsigned int), d.stream)) != cudaSuccess) {
            err = cuda_msg(e, "memset");
            return MC_ERR_CUDA;
        }
        cudaEventRecord(d.ev[1], d.stream);
        if ((e = launch_history_fp64(d.dt, A, replay, grid, block, d.stream)) != cudaSuccess) {
            err = cuda_msg(e, "history kernel launch");
            return MC_ERR_CUDA;
        }
        cudaEventRecord(d.ev[2], d.stream);
        if ((replay && (e = launch_fold_ordered(A.hist, cn, ld, d.dt.n_bins, d.d_sum, d.d_sq, d.stream)) != cudaSuccess) ||
            (e = launch_fold_exact(A.hist, cn, ld, d.dt.n_bins, d.d_exact, replay ? nullptr : d.d_sum,
                                   replay ? nullptr : d.d_sq, d.stream)) != cudaSuccess) {
            err = cuda_msg(e, "fold kernel launch");
            return MC_ERR_CUDA;
        }
        launches += replay ? 3 : 2;
        // a limb absorbs 2^31 additions of 32-bit digits
        unnormalized += cn;
        if (unnormalized >= (1ull << 30)) {
            if ((e = launch_exact_normalize(d.d_exact, d.dt.n_bins, d.stream)) != cudaSuccess) {
                err = cuda_msg(e, "exact sums");
                return MC_ERR_CUDA;
            }
            unnormalized = 0;
            ++launches;
        }
        cudaEventRecord(d.ev[3], d.stream);
        if (want_digest && (e = cudaMemcpyAsync(d.digests.data() + c0, A.digest, cn * sizeof(uint64_t),
                                                cudaMemcpyDeviceToHost, d.stream)) != cudaSuccess) {
            err = cuda_msg(e, "digests");
            return MC_ERR_CUDA;
        }
        const bool last = c0 + chunk >= n;
        if (last) {
            if ((e = launch_exact_normalize(d.d_exact, d.dt.n_bins, d.stream)) != cudaSuccess) {
                err = cuda_msg(e, "exact sums");
                return MC_ERR_CUDA;
            }
            ++launches;
            cudaEventRecord(d.ev_end, d.stream);
        }
        if ((e = cudaMemcpyAsync(d.h_stage, misc, kCtlBytes, cudaMemcpyDeviceToHost, d.stream)) != cudaSuccess ||
            (e = cudaStreamSynchronize(d.stream)) != cudaSuccess) {
            err = cuda_msg(e, "history kernel");
            return MC_ERR_CUDA;
        }
        float a = 0.f, b = 0.f;
        cudaEventElapsedTime(&a, d.ev[1], d.ev[2]);
        cudaEventElapsedTime(&b, d.ev[2], d.ev[3]);
        t_transport += a;
        t_fold += b;
        int hs = 0;
        std::memcpy(&hs, d.h_stage + kCtlStatus, sizeof(hs));
        if (hs != DS_OK) {
            err = device_status_text(hs);
            if (hs == DS_OVERFLOW) err += " (raise mc_tune.stack_depth)";
            return status_from_device(hs);
        }
    }
    float total = 0.f;
    cudaEventElapsedTime(&total, d.ev[0], d.ev_end);
    unsigned long long cnt[kNumCounters];
    std::memcpy(cnt, d.h_stage + kCtlCounters, sizeof(cnt));
    mc_counters &L = d.last;
    L.flights = cnt[0]; L.collisions = cnt[1]; L.crossings = cnt[2]; L.tally_updates = cnt[3];
    L.particles = cnt[4]; L.splits = cnt[5]; L.xs_evals = cnt[6]; L.freegas_iters = cnt[7];
    L.nuc_lookups = cnt[8];
    L.histories = n;
    L.transport_ms = t_transport;
    L.fold_ms = t_fold;
    L.total_ms = total;
    L.launches = launches;
    d.histories += n;
    d.ntrack += L.flights;
    d.exact_valid = exact_was_valid;
    return MC_OK;
}

}  // namespace mc
