// mc_history.cu -- launches of the FP64 transport, and the replay mode's
// kernels (built with -fmad=false; the plain mode's are mc_history_plain.cu).
#include <algorithm>

#include "mc_fold.cuh"
#include "mc_history_kernels.cuh"

namespace mc {

void launch_history_plain(const DevTables &T, const HistoryArgs &A, int grid, int block, cudaStream_t st);

size_t fp64_particle_bytes() { return sizeof(PartD); }

// One FP64 instruction takes a scheduler's pipe 64 cycles and more, for one
// lane as for 32.  Few histories are therefore spread over all schedulers with
// as few lanes of a warp each (3,001 duct histories: 4.8 ms, in full warps 5.6
// ms); beyond one full warp per scheduler, CTAs are added until every history
// has a lane or the registers run out.
HistoryShape history_fp64_shape(uint64_t n, bool multigroup)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    sms = std::max(sms, 1);
    const uint64_t warps = (uint64_t)sms * (kBlock / 32);
    if (n <= warps) return {(int)std::max<uint64_t>(1, (n + 3) / 4), 1};
    if (n <= warps * 32) return {sms, (int)((n + warps - 1) / warps)};
    const uint64_t per_sm = (n + warps * 32 - 1) / (warps * 32);
    return {sms * (int)std::min<uint64_t>(per_sm, (uint64_t)ctas_per_sm(multigroup ? F_MG : F_CE)), 32};
}

cudaError_t launch_history_fp64(const DevTables &T, const HistoryArgs &A, bool replay, int grid, int block,
                                cudaStream_t st)
{
    if (A.n_params > 0 && (!replay || A.n_params > kMaxParams)) return cudaErrorInvalidValue;
    const long long cols = A.n_params > 0 ? T.n_bins * (1 + (long long)(A.n_cols > A.n_params ? A.n_cols : A.n_params))
                                          : T.n_bins;
    if (cols > 0) {
        const cudaError_t e = cudaMemsetAsync(A.hist, 0, (size_t)cols * A.hist_ld * sizeof(double), st);
        if (e != cudaSuccess) return e;
    }
    if (A.n_params > 0) {
        k_history_fp64<true, F_LR><<<grid, block, 0, st>>>(T, A);
    } else if (!replay) {
        launch_history_plain(T, A, grid, block, st);
    } else if (T.mg_groups > 0) {
        k_history_fp64<true, F_MG><<<grid, block, 0, st>>>(T, A);
    } else {
        k_history_fp64<true, F_CE><<<grid, block, 0, st>>>(T, A);
    }
    return cudaGetLastError();
}

cudaError_t launch_fold_ordered(const double *hist, uint32_t n, uint64_t ld, long long n_cols, double *sum,
                                double *sq, cudaStream_t st)
{
    if (n_cols <= 0 || n == 0) return cudaSuccess;
    k_fold_ordered<<<dim3((unsigned)n_cols, 2), kFoldThreads, 0, st>>>(hist, n, ld, sum, sq);
    return cudaGetLastError();
}

}  // namespace mc
