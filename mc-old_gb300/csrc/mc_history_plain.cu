// mc_history_plain.cu -- the plain mode's FP64 transport kernels.  They need not
// repeat the CPU's roundings: built with FMA contraction, a product and a sum
// are one instruction of the FP64 pipe that bounds them and one rounding
// instead of two (200,000 shield histories 33.2 -> 31.3 ms, 2,000,000 deep-slab
// histories 3.67 -> 3.44 ms).
#include "mc_history_kernels.cuh"

namespace mc {

void launch_history_plain(const DevTables &T, const HistoryArgs &A, int grid, int block, cudaStream_t st)
{
    if (T.mg_groups > 0) k_history_fp64<false, F_MG><<<grid, block, 0, st>>>(T, A);
    else k_history_fp64<false, F_CE><<<grid, block, 0, st>>>(T, A);
}

}  // namespace mc
