// mc_event_mgx.cu -- the per-thread kernels (k_track) for multigroup problems with time filters
// or the particle comb.  Philox refills as in mc_event_mg.cu.
#define MC_EV_RNG_OUTLINE 1
#include "mc_event_kernels.cuh"

namespace mc {
namespace ev {

EvKernel pick_track_mgx(int minb, bool batch) { return pick_track<FL_MGX>(minb, batch); }

}  // namespace ev
}  // namespace mc
