// mc_event_mgs.cu -- the per-thread kernels (k_track) for multigroup problems with estimators
// without records, and neither time filters nor the particle comb.  Philox refills as in mc_event_mg.cu.
#define MC_EV_RNG_OUTLINE 1
#include "mc_event_kernels.cuh"

namespace mc {
namespace ev {

EvKernel pick_track_mgs(int minb, bool batch) { return pick_track<FL_MGS>(minb, batch); }

}  // namespace ev
}  // namespace mc
