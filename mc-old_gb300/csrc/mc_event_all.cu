// mc_event_all.cu -- the per-thread kernels (k_track) for continuous-energy problems with time filters,
// estimators without records or the particle comb, and for batches that mix them with multigroup problems.
#include "mc_event_kernels.cuh"

namespace mc {
namespace ev {

EvKernel pick_track_all(int minb, bool batch) { return pick_track<FL_ALL>(minb, batch); }

}  // namespace ev
}  // namespace mc
