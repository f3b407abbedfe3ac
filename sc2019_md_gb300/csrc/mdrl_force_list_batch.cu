/*
 * mdrl_force_list_batch.cu — the list force-kernel instantiations for the half-shell replicas of a batch (per-unit shift); one
 * instantiation set per translation unit so that the sets compile in parallel.
 */
#include "mdrl_force_list.cuh"

namespace mdrl {

template list_fn pick_force_list<kDiffShift, true>(int, bool, bool, bool, bool);

}  // namespace mdrl
