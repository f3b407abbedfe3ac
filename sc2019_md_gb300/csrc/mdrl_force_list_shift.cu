/*
 * mdrl_force_list_shift.cu — the list force-kernel instantiations for one system, the per-unit shift of the reference's difference rule; one
 * instantiation set per translation unit so that the sets compile in parallel.
 */
#include "mdrl_force_list.cuh"

namespace mdrl {

template list_fn pick_force_list<kDiffShift, false>(int, bool, bool, bool, bool);

}  // namespace mdrl
