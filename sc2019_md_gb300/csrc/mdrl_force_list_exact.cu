/*
 * mdrl_force_list_exact.cu — the list force-kernel instantiations for one system, the exact-difference rule; one
 * instantiation set per translation unit so that the sets compile in parallel.
 */
#include "mdrl_force_list.cuh"

namespace mdrl {

template list_fn pick_force_list<kDiffExact, false>(int, bool, bool, bool, bool);

}  // namespace mdrl
