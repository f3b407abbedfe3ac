/*
 * mdrl_force_list_pairs.cu — the list force-kernel instantiations for a batch's replicas with fewer than 3 cells per axis whose edges all
 * exceed 2 rc (per-pair wrap); one
 * instantiation set per translation unit so that the sets compile in parallel.
 */
#include "mdrl_force_list.cuh"

namespace mdrl {

template list_fn pick_force_list<kDiffWrap, true>(int, bool, bool, bool, bool);

}  // namespace mdrl
