/*
 * mdrl_force_narrow.cu — the instantiations of the default tile's one-warp-per-unit kernel; a
 * translation unit of their own so that the sets compile in parallel.
 */
#include "mdrl_force_narrow.cuh"

namespace mdrl {

template narrow_fn pick_force_narrow<kDiffShift>(int, bool, bool, bool);
template narrow_fn pick_force_narrow<kDiffExact>(int, bool, bool, bool);

}  // namespace mdrl
