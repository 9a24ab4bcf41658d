// tiers_one_int.cu -- the move tier kernels for one graph, integer tables.
#define NIDO_TIER_KERNELS
#include "move_tiers.cuh"

namespace nido {
template struct TierKernels<false, true, false>;
template struct TierKernels<false, true, true>;
}  // namespace nido
