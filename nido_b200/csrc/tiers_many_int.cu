// tiers_many_int.cu -- the move tier kernels for many graphs, integer tables.
#define NIDO_TIER_KERNELS
#include "move_tiers.cuh"

namespace nido {
template struct TierKernels<true, true, false>;
template struct TierKernels<true, true, true>;
}  // namespace nido
