// tiers_one_fp.cu -- the move tier kernels for one graph, FP64 tables.
#define NIDO_TIER_KERNELS
#include "move_tiers.cuh"

namespace nido {
template struct TierKernels<false, false, false>;
template struct TierKernels<false, false, true>;
}  // namespace nido
