// tiers_many_fp.cu -- the move tier kernels for many graphs, FP64 tables.
#define NIDO_TIER_KERNELS
#include "move_tiers.cuh"

namespace nido {
template struct TierKernels<true, false, false>;
template struct TierKernels<true, false, true>;
}  // namespace nido
