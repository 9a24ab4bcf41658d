// phase_loop_one_fp.cu -- the persistent phase loop for one graph, FP64 tables.
#define NIDO_LOOP_KERNELS
#include "phase_loop.cuh"

namespace nido {
template struct PhaseLoopKernel<false, false>;
}  // namespace nido
