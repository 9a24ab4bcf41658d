// phase_loop_many_fp.cu -- the persistent phase loop for many graphs, FP64 tables.
#define NIDO_LOOP_KERNELS
#include "phase_loop.cuh"

namespace nido {
template struct PhaseLoopKernel<true, false>;
}  // namespace nido
