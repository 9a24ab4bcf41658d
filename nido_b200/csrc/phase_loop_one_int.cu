// phase_loop_one_int.cu -- the persistent phase loop for one graph, integer tables.
#define NIDO_LOOP_KERNELS
#include "phase_loop.cuh"

namespace nido {
template struct PhaseLoopKernel<false, true>;
}  // namespace nido
