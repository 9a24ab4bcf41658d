// phase_loop_many_int.cu -- the persistent phase loop for many graphs, integer tables.
#define NIDO_LOOP_KERNELS
#include "phase_loop.cuh"

namespace nido {
template struct PhaseLoopKernel<true, true>;
}  // namespace nido
