// pe_kernels_lockstep.cu — the tail kernel with inline shadow rays (pe_integrator.cuh), compiled on their own.
#include "pe_integrator.cuh"

namespace pe {
#define PE_K(...) template __global__ void __VA_ARGS__ PE_TAIL_ARGS;
PE_LOCKSTEP_KERNELS(PE_K)
#undef PE_K
} // namespace pe
