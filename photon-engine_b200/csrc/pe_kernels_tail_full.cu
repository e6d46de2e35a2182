// pe_kernels_tail_full.cu — the tail kernels of every other scene (pe_integrator.cuh), compiled on their own.
#include "pe_integrator.cuh"

namespace pe {
#define PE_K(...) template __global__ void __VA_ARGS__ PE_TAIL_WARPS_ARGS;
PE_TAIL_WARPS_FULL_KERNELS(PE_K)
#undef PE_K
} // namespace pe
