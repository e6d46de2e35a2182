// pe_kernels_tail_lean.cu — the tail kernels of lean-shading scenes (pe_integrator.cuh), compiled on their own.
#include "pe_integrator.cuh"

namespace pe {
#define PE_K(...) template __global__ void __VA_ARGS__ PE_TAIL_WARPS_ARGS;
PE_TAIL_WARPS_LEAN_KERNELS(PE_K)
#undef PE_K
} // namespace pe
