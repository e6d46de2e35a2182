// pe_kernels_full.cu — the full shading kernels (pe_integrator.cuh), compiled on their own.
#include "pe_integrator.cuh"

namespace pe {
#define PE_K(...) template __global__ void __VA_ARGS__ PE_SHADE_ARGS;
PE_FULL_KERNELS(PE_K)
#undef PE_K
} // namespace pe
