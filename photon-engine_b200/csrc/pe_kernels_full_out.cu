// pe_kernels_full_out.cu — the full shading kernels that record AOVs and render passes (pe_integrator.cuh), compiled on their own.
#include "pe_integrator.cuh"

namespace pe {
#define PE_K(...) template __global__ void __VA_ARGS__ PE_SHADE_ARGS;
PE_FULL_OUT_KERNELS(PE_K)
#undef PE_K
} // namespace pe
