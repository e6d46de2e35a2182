// pe_kernels_lean_out.cu — the lean shading kernels that record AOVs and render passes (pe_integrator.cuh), compiled on their own.
#include "pe_integrator.cuh"

namespace pe {
#define PE_INSTANTIATE(...) template __global__ void __VA_ARGS__ PE_SHADE_ARGS;
PE_LEAN_OUT_KERNELS(PE_INSTANTIATE)
#undef PE_INSTANTIATE
} // namespace pe
