// pe_kernels_lean_out.cu — the per-key shading kernels of plain surface scenes that record AOVs or passes (pe_integrator.cuh),
// compiled on their own.
#include "pe_integrator.cuh"

namespace pe {
#define PE_K(...) template __global__ void __VA_ARGS__ PE_SHADE_ARGS;
PE_LEAN_KEYS(PE_SHADE_KEY, true)
#undef PE_K
} // namespace pe
