// pe_kernels_media.cu — the shading kernel of scenes with media or walks (pe_integrator.cuh),
// compiled on its own.
#include "pe_integrator.cuh"

namespace pe {
#define PE_K(...) template __global__ void __VA_ARGS__ PE_SHADE_ARGS;
PE_MEDIA_KERNELS(PE_K)
#undef PE_K
} // namespace pe
