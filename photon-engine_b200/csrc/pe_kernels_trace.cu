// pe_kernels_trace.cu — the closest-hit and any-hit kernels (pe_integrator.cuh), compiled on their own.
#include "pe_integrator.cuh"

namespace pe {
#define PE_K(...) template __global__ void __VA_ARGS__ PE_TRACE_ARGS;
PE_TRACE_KERNELS(PE_K)
#undef PE_K
#define PE_K(...) template __global__ void __VA_ARGS__ PE_BINARY_ARGS;
PE_BINARY_KERNELS(PE_K)
#undef PE_K
#define PE_K(...) template __global__ void __VA_ARGS__ PE_SHADOW_ARGS;
PE_SHADOW_KERNELS(PE_K)
#undef PE_K
} // namespace pe
