// Kernels of the mixed-precision solves (FP32 inner iterations, FP64
// refinement) with tiled or Jacobi-sweep IC(0), compiled with fused multiply-adds (--fmad=true) and a
// reciprocal diagonal; they make no bitwise claim.
#define TFLOWS_KNS fma
#define TFLOWS_FP64_RECIP_DIAG 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* mixed_kernel(KernelId id) {
    switch (id) {
        case KernelId::MixedRestart: return (const void*)fma::mixed_kernel<0>;
        case KernelId::MixedReliable: return (const void*)fma::mixed_kernel<1>;
        case KernelId::MixedCgs: return (const void*)fma::mixed_kernel<2>;
        case KernelId::BatchReliable: return (const void*)fma::batch_kernel<2>;
        default: return nullptr;
    }
}

}  // namespace tflows
