// As krylov_diag.cu, with fused multiply-adds and a reciprocal diagonal:
// TFLOWS_FP64_FMA and the mixed solves.
#define TFLOWS_KNS fma_diag
#define TFLOWS_FP64_RECIP_DIAG 1
#define TFLOWS_FOR_DIAG 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* fma_diag_kernel(KernelId id) {
    switch (id) {
        case KernelId::Cg: return (const void*)fma_diag::krylov_kernel<double, 0>;
        case KernelId::CgFused: return (const void*)fma_diag::krylov_kernel<double, 1>;
        case KernelId::CgNone: return (const void*)fma_diag::krylov_kernel<double, 5>;
        case KernelId::CgNoneFused: return (const void*)fma_diag::krylov_kernel<double, 6>;
        case KernelId::Cgs: return (const void*)fma_diag::krylov_kernel<double, 2>;
        case KernelId::BicgTrue: return (const void*)fma_diag::krylov_kernel<double, 3>;
        case KernelId::MixedRestart: return (const void*)fma_diag::mixed_kernel<0>;
        case KernelId::MixedReliable: return (const void*)fma_diag::mixed_kernel<1>;
        case KernelId::MixedApart: return (const void*)fma_diag::mixed_kernel<3>;
        case KernelId::MixedCgs: return (const void*)fma_diag::mixed_kernel<2>;
        case KernelId::BatchFp64: return (const void*)fma_diag::batch_kernel<0>;
        case KernelId::BatchReliable: return (const void*)fma_diag::batch_kernel<2>;
        default: return nullptr;
    }
}

}  // namespace tflows
