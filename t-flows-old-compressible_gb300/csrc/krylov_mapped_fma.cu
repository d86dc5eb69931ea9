// As krylov_mapped.cu, with fused multiply-adds and a reciprocal diagonal:
// TFLOWS_FP64_FMA and the mixed solves.
#define TFLOWS_KNS fma_mapped
#define TFLOWS_FP64_RECIP_DIAG 1
#define TFLOWS_FOR_MAPPED 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* fma_mapped_kernel(KernelId id) {
    switch (id) {
        case KernelId::Cg: return (const void*)fma_mapped::krylov_kernel<double, 0>;
        case KernelId::CgFused: return (const void*)fma_mapped::krylov_kernel<double, 1>;
        case KernelId::Cgs: return (const void*)fma_mapped::krylov_kernel<double, 2>;
        case KernelId::IcApply: return (const void*)fma_mapped::krylov_kernel<double, 8>;
        case KernelId::MixedRestart: return (const void*)fma_mapped::mixed_kernel<0>;
        case KernelId::MixedReliable: return (const void*)fma_mapped::mixed_kernel<1>;
        case KernelId::MixedCgs: return (const void*)fma_mapped::mixed_kernel<2>;
        default: return nullptr;
    }
}

}  // namespace tflows
