// The mixed-precision CGS and batch kernels: as krylov_mixed.cu, in a unit of
// their own, so that the two compile side by side.
#define TFLOWS_KNS fma
#define TFLOWS_FP64_RECIP_DIAG 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* mixed_batch_kernel(KernelId id) {
    switch (id) {
        case KernelId::MixedCgs: return (const void*)fma::mixed_kernel<2>;
        case KernelId::BatchMixed: return (const void*)fma::batch_kernel<1>;
        default: return nullptr;
    }
}

}  // namespace tflows
