// As krylov_batch.cu, with fused multiply-adds and a reciprocal diagonal.
#define TFLOWS_KNS fma_any
#define TFLOWS_FP64_RECIP_DIAG 1
#define TFLOWS_FOR_ANY 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* fma_batch_kernel(KernelId id) {
    switch (id) {
        case KernelId::BatchFp64: return (const void*)fma_any::batch_kernel<0>;
        default: return nullptr;
    }
}

}  // namespace tflows
