// As krylov_box_batch.cu, with fused multiply-adds and a reciprocal diagonal:
// TFLOWS_FP64_FMA and the mixed solves.
#define TFLOWS_KNS fma_boxes
#define TFLOWS_FP64_RECIP_DIAG 1
#define TFLOWS_FOR_BOX_BATCH 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* fma_box_batch_kernel(KernelId id) {
    switch (id) {
        case KernelId::BatchFp64: return (const void*)fma_boxes::batch_kernel<0>;
        case KernelId::BatchReliable: return (const void*)fma_boxes::batch_kernel<2>;
        default: return nullptr;
    }
}

}  // namespace tflows
