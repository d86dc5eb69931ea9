// As krylov_batch_fma.cu: batches of mixed solves.
#define TFLOWS_KNS fma_any
#define TFLOWS_FP64_RECIP_DIAG 1
#define TFLOWS_FOR_ANY 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* mixed_batch_kernel(KernelId id) {
    switch (id) {
        case KernelId::BatchMixed: return (const void*)fma_any::batch_kernel<1>;
        default: return nullptr;
    }
}

}  // namespace tflows
