// The batch kernel in reference arithmetic.
#define TFLOWS_KNS ref_any
#define TFLOWS_FOR_ANY 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* ref_batch_kernel(KernelId id) {
    switch (id) {
        case KernelId::BatchFp64: return (const void*)ref_any::batch_kernel<0>;
        default: return nullptr;
    }
}

}  // namespace tflows
