// The kernel of batches of boxes in reference arithmetic.
#define TFLOWS_KNS ref_boxes
#define TFLOWS_FOR_BOX_BATCH 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* ref_box_batch_kernel(KernelId id) {
    switch (id) {
        case KernelId::BatchFp64: return (const void*)ref_boxes::batch_kernel<0>;
        default: return nullptr;
    }
}

}  // namespace tflows
