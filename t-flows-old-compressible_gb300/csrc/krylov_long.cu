// Solvers in reference arithmetic on rows longer than a hexahedron's.
#define TFLOWS_KNS ref_long
#define TFLOWS_FOR_LONG 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* ref_long_kernel(KernelId id) {
    switch (id) {
        case KernelId::Cg:
        case KernelId::CgFused: return (const void*)ref_long::krylov_kernel<double, 4>;
        case KernelId::Cgs: return (const void*)ref_long::krylov_kernel<double, 2>;
        default: return nullptr;
    }
}

}  // namespace tflows
