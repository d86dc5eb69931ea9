// Solvers in reference arithmetic with the diagonal or no preconditioner.
#define TFLOWS_KNS ref_diag
#define TFLOWS_FOR_DIAG 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* ref_diag_kernel(KernelId id) {
    switch (id) {
        case KernelId::Cg: return (const void*)ref_diag::krylov_kernel<double, 0>;
        case KernelId::CgFused: return (const void*)ref_diag::krylov_kernel<double, 1>;
        case KernelId::CgNone: return (const void*)ref_diag::krylov_kernel<double, 5>;
        case KernelId::CgNoneFused: return (const void*)ref_diag::krylov_kernel<double, 6>;
        case KernelId::Cgs: return (const void*)ref_diag::krylov_kernel<double, 2>;
        case KernelId::BicgTrue: return (const void*)ref_diag::krylov_kernel<double, 3>;
        case KernelId::BatchFp64: return (const void*)ref_diag::batch_kernel<0>;
        default: return nullptr;
    }
}

}  // namespace tflows
