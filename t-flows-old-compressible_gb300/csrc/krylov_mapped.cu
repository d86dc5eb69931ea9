// Solvers in reference arithmetic with tiled IC(0) on boxes in other numberings.
#define TFLOWS_KNS ref_mapped
#define TFLOWS_FOR_MAPPED 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* ref_mapped_kernel(KernelId id) {
    switch (id) {
        case KernelId::Cg: return (const void*)ref_mapped::krylov_kernel<double, 0>;
        case KernelId::CgFused: return (const void*)ref_mapped::krylov_kernel<double, 1>;
        case KernelId::Cgs: return (const void*)ref_mapped::krylov_kernel<double, 2>;
        case KernelId::IcApply: return (const void*)ref_mapped::krylov_kernel<double, 8>;
        default: return nullptr;
    }
}

}  // namespace tflows
