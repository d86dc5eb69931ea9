// Solvers in reference arithmetic with level-ordered exact IC(0).
#define TFLOWS_KNS ref_level
#define TFLOWS_FOR_LEVEL 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* ref_level_kernel(KernelId id) {
    switch (id) {
        case KernelId::Cg: return (const void*)ref_level::krylov_kernel<double, 0>;
        case KernelId::CgFused: return (const void*)ref_level::krylov_kernel<double, 1>;
        case KernelId::Cgs: return (const void*)ref_level::krylov_kernel<double, 2>;
        case KernelId::IcApply: return (const void*)ref_level::krylov_kernel<double, 8>;
        default: return nullptr;
    }
}

}  // namespace tflows
