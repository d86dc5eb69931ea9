// FP64 kernels of the contracted build (TFLOWS_FP64_FMA) with tiled or
// Jacobi-sweep IC(0): the same solver code as krylov.cu, compiled with fused multiply-adds (--fmad=true) and a
// reciprocal diagonal for the Jacobi preconditioner -- the reference's
// recurrences with about half the FP64 instructions (GB300's FP64 pipe, not
// its memory, bounds the reference-arithmetic build); results differ from the
// reference's only by rounding.
#define TFLOWS_KNS fma
#define TFLOWS_FP64_RECIP_DIAG 1
#include "internal.h"
#include "solver_entry.cuh"

namespace tflows {

const void* fma_kernel(KernelId id) {
    switch (id) {
        case KernelId::Cg: return (const void*)fma::krylov_kernel<double, 0>;
        case KernelId::CgFused: return (const void*)fma::krylov_kernel<double, 1>;
        case KernelId::Cgs: return (const void*)fma::krylov_kernel<double, 2>;
        case KernelId::IcApply: return (const void*)fma::krylov_kernel<double, 8>;
        case KernelId::BatchFp64: return (const void*)fma::batch_kernel<0>;
        default: return nullptr;  // Prec1 (TFLOWS_FP64 semantics) lives in krylov.cu only
    }
}

}  // namespace tflows
