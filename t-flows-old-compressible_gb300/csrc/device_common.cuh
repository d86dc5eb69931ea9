// Device-side building blocks shared by the Krylov kernels (sm_103a).
//
// * memory-model helpers (relaxed / acquire / release accesses at gpu scope)
// * a grid barrier for persistent cooperative launches whose every wait is
//   bounded by the SM cycle counter and by a shared abort flag
// * value-as-flag cells for the sync-free triangular sweeps: a cell holds a
//   signalling-NaN sentinel until its producer stores the computed value
//   (arithmetic never yields a signalling NaN, so a stored result can never
//   be mistaken for the sentinel)
// * deterministic block and grid reductions (fixed summation tree)
#pragma once

#include "fp64_div.cuh"

#include <cstdint>
#include <cuda_runtime.h>

namespace tflows {

constexpr int kWarp = 32;

// ---- status codes (mirror include/tflows_krylov.h) -------------------------
enum : int {
    ST_OK = 0, ST_NOT_CONVERGED = 1, ST_BREAKDOWN = 2, ST_NONFINITE = 3,
    ST_TIMEOUT = 4, ST_BAD_INPUT = 5, ST_CUDA_ERROR = 6
};

// Exit kinds of the reference control flow (Process/CG.f90:69-72,105-108,255).
enum : int { EXIT_BNRM = 1, EXIT_INIRES = 2, EXIT_CONVERGED = 3, EXIT_MAXITER = 4,
             EXIT_ABORT = 5, EXIT_NONFINITE = 6 };

// Per-solve device record (one per system), written by block 0.
struct DevState {
    int status;
    int exit_kind;
    int iterations;      // reference-visible iteration count
    int inner_iters;     // mixed mode: total inner iterations
    int refinements;     // mixed mode: refinement steps
    int timeout_where;   // which wait timed out (diagnostics)
    double ini_res;
    double fin_res;
    double bnrm2;
    double group_ns;     // batched launches: the system's own solve time
    double pad[2];
};

// Nanosecond clock shared by all SMs (measurement only; waits use clock64).
__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Control block shared by all blocks of one persistent launch.
struct DevCtl {
    unsigned long long bar;  // monotonically increasing arrival counter; kBarAbort once aborted
    int status;              // first error status raised
    int where;
};

// Wait limits are measured in SM clock cycles (clock64: monotonic and local
// to the SM, unlike the host-synchronised %globaltimer); the host converts
// the limit in seconds with the device's highest SM clock, so the real limit
// is never shorter than requested.

__device__ __forceinline__ long long ld_relaxed_s64(const long long* p) {
    long long v;
    asm volatile("ld.relaxed.gpu.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int ld_relaxed_s32(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_s64(long long* p, long long v) {
    asm volatile("st.relaxed.gpu.global.s64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed_s32(int* p, int v) {
    asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_add_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Raise an abort: first status wins.  One bit of the barrier's counter ends
// every barrier, as it lifts the counter past any target, and every other wait,
// which polls the same word: a warp that has left a wait for it is met by a
// barrier that fails for its whole block.
constexpr unsigned long long kBarAbort = 1ull << 62;
__device__ __forceinline__ void raise_abort(DevCtl* c, int status, int where) {
    if (atomicCAS(&c->status, 0, status) == 0) c->where = where;
    atomicOr(&c->bar, kBarAbort);
}
__device__ __forceinline__ bool aborted(const DevCtl* c) {
    return (unsigned long long)ld_relaxed_s64(reinterpret_cast<const long long*>(&c->bar)) >= kBarAbort;
}

// ---- asynchronous copies global -> shared (per thread, in commit groups) ----------
__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
// 16 bytes through L2 only; both addresses 16-byte aligned.  (The predicates
// of these copies are part of the instruction: a branch around each of a few
// copies costs more than the copies.)
__device__ __forceinline__ void cp_async16(unsigned dst, const void* src, bool p = true) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t"
        "@q cp.async.cg.shared.global [%0], [%1], 16;\n\t}" ::"r"(dst), "l"(src), "r"((unsigned)p)
        : "memory");
}
// One value of 4 or 8 bytes, naturally aligned.
template <int BYTES>
__device__ __forceinline__ void cp_async(unsigned dst, const void* src, bool p) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t"
        "@q cp.async.ca.shared.global [%0], [%1], %2;\n\t}" ::"r"(dst), "l"(src), "n"(BYTES),
        "r"((unsigned)p)
        : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Waits until at most N of this thread's groups are in flight.
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ---- value-as-flag cells ------------------------------------------------------
template <typename T> struct Cell;
template <> struct Cell<double> {
    using bits_t = long long;
    static constexpr long long kSentinel = 0x7FF4242424242424LL;  // signalling NaN
    __device__ static __forceinline__ bits_t bits(double v) { return __double_as_longlong(v); }
    __device__ static __forceinline__ double value(bits_t b) { return __longlong_as_double(b); }
    __device__ static __forceinline__ bits_t load(const double* p) {
        return ld_relaxed_s64(reinterpret_cast<const long long*>(p));
    }
    __device__ static __forceinline__ void store(double* p, double v) {
        st_relaxed_s64(reinterpret_cast<long long*>(p), __double_as_longlong(v));
    }
    __device__ static __forceinline__ double sentinel() { return __longlong_as_double(kSentinel); }
};
template <> struct Cell<float> {
    using bits_t = int;
    static constexpr int kSentinel = 0x7FA42424;  // signalling NaN
    __device__ static __forceinline__ bits_t bits(float v) { return __float_as_int(v); }
    __device__ static __forceinline__ float value(bits_t b) { return __int_as_float(b); }
    __device__ static __forceinline__ bits_t load(const float* p) {
        return ld_relaxed_s32(reinterpret_cast<const int*>(p));
    }
    __device__ static __forceinline__ void store(float* p, float v) {
        st_relaxed_s32(reinterpret_cast<int*>(p), __float_as_int(v));
    }
    __device__ static __forceinline__ float sentinel() { return __int_as_float(kSentinel); }
};

// ---- reductions ---------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The block's shared scratch of publish: 3 values of 16 warps x 16 lanes.
__device__ __forceinline__ double* reduce_smem() {
    __shared__ double s[3 * 16 * 16];
    return s;
}

// Persistent-launch context kept in registers / shared memory of each block.
struct Grid {
    DevCtl* ctl;
    double* partials;   // [slots][nblocks]
    long long timeout_cyc;
    unsigned long long target;  // thread 0 only
    int nblocks;
    int wg;   // global warp index
    int nw;   // warps in the grid
    int lane;
    int tid;  // thread index within the group of blocks solving one system
    int nt;   // threads in the group
    int bid;  // block index within the group
    unsigned epoch;  // tiled IC sweeps: number of the current apply
    int stall;      // test hook: block 0 skips its first barrier arrival
};

// A "grid" here is the group of `nb` blocks (starting at block `b0` of the
// launch) that solves one system: barriers, partial sums and work
// distribution are all relative to the group, so one launch can carry many
// independent solves.
__device__ __forceinline__ void grid_init_group(Grid& g, DevCtl* ctl, double* partials,
                                                long long timeout_cyc, int b0, int nb) {
    g.ctl = ctl;
    g.partials = partials;
    g.timeout_cyc = timeout_cyc;
    g.target = 0;
    g.nblocks = nb;
    g.bid = blockIdx.x - b0;
    g.lane = threadIdx.x & 31;
    g.tid = g.bid * blockDim.x + threadIdx.x;
    g.nt = nb * blockDim.x;
    g.wg = g.tid >> 5;
    g.nw = g.nt >> 5;
    g.epoch = 0;
    g.stall = 0;
}

__device__ __forceinline__ void grid_init(Grid& g, DevCtl* ctl, double* partials,
                                          long long timeout_cyc) {
    grid_init_group(g, ctl, partials, timeout_cyc, 0, gridDim.x);
}

// Grid-wide barrier with release/acquire ordering (every write before the
// barrier is visible to every read after it).  Returns false when the
// launch was aborted (timeout or error raised anywhere).  The block's
// threads meet at __syncthreads, then thread 0 arrives with a release add
// and waits with acquire loads; the release is cumulative over the writes
// the block barrier ordered before it and the acquire orders every read
// after the closing block barrier, so no separate fence is needed (a fence
// on each side cost 0.9 us of a 6.6 us barrier with 304 blocks).
__device__ __forceinline__ bool grid_sync(Grid& g, int where) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        g.target += (unsigned long long)g.nblocks;
        if (g.stall && g.bid == 0) g.stall = 0;  // withheld: the barrier cannot complete
        else red_release_add_u64(&g.ctl->bar, 1ull);
        long long t0 = 0;
        unsigned spins = 0;
        unsigned long long v;
        while ((v = ld_acquire_u64(&g.ctl->bar)) < g.target) {
            if ((++spins & 255u) == 0u) {
                const long long t = clock64();
                if (t0 == 0) t0 = t;
                else if (t - t0 > g.timeout_cyc) raise_abort(g.ctl, ST_TIMEOUT, where);
            }
        }
        s_ok = v < kBarAbort;
    }
    __syncthreads();
    return s_ok != 0;
}

// Publish this block's K partial sums into slot range [slot, slot+K), K <= 3;
// the grid_sync that follows every publish orders the stores before its
// arrival.  GB300 does 2 FP64 additions per clock and SM, so a shuffle tree
// in every warp would hold the pipe for 80 cycles per warp and value: the
// lanes' values are halved once by shuffle, and one warp per value adds what
// the warps left in shared memory.  A reduction of three values with its
// barrier took 16.5 us with a tree per warp and one warp for all totals, and
// takes 9.1, in 608 blocks of 256 threads; 6.8 and 3.2 in 152.
template <int K>
__device__ __forceinline__ void publish(Grid& g, int slot, const double (&v)[K]) {
    constexpr int kHalf = kWarp / 2, kMaxWarps = 16;
    static_assert(K <= 3, "");
    double* const sm = reduce_smem();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double s = v[k] + __shfl_down_sync(0xffffffffu, v[k], kHalf);
        if (lane < kHalf) sm[(k * kMaxWarps + warp) * kHalf + lane] = s;
    }
    __syncthreads();
    for (int k = warp; k < K; k += nw) {
        // lane l adds entries l, l + 32, ...: two chains of at most four
        double a = 0.0, b = 0.0;
        const double* const p = sm + k * kMaxWarps * kHalf;
#pragma unroll
        for (int j = 0; j < kMaxWarps / 4; ++j) {
            const int e = j * 2 * kWarp + lane;
            if (e < nw * kHalf) a += p[e];
            if (e + kWarp < nw * kHalf) b += p[e + kWarp];
        }
        const double s = warp_sum(a + b);
        if (lane == 0) g.partials[(size_t)(slot + k) * g.nblocks + g.bid] = s;
    }
}

// After a grid_sync: every block computes the same K totals in the same
// order (deterministic), one warp per value, broadcast through shared memory
// together with what one thread derives from each: ext[k] = post(k, total).
// (A division or a square root by every thread would hold the FP64 pipe for
// some 160 cycles per warp, 2.6 us on an SM full of them.)
template <int K, typename Post>
__device__ __forceinline__ void totals(Grid& g, int slot, double (&res)[K], double (&ext)[K], Post post) {
    __shared__ double s_tot[K], s_ext[K];
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int k = warp; k < K; k += nw) {
        const long long* src =
            reinterpret_cast<const long long*>(g.partials + (size_t)(slot + k) * g.nblocks);
        // each lane's partials eight at a time: loads ahead of their sums,
        // summed as a tree
        double s = 0.0;
        for (int b0 = g.lane; b0 < g.nblocks; b0 += 32 * 8) {
            double w[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                w[u] = __longlong_as_double(b0 + 32 * u < g.nblocks ? ld_relaxed_s64(src + b0 + 32 * u) : 0);
            if (b0 - g.lane + 32 < g.nblocks) {
                if (b0 - g.lane + 128 < g.nblocks) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) w[u] += w[u + 4];
                }
                w[0] += w[2];
                w[1] += w[3];
                w[0] += w[1];
            }
            s += w[0];
        }
        s = warp_sum(s);
        if (g.lane == 0) {
            s_tot[k] = s;
            s_ext[k] = post(k, s);
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) {
        res[k] = s_tot[k];
        ext[k] = s_ext[k];
    }
    // no closing block barrier: the next write of s_tot comes after the
    // next grid_sync, whose opening __syncthreads every thread reaches after
    // reading these totals
}
template <int K>
__device__ __forceinline__ void totals(Grid& g, int slot, double (&res)[K]) {
    double ext[K];
    totals<K>(g, slot, res, ext, [](int, double) { return 0.0; });
}

// sqrt(t) < tol as a comparison of t: the least t whose (rounded, monotonic)
// square root is not below tol.  Set by one thread; lives in shared memory.
struct NormTest {
    double tol, least;
    bool direct;  // tol^2 is not a comfortable number: compare square roots
    __device__ void set(double tol_) {  // by one thread
        tol = tol_;
        direct = !(tol <= 0.0) && !(tol > 1e-140 && tol < 1e140);
        double t = 0.0;  // tol <= 0: no norm is below it
        if (tol > 0.0 && !direct) {
            t = tol * tol;
            while (sqrt(t) >= tol) t = __longlong_as_double(__double_as_longlong(t) - 1);
            while (sqrt(t) < tol) t = __longlong_as_double(__double_as_longlong(t) + 1);
        }
        least = t;
    }
    // t: a sum of squares (not negative, or not a number)
    __device__ bool below(double t) const { return direct ? sqrt(t) < tol : t < least; }
};

// A solver's scalars, one copy per block in shared memory.  Only the threads
// that form totals (lane 0 of a summing warp) read and write them between
// barriers; what every thread needs comes with the totals.
struct Scalars {
    double rho, rho_old;  // (r, z) of the current iteration and of the one before
    double beta;
    double rr;            // ||r||^2 at the end of the last iteration
    NormTest conv, refine;
};
__device__ __forceinline__ Scalars& scalars() {
    __shared__ Scalars s;
    return s;
}

}  // namespace tflows
