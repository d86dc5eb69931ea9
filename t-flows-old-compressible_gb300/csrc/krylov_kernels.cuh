// Persistent Krylov solvers (CG / CGS with diagonal or IC(0) preconditioning)
// for the T-FlowS compressed-row systems, in FP64 (reference arithmetic) or
// FP32 (inner solves of the mixed-precision refinement).
//
// Matrix storage on the device is SELL-32: the rows are cut into slices of
// 32 consecutive rows; within a slice entry t of row (32*s + lane) sits at
// soff[s] + 32*t + lane, so a warp reading entry t of its 32 rows touches
// 32 consecutive words.  Each row keeps its entries in the caller's stored
// order, so every per-row sum runs left to right exactly as the reference's
// loops do (Process/CG.f90:193-199, Resid.f90:28-33); padding slots carry
// column -1 and are skipped.  In the reference-arithmetic build (--fmad=false)
// every a*b+c is a rounded product followed by a rounded sum, as in the
// reference; the contracted build fuses them (solver_entry.cuh).
//
// One cooperative launch runs a whole solve.  Phases are separated by the
// bounded grid barrier of device_common.cuh; the three scalar all-reduces
// per iteration of the reference (glosum, Parallel/Double/GloSum.f90:20-28)
// become block partial sums combined in a fixed order by every block, so
// alpha, beta and the convergence test never leave the device.
//
// IC(0) preconditioning (Process/Prec1.f90:51-59 and CG.f90:135-156) runs as
// sync-free triangular sweeps: rows are visited in wavefront-level order
// (levels padded to whole warps, so no warp waits on itself) and each row
// waits only for the specific earlier rows it reads, through value-as-flag
// cells.  Rows therefore combine the same operands in the same order as the
// sequential sweep: the preconditioner output is bit-identical to it.
#pragma once

#include "device_common.cuh"
#include "fp64_int.cuh"

#include <type_traits>

namespace tflows {

constexpr double kTiny = 1.0e-64;  // Library/allp_mod.f90:31
// TINY in the working precision: FP32 has no such number and 1e-64 rounds
// to zero there, so the FP32 inner solves divide by D itself.
template <typename T>
__device__ __forceinline__ T tiny_v() {
    if constexpr (sizeof(T) == 8) return T(kTiny);
    else return T(0);
}

// Reduction slots in the partials array (each slot = one value per block).
enum : int { SLOT_A = 0, SLOT_B = 4, SLOT_C = 8, SLOT_D = 12, NUM_SLOTS = 16 };

// Tiled IC(0) sweeps on a box (7-point stencil): numbered row = x + nx (y +
// ny z), or in any way that numbers a cell after its three neighbours before
// it along x, y and z, as the blocks of a block-structured mesh do (the
// sweeps' order of dependence is the same; `row` then leads from a cell to its
// row, and `ord` keeps the order of each row's sum).  A warp owns a patch of 8 x 4 columns of
// the box over all z, one column per lane, and walks the wavefront: at step s
// lane (mx, my) solves the cell z = s - mx - my of its column.  A tile is the
// patches of one block, at most two of them side by side in x.
// What a step reads -- the three factor entries and the pivot of 32 cells --
// is one contiguous record of the patch, records in step order.  The backward
// sweep runs the same code in mirrored coordinates (x, y, z and the lanes
// counted from the far end), with its own records.  Each sweeping warp has
// three more warps: one stages what it reads, one fetches its edges from
// other blocks, one drains what it writes.
constexpr int kPatchX = 8, kPatchY = 4;          // columns of a patch
constexpr int kSkew = kPatchX + kPatchY - 2;     // steps a patch takes beyond nz
constexpr int kTileK = 4;                        // steps per chunk (staging and hand-off unit)
constexpr int kRing = 32;                        // steps of the per-warp ring (power of two)
constexpr int kRowS = kPatchX + 1;               // elements of a ring slot: a column and
constexpr int kSlot = kRowS * (kPatchY + 1);     // a row more than the patch
constexpr int kWarpsPerPatch = 4;
constexpr int kMaxSweepWarps = 4;

// Chunks of records staged per patch, the one in use included.  Two more
// cover an L2 miss at FP64 step times; the BF16 records are small enough for
// a fourth within two blocks per SM.
__host__ __device__ constexpr int tile_stages(unsigned coef_bytes) { return coef_bytes == 2 ? 4 : 3; }

template <typename T>
struct Tiles {
    int on;            // 1: IC applies of this solve run the tiled sweeps
    int nx, ny, nz;    // box dimensions
    int sw;            // sweeping warps per block = patches per tile (1, 2 or 4)
    int ntx, nty;      // tiles along x and y
    int chunks;        // ceil((nz + kSkew) / kTileK)
    int lu_bf16;       // factor entries stored as BF16 bit patterns (FP32 solves)
    unsigned char* rec[2];   // forward / backward records, [patch][step]
    T* mid;                  // what the backward sweep starts from, [patch][step][lane]
    unsigned char* edge[2];  // forward / backward edge words, [patch][tile_edge_words]
    // A box in another numbering: the row of cell x + nx (y + ny z) (null: the
    // cell itself), and the order in which each row adds its three
    // neighbours, [patch][chunk][lane], one byte per step (reference
    // arithmetic; null: kBoxOrder)
    const int* row;
    unsigned* ord[2];
};
// Two bits per place: which of a record's entries is added first, second, third.
constexpr unsigned kBoxOrder = 0 | 1 << 2 | 2 << 4;
constexpr unsigned kBoxOrders = kBoxOrder * 0x01010101u;

// Edge words of a patch: per step of the reading patch its four edge cells
// along x, then the eight along y.
__host__ __device__ constexpr unsigned tile_edge_words(int chunks) {
    return (unsigned)chunks * kTileK * (kPatchX + kPatchY);
}

// Bytes of one record: three factor entries and the pivot of 32 cells.
__host__ __device__ constexpr unsigned tile_rec_bytes(unsigned coef_bytes, unsigned val_bytes) {
    return 32u * (3u * coef_bytes + val_bytes);
}
// An edge word: the value and the epoch it belongs to, 8 bytes per 32 bits of value.
__host__ __device__ constexpr unsigned tile_edge_bytes(unsigned val_bytes) { return 2u * val_bytes; }
// Shared memory of one sweeping warp: the ring, the staged records, the
// staged middle values.  Ring slot s holds what the lanes compute at step s,
// and the column and the row of the patches before it that step s + 1 reads.
__host__ __device__ constexpr unsigned tile_warp_smem(unsigned coef_bytes, unsigned val_bytes) {
    return kRing * kSlot * val_bytes +
           tile_stages(coef_bytes) * kTileK * (tile_rec_bytes(coef_bytes, val_bytes) + 32u * val_bytes);
}
__host__ __device__ constexpr unsigned tile_smem_bytes(int sw, unsigned coef_bytes, unsigned val_bytes) {
    return 128u + sw * tile_warp_smem(coef_bytes, val_bytes);
}

template <typename T>
struct Mat {
    int n;
    int nslices;
    const long long* __restrict__ soff;  // nslices + 1 slice offsets (elements)
    int width;                           // entries per row of every slice (0: they differ)
    int narrow;                          // 1: products by product_rows (FP32: no row has more than 8 entries)
    const int* __restrict__ scol;        // SELL column indices, -1 = padding
    // Column patterns (null when the topology has none): row i's entry t is
    // at column i + poff[8 * spat[i] + t], absent where that offset is
    // kNoCol (i + kNoCol < 0 for every row); the same columns as `scol`, in
    // the same order, read as one byte per row instead of four per entry.
    const unsigned char* __restrict__ spat;
    const int* __restrict__ poff;
    const T* __restrict__ sval;          // SELL values
    const int* __restrict__ meta;        // per row: length | diag slot << 16
    const int* __restrict__ perm_f;      // forward level order, 32-padded, -1 pads
    const int* __restrict__ perm_b;      // backward level order
    // BF16 copy of the SELL values (bit patterns), read by the IC sweeps in
    // place of `sval` when set (the off-diagonal factor entries)
    const unsigned short* __restrict__ lu16;
    int nchunk_f;
    int nchunk_b;
    int wide_f;  // chunks in the widest forward / backward level
    int wide_b;
    int sweep_mult;  // sweep warps per chunk of the widest level (0 = default)
    int sweep_sleep; // longest pause between polls of a sweep cell, ns (0: none)
    int sweep_gate;  // 1: a waiting warp polls one representative cell first
    Tiles<T> tile;   // tiled IC sweeps (tile.on = 0: level-ordered sweeps)
};

template <typename T>
struct Vecs {
    T* x;   // solution (in/out)
    T* r;   // in: right-hand side, out: final recursive residual
    T* p;   // search direction (CGS: p1)
    T* q;   // A p (CGS: q1)
    T* z;   // preconditioned residual (CG)
    T* w;   // IC forward-sweep cells (sentinel between sweeps)
    T* D;   // Prec1 output
    T* r2;  // CGS: shadow residual
    T* u1;
    T* u2;
    T* v2;
    T* p2;
    T* t;   // CGS: u1 + q1
    T* s;   // scratch of the Jacobi-sweep IC apply (FP32 inner solves)
};

struct SolveCfg {
    int method;     // 0 CG, 2 CGS (BiCG runs as CG)
    int prec;       // 1 diagonal, 2 IC(0), other = none
    int maxiter;
    double tol;     // absolute, compared as error < tol
    int x_is_zero;  // skip Resid's product (x0 = 0)
    int do_prec1;   // compute D (Prec1) in this launch
    int tol_is_relative;  // tol multiplies ||b||
    int ic_sweeps;  // prec 2: 0 = exact triangular sweeps, k > 0 = k Jacobi sweeps each
    int fuse_dir;   // FP64 CG: form the search direction inside the product
};

struct SolveOut {
    int exit_kind;
    int iterations;
    double ini_res;
    double fin_res;
    double bnrm2;
};

// Rows in SELL order: row i = 32*slice + lane (used by the matrix phases).
#define TF_FOR_ROWS(g, m, i)                                        \
    for (int s__ = (g).wg; s__ < (m).nslices; s__ += (g).nw)        \
        for (int i = s__ * kWarp + (g).lane, once__ = 1; once__; once__ = 0) \
            if (i < (m).n)

// Four consecutive rows per thread with 16-byte vector accesses (the vector
// phases).  Every work vector is padded to a multiple of 32 elements, so the
// group i..i+3 is in bounds; contributions of rows >= n are masked.
#define TF_FOR4(g, m, i) for (int i = 4 * (g).tid; i < (m).n; i += 4 * (g).nt)

template <typename T>
struct V4 {
    T a[4];
};
__device__ __forceinline__ V4<float> ld4(const float* p) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    return {{v.x, v.y, v.z, v.w}};
}
__device__ __forceinline__ void st4(float* p, const V4<float>& v) {
    *reinterpret_cast<float4*>(p) = make_float4(v.a[0], v.a[1], v.a[2], v.a[3]);
}
// Doubles as one 32-byte access: two of 16 bytes write every sector twice to
// L2 (a warp's 16-byte stores at a 32-byte stride fill half of each).
__device__ __forceinline__ V4<double> ld4(const double* p) {
    const double4_32a v = *reinterpret_cast<const double4_32a*>(p);
    return {{v.x, v.y, v.z, v.w}};
}
__device__ __forceinline__ void st4(double* p, const V4<double>& v) {
    *reinterpret_cast<double4_32a*>(p) = make_double4_32a(v.a[0], v.a[1], v.a[2], v.a[3]);
}

// Dot-product partials accumulate per thread in the working precision (FP64
// sums in FP64 mode; FP32 sums in the FP32 inner solves, where a per-element
// FP64 accumulation would load GB300's narrow FP64 pipe) and are combined
// across threads and blocks in FP64.
template <int K, typename T>
__device__ __forceinline__ void publish_t(Grid& g, int slot, const T (&v)[K]) {
    double d[K];
#pragma unroll
    for (int k = 0; k < K; ++k) d[k] = (double)v[k];
    publish<K>(g, slot, d);
}

// Jacobi step z = r / D.  The reference-arithmetic build keeps the
// reference's correctly rounded division; the contracted build
// (TFLOWS_FP64_RECIP_DIAG) and the FP32 inner solves hold 1/D and multiply.
#ifdef TFLOWS_FP64_RECIP_DIAG
constexpr bool kIntProducts = false;
constexpr bool kRecipDiag64 = true;
__device__ __forceinline__ double jacobi(double r, double dinv) { return r * dinv; }
#else
constexpr bool kRecipDiag64 = false;
constexpr bool kIntProducts = true;
__device__ __forceinline__ double jacobi(double r, double d) { return div_rn(r, d); }
#endif
__device__ __forceinline__ float jacobi(float r, float dinv) { return r * dinv; }

// What the unit's solvers are built for.  Code that a solve never runs costs
// the rest of its kernel registers (64 a thread, spilled beyond): with the
// products of long rows beside those of boxes a diagonal CG lost 2 to 5 %.
// Apart, against one kernel for everything, us per iteration: 64^3 diagonal in
// reference arithmetic 24.3 -> 23.0, multiply-adds 19.5 -> 18.5; 128^3 mixed
// diagonal 52.8 -> 50.8, with IC(0) 331 -> 323; 100 x 87 x 75 cells numbered in
// blocks, IC(0), reference arithmetic 576 -> 512, mixed 209 -> 198.
// * TFLOWS_FOR_DIAG: the diagonal or no preconditioner, short rows;
// * TFLOWS_FOR_LONG: those and Jacobi-sweep IC(0), long rows (product_columns);
// * TFLOWS_FOR_LEVEL: exact IC(0) by level-ordered sweeps, any rows;
// * TFLOWS_FOR_MAPPED: tiled IC(0) on boxes in other numberings;
// * TFLOWS_FOR_BOX_BATCH: the diagonal, tiled IC(0) on boxes in their own
//   numbering and Jacobi-sweep IC(0), short rows (batches of such systems);
// * TFLOWS_FOR_ANY: everything (batches of any others);
// * none of these: tiled IC(0) on boxes in their own numbering and Jacobi-sweep
//   IC(0), short rows.
#if defined(TFLOWS_FOR_DIAG)
constexpr bool kDiagPrec = true, kJacobiIc = false, kTiledIc = false, kLevelIc = false;
constexpr bool kShortRows = true, kLongRows = false;
#elif defined(TFLOWS_FOR_LONG)
constexpr bool kDiagPrec = true, kJacobiIc = true, kTiledIc = false, kLevelIc = false;
constexpr bool kShortRows = false, kLongRows = true;
#elif defined(TFLOWS_FOR_LEVEL)
constexpr bool kDiagPrec = false, kJacobiIc = false, kTiledIc = false, kLevelIc = true;
constexpr bool kShortRows = true, kLongRows = true;
#elif defined(TFLOWS_FOR_MAPPED)
constexpr bool kDiagPrec = false, kJacobiIc = false, kTiledIc = true, kLevelIc = false;
constexpr bool kShortRows = true, kLongRows = false;
#elif defined(TFLOWS_FOR_BOX_BATCH)
constexpr bool kDiagPrec = true, kJacobiIc = true, kTiledIc = true, kLevelIc = false;
constexpr bool kShortRows = true, kLongRows = false;
#elif defined(TFLOWS_FOR_ANY)
constexpr bool kDiagPrec = true, kJacobiIc = true, kTiledIc = true, kLevelIc = true;
constexpr bool kShortRows = true, kLongRows = true;
#else
constexpr bool kDiagPrec = false, kJacobiIc = true, kTiledIc = true, kLevelIc = false;
constexpr bool kShortRows = true, kLongRows = false;
#endif
// (batches keep the direction inside the product on any rows)
constexpr bool kApart = kLongRows && !(kDiagPrec && kLevelIc);
__device__ __forceinline__ int prec_of(int prec) {
    if (!kDiagPrec) return 2;
    if (!kJacobiIc && !kTiledIc && !kLevelIc) return prec == 1 ? 1 : 0;
    return prec == 1 || prec == 2 ? prec : 0;
}

__device__ __forceinline__ double divide(double a, double b) { return div_rn(a, b); }
__device__ __forceinline__ float divide(float a, float b) { return a / b; }

// Offset marking an absent entry of a column pattern: patterns are built
// only for fewer than 2^30 rows, so i + kNoCol is negative for every row.
constexpr int kNoCol = -(1 << 30);

// The first 8 column indices of row i = 32*s + lane of a slice of width
// w <= 8 (negative where the row has no entry): from the row's column
// pattern (two 16-byte loads of a table that stays in L1, one add per
// entry) when the topology has patterns, else from the SELL column array.
template <typename T>
__device__ __forceinline__ void sell_cols8(const Mat<T>& m, int s, int lane, int w, long long b0,
                                          int (&c)[8]) {
    if (m.spat) {
        const int i = s * kWarp + lane;
        const int4* po = reinterpret_cast<const int4*>(m.poff) + 2 * (int)m.spat[i];
        const int4 a = __ldg(po), b = __ldg(po + 1);
        c[0] = i + a.x;
        c[1] = i + a.y;
        c[2] = i + a.z;
        c[3] = i + a.w;
        c[4] = i + b.x;
        c[5] = i + b.y;
        c[6] = i + b.z;
        c[7] = i + b.w;
    } else {
        const int* cp = m.scol + b0 + lane;
#pragma unroll
        for (int t = 0; t < 8; ++t) c[t] = t < w ? cp[32 * t] : -1;
    }
}

// FP32 products in difference form.  The FP32 copy of a matrix keeps its
// off-diagonal entries rounded to FP32 but holds, in the diagonal slot, the
// row sum c_i (summed in FP64, then rounded); a product is then formed as
//     q_i = c_i x_i + sum_{j != i} a_ij (x_j - x_i),
// the same number in exact arithmetic.  Rounding each entry separately would
// perturb every row sum by ~6e-8 |a_ii|; for the pressure-correction
// operator -- a graph Laplacian whose rows sum to zero except at Dirichlet
// cells -- that shifts the smallest eigenvalues, so FP32 inner CG iterations
// converge towards a different operator and each FP64 refinement pays for
// it (measured: 112 instead of 84 iterations at 24^3; reliable updates
// stalling at 256^3).  In difference form the rounding error of a product
// scales with the variation of x, and the near null space of the operator
// (smooth x) is kept.  The FP64 matrices keep the reference's plain sums.
template <typename T>
__device__ __forceinline__ T diff_term(T a, T xj, T xi, bool diag) {
    return diag ? a * xi : a * (xj - xi);
}

// q_i = sum_j a_ij x_j over row i = 32*s + lane, left to right from 0 (FP32:
// in difference form).  Rows of at most 8 stored entries (every hex or prism
// cell) take a fully unrolled path: all index and value loads issue before
// the gathers.
template <typename T, typename X>
__device__ __forceinline__ T sell_row(const Mat<T>& m, int s, int lane, const X* __restrict__ xv) {
    const long long b0 = m.soff[s];
    const int w = (int)((m.soff[s + 1] - b0) >> 5);
    const int* cp = m.scol + b0 + lane;
    const T* vp = m.sval + b0 + lane;
    const int i = s * kWarp + lane;
    T acc = T(0);
    if (w <= 8) {
        int c[8];
        T v[8], xx[8];
        sell_cols8(m, s, lane, w, b0, c);
#pragma unroll
        for (int t = 0; t < 8; ++t) v[t] = t < w ? vp[32 * t] : T(0);
#pragma unroll
        for (int t = 0; t < 8; ++t) xx[t] = c[t] >= 0 ? T(xv[c[t]]) : T(0);
        if constexpr (sizeof(T) == 4) {
            T xi = T(0);
#pragma unroll
            for (int t = 0; t < 8; ++t)
                if (c[t] == i) xi = xx[t];
#pragma unroll
            for (int t = 0; t < 8; ++t)
                if (c[t] >= 0) acc = acc + diff_term(v[t], xx[t], xi, c[t] == i);
            return acc;
        }
#pragma unroll
        for (int t = 0; t < 8; ++t)
            if (c[t] >= 0) acc = acc + v[t] * xx[t];
        return acc;
    }
    if constexpr (sizeof(T) == 4) {
        const T xi = i < m.n ? T(xv[i]) : T(0);
        for (int t = 0; t < w; ++t) {
            const int c = cp[32 * t];
            if (c >= 0) acc = acc + diff_term(vp[32 * t], T(xv[c]), xi, c == i);
        }
        return acc;
    }
    for (int t = 0; t < w; ++t) {
        const int c = cp[32 * t];
        if (c >= 0) acc = acc + vp[32 * t] * T(xv[c]);
    }
    return acc;
}

// a * b of a reference-arithmetic product: on the integer pipe in the build
// whose sums are separate (fp64_int.cuh), which the FP64 pipe bounds.
template <typename T>
__device__ __forceinline__ T prod(T a, T b) {
    if constexpr (sizeof(T) == 8 && kIntProducts) return mul_rn(a, b);
    else return a * b;
}

// q_i = sum_j a_ij (z_j + beta p_j): the product with the next search
// direction formed inside the gather (FP32 inner solves), so the update
// p = z + beta p needs no pass of its own and no grid barrier.  `first`:
// p = z.  The direction is formed with one fused multiply-add, exactly as
// the row's owner forms its own entry (fused_dir), so every product sees the
// same vector the iteration stores.
__device__ __forceinline__ float fused_dir(float z, float beta, float p, bool first) {
    return first ? z : __fmaf_rn(beta, p, z);
}
// FP64: z + beta p written as the separate update pass writes it, so each
// build (contracted or not) forms the same value either way.
__device__ __forceinline__ double fused_dir(double z, double beta, double p, bool first) {
    return first ? z : z + beta * p;
}

// Entries of a row loaded ahead of their use.  FP64: a hexahedron's row has
// seven (the FP64 pipe also does what a predicate turns off, so an eighth
// that no row has would cost as much as the others).  Longer rows:
// product_columns.
template <typename T>
constexpr int kRowAhead = sizeof(T) == 8 ? 7 : 8;

// ---- the phases of an iteration ------------------------------------------------
// They are inlined: as functions of their own they cost 30 us per iteration
// at 4.1 M rows (registers saved around each call go through L2, and their
// pointers lose the global address space).  The solver around them therefore
// keeps its scalars in shared memory (Scalars), so that a loop has nearly the
// whole register budget of 64.

// q = A p over this warp's slices; returns the thread's sum of w_i q_i.  With
// DIR the search direction is formed in the gather (p_i = z_i + beta p_i, or
// z_i when `first`), stored to pn, and takes the place of w: the same
// direction and the same q as a separate update pass followed by the
// product, bit for bit, with one vector pass and one grid barrier less.
// Bound by DRAM (FP32, and FP64 sums with fused multiply-adds on large
// systems) or by the FP64 pipe's 2 lanes per clock and SM (separate products
// and sums, of which the products go to the integer pipe).  The loads of a
// row's first entries are in flight before their first use, with the pattern
// of the next row, so that nothing waits twice; the values are streamed past
// L1, whose lines the gathers of neighbouring warps share.  Of a CG iteration
// on 161 x 150 x 170 cells (512 x 304 threads) against an explicit column per
// entry, an offset per slice, values through L1 and every FP64 operation on
// its pipe: FP64 322 -> 176 us (238 with the products on the FP64 pipe), fused
// multiply-adds 144 -> 132, FP32 105 -> 85.  Values staged through shared
// memory by asynchronous copies cost 7 % to 15 %: what they hold is taken from L1.
template <typename T, bool DIR, bool COLUMNS>
__device__ __forceinline__ T product_rows(const Mat<T>& m, int wg, int nw, const T* __restrict__ z,
                                            const T* __restrict__ p, T* __restrict__ pn, T* __restrict__ q,
                                            const T* __restrict__ w, T beta, bool first) {
    constexpr int kAhead = kRowAhead<T>;
    const int lane = threadIdx.x & 31, n = m.n, nslices = m.nslices;
    T sum = T(0);
    unsigned id = !COLUMNS && wg < nslices ? m.spat[wg * kWarp + lane] : 0;
    for (int s = wg; s < nslices; s += nw) {
        const int i = s * kWarp + lane;
        long long b0 = (long long)s * (kWarp * m.width);
        int ww = m.width;
        if (!ww) {
            b0 = m.soff[s];
            ww = (int)((m.soff[s + 1] - b0) >> 5);
        }
        T v[kAhead];
#pragma unroll
        for (int t = 0; t < kAhead; ++t) v[t] = t < ww ? __ldcs(m.sval + b0 + 32 * t + lane) : T(0);
        int c[kAhead];
        const unsigned pat = id;
        if (COLUMNS) {
#pragma unroll
            for (int t = 0; t < kAhead; ++t) c[t] = t < ww ? __ldcs(m.scol + b0 + 32 * t + lane) : -1;
        } else {
            const int4* const po = reinterpret_cast<const int4*>(m.poff) + 2 * pat;
            const int4 a = __ldg(po), b = __ldg(po + 1);
            id = s + nw < nslices ? m.spat[(s + nw) * kWarp + lane] : 0;
            c[0] = i + a.x; c[1] = i + a.y; c[2] = i + a.z; c[3] = i + a.w;
            c[4] = i + b.x; c[5] = i + b.y; c[6] = i + b.z;
            if (kAhead == 8) c[kAhead - 1] = i + b.w;
        }
        T xi = T(0);  // the row's own direction (FP32 and DIR)
        if ((DIR || sizeof(T) == 4) && i < n)
            xi = DIR ? fused_dir(z[i], beta, first ? T(0) : p[i], first) : p[i];
        T x[kAhead], acc = T(0);
#pragma unroll
        for (int t = 0; t < kAhead; ++t) {
            const T pt = c[t] >= 0 && !(DIR && first) ? p[c[t]] : T(0);
            x[t] = DIR ? (c[t] >= 0 ? fused_dir(z[c[t]], beta, pt, first) : T(0)) : pt;
        }
#pragma unroll
        for (int t = 0; t < kAhead; ++t)
            if (c[t] >= 0) {
                if constexpr (sizeof(T) == 4) acc = acc + diff_term(v[t], x[t], xi, c[t] == i);
                else acc = acc + (DIR ? v[t] * x[t] : prod(v[t], x[t]));
            }
        if constexpr (kAhead < 8) {
#pragma unroll 1
            for (int t = kAhead; t < ww; ++t) {
                const int j = COLUMNS ? m.scol[b0 + 32 * t + lane] : i + m.poff[8 * pat + t];
                if (j < 0) continue;
                T xt = first && DIR ? T(0) : p[j];
                if (DIR) xt = fused_dir(z[j], beta, xt, first);
                const T vt = m.sval[b0 + 32 * t + lane];
                acc = acc + (DIR ? vt * xt : prod(vt, xt));
            }
        }
        if (i < n) {
            q[i] = acc;
            if (DIR) pn[i] = xi;
            sum += (DIR ? xi : w[i]) * acc;
        }
    }
    return sum;
}

// The same for longer rows (explicit columns), eight entries loaded ahead of
// their use; not beside the loop above where registers count.  A CG iteration on 128^3 rows of 15 entries against one entry at a time, and
// against the form above in FP64: FP32 269 -> 92 us, multiply-adds 191 -> 124,
// reference arithmetic 228 -> 152; 64^3: 40 -> 24, 32.1 -> 29.3, 41.8 -> 35.1.
template <typename T, bool DIR>
__device__ __forceinline__ T columns_loop(const Mat<T>& m, int wg, int nw, const T* __restrict__ z,
                                          const T* __restrict__ p, T* __restrict__ pn, T* __restrict__ q,
                                          const T* __restrict__ w, T beta, bool first) {
    constexpr int kAhead = 8;
    const int lane = threadIdx.x & 31, n = m.n, nslices = m.nslices, width = m.width;
    const long long* __restrict__ const soff = m.soff;
    const int* __restrict__ const cols = m.scol;
    const T* __restrict__ const vals = m.sval;
    __builtin_assume(__isGlobal(p) && __isGlobal(q) && __isGlobal(cols) && __isGlobal(vals));
    if (DIR) __builtin_assume(__isGlobal(z) && __isGlobal(pn));
    else __builtin_assume(__isGlobal(w));
    T sum = T(0);
    for (int s = wg; s < nslices; s += nw) {
        const int i = s * kWarp + lane;
        const long long b0 = width ? (long long)s * (kWarp * width) : soff[s];
        const int ww = width ? width : (int)((soff[s + 1] - b0) >> 5);
        const int* const cp = cols + b0 + lane;
        const T* const vp = vals + b0 + lane;
        T xi = T(0), acc = T(0);  // xi: the row's own direction (FP32 and DIR)
        if ((DIR || sizeof(T) == 4) && i < n)
            xi = DIR ? fused_dir(z[i], beta, first ? T(0) : p[i], first) : p[i];
#pragma unroll 1
        for (int t0 = 0; t0 < ww; t0 += kAhead) {
            int c[kAhead];
            T v[kAhead], x[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                c[u] = t0 + u < ww ? __ldcs(cp + 32 * (t0 + u)) : -1;
                v[u] = t0 + u < ww ? __ldcs(vp + 32 * (t0 + u)) : T(0);
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const T pt = c[u] >= 0 && !(DIR && first) ? p[c[u]] : T(0);
                x[u] = DIR ? (c[u] >= 0 ? fused_dir(z[c[u]], beta, pt, first) : T(0)) : pt;
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (c[u] >= 0) {
                    if constexpr (sizeof(T) == 4) acc = acc + diff_term(v[u], x[u], xi, c[u] == i);
                    else acc = acc + (DIR ? v[u] * x[u] : prod(v[u], x[u]));
                }
        }
        if (i < n) {
            q[i] = acc;
            if (DIR) pn[i] = xi;
            sum += (DIR ? xi : w[i]) * acc;
        }
    }
    return sum;
}

template <typename T, bool DIR>
__device__ __noinline__ T product_columns(const Mat<T>& m, int wg, int nw, const T* z, const T* p, T* pn, T* q,
                                          const T* w, T beta, bool first) {
    return columns_loop<T, DIR>(m, wg, nw, z, p, pn, q, w, beta, first);
}

template <typename T, bool DIR>
__device__ __forceinline__ T product_phase(const Mat<T>& m, int wg, int nw, const T* z, const T* p, T* pn,
                                           T* q, const T* w, T beta, bool first) {
    if constexpr (!kShortRows) {
        return columns_loop<T, DIR>(m, wg, nw, z, p, pn, q, w, beta, first);
    } else {
        if constexpr (kLongRows) {
            if (!m.narrow) return product_columns<T, DIR>(m, wg, nw, z, p, pn, q, w, beta, first);
        }
        if (m.spat) return product_rows<T, DIR, false>(m, wg, nw, z, p, pn, q, w, beta, first);
        return product_rows<T, DIR, true>(m, wg, nw, z, p, pn, q, w, beta, first);
    }
}

// p = z + beta p, or z when `first` (CG.f90:178-187).
template <typename T>
__device__ __forceinline__ void direction_phase(int tid, int nt, int n, const T* __restrict__ z,
                                             T* __restrict__ p, T beta, bool first) {
    if (first) {
        for (int i = 4 * tid; i < n; i += 4 * nt) st4(p + i, ld4(z + i));
        return;
    }
    for (int i = 4 * tid; i < n; i += 4 * nt) {
        const V4<T> zz = ld4(z + i);
        V4<T> pp = ld4(p + i);
#pragma unroll
        for (int u = 0; u < 4; ++u) pp.a[u] = zz.a[u] + prod(beta, pp.a[u]);
        st4(p + i, pp);
    }
}

// x += alfa p, r -= alfa q (CG.f90:226-253), z = M^-1 r with the diagonal;
// the thread's sums of r r, r z and (with `count`) the entries of x and r
// that are numbers.
template <typename T>
struct Sums3 {
    T a[3];
};
template <bool COUNT, typename T>
__device__ __forceinline__ Sums3<T> update_loop(int tid, int nt, int n, T* __restrict__ x, T* __restrict__ r,
                                                const T* __restrict__ p, const T* __restrict__ q,
                                                const T* __restrict__ D, T* __restrict__ z, T alfa,
                                                bool diag) {
    Sums3<T> out;
    T rr_ = T(0), rz_ = T(0), cnt = T(0);
    for (int i = 4 * tid; i < n; i += 4 * nt) {
        V4<T> xx = ld4(x + i), rr = ld4(r + i);
        const V4<T> pp = ld4(p + i), qq = ld4(q + i);
        V4<T> dd, zz;
        if (diag) dd = ld4(D + i);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            xx.a[u] = xx.a[u] + prod(alfa, pp.a[u]);
            rr.a[u] = rr.a[u] - prod(alfa, qq.a[u]);
            if (diag) zz.a[u] = jacobi(rr.a[u], dd.a[u]);
            if (i + u < n) {
                rr_ += rr.a[u] * rr.a[u];
                if (diag) rz_ += rr.a[u] * zz.a[u];
                if (COUNT)
                    cnt += (xx.a[u] == xx.a[u] ? T(1) : T(0)) + (rr.a[u] == rr.a[u] ? T(1) : T(0));
            }
        }
        st4(x + i, xx);
        st4(r + i, rr);
        if (diag) st4(z + i, zz);
    }
    out.a[0] = rr_;
    out.a[1] = rz_;
    out.a[2] = cnt;
    return out;
}
template <typename T>
__device__ __noinline__ Sums3<T> update_count(int tid, int nt, int n, T* x, T* r, const T* p, const T* q,
                                              const T* D, T* z, T alfa, bool diag) {
    return update_loop<true>(tid, nt, n, x, r, p, q, D, z, alfa, diag);
}
template <typename T>
__device__ __forceinline__ Sums3<T> update_phase(int tid, int nt, int n, T* x, T* r, const T* p, const T* q,
                                                 const T* D, T* z, T alfa, bool diag, bool count) {
    if (count) return update_count(tid, nt, n, x, r, p, q, D, z, alfa, diag);
    return update_loop<false>(tid, nt, n, x, r, p, q, D, z, alfa, diag);
}

// r_i <- r_i - a_i1 x_1 - a_i2 x_2 - ... (Process/Resid.f90:28-33 order;
// FP32: r_i - (the difference-form product)).
template <typename T, typename X>
__device__ __forceinline__ T sell_resid_row(const Mat<T>& m, int s, int lane, T ri,
                                            const X* __restrict__ xv) {
    if constexpr (sizeof(T) == 4) return ri - sell_row(m, s, lane, xv);
    const long long b0 = m.soff[s];
    const int w = (int)((m.soff[s + 1] - b0) >> 5);
    const int* cp = m.scol + b0 + lane;
    const T* vp = m.sval + b0 + lane;
    if (w <= 8) {
        int c[8];
        T v[8], xx[8];
        sell_cols8(m, s, lane, w, b0, c);
#pragma unroll
        for (int t = 0; t < 8; ++t) v[t] = t < w ? vp[32 * t] : T(0);
#pragma unroll
        for (int t = 0; t < 8; ++t) xx[t] = c[t] >= 0 ? T(xv[c[t]]) : T(0);
#pragma unroll
        for (int t = 0; t < 8; ++t)
            if (c[t] >= 0) ri = ri - v[t] * xx[t];
        return ri;
    }
    for (int t = 0; t < w; ++t) {
        const int c = cp[32 * t];
        if (c >= 0) ri = ri - vp[32 * t] * T(xv[c]);
    }
    return ri;
}

// An off-diagonal factor entry for the IC sweeps: the BF16 copy when the
// matrix carries one (FP32 inner solves with ic_bf16), else the SELL value.
// BF16 -> FP32 is exact (the bit pattern shifted into the high half).
template <typename T>
__device__ __forceinline__ T lu_val(const Mat<T>& m, long long k) {
    if constexpr (sizeof(T) == 4) {
        if (m.lu16) return __uint_as_float((unsigned)m.lu16[k] << 16);
    }
    return m.sval[k];
}

template <typename T>
__device__ __forceinline__ T diag_value(const Mat<T>& m, int i) {
    const int dslot = m.meta[i] >> 16;
    return m.sval[m.soff[i >> 5] + (i & 31) + 32LL * dslot];
}

// ---- sync-free level-ordered sweeps ----------------------------------------
// Rows are visited in wavefront-level order in chunks of 32 rows of one
// level (levels padded to whole warps); warp w takes chunks w, w+nw, ... in
// increasing order.  A row waits only for the specific earlier rows it reads,
// through their value-as-flag cells; every index, coefficient and own-row
// operand is loaded before the first wait, so a row's critical path is one
// cell load per dependency.  A chunk only ever waits on rows of lower levels,
// which sit in chunks of lower index, so with all warps resident the sweep
// cannot deadlock.
constexpr int kSweepMax = 8;  // dependencies prefetched per row
// Warps taking part in a sweep: at most `per_chunk` (a tuning parameter,
// default 4) per chunk of the widest level, so that a warp's next chunk is
// only a few levels ahead of the front and its polls rarely spin long.
constexpr int kSweepWarpsPerChunk = 4;

__device__ __forceinline__ int sweep_warps(const Grid& g, int wide, int per_chunk) {
    const int want = max(1, wide * (per_chunk > 0 ? per_chunk : kSweepWarpsPerChunk));
    return want < g.nw ? want : g.nw;
}

// One chunk of a level-ordered sweep.  Each lane owns one row; every index,
// coefficient and own-row operand is loaded before the first poll.  The
// warp then polls its rows' not-yet-ready dependency cells together, and a
// lane computes and publishes its row as soon as its own dependencies are
// in, without waiting for the other lanes, so a level's rows become visible
// one handoff after their inputs rather than after the slowest lane of the
// chunk.  Rows with more than kSweepMax dependencies wait one cell at a time.
// KIND 0: forward  acc = rhs - sum a_t cell_t,   result = acc * D_row
// KIND 1: backward acc = mid - sum a_t cell_t,   result = acc * D_row
// KIND 2: pivots   acc = a_ii - sum cell_t a_t a_t, result = 1 / acc
template <int KIND, typename T, typename Pub>
__device__ __forceinline__ bool sweep_chunk(const Grid& g, const Mat<T>& m, int row, int t0, int t1,
                                            long long base, T acc, T dmul, const T* cells,
                                            int where, Pub publish_row) {
    using C = Cell<T>;
    const int n = row >= 0 ? t1 - t0 : 0;
    const bool longrow = n > kSweepMax;  // rare: walked with a cursor instead
    int c[kSweepMax];
    T a[kSweepMax], v[kSweepMax];
    unsigned pending = 0;
#pragma unroll
    for (int u = 0; u < kSweepMax; ++u) {
        const bool use = !longrow && u < n;
        c[u] = use ? m.scol[base + 32LL * (t0 + u)] : 0;
        a[u] = use ? lu_val(m, base + 32LL * (t0 + u)) : T(0);
        v[u] = T(0);
        if (use) pending |= 1u << u;
    }
    int cursor = t0;
    bool done = row < 0;
    // Gate: while the chunk's inputs are far from ready, one lane polls one
    // representative cell (its dependency nearest in row order: the last
    // lower entry forward, the first upper entry backward) instead of every
    // lane polling every cell; the whole warp polls once it is in.  This
    // keeps thousands of early warps from loading L2 with polls.
    int gate_lane = -1, gate_col = 0;
    if (m.sweep_gate) {
        int rc = 0;
#pragma unroll
        for (int u = 0; u < kSweepMax; ++u)
            if (KIND == 1 ? u == 0 : u == n - 1) rc = c[u];
        const unsigned has = __ballot_sync(0xffffffffu, !longrow && n > 0);
        gate_lane = has ? __ffs(has) - 1 : -1;
        gate_col = __shfl_sync(0xffffffffu, rc, gate_lane < 0 ? 0 : gate_lane);
    }
    bool gated = gate_lane >= 0;
    const long long start = clock64();
    unsigned spins = 0;
    while (true) {
        if (gated) {
            int ready = 0;
            if (g.lane == gate_lane) ready = C::load(cells + gate_col) != C::kSentinel;
            gated = !__shfl_sync(0xffffffffu, ready, gate_lane);
        }
        if (!done && !gated) {
            if (longrow) {
                while (cursor < t1) {
                    const auto b = C::load(cells + m.scol[base + 32LL * cursor]);
                    if (b == C::kSentinel) break;
                    const T av = lu_val(m, base + 32LL * cursor);
                    const T vv = C::value(b);
                    acc = KIND == 2 ? acc - vv * av * av : acc - av * vv;
                    ++cursor;
                }
                if (cursor == t1) {
                    publish_row(KIND == 2 ? divide(T(1), acc) : acc * dmul);
                    done = true;
                }
            } else {
#pragma unroll
                for (int u = 0; u < kSweepMax; ++u) {
                    if (pending & (1u << u)) {
                        const auto b = C::load(cells + c[u]);
                        if (b != C::kSentinel) {
                            v[u] = C::value(b);
                            pending &= ~(1u << u);
                        }
                    }
                }
                if (!pending) {
                    // every input present: sum in slot order (the reference's order)
#pragma unroll
                    for (int u = 0; u < kSweepMax; ++u)
                        if (u < n) acc = KIND == 2 ? acc - v[u] * a[u] * a[u] : acc - a[u] * v[u];
                    publish_row(KIND == 2 ? divide(T(1), acc) : acc * dmul);
                    done = true;
                }
            }
        }
        if (__all_sync(0xffffffffu, done)) return true;
        // back off while the inputs are far from ready (a chunk several
        // levels ahead of the front), never more than m.sweep_sleep ns
        ++spins;
        if (m.sweep_sleep > 0 && spins > 4u)
            __nanosleep(min((unsigned)m.sweep_sleep, 8u << min(spins - 4u, 10u)));
        if ((spins & 63u) == 0u) {
            bool quit = aborted(g.ctl);
            if (!quit && clock64() - start > g.timeout_cyc) {
                raise_abort(g.ctl, ST_TIMEOUT, where);
                quit = true;
            }
            if (__any_sync(0xffffffffu, quit)) return false;
        }
    }
}

// ---- Prec1 -----------------------------------------------------------------
// prec 1: D_i = a_ii; prec 2: D_i = 1 / (a_ii - sum_{k<i} D_k a_ik a_ik);
// otherwise D_i = 1 (Process/Prec1.f90:45-67).  IC ends with a grid barrier.
template <typename T>
__device__ __noinline__ bool prec1_phase(Grid& g, const Mat<T>& m, T* D, int prec) {
    if (prec == 2) {
        TF_FOR_ROWS(g, m, i) { D[i] = Cell<T>::sentinel(); }
        if (!grid_sync(g, 10)) return false;
        bool ok = true;
        const int nws = sweep_warps(g, m.wide_f, m.sweep_mult);
        for (int ch = g.wg; g.wg < nws && ch < m.nchunk_f && ok; ch += nws) {
            const int row = m.perm_f[ch * kWarp + g.lane];
            int dslot = 0;
            long long base = 0;
            T aii = T(1);
            if (row >= 0) {
                dslot = m.meta[row] >> 16;
                base = m.soff[row >> 5] + (row & 31);
                aii = m.sval[base + 32LL * dslot];
            }
            ok = sweep_chunk<2>(g, m, row, 0, dslot, base, aii, T(1), D, 11,
                                [&](T d) { Cell<T>::store(D + row, d); });
        }
        const bool synced = grid_sync(g, 12);
        return ok && synced;
    }
    // with a reciprocal diagonal (contracted FP64 build) D holds 1 / a_ii
    TF_FOR_ROWS(g, m, i) {
        D[i] = (prec == 1) ? (sizeof(T) == 8 && kRecipDiag64 ? divide(T(1), diag_value(m, i))
                                                            : diag_value(m, i))
                           : T(1);
    }
    return true;  // made visible by the caller's next barrier
}

// What an IC apply does with each row of its result besides storing it:
// kRowNone nothing, kRowDot sums rhs_row z_row, kRowAxpy x_row += alfa z_row.
enum : int { kRowNone = 0, kRowDot = 1, kRowAxpy = 2 };
template <int OP, typename T>
struct RowOp {
    T alfa, *x;
    T dot;
    __device__ __forceinline__ void operator()(int row, T z, T rhs) {
        if (OP == kRowDot) dot += rhs * z;
        if (OP == kRowAxpy) x[row] = x[row] + alfa * z;
    }
};
template <typename T>
struct Applied {
    bool ok;
    T dot;
};

// ---- IC(0) apply -------------------------------------------------------------
// z = [(D~+U)^-1 D~ (D~+L)^-1] rhs with D~ = 1/D, computed as the reference
// does: forward w_i = D_i (rhs_i - sum_{k<i} a_ik w_k); middle
// w_i / (D_i + TINY); backward z_i = D_i (mid_i - sum_{k>i} a_ik z_k).
// `w` cells must hold the sentinel on entry and hold it again on exit.
// The backward phase runs `epi` (RowOp) per row.  Inlined, narrow levels took 2
// to 4 % longer in mixed precision and wide ones 4 % less.
template <typename T, typename Epi>
__device__ __noinline__ Applied<T> ic_apply(Grid& g, const Mat<T>& m, const T* D, const T* rhs, T* w, T* z,
                                            Epi epi) {
    bool ok = true;
    const int nwf = sweep_warps(g, m.wide_f, m.sweep_mult);
    for (int ch = g.wg; g.wg < nwf && ch < m.nchunk_f && ok; ch += nwf) {
        const int row = m.perm_f[ch * kWarp + g.lane];
        int dslot = 0;
        long long base = 0;
        T r0 = T(0), d = T(0);
        if (row >= 0) {
            dslot = m.meta[row] >> 16;
            base = m.soff[row >> 5] + (row & 31);
            r0 = rhs[row];
            d = D[row];
            z[row] = Cell<T>::sentinel();
        }
        ok = sweep_chunk<0>(g, m, row, 0, dslot, base, r0, d, w, 20,
                            [&](T val) { Cell<T>::store(w + row, val); });
    }
    if (!grid_sync(g, 21) || !ok) return {false, T(0)};
    const int nwb = sweep_warps(g, m.wide_b, m.sweep_mult);
    for (int ch = g.wg; g.wg < nwb && ch < m.nchunk_b && ok; ch += nwb) {
        const int row = m.perm_b[ch * kWarp + g.lane];
        int dslot = 0, len = 0;
        long long base = 0;
        T mid = T(0), d = T(0);
        if (row >= 0) {
            const int meta = m.meta[row];
            len = meta & 0xFFFF;
            dslot = meta >> 16;
            base = m.soff[row >> 5] + (row & 31);
            d = D[row];
            mid = divide(w[row], d + tiny_v<T>());
        }
        ok = sweep_chunk<1>(g, m, row, dslot + 1, row >= 0 ? len : dslot + 1, base, mid, d, z, 22,
                            [&](T zi) {
                                Cell<T>::store(z + row, zi);
                                w[row] = Cell<T>::sentinel();
                                epi(row, zi, rhs[row]);
                            });
    }
    return {ok, epi.dot};
}

// ---- IC(0) apply by Jacobi sweeps (FP32 inner solves, ic_sweeps = k > 0) ----
// Each triangular solve of the exact apply is replaced by k Jacobi sweeps
//     y^s_i = D_i (f_i - sum_{t in the triangle of row i} a_it y^(s-1)_t),
//     y^0   = D f,
// every sweep one fully parallel pass over one triangle (no waits between
// rows, a grid barrier between sweeps); the middle step y_i / (D_i + TINY)
// is folded into the last forward sweep.  For a symmetric matrix the
// backward sweeps are the transposes of the forward ones, so the operator is
// fixed and symmetric and CG stays valid; it tends to the exact IC(0) apply
// as k grows (after k = number of levels it is exact).
//
// One pass, bound by DRAM and L1/L2 latency.  What the loop reads of the grid
// and the matrix is taken into registers first (behind references it is read
// again after every store), in global space, with the next row's pattern and
// length a trip ahead; a row of a box has three entries in a triangle, so four
// are loaded together and a loop takes the rest (the FP64 pipe also does what
// a predicate turns off); LONG: four at a time, which costs a box 6 % (128^3
// rows of 15 entries, one sweep per triangle, mixed: 481 -> 262 us with the
// products of such rows).  FP32: a function of its own (inlined beside the tiled
// sweeps, 240^3 cells took 809 us per iteration, so 750; two sweeps 1383 and
// 1264).  A CG iteration with one / two sweeps per triangle, 161 x 150 x 170
// cells, against eight entries and explicit columns in 608 blocks of 256:
// FP32 269 -> 260 / 395 -> 389 us, multiply-adds 473 -> 361 / 670 -> 505.
constexpr int kTriAhead = 4;

template <bool FWD, bool LONG, typename T, typename Fin>
__device__ __forceinline__ void tri_jacobi(const Grid& g, const Mat<T>& m, const T* __restrict__ D,
                                           const T* __restrict__ f, const T* __restrict__ y,
                                           T* __restrict__ out, Fin fin) {
    const int n = m.n, nslices = m.nslices, wg = g.wg, nw = g.nw, lane = threadIdx.x & 31, width = m.width;
    const int* __restrict__ const metas = m.meta;
    const int* __restrict__ const cols = m.scol;
    const int* __restrict__ const offs = m.poff;
    const unsigned char* __restrict__ const pats = m.spat;
    const long long* __restrict__ const soff = m.soff;
    const T* __restrict__ const vals = m.sval;
    const unsigned short* __restrict__ const lu16 = m.lu16;
    auto value = [&](long long k) {
        if constexpr (sizeof(T) == 4) {
            if (lu16) return __uint_as_float((unsigned)lu16[k] << 16);
        }
        return vals[k];
    };
    __builtin_assume(__isGlobal(D) && __isGlobal(f) && __isGlobal(out) && __isGlobal(vals) && __isGlobal(metas));
    // (the next row's pattern and length are loaded a trip ahead)
    int i = wg * kWarp + lane;
    int meta_next = i < n ? metas[i] : 0;
    unsigned pat_next = pats && i < n ? pats[i] : 0;
    for (int s = wg; s < nslices; s += nw) {
        i = s * kWarp + lane;
        if (i >= n) continue;
        const int meta = meta_next, next = i + nw * kWarp;
        const int* const po = pats ? offs + 8 * pat_next : nullptr;
        if (next < n) {
            meta_next = metas[next];
            if (pats) pat_next = pats[next];
        }
        const int dslot = meta >> 16;
        const int t0 = FWD ? 0 : dslot + 1;
        const int nt = (FWD ? dslot : (meta & 0xFFFF)) - t0;
        const long long base = (width ? (long long)s * (kWarp * width) : soff[s]) + lane + 32LL * t0;
        auto column = [&](int u) { return po ? i + po[t0 + u] : cols[base + 32LL * u]; };
        T acc = f[i];
        const T di = D[i];
#pragma unroll 1
        for (int u0 = 0; u0 < (LONG ? nt : 1); u0 += kTriAhead) {
            int c[kTriAhead];
            T a[kTriAhead], yv[kTriAhead];
#pragma unroll
            for (int u = 0; u < kTriAhead; ++u) {
                c[u] = u0 + u < nt ? column(u0 + u) : 0;
                a[u] = u0 + u < nt ? value(base + 32LL * (u0 + u)) : T(0);
            }
#pragma unroll
            for (int u = 0; u < kTriAhead; ++u)
                yv[u] = u0 + u < nt ? (y ? y[c[u]] : D[c[u]] * f[c[u]]) : T(0);
#pragma unroll
            for (int u = 0; u < kTriAhead; ++u)
                if (u0 + u < nt) acc = acc - a[u] * yv[u];
        }
        if constexpr (!LONG) {
#pragma unroll 1
            for (int u = kTriAhead; u < nt; ++u) {
                const int j = column(u);
                acc = acc - value(base + 32LL * u) * (y ? y[j] : D[j] * f[j]);
            }
        }
        out[i] = fin(i, acc * di);
    }
}

// k forward sweeps ping-pong between w and s (the last one stores the middle
// vector), k backward sweeps between z and the other buffer, the last one
// into z with `epi` (RowOp) fused.  No barrier after the last sweep.
template <bool LONG, typename T, typename Epi>
__device__ __forceinline__ Applied<T> jacobi_apply(Grid& g, const Mat<T>& m, const T* D, const T* rhs, T* w, T* sb,
                                T* z, int k, Epi epi) {
    T* fb[2] = {w, sb};
    for (int sw = 1; sw <= k; ++sw) {
        const T* y = sw == 1 ? nullptr : fb[(sw - 1) & 1];
        T* o = fb[sw & 1];
        if (sw < k)
            tri_jacobi<true, LONG>(g, m, D, rhs, y, o, [](int, T v) { return v; });
        else
            tri_jacobi<true, LONG>(g, m, D, rhs, y, o, [&](int i, T v) { return v / (D[i] + tiny_v<T>()); });
        if (!grid_sync(g, 23)) return {false, T(0)};
    }
    const T* mid = fb[k & 1];
    T* bb[2] = {z, fb[(k + 1) & 1]};
    for (int sw = 1; sw <= k; ++sw) {
        const T* y = sw == 1 ? nullptr : bb[(k - sw + 1) & 1];
        T* o = bb[(k - sw) & 1];
        if (sw < k) {
            tri_jacobi<false, LONG>(g, m, D, mid, y, o, [](int, T v) { return v; });
            if (!grid_sync(g, 24)) return {false, T(0)};
        } else {
            tri_jacobi<false, LONG>(g, m, D, mid, y, o, [&](int i, T v) {
                epi(i, v, rhs[i]);
                return v;
            });
        }
    }
    return {true, epi.dot};
}
template <bool LONG, typename T, typename Epi>
__device__ __noinline__ Applied<T> jacobi_function(Grid& g, const Mat<T>& m, const T* D, const T* rhs, T* w, T* sb,
                                                   T* z, int k, Epi epi) {
    return jacobi_apply<LONG>(g, m, D, rhs, w, sb, z, k, epi);
}

// ---- tiled IC(0) sweeps (boxes) ------------------------------------------------
// Forward: row (x, y, z) needs (x, y, z-1), (x, y-1, z), (x-1, y, z), in the
// stored order of its lower entries (columns ascending, CG.f90:135-142).  The
// first is the lane's own last result, the other two lie in the step before
// of the patch's ring in shared memory, one lane or one row before; the
// ring's edge column and row belong to the patches beside it.  Backward mirrors it (x+1, y+1,
// z+1).  Each row combines the same operands in the same order as the
// sequential sweep (CG.f90:135-156), so in the reference-arithmetic build the
// result is bit-identical to it and to the level-ordered sweeps.
//
// The sweep is a chain of nx + ny + nz - 2 dependent cells, so the time of a
// step, not its bytes, bounds it.  Hence one warp per patch with no block
// barrier inside the sweep, and nothing but the cells' own arithmetic in that
// warp: per step it loads a record, the right-hand side and two neighbours
// from shared memory, at constant offsets from one ring position per chunk,
// and stores the result there, for its own next step and for the patches
// after it; cells outside the box compute 0, and chunks inside it skip the
// test.  Everything else is done by three more warps per patch: one stages
// records, right-hand side and middle values with asynchronous copies
// `tile_stages` chunks deep, one fetches the edges from other blocks, one
// drains the results, in z slabs that all lanes touch at the same z
// (coalesced), and publishes the edges for other blocks.  The warps hand over
// once per chunk of kTileK steps through progress counters in shared memory.
// Each of these loops is one warp's instruction latency, so they test with
// predicates rather than branches, and patches and chunks inside the box take
// paths without tests.  Edges between blocks are words in
// global memory that carry value and epoch in one 8-byte store, so that no
// fence and no reset is needed; a reader loads the words of the chunks ahead
// and polls (bounded) only those that were not there yet.
//
// Tiles are taken in increasing index forward and decreasing backward, each
// depending only on tiles before it, and all blocks are resident, so no
// sweep can deadlock; the backward sweep of a tile needs the forward sweep of
// that tile only, which the same warps ran, so no grid barrier separates the
// two.

// Edge words: relaxed 8-byte stores and loads at gpu scope, predicated.
__device__ __forceinline__ void st_word(unsigned char* p, unsigned long long w, bool on) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.relaxed.gpu.global.u64 [%0], %1;\n\t}" ::"l"(p),
        "l"(w), "r"((unsigned)on)
        : "memory");
}
__device__ __forceinline__ void ld_word(const unsigned char* p, unsigned long long& w, bool on) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.relaxed.gpu.global.u64 %0, [%1];\n\t}"
        : "+l"(w)
        : "l"(p), "r"((unsigned)on)
        : "memory");
}
template <typename T> struct EdgeWord;
template <> struct EdgeWord<float> {
    unsigned long long w = 0;
    __device__ static void store(unsigned char* p, float v, unsigned epoch, bool on) {
        st_word(p, (unsigned long long)__float_as_uint(v) << 32 | epoch, on);
    }
    __device__ void load(const unsigned char* p, bool on) { ld_word(p, w, on); }
    __device__ bool ready(unsigned epoch) const { return (unsigned)w == epoch; }
    __device__ float value() const { return __uint_as_float((unsigned)(w >> 32)); }
};
template <> struct EdgeWord<double> {
    unsigned long long h = 0, l = 0;
    __device__ static void store(unsigned char* p, double v, unsigned epoch, bool on) {
        const unsigned long long b = (unsigned long long)__double_as_longlong(v);
        st_word(p, (b & 0xffffffff00000000ull) | epoch, on);
        st_word(p + 8, b << 32 | epoch, on);
    }
    __device__ void load(const unsigned char* p, bool on) {
        ld_word(p, h, on);
        ld_word(p + 8, l, on);
    }
    __device__ bool ready(unsigned epoch) const {
        return (unsigned)h == epoch && (unsigned)l == epoch;
    }
    __device__ double value() const {
        return __longlong_as_double((long long)((h & 0xffffffff00000000ull) | l >> 32));
    }
};

// Record of one step for one lane: factor entries a[0..2] and the pivot d.
template <typename L, typename T> struct TileRec {  // FP32 / FP64 entries
    T a[3], d;
    __device__ __forceinline__ void load(const unsigned char* r, int lane) {
        if constexpr (sizeof(T) == 4) {
            const float4 v = reinterpret_cast<const float4*>(r)[lane];
            a[0] = v.x; a[1] = v.y; a[2] = v.z; d = v.w;
        } else {
            const double2 u = reinterpret_cast<const double2*>(r)[lane];
            const double2 v = reinterpret_cast<const double2*>(r + 512)[lane];
            a[0] = u.x; a[1] = u.y; a[2] = v.x; d = v.y;
        }
    }
    // where entry f (3: the pivot) of lane's cell sits in a record
    __host__ __device__ static constexpr unsigned at(int f, int lane) {
        return sizeof(T) == 4 ? 16u * lane + 4u * f : (f & 2 ? 512u : 0u) + 16u * lane + 8u * (f & 1);
    }
};
template <> struct TileRec<unsigned short, float> {  // BF16 entries, FP32 pivot
    float a[3], d;
    __device__ __forceinline__ void load(const unsigned char* r, int lane) {
        const uint2 v = reinterpret_cast<const uint2*>(r)[lane];
        const unsigned w = reinterpret_cast<const unsigned short*>(r + 256)[lane];
        a[0] = __uint_as_float(v.x << 16);
        a[1] = __uint_as_float(v.x & 0xffff0000u);
        a[2] = __uint_as_float(w << 16);
        d = __uint_as_float(v.y);
    }
    __host__ __device__ static constexpr unsigned at(int f, int lane) {
        return f == 3 ? 8u * lane + 4u : f == 2 ? 256u + 2u * lane : 8u * lane + 2u * f;
    }
};

// The contracted FP64 build scales the factor entries by the row's pivot, so
// that a step's chain is two multiply-adds instead of three and a product
// (an FP64 operation takes about 80 cycles here): forward w = D f - sum (D a)
// w, backward z = w - sum (D a) z, w itself being D times the middle value.
template <typename T> constexpr bool kScaledRec = sizeof(T) == 8 && kRecipDiag64;

// Patch `pt` of the tile grid (patch order within a tile: x first).
template <typename T>
__device__ __forceinline__ void patch_origin(const Tiles<T>& tl, int pt, int& x0, int& y0) {
    const int k = pt / tl.sw, w = pt % tl.sw, px = tl.sw > 1 ? 2 : 1;
    x0 = (px * (k % tl.ntx) + w % px) * kPatchX;
    y0 = (tl.sw / px * (k / tl.ntx) + w / px) * kPatchY;
}

// The cell of lane `lane` of a patch at step s in direction `dir`; false
// where there is none.
template <typename T>
__device__ __forceinline__ bool patch_cell(const Tiles<T>& tl, int dir, int x0, int y0, int s,
                                           int lane, int& x, int& y, int& z) {
    const int mx = lane % kPatchX, my = lane / kPatchX;
    z = s - mx - my;
    x = x0 + (dir ? kPatchX - 1 - mx : mx);
    y = y0 + (dir ? kPatchY - 1 - my : my);
    const bool in = x < tl.nx && y < tl.ny && z >= 0 && z < tl.nz;
    if (dir) z = tl.nz - 1 - z;
    return in;
}

// Tiles that block `bid` of a group of `nblocks` takes.
template <typename T>
__device__ __forceinline__ int tiles_of(const Tiles<T>& tl, int bid, int nblocks) {
    const int n = tl.ntx * tl.nty;
    return bid < n ? (n - 1 - bid) / nblocks + 1 : 0;
}

// Once per solve, before the first apply (a grid barrier must follow): the
// pivots into both record kinds, epoch 0 into every edge word.
template <typename T>
__device__ __noinline__ void tiles_init(Grid& g, const Mat<T>& m, const T* __restrict__ D) {
    const Tiles<T>& tl = m.tile;
    const unsigned cb = tl.lu_bf16 ? 2u : (unsigned)sizeof(T);
    const unsigned rec = tile_rec_bytes(cb, sizeof(T));
    const int sp = tl.chunks * kTileK, patches = tl.ntx * tl.nty * tl.sw;
    const long long total = (long long)patches * sp * 32;
    for (long long i = g.tid; i < total; i += g.nt) {
        const int lane = (int)(i & 31);
        const long long ps = i >> 5;
        const int s = (int)(ps % sp), pt = (int)(ps / sp);
        int x0, y0, x, y, z;
        patch_origin(tl, pt, x0, y0);
        for (int dir = 0; dir < 2; ++dir) {
            const bool in = patch_cell(tl, dir, x0, y0, s, lane, x, y, z);
            const unsigned at = cb == sizeof(T) ? TileRec<T, T>::at(3, lane)
                                                : TileRec<unsigned short, float>::at(3, lane);
            const int cell = x + tl.nx * (y + tl.ny * z);
            const T d = in ? D[tl.row ? tl.row[cell] : cell] : T(0);
            unsigned char* const r = tl.rec[dir] + ps * rec;
            *reinterpret_cast<T*>(r + at) = d;
            if constexpr (kScaledRec<T>)
                for (int f = 0; f < 3; ++f) *reinterpret_cast<T*>(r + TileRec<T, T>::at(f, lane)) *= d;
        }
    }
    const long long words = (long long)patches * tile_edge_words(tl.chunks) * (sizeof(T) / 4);
    for (int dir = 0; dir < 2; ++dir)
        for (long long i = g.tid; i < words; i += g.nt)
            reinterpret_cast<unsigned long long*>(tl.edge[dir])[i] = 0ull;
    g.epoch = 0;
}

// Progress counters in shared memory: chunks done in this apply.
__device__ __forceinline__ int progress_load(unsigned a) {
    int v;
    asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
// (by lane 0, after a __syncwarp that orders the other lanes' accesses)
__device__ __forceinline__ void progress_store(unsigned a, int v, int lane) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.eq.s32 q, %2, 0;\n\t@q st.release.cta.shared.s32 [%0], %1;\n\t}" ::"r"(a),
        "r"(v), "r"(lane)
        : "memory");
}

// The bounded wait of a warp: until ok() holds on every lane.  False: the
// launch is aborted.
template <typename Ok>
__device__ __forceinline__ bool tile_wait(DevCtl* ctl, long long limit, int where, Ok ok) {
    if (!__all_sync(0xffffffffu, ok())) {
        const long long t0 = clock64();
        unsigned spins = 0;
        do {
            if ((++spins & 63u) == 0u) {
                bool quit = aborted(ctl);
                if (!quit && clock64() - t0 > limit) {
                    raise_abort(ctl, ST_TIMEOUT, where);
                    quit = true;
                }
                if (__any_sync(0xffffffffu, quit)) return false;
            }
        } while (!__all_sync(0xffffffffu, ok()));
    }
    __syncwarp();
    return true;
}

// One sweep over this block's tiles, forward (BWD = 0) or backward.  Forward
// reads rhs and writes tl.mid; backward reads tl.mid and rhs and writes zout,
// with epi (RowOp) per row.  Not ok: a wait gave up (the launch is aborted).
template <int BWD, bool MAP, typename L, typename T, typename Epi>
__device__ __forceinline__ Applied<T> tile_sweep(DevCtl* ctl, long long limit, int bid, int nblocks,
                                              unsigned epoch, int first, const Mat<T>& m,
                                              const T* __restrict__ rhs, T* __restrict__ zout, Epi epi) {
    extern __shared__ __align__(128) unsigned char tf_smem[];
    const Tiles<T>& tl = m.tile;
    constexpr unsigned kRec = tile_rec_bytes(sizeof(L), sizeof(T));
    constexpr unsigned kChunkRec = kTileK * kRec;
    constexpr int kStages = tile_stages(sizeof(L));
    constexpr unsigned kEdge = tile_edge_bytes(sizeof(T));
    constexpr unsigned kWarpB = tile_warp_smem(sizeof(L), sizeof(T));
    constexpr int kDn = BWD ? -1 : 1;  // towards the patches after
    // A ring slot is filled again 32 steps on; staging runs ahead of its chunk
    // by the skew, draining a slab lags by it, so the drained chunk may be
    // this many behind the one filled.
    constexpr int kDrainLag = (kRing - kSkew) / kTileK - 1;
    constexpr int kNever = -(1 << 20);  // an offset that any progress meets
    const int lane = threadIdx.x & 31, sw = tl.sw, px = sw > 1 ? 2 : 1, swy = sw / px;
    // roles: 0 sweeps, 1 stages, 2 drains, 3 fetches edges
    const int wid = threadIdx.x >> 5, role = wid / sw, w = wid % sw;
    const int chunks = tl.chunks, nz = tl.nz;
    const int mine = tiles_of(tl, bid, nblocks);
    if (role >= kWarpsPerPatch) return {true, T(0)};
    const unsigned prog = smem_u32(tf_smem) + 4 * w;  // chunks swept, staged, drained, fetched
    const unsigned staged = prog + 4 * kMaxSweepWarps, drained = staged + 4 * kMaxSweepWarps,
                   fetched = drained + 4 * kMaxSweepWarps;
    T* const ring = reinterpret_cast<T*>(tf_smem + 128 + w * kWarpB);
    unsigned char* const s_rec = tf_smem + 128 + w * kWarpB + kRing * kSlot * sizeof(T);
    T* const s_mid = reinterpret_cast<T*>(s_rec + kStages * kChunkRec) + lane;
    const int mx = lane % kPatchX, my = lane / kPatchX, skew = mx + my;
    T* const own = ring + (my + 1) * kRowS + mx + 1;  // this lane's cell in slot 0
    for (int q = 0; q < mine; ++q) {
        const int base = first + q * chunks;
        const int k = bid + (BWD ? mine - 1 - q : q) * nblocks;
        const int tx = k % tl.ntx, ty = k / tl.ntx, wx = w % px, wy = w / px;
        const int x0 = (px * tx + wx) * kPatchX, y0 = (swy * ty + wy) * kPatchY;
        if (x0 >= tl.nx || y0 >= tl.ny) {  // no such patch: nothing to hand over
            progress_store(prog + 4 * kMaxSweepWarps * role, base + chunks, lane);
            continue;
        }
        // the patches before (up) and after (dn) this one along x and y:
        // 0 none, 1 in this block, 2 in another block
        const int hi_x = x0 + kPatchX < tl.nx ? (wx < px - 1 ? 1 : 2) : 0;
        const int lo_x = wx > 0 ? 1 : (tx > 0 ? 2 : 0);
        const int hi_y = y0 + kPatchY < tl.ny ? (wy < swy - 1 ? 1 : 2) : 0;
        const int lo_y = wy > 0 ? 1 : (ty > 0 ? 2 : 0);
        const int up_x = BWD ? hi_x : lo_x, up_y = BWD ? hi_y : lo_y;
        const int dn_x = BWD ? lo_x : hi_x, dn_y = BWD ? lo_y : hi_y;
        const bool far = up_x == 2 || up_y == 2;
        const int x = x0 + (BWD ? kPatchX - 1 - mx : mx), y = y0 + (BWD ? kPatchY - 1 - my : my);
        const bool whole = x0 + kPatchX <= tl.nx && y0 + kPatchY <= tl.ny;
        const unsigned nzl = x < tl.nx && y < tl.ny ? nz : 0;  // this lane's cells: z in [0, nzl)
        unsigned pos = (unsigned)base * kTileK & (kRing - 1);  // first slot of the chunk
        int st = base % kStages;                               // its stage
        if (role == 0) {
            // ---- sweeping.  Lanes 0..3 watch the neighbours in this block,
            // lanes 4 to 6 the warps that stage, drain and fetch.  At the same
            // z the patch before runs kPatchX steps ahead along x and kPatchY
            // along y; the patches after may lag by what their rings hold.
            unsigned watch = prog;
            int off = kNever;
            if (lane == 0 && up_x == 1) { watch = prog - 4 * (unsigned)kDn; off = (kPatchX + 2 * kTileK - 2) / kTileK; }
            if (lane == 1 && up_y == 1) { watch = prog - 4 * (unsigned)(px * kDn); off = (kPatchY + 2 * kTileK - 2) / kTileK; }
            if (lane == 2 && dn_x == 1) { watch = prog + 4 * (unsigned)kDn; off = -(kRing / kTileK - 1); }
            if (lane == 3 && dn_y == 1) { watch = prog + 4 * (unsigned)(px * kDn); off = -(kRing / kTileK - 1); }
            if (lane == 4) { watch = staged; off = 1; }
            if (lane == 5) { watch = drained; off = -kDrainLag; }
            if (lane == 6 && far) { watch = fetched; off = 1; }
            // edge cells go into the edge column / row of the patch after, 8 /
            // 4 slots back; the other lanes store their own cell again
            const bool give_x = dn_x == 1 && mx == kPatchX - 1, give_y = dn_y == 1 && my == kPatchY - 1;
            T* const to_x = give_x ? own + kDn * (int)(kWarpB / sizeof(T)) - kPatchX : own;
            T* const to_y = give_y ? own + px * kDn * (int)(kWarpB / sizeof(T)) - kPatchY * kRowS : own;
            const unsigned back_x = give_x ? kPatchX : 0, back_y = give_y ? kPatchY : 0;
            T prev = T(0);
            constexpr bool kOrders = MAP && sizeof(T) == 8 && !kScaledRec<T>;
            const unsigned* const ords =
                kOrders ? tl.ord[BWD] + (size_t)(k * sw + w) * chunks * 32 + lane : nullptr;
            unsigned ord_next = kOrders ? ords[0] : kBoxOrders;
            for (int c = 0; c < chunks; ++c) {
                const unsigned ord = ord_next;
                if (kOrders && c + 1 < chunks) ord_next = ords[(c + 1) * 32];
                const int target = base + min(c + off, chunks);
                if (!tile_wait(ctl, limit, BWD ? 28 : 26,
                               [&] { return progress_load(watch) - target >= 0; }))
                    return {false, T(0)};
                const unsigned char* const rc = s_rec + st * kChunkRec;
                const T* const mc = s_mid + st * (kTileK * 32);
                T* const cur = own + pos * kSlot;
                const T* const before = own + ((pos - 1) & (kRing - 1)) * kSlot;
                T* const gx = to_x + ((pos - back_x) & (kRing - 1)) * kSlot;
                T* const gy = to_y + ((pos - back_y) & (kRing - 1)) * kSlot;
                auto steps = [&](auto all_inside, auto box_order) {
                    TileRec<L, T> r[kTileK];
                    T f[kTileK];
#pragma unroll
                    for (int u = 0; u < kTileK; ++u) {
                        r[u].load(rc + u * kRec, lane);
                        f[u] = BWD ? mc[u * 32] : cur[u * kSlot];
                        if (!BWD && kScaledRec<T>) f[u] = f[u] * r[u].d;
                    }
#pragma unroll
                    for (int u = 0; u < kTileK; ++u) {
                        // absent neighbours have entry 0 and value 0
                        const T* const nb = u == 0 ? before : cur + (u - 1) * kSlot;
                        const T vx = nb[-1], vy = nb[-kRowS];
                        T v;
                        if (kScaledRec<T>) {
                            v = f[u] - r[u].a[BWD ? 2 : 0] * prev;
                            v = v - r[u].a[1] * vy;
                            v = v - r[u].a[BWD ? 0 : 2] * vx;
                        } else if (BWD && sizeof(T) == 4) {
                            T a = r[u].a[2] * prev;  // the middle value is w, D times its own
                            a = a + r[u].a[1] * vy;
                            a = a + r[u].a[0] * vx;
                            v = f[u] - a * r[u].d;
                        } else {
                            T a = f[u];
                            if (decltype(box_order)::value) {
                                a = a - r[u].a[0] * (BWD ? vx : prev);
                                a = a - r[u].a[1] * vy;
                                a = a - r[u].a[2] * (BWD ? prev : vx);
                            } else {
                                const T t0 = r[u].a[0] * (BWD ? vx : prev), t1 = r[u].a[1] * vy,
                                        t2 = r[u].a[2] * (BWD ? prev : vx);
#pragma unroll
                                for (int e = 0; e < 3; ++e) {
                                    const unsigned which = ord >> (8 * u + 2 * e) & 3u;
                                    a = a - (which == 0 ? t0 : which == 1 ? t1 : t2);
                                }
                            }
                            v = a * r[u].d;
                        }
                        if (!decltype(all_inside)::value)
                            v = (unsigned)(c * kTileK + u - skew) < nzl ? v : T(0);
                        prev = v;
                        cur[u * kSlot] = v;
                        gx[u * kSlot] = v;
                        gy[u * kSlot] = v;
                        __syncwarp();
                    }
                };
                bool ordered = true;
                if constexpr (kOrders) {
                    ordered = __all_sync(0xffffffffu, ord == kBoxOrders);
                    if (!ordered) steps(std::false_type{}, std::false_type{});
                }
                if (!ordered) {
                } else if (whole && c * kTileK >= kSkew && (c + 1) * kTileK <= nz)
                    steps(std::true_type{}, std::true_type{});
                else
                    steps(std::false_type{}, std::true_type{});
                progress_store(prog, base + c + 1, lane);
                pos = (pos + kTileK) & (kRing - 1);
                st = st + 1 == kStages ? 0 : st + 1;
            }
            continue;
        }
        const int pt = k * sw + w;
        const unsigned words = tile_edge_words(chunks), ywords = chunks * (kTileK * kPatchY);
        const int nxy = tl.nx * tl.ny, zstep = BWD ? -nxy : nxy;
        const int row0 = x + tl.nx * y + (BWD ? nxy * (nz - 1) : 0);  // z = 0 of the direction
        T* const mid = tl.mid + (size_t)pt * chunks * kTileK * 32;
        // Edge words: lane (xq, xe) of the first 16 has edge cell xe along x
        // of step xq of the chunk, lane (my, mx) cell mx along y of step my.
        const int xq = lane / kPatchY, xe = lane % kPatchY;
        const bool row_in = lane < kTileK * kPatchY && y0 + (BWD ? kPatchY - 1 - xe : xe) < tl.ny;
        if (role == 1) {
            // ---- staging.  Chunk i: the records; forward four slabs of the
            // right-hand side, each lane its own column, into the slots of
            // their steps; backward the middle values of the steps.  kFlight
            // chunks stay in flight behind the one handed over.
            constexpr int kFlight = kStages - 2;
            if (BWD && q == 0) {  // it starts from what the forward sweep drained
                if (!tile_wait(ctl, limit, 29, [&] { return progress_load(drained) - base >= 0; }))
                    return {false, T(0)};
            }
            // lane 0: the stage is free; the others: the ring slots are
            // drained (the reference's middle step also reads the pivots)
            const unsigned watch = lane ? drained : prog;
            const int off = !lane || (!BWD && sizeof(T) == 8 && !kRecipDiag64) ? -(kStages - 1) : -kDrainLag;
            const unsigned char* rec_src = tl.rec[BWD] + (size_t)pt * chunks * kChunkRec + lane * 16;
            const T* src = BWD ? mid + (nz + kSkew - 1) * 32 + (31 - lane) : rhs + row0;
            const unsigned s_rec_a = smem_u32(s_rec) + lane * 16, s_mid_a = smem_u32(s_mid),
                           own_a = smem_u32(own);
            // (another numbering: the rows of the next chunk's slabs)
            const int* const rows = MAP ? tl.row + row0 : nullptr;
            int next[kTileK];
            if (!BWD && MAP)
#pragma unroll
                for (int u = 0; u < kTileK; ++u) next[u] = (unsigned)u < nzl ? rows[u * nxy] : 0;
            for (int i = 0; i < chunks + kFlight; ++i) {
                if (i < chunks) {
                    const int target = base + i + off;
                    if (!tile_wait(ctl, limit, BWD ? 29 : 27,
                                   [&] { return progress_load(watch) - target >= 0; })) {
                        cp_async_wait<0>();
                        return {false, T(0)};
                    }
                    const unsigned d = s_rec_a + st * kChunkRec;
#pragma unroll
                    for (unsigned o = 0; o < kChunkRec; o += 512) {
                        if (kChunkRec - o >= 512) cp_async16(d + o, rec_src + o);
                        else cp_async16(d + o, rec_src + o, lane * 16 < kChunkRec - o);
                    }
                    rec_src += kChunkRec;
                    if (!BWD && MAP) {
#pragma unroll
                        for (int u = 0; u < kTileK; ++u) {
                            const int z = i * kTileK + u;
                            cp_async<sizeof(T)>(
                                own_a + ((pos + u + skew) & (kRing - 1)) * (unsigned)(kSlot * sizeof(T)),
                                rhs + next[u], (unsigned)z < nzl);
                            next[u] = (unsigned)(z + kTileK) < nzl ? rows[(z + kTileK) * nxy] : 0;
                        }
                    } else if (!BWD) {
#pragma unroll
                        for (int u = 0; u < kTileK; ++u) {
                            cp_async<sizeof(T)>(
                                own_a + ((pos + u + skew) & (kRing - 1)) * (unsigned)(kSlot * sizeof(T)), src,
                                (unsigned)(i * kTileK + u) < nzl);
                            src += nxy;
                        }
                    } else {
                        const unsigned md = s_mid_a + st * (unsigned)(kTileK * 32 * sizeof(T));
#pragma unroll
                        for (int u = 0; u < kTileK; ++u)
                            cp_async<sizeof(T)>(md + u * (unsigned)(32 * sizeof(T)), src - u * 32,
                                                (unsigned)(i * kTileK + u - skew) < nzl);
                        src -= kTileK * 32;
                    }
                    // no patch before: its edge cells are 0 (step s reads slot s - 1)
                    if (up_x == 0 && lane < kTileK * kPatchY)
                        ring[((pos + xq - 1) & (kRing - 1)) * kSlot + (xe + 1) * kRowS] = T(0);
                    if (up_y == 0) ring[((pos + my - 1) & (kRing - 1)) * kSlot + mx + 1] = T(0);
                    pos = (pos + kTileK) & (kRing - 1);
                    st = st + 1 == kStages ? 0 : st + 1;
                }
                cp_async_commit();
                cp_async_wait<kFlight>();
                __syncwarp();
                if (i >= kFlight) progress_store(staged, base + i - kFlight + 1, lane);
            }
            continue;
        }
        if (role == 3) {
            // ---- fetching edges from other blocks.  The words of two chunks
            // ahead are on their way while a chunk waits for its own; two sets
            // of registers take turns, as moving a word on would wait for it.
            if (!far) {
                progress_store(fetched, base + chunks, lane);
                continue;
            }
            const bool want_x = up_x == 2 && row_in, want_y = up_y == 2 && x < tl.nx;
            const unsigned char* const in_x =
                tl.edge[BWD] + ((size_t)((k - kDn) * sw + w + (px - 1) * kDn) * words + lane) * kEdge;
            const unsigned char* const in_y =
                tl.edge[BWD] + ((size_t)((k - kDn * tl.ntx) * sw + (BWD ? wx : wx + px * (swy - 1))) * words +
                                ywords + lane) * kEdge;
            EdgeWord<T> ax, ay, bx, by;
            auto has_x = [&](int c) { return want_x && (unsigned)(c * kTileK + xq - xe) < (unsigned)nz; };
            auto has_y = [&](int c) { return want_y && (unsigned)(c * kTileK + my - mx) < (unsigned)nz; };
            auto fetch = [&](int c, EdgeWord<T>& ex, EdgeWord<T>& ey) {
                ex.load(in_x + c * (kTileK * kPatchY * kEdge), has_x(c));
                ey.load(in_y + c * (kTileK * kPatchX * kEdge), has_y(c));
            };
            auto edges_in = [&](int c, EdgeWord<T>& ex, EdgeWord<T>& ey) {
                const bool hx = has_x(c), hy = has_y(c);
                const unsigned char* const cx = in_x + c * (kTileK * kPatchY * kEdge);
                const unsigned char* const cy = in_y + c * (kTileK * kPatchX * kEdge);
                // (the slots' last readers: the chunk before 32 steps ago)
                const int room = base + c - (kRing / kTileK - 1);
                bool again = false;
                if (!tile_wait(ctl, limit, BWD ? 29 : 27, [&] {
                        const bool nx_ = hx && !ex.ready(epoch), ny_ = hy && !ey.ready(epoch);
                        ex.load(cx, again && nx_);
                        ey.load(cy, again && ny_);
                        again = true;
                        const bool here = (!hx || ex.ready(epoch)) && (!hy || ey.ready(epoch));
                        return here & (progress_load(prog) - room >= 0);
                    }))
                    return false;
                // step s reads its edges from slot s - 1
                if (hx) ring[((pos + xq - 1) & (kRing - 1)) * kSlot + (xe + 1) * kRowS] = ex.value();
                if (hy) ring[((pos + my - 1) & (kRing - 1)) * kSlot + mx + 1] = ey.value();
                __syncwarp();
                progress_store(fetched, base + c + 1, lane);
                pos = (pos + kTileK) & (kRing - 1);
                fetch(c + 2, ex, ey);
                return true;
            };
            fetch(0, ax, ay);
            fetch(1, bx, by);
            for (int c = 0; c < chunks; ++c)
                if (!(c & 1 ? edges_in(c, bx, by) : edges_in(c, ax, ay))) return {false, T(0)};
            continue;
        }
        // ---- draining
        unsigned char* const out_x = tl.edge[BWD] + ((size_t)pt * words + lane) * kEdge;
        unsigned char* const out_y = out_x + (size_t)ywords * kEdge;
        const bool far_x = dn_x == 2 && row_in, far_y = dn_y == 2 && x < tl.nx, publish_far = dn_x == 2 || dn_y == 2;
        // (another numbering: the rows of the next chunk's slabs)
        int next[kTileK];
        if (BWD && MAP)
#pragma unroll
            for (int u = 0; u < kTileK; ++u)
                next[u] = (unsigned)(u - kSkew) < nzl ? tl.row[row0 + (u - kSkew) * zstep] : 0;
        for (int c = 0; c < chunks; ++c) {
            const int z0 = c * kTileK - kSkew;  // backward: first of the slabs whose last lane is done
            const bool inside = whole && z0 >= 0 && z0 + kTileK <= nz;
            T rpre[kTileK];  // their right-hand side
            int rows[kTileK];
            if (BWD && MAP) {
#pragma unroll
                for (int u = 0; u < kTileK; ++u) {
                    rows[u] = next[u];
                    rpre[u] = (unsigned)(z0 + u) < nzl ? rhs[rows[u]] : T(0);
                    const int z = z0 + kTileK + u;
                    next[u] = (unsigned)z < nzl ? tl.row[row0 + z * zstep] : 0;
                }
            } else if (BWD) {
                if (inside) {
#pragma unroll
                    for (int u = 0; u < kTileK; ++u) rpre[u] = rhs[row0 + (z0 + u) * zstep];
                } else {
#pragma unroll
                    for (int u = 0; u < kTileK; ++u)
                        rpre[u] = (unsigned)(z0 + u) < nzl ? rhs[row0 + (z0 + u) * zstep] : T(0);
                }
            }
            const int target = base + c + 1;
            if (!tile_wait(ctl, limit, BWD ? 29 : 27,
                           [&] { return progress_load(prog) - target >= 0; }))
                return {false, T(0)};
            if (publish_far) {
                const int tx_ = c * kTileK + xq - (kPatchX - 1), ty_ = c * kTileK + my - (kPatchY - 1);  // the reader's steps
                EdgeWord<T>::store(out_x + (c * kTileK - (kPatchX - 1)) * (int)(kPatchY * kEdge),
                                   ring[(pos + (xq & (kTileK - 1))) * kSlot + (xe + 1) * kRowS + kPatchX], epoch,
                                   far_x && (unsigned)(tx_ - xe) < (unsigned)nz);
                EdgeWord<T>::store(out_y + (c * kTileK - (kPatchY - 1)) * (int)(kPatchX * kEdge),
                                   ring[(pos + my) * kSlot + kPatchY * kRowS + mx + 1], epoch,
                                   far_y && (unsigned)(ty_ - mx) < (unsigned)nz);
            }
            if (!BWD) {
                // the middle step w / (D + TINY) of CG.f90:144-146 in the
                // reference's arithmetic; the others go on from w itself
                T* const mp = mid + c * (kTileK * 32) + lane;
                const T* const vp = own + pos * kSlot;
                const unsigned char* const rc = s_rec + st * kChunkRec;
#pragma unroll
                for (int u = 0; u < kTileK; ++u) {
                    T v = vp[u * kSlot];
                    if constexpr (sizeof(T) == 8 && !kRecipDiag64)
                        v = div_rn(v, *reinterpret_cast<const T*>(rc + u * kRec + TileRec<L, T>::at(3, lane)) +
                                          tiny_v<T>());
                    mp[u * 32] = v;
                }
            } else {
                auto flush = [&](int u, int row) {
                    const T v = own[((pos - kSkew + u + skew) & (kRing - 1)) * kSlot];
                    zout[row] = v;
                    epi(row, v, rpre[u]);
                };
                if (MAP) {
#pragma unroll
                    for (int u = 0; u < kTileK; ++u)
                        if ((unsigned)(z0 + u) < nzl) flush(u, rows[u]);
                } else if (inside) {
#pragma unroll
                    for (int u = 0; u < kTileK; ++u) flush(u, row0 + (z0 + u) * zstep);
                } else {
#pragma unroll
                    for (int u = 0; u < kTileK; ++u)
                        if ((unsigned)(z0 + u) < nzl) flush(u, row0 + (z0 + u) * zstep);
                }
            }
            __syncwarp();
            progress_store(drained, base + c + 1, lane);
            pos = (pos + kTileK) & (kRing - 1);
            st = st + 1 == kStages ? 0 : st + 1;
        }
    }
    return {true, epi.dot};
}

// z = IC(0) apply of rhs by the tiled sweeps, epi (RowOp) per row.
template <bool MAP, typename L, typename T, typename Epi>
__device__ __forceinline__ Applied<T> ic_tiled_apply(Grid& g, const Mat<T>& m, const T* rhs, T* z, Epi epi) {
    extern __shared__ __align__(128) unsigned char tf_smem[];
    const int chunks = tiles_of(m.tile, g.bid, g.nblocks) * m.tile.chunks;
    ++g.epoch;
    // The counters start at 0 in each apply, so that they stay within one
    // apply's chunks however long the solve (a grid barrier separates the
    // applies: no warp reads them any more).
    if (threadIdx.x < kWarpsPerPatch * kMaxSweepWarps) reinterpret_cast<int*>(tf_smem)[threadIdx.x] = 0;
    __syncthreads();
    // (all warps of the block go on to the backward sweep: its waits end by
    // the abort flag if the forward sweep of another warp gave up)
    const RowOp<kRowNone, T> none{T(0), nullptr, T(0)};
    const bool ok =
        tile_sweep<0, MAP, L, T>(g.ctl, g.timeout_cyc, g.bid, g.nblocks, g.epoch, 0, m, rhs, z, none).ok;
    Applied<T> a =
        tile_sweep<1, MAP, L, T>(g.ctl, g.timeout_cyc, g.bid, g.nblocks, g.epoch, chunks, m, rhs, z, epi);
    a.ok = a.ok && ok;
    return a;
}

// On a box in another numbering, beside the box's own: a function, as the rows'
// look-up and the order of their sums would cost the box numbering 4 to 7 % of
// an apply (reference arithmetic, 109 x 83 x 97 cells: 527 -> 566 us per
// iteration).
template <typename L, typename T, typename Epi>
__device__ __noinline__ Applied<T> ic_mapped_apply(Grid& g, const Mat<T>& m, const T* rhs, T* z, Epi epi) {
    return ic_tiled_apply<true, L>(g, m, rhs, z, epi);
}

// The IC(0) apply the solve was configured for: `sweeps` Jacobi sweeps per
// triangle (FP32 inner solves and contracted FP64 solves), else the exact
// apply -- tiled sweeps on a box, level-ordered sync-free
// sweeps otherwise.  OP, alfa, x: what is done with each row (RowOp); the
// thread's sum of kRowDot in `dot`.
template <int OP, typename T>
__device__ __forceinline__ bool ic_precond(Grid& g, const Mat<T>& m, Vecs<T>& v, int sweeps,
                                           const T* rhs, T* z, T& dot, T alfa = T(0), T* x = nullptr) {
    const RowOp<OP, T> epi{alfa, x, T(0)};
    Applied<T> a{false, T(0)};
    if (kJacobiIc && (sweeps > 0 || !(kTiledIc || kLevelIc))) {
        if constexpr (!kShortRows) a = jacobi_function<true>(g, m, v.D, rhs, v.w, v.s, z, sweeps, epi);
        else if constexpr (sizeof(T) == 4) a = jacobi_function<false>(g, m, v.D, rhs, v.w, v.s, z, sweeps, epi);
        else if constexpr (kJacobiIc) a = jacobi_apply<false>(g, m, v.D, rhs, v.w, v.s, z, sweeps, epi);
    } else if (kTiledIc && (!kLevelIc || m.tile.on)) {
        if constexpr (kTiledIc && !kJacobiIc) {  // TFLOWS_FOR_MAPPED
            if constexpr (sizeof(T) == 4)
                a = m.tile.lu_bf16 ? ic_tiled_apply<true, unsigned short>(g, m, rhs, z, epi)
                                   : ic_tiled_apply<true, T>(g, m, rhs, z, epi);
            else
                a = ic_tiled_apply<true, T>(g, m, rhs, z, epi);
        } else if constexpr (kTiledIc) {
            const bool mapped = kLevelIc && m.tile.row;
            if constexpr (sizeof(T) == 4) {
                if (mapped)
                    a = m.tile.lu_bf16 ? ic_mapped_apply<unsigned short>(g, m, rhs, z, epi)
                                       : ic_mapped_apply<T>(g, m, rhs, z, epi);
                else
                    a = m.tile.lu_bf16 ? ic_tiled_apply<false, unsigned short>(g, m, rhs, z, epi)
                                       : ic_tiled_apply<false, T>(g, m, rhs, z, epi);
            } else {
                a = mapped ? ic_mapped_apply<T>(g, m, rhs, z, epi) : ic_tiled_apply<false, T>(g, m, rhs, z, epi);
            }
        }
    } else if constexpr (kLevelIc) {
        a = ic_apply(g, m, v.D, rhs, v.w, z, epi);
    }
    dot = a.dot;
    return a.ok;
}

template <typename T>
__device__ __forceinline__ bool finite_val(T v) { return isfinite(v); }

// The end of an iteration: the totals of r r and of the second sum, and of the
// third (finite entries of x and r) only once the residual has turned
// non-finite.  beta, the ratio of the next rho (total `num`) and the current
// one, which it replaces, is formed by the summing thread (`next_rho`).
struct IterEnd {
    double rr;       // ||r||^2
    double beta;
    bool converged;
    bool all_nan;    // (with `all`) no entry of x and r is a number
};
template <typename T>
__device__ __forceinline__ bool reduce_end(Grid& g, int slot, const T (&a)[3], bool all, int where, int num,
                                           bool next_rho, IterEnd& e) {
    e.all_nan = false;
    if (all) {
        const T c[1] = {a[2]};
        publish_t<1>(g, slot + 2, c);
        if (!grid_sync(g, where)) return false;
        double t[1];
        totals<1>(g, slot + 2, t);
        e.all_nan = t[0] == 0.0;
    }
    const T b[2] = {a[0], a[1]};
    publish_t<2>(g, slot, b);
    if (!grid_sync(g, where)) return false;
    double u[2], x[2];
    totals<2>(g, slot, u, x, [&](int k, double s) {
        double r = 0.0;
        if (k == num && next_rho) {
            r = div_rn(s, scalars().rho);
            scalars().rho = s;
        }
        if (k == 0) scalars().rr = s;
        return r;
    });
    e.rr = u[0];
    e.beta = x[num];
    e.converged = scalars().conv.below(u[0]);
    return true;
}

// ---- the reference prologue: Prec1, ||b||, Resid, IniRes -------------------
// Returns false when the launch aborted or an early exit was taken (out
// records which).  On return true, the block's scalars hold the tolerance and,
// for prec 1 / 0, rho = (r0, M^-1 r0) (z written for prec 1).
template <typename T>
__device__ __noinline__ bool prologue(Grid& g, const Mat<T>& m, Vecs<T>& v, const SolveCfg& cfg, SolveOut& out,
                         bool store_z) {
    if (cfg.do_prec1 && !prec1_phase(g, m, v.D, cfg.prec)) {
        out.exit_kind = EXIT_ABORT;
        return false;
    }
    // (IC pivots complete: prec1_phase ends with a barrier; the barrier
    // below orders the tiled layout before the first apply)
    if (kTiledIc && cfg.do_prec1 && cfg.prec == 2 && m.tile.on) tiles_init(g, m, v.D);
    T acc[1] = {T(0)};
    TF_FOR4(g, m, i) {
        const V4<T> r = ld4(v.r + i);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u < m.n) acc[0] += r.a[u] * r.a[u];
    }
    publish_t<1>(g, SLOT_A, acc);
    if (!grid_sync(g, 30)) { out.exit_kind = EXIT_ABORT; return false; }
    double tot[1], nrm[1];
    totals<1>(g, SLOT_A, tot, nrm, [](int, double s) { return sqrt(s); });
    const double bnrm2 = nrm[0];
    double tol = cfg.tol;
    out.bnrm2 = bnrm2;
    if (cfg.tol_is_relative) tol = tol * bnrm2;
    if (bnrm2 < tol || (cfg.tol_is_relative && bnrm2 == 0.0)) {
        out.exit_kind = EXIT_BNRM;
        out.iterations = 0;
        return false;
    }
    T a2[2] = {T(0), T(0)};
    for (int s = g.wg; s < m.nslices; s += g.nw) {
        const int i = s * kWarp + g.lane;
        T ri = i < m.n ? v.r[i] : T(0);
        if (!cfg.x_is_zero) ri = sell_resid_row(m, s, g.lane, ri, v.x);
        if (i < m.n) {
            v.r[i] = ri;
            a2[0] += ri * ri;
            if (store_z) {
                if (cfg.prec == 1) {
                    const T zi = jacobi(ri, v.D[i]);
                    v.z[i] = zi;
                    a2[1] += ri * zi;
                }
            }
        }
    }
    publish_t<2>(g, SLOT_B, a2);
    if (!grid_sync(g, 31)) { out.exit_kind = EXIT_ABORT; return false; }
    double t2[2], e2[2];
    totals<2>(g, SLOT_B, t2, e2, [](int k, double s) { return k == 0 ? sqrt(s) : 0.0; });
    const double err = e2[0];
    out.ini_res = err;
    out.fin_res = err;
    if (err < tol) {
        out.exit_kind = EXIT_INIRES;
        out.iterations = 0;
        return false;
    }
    if (threadIdx.x == 0) {
        scalars().conv.set(tol);
        scalars().rho = cfg.prec == 1 ? t2[1] : t2[0];
    }
    __syncthreads();
    return true;
}

// ---- CG (Process/CG.f90:113-259; also BiCG, whose iterates are CG's) --------
// FUSE: the search direction formed inside the product, 1 always, 0 never, -1
// as cfg.fuse_dir says (two forms of the product in one kernel).  PREC: the
// preconditioner where the kernel has but one, -1 as prec_of says.
template <int FUSE, int PREC, typename T>
__device__ void cg_solve(Grid& g, const Mat<T>& m, Vecs<T>& v, const SolveCfg& cfg, SolveOut& out) {
    if (!prologue(g, m, v, cfg, out, true)) return;
    const int prec = PREC < 0 ? prec_of(cfg.prec) : PREC;
    const T* z = prec == 0 ? v.r : v.z;
    bool nonfinite = false;
    int iter = 1;
    T beta = T(0);
    IterEnd e;
    // search direction; formed inside the product it alternates between p and t
    T* pcur = v.p;
    T* pnext = v.t;
    for (; iter <= cfg.maxiter; ++iter) {
        if (prec == 2) {
            T a[1];
            const bool ok = ic_precond<kRowDot>(g, m, v, cfg.ic_sweeps, v.r, v.z, a[0]);
            publish_t<1>(g, SLOT_A, a);
            if (!grid_sync(g, 41) || !ok) { out.exit_kind = EXIT_ABORT; return; }
            double t[1], x[1];
            totals<1>(g, SLOT_A, t, x, [&](int, double s) {
                const double b = iter == 1 ? 0.0 : div_rn(s, scalars().rho);
                scalars().rho = s;
                return b;
            });
            beta = T(x[0]);
        }
        // The new search direction formed inside the product, into the other
        // p buffer (no separate update pass, one barrier less per
        // iteration): always in the FP32 inner solves; in FP64 where the
        // host asked for it (small systems -- on larger ones gathering z and
        // p and forming z + beta p per neighbour on the FP64 pipe costs more
        // than the pass it saves).
        T a1[1];
        if (FUSE < 0 ? cfg.fuse_dir != 0 : FUSE != 0) {
            T* const pnew = pnext;
            a1[0] = product_phase<T, true>(m, g.wg, g.nw, z, pcur, pnew, v.q, nullptr, beta, iter == 1);
            pnext = pcur;
            pcur = pnew;
        } else {
            direction_phase(g.tid, g.nt, m.n, z, v.p, beta, iter == 1);
            if (!grid_sync(g, 42)) { out.exit_kind = EXIT_ABORT; return; }
            // q = A p; (p, q)  (CG.f90:193-218)
            a1[0] = product_phase<T, false>(m, g.wg, g.nw, nullptr, v.p, nullptr, v.q, v.p, T(0), false);
        }
        publish_t<1>(g, SLOT_C, a1);
        if (!grid_sync(g, 43)) { out.exit_kind = EXIT_ABORT; return; }
        double t1[1], x1[1];
        totals<1>(g, SLOT_C, t1, x1, [&](int, double s) { return div_rn(scalars().rho, s); });
        const T alfa = T(x1[0]);
        // x += alfa p; r -= alfa q; ||r||; next z and rho  (CG.f90:226-253)
        const Sums3<T> a3 =
            update_phase(g.tid, g.nt, m.n, v.x, v.r, pcur, v.q, v.D, v.z, alfa, prec == 1, nonfinite);
        if (!reduce_end(g, SLOT_D, a3.a, nonfinite, 44, prec == 1 ? 1 : 0, prec != 2, e)) {
            out.exit_kind = EXIT_ABORT;
            return;
        }
        beta = T(e.beta);
        if (e.converged) {
            out.exit_kind = EXIT_CONVERGED;
            out.iterations = iter;
            out.fin_res = sqrt(e.rr);
            return;
        }
        if (!finite_val(e.rr)) {
            // From here on the reference keeps iterating on non-finite
            // values; once every x and r entry is NaN nothing changes any
            // more, so the remaining iterations can be skipped.
            if (e.all_nan) {
                out.exit_kind = EXIT_NONFINITE;
                out.iterations = cfg.maxiter + 1;
                out.fin_res = sqrt(e.rr);
                return;
            }
            nonfinite = true;
        }
    }
    out.exit_kind = EXIT_MAXITER;
    out.iterations = iter;
    if (iter > 1) out.fin_res = sqrt(scalars().rr);
}

// ---- CGS (Process/CGS.f90:112-333) -------------------------------------------
template <typename T>
__device__ void cgs_solve(Grid& g, const Mat<T>& m, Vecs<T>& v, const SolveCfg& cfg, SolveOut& out) {
    if (!prologue(g, m, v, cfg, out, false)) return;
    T beta = T(0);
    IterEnd e;
    const int prec = prec_of(cfg.prec);
    // r2 = r1 (CGS.f90:84-86); rho = (r1, r2) for the first iteration.
    T a0[1] = {T(0)};
    TF_FOR4(g, m, i) {
        const V4<T> r = ld4(v.r + i);
        st4(v.r2 + i, r);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u < m.n) a0[0] += r.a[u] * r.a[u];
    }
    publish_t<1>(g, SLOT_A, a0);
    if (!grid_sync(g, 50)) { out.exit_kind = EXIT_ABORT; return; }
    double t0[1], x0[1];
    totals<1>(g, SLOT_A, t0, x0, [](int, double s) { return scalars().rho = s; });
    bool nonfinite = false;
    int iter = 1;
    for (; iter <= cfg.maxiter; ++iter) {
        // u1 = r1 + beta q1; u2 = u1 + beta (q1 + beta u2); p2 = M^-1 u2
        TF_FOR4(g, m, i) {
            const V4<T> rr = ld4(v.r + i);
            V4<T> u1, u2, p2;
            if (iter == 1) {
                u1 = rr;
                u2 = rr;
            } else {
                const V4<T> q1 = ld4(v.q + i);
                u2 = ld4(v.u2 + i);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    u1.a[u] = rr.a[u] + beta * q1.a[u];
                    u2.a[u] = u1.a[u] + beta * (q1.a[u] + beta * u2.a[u]);
                }
            }
            st4(v.u1 + i, u1);
            st4(v.u2 + i, u2);
            if (prec == 1) {
                const V4<T> dd = ld4(v.D + i);
#pragma unroll
                for (int u = 0; u < 4; ++u) p2.a[u] = jacobi(u2.a[u], dd.a[u]);
                st4(v.p2 + i, p2);
            } else if (prec != 2) {
                st4(v.p2 + i, u2);
            }
        }
        if (!grid_sync(g, 51)) { out.exit_kind = EXIT_ABORT; return; }
        if (prec == 2) {
            T none;
            const bool ok = ic_precond<kRowNone>(g, m, v, cfg.ic_sweeps, v.u2, v.p2, none);
            if (!grid_sync(g, 53) || !ok) { out.exit_kind = EXIT_ABORT; return; }
        }
        // v2 = A p2; alfa = rho / (r2, v2)
        const T a1[1] = {product_phase<T, false>(m, g.wg, g.nw, nullptr, v.p2, nullptr, v.v2, v.r2, T(0), false)};
        publish_t<1>(g, SLOT_B, a1);
        if (!grid_sync(g, 54)) { out.exit_kind = EXIT_ABORT; return; }
        double t1[1], x1[1];
        totals<1>(g, SLOT_B, t1, x1, [&](int, double s) { return div_rn(scalars().rho, s); });
        const T alfa = T(x1[0]);
        // q1 = u1 - alfa v2; p1 = M^-1 (u1 + q1); x += alfa p1
        TF_FOR4(g, m, i) {
            const V4<T> u1 = ld4(v.u1 + i), v2 = ld4(v.v2 + i);
            V4<T> q1, tt;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                q1.a[u] = u1.a[u] - alfa * v2.a[u];
                tt.a[u] = u1.a[u] + q1.a[u];
            }
            st4(v.q + i, q1);
            if (prec == 2) {
                st4(v.t + i, tt);
            } else {
                V4<T> p1 = tt, xx = ld4(v.x + i);
                if (prec == 1) {
                    const V4<T> dd = ld4(v.D + i);
#pragma unroll
                    for (int u = 0; u < 4; ++u) p1.a[u] = jacobi(tt.a[u], dd.a[u]);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) xx.a[u] = xx.a[u] + alfa * p1.a[u];
                st4(v.p + i, p1);
                st4(v.x + i, xx);
            }
        }
        if (!grid_sync(g, 55)) { out.exit_kind = EXIT_ABORT; return; }
        if (prec == 2) {
            T none;
            const bool ok = ic_precond<kRowAxpy>(g, m, v, cfg.ic_sweeps, v.t, v.p, none, alfa, v.x);
            if (!grid_sync(g, 57) || !ok) { out.exit_kind = EXIT_ABORT; return; }
        }
        // q2 = A p1; r1 -= alfa q2; ||r1||; next rho = (r1, r2)
        T a3[3] = {T(0), T(0), T(0)};
        for (int s = g.wg; s < m.nslices; s += g.nw) {
            const int i = s * kWarp + g.lane;
            const T q2 = sell_row(m, s, g.lane, v.p);
            if (i < m.n) {
                const T ri = v.r[i] - alfa * q2;
                v.r[i] = ri;
                a3[0] += ri * ri;
                a3[1] += ri * v.r2[i];
                if (nonfinite) {
                    const T xi = v.x[i];
                    a3[2] += (xi == xi ? T(1) : T(0)) + (ri == ri ? T(1) : T(0));
                }
            }
        }
        if (!reduce_end(g, SLOT_C, a3, nonfinite, 58, 1, true, e)) {
            out.exit_kind = EXIT_ABORT;
            return;
        }
        beta = T(e.beta);
        if (e.converged) {
            out.exit_kind = EXIT_CONVERGED;
            out.iterations = iter;
            out.fin_res = sqrt(e.rr);
            return;
        }
        if (!finite_val(e.rr)) {
            if (e.all_nan) {
                out.exit_kind = EXIT_NONFINITE;
                out.iterations = cfg.maxiter + 1;
                out.fin_res = sqrt(e.rr);
                return;
            }
            nonfinite = true;
        }
    }
    out.exit_kind = EXIT_MAXITER;
    out.iterations = iter;
    if (iter > 1) out.fin_res = sqrt(scalars().rr);
}

// ---- BiCG with the transposed shadow sequence (extension) ---------------------
// The textbook preconditioned BiCG (the shadow residual is multiplied by A^T,
// whose values mT holds in A's pattern), for nonsymmetric systems where the
// reference's "bicg" (shadow multiplied by A, i.e. CG) may fail.  Diagonal
// or no preconditioning (M^T = M).  Same control flow and outputs as cg_solve.
template <typename T>
__device__ void bicg_true_solve(Grid& g, const Mat<T>& m, const Mat<T>& mT, Vecs<T>& v,
                                const SolveCfg& cfg, SolveOut& out) {
    if (!prologue(g, m, v, cfg, out, false)) return;
    T beta = T(0);
    IterEnd e;
    const bool diag = cfg.prec == 1;
    T* z2 = v.u1;
    T* q2 = v.v2;
    // shadow r2 = r; z = M^-1 r, z2 = M^-1 r2; rho = (z, r2)
    T a0[1] = {T(0)};
    TF_FOR4(g, m, i) {
        const V4<T> r = ld4(v.r + i);
        V4<T> z = r;
        if (diag) {
            const V4<T> d = ld4(v.D + i);
#pragma unroll
            for (int u = 0; u < 4; ++u) z.a[u] = jacobi(r.a[u], d.a[u]);
        }
        st4(v.r2 + i, r);
        st4(v.z + i, z);
        st4(z2 + i, z);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u < m.n) a0[0] += z.a[u] * r.a[u];
    }
    publish_t<1>(g, SLOT_A, a0);
    if (!grid_sync(g, 60)) { out.exit_kind = EXIT_ABORT; return; }
    double t0[1], x0[1];
    totals<1>(g, SLOT_A, t0, x0, [](int, double s) { return scalars().rho = s; });
    int iter = 1;
    for (; iter <= cfg.maxiter; ++iter) {
        TF_FOR4(g, m, i) {
            const V4<T> z = ld4(v.z + i), zz = ld4(z2 + i);
            V4<T> p = z, pp = zz;
            if (iter > 1) {
                p = ld4(v.p + i);
                pp = ld4(v.p2 + i);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    p.a[u] = z.a[u] + beta * p.a[u];
                    pp.a[u] = zz.a[u] + beta * pp.a[u];
                }
            }
            st4(v.p + i, p);
            st4(v.p2 + i, pp);
        }
        if (!grid_sync(g, 61)) { out.exit_kind = EXIT_ABORT; return; }
        T a1[1] = {T(0)};
        for (int s = g.wg; s < m.nslices; s += g.nw) {
            const int i = s * kWarp + g.lane;
            const T qi = sell_row(m, s, g.lane, v.p);
            const T q2i = sell_row(mT, s, g.lane, v.p2);
            if (i < m.n) {
                v.q[i] = qi;
                q2[i] = q2i;
                a1[0] += v.p2[i] * qi;
            }
        }
        publish_t<1>(g, SLOT_B, a1);
        if (!grid_sync(g, 62)) { out.exit_kind = EXIT_ABORT; return; }
        double t1[1], x1[1];
        totals<1>(g, SLOT_B, t1, x1, [&](int, double s) { return div_rn(scalars().rho, s); });
        const T alfa = T(x1[0]);
        T a3[3] = {T(0), T(0), T(0)};
        TF_FOR4(g, m, i) {
            V4<T> x = ld4(v.x + i), r = ld4(v.r + i), rr = ld4(v.r2 + i);
            const V4<T> p = ld4(v.p + i), q = ld4(v.q + i), qq = ld4(q2 + i);
            V4<T> z, zz, d;
            if (diag) d = ld4(v.D + i);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                x.a[u] = x.a[u] + alfa * p.a[u];
                r.a[u] = r.a[u] - alfa * q.a[u];
                rr.a[u] = rr.a[u] - alfa * qq.a[u];
                z.a[u] = diag ? jacobi(r.a[u], d.a[u]) : r.a[u];
                zz.a[u] = diag ? jacobi(rr.a[u], d.a[u]) : rr.a[u];
                if (i + u < m.n) {
                    a3[0] += r.a[u] * r.a[u];
                    a3[1] += z.a[u] * rr.a[u];
                }
            }
            st4(v.x + i, x);
            st4(v.r + i, r);
            st4(v.r2 + i, rr);
            st4(v.z + i, z);
            st4(z2 + i, zz);
        }
        if (!reduce_end(g, SLOT_C, a3, false, 63, 1, true, e)) { out.exit_kind = EXIT_ABORT; return; }
        beta = T(e.beta);
        if (e.converged) {
            out.exit_kind = EXIT_CONVERGED;
            out.iterations = iter;
            out.fin_res = sqrt(e.rr);
            return;
        }
        if (!finite_val(e.rr)) {
            out.exit_kind = EXIT_NONFINITE;
            out.iterations = cfg.maxiter + 1;
            out.fin_res = sqrt(e.rr);
            return;
        }
    }
    out.exit_kind = EXIT_MAXITER;
    out.iterations = iter;
    if (iter > 1) out.fin_res = sqrt(scalars().rr);
}

// ---- mixed precision: FP32 inner Krylov inside FP64 iterative refinement ---------
// Outer loop in FP64: r = b - A x with the FP64 values (exact row order),
// ||r|| and the convergence test; inner solve of A d = r in FP32 (FP32 SELL
// values and vectors, FP64 reductions) by the same CG / CGS code with a
// relative tolerance; x += d in FP64.  The preconditioner setup (Prec1) runs
// once in FP64 and is rounded to FP32.
struct MixedCfg {
    int method;
    int prec;
    int max_ref;
    int maxiter;         // cap on the total number of FP32 iterations
    int restart;         // 1: restarted refinement; 0: reliable updates (CG)
    int inner_maxiter;
    double tol;
    double inner_rtol;
    int tol_is_relative;
    int x_is_zero;
    int ic_sweeps;       // prec 2: 0 exact sweeps, k > 0 Jacobi sweeps
    int fuse_dir;        // reliable updates: form the search direction inside the product
};

struct MixedOut {
    int exit_kind;
    int iterations;   // total inner iterations
    int refinements;
    double ini_res;
    double fin_res;
    double bnrm2;
};

// r64 = b - A x64, r32 = (float) r64, d32 = 0; returns ||r64|| (after a barrier).
__device__ __forceinline__ bool mixed_residual(Grid& g, const Mat<double>& m64, const double* b64,
                                               const double* x64, double* r64, float* r32,
                                               float* d32, bool x_zero, double& err) {
    double a[1] = {0.0};
    for (int s = g.wg; s < m64.nslices; s += g.nw) {
        const int i = s * kWarp + g.lane;
        double ri = i < m64.n ? b64[i] : 0.0;
        if (!x_zero) ri = sell_resid_row(m64, s, g.lane, ri, x64);
        if (i < m64.n) {
            r64[i] = ri;
            r32[i] = (float)ri;
            if (d32) d32[i] = 0.0f;
            a[0] += ri * ri;
        }
    }
    publish<1>(g, SLOT_D + 3, a);
    if (!grid_sync(g, 70)) return false;
    double t[1], e[1];
    totals<1>(g, SLOT_D + 3, t, e, [](int, double s) { return sqrt(s); });
    err = e[0];
    return true;
}

template <bool CGS>
__device__ __forceinline__ void mixed_solve(Grid& g, const Mat<double>& m64, const Mat<float>& m32, double* x64,
                            double* r64, const double* b64, double* D64, Vecs<float>& v32,
                            const MixedCfg& c, MixedOut& out) {
    out.exit_kind = EXIT_ABORT;
    if (!prec1_phase(g, m64, D64, c.prec)) return;
    // D64 was written in slice order; the next pass reads it four rows per
    // thread, so it must be complete first.
    if (!grid_sync(g, 74)) return;
    double acc[1] = {0.0};
    TF_FOR4(g, m64, i) {
        const V4<double> d = ld4(D64 + i), bb = ld4(b64 + i);
        V4<float> df, wf;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            // FP32 solves hold 1/D for the diagonal preconditioner
            df.a[u] = c.prec == 1 ? (float)(kRecipDiag64 ? d.a[u] : div_rn(1.0, d.a[u]))
                                  : (float)d.a[u];
            wf.a[u] = Cell<float>::sentinel();
            if (i + u < m64.n) acc[0] += bb.a[u] * bb.a[u];
        }
        st4(v32.D + i, df);
        st4(v32.w + i, wf);
    }
    publish<1>(g, SLOT_A, acc);
    if (!grid_sync(g, 71)) return;
    // (the residual pass below ends with a barrier before the first apply)
    if (kTiledIc && c.prec == 2 && m32.tile.on) tiles_init(g, m32, v32.D);
    double tot[1], nrm[1];
    totals<1>(g, SLOT_A, tot, nrm, [](int, double s) { return sqrt(s); });
    const double bnrm2 = nrm[0];
    out.bnrm2 = bnrm2;
    double tol = c.tol_is_relative ? c.tol * bnrm2 : c.tol;
    if (bnrm2 < tol || (c.tol_is_relative && bnrm2 == 0.0)) {
        out.exit_kind = EXIT_BNRM;
        out.iterations = 0;
        return;
    }
    double err;
    if (!mixed_residual(g, m64, b64, x64, r64, v32.r, v32.x, c.x_is_zero != 0, err)) return;
    out.ini_res = err;
    out.fin_res = err;
    if (err < tol) {
        out.exit_kind = EXIT_INIRES;
        out.iterations = 0;
        return;
    }
    SolveCfg ci;
    ci.method = c.method;
    ci.prec = c.prec;
    ci.maxiter = c.inner_maxiter;
    ci.tol = c.inner_rtol;
    ci.x_is_zero = 1;
    ci.do_prec1 = 0;
    ci.tol_is_relative = 1;
    ci.ic_sweeps = c.ic_sweeps;
    int total = 0, stall = 0;
    double prev = err;
    for (int ref = 1; ref <= c.max_ref; ++ref) {
        ci.maxiter = min(c.inner_maxiter, c.maxiter - total);
        if (ci.maxiter <= 0) break;
        SolveOut oi;
        oi.exit_kind = 0;
        oi.iterations = 0;
        oi.fin_res = 0.0;
        if constexpr (CGS) cgs_solve<float>(g, m32, v32, ci, oi);
        else cg_solve<1, -1>(g, m32, v32, ci, oi);
        if (oi.exit_kind == EXIT_ABORT) return;
        total += oi.exit_kind == EXIT_MAXITER || oi.exit_kind == EXIT_NONFINITE ? ci.maxiter
                                                                                 : oi.iterations;
        out.iterations = total;
        out.refinements = ref;
        if (!isfinite(oi.fin_res)) {
            out.exit_kind = EXIT_NONFINITE;
            return;
        }
        TF_FOR4(g, m64, i) {
            V4<double> xx = ld4(x64 + i);
            const V4<float> d = ld4(v32.x + i);
#pragma unroll
            for (int u = 0; u < 4; ++u) xx.a[u] = xx.a[u] + (double)d.a[u];
            st4(x64 + i, xx);
        }
        if (!grid_sync(g, 72)) return;
        // r = b - A x; d32 is kept (not cleared) until the step is accepted
        double err_new;
        if (!mixed_residual(g, m64, b64, x64, r64, v32.r, nullptr, false, err_new)) return;
        if (!(err_new <= 10.0 * prev)) {
            // The correction made the true residual grow tenfold (the inner
            // iteration diverged in FP32): take the step back and stop.  (CG
            // minimises the error in the A-norm, so a smaller rise of the
            // residual norm is normal and is kept.)
            TF_FOR4(g, m64, i) {
                V4<double> xx = ld4(x64 + i);
                const V4<float> d = ld4(v32.x + i);
#pragma unroll
                for (int u = 0; u < 4; ++u) xx.a[u] = xx.a[u] - (double)d.a[u];
                st4(x64 + i, xx);
            }
            if (!grid_sync(g, 73)) return;
            if (!mixed_residual(g, m64, b64, x64, r64, v32.r, v32.x, false, err)) return;
            out.fin_res = err;
            out.exit_kind = isfinite(err_new) ? EXIT_MAXITER : EXIT_NONFINITE;
            return;
        }
        err = err_new;
        TF_FOR4(g, m64, i) { st4(v32.x + i, V4<float>{{0.f, 0.f, 0.f, 0.f}}); }
        out.fin_res = err;
        if (err < tol) {
            out.exit_kind = EXIT_CONVERGED;
            return;
        }
        stall = err > 0.9 * prev ? stall + 1 : 0;
        if (stall >= 6) break;
        prev = err;
    }
    out.exit_kind = EXIT_MAXITER;
}

// ---- mixed precision CG with reliable updates ---------------------------------
// Drift between the true and the FP32 recursive residual, relative to the
// latter, above which a reliable update also restarts the search direction.
constexpr double kReliableDrift = 0.3;

// The search direction in a pass of its own, then the product with explicit
// columns (a function of its own: registers).
static __device__ __noinline__ bool product_apart(Grid& g, const Mat<float>& m, const float* z, float* p,
                                                  float* q, float beta, bool first, float& sum) {
    direction_phase(g.tid, g.nt, m.n, z, p, beta, first);
    if (!grid_sync(g, 84)) return false;
    sum = columns_loop<float, false>(m, g.wg, g.nw, nullptr, p, nullptr, q, p, 0.0f, false);
    return true;
}

// One FP32 preconditioned CG iteration stream (FP32 values and vectors, FP64
// reductions).  Whenever its recursive residual has dropped by `inner_rtol`
// since the last refinement (or below the tolerance), the FP32 correction is
// added to x in FP64, the true residual b - A x is recomputed with the FP64
// values, the convergence test ||r|| < tol is made on it in FP64, and the
// FP32 residual is replaced by it.  Unlike a restarted refinement the search
// direction is kept, so the iteration count stays close to the FP64 solve's.
template <bool APART>
__device__ __forceinline__ void mixed_cg_reliable(Grid& g, const Mat<double>& m64, const Mat<float>& m32,
                                  double* x64, double* r64, const double* b64, double* D64,
                                  double* xbest, Vecs<float>& v, const MixedCfg& c,
                                  MixedOut& out) {
    out.exit_kind = EXIT_ABORT;
    const int prec = prec_of(c.prec);
    if (!prec1_phase(g, m64, D64, c.prec)) return;
    if (!grid_sync(g, 80)) return;
    double acc[1] = {0.0};
    TF_FOR4(g, m64, i) {
        const V4<double> d = ld4(D64 + i), bb = ld4(b64 + i);
        V4<float> df, wf;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            // FP32 solves hold 1/D for the diagonal preconditioner
            df.a[u] = c.prec == 1 ? (float)(kRecipDiag64 ? d.a[u] : div_rn(1.0, d.a[u]))
                                  : (float)d.a[u];
            wf.a[u] = Cell<float>::sentinel();
            if (i + u < m64.n) acc[0] += bb.a[u] * bb.a[u];
        }
        st4(v.D + i, df);
        st4(v.w + i, wf);
    }
    publish<1>(g, SLOT_A, acc);
    if (!grid_sync(g, 81)) return;
    if (kTiledIc && c.prec == 2 && m32.tile.on) tiles_init(g, m32, v.D);
    double tot[1], nrm[1];
    totals<1>(g, SLOT_A, tot, nrm, [](int, double s) { return sqrt(s); });
    const double bnrm2 = nrm[0];
    out.bnrm2 = bnrm2;
    const double tol = c.tol_is_relative ? c.tol * bnrm2 : c.tol;
    if (bnrm2 < tol || (c.tol_is_relative && bnrm2 == 0.0)) {
        out.exit_kind = EXIT_BNRM;
        out.iterations = 0;
        return;
    }
    const float* z = prec == 0 ? v.r : v.z;
    // r64 = b - A x; r = (float) r64; xl = 0; ||r||; z = M^-1 r (diag) and (r, z)
    // (with `drift`: also ||r_true - r_recursive||^2 into drift, the FP32
    // recursive residual being the one in v.r before it is replaced)
    auto refresh = [&](bool x_zero, double& err, double& rz, double* drift) -> bool {
        double a[3] = {0.0, 0.0, 0.0};
        for (int s = g.wg; s < m64.nslices; s += g.nw) {
            const int i = s * kWarp + g.lane;
            double ri = i < m64.n ? b64[i] : 0.0;
            if (!x_zero) ri = sell_resid_row(m64, s, g.lane, ri, x64);
            if (i < m64.n) {
                r64[i] = ri;
                const float rf = (float)ri;
                if (drift) {
                    const double dr = ri - (double)v.r[i];
                    a[2] += dr * dr;
                }
                v.r[i] = rf;
                v.x[i] = 0.0f;
                a[0] += ri * ri;
                if (prec == 1) {
                    const float zf = rf * v.D[i];
                    v.z[i] = zf;
                    a[1] += double(rf * zf);
                } else if (prec == 0) {
                    a[1] += double(rf * rf);
                }
            }
        }
        publish<3>(g, SLOT_D, a);
        if (!grid_sync(g, 82)) return false;
        double t[3], e[3];
        totals<3>(g, SLOT_D, t, e, [](int k, double s) { return k == 1 ? 0.0 : sqrt(s); });
        err = e[0];
        rz = t[1];
        if (drift) *drift = e[2];
        return true;
    };
    // rho = (r, M^-1 r), beta its ratio to the rho before
    auto ic = [&](float& beta) -> bool {
        float a[1];
        const bool ok = ic_precond<kRowDot>(g, m32, v, c.ic_sweeps, v.r, v.z, a[0]);
        publish_t<1>(g, SLOT_A, a);
        if (!grid_sync(g, 83) || !ok) return false;
        double t[1], e[1];
        totals<1>(g, SLOT_A, t, e, [&](int, double s) {
            const double b = div_rn(s, scalars().rho);
            scalars().rho = s;
            return b;
        });
        beta = (float)e[0];
        return true;
    };
    double err, rz;
    const double delta = c.inner_rtol > 0.0 && c.inner_rtol < 1.0 ? c.inner_rtol : 0.1;
    if (!refresh(c.x_is_zero != 0, err, rz, nullptr)) return;
    out.ini_res = err;
    out.fin_res = err;
    if (err < tol) {
        out.exit_kind = EXIT_INIRES;
        out.iterations = 0;
        return;
    }
    float beta = 0.0f;
    if (threadIdx.x == 0) {
        scalars().rho = rz;
        scalars().conv.set(tol);
        scalars().refine.set(delta * err);
    }
    __syncthreads();
    if (prec == 2 && !ic(beta)) return;
    // best FP64 iterate so far (returned if the iteration later diverges)
    auto keep_best = [&]() {
        TF_FOR4(g, m64, i) { st4(xbest + i, ld4(x64 + i)); }
    };
    keep_best();
    double prev = err, best = err;
    int nref = 0, stall = 0, it = 1;
    bool diverged = false, fresh = false;
    float *pcur = v.p, *pnext = v.t;
    for (; it <= c.maxiter; ++it) {
        const bool along = it == 1 || fresh;  // p = z
        float a1[1];
        if (APART) {
            direction_phase(g.tid, g.nt, m32.n, z, pcur, beta, along);
            if (!grid_sync(g, 84)) return;
            a1[0] = product_phase<float, false>(m32, g.wg, g.nw, nullptr, pcur, nullptr, v.q, pcur, 0.0f, false);
        } else if (!kApart || c.fuse_dir) {
            // the direction formed inside the product, into the other buffer
            a1[0] = product_phase<float, true>(m32, g.wg, g.nw, z, pcur, pnext, v.q, nullptr, beta, along);
            float* const pold = pcur;
            pcur = pnext;
            pnext = pold;
        } else if (!product_apart(g, m32, z, pcur, v.q, beta, along, a1[0])) {
            return;
        }
        fresh = false;
        publish_t<1>(g, SLOT_C, a1);
        if (!grid_sync(g, 85)) return;
        double t1[1], e1[1];
        totals<1>(g, SLOT_C, t1, e1, [&](int, double s) { return div_rn(scalars().rho, s); });
        const float alfa = (float)e1[0];
        const Sums3<float> u3 =
            update_phase(g.tid, g.nt, m32.n, v.x, v.r, pcur, v.q, v.D, v.z, alfa, prec == 1, false);
        const float a3[2] = {u3.a[0], u3.a[1]};
        publish_t<2>(g, SLOT_B, a3);
        if (!grid_sync(g, 86)) return;
        double t3[2], e3[2];
        totals<2>(g, SLOT_B, t3, e3, [&](int k, double s) {  // next beta; whether to refine
            if (k == 0 && prec != 0) return scalars().refine.below(s) || scalars().conv.below(s) ? 1.0 : 0.0;
            if (prec == 2 || k != (prec == 1 ? 1 : 0)) return 0.0;
            const double b = div_rn(s, scalars().rho);
            scalars().rho_old = scalars().rho;
            scalars().rho = s;
            return b;
        });
        out.iterations = it;
        if (!isfinite(t3[0])) {
            out.exit_kind = EXIT_NONFINITE;
            return;
        }
        beta = (float)e3[prec == 1 ? 1 : 0];
        const bool refine = prec != 0 ? e3[0] != 0.0
                                      : scalars().refine.below(t3[0]) || scalars().conv.below(t3[0]);
        if (refine) {
            const double rnorm = sqrt(t3[0]);
            // refinement: x += xl in FP64, true residual, FP64 test
            TF_FOR4(g, m64, i) {
                V4<double> xd = ld4(x64 + i);
                const V4<float> xl = ld4(v.x + i);
#pragma unroll
                for (int u = 0; u < 4; ++u) xd.a[u] = xd.a[u] + (double)xl.a[u];
                st4(x64 + i, xd);
            }
            if (!grid_sync(g, 87)) return;
            double drift = 0.0;
            if (!refresh(false, err, rz, &drift)) return;
            out.fin_res = err;
            out.refinements = ++nref;
            // Keep the search direction only while the recursive residual
            // it was built with is still close to the true one; a larger
            // drift (FP32 recurrences on large, ill-conditioned systems)
            // restarts it from the new preconditioned residual.
            fresh = drift > kReliableDrift * rnorm;
            if (err < tol) {
                out.exit_kind = EXIT_CONVERGED;
                return;
            }
            if (!isfinite(err)) {
                out.exit_kind = EXIT_NONFINITE;
                return;
            }
            if (err < best) {
                best = err;
                keep_best();
            } else if (err > 1e3 * best) {
                diverged = true;
                break;
            }
            stall = err > 0.999 * prev ? stall + 1 : 0;
            if (stall >= 4) break;
            prev = err;
            // the next rho is that of the refreshed residual; beta its ratio
            // to the rho of the direction kept
            if (threadIdx.x == 0) {
                scalars().refine.set(delta * err);
                if (prec != 2) {
                    scalars().beta = div_rn(rz, scalars().rho_old);
                    scalars().rho = rz;
                }
            }
            __syncthreads();
            if (prec != 2) beta = (float)scalars().beta;
        }
        if (prec == 2 && !ic(beta)) return;
    }
    // out of iterations: fold the pending correction into x, and fall back
    // to the best iterate if this one is worse
    if (!diverged) {
        TF_FOR4(g, m64, i) {
            V4<double> xd = ld4(x64 + i);
            const V4<float> xl = ld4(v.x + i);
#pragma unroll
            for (int u = 0; u < 4; ++u) xd.a[u] = xd.a[u] + (double)xl.a[u];
            st4(x64 + i, xd);
        }
        if (!grid_sync(g, 88)) return;
        if (!refresh(false, err, rz, nullptr)) return;
    }
    if (diverged || !(err <= best)) {
        TF_FOR4(g, m64, i) { st4(x64 + i, ld4(xbest + i)); }
        if (!grid_sync(g, 89)) return;
        if (!refresh(false, err, rz, nullptr)) return;
    }
    out.fin_res = err;
    out.exit_kind = err < tol ? EXIT_CONVERGED : EXIT_MAXITER;
}

}  // namespace tflows
