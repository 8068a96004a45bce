// Persistent solver kernel: the whole Newton loop (device evaluation, MNA
// stamping through the stamp map, FP64 residual, right-preconditioned
// BiCGSTAB, voltage limiting, convergence test) or a linear solve with FP64
// iterative refinement, in ONE launch: a block, a thread-block cluster or a
// cooperative grid.
//
// Algorithms followed:
//   Newton loop       src/solver/newton.rs:153-488 (newton_solve)
//   BiCGSTAB          src/solver/bicgstab.rs:56-189 (bicgstab_with_params),
//                     same operation order; breakdown tests made scale-free
//                     (see krylov()) and optionally followed by a restart
//   Jacobi            src/solver/gpu.rs:177-190, newton.rs:340-361
//   convergence       src/solver/ds_nonlinear_shaders.rs:1256-1297
//
// Each outer iteration solves the correction equation J d = b - J x in the
// Krylov precision (FP32 or FP64) and updates x in FP64.  With the reference's
// stopping rule ||b - J x_new|| < tol ||b|| (bicgstab.rs:98, 161) this is the
// reference's linear solve with a warm start; mixed precision adds an inner
// relative tolerance and falls back to an FP64 Krylov solve when the FP32 one
// fails or stalls (contraction worse than 0.5).
//
// Work split: block b owns rows [b*n/G, (b+1)*n/G).  Vector phases map one
// thread per row; SpMV phases map LPR lanes per row (sub-warp CSR).  Device
// phases are grid-strided over devices / touched slots.  Phases are separated
// by team synchronisations (GridTeam); dot products are reduced
// deterministically (per-block values, then every block sums them all in one
// fixed order), so all blocks hold bit-identical scalars and take the same branch.
#pragma once

#include <cstdint>
#include <type_traits>

#include "common.cuh"
#include "devices.cuh"

namespace ohm {

enum KrylovCode : int {
    kKrylovAbort = -1,        // a barrier gave up; leave the kernel
    kKrylovRunning = 0,
    kKrylovConverged = 1,
    kKrylovMaxIter = 2,
    kKrylovBreakRho = 3,
    kKrylovBreakRv = 4,
    kKrylovBreakTt = 5,
    kKrylovBreakOmega = 6,
    kKrylovNan = 7,
};

enum SolveStatus : int {
    kOk = 0,
    kErrSolve = 1,
    kErrNewtonNotConverged = 2,
    kErrNewtonNumerical = 3,
    kErrTimeout = 5,
};

enum PrecondKind : int { kPcAuto = 0, kPcJacobi = 1, kPcIsai = 2, kPcNone = 3 };

// Threads per block of the persistent solver (one block per SM).  512 threads
// have 128 registers each and half the per-warp overhead of a phase (barriers,
// reductions, address arithmetic) of 1024 threads with 64: DC of the 500 x 500
// diode mesh 382 -> 234 ms, of a 100 x 100 one 31.7 -> 24.7 ms (256 threads:
// 276 and 26.5 ms).
constexpr int kSolverBlock = 512;
// Threads per block of its global-memory form (GlobalTeam): the phases of
// krylov() and krylov_isai() wait for loads from L2 and HBM, and 512 threads
// have too few in flight (us per iteration at 512 -> 1024 threads: 2000 x 2000
// mesh 525 -> 357, the same in FP32 474 -> 288, 1000 x 1000 mesh in random order
// 163 -> 113).
constexpr int kWideBlock = 1024;

// Breakdown test: |(a, b)| < kBreakdownRel * ||a|| ||b||.  The reference's
// absolute 1e-30 (bicgstab.rs:107, :125) depends on the units of the
// residual; a relative test only fires on (near-)exact orthogonality.
constexpr double kBreakdownRel = 1e-24;

struct DeviceInfo {
    int status;
    int krylov_code;
    int iterations;          // Newton iterations, or refinement sweeps for a linear solve
    int error_iteration;
    long long krylov_iterations;
    int fp64_fallbacks;      // mixed precision: Krylov solves redone in FP64
    int krylov_restarts;
    double max_residual;     // last max|x - x_old|
    double final_residual;   // ||b - A x||_2 (FP64) at exit, linear mode
    double b_norm;
    int continuation_steps;  // Newton runs of the DC continuation after the direct attempt
    int continuation_kind;   // kContNone / kContSource / kContGmin / kContPseudo: last stage used
};

// DC continuation stages (src/analysis/dc.rs:60-290).
enum ContKind : int { kContNone = 0, kContSource = 1, kContGmin = 2, kContPseudo = 3 };

struct KernelArgs {
    // CSR system (u32 indices, FP64 assembled values, FP32 copy for mixed)
    int n, nnz;
    const uint32_t *row_ptr, *col;
    double *vals64;
    float *vals32;
    const double *base_vals;    // Newton: values without device stamps
    const double *base_b;
    double *b;                  // assembled rhs (linear: the rhs)
    double *x;                  // FP64 iterate (in: initial guess, out: solution)
    double *x_prev;             // FP64 previous Newton iterate
    double *r64;                // FP64 residual b - A x
    double *dx;                 // FP64 correction from the Krylov solve

    // block-Jacobi preconditioner (1x1, or 2x2 pairs for zero-diagonal rows)
    int precond;
    const int32_t *partner;     // -1: unpaired
    const uint32_t *diag_slot;  // CSR slot of (i,i), kSentinel if absent
    const uint32_t *off_slot;   // CSR slot of (i, partner(i))
    const uint8_t *rowflag;     // 1: row i or one of its columns is paired
    void *pc_part;              // Krylov-precision coefficient on the partner

    // Krylov state.  rec0/rec1: per-row records {p, v, r, c} (c = the
    // preconditioner's self coefficient), double-buffered; the SpMV of each
    // phase gathers one record (one 32-byte sector in FP64) per nonzero and
    // forms M^-1 p or M^-1 s on the fly.  Other vectors: own rows only.
    void *rec0, *rec1, *rhat, *s, *t, *phat, *shat, *d;

    // nonlinear devices and the stamp map
    int nd, nq, nm;
    const DiodeDesc *diodes;
    const BjtDesc *bjts;
    const MosfetDesc *mosfets;
    const double *bjt_vaf;      // may be null
    double *mstamp, *rstamp;    // per-device stamp values
    int n_mslots;
    const uint32_t *mslot, *mslot_ptr, *mslot_ids;
    int n_rrows;
    const uint32_t *rrow, *rrow_ptr, *rrow_ids;
    unsigned long long *node_scale;

    // Long rows / long stamp segments handled by the whole team (see
    // spmv_long and the stamp pass).  longflag[i] = 1 for a long row.
    int n_long, n_long_chunks;
    const uint8_t *longflag;
    const uint32_t *long_row, *long_chunk_ptr, *long_chunk_owner, *long_chunk_beg, *long_chunk_end;
    double *long_part;
    // stamp segments (index k over mslots then rrows) with many contributions
    int n_lseg, n_lseg_chunks;
    const uint32_t *lseg, *lseg_chunk_ptr, *lseg_chunk_owner, *lseg_chunk_beg, *lseg_chunk_end;
    const uint8_t *lseg_flag;    // per mslot/rrow entry: 1 if handled as a long segment
    double *lseg_part;

    // DC continuation (src/analysis/dc.rs): bit 0 = on failure of the direct
    // Newton solve, run source stepping (MOSFET circuits), GMIN stepping and
    // pseudo-transient continuation on the device; bit 1 (testing) = treat
    // the true-GMIN solve after GMIN stepping as failed.  n_nodes: node rows come
    // first (MNA order).  stampflag per row: bit 0 = its diagonal slot is
    // written by the stamp map, bit 1 = its rhs entry is.  x_good: last
    // converged continuation point (size n).
    int continuation;
    int n_nodes;
    const uint8_t *stampflag;
    double *x_good;

    // control
    int newton;                 // 1: Newton loop, 0: linear solve (+ refinement)
    int mixed;                  // 1: FP32 Krylov with FP64 fallback
    int max_outer;              // Newton iterations or refinement sweeps
    double abs_tol, rel_tol;    // Newton convergence
    int max_krylov;
    double krylov_tol;          // ||r|| < krylov_tol * ||b||  (bicgstab.rs:98)
    double inner_rtol;          // ... or < inner_rtol * ||r0|| (inexact inner solve)
    int forcing;                // 1: Eisenstat-Walker inner tolerance, floor inner_rtol
    double eta_max;             // Eisenstat-Walker upper bound
    int fp32_max_iterations;    // mixed: iteration cap of an FP32 attempt before FP64
    double fp32_min_eta;        // mixed Newton: inner tolerances below this go straight to FP64
    int max_restarts;           // restarts with r_hat = r after a breakdown
    double *trace;              // optional per-outer-iteration record (kTraceCols doubles)
    int trace_cap;
    int require_true_residual;  // linear: fail unless the FP64 residual meets the tolerance

    // ISAI(1): augmented pattern (A + diagonal), Chow-Patel product lists,
    // factor values (double-buffered), M_L / M_U (CSR values + column lists)
    const uint32_t *aug_rp, *aug_col, *aug_diag;
    const int32_t *aug_map;
    const uint32_t *cp_ptr, *cp_pair;
    double *isai_f0, *isai_f1;
    const uint32_t *ml_rp, *ml_col, *ml_cp, *ml_row, *ml_pos;
    double *ml_val;
    const uint32_t *mu_rp, *mu_col, *mu_cp, *mu_row, *mu_pos;
    double *mu_val;

    double *partials;           // >= 8 * gridDim.x doubles (two alternating regions)
    GridSync gs;
    DeviceInfo *info;
    // dynamic shared memory of the launch: when > 0 the Krylov solve keeps each
    // block's slice there as far as it fits (krylov_slice()).  nnz_long:
    // nonzeros of the long rows (host side, sizes that slice).  cluster: the
    // grid is one thread-block cluster.  slice_col and slice_val (5
    // entries per 4 nonzeros), slice_export (u8 per row), cself and rself (8
    // bytes per row) are that solve's workspace.
    // scatter (host side): how far the rows of a block reach (ohm_scatter()).
    int smem_bytes;
    int64_t nnz_long;
    int cluster;
    int scatter;
    uint16_t *slice_col;
    double *slice_val;
    uint8_t *slice_export;
    void *cself, *rself;
};

// Columns of the per-outer-iteration trace: FP32 Krylov iterations, FP64
// Krylov iterations, ||b - J x|| (FP64) before the solve, inner tolerance
// used, max|x - x_old| after limiting, restarts.
constexpr int kTraceCols = 6;

// What a block knows about its slice of the system (krylov_slice()), built at
// the first Krylov solve of a launch: H halo rows, matrix slices of 32 W entries.
enum SliceState : int {
    kSliceNone = 0,     // not built yet
    kSliceChip = 1,     // everything in shared memory
    kSliceStream = 2,   // gather vector in shared memory, matrix slices in global memory
    kSliceCsr = 3,      // gather vector in shared memory, the matrix in CSR form
    kSliceNo = 4,       // does not fit: global-memory solve
};
struct SliceMap {
    int state, H, W, pairs;   // W: padded nonzeros / 32
};

// A team is the set of threads that solves one system: the whole grid (one
// large circuit, GridTeam) or one block (one circuit of a batch, BlockTeam).
// Both expose the rows this block owns [r0, r1), a thread index / stride over
// the team for device- and slot-parallel loops, sync() and deterministic
// all-reductions whose results are bit-identical in every thread.
// A grid of one block synchronises within the block; a grid of up to 16
// blocks is launched as one cluster and meets at cluster barriers with its
// dot products exchanged through distributed shared memory; larger grids
// meet at the counter barrier.  The sums have the same order in all three.
// SLICES: whether the kernel has krylov_slice(); without it (kWideBlock
// threads) the team works from global memory.
template <bool SLICES>
struct GridTeamT {
    static constexpr bool kSlices = SLICES;
    int G, bid, r0, r1, gtid, gstride;
    double *smem;
    double *partials;
    bool cluster;
    GridSync gs;
    SliceMap map;

    __device__ __forceinline__ void init(const KernelArgs &a) {
        G = gridDim.x;
        bid = blockIdx.x;
        r0 = (int)(((long long)a.n * bid) / G);
        r1 = (int)(((long long)a.n * (bid + 1)) / G);
        gtid = bid * blockDim.x + threadIdx.x;
        gstride = G * blockDim.x;
        smem = reduce_buffers().warp;
        partials = a.partials;
        cluster = a.cluster != 0;
        gs = a.gs;
        map.state = kSliceNone;
        reduce_buffers_init();
        if (cluster) cluster_barrier();     // peers' shared memory exists from here on
    }
    __device__ __forceinline__ bool sync() {
        if (gridDim.x == 1) { __syncthreads(); return true; }
        if (cluster) { cluster_barrier(); return true; }
        return grid_barrier(gs);
    }
    __device__ __forceinline__ bool leader() const { return blockIdx.x == 0 && threadIdx.x == 0; }
    template <int NV, bool MAX = false, typename Fin>
    __device__ __forceinline__ bool reduce_then(const double (&v)[NV], Fin fin) {
        return team_reduce_then<NV, MAX>((int)gridDim.x, (int)blockIdx.x, cluster, partials, gs, v, fin);
    }
    template <int NV, bool MAX>
    __device__ __forceinline__ bool reduce(double (&v)[NV]) {
        double *res = reduce_buffers().res;
        const bool ok = reduce_then<NV, MAX>(v, [&](const double (&t)[NV], bool writer) {
            if (writer) {
#pragma unroll
                for (int k = 0; k < NV; ++k) res[k] = t[k];
            }
        });
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] = res[k];
        return ok;
    }
    template <int NV>
    __device__ __forceinline__ bool allreduce(double (&v)[NV]) { return reduce<NV, false>(v); }
    template <int NV>
    __device__ __forceinline__ bool allmax(double (&v)[NV]) { return reduce<NV, true>(v); }
};

using GridTeam = GridTeamT<true>;
using GlobalTeam = GridTeamT<false>;
template <class Team>
constexpr int kTeamBlock = Team::kSlices ? kSolverBlock : kWideBlock;

struct BlockTeam {
    static constexpr bool kSlices = true;
    int r0, r1, gtid, gstride;
    double *smem;
    SliceMap map;

    template <int NV, bool MAX = false, typename Fin>
    __device__ __forceinline__ bool reduce_then(const double (&v)[NV], Fin fin) {
        return team_reduce_then<NV, MAX>(1, 0, false, nullptr, GridSync{nullptr, nullptr}, v, fin);
    }

    __device__ __forceinline__ bool sync() { __syncthreads(); return true; }
    __device__ __forceinline__ bool leader() const { return threadIdx.x == 0; }
    template <int NV>
    __device__ __forceinline__ bool allreduce(double (&v)[NV]) { block_sum<NV>(v, smem); return true; }
    template <int NV>
    __device__ __forceinline__ bool allmax(double (&v)[NV]) { block_max<NV>(v, smem); return true; }
};

template <typename T>
__device__ __forceinline__ T cvt(double x) { return (T)x; }

// y_i = sum_j A_ij x(j) for the rows of this block, where x(j, slow) is a
// gather functor; `f(row, y_i)` runs on the first lane of each row group.
// Each group keeps kRowsInFlight rows in flight (their row pointers, nonzeros
// and gathers are issued together), so the dependent L2 round trips of one row
// overlap those of the others.  All lanes of a warp run the same number of
// tiles and inner steps, so the group shuffles are safe.  `slow` is the row's
// flag from `rowflag` (false when null).  rp is indexed by row - rp_off (a
// block's local CSR slice has rp_off = its first row).
constexpr int kRowsInFlight = 4;

template <int LPR, typename Acc, typename TA, typename X, typename F, int U = kRowsInFlight, bool PIPE = false,
          typename TR, typename TC>
__device__ __forceinline__ void spmv_rows(const TR *__restrict__ rp, const TC *__restrict__ col,
                                          const TA *__restrict__ val, const uint8_t *rowflag,
                                          int r0, int r1, X x, F f, const uint8_t *skip = nullptr,
                                          int rp_off = 0) {
    const int lane = threadIdx.x % LPR;
    const int group = threadIdx.x / LPR;
    const int ngroups = blockDim.x / LPR;
    for (int tile = r0; tile < r1; tile += ngroups * U) {
        int row[U];
        uint32_t beg[U], end[U];
        bool slow[U];
        Acc acc[U];
        uint32_t len = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            row[u] = tile + group + u * ngroups;
            const bool ok = row[u] < r1 && !(skip != nullptr && skip[row[u]] != 0);
            beg[u] = ok ? rp[row[u] - rp_off] : 0u;
            end[u] = ok ? rp[row[u] - rp_off + 1] : 0u;
            slow[u] = ok && rowflag != nullptr && rowflag[row[u]] != 0;
            acc[u] = Acc(0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) len = max(len, end[u] - beg[u]);
        // the longest row of the group decides the step count; shuffles below
        // need every lane of the warp, so take the warp-wide maximum
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) len = max(len, __shfl_xor_sync(0xffffffffu, len, o));
        if constexpr (PIPE) {
            // rows in shared memory: unrolled, so the gathers of several
            // nonzeros are in flight together
#pragma unroll 4
            for (uint32_t off = lane; off < len; off += LPR) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t k = beg[u] + off;
                    if (k < end[u]) acc[u] += (Acc)val[k] * (Acc)x((int)col[k], slow[u]);
                }
            }
        } else {
            for (uint32_t off = lane; off < len; off += LPR) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t k = beg[u] + off;
                    if (k < end[u]) acc[u] += (Acc)val[k] * (Acc)x((int)col[k], slow[u]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int o = LPR / 2; o > 0; o >>= 1) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o, LPR);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (lane == 0 && row[u] < r1 && !(skip != nullptr && skip[row[u]] != 0)) f(row[u], (double)acc[u]);
    }
}

// Block of the team that finishes team-shared work item q (grid teams: block
// q mod G; BlockTeam: its only block), and whether this block owns row i.
template <class Team>
__device__ __forceinline__ bool team_owns_item(const Team &g, int q) {
    if constexpr (!std::is_same<Team, BlockTeam>::value) return q % g.G == g.bid;
    else return true;
}

// Long rows (a hub node such as a supply rail, whose row holds a nonzero per
// connected device) are skipped by spmv_rows and computed by the whole team:
// one warp per chunk of at most a couple of hundred nonzeros writes a partial
// (4 nonzeros per lane, their loads issued together), a team sync, then the
// block that owns the row sums its partials with all its threads (a fixed
// tree, so the value does not depend on timing) and calls f(row, y) like
// spmv_rows does, on one thread.  The callback may therefore use the owning
// block's shared memory.  Returns false if the sync gave up.
template <typename Acc, class Team, typename TA, typename X, typename F>
__device__ __forceinline__ bool spmv_long(const KernelArgs &a, Team &g, const uint32_t *__restrict__ col,
                                          const TA *__restrict__ val, const uint8_t *rowflag, X x, F f) {
    if (a.n_long == 0) return true;
    const int lane = threadIdx.x & 31;
    const int warp = g.gtid >> 5, nwarps = g.gstride >> 5;
    for (int c = warp; c < a.n_long_chunks; c += nwarps) {
        const uint32_t row = a.long_row[a.long_chunk_owner[c]];
        const bool slow = rowflag != nullptr && rowflag[row] != 0;
        Acc acc = Acc(0);
        const uint32_t kend = a.long_chunk_end[c];
#pragma unroll 4
        for (uint32_t k = a.long_chunk_beg[c] + lane; k < kend; k += 32)
            acc += (Acc)val[k] * (Acc)x((int)col[k], slow);
        double s = (double)acc;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) a.long_part[c] = s;
    }
    if (!g.sync()) return false;
    for (int j = 0; j < a.n_long; ++j) {
        const int row = (int)a.long_row[j];
        if (row < g.r0 || row >= g.r1) continue;          // uniform over the block
        double v[1] = {0.0};
        for (uint32_t c = a.long_chunk_ptr[j] + threadIdx.x; c < a.long_chunk_ptr[j + 1]; c += blockDim.x)
            v[0] += a.long_part[c];
        block_sum<1>(v, g.smem);
        if (threadIdx.x == 0) f(row, v[0]);
    }
    return true;
}

// Per-row Krylov record: p, v, r and the preconditioner's self coefficient.
template <typename T>
struct alignas(4 * sizeof(T)) KRec {
    T p, v, r, c;
};

#define OHM_SYNC_OR(ret)                \
    do {                                \
        if (!g.sync()) return ret;      \
    } while (0)

struct KrylovOut {
    int iterations;
    int restarts;
};

// Dynamic shared memory of the grid-team kernels: the Krylov solve keeps
// each block's own-row state and CSR slice here when the launch provides
// enough of it (KernelArgs::smem_bytes).
extern __shared__ __align__(128) unsigned char ohm_dsmem[];

// Exclusive prefix sum over the block of one value per thread (in thread
// order); *total receives the block sum.  `scratch` holds >= 33 words.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *scratch, uint32_t *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = (blockDim.x + 31) >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    __syncthreads();
    if (lane == 31) scratch[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < nwarps ? scratch[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        scratch[lane] = w;                       // inclusive prefix of warp sums
        if (lane == 31) scratch[32] = w;
    }
    __syncthreads();
    const uint32_t before = (warp > 0 ? scratch[warp - 1] : 0u) + inc - v;
    *total = scratch[32];
    __syncthreads();
    return before;
}

// A breakdown at a residual more than ten times the initial one (||W r||,
// compared as squares) gives the solve's work up, once: back to d = 0 and
// r = r64, with the shadow residual r64 + g r, g = ||r64|| / ||r|| (its product
// with r64 is not small: a breakdown of rho makes r orthogonal to the first
// shadow residual).  Such breakdowns come after a spike of the recurrence; 4
// of 440 solves of a 600 x 600 diode mesh (1.0 V, 5 % diodes) met one, at 140 to
// 2.6e8 times the initial residual, and one of them then spent the rest of its
// 20,000 iterations above it.  FP64 solves only (the FP32 attempts have few
// iterations and an FP64 solve after them), and only where no DC continuation
// follows a failure: its direct attempts often cannot succeed, and trying them
// longer took most of a batch's time (ten batches of 512 amplifiers 1.40 -> 1.89
// s).
constexpr double kRestartFromStart = 100.0;
template <typename T>
__device__ __forceinline__ bool restarts_from_start(const KernelArgs &a) {
    return sizeof(T) == 8 && a.continuation == 0;
}

// |x| < rel sqrt(y), compared as squares: a square root is 120 cycles on the
// one lane that every thread waits for.  Where a square would leave the
// normal range the root decides.  krylov() and krylov_slice() share these
// tests: blocks of one team may run either form, and all of them have to take
// the same branch.
__device__ __forceinline__ bool below_root(double x, double rel, double y) {
    const double x2 = x * x, y2 = rel * rel * y;
    if (x2 > 1e-290 && x2 < 1e290 && y2 > 1e-290 && y2 < 1e290) return x2 < y2;
    return !(fabs(x) >= rel * sqrt(y));
}
// sqrt(y) < tol, tol2 = tol^2.
__device__ __forceinline__ bool root_below(double y, double tol, double tol2) {
    return tol2 > 1e-290 && tol2 < 1e290 ? y < tol2 : sqrt(y) < tol;
}

// Right-preconditioned BiCGSTAB on J d = r64 in precision T, d0 = 0, with
// the reference's operation order (bicgstab.rs:104-183) and three grid
// synchronisations per iteration:
//   AB: p = (p - w v) b + r and v = A M^-1 p  (M^-1 p formed on the fly per
//       gathered record), reduce (r_hat, v), (v, v)
//   CD: s = r - a v and t = A M^-1 s (on the fly), reduce (s, s), (t, s), (t, t)
//   E : d += a phat + w shat; r = s - w t, reduce (r_hat, r), (r, r)
// phat = M^-1 p, s and shat = M^-1 s are re-formed from the row's record
// where they are needed instead of being stored (the same expressions, so
// the same values).  The early exit on ||s|| (bicgstab.rs:134-139) is taken
// after CD; t is then simply unused.  Stops when ||r|| < max(tol_floor,
// inner_rtol * ||r0||).  On success the correction is left in a.dx (FP64)
// for the rows of this block.
//
// This is the global-memory form (slices whose gathered vector does not fit in
// shared memory, and OHM_KRYLOV_LAYOUT_GLOBAL); krylov_slice() is the same
// iteration with each block's slice in shared memory.
//
// Newton solves measure that stopping norm on the diagonally scaled residual
// W r, w_i = 1/|J_ii| (1 for a zero diagonal): volts instead of amperes, so a
// junction row with a huge conductance cannot hide unresolved corrections on
// the other rows behind a relative tolerance.  Linear solves keep the
// reference's unscaled ||r|| < tol ||b||.
template <typename T, int LPR, class Team>
__device__ __forceinline__ int krylov(const KernelArgs &a, Team &g, double tol_floor, double inner_rtol,
                                      int max_it, bool accept_partial, KrylovOut &out) {
    using Acc = T;   // FP32 SpMV accumulates in FP32, FP64 in FP64; dots always in FP64
    const int r0 = g.r0, r1 = g.r1;
    KRec<T> *cur = (KRec<T> *)a.rec0, *nxt = (KRec<T> *)a.rec1;
    T *pc_part = (T *)a.pc_part;
    const int32_t *partner = a.partner;
    const T *A;
    if constexpr (sizeof(T) == 4) A = (const T *)a.vals32; else A = (const T *)a.vals64;
    out.iterations = 0;
    out.restarts = 0;
    const bool wt = a.newton != 0;

    T *rhat = (T *)a.rhat + r0, *t = (T *)a.t + r0;   // own rows, local index
    // 8 bytes a row in either precision, as krylov_slice() keeps it: blocks of
    // one team that run different forms must not overlap
    T *d = (T *)((double *)a.d + r0);
    T *s_pair = (T *)a.s;   // s of the rows of 2x2 pairs (read by the partner in E)
    double *w = a.dx + r0;
    auto own = [&](KRec<T> *buf, int i) -> KRec<T> { return buf[i]; };
    // (as in krylov_slice(): with other preconditioners its blocks leave no s_pair)
    const bool pairs = a.precond == kPcAuto;
    auto is_paired = [&](int i) -> bool { return pairs && partner[i] >= 0; };

    double r0norm = 0.0, abs_tol = 0.0, tol2 = 0.0;     // stopping norm (scaled for Newton)
    double rr0 = 0.0, rw0 = 0.0;
    double rr_cur = 0.0, rw_cur = 0.0;    // ||r||^2, ||W r||^2
    double rhat2 = 0.0;                   // ||r_hat||^2
    double rho_new = 0.0;                 // (r_hat, r)
    double rho = 1.0, alpha = 1.0, omega = 1.0, mix = 0.0;
    int code = kKrylovRunning;
    int it = 0;

    // restart: r_hat = r, p = v = 0.  The shadow residual r_hat = b
    // (bicgstab.rs:87) can be orthogonal to later residuals when b lives on a
    // few source rows.
#define OHM_RESTART()                                                          \
    do {                                                                       \
        for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {              \
            KRec<T> q = own(cur, i);                                           \
            q.p = T(0); q.v = T(0);                                            \
            cur[i] = q;                                                        \
            rhat[i - r0] = q.r;                                                \
        }                                                                      \
        OHM_SYNC_OR(kKrylovAbort);                                             \
        rho = 1.0; alpha = 1.0; omega = 1.0;                                   \
        rho_new = rr_cur; rhat2 = rr_cur;                                      \
        ++out.restarts;                                                        \
    } while (0)

    // M^-1 applied to a row's own vector u (the self coefficient c of the
    // row's record, plus the partner term for a 2x2 pair): the same
    // expression as in the gathers below, so the same rounding.
    auto pc_apply = [&](int i, double c, T u, bool pair, T u_partner) -> T {
        double z = c * (double)u;
        if (pair) z += (double)pc_part[i] * (double)u_partner;
        return cvt<T>(z);
    };

    for (bool again = false;; again = true) {       // twice at most (kRestartFromStart)
        // ---- start: r = r64, r_hat = r (again: r64 + g r), p = v = d = 0;
        //      preconditioner coefficients ----
        double acc0[4] = {0.0, 0.0, 0.0, 0.0};     // ||r||^2, ||W r||^2, (r_hat, r), ||r_hat||^2
        KRec<T> *const old = cur;
        cur = (KRec<T> *)a.rec0;
        nxt = (KRec<T> *)a.rec1;
        for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
            const int li = i - r0;
            const T rt = cvt<T>(a.r64[i]);
            double cs = 0.0, cp = 0.0;
            const uint32_t ds = a.diag_slot[i];
            const double aii = ds == kSentinel ? 0.0 : a.vals64[ds];
            const double wi = (wt && fabs(aii) > 1e-30) ? 1.0 / fabs(aii) : 1.0;
            if (wt) w[li] = wi;
            if (a.precond != kPcNone) {
                const int pi = partner[i];
                if (a.precond == kPcAuto && pi >= 0) {
                    const double akk = a.diag_slot[pi] == kSentinel ? 0.0 : a.vals64[a.diag_slot[pi]];
                    const double aik = a.vals64[a.off_slot[i]];
                    const double aki = a.vals64[a.off_slot[pi]];
                    const double det = aii * akk - aik * aki;
                    if (fabs(det) > 1e-300) { cs = akk / det; cp = -aik / det; }
                } else if (fabs(aii) > 1e-30) {
                    cs = 1.0 / aii;
                } else if (a.precond == kPcAuto) {
                    cs = 1.0;   // unpaired zero diagonal: identity keeps M^-1 nonsingular
                }
            } else {
                cs = 1.0;
            }
            const T rh = again ? cvt<T>(fma(mix, (double)old[i].r, (double)rt)) : rt;
            KRec<T> q;
            q.p = T(0); q.v = T(0); q.r = rt; q.c = cvt<T>(cs);
            cur[i] = q;
            pc_part[i] = cvt<T>(cp);
            rhat[li] = rh;
            d[li] = T(0);
            acc0[0] += (double)rt * (double)rt;
            acc0[1] += (wi * (double)rt) * (wi * (double)rt);
            acc0[2] += (double)rh * (double)rt;
            acc0[3] += (double)rh * (double)rh;
        }
        {
            if (!g.template allreduce<4>(acc0)) return kKrylovAbort;
        }
        rr_cur = acc0[0]; rw_cur = acc0[1]; rho_new = acc0[2]; rhat2 = acc0[3];
        rho = 1.0; alpha = 1.0; omega = 1.0;
        if (!again) {
            rr0 = rr_cur;
            rw0 = rw_cur;
            r0norm = sqrt(rw_cur);
            abs_tol = fmax(tol_floor, inner_rtol * r0norm);
            tol2 = abs_tol * abs_tol;
            if (!isfinite(r0norm)) { code = kKrylovNan; break; }
            if (r0norm < abs_tol || r0norm == 0.0) { code = kKrylovConverged; break; }
        }
        const bool try_start = restarts_from_start<T>(a);
        bool back = false;
        for (; it < max_it; ++it) {
            if (below_root(rho_new, kBreakdownRel, rhat2 * rr_cur)) {
                if (out.restarts < a.max_restarts && rr_cur > 0.0) {
                    back = try_start && !again && rw_cur > kRestartFromStart * rw0;
                    if (back) break;
                    OHM_RESTART();
                } else {
                    code = kKrylovBreakRho;
                    break;
                }
            }
            const double beta = (rho_new / rho) * (alpha / omega);
            rho = rho_new;
            const double om = omega;
            // ---------------- AB: p update and v = A M^-1 p ----------------
            auto pnew = [&](const KRec<T> &q) -> T {
                return cvt<T>(((double)q.p + (-om) * (double)q.v) * beta + (double)q.r);
            };
            auto phat_at = [&](int j, bool slow) -> T {
                const KRec<T> q = cur[j];
                double z = (double)q.c * (double)pnew(q);
                if (slow) {
                    const int pj = partner[j];
                    if (pj >= 0) z += (double)pc_part[j] * (double)pnew(cur[pj]);
                }
                return cvt<T>(z);
            };
            double acc1[2] = {0.0, 0.0};
            auto ab_row = [&](int i, double y) {
                const KRec<T> q = own(cur, i);
                KRec<T> n;
                n.p = pnew(q);
                n.v = cvt<T>(y);
                n.r = q.r;
                n.c = q.c;
                nxt[i] = n;
                acc1[0] += (double)rhat[i - r0] * (double)n.v;
                acc1[1] += (double)n.v * (double)n.v;
            };
            spmv_rows<LPR, Acc>(a.row_ptr, a.col, A, a.rowflag, r0, r1, phat_at, ab_row, a.longflag);
            if (!spmv_long<Acc>(a, g, a.col, A, a.rowflag, phat_at, ab_row)) return kKrylovAbort;
            {
                if (!g.template allreduce<2>(acc1)) return kKrylovAbort;
            }
            if (below_root(acc1[0], kBreakdownRel, rhat2 * acc1[1])) {
                if (out.restarts < a.max_restarts && rr_cur > 0.0) {
                    if (it + 1 >= max_it) {
                        // the limit comes first, with no restart and no sync,
                        // as in krylov_scalars_step()
                        ++out.restarts;
                        ++it;
                        code = kKrylovMaxIter;
                        break;
                    }
                    back = try_start && !again && rw_cur > kRestartFromStart * rw0;
                    if (back) { ++it; break; }
                    OHM_RESTART();        // cur still holds r; restart from it
                    continue;
                }
                code = kKrylovBreakRv;
                break;
            }
            alpha = rho / acc1[0];
            const double al = alpha;
            // phat of an own row from its record in nxt (p is the new p)
            auto phat_own = [&](int i, const KRec<T> &q) -> T {
                const bool pair = is_paired(i);
                return pc_apply(i, (double)q.c, q.p, pair, pair ? nxt[partner[i]].p : T(0));
            };
            // ---------------- CD: s = r - a v and t = A M^-1 s ----------------
            auto s_of = [&](const KRec<T> &q) -> T {
                return cvt<T>((double)q.r + (-al) * (double)q.v);
            };
            auto shat_at = [&](int j, bool slow) -> T {
                const KRec<T> q = nxt[j];
                double z = (double)q.c * (double)s_of(q);
                if (slow) {
                    const int pj = partner[j];
                    if (pj >= 0) z += (double)pc_part[j] * (double)s_of(nxt[pj]);
                }
                return cvt<T>(z);
            };
            double acc3[4] = {0.0, 0.0, 0.0, 0.0};   // (s,s), (t,s), (t,t), ||W s||^2
            auto cd_row = [&](int i, double y) {
                const T si = s_of(own(nxt, i));
                const T ti = cvt<T>(y);
                t[i - r0] = ti;
                if (is_paired(i)) s_pair[i] = si;
                const double ws = wt ? w[i - r0] * (double)si : (double)si;
                acc3[0] += (double)si * (double)si;
                acc3[1] += (double)ti * (double)si;
                acc3[2] += (double)ti * (double)ti;
                acc3[3] += ws * ws;
            };
            spmv_rows<LPR, Acc>(a.row_ptr, a.col, A, a.rowflag, r0, r1, shat_at, cd_row, a.longflag);
            if (!spmv_long<Acc>(a, g, a.col, A, a.rowflag, shat_at, cd_row)) return kKrylovAbort;
            {
                if (!g.template allreduce<4>(acc3)) return kKrylovAbort;
            }
            if (root_below(acc3[3], abs_tol, tol2)) {   // early exit (bicgstab.rs:134-139)
                for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
                    const T ph = phat_own(i, own(nxt, i));
                    d[i - r0] = cvt<T>((double)d[i - r0] + al * (double)ph);
                }
                code = kKrylovConverged;
                ++it;
                break;
            }
            if (!(acc3[2] > 0.0)) { code = kKrylovBreakTt; break; }
            omega = acc3[1] / acc3[2];
            // ---------------- E: d, r updates ----------------
            double acc4[3] = {0.0, 0.0, 0.0};   // (r_hat, r), ||r||^2, ||W r||^2
            for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
                const int li = i - r0;
                const KRec<T> q = own(nxt, i);
                const bool pair = is_paired(i);
                const int pi = pair ? partner[i] : i;
                // the partner's p and s as formed in AB / CD (its r changes in this loop)
                const T ph = pc_apply(i, (double)q.c, q.p, pair, pair ? nxt[pi].p : T(0));
                const T si = s_of(q);
                const T sh = pc_apply(i, (double)q.c, si, pair, pair ? s_pair[pi] : T(0));
                d[li] = cvt<T>(((double)d[li] + al * (double)ph) + omega * (double)sh);
                const T rt = cvt<T>((double)si + (-omega) * (double)t[li]);
                nxt[i].r = rt;
                const double wr = wt ? w[li] * (double)rt : (double)rt;
                acc4[0] += (double)rhat[li] * (double)rt;
                acc4[1] += (double)rt * (double)rt;
                acc4[2] += wr * wr;
            }
            {
                if (!g.template allreduce<3>(acc4)) return kKrylovAbort;
            }
            { KRec<T> *tmp = cur; cur = nxt; nxt = tmp; }
            rho_new = acc4[0];
            rr_cur = acc4[1];
            rw_cur = acc4[2];
            if (!isfinite(acc4[2])) { code = kKrylovNan; ++it; break; }
            if (root_below(acc4[2], abs_tol, tol2)) { code = kKrylovConverged; ++it; break; }
            if (fabs(omega) < 1e-30) { code = kKrylovBreakOmega; ++it; break; }
            if (accept_partial && it + 1 == max_it && sqrt(acc4[2]) <= 0.5 * r0norm) {
                code = kKrylovConverged;          // inexact inner solve accepted
                ++it;
                break;
            }
        }
        if (!back) {
            if (code == kKrylovRunning) code = kKrylovMaxIter;
            break;
        }
        mix = sqrt(rr0 / rr_cur);
        ++out.restarts;
    }
#undef OHM_RESTART
    out.iterations = it;
    if (code == kKrylovConverged)
        for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) a.dx[i] = (double)d[i - r0];
    return code;
}

}  // namespace ohm

#include "isai.cuh"

namespace ohm {

// krylov() with each block's slice of the system in shared memory.
//
// What bounds it: the working set sits on the chip, so an iteration is a
// chain of latencies (three team reductions, and in each SpMV phase the round
// trip to the neighbours' rows) and of issued instructions.  So:
//   * each phase first forms the vector that the product gathers (M^-1 p or
//     M^-1 s) once per row into shared memory, z: the block's own rows from
//     its own state, the rows of other blocks that its nonzeros touch (the
//     halo: about 1,000 rows for the 8,400 nonzeros of a 1,690-row slice of a
//     500 x 500 mesh) from the records that their owners publish, every
//     remote record fetched once and all of them at the same time;
//   * the matrix is stored in slices of 32 rows padded to their longest row,
//     entry k of the 32 rows side by side (16-bit local columns; padding has
//     value 0 and the column of a zero): a warp's loads are consecutive, the
//     product costs three shared-memory loads and an FMA per nonzero;
//   * own-row state is one array per field (no bank conflicts), and only rows
//     in someone's halo are published (slice_export);
//   * the scalars of the recurrence live in shared memory and are updated by
//     one lane inside the reductions (KrylovScalars): every thread repeating
//     the divisions and square roots cost 300 of 1,350 instructions per warp
//     and iteration, and the registers that held them were spilled.
// Measured together with the cluster teams and the cheaper reductions (B200,
// 512 threads a block), before -> after: DC of the 500 x 500 diode mesh (one
// block per SM, 1,690 rows each) 340 -> 238 ms, 23.5 -> 16 us per BiCGSTAB
// iteration; 100 x 100 mesh (a cluster of 10) 47 -> 27 ms; 600 x 600 mesh
// (stream layout) 760 -> 473 ms; 200 steps of a 401-row transient (one block)
// 116 -> 44 ms.
// The values and their order are krylov()'s, so the results are bit-identical
// (fma is written out where two phases share code: a product merged from two
// branches is not contracted).
//
// Layouts, chosen per block when the slice map is built:
//   chip   everything in shared memory;
//   stream (larger slices) z and the vectors, in the order of their traffic,
//          while they fit; the 32-row slices of the matrix in global memory,
//          the values of as many as still fit on the chip (600 x 600 mesh,
//          2,432 rows a block: 2 % of a solve);
//   csr    (several lanes per row, or rows too uneven to pad) vectors as in
//          `stream`; the matrix in compact rows with local column indices, on
//          the chip where it fits.  Blocks with a few long rows: without it they
//          ran krylov() (whole linear solves, 54 of 27,200 rows with 100 entries
//          15.8 -> 6.8 ms, 400 of 200,000 31.5 -> 13.8 ms; 20 steps of a
//          1,200-stage CMOS chain 61 -> 21 ms);
//   none   z does not fit, or the halo overflows its table: krylov().
// A block chooses for itself: blocks exchange data only through the published
// records and the reductions (one without a slice marks every column of its
// rows for export).
constexpr uint32_t kHaloPaired = 0x80000000u;    // halo entry: the row is half of a 2x2 pair
constexpr uint8_t kRowPaired = 1, kRowExport = 2, kRowLong = 4;

__host__ __device__ __forceinline__ uint32_t up16(uint32_t x) { return (x + 15u) & ~15u; }

// Byte offsets in dynamic shared memory: slice starts at 0 (csr: the rows'
// first nonzeros), halo list, row flags, columns of the matrix slices (32 W entries; none when they are in
// global memory), z (R + H rows and a zero), eight own-row vectors of eight
// bytes a row in either Krylov precision, values of the matrix slices.
struct SliceOffsets {
    uint32_t halo, flag, col, z, vec, vec_bytes, val, end;
};
__host__ __device__ __forceinline__ SliceOffsets slice_offsets(uint32_t R, uint32_t H, uint32_t W, bool csr) {
    SliceOffsets o;
    o.halo = up16(4u * ((csr ? R : (R + 31u) / 32u) + 1u));
    o.flag = o.halo + up16(4u * H);
    o.col = o.flag + up16(R);
    o.z = o.col + 64u * W;
    o.vec = o.z + up16(8u * (R + H + 1u));
    o.vec_bytes = up16(8u * R);
    o.val = o.vec + 8u * o.vec_bytes;
    o.end = o.val + 256u * W;
    return o;
}

template <class Team>
__device__ __forceinline__ bool team_of_one(const Team &g) {
    if constexpr (!std::is_same<Team, BlockTeam>::value) return g.G == 1;
    else return true;
}

// Teams that can take the csr layout.  Not the one-lane kernels of a batch: a
// third form of the solve raised their spills (944 against 564 bytes at 128
// registers).
template <int LPR, class Team>
constexpr bool kHasCsr = LPR > 1 || std::is_same<Team, GridTeam>::value;

// Room for the padded matrix slices of nonzeros [k0, k1) in global memory
// (slice_val / slice_col hold 5 entries for every 4 nonzeros).
__device__ __forceinline__ uint32_t slice_start(uint32_t k) { return k + k / 4u; }

// Builds the block's slice map (once per launch; once per circuit in a
// batch): halo rows numbered through a hash table at the top of the dynamic
// shared memory, row flags, matrix slices' columns.  Returns false when a
// team sync gave up.
template <int LPR, class Team>
__device__ __forceinline__ bool slice_map(const KernelArgs &a, Team &g) {
    __shared__ int s_count, s_fail;
    const int r0 = g.r0, r1 = g.r1, R = r1 - r0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const bool lone = team_of_one(g), pairs = a.precond == kPcAuto;
    SliceMap m{kSliceNo, 0, 0, 0};
    g.map = m;
    if (a.smem_bytes == 0) return true;      // uniform over the team
    const uint32_t room = (uint32_t)a.smem_bytes & ~15u;
    auto row_len = [&](int i) -> uint32_t {
        if (a.longflag != nullptr && a.longflag[i] != 0) return 0u;
        return a.row_ptr[i + 1] - a.row_ptr[i];
    };
    uint32_t bits = 0;
    while ((8ull << (bits + 1)) <= (unsigned long long)a.smem_bytes / 2 && bits < 14) ++bits;
    const uint32_t cap = lone ? 0u : 1u << bits;
    uint32_t *key = (uint32_t *)(ohm_dsmem + room) - 2u * cap, *id = key + cap;
    const int nsl = (R + 31) / 32;
    uint32_t *sl = (uint32_t *)ohm_dsmem;
    bool fail = up16(4u * (nsl + 1u)) > room - 8u * cap;
    // widths of the 32-row slices
    for (int s = warp; !fail && s < nsl; s += nwarps) {
        const int li = s * 32 + lane;
        uint32_t w = li < R ? row_len(r0 + li) : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w = max(w, __shfl_xor_sync(0xffffffffu, w, o));
        if (lane == 0) sl[s] = w;
    }
    if (!lone) {
        for (uint32_t q = threadIdx.x; q < cap; q += blockDim.x) key[q] = kSentinel;
        if (threadIdx.x == 0) { s_count = 0; s_fail = 0; }
        const uint8_t all = a.n_long > 0 ? 1 : 0;     // the chunks of a long row gather records anywhere
        for (int i = r0 + (int)threadIdx.x; i < r1; i += blockDim.x) a.slice_export[i] = all;
        if (!g.sync()) return false;
        for (int li = threadIdx.x; li < R; li += blockDim.x) {
            const int i = r0 + li;
            if (pairs && a.partner[i] >= 0) a.slice_export[a.partner[i]] = 1;
            const uint32_t k0 = a.row_ptr[i], k1 = k0 + row_len(i);
            for (uint32_t k = k0; k < k1; ++k) {
                const uint32_t j = a.col[k];
                if ((int)j >= r0 && (int)j < r1) continue;
                uint32_t pos = (j * 2654435761u) >> (32u - bits), tries = 0;
                for (; tries < cap; ++tries, pos = (pos + 1u) & (cap - 1u)) {
                    const uint32_t old = atomicCAS(&key[pos], kSentinel, j);
                    if (old == j) break;
                    if (old == kSentinel) {
                        const int slot = atomicAdd(&s_count, 1);
                        id[pos] = (uint32_t)slot;
                        a.slice_export[j] = 1;
                        if (pairs && a.partner[j] >= 0) a.slice_export[a.partner[j]] = 1;
                        if (slot >= (int)(cap / 4u * 3u)) s_fail = 1;
                        break;
                    }
                }
                if (tries == cap) s_fail = 1;
                if (*(volatile int *)&s_fail) break;
            }
            if (*(volatile int *)&s_fail) break;
        }
        __syncthreads();
        m.H = s_count;
        fail = fail || s_fail != 0;
    } else {
        __syncthreads();
    }
    // slice starts: block scan of the widths over contiguous chunks of slices
    if (!fail) {
        const int chunk = (nsl + (int)blockDim.x - 1) / (int)blockDim.x;
        const int c0 = min(nsl, (int)threadIdx.x * chunk), c1 = min(nsl, c0 + chunk);
        uint32_t mine = 0, total = 0;
        for (int s = c0; s < c1; ++s) mine += sl[s];
        uint32_t at = block_exclusive_scan(mine, (uint32_t *)g.smem, &total);
        for (int s = c0; s < c1; ++s) {
            const uint32_t w = sl[s];
            sl[s] = at;
            at += w;
        }
        if (threadIdx.x == 0) sl[nsl] = total;
        m.W = (int)total;
        __syncthreads();
    }
    const uint32_t below = room - 8u * cap;      // the table stays until the columns are known
    const uint32_t g0 = slice_start(a.row_ptr[r0]);
    fail = fail || R + m.H >= 0xFFFF;
    const bool pads = LPR == 1 && m.W <= 0xFFFF;        // (the offsets below fit 32 bits)
    if (!fail) {
        const SliceOffsets chip = slice_offsets((uint32_t)R, (uint32_t)m.H, pads ? (uint32_t)m.W : 0u, false);
        const SliceOffsets rest = slice_offsets((uint32_t)R, (uint32_t)m.H, 0u, false);
        const SliceOffsets csr = slice_offsets((uint32_t)R, (uint32_t)m.H, 0u, true);
        if (pads && chip.end <= room && chip.z <= below) m.state = kSliceChip;
        else if (pads && rest.vec <= room && rest.z <= below && a.slice_val != nullptr &&
                 32u * m.W <= slice_start(a.row_ptr[r1]) - g0) m.state = kSliceStream;
        else if (kHasCsr<LPR, Team> && csr.vec <= room && csr.z <= below && a.slice_col != nullptr)
            m.state = kSliceCsr;
    }
    const SliceOffsets o = slice_offsets((uint32_t)R, (uint32_t)m.H, m.state == kSliceChip ? (uint32_t)m.W : 0u,
                                         m.state == kSliceCsr);
    if (m.state == kSliceNo && !lone) {
        // krylov() on this block gathers the record of every column
        for (int i = r0 + (int)threadIdx.x; i < r1; i += blockDim.x)
            for (uint32_t k = a.row_ptr[i]; k < a.row_ptr[i + 1]; ++k) {
                const uint32_t j = a.col[k];
                a.slice_export[j] = 1;
                if (pairs && a.partner[j] >= 0) a.slice_export[a.partner[j]] = 1;
            }
    }
    if (m.state != kSliceNo) {
        uint32_t *hl = (uint32_t *)(ohm_dsmem + o.halo);
        auto local = [&](uint32_t j) -> uint16_t {
            if (lone || ((int)j >= r0 && (int)j < r1)) return (uint16_t)(j - (uint32_t)r0);
            uint32_t pos = (j * 2654435761u) >> (32u - bits);
            while (key[pos] != j) pos = (pos + 1u) & (cap - 1u);     // inserted above
            return (uint16_t)(R + id[pos]);
        };
        if (m.state == kSliceCsr) {
            // (the widths that these replace were last read before the scan)
            for (int li = threadIdx.x; li <= R; li += blockDim.x) sl[li] = a.row_ptr[r0 + li];
            for (int li = threadIdx.x; li < R; li += blockDim.x) {
                const uint32_t k0 = a.row_ptr[r0 + li], k1 = k0 + row_len(r0 + li);
                for (uint32_t k = k0; k < k1; ++k) a.slice_col[k] = local(a.col[k]);
            }
        }
        for (uint32_t q = threadIdx.x; q < cap; q += blockDim.x)
            if (key[q] != kSentinel)
                hl[id[q]] = key[q] | (pairs && a.partner[key[q]] >= 0 ? kHaloPaired : 0u);
        if (m.state != kSliceCsr) {
            uint16_t *lc = m.state == kSliceChip ? (uint16_t *)(ohm_dsmem + o.col) : a.slice_col + g0;
            for (int s = warp; s < nsl; s += nwarps) {
                const int li = s * 32 + lane;
                const uint32_t b = sl[s], e = sl[s + 1];
                const uint32_t k0 = li < R ? a.row_ptr[r0 + li] : 0u, len = li < R ? row_len(r0 + li) : 0u;
                for (uint32_t k = 0; k < e - b; ++k)
                    lc[(b + k) * 32u + lane] = k < len ? local(a.col[k0 + k]) : (uint16_t)(R + m.H);
            }
        }
    }
    if (!lone && !g.sync()) return false;               // everyone's exports are marked
    int any = 0;
    if (m.state != kSliceNo) {
        uint8_t *flag = ohm_dsmem + o.flag;
        for (int li = threadIdx.x; li < R; li += blockDim.x) {
            const int i = r0 + li;
            uint8_t f = 0;
            if (pairs && a.partner[i] >= 0) { f |= kRowPaired; any = 1; }
            if (!lone && a.slice_export[i] != 0) f |= kRowExport;
            if (a.longflag != nullptr && a.longflag[i] != 0) f |= kRowLong;
            flag[li] = f;
        }
    }
    m.pairs = __syncthreads_or(any);
    g.map = m;
    return true;
}

// The recurrence's scalars and control, one copy per block in shared memory,
// written by one lane of warp 0 inside the reductions (identical in every
// block).
enum KrylovPhase : int { kPhaseStart, kPhaseAB, kPhaseCD, kPhaseE, kPhaseDone };
struct KrylovScalars {
    double beta, om, al, omega;                     // read by every thread
    double rho, rho_new, rr, rhat2, abs_tol, r0norm, tol2;
    double rw, rr0, rw0, mix;                       // ||W r||^2, initial norms, kRestartFromStart's g
    int phase, restart, early, code, it, restarts, flip, again;
};

// What follows a reduction: s holds its totals, q the scalars.
struct KrylovLimits {
    double tol_floor, inner_rtol;
    int max_it, max_restarts;
    bool accept_partial, try_start;
};
__device__ __forceinline__ void krylov_scalars_step(KrylovScalars &q, const double (&s)[4], const KrylovLimits &lim) {
    bool top = false, restart = false, back = false;
    const int phase = q.phase;
    int code = kKrylovRunning, next = kPhaseDone;
    if (phase == kPhaseStart && q.again) {          // back at the start
        q.rr = s[0];
        q.rw = s[1];
        q.rho_new = s[2];
        q.rhat2 = s[3];
        q.rho = q.al = q.omega = 1.0;
        q.flip = 1;
        top = true;
    } else if (phase == kPhaseStart) {              // ||r||^2, ||W r||^2, (r_hat, r), ||r_hat||^2
        const double r0norm = sqrt(s[1]);
        const double abs_tol = fmax(lim.tol_floor, lim.inner_rtol * r0norm);
        q.r0norm = r0norm;
        q.abs_tol = abs_tol;
        q.tol2 = abs_tol * abs_tol;
        q.rr = q.rr0 = s[0];
        q.rw = q.rw0 = s[1];
        q.rho_new = s[2];
        q.rhat2 = s[3];
        q.rho = q.al = q.omega = 1.0;
        q.it = q.restarts = 0;
        q.early = 0;
        q.flip = 1;                                 // toggled at the top: cur = rec0
        if (!isfinite(r0norm)) code = kKrylovNan;
        else if (r0norm < abs_tol || r0norm == 0.0) code = kKrylovConverged;
        else top = true;
    } else if (phase == kPhaseAB) {                 // (r_hat, v), ||v||^2
        if (below_root(s[0], kBreakdownRel, q.rhat2 * s[1])) {
            if (q.restarts < lim.max_restarts && q.rr > 0.0) {
                ++q.it;                             // cur still holds r; restart from it
                q.flip ^= 1;
                restart = top = true;
            } else {
                code = kKrylovBreakRv;
            }
        } else {
            q.al = q.rho / s[0];
            next = kPhaseCD;
        }
    } else if (phase == kPhaseCD) {                 // (s,s), (t,s), (t,t), ||W s||^2
        if (root_below(s[3], q.abs_tol, q.tol2)) {  // early exit (bicgstab.rs:134-139)
            code = kKrylovConverged;
            q.early = 1;
            ++q.it;
        } else if (!(s[2] > 0.0)) {
            code = kKrylovBreakTt;
        } else {
            q.omega = s[1] / s[2];
            next = kPhaseE;
        }
    } else {                                        // (r_hat, r), ||r||^2, ||W r||^2
        q.rho_new = s[0];
        q.rr = s[1];
        q.rw = s[2];
        ++q.it;
        if (!isfinite(s[2])) code = kKrylovNan;
        else if (root_below(s[2], q.abs_tol, q.tol2)) code = kKrylovConverged;
        else if (fabs(q.omega) < 1e-30) code = kKrylovBreakOmega;
        else if (lim.accept_partial && q.it == lim.max_it && sqrt(s[2]) <= 0.5 * q.r0norm)
            code = kKrylovConverged;                // inexact inner solve accepted
        else top = true;
    }
    if (top) {
        // top of an iteration: limit, rho breakdown test (restart with r_hat
        // = r, p = v = 0, or stop), beta
        q.flip ^= 1;
        const bool stop = q.it >= lim.max_it;
        if (!restart && !stop && below_root(q.rho_new, kBreakdownRel, q.rhat2 * q.rr)) {
            if (q.restarts < lim.max_restarts && q.rr > 0.0) restart = true;
            else code = kKrylovBreakRho;
        }
        if (stop) code = kKrylovMaxIter;
        back = restart && !stop && lim.try_start && !q.again && q.rw > kRestartFromStart * q.rw0;
        if (back) {
            ++q.restarts;
            q.again = 1;
            q.mix = sqrt(q.rr0 / q.rr);
        } else if (restart) {
            ++q.restarts;
            q.rho = 1.0; q.al = 1.0; q.omega = 1.0;
            q.rho_new = q.rr; q.rhat2 = q.rr;
        }
        if (code == kKrylovRunning) {
            q.beta = (q.rho_new / q.rho) * (q.al / q.omega);
            q.om = q.omega;
            q.rho = q.rho_new;
            next = kPhaseAB;
        }
    }
    if (back) next = kPhaseStart;
    q.restart = restart && !back ? 1 : 0;
    q.code = code;
    q.phase = code == kKrylovRunning ? next : kPhaseDone;
}

// Where the own-row vectors and the matrix slices are in the stream and csr
// layouts, in shared memory and read again in every phase: held in registers
// they were spilled.
enum SliceVec : int { kVecR, kVecV, kVecP, kVecC, kVecT, kVecRhat, kVecD, kVecW, kSliceVecs };
struct SliceView {
    void *ptr[kSliceVecs];
    const uint16_t *lcol;
    void *lval, *sval;      // stream: values of the matrix slices, the first n_sval slices on the chip
    int n_sval;             // csr: 1 when lcol and lval are on the chip
};

// The solve on a built slice map: a loop over phases around one reduction, so
// that the code of an iteration stays small (written out, with a reduction
// and a product per phase, an iteration streamed 40 KB of instructions
// through the instruction caches, and their misses took most of it).
template <typename T, int LPR, int MODE, class Team>
__device__ __forceinline__ int krylov_slice(const KernelArgs &a, Team &g, double tol_floor, double inner_rtol,
                                            int max_it, bool accept_partial, KrylovOut &out) {
    using Acc = T;
    __shared__ KrylovScalars S;
    __shared__ SliceView V_;
    const volatile SliceView &V = V_;
    const int r0 = g.r0, r1 = g.r1, R = r1 - r0, H = g.map.H;
    const bool pairs = g.map.pairs != 0, wt = a.newton != 0, lone = team_of_one(g), has_long = a.n_long > 0;
    const T *A;
    if constexpr (sizeof(T) == 4) A = (const T *)a.vals32; else A = (const T *)a.vals64;
    const SliceOffsets o = slice_offsets((uint32_t)R, (uint32_t)H, MODE == kSliceChip ? (uint32_t)g.map.W : 0u,
                                         MODE == kSliceCsr);
    const uint32_t k0 = MODE == kSliceCsr ? a.row_ptr[r0] : 0u, nb = MODE == kSliceCsr ? a.row_ptr[r1] - k0 : 0u;
    if (threadIdx.x == 0) {
        if constexpr (MODE != kSliceChip) {
            // in the order of their traffic while they fit, the rest in the
            // workspace (own rows, local index)
            const uint32_t room = (uint32_t)a.smem_bytes & ~15u;
            void *const spill[kSliceVecs] = {(T *)a.rself + r0, (T *)a.shat + r0, (T *)a.phat + r0,
                                             (T *)a.cself + r0, (T *)a.t + r0,    (T *)a.rhat + r0,
                                             (double *)a.d + r0, a.dx + r0};
            uint32_t at = o.vec;
            for (int k = 0; k < kSliceVecs; ++k) {
                const bool fits = at + o.vec_bytes <= room;
                V_.ptr[k] = fits ? (void *)(ohm_dsmem + at) : spill[k];
                if (fits) at += o.vec_bytes;
            }
            const uint32_t g0 = MODE == kSliceStream ? slice_start(a.row_ptr[r0]) : 0u;
            V_.lcol = a.slice_col + g0;
            V_.lval = (void *)((T *)(a.slice_val + g0));
            // what is left holds the values of the first slices
            int fits = 0;
            if constexpr (MODE == kSliceStream) {
                const uint32_t *starts = (const uint32_t *)ohm_dsmem;
                const uint32_t cols = at < room ? (room - at) / 256u : 0u;
                while (fits < (R + 31) / 32 && starts[fits + 1] <= cols) ++fits;
            }
            if constexpr (MODE == kSliceCsr) {
                // columns and values on the chip where both fit (both arrays
                // are indexed by the CSR position)
                const unsigned long long need = up16(2u * nb) + 8ull * nb;
                if (at <= room && need <= room - at) {
                    V_.lcol = (const uint16_t *)(ohm_dsmem + at) - k0;
                    V_.lval = (void *)((T *)(ohm_dsmem + at + up16(2u * nb)) - k0);
                    fits = 1;
                } else {
                    V_.lval = (void *)A;
                }
            }
            V_.sval = (void *)(ohm_dsmem + at);
            V_.n_sval = fits;
        }
        ((T *)(ohm_dsmem + o.z))[R + H] = T(0);          // the padding's column
        S.phase = kPhaseStart;
        S.again = 0;
    }
    __syncthreads();
    // On the chip the own-row vectors are one stride apart, so a row's fields
    // are one index and eight offsets.
    auto vec = [&](int k) -> void * {
        if constexpr (MODE == kSliceChip) return (void *)(ohm_dsmem + o.vec + (uint32_t)k * o.vec_bytes);
        else return V.ptr[k];
    };
    auto vecT = [&](int k) -> T * { return (T *)vec(k); };
    auto zvec = [&]() -> T * { return (T *)(ohm_dsmem + o.z); };
    auto flags = [&]() -> const uint8_t * { return ohm_dsmem + o.flag; };
    auto lvals = [&](int s) -> T * {        // values of matrix slice s
        if constexpr (MODE == kSliceChip) return (T *)(ohm_dsmem + o.val);
        else return (T *)(s < V.n_sval ? V.sval : V.lval);
    };
    auto lcols = [&]() -> const uint16_t * {
        if constexpr (MODE == kSliceChip) return (const uint16_t *)(ohm_dsmem + o.col);
        else return V.lcol;
    };
    const KrylovLimits lim{tol_floor, inner_rtol, max_it, a.max_restarts, accept_partial, restarts_from_start<T>(a)};

    for (;;) {
        const int phase = S.phase;
        if (phase == kPhaseDone) break;
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        if (phase == kPhaseE) {
            // ---- E: d += w M^-1 s, r = s - w t; (r_hat, r), ||r||^2, ||W r||^2 ----
            const double omega = S.omega;
            T *r = vecT(kVecR);
            const T *z = zvec(), *t = vecT(kVecT), *rhat = vecT(kVecRhat);
            double *d = (double *)vec(kVecD);
            const double *w = (const double *)vec(kVecW);
            const uint8_t *flag = flags();
            KRec<T> *nxt = (KRec<T> *)(S.flip ? a.rec0 : a.rec1);
#pragma unroll 1
            for (int li = threadIdx.x; li < R; li += blockDim.x) {
                const T si = r[li];
                d[li] = (double)cvt<T>(fma(omega, (double)z[li], d[li]));
                const T rt = cvt<T>(fma(-omega, (double)t[li], (double)si));
                r[li] = rt;
                if (flag[li] & kRowExport) nxt[r0 + li].r = rt;
                const double wr = wt ? w[li] * (double)rt : (double)rt;
                acc[0] = fma((double)rhat[li], (double)rt, acc[0]);
                acc[1] = fma((double)rt, (double)rt, acc[1]);
                acc[2] = fma(wr, wr, acc[2]);
            }
        } else if (phase != kPhaseStart) {
            // ---- AB: p update, v = A M^-1 p; (r_hat, v), ||v||^2 ----
            // ---- CD: s = r - a v (kept in r), d += a M^-1 p, t = A M^-1 s;
            //      (s, s), (t, s), (t, t), ||W s||^2 ----
            const bool cd = phase == kPhaseCD;
            KRec<T> *cur = (KRec<T> *)(S.flip ? a.rec1 : a.rec0), *nxt = (KRec<T> *)(S.flip ? a.rec0 : a.rec1);
            if (!cd && S.restart) {
                const uint8_t *flag = flags();
                T *p = vecT(kVecP), *v = vecT(kVecV), *r = vecT(kVecR), *c = vecT(kVecC), *rhat = vecT(kVecRhat);
#pragma unroll 1
                for (int li = threadIdx.x; li < R; li += blockDim.x) {
                    p[li] = T(0);
                    v[li] = T(0);
                    rhat[li] = r[li];
                    if (flag[li] & kRowExport) cur[r0 + li] = KRec<T>{T(0), T(0), r[li], c[li]};
                }
                OHM_SYNC_OR(kKrylovAbort);
            }
            // the vector that M^-1 is applied to: p's update or s
            const double kv = cd ? -S.al : -S.om, beta = S.beta;
            auto u3 = [&](T pp, T vv, T rr) -> T {
                const double base = cd ? (double)rr : (double)pp;
                const double x = fma(kv, (double)vv, base);
                return cvt<T>(cd ? x : fma(x, beta, (double)rr));
            };
            auto u = [&](const KRec<T> &q) -> T { return u3(q.p, q.v, q.r); };
            const KRec<T> *buf = cd ? nxt : cur;
            T *const up = cd ? vecT(kVecR) : vecT(kVecP);        // where the own rows of it are kept
            {
                // z of the halo rows from their published records; the first
                // one is fetched before the own rows' work, so its round trip
                // overlaps it
                const uint32_t *hl = (const uint32_t *)(ohm_dsmem + o.halo);
                T *z = zvec();
                int h = threadIdx.x;
                uint32_t e = 0;
                KRec<T> q{};
                if (h < H) {
                    e = hl[h];
                    q = buf[e & ~kHaloPaired];
                }
                {
                    const T *p = vecT(kVecP), *v = vecT(kVecV), *r = vecT(kVecR), *c = vecT(kVecC);
                    double *d = (double *)vec(kVecD);
                    const double al = S.al;
#pragma unroll 1
                    for (int li = threadIdx.x; li < R; li += blockDim.x) {
                        const T un = u3(p[li], v[li], r[li]);
                        if (cd) d[li] = fma(al, (double)z[li], d[li]);
                        up[li] = un;
                        z[li] = cvt<T>((double)c[li] * (double)un);
                    }
                }
                while (h < H) {
                    double zz = (double)q.c * (double)u(q);
                    if (e & kHaloPaired) {
                        const uint32_t j = e & ~kHaloPaired;
                        zz = fma((double)((const T *)a.pc_part)[j], (double)u(buf[a.partner[j]]), zz);
                    }
                    z[R + h] = cvt<T>(zz);
                    h += blockDim.x;
                    if (h >= H) break;
                    e = hl[h];
                    q = buf[e & ~kHaloPaired];
                }
            }
            if (pairs) {
                // own paired rows: the partner's term
                __syncthreads();
                const uint8_t *flag = flags();
                const T *c = vecT(kVecC);
                T *z = zvec();
#pragma unroll 1
                for (int li = threadIdx.x; li < R; li += blockDim.x) {
                    if (!(flag[li] & kRowPaired)) continue;
                    const int pi = a.partner[r0 + li];
                    const T other = (pi >= r0 && pi < r1) ? up[pi - r0] : u(buf[pi]);
                    double zz = (double)c[li] * (double)up[li];
                    zz = fma((double)((const T *)a.pc_part)[r0 + li], (double)other, zz);
                    z[li] = cvt<T>(zz);
                    if (cd && !lone) ((T *)a.s)[r0 + li] = up[li];
                }
            }
            __syncthreads();
            // y = A z on the own rows
            const uint8_t *flag = flags();
            auto row = [&](int i, double y) {
                const int li = i - r0;
                const T yt = cvt<T>(y), ui = up[li];
                if (cd) {
                    vecT(kVecT)[li] = yt;
                    const double ws = wt ? ((const double *)vec(kVecW))[li] * (double)ui : (double)ui;
                    acc[0] = fma((double)ui, (double)ui, acc[0]);
                    acc[1] = fma((double)yt, (double)ui, acc[1]);
                    acc[2] = fma((double)yt, (double)yt, acc[2]);
                    acc[3] = fma(ws, ws, acc[3]);
                } else {
                    vecT(kVecV)[li] = yt;
                    if (flag[li] & kRowExport) nxt[i] = KRec<T>{ui, yt, vecT(kVecR)[li], vecT(kVecC)[li]};
                    acc[0] = fma((double)vecT(kVecRhat)[li], (double)yt, acc[0]);
                    acc[1] = fma((double)yt, (double)yt, acc[1]);
                }
            };
            if constexpr (MODE == kSliceCsr) {
                const T *z = zvec();
                auto zx = [&](int j, bool) -> T { return z[j]; };
                spmv_rows<LPR, Acc, T, decltype(zx), decltype(row), kRowsInFlight, LPR == 1>(
                    (const uint32_t *)ohm_dsmem, lcols(), (const T *)V.lval, (const uint8_t *)nullptr, r0, r1, zx,
                    row, a.longflag, r0);
            } else {
                const int lane = threadIdx.x & 31;
                const uint32_t *sl = (const uint32_t *)ohm_dsmem;
                const T *z = zvec();
                const uint16_t *lcol = lcols();
#pragma unroll 1
                for (int li = threadIdx.x; li - lane < R; li += blockDim.x) {
                    const int s = li >> 5;
                    const T *lval = lvals(s);
                    const uint32_t e = sl[s + 1] * 32u;
                    uint32_t k = sl[s] * 32u + lane;
                    Acc y = Acc(0);
#pragma unroll 1
                    for (; k + 96u < e; k += 128u) {
                        const T z0 = z[lcol[k]], z1 = z[lcol[k + 32u]], z2 = z[lcol[k + 64u]], z3 = z[lcol[k + 96u]];
                        y += (Acc)lval[k] * (Acc)z0;
                        y += (Acc)lval[k + 32u] * (Acc)z1;
                        y += (Acc)lval[k + 64u] * (Acc)z2;
                        y += (Acc)lval[k + 96u] * (Acc)z3;
                    }
                    if (MODE == kSliceStream && sl[s + 1] - sl[s] < 4u) {
                        // short rows (a ladder's) from global memory in one
                        // round trip, not one per entry
                        if (k < e) {
                            const bool b1 = k + 32u < e, b2 = k + 64u < e;
                            const uint16_t c0 = lcol[k], c1 = b1 ? lcol[k + 32u] : c0, c2 = b2 ? lcol[k + 64u] : c0;
                            const T v0 = lval[k], v1 = b1 ? lval[k + 32u] : T(0), v2 = b2 ? lval[k + 64u] : T(0);
                            y += (Acc)v0 * (Acc)z[c0];
                            if (b1) y += (Acc)v1 * (Acc)z[c1];
                            if (b2) y += (Acc)v2 * (Acc)z[c2];
                        }
                    } else {
#pragma unroll 1
                        for (; k < e; k += 32u) y += (Acc)lval[k] * (Acc)z[lcol[k]];
                    }
                    if (li < R && !(has_long && (flag[li] & kRowLong))) row(r0 + li, (double)y);
                }
            }
            if (has_long) {
                // a block alone publishes no records: z holds every row
                auto z_at = [&](int j, bool slow) -> T {
                    if (lone) return zvec()[j];
                    const KRec<T> q = buf[j];
                    double zz = (double)q.c * (double)u(q);
                    if (slow) {
                        const int pj = a.partner[j];
                        if (pj >= 0) zz = fma((double)((const T *)a.pc_part)[j], (double)u(buf[pj]), zz);
                    }
                    return cvt<T>(zz);
                };
                if (!spmv_long<Acc>(a, g, a.col, A, a.rowflag, z_at, row)) return kKrylovAbort;
            }
        } else {
            // ---- start: matrix slices' values, r = r64, r_hat = r (again:
            //      r64 + g r), p = v = d = 0, preconditioner coefficients;
            //      ||r||^2, ||W r||^2, (r_hat, r), ||r_hat||^2 ----
            const bool again = S.again != 0;
            const double mix = S.mix;
            const uint8_t *flag = flags();
            if constexpr (MODE == kSliceCsr) {
                if (V.n_sval) {
                    uint16_t *lc = (uint16_t *)V.lcol + k0;
                    T *lv = (T *)V.lval + k0;
#pragma unroll 4
                    for (uint32_t k = threadIdx.x; k < nb; k += blockDim.x) {
                        lc[k] = a.slice_col[k0 + k];
                        lv[k] = A[k0 + k];
                    }
                }
            } else {
                const int lane = threadIdx.x & 31;
                const uint32_t *sl = (const uint32_t *)ohm_dsmem;
#pragma unroll 1
                for (int li = threadIdx.x; li - lane < R; li += blockDim.x) {
                    const int s = li >> 5;
                    T *lval = lvals(s);
                    const uint32_t b = sl[s], width = sl[s + 1] - b;
                    uint32_t k0 = 0, len = 0;
                    if (li < R && !(flag[li] & kRowLong)) {
                        k0 = a.row_ptr[r0 + li];
                        len = a.row_ptr[r0 + li + 1] - k0;
                    }
#pragma unroll 4
                    for (uint32_t k = 0; k < width; ++k) lval[(b + k) * 32u + lane] = k < len ? A[k0 + k] : T(0);
                }
            }
            T *p = vecT(kVecP), *v = vecT(kVecV), *r = vecT(kVecR), *c = vecT(kVecC), *rhat = vecT(kVecRhat);
            double *d = (double *)vec(kVecD), *w = (double *)vec(kVecW);
#pragma unroll 1
            for (int li = threadIdx.x; li < R; li += blockDim.x) {
                const int i = r0 + li;
                const T rt = cvt<T>(a.r64[i]);
                double cs = 0.0, cp = 0.0;
                const uint32_t ds = a.diag_slot[i];
                const double aii = ds == kSentinel ? 0.0 : a.vals64[ds];
                const double wi = (wt && fabs(aii) > 1e-30) ? 1.0 / fabs(aii) : 1.0;
                if (wt) w[li] = wi;
                if (a.precond != kPcNone) {
                    if (flag[li] & kRowPaired) {
                        const int pi = a.partner[i];
                        const double akk = a.diag_slot[pi] == kSentinel ? 0.0 : a.vals64[a.diag_slot[pi]];
                        const double aik = a.vals64[a.off_slot[i]];
                        const double aki = a.vals64[a.off_slot[pi]];
                        const double det = aii * akk - aik * aki;
                        if (fabs(det) > 1e-300) { cs = akk / det; cp = -aik / det; }
                        ((T *)a.pc_part)[i] = cvt<T>(cp);
                    } else if (fabs(aii) > 1e-30) {
                        cs = 1.0 / aii;
                    } else if (a.precond == kPcAuto) {
                        cs = 1.0;   // unpaired zero diagonal: identity keeps M^-1 nonsingular
                    }
                } else {
                    cs = 1.0;
                }
                const T rh = again ? cvt<T>(fma(mix, (double)r[li], (double)rt)) : rt;
                p[li] = T(0);
                v[li] = T(0);
                r[li] = rt;
                c[li] = cvt<T>(cs);
                rhat[li] = rh;
                d[li] = 0.0;
                if (flag[li] & kRowExport) ((KRec<T> *)a.rec0)[i] = KRec<T>{T(0), T(0), rt, cvt<T>(cs)};
                acc[0] = fma((double)rt, (double)rt, acc[0]);
                acc[1] = fma(wi * (double)rt, wi * (double)rt, acc[1]);
                acc[2] = fma((double)rh, (double)rt, acc[2]);
                acc[3] = fma((double)rh, (double)rh, acc[3]);
            }
        }
        if (!g.template reduce_then<4>(acc, [&](const double (&s)[4], bool writer) {
                if (writer) krylov_scalars_step(S, s, lim);
            }))
            return kKrylovAbort;
    }
    const int code = S.code;
    if (code == kKrylovConverged) {
        // an early exit left d + a M^-1 p unrounded
        const bool early = S.early != 0;
        const double *d = (const double *)vec(kVecD);
#pragma unroll 1
        for (int li = threadIdx.x; li < R; li += blockDim.x)
            a.dx[r0 + li] = early ? (double)cvt<T>(d[li]) : d[li];
    }
    out.iterations = S.it;
    out.restarts = S.restarts;
    __syncthreads();                                   // S is rewritten by the next solve
    return code;
}

// One Krylov solve of J d = r64 with the configured preconditioner.
template <typename T, int LPR, class Team>
__device__ __forceinline__ int krylov_any(const KernelArgs &a, Team &g, double tol_floor, double inner_rtol,
                                          int max_it, bool accept_partial, KrylovOut &out) {
    if (a.precond == kPcIsai) return krylov_isai<T, LPR>(a, g, tol_floor, inner_rtol, max_it, accept_partial, out);
    if constexpr (Team::kSlices) {
        if (g.map.state == kSliceNone && !slice_map<LPR>(a, g)) return kKrylovAbort;
        if constexpr (LPR == 1) {
            if (g.map.state == kSliceChip)
                return krylov_slice<T, LPR, kSliceChip>(a, g, tol_floor, inner_rtol, max_it, accept_partial, out);
            if (g.map.state == kSliceStream)
                return krylov_slice<T, LPR, kSliceStream>(a, g, tol_floor, inner_rtol, max_it, accept_partial, out);
        }
        if constexpr (kHasCsr<LPR, Team>) {
            if (g.map.state == kSliceCsr)
                return krylov_slice<T, LPR, kSliceCsr>(a, g, tol_floor, inner_rtol, max_it, accept_partial, out);
        }
    }
    return krylov<T, LPR>(a, g, tol_floor, inner_rtol, max_it, accept_partial, out);
}

// One Newton run (or a linear solve with refinement).  RunCfg modifies the
// system the way the reference's continuation steps do (gmin_newton_step,
// dc.rs:297-330, and the rhs scalings of dc.rs:355-400 and :520-560):
//   gshift  added to the diagonal of every node row,
//   src     scale of the base rhs (the independent sources),
//   pt      pseudo-transient anchor: b_i += pt * x_good_i on node rows.
// The modifications are applied only when a.continuation is set.
struct RunCfg {
    double gshift, src, pt;
    int max_outer, max_krylov;
    bool trace;
};

struct RunOut {
    int status, kcode, outer_done, err_iter, fallbacks, restarts;
    long long kiters;
    double last_dmax, bnorm_last, final_res;
};

// Device evaluation and stamping at a.x: every slot / rhs row touched by a
// device becomes base + its contributions in canonical order (the stamp map;
// slots and rows with many contributions are summed by warps in chunks
// first), the rhs rows scaled by cfg.src; then the continuation terms when
// a.continuation is set.  Untouched slots and rows are not written.  A false
// return means a team sync gave up.
template <class Team>
__device__ __forceinline__ bool assemble(const KernelArgs &a, Team &g, const RunCfg &cfg,
                                         const double *__restrict__ base_vals,
                                         const double *__restrict__ base_b) {
    const int gtid = g.gtid, gstride = g.gstride;
    const int ndev = a.nd + a.nq + a.nm;
    for (int k = gtid; k < ndev; k += gstride) {
        if (k < a.nd) {
            diode_stamps(a.diodes[k], a.x, a.mstamp + 4 * (size_t)k, a.rstamp + 2 * (size_t)k);
        } else if (k < a.nd + a.nq) {
            const int q = k - a.nd;
            const double vaf = a.bjt_vaf ? a.bjt_vaf[q] : __longlong_as_double(0x7ff0000000000000LL);
            bjt_stamps(a.bjts[q], vaf, a.x, a.mstamp + 4 * (size_t)a.nd + 9 * (size_t)q,
                       a.rstamp + 2 * (size_t)a.nd + 3 * (size_t)q);
        } else {
            const int m = k - a.nd - a.nq;
            mosfet_stamps(a.mosfets[m], a.x,
                          a.mstamp + 4 * (size_t)a.nd + 9 * (size_t)a.nq + 6 * (size_t)m,
                          a.rstamp + 2 * (size_t)a.nd + 3 * (size_t)a.nq + 2 * (size_t)m);
        }
    }
    OHM_SYNC_OR(false);
    // stamp map: each touched slot / row = base + contributions in canonical order;
    // entries with many contributions are summed by warps in chunks first
    if (a.n_lseg) {
        // chunks of a few dozen contributions per warp (their index and value
        // loads issued together), then each long segment's partials summed
        // by one block with a fixed tree
        const int lane = threadIdx.x & 31;
        for (int c = gtid >> 5; c < a.n_lseg_chunks; c += gstride >> 5) {
            const bool mat = (int)a.lseg[a.lseg_chunk_owner[c]] < a.n_mslots;
            const uint32_t *ids = mat ? a.mslot_ids : a.rrow_ids;
            const double *src = mat ? a.mstamp : a.rstamp;
            double acc = 0.0;
            const uint32_t jend = a.lseg_chunk_end[c];
#pragma unroll 4
            for (uint32_t j = a.lseg_chunk_beg[c] + lane; j < jend; j += 32) acc += src[ids[j]];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0) a.lseg_part[c] = acc;
        }
        OHM_SYNC_OR(false);
        for (int q = 0; q < a.n_lseg; ++q) {
            if (!team_owns_item(g, q)) continue;            // uniform over the block
            double v[1] = {0.0};
            for (uint32_t c = a.lseg_chunk_ptr[q] + threadIdx.x; c < a.lseg_chunk_ptr[q + 1]; c += blockDim.x)
                v[0] += a.lseg_part[c];
            block_sum<1>(v, g.smem);
            const double acc = v[0];
            if (threadIdx.x == 0) {
                const int k = (int)a.lseg[q];
                if (k < a.n_mslots) {
                    const uint32_t slot = a.mslot[k];
                    const double v = base_vals[slot] + acc;
                    a.vals64[slot] = v;
                    if (a.vals32) a.vals32[slot] = (float)v;
                } else {
                    const uint32_t row = a.rrow[k - a.n_mslots];
                    a.b[row] = cfg.src * base_b[row] + acc;
                }
            }
        }
    }
    for (int k = gtid; k < a.n_mslots + a.n_rrows; k += gstride) {
        if (a.lseg_flag != nullptr && a.lseg_flag[k]) continue;
        if (k < a.n_mslots) {
            const uint32_t slot = a.mslot[k];
            double acc = base_vals[slot];
            for (uint32_t j = a.mslot_ptr[k]; j < a.mslot_ptr[k + 1]; ++j) acc += a.mstamp[a.mslot_ids[j]];
            a.vals64[slot] = acc;
            if (a.vals32) a.vals32[slot] = (float)acc;
        } else {
            const int q = k - a.n_mslots;
            const uint32_t row = a.rrow[q];
            double acc = cfg.src * base_b[row];
            for (uint32_t j = a.rrow_ptr[q]; j < a.rrow_ptr[q + 1]; ++j) acc += a.rstamp[a.rrow_ids[j]];
            a.b[row] = acc;
        }
    }
    OHM_SYNC_OR(false);
    if (a.continuation) {
        // continuation terms on top of the assembled system; rows the
        // stamp map does not write restart from their base values
        for (int i = gtid; i < a.n; i += gstride) {
            const uint8_t f = a.stampflag[i];
            const bool node = i < a.n_nodes;
            const uint32_t ds = a.diag_slot[i];
            if (node && ds != kSentinel) {
                const double v = ((f & 1) ? a.vals64[ds] : base_vals[ds]) + cfg.gshift;
                a.vals64[ds] = v;
                if (a.vals32) a.vals32[ds] = (float)v;
            }
            double bv = (f & 2) ? a.b[i] : cfg.src * base_b[i];
            if (node && cfg.pt != 0.0) bv += cfg.pt * a.x_good[i];
            a.b[i] = bv;
        }
        OHM_SYNC_OR(false);
    }
    return true;
}

// The Newton loop for one system, run by a team; results in `o` (identical in
// every thread).  A false return means a grid barrier gave up.
template <int LPR, class Team>
__device__ __forceinline__ bool newton_run(const KernelArgs &a, Team &g, const RunCfg &cfg, RunOut &o) {
    const int r0 = g.r0, r1 = g.r1, gtid = g.gtid, gstride = g.gstride;

    int status = kOk, kcode = kKrylovRunning, outer_done = 0, err_iter = 0;
    int fallbacks = 0, restarts = 0;
    long long kiters = 0;
    double last_dmax = 0.0, bnorm_last = 0.0, final_res = -1.0;
    double fnorm_prev = -1.0, eta_prev = a.eta_max;

    for (int outer = 0; outer < cfg.max_outer; ++outer) {
        // ---------------- device evaluation + stamping (Newton) ----------------
        if (a.newton) {
            if (!assemble(a, g, cfg, a.base_vals, a.base_b)) return false;
        }

        // -------------------------- FP64 residual r64 = b - A x -------------------------
        // ||b||^2, ||r||^2, and for Newton the scaled ||W b||^2, ||W r||^2
        // (w_i = 1/|J_ii|, the stopping scale of krylov()).  A non-finite
        // entry makes ||r||^2 non-finite.
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        const double *xv = a.x;
        auto x_at = [&](int j, bool) -> double { return xv[j]; };
        auto res_row = [&](int i, double ax) {
            const double bi = a.b[i];
            const double ri = bi - ax;
            a.r64[i] = ri;
            acc[0] += bi * bi;
            acc[1] += ri * ri;
            if (a.newton) {
                const uint32_t ds = a.diag_slot[i];
                const double aii = ds == kSentinel ? 0.0 : a.vals64[ds];
                const double wi = fabs(aii) > 1e-30 ? 1.0 / fabs(aii) : 1.0;
                acc[2] += (wi * bi) * (wi * bi);
                acc[3] += (wi * ri) * (wi * ri);
            }
        };
        spmv_rows<LPR, double>(a.row_ptr, a.col, a.vals64, (const uint8_t *)nullptr, r0, r1, x_at, res_row,
                               a.longflag);
        if (!spmv_long<double>(a, g, a.col, a.vals64, (const uint8_t *)nullptr, x_at, res_row)) return false;
        {
            if (!g.template allreduce<4>(acc)) return false;
        }
        const double bnorm = sqrt(acc[0]);
        const double bnorm_w = a.newton ? sqrt(acc[2]) : bnorm;   // Krylov stopping scale
        const double fnorm_w = a.newton ? sqrt(acc[3]) : sqrt(acc[1]);
        const double rnorm64 = sqrt(acc[1]);
        bnorm_last = bnorm;
        if (a.newton && !isfinite(acc[1])) {
            // non-finite assembled system (newton.rs:258-263)
            status = kErrNewtonNumerical;
            err_iter = outer;
            outer_done = outer;
            break;
        }
        if (!a.newton && (rnorm64 < a.krylov_tol * bnorm || bnorm < 1e-30)) {
            // converged before this sweep (bicgstab.rs:91-95 for b = 0)
            kcode = kKrylovConverged;
            outer_done = outer;
            final_res = rnorm64;
            break;
        }

        // ISAI(1) factorisation of the current matrix (once per outer iteration
        // of a Newton solve, once for a linear solve)
        if (a.precond == kPcIsai && (a.newton || outer == 0)) {
            if (!isai_setup(a, g)) return false;
        }

        // -------------------------------- BiCGSTAB ---------------------------------
        const double floor_tol = a.krylov_tol * bnorm_w;
        // Inner tolerance: constant, or Eisenstat-Walker choice 2 (gamma 0.9,
        // exponent 2, safeguarded) on the scaled Newton residual ||W (b - J x)||.
        double eta = a.inner_rtol;
        if (a.newton && a.forcing == 1) {
            if (fnorm_prev > 0.0) {
                const double ratio = fnorm_w / fnorm_prev;
                eta = 0.9 * ratio * ratio;
                const double guard = 0.9 * eta_prev * eta_prev;
                if (guard > 0.1) eta = fmax(eta, guard);
            } else {
                eta = a.eta_max;
            }
            eta = fmin(fmax(eta, a.inner_rtol), a.eta_max);
            eta_prev = eta;
            fnorm_prev = fnorm_w;
        }
        KrylovOut ko{0, 0};
        int it32 = 0, it64 = 0;
        bool run64 = true;
        if (a.mixed && !(a.newton && eta < a.fp32_min_eta)) {
            kcode = krylov_any<float, LPR>(a, g, floor_tol, eta, min(a.fp32_max_iterations, cfg.max_krylov), true, ko);
            if (kcode == kKrylovAbort) return false;
            it32 = ko.iterations;
            restarts += ko.restarts;
            run64 = kcode != kKrylovConverged;
            if (run64) ++fallbacks;    // FP32 failed or stalled: redo this solve in FP64
        }
        if (run64) {
            kcode = krylov_any<double, LPR>(a, g, floor_tol, eta, cfg.max_krylov, false, ko);
            if (kcode == kKrylovAbort) return false;
            it64 = ko.iterations;
            restarts += ko.restarts;
        }
        kiters += it32 + it64;
        if (cfg.trace && a.trace && outer < a.trace_cap && g.leader()) {
            double *tr = a.trace + (size_t)outer * kTraceCols;
            tr[0] = it32; tr[1] = it64; tr[2] = rnorm64; tr[3] = eta; tr[4] = -1.0; tr[5] = ko.restarts;
        }
        if (kcode != kKrylovConverged) {
            status = kErrSolve;
            err_iter = outer;
            outer_done = outer;
            break;
        }

        // -------------------------------- update ----------------------------------
        if (!a.newton) {
            for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) a.x[i] = a.x[i] + a.dx[i];
            OHM_SYNC_OR(false);
            outer_done = outer + 1;
            continue;      // next refinement sweep recomputes the FP64 residual
        }
        for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
            const double xo = a.x[i];
            a.x_prev[i] = xo;
            a.x[i] = xo + a.dx[i];
            a.node_scale[i] = 0x3FF0000000000000ULL;   // 1.0
        }
        OHM_SYNC_OR(false);
        {
            const int ndev = a.nd + a.nq + a.nm;
            for (int k = gtid; k < ndev; k += gstride) {
                if (k < a.nd) diode_limit(a.diodes[k], a.x_prev, a.x, a.node_scale);
                else if (k < a.nd + a.nq) bjt_limit(a.bjts[k - a.nd], a.x_prev, a.x, a.node_scale);
                else mosfet_limit(a.mosfets[k - a.nd - a.nq], a.x_prev, a.x, a.node_scale);
            }
        }
        OHM_SYNC_OR(false);
        {
            double mx[3] = {0.0, 0.0, 0.0};   // max|dx|, max|x|, non-finite count
            for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
                const double sc = __longlong_as_double((long long)a.node_scale[i]);
                const double xo = a.x_prev[i];
                double xn = a.x[i];
                if (sc < 1.0) { xn = xo + (xn - xo) * sc; a.x[i] = xn; }
                if (!isfinite(xn)) mx[2] += 1.0;
                mx[0] = fmax(mx[0], fabs(xn - xo));
                mx[1] = fmax(mx[1], fabs(xn));
            }
            if (!g.template allmax<3>(mx)) return false;
            last_dmax = mx[0];
            outer_done = outer + 1;
            if (cfg.trace && a.trace && outer < a.trace_cap && g.leader())
                a.trace[(size_t)outer * kTraceCols + 4] = mx[0];
            if (mx[2] > 0.0) { status = kErrNewtonNumerical; err_iter = outer; break; }
            if (mx[0] < a.abs_tol + a.rel_tol * mx[1]) { status = kOk; break; }
            if (outer + 1 == cfg.max_outer) status = kErrNewtonNotConverged;
        }
    }

    // final FP64 residual of a linear solve (reported; the refinement test in mixed mode)
    if (!a.newton && status == kOk && final_res < 0.0) {
        double acc[1] = {0.0};
        const double *xv = a.x;
        auto x_at = [&](int j, bool) -> double { return xv[j]; };
        auto fin_row = [&](int i, double ax) {
            const double ri = a.b[i] - ax;
            acc[0] += ri * ri;
        };
        spmv_rows<LPR, double>(a.row_ptr, a.col, a.vals64, (const uint8_t *)nullptr, r0, r1, x_at, fin_row,
                               a.longflag);
        if (!spmv_long<double>(a, g, a.col, a.vals64, (const uint8_t *)nullptr, x_at, fin_row)) return false;
        if (!g.template allreduce<1>(acc)) return false;
        final_res = sqrt(acc[0]);
        if (a.require_true_residual && !(final_res < a.krylov_tol * bnorm_last)) {
            // refinement sweeps exhausted without reaching the FP64 tolerance
            status = kErrSolve;
            if (kcode == kKrylovConverged) kcode = kKrylovMaxIter;
        }
    }

    o.status = status;
    o.kcode = kcode;
    o.outer_done = outer_done;
    o.err_iter = err_iter;
    o.fallbacks = fallbacks;
    o.restarts = restarts;
    o.kiters = kiters;
    o.last_dmax = last_dmax;
    o.bnorm_last = bnorm_last;
    o.final_res = final_res;
    return true;
}

// x[own rows] = src (or 0 when src is null), then a team sync.
template <class Team>
__device__ __forceinline__ bool team_copy(Team &g, double *dst, const double *src) {
    for (int i = g.r0 + threadIdx.x; i < g.r1; i += blockDim.x) dst[i] = src ? src[i] : 0.0;
    return g.sync();
}

// BiCGSTAB cap of an intermediate continuation step: the reference's
// fail-fast limits (dc.rs:171-174, :391-393, :531-536), scaled by 4 for the
// tighter inner tolerance used here, never above the caller's limit.
__device__ __forceinline__ int cont_cap(const KernelArgs &a, int reference_cap) {
    return min(a.max_krylov, 4 * reference_cap);
}

// One system solved by a team: the direct Newton run (or linear solve), then,
// when a.continuation is set and the direct run failed, the reference's
// nonlinear DC strategy (run_nonlinear, src/analysis/dc.rs:60-290) on the
// device: source stepping for circuits with MOSFETs (run_source_stepping,
// :495-645: start at 0.1, grow by twice the last successful step, halve on
// failure, at most 20 subdivisions), adaptive GMIN stepping (:160-253: from
// 0.1, 1000x drops, 10x subdivisions from the last good level, at most 13),
// a solve at the true GMIN, then pseudo-transient continuation from the last
// GMIN point (:331-490: alpha from 0.1, 100x drops, at most 7 subdivisions,
// b += alpha x_good on node rows) and a final true-DC solve.  The final
// solves take the reference's own Newton limits (50 after GMIN stepping, 25
// after pseudo-transient), the direct attempt the caller's.  The reference's
// CPU sparse-LU retries have no counterpart.  The stages form a state machine
// around one newton_run call site.  The leader writes `*info`; a false
// return means a grid barrier gave up.
template <int LPR, class Team>
__device__ __forceinline__ bool solve_body(const KernelArgs &a, Team &g, DeviceInfo *info) {
    enum { kDirect, kSource, kGmin, kGminFinal, kPseudo, kPseudoFinal };
    RunOut o;
    RunCfg c{0.0, 1.0, 0.0, a.max_outer, a.max_krylov, true};
    int stage = kDirect, steps = 0, kind = kContNone, subdiv = 0;
    bool have_good = false;
    double last = 0.0, target = 0.0;
    long long kiters = 0;
    int fallbacks = 0, restarts = 0;
    for (;;) {
        if (!newton_run<LPR>(a, g, c, o)) return false;
        kiters += o.kiters;
        fallbacks += o.fallbacks;
        restarts += o.restarts;
        if (stage != kDirect) ++steps;
        const bool ok = o.status == kOk;
        bool finished = false, save_good = false;
        int xsrc = -1;                  // next start: -1 keep x, 0 zeros, 1 x_good
        switch (stage) {
            case kDirect:
                if (ok || !(a.newton && a.continuation)) { finished = true; break; }
                have_good = false;
                subdiv = 0;
                xsrc = 0;
                if (a.nm > 0) {
                    stage = kSource; kind = kContSource; last = 0.0; target = 0.1;
                    c = RunCfg{0.0, target, 0.0, 30, cont_cap(a, 200), false};
                } else {
                    stage = kGmin; kind = kContGmin; last = 1.0; target = 1e-1;
                    c = RunCfg{target, 1.0, 0.0, 15, cont_cap(a, 300), false};
                }
                break;
            case kSource:
                if (ok) {
                    save_good = true;
                    have_good = true;
                    const double prev_step = target - last;
                    last = target;
                    subdiv = 0;
                    if (fabs(target - 1.0) < 1e-12) { finished = true; break; }
                    target = fmin(target + 2.0 * prev_step, 1.0);
                    xsrc = -1;
                    c.src = target;
                    break;
                }
                target = last + 0.5 * (target - last);
                if (++subdiv > 20 || target - last < 1e-6) {
                    stage = kGmin; kind = kContGmin; have_good = false; subdiv = 0; last = 1.0; target = 1e-1;
                    xsrc = 0;
                    c = RunCfg{target, 1.0, 0.0, 15, cont_cap(a, 300), false};
                } else {
                    xsrc = have_good ? 1 : 0;
                    c.src = target;
                }
                break;
            case kGmin:
                if (ok) {
                    save_good = true;
                    have_good = true;
                    last = target;
                    subdiv = 0;
                    target *= 1e-3;
                } else {
                    if (++subdiv > 13) { finished = true; break; }
                    target = last * pow(10.0, -(double)subdiv);
                }
                xsrc = have_good ? 1 : 0;
                if (target > 1e-13) {
                    c = RunCfg{target, 1.0, 0.0, 15, cont_cap(a, 300), false};
                } else {
                    stage = kGminFinal;       // NewtonParams::default(): 50 iterations (dc.rs:255-262)
                    c = RunCfg{0.0, 1.0, 0.0, 50, a.max_krylov, false};
                }
                break;
            case kGminFinal:
                // continuation bit 1 (testing): count this solve as failed so
                // that the pseudo-transient stage runs
                if ((ok && !(a.continuation & 2)) || !have_good) { finished = true; break; }
                stage = kPseudo; kind = kContPseudo; last = 1.0; target = 1e-1; subdiv = 0;
                xsrc = 1;
                c = RunCfg{target, 1.0, target, 20, cont_cap(a, 500), false};
                break;
            case kPseudo:
                if (ok) {
                    save_good = true;
                    last = target;
                    subdiv = 0;
                    target *= 1e-2;
                } else {
                    if (++subdiv > 7) { finished = true; break; }
                    target = last * pow(10.0, -(double)subdiv);
                }
                xsrc = 1;
                if (target > 1e-8) {
                    c = RunCfg{target, 1.0, target, 20, cont_cap(a, 500), false};
                } else {
                    stage = kPseudoFinal;     // 25 iterations (dc.rs:449-454)
                    c = RunCfg{0.0, 1.0, 0.0, 25, a.max_krylov, false};
                }
                break;
            default:
                finished = true;
                break;
        }
        if (save_good && !team_copy(g, a.x_good, a.x)) return false;
        if (finished) break;
        if (xsrc == 0 && !team_copy(g, a.x, (const double *)nullptr)) return false;
        if (xsrc == 1 && !team_copy(g, a.x, a.x_good)) return false;
    }
    if (g.leader()) {
        info->status = o.status;
        info->krylov_code = o.kcode;
        info->iterations = o.outer_done;
        info->error_iteration = o.err_iter;
        info->krylov_iterations = kiters;
        info->fp64_fallbacks = fallbacks;
        info->krylov_restarts = restarts;
        info->max_residual = o.last_dmax;
        info->final_residual = o.final_res;
        info->b_norm = o.bnorm_last;
        info->continuation_steps = steps;
        info->continuation_kind = kind;
    }
    return true;
}

// One large system per launch: the whole (co-resident) grid is the team.
template <int LPR>
__global__ void __launch_bounds__(kSolverBlock, 1) persistent_solver(const __grid_constant__ KernelArgs a) {
    GridTeam g;
    g.init(a);
    solve_body<LPR>(a, g, a.info);
}
template <int LPR>
__global__ void __launch_bounds__(kWideBlock, 1) persistent_solver_wide(const __grid_constant__ KernelArgs a) {
    GlobalTeam g;
    g.init(a);
    solve_body<LPR>(a, g, a.info);
}


#undef OHM_SYNC_OR

}  // namespace ohm
