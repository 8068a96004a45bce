// Internal declarations shared by the C-ABI translation units.
#pragma once

#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <string>

#include "../../include/ohm.h"
#include "solver_kernel.cuh"

using ohm::DeviceInfo;

// A grid-team kernel with Krylov slices (kSolverBlock threads) and its
// global-memory form (kWideBlock threads).
template <typename Fn>
struct KernelPair {
    Fn slices, wide;
};

// The persistent solver per lanes per row, instantiated in solver_k*.cu.
using KernelFn = void (*)(ohm::KernelArgs);
template <int LPR>
KernelPair<KernelFn> persistent_kernel_for();
template <>
KernelPair<KernelFn> persistent_kernel_for<1>();
template <>
KernelPair<KernelFn> persistent_kernel_for<4>();
template <>
KernelPair<KernelFn> persistent_kernel_for<8>();
template <>
KernelPair<KernelFn> persistent_kernel_for<16>();
template <>
KernelPair<KernelFn> persistent_kernel_for<32>();

// Records the message for ohm_last_error() and returns `st`.
ohm_status ohm_fail(ohm_status st, const char *fmt, ...);

#define CUDA_TRY(expr)                                                                      \
    do {                                                                                    \
        cudaError_t e_ = (expr);                                                            \
        if (e_ != cudaSuccess)                                                              \
            return ohm_fail(OHM_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e_));  \
    } while (0)

// ---------------------------------------------------------------- context --
struct ohm_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    int num_sms = 0;
    // barrier words + info block
    unsigned int *sync_words = nullptr;   // [count, gen, error(int)]
    DeviceInfo *info_dev = nullptr;
    DeviceInfo *info_host = nullptr;      // pinned
    double *dot_scratch = nullptr;        // for ohm_dot
    int krylov_layout = 0;                    // OHM_KRYLOV_LAYOUT_*
    // Objects created on this context (plans, buffers, matrices).  Destroying
    // the context while some are alive defers the release to the last one.
    int live_objects = 0;
    bool destroy_pending = false;
};

// Where a persistent-solver launch puts its barrier words and status block.
struct LaunchTarget {
    int num_sms;
    cudaStream_t stream;
    unsigned int *sync_words;        // 4 words: count, generation, error, spare
    ohm::DeviceInfo *info_dev;
    ohm::DeviceInfo *info_host;      // host copy target (pinned or not)
    int max_grid;                    // 0: no cap beyond the co-residency limit
    int krylov_layout;               // OHM_KRYLOV_LAYOUT_* (0 when not given)
};
ohm_status ohm_launch_persistent(const LaunchTarget &t, ohm::KernelArgs &a, int64_t nnz, int *launches);
ohm_status ohm_finish_persistent(const LaunchTarget &t, ohm_solve_info *info, int launches);
ohm_status ohm_check_krylov(const ohm_krylov_params *p);
// Most dynamic shared memory that a block of `fn` can have (a multiple of 16,
// 1 KB kept free), the kernel's limit raised to it; 0 on failure.  The limit
// belongs to the function, whatever the context or the thread: every launch
// sets the same one, since a smaller one set by a call on another thread would
// make a launch fail that needs more.
int ohm_max_dynamic_smem(const void *fn);

// How far the rows of a system's blocks reach, from its pattern on the host:
// kScatterNear when the columns that a block shares with others fit its halo
// table (krylov_slice()), kScatterWide when they do so with one block per
// kTeamRows rows but not in a cluster of kMaxTeamCluster, kScatterFar when they
// do not: such a system (rows in random order, a random graph) runs krylov() in
// every block, which wants its shared memory as L1 and 1,024 threads (us per
// iteration with 512 threads that reserved a slice -> so: 500 x 500 mesh in
// random order 54 -> 35, 700 x 700 91 -> 55, 1000 x 1000 243 -> 117).
enum Scatter : int { kScatterNear = 0, kScatterWide = 1, kScatterFar = 2 };
int ohm_scatter(int64_t n, int64_t n_devices, int num_sms, const uint32_t *row_ptr, const uint32_t *col);

// Grid, block, kernel form, dynamic shared memory (a.smem_bytes) and
// synchronisation (a.cluster) of a grid-team kernel over a.n rows.
constexpr int kMaxTeamCluster = 16, kTeamOneBlock = 1024, kTeamRows = 512, kTeamClusterRows = 1700,
              kTeamRowNnz = 6;
struct TeamShape {
    int grid = 1, block = ohm::kSolverBlock;
    bool wide = false;
};
ohm_status ohm_team_shape(const void *slices, const void *wide, int num_sms, int max_grid, int krylov_layout,
                          int64_t nnz, ohm::KernelArgs &a, TeamShape &s);
template <typename Fn>
ohm_status ohm_team_kernel(const KernelPair<Fn> &k, int num_sms, int max_grid, int krylov_layout, int64_t nnz,
                           ohm::KernelArgs &a, TeamShape &s, Fn &fn) {
    const ohm_status st = ohm_team_shape((const void *)k.slices, (const void *)k.wide, num_sms, max_grid,
                                         krylov_layout, nnz, a, s);
    fn = s.wide ? k.wide : k.slices;
    return st;
}
// Launch configuration of that shape: one cluster, or a cooperative grid.
struct TeamLaunch {
    cudaLaunchConfig_t config = {};
    cudaLaunchAttribute attr[1] = {};
    TeamLaunch(const TeamShape &s, const ohm::KernelArgs &a, cudaStream_t stream) {
        config.gridDim = dim3(s.grid);
        config.blockDim = dim3(s.block);
        config.dynamicSmemBytes = (size_t)a.smem_bytes;
        config.stream = stream;
        if (a.cluster) {
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = s.grid;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        } else {
            attr[0].id = cudaLaunchAttributeCooperative;
            attr[0].val.cooperative = 1;
        }
        config.attrs = attr;
        config.numAttrs = 1;
    }
    TeamLaunch(const TeamLaunch &) = delete;
};
// Kernel arguments of a Newton solve on a plan (validated params), its
// context, and the launch of a plan-sized persistent kernel (api.cu).
ohm_status ohm_plan_kernel_args(ohm_plan *p, const ohm_newton_params *np, double *x_dev, ohm::KernelArgs &a,
                                int64_t *nnz);
ohm_ctx *ohm_plan_context(ohm_plan *p);
// Copies the plan's base rhs back into its assembled rhs (a Newton solve
// re-stamps only the rows that devices touch, so a run that assembled
// another rhs into the plan, such as a transient step, must restore it).
cudaError_t ohm_plan_restore_rhs(ohm_plan *p);
// J(x) values of a plan's system at a device x, on base values base_vals_dev
// (the plan's conductance base when null), written to J_out (nnz doubles).
ohm_status ohm_plan_jacobian_device(ohm_plan *p, const double *x_dev, const double *base_vals_dev, double *J_out);
// A device linear system of fixed pattern (uploaded once, with its
// preconditioner structure and Krylov workspace) solved for new values and
// right-hand sides; FP64.  x starts from zero.
struct ohm_linsys;
ohm_status ohm_linsys_create(ohm_ctx *c, int64_t n, int64_t nnz, const uint32_t *h_rp, const uint32_t *h_col,
                             const double *h_val, ohm_linsys **out);
ohm_status ohm_linsys_solve(ohm_linsys *L, double *d_vals, double *d_b, double *d_x, const ohm_krylov_params *p,
                            ohm_solve_info *info);
void ohm_linsys_destroy(ohm_linsys *L);
cudaError_t ohm_f64_to_f32(const double *in, float *out, int64_t n, cudaStream_t s);

// Child-object bookkeeping (see ohm_ctx::live_objects).
void ohm_ctx_retain(ohm_ctx *c);
void ohm_ctx_release(ohm_ctx *c);

struct ohm_buf {
    ohm_ctx *ctx;
    double *d;
    int64_t n;
};

struct ohm_csr {
    ohm_ctx *ctx;
    int64_t n, nnz;
    uint32_t *rp, *col;
    double *val;
};

// Device memory of the library's buffers comes from a per-device cache
// (pool.cu).  Every buffer is released with ohm_pool_free after the work on
// it has completed (the owner synchronises its stream first).
cudaError_t ohm_pool_alloc(void **p, size_t bytes);
void ohm_pool_free(void *p);
void ohm_pool_trim(int device);

template <typename T>
inline cudaError_t dalloc(T **p, size_t count) {
    *p = nullptr;
    if (count == 0) count = 1;
    return ohm_pool_alloc((void **)p, count * sizeof(T));
}

