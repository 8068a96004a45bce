// AC sweep: A(f) x(f) = b_ac with A(f) = G + j 2 pi f C for many frequency
// points in one launch (src/analysis/ac.rs:56-70 solves them one at a time).
//
// One thread-block cluster per frequency point where its shared memory holds
// the point, else one thread block per point (or a team of them), taken from
// a work queue; each runs a complex FP64 right-preconditioned BiCGSTAB with the reference's operation
// order (src/solver/gpu.rs:608-690: conjugated dots sum(conj(x) y), stop at
// ||r|| < tol ||b||).  A(f) is never stored: the SpMV reads the shared G and
// C values of one pattern and forms g + j w c per nonzero, so every
// frequency's matrix traffic hits the same L2-resident arrays.
#include <cuda_runtime.h>

#include <algorithm>
#include <numeric>
#include <cmath>
#include <cstring>
#include <vector>

#include "host_util.h"

using namespace ohm;

namespace {

constexpr int kAcBlock = 256;       // points >> SMs: several blocks per SM
constexpr int kAcWideBlock = 1024;  // points <= SMs on a large system: one wide block per point
constexpr int kAcVecs = 11;        // x r rhat p v s t phat shat m_self m_part

struct AcDev {
    int code, iterations, restarts, pad;
    double rnorm, bnorm;
};

struct AcArgs {
    int n, n_freq, precond, max_it, max_restarts;
    double tol;
    const uint32_t *rp, *col;
    const double *g, *c;               // c may be null
    const double2 *b;
    const double *omega;               // per frequency point of this launch
    const int32_t *partner;
    const uint32_t *diag_slot, *off_slot;
    double2 *work;                     // vecs * n per frequency point
    int vecs;
    AcDev *info;
    unsigned int *queue;
    // Team mode (fewer points than resident blocks): block b works on point
    // blk_point[b] as member blk_member[b] of point_team[q] blocks, with a
    // per-point barrier counter and reduction partials [2][4][kAcMaxTeam].
    int team_mode;
    const int32_t *blk_point, *blk_member, *point_team;
    unsigned long long *team_count;
    double *team_part;
    int *team_error;
};

constexpr int kAcMaxTeam = 8;

// The blocks solving one frequency point.  A one-block team (TEAM false, the
// queue mode) synchronises and reduces within the block; a team of T blocks
// splits the rows evenly and meets at a bounded barrier on the point's
// arrival counter, its dot products summed from per-member partials in
// member order (identical in every member).
template <bool TEAM>
struct AcTeam {
    int T, m, r0, r1;
    unsigned long long *count;
    unsigned long long epoch;
    double *part;
    int red;
    int *error;
    double *smem;

    __device__ __forceinline__ bool sync() {
        if constexpr (!TEAM) { __syncthreads(); return true; }
        __shared__ int s_ok;
        epoch += (unsigned long long)T;
        __syncthreads();
        if (threadIdx.x == 0) {
            red_release_add_u64(count, 1ull);
            int ok = 1;
            uint32_t spins = 0;
            while (ld_acquire_u64(count) < epoch) {
                if (++spins > kBarrierSpinLimit || *(volatile int *)error != 0) {
                    atomicCAS(error, 0, kStatusTimeout);
                    ok = 0;
                    break;
                }
                if (spins > kTightSpins) __nanosleep(64);
            }
            s_ok = ok;
        }
        __syncthreads();
        return s_ok != 0;
    }
    template <int NV>
    __device__ __forceinline__ bool sum(double (&v)[NV]) {
        block_sum<NV>(v, smem);
        if constexpr (!TEAM) return true;
        double *p = part + (size_t)(red & 1) * 4 * kAcMaxTeam;
        ++red;
        if (threadIdx.x == 0)
            for (int k = 0; k < NV; ++k) p[k * kAcMaxTeam + m] = v[k];
        if (!sync()) return false;
        for (int k = 0; k < NV; ++k) {
            double x = 0.0;
            for (int j = 0; j < T; ++j) x += __ldcg(p + k * kAcMaxTeam + j);
            v[k] = x;
        }
        return true;
    }
};

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// conj(a) * b
__device__ __forceinline__ double2 cdotc(double2 a, double2 b) {
    return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ double cabs2(double2 a) { return a.x * a.x + a.y * a.y; }
__device__ __forceinline__ double2 cdiv(double2 a, double2 b) {
    const double d = cabs2(b);
    return make_double2((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}
__device__ __forceinline__ double2 cval(const AcArgs &A, uint32_t k, double w) {
    return make_double2(A.g[k], A.c ? w * A.c[k] : 0.0);
}

// Block-Jacobi coefficients of row i at this frequency: the row's own
// (returned) and its partner's (cp).
__device__ __forceinline__ double2 ac_precond(const AcArgs &A, int i, double w, double2 &cp) {
    double2 cs = make_double2(0.0, 0.0);
    cp = make_double2(0.0, 0.0);
    const uint32_t ds = A.diag_slot[i];
    const double2 aii = ds == kSentinel ? make_double2(0.0, 0.0) : cval(A, ds, w);
    const int pi = A.partner[i];
    if (A.precond == kPcNone) {
        cs = make_double2(1.0, 0.0);
    } else if (A.precond == kPcAuto && pi >= 0) {
        // [[a_ii a_ik] [a_ki a_kk]]^-1, the row-i half
        const uint32_t dk = A.diag_slot[pi];
        const double2 akk = dk == kSentinel ? make_double2(0.0, 0.0) : cval(A, dk, w);
        const double2 aik = cval(A, A.off_slot[i], w), aki = cval(A, A.off_slot[pi], w);
        const double2 det = csub(cmul(aii, akk), cmul(aik, aki));
        if (cabs2(det) > 1e-300) {
            cs = cdiv(akk, det);
            cp = cdiv(make_double2(-aik.x, -aik.y), det);
        }
    } else if (cabs2(aii) > 1e-30) {
        cs = cdiv(make_double2(1.0, 0.0), aii);        // gpu.rs:300-313
    } else if (A.precond == kPcAuto) {
        cs = make_double2(1.0, 0.0);
    }
    return cs;
}

// y_i = sum_k A(f)_ik x_k for rows [r0, r1), LPR lanes per row; f(i, y).
template <int LPR, typename F>
__device__ __forceinline__ void cspmv(const AcArgs &A, double w, const double2 *x, int r0, int r1, F f) {
    const int lane = threadIdx.x % LPR, group = threadIdx.x / LPR, ngroups = blockDim.x / LPR;
    for (int base = r0; base < r1; base += ngroups) {
        const int i = base + group;
        const bool ok = i < r1;
        const uint32_t b = ok ? A.rp[i] : 0u, e = ok ? A.rp[i + 1] : 0u;
        uint32_t len = e - b;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) len = max(len, __shfl_xor_sync(0xffffffffu, len, o));
        double2 acc = make_double2(0.0, 0.0);
        for (uint32_t off = lane; off < len; off += LPR) {
            const uint32_t k = b + off;
            if (k < e) acc = cadd(acc, cmul(cval(A, k, w), x[A.col[k]]));
        }
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) {
            acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o, LPR);
            acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o, LPR);
        }
        if (ok && lane == 0) f(i, acc);
    }
}

// One frequency point solved by team g (rows [g.r0, g.r1) of this block).
// Returns false when a team barrier gave up.
template <int LPR, bool TEAM>
__device__ bool ac_point(const AcArgs &A, int q, AcTeam<TEAM> &g) {
    const int n = A.n, r0 = g.r0, r1 = g.r1;
    {
        const double w = A.omega[q];
        // (a constant: with A.vecs the team kernel spilled 196 bytes, not 44)
        double2 *W = A.work + (size_t)q * kAcVecs * n;
        double2 *x = W, *r = W + n, *rh = W + 2 * (size_t)n, *p = W + 3 * (size_t)n, *v = W + 4 * (size_t)n;
        double2 *s = W + 5 * (size_t)n, *t = W + 6 * (size_t)n, *ph = W + 7 * (size_t)n, *sh = W + 8 * (size_t)n;
        double2 *ms = W + 9 * (size_t)n, *mp = W + 10 * (size_t)n;

        // preconditioner coefficients for this frequency, and the start vectors
        double acc0[1] = {0.0};
        for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
            double2 cp;
            const double2 cs = ac_precond(A, i, w, cp);
            ms[i] = cs;
            mp[i] = cp;
            const double2 bi = A.b[i];
            x[i] = make_double2(0.0, 0.0);
            r[i] = bi;
            rh[i] = bi;
            p[i] = make_double2(0.0, 0.0);
            v[i] = make_double2(0.0, 0.0);
            acc0[0] += cabs2(bi);
        }
        if (!g.sum<1>(acc0)) return false;
        const double bnorm = sqrt(acc0[0]);
        int code = kKrylovRunning, it = 0, restarts = 0;
        double rnorm = bnorm;
        if (!(bnorm >= 1e-30)) {
            code = isfinite(bnorm) ? kKrylovConverged : kKrylovNan;    // b = 0: x = 0 (gpu.rs:618-621)
        } else {
            const double abs_tol = A.tol * bnorm;
            double2 rho = make_double2(1.0, 0.0), alpha = rho, omega = rho;
            double2 rho_new = make_double2(acc0[0], 0.0);
            double rr = acc0[0], rh2 = acc0[0];
            auto restart = [&]() -> bool {
                for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
                    rh[i] = r[i];
                    p[i] = make_double2(0.0, 0.0);
                    v[i] = make_double2(0.0, 0.0);
                }
                if (!g.sync()) return false;
                rho = make_double2(1.0, 0.0);
                alpha = rho;
                omega = rho;
                rho_new = make_double2(rr, 0.0);
                rh2 = rr;
                ++restarts;
                return true;
            };
            for (; it < A.max_it; ++it) {
                if (!(sqrt(cabs2(rho_new)) >= kBreakdownRel * sqrt(rh2 * rr))) {
                    if (restarts < A.max_restarts && rr > 0.0) { if (!restart()) return false; }
                    else { code = kKrylovBreakRho; break; }
                }
                const double2 beta = cmul(cdiv(rho_new, rho), cdiv(alpha, omega));
                rho = rho_new;
                for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x)
                    p[i] = cadd(cmul(csub(p[i], cmul(omega, v[i])), beta), r[i]);
                if (!g.sync()) return false;
                for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
                    double2 z = cmul(ms[i], p[i]);
                    const int pi = A.partner[i];
                    if (pi >= 0) z = cadd(z, cmul(mp[i], p[pi]));
                    ph[i] = z;
                }
                if (!g.sync()) return false;
                double a1[4] = {0.0, 0.0, 0.0, 0.0};     // r_hat^H v, ||v||^2
                cspmv<LPR>(A, w, ph, r0, r1, [&](int i, double2 y) {
                    v[i] = y;
                    const double2 d = cdotc(rh[i], y);
                    a1[0] += d.x;
                    a1[1] += d.y;
                    a1[2] += cabs2(y);
                });
                if (!g.sum<4>(a1)) return false;
                const double2 rhv = make_double2(a1[0], a1[1]);
                if (!(sqrt(cabs2(rhv)) >= kBreakdownRel * sqrt(rh2 * a1[2]))) {
                    if (restarts < A.max_restarts && rr > 0.0) {
                        if (!restart()) return false;
                        continue;
                    }
                    code = kKrylovBreakRv;
                    break;
                }
                alpha = cdiv(rho, rhv);
                double a2[1] = {0.0};
                for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
                    const double2 si = csub(r[i], cmul(alpha, v[i]));
                    s[i] = si;
                    a2[0] += cabs2(si);
                }
                if (!g.sum<1>(a2)) return false;
                if (sqrt(a2[0]) < abs_tol) {                     // gpu.rs:646-650
                    for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) x[i] = cadd(x[i], cmul(alpha, ph[i]));
                    rnorm = sqrt(a2[0]);
                    code = kKrylovConverged;
                    ++it;
                    break;
                }
                for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
                    double2 z = cmul(ms[i], s[i]);
                    const int pi = A.partner[i];
                    if (pi >= 0) z = cadd(z, cmul(mp[i], s[pi]));
                    sh[i] = z;
                }
                if (!g.sync()) return false;
                double a3[3] = {0.0, 0.0, 0.0};          // t^H s, t^H t
                cspmv<LPR>(A, w, sh, r0, r1, [&](int i, double2 y) {
                    t[i] = y;
                    const double2 d = cdotc(y, s[i]);
                    a3[0] += d.x;
                    a3[1] += d.y;
                    a3[2] += cabs2(y);
                });
                if (!g.sum<3>(a3)) return false;
                if (!(a3[2] > 0.0)) { code = kKrylovBreakTt; break; }
                omega = cdiv(make_double2(a3[0], a3[1]), make_double2(a3[2], 0.0));
                double a4[3] = {0.0, 0.0, 0.0};          // r_hat^H r, ||r||^2
                for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
                    x[i] = cadd(cadd(x[i], cmul(alpha, ph[i])), cmul(omega, sh[i]));
                    const double2 ri = csub(s[i], cmul(omega, t[i]));
                    r[i] = ri;
                    const double2 d = cdotc(rh[i], ri);
                    a4[0] += d.x;
                    a4[1] += d.y;
                    a4[2] += cabs2(ri);
                }
                if (!g.sum<3>(a4)) return false;
                rho_new = make_double2(a4[0], a4[1]);
                rr = a4[2];
                rnorm = sqrt(rr);
                if (!isfinite(rnorm)) { code = kKrylovNan; ++it; break; }
                if (rnorm < abs_tol) { code = kKrylovConverged; ++it; break; }
                if (!(cabs2(omega) > 1e-60)) { code = kKrylovBreakOmega; ++it; break; }
            }
            if (code == kKrylovRunning) code = kKrylovMaxIter;
        }
        __syncthreads();
        if (g.m == 0 && threadIdx.x == 0) {
            AcDev &d = A.info[q];
            d.code = code;
            d.iterations = it;
            d.restarts = restarts;
            d.rnorm = rnorm;
            d.bnorm = bnorm;
        }
        __syncthreads();
    }
    return true;
}

// Team mode (cooperative launch, fewer points than resident blocks): block
// b solves point blk_point[b] with the other members of its team.
template <int LPR>
__global__ void __launch_bounds__(kAcWideBlock) ac_team_kernel(AcArgs A) {
    __shared__ double smem[32 * 4];
    AcTeam<true> g;
    g.smem = smem;
    g.epoch = 0;
    g.red = 0;
    const int q = A.blk_point[blockIdx.x];
    g.T = A.point_team[q];
    g.m = A.blk_member[blockIdx.x];
    g.r0 = (int)(((long long)A.n * g.m) / g.T);
    g.r1 = (int)(((long long)A.n * (g.m + 1)) / g.T);
    g.count = A.team_count + q;
    g.part = A.team_part + (size_t)q * 8 * kAcMaxTeam;
    g.error = A.team_error;
    ac_point<LPR, true>(A, q, g);
}

// Queue mode: each block takes points from the queue and solves each alone.
template <int LPR, int BLOCK>
__global__ void __launch_bounds__(BLOCK) ac_sweep_kernel(AcArgs A) {
    __shared__ double smem[32 * 4];
    __shared__ int s_q;
    AcTeam<false> g;
    g.smem = smem;
    g.epoch = 0;
    g.red = 0;
    g.T = 1;
    g.m = 0;
    g.r0 = 0;
    g.r1 = A.n;
    g.count = nullptr;
    g.part = nullptr;
    g.error = nullptr;
    for (;;) {
        if (threadIdx.x == 0) s_q = (int)atomicAdd(A.queue, 1u);
        __syncthreads();
        const int q = s_q;
        __syncthreads();
        if (q >= A.n_freq) return;
        ac_point<LPR, false>(A, q, g);
    }
}

// ---------------------------------------------------------- cluster form --
// One frequency point per thread-block cluster, everything that an iteration
// touches on the chip: p, v, r (s), t, r_hat, the preconditioner and the
// gathered vector z = M^-1 p or M^-1 s of each block's rows in shared memory
// (112 bytes a row), the matrix in 32-row slices (G and j w C apart, 16-bit
// local columns) streamed from L2, where all points share it.  Blocks meet at
// cluster barriers: own z, one barrier, the halo rows of z fetched once each
// from their owners' shared memory, the product, one reduction.  The
// recurrence's scalars are updated by one lane inside the reductions.
//
// What bounds it: latency (five cluster barriers and reductions an iteration)
// and issued instructions, so a cluster is the smallest that holds a point
// (throughput is points in flight / time per iteration, and the fixed part of
// an iteration does not shrink with more blocks; 10,002 rows x 90 points on
// clusters of 5 / 6 / 8 / 10 / 16: 71 / 75 / 85 / 92 / 140 ms).  The block and
// team forms above keep their vectors in global memory (158 MB for those 90
// points, more than L2 holds).  Before -> after: 10,002 rows x 90 points 160
// -> 60 ms, 3,002 x 90 33 -> 15 ms, 902 x 90 11.0 -> 4.3 ms, 902 x 540 24 ->
// 15 ms, 92 x 720 9.9 -> 9.7 ms, 30,602 x 27 361 -> 109 ms, so every system
// that fits a cluster of 16 takes this form.
constexpr int kAcClusterBlock = 512;
constexpr int kAcClusterMax = 16;
constexpr int kAcRowBytes = 7 * 16;        // p v r t rh ms z

struct AcClusterArgs {
    int C, smem_bytes, any_pair;
    const uint32_t *sl_ptr;                // per 32-row slice of each block: first entry / 32 (slice_base[b] + s)
    const uint32_t *slice_base;            // per block: first slice in sl_ptr
    const uint16_t *col;                   // local columns, 32 entries per slice column
    const double *gval, *cval;             // G and C in the same places (cval may be null)
    const uint32_t *halo_ptr, *halo;       // per block: places of its halo rows
    const uint32_t *pair_ptr, *pair_row;   // per block: its rows in 2x2 pairs (local index) ...
    const uint32_t *pair_place;            // ... and their partners' places
    const uint32_t *place_partner;         // per row in a pair: the partner's place
};

// A place: block rank in the upper bits, local row in the lower; for a halo
// row, bit kPlacePaired marks half of a 2x2 pair.
constexpr uint32_t kPlaceBits = 20, kPlacePaired = 0x80000000u;

struct AcScalars {
    double2 beta, om, al, omega, rho, rho_new;
    double rr, rh2, bnorm, abs_tol, tol2, rnorm;
    int phase, restart, code, it, restarts, q;
};

// Entry of an own-row array (at the same offset in every block) at a place.
__device__ __forceinline__ double2 ld_place(const double2 *base, uint32_t place) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(base + (place & ((1u << kPlaceBits) - 1u)));
    uint32_t r;
    double2 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(r) : "r"(a), "r"((place & ~kPlacePaired) >> kPlaceBits));
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(r) : "memory");
    return v;
}

// !(sqrt(x) >= rel sqrt(y)) through squares (see below_root()).
__device__ __forceinline__ bool root_below_root(double x, double rel, double y) {
    const double y2 = rel * rel * y;
    if (x > 1e-290 && x < 1e290 && y2 > 1e-290 && y2 < 1e290) return x < y2;
    return !(sqrt(x) >= rel * sqrt(y));
}

// One lane: what follows a reduction (totals s), the same tests and order as
// ac_point().
__device__ __forceinline__ void ac_scalars_step(AcScalars &q, const double (&s)[4], const AcArgs &A) {
    bool top = false, restart = false;
    int code = kKrylovRunning, next = kPhaseDone;
    const double2 one = make_double2(1.0, 0.0);
    if (q.phase == kPhaseStart) {
        q.bnorm = q.rnorm = sqrt(s[0]);
        q.abs_tol = A.tol * q.bnorm;
        q.tol2 = q.abs_tol * q.abs_tol;
        q.rr = q.rh2 = s[0];
        q.rho_new = make_double2(s[0], 0.0);
        q.rho = q.al = q.omega = one;
        q.it = q.restarts = 0;
        if (!(q.bnorm >= 1e-30)) code = isfinite(q.bnorm) ? kKrylovConverged : kKrylovNan;   // b = 0: x = 0
        else top = true;
    } else if (q.phase == kPhaseAB) {
        const double2 rhv = make_double2(s[0], s[1]);
        if (root_below_root(cabs2(rhv), kBreakdownRel, q.rh2 * s[2])) {
            if (q.restarts < A.max_restarts && q.rr > 0.0) {
                ++q.it;
                restart = top = true;
            } else {
                code = kKrylovBreakRv;
            }
        } else {
            q.al = cdiv(q.rho, rhv);
            next = kPhaseCD;
        }
    } else if (q.phase == kPhaseCD) {              // |s|^2, t^H s, |t|^2
        if (root_below(s[0], q.abs_tol, q.tol2)) {
            code = kKrylovConverged;
            q.rnorm = sqrt(s[0]);
            ++q.it;
        } else if (!(s[3] > 0.0)) {
            code = kKrylovBreakTt;
        } else {
            q.omega = cdiv(make_double2(s[1], s[2]), make_double2(s[3], 0.0));
            next = kPhaseE;
        }
    } else {
        q.rho_new = make_double2(s[0], s[1]);
        q.rr = s[2];
        ++q.it;
        if (!isfinite(s[2])) code = kKrylovNan;
        else if (root_below(s[2], q.abs_tol, q.tol2)) code = kKrylovConverged;
        else if (!(cabs2(q.omega) > 1e-60)) code = kKrylovBreakOmega;
        else top = true;
    }
    if (top) {
        const bool stop = q.it >= A.max_it;
        if (!restart && !stop && root_below_root(cabs2(q.rho_new), kBreakdownRel, q.rh2 * q.rr)) {
            if (q.restarts < A.max_restarts && q.rr > 0.0) restart = true;
            else code = kKrylovBreakRho;
        }
        if (stop) code = kKrylovMaxIter;
        if (restart) {
            ++q.restarts;
            q.rho = q.al = q.omega = one;
            q.rho_new = make_double2(q.rr, 0.0);
            q.rh2 = q.rr;
        }
        if (code == kKrylovRunning) {
            q.beta = cmul(cdiv(q.rho_new, q.rho), cdiv(q.al, q.omega));
            q.om = q.omega;
            q.rho = q.rho_new;
            next = kPhaseAB;
        }
    }
    if (code != kKrylovRunning && q.phase != kPhaseStart && code != kKrylovConverged) q.rnorm = sqrt(q.rr);
    if (code == kKrylovConverged && q.phase == kPhaseE) q.rnorm = sqrt(q.rr);
    q.restart = restart ? 1 : 0;
    q.code = code;
    q.phase = code == kKrylovRunning ? next : kPhaseDone;
}

__global__ void __launch_bounds__(kAcClusterBlock, 1) ac_cluster_kernel(const __grid_constant__ AcArgs A,
                                                                        const __grid_constant__ AcClusterArgs K) {
    __shared__ AcScalars S;
    const int C = K.C, rank = (int)(blockIdx.x % (unsigned)C), n = A.n;
    const int r0 = (int)(((long long)n * rank) / C), r1 = (int)(((long long)n * (rank + 1)) / C), R = r1 - r0;
    const int stride = (n + C - 1) / C;            // rows of the largest block: uniform offsets
    const int lane = threadIdx.x & 31;
    double2 *p = (double2 *)ohm_dsmem, *v = p + stride, *r = v + stride, *t = r + stride, *rh = t + stride,
            *ms = rh + stride, *z = ms + stride;
    const int H = (int)(K.halo_ptr[rank + 1] - K.halo_ptr[rank]);
    uint32_t *halo = (uint32_t *)(z + R + H + 1);
    for (int h = threadIdx.x; h < H; h += blockDim.x) halo[h] = K.halo[K.halo_ptr[rank] + h];
    const uint32_t *sl = K.sl_ptr + K.slice_base[rank];
    const GridSync none{nullptr, nullptr};
    reduce_buffers_init();
    if (C > 1) cluster_barrier();
    auto team_sync = [&]() { if (C > 1) cluster_barrier(); else __syncthreads(); };
    for (;;) {
        // next point: the cluster's first block takes it and tells the others
        if (rank == 0 && threadIdx.x == 0) {
            const int q = (int)atomicAdd(A.queue, 1u);
            for (int k = 0; k < C; ++k) {
                const uint32_t a = (uint32_t)__cvta_generic_to_shared(&S.q);
                uint32_t b;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(k));
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(b), "r"(q) : "memory");
            }
        }
        team_sync();
        const int q = S.q;
        if (q >= A.n_freq) return;
        const double w = A.omega[q];
        double2 *W = A.work + (size_t)q * A.vecs * n;
        double2 *x = W + r0, *mp = W + n;           // x and, for 2x2 pairs, the partner's coefficient
        if (threadIdx.x == 0) S.phase = kPhaseStart;
        __syncthreads();
        for (;;) {
            const int phase = S.phase;
            if (phase == kPhaseDone) break;
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
            if (phase == kPhaseE) {
                const double2 omega = S.omega;
#pragma unroll 4
                for (int li = threadIdx.x; li < R; li += blockDim.x) {
                    x[li] = cadd(x[li], cmul(omega, z[li]));
                    const double2 ri = csub(r[li], cmul(omega, t[li]));
                    r[li] = ri;
                    const double2 d = cdotc(rh[li], ri);
                    acc[0] += d.x;
                    acc[1] += d.y;
                    acc[2] += cabs2(ri);
                }
            } else if (phase != kPhaseStart) {
                const bool cd = phase == kPhaseCD;
                const double2 al = S.al;
                if (!cd && S.restart) {
#pragma unroll 1
                    for (int li = threadIdx.x; li < R; li += blockDim.x) {
                        rh[li] = r[li];
                        p[li] = make_double2(0.0, 0.0);
                        v[li] = make_double2(0.0, 0.0);
                    }
                }
                // p's update, or s (kept in r) and x += alpha M^-1 p; z = M^-1 of it
                const double2 beta = S.beta, om = S.om;
#pragma unroll 4
                for (int li = threadIdx.x; li < R; li += blockDim.x) {
                    double2 u;
                    if (cd) {
                        u = csub(r[li], cmul(al, v[li]));
                        x[li] = cadd(x[li], cmul(al, z[li]));
                        r[li] = u;
                    } else {
                        u = cadd(cmul(csub(p[li], cmul(om, v[li])), beta), r[li]);
                        p[li] = u;
                    }
                    z[li] = cmul(ms[li], u);
                }
                team_sync();
                double2 *u = cd ? r : p;
#pragma unroll 2
                for (int h = threadIdx.x; h < H; h += blockDim.x) {
                    const uint32_t at = halo[h];
                    if (!(at & kPlacePaired)) {
                        z[R + h] = ld_place(z, at);
                    } else {
                        const int q1 = (int)((at & ~kPlacePaired) >> kPlaceBits);
                        const int j = (int)(((long long)n * q1) / C) + (int)(at & ((1u << kPlaceBits) - 1u));
                        z[R + h] = cadd(cmul(ld_place(ms, at), ld_place(u, at)), cmul(mp[j], ld_place(u, K.place_partner[j])));
                    }
                }
                if (K.any_pair) {
                    const uint32_t k1 = K.pair_ptr[rank + 1];
                    for (uint32_t k = K.pair_ptr[rank] + threadIdx.x; k < k1; k += blockDim.x) {
                        const int li = (int)K.pair_row[k];
                        z[li] = cadd(z[li], cmul(mp[r0 + li], ld_place(u, K.pair_place[k])));
                    }
                }
                __syncthreads();
#pragma unroll 1
                for (int li = threadIdx.x; li - lane < R; li += blockDim.x) {
                    const uint32_t e = sl[(li >> 5) + 1] * 32u;
                    uint32_t k = sl[li >> 5] * 32u + lane;
                    double2 y = make_double2(0.0, 0.0);
#pragma unroll 5
                    for (; k < e; k += 32u) {
                        const double2 a = make_double2(K.gval[k], K.cval ? w * K.cval[k] : 0.0);
                        y = cadd(y, cmul(a, z[K.col[k]]));
                    }
                    if (li < R) {
                        if (cd) {
                            const double2 si = r[li], d = cdotc(y, si);
                            t[li] = y;
                            acc[0] += cabs2(si);
                            acc[1] += d.x;
                            acc[2] += d.y;
                            acc[3] += cabs2(y);
                        } else {
                            const double2 d = cdotc(rh[li], y);
                            v[li] = y;
                            acc[0] += d.x;
                            acc[1] += d.y;
                            acc[2] += cabs2(y);
                        }
                    }
                }
            } else {
#pragma unroll 1
                for (int li = threadIdx.x; li < R; li += blockDim.x) {
                    const int i = r0 + li;
                    double2 cp;
                    ms[li] = ac_precond(A, i, w, cp);
                    if (K.any_pair) mp[i] = cp;
                    const double2 bi = A.b[i];
                    x[li] = make_double2(0.0, 0.0);
                    r[li] = bi;
                    rh[li] = bi;
                    p[li] = make_double2(0.0, 0.0);
                    v[li] = make_double2(0.0, 0.0);
                    acc[0] += cabs2(bi);
                }
                if (threadIdx.x == 0) z[R + H] = make_double2(0.0, 0.0);   // the padding's column
            }
            // never false: no counter barrier in a cluster
            team_reduce_then<4, false>(C, rank, C > 1, nullptr, none, acc, [&](const double (&s)[4], bool writer) {
                if (writer) ac_scalars_step(S, s, A);
            });
        }
        if (rank == 0 && threadIdx.x == 0) {
            AcDev &d = A.info[q];
            d.code = S.code;
            d.iterations = S.it;
            d.restarts = S.restarts;
            d.rnorm = S.rnorm;
            d.bnorm = S.bnorm;
        }
        team_sync();                                // S and the vectors are reused
    }
}

using AcFn = void (*)(AcArgs);

// Host side of the cluster form: cluster size, halo rows and 32-row slices of
// every block, and the nonzeros' local columns in CSR order.  The slices
// themselves are filled on the device (ac_fill_slices()).
struct AcSlices {
    int C = 0, smem_bytes = 0;
    uint32_t entries = 0;                               // padded nonzeros / 32
    std::vector<uint32_t> sl_ptr, sl_row, sl_end, sl_pad;   // per slice (and one more per block): entries so far,
                                                            // its rows, the padding's column
    std::vector<uint32_t> slice_base, halo_ptr, halo, pair_ptr, pair_row, pair_place, place_partner;
    std::vector<uint16_t> lcol;

    // The smallest cluster whose blocks hold their part of a point in `avail`
    // bytes of shared memory; false when none does, or when its blocks fetch more
    // halo rows than they own (10,000 rows of 15 scattered entries, whole calls:
    // one point 2.0 ms in the block form, 4.0 ms so; 100 points 10.8 and 9.3;
    // with a fifth as many halo rows as own ones 2.2 and 2.1 ms).  One pass over the
    // nonzeros where it can be: a size is tried only when its middle block
    // fits, and none when the middle block of the largest cluster does not
    // (a larger cluster's blocks hold fewer rows and touch no more).
    // (With every size tried in full and the slices filled here, the
    // set-up of 10,000 rows of 40 entries took longer than their solve: one
    // point 3.9 ms in the block form, 22.7 ms so.)
    bool build(int64_t n, const uint32_t *rp, const uint32_t *cl, int64_t avail, const std::vector<int32_t> &partner,
               bool any_pair) {
        const int c_max = (int)std::min<int64_t>(kAcClusterMax, n);
        std::vector<int32_t> at(n, -1);
        lcol.resize(rp[n]);
        C = c_max;
        if (!start(n, avail) || !block(n, rp, cl, C / 2, avail, at)) return false;
        const int64_t touched = (n + C - 1) / C + (int64_t)halo.size();     // a larger block touches no fewer
        for (C = 1; C <= c_max; ++C) {
            if (!start(n, avail)) continue;
            if (C > 1 && touched > 2 * ((n + C - 1) / C)) return false;     // more halo rows than own ones
            if (C > 1 && !block(n, rp, cl, C / 2, avail, at)) continue;
            if ((int64_t)halo.size() > (n + C - 1) / C) return false;
            start(n, avail);
            bool ok = true;
            for (int b = 0; b < C && ok; ++b) ok = block(n, rp, cl, b, avail, at);
            if (ok) break;
        }
        if (C > c_max || (int64_t)halo.size() > n) return false;
        // halo rows and partners as places
        auto place = [&](int64_t j) -> uint32_t {
            int64_t q = (j * C) / n;
            while (j >= n * (q + 1) / C) ++q;
            return (uint32_t)((q << kPlaceBits) | (j - n * q / C));
        };
        for (uint32_t &h : halo) h = place(h) | (partner[h] >= 0 ? kPlacePaired : 0u);
        pair_ptr.assign(1, 0);
        if (any_pair) place_partner.assign(n, 0);
        for (int b = 0; b < C; ++b) {
            const int64_t r0 = n * b / C, r1 = n * (b + 1) / C;
            for (int64_t i = any_pair ? r0 : r1; i < r1; ++i) {
                if (partner[i] < 0) continue;
                place_partner[i] = place(partner[i]);
                pair_row.push_back((uint32_t)(i - r0));
                pair_place.push_back(place_partner[i]);
            }
            pair_ptr.push_back((uint32_t)pair_row.size());
        }
        return true;
    }

private:
    bool start(int64_t n, int64_t avail) {
        sl_ptr.clear(); sl_row.clear(); sl_end.clear(); sl_pad.clear(); slice_base.clear(); halo.clear();
        halo_ptr.assign(1, 0);
        entries = 0;
        smem_bytes = 0;
        return ((n + C - 1) / C) * kAcRowBytes + 16 * 64 <= avail;
    }
    // Appends block b; false when it does not fit.  at: -1 everywhere, and again afterwards.
    bool block(int64_t n, const uint32_t *rp, const uint32_t *cl, int b, int64_t avail, std::vector<int32_t> &at) {
        const int64_t r0 = n * b / C, r1 = n * (b + 1) / C, R = r1 - r0, stride = (n + C - 1) / C;
        const size_t h0 = halo.size();
        // 16 bytes of z and 4 of its place for a halo row, and a zero
        const int64_t h_fit = std::min<int64_t>((avail - stride * kAcRowBytes - 32) / 20, 0xFFFE - R);
        bool ok = true;
        for (uint32_t k = rp[r0]; k < rp[r1] && ok; ++k) {
            const int64_t j = cl[k];
            if (j >= r0 && j < r1) {
                lcol[k] = (uint16_t)(j - r0);
                continue;
            }
            if (at[j] < 0) {
                ok = (int64_t)(halo.size() - h0) < h_fit;
                at[j] = (int32_t)(R + (int64_t)(halo.size() - h0));
                halo.push_back((uint32_t)j);
            }
            lcol[k] = (uint16_t)at[j];
        }
        for (size_t h = h0; h < halo.size(); ++h) at[halo[h]] = -1;
        const int64_t H = (int64_t)(halo.size() - h0);
        halo_ptr.push_back((uint32_t)halo.size());
        slice_base.push_back((uint32_t)sl_ptr.size());
        for (int64_t s = r0; s < r1 && ok; s += 32) {
            uint32_t width = 0;
            for (int64_t i = s; i < std::min(r1, s + 32); ++i) width = std::max(width, rp[i + 1] - rp[i]);
            slice(s, std::min(r1, s + 32), R + H);
            entries += width;
            ok = 32ull * entries <= 2ull * (uint64_t)rp[n] + 4096;      // else rows too uneven to pad
        }
        slice(r1, r1, R + H);
        smem_bytes = std::max(smem_bytes, (int)(stride * kAcRowBytes + 20 * H + 32));
        return ok;
    }
    void slice(int64_t row, int64_t end, int64_t pad) {
        sl_ptr.push_back(entries);
        sl_row.push_back((uint32_t)row);
        sl_end.push_back((uint32_t)end);
        sl_pad.push_back((uint32_t)pad);
    }
};

// Fills the matrix slices from the CSR arrays: one warp a slice, its lanes the
// slice's rows.  Padding has value 0 and the column of a zero.
__global__ void ac_fill_slices(int n_slices, const uint32_t *__restrict__ sl_ptr, const uint32_t *__restrict__ sl_row,
                               const uint32_t *__restrict__ sl_end, const uint32_t *__restrict__ sl_pad,
                               const uint32_t *__restrict__ rp, const uint16_t *__restrict__ lcol,
                               const double *__restrict__ g, const double *__restrict__ c, uint16_t *col, double *gval,
                               double *cval) {
    const int s = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (s >= n_slices || sl_row[s] == sl_end[s]) return;       // (a block's last entry has no rows)
    const uint32_t i = sl_row[s] + lane, end = sl_end[s], pad = sl_pad[s], e0 = sl_ptr[s];
    const uint32_t width = sl_ptr[s + 1] - e0;
    const uint32_t k0 = i < end ? rp[i] : 0u, len = i < end ? rp[i + 1] - k0 : 0u;
    for (uint32_t k = 0; k < width; ++k) {
        const size_t e = (size_t)(e0 + k) * 32 + lane;
        const bool in = k < len;
        col[e] = in ? lcol[k0 + k] : (uint16_t)pad;
        gval[e] = in ? g[k0 + k] : 0.0;
        if (c) cval[e] = in ? c[k0 + k] : 0.0;
    }
}

AcFn pick_ac(double avg, bool wide) {
    if (wide) {
        if (avg <= 3.0) return ac_sweep_kernel<2, kAcWideBlock>;
        if (avg <= 12.0) return ac_sweep_kernel<4, kAcWideBlock>;
        return ac_sweep_kernel<8, kAcWideBlock>;
    }
    if (avg <= 3.0) return ac_sweep_kernel<2, kAcBlock>;
    if (avg <= 12.0) return ac_sweep_kernel<4, kAcBlock>;
    return ac_sweep_kernel<8, kAcBlock>;
}

AcFn pick_ac_team(double avg) {
    if (avg <= 3.0) return ac_team_kernel<2>;
    if (avg <= 12.0) return ac_team_kernel<4>;
    return ac_team_kernel<8>;
}

}  // namespace

extern "C" ohm_status ohm_ac_sweep(ohm_ctx *c, int64_t n, int64_t nnz, const uint32_t *row_ptr, const uint32_t *col,
                                   const double *g_values, const double *c_values, const double *b_re_im,
                                   int64_t n_freq, const double *freqs_hz, const ohm_krylov_params *params,
                                   double *x_re_im, ohm_ac_point_info *points) {
    if (!c || !params || n_freq < 0) return ohm_fail(OHM_ERR_INVALID_ARG, "bad arguments");
    ohm_status st = ohm_check_krylov(params);
    if (st != OHM_OK) return st;
    if (params->precond == OHM_PRECOND_ISAI1)
        return ohm_fail(OHM_ERR_INVALID_ARG, "the AC sweep uses block Jacobi, Jacobi or no preconditioner");
    if (n_freq == 0 || n == 0) return OHM_OK;
    if (!b_re_im || !x_re_im || !freqs_hz || (nnz && !g_values))
        return ohm_fail(OHM_ERR_INVALID_ARG, "null array");
    st = check_csr(n, nnz, row_ptr, col);
    if (st != OHM_OK) return st;
    for (int64_t k = 0; k < n_freq; ++k)
        if (!std::isfinite(freqs_hz[k])) return ohm_fail(OHM_ERR_INVALID_ARG, "frequency %lld is not finite", (long long)k);
    CUDA_TRY(cudaSetDevice(c->device));
    // block-Jacobi pairing from the real part's structure
    std::vector<char> touched(nnz, 0);
    PcHost pc;
    build_precond(n, row_ptr, col, g_values, touched, params->precond == OHM_PRECOND_AUTO, pc);
    // cluster form where a point fits a cluster's shared memory
    AcSlices slices;
    AcClusterArgs K{};
    std::vector<uint32_t> words;
    int clusters = 0;
    cudaLaunchAttribute cl_attr[1];
    cudaLaunchConfig_t cl_cfg = {};
    if (n >= 1) {
        const int avail = ohm_max_dynamic_smem((const void *)ac_cluster_kernel);
        if (avail > 0 && slices.build(n, row_ptr, col, avail, pc.partner, pc.any_pair) &&
            cudaFuncSetAttribute(ac_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            cl_attr[0].id = cudaLaunchAttributeClusterDimension;
            cl_attr[0].val.clusterDim.x = (unsigned)slices.C;
            cl_attr[0].val.clusterDim.y = cl_attr[0].val.clusterDim.z = 1;
            cl_cfg.gridDim = dim3((unsigned)slices.C);
            cl_cfg.blockDim = dim3(kAcClusterBlock);
            cl_cfg.dynamicSmemBytes = (size_t)slices.smem_bytes;
            cl_cfg.stream = c->stream;
            cl_cfg.attrs = cl_attr;
            cl_cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&clusters, ac_cluster_kernel, &cl_cfg) != cudaSuccess) clusters = 0;
        }
        (void)cudaGetLastError();
    }
    const int vecs = clusters > 0 ? 2 : kAcVecs;
    // frequency groups sized so the per-point workspace stays under ~4 GB
    const size_t per_point = (size_t)vecs * n * sizeof(double2);
    const int64_t group = std::max<int64_t>(1, std::min<int64_t>(n_freq, ((size_t)4 << 30) / per_point));
    std::vector<void *> allocs;
    auto put = [&](auto **dst, const auto *src, size_t count) -> cudaError_t {
        cudaError_t e = dalloc(dst, count);
        if (e == cudaSuccess) allocs.push_back((void *)*dst);
        if (e == cudaSuccess && src && count)
            e = cudaMemcpyAsync(*dst, src, count * sizeof(**dst), cudaMemcpyHostToDevice, c->stream);
        return e;
    };
    AcArgs A{};
    uint32_t *d_rp = nullptr, *d_col = nullptr, *d_diag = nullptr, *d_off = nullptr;
    double *d_g = nullptr, *d_c = nullptr, *d_omega = nullptr;
    double2 *d_b = nullptr, *d_work = nullptr;
    int32_t *d_partner = nullptr;
    AcDev *d_info = nullptr;
    unsigned int *d_queue = nullptr;
    cudaError_t e = put(&d_rp, row_ptr, n + 1);
    if (e == cudaSuccess) e = put(&d_col, col, nnz);
    if (e == cudaSuccess) e = put(&d_g, g_values, nnz);
    if (e == cudaSuccess && c_values) e = put(&d_c, c_values, nnz);
    if (e == cudaSuccess) e = put(&d_b, (const double2 *)b_re_im, n);
    if (e == cudaSuccess) e = put(&d_partner, pc.partner.data(), n);
    if (e == cudaSuccess) e = put(&d_diag, pc.diag_slot.data(), n);
    if (e == cudaSuccess) e = put(&d_off, pc.off_slot.data(), n);
    if (e == cudaSuccess) e = put(&d_omega, (const double *)nullptr, group);
    if (e == cudaSuccess) e = put(&d_work, (const double2 *)nullptr, (size_t)group * vecs * n);
    if (e == cudaSuccess) e = put(&d_info, (const AcDev *)nullptr, group);
    if (e == cudaSuccess) e = put(&d_queue, (const unsigned int *)nullptr, 1);
    A.n = (int)n;
    A.precond = params->precond == OHM_PRECOND_NONE ? kPcNone
              : (params->precond == OHM_PRECOND_JACOBI ? kPcJacobi : kPcAuto);
    A.max_it = params->max_iterations;
    A.max_restarts = std::max(0, params->max_restarts);
    A.tol = params->tolerance;
    A.rp = d_rp; A.col = d_col; A.g = d_g; A.c = d_c; A.b = d_b; A.omega = d_omega;
    A.partner = d_partner; A.diag_slot = d_diag; A.off_slot = d_off;
    A.work = d_work; A.info = d_info; A.queue = d_queue;
    A.vecs = vecs;
    if (clusters > 0) {
        K.C = slices.C;
        K.smem_bytes = slices.smem_bytes;
        K.any_pair = pc.any_pair ? 1 : 0;
        // the index arrays as one upload
        const std::vector<uint32_t> *parts[] = {&slices.sl_ptr,   &slices.sl_row, &slices.sl_end,   &slices.sl_pad,
                                                &slices.slice_base, &slices.halo_ptr, &slices.halo, &slices.pair_ptr,
                                                &slices.pair_row, &slices.pair_place, &slices.place_partner};
        size_t first[11];
        for (int q = 0; q < 11; ++q) {
            first[q] = words.size();
            words.insert(words.end(), parts[q]->begin(), parts[q]->end());
        }
        uint32_t *u = nullptr;
        uint16_t *lc = nullptr, *h = nullptr;
        double *gv = nullptr, *cv = nullptr;
        const size_t padded = 32 * (size_t)slices.entries;
        if (e == cudaSuccess) e = put(&u, words.data(), words.size());
        if (e == cudaSuccess) e = put(&lc, slices.lcol.data(), slices.lcol.size());
        if (e == cudaSuccess) e = put(&h, (const uint16_t *)nullptr, padded);
        if (e == cudaSuccess) e = put(&gv, (const double *)nullptr, padded);
        if (e == cudaSuccess && c_values) e = put(&cv, (const double *)nullptr, padded);
        K.sl_ptr = u + first[0]; K.slice_base = u + first[4]; K.halo_ptr = u + first[5]; K.halo = u + first[6];
        K.pair_ptr = u + first[7]; K.pair_row = u + first[8]; K.pair_place = u + first[9];
        K.place_partner = u + first[10];
        K.col = h; K.gval = gv; K.cval = cv;
        if (e == cudaSuccess) {
            const int n_slices = (int)slices.sl_ptr.size();
            ac_fill_slices<<<(n_slices + 7) / 8, 256, 0, c->stream>>>(n_slices, K.sl_ptr, u + first[1], u + first[2],
                                                                      u + first[3], d_rp, lc, d_g, d_c, h, gv, cv);
            e = cudaGetLastError();
        }
    }
    // a point per SM at most: give each point a whole SM when the system is large
    const bool wide = n >= 2048 && n_freq <= c->num_sms;
    const int block = wide ? kAcWideBlock : kAcBlock;
    AcFn fn = pick_ac((double)nnz / (double)n, wide);
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, block, 0);
    std::vector<double> omega(group);
    std::vector<AcDev> hinfo(group);
    int64_t failed = -1;
    AcDev fail_info{};
    // Team mode: with fewer points than resident blocks, the spare blocks
    // join the lowest-frequency points (the slowest: the conductances
    // dominate) as teams of up to kAcMaxTeam blocks of >= 1024 rows each.
    const int total_blocks = std::max(per_sm, 1) * c->num_sms;
    const int tmax = (int)std::min<int64_t>(kAcMaxTeam, std::max<int64_t>(1, n / 1024));
    const AcFn fn_team = pick_ac_team((double)nnz / (double)n);
    int team_per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&team_per_sm, fn_team, kAcWideBlock, 0);
    // the team kernel must be co-resident: no more teamed blocks than it can hold
    const bool team_capable = wide && tmax >= 2 && group < total_blocks && team_per_sm * c->num_sms >= total_blocks;
    int32_t *d_blk_point = nullptr, *d_blk_member = nullptr, *d_point_team = nullptr;
    unsigned long long *d_team_count = nullptr;
    double *d_team_part = nullptr;
    int *d_team_error = nullptr;
    std::vector<int32_t> h_blk_point, h_blk_member, h_point_team;
    if (team_capable) {
        if (e == cudaSuccess) e = put(&d_blk_point, (const int32_t *)nullptr, total_blocks);
        if (e == cudaSuccess) e = put(&d_blk_member, (const int32_t *)nullptr, total_blocks);
        if (e == cudaSuccess) e = put(&d_point_team, (const int32_t *)nullptr, group);
        if (e == cudaSuccess) e = put(&d_team_count, (const unsigned long long *)nullptr, group);
        if (e == cudaSuccess) e = put(&d_team_part, (const double *)nullptr, (size_t)group * 8 * kAcMaxTeam);
        if (e == cudaSuccess) e = put(&d_team_error, (const int *)nullptr, 1);
        A.blk_point = d_blk_point; A.blk_member = d_blk_member; A.point_team = d_point_team;
        A.team_count = d_team_count; A.team_part = d_team_part; A.team_error = d_team_error;
    }
    int team_err_host = 0;
    for (int64_t f0 = 0; e == cudaSuccess && f0 < n_freq; f0 += group) {
        const int64_t m = std::min(group, n_freq - f0);
        for (int64_t k = 0; k < m; ++k) omega[k] = 2.0 * 3.14159265358979323846 * freqs_hz[f0 + k];   // ac.rs:57
        e = cudaMemcpyAsync(d_omega, omega.data(), m * sizeof(double), cudaMemcpyHostToDevice, c->stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(d_queue, 0, sizeof(unsigned int), c->stream);
        A.n_freq = (int)m;
        // team sizes: the same base size for every point, one more block for
        // the lowest frequencies while blocks are left
        int teamed = 0;
        if (clusters == 0 && team_capable && m < total_blocks) {
            const int base = std::min<int>(tmax, (int)(total_blocks / m));
            int spare = base < tmax ? total_blocks - base * (int)m : 0;
            std::vector<int32_t> by_freq((size_t)m);
            std::iota(by_freq.begin(), by_freq.end(), 0);
            std::stable_sort(by_freq.begin(), by_freq.end(), [&](int32_t x, int32_t y) { return omega[x] < omega[y]; });
            h_point_team.assign((size_t)m, base);
            for (int32_t q : by_freq) {
                if (spare == 0) break;
                ++h_point_team[q];
                --spare;
            }
            h_blk_point.clear();
            h_blk_member.clear();
            for (int64_t q = 0; q < m; ++q)
                for (int j = 0; j < h_point_team[q]; ++j) {
                    h_blk_point.push_back((int32_t)q);
                    h_blk_member.push_back(j);
                }
            if (base > 1 || h_point_team[by_freq[0]] > 1) teamed = (int)h_blk_point.size();
        }
        if (clusters > 0) {
            cl_cfg.gridDim = dim3((unsigned)(slices.C * (int)std::min<int64_t>(clusters, m)));
            if (e == cudaSuccess) e = cudaLaunchKernelEx(&cl_cfg, ac_cluster_kernel, A, K);
        } else if (teamed > 0) {
            A.team_mode = 1;
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(d_blk_point, h_blk_point.data(), teamed * sizeof(int32_t), cudaMemcpyHostToDevice,
                                    c->stream);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(d_blk_member, h_blk_member.data(), teamed * sizeof(int32_t),
                                    cudaMemcpyHostToDevice, c->stream);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(d_point_team, h_point_team.data(), m * sizeof(int32_t), cudaMemcpyHostToDevice,
                                    c->stream);
            if (e == cudaSuccess) e = cudaMemsetAsync(d_team_count, 0, m * sizeof(unsigned long long), c->stream);
            if (e == cudaSuccess) e = cudaMemsetAsync(d_team_error, 0, sizeof(int), c->stream);
            void *args[] = {&A};
            if (e == cudaSuccess)
                e = cudaLaunchCooperativeKernel((void *)fn_team, dim3(teamed), dim3(kAcWideBlock), args, 0, c->stream);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(&team_err_host, d_team_error, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
        } else {
            A.team_mode = 0;
            const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)total_blocks, m));
            if (e == cudaSuccess) {
                fn<<<grid, block, 0, c->stream>>>(A);
                e = cudaGetLastError();
            }
        }
        // x of every point: the first of its kAcVecs vectors
        for (int64_t k = 0; e == cudaSuccess && k < m; ++k)
            e = cudaMemcpyAsync(x_re_im + 2 * (size_t)(f0 + k) * n, d_work + (size_t)k * vecs * n,
                                n * sizeof(double2), cudaMemcpyDeviceToHost, c->stream);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(hinfo.data(), d_info, m * sizeof(AcDev), cudaMemcpyDeviceToHost, c->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
        if (e == cudaSuccess && team_err_host != 0) break;
        for (int64_t k = 0; e == cudaSuccess && k < m; ++k) {
            const AcDev &d = hinfo[k];
            if (points) {
                ohm_ac_point_info &o = points[f0 + k];
                o.krylov_code = d.code;
                o.iterations = d.iterations;
                o.restarts = d.restarts;
                o.reserved = 0;
                o.residual_norm = d.rnorm;
                o.b_norm = d.bnorm;
            }
            if (d.code != kKrylovConverged && failed < 0) { failed = f0 + k; fail_info = d; }
        }
    }
    cudaStreamSynchronize(c->stream);
    for (void *q : allocs) ohm_pool_free(q);
    if (e != cudaSuccess) return ohm_fail(OHM_ERR_CUDA, "AC sweep: %s", cudaGetErrorString(e));
    if (team_err_host != 0) return ohm_fail(OHM_ERR_TIMEOUT, "AC sweep: a team barrier wait gave up");
    if (failed >= 0)
        return ohm_fail(OHM_ERR_SOLVE, "BiCGSTAB did not converge at frequency point %lld (%.6e Hz, code %d)",
                        (long long)failed, freqs_hz[failed], fail_info.code);
    return OHM_OK;
}

// LinearSolver::solve_complex (src/solver/mod.rs:27-34, gpu.rs:210-735): one
// complex system A x = b as a one-point sweep with G = Re A, C = Im A and
// f = 1 / (2 pi), so that w = 2 pi f is exactly 1.0 and A(f) = A.
extern "C" ohm_status ohm_solve_complex(ohm_ctx *c, int64_t n, int64_t nnz, const uint32_t *row_ptr,
                                        const uint32_t *col, const double *values_re_im, const double *b_re_im,
                                        double *x_re_im, const ohm_krylov_params *params, ohm_ac_point_info *info) {
    if (!c || !params || n < 0 || nnz < 0) return ohm_fail(OHM_ERR_INVALID_ARG, "bad arguments");
    if (info) std::memset(info, 0, sizeof *info);
    if (n == 0) return OHM_OK;
    if (!row_ptr || !b_re_im || !x_re_im || (nnz && (!col || !values_re_im)))
        return ohm_fail(OHM_ERR_INVALID_ARG, "null array");
    std::vector<double> re((size_t)nnz), im((size_t)nnz);
    for (int64_t k = 0; k < nnz; ++k) {
        re[k] = values_re_im[2 * k];
        im[k] = values_re_im[2 * k + 1];
    }
    const double f = 1.0 / (2.0 * 3.14159265358979323846);
    ohm_ac_point_info pt{};
    const ohm_status st =
        ohm_ac_sweep(c, n, nnz, row_ptr, col, re.data(), im.data(), b_re_im, 1, &f, params, x_re_im, &pt);
    if (info) *info = pt;
    return st;
}
