// Shared device helpers for the persistent solver kernels: bounded grid
// barrier, deterministic block / grid reductions, small numeric helpers.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace ohm {

constexpr uint32_t kSentinel = 0xFFFFFFFFu;   // u32::MAX, ground / absent slot

// Device status words shared by all kernels (ohm_status values).
constexpr int kStatusOk = 0;
constexpr int kStatusTimeout = 5;

// Upper bound on one barrier wait: spin iterations (tight for the first
// kTightSpins, then __nanosleep(64)); about 2-3 s in total.  A wait that runs
// out records kStatusTimeout and the kernel returns; with a cooperative launch
// every block is resident, so a healthy barrier never comes near the bound.
// Clusters wait at the hardware's barrier, which has no bound to set: their
// blocks are scheduled together, take the same branches (decided on reductions
// that are bit-identical in every block) and leave only at the same points, and
// the barrier does not count threads that have left.
constexpr uint32_t kBarrierSpinLimit = 1u << 22;
constexpr uint32_t kTightSpins = 2048;

struct GridSync {
    unsigned long long *count;   // arrivals since launch (monotone, zeroed per launch)
    int *error;                  // first error recorded by any block (0 = none)
};

__device__ __forceinline__ void red_release_add_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Warp totals (sum, or max when MAX) of NV <= 4 values by the xor tree
// 16, 8, 4, 2, 1.  The first steps exchange halves: after step 16 the lanes
// with bit 4 set hold the upper half of the values, after step 8 (NV > 2)
// each lane holds one, so 4 values cost 6 double shuffles instead of 20 with
// the same pairs summed in the same tree (bit-identical totals).  A block of
// 32 warps is bound by the SM's shuffle rate here: 4 values took 1.2 us as 20
// shuffles a warp (of a 1.5 us one-block all-reduce).
// Value warp_value<NV>(lane) is returned on each lane (NV 3 counts as 4; the
// lanes of the missing value return 0).
template <int NV>
__device__ __forceinline__ int warp_value(int lane) {
    return NV == 1 ? 0 : (NV == 2 ? (lane >> 4) & 1 : ((lane >> 4) & 1) * 2 + ((lane >> 3) & 1));
}
template <int NV>
constexpr int kWarpValueLanes = NV == 1 ? 32 : (NV == 2 ? 16 : 8);   // lanes that hold one value's total

template <bool MAX>
__device__ __forceinline__ double combine2(double x, double y) { return MAX ? fmax(x, y) : x + y; }

template <int NV, bool MAX>
__device__ __forceinline__ double warp_totals(const double (&v)[NV], int lane) {
    static_assert(NV >= 1 && NV <= 4, "1 to 4 values");
    double x;
    int o = 16;
    if constexpr (NV == 1) {
        x = v[0];
    } else if constexpr (NV == 2) {
        const bool hi = lane & 16;
        const double keep = hi ? v[1] : v[0], send = hi ? v[0] : v[1];
        x = combine2<MAX>(keep, __shfl_xor_sync(0xffffffffu, send, 16));
        o = 8;
    } else {
        const double v3 = NV == 4 ? v[NV - 1] : 0.0;
        const bool hi = lane & 16, mid = lane & 8;
        double k0 = hi ? v[2] : v[0], k1 = hi ? v3 : v[1];
        const double s0 = hi ? v[0] : v[2], s1 = hi ? v[1] : v3;
        k0 = combine2<MAX>(k0, __shfl_xor_sync(0xffffffffu, s0, 16));
        k1 = combine2<MAX>(k1, __shfl_xor_sync(0xffffffffu, s1, 16));
        x = combine2<MAX>(mid ? k1 : k0, __shfl_xor_sync(0xffffffffu, mid ? k0 : k1, 8));
        o = 4;
    }
#pragma unroll
    for (; o > 0; o >>= 1) x = combine2<MAX>(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}

// Every lane receives all NV totals of warp_totals().
template <int NV, bool MAX>
__device__ __forceinline__ void warp_totals_all(const double (&v)[NV], int lane, double (&t)[NV]) {
    const double x = warp_totals<NV, MAX>(v, lane);
    if constexpr (NV == 1) {
        t[0] = x;
    } else {
#pragma unroll
        for (int k = 0; k < NV; ++k)
            t[k] = __shfl_sync(0xffffffffu, x, NV == 2 ? 16 * k : 16 * (k >> 1) + 8 * (k & 1));
    }
}

// First stage of every reduction: each warp's totals to smem[k * 32 + warp].
template <int NV, bool MAX>
__device__ __forceinline__ void warp_partials(const double (&v)[NV], double *smem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double x = warp_totals<NV, MAX>(v, lane);
    const int k = warp_value<NV>(lane);
    if (lane % kWarpValueLanes<NV> == 0 && k < NV) smem[k * 32 + warp] = x;
}

// All-reduce of NV <= 4 doubles over the block (sum, or max when MAX) with a
// fixed tree, so identical inputs give identical outputs; the result is valid
// in every thread.  smem holds >= 32 * NV doubles and may be reused right
// away by another reduction.
template <int NV, bool MAX>
__device__ __forceinline__ void block_allreduce(double (&v)[NV], double *smem) {
    __shared__ double s_res[4];
    const int lane = threadIdx.x & 31;
    const int nwarps = (blockDim.x + 31) >> 5;
    warp_partials<NV, MAX>(v, smem);
    __syncthreads();
    if (threadIdx.x < 32) {
        double w[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) w[k] = lane < nwarps ? smem[k * 32 + lane] : 0.0;
        const double x = warp_totals<NV, MAX>(w, lane);
        const int k = warp_value<NV>(lane);
        if (lane % kWarpValueLanes<NV> == 0 && k < NV) s_res[k] = x;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = s_res[q];
}

template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double *smem) { block_allreduce<NV, false>(v, smem); }
template <int NV>
__device__ __forceinline__ void block_max(double (&v)[NV], double *smem) { block_allreduce<NV, true>(v, smem); }

// Cluster barrier (release / acquire, every thread of every block of the
// cluster): 0.33 us for 2 to 16 blocks, against 1.0-1.13 us for the counter
// barrier below.
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();       // the aligned forms want the whole warp together
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Shared memory of the team's reductions and barriers: warp values, results,
// the mailbox that the other blocks of a cluster write to, and the barrier
// state.  One copy per kernel at an address that the compiler knows: state in
// registers would be spilled around the Krylov loop, and a spilled value
// comes back from L2 after every acquire (which empties L1).
struct ReduceBuffers {
    double warp[4 * 32], res[4], box[2 * 4 * 16];
    unsigned long long epoch;           // arrivals that complete the last barrier
    int ok, turn;
};
__device__ __forceinline__ ReduceBuffers &reduce_buffers() {
    __shared__ ReduceBuffers b;
    return b;
}
__device__ __forceinline__ void reduce_buffers_init() {
    if (threadIdx.x == 0) {
        ReduceBuffers &b = reduce_buffers();
        b.epoch = 0;
        b.turn = 0;
        b.ok = 1;
    }
    __syncthreads();
}

// Thread 0: arrive at the grid's barrier number epoch / G and wait for it.
__device__ __forceinline__ bool grid_arrive_wait(unsigned long long *count, int *error, unsigned long long epoch) {
    red_release_add_u64(count, 1ull);
    uint32_t spins = 0;
    while (ld_acquire_u64(count) < epoch) {
        if (++spins > kBarrierSpinLimit) {
            atomicCAS(error, 0, kStatusTimeout);
            return false;
        }
        if (spins > kTightSpins) __nanosleep(64);
    }
    return true;
}

// Grid-wide barrier for co-resident (cooperatively launched) blocks on a
// monotone arrival counter: barrier number k completes when the counter
// reaches k * gridDim.x, so nothing is reset and a block never waits on a
// generation flag.  The release add publishes this block's writes (bar.sync
// orders the other threads' writes before it); the acquire load orders
// everything after.  Returns false when the wait gave up; the caller must
// then leave the kernel.
__device__ __forceinline__ bool grid_barrier(const GridSync &gs) {
    ReduceBuffers &b = reduce_buffers();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned long long e = b.epoch + gridDim.x;
        b.epoch = e;
        b.ok = grid_arrive_wait(gs.count, gs.error, e) ? 1 : 0;
    }
    __syncthreads();
    return b.ok != 0;
}

// Reduction of NV <= 4 values over a team of G blocks (sum, or max when MAX)
// in one team barrier: warps reduce to shared memory; the block's values go
// to every block's mailbox through distributed shared memory (one cluster:
// warp k, value k) or to the partials (grid of co-resident blocks, 2 x 4 x G
// doubles: warp 0, whose lane 0 arrives with release and waits, bounded, with
// acquire); then warp 0 sums the blocks' values, lane-strided in block order
// and by a fixed shuffle tree, and calls fin(totals, writer), `writer` true
// on one lane.  What that lane stores to shared memory is visible to every
// thread of the block afterwards.  The order is the same in all three forms
// and fixed, so every block holds bit-identical results.  The mailbox and the
// partials are two regions used alternately: a block may write reduction
// j + 1 while a slower one still reads reduction j, never j + 2.  Returns
// false when a barrier wait gave up.
template <int NV, bool MAX, typename Fin>
__device__ __forceinline__ bool team_reduce_then(int G, int rank, bool cluster, double *partials,
                                                 const GridSync &gs, const double (&v)[NV], Fin fin) {
    ReduceBuffers &buf = reduce_buffers();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = (blockDim.x + 31) >> 5;
    warp_partials<NV, MAX>(v, buf.warp);
    __syncthreads();
    const int half = buf.turn & 1;
    if (cluster) {
        if (warp < NV) {
            double y = lane < nwarps ? buf.warp[warp * 32 + lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) y = combine2<MAX>(y, __shfl_xor_sync(0xffffffffu, y, o));
            if (lane < G) {
                const uint32_t local = (uint32_t)__cvta_generic_to_shared(buf.box + half * 64 + warp * 16 + rank);
                uint32_t remote;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(lane));
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote), "d"(y) : "memory");
            }
        }
        cluster_barrier();
    }
    if (warp == 0) {
        double w[NV], tot[NV];
        bool ok = true;
        if (cluster) {
#pragma unroll
            for (int k = 0; k < NV; ++k) w[k] = lane < G ? combine2<MAX>(0.0, buf.box[half * 64 + k * 16 + lane]) : 0.0;
        } else {
#pragma unroll
            for (int k = 0; k < NV; ++k) w[k] = lane < nwarps ? buf.warp[k * 32 + lane] : 0.0;
            if (G > 1) {
                double *p = partials + (size_t)half * 4 * G;
                const double x = warp_totals<NV, MAX>(w, lane);
                const int kv = warp_value<NV>(lane);
                if (lane % kWarpValueLanes<NV> == 0 && kv < NV) p[kv * G + rank] = x;
                __syncwarp();
                if (lane == 0) {
                    const unsigned long long e = buf.epoch + (unsigned)G;
                    buf.epoch = e;
                    ok = grid_arrive_wait(gs.count, gs.error, e);
                    buf.ok = ok ? 1 : 0;
                }
                ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
#pragma unroll
                for (int k = 0; k < NV; ++k) w[k] = 0.0;
                // five loads per value and lane in flight (160 blocks); with
                // the trip count left to the compiler its remainder loop took
                // one round trip per load, 4 us of every reduction
                for (int j0 = lane; j0 - lane < G; j0 += 160) {
#pragma unroll
                    for (int q = 0; q < 5; ++q) {
                        const int j = j0 + 32 * q;
#pragma unroll
                        for (int k = 0; k < NV; ++k) w[k] = combine2<MAX>(w[k], j < G ? __ldcg(p + k * G + j) : 0.0);
                    }
                }
            }
        }
        warp_totals_all<NV, MAX>(w, lane, tot);
        if (ok) fin(tot, lane == 0);
        if (lane == 0) buf.turn = buf.turn + 1;
    }
    __syncthreads();
    return buf.ok != 0;
}

}  // namespace ohm
