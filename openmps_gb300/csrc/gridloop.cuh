// gridloop.cuh - grid-wide sums and barriers of the single-launch solver loops.
//
// A conjugate-gradient iteration on these systems is a few microseconds of work between
// two dot products.  As separate kernels under a graph's WHILE node an iteration of the
// 1,850-row dam break cost 30 us, almost all of it kernel boundaries, ticket reductions
// and the node's own turnaround; in one launch it costs its memory round trips and the
// exchanges below.
//
// loop_reduce is a sum and a barrier at once.  Every block adds the same partial sums in the
// same order, so the totals are equal in all blocks, bit for bit, and the same run to run.
// Two forms (GB300, measured back to back with a one-value sum over 576 threads a block):
//   cluster  one cluster of up to 16 blocks: partial sums through distributed shared memory
//            and the hardware's cluster barrier (0.4-0.9 us for the exchange alone);
//   grid     a cooperative launch: partial sums through L2 and an arrival counter that one
//            thread per block polls (2.3 us for the exchange at 152 blocks on two dies; 152
//            threads per block polling the other blocks' slots took 4.8-5.5 us).
// GB300's FP64 pipe takes a warp-wide addition (or conversion) every 64 cycles per scheduler
// and answers after 64, so a five-level shuffle tree takes 605: the block's sum runs on four
// warps, one per scheduler, over the threads that hold values only, and what follows from the
// totals (divisions) on one thread.  (The sums in fixed point on the integer pipe, limbs added
// by redux.sync and correctly rounded, took 900 cycles a warp and were dropped.)
//
// The grid form's wait is bounded (LoopReduce::wait_clocks): a block whose wait runs out gets
// false and leaves its loop, and so do the others at the next exchange, where its arrival is
// missing.  At a loop's last exchange the others may pass: what a block reports then stands
// beside their result (CgScalars::timed_out).
#pragma once

#include "common.cuh"

namespace mpsgb {

constexpr int kLoopThreads = 512;  // one block per SM, 128 registers a thread
constexpr int kLoopMaxBlocks = 256;
constexpr int kLoopMaxValues = 3;
constexpr int kLoopCluster = 16;                     // blocks of the cluster form
constexpr long long kLoopWaitClocks = 4000000000LL;  // default bound of a wait, about two seconds
// global words of the grid form: the arrival counter (zeroed by clear_slots in a kernel
// before the loop), then two sets of partial sums used in turn (a set is written again two
// rounds later, when every block has arrived at the round between and so has read it)
constexpr int kLoopSlots = 16 + 2 * kLoopMaxValues * kLoopMaxBlocks;  // 8-byte words

// shared memory of loop_reduce
struct LoopReduce {
    double lanes[kLoopMaxValues][kLoopThreads];
    double cluster[2][kLoopMaxValues][kLoopCluster];
    double warps[kLoopMaxValues][4];
    double total[kLoopMaxValues];
    long long wait_clocks;  // bound of the grid form's wait, set and read by thread 0
};

struct LoopSync {
    double* slots;
    unsigned arrived;  // arrivals after the next round
    int round;         // 0, 1, 0, ...
};

// Blocks of the grid form on `sms` SMs: one each where the device launches cooperatively (all
// blocks of a launch must be resident at once), else a single one, which waits for nobody.
inline cudaError_t loop_grid_blocks(int dev, int sms, int* blocks) {
    int coop = 0;
    const cudaError_t e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    *blocks = !coop ? 1 : sms < kLoopMaxBlocks ? sms : kLoopMaxBlocks;
    return e;
}

// Readies the slots for the loop kernel launched after this one (any grid).
__device__ __forceinline__ void clear_slots(double* slots) {
    if (slots && blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<unsigned*>(slots) = 0u;
}

// Before the first exchange of the cluster form: every block of the cluster has started.
__device__ __forceinline__ void loop_cluster_start() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ double loop_warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Grid-wide sums of NV values (NV = 0: a barrier), then then(totals) in warp 0 alone,
// whose thread 0 leaves what the block needs in shared memory.  Called by all threads of all blocks
// (at least 128 threads a block); only the first `active` threads of this block hold values.
// What the grid's threads wrote before the call is visible after it.
template <bool kCluster, int NV, class Then>
__device__ __forceinline__ bool loop_reduce(LoopSync& ls, LoopReduce& sh, const double* v, int active, Then then) {
    const int t = static_cast<int>(threadIdx.x), w = t >> 5, lane = t & 31;
    const int G = static_cast<int>(gridDim.x);
    const int round = ls.round;
    ls.round ^= 1;
    double* slot = ls.slots + 16 + round * kLoopMaxValues * kLoopMaxBlocks;
    if (NV > 0) {
        if (t < active) {
#pragma unroll
            for (int i = 0; i < NV; i++) sh.lanes[i][t] = v[i];
        }
        __syncthreads();
        if (t < 128) {
            double s[NV > 0 ? NV : 1];
#pragma unroll
            for (int i = 0; i < NV; i++) s[i] = t < active ? sh.lanes[i][t] : 0.0;
            for (int k = t + 128; k < active; k += 128) {
#pragma unroll
                for (int i = 0; i < NV; i++) s[i] += sh.lanes[i][k];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                for (int i = 0; i < NV; i++) s[i] += __shfl_down_sync(0xffffffffu, s[i], o);
            }
            if (lane == 0) {
#pragma unroll
                for (int i = 0; i < NV; i++) sh.warps[i][w] = s[i];
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
        }
    } else if (!kCluster) {
        __syncthreads();
    }
    double mine = 0.0;  // warp i: this block's sum of value i
    if (NV > 0 && w < NV) mine = (sh.warps[w][0] + sh.warps[w][1]) + (sh.warps[w][2] + sh.warps[w][3]);
    if constexpr (kCluster) {
        if (NV > 0 && w < NV && lane < G) {  // this block's sums to every block of the cluster
            uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(&sh.cluster[round][w][blockIdx.x]));
            asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(lane));
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(mine) : "memory");
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        if (NV > 0 && w < NV && lane == 0) __stcg(slot + w * kLoopMaxBlocks + blockIdx.x, mine);
        if (NV > 1 && w < NV) asm volatile("bar.sync 2, %0;" ::"n"(32 * (NV > 0 ? NV : 1)) : "memory");
        int late = 0;
        if (t == 0) {
            unsigned* count = reinterpret_cast<unsigned*>(ls.slots);
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
            const long long t0 = clock64();
            unsigned seen;
            while (true) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
                if (static_cast<int>(seen - ls.arrived) >= 0) break;
                if (clock64() - t0 >= sh.wait_clocks) {
                    late = 1;
                    break;
                }
            }
        }
        ls.arrived += static_cast<unsigned>(G);
        if (__syncthreads_or(late)) return false;
    }
    if (NV > 0) {
        if (w < NV) {  // one warp per value
            double s;
            if constexpr (kCluster) {
                s = lane < G ? sh.cluster[round][w][lane] : 0.0;
#pragma unroll
                for (int o = kLoopCluster / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            } else {
                constexpr int kPer = kLoopMaxBlocks / 32;
                double x[kPer];
#pragma unroll
                for (int k = 0; k < kPer; k++)
                    x[k] = lane + 32 * k < G ? __ldcg(slot + w * kLoopMaxBlocks + lane + 32 * k) : 0.0;
                // pairs of blocks that exist only: each addition takes the pipe 64 cycles
#pragma unroll
                for (int d = 1; d < kPer; d *= 2) {
#pragma unroll
                    for (int k = 0; k + d < kPer; k += 2 * d)
                        if (32 * (k + d) < G) x[k] += x[k + d];
                }
                s = loop_warp_sum(x[0]);
            }
            if (lane == 0) sh.total[w] = s;
            if (NV > 1) asm volatile("bar.sync 2, %0;" ::"n"(32 * (NV > 0 ? NV : 1)) : "memory");
            if (NV == 1) __syncwarp();
            if (w == 0) then(sh.total);
        }
        __syncthreads();
    }
    return true;
}

}  // namespace mpsgb
