// gridsum.cuh -- grid-wide sums that are also grid barriers, for persistent
// kernels whose phases are a few microseconds long.
//
// A barrier is an arrival counter: one thread of every block adds 1 with
// release order and polls the counter with acquire order until all have (1.25
// us for 148 blocks, as cooperative_groups' grid.sync; 0.5 us of it is one
// trip to L2 and back).  A sum adds one coalesced read of the blocks' partials
// (0.4 us), where grid.sync with a shared-memory fold by every block of 592
// partials took about 4 us.  Polling the partials themselves, each with an
// epoch beside it, needs no counter but took 4.2 us at 148 blocks: strong
// loads of many words are served one by one.
//
// Partials alternate between two sets, so a block that runs ahead writes the
// other set while the slow ones still read this one (it cannot pass the next
// sum before they arrive).  The counter runs on over the launches that share
// it: a launch starts from the epoch that the last one left in memory, so
// every launch must take grid_begin, at least one sum or barrier, and
// grid_end.
//
// The blocks must be co-resident (cooperative launch).  Waits are bounded:
// after SPIN_LIMIT polls the block sets *err and goes on, so a launch always
// ends and the host reports the error.
#pragma once

#include "device.cuh"

namespace pdhcg {

constexpr int SPIN_LIMIT = 1 << 22;

struct GridSlots {
    double *part;               // [2][stride] partials: value k of block b at k * blocks + b
    int stride;
    unsigned long long *state;  // [0] arrivals, [1] epoch of the last barrier (both start at 0)
    int *err;                   // set when a wait ran out
    unsigned long long epoch;   // device side: barriers taken so far
};

__device__ __forceinline__ void grid_begin(GridSlots &S) { S.epoch = S.state[1]; }

// every block has taken its last barrier of this launch
__device__ __forceinline__ void grid_end(const GridSlots &S)
{
    if (blockIdx.x == 0 && threadIdx.x == 0)
        S.state[1] = S.epoch;
}

// one thread per block, after a block barrier: arrive and wait for the others
__device__ __forceinline__ void grid_arrive_wait(const GridSlots &S)
{
    const unsigned long long want = (S.epoch + 1) * gridDim.x;
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(S.state) : "memory");
    for (int spin = 0;; ++spin) {
        unsigned long long have;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(have) : "l"(S.state) : "memory");
        if (have >= want)
            return;
        // past the limit, or another wait already was: give up for good
        if (spin >= SPIN_LIMIT || ((spin & 1023) == 1023 && *(volatile int *)S.err)) {
            *S.err = 1;
            return;
        }
    }
}

// Barrier over the grid: what any thread wrote to global memory before it is
// visible after it to L2-level loads (__ldcg) and to plain loads.
__device__ __forceinline__ void grid_barrier(GridSlots &S)
{
    __syncthreads();
    if (gridDim.x > 1) {
        if (threadIdx.x == 0)
            grid_arrive_wait(S);
        __syncthreads();
    }
    ++S.epoch;
}

// this launch's partials of value k
__device__ __forceinline__ double *grid_part(const GridSlots &S, int k)
{
    return S.part + (S.epoch & 1) * (size_t)S.stride + (size_t)k * gridDim.x;
}

// one warp: sum, or maximum of non-negative values, of p[0, blocks) in block
// order over the lanes' strides
__device__ __forceinline__ double grid_part_fold(const double *p, int lane, bool mx)
{
    const int nb = gridDim.x;
    double a = 0.0;
#pragma unroll 5
    for (int b = lane; b < nb; b += 32) {
        const double v = __ldcg(p + b);
        a = mx ? fmax(a, v) : a + v;
    }
    return mx ? warp_max(a) : warp_sum(a);
}

// K values per thread (bit k of is_max: maximum of non-negative values, else
// sum) folded over the grid, warp by warp and block by block in a fixed
// order; also a barrier, as grid_barrier.  NW >= K warps per block; sh: K *
// (NW + 1) doubles.
template <int K, int NW>
__device__ __forceinline__ void grid_fold(double (&v)[K], unsigned is_max, GridSlots &S, double *sh)
{
    static_assert(K <= NW, "a warp per value");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double w = (is_max >> k) & 1u ? warp_max(v[k]) : warp_sum(v[k]);
        if (lane == 0)
            sh[k * NW + warp] = w;
    }
    __syncthreads();
    const bool mx = warp < K && ((is_max >> warp) & 1u);
    double a = 0.0;
    if (warp < K) {
        a = lane < NW ? sh[warp * NW + lane] : 0.0;
        a = mx ? warp_max(a) : warp_sum(a);
    }
    if (gridDim.x > 1) {
        if (warp < K && lane == 0)
            __stcg(grid_part(S, warp) + blockIdx.x, a);
        __syncthreads();
        if (threadIdx.x == 0)
            grid_arrive_wait(S);
        __syncthreads();
        if (warp < K)
            a = grid_part_fold(grid_part(S, warp), lane, mx);
    }
    if (warp < K && lane == 0)
        sh[K * NW + warp] = a;
    ++S.epoch;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k)
        v[k] = sh[K * NW + k];
    __syncthreads();
}

// One value per thread, summed over the grid; also a barrier.  NW warps per
// block; sh: NW + 1 doubles.
template <int NW>
__device__ __forceinline__ double grid_sum(double v, GridSlots &S, double *sh)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_sum(v);
    if (lane == 0)
        sh[warp] = v;
    __syncthreads();
    if (warp == 0) {
        double a = lane < NW ? sh[lane] : 0.0;
        a = warp_sum(a);
        if (gridDim.x > 1) {
            double *p = grid_part(S, 0);
            if (lane == 0) {
                __stcg(p + blockIdx.x, a);
                grid_arrive_wait(S);
            }
            __syncwarp();
            a = grid_part_fold(p, lane, false);
        }
        if (lane == 0)
            sh[NW] = a;
    }
    ++S.epoch;
    __syncthreads();
    return sh[NW];
}

} // namespace pdhcg
