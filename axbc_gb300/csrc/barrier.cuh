// The grid barrier of the persistent (cooperative) kernels.
#pragma once

#include "common.cuh"

// Wait budget of one barrier in SM clock cycles (about 4 s at 2 GHz): a wait
// that runs out records its site and every block returns; the host reports
// AXBC_ERR_TIMEOUT.
#define AXBC_BAR_BUDGET (1ll << 33)

__device__ __forceinline__ unsigned vload_u(const unsigned *p) { return *(const volatile unsigned *)p; }
__device__ __forceinline__ int vload_i(const int *p) { return *(const volatile int *)p; }

// All blocks of the cooperative grid meet here; `epoch` counts the launch's
// barriers, the same in every block.  Thread 0 of each block fences, adds one to
// the arrival count and waits: without a lead until the count reaches the
// barrier's total, with one until the last block to arrive has run lead() with
// its first warp and says so (gen).  The fences before arriving and after the
// wait make the block's later loads see what every block wrote before.  A wait
// polls without sleeping at first (a barrier of 152 blocks took 3.1 us with a
// sleep in every poll and a generation word to be flipped for each).  Returns
// false when this wait, or an earlier one of any block, ran out of its budget.
struct NoLead {
    __device__ void operator()() const {}
};
template <class F> struct HasLead {
    static constexpr bool yes = true;
};
template <> struct HasLead<NoLead> {
    static constexpr bool yes = false;
};
template <class F>
__device__ __forceinline__ bool grid_barrier(GridSync *gs, long long budget, int site, unsigned &epoch, const F &lead)
{
    __shared__ int s_role;  // 1 leader, 0 released, -1 failed
    const unsigned mine = ++epoch, total = mine * gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned arrived = atomicAdd(&gs->count, 1u) + 1;
        int role = HasLead<F>::yes && arrived == total ? 1 : 0;
        if (role == 0 && arrived != total) {
            const long long t0 = clock64();
            for (unsigned polls = 1;; polls++) {
                if (HasLead<F>::yes ? (int)(vload_u(&gs->gen) - mine) >= 0 : (int)(vload_u(&gs->count) - total) >= 0)
                    break;
                if (polls % 32) continue;
                if (vload_i(&gs->err)) {
                    role = -1;
                    break;
                }
                if (clock64() - t0 > budget) {
                    atomicCAS(&gs->err, 0, site);
                    role = -1;
                    break;
                }
                if (polls >= 1024) __nanosleep(64);
            }
        }
        __threadfence();
        s_role = role;
    }
    __syncthreads();
    const int role = s_role;
    if (HasLead<F>::yes && role == 1) {
        if (threadIdx.x < 32) lead();
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicExch(&gs->gen, mine);
        }
    }
    return role >= 0;
}
