// Barrier of the kernels that keep a whole level resident: over a cluster by the
// hardware, or over a cooperative grid by a counter in global memory whose wait
// is bounded.
#pragma once

namespace p2 {

constexpr unsigned kResSpin = 1u << 22;  // polls of the grid barrier before it gives up (seconds)

struct GridBarrier {
    unsigned *count;  // [0] arrivals, [1] blocks done; both 0 between launches
    double *error;    // set to 1 when a wait ran out
};

// Barrier over the cluster or the whole grid; false when the wait ran out.
template <bool kCluster>
__device__ __forceinline__ bool res_sync(GridBarrier B, unsigned &target, bool *ok)
{
    if (kCluster) {
        asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
        return true;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        target += gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(B.count) : "memory");
        unsigned v = 0, spins = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(B.count) : "memory");
        } while ((int)(v - target) < 0 && ++spins < kResSpin);
        *ok = (int)(v - target) >= 0;
        if (!*ok) *B.error = 1.0;
    }
    __syncthreads();
    return *ok;
}

// At the end of a grid's kernel: the last block to leave clears the counters for the next launch.
__device__ __forceinline__ void res_leave(GridBarrier B)
{
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(B.count + 1, 1u) == gridDim.x - 1) {
        B.count[0] = 0;
        B.count[1] = 0;
    }
}

}  // namespace p2
