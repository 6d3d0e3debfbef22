// Barrier over the blocks of one cooperative launch (all resident at once), for the kernels that run
// several steps in one launch.
#pragma once
#include <algorithm>
#include <mutex>

#include "wg_internal.h"

namespace wg {

// polls of a waiting block before it gives up (each a trip to L2: a few seconds; a phase of a step
// takes well under a millisecond)
constexpr int kBarrierPolls = 1 << 22;
constexpr int kErrBarrier = 105;

__device__ __forceinline__ unsigned ldAcquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int flagNow(const int* f) { return *(const volatile int*)f; }

// Every thread of every block calls it; counter starts at zero. False when the wait ran out (FL_ERR is
// then kErrBarrier): the caller returns. `ok` is a shared word of the block. What any thread wrote before
// is visible to every thread after it.
__device__ __forceinline__ bool gridBarrier(unsigned* counter, int* dFlags, int* ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned n = gridDim.x, mine = atomicAdd(counter, 1u);
        const unsigned target = (mine / n + 1u) * n;
        int good = 1;
        for (int q = 0; ldAcquire(counter) < target; q++)
            if (q >= kBarrierPolls || flagNow(dFlags + FL_ERR) == kErrBarrier) {
                atomicCAS(dFlags + FL_ERR, 0, kErrBarrier);
                good = 0;
                break;
            }
        __threadfence();
        *ok = good;
    }
    __syncthreads();
    return *ok != 0;
}
__device__ __forceinline__ unsigned long long nowNs() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// streaming multiprocessors of the current device
static int smCount() {
    static std::mutex mu;
    static int n[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    std::lock_guard<std::mutex> lk(mu);
    if (!n[dev] && (cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n[dev] < 1)) n[dev] = 1;
    return n[dev];
}

// blocks that a launch of several steps over so many items can use: one on each SM, a warp for 32 items
static int stepsBlocks(int64_t items) { return (int)std::min<int64_t>(std::max<int64_t>((items + 31) / 32, 1), smCount()); }

// Whether kernel f can be launched with a block on every SM at once.
static bool stepsFit(const void* f, int threads, size_t shared) {
    int most = 0;
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&most, f, threads, shared) != cudaSuccess || most < 1) {
        cudaGetLastError();
        return false;
    }
    return true;
}
}  // namespace wg
