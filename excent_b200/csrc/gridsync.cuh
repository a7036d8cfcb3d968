// gridsync.cuh -- a barrier over every block of a cooperative launch.
//
// The persistent solve kernels run all their passes in one launch and order
// the phases of a pass with this barrier. Measured on a B200: 1.3 us for 148
// blocks of up to 1024 threads, 1.85 us for 444 and 3.1 us for 888 of 256,
// against about 10 us for each kernel node of the graph loops it replaces;
// hence one large block per SM. The wait is bounded: past its limit it marks
// the barrier failed, every block leaves, and the host reports an error.
#pragma once
#include <cuda_runtime.h>

namespace excent {

struct GridBar {
    unsigned arrived;   // blocks arrived, over the whole launch
    unsigned failed;    // a wait gave up
};
// Polls take about half a microsecond: the limit is over half a minute of waiting in one phase.
static constexpr unsigned GRID_SPIN_LIMIT = 1u << 26;

// Wait until every block of the launch has arrived as often as this one.
// `epoch` starts at 0 in every thread and belongs to the barrier. Memory
// written before the barrier by any thread is visible after it to all (the
// acquire also drops stale L1 lines). False: a wait gave up; leave the kernel.
__device__ __forceinline__ bool grid_sync(GridBar* b, unsigned& epoch) {
    __shared__ int s_ok;
    epoch += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        // release: what the block's threads wrote before (ordered by the block barrier) comes first
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&b->arrived) : "memory");
        int ok = 0;
        for (unsigned it = 0; it < GRID_SPIN_LIMIT; it++) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&b->arrived) : "memory");
            if ((int)(v - epoch) >= 0) { ok = 1; break; }
            if ((it & 1023u) == 1023u && *(volatile unsigned*)&b->failed) break;
        }
        if (!ok) atomicExch(&b->failed, 1u);
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Launch `kernel` as a cooperative launch; `bar` is zeroed first, on the
// stream (null: it is zero already).
template <typename Args>
static inline cudaError_t launch_grid(void (*kernel)(Args), int blocks, int threads, size_t smem, Args& a, GridBar* bar,
                                      cudaStream_t st) {
    if (bar) {
        const cudaError_t rc = cudaMemsetAsync(bar, 0, sizeof(GridBar), st);
        if (rc != cudaSuccess) return rc;
    }
    void* args[] = {&a};
    return cudaLaunchCooperativeKernel((const void*)kernel, dim3((unsigned)blocks), dim3((unsigned)threads), args, smem,
                                       st);
}

}  // namespace excent
