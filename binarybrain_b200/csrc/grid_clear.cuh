// Clearing a buffer inside the kernel that afterwards adds to it, instead of by a memset in front: for kernels of a few microseconds the
// memset costs about 3 us of the GPU's time (its own, and the overlap of launches that it breaks) and 2 us of the host's.
//
// The buffer is cut into slices of kClearSlice floats.  Every CTA, when it starts, claims slices until none is left, so that a slice is
// always in the hands of a CTA that runs, whichever CTAs the GPU has room for; before its first addition a CTA waits until all slices are
// cleared.  That wait therefore ends without any CTA that has not started; it is bounded all the same, and a CTA whose wait has run out
// records the fault and makes its gradients NaN.  The last CTA to pass the wait resets the counters for the next kernel of the stream, which
// touches them after its grid_dependency() only.
#pragma once

#include "common.cuh"
#include "async_copy.cuh"

namespace bb200 {

struct GridClear {
    float *dst;                 // nullptr: the launcher has cleared the buffer
    unsigned *counters;         // [3]: slices claimed, slices cleared, CTAs done with waiting; zero before and after the kernel
    int *fault;
    size_t floats;
};

constexpr int kClearSlice = 8192;

// Fills in `c`, or clears the buffer by a memset where the stream has no counters; returns a status.
inline int grid_clear_setup(GridClear &c, float *dst, size_t floats, cudaStream_t st)
{
    c = GridClear{};
    c.counters = floats > 0 && floats < ((size_t)1 << 40) ? stream_counters(st) : nullptr;
    c.fault = fault_word();
    if (c.counters == nullptr || c.fault == nullptr) {
        BB200_CUDA(cudaMemsetAsync(dst, 0, sizeof(float) * floats, st));
        return BBCU_OK;
    }
    c.dst = dst;
    c.floats = floats;
    return BBCU_OK;
}

// All threads of the CTA.
__device__ __forceinline__ void grid_clear_slices(const GridClear &c)
{
    __shared__ unsigned s_claim;
    if (c.dst == nullptr) return;
    const unsigned slices = (unsigned)((c.floats + kClearSlice - 1) / kClearSlice);
    const bool aligned = (reinterpret_cast<uintptr_t>(c.dst) & 15) == 0;
    for (;;) {
        if (threadIdx.x == 0) s_claim = atomicAdd(c.counters, 1u);
        __syncthreads();
        const unsigned k = s_claim;
        if (k >= slices) return;                              // (every thread leaves here, after the same barrier)
        const size_t begin = (size_t)k * kClearSlice;
        const int n = (int)(c.floats - begin < (size_t)kClearSlice ? c.floats - begin : (size_t)kClearSlice);
        const int quads = aligned ? n / 4 : 0;
        float *p = c.dst + begin;
        for (int i = threadIdx.x; i < quads; i += blockDim.x) reinterpret_cast<float4 *>(p)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int i = 4 * quads + threadIdx.x; i < n; i += blockDim.x) p[i] = 0.0f;
        __threadfence();
        __syncthreads();                                      // the slice is written, and s_claim read, by all
        if (threadIdx.x == 0) atomicAdd(c.counters + 1, 1u);
    }
}

// One thread of the CTA, once; a barrier of the CTA has to follow before the first addition.  Where the buffer is not cleared after a second or
// so, what follows is no gradient: the 64 table gradients of the CTA's node and the `n` floats of `factors`, shared memory that every addition
// to the buffer is multiplied by, become NaN.  (Leaving the kernel instead cost the ordinary call 1 us: the branch, and loads held back by it.)
__device__ __forceinline__ void grid_clear_wait(const GridClear &c, float *dW_row, float *factors, int n)
{
    if (c.dst == nullptr) return;
    const unsigned slices = (unsigned)((c.floats + kClearSlice - 1) / kClearSlice);
    unsigned done = 0;
    int tries = 0;
    for (; tries < (1 << 20); ++tries) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(done) : "l"(c.counters + 1) : "memory");
        if (done >= slices) break;
        __nanosleep(64);
    }
    if (done < slices) {
        atomicCAS(c.fault, 0, kFaultBarrierTimeout);
        for (int i = 0; i < 64; ++i) dW_row[i] = __int_as_float(0x7fffffff);
        for (int i = 0; i < n; ++i) factors[i] = __int_as_float(0x7fffffff);
    }
    __threadfence();
    if (atomicAdd(c.counters + 2, 1u) == gridDim.x - 1) {     // nobody looks at the counters any more
        c.counters[0] = 0u;
        c.counters[1] = 0u;
        c.counters[2] = 0u;
    }
}

}   // namespace bb200
