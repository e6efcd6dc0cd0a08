// Processing order of a paired batch on the device: a counting sort of the
// pairs by the shape of their DP (rows = the longer side, columns = the
// shorter), the largest first, so that the lanes of a warp run loops of
// near-equal length.  64 classes a side: steps of 8 points up to 256, then
// eighths of an octave (lengths from 3,584 share the last); pairs of a class in
// any order.
//
// Bound by launches and by the latency of its atomics, not by its 12 bytes a
// pair.  A call with 100,000 pairs of 20..200 points and this order takes 742 us
// where one with a 31-bit radix sort and its key passes took 835.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace tsm {

constexpr int kOrderClasses = 64 * 64;
constexpr int kOrderThreads = 1024;
constexpr int kOrderInts = 2 * kOrderClasses;  // workspace: class counts, class cursors

__device__ __forceinline__ int side_class(int n) {
    if (n <= 256) return max(n, 0) + 7 >> 3;  // 0 .. 32
    const int e = 31 - __clz(n);              // 8 ..
    return min(63, 33 + (e - 8) * 8 + ((n >> (e - 3)) & 7));
}
// Class 0: the largest pairs.
__device__ __forceinline__ int order_class(int na, int nb) {
    return kOrderClasses - 1 - (side_class(max(na, nb)) * 64 + side_class(min(na, nb)));
}

__global__ void __launch_bounds__(kOrderThreads) order_count(const int32_t* __restrict__ len_a,
                                                             const int32_t* __restrict__ len_b, int64_t n,
                                                             int* __restrict__ ws) {
    __shared__ int hist[kOrderClasses];
    for (int c = threadIdx.x; c < kOrderClasses; c += kOrderThreads) hist[c] = 0;
    __syncthreads();
    for (int64_t k = (int64_t)blockIdx.x * kOrderThreads + threadIdx.x; k < n; k += (int64_t)gridDim.x * kOrderThreads)
        atomicAdd(&hist[order_class(len_a[k], len_b[k])], 1);
    __syncthreads();
    for (int c = threadIdx.x; c < kOrderClasses; c += kOrderThreads)
        if (hist[c]) atomicAdd(ws + c, hist[c]);
}

// The same grid as order_count: each CTA counts its pairs again, takes a range
// of every class it has and writes its pairs there.
__global__ void __launch_bounds__(kOrderThreads) order_scatter(const int32_t* __restrict__ len_a,
                                                               const int32_t* __restrict__ len_b, int64_t n,
                                                               int* __restrict__ ws, int32_t* __restrict__ order) {
    __shared__ int hist[kOrderClasses];
    __shared__ int base[kOrderClasses];
    __shared__ int tot[kOrderThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int PER = kOrderClasses / kOrderThreads;  // classes per thread of the scan
    int v[PER], sum = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        v[i] = sum;
        sum += ws[threadIdx.x * PER + i];
    }
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) tot[warp] = x;
    for (int c = threadIdx.x; c < kOrderClasses; c += kOrderThreads) hist[c] = 0;
    __syncthreads();
    int before = x - sum;
    for (int w = 0; w < warp; ++w) before += tot[w];
#pragma unroll
    for (int i = 0; i < PER; ++i) base[threadIdx.x * PER + i] = before + v[i];
    for (int64_t k = (int64_t)blockIdx.x * kOrderThreads + threadIdx.x; k < n; k += (int64_t)gridDim.x * kOrderThreads)
        atomicAdd(&hist[order_class(len_a[k], len_b[k])], 1);
    __syncthreads();
    for (int c = threadIdx.x; c < kOrderClasses; c += kOrderThreads)
        if (hist[c]) base[c] += atomicAdd(ws + kOrderClasses + c, hist[c]);
    __syncthreads();
    for (int64_t k = (int64_t)blockIdx.x * kOrderThreads + threadIdx.x; k < n; k += (int64_t)gridDim.x * kOrderThreads)
        order[atomicAdd(&base[order_class(len_a[k], len_b[k])], 1)] = (int32_t)k;
}

}  // namespace tsm
