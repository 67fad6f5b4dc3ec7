/*
 * The processing order of a per-frame batch: the frames with the weakest LLRs
 * first, so that those which need many iterations do not start last and leave
 * the device to a few of them.  Any order gives the same results.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "ldpc_device.h"

namespace drxg {

namespace {

constexpr int kOrderThreads = 512;
constexpr int kOrderBins = 1024;

/* A warp takes a frame: its key is the mean |LLR| of every fourth 512-byte
 * piece (aligned 16-byte loads inside the row), in eighths.  The last block to
 * finish sorts the keys by counting.  Bound by the loads' latency and the sort's
 * (1024 normal frames about 10 us, 4096 about 15). */
__global__ void __launch_bounds__(kOrderThreads) k_order(const int8_t* __restrict__ llr, size_t stride, int N, int n,
                                                         int* __restrict__ keys, int32_t* __restrict__ order,
                                                         unsigned* ticket)
{
    __shared__ int hist[kOrderBins];
    __shared__ int wsum[kOrderThreads / 32];
    __shared__ bool last;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nwarps = kOrderThreads / 32;
    for (int f = blockIdx.x * nwarps + warp; f < n; f += gridDim.x * nwarps) {
        const int8_t* row = llr + (size_t)f * stride;
        const int skip = (int)((16 - ((uintptr_t)row & 15)) & 15);
        const uint4* v = (const uint4*)(row + skip);
        const int nv = (N - skip) / 16;
        unsigned sum = 0;
        int cnt = 0;
#pragma unroll 8
        for (int i = lane; i < nv; i += 128) {
            const uint4 w = __ldg(v + i);
            sum = __dp4a(__vabs4(w.x), 0x01010101u, sum);
            sum = __dp4a(__vabs4(w.y), 0x01010101u, sum);
            sum = __dp4a(__vabs4(w.z), 0x01010101u, sum);
            sum = __dp4a(__vabs4(w.w), 0x01010101u, sum);
            cnt += 16;
        }
        sum = __reduce_add_sync(~0u, sum);
        cnt = __reduce_add_sync(~0u, cnt);
        if (lane == 0)
            keys[f] = min(kOrderBins - 1, (int)(sum * 8 / max(cnt, 1)));
    }
    __syncthreads();
    if (t == 0) {
        __threadfence();
        last = atomicAdd(ticket, 1) == gridDim.x - 1;
    }
    for (int i = t; i < kOrderBins; i += kOrderThreads)
        hist[i] = 0;
    __syncthreads();
    if (!last)
        return;
    __threadfence();
#pragma unroll 8
    for (int f = t; f < n; f += kOrderThreads)
        atomicAdd(&hist[__ldcg(keys + f)], 1);
    __syncthreads();
    /* exclusive prefix sums of the bins, two per thread */
    static_assert(kOrderBins == 2 * kOrderThreads, "two bins per thread");
    const int a = hist[2 * t], b = hist[2 * t + 1];
    int s = a + b;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const int o = __shfl_up_sync(~0u, s, d);
        if (lane >= d)
            s += o;
    }
    if (lane == 31)
        wsum[warp] = s;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; w++)
        before += wsum[w];
    hist[2 * t] = before + s - a - b;
    hist[2 * t + 1] = before + s - b;
    __syncthreads();
#pragma unroll 8
    for (int f = t; f < n; f += kOrderThreads)
        order[atomicAdd(&hist[__ldcg(keys + f)], 1)] = f;
}

}  // namespace

cudaError_t launch_order(const int8_t* llr, size_t stride, int N, int n, void* scratch, unsigned* ticket, int sms,
                         cudaStream_t s)
{
    int32_t* order = (int32_t*)scratch;
    const int blocks = std::min((n + kOrderThreads / 32 - 1) / (kOrderThreads / 32), 2 * sms);
    k_order<<<blocks, kOrderThreads, 0, s>>>(llr, stride, N, n, order + kOrderFrames, order, ticket);
    return cudaGetLastError();
}

}  // namespace drxg
