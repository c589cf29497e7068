// counts.cuh -- event counters of the collision kernels.
#pragma once

#include <cuda_runtime.h>

namespace pgd {

using u64 = unsigned long long;

// Adds the threads' counts to counts[at[k]], one atomic per block and count
// (one per thread at the same address is 1 to 2 ns each, one after the other:
// 90 us of a swarm step's MCC).  Every thread of the block takes part.
template <int N>
__device__ __forceinline__ void add_counts(u64* counts, const int (&at)[N], const u64 (&v)[N]) {
    __shared__ u64 sum[N];
    if (threadIdx.x < N) sum[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k) {
        u64 x = v[k];
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
        if ((threadIdx.x & 31) == 0 && x) atomicAdd(&sum[k], x);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k)
        if (threadIdx.x == k && sum[k]) atomicAdd(counts + at[k], sum[k]);
}

}  // namespace pgd
