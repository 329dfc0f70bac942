// fem_reduce.cuh -- block sums of FP64 values.
//
// A warp instruction of the FP64 pipe takes 16 cycles of the SM on GB300, so the
// usual tree (five shuffle steps in every warp, then in one) costs a block of 8
// warps 45 of them per value: for short vectors more than the work that is
// summed.  Here the threads leave their values in shared memory and one warp per
// value adds them, 256 / 32 per lane and then five steps: 12 instructions.
#pragma once

namespace fem {

__device__ __forceinline__ double warp_total(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// out[k] += sum over the block of v[k] (one atomic each).  NT = blockDim.x, a
// multiple of 32 * EVERY; only threads with threadIdx.x % EVERY == 0 hold values.
// The block may call it again (another instance) after a barrier of its own.
template <int NT, int EVERY, int NV>
__device__ __forceinline__ void block_sum_add(const double (&v)[NV], double* const (&out)[NV]) {
    constexpr int N = NT / EVERY;
    static_assert(N % 32 == 0 && NV <= NT / 32, "whole warps");
    __shared__ double red[NV][N];
    if (threadIdx.x % EVERY == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) red[k][threadIdx.x / EVERY] = v[k];
    }
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (w >= NV) return;
    double s = red[w][lane];
#pragma unroll
    for (int i = 1; i < N / 32; ++i) s += red[w][lane + 32 * i];
    s = warp_total(s);
    double* o = out[0];
#pragma unroll
    for (int k = 1; k < NV; ++k)
        if (w == k) o = out[k];
    if (lane == 0) atomicAdd(o, s);
}

// A sum over the grid is kept in parts: an FP64 atomic of every block to one address
// takes 10 ns.  part_of: where the block adds; parts_total: the total, by a whole warp.
constexpr int kSumParts = 8;
__device__ __forceinline__ double* part_of(double* sum) { return sum + blockIdx.x % kSumParts; }
__device__ __forceinline__ double parts_total(const double* sum) {
    double t = sum[threadIdx.x % kSumParts];
#pragma unroll
    for (int o = kSumParts / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

}  // namespace fem
