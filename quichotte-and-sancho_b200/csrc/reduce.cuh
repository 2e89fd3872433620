// reduce.cuh -- sums over many blocks finished by the block that arrives last: one launch, and the
// partial sums added in a fixed order (the result does not depend on which block that is).
#pragma once
#include "qs_common.cuh"

namespace qs {

// True in every thread of the last of `total` blocks to call this with the counter (zero before
// the launch, zero again after it); what the blocks wrote before their call is then visible.
__device__ __forceinline__ bool last_block(int *cnt, int total) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(cnt, 1) == total - 1;
        if (last) *cnt = 0;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// out[j] = op_b part[b stride + j] for j < nv <= blockDim.x, over nb partials, by the whole block:
// groups of lanes take every blockDim / (nv rounded up to a power of two)-th partial, and one
// thread per value adds the groups' sums. max_first: the maximum for j = 0.
__device__ __forceinline__ void part_reduce(const double *part, int nb, int stride, int nv, bool max_first, double *sh,
                                            double *out) {
    int p = 1;
    while (p < nv) p *= 2;
    const int j = threadIdx.x & (p - 1), grp = threadIdx.x / p, ng = blockDim.x / p;
    const bool mx = max_first && j == 0;
    double s = 0.0;
    if (j < nv) {
#pragma unroll 8
        for (int b = grp; b < nb; b += ng) {
            const double v = __ldcg(part + (int64_t)b * stride + j);
            s = mx ? fmax(s, v) : s + v;
        }
    }
    sh[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x < nv) {
        s = sh[j];
        for (int q = 1; q < ng; q++) s = mx ? fmax(s, sh[q * p + j]) : s + sh[q * p + j];
        out[j] = s;
    }
}

}  // namespace qs
