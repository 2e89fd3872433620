// noalloc.cu -- qs_invert_batched_noalloc: the batched Dyson inversion for callers that
// cannot allocate GPU memory.
//
// Who needs it: a caller whose device memory is all handed out by someone else, e.g. a
// solver embedded in a larger GPU application that owns a fixed memory pool or arena and
// forbids allocations behind its back, or a latency-critical loop that cannot afford the
// device-wide synchronisation cudaMalloc/cudaFree may cause. Such a caller already holds
// its matrices and outputs in device memory and only needs the inversion itself.
//
// The elimination runs in shared memory (small orders or batches) or in the caller's matrices
// themselves, so the call needs no workspace at all: it allocates nothing, keeps nothing between
// calls, and calls on different matrices may overlap on any streams and threads.
#include <cstdio>

#include "qs_common.cuh"

constexpr int QS_NOALLOC_MAX_N = 512;  // the kernels' limit

extern "C" int qs_invert_batched_noalloc(int N, int batch, double *A, int *info, void *stream) {
    if (N < 1 || N > QS_NOALLOC_MAX_N || batch < 0) {
        std::fprintf(stderr, "qs_invert_batched_noalloc: N = %d, batch = %d rejected: needs 1 <= N <= %d and batch >= 0\n",
                     N, batch, QS_NOALLOC_MAX_N);
        return QS_ERR_NOALLOC_LIMIT;
    }
    if (batch == 0) return 0;
    if (!A || !info) return -1;
    cudaStream_t st = (cudaStream_t)stream;
    const cudaError_t e = cudaMemsetAsync(info, 0, sizeof(int) * (size_t)batch, st);  // 0: no zero pivot
    if (e != cudaSuccess) return -(int)e;
    return qs::invert_batched_dev(st, N, batch, (qs::zc *)A, nullptr, info, true);
}
