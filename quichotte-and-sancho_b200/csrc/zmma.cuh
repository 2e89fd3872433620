// zmma.cuh -- complex products on the FP64 tensor cores from matrices in shared memory.
#pragma once
#include "qs_common.cuh"

namespace qs {

// Position of element (i, j) of an N x N complex matrix in shared memory: column-major with the
// leading dimension padded to a multiple of 8, the row index XORed with a permutation of j mod 8.
// The eight lanes that a 16-byte access serves at a time touch eight different bank groups for all
// fragment shapes below: 2 rows x 4 columns (A, and B transposed), 4 rows x 2 columns (B), 2 rows x
// 4 even or odd columns (C), and for 8 rows of a column.
__device__ __forceinline__ int xr(int j) { return ((j ^ (j >> 2)) & 1) << 2 | (j & 2); }
__host__ __device__ __forceinline__ int smem_ld(int N) { return (N + 7) & ~7; }
__device__ __forceinline__ int at(int i, int j, int N) { return (i + j * smem_ld(N)) ^ xr(j); }
// values of a matrix with its columns padded to a multiple of 8, and the row tiles of 16 that
// reach beyond the last column
__host__ __device__ __forceinline__ int smem_units(int N) { return smem_ld(N) * smem_ld(N) + 8; }

// D = A B + D with A 16x8, B 8x8 in FP64: a_i = A(g + 8(i&1), t + 4(i>>1)), i < 4;
// b_i = B(t + 4i, g), i < 2; c_i = C(g + 8(i>>1), 2t + (i&1)) (g = lane / 4, t = lane % 4)
__device__ __forceinline__ void dmma1688(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

}  // namespace qs
