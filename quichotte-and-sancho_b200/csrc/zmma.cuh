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

// the same over k = 16: a_i = A(g + 8(i&1), t + 4(i>>1)), i < 8; b_i = B(t + 4i, g), i < 4
__device__ __forceinline__ void dmma16816(double (&c)[4], const double (&a)[8], const double (&b)[4]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
        "{%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]), "d"(b[1]),
          "d"(b[2]), "d"(b[3]));
}
// complex C += A B over k = 16 from the fragments u and b
__device__ __forceinline__ void zmma16(double (&cr)[4], double (&ci)[4], const zc (&u)[8], const zc (&b)[4]) {
    double ar[8], ai[8], br[4], bi[4], nbi[4];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        ar[q] = u[q].x;
        ai[q] = u[q].y;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        br[q] = b[q].x;
        bi[q] = b[q].y;
        nbi[q] = -b[q].y;
    }
    dmma16816(cr, ar, br);
    dmma16816(ci, ar, bi);
    dmma16816(cr, ai, nbi);
    dmma16816(ci, ai, br);
}
// the same with A in shared memory, over the 16 columns of a panel or (!wide) its only 8: lo, hi the lane's values
// (row g of the tile, row g + 8 is 8 further) in columns t4 and t4 + 4, those in t4 + 8 and t4 + 12 are 8 ld further
__device__ __forceinline__ void zmma_panel(double (&cr)[4], double (&ci)[4], const zc *lo, const zc *hi, int ld, const zc (&b)[4],
                                           bool wide) {
    if (wide) {
        const zc u[8] = {lo[0], lo[8], hi[0], hi[8], lo[8 * ld], lo[8 * ld + 8], hi[8 * ld], hi[8 * ld + 8]};
        zmma16(cr, ci, u, b);
    } else {
        const zc u0 = lo[0], u1 = lo[8], u2 = hi[0], u3 = hi[8];
        const double ar[4] = {u0.x, u1.x, u2.x, u3.x}, ai[4] = {u0.y, u1.y, u2.y, u3.y};
        const double br[2] = {b[0].x, b[1].x}, bi[2] = {b[0].y, b[1].y}, nbi[2] = {-b[0].y, -b[1].y};
        dmma1688(cr, ar, br);
        dmma1688(ci, ar, bi);
        dmma1688(cr, ai, nbi);
        dmma1688(ci, ai, br);
    }
}

}  // namespace qs
