// gauss.cuh -- one column of a Gauss-Jordan panel with a row per lane, PB columns of it in registers:
// the pivot search within a warp, the reciprocal, and the elimination of the lane's row.
#pragma once
#include "qs_common.cuh"

namespace qs {

constexpr int PB = 8;  // panel width

// 1 / a without overflow or underflow of the intermediate |a|^2: a is scaled by the power of two
// that brings its larger part to [1, 2)
__device__ __forceinline__ zc scaled_recip(zc a) {
    const unsigned h = max((unsigned)__double2hiint(a.x) & 0x7fffffffu, (unsigned)__double2hiint(a.y) & 0x7fffffffu) >> 20;
    const double s = __hiloint2double((int)(min(max(2046 - (int)h, 1), 2046) << 20), 0);  // 2^(1023 - h)
    const double x = a.x * s, y = a.y * s, d = s / fma(x, x, y * y);
    return zc{x * d, -y * d};
}

// |Re| + |Im| >= 0, so its bit pattern orders like its value (a NaN is a large key: a row is
// always found); 0 marks a row that is used or beyond the matrix
__device__ __forceinline__ unsigned long long pivot_key(zc v, bool open) {
    return open ? (unsigned long long)__double_as_longlong(cabs1(v)) + 1 : 0;
}
// the first lane with the warp's largest key (the first maximum, as izamax)
__device__ __forceinline__ int warp_pivot(unsigned long long key) {
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    return __ffs(__ballot_sync(0xffffffffu, hi == mh && lo == ml)) - 1;
}
// R -= m row, with 1 at column c of the pivot row
__device__ __forceinline__ void eliminate(zc (&R)[PB], int c, zc m, const zc (&row)[PB]) {
#pragma unroll
    for (int j = 0; j < PB; j++) {
        if (j == c) {
            R[j] = R[j] - m;
        } else {
            const zc r = row[j];
            R[j].x = fma(-m.x, r.x, R[j].x);
            R[j].y = fma(-m.x, r.y, R[j].y);
            R[j].x = fma(m.y, r.y, R[j].x);
            R[j].y = fma(-m.y, r.x, R[j].y);
        }
    }
}

}  // namespace qs
