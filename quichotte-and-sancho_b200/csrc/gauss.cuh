// gauss.cuh -- the panels of the blocked Gauss-Jordan elimination (dyson_blk.cu, dyson_l2.cu): 16 columns, a
// row per lane in registers, partial pivoting without row exchanges.
#pragma once
#include "qs_common.cuh"

namespace qs {

constexpr int PB = 16;  // panel width: the k extent of one FP64 tensor-core product

// 1 / a without overflow or underflow of the intermediate |a|^2: a is scaled by the power of two
// that brings its larger part to [1, 2). (An infinite a gives NaN.)
__device__ __forceinline__ zc scaled_recip(zc a) {
    const unsigned h = max((unsigned)__double2hiint(a.x) & 0x7fffffffu, (unsigned)__double2hiint(a.y) & 0x7fffffffu) >> 20;
    const double s = __hiloint2double((int)(min(max(2046 - (int)h, 1), 2046) << 20), 0);  // 2^(1023 - h)
    const double x = a.x * s, y = a.y * s, d = s / fma(x, x, y * y);
    return zc{x * d, -y * d};
}

// |Re| + |Im| >= 0, so its bit pattern orders like its value (a NaN is a large key: a row is
// always found); 0 marks a row that is used or beyond the matrix
constexpr unsigned long long INF_KEY = 0x7ff0000000000001ull;  // of an infinite sum
__device__ __forceinline__ unsigned long long pivot_key(zc v, bool open) {
    return open ? (unsigned long long)__double_as_longlong(cabs1(v)) + 1 : 0;
}
// the lane with the warp's largest key, among equals the one whose row has the lowest place
__device__ __forceinline__ int warp_pivot(unsigned long long key, int place) {
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    const bool top = hi == mh && lo == ml;
    unsigned m = __ballot_sync(0xffffffffu, top);
    if (m & (m - 1)) {
        const unsigned first = __reduce_min_sync(0xffffffffu, top ? (unsigned)place : 0xffffffffu);
        m = __ballot_sync(0xffffffffu, top && (unsigned)place == first);
    }
    return __ffs(m) - 1;
}

// What the panel warps of a matrix exchange. NBUF = 2: the steps alternate between two buffers, one barrier
// each; 1: two barriers a step, for the order whose matrix leaves no room.
template <int PW, int NBUF> struct PanelExchange {
    zc row[NBUF][PW][PB];  // each panel warp's candidate: 1 / pivot, then the rest of its row
    zc extra[PB];
    unsigned long long key[NBUF][PW];
    int at[NBUF][PW];             // its place << 16 | its row
    int first_zero;               // 1 + the first step with a zero pivot (LAPACK's INFO), 0 if none
    unsigned char perm[32 * PW];  // pivot row of a step
};

// Steps k0 .. k0 + kb - 1 on the columns k0 .. k0 + WD - 1 of a matrix of order N (WD = 8 where there are no more), lane
// `row` holding its row's values in R (zero beyond the columns). R[j] is column (c + j) mod WD at step c, so that
// the current one is always R[0] and the loop need not be unrolled; afterwards R[j] is column (kb + j) mod WD.
// `place` is where row exchanges would have the row by now: used rows stand before step k, and the first of
// several largest candidates is the one that LAPACK's izamax finds. Returns whether the row became a pivot row.
// The operations on every value, and their order, are those of the elimination with row exchanges
//   row_k = row_p / pivot, row_i -= a_ik row_k
// so that the rounding of an inverse, which the sharp levels of a long molecule enlarge by 10^5 and more, is
// that of the elimination with row exchanges too.
template <int WD, int PW, int NBUF, class SYNC>
__device__ __forceinline__ bool eliminate_steps(PanelExchange<PW, NBUF> &e, int npw, zc (&R)[WD], int row, int N, int k0, int kb,
                                                int &place, bool zero_of_inf, SYNC sync) {
    const int lane = row & 31, warp = PW == 1 ? 0 : row >> 5;
    bool mine = false;
#pragma unroll 1
    for (int c = 0; c < kb; c++) {
        const int k = k0 + c, b = NBUF == 2 ? c & 1 : 0;
        const unsigned long long key = pivot_key(R[0], row < N && place >= k);
        const zc own = scaled_recip(R[0]);  // in case this row is chosen
        __syncwarp();
        if (lane == warp_pivot(key, place)) {
            e.row[b][warp][0] = own;
#pragma unroll
            for (int j = 1; j < WD; j++) e.row[b][warp][j] = R[j];
            e.key[b][warp] = key;
            e.at[b][warp] = place << 16 | row;
        }
        sync();
        int wb = 0, at = e.at[b][0];
        unsigned long long bk = e.key[b][0];
        if constexpr (PW > 1) {
#pragma unroll
            for (int q = 1; q < PW; q++) {
                if (q >= npw) break;
                const unsigned long long ck = e.key[b][q];
                const int ca = e.at[b][q];
                if (ck > bk || (ck == bk && ca < at)) {
                    bk = ck;
                    at = ca;
                    wb = q;
                }
            }
        }
        // a pivot whose key is that of +0: singular from here on (every lane sees the same)
        const bool zero = bk == 1;
        const int fz = e.first_zero;
        // the pivot row over its pivot, a value a lane; a copy for each warp, where its own candidate stood
        zc *S = warp == wb ? e.extra : e.row[b][warp];
        if (lane < WD) {
            const bool none = zero || (fz != 0 && fz <= k) || (zero_of_inf && bk == INF_KEY);
            const zc inv = none ? zc{0, 0} : e.row[b][wb][0], v = e.row[b][wb][lane];
            S[lane] = lane == 0 ? inv : v * inv;
        }
        if constexpr (NBUF == 1 && PW > 1) sync();
        else __syncwarp();
        const zc f = R[0];
        if (row == (at & 0xffff)) {
            mine = true;
            place = k;
            e.perm[k] = (unsigned char)row;
            if (zero && fz == 0) e.first_zero = k + 1;
            const zc inv = S[0];
#pragma unroll
            for (int j = 1; j < WD; j++) R[j - 1] = S[j];
            R[WD - 1] = inv;
        } else {
            if (place == k) place = at >> 16;
            zc first;
#pragma unroll
            for (int j = 0; j < WD; j++) {
                const zc r = S[j];
                zc t = j == 0 ? zc{0, 0} : R[j];
                t.x = fma(-f.x, r.x, t.x);
                t.x = fma(f.y, r.y, t.x);
                t.y = fma(-f.x, r.y, t.y);
                t.y = fma(-f.y, r.x, t.y);
                if (j == 0) first = t;
                else R[j - 1] = t;
            }
            R[WD - 1] = first;
        }
    }
    return mine;
}

// The panel of kb <= 16 columns in shared memory, lane `row` doing its row: value c at col(c)
template <int WD, int PW, int NBUF, class COL, class SYNC>
__device__ __forceinline__ bool eliminate_columns(PanelExchange<PW, NBUF> &e, int npw, int row, int N, int k0, int kb, int &place,
                                                  bool zero_of_inf, COL col, SYNC sync) {
    zc R[WD];
#pragma unroll
    for (int c = 0; c < WD; c++) R[c] = row < N && c < kb ? *col(c) : zc{0, 0};
    const bool mine = eliminate_steps<WD>(e, npw, R, row, N, k0, kb, place, zero_of_inf, sync);
    if (row < N)
#pragma unroll
        for (int j = 0; j < WD; j++) {
            const int c = (kb + j) & (WD - 1);
            if (c < kb) *col(c) = R[j];
        }
    return mine;
}
template <int PW, int NBUF, class COL, class SYNC>
__device__ __forceinline__ bool eliminate_panel(PanelExchange<PW, NBUF> &e, int npw, int row, int N, int k0, int kb, int &place,
                                                bool zero_of_inf, COL col, SYNC sync) {
    return kb > 8 ? eliminate_columns<PB>(e, npw, row, N, k0, kb, place, zero_of_inf, col, sync)
                  : eliminate_columns<8>(e, npw, row, N, k0, kb, place, zero_of_inf, col, sync);
}

}  // namespace qs
