// dyson_l2.cu -- the elimination of dyson_blk.cu for matrices in global memory (orders up to 256):
// in two levels, so that each value outside the current columns is read and written once per 32 steps.
//
// The matrix is where G goes (or in the block's slot of a workspace); the matrices of the resident
// blocks stay in L2. Per 32 columns K:
//   panel    the N x 32 columns in shared memory go through the 8-wide panels and updates of
//            dyson_blk: a row per lane, implicit pivoting, FP64 tensor cores
//   update   every other column, 8 a warp: A[i, j] = (i a pivot row of the 32 ? 0 : A[i, j]) +
//            sum_t A[i, K_t] A[p_t, j]. The 32 pivot-row values of its columns are in registers, the next
//            16 rows arrive while the present ones are multiplied
//   columns  column k of the eliminated matrix is column p_k of the inverse: it goes to that place, and the
//            column that stood there to one that became free. So the matrix needs no second copy; rows are
//            put in order, with the factors of their pivots, by one last pass over each column.
//
// Bound: FP64 rate (8 N^3 flops), and the panels' chain of about 1100 cycles a column, 2000 to 2900
// while the other blocks' tensor instructions keep the FP64 pipe. Up to 128 states four warps make a
// block, and three (N = 128) or four (N = 96) blocks an SM: their chains overlap each other and the
// updates. Above, eight warps and two blocks, where the matrices (175 MB at N = 192) no longer stay in L2.
// Of 750k cycles a matrix at N = 120 (three blocks an SM) the panels take 200k, their inner updates
// 70k, the update 280k, the build and the copies 200k.
// Measured on B200, batched inversion (8 N^3 flops a matrix), against one block an SM with the matrix in
// shared memory: 96 x 4000 2.77 -> 1.60 ms, 120 x 4096 4.06 -> 3.3 (17 TFLOP/s), 120 x 300 0.43 -> 0.34;
// against 16-wide panels with row exchanges in global memory: 192 x 1201 7.5 -> 3.9 ms (17 TFLOP/s).
// As Dyson step: 120 x 4096 4.6 -> 3.8 ms, 192 x 1201 7.5 -> 4.4 ms.
#include <algorithm>

#include "gauss.cuh"
#include "zmma.cuh"

namespace qs {
namespace {

__device__ __forceinline__ void cpa16(void *dst, const void *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

constexpr int OB = 32;             // columns of the outer level
constexpr int L2_MAXN = 256;

template <int MAXN> struct ExchangeL2 {
    static constexpr int MAXPW = MAXN / 32;
    zc row[2][MAXPW][PB];  // each panel warp's candidate row; steps alternate between the two
    zc inv[2][MAXPW];
    unsigned long long key[2][MAXPW];
    int idx[2][MAXPW];
    unsigned used[MAXPW], used_o[MAXPW];  // rows that became pivot rows in this panel, in these 32 columns
    int first_zero;                       // 1 + the first step with a zero pivot (LAPACK's INFO), 0 if none
    zc scale[MAXN];                    // 1 / pivot of a row
    unsigned char perm[MAXN];          // pivot row of a step
    short at_col[MAXN], col_at[MAXN];  // where a column is, and which one a place holds
};

// W warps, a row of the panel per lane: N <= 32 W
template <int W, int MINB>
__global__ void __launch_bounds__(32 * W, MINB) dyson_l2(DysonArgs a) {
    constexpr int MAXPW = W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ExchangeL2<32 * W> e;
    const int N = a.N, tid = threadIdx.x;
    constexpr int nthr = 32 * W;
    const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    zc *P = (zc *)smem_raw;  // the columns K: (i, c) at at(i, c, N)
    const bool whole = a.Ain || a.nA == N;  // every state is active
    const int ld = smem_ld(N), mtiles = (N + 15) / 16, PW = (N + 31) / 32;
    const int a0 = (g ^ xr(t4)) + t4 * ld, a1 = (g ^ xr(t4 + 4)) + (t4 + 4) * ld;
    const int e0 = (g ^ xr(2 * t4)) + 2 * t4 * ld, e1 = (g ^ xr(2 * t4 + 1)) + (2 * t4 + 1) * ld;
    for (int iw = a.iw0 + blockIdx.x; iw < a.iw1; iw += gridDim.x) {
        zc *M = a.inplace ? a.Gout + (size_t)(iw - a.iw0) * N * N : a.ws + (size_t)blockIdx.x * N * N;
        if (a.Ain && a.inplace) {  // the matrix is there
        } else if (a.Ain) {
            const zc *A = a.Ain + (size_t)(iw - a.iw0) * N * N;
            for (int idx = tid; idx < N * N; idx += nthr) M[idx] = A[idx];
        } else {
            // a warp takes 8 x 32 values at a time, their loads together
            constexpr int NC = 8 / MAXPW;
            const double w = a.omega[iw];
            const zc *SR = a.Sig + iw * a.sig_ld;
            for (int j0 = NC * warp; j0 < N; j0 += NC * W) {
                zc v[8], sg[8];
                bool with[8];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int i = min(lane + 32 * (u % MAXPW), N - 1), j = min(j0 + u / MAXPW, N - 1);
                    v[u] = a.Hemb[i + j * N];
                    const int pi = whole ? i : a.pos[i], pj = whole ? j : a.pos[j];
                    with[u] = a.use_sigma && pi >= 0 && pj >= 0;
                    sg[u] = with[u] && a.order2 ? sig_r(SR, pi, pj) : zc{0, 0};
                }
                if (a.use_sigma) {
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        const int i = min(lane + 32 * (u % MAXPW), N - 1), j = min(j0 + u / MAXPW, N - 1);
                        if (with[u]) v[u] = v[u] - (a.Sig1[i + j * N] + sg[u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int i = lane + 32 * (u % MAXPW), j = j0 + u / MAXPW;
                    if (i == j) v[u].x += w;
                    if (i < N && j < N) M[i + j * N] = v[u];
                }
            }
        }
        for (int i = tid; i < N; i += nthr) e.at_col[i] = e.col_at[i] = (short)i;
        if (tid == 0) e.first_zero = 0;
        const bool is_panel = warp < PW;
        bool open = is_panel && tid < N;  // this lane's row is not used yet
        __syncthreads();
#pragma unroll 1
        for (int k0 = 0; k0 < N; k0 += OB) {
            const int kb = min(OB, N - k0);
            // ---- the columns K into shared memory; columns beyond N are zero
            for (int c = warp; c < OB; c += W) {
                const zc *src = M + (c < kb ? e.at_col[k0 + c] : 0) * N;
                for (int i = lane; i < N; i += 32) {
                    if (c < kb) cpa16(&P[at(i, c, N)], src + i);
                    else P[at(i, c, N)] = zc{0, 0};
                }
            }
            asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
            if (tid < MAXPW) e.used_o[tid] = 0;
            __syncthreads();
#pragma unroll 1
            for (int k1 = 0; k1 < kb; k1 += PB) {
                if (is_panel) {
                    zc R[PB];
#pragma unroll
                    for (int c = 0; c < PB; c++) R[c] = tid < N ? P[at(tid, k1 + c, N)] : zc{0, 0};
                    bool mine = false;
#pragma unroll
                    for (int c = 0; c < PB; c++) {
                        const int k = k0 + k1 + c, b = c & 1;
                        if (k >= N) break;
                        const unsigned long long key = pivot_key(R[c], open);
                        const zc inv = scaled_recip(R[c]);  // in case this row is chosen
                        if (lane == warp_pivot(key)) {
#pragma unroll
                            for (int j = 0; j < PB; j++)
                                if (j != c) e.row[b][warp][j] = R[j];
                            e.inv[b][warp] = inv;
                            e.key[b][warp] = key;
                            e.idx[b][warp] = tid;
                        }
                        asm volatile("bar.sync 1, %0;\n" ::"r"(32 * PW) : "memory");
                        int wb = 0;
                        unsigned long long bk = e.key[b][0];
#pragma unroll
                        for (int q = 1; q < MAXPW; q++) {
                            if (q >= PW) break;
                            const unsigned long long ck = e.key[b][q];
                            if (ck > bk) {
                                bk = ck;
                                wb = q;
                            }
                        }
                        const int p = e.idx[b][wb];
                        zc pinv = e.inv[b][wb];
                        const bool zero = bk == 1;
                        const int fz = e.first_zero;
                        if (zero || (fz != 0 && fz <= k)) pinv = zc{0, 0};
                        zc m = R[c] * pinv;
                        const bool is = tid == p;
                        R[c] = is ? zc{1, 0} : zc{0, 0};
                        if (is) {
                            open = false;
                            mine = true;
                            e.scale[p] = pinv;
                            m = zc{0, 0};
                            e.perm[k] = (unsigned char)p;
                            if (zero && fz == 0) e.first_zero = k + 1;
                        }
                        eliminate(R, c, m, e.row[b][wb]);
                    }
                    if (tid < N)
#pragma unroll
                        for (int c = 0; c < PB; c++)
                            if (k0 + k1 + c < N) P[at(tid, k1 + c, N)] = R[c];
                    const unsigned u = __ballot_sync(0xffffffffu, mine);
                    if (lane == 0) {
                        e.used[warp] = u;
                        e.used_o[warp] |= u;
                    }
                }
                __syncthreads();
                // ---- the other 8-column tiles of K: their pivot-row values first
                const int p0 = k0 + k1 + t4 < N ? e.perm[k0 + k1 + t4] : -1;
                const int p1 = k0 + k1 + t4 + 4 < N ? e.perm[k0 + k1 + t4 + 4] : -1;
                constexpr int CTS = OB / PB;
                zc v0[CTS], v1[CTS];
#pragma unroll
                for (int ct = 0; ct < CTS; ct++) {
                    const zc *col = P + (8 * ct + g) * ld;
                    v0[ct] = p0 >= 0 ? col[p0 ^ xr(g)] : zc{0, 0};
                    v1[ct] = p1 >= 0 ? col[p1 ^ xr(g)] : zc{0, 0};
                }
                __syncthreads();
                const zc *Ap0 = P + k1 * ld + a0, *Ap1 = P + k1 * ld + a1;
#pragma unroll 1
                for (int rt = warp; rt < mtiles; rt += W) {
                    const int i0 = 16 * rt;
                    const unsigned um = e.used[i0 >> 5] >> (i0 & 31);  // pivot rows of this tile
                    const bool ug = (um >> g) & 1, uh = (um >> (g + 8)) & 1, low = i0 + 8 < N;
                    const zc u0 = Ap0[i0], u1 = Ap0[i0 + 8], u2 = Ap1[i0], u3 = Ap1[i0 + 8];
                    const double ar[4] = {u0.x, u1.x, u2.x, u3.x}, ai[4] = {u0.y, u1.y, u2.y, u3.y};
#pragma unroll
                    for (int ct = 0; ct < CTS; ct++) {
                        if (ct == k1 / PB || 8 * ct >= kb) continue;
                        zc *Cp0 = P + 8 * ct * ld + e0 + i0, *Cp1 = P + 8 * ct * ld + e1 + i0;
                        const zc w0 = Cp0[0], w1 = Cp1[0], w2 = Cp0[8], w3 = Cp1[8];
                        double cr[4] = {ug ? 0.0 : w0.x, ug ? 0.0 : w1.x, uh ? 0.0 : w2.x, uh ? 0.0 : w3.x};
                        double ci[4] = {ug ? 0.0 : w0.y, ug ? 0.0 : w1.y, uh ? 0.0 : w2.y, uh ? 0.0 : w3.y};
                        const double br[2] = {v0[ct].x, v1[ct].x}, bi[2] = {v0[ct].y, v1[ct].y};
                        const double nbi[2] = {-v0[ct].y, -v1[ct].y};
                        dmma1688(cr, ar, br);
                        dmma1688(ci, ar, bi);
                        dmma1688(cr, ai, nbi);
                        dmma1688(ci, ai, br);
                        Cp0[0] = zc{cr[0], ci[0]};
                        Cp1[0] = zc{cr[1], ci[1]};
                        if (low) {  // (the last tile's lower half may lie in the next column)
                            Cp0[8] = zc{cr[2], ci[2]};
                            Cp1[8] = zc{cr[3], ci[3]};
                        }
                    }
                }
                __syncthreads();
            }
            // ---- the other columns, 8 a warp: column q of them is q or, beyond K, q + kb
            const int nq = N - kb;
#pragma unroll 1
            for (int q0 = 8 * warp; q0 < nq; q0 += 8 * W) {
                auto column = [&](int q) {
                    q = min(q, nq - 1);
                    return M + e.at_col[q < k0 ? q : q + kb] * N;
                };
                const zc *Bc = column(q0 + g);
                zc b[OB / 4];
#pragma unroll
                for (int s = 0; s < OB / 4; s++) {
                    const int t = 4 * s + t4;
                    b[s] = t < kb ? Bc[e.perm[k0 + t]] : zc{0, 0};
                }
                __syncwarp();  // before other lanes of this warp rewrite the pivot rows
                zc *C0 = column(q0 + 2 * t4), *C1 = column(q0 + 2 * t4 + 1);
                const bool s0 = q0 + 2 * t4 < nq, s1 = q0 + 2 * t4 + 1 < nq;
                zc n0 = C0[g], n1 = C1[g], n2 = C0[g + 8], n3 = C1[g + 8];  // (N > 16)
#pragma unroll 1
                for (int rt = 0; rt < mtiles; rt++) {
                    const int i0 = 16 * rt;
                    const unsigned um = e.used_o[i0 >> 5] >> (i0 & 31);
                    const bool ug = (um >> g) & 1, uh = (um >> (g + 8)) & 1;
                    double cr[4] = {ug ? 0.0 : n0.x, ug ? 0.0 : n1.x, uh ? 0.0 : n2.x, uh ? 0.0 : n3.x};
                    double ci[4] = {ug ? 0.0 : n0.y, ug ? 0.0 : n1.y, uh ? 0.0 : n2.y, uh ? 0.0 : n3.y};
                    const int ng = min(i0 + 16 + g, N - 1), nh = min(i0 + 24 + g, N - 1);
                    n0 = C0[ng];
                    n1 = C1[ng];
                    n2 = C0[nh];
                    n3 = C1[nh];
#pragma unroll
                    for (int s = 0; s < OB / 8; s++) {
                        const zc *Ap0 = P + 8 * s * ld + a0 + i0, *Ap1 = P + 8 * s * ld + a1 + i0;
                        const zc u0 = Ap0[0], u1 = Ap0[8], u2 = Ap1[0], u3 = Ap1[8];
                        const double ar[4] = {u0.x, u1.x, u2.x, u3.x}, ai[4] = {u0.y, u1.y, u2.y, u3.y};
                        const double br[2] = {b[2 * s].x, b[2 * s + 1].x}, bi[2] = {b[2 * s].y, b[2 * s + 1].y};
                        const double nbi[2] = {-b[2 * s].y, -b[2 * s + 1].y};
                        dmma1688(cr, ar, br);
                        dmma1688(ci, ar, bi);
                        dmma1688(cr, ai, nbi);
                        dmma1688(ci, ai, br);
                    }
                    const bool r0 = i0 + g < N, r1 = i0 + g + 8 < N;
                    if (s0 && r0) C0[i0 + g] = zc{cr[0], ci[0]};
                    if (s1 && r0) C1[i0 + g] = zc{cr[1], ci[1]};
                    if (s0 && r1) C0[i0 + g + 8] = zc{cr[2], ci[2]};
                    if (s1 && r1) C1[i0 + g + 8] = zc{cr[3], ci[3]};
                }
            }
            __syncthreads();
            // ---- column c of K belongs at t = p_c; a column found there (none of K's) moves to a place of K
            // that no column of K goes to
            const bool in = lane < kb;
            const int from = in ? e.at_col[k0 + lane] : 0, t = in ? e.perm[k0 + lane] : 0;
            const int there = e.col_at[t];
            const bool moves = in && (there < k0 || there >= k0 + kb);
            const unsigned freed = __ballot_sync(0xffffffffu, in && !((e.used_o[from >> 5] >> (from & 31)) & 1));
            const unsigned moving = __ballot_sync(0xffffffffu, moves);
            const int fl = moves ? __fns(freed, 0, __popc(moving & ((1u << lane) - 1)) + 1) : lane;
            const int to = __shfl_sync(0xffffffffu, from, fl);
            for (int c = warp; c < kb; c += W) {
                const int tc = __shfl_sync(0xffffffffu, t, c), dst = __shfl_sync(0xffffffffu, to, c);
                zc v[MAXPW];
                const bool mv = (moving >> c) & 1;
#pragma unroll
                for (int q = 0; q < MAXPW; q++) {
                    const int i = lane + 32 * q;
                    if (mv && i < N) v[q] = M[i + tc * N];
                }
#pragma unroll
                for (int q = 0; q < MAXPW; q++) {
                    const int i = lane + 32 * q;
                    if (i >= N) continue;
                    if (mv) M[i + dst * N] = v[q];
                    M[i + tc * N] = P[at(i, c, N)];
                }
            }
            __syncthreads();
            if (warp == 0) {
                if (moves) {
                    e.at_col[there] = (short)to;
                    e.col_at[to] = (short)there;
                }
                if (in) {
                    e.at_col[k0 + lane] = (short)t;
                    e.col_at[t] = (short)(k0 + lane);
                }
            }
            __syncthreads();
        }
        if (e.first_zero && tid == 0) {
            if (a.info) atomicMin(a.info, iw + 1);
            if (a.info_each) a.info_each[iw - a.iw0] = e.first_zero;
        }
        // ---- rows in order, times their factors; column c is in its place
        const bool part = a.out_mode == 0 && !whole;  // the active block alone
        const int nout = part ? a.nA : N;
        zc *G = a.out_mode == 0 ? a.Gout + (size_t)iw * nout * nout : a.Gout + (size_t)(iw - a.iw0) * nout * nout;
        for (int c = warp; c < nout; c += W) {
            const zc *col = M + (part ? a.act[c] : c) * N;
            zc v[MAXPW];
#pragma unroll
            for (int q = 0; q < MAXPW; q++) {
                const int k = lane + 32 * q;
                if (k < nout) {
                    const int p = e.perm[part ? a.act[k] : k];
                    v[q] = col[p] * e.scale[p];
                }
            }
            __syncwarp();  // in place: the column is read before it is rewritten
#pragma unroll
            for (int q = 0; q < MAXPW; q++) {
                const int k = lane + 32 * q;
                if (k < nout) G[k + c * nout] = v[q];
            }
        }
        __syncthreads();
    }
}

template <int W, int MINB> int run(cudaStream_t st, const DysonArgs &a) {
    const void *fn = (const void *)dyson_l2<W, MINB>;
    cudaError_t e = smem_cap(fn);
    if (e != cudaSuccess) return -(int)e;
    // as many blocks as fit at once (228 KB of shared memory an SM, 1 KB of it the system's for each block)
    const size_t sm = sizeof(zc) * (OB * smem_ld(a.N) + 8);
    const int fit = std::min<int>(MINB, (228 << 10) / (sm + sizeof(ExchangeL2<32 * W>) + 1024));
    const int blocks = a.inplace ? 148 * std::max(fit, 1) : std::min(148 * std::max(fit, 1), DYSON_L2_SLOTS);
    dyson_l2<W, MINB><<<std::min(a.iw1 - a.iw0, blocks), 32 * W, sm, st>>>(a);
    e = cudaGetLastError();
    return e == cudaSuccess ? 0 : -(int)e;
}

}  // namespace

bool dyson_l2_fits(int N) { return N <= L2_MAXN; }

int launch_dyson_l2(cudaStream_t st, const DysonArgs &a) { return a.N <= 128 ? run<4, 4>(st, a) : run<8, 2>(st, a); }

}  // namespace qs
