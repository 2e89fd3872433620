// dyson_l2.cu -- the elimination of dyson_blk.cu for matrices in global memory (orders up to 256):
// in two levels, so that each value outside the current columns is read and written once per 32 steps.
//
// The matrix is where G goes (or in the block's slot of a workspace); the matrices of the resident
// blocks stay in L2. Per 32 columns K, two panels of 16, in shared memory:
//   panels   the first one's columns by a row per lane with implicit pivoting (gauss.cuh), its update of the
//            second one's columns on the FP64 tensor cores, the second one's columns
//   update   every other column, 8 a warp, the two panels one after the other on values in registers:
//            A[i, j] = (i a pivot row of the panel ? 0 : A[i, j]) + sum_t A[i, K_t] A[p_t, j]. The pivot-row
//            values of the first panel are loaded; those of the second have to be what the first one makes of them,
//            so its 16 pivot rows are formed ahead as a tile of their own. The next 16 rows arrive while
//            the present ones are multiplied. Then the second panel's update of the first one's columns, whose
//            values after the first panel all of this has used
//   columns  column k of the eliminated matrix is column p_k of the inverse: it goes to that place, and the
//            column that stood there to one that became free. So the matrix needs no second copy; rows are
//            put in order by one last pass over each column.
// As in dyson_blk.cu, the operations on a value are those of the elimination with row exchanges in panels of 16,
// bit for bit (one update of depth 32 from panels of 8: 120 x 4096 3.29 ms, here 3.46; 192 x 1201 3.82 and 4.27).
//
// Bound: FP64 rate (8 N^3 flops: 17 TFLOP/s at 120 x 4096, 16 at 192 x 1201), and the panels' chain, stretched while
// the other blocks' tensor instructions keep the FP64 pipe. Up to 128 states four warps make a
// block, and three (N = 128) or four (N = 96) blocks an SM: their chains overlap each other and the
// updates. Four need 128 registers a thread, which spill; from 97 on there is room for three blocks at most, and
// with 168 registers 120 x 4096 takes 3.46 ms instead of 3.68. Above 128, eight warps and two blocks, where the
// matrices (175 MB at N = 192) no longer stay in L2.
// Measured on B200, batched inversion, against one block an SM with the matrix in shared memory:
// 96 x 4000 3.21 -> 1.91 ms, 120 x 4096 4.83 -> 3.46, 120 x 300 0.51 -> 0.39; against 16-wide panels with row
// exchanges in global memory: 192 x 1201 7.5 -> 4.3 ms.
#include <algorithm>

#include "gauss.cuh"
#include "zmma.cuh"

namespace qs {
namespace {

__device__ __forceinline__ void cpa16(void *dst, const void *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

constexpr int OB = 2 * PB;         // columns of the outer level: two panels
constexpr int L2_MAXN = 256;

template <int W> struct ExchangeL2 : PanelExchange<W, 2> {
    unsigned used[2][W];                   // rows that became pivot rows in the first and in the second panel
    short at_col[32 * W], col_at[32 * W];  // where a column is, and which one a place holds
};

// the B fragment (k = 16, n = 8) of a 16 x 8 result that the warp holds as accumulators
__device__ __forceinline__ void as_b(const double (&cr)[4], const double (&ci)[4], zc (&b)[4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        // row t4 + 4 q, column g: lane 4 (row mod 8) + g / 2, value 2 (row / 8) + g mod 2
        const int from = 4 * (t4 + 4 * (q & 1)) + (g >> 1), v = 2 * (q >> 1);
        const double x0 = __shfl_sync(0xffffffffu, cr[v], from), x1 = __shfl_sync(0xffffffffu, cr[v + 1], from);
        const double y0 = __shfl_sync(0xffffffffu, ci[v], from), y1 = __shfl_sync(0xffffffffu, ci[v + 1], from);
        b[q] = g & 1 ? zc{x1, y1} : zc{x0, y0};
    }
}

// W warps, a row of the panel per lane: N <= 32 W
template <int W, int MINB>
__global__ void __launch_bounds__(32 * W, MINB) dyson_l2(DysonArgs a) {
    constexpr int MAXPW = W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ExchangeL2<W> e;
    const int N = a.N, tid = threadIdx.x;
    constexpr int nthr = 32 * W;
    const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    zc *P = (zc *)smem_raw;  // the columns K: (i, c) at at(i, c, N)
    const bool whole = a.Ain || a.nA == N;  // every state is active
    const int ld = smem_ld(N), mtiles = (N + 15) / 16, PW = (N + 31) / 32;
    const int a0 = (g ^ xr(t4)) + t4 * ld, a1 = (g ^ xr(t4 + 4)) + (t4 + 4) * ld;
    const int e0 = (g ^ xr(2 * t4)) + 2 * t4 * ld, e1 = (g ^ xr(2 * t4 + 1)) + (2 * t4 + 1) * ld;
    auto panel_sync = [&] { asm volatile("bar.sync 1, %0;\n" ::"r"(32 * PW) : "memory"); };
    // rows of tile i0 in the mask: g, g + 8
    auto rows_used = [&](int panel, int i0, bool &ug, bool &uh) {
        const unsigned um = e.used[panel][i0 >> 5] >> (i0 & 31);
        ug = (um >> g) & 1;
        uh = (um >> (g + 8)) & 1;
    };
    // the 16 columns of panel `by` applied to the other panel of K, in place: a warp's row tiles, after the
    // pivot-row values of all its columns were read
    auto cross_update = [&](int by, int k0, int kb) {
        const int other = 1 - by, c0 = PB * other, nb = min(PB, kb - PB * by), nc = min(PB, kb - c0);
        zc v[2][4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int t = t4 + 4 * q, p = t < nb ? e.perm[k0 + PB * by + t] : -1;
#pragma unroll
            for (int ct = 0; ct < 2; ct++) v[ct][q] = p >= 0 ? P[(c0 + 8 * ct + g) * ld + (p ^ xr(g))] : zc{0, 0};
        }
        __syncthreads();
#pragma unroll 1
        for (int rt = warp; rt < mtiles; rt += W) {
            const int i0 = 16 * rt;
            const bool low = i0 + 8 < N;
            bool ug, uh;
            rows_used(by, i0, ug, uh);
#pragma unroll
            for (int ct = 0; ct < 2; ct++) {
                if (8 * ct >= nc) continue;
                zc *Cp0 = P + (c0 + 8 * ct) * ld + e0 + i0, *Cp1 = P + (c0 + 8 * ct) * ld + e1 + i0;
                const zc w0 = Cp0[0], w1 = Cp1[0], w2 = Cp0[8], w3 = Cp1[8];
                double cr[4] = {ug ? 0.0 : w0.x, ug ? 0.0 : w1.x, uh ? 0.0 : w2.x, uh ? 0.0 : w3.x};
                double ci[4] = {ug ? 0.0 : w0.y, ug ? 0.0 : w1.y, uh ? 0.0 : w2.y, uh ? 0.0 : w3.y};
                zmma_panel(cr, ci, P + PB * by * ld + a0 + i0, P + PB * by * ld + a1 + i0, ld, v[ct], nb > 8);
                Cp0[0] = zc{cr[0], ci[0]};
                Cp1[0] = zc{cr[1], ci[1]};
                if (low) {  // (the last tile's lower half may lie in the next column)
                    Cp0[8] = zc{cr[2], ci[2]};
                    Cp1[8] = zc{cr[3], ci[3]};
                }
            }
        }
        __syncthreads();
    };
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
        int place = tid;  // of this lane's row
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
            __syncthreads();
#pragma unroll 1
            for (int h = 0; PB * h < kb; h++) {
                if (is_panel) {
                    const int c0 = PB * h, nb = min(PB, kb - c0);
                    const bool mine = eliminate_panel(e, PW, tid, N, k0 + c0, nb, place, a.zero_of_inf,
                                                      [&](int c) { return P + at(tid, c0 + c, N); }, panel_sync);
                    const unsigned u = __ballot_sync(0xffffffffu, mine);
                    if (lane == 0) e.used[h][warp] = u;
                }
                __syncthreads();
                // ---- after the last panel, the other columns, 8 a warp, both panels in turn: column q of them is
                // q or, beyond K, q + kb
                const int nq = PB * (h + 1) < kb ? 0 : N - kb;
#pragma unroll 1
                for (int q0 = 8 * warp; q0 < nq; q0 += 8 * W) {
                    auto column = [&](int q) {
                        q = min(q, nq - 1);
                        return M + e.at_col[q < k0 ? q : q + kb] * N;
                    };
                    const zc *Bc = column(q0 + g);
                    zc *C0 = column(q0 + 2 * t4), *C1 = column(q0 + 2 * t4 + 1);
                    zc b1[4], b2[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int t = t4 + 4 * q;
                        b1[q] = t < kb ? Bc[e.perm[k0 + t]] : zc{0, 0};
                        b2[q] = zc{0, 0};
                    }
                    if (kb > PB) {
                        // the second panel's pivot rows after the first panel
                        const int r0 = PB + g < kb ? e.perm[k0 + PB + g] : -1, r1 = PB + g + 8 < kb ? e.perm[k0 + PB + g + 8] : -1;
                        const zc z{0, 0}, w0 = r0 >= 0 ? C0[r0] : z, w1 = r0 >= 0 ? C1[r0] : z, w2 = r1 >= 0 ? C0[r1] : z,
                                 w3 = r1 >= 0 ? C1[r1] : z;
                        double cr[4] = {w0.x, w1.x, w2.x, w3.x}, ci[4] = {w0.y, w1.y, w2.y, w3.y};
                        zc u[8];
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            const int r = q & 1 ? r1 : r0, c = t4 + 4 * (q >> 1);
                            u[q] = r >= 0 ? P[at(r, c, N)] : z;
                        }
                        zmma16(cr, ci, u, b1);
                        as_b(cr, ci, b2);
                    }
                    __syncwarp();  // before other lanes of this warp rewrite the pivot rows
                    const bool s0 = q0 + 2 * t4 < nq, s1 = q0 + 2 * t4 + 1 < nq;
                    zc n0 = C0[g], n1 = C1[g], n2 = C0[g + 8], n3 = C1[g + 8];  // (N > 16)
#pragma unroll 1
                    for (int rt = 0; rt < mtiles; rt++) {
                        const int i0 = 16 * rt;
                        bool ug, uh;
                        rows_used(0, i0, ug, uh);
                        double cr[4] = {ug ? 0.0 : n0.x, ug ? 0.0 : n1.x, uh ? 0.0 : n2.x, uh ? 0.0 : n3.x};
                        double ci[4] = {ug ? 0.0 : n0.y, ug ? 0.0 : n1.y, uh ? 0.0 : n2.y, uh ? 0.0 : n3.y};
                        const int ng = min(i0 + 16 + g, N - 1), nh = min(i0 + 24 + g, N - 1);
                        n0 = C0[ng];
                        n1 = C1[ng];
                        n2 = C0[nh];
                        n3 = C1[nh];
                        zmma_panel(cr, ci, P + a0 + i0, P + a1 + i0, ld, b1, kb > 8);
                        if (kb > PB) {
                            rows_used(1, i0, ug, uh);
                            cr[0] = ug ? 0.0 : cr[0];
                            cr[1] = ug ? 0.0 : cr[1];
                            cr[2] = uh ? 0.0 : cr[2];
                            cr[3] = uh ? 0.0 : cr[3];
                            ci[0] = ug ? 0.0 : ci[0];
                            ci[1] = ug ? 0.0 : ci[1];
                            ci[2] = uh ? 0.0 : ci[2];
                            ci[3] = uh ? 0.0 : ci[3];
                            zmma_panel(cr, ci, P + PB * ld + a0 + i0, P + PB * ld + a1 + i0, ld, b2, kb > PB + 8);
                        }
                        const bool r0 = i0 + g < N, r1 = i0 + g + 8 < N;
                        if (s0 && r0) C0[i0 + g] = zc{cr[0], ci[0]};
                        if (s1 && r0) C1[i0 + g] = zc{cr[1], ci[1]};
                        if (s0 && r1) C0[i0 + g + 8] = zc{cr[2], ci[2]};
                        if (s1 && r1) C1[i0 + g + 8] = zc{cr[3], ci[3]};
                    }
                }
                // ---- the panel applied to the other one (the second to the first's old values once they are not
                // needed any more)
                if (kb > PB) {
                    if (h) __syncthreads();
                    cross_update(h, k0, kb);
                }
            }
            __syncthreads();
            // ---- column c of K belongs at t = p_c; a column found there (none of K's) moves to a place of K
            // that no column of K goes to
            const bool in = lane < kb;
            const int from = in ? e.at_col[k0 + lane] : 0, t = in ? e.perm[k0 + lane] : 0;
            const int there = e.col_at[t];
            const bool moves = in && (there < k0 || there >= k0 + kb);
            const unsigned taken = e.used[0][from >> 5] | (kb > PB ? e.used[1][from >> 5] : 0u);
            const unsigned freed = __ballot_sync(0xffffffffu, in && !((taken >> (from & 31)) & 1));
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
        // ---- rows in order; column c is in its place
        const bool part = a.out_mode == 0 && !whole;  // the active block alone
        const int nout = part ? a.nA : N;
        zc *G = a.out_mode == 0 ? a.Gout + (size_t)iw * nout * nout : a.Gout + (size_t)(iw - a.iw0) * nout * nout;
        for (int c = warp; c < nout; c += W) {
            const zc *col = M + (part ? a.act[c] : c) * N;
            zc v[MAXPW];
#pragma unroll
            for (int q = 0; q < MAXPW; q++) {
                const int k = lane + 32 * q;
                if (k < nout) v[q] = col[e.perm[part ? a.act[k] : k]];
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
    const int fit = std::min<int>(MINB, (228 << 10) / (sm + sizeof(ExchangeL2<W>) + 1024));
    const int blocks = a.inplace ? 148 * std::max(fit, 1) : std::min(148 * std::max(fit, 1), DYSON_L2_SLOTS);
    dyson_l2<W, MINB><<<std::min(a.iw1 - a.iw0, blocks), 32 * W, sm, st>>>(a);
    e = cudaGetLastError();
    return e == cudaSuccess ? 0 : -(int)e;
}

}  // namespace

bool dyson_l2_fits(int N) { return N <= L2_MAXN; }

int launch_dyson_l2(cudaStream_t st, const DysonArgs &a) {
    return a.N <= 96 ? run<4, 4>(st, a) : a.N <= 128 ? run<4, 3>(st, a) : run<8, 2>(st, a);
}

}  // namespace qs
