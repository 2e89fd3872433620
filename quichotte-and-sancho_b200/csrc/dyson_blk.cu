// dyson_blk.cu -- G^r(w) = [hbar w - H + (i/2hbar)(GammaL+GammaR) - Sigma^r(w)]^-1 for every energy, and
// batched inversion (invert_complex, common/linear_algebra.f90:58-88): blocked in-place Gauss-Jordan
// elimination with partial pivoting in shared memory, one matrix per warp (N <= 32) or block
// (N <= 120).
//
// Panels of 8 columns K = [k0, k0 + 8), one column tile of the FP64 tensor cores:
//   panel   PW = ceil(N / 32) warps hold one row of the panel per lane in registers. Per column every
//           warp finds its best row (integer warp reductions on the bits of |Re| + |Im|) and
//           publishes that row and its reciprocal; after one barrier every lane picks the best
//           warp's and eliminates its own row
//   update  every other column tile j by one warp, complex products of four real DMMAs:
//           A[i, j] = (i a pivot row of the panel ? 0 : A[i, j]) + sum_t A[i, K_t] A[p_t, j],
//           with the pivot rows A[p_t, j] read into registers first
// Rows are never exchanged: a row is used once, as pivot row p_k of step k. With the pivot on
// (p_k, k) elimination exchanges y_{p_k} and x_k, so that in the end row p_k holds row k of the
// inverse and column k its column p_k; the output is written through that permutation. Elimination
// is homogeneous in a row, so a pivot row is not divided by its pivot either: it keeps its values
// (1 in column k) and gets the factor 1 / pivot on output.
//
// Bound: the panel's columns are a chain of about 500 cycles (search, row, barrier, 32 DFMA); the
// update runs at the FP64 rate. Small matrices share an SM (20 of order 24, 5 of order 40), so
// that panels and updates of different ones overlap.
//
// Measured on B200, batched inversion (8 N^3 flops a matrix), against the kernels this replaces
// (row exchanges, 16-wide panels, one block a matrix, or everything through a global workspace):
// N = 120 8.9 -> 13.9 TFLOP/s; as Dyson of 40 states x 5003 energies 0.99 -> 0.39 ms,
// 24 x 32768 3.05 -> 0.48 ms, 48 x 4001 1.58 -> 0.36 ms. At N = 120 a matrix takes 280k cycles: the
// panels 128k (1070 a column), the updates 125k (107k at the DMMA rate), load and output 30k.
// Tried instead for N <= 96: the whole matrix in registers, rank-1 updates (4-9 TFLOP/s: the
// per-step work of every warp, column and row exchange and selects, outweighs the update).
#include <algorithm>
#include <climits>

#include "gauss.cuh"
#include "zmma.cuh"

namespace qs {
namespace {

template <int PW> struct Exchange {
    zc row[2][PW][PB];  // each panel warp's candidate row; steps alternate between the two
    zc inv[2][PW];
    unsigned long long key[2][PW];
    int idx[2][PW];
    unsigned used[PW];      // rows (bits) that became pivot rows in this panel
    int first_zero;         // 1 + the first step with a zero pivot (LAPACK's INFO), 0 if none
    int pad;
    unsigned char perm[32 * PW], step[32 * PW];  // pivot row of a step, step of a row
};

// PW panel warps, W warps a matrix, MPB matrices a block (more than one only for W = 1).
template <int PW, int W, int MPB, int MINB>
__global__ void __launch_bounds__(32 * W * MPB, MINB) dyson_blk(DysonArgs a) {
    static_assert(MPB == 1 || W == 1, "several matrices a block: one warp each");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ Exchange<PW> exs[MPB];
    const int N = a.N, nA = a.nA, slot = W == 1 ? threadIdx.x >> 5 : 0, tid = W == 1 ? threadIdx.x & 31 : threadIdx.x;
    constexpr int nthr = 32 * W;
    const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    Exchange<PW> &e = exs[slot];
    zc *M = (zc *)smem_raw + (size_t)slot * smem_units(N);
    const int mtiles = (N + 15) / 16, ntiles = (N + 7) / 8;
    auto sync = [] {
        if constexpr (W == 1) __syncwarp();
        else __syncthreads();
    };
    auto panel_sync = [] {
        if constexpr (W == 1) __syncwarp();
        else if constexpr (PW == W) __syncthreads();
        else if constexpr (PW == 1) __syncwarp();
        else asm volatile("bar.sync 1, %0;\n" ::"n"(32 * PW) : "memory");
    };
    const bool whole = a.Ain || nA == N;           // every state is active
    const int di = nthr % N, dj = nthr / N;        // the step from one element of a thread to its next
    constexpr int NB = PW == 1 ? 6 : 4;
    for (int iw = a.iw0 + blockIdx.x * MPB + slot; iw < a.iw1; iw += gridDim.x * MPB) {
        if (a.Ain) {
            const zc *A = a.Ain + (size_t)(iw - a.iw0) * N * N;
#pragma unroll 4
            for (int idx = tid; idx < N * N; idx += nthr) M[at(idx % N, idx / N, N)] = A[idx];
        } else {
            const double w = a.omega[iw];
            const zc *SR = a.Sig + iw * a.sig_ld;
            // NB values a thread at a time: their loads together, those of Sigma2 first
            int i = tid % N, j = tid / N;
            for (int idx = tid; idx < N * N; idx += NB * nthr) {
                zc v[NB], sg[NB];
                int at_s[NB];
                bool with[NB];
#pragma unroll
                for (int u = 0; u < NB; u++) {
                    at_s[u] = j < N ? at(i, j, N) : -1;
                    with[u] = a.use_sigma && j < N;
                    int pi = i, pj = j;
                    if (!whole && with[u]) {
                        pi = a.pos[i];
                        pj = a.pos[j];
                        with[u] = pi >= 0 && pj >= 0;
                    }
                    sg[u] = with[u] && a.order2 ? sig_r(SR, pi, pj) : zc{0, 0};
                    v[u] = j < N ? a.Hemb[idx + u * nthr] : zc{0, 0};
                    if (i == j) v[u].x += w;
                    i += di;
                    j += dj + (i >= N);
                    i -= i >= N ? N : 0;
                }
#pragma unroll
                for (int u = 0; u < NB; u++) {
                    if (with[u]) v[u] = v[u] - (a.Sig1[idx + u * nthr] + sg[u]);
                    if (at_s[u] >= 0) M[at_s[u]] = v[u];
                }
            }
        }
        // the columns that pad the last tile: zero operands (rows beyond N reach rows beyond N only)
        for (int t = N * smem_ld(N) + tid; t < smem_units(N); t += nthr) M[t] = zc{0, 0};
        if (tid == 0) e.first_zero = 0;
        const bool is_panel = warp < PW;
        bool open = is_panel && tid < N;  // this lane's row is not used yet
        zc scale{0, 0};                   // the factor it lacks since its step
        sync();
#pragma unroll 1
        for (int k0 = 0; k0 < N; k0 += PB) {
            if (is_panel) {
                zc R[PB];
#pragma unroll
                for (int c = 0; c < PB; c++) R[c] = (tid < N && k0 + c < N) ? M[at(tid, k0 + c, N)] : zc{0, 0};
                bool mine = false;
#pragma unroll
                for (int c = 0; c < PB; c++) {
                    const int k = k0 + c, b = c & 1;
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
                    panel_sync();
                    int wb = 0;
                    if constexpr (PW > 1) {
                        unsigned long long bk = e.key[b][0];
#pragma unroll
                        for (int q = 1; q < PW; q++) {
                            const unsigned long long ck = e.key[b][q];
                            if (ck > bk) {
                                bk = ck;
                                wb = q;
                            }
                        }
                    }
                    const int p = e.idx[b][wb];
                    zc pinv = e.inv[b][wb];
                    // a pivot whose key is that of +0: singular from here on (every lane sees the same)
                    const bool zero = e.key[b][wb] == 1;
                    const int fz = e.first_zero;
                    if (zero || (fz != 0 && fz <= k)) pinv = zc{0, 0};
                    zc m = R[c] * pinv;
                    const bool is = tid == p;
                    R[c] = is ? zc{1, 0} : zc{0, 0};
                    if (is) {
                        open = false;
                        mine = true;
                        scale = pinv;
                        m = zc{0, 0};
                        e.perm[k] = (unsigned char)p;
                        e.step[p] = (unsigned char)k;
                        if (zero && fz == 0) e.first_zero = k + 1;
                    }
                    eliminate(R, c, m, e.row[b][wb]);
                }
                if (tid < N)
#pragma unroll
                    for (int c = 0; c < PB; c++)
                        if (k0 + c < N) M[at(tid, k0 + c, N)] = R[c];
                const unsigned u = __ballot_sync(0xffffffffu, mine);
                if (lane == 0) e.used[warp] = u;
            }
            sync();
            // the lane's places in the fragments of column tile 0: A(g, t4 [+ 4]), C(g, 2 t4 [+ 1])
            const int ld = smem_ld(N), kb = min(PB, N - k0);
            const int a0 = (g ^ xr(t4)) + t4 * ld, a1 = (g ^ xr(t4 + 4)) + (t4 + 4) * ld;
            const int e0 = (g ^ xr(2 * t4)) + 2 * t4 * ld, e1 = (g ^ xr(2 * t4 + 1)) + (2 * t4 + 1) * ld;
            const int p0 = t4 < kb ? e.perm[k0 + t4] : -1, p1 = t4 + 4 < kb ? e.perm[k0 + t4 + 4] : -1;
            for (int ct = warp; ct < ntiles; ct += W) {
                if (ct == k0 / PB) continue;
                const int j0 = 8 * ct;
                const zc v0 = p0 >= 0 ? M[j0 * ld + g * ld + (p0 ^ xr(g))] : zc{0, 0};
                const zc v1 = p1 >= 0 ? M[j0 * ld + g * ld + (p1 ^ xr(g))] : zc{0, 0};
                const double br[2] = {v0.x, v1.x}, bi[2] = {v0.y, v1.y}, nbi[2] = {-v0.y, -v1.y};
                __syncwarp();  // the fragments are read before other lanes of this warp rewrite the pivot rows
                const zc *Ap0 = M + k0 * ld + a0, *Ap1 = M + k0 * ld + a1;
                zc *Cp0 = M + j0 * ld + e0, *Cp1 = M + j0 * ld + e1;
#pragma unroll 2
                for (int rt = 0; rt < mtiles; rt++) {
                    const int i0 = 16 * rt;
                    const unsigned um = e.used[i0 >> 5] >> (i0 & 31);  // pivot rows of this tile
                    const bool ug = (um >> g) & 1, uh = (um >> (g + 8)) & 1, low = i0 + 8 < N;
                    const zc u0 = Ap0[i0], u1 = Ap0[i0 + 8], u2 = Ap1[i0], u3 = Ap1[i0 + 8];
                    const double ar[4] = {u0.x, u1.x, u2.x, u3.x}, ai[4] = {u0.y, u1.y, u2.y, u3.y};
                    const zc w0 = Cp0[i0], w1 = Cp1[i0], w2 = Cp0[i0 + 8], w3 = Cp1[i0 + 8];
                    double cr[4] = {ug ? 0.0 : w0.x, ug ? 0.0 : w1.x, uh ? 0.0 : w2.x, uh ? 0.0 : w3.x};
                    double ci[4] = {ug ? 0.0 : w0.y, ug ? 0.0 : w1.y, uh ? 0.0 : w2.y, uh ? 0.0 : w3.y};
                    dmma1688(cr, ar, br);
                    dmma1688(ci, ar, bi);
                    dmma1688(cr, ai, nbi);
                    dmma1688(ci, ai, br);
                    Cp0[i0] = zc{cr[0], ci[0]};
                    Cp1[i0] = zc{cr[1], ci[1]};
                    if (low) {  // (the last tile's lower half may lie in the next column)
                        Cp0[i0 + 8] = zc{cr[2], ci[2]};
                        Cp1[i0 + 8] = zc{cr[3], ci[3]};
                    }
                }
            }
            sync();
        }
        if (e.first_zero && tid == 0) {
            if (a.info) atomicMin(a.info, iw + 1);
            if (a.info_each) a.info_each[iw - a.iw0] = e.first_zero;
        }
        // scale the rows in place (their lanes know the factors), then write through the permutation
        if (is_panel && tid < N) {
            for (int j = 0; j < N; j++) {
                zc &m = M[at(tid, j, N)];
                m = m * scale;
            }
        }
        sync();
        const bool part = a.out_mode == 0 && !whole;  // the active block alone
        const int nout = part ? nA : N;
        zc *G = a.out_mode == 0 ? a.Gout + (size_t)iw * nout * nout : a.Gout + (size_t)(iw - a.iw0) * nout * nout;
        if (part) {
            for (int idx = tid; idx < nout * nout; idx += nthr) {
                G[idx] = M[at(e.perm[a.act[idx % nout]], e.step[a.act[idx / nout]], N)];
            }
        } else {
            int k = tid % N, c = tid / N;
#pragma unroll 4
            for (int idx = tid; idx < N * N; idx += nthr) {
                G[idx] = M[at(e.perm[k], e.step[c], N)];
                k += di;
                c += dj + (k >= N);
                k -= k >= N ? N : 0;
            }
        }
        sync();
    }
}

template <int PW, int W, int MPB, int MINB> int run(cudaStream_t st, const DysonArgs &a) {
    const void *fn = (const void *)dyson_blk<PW, W, MPB, MINB>;
    const size_t sm = sizeof(zc) * smem_units(a.N) * MPB;
    if (sm > 40 << 10) {
        const cudaError_t e = smem_cap(fn);
        if (e != cudaSuccess) return -(int)e;
    }
    const int need = (a.iw1 - a.iw0 + MPB - 1) / MPB;
    dyson_blk<PW, W, MPB, MINB><<<std::min(need, 148 * 16), 32 * W * MPB, sm, st>>>(a);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : -(int)e;
}

}  // namespace

int launch_dyson_blk(cudaStream_t st, const DysonArgs &a) {
    // warps: enough for the column tiles of an update in one or two rounds, few enough that several
    // blocks share an SM as long as their matrices fit
    const int N = a.N;
    if (N <= 32) return run<1, 1, 4, 5>(st, a);
    if (N <= 64) return run<2, 4, 1, 5>(st, a);
    if (N <= 80) return run<3, 8, 1, 2>(st, a);
    if (N <= 96) return run<3, 11, 1, 1>(st, a);
    return run<4, 15, 1, 1>(st, a);
}

}  // namespace qs
