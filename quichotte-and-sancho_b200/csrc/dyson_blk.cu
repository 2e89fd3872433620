// dyson_blk.cu -- G^r(w) = [hbar w - H + (i/2hbar)(GammaL+GammaR) - Sigma^r(w)]^-1 for every energy, and
// batched inversion (invert_complex, common/linear_algebra.f90:58-88): blocked in-place Gauss-Jordan
// elimination with partial pivoting in shared memory, one matrix per warp (N <= 32) or block
// (N <= 120).
//
// Panels of 16 columns K = [k0, k0 + 16), the k extent of an FP64 tensor-core product:
//   panel   PW = ceil(N / 32) warps hold one row of the panel per lane in registers (gauss.cuh). Per column
//           every warp finds its best row (integer warp reductions on the bits of |Re| + |Im|) and
//           publishes that row and its reciprocal; after one barrier every warp picks the best
//           warp's, divides it, a value a lane, and every lane eliminates its own row
//   update  every other column tile j (8 columns) by one warp, complex products of four real DMMAs:
//           A[i, j] = (i a pivot row of the panel ? 0 : A[i, j]) + sum_t A[i, K_t] A[p_t, j],
//           with the pivot rows A[p_t, j] read into registers first
// Rows are never exchanged: a row is used once, as pivot row p_k of step k. With the pivot on
// (p_k, k) elimination exchanges y_{p_k} and x_k, so that in the end row p_k holds row k of the
// inverse and column k its column p_k; the output is written through that permutation.
//
// The operations on a value are those of the elimination with row exchanges in panels of 16, bit for bit. Panels of 8
// with undivided pivot rows took 0.41 ms where these take 0.48 (24 x 32768; 48 x 4000 0.33 and 0.41, 80 x 4096 1.32
// and 1.55), but rounded differently: spectra of 48 first-order states moved by up to 2e-9 (their sharp levels are
// not determined better), and results are to stay what they were.
//
// Bound: the chain of a panel's column (search, row, barrier, reciprocal, division, 64 DFMA); the
// update runs at the FP64 rate. Small matrices share an SM (16 of order 24, 4 of order 40; the panel's
// registers), so that panels and updates of different ones overlap.
//
// Measured on B200, batched inversion, against the elimination with row exchanges (one block a matrix, or
// everything through a global workspace): as Dyson of 48 states x 4001 energies 1.58 -> 0.41 ms, 40 x 5003
// 0.99 -> 0.41, 24 x 32768 3.05 -> 0.48, 120 x 148 0.18 ms.
// Tried instead: the whole matrix in registers, rank-1 updates (4-9 TFLOP/s: the per-step work of every
// warp, column and row exchange and selects, outweighs the update); the pivot row taken over by selects
// instead of a branch (24 x 32768 0.53 ms); its division by the candidate lane before the barrier (0.49).
#include <algorithm>
#include <climits>

#include "gauss.cuh"
#include "zmma.cuh"

namespace qs {
namespace {

template <int PW, int NBUF> struct Exchange : PanelExchange<PW, NBUF> {
    unsigned used[PW];                            // rows (bits) that became pivot rows in this panel
    unsigned char step[32 * PW];  // step of a pivot row
};

// PW panel warps, W warps a matrix, MPB matrices a block (more than one only for W = 1).
template <int PW, int W, int MPB, int MINB, int NBUF>
__global__ void __launch_bounds__(32 * W * MPB, MINB) dyson_blk(DysonArgs a) {
    static_assert(MPB == 1 || W == 1, "several matrices a block: one warp each");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ Exchange<PW, NBUF> exs[MPB];
    const int N = a.N, nA = a.nA, slot = W == 1 ? threadIdx.x >> 5 : 0, tid = W == 1 ? threadIdx.x & 31 : threadIdx.x;
    constexpr int nthr = 32 * W;
    const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    Exchange<PW, NBUF> &e = exs[slot];
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
                bool with[NB], diag[NB];
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
                    diag[u] = i == j;
                    i += di;
                    j += dj + (i >= N);
                    i -= i >= N ? N : 0;
                }
#pragma unroll
                for (int u = 0; u < NB; u++) {
                    if (with[u]) v[u] = v[u] - (a.Sig1[idx + u * nthr] + sg[u]);
                    if (diag[u]) v[u].x += w;
                    if (at_s[u] >= 0) M[at_s[u]] = v[u];
                }
            }
        }
        // the columns that pad the last tile: zero operands (rows beyond N reach rows beyond N only)
        for (int t = N * smem_ld(N) + tid; t < smem_units(N); t += nthr) M[t] = zc{0, 0};
        if (tid == 0) e.first_zero = 0;
        const bool is_panel = warp < PW;
        int place = tid;  // of this lane's row
        sync();
#pragma unroll 1
        for (int k0 = 0; k0 < N; k0 += PB) {
            const int kb = min(PB, N - k0);
            if (is_panel) {
                const bool mine = eliminate_panel(e, PW, tid, N, k0, kb, place, a.zero_of_inf, [&](int c) { return M + at(tid, k0 + c, N); },
                                                  panel_sync);
                if (mine) e.step[tid] = (unsigned char)place;
                const unsigned u = __ballot_sync(0xffffffffu, mine);
                if (lane == 0) e.used[warp] = u;
            }
            sync();
            // the lane's places in the fragments of column tile 0: A(g, t4 [+ 4]), C(g, 2 t4 [+ 1])
            const int ld = smem_ld(N);
            const int a0 = (g ^ xr(t4)) + t4 * ld, a1 = (g ^ xr(t4 + 4)) + (t4 + 4) * ld;
            const int e0 = (g ^ xr(2 * t4)) + 2 * t4 * ld, e1 = (g ^ xr(2 * t4 + 1)) + (2 * t4 + 1) * ld;
            int p[4];
#pragma unroll
            for (int q = 0; q < 4; q++) p[q] = t4 + 4 * q < kb ? e.perm[k0 + t4 + 4 * q] : -1;
            for (int ct = warp; ct < ntiles; ct += W) {
                const int j0 = 8 * ct;
                if (j0 >= k0 && j0 < k0 + kb) continue;
                zc v[4];
#pragma unroll
                for (int q = 0; q < 4; q++) v[q] = p[q] >= 0 ? M[j0 * ld + g * ld + (p[q] ^ xr(g))] : zc{0, 0};
                __syncwarp();  // the fragments are read before other lanes of this warp rewrite the pivot rows
                const zc *Ap0 = M + k0 * ld + a0, *Ap1 = M + k0 * ld + a1;
                zc *Cp0 = M + j0 * ld + e0, *Cp1 = M + j0 * ld + e1;
#pragma unroll 1
                for (int rt = 0; rt < mtiles; rt++) {
                    const int i0 = 16 * rt;
                    const unsigned um = e.used[i0 >> 5] >> (i0 & 31);  // pivot rows of this tile
                    const bool ug = (um >> g) & 1, uh = (um >> (g + 8)) & 1, low = i0 + 8 < N;
                    const zc w0 = Cp0[i0], w1 = Cp1[i0], w2 = Cp0[i0 + 8], w3 = Cp1[i0 + 8];
                    double cr[4] = {ug ? 0.0 : w0.x, ug ? 0.0 : w1.x, uh ? 0.0 : w2.x, uh ? 0.0 : w3.x};
                    double ci[4] = {ug ? 0.0 : w0.y, ug ? 0.0 : w1.y, uh ? 0.0 : w2.y, uh ? 0.0 : w3.y};
                    zmma_panel(cr, ci, Ap0 + i0, Ap1 + i0, ld, v, kb > 8);
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
        // through the permutation
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

template <int PW, int W, int MPB, int MINB, int NBUF> int run(cudaStream_t st, const DysonArgs &a) {
    const void *fn = (const void *)dyson_blk<PW, W, MPB, MINB, NBUF>;
    const size_t sm = sizeof(zc) * smem_units(a.N) * MPB;
    if (sm > 40 << 10) {
        const cudaError_t e = smem_cap(fn);
        if (e != cudaSuccess) return -(int)e;
    }
    const int need = (a.iw1 - a.iw0 + MPB - 1) / MPB;
    dyson_blk<PW, W, MPB, MINB, NBUF><<<std::min(need, 148 * 16), 32 * W * MPB, sm, st>>>(a);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : -(int)e;
}

}  // namespace

int launch_dyson_blk(cudaStream_t st, const DysonArgs &a) {
    // warps: enough for the column tiles of an update in one or two rounds, few enough that several
    // blocks share an SM as long as their matrices fit
    const int N = a.N;
    if (N <= 32) return run<1, 1, 4, 4, 2>(st, a);
    if (N <= 64) return run<2, 4, 1, 4, 2>(st, a);
    if (N <= 80) return run<3, 8, 1, 2, 2>(st, a);
    if (N <= 96) return run<3, 11, 1, 1, 2>(st, a);
    return run<4, 15, 1, 1, 1>(st, a);
}

}  // namespace qs
