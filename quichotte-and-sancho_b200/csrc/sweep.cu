// sweep.cu -- the energy sweep (sweep / G_at_energy, src/scf.f90:280-415) as batched
// kernels over the whole energy grid:
//   dyson_gj        G^r(w) = [hbar w - H + (i/2hbar)(GammaL+GammaR) - Sigma^r(w)]^-1 by
//                   in-place Gauss-Jordan elimination with partial pivoting for orders above
//                   256, one block per energy (invert_complex, common/linear_algebra.f90:58-88);
//                   dyson_blk.cu and dyson_l2.cu have the smaller ones
//   keldysh_scf2    G^< = G^r Sigma^< G^a on the active block as two complex GEMMs per
//                   energy, written straight into the SCF vector with its diagonals
//                   (modes M_INIT2 / M_SCF2, src/scf.f90:340-355), for blocks above 256 states;
//                   keldysh_sm.cu and keldysh_rows.cu have the smaller ones
//   final_outputs   modes M_SCF1 / M_FINAL (src/scf.f90:357-410): on-site and intra-atom
//                   blocks of G^<, Im G^r_ii, the current integrand
// plus the reductions over energies (equal_time_lesser, gather_onsite, gather_atoms,
// Current, the sanity sums) and the pack_gf / unpack_gf layout conversions.
#include <algorithm>
#include <cmath>
#include <mutex>

#include "qs_common.cuh"
#include "reduce.cuh"

namespace qs {


// ---------------------------------------------------------------------------------
// Block-wide argmax of cabs1 over rows k..N-1 of column k (first maximum wins, as
// LAPACK's izamax).
// ---------------------------------------------------------------------------------
__device__ __forceinline__ void warp_argmax(double &v, int &i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        double v2 = __shfl_down_sync(0xffffffffu, v, o);
        int i2 = __shfl_down_sync(0xffffffffu, i, o);
        if (v2 > v || (v2 == v && i2 < i)) {
            v = v2;
            i = i2;
        }
    }
}

__global__ void __launch_bounds__(512) dyson_gj(DysonArgs a) {
    const int N = a.N;
    __shared__ unsigned short perm[512];
    __shared__ double wv[16];
    __shared__ int wi[16];
    __shared__ int piv_s;
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int NG = nthr / N;  // threads per row in the update (>= 1, N <= 512)
    const int myrow = tid % N, mygrp = tid / N;
    const bool upd = mygrp < NG;

    for (int iw = a.iw0 + blockIdx.x; iw < a.iw1; iw += gridDim.x) {
        zc *M = a.inplace ? a.Gout + (size_t)(iw - a.iw0) * N * N : a.ws + (size_t)blockIdx.x * N * N;
        // ---- build w1 = Hemb - (Sig1 + Sigma2^r(w)) on act x act, + hbar w on the diagonal
        if (a.Ain && a.inplace) {  // the matrix is there
        } else if (a.Ain) {
            const zc *A = a.Ain + (size_t)(iw - a.iw0) * N * N;
            for (int idx = tid; idx < N * N; idx += nthr) M[idx] = A[idx];
        } else {
            const double w = a.omega[iw];
            const zc *SR = a.Sig + iw * a.sig_ld;
            for (int idx = tid; idx < N * N; idx += nthr) {
                int i = idx % N, j = idx / N;
                zc v = a.Hemb[idx];
                if (a.use_sigma) {
                    int pi = a.pos[i], pj = a.pos[j];
                    if (pi >= 0 && pj >= 0) {
                        zc s = a.Sig1[idx];
                        if (a.order2) s = s + sig_r(SR, pi, pj);
                        v = v - s;
                    }
                }
                if (i == j) v.x += w;
                M[idx] = v;
            }
        }
        __syncthreads();
        bool singular = false;
        int first_zero = 0;  // 1 + the first step with a zero pivot (LAPACK's INFO)
        // ---- Gauss-Jordan with row interchanges
        for (int k = 0; k < N; k++) {
            // pivot search
            double v = -1.0;
            int vi = N;
            for (int i = k + tid; i < N; i += nthr) {
                double c = cabs1(M[i + (size_t)k * N]);
                if (c > v) { v = c; vi = i; }
            }
            warp_argmax(v, vi);
            if ((tid & 31) == 0) { wv[tid >> 5] = v; wi[tid >> 5] = vi; }
            __syncthreads();
            if (tid < 32) {
                int nw = nthr >> 5;
                v = tid < nw ? wv[tid] : -1.0;
                vi = tid < nw ? wi[tid] : N;
                warp_argmax(v, vi);
                if (vi >= N) vi = k;  // no comparable entry (NaN column): keep row k, in range
                if (tid == 0) { piv_s = vi; perm[k] = vi; }
            }
            __syncthreads();
            const int p = piv_s;
            if (p != k) {
                for (int j = tid; j < N; j += nthr) {
                    zc t = M[k + (size_t)j * N];
                    M[k + (size_t)j * N] = M[p + (size_t)j * N];
                    M[p + (size_t)j * N] = t;
                }
                __syncthreads();
            }
            zc pivot = M[k + (size_t)k * N];
            if (pivot.x == 0.0 && pivot.y == 0.0) {
                if (!singular) first_zero = k + 1;
                singular = true;
            }
            zc inv = singular ? zc{0.0, 0.0} : crecip(pivot);
            zc f = upd ? M[myrow + (size_t)k * N] : zc{0.0, 0.0};
            __syncthreads();
            // scale the pivot row (M[k][k] is replaced by 1 first, so it ends as 1/pivot)
            for (int j = tid; j < N; j += nthr) {
                zc t = (j == k) ? zc{1.0, 0.0} : M[k + (size_t)j * N];
                M[k + (size_t)j * N] = t * inv;
            }
            __syncthreads();
            // rank-1 update of every other row (column k is replaced by 0 first)
            if (upd && myrow != k) {
                for (int j = mygrp; j < N; j += NG) {
                    zc t = (j == k) ? zc{0.0, 0.0} : M[myrow + (size_t)j * N];
                    zc r = M[k + (size_t)j * N];
                    t.x = fma(-f.x, r.x, t.x);
                    t.x = fma(f.y, r.y, t.x);
                    t.y = fma(-f.x, r.y, t.y);
                    t.y = fma(-f.y, r.x, t.y);
                    M[myrow + (size_t)j * N] = t;
                }
            }
            __syncthreads();
        }
        // undo the row interchanges by column interchanges in reverse order
        if (tid < N) {
            for (int k = N - 1; k >= 0; k--) {
                int p = perm[k];
                if (p != k) {
                    zc t = M[tid + (size_t)k * N];
                    M[tid + (size_t)k * N] = M[tid + (size_t)p * N];
                    M[tid + (size_t)p * N] = t;
                }
            }
        }
        __syncthreads();
        if (singular && tid == 0) {
            if (a.info) atomicMin(a.info, iw + 1);
            if (a.info_each) a.info_each[iw - a.iw0] = first_zero;
        }
        // ---- output
        if (a.inplace) {
        } else if (a.out_mode == 0) {
            const int nA = a.nA;
            zc *G = a.Gout + (size_t)iw * nA * nA;
            for (int idx = tid; idx < nA * nA; idx += nthr) {
                int p = idx % nA, q = idx / nA;
                G[idx] = M[a.act[p] + (size_t)a.act[q] * N];
            }
        } else {
            zc *G = a.Gout + (size_t)(iw - a.iw0) * N * N;
            for (int idx = tid; idx < N * N; idx += nthr) G[idx] = M[idx];
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------
// Block-level complex GEMM C(MxN) = A(MxK) B(KxN) over 32x32 output tiles, 256 threads,
// each thread 2x2 outputs. Operands come from loader functors; the store functor gets
// (i, j, value). With `upper`, tiles strictly below the diagonal are skipped.
// ---------------------------------------------------------------------------------
constexpr int TB = 32, TK = 16;

template <class LA, class LB, class ST>
__device__ void cta_gemm(int M, int N, int K, LA la, LB lb, ST st, zc *sA, zc *sB, bool upper) {
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int mt = (M + TB - 1) / TB, nt = (N + TB - 1) / TB;
    for (int tile = 0; tile < mt * nt; tile++) {
        const int bi = tile % mt, bj = tile / mt;
        if (upper && bi > bj) continue;
        zc acc[2][2] = {{{0, 0}, {0, 0}}, {{0, 0}, {0, 0}}};
        for (int k0 = 0; k0 < K; k0 += TK) {
            // sA[kk][r] (TK x TB), sB[kk][c] (TK x TB)
            for (int idx = tid; idx < TB * TK; idx += 256) {
                int r = idx % TB, kk = idx / TB;
                int i = bi * TB + r, k = k0 + kk;
                sA[kk * TB + r] = (i < M && k < K) ? la(i, k) : zc{0, 0};
            }
            for (int idx = tid; idx < TB * TK; idx += 256) {
                int kk = idx % TK, c = idx / TK;
                int j = bj * TB + c, k = k0 + kk;
                sB[kk * TB + c] = (j < N && k < K) ? lb(k, j) : zc{0, 0};
            }
            __syncthreads();
#pragma unroll
            for (int kk = 0; kk < TK; kk++) {
                zc a0 = sA[kk * TB + ty], a1 = sA[kk * TB + ty + 16];
                zc b0 = sB[kk * TB + tx], b1 = sB[kk * TB + tx + 16];
                cfma(acc[0][0], a0, b0);
                cfma(acc[0][1], a0, b1);
                cfma(acc[1][0], a1, b0);
                cfma(acc[1][1], a1, b1);
            }
            __syncthreads();
        }
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
                int i = bi * TB + ty + 16 * r, j = bj * TB + tx + 16 * c;
                if (i < M && j < N) st(i, j, acc[r][c]);
            }
    }
}

// element idx of an nA x nA matrix walked by 2x2 site blocks (rows fastest inside a block, then
// the blocks of a column): adjacent lanes touch whole 64-byte blocks of the packed layout and
// runs of the column-major one
__device__ __forceinline__ void block_order(int idx, int nA, int &i, int &j) {
    const int e = idx & 3, q = idx >> 2, s = nA >> 1;
    i = 2 * (q % s) + (e & 1);
    j = 2 * (q / s) + (e >> 1);
}

// modes M_INIT2 / M_SCF2: T = G^r SL, G^< = T G^r^dagger (upper triangle), packed.
__global__ void __launch_bounds__(256) keldysh_scf2(KeldyshArgs a) {
    __shared__ zc sA[TB * TK], sB[TB * TK];
    const int nA = a.nA, nfull = nA * nA;
    zc *T = a.Tws + (size_t)blockIdx.x * nfull;
    for (int iw = blockIdx.x; iw < a.n; iw += gridDim.x) {
        const zc *G = a.G + (size_t)iw * nfull;
        const double w = a.omega[iw];
        const double fL = fermi_d(w, *a.V, a.mu, a.beta), fR = fermi_d(w, 0.0, a.mu, a.beta);
        const zc *SL2 = a.Sig ? a.Sig + iw * a.sig_ld : nullptr;
        // SL = i (fL GamL_s + fR GamR_s) / hbar  (+ Sigma2^<)   (src/scf.f90:333-336)
        auto ldSL = [&](int k, int j) {
            size_t idx = k + (size_t)j * nA;
            zc g{fL * a.GamLs[idx].x + fR * a.GamRs[idx].x, fL * a.GamLs[idx].y + fR * a.GamRs[idx].y};
            zc s{-g.y, g.x};
            if (SL2) s = s + sig_l(SL2, k, j);
            return s;
        };
        cta_gemm(
            nA, nA, nA, [&](int i, int k) { return G[i + (size_t)k * nA]; }, ldSL,
            [&](int i, int j, zc v) { T[i + (size_t)j * nA] = v; }, sA, sB, false);
        __syncthreads();
        double *blk = a.out + (size_t)iw * a.nblk;
        const double *xb = a.xsub ? a.xsub + (size_t)iw * a.nblk : nullptr;
        cta_gemm(
            nA, nA, nA, [&](int i, int k) { return T[i + (size_t)k * nA]; },
            [&](int k, int j) { return conj(G[j + (size_t)k * nA]); },
            [&](int i, int j, zc v) {
                if (i < j) {
                    const int o = dl_l(i, j);
                    blk[o] = xb ? v.x - xb[o] : v.x;
                    blk[o + 1] = xb ? v.y - xb[o + 1] : v.y;
                } else if (i == j) {
                    const int o = dl_d(i);
                    blk[o] = xb ? v.y - xb[o] : v.y;
                    if (a.gLd) a.gLd[(size_t)iw * nA + i] = v;
                }
            },
            sA, sB, true);
        // G^r part of the block
        for (int idx = threadIdx.x; idx < nfull; idx += blockDim.x) {
            int i, j;
            block_order(idx, nA, i, j);
            const zc g = G[i + (size_t)j * nA];
            const int o = dl_r(i, j);
            blk[o] = xb ? g.x - xb[o] : g.x;
            blk[o + 1] = xb ? g.y - xb[o + 1] : g.y;
            if (i == j && a.gRd) a.gRd[(size_t)iw * nA + i] = g;
        }
        __syncthreads();
    }
}

// modes M_SCF1 and M_FINAL (src/scf.f90:357-410)
__global__ void __launch_bounds__(256) final_outputs(FinalArgs a) {
    __shared__ zc sA[TB * TK], sB[TB * TK];
    __shared__ zc Xs[32 * 32];  // nCL <= 32 (checked in qs_create)
    const int N = a.N, nS = a.nS;
    const bool fin = (a.mode == M_FINAL);
    const int Mrows = fin ? N : a.nA;
    zc *T = a.Tws + (size_t)blockIdx.x * Mrows * nS;
    for (int iw = a.iw0 + blockIdx.x; iw < a.iw1; iw += gridDim.x) {
        const zc *G = a.G + (size_t)(iw - a.iw0) * N * N;
        auto g = [&](int i, int j) { return G[i + (size_t)j * N]; };
        const double w = a.omega[iw];
        const double fL = fermi_d(w, a.V, a.mu, a.beta), fR = fermi_d(w, 0.0, a.mu, a.beta);
        const zc *SL2 = a.Sig ? a.Sig + iw * sig_stride(a.nA) : nullptr;
        auto ldSL = [&](int k, int j) {
            size_t idx = k + (size_t)j * nS;
            zc gg{fL * a.GamLs[idx].x + fR * a.GamRs[idx].x, fL * a.GamLs[idx].y + fR * a.GamRs[idx].y};
            zc s{-gg.y, gg.x};
            if (SL2) s = s + sig_l(SL2, k, j);
            return s;
        };
        // T = w1(rows, sup) SL
        cta_gemm(
            Mrows, nS, nS, [&](int i, int k) { return g(fin ? i : a.act[i], a.sup[k]); }, ldSL,
            [&](int i, int j, zc v) { T[i + (size_t)j * Mrows] = v; }, sA, sB, false);
        __syncthreads();
        // sum_q T(r, q) conj(w1(c, sup(q)))
        auto blkv = [&](int r, int c) {
            zc acc{0, 0};
            for (int q = 0; q < nS; q++) cfma_conj(acc, T[r + (size_t)q * Mrows], g(c, a.sup[q]));
            return acc;
        };
        if (fin) {
            for (int i = threadIdx.x; i < N; i += blockDim.x) a.dosd[(size_t)iw * N + i] = g(i, i).y;
            for (int t = threadIdx.x; t < 4 * a.N_sites; t += blockDim.x) {
                int s = t >> 2, e = t & 3, aa = e & 1, bb = e >> 1;
                a.onsL[(size_t)iw * 4 * a.N_sites + t] = blkv(2 * s + aa, 2 * s + bb);
            }
            if (a.atomL) {
                for (int at = 0; at < a.N_atoms; at++) {
                    int lo = 2 * (a.atom_first[at] - 1), m = 2 * a.atom_norb[at];
                    for (int t = threadIdx.x; t < m * m; t += blockDim.x) {
                        int aa = t % m, bb = t / m;
                        a.atomL[(size_t)iw * a.atomL_ld + a.atom_off[at] + t] = blkv(lo + aa, lo + bb);
                    }
                }
            }
            // current integrand through the left lead (src/scf.f90:390-409)
            const int nCL = a.nCL;
            for (int t = threadIdx.x; t < nCL * nCL; t += blockDim.x) {
                int k = t % nCL, aa = t / nCL;
                int ck = a.cl[k], ca = a.cl[aa];
                zc glc = blkv(ck, ca);
                zc gka = g(ck, ca), gak = conj(g(ca, ck));
                zc gg = glc + gka - gak;
                Xs[t] = zc{(fL - 1.0) * glc.x - fL * gg.x, (fL - 1.0) * glc.y - fL * gg.y};
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                zc tu{0, 0}, td{0, 0};
                for (int aa = 0; aa < nCL; aa++) {
                    zc mc{0, 0};
                    for (int k = 0; k < nCL; k++) cfma(mc, a.GamLcl[aa + (size_t)k * nCL], Xs[k + (size_t)aa * nCL]);
                    mc = zc{-mc.y, mc.x};
                    if ((a.cl[aa] & 1) == 0) tu = tu + mc;  // 0-based even = spin up
                    else td = td + mc;
                }
                a.trU[iw] = tu.x / (2.0 * PI);
                a.trD[iw] = td.x / (2.0 * PI);
            }
        } else {
            for (int k = threadIdx.x; k < a.nA; k += blockDim.x) {
                int ak = a.act[k];
                a.gRd[(size_t)iw * a.nA + k] = g(ak, ak);
                a.gLd[(size_t)iw * a.nA + k] = blkv(k, ak);
            }
            for (int t = threadIdx.x; t < 4 * a.N_sites; t += blockDim.x) {
                int s = t >> 2, e = t & 3, aa = e & 1, bb = e >> 1;
                if (!a.site_int[s]) continue;
                int lo = 2 * s, p1 = a.pos[lo];
                a.onsL[(size_t)iw * 4 * a.N_sites + t] = blkv(p1 + aa, lo + bb);
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------
// Reductions over energies: out[c] = sum_r A[r*ld + c], deterministic. CB columns (a power of
// two <= 32) x 256 / CB rows a step and block; gridDim.y blocks share the rows of a column group,
// and the last to arrive adds their partials. The first version gave a column group to one
// block: 16384 rows were then 2048 dependent steps (0.4 ms); measured now: 24 columns x 32768
// rows 0.51 ms -> 7 us.
// ---------------------------------------------------------------------------------
template <typename V>
__global__ void __launch_bounds__(256) colsum(const V *__restrict__ A, const V *__restrict__ B, int64_t ld, int ncols,
                                              int64_t nrows, int CB, V *__restrict__ out, V *__restrict__ part,
                                              int *__restrict__ cnt) {
    __shared__ V sh[256];
    const int cl = threadIdx.x & (CB - 1), c = blockIdx.x * CB + cl, rl = threadIdx.x / CB, R = 256 / CB;
    const int RB = gridDim.y, grp = blockIdx.z * gridDim.x + blockIdx.x;
    const V *src = blockIdx.z ? B : A;
    const int64_t per = (nrows + RB - 1) / RB, r0 = blockIdx.y * per, r1 = r0 + per < nrows ? r0 + per : nrows;
    // the block's sum of a value per thread over the threads of a column
    auto block_total = [&](V v) {
        sh[threadIdx.x] = v;
        __syncthreads();
        for (int w = R / 2; w > 0; w >>= 1) {
            if (rl < w) sh[threadIdx.x] = sh[threadIdx.x] + sh[threadIdx.x + w * CB];
            __syncthreads();
        }
        return sh[cl];
    };
    V acc{};
    if (c < ncols)
#pragma unroll 4
        for (int64_t r = r0 + rl; r < r1; r += R) acc = acc + src[r * ld + c];
    V tot = block_total(acc);
    if (RB > 1) {
        if (rl == 0) part[(grp * RB + blockIdx.y) * CB + cl] = tot;
        if (!last_block(cnt + grp, RB)) return;
        acc = V{};
        for (int b = rl; b < RB; b += R) acc = acc + part[(grp * RB + b) * CB + cl];
        tot = block_total(acc);
    }
    if (rl == 0 && c < ncols) out[blockIdx.z * ncols + c] = tot;
}

// The on-site sums that are the SCF vector at first order, in an order that does not depend on the grid: eight
// chains a column, rows r = 0..7 (mod 8) in turn, then the chains one after the other. Levels of width 1e-6 t turn the
// last bits of such a sum into 1e-10 of their spectra. A block has 4 columns: 256 threads bring tiles of 128 rows
// into shared memory, four under way, 32 of them add. Bound: the chains, one dependent addition for eight rows
// (40 cycles: 96 columns x 4001 energies 12 us, 24 x 32768 85 us, where colsum takes 6 and 12).
constexpr int SUM_COLS = 4, SUM_ROWS = 128, SUM_STAGES = 5;
__global__ void __launch_bounds__(256) chain_sums(const zc *__restrict__ A, int64_t ld, int ncols, int64_t nrows, zc *__restrict__ out) {
    __shared__ zc tile[SUM_STAGES][SUM_ROWS][SUM_COLS], chain[8][SUM_COLS];
    const int c0 = blockIdx.x * SUM_COLS, c = threadIdx.x % SUM_COLS, l = threadIdx.x / SUM_COLS;
    const int tiles = (int)((nrows + SUM_ROWS - 1) / SUM_ROWS);
    auto load = [&](int t) {
        if (t < tiles) {
            for (int r = l; r < SUM_ROWS; r += 256 / SUM_COLS) {
                const int64_t row = (int64_t)t * SUM_ROWS + r;
                const bool in = row < nrows && c0 + c < ncols;  // (else zero)
                const unsigned d = (unsigned)__cvta_generic_to_shared(&tile[t % SUM_STAGES][r][c]);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(in ? A + row * ld + c0 + c : A), "r"(in ? 16 : 0)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int t = 0; t < SUM_STAGES - 1; t++) load(t);
    zc acc{};
    for (int t = 0; t < tiles; t++) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(SUM_STAGES - 2) : "memory");
        __syncthreads();
        load(t + SUM_STAGES - 1);  // where tile t - 1 was
        if (l < 8) {
            const zc(*x)[SUM_COLS] = tile[t % SUM_STAGES];
#pragma unroll
            for (int r = 0; r < SUM_ROWS; r += 8) acc = acc + x[r + l][c];
        }
    }
    if (l < 8) chain[l][c] = acc;
    __syncthreads();
    if (l == 0 && c0 + c < ncols) {
        zc s = chain[0][c];
        for (int q = 1; q < 8; q++) s = s + chain[q][c];
        out[c0 + c] = s;
    }
}

int sum_in_order(qs_handle *h, const zc *d_A, int64_t ld, int ncols, int64_t nrows, zc *d_out) {
    if (ncols <= 0) return 0;
    int pi = prof_begin(h, K_REDUCE);
    chain_sums<<<(ncols + SUM_COLS - 1) / SUM_COLS, 256, 0, h->stream>>>(d_A, ld, ncols, nrows, d_out);
    prof_end(h, pi);
    QS_CUDA(h, cudaGetLastError());
    return 0;
}

namespace {
constexpr int PIN_SLOTS = 64, PIN_DOUBLES = 2560;
std::mutex g_pin_mu;
double *g_pin = nullptr;
bool g_pin_tried = false, g_pin_used[PIN_SLOTS];
}  // namespace

void host_scratch(qs_handle *h, int states) {
    const size_t need = 4 * (size_t)states + 1 + PIN_BROYDEN;
    h->pin_states = states;
    if (need <= PIN_DOUBLES) {
        std::lock_guard<std::mutex> lk(g_pin_mu);
        if (!g_pin_tried) {
            g_pin_tried = true;
            if (cudaHostAlloc((void **)&g_pin, sizeof(double) * PIN_SLOTS * PIN_DOUBLES, cudaHostAllocPortable) != cudaSuccess) {
                cudaGetLastError();
                g_pin = nullptr;
            }
        }
        for (int k = 0; g_pin && k < PIN_SLOTS; k++)
            if (!g_pin_used[k]) {
                g_pin_used[k] = true;
                h->pin = g_pin + (size_t)k * PIN_DOUBLES;
                return;
            }
    }
    h->pin_own.resize(need);
    h->pin = h->pin_own.data();
}

void host_scratch_release(qs_handle *h) {
    std::lock_guard<std::mutex> lk(g_pin_mu);
    if (g_pin && h->pin >= g_pin && h->pin < g_pin + (size_t)PIN_SLOTS * PIN_DOUBLES)
        g_pin_used[(h->pin - g_pin) / PIN_DOUBLES] = false;
    h->pin = nullptr;
}

int reduce_scratch(qs_handle *h, int states) {
    host_scratch(h, states);
    int rc = dalloc(h, (void **)&h->d_rpart, sizeof(double) * REDUCE_PART);
    return rc ? rc : dalloc(h, (void **)&h->d_rcnt, sizeof(int) * REDUCE_CNT);
}

template <typename V>
static int launch_colsum(qs_handle *h, const V *A, const V *B, int64_t ld, int ncols, int64_t nrows, V *out) {
    if (ncols <= 0) return 0;
    int CB = 1;
    while (CB < 32 && CB < ncols) CB *= 2;
    const int gx = (ncols + CB - 1) / CB, gz = B ? 2 : 1, R = 256 / CB;
    // at least eight rows a thread, at most four blocks an SM
    const int RB = (int)std::max<int64_t>(1, std::min<int64_t>((nrows + 8 * R - 1) / (8 * R), REDUCE_BLOCKS / (gx * gz)));
    int pi = prof_begin(h, K_REDUCE);
    colsum<V><<<dim3(gx, RB, gz), 256, 0, h->stream>>>(A, B, ld, ncols, nrows, CB, out, (V *)h->d_rpart, h->d_rcnt);
    prof_end(h, pi);
    QS_CUDA(h, cudaGetLastError());
    return 0;
}
int sum_over_energies(qs_handle *h, const zc *d_A, int64_t ld, int ncols, int64_t nrows, zc *d_out, const zc *d_B) {
    return launch_colsum<zc>(h, d_A, d_B, ld, ncols, nrows, d_out);
}
int sum_over_energies_real(qs_handle *h, const double *d_A, int64_t ld, int ncols, int64_t nrows, double *d_out) {
    return launch_colsum<double>(h, d_A, nullptr, ld, ncols, nrows, d_out);
}

// ---------------------------------------------------------------------------------
// pack_gf layout <-> device layout, per energy block of 3 nA^2 doubles through the table of
// positions (d_dl_perm, built in sigma2_setup)
// ---------------------------------------------------------------------------------
__global__ void ref_dl_perm(int64_t nblk, int64_t Nw, const int *__restrict__ perm, const double *__restrict__ src,
                            double *__restrict__ dst, int to_dl) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < Nw * nblk; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t w = t / nblk, d = w * nblk + perm[t - w * nblk];
        if (to_dl) dst[d] = src[t];
        else dst[t] = src[d];
    }
}

int convert_ref_to_dl(qs_handle *h, const double *ref, double *dl) {
    count_launch();
    ref_dl_perm<<<1184, 256, 0, h->stream>>>(h->nblk, h->n, h->d_dl_perm, ref, dl, 1);
    return (int)cudaGetLastError();
}
int convert_dl_to_ref(qs_handle *h, const double *dl, double *ref) {
    count_launch();
    ref_dl_perm<<<1184, 256, 0, h->stream>>>(h->nblk, h->n, h->d_dl_perm, dl, ref, 0);
    return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------------
constexpr int GJ_THREADS = 512;  // the unblocked kernel, N <= 512

// Up to 80 states several matrices share an SM's memory (dyson_blk: 64 x 4000 0.79 ms, dyson_l2 0.82; 80 x 148 0.09
// and 0.13, if 80 x 4000 1.52 and 1.42). From there to DYSON_SMEM_MAXN dyson_blk holds one matrix an SM, the faster
// form while there is one for each SM at most (96 x 148 0.121 ms, dyson_l2 0.164; 120 x 170 0.342 and
// 0.300, 96 x 4000 3.21 and 1.91); it is also the one that needs no workspace when G is a part of the matrix.
static int run_dyson(cudaStream_t st, const DysonArgs &a) {
    if (a.N <= 80 || (dyson_fits_smem(a.N) && (!a.inplace || a.iw1 - a.iw0 <= 148))) return launch_dyson_blk(st, a);
    if (dyson_l2_fits(a.N)) return launch_dyson_l2(st, a);
    dyson_gj<<<std::min(a.iw1 - a.iw0, DYSON_L2_SLOTS), GJ_THREADS, 0, st>>>(a);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : -(int)e;
}

static int launch_dyson(qs_handle *h, DysonArgs &a) {
    int pi = prof_begin(h, K_DYSON);
    // in global memory the matrices are built and inverted where G goes if G has their order: one
    // copy less, and no slot that the next matrix of the block waits for
    a.inplace = a.out_mode == 1 || a.nA == a.N;
    a.ws = h->d_Gws;
    const int rc = run_dyson(h->stream, a);
    prof_end(h, pi);
    QS_CUDA(h, (cudaError_t)-rc);
    return 0;
}

int invert_batched_dev(cudaStream_t st, int N, int batch, zc *d_A, int *d_min, int *d_each, bool zero_of_inf) {
    DysonArgs a{};
    a.N = N;
    a.iw1 = batch;
    a.Ain = d_A;
    a.out_mode = 1;
    a.Gout = d_A;
    a.info = d_min;
    a.info_each = d_each;
    a.inplace = 1;
    a.zero_of_inf = zero_of_inf || N < 16;
    count_launch();
    return run_dyson(st, a);
}

int set_voltage(qs_handle *h, double V) {
    if (V == h->V_dev) return 0;
    QS_CUDA(h, cudaMemcpyAsync(h->d_V, &V, sizeof(double), cudaMemcpyHostToDevice, h->stream));
    h->V_dev = V;
    return 0;
}

// final_rows (keldysh_rows.cu): every state active, the left contact states within one block of 32 rows
static bool final_rows_fits(const qs_handle *h, int mode) {
    return mode == M_FINAL && h->order == 2 && h->nA == h->Norb && h->nS == h->Norb && keldysh_rows_fits(h->Norb) &&
           (h->cl.empty() || h->cl.front() / 32 == h->cl.back() / 32);
}

// sweep(mode) over all energies (src/scf.f90:280-290).
//   M_INIT2 / M_SCF2: output into d_out (SCF vector, DL); M_SCF2 subtracts d_x.
//   M_SCF1 / M_FINAL: per-energy arrays of the handle.
int sweep(qs_handle *h, int mode, double V, bool use_sigma, double *d_out, const double *d_x, bool fp32) {
    const int N = h->Norb, nA = h->nA, n = h->n;
    DysonArgs a{};
    a.N = N;
    a.nA = nA;
    a.Hemb = h->d_Hemb;
    a.Sig1 = h->d_Sig1;
    a.Sig = h->d_Sig;
    a.sig_ld = sig_stride(nA);
    a.pos = h->d_pos;
    a.act = h->d_act;
    a.omega = h->d_omega;
    a.use_sigma = use_sigma;
    a.order2 = (h->order == 2);
    a.info = h->d_info;
    a.zero_of_inf = N < 16;
    int rc;
    if (mode == M_INIT2 || mode == M_SCF2) {
        a.iw0 = 0;
        a.iw1 = n;
        a.out_mode = 0;
        a.Gout = h->d_G;
        // one form per order
        const int form = dyson_l2_fits(N) ? DYSON_BLOCKED : DYSON_UNBLOCKED;
        rc = tune_launch(h, TUNE_DYSON, tune_key(N, n), &form, 1, form, [&](int) { return launch_dyson(h, a); });
        if (rc) return rc;
        KeldyshArgs k{};
        k.nA = nA;
        k.n = n;
        k.nblk = h->nblk;
        k.G = h->d_G;
        k.Sig = (use_sigma && h->order == 2) ? h->d_Sig : nullptr;
        k.sig_ld = sig_stride(nA);
        k.GamLs = h->d_GamLs;
        k.GamRs = h->d_GamRs;
        k.omega = h->d_omega;
        if ((rc = set_voltage(h, V))) return rc;
        k.V = h->d_V;
        k.mu = h->mu;
        k.beta = h->beta;
        k.out = d_out;
        k.xsub = (mode == M_SCF2) ? d_x : nullptr;
        k.gRd = h->d_gRd;
        k.gLd = h->d_gLd;
        k.Tws = h->d_T;
        k.err = h->d_info + 1;
        k.cidx = h->d_kd_cidx;
        k.nc = (h->nS == nA) ? h->kd_nc : -1;
        auto launch_k = [&](int v) -> int {
            if (v == KELDYSH_TF32) return launch_keldysh_tf32(h, k);
            if (v == KELDYSH_TC) return keldysh_sm_fits(nA) ? launch_keldysh_sm(h, k) : launch_keldysh_rows(h, k);
            int pi = prof_begin(h, K_KELDYSH);
            keldysh_scf2<<<(int)std::min<size_t>(h->T_slots, (size_t)n), 256, 0, h->stream>>>(k);
            prof_end(h, pi);
            QS_CUDA(h, cudaGetLastError());
            return 0;
        };
        // one FP64 form per order
        const int fp64 = keldysh_rows_fits(nA) ? KELDYSH_TC : KELDYSH_CUDA;
        // the FP32 phase of a QS_PREC_MIXED solve: the 3xTF32 kernel on the fifth-generation
        // tensor cores is a candidate too, kept only where it is the fastest
        if (fp32 && mode == M_SCF2 && keldysh_tf32_fits(nA)) {
            const int c3[2] = {KELDYSH_TF32, fp64};
            return tune_launch(h, TUNE_KELDYSH32, tune_key(nA, n), c3, 2, fp64, launch_k);
        }
        return tune_launch(h, TUNE_KELDYSH, tune_key(nA, n), &fp64, 1, fp64, launch_k);
    }
    // chunked full inversion + per-energy outputs
    const int Mrows = (mode == M_FINAL) ? N : nA;
    for (int iw0 = 0; iw0 < n; iw0 += (int)h->G_chunk) {
        int iw1 = std::min(n, iw0 + (int)h->G_chunk);
        a.iw0 = iw0;
        a.iw1 = iw1;
        a.out_mode = 1;
        a.Gout = h->d_G;
        if ((rc = launch_dyson(h, a))) return rc;
        FinalArgs f{};
        f.N = N;
        f.nS = h->nS;
        f.nA = nA;
        f.nCL = h->nCL;
        f.N_sites = h->N_sites;
        f.N_atoms = h->N_atoms;
        f.iw0 = iw0;
        f.iw1 = iw1;
        f.mode = mode;
        f.G = h->d_G;
        f.sup = h->d_sup;
        f.act = h->d_act;
        f.pos = h->d_pos;
        f.cl = h->d_cl;
        f.site_int = h->d_site_int;
        f.atom_first = h->d_atom_first;
        f.atom_norb = h->d_atom_norb;
        f.atom_off = h->d_atom_off;
        f.GamLs = h->d_GamLs;
        f.GamRs = h->d_GamRs;
        f.GamLcl = h->d_GamLcl;
        f.Sig = (use_sigma && h->order == 2) ? h->d_Sig : nullptr;
        f.omega = h->d_omega;
        f.V = V;
        f.mu = h->mu;
        f.beta = h->beta;
        f.Tws = h->d_T;
        f.dosd = h->d_dosd;
        f.trU = h->d_trU;
        f.trD = h->d_trD;
        f.onsL = h->d_onsL;
        f.atomL = h->has_atomL ? h->d_atomL : nullptr;
        f.atomL_ld = h->has_atomL ? h->atom_off.back() : 0;
        f.gRd = h->d_gRd;
        f.gLd = h->d_gLd;
        f.cidx = h->d_kd_cidx;
        f.nc = h->kd_nc;
        if (final_rows_fits(h, mode)) {
            if ((rc = launch_final_rows(h, f))) return rc;
            continue;
        }
        size_t per = (size_t)Mrows * h->nS;
        int nb = (int)std::min<size_t>(std::min<size_t>(h->T_bytes / (sizeof(zc) * std::max<size_t>(per, 1)), 148 * 8),
                                       (size_t)(iw1 - iw0));
        nb = std::max(nb, 1);
        int pi = prof_begin(h, K_FINAL);
        final_outputs<<<nb, 256, 0, h->stream>>>(f);
        prof_end(h, pi);
        QS_CUDA(h, cudaGetLastError());
    }
    return 0;
}

}  // namespace qs
