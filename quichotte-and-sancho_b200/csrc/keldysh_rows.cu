// keldysh_rows.cu -- products with the rows of T = G^r SL in shared memory: the outputs of the final sweep
// (final_rows, below) and the Keldysh step of the sweep (modes M_INIT2 / M_SCF2, src/scf.f90:333-355) for
// active blocks of 49 to 256 states: G^< = G^r SL G^r^dagger with SL = i (f_L Gamma_L + f_R Gamma_R) +
// Sigma2^<, written with G^r into the packed vector minus x.
//
// One block per (energy, 32 rows). The rows of G^r are held in shared memory for all k, the other operand
// streams from L2 straight into fragment registers, one k step of 8 ahead (a fragment has one user, and
// the tensor instructions of a step take longer than an L2 load), so a product has no barrier inside:
//   T = G SL      for the 32 rows, two 8-column tiles a warp; T overwrites the rows of G^r
//   G^< = T G^+   for the column tiles that touch the upper triangle
// The lead matrices are non-zero on the contact states only: their term is added to those columns of T.
// Without Sigma2^< (the non-interacting start) T has no other columns, and both products skip the k
// steps without a contact.
//
// Bound: FP64 rate (12 nA^3 flops an energy against 72 nA^2 bytes). Blocks of one energy follow each
// other, so G^r and Sigma^< come from L2; two blocks share an SM up to 128 states, so that one's copies
// and stores overlap another's products. Measured on B200 per launch: 120 states x 4096 energies
// 5.1 -> 4.5 ms (one block an SM with 16-deep panels of both operands in shared memory, SL and T through
// scratch matrices), 192 x 1201 10.1 -> 5.0 ms (32x32-tile CUDA-core GEMMs), the tensor pipe 69 % busy;
// 64 x 4096 0.84 -> 0.61, 80 x 4096 1.43 -> 1.22 (one energy a block with both operands in shared memory).
// Touching a loaded value (its sign) before the step that uses it cost 30 %.
#include <algorithm>

#include "zmma.cuh"

namespace qs {
namespace {

constexpr int RB = 32;        // rows a block: two row tiles
constexpr int CT = 2;         // column tiles a warp
constexpr int NC_CORR = 16;   // contact states up to which the lead term is a correction of T

__device__ __forceinline__ void cpa16(void *dst, const void *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

// C(32 rows, CT column tiles) = A B over the k steps of kmask: A from the panel, the lane's two
// values of B(k step, column tile u) as fix(kc, u, half, value loaded from at(kc, u, half)). The loads are
// of the next step and are not touched before it, so that nothing waits for them. mt[u] row
// tiles of column tile u are needed.
template <class AT, class FIX>
__device__ __forceinline__ void panel_product(const zc *P, unsigned kmask, const int (&mt)[CT], AT from, FIX fix,
                                              double (&cr)[CT][2][4], double (&ci)[CT][2][4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int a0 = (g ^ xr(t4)) + t4 * RB, a1 = (g ^ xr(t4 + 4)) + (t4 + 4) * RB;
#pragma unroll
    for (int u = 0; u < CT; u++)
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int q = 0; q < 4; q++) cr[u][m][q] = ci[u][m][q] = 0.0;
    const int mtop = max(mt[0], mt[1]);
    if (mtop == 0 || kmask == 0) return;
    zc next[CT][2];
    int kc = __ffs(kmask) - 1;
#pragma unroll
    for (int u = 0; u < CT; u++)
#pragma unroll
        for (int hh = 0; hh < 2; hh++) next[u][hh] = *from(kc, u, hh);
#pragma unroll 1
    for (;;) {
        kmask &= kmask - 1;
        const int kn = kmask ? __ffs(kmask) - 1 : kc;
        zc v[CT][2];
#pragma unroll
        for (int u = 0; u < CT; u++)
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
                v[u][hh] = fix(kc, u, hh, next[u][hh]);
                next[u][hh] = *from(kn, u, hh);
            }
#pragma unroll
        for (int m = 0; m < 2; m++) {
            if (m >= mtop) break;
            const zc *Ap0 = P + 8 * kc * RB + 16 * m + a0, *Ap1 = P + 8 * kc * RB + 16 * m + a1;
            const zc u0 = Ap0[0], u1 = Ap0[8], u2 = Ap1[0], u3 = Ap1[8];
            const double ar[4] = {u0.x, u1.x, u2.x, u3.x}, ai[4] = {u0.y, u1.y, u2.y, u3.y};
// the column tiles in turn: an instruction that adds to the same accumulators is four away
#pragma unroll
            for (int part = 0; part < 2; part++)
#pragma unroll
                for (int u = 0; u < CT; u++) {
                    const double br[2] = {v[u][0].x, v[u][1].x}, bi[2] = {v[u][0].y, v[u][1].y};
                    const double nbi[2] = {-v[u][0].y, -v[u][1].y};
                    if (m >= mt[u]) continue;
                    if (part == 0) {
                        dmma1688(cr[u][m], ar, br);
                        dmma1688(ci[u][m], ar, bi);
                    } else {
                        dmma1688(cr[u][m], ai, nbi);
                        dmma1688(ci[u][m], ai, br);
                    }
                }
        }
        if (!kmask) break;
        kc = kn;
    }
}

// The rows r0 .. r0 + 31 of T = G SL in the panel P ((r, k) at at(r, k, RB)), with hook() called while it holds
// those of G. kmask: the k steps in which T has columns other than zero; cr, ci are scratch.
template <class HOOK>
__device__ __forceinline__ void rows_of_T(zc *P, unsigned char (&contact)[256], int N, int r0, const zc *G, const zc *SL,
                                          const zc *GamLs, const zc *GamRs, const int *cidx, int nc, double fL, double fR,
                                          unsigned &kmask, double (&cr)[CT][2][4], double (&ci)[CT][2][4], HOOK hook) {
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3, nw = nthr >> 5;
    const int nk = (N + 7) / 8, rows = min(RB, N - r0), mrows = (rows + 15) / 16;
    const bool corr = nc >= 0 && nc <= NC_CORR;  // else the leads enter as a matrix
    auto lead = [&](int k, int j) {
        const zc gl = GamLs[k + j * N], gr = GamRs[k + j * N];
        return zc{-(fL * gl.y + fR * gr.y), fL * gl.x + fR * gr.x};
    };
    for (int k = warp; k < 8 * nk; k += nw) {
        if (lane < rows && k < N) cpa16(&P[at(lane, k, RB)], G + r0 + lane + k * N);
        else P[at(lane, k, RB)] = zc{0, 0};  // rows and columns beyond N: zero operands
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (int i = tid; i < 256; i += nthr) contact[i] = 0;
    __syncthreads();
    if (corr && tid < nc) contact[cidx[tid]] = 1;
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    hook();
    // the k steps: all, or those with a contact if T has only their columns
    const unsigned all = nk == 32 ? 0xffffffffu : (1u << nk) - 1;
    kmask = all;
    if (!SL && corr) {
        kmask = 0;
        for (int q = 0; q < nc; q++) kmask |= 1u << (cidx[q] >> 3);
    }
    {
        int mt[CT];
#pragma unroll
        for (int u = 0; u < CT; u++) mt[u] = (warp + u * nw < nk && (SL || !corr)) ? mrows : 0;
        // (beyond N the last element is loaded, and replaced by zero)
        panel_product(
            P, kmask, mt,
            [&](int kc, int u, int hh) {
                const int j = min(8 * (warp + u * nw) + g, N - 1), k = min(8 * kc + 4 * hh + t4, N - 1);
                return SL ? sig_l_at(SL, k, j) : G;
            },
            [&](int kc, int u, int hh, zc v) {
                const int j = 8 * (warp + u * nw) + g, k = 8 * kc + 4 * hh + t4;
                if ((k >> 1) > (j >> 1)) v.x = -v.x;
                if (!SL || j >= N || k >= N) v = zc{0, 0};
                if (!corr && j < N && k < N) v = v + lead(k, j);
                return v;
            },
            cr, ci);
    }
    if (corr) {
#pragma unroll
        for (int u = 0; u < CT; u++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int c = 8 * (warp + u * nw) + 2 * t4 + e;
                if (c >= N || !contact[c]) continue;
                for (int q = 0; q < nc; q++) {
                    const int k = cidx[q];
                    const zc l = lead(k, c);
#pragma unroll
                    for (int m = 0; m < 2; m++)
#pragma unroll
                        for (int hh = 0; hh < 2; hh++) {
                            zc v{cr[u][m][2 * hh + e], ci[u][m][2 * hh + e]};
                            cfma(v, P[at(16 * m + 8 * hh + g, k, RB)], l);
                            cr[u][m][2 * hh + e] = v.x;
                            ci[u][m][2 * hh + e] = v.y;
                        }
                }
            }
    }
    __syncthreads();  // every warp has read the rows of G^r
#pragma unroll
    for (int u = 0; u < CT; u++)
        if (warp + u * nw < nk)
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int q = 0; q < 4; q++)
                    P[at(16 * m + 8 * (q >> 1) + g, 8 * (warp + u * nw) + 2 * t4 + (q & 1), RB)] = zc{cr[u][m][q], ci[u][m][q]};
    __syncthreads();
}

__global__ void __launch_bounds__(512, 1) keldysh_rows(KeldyshArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned char contact[256];  // 1 for a contact state
    const int N = a.nA, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3, nw = blockDim.x >> 5;
    const int nk = (N + 7) / 8, nrb = (N + RB - 1) / RB;
    const int iw = blockIdx.x / nrb, r0 = RB * (blockIdx.x % nrb), rows = min(RB, N - r0), mrows = (rows + 15) / 16;
    zc *P = (zc *)smem_raw;
    const zc *G = a.G + (size_t)iw * N * N;
    const double w = a.omega[iw];
    double *blk = a.out + (size_t)iw * a.nblk;
    const double *xb = a.xsub ? a.xsub + (size_t)iw * a.nblk : nullptr;
    // G^r minus x, by 2x2 site blocks: a warp takes the rows' 16 blocks of a site column as two
    // halves, four columns at a time
    auto pack = [&]() {
        for (int J0 = warp; J0 < N / 2; J0 += 4 * nw) {
            zc xv[8];
            int o[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int J = J0 + (u >> 1) * nw, i = 16 * (u & 1) + 2 * (lane >> 2) + (lane & 1), j = 2 * J + ((lane >> 1) & 1);
                o[u] = i < rows && J < N / 2 ? dl_r(r0 + i, j) : -1;
                xv[u] = xb && o[u] >= 0 ? *(const zc *)(xb + o[u]) : zc{0, 0};
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                if (o[u] < 0) continue;
                const int J = J0 + (u >> 1) * nw, i = 16 * (u & 1) + 2 * (lane >> 2) + (lane & 1), j = 2 * J + ((lane >> 1) & 1);
                const zc v = P[at(i, j, RB)];
                *(zc *)(blk + o[u]) = v - xv[u];
                if (r0 + i == j && a.gRd) a.gRd[(size_t)iw * N + j] = v;
            }
        }
    };
    unsigned kmask;
    double cr[CT][2][4], ci[CT][2][4];
    rows_of_T(P, contact, N, r0, G, a.Sig ? a.Sig + iw * a.sig_ld : nullptr, a.GamLs, a.GamRs, a.cidx, a.nc,
              fermi_d(w, *a.V, a.mu, a.beta), fermi_d(w, 0.0, a.mu, a.beta), kmask, cr, ci, pack);
    // ---- G^< = T G^+ in the column tiles from the diagonal on
    int mt[CT];
#pragma unroll
    for (int u = 0; u < CT; u++) {
        const int ct = r0 / 8 + warp + u * nw;
        mt[u] = ct >= nk ? 0 : 8 * ct + 7 < r0 + 16 ? 1 : mrows;
    }
    panel_product(
        P, kmask, mt,
        [&](int kc, int u, int hh) {
            const int j = min(r0 + 8 * (warp + u * nw) + g, N - 1), k = min(8 * kc + 4 * hh + t4, N - 1);
            return G + j + k * N;
        },
        [&](int kc, int u, int hh, zc v) {
            const int j = r0 + 8 * (warp + u * nw) + g, k = 8 * kc + 4 * hh + t4;
            return j < N && k < N ? conj(v) : zc{0, 0};
        },
        cr, ci);
#pragma unroll
    for (int u = 0; u < CT; u++)
#pragma unroll
        for (int m = 0; m < 2; m++) {
            if (m >= mt[u]) continue;
            int o[4];
            zc xv[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int r = r0 + 16 * m + 8 * (q >> 1) + g, c = r0 + 8 * (warp + u * nw) + 2 * t4 + (q & 1);
                o[q] = c >= N || r > c ? -1 : r < c ? dl_l(r, c) : dl_d(r);
                xv[q] = zc{0, 0};
                if (xb && o[q] >= 0) {
                    if (r < c) xv[q] = *(const zc *)(xb + o[q]);
                    else xv[q].y = xb[o[q]];
                }
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int r = r0 + 16 * m + 8 * (q >> 1) + g, c = r0 + 8 * (warp + u * nw) + 2 * t4 + (q & 1);
                if (o[q] < 0) continue;
                if (r < c) {
                    *(zc *)(blk + o[q]) = zc{cr[u][m][q] - xv[q].x, ci[u][m][q] - xv[q].y};
                } else {
                    blk[o[q]] = ci[u][m][q] - xv[q].y;
                    if (a.gLd) a.gLd[(size_t)iw * N + r] = zc{cr[u][m][q], ci[u][m][q]};
                }
            }
        }
}

// mode M_FINAL (src/scf.f90:357-410) where every state is active: the blocks of G^< that the outputs need are dot
// products of rows of T and of G, four lanes each. The block whose rows hold the left contact states does the
// current integrand. Per launch, against one block an energy with CUDA-core tiles and T in global scratch:
// 24 states x 32768 energies 0.98 -> 0.53 ms, 40 x 5003 0.65 -> 0.27, 120 x 4096 5.7 -> 2.5, 192 x 1201 6.7 -> 3.0.
__global__ void __launch_bounds__(512, 1) final_rows(FinalArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned char contact[256];
    __shared__ double Xs[32 * 32];  // nCL <= 32 (checked in qs_create)
    const int N = a.N, tid = threadIdx.x, nthr = blockDim.x, nrb = (N + RB - 1) / RB;
    const int iw = a.iw0 + blockIdx.x / nrb, r0 = RB * (blockIdx.x % nrb), rows = min(RB, N - r0);
    zc *P = (zc *)smem_raw;
    const zc *G = a.G + (size_t)(iw - a.iw0) * N * N;
    const double w = a.omega[iw];
    const double fL = fermi_d(w, a.V, a.mu, a.beta), fR = fermi_d(w, 0.0, a.mu, a.beta);
    unsigned kmask;
    double cr[CT][2][4], ci[CT][2][4];
    rows_of_T(P, contact, N, r0, G, a.Sig ? a.Sig + iw * sig_stride(N) : nullptr, a.GamLs, a.GamRs, a.cidx, a.nc, fL, fR,
              kmask, cr, ci, [&]() {
                  for (int i = tid; i < rows; i += nthr) a.dosd[(size_t)iw * N + r0 + i] = P[at(i, r0 + i, RB)].y;
              });
    // G^<(r, c), r = r0 + i; all four lanes of a group get it
    const int sub = tid & 3;
    auto dot = [&](int i, int c) {
        zc v{0, 0};
#pragma unroll 4
        for (int q = sub; q < N; q += 4) cfma_conj(v, P[at(i, q, RB)], G[c + q * N]);
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        }
        return v;
    };
    // the groups of a warp stay together: the last ones repeat an entry
    auto each = [&](int count, auto entry) {
        for (int t0 = tid >> 5 << 3; t0 < count; t0 += nthr >> 2) {
            const int t = t0 + ((tid & 31) >> 2);
            entry(min(t, count - 1), t < count && sub == 0);
        }
    };
    each(2 * rows, [&](int t, bool keep) {
        const int s = (r0 >> 1) + (t >> 2), aa = t & 1, bb = (t >> 1) & 1;
        const zc v = dot(2 * (t >> 2) + aa, 2 * s + bb);
        if (keep) a.onsL[(size_t)iw * 4 * a.N_sites + 4 * s + aa + 2 * bb] = v;
    });
    if (a.atomL) {
        for (int k = 0; k < a.N_atoms; k++) {
            const int lo = 2 * (a.atom_first[k] - 1), m = 2 * a.atom_norb[k];
            const int b0 = max(lo, r0), b1 = min(lo + m, r0 + rows);  // its rows in this block
            if (b0 >= b1) continue;
            each((b1 - b0) * m, [&](int t, bool keep) {
                const int r = b0 + t % (b1 - b0), c = lo + t / (b1 - b0);
                const zc v = dot(r - r0, c);
                if (keep) a.atomL[(size_t)iw * a.atomL_ld + a.atom_off[k] + (r - lo) + (c - lo) * m] = v;
            });
        }
    }
    // current integrand through the left lead (src/scf.f90:390-409)
    const int nCL = a.nCL;
    if (nCL == 0 ? r0 != 0 : a.cl[0] / RB != r0 / RB) return;
    if (nCL > 0)
        each(nCL * nCL, [&](int t, bool keep) {
            const int k = t % nCL, aa = t / nCL, ck = a.cl[k], ca = a.cl[aa];
            const zc glc = dot(ck - r0, ca), gg = glc + G[ck + ca * N] - conj(G[ca + ck * N]);
            const zc x{(fL - 1.0) * glc.x - fL * gg.x, (fL - 1.0) * glc.y - fL * gg.y};
            const zc m = a.GamLcl[aa + k * nCL] * x;
            if (keep) Xs[t] = -m.y;  // Re i GammaL x
        });
    __syncthreads();
    if (tid < 2) {  // spin up: even states
        double tr = 0;
        for (int aa = 0; aa < nCL; aa++)
            if ((a.cl[aa] & 1) == tid)
                for (int k = 0; k < nCL; k++) tr += Xs[k + aa * nCL];
        (tid ? a.trD : a.trU)[iw] = tr / (2.0 * PI);
    }
}

}  // namespace

static int rows_threads(int N) { return 32 * (((N + 7) / 8 + CT - 1) / CT); }
static size_t rows_smem(int N) { return sizeof(zc) * RB * 8 * ((N + 7) / 8); }


bool keldysh_rows_fits(int nA) { return nA <= 256; }

int launch_keldysh_rows(qs_handle *h, const KeldyshArgs &k) {
    const int nrb = (k.nA + RB - 1) / RB;
    QS_CUDA(h, smem_cap((const void *)keldysh_rows));
    int pi = prof_begin(h, K_KELDYSH);
    keldysh_rows<<<k.n * nrb, rows_threads(k.nA), rows_smem(k.nA), h->stream>>>(k);
    prof_end(h, pi);
    QS_CUDA(h, cudaGetLastError());
    return 0;
}

int launch_final_rows(qs_handle *h, const FinalArgs &f) {
    QS_CUDA(h, smem_cap((const void *)final_rows));
    int pi = prof_begin(h, K_FINAL);
    final_rows<<<(f.iw1 - f.iw0) * ((f.N + RB - 1) / RB), rows_threads(f.N), rows_smem(f.N), h->stream>>>(f);
    prof_end(h, pi);
    QS_CUDA(h, cudaGetLastError());
    return 0;
}

}  // namespace qs
