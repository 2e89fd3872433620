// keldysh_rows.cu -- the Keldysh step of the sweep (modes M_INIT2 / M_SCF2, src/scf.f90:333-355) for
// active blocks of 81 to 256 states: G^< = G^r SL G^r^dagger with SL = i (f_L Gamma_L + f_R Gamma_R) +
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
// scratch matrices), 192 x 1201 10.1 -> 5.0 ms (32x32-tile CUDA-core GEMMs), the tensor pipe 69 % busy.
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

__global__ void __launch_bounds__(512, 1) keldysh_rows(KeldyshArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned char contact[256];  // 1 + index of a contact state, 0 for the others
    const int N = a.nA, tid = threadIdx.x, nthr = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3, nw = nthr >> 5;
    const int nk = (N + 7) / 8, nrb = (N + RB - 1) / RB;
    const int iw = blockIdx.x / nrb, r0 = RB * (blockIdx.x % nrb), rows = min(RB, N - r0), mrows = (rows + 15) / 16;
    const bool corr = a.nc >= 0 && a.nc <= NC_CORR;  // else the leads enter as a matrix
    zc *P = (zc *)smem_raw;                           // rows r0 .. r0 + 31 of G^r, then of T: (r, k) at at(r, k, RB)
    const zc *G = a.G + (size_t)iw * N * N;
    const zc *SL = a.Sig ? a.Sig + iw * a.sig_ld : nullptr;
    const double w = a.omega[iw];
    const double fL = fermi_d(w, a.V, a.mu, a.beta), fR = fermi_d(w, 0.0, a.mu, a.beta);
    auto lead = [&](int k, int j) {
        const zc gl = a.GamLs[k + j * N], gr = a.GamRs[k + j * N];
        return zc{-(fL * gl.y + fR * gr.y), fL * gl.x + fR * gr.x};
    };
    for (int k = warp; k < 8 * nk; k += nw) {
        if (lane < rows && k < N) cpa16(&P[at(lane, k, RB)], G + r0 + lane + k * N);
        else P[at(lane, k, RB)] = zc{0, 0};  // rows and columns beyond N: zero operands
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (int i = tid; i < 256; i += nthr) contact[i] = 0;
    __syncthreads();
    if (corr && tid < a.nc) contact[a.cidx[tid]] = (unsigned char)(tid + 1);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    double *blk = a.out + (size_t)iw * a.nblk;
    const double *xb = a.xsub ? a.xsub + (size_t)iw * a.nblk : nullptr;
    // ---- G^r minus x, by 2x2 site blocks: a warp takes the rows' 16 blocks of a site column as two
    // halves, four columns at a time
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
    // ---- T = G SL; the k steps: all, or those with a contact if T has only their columns
    const unsigned all = nk == 32 ? 0xffffffffu : (1u << nk) - 1;
    unsigned kmask = all;
    if (!SL && corr) {
        kmask = 0;
        for (int q = 0; q < a.nc; q++) kmask |= 1u << (a.cidx[q] >> 3);
    }
    double cr[CT][2][4], ci[CT][2][4];
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
                for (int q = 0; q < a.nc; q++) {
                    const int k = a.cidx[q];
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

}  // namespace

bool keldysh_rows_fits(int nA) { return nA <= 256; }

int launch_keldysh_rows(qs_handle *h, const KeldyshArgs &k) {
    const int nk = (k.nA + 7) / 8, nrb = (k.nA + RB - 1) / RB;
    QS_CUDA(h, smem_cap((const void *)keldysh_rows));
    int pi = prof_begin(h, K_KELDYSH);
    keldysh_rows<<<k.n * nrb, 32 * ((nk + CT - 1) / CT), sizeof(zc) * RB * 8 * nk, h->stream>>>(k);
    prof_end(h, pi);
    QS_CUDA(h, cudaGetLastError());
    return 0;
}

}  // namespace qs
