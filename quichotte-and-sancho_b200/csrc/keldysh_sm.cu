// keldysh_sm.cu -- the Keldysh step of the sweep (modes M_INIT2 / M_SCF2, src/scf.f90:333-355) for
// active blocks up to 48: G^< = G^r SL G^r^dagger with SL = i (f_L Gamma_L + f_R Gamma_R) + Sigma2^<,
// written with G^r into the packed vector minus x.
//
// One block per energy with G^r and SL in shared memory, both products on the FP64 tensor cores:
//   T = G SL      a warp computes an 8-column tile of T for all rows and writes it over the same
//                 columns of SL, which no other warp reads
//   G^< = T G^+   the 16 x 8 tiles that touch the upper triangle, shared out over the warps, straight
//                 to the output (their x values are loaded before the products)
// Sigma2^< is stored as its upper site blocks; the lower ones are filled in on the way into shared
// memory, and the lead matrices are added on the contact states only.
// Bound: HBM (G^r, Sigma^<, x in, F out: 72 nA^2 bytes) and the FP64 rate (12 nA^3 flops) are close to
// each other at these orders; several blocks share an SM, so that one's loads and stores overlap
// another's products. Measured on B200 per launch, against 32x32-tile CUDA-core GEMMs through a
// scratch matrix: 24 states x 32768 energies 1.45 -> 0.55 ms, 40 x 5003 0.89 -> 0.28, 16 x 4096
// 0.10 -> 0.039.
#include <algorithm>

#include "zmma.cuh"

namespace qs {
namespace {

__device__ __forceinline__ void cpa16(void *dst, const void *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

// MT = row tiles (16 rows) of the block; blockDim = 32 x column tiles (8 columns)
template <int MT, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) keldysh_sm(KeldyshArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int N = a.nA, tid = threadIdx.x, nthr = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3, nt = (N + 7) / 8;
    const int ld = smem_ld(N), nw = nthr >> 5, sites = N / 2, nk = nt;  // k steps of 8
    zc *G = (zc *)smem_raw, *S = G + smem_units(N);
    // rows and columns beyond N stay zero, so that the k loops need no bounds (rows of results
    // beyond N are not stored)
    for (int t = tid; t < 2 * smem_units(N); t += nthr) G[t] = zc{0, 0};
    // the lane's places in the fragments: A(g + .., k = t4 [+ 4] + ..) of G or S, B(k, g + ..) of S
    const int a0 = (g ^ xr(t4)) + t4 * ld, a1 = (g ^ xr(t4 + 4)) + (t4 + 4) * ld;
    const int b0 = (t4 ^ xr(g)) + g * ld, b1 = ((t4 + 4) ^ xr(g)) + g * ld;
    const int e0 = (g ^ xr(2 * t4)) + 2 * t4 * ld, e1 = (g ^ xr(2 * t4 + 1)) + (2 * t4 + 1) * ld;  // C(g + .., 2 t4 [+ 1])
    __syncthreads();
    for (int iw = blockIdx.x; iw < a.n; iw += gridDim.x) {
        const zc *Gg = a.G + (size_t)iw * N * N;
        const double w = a.omega[iw];
        const double fL = fermi_d(w, *a.V, a.mu, a.beta), fR = fermi_d(w, 0.0, a.mu, a.beta);
        for (int j = warp; j < N; j += nw)
            for (int i = lane; i < N; i += 32) cpa16(&G[at(i, j, N)], Gg + i + j * N);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        if (a.Sig) {
            // site pairs I <= J, four lanes each: an element (i, j) and its mirror image
            for (int J = warp; J < sites; J += nw) {
                const zc *Sg = a.Sig + iw * a.sig_ld + sig_block(0, J) + 8;
                for (int t = lane; t < 4 * (J + 1); t += 32) {
                    const int I = t >> 2, i = 2 * I + (t & 1), j = 2 * J + ((t >> 1) & 1);
                    const zc v = Sg[12 * I + (t & 3)];
                    S[at(i, j, N)] = v;
                    if (I < J) S[at(j, i, N)] = zc{-v.x, v.y};
                }
            }
        } else {
            for (int j = warp; j < N; j += nw)
                for (int i = lane; i < N; i += 32) S[at(i, j, N)] = zc{0, 0};
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        // the leads: the contact states' block, or everything when they are not known
        const int nc = a.nc >= 0 ? a.nc : N;
        for (int t = tid; t < nc * nc; t += nthr) {
            const int i = a.nc >= 0 ? a.cidx[t % nc] : t % nc, j = a.nc >= 0 ? a.cidx[t / nc] : t / nc;
            const zc gl = a.GamLs[i + j * N], gr = a.GamRs[i + j * N], s = S[at(i, j, N)];
            S[at(i, j, N)] = zc{s.x - (fL * gl.y + fR * gr.y), s.y + (fL * gl.x + fR * gr.x)};
        }
        __syncthreads();
        // ---- T = G SL, columns 8 warp .. 8 warp + 7, in place of SL
        {
            const int j0 = 8 * warp;
            double cr[MT][4], ci[MT][4];
#pragma unroll
            for (int m = 0; m < MT; m++)
#pragma unroll
                for (int q = 0; q < 4; q++) cr[m][q] = ci[m][q] = 0.0;
            const zc *Ap0 = G + a0, *Ap1 = G + a1, *Bp0 = S + j0 * ld + b0, *Bp1 = S + j0 * ld + b1;
#pragma unroll 1
            for (int kc = 0; kc < nk; kc++) {
                const zc v0 = *Bp0, v1 = *Bp1;
                const double br[2] = {v0.x, v1.x}, bi[2] = {v0.y, v1.y}, nbi[2] = {-v0.y, -v1.y};
#pragma unroll
                for (int m = 0; m < MT; m++) {
                    const zc u0 = Ap0[16 * m], u1 = Ap0[16 * m + 8], u2 = Ap1[16 * m], u3 = Ap1[16 * m + 8];
                    const double ar[4] = {u0.x, u1.x, u2.x, u3.x}, ai[4] = {u0.y, u1.y, u2.y, u3.y};
                    dmma1688(cr[m], ar, br);
                    dmma1688(ci[m], ar, bi);
                    dmma1688(cr[m], ai, nbi);
                    dmma1688(ci[m], ai, br);
                }
                Ap0 += 8 * ld;
                Ap1 += 8 * ld;
                Bp0 += 8;
                Bp1 += 8;
            }
            __syncwarp();
#pragma unroll
            for (int m = 0; m < MT; m++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int dr = 16 * m + 8 * (q >> 1), c = j0 + 2 * t4 + (q & 1);
                    if (dr + g < N && c < N) S[j0 * ld + dr + ((q & 1) ? e1 : e0)] = zc{cr[m][q], ci[m][q]};
                }
        }
        __syncthreads();
        double *blk = a.out + (size_t)iw * a.nblk;
        const double *xb = a.xsub ? a.xsub + (size_t)iw * a.nblk : nullptr;
        // ---- the upper triangle of T G^+: tile u in column-major order of the tiles (rt <= (8 ct + 7) / 16)
        int rt = warp, ct = 0;
        for (;;) {
            while (ct < nt && rt >= min((8 * ct + 7) / 16 + 1, (N + 15) / 16)) {
                rt -= min((8 * ct + 7) / 16 + 1, (N + 15) / 16);
                ct++;
            }
            if (ct >= nt) break;
            const int r0 = 16 * rt, c0 = 8 * ct;
            zc xv[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int r = r0 + g + 8 * (q >> 1), c = c0 + 2 * t4 + (q & 1);
                xv[q] = zc{0, 0};
                if (xb && c < N) {
                    if (r < c) xv[q] = *(const zc *)(xb + dl_l(r, c));
                    else if (r == c) xv[q].y = xb[dl_d(r)];
                }
            }
            double cr[4] = {0, 0, 0, 0}, ci[4] = {0, 0, 0, 0};
            const zc *Ap0 = S + r0 + a0, *Ap1 = S + r0 + a1, *Bp0 = G + c0 + a0, *Bp1 = G + c0 + a1;  // B(k, n) = conj G(n, k)
#pragma unroll 2
            for (int kc = 0; kc < nk; kc++) {
                const zc v0 = *Bp0, v1 = *Bp1, u0 = Ap0[0], u1 = Ap0[8], u2 = Ap1[0], u3 = Ap1[8];
                const double br[2] = {v0.x, v1.x}, bi[2] = {-v0.y, -v1.y}, nbi[2] = {v0.y, v1.y};
                const double ar[4] = {u0.x, u1.x, u2.x, u3.x}, ai[4] = {u0.y, u1.y, u2.y, u3.y};
                dmma1688(cr, ar, br);
                dmma1688(ci, ar, bi);
                dmma1688(cr, ai, nbi);
                dmma1688(ci, ai, br);
                Ap0 += 8 * ld;
                Ap1 += 8 * ld;
                Bp0 += 8 * ld;
                Bp1 += 8 * ld;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int r = r0 + g + 8 * (q >> 1), c = c0 + 2 * t4 + (q & 1);
                if (c >= N || r > c) continue;
                if (r < c) {
                    *(zc *)(blk + dl_l(r, c)) = zc{cr[q] - xv[q].x, ci[q] - xv[q].y};
                } else {
                    blk[dl_d(r)] = ci[q] - xv[q].y;
                    if (a.gLd) a.gLd[(size_t)iw * N + r] = zc{cr[q], ci[q]};
                }
            }
            rt += nthr >> 5;
        }
        // ---- G^r minus x, by 2x2 site blocks
        for (int J = warp; J < sites; J += nw)
            for (int t = lane; t < 4 * sites; t += 32) {
                const int i = 2 * (t >> 2) + (t & 1), j = 2 * J + ((t >> 1) & 1), o = dl_r(i, j);
                const zc v = G[at(i, j, N)];
                *(zc *)(blk + o) = xb ? v - *(const zc *)(xb + o) : v;
                if (i == j && a.gRd) a.gRd[(size_t)iw * N + i] = v;
            }
        __syncthreads();  // G and SL are reloaded for the next energy
    }
}

template <int MT, int MAXT, int MINB> int run(qs_handle *h, const KeldyshArgs &k) {
    const void *fn = (const void *)keldysh_sm<MT, MAXT, MINB>;
    const size_t sm = 2 * sizeof(zc) * smem_units(k.nA);
    QS_CUDA(h, smem_cap(fn));
    const int thr = 32 * ((k.nA + 7) / 8);
    int pi = prof_begin(h, K_KELDYSH);
    keldysh_sm<MT, MAXT, MINB><<<std::min(k.n, 148 * 16), thr, sm, h->stream>>>(k);
    prof_end(h, pi);
    QS_CUDA(h, cudaGetLastError());
    return 0;
}

}  // namespace

// above, blocks of 32 rows are faster: one energy's two matrices leave room for one or two blocks an SM
// (per launch, 4096 energies: 48 states 0.32 ms here, 0.39 by rows; 56 0.74 and 0.53; 80 1.43 and 1.22)
bool keldysh_sm_fits(int nA) { return nA <= 48; }

int launch_keldysh_sm(qs_handle *h, const KeldyshArgs &k) {
    switch ((k.nA + 15) / 16) {
        case 1: return run<1, 64, 12>(h, k);
        case 2: return run<2, 128, 7>(h, k);
        default: return run<3, 192, 3>(h, k);
    }
}

}  // namespace qs
