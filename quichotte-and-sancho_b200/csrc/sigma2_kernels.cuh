// sigma2_kernels.cuh -- the three FFT kernels of the second-order self-energies
// (sigma2_compute, src/self_energies.f90:135-219), templates over the element type and the
// length of the transform; sigma2.cu describes the method and chooses the instances.
#pragma once
#include "fft.cuh"
#include "sigma2.cuh"

namespace qs {

// resident blocks an SM asked of the register allocator: a radix-R1 butterfly holds 4 R1 registers
// of data, and the kernels are bound by the memory latency they can hide
constexpr int s2_minb(int R1) { return R1 <= 8 ? 4 : R1 <= 12 ? 3 : 2; }

constexpr int S2_E = 12;  // complex values of a site pair: R_IJ, R_JI, L_IJ (2x2 blocks, rows fastest)

// ---------------------------------------------------------------------------------
// Kernel A: forward length-N1 transforms of the zero-padded energies, and the twiddle
// W_Nf^{m2 l1}. Item = one site pair x GA adjacent m2 (w = N2 m1 + m2), items with the pair
// fastest: the blocks in flight read neighbouring 192-byte pieces of the same energies.
//   pass 1 reads X straight into registers (192-byte runs, every load of a butterfly in
//   flight), pass 2 writes Y straight from registers (runs of GA x 192 bytes: whole lines)
// Bound: HBM (reads n, writes Nf values of each of the 12 sequences, zero padding not read).
// ---------------------------------------------------------------------------------
template <typename T, int R1, int R2>
__global__ void __launch_bounds__(S2_THREADS, s2_minb(R1)) sig2_fwdA(Sig2A a) {
    constexpr int N1 = R1 * R2, GA = S2_GA, W = GA * S2_E;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx<T> *S = (cplx<T> *)smem_raw;  // [position][m2][e]
    cplx<T> *twL = S + N1 * W;         // W_N1^m
    cplx<T> *twC = twL + N1;           // W_Nf^{m2 l1} of the item's m2: [l1][m2]
    int twm = -1;                      // the m20 they are for
    for (int m = threadIdx.x; m < N1; m += blockDim.x) twL[m] = cvt<T>(a.tw[m * a.N2]);
    __syncthreads();
    for (int it = blockIdx.x; it < a.nitems; it += gridDim.x) {
        const int ip = it % a.npairs, m20 = (it / a.npairs) * GA;
        const int2 pr = a.pairs[ip];
        const bool diag = pr.x == pr.y;
        if (m20 != twm) {
            for (int t = threadIdx.x; t < N1 * GA; t += blockDim.x) twC[t] = cvt<T>(a.tw[(m20 + t % GA) * (t / GA)]);
            twm = m20;
        }
        const double *base = a.X + dl_block(pr.x, pr.y);
        for (int idx = threadIdx.x; idx < W * R2; idx += blockDim.x) {
            const int e = idx % S2_E, g = (idx / S2_E) % GA, j = idx / W;
            const int64_t w0 = (int64_t)a.N2 * j + m20 + g;
            cplx<T> v[R1];
            if (!diag) {
#pragma unroll
                for (int r = 0; r < R1; r++) {
                    const int64_t w = w0 + (int64_t)a.N2 * R2 * r;
                    v[r] = w < a.n ? cvt<T>(*(const zc *)(base + w * a.nblk + 2 * e)) : cplx<T>{0, 0};
                }
            } else {
                // R twice (R_JI = R_IJ), then L_00, L_10 = -conj L_01, L_01, L_11 from L_01 and the two Im L_ii
#pragma unroll
                for (int r = 0; r < R1; r++) {
                    const int64_t w = w0 + (int64_t)a.N2 * R2 * r;
                    zc x{0, 0};
                    if (w < a.n) {
                        const double *b = base + w * a.nblk;
                        if (e < 8) x = *(const zc *)(b + 2 * (e & 3));
                        else if (e == 8) x.y = b[10];
                        else if (e == 11) x.y = b[11];
                        else {
                            x = *(const zc *)(b + 8);
                            if (e == 9) x.x = -x.x;
                        }
                    }
                    v[r] = cvt<T>(x);
                }
            }
            dft<T, R1, -1>(v);
            S[j * W + idx % W] = v[0];
#pragma unroll
            for (int q = 1; q < R1; q++) S[(q * R2 + j) * W + idx % W] = v[q] * twL[j * q];
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < W * R1; idx += blockDim.x) {
            const int e = idx % S2_E, g = (idx / S2_E) % GA, k = idx / W;
            cplx<T> v[R2];
#pragma unroll
            for (int j = 0; j < R2; j++) v[j] = S[(k * R2 + j) * W + idx % W];
            dft<T, R2, -1>(v);
            const int m2 = m20 + g;
            cplx<T> *y = (cplx<T> *)a.Y + ((size_t)ip * N1 * a.N2 + m2) * S2_E + e;
#pragma unroll
            for (int t = 0; t < R2; t++) {
                const int l1 = k + R1 * t;
                y[(size_t)l1 * a.N2 * S2_E] = v[t] * twC[l1 * GA + g];
            }
        }
        __syncthreads();  // S is rewritten by the next item
    }
}

// 2x2 complex blocks
template <typename T> struct B2 { cplx<T> a[2][2]; };
template <typename T> __device__ __forceinline__ B2<T> mm2(const B2<T> &X, const B2<T> &Y) {
    B2<T> Z;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            Z.a[i][j] = X.a[i][0] * Y.a[0][j];
            cfma(Z.a[i][j], X.a[i][1], Y.a[1][j]);
        }
    return Z;
}
template <typename T> __device__ __forceinline__ B2<T> dag2(const B2<T> &X) {
    B2<T> Z;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) Z.a[i][j] = conj(X.a[j][i]);
    return Z;
}
// adj2 (src/self_energies.f90:222-228): Tr(M) 1 - M
template <typename T> __device__ __forceinline__ B2<T> adj2(const B2<T> &M) {
    B2<T> A;
    A.a[0][0] = M.a[1][1];
    A.a[0][1] = -M.a[0][1];
    A.a[1][0] = -M.a[1][0];
    A.a[1][1] = M.a[0][0];
    return A;
}
template <typename T> __device__ __forceinline__ cplx<T> det2(const B2<T> &M) {
    cplx<T> d = M.a[0][0] * M.a[1][1];
    cfma(d, -M.a[0][1], M.a[1][0]);
    return d;
}
// det(X + Y) - det X - det Y
template <typename T> __device__ __forceinline__ cplx<T> polar2(const B2<T> &X, const B2<T> &Y) {
    cplx<T> d = X.a[0][0] * Y.a[1][1];
    cfma(d, X.a[1][1], Y.a[0][0]);
    cfma(d, -X.a[0][1], Y.a[1][0]);
    cfma(d, -X.a[1][0], Y.a[0][1]);
    return d;
}

// The per-frequency algebra of src/self_energies.f90:175-199 for a pair (I, J): from
// r = R_IJ(l), L = L_IJ(l) and rp = R_JI(-l) the outputs sR_IJ(l), sL_IJ(l) and sR_JI(-l).
// With a_IJ(l) = rp^+, a_JI(-l) = r^+, L_JI(-l) = -L^+ and G = L + r - a the reference forms
//   sR_IJ = r adj(L_JI G_IJ) + L adj(L_JI r + a_JI L),   sL_IJ = L adj(G_JI L).
// adj is linear and adj(XY) = adj(Y) adj(X), X adj(X) = det(X) 1, and X adj(Y) + Y adj(X) is
// the scalar polar2(X, Y), so that
//   sR_IJ = [(det r + polar(r, L)) 1 - r adj(a_IJ)] adj(L_JI) + det(L) adj(a_JI),
//   sL_IJ = det(L) adj(G_JI),
// and sR_JI(-l) likewise with the two sites exchanged; sL_JI(-l) = -sL_IJ(l)^+ needs no
// computation (Sigma^< is anti-Hermitian). 58 complex products instead of 112.
template <typename T>
__device__ __forceinline__ void pair_algebra(const B2<T> &r, const B2<T> &rp, const B2<T> &L, B2<T> &sR, B2<T> &sRp,
                                             B2<T> &sL) {
    const B2<T> ar = adj2(dag2(r)), arp = adj2(dag2(rp)), aL = adj2(L), Ld = dag2(L), aLd = adj2(Ld);
    const cplx<T> dL = det2(L), dLc = conj(dL);
    {
        const cplx<T> s = det2(r) + polar2(r, L);
        B2<T> M = mm2(r, arp);
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) M.a[i][j] = (i == j) ? M.a[i][j] - s : M.a[i][j];  // r adj(a_IJ) - s, times adj(L^+)
        sR = mm2(M, aLd);
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) cfma(sR.a[i][j], dL, ar.a[i][j]);
    }
    {
        const cplx<T> s = det2(rp) - polar2(rp, Ld);
        B2<T> M = mm2(rp, ar);
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) M.a[i][j] = (i == j) ? s - M.a[i][j] : -M.a[i][j];
        sRp = mm2(M, aL);
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) cfma(sRp.a[i][j], dLc, arp.a[i][j]);
    }
    // G_JI(-l) = -(L + r - rp^+)^+ = rp - r^+ - L^+
    B2<T> G;
    const B2<T> rd = dag2(r);
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) G.a[i][j] = rp.a[i][j] - rd.a[i][j] - Ld.a[i][j];
    const B2<T> aG = adj2(G);
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) sL.a[i][j] = dL * aG.a[i][j];
}

// ---------------------------------------------------------------------------------
// Kernel B: the spectra (length-N2 transforms over m2), the 2x2 algebra, the inverse length-N2
// transforms, in place in Y. Item = one site pair and the column pair {c, N1 - c}: the partner
// -l of a frequency l = l1 + N1 l2 lies in the other column, and one thread's task (a
// frequency l) reads R_IJ(l), L_IJ(l) and R_JI(-l) and writes its three outputs over them, so
// the whole item lives in one buffer. Pass 2 leaves the spectrum in the order it reads
// (X[q + R1 t] at position q R2 + t) and the inverse starts from that order: no exchange
// beyond the one between the passes. Shared-memory rows of 24 values (both columns) are
// padded to 25: the algebra's lanes, one row each, then start on different banks.
// Bound: HBM (reads and writes Y once); the FP64 work of the algebra and the transforms is
// about half of that time.
// ---------------------------------------------------------------------------------
template <typename T, int R1, int R2>
__global__ void __launch_bounds__(S2_THREADS, s2_minb(R1 > 9 ? R1 : 9)) sig2_mid(Sig2B a) {
    constexpr int N2 = R1 * R2, LD = 2 * S2_E + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx<T> *S = (cplx<T> *)smem_raw;  // [position][column][e]
    cplx<T> *twL = S + N2 * LD;        // W_N2^m
    for (int m = threadIdx.x; m < N2; m += blockDim.x) twL[m] = cvt<T>(a.tw[m * a.N1]);
    __syncthreads();
    const int ncp = a.N1 / 2 + 1;
    for (int it = blockIdx.x; it < a.nitems; it += gridDim.x) {
        const int ip = it / ncp, c0 = it % ncp, c1 = (a.N1 - c0) % a.N1;
        const bool two = c0 != c1;
        cplx<T> *Yp = (cplx<T> *)a.Y + (size_t)ip * a.N1 * N2 * S2_E;
        // forward pass 1: global -> registers -> S
        for (int idx = threadIdx.x; idx < 2 * S2_E * R2; idx += blockDim.x) {
            const int ce = idx % (2 * S2_E), col = ce / S2_E, e = ce % S2_E, j = idx / (2 * S2_E);
            if (col && !two) continue;
            const cplx<T> *y = Yp + (size_t)(col ? c1 : c0) * N2 * S2_E + e;
            cplx<T> v[R1];
#pragma unroll
            for (int r = 0; r < R1; r++) v[r] = y[(j + R2 * r) * S2_E];
            dft<T, R1, -1>(v);
            S[j * LD + ce] = v[0];
#pragma unroll
            for (int q = 1; q < R1; q++) S[(q * R2 + j) * LD + ce] = v[q] * twL[j * q];
        }
        __syncthreads();
        // forward pass 2, in place
        for (int idx = threadIdx.x; idx < 2 * S2_E * R1; idx += blockDim.x) {
            const int ce = idx % (2 * S2_E), k = idx / (2 * S2_E);
            if (ce >= S2_E && !two) continue;
            cplx<T> v[R2];
#pragma unroll
            for (int j = 0; j < R2; j++) v[j] = S[(k * R2 + j) * LD + ce];
            dft<T, R2, -1>(v);
#pragma unroll
            for (int t = 0; t < R2; t++) S[(k * R2 + t) * LD + ce] = v[t];
        }
        __syncthreads();
        // the algebra, one frequency a task, in place
        for (int idx = threadIdx.x; idx < (two ? 2 : 1) * N2; idx += blockDim.x) {
            const int pos = idx % N2, col = idx / N2;
            // position of -l: l2 = k + R1 t at k R2 + t; column 0 maps l2 to N2 - l2, the others to N2 - 1 - l2
            int pm = N2 - 1 - pos;
            if (c0 == 0) {
                const int k = pos / R2, t = pos % R2;
                pm = (k == 0) ? (R2 - t) % R2 : (R1 - k) * R2 + (R2 - 1 - t);
            }
            cplx<T> *s0 = S + pos * LD + col * S2_E;                       // R_IJ(l), L_IJ(l)
            cplx<T> *s1 = S + pm * LD + (two ? 1 - col : 0) * S2_E + 4;  // R_JI(-l)
            B2<T> r, L, rp, sR, sRp, sL;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                r.a[e & 1][e >> 1] = s0[e];
                L.a[e & 1][e >> 1] = s0[8 + e];
                rp.a[e & 1][e >> 1] = s1[e];
            }
            pair_algebra(r, rp, L, sR, sRp, sL);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                s0[e] = sR.a[e & 1][e >> 1];
                s0[8 + e] = sL.a[e & 1][e >> 1];
                s1[e] = sRp.a[e & 1][e >> 1];
            }
        }
        __syncthreads();
        // inverse over t, in place: d[k][j] = W_N2^{-jk} sum_t X[k + R1 t] W_R2^{-jt}
        for (int idx = threadIdx.x; idx < 2 * S2_E * R1; idx += blockDim.x) {
            const int ce = idx % (2 * S2_E), k = idx / (2 * S2_E);
            if (ce >= S2_E && !two) continue;
            cplx<T> v[R2];
#pragma unroll
            for (int t = 0; t < R2; t++) v[t] = S[(k * R2 + t) * LD + ce];
            dft<T, R2, 1>(v);
            S[k * R2 * LD + ce] = v[0];
#pragma unroll
            for (int j = 1; j < R2; j++) S[(k * R2 + j) * LD + ce] = v[j] * conj(twL[j * k]);
        }
        __syncthreads();
        // inverse over k: x[j + R2 r] = sum_k d[k][j] W_R1^{-kr}, registers -> global
        for (int idx = threadIdx.x; idx < 2 * S2_E * R2; idx += blockDim.x) {
            const int ce = idx % (2 * S2_E), col = ce / S2_E, e = ce % S2_E, j = idx / (2 * S2_E);
            if (col && !two) continue;
            cplx<T> *y = Yp + (size_t)(col ? c1 : c0) * N2 * S2_E + e;
            cplx<T> v[R1];
#pragma unroll
            for (int k = 0; k < R1; k++) v[k] = S[(k * R2 + j) * LD + ce];
            dft<T, R1, 1>(v);
#pragma unroll
            for (int r = 0; r < R1; r++) y[(j + R2 * r) * S2_E] = v[r];
        }
        __syncthreads();  // S is rewritten by the next item
    }
}

// ---------------------------------------------------------------------------------
// Kernel C: the twiddle W_Nf^{-m2 l1}, inverse length-N1 transforms, scaling by
// U_I U_J hbar^2 (delta/2pi)^2 / Nf, the first n energies -> Sigma[w][pair]. Items as in kernel A.
// Bound: HBM (reads Nf, writes n values of each of the 12 sequences).
// ---------------------------------------------------------------------------------
template <typename T, int R1, int R2>
__global__ void __launch_bounds__(S2_THREADS, s2_minb(R1)) sig2_invC(Sig2C a) {
    constexpr int N1 = R1 * R2, GA = S2_GA, W = GA * S2_E;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx<T> *S = (cplx<T> *)smem_raw;  // [position][m2][e]
    cplx<T> *twL = S + N1 * W;         // W_N1^-m
    cplx<T> *twC = twL + N1;           // W_Nf^{-m2 l1} of the item's m2: [l1][m2]
    int twm = -1;                      // the m20 they are for
    for (int m = threadIdx.x; m < N1; m += blockDim.x) twL[m] = conj(cvt<T>(a.tw[m * a.N2]));
    __syncthreads();
    for (int it = blockIdx.x; it < a.nitems; it += gridDim.x) {
        const int ip = it % a.npairs, m20 = (it / a.npairs) * GA;
        const int2 pr = a.pairs[ip];
        const double c = a.scale[ip];
        if (m20 != twm) {
            for (int t = threadIdx.x; t < N1 * GA; t += blockDim.x)
                twC[t] = conj(cvt<T>(a.tw[(m20 + t % GA) * (t / GA)]));
            twm = m20;
            __syncthreads();
        }
        for (int idx = threadIdx.x; idx < W * R2; idx += blockDim.x) {
            const int e = idx % S2_E, g = (idx / S2_E) % GA, j = idx / W;
            const int m2 = m20 + g;
            const cplx<T> *y = (const cplx<T> *)a.Y + ((size_t)ip * N1 * a.N2 + m2) * S2_E + e;
            cplx<T> v[R1];
#pragma unroll
            for (int r = 0; r < R1; r++) v[r] = y[(size_t)(j + R2 * r) * a.N2 * S2_E];
#pragma unroll
            for (int r = 0; r < R1; r++) v[r] = v[r] * twC[(j + R2 * r) * GA + g];
            dft<T, R1, 1>(v);
            S[j * W + idx % W] = v[0];
#pragma unroll
            for (int q = 1; q < R1; q++) S[(q * R2 + j) * W + idx % W] = v[q] * twL[j * q];
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < W * R1; idx += blockDim.x) {
            const int e = idx % S2_E, g = (idx / S2_E) % GA, k = idx / W;
            cplx<T> v[R2];
#pragma unroll
            for (int j = 0; j < R2; j++) v[j] = S[(k * R2 + j) * W + idx % W];
            dft<T, R2, 1>(v);
            zc *s = a.Sig + sig_block(pr.x, pr.y) + e;
#pragma unroll
            for (int t = 0; t < R2; t++) {
                const int64_t w = (int64_t)a.N2 * (k + R1 * t) + m20 + g;
                if (w < a.n) s[w * a.sig_ld] = zc{c * (double)v[t].x, c * (double)v[t].y};
            }
        }
        __syncthreads();  // S is rewritten by the next item
    }
}

// the shared memory of the kernels at a length
template <typename T> constexpr size_t sig2_smem_A(int N1) { return sizeof(cplx<T>) * (size_t)N1 * (S2_GA * S2_E + 1 + S2_GA); }
template <typename T> constexpr size_t sig2_smem_B(int N2) { return sizeof(cplx<T>) * (size_t)N2 * (2 * S2_E + 1 + 1); }

}  // namespace qs
