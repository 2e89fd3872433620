// sancho_fft.cu -- SANCHO's bubbles and self-energies (src/self_energies.f90:49-207) as transforms over
// the energy index.
//
// All sums over energies are convolutions or correlations of two sequences, one of at most n and one of at
// most 2 n - 1 values, of which 2 n - 1 or n results are needed: a cyclic length L >= 2 n - 1 gives them
// exactly. With A^ the transform of a sequence A(k),
//   sum_k A(k) B(q - k)  ->  A^ B^           sum_k A(k) B(k - m)  ->  A^ conj(FFT[conj B])
// and since G^< and G^> are anti-Hermitian and G^a = (G^r)^+, conj B of an element (j, i) is an element (i, j)
// again: all factors belong to one element, with r, a, l, g the spectra of its G^r, G^a, G^<, G^> = l + r - a:
//   chi^> = -g l*    chi^< = -l g*    chi^r = l r* - r l*    chi^a = l a* - a l*       (particle-hole bubbles)
//   phi^> = g g      phi^< = l l      phi^r = r (g + l)      phi^a = a (g + l)         (particle-particle)
//   Sigma^< = l X^< - g* P^<          Sigma^r = r X^> + l X^r + r* P^> - g* P^r
// with X = chi, P absent for Sigma2, and X = D, P the products of bubbles for Sigma3 (bubbles of the
// products are formed at each lag, so chi and phi are transformed back and the products forward again).
//
// One block per sequence, the sequence in shared memory, in place: three (L <= 4096) or four register
// butterflies with a barrier each. The forward transform leaves its values in the order in which the
// inverse takes them, and the products are pointwise, so nothing is reordered.
//
// The direct sums it replaces cost 12 (bubbles) and 6 multiply-adds per pair of energies and element;
// they remain for grids whose sequences do not fit in shared memory. Bound: the latency of the few
// launches (10 sites x 883 energies, order 3: 24 transforms of 1792 values an element, 2.3 MFLOP; 2.9 MB per
// array, all in L2).
#include <algorithm>

#include "fft.cuh"
#include "sancho_fft.cuh"

namespace qs {
namespace {

__host__ __device__ __forceinline__ int pad(int p) { return p + (p >> 4); }  // bank groups of 8 words
constexpr int SA_LMAX = 13440;  // the longest product of radices with pad(L) * 16 bytes within SMEM_MAX

// one pass over blocks of Ns = R M values: forward (S < 0) butterfly then twiddle, backward the reverse
template <int R, int S> __device__ __forceinline__ void pass(zc *s, int L, int Ns, const zc *__restrict__ tw) {
    const int M = Ns / R, step = L / Ns;
    for (int b = threadIdx.x; b < L / R; b += blockDim.x) {
        const int j = b % M, base = (b / M) * Ns + j;
        zc v[R];
#pragma unroll
        for (int q = 0; q < R; q++) {
            v[q] = s[pad(base + M * q)];
            if (S > 0 && q > 0) v[q] = v[q] * conj(tw[j * q * step]);
        }
        dft<double, R, S>(v);
#pragma unroll
        for (int q = 0; q < R; q++) {
            if (S < 0 && q > 0) v[q] = v[q] * tw[j * q * step];
            s[pad(base + M * q)] = v[q];
        }
    }
}

// the whole transform; values in natural order before a forward and after a backward one
template <int S> __device__ __forceinline__ void transform(zc *s, const SaPlan &p, const zc *__restrict__ tw) {
    int Ns = p.L;
    if (S > 0)
        for (int k = 0; k + 1 < p.nst; k++) Ns /= p.rad[k];
#pragma unroll 1
    for (int k = 0; k < p.nst; k++) {
        const int R = p.rad[S < 0 ? k : p.nst - 1 - k];
        __syncthreads();
        switch (R) {
            case 4: pass<4, S>(s, p.L, Ns, tw); break;
            case 5: pass<5, S>(s, p.L, Ns, tw); break;
            case 6: pass<6, S>(s, p.L, Ns, tw); break;
            case 7: pass<7, S>(s, p.L, Ns, tw); break;
            case 8: pass<8, S>(s, p.L, Ns, tw); break;
            case 9: pass<9, S>(s, p.L, Ns, tw); break;
            case 10: pass<10, S>(s, p.L, Ns, tw); break;
            case 12: pass<12, S>(s, p.L, Ns, tw); break;
            case 14: pass<14, S>(s, p.L, Ns, tw); break;
            default: pass<16, S>(s, p.L, Ns, tw);
        }
        if (S < 0) Ns /= R;
        else if (k + 1 < p.nst) Ns *= p.rad[p.nst - 2 - k];
    }
    __syncthreads();
}

// forward transforms of nseq sequences per element: value p of len (stride len) stands at p - shift mod L
struct SaFwd {
    SaPlan p;
    const zc *tw;
    const zc *src[6];
    zc *dst[6];  // [e L + position]
    int len[6], shift[6];
};
__global__ void __launch_bounds__(256) sa_forward(SaFwd a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    zc *s = (zc *)smem_raw;
    const int e = blockIdx.x, q = blockIdx.y, L = a.p.L, len = a.len[q], shift = a.shift[q];
    const zc *src = a.src[q] + (size_t)e * len;
    for (int i = threadIdx.x; i < L; i += blockDim.x) {
        int p = i + shift;
        if (p >= L) p -= L;
        s[pad(i)] = p < len ? src[p] : zc{0, 0};
    }
    transform<-1>(s, a.p, a.tw);
    zc *d = a.dst[q] + (size_t)e * L;
    for (int i = threadIdx.x; i < L; i += blockDim.x) d[i] = s[pad(i)];
}

__device__ __forceinline__ zc mul_conj(zc a, zc b) { return zc{fma(a.y, b.y, a.x * b.x), fma(a.y, b.x, -a.x * b.y)}; }

enum { S_L = 0, S_R, CHI, PHI = CHI + 4 };  // results of sa_backward: Sigma^<, Sigma^r, four bubbles each
struct SaBwd {
    SaPlan p;
    int Na, n, first;                // grid.y = 0 is result `first`
    const zc *tw;
    const zc *r, *a, *l;             // spectra of G^r, G^a, G^<
    const zc *X[3], *P[3];           // spectra of D and P: >, <, r (third: Sigma3), else nullptr
    const double *U;
    double pp;
    zc *SL, *SR, *chi[4], *phi[4];
};
template <bool THIRD> __global__ void __launch_bounds__(256) sa_backward(SaBwd a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    zc *s = (zc *)smem_raw;
    const int e = blockIdx.x, t = a.first + blockIdx.y, L = a.p.L, n = a.n, Nm = 2 * n - 1;
    const size_t o = (size_t)e * L;
    for (int i = threadIdx.x; i < L; i += blockDim.x) {
        const zc l = a.l[o + i], r = a.r[o + i], ad = a.a[o + i], g = (l + r) - ad;
        zc v;
        if (THIRD) {
            if (t == S_L) {
                v = l * a.X[1][o + i] - mul_conj(a.P[1][o + i], g);
            } else {
                v = r * a.X[0][o + i];
                cfma(v, l, a.X[2][o + i]);
                v = v + mul_conj(a.P[0][o + i], r) - mul_conj(a.P[2][o + i], g);
            }
        } else {
            const zc cl = -mul_conj(l, g);
            switch (t) {
                case S_L: v = l * cl; break;
                case S_R: {
                    v = r * -mul_conj(g, l);
                    cfma(v, l, mul_conj(l, r) - mul_conj(r, l));
                    break;
                }
                case CHI: v = -mul_conj(g, l); break;
                case CHI + 1: v = cl; break;
                case CHI + 2: v = mul_conj(l, r) - mul_conj(r, l); break;
                case CHI + 3: v = mul_conj(l, ad) - mul_conj(ad, l); break;
                case PHI: v = g * g; break;
                case PHI + 1: v = l * l; break;
                case PHI + 2: v = r * (g + l); break;
                default: v = ad * (g + l);
            }
        }
        s[pad(i)] = v;
    }
    transform<1>(s, a.p, a.tw);
    if (t < CHI) {
        // -(i hbar)^2 = 1 and -(i hbar)^3 = i (hbar = 1); the bubbles' own delta / 2 pi at second order
        const double c = a.U[e % a.Na] * a.U[e / a.Na] * a.pp * (THIRD ? 1.0 : a.pp) / L;
        zc *out = (t == S_L ? a.SL : a.SR) + e;
        const size_t ld = (size_t)a.Na * a.Na;
        for (int w = threadIdx.x; w < n; w += blockDim.x) {
            const zc v = s[pad(w)];
            out[w * ld] = THIRD ? zc{-c * v.y, c * v.x} : zc{c * v.x, c * v.y};
        }
    } else {
        const double c = a.pp / L;
        const int shift = t < PHI ? n - 1 : 0;  // chi(m) at m + n - 1
        zc *out = (t < PHI ? a.chi[t - CHI] : a.phi[t - PHI]) + (size_t)e * Nm;
        for (int p = threadIdx.x; p < Nm; p += blockDim.x) {
            const int i = p >= shift ? p - shift : p - shift + L;
            out[p] = c * s[pad(i)];
        }
    }
}

__global__ void sa_twiddle(int L, zc *tw) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= L) return;
    // a quarter turn at a time, so that the argument's rounding stays below half an ulp of the result
    const int q = (int)(4 * (int64_t)k / L);
    double sn, cs;
    sincospi((double)(4 * (int64_t)k - (int64_t)q * L) / (2.0 * L), &sn, &cs);
    tw[k] = q == 0 ? zc{cs, -sn} : q == 1 ? zc{-sn, -cs} : q == 2 ? zc{-cs, sn} : zc{sn, cs};
}

int threads(const SaPlan &p) { return p.L <= 2048 ? 128 : 256; }
size_t smem(const SaPlan &p) { return sizeof(zc) * (pad(p.L - 1) + 1); }

template <class K, class A> int launch(cudaStream_t st, K kernel, dim3 grid, const SaPlan &p, const A &a) {
    // (up to 40 KB need no attribute)
    cudaError_t e = smem(p) > 40 << 10 ? smem_cap((const void *)kernel) : cudaSuccess;
    if (e == cudaSuccess) {
        count_launch();
        kernel<<<grid, threads(p), smem(p), st>>>(a);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? 0 : -(int)e;
}

}  // namespace

SaPlan sa_plan(int n) {
    static const int R[] = {16, 14, 12, 10, 9, 8, 7, 6, 5, 4};
    SaPlan best;
    if (2 * n - 1 > SA_LMAX) return best;
    const int need = std::max(2 * n - 1, 16);
    const int nst = need <= 256 ? 2 : need <= 4096 ? 3 : 4;
    for (int a : R)
        for (int b : R)
            for (int c : R)
                for (int d : R) {
                    if (b > a || c > b || d > c) continue;
                    const int rad[4] = {a, b, nst > 2 ? c : 1, nst > 3 ? d : 1};
                    const int L = rad[0] * rad[1] * rad[2] * rad[3];
                    if (L < need || L > SA_LMAX || (best.L && L >= best.L)) continue;
                    best.L = L;
                    best.nst = nst;
                    std::copy(rad, rad + 4, best.rad);
                }
    return best;
}

int sa_twiddles(cudaStream_t st, const SaPlan &p, zc *tw) {
    count_launch();
    sa_twiddle<<<(p.L + 255) / 256, 256, 0, st>>>(p.L, tw);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : -(int)e;
}

static SaBwd backward(const SaFft &f) {
    SaBwd b{};
    b.p = f.p;
    b.Na = f.Na;
    b.n = f.n;
    b.tw = f.tw;
    b.U = f.U;
    b.pp = f.pp;
    return b;
}

int sa_fft_second(cudaStream_t st, const SaFft &f, int order) {
    // the spectra of G^r, G^a, G^< stand where nothing is needed now: the products, or chi at order 2
    zc *const *hat = order == 3 ? f.D : f.chi;
    SaFwd a{};
    a.p = f.p;
    a.tw = f.tw;
    for (int q = 0; q < 3; q++) {
        a.src[q] = f.E[q];
        a.dst[q] = hat[q];
        a.len[q] = f.n;
    }
    const int nf = f.Na * f.Na;
    int rc = launch(st, sa_forward, dim3(nf, 3), f.p, a);
    if (rc) return rc;
    SaBwd b = backward(f);
    b.r = hat[0];
    b.a = hat[1];
    b.l = hat[2];
    b.SL = f.S2L;
    b.SR = f.S2R;
    if (order == 3)
        for (int q = 0; q < 4; q++) {
            b.chi[q] = f.chi[q];
            b.phi[q] = f.phi[q];
        }
    return launch(st, sa_backward<false>, dim3(nf, order == 3 ? 10 : 2), f.p, b);
}

int sa_fft_third(cudaStream_t st, const SaFft &f) {
    // the spectra of D and P take the place of chi and phi, those of G_in of the rest and of D^>
    SaFwd a{};
    a.p = f.p;
    a.tw = f.tw;
    for (int q = 0; q < 6; q++) {
        a.src[q] = q < 3 ? f.D[q] : f.P[q - 3];
        a.dst[q] = q < 3 ? f.chi[q] : f.phi[q - 3];
        a.len[q] = 2 * f.n - 1;
        a.shift[q] = q < 3 ? f.n - 1 : 0;
    }
    const int nf = f.Na * f.Na;
    int rc = launch(st, sa_forward, dim3(nf, 6), f.p, a);
    if (rc) return rc;
    zc *hat[3] = {f.chi[3], f.phi[3], f.D[0]};
    for (int q = 0; q < 3; q++) {
        a.src[q] = f.E[q];
        a.dst[q] = hat[q];
        a.len[q] = f.n;
        a.shift[q] = 0;
    }
    if ((rc = launch(st, sa_forward, dim3(nf, 3), f.p, a))) return rc;
    SaBwd b = backward(f);
    b.r = hat[0];
    b.a = hat[1];
    b.l = hat[2];
    for (int q = 0; q < 3; q++) {
        b.X[q] = f.chi[q];
        b.P[q] = f.phi[q];
    }
    b.SL = f.S3L;
    b.SR = f.S3R;
    return launch(st, sa_backward<true>, dim3(nf, 2), f.p, b);
}

}  // namespace qs
