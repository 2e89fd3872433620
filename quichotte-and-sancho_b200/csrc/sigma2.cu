// sigma2.cu -- second-order self-energies Sigma2^r, Sigma2^< for all energies at once
// (sigma2_compute, src/self_energies.f90:135-219), as three FFT kernels over the energy
// axis with the 2x2 spin algebra fused between the forward and the inverse transforms.
//
// The reference zero-pads G_ij(w) from n to Nf >= 2n-1, forward-transforms every active element
// of G^r and G^<, forms per site pair (I,J) and frequency l the 2x2 products of blocks (I,J) at
// +l and (J,I) at -l, and inverse-transforms the result (scaled by
// c = U_I U_J hbar^2 (delta/2pi)^2 / Nf) back to the first n energies. Any Nf >= 2n-1 gives the
// same sums; the reference takes the next length with factors 2, 3, 5, 7 (good_fft_size).
//
// Here Nf = N1*N2 is the smallest product of two lengths that have kernels (5 % above 2n-1 on
// average, 14 % at most from n = 200 on, 25 % from 129; 256 for all shorter grids), and every transform is split in the four-step way (w = N2 m1 + m2,
// l = l1 + N1 l2):
//   kernel A  length-N1 FFTs over m1, twiddle W^{m2 l1}                          -> Y[l1][m2]
//   kernel B  per column pair {l1, N1-l1}: length-N2 FFTs over m2 (the spectrum), the 2x2
//             algebra (the partner -l of l = l1 + N1 l2 lies in column N1-l1), inverse
//             length-N2 FFTs, in place
//   kernel C  twiddle W^{-m2 l1}, inverse length-N1 FFTs over l1, scale by c, the first n
//             energies                                                           -> Sigma[w]
// The unit of all three is a site pair I <= J with its 12 sequences R_IJ, R_JI, L_IJ side by
// side: G^< and Sigma^< are anti-Hermitian (unpack_gf rebuilds G^<_ji = -conj(G^<_ij),
// common/linear_algebra.f90:222-223), so FL_JI(l) = -FL_IJ(-l)^+ and neither is transformed.
// The SCF vector, Y and Sigma keep a pair's 12 values together (192 bytes), so every global
// access is a run of at least 192 bytes whatever the transform length.
//
// Measured on B200 per launch (A / B / C, FP64), with the sequence-major spectra, runtime radices and
// runs of 16 to 64 bytes before: 120 states x 4096 energies 2.23 / 3.96 / 2.54 -> 1.06 / 1.45 /
// 0.83 ms (4.1, 4.0 and 5.2 TB/s of the bytes they cannot avoid); 192 x 1201: 5.3 / 11.6 / 7.0 ->
// 0.74 / 1.41 / 0.57 ms; 24 x 32768: 2.96 / 1.23 / 2.90 -> 0.44 / 0.68 / 0.42 ms.
#include <algorithm>
#include <cmath>

#include "sigma2.cuh"

namespace qs {

// the lengths with kernels (QS_FFT_LENGTHS of fft.cuh)
static const int S2_LENGTHS[] = {16, 20, 24, 28, 32, 36, 40, 48, 56, 64, 72, 80, 96, 112, 128, 144, 160, 192, 224, 256};

FftPlan sigma2_plan(int n) {
    FftPlan best{0, 0, 0};
    for (int n1 : S2_LENGTHS)
        for (int n2 : S2_LENGTHS) {
            const int nf = n1 * n2;
            if (n2 > n1 || nf < 2 * n - 1) continue;
            // the shortest; among equals the most balanced split
            if (!best.Nf || nf < best.Nf || (nf == best.Nf && n1 < best.N1)) best = FftPlan{nf, n1, n2};
        }
    return best;
}

int sigma2_count_pairs(const qs_handle *h) {
    int k = 0;
    for (int J = 0; J < h->nAs; J++)
        for (int I = 0; I <= J; I++) k += h->U_site[h->act[2 * I]] * h->U_site[h->act[2 * J]] != 0.0;
    return k;
}

// The reference's padded length and the split this solver used to give it: grids whose length
// has no divisor that keeps N1 <= 512 are refused (all above 65536, and a few below).
static bool reference_length_fits(int n, int &Nf) {
    for (Nf = 2 * n - 1;; Nf++) {
        int m = Nf;
        for (int r : {2, 3, 5, 7})
            while (m % r == 0) m /= r;
        if (m == 1) break;
    }
    int best = 1;
    const double sq = std::sqrt((double)Nf);
    for (int d = 1; d <= 128; d++)
        if (Nf % d == 0 && std::fabs(d - sq) < std::fabs(best - sq)) best = d;
    return Nf / best <= 512;
}

template <typename T> static Sig2Fn fwdA_fn(int L) { return sizeof(T) == 8 ? sig2_fwdA_fn64(L) : sig2_fwdA_fn32(L); }
template <typename T> static Sig2Fn mid_fn(int L) { return sizeof(T) == 8 ? sig2_mid_fn64(L) : sig2_mid_fn32(L); }
template <typename T> static Sig2Fn invC_fn(int L) { return sizeof(T) == 8 ? sig2_invC_fn64(L) : sig2_invC_fn32(L); }

template <typename T> static int sigma2_attributes(qs_handle *h) {
    int k = 0;
    for (const Sig2Fn &f : {fwdA_fn<T>(h->fft.N1), mid_fn<T>(h->fft.N2), invC_fn<T>(h->fft.N1)}) {
        if (!f.fn) {
            h->err = "sigma2: no kernel for a transform length";
            return -1;
        }
        QS_CUDA(h, smem_cap(f.fn));
        QS_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&h->sig2_occ[sizeof(T) == 8][k], f.fn, S2_THREADS, f.smem));
        k++;
    }
    return 0;
}

int sigma2_setup(qs_handle *h) {
    const int n = h->n, nA = h->nA;
    int Nref;
    if (!reference_length_fits(n, Nref) || !sigma2_plan(n).Nf) {
        h->err = "sigma2: FFT length " + std::to_string(Nref) + " needs N1 <= 512 and N2 <= 128";
        return -1;
    }
    FftPlan &fp = h->fft;
    fp = sigma2_plan(n);
    // twiddles W_Nf^k in extended precision
    std::vector<zc> tw(fp.Nf);
    for (int k = 0; k < fp.Nf; k++) {
        long double a = -2.0L * 3.141592653589793238462643383279502884L * (long double)k / (long double)fp.Nf;
        tw[k] = zc{(double)cosl(a), (double)sinl(a)};
    }
    int rc;
    if ((rc = dalloc(h, (void **)&h->d_tw, sizeof(zc) * fp.Nf))) return rc;
    QS_CUDA(h, cudaMemcpyAsync(h->d_tw, tw.data(), sizeof(zc) * fp.Nf, cudaMemcpyHostToDevice, h->stream));
    // the pack_gf block's elements (Re G^r row-major | Im G^r | Re G^< strict upper row-major |
    // Im G^< upper row-major) in a device block
    std::vector<int> perm;
    perm.reserve((size_t)3 * nA * nA);
    for (int part = 0; part < 2; part++)
        for (int i = 0; i < nA; i++)
            for (int j = 0; j < nA; j++) perm.push_back(dl_r(i, j) + part);
    for (int i = 0; i < nA; i++)
        for (int j = i + 1; j < nA; j++) perm.push_back(dl_l(i, j));
    for (int i = 0; i < nA; i++)
        for (int j = i; j < nA; j++) perm.push_back(i == j ? dl_d(i) : dl_l(i, j) + 1);
    if ((rc = dalloc(h, (void **)&h->d_dl_perm, sizeof(int) * perm.size()))) return rc;
    QS_CUDA(h, cudaMemcpyAsync(h->d_dl_perm, perm.data(), sizeof(int) * perm.size(), cudaMemcpyHostToDevice, h->stream));
    if ((rc = dalloc(h, (void **)&h->d_Y, sizeof(zc) * y_elems(h)))) return rc;
    if ((rc = dalloc(h, (void **)&h->d_Sig, sizeof(zc) * (size_t)sig_stride(nA) * n))) return rc;
    // interacting pairs and their scale c = U_I U_J hbar^2 (delta/2pi)^2 / Nf
    const double pp = h->delta / (2.0 * PI);
    std::vector<double> scale;
    std::vector<int2> pairs;
    for (int J = 0; J < h->nAs; J++)
        for (int I = 0; I <= J; I++) {
            const double up = h->U_site[h->act[2 * I]] * h->U_site[h->act[2 * J]];
            if (up == 0.0) continue;
            pairs.push_back(int2{I, J});
            scale.push_back(up * pp * pp / (double)fp.Nf);
        }
    h->sig2_npairs = (int)pairs.size();
    if ((rc = dalloc(h, (void **)&h->sig2_scale, sizeof(double) * std::max<size_t>(pairs.size(), 1)))) return rc;
    if ((rc = dalloc(h, (void **)&h->sig2_pairs, sizeof(int2) * std::max<size_t>(pairs.size(), 1)))) return rc;
    if (!pairs.empty()) {
        QS_CUDA(h, cudaMemcpyAsync(h->sig2_scale, scale.data(), sizeof(double) * scale.size(), cudaMemcpyHostToDevice, h->stream));
        QS_CUDA(h, cudaMemcpyAsync(h->sig2_pairs, pairs.data(), sizeof(int2) * pairs.size(), cudaMemcpyHostToDevice, h->stream));
    }
    if ((rc = sigma2_attributes<double>(h))) return rc;
    if (h->precision == QS_PREC_MIXED && (rc = sigma2_attributes<float>(h))) return rc;
    // every buffer is zeroed on h->stream by dalloc: the tables are copied on the same
    // stream (after the zeroing) and the host staging vectors must outlive the copies
    QS_CUDA(h, cudaStreamSynchronize(h->stream));
    return 0;
}

// as many blocks as fit at once (occ per SM) walk the items
template <typename P> static int launch_sig2(qs_handle *h, int fam, const Sig2Fn &f, const P &p, int occ) {
    P arg = p;
    void *args[] = {&arg};
    const int pi = prof_begin(h, fam);
    const cudaError_t e = cudaLaunchKernel(f.fn, dim3(std::min(p.nitems, 148 * std::max(occ, 1))), dim3(S2_THREADS), args,
                                           f.smem, h->stream);
    prof_end(h, pi);
    QS_CUDA(h, e);
    return 0;
}

// Y holds FP32 spectra when T = float (in the first half of the same allocation)
template <typename T> static int sigma2_run(qs_handle *h, const double *d_x) {
    const FftPlan &fp = h->fft;
    if (h->sig2_npairs == 0) return 0;
    const int itemsAC = h->sig2_npairs * (fp.N2 / S2_GA);
    const Sig2A a{d_x, h->nblk, h->n, fp.N2, h->sig2_npairs, itemsAC, h->sig2_pairs, h->d_tw, h->d_Y};
    const Sig2B b{h->d_Y, fp.N1, h->sig2_npairs * (fp.N1 / 2 + 1), h->d_tw};
    const Sig2C c{h->d_Y, h->d_Sig, sig_stride(h->nA), h->n, fp.N2, h->sig2_npairs, itemsAC, h->sig2_pairs, h->sig2_scale,
                  h->d_tw};
    const int *occ = h->sig2_occ[sizeof(T) == 8];
    int rc;
    if ((rc = launch_sig2(h, K_SIG2A, fwdA_fn<T>(fp.N1), a, occ[0]))) return rc;
    if ((rc = launch_sig2(h, K_SIG2B, mid_fn<T>(fp.N2), b, occ[1]))) return rc;
    return launch_sig2(h, K_SIG2C, invC_fn<T>(fp.N1), c, occ[2]);
}

int sigma2_compute(qs_handle *h, const double *d_x, bool fp32) {
    if (fp32) {
        if (h->precision != QS_PREC_MIXED) {
            h->err = "sigma2: FP32 transforms need a QS_PREC_MIXED handle";
            return -1;
        }
        return sigma2_run<float>(h, d_x);
    }
    return sigma2_run<double>(h, d_x);
}

__global__ void sig2_unblock(int nA, int64_t n, const zc *__restrict__ Sig, zc *__restrict__ SR, zc *__restrict__ SL) {
    const int nf = nA * nA;
    const int64_t ld = sig_stride(nA);
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n * nf; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t w = t / nf;
        const int e = (int)(t - w * nf), i = e % nA, j = e / nA;
        SR[t] = sig_r(Sig + w * ld, i, j);
        SL[t] = sig_l(Sig + w * ld, i, j);
    }
}

int sigma2_unblock(qs_handle *h, zc *SR, zc *SL) {
    count_launch();
    sig2_unblock<<<1184, 256, 0, h->stream>>>(h->nA, h->n, h->d_Sig, SR, SL);
    QS_CUDA(h, cudaGetLastError());
    return 0;
}

}  // namespace qs
