// sancho_fft.cuh -- SANCHO's bubbles and self-energies (src/self_energies.f90:49-207) as transforms over
// the energy index.
#pragma once
#include "qs_common.cuh"

namespace qs {

// a transform of length L = rad[0] .. rad[nst - 1]
struct SaPlan {
    int L = 0, nst = 0;
    int rad[4] = {1, 1, 1, 1};
};
// the shortest one for a grid of n energies (L >= 2 n - 1); L = 0 where a sequence does not fit in
// shared memory: n above 6720
SaPlan sa_plan(int n);

struct SaFft {
    int Na, n;
    SaPlan p;
    const zc *tw;           // exp(-2 pi i k / L), L values (sa_twiddles)
    const double *U;
    double pp;              // delta / 2 pi
    zc *const *E;           // G_in: r, a, <, >, [e n + k]
    zc *const *chi, *const *phi, *const *D, *const *P;  // as in the handle; room for Na^2 L values each
    zc *S2R, *S2L, *S3R, *S3L;                          // [e + w Na^2]
};
int sa_twiddles(cudaStream_t st, const SaPlan &p, zc *tw);
// Sigma2, and at order 3 chi and phi (ph: > , <, r, a at [e (2 n - 1) + p]) of G_in
int sa_fft_second(cudaStream_t st, const SaFft &f, int order);
// Sigma3 from the products D and P of the bubbles
int sa_fft_third(cudaStream_t st, const SaFft &f);

}  // namespace qs
