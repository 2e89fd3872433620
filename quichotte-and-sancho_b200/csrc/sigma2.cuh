// sigma2.cuh -- what sigma2.cu and the files with the instances of its kernels share.
#pragma once
#include "qs_common.cuh"

namespace qs {

constexpr int S2_THREADS = 192, S2_GA = 2;  // threads a block; m2 columns of an item of kernels A and C

// an entry of the kernel tables: the function of a length, its shared memory
struct Sig2Fn {
    const void *fn;
    size_t smem;
};

struct Sig2A {
    const double *X;  // SCF vector
    int64_t nblk;
    int n, N2, npairs, nitems;
    const int2 *pairs;
    const zc *tw;  // W_Nf^k
    void *Y;       // [pair][l1][m2][12]
};
struct Sig2B {
    void *Y;
    int N1, nitems;
    const zc *tw;
};
struct Sig2C {
    const void *Y;
    zc *Sig;         // [w][pair][12]
    int64_t sig_ld;  // values per energy
    int n, N2, npairs, nitems;
    const int2 *pairs;
    const double *scale;  // per pair
    const zc *tw;
};

// the instance of a kernel for the length L (sigma2_{a,b,c}{64,32}.cu); fn = nullptr if it has none
Sig2Fn sig2_fwdA_fn64(int L);
Sig2Fn sig2_mid_fn64(int L);
Sig2Fn sig2_invC_fn64(int L);
Sig2Fn sig2_fwdA_fn32(int L);
Sig2Fn sig2_mid_fn32(int L);
Sig2Fn sig2_invC_fn32(int L);

}  // namespace qs
