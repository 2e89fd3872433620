// sigma2_b64.cu -- the FP64 instances of sig2_mid (sigma2_kernels.cuh).
#include "sigma2_kernels.cuh"

namespace qs {

Sig2Fn sig2_mid_fn64(int L) {
#define QS_CASE(R1, R2) \
    if (L == R1 * R2) return {(const void *)sig2_mid<double, R1, R2>, sig2_smem_B<double>(L)};
    QS_FFT_LENGTHS(QS_CASE)
#undef QS_CASE
    return {nullptr, 0};
}

}  // namespace qs
