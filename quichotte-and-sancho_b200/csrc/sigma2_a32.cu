// sigma2_a32.cu -- the FP32 instances of sig2_fwdA (sigma2_kernels.cuh).
#include "sigma2_kernels.cuh"

namespace qs {

Sig2Fn sig2_fwdA_fn32(int L) {
#define QS_CASE(R1, R2) \
    if (L == R1 * R2) return {(const void *)sig2_fwdA<float, R1, R2>, sig2_smem_A<float>(L)};
    QS_FFT_LENGTHS(QS_CASE)
#undef QS_CASE
    return {nullptr, 0};
}

}  // namespace qs
