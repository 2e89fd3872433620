// fft.cuh -- transforms of length L = R1 R2 for kernels that hold many sequences side by side
// in shared memory, two register butterflies and one shared-memory exchange per transform.
//
// Conventions are FFTW's, as the reference uses them (src/self_energies.f90:102-103,129,
// 205,208): sign = -1 is the forward transform sum_j x_j exp(-2 pi i jk/L), sign = +1 the
// backward one, both unnormalised.
//
// With x[j + R2 r], j < R2, r < R1:
//   pass 1 (R2 butterflies of radix R1):  b[q][j] = W_L^{jq} sum_r x[j + R2 r] W_R1^{rq}
//   pass 2 (R1 butterflies of radix R2):  X[q + R1 t] = sum_j b[q][j] W_R2^{jt}
// A thread computes one butterfly of one sequence in registers. The sequences of a tile are
// the fastest index in shared and global memory (12 spin components of a site pair times one
// or two neighbouring columns), so that the lanes of a warp touch consecutive 16-byte words
// in both passes whatever the radix: no bank conflicts and no index padding.
#pragma once
#include "qs_common.cuh"

namespace qs {

// an FP64 twiddle at the kernel's element type
template <typename T> __device__ __forceinline__ cplx<T> cvt(zc v) { return cplx<T>{(T)v.x, (T)v.y}; }

// cos(2 pi k / R); k is a constant once the loops around it are unrolled
template <int R> __device__ __forceinline__ double cosv(int k) {
    if constexpr (R == 3) {
        const double t[3] = {1.0, -0.5, -0.5};
        return t[k];
    } else if constexpr (R == 5) {
        const double t[5] = {1.0, 0.30901699437494745, -0.8090169943749475, -0.8090169943749475,
            0.30901699437494745};
        return t[k];
    } else if constexpr (R == 6) {
        const double t[6] = {1.0, 0.5, -0.5, -1.0, -0.5, 0.5};
        return t[k];
    } else if constexpr (R == 7) {
        const double t[7] = {1.0, 0.6234898018587335, -0.2225209339563144, -0.9009688679024191,
            -0.9009688679024191, -0.2225209339563144, 0.6234898018587335};
        return t[k];
    } else if constexpr (R == 9) {
        const double t[9] = {1.0, 0.766044443118978, 0.17364817766693036, -0.5, -0.9396926207859084,
            -0.9396926207859084, -0.5, 0.17364817766693036, 0.766044443118978};
        return t[k];
    } else if constexpr (R == 10) {
        const double t[10] = {1.0, 0.8090169943749475, 0.30901699437494745, -0.30901699437494745,
            -0.8090169943749475, -1.0, -0.8090169943749475, -0.30901699437494745, 0.30901699437494745,
            0.8090169943749475};
        return t[k];
    } else if constexpr (R == 12) {
        const double t[12] = {1.0, 0.8660254037844386, 0.5, 0.0, -0.5, -0.8660254037844386, -1.0,
            -0.8660254037844386, -0.5, 0.0, 0.5, 0.8660254037844386};
        return t[k];
    } else if constexpr (R == 14) {
        const double t[14] = {1.0, 0.9009688679024191, 0.6234898018587335, 0.2225209339563144,
            -0.2225209339563144, -0.6234898018587335, -0.9009688679024191, -1.0, -0.9009688679024191,
            -0.6234898018587335, -0.2225209339563144, 0.2225209339563144, 0.6234898018587335,
            0.9009688679024191};
        return t[k];
    } else if constexpr (R == 16) {
        const double t[16] = {1.0, 0.9238795325112867, 0.7071067811865476, 0.3826834323650898, 0.0,
            -0.3826834323650898, -0.7071067811865476, -0.9238795325112867, -1.0, -0.9238795325112867,
            -0.7071067811865476, -0.3826834323650898, 0.0, 0.3826834323650898, 0.7071067811865476,
            0.9238795325112867};
        return t[k];
    }
    return 0.0;
}
// sin(2 pi k / R); k is a constant once the loops around it are unrolled
template <int R> __device__ __forceinline__ double sinv(int k) {
    if constexpr (R == 3) {
        const double t[3] = {0.0, 0.8660254037844386, -0.8660254037844386};
        return t[k];
    } else if constexpr (R == 5) {
        const double t[5] = {0.0, 0.9510565162951535, 0.5877852522924731, -0.5877852522924731,
            -0.9510565162951535};
        return t[k];
    } else if constexpr (R == 6) {
        const double t[6] = {0.0, 0.8660254037844386, 0.8660254037844386, 0.0, -0.8660254037844386,
            -0.8660254037844386};
        return t[k];
    } else if constexpr (R == 7) {
        const double t[7] = {0.0, 0.7818314824680298, 0.9749279121818236, 0.4338837391175581,
            -0.4338837391175581, -0.9749279121818236, -0.7818314824680298};
        return t[k];
    } else if constexpr (R == 9) {
        const double t[9] = {0.0, 0.6427876096865394, 0.984807753012208, 0.8660254037844386, 0.3420201433256687,
            -0.3420201433256687, -0.8660254037844386, -0.984807753012208, -0.6427876096865394};
        return t[k];
    } else if constexpr (R == 10) {
        const double t[10] = {0.0, 0.5877852522924731, 0.9510565162951535, 0.9510565162951535,
            0.5877852522924731, 0.0, -0.5877852522924731, -0.9510565162951535, -0.9510565162951535,
            -0.5877852522924731};
        return t[k];
    } else if constexpr (R == 12) {
        const double t[12] = {0.0, 0.5, 0.8660254037844386, 1.0, 0.8660254037844386, 0.5, 0.0, -0.5,
            -0.8660254037844386, -1.0, -0.8660254037844386, -0.5};
        return t[k];
    } else if constexpr (R == 14) {
        const double t[14] = {0.0, 0.4338837391175581, 0.7818314824680298, 0.9749279121818236,
            0.9749279121818236, 0.7818314824680298, 0.4338837391175581, 0.0, -0.4338837391175581,
            -0.7818314824680298, -0.9749279121818236, -0.9749279121818236, -0.7818314824680298,
            -0.4338837391175581};
        return t[k];
    } else if constexpr (R == 16) {
        const double t[16] = {0.0, 0.3826834323650898, 0.7071067811865476, 0.9238795325112867, 1.0,
            0.9238795325112867, 0.7071067811865476, 0.3826834323650898, 0.0, -0.3826834323650898,
            -0.7071067811865476, -0.9238795325112867, -1.0, -0.9238795325112867, -0.7071067811865476,
            -0.3826834323650898};
        return t[k];
    }
    return 0.0;
}
// v * exp(S 2 pi i k / R) for a k known at compile time (after unrolling): no multiplication
// for the multiples of a quarter turn, one per component for the odd eighths
template <typename T, int R, int S> __device__ __forceinline__ cplx<T> mul_root(cplx<T> v, int k) {
    k %= R;
    if (S < 0) k = (R - k) % R;
    if (k == 0) return v;
    if (4 * k == R) return {-v.y, v.x};
    if (2 * k == R) return {-v.x, -v.y};
    if (4 * k == 3 * R) return {v.y, -v.x};
    const T h = (T)0.70710678118654752440084436210484903928;
    if (8 * k == R) return {h * (v.x - v.y), h * (v.x + v.y)};
    if (8 * k == 3 * R) return {-h * (v.x + v.y), h * (v.x - v.y)};
    if (8 * k == 5 * R) return {h * (v.y - v.x), -h * (v.x + v.y)};
    if (8 * k == 7 * R) return {h * (v.x + v.y), h * (v.y - v.x)};
    const T c = (T)cosv<R>(k), s = (T)sinv<R>(k);
    return {v.x * c - v.y * s, v.x * s + v.y * c};
}

// the inner split R = P Q of a composite radix
__host__ __device__ constexpr int dft_p(int R) {
    return R == 16 ? 4 : R == 14 ? 2 : R == 12 ? 3 : R == 10 ? 2 : R == 9 ? 3 : R == 8 ? 2 : R == 6 ? 2 : 1;
}

// DFT of R points in registers, natural order in and out
template <typename T, int R, int S> __device__ __forceinline__ void dft(cplx<T> (&v)[R]) {
    if constexpr (R == 2) {
        const cplx<T> a = v[0], b = v[1];
        v[0] = a + b;
        v[1] = a - b;
    } else if constexpr (R == 4) {
        const cplx<T> s02 = v[0] + v[2], d02 = v[0] - v[2], s13 = v[1] + v[3], d = v[1] - v[3];
        const cplx<T> d13 = S < 0 ? cplx<T>{d.y, -d.x} : cplx<T>{-d.y, d.x};
        v[0] = s02 + s13;
        v[2] = s02 - s13;
        v[1] = d02 + d13;
        v[3] = d02 - d13;
    } else if constexpr (R == 3 || R == 5 || R == 7) {
        // pairs (r, R - r): the cosine terms act on their sums, the sine terms on their differences
        constexpr int H = R / 2;
        cplx<T> s[H], d[H];
#pragma unroll
        for (int r = 0; r < H; r++) {
            s[r] = v[r + 1] + v[R - 1 - r];
            d[r] = v[r + 1] - v[R - 1 - r];
        }
        const cplx<T> x0 = v[0];
#pragma unroll
        for (int r = 0; r < H; r++) v[0] = v[0] + s[r];
#pragma unroll
        for (int q = 1; q <= H; q++) {
            cplx<T> a = x0, b{0, 0};
#pragma unroll
            for (int r = 0; r < H; r++) {
                const int m = ((r + 1) * q) % R;
                const T c = (T)cosv<R>(m), sn = (T)S * (T)sinv<R>(m);
                a.x = fma(c, s[r].x, a.x);
                a.y = fma(c, s[r].y, a.y);
                b.x = fma(-sn, d[r].y, b.x);  // i sn d
                b.y = fma(sn, d[r].x, b.y);
            }
            v[q] = a + b;
            v[R - q] = a - b;
        }
    } else {
        constexpr int P = dft_p(R), Q = R / P;
        static_assert(P * Q == R && P > 1, "a composite radix of the table");
        cplx<T> b[P][Q];
#pragma unroll
        for (int j = 0; j < Q; j++) {
            cplx<T> u[P];
#pragma unroll
            for (int r = 0; r < P; r++) u[r] = v[j + Q * r];
            dft<T, P, S>(u);
#pragma unroll
            for (int q = 0; q < P; q++) b[q][j] = mul_root<T, R, S>(u[q], j * q);
        }
#pragma unroll
        for (int q = 0; q < P; q++) {
            dft<T, Q, S>(b[q]);
#pragma unroll
            for (int t = 0; t < Q; t++) v[q + P * t] = b[q][t];
        }
    }
}

// The transform lengths that have kernels, and their split L = R1 R2 with R1 >= R2. The radices
// are 4..16 and the lengths 11 to 25 % apart, so that a product of two of them lies a few percent above
// any length from 400 up to 65536.
#define QS_FFT_LENGTHS(X) \
    X(4, 4) X(5, 4) X(6, 4) X(7, 4) X(8, 4) X(6, 6) X(8, 5) X(8, 6) X(8, 7) X(8, 8) X(9, 8) X(10, 8) X(12, 8) X(14, 8) \
    X(16, 8) X(12, 12) X(16, 10) X(16, 12) X(16, 14) X(16, 16)

}  // namespace qs
