// qs_common.cuh -- shared definitions of the B200 NEGF solver.
//
// Device data layout (HBM), with nA active states, n energies, Nf padded FFT length:
//   X, F, Fold, xold   SCF vectors, energy-major: block w (3 nA^2 doubles) holds the site
//                      pairs I <= J, J by J (site = two consecutive active states): for I < J
//                      12 complex values, the 2x2 blocks G^r_IJ, G^r_JI, G^<_IJ (rows fastest);
//                      for I = J G^r_II, the element G^<_01 of the block and its two Im G^<_aa.
//                      This is a fixed permutation of the reference's pack_gf block
//                      (common/linear_algebra.f90:155-191), so every Broyden quantity
//                      (norms, dots, updates) is the reference's up to summation order.
//   Sig                Sigma2 for each energy: per site pair (I <= J, index J(J+1)/2 + I)
//                      the 12 values Sigma^r_IJ, Sigma^r_JI, Sigma^<_IJ; the lower blocks of
//                      Sigma^< follow from Sigma^<_JI = -Sigma^<_IJ^+. Zero for pairs without
//                      interaction (written once, at creation).
//   Y                  FFT intermediates of the interacting pairs: [pair][l1][m2][12] of the
//                      four-step split Nf = N1*N2, spectra and inverse transforms in place.
//   gRd, gLd           diagonals (n x nA complex) for the sanity check.
//   onsL, dosd, atomL, trU, trD   final-sweep arrays, energy-major (reference layout).
#pragma once
#include <cmath>
#include <functional>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "qsb200.h"

namespace qs {

template <typename T>
struct __align__(2 * sizeof(T)) cplx {
    T x, y;
};
using zc = cplx<double>;
using cc = cplx<float>;

template <typename T> __host__ __device__ __forceinline__ cplx<T> mk(T a, T b) { return cplx<T>{a, b}; }
template <typename T> __host__ __device__ __forceinline__ cplx<T> operator+(cplx<T> a, cplx<T> b) { return {a.x + b.x, a.y + b.y}; }
template <typename T> __host__ __device__ __forceinline__ cplx<T> operator-(cplx<T> a, cplx<T> b) { return {a.x - b.x, a.y - b.y}; }
template <typename T> __host__ __device__ __forceinline__ cplx<T> operator-(cplx<T> a) { return {-a.x, -a.y}; }
template <typename T> __host__ __device__ __forceinline__ cplx<T> operator*(cplx<T> a, cplx<T> b) {
    return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
template <typename T> __host__ __device__ __forceinline__ cplx<T> operator*(T s, cplx<T> a) { return {s * a.x, s * a.y}; }
template <typename T> __host__ __device__ __forceinline__ cplx<T> conj(cplx<T> a) { return {a.x, -a.y}; }
// a += b*c (complex fused multiply-add)
template <typename T> __host__ __device__ __forceinline__ void cfma(cplx<T> &a, cplx<T> b, cplx<T> c) {
    a.x = fma(b.x, c.x, a.x);
    a.x = fma(-b.y, c.y, a.x);
    a.y = fma(b.x, c.y, a.y);
    a.y = fma(b.y, c.x, a.y);
}
// a += b*conj(c)
template <typename T> __host__ __device__ __forceinline__ void cfma_conj(cplx<T> &a, cplx<T> b, cplx<T> c) {
    a.x = fma(b.x, c.x, a.x);
    a.x = fma(b.y, c.y, a.x);
    a.y = fma(-b.x, c.y, a.y);
    a.y = fma(b.y, c.x, a.y);
}
template <typename T> __host__ __device__ __forceinline__ T cabs1(cplx<T> a) { return fabs(a.x) + fabs(a.y); }
// 1/a by Smith's method (no overflow for |a| near the range limits)
template <typename T> __device__ __forceinline__ cplx<T> crecip(cplx<T> a) {
    if (fabs(a.x) >= fabs(a.y)) {
        T r = a.y / a.x, d = a.x + a.y * r;
        return {T(1) / d, -r / d};
    } else {
        T r = a.x / a.y, d = a.y + a.x * r;
        return {r / d, T(-1) / d};
    }
}

// offset (doubles) of the pair (I <= J) in a block of an SCF vector
__host__ __device__ __forceinline__ int dl_block(int I, int J) { return 12 * J * J + 24 * I; }
// offsets of G^r_ij, of G^<_ij (i < j) and of Im G^<_ii
__host__ __device__ __forceinline__ int dl_r(int i, int j) {
    const int I = i >> 1, J = j >> 1, e = 2 * ((i & 1) + 2 * (j & 1));
    return I <= J ? dl_block(I, J) + e : dl_block(J, I) + 8 + e;
}
__host__ __device__ __forceinline__ int dl_l(int i, int j) {
    const int I = i >> 1, J = j >> 1;
    return I < J ? dl_block(I, J) + 16 + 2 * ((i & 1) + 2 * (j & 1)) : dl_block(I, I) + 8;
}
__host__ __device__ __forceinline__ int dl_d(int i) { return dl_block(i >> 1, i >> 1) + 10 + (i & 1); }
// the pair (I <= J) in an energy's Sigma2, its values, Sigma^r_ij and Sigma^<_ij
__host__ __device__ __forceinline__ int64_t sig_block(int I, int J) { return (int64_t)12 * (J * (J + 1) / 2 + I); }
__host__ __device__ __forceinline__ int64_t sig_stride(int nA) { return (int64_t)3 * (nA / 2) * (nA + 2); }
__device__ __forceinline__ zc sig_r(const zc *S, int i, int j) {
    const int I = i >> 1, J = j >> 1, e = (i & 1) + 2 * (j & 1);
    return S[I <= J ? sig_block(I, J) + e : sig_block(J, I) + 4 + e];
}
// the stored element that Sigma^<_ij equals (upper blocks) or is minus the conjugate of (lower ones)
__device__ __forceinline__ const zc *sig_l_at(const zc *S, int i, int j) {
    const int I = i >> 1, J = j >> 1;
    return S + (I <= J ? sig_block(I, J) + 8 + (i & 1) + 2 * (j & 1) : sig_block(J, I) + 8 + (j & 1) + 2 * (i & 1));
}
__device__ __forceinline__ zc sig_l(const zc *S, int i, int j) {
    const zc v = *sig_l_at(S, i, j);
    return (i >> 1) <= (j >> 1) ? v : zc{-v.x, v.y};
}

constexpr double PI = 3.14159265358979323846;
constexpr int SMEM_MAX = 232448;  // max dynamic shared memory per block on sm_100 (227 KB)

// The Gauss-Jordan kernel keeps the N x N complex matrix in shared memory when it fits next to its
// 1.6 KB of static shared memory.
constexpr int DYSON_SMEM_MAXN = 120;
inline bool dyson_fits_smem(int N) { return N <= DYSON_SMEM_MAXN; }

// the four-step split of the padded length Nf = N1 * N2 (>= 2 n - 1)
struct FftPlan {
    int Nf, N1, N2;
};

// ---------------------------------------------------------------------------------
// The solver handle (one per qs_create).
// ---------------------------------------------------------------------------------
struct DeviceBuf {
    void *p = nullptr;
    size_t bytes = 0;
};

}  // namespace qs

namespace qs {
// kernel families timed by the optional profiler (qs_profile)
enum KernelFamily { K_DYSON = 0, K_KELDYSH, K_SIG2A, K_SIG2B, K_SIG2C, K_FINAL, K_BROYDEN, K_REDUCE, K_OTHER, K_NFAM };
}  // namespace qs

struct qs_handle {
    // optional per-launch CUDA-event timing on the solver stream
    bool prof_on = false;
    std::vector<cudaEvent_t> prof_ev;           // pool, 2 per timed launch
    std::vector<int> prof_fam;                  // family of launch i (events 2i, 2i+1)
    double prof_ms[qs::K_NFAM] = {0};
    int64_t prof_count[qs::K_NFAM] = {0};
    // problem (host copies)
    int Norb = 0, N_sites = 0, N_atoms = 0, order = 0, n = 0, device = 0, precision = 0;
    double mu = 0, beta = 0, delta = 0, alpha_mix = 0.5, tolf = 1e-6, tolf_order1 = 1e-8;
    int nhist = 16, maxscf = 300;
    double mixed_switch = 1e-4;  // QS_PREC_MIXED: FP32 max|F| below which the residual turns FP64
    bool single = true;
    std::vector<double> H, GammaL, GammaR, U_site, omega;  // complex arrays as double pairs
    std::vector<int> atom_norb, atom_first;
    // active subspace (setup_storage), 0-based indices
    int nA = 0, nS = 0, nCL = 0, nAs = 0, n_int_sites = 0;
    std::vector<int> act, pos, sup, cl, asite;
    std::vector<char> site_int, site_act;
    bool has_atomL = false;
    std::vector<int> atom_off;
    int64_t n_vec = 0, nblk = 0;
    // device model arrays
    qs::zc *d_Hemb = nullptr, *d_Sig1 = nullptr, *d_GamLs = nullptr, *d_GamRs = nullptr, *d_GamLcl = nullptr;
    int *d_pos = nullptr;
    int *d_kd_cidx = nullptr;  // contact states of GamLs / GamRs (the lead terms of SL)
    int kd_nc = -1;
    int *d_act = nullptr, *d_sup = nullptr, *d_cl = nullptr, *d_atom_first = nullptr, *d_atom_norb = nullptr,
        *d_atom_off = nullptr, *d_site_int = nullptr;
    double *d_omega = nullptr, *d_U = nullptr;
    // SCF vectors and Broyden history (order 2: n_vec doubles; order 1: tiny)
    double *d_x = nullptr, *d_F = nullptr, *d_Fold = nullptr, *d_xold = nullptr;
    void *d_hdF = nullptr, *d_hU = nullptr;  // nhist columns, float (single history) or double
    // second-order self-energies and the FFT
    qs::FftPlan fft{};
    qs::zc *d_tw = nullptr;  // W_Nf^k
    qs::zc *d_Sig = nullptr;
    qs::zc *d_Y = nullptr;          // y_elems values: the FFT intermediates, then the sweep's scratch
    int *d_dl_perm = nullptr;       // position in a device block of each element of a pack_gf block
    double *sig2_scale = nullptr;   // U_I U_J hbar^2 (delta/2pi)^2 / Nf per interacting site pair
    int2 *sig2_pairs = nullptr;     // interacting site pairs I <= J
    int sig2_npairs = 0;
    int sig2_occ[2][3] = {};        // resident blocks per SM of kernels A, B, C: FP32, FP64 forms
    // sweep scratch
    qs::zc *d_G = nullptr;  // Dyson output (G_AA for all energies, or full G for a chunk)
    size_t G_chunk = 0;     // energies per chunk in full-G mode
    bool small_chunks = false;  // order 2: no memory beyond G_AA of every energy for them
    qs::zc *d_T = nullptr;  // per-CTA GEMM scratch
    size_t T_slots = 0, T_bytes = 0;
    qs::zc *d_Gws = nullptr;  // Gauss-Jordan workspace for orders above the shared-memory limit when nA < N
    size_t ws_slots = 0;
    qs::zc *d_gRd = nullptr, *d_gLd = nullptr, *d_onsL = nullptr, *d_atomL = nullptr;
    double *d_dosd = nullptr, *d_trU = nullptr, *d_trD = nullptr;
    qs::zc *d_Glt0 = nullptr;  // G^<(t=0) on-site blocks, 4 per site
    double *d_red = nullptr;   // reduction scratch
    size_t red_len = 0;
    double *d_rpart = nullptr;  // partial sums of the reductions over energies, REDUCE_PART doubles
    int *d_rcnt = nullptr;      // their arrival counters, REDUCE_CNT ints (zero between launches)
    int *d_info = nullptr;     // first singular energy (+1), 0 if none
    // page-locked host memory of the values read in every step (host_scratch): 4 doubles a state
    // (the sanity sums), then d_info, the norms, the Gram column and gamma
    double *pin = nullptr;
    int pin_states = 0;
    std::vector<double> pin_own;  // in its place when the pool has no slot
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    // host state
    std::vector<double> G_less_t0, G_less_obs, Sig1;  // Norb*Norb complex
    double J_up = 0, J_down = 0;
    bool have_x = false, final_done = false;
    std::vector<double> x1_host;  // order-1 SCF vector
    std::string err;
    size_t bytes_allocated = 0;
    std::vector<void *> allocs;
    // CUDA graphs of the FP64 residual's launches, one per (x, F) the Broyden loop uses (x and F
    // alternate between two buffers each): replayed instead of re-launching, at every voltage
    struct ResidualGraph {
        const double *x = nullptr;
        double *F = nullptr;
        cudaGraphExec_t exec = nullptr;
        int64_t launches = 0;  // kernels in the graph (added to the launch count per replay)
    };
    ResidualGraph graphs[4];
    double *d_V = nullptr;     // the voltage the Keldysh kernels read, and its value (NaN: none yet)
    double V_dev = NAN;
    bool graphs_off = false;   // a capture failed: eager launches from then on
    int64_t graph_replays = 0;
};

namespace qs {

// error handling: every CUDA call inside the library goes through this
#define QS_CUDA(h, call)                                                                        \
    do {                                                                                        \
        cudaError_t _e = (call);                                                                \
        if (_e != cudaSuccess) {                                                                \
            (h)->err = std::string(#call) + ": " + cudaGetErrorString(_e);                      \
            return -(int)_e;                                                                     \
        }                                                                                       \
    } while (0)

int dalloc(qs_handle *h, void **p, size_t bytes);
// scratch of the reductions over energies: one partial per block for at most REDUCE_BLOCKS blocks
// of 32 complex columns, a counter per group of blocks that share an output
constexpr int REDUCE_BLOCKS = 592, REDUCE_PART = REDUCE_BLOCKS * 64, REDUCE_CNT = REDUCE_BLOCKS;
int reduce_scratch(qs_handle *h, int states);
// h->pin from a process-wide pool of page-locked slots (64 of 20 KB, allocated with the first handle), so that
// the small copies of a step neither block the host nor synchronise; a handle that gets no slot uses
// ordinary memory. Returned by release_all.
void host_scratch(qs_handle *h, int states);
void host_scratch_release(qs_handle *h);
inline int *pin_info(qs_handle *h) { return (int *)(h->pin + 4 * (size_t)h->pin_states); }
inline double *pin_broyden(qs_handle *h) { return h->pin + 4 * (size_t)h->pin_states + 1; }
constexpr int PIN_BROYDEN = 4 + 3 * 32;  // norms, (Gram, dF^T F) pairs, gamma
// The dynamic shared-memory cap of a kernel is a process-wide attribute: it is always set
// to the device maximum (a cap, not a reservation), so that handles that size the same
// kernel differently, on other threads, never lower it under each other's launches.
inline cudaError_t smem_cap(const void *kernel) {
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(SMEM_MAX - fa.sharedSizeBytes));
}

// every kernel launch of the library is counted (qs_kernel_launches)
void count_launch();
void count_launches(int64_t k);
// bracket a launch with events when profiling is on: idx = prof_begin(...); launch; prof_end(h, idx)
int prof_begin(qs_handle *h, int fam, bool count = true);
void prof_end(qs_handle *h, int idx);

__device__ __forceinline__ double fermi_d(double w, double V, double mu, double beta) {
    // src/green_functions.f90:74-84 (hbar = 1)
    double arg = (w - mu + V) * beta;
    return 1.0 / (exp(fmin(arg, 700.0)) + 1.0);
}

// arguments of the Gauss-Jordan kernels
struct DysonArgs {
    int N, nA, iw0, iw1;
    const zc *Hemb, *Sig1, *Sig;
    int64_t sig_ld;
    const int *pos;  // full index -> active index, -1 if inactive
    const int *act;
    const double *omega;
    int use_sigma, order2;
    int out_mode;  // 0: G_AA for energy iw at Gout[iw*nA^2]; 1: full G at Gout[(iw-iw0)*N^2]
    zc *Gout;
    zc *ws;        // global workspace (N^2 per block) when the matrix is not in shared memory
    int *info;     // min over energies of (iw + 1) with a zero pivot; INT_MAX if none
    const zc *Ain; // batched-inversion mode: matrices to invert (nullptr for the sweep)
    int *info_each;
    int zero_of_inf;  // 1 / inf = 0 for a pivot, else NaN: orders below 16, and qs_invert_batched_noalloc
    int inplace;   // kernels whose matrix is in global memory: in Gout itself (N x N each) instead of ws
};
// the blocked elimination in shared memory (dyson_blk.cu), N <= DYSON_SMEM_MAXN; 0 or a CUDA error (< 0)
int launch_dyson_blk(cudaStream_t st, const DysonArgs &a);
// the same with the matrix in global memory (dyson_l2.cu), 16 < N <= 256; DYSON_L2_SLOTS workspaces unless inplace
constexpr int DYSON_L2_SLOTS = 2 * 148;
int launch_dyson_l2(cudaStream_t st, const DysonArgs &a);
bool dyson_l2_fits(int N);

// arguments of the Keldysh kernels (sweep modes M_INIT2 / M_SCF2)
struct KeldyshArgs {
    int nA, n;
    int64_t nblk;
    const zc *G;     // G_AA per energy (nA^2 complex)
    const zc *Sig;   // Sigma2 per energy, or nullptr
    int64_t sig_ld;  // its values per energy
    const zc *GamLs, *GamRs;
    const double *omega;
    const double *V;    // in device memory: a captured step serves every voltage
    double mu, beta;
    double *out;        // DL blocks (SCF vector)
    const double *xsub; // subtracted (F = out - x), or nullptr
    zc *gRd, *gLd;      // diagonals, or nullptr
    zc *Tws;            // per-block scratch, nA^2 complex
    int *err;           // set to 1 if a bounded tensor-core wait gave up (tcgen05 kernel)
    const int *cidx;    // the contact states: rows/columns where GamLs or GamRs is non-zero
    int nc;             // their number (-1: not known)
};
// arguments of the per-energy outputs (sweep modes M_SCF1 / M_FINAL)
struct FinalArgs {
    int N, nS, nA, nCL, N_sites, N_atoms, iw0, iw1, mode;
    const zc *G;  // full G per energy of the chunk
    const int *sup, *act, *pos, *cl, *site_int, *atom_first, *atom_norb, *atom_off;
    const zc *GamLs, *GamRs, *GamLcl, *Sig;
    const double *omega;
    double V, mu, beta;
    zc *Tws;
    double *dosd, *trU, *trD;
    zc *onsL, *atomL, *gRd, *gLd;
    int atomL_ld;
    const int *cidx;  // the contact states, as in KeldyshArgs
    int nc;
};
// the Keldysh step with both operands in shared memory (keldysh_sm.cu): nA <= 48
int launch_keldysh_sm(qs_handle *h, const KeldyshArgs &k);
bool keldysh_sm_fits(int nA);
// the same by blocks of 32 rows (keldysh_rows.cu): nA <= 256
int launch_keldysh_rows(qs_handle *h, const KeldyshArgs &k);
bool keldysh_rows_fits(int nA);
int launch_final_rows(qs_handle *h, const FinalArgs &f);
// the FP32-phase Keldysh step of a QS_PREC_MIXED solve on the fifth-generation tensor cores
// (keldysh_tf32.cu): 32 <= nA <= 128; returns -1 for other sizes
int launch_keldysh_tf32(qs_handle *h, const KeldyshArgs &k);
bool keldysh_tf32_fits(int nA);

// launchers (implemented in the .cu files)
int sigma2_setup(qs_handle *h);
// the padded transform length and its split for a grid of n energies; {0, 0, 0} if there is none
FftPlan sigma2_plan(int n);
// interacting site pairs I <= J of a handle
int sigma2_count_pairs(const qs_handle *h);
// values of the handle's d_Y and of the sweep's per-block scratch at its end (order 2)
size_t sweep_scratch_elems(const qs_handle *h);
size_t y_elems(const qs_handle *h);
// Sigma2^r, Sigma2^< as n blocks of nA x nA, column-major
int sigma2_unblock(qs_handle *h, zc *SR, zc *SL);
// fp32: FFTs, 2x2 algebra and spectra in FP32 (QS_PREC_MIXED handles), Sigma written in FP64
int sigma2_compute(qs_handle *h, const double *d_x, bool fp32 = false);
// autotuner (autotune.cu): kinds of decisions and the variants they choose between (kinds 2 and 3
// are no longer decided: the Sigma2 kernels have one form per length)
// TUNE_KELDYSH32: the Keldysh step of a mixed solve's FP32 phase, where the 3xTF32 tensor-core
// kernel (keldysh_tf32.cu) competes with the two FP64 ones
enum TuneKind { TUNE_DYSON = 0, TUNE_KELDYSH = 1, TUNE_KELDYSH32 = 4 };
// DYSON_BLOCKED: dyson_blk or dyson_l2 by the order
enum { DYSON_BLOCKED = 1, DYSON_UNBLOCKED = 2, KELDYSH_TC = 1, KELDYSH_CUDA = 2, KELDYSH_TF32 = 3 };
// the size key of a decision: the matrix order and the octave of the grid length (how many
// energies each SM gets changes which variant wins)
inline int tune_key(int order, int n) {
    int lg = 0;
    while ((2 << lg) <= n) lg++;
    return order + 1024 * lg;
}
int tune_get(int kind, int size);
bool tune_enabled();
void tune_put(int kind, int size, int choice);
// launch(cand[c]) for the recorded choice of (kind, size); the first time, every candidate
// is launched and timed and the fastest recorded. fallback: the choice without tuning.
int tune_launch(qs_handle *h, int kind, int size, const int *cand, int ncand, int fallback,
                const std::function<int(int)> &launch);
// max |v_i| over a device vector (uses the Broyden reduction scratch)
int vec_maxabs(qs_handle *h, const double *d_v, int64_t n, double &mx);
int equal_time_lesser_sigma1(qs_handle *h, const double *d_x);
// h->d_V = V, on the handle's stream
int set_voltage(qs_handle *h, double V);
enum SweepMode { M_INIT2 = 1, M_SCF2 = 2, M_SCF1 = 3, M_FINAL = 4 };
// fp32: the FP32 phase of a QS_PREC_MIXED solve (M_SCF2 only: tensor-core Keldysh products)
int sweep(qs_handle *h, int mode, double V, bool use_sigma, double *d_out, const double *d_x, bool fp32 = false);
// d_out[c] = sum over rows of d_A[r ld + c]; with d_B, its sums behind them at d_out[ncols + c]
int sum_over_energies(qs_handle *h, const zc *d_A, int64_t ld, int ncols, int64_t nrows, zc *d_out,
                      const zc *d_B = nullptr);
int sum_over_energies_real(qs_handle *h, const double *d_A, int64_t ld, int ncols, int64_t nrows, double *d_out);
// the same for d_A alone, added in an order that does not depend on the grid (the vector of order 1)
int sum_in_order(qs_handle *h, const zc *d_A, int64_t ld, int ncols, int64_t nrows, zc *d_out);
// batch N x N column-major matrices inverted in place; d_min (or nullptr) receives the smallest
// 1 + b of a singular one, d_each[b] 1 + the step of its first zero pivot
int invert_batched_dev(cudaStream_t st, int N, int batch, zc *d_A, int *d_min, int *d_each, bool zero_of_inf = false);
int convert_ref_to_dl(qs_handle *h, const double *ref, double *dl);
int convert_dl_to_ref(qs_handle *h, const double *dl, double *ref);

// check_diag_sanity (common/scf_checks.f90:59-91) from the per-state sums over energies:
// sumL[i] = sum_w G^<_ii(w), sumRim[i] = sum_w Im G^r_ii(w); state_index maps i to the
// reported (0-based) state label, or nullptr for i itself
struct SanityOut {
    bool runaway = false, unphysical = false;
    int i_worst = 1;
    double n_worst = 0.5, w_worst = 1.0;
};
SanityOut check_diag_sanity(int nb, const std::vector<zc> &sumL, const std::vector<double> &sumRim, double delta,
                            const int *state_index);
void release_all(qs_handle *h);

// Broyden (common/broyden_mixing.f90) on device vectors; the residual is a host callback
// that fills F (device) from x (device) and may set abort.
struct BroydenResidual {
    virtual int operator()(const double *d_x, double *d_F, bool &abort) = 0;
    // called once the stream has been waited for after operator(): what it left to be read then
    virtual int complete(bool &abort) { return 0; }
    // true if the residual just evaluated used another precision than the one before: the
    // (dF, u) pair of this step would mix two different residual functions and is not
    // stored, and the history built on the other function is dropped
    virtual bool precision_changed() const { return false; }
    virtual ~BroydenResidual() = default;
};
struct BroydenOut {
    bool converged = false;
    int n_iter = 0, n_resets = 0;
    double fmax = 0;
    bool aborted = false;
    std::vector<qs_scf_step> log;
};
// column stride (elements) of the Broyden history: n rounded up to a multiple of 4, so that
// every column starts on a 16-byte boundary for the kernels' 4-wide vector accesses
inline int64_t broyden_ld(int64_t n) { return (n + 3) & ~(int64_t)3; }
int broyden_solve_dev(qs_handle *h, BroydenResidual &res, double *&d_x, double *&d_F, double *&d_Fold,
                      double *&d_xold, void *d_hdF, void *d_hU, int64_t n, double alpha_mix, int nhist, int maxscf,
                      double tolf, bool sp, BroydenOut &out);

}  // namespace qs
