// Internal (C++) interfaces shared between the translation units of the
// native library.  The public boundary is the C ABI in include/jaxhps_gb300.h.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "hps_common.cuh"

struct CUtensorMap_st;   // CUtensorMap of cuda.h

namespace hps {

// D = alpha*A@B + beta*C over a strided batch (row-major).  C may be null
// (then beta is ignored) and may alias D.  digits: FP64 and complex128 products
// may run on the digit kernels (gemm_f64_tc.cu) by the rule for their sizes,
// where the caller knows that no large entry of A's rows meets only small ones
// of B's columns.
template <class T>
cudaError_t gemm_batched(int M, int N, int K, T alpha, const T* A, long long lda, long long sA,
                         const T* B, long long ldb, long long sB, T beta, const T* C, long long ldc,
                         long long sC, T* D, long long ldd, long long sD, int batch, cudaStream_t st,
                         bool digits = true);

// Batched inverse by Gauss-Jordan elimination with partial (row) pivoting.
// X may alias A.  info[b] = 0 on success, k+1 if the k-th pivot was zero.
// flags: INV_TENSOR_MEMORY lets FP32 blocks of 64 < n <= 224 use the
// tensor-memory kernel (while inverse_tc_policy() is 1); INV_BLOCK_RECURSIVE
// lets FP32 matrices of n >= 224 use the recursive 2 x 2 block inversion
// (pivots within its smallest blocks only; while inverse_rec_policy() is 1).
enum InverseFlags : int { INV_TENSOR_MEMORY = 1, INV_BLOCK_RECURSIVE = 2 };
size_t inverse_workspace_bytes(int dtype, int n, int batch);
template <class T>
cudaError_t inverse_batched(int n, const T* A, long long lda, long long sA, T* X, long long ldx,
                            long long sX, int batch, int* info, void* ws, size_t ws_bytes,
                            cudaStream_t st, int flags = 0);
// FP64 / complex128 inverses refined from the single-precision one
// (inverse_refined.cu), for n > 64: info[b] = 0, or INV_NOT_REFINED where the
// refinement does not reach FP64 (X[b] is then not the inverse).  X may alias
// A; info is needed.
constexpr int INV_NOT_REFINED = -2;
bool inverse_refined_takes(int dtype, int n);
size_t inverse_refined_workspace_bytes(int dtype, int n, int batch);
template <class T>
cudaError_t inverse_refined(int n, const T* A, long long lda, long long sA, T* X, long long ldx, long long sX, int batch,
                            int* info, void* ws, size_t ws_bytes, cudaStream_t st);
int inverse_rec_policy();
int set_inverse_rec_policy(int policy);

// FP32 GEMM on the tensor cores (TF32 split into hi + lo, three products);
// gemm_tc_error() reports whether a CTA's bounded wait ever ran out.
cudaError_t gemm_tf32x3(int M, int N, int K, float alpha, const float* A, long long lda, long long sA,
                        const float* B, long long ldb, long long sB, float beta, const float* C, long long ldc,
                        long long sC, float* D, long long ldd, long long sD, int batch, cudaStream_t st);
cudaError_t gemm_tf32x3_c64(int M, int N, int K, float alpha, const c64* A, long long lda, long long sA,
                            const c64* B, long long ldb, long long sB, float beta, const c64* C, long long ldc,
                            long long sC, c64* D, long long ldd, long long sD, int batch, cudaStream_t st);
// Warp-specialised TMA + tcgen05 3xTF32 kernel for N <= 64 (gemm_tc.cu):
// cudaErrorNotSupported for layouts it does not take (gemm_tma_supported).
bool gemm_tma_supported(int M, int N, int K, const float* A, long long lda, long long sA, const float* B,
                        long long ldb, long long sB, int batch);
cudaError_t gemm_tma_f32(int M, int N, int K, float alpha, const float* A, long long lda, long long sA,
                         const float* B, long long ldb, long long sB, float beta, const float* C, long long ldc,
                         long long sC, float* D, long long ldd, long long sD, int batch, cudaStream_t st);
// The same products in 128 x 128 tiles with TMA loads and specialised warps
// (gemm_tc_wide.cu); cudaErrorNotSupported for layouts TMA does not take
// (16-byte aligned bases, rows and batch strides).
cudaError_t gemm_wide_f32(int M, int N, int K, float alpha, const float* A, long long lda, long long sA, const float* B,
                          long long ldb, long long sB, float beta, const float* C, long long ldc, long long sC, float* D,
                          long long ldd, long long sD, int batch, cudaStream_t st);
cudaError_t gemm_wide_c64(int M, int N, int K, float alpha, const c64* A, long long lda, long long sA, const c64* B,
                          long long ldb, long long sB, float beta, const c64* C, long long ldc, long long sC, c64* D,
                          long long ldd, long long sD, int batch, cudaStream_t st);
// Tensor map of a batch of row-major FP32 matrices (d0 inner): box0 x box1
// boxes, 128-byte swizzled or plain; false where TMA does not take it.
bool tma_map_f32(::CUtensorMap_st* map, const float* base, long long d0, long long d1, long long d2, long long ld,
                 long long sb, int box0, int box1, bool swizzle);
// FP64 / complex128 products (real alpha, beta) from 8-bit digits on the FP16
// tensor cores (gemm_f64_tc.cu).  K >= 1; D may alias C only.  `skip`: device
// flags, one per product of the batch; where set, the product is left out.
cudaError_t gemm_f64_tc(int M, int N, int K, double alpha, const double* A, long long lda, long long sA,
                        const double* B, long long ldb, long long sB, double beta, const double* C, long long ldc,
                        long long sC, double* D, long long ldd, long long sD, int batch, cudaStream_t st,
                        const int* skip = nullptr);
cudaError_t gemm_c128_tc(int M, int N, int K, double alpha, const c128* A, long long lda, long long sA, const c128* B,
                         long long ldb, long long sB, double beta, const c128* C, long long ldc, long long sC, c128* D,
                         long long ldd, long long sD, int batch, cudaStream_t st,
                         const int* skip = nullptr);
// Products of blocks of the same matrices in one launch of the digit kernel
// (gemm_f64_tc.cu): for every group, rows m0 .. m0 + m - 1 and columns n0 ..
// n0 + n - 1 of D = alpha A B + beta C with K running over the columns of A and
// rows of B of its segments.  T = double or c128.  The groups' blocks of D do
// not overlap; D may alias C only.
constexpr int GEMM_GROUPS = 32, GEMM_SEGS = 4;
struct GemmGroup {
  int m0, m, n0, n, segs, k0[GEMM_SEGS], len[GEMM_SEGS];
};
template <class T>
cudaError_t gemm_groups(const GemmGroup* groups, int n, double alpha, const T* A, long long lda, long long sA, const T* B,
                        long long ldb, long long sB, double beta, const T* C, long long ldc, long long sC, T* D,
                        long long ldd, long long sD, int batch, cudaStream_t st);
// The same for T = float or c64 in multiply-adds (gemm.cu), D = alpha A B (+ D).
template <class T>
cudaError_t gemm_groups_simt(const GemmGroup* groups, int n, T alpha, const T* A, long long lda, long long sA, const T* B,
                             long long ldb, long long sB, bool add_d, T* D, long long ldd, long long sD, int batch,
                             cudaStream_t st);
// D += A B for the rows of the groups (their n0 and n are not used) and N <= 8
// columns, any type (gemm.cu); M rows in all.
template <class T>
cudaError_t skinny_groups(const GemmGroup* groups, int n, int M, int N, const T* A, long long lda, long long sA,
                          const T* B, long long ldb, long long sB, T* D, long long ldd, long long sD, int batch,
                          cudaStream_t st);
// Products of operands split into FP16 digits ahead of them (gemm_digits.cu),
// batches of real (M x N x K) products; complex ones by their real views: A's
// rows of (re, im), N and K doubled, B (K / 2 x N / 2) complex (`cplx`).
// digit_rows / digit_cols write the leading `digits` (8, 6 or 4) of A and B
// and the largest high words of their rows (batch, M) or columns (batch, N) to
// `top`; with `round` (4 digits) B becomes what they hold.  digit_product:
// D = (neg ? -1 : 1) A B + C from the digits t + u < max(da, db), for (da, db) =
// (8, 8), (8, 4), (6, 6) or (4, 4), to 2^-60, 2^-60, 2^-47 and 2^-31 of the
// largest product of a row's and a column's entries; NaN where a row of A or a
// column of B holds an infinity or a NaN, zeros where all are below 2^-958.  C may alias D.  Leading dimensions and strides in doubles;
// `skip` as above.
size_t digit_rows_bytes(int M, int K, int digits);
size_t digit_cols_bytes(int N, int K, int digits);
cudaError_t digit_rows(int digits, int M, int K, const double* X, long long ldx, long long sX, int* top, void* out,
                       int batch, const int* skip, cudaStream_t st);
cudaError_t digit_cols(int digits, bool cplx, bool round, int N, int K, double* X, long long ldx, long long sX, int* top,
                       void* out, int batch, const int* skip, cudaStream_t st);
cudaError_t digit_product(int da, int db, int M, int N, int K, bool cplx, bool neg, const void* A, const int* ta,
                          const void* B, const int* tb, const double* C, long long ldc, long long sC, double* D,
                          long long ldd, long long sD, int batch, const int* skip, cudaStream_t st);
// Device addresses of the tensor-core kernels' failure flag and wait limit.
cudaError_t tc_wait_state(int** err, const long long** limit);
int gemm_tc_error();
// Reads the flag and clears it (both synchronise with the device).
int gemm_tc_error_reset();
// Spin limits of the bounded waits on the current device (polls < 0: keep);
// the previous value is returned through `previous` when it is not null.
cudaError_t set_tc_spin_limit(long long polls, long long* previous);
cudaError_t set_panel_spin_limit(long long polls, long long* previous);
cudaError_t set_itc_spin_limit(long long polls, long long* previous);

// FP32 batched inverse with the tableau in tensor memory (inverse_tc.cu),
// for 64 < n <= 224; used by inverse_batched<float> for the calls that pass
// tensor_memory = true while inverse_tc_policy() is 1, for every call at 2.
bool inverse_tc_supported(int n);
cudaError_t inverse_tc_f32(int n, const float* A, long long lda, long long sA, float* X, long long ldx,
                           long long sX, int batch, int* info, cudaStream_t st);
int inverse_tc_policy();
int set_inverse_tc_policy(int policy);

// Autotuning table of the FP32 products (gemm.cu): per-shape kernel variant,
// a forced variant for timing, and the shape recorder.
int gemm_tune_set(int M, int N, int K, int batch, int variant);
void gemm_tune_clear();
int gemm_force_variant(int variant);
// Whether FP32 products may be grouped on the SIMT tiles: no variant forced, no
// policy that sends every product to the tensor cores.
bool gemm_simt_blocks();
long long gemm_shapes(int mode, long long* out, long long cap);
// Whether that policy lets FP64 products use the tensor cores.
bool f64_products_on_tensor_cores();
// Sets the tensor-core policy of gemm_batched (0, 1, 2); returns the old one.
int set_gemm_policy(int p);

// Largest n served by the register-resident single-CTA kernel.
int inverse_small_nmax(int dtype);

// Number of kernels this library has launched (process-wide), reported by
// hps_launch_count().  Every launch site calls note_launch().
void note_launch();

// Kernel classes for the live profiler (hps_profile_begin/end).
// 5-7 single out the kernels that carry most of a mixed-precision step: the
// TMA GEMM (work in algorithmic bytes), the FP32-pair residual update (bytes)
// and the tensor-memory leaf inverse (flops).
enum KernelClass : int {
  KC_GEMM = 1,
  KC_INVERSE = 2,
  KC_MOVE = 3,
  KC_RESIDUAL = 4,
  KC_GEMM_TMA = 5,
  KC_RESIDUAL_DF = 6,
  KC_INVERSE_TC = 7
};

// RAII scope placed around one kernel launch (or a sequence of them): when
// the profiler is armed for `cls`, records a CUDA event pair on `st` around
// it and adds its algorithmic flop (or byte) count.  Scopes opened inside
// another scope record nothing; the outermost one owns the time.
struct ProfScope {
  bool on;
  cudaStream_t st;
  int slot;
  ProfScope(int cls, cudaStream_t st, double work);
  ~ProfScope();
};

// Records an error message for hps_last_error().
void set_error(const char* fmt, ...);

}  // namespace hps
