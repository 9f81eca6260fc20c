// FP64 and complex128 batched inverses from the single-precision inverse and
// the residual iteration (Schulz, 1933; its fourth-order form first):
//
//   X0 = inverse of A in FP32 / complex64         (inverse*.cu)
//   R  = I - A X0,  X1 = X0 + X0 (R + R^2 + R^3)
//   R  = I - A X1,  X  = X1 + X1 R                where the first R was not small
//
// X0 comes from whichever single-precision kernel its size selects, the block
// inversions among them, which pivot inside blocks of 16 only: on matrices whose
// leading blocks are nearly singular (indefinite leaves of 400 points and more
// with two wavelengths and more across) it may be no starting point.  The second
// residual is what guards the result.
// The products with A and with X run on the digit kernels (gemm_f64_tc.cu,
// FP64 and better, or gemm_digits.cu with the digits that a step needs), the
// powers of R, corrections of R, in single precision: they leave an error of
// about |R|^2 2^-21, so a matrix whose R has row sums of at most 5e-5 is done
// after the first step (leaves: 2e-6 per entry, row sums 2e-5) and left out of
// the second; the others (interface and impedance matrices, up to 1e-2) have
// |R| of at most 1e-8 there, and R^2 is left.  The result carries the rounding
// of R (1e-16) and no elimination's growth.
// The digits each step needs: A always 8 (62 bits); X0 is rounded to 4 (32
// bits, it has 24 good ones) and is from then on that matrix, so that its
// residual is exact with 26 of the 36 digit products; X0 (R + R^2 + R^3) with 6
// is good to 2^-47 |R|, below the single-precision powers; X1 keeps 8 in its
// residual; X1 R with 4 is good to 2^-31 |R|, 5e-18.
//
// Why: elimination is a chain of n dependent pivots.  Its panels are bound by
// the FP64 pipe (two multiply-adds per SM and clock) for many matrices and by
// the pivot exchange for few (3.3 us a column on a cluster), and its
// rank-32 updates read and write the whole matrix n / 32 times; the products
// of size n do not wait for one another's columns.
// A matrix whose second residual is not small, whose single-precision inverse
// met a zero pivot or an overflow, or whose columns are graded (done_kernel)
// gets info = INV_NOT_REFINED, and the caller runs the elimination.
#include "hps_common.cuh"
#include "hps_internal.h"

namespace hps {

namespace {

template <class T> struct Low;
template <> struct Low<double> { using type = float; };
template <> struct Low<c128> { using type = c64; };

__device__ __forceinline__ float to_low(double v) { return (float)v; }
__device__ __forceinline__ c64 to_low(c128 v) { return c64{(float)v.x, (float)v.y}; }
__device__ __forceinline__ double to_high(float v) { return (double)v; }
__device__ __forceinline__ c128 to_high(c64 v) { return c128{(double)v.x, (double)v.y}; }
__device__ __forceinline__ float mag(float v) { return fabsf(v); }
__device__ __forceinline__ float mag(c64 v) { return fabsf(v.x) + fabsf(v.y); }

constexpr int RF_NT = 256;

// The larger part's magnitude as the upper word of its bits.
__device__ __forceinline__ uint32_t top_word(double v) { return (uint32_t)__double2hiint(v) & 0x7fffffffu; }
__device__ __forceinline__ uint32_t top_word(c128 v) { return max(top_word(v.x), top_word(v.y)); }

// out (contiguous) = A in single precision, and the columns' spans: RF_ONE less
// the binary orders by which a column's largest entry lies below its own row's
// largest, the best of the rows (0: a column of zeros).  A warp per row, which
// it reads twice (the second time from L1); a CTA's spans meet in shared memory.
constexpr int RF_ONE = 64, RF_COLS = 4096;
template <class T, class L>
__global__ void __launch_bounds__(RF_NT) lower_kernel(int n, const T* __restrict__ A, long long lda, long long sA, L* out,
                                                      int* span) {
  __shared__ int best[RF_COLS];
  const long long b = blockIdx.y, nn = (long long)n * n;
  const int lane = threadIdx.x & 31, step = gridDim.x * (RF_NT / 32);
  for (int c0 = 0; c0 < n; c0 += RF_COLS) {
    const int c1 = min(n, c0 + RF_COLS);
    for (int j = c0 + threadIdx.x; j < c1; j += RF_NT) best[j - c0] = 0;
    __syncthreads();
    for (int i = blockIdx.x * (RF_NT / 32) + (threadIdx.x >> 5); i < n; i += step) {
      const T* a = A + b * sA + i * lda;
      uint32_t m = 0;
#pragma unroll 4
      for (int j = lane; j < n; j += 32) m = max(m, top_word(a[j]));
      const int e = (int)(__reduce_max_sync(0xffffffffu, m) >> 20);
#pragma unroll 4
      for (int j = c0 + lane; j < c1; j += 32) {
        const T v = a[j];
        out[b * nn + (long long)i * n + j] = to_low(v);
        const uint32_t w = top_word(v);
        const int s = w ? max(1, RF_ONE + (int)(w >> 20) - e) : 0;
        if (s > best[j - c0]) atomicMax(&best[j - c0], s);
      }
    }
    __syncthreads();
    for (int j = c0 + threadIdx.x; j < c1; j += RF_NT)
      if (best[j - c0] > span[b * n + j]) atomicMax(span + b * n + j, best[j - c0]);
    __syncthreads();
  }
}

// out = in, with zeros for what is not finite (a singular or overflowing
// matrix: its residual is then not small, and no product meets infinities)
template <class T, class L>
__global__ void __launch_bounds__(RF_NT) raise_kernel(long long total, const L* __restrict__ in, T* out) {
  for (long long e = blockIdx.x * (long long)RF_NT + threadIdx.x; e < total; e += (long long)gridDim.x * RF_NT)
    out[e] = mag(in[e]) < __int_as_float(0x7f800000) ? to_high(in[e]) : zero<T>();
}

// R (= -A X) += I, its single-precision copy (first step), and the largest row
// sum per matrix (as the bits of a float; NaN as infinity): a warp per row
template <class T, class L>
__global__ void __launch_bounds__(RF_NT) residual_kernel(int n, T* R, L* low, int* top, const int* __restrict__ skip) {
  const long long b = blockIdx.y, nn = (long long)n * n;
  if (skip && skip[b]) return;
  const int lane = threadIdx.x & 31;
  float most = 0.f;
  for (int i = blockIdx.x * (RF_NT / 32) + (threadIdx.x >> 5); i < n; i += gridDim.x * (RF_NT / 32)) {
    T* r = R + b * nn + (long long)i * n;
    float sum = 0.f;
    for (int j = lane; j < n; j += 32) {
      T v = r[j];
      if (j == i) r[j] = v = add(v, one<T>());
      const L l = to_low(v);
      if (low) low[b * nn + (long long)i * n + j] = l;
      sum += mag(l);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    most = fmaxf(most, sum == sum ? sum : __int_as_float(0x7f800000));
  }
  if (lane == 0 && most > 0.f) atomicMax(top + b, __float_as_int(most));
}

// R += Q
template <class T, class L>
__global__ void __launch_bounds__(RF_NT) add_powers_kernel(long long total, T* R, const L* __restrict__ Q) {
  for (long long e = blockIdx.x * (long long)RF_NT + threadIdx.x; e < total; e += (long long)gridDim.x * RF_NT)
    R[e] = add(R[e], to_high(Q[e]));
}

// X (strided) = the first iterate where that is the result
template <class T>
__global__ void __launch_bounds__(RF_NT) keep_kernel(int n, const T* __restrict__ Q, T* X, long long ldx, long long sX,
                                                     const int* __restrict__ skip) {
  const long long b = blockIdx.y, nn = (long long)n * n;
  if (!skip[b]) return;
  for (long long e = blockIdx.x * (long long)RF_NT + threadIdx.x; e < nn; e += (long long)gridDim.x * RF_NT) {
    const long long i = e / n;
    X[b * sX + i * ldx + (e - i * n)] = Q[b * nn + e];
  }
}

// After the first residual: the matrices that need no second step, and those
// whose columns are graded.  The products with A cut its entries 2^-62 below
// their row's largest, which its residual, formed with the same cut entries,
// cannot show; elimination rounds a column relative to the column.  As long as
// every column's largest entry lies within 2^9 of its row's largest, the cut
// stays below 2^-53 of the column (columns of 96 scaled by 2^-k, error of the
// inverse's rows: 2e-16 at k = 9, elimination 6e-16; 2.5e-15 at 12, 6e-13 at 20,
// all of them with residuals below 1e-10).
constexpr int RF_SPAN = 9;
__global__ void __launch_bounds__(128) done_kernel(int n, const int* __restrict__ span, int* low_info, int* top, int* skip) {
  const long long b = blockIdx.x;
  int least = RF_ONE;
  for (int j = threadIdx.x; j < n; j += 128) least = min(least, span[b * n + j]);
  const bool graded = __syncthreads_or(least < RF_ONE - RF_SPAN);
  if (threadIdx.x) return;
  if (graded) low_info[b] = INV_NOT_REFINED;
  skip[b] = (low_info[b] == 0 && __int_as_float(top[b]) <= 5e-5f) ? 1 : 0;
  if (!skip[b]) top[b] = 0;
}

// After the second one.
__global__ void verdict_kernel(int batch, const int* __restrict__ low_info, const int* __restrict__ top,
                               const int* __restrict__ skip, int* info) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  info[b] = (skip[b] || (low_info[b] == 0 && __int_as_float(top[b]) <= 1e-8f)) ? 0 : INV_NOT_REFINED;
}

template <class T>
cudaError_t digits_gemm(int n, double alpha, const T* A, long long lda, long long sA, const T* B, long long sB,
                        const T* C, T* D, long long ldd, long long sD, int batch, cudaStream_t st, const int* skip) {
  if constexpr (DTypeOf<T>::value == F64)
    return gemm_f64_tc(n, n, n, alpha, A, lda, sA, B, n, sB, 1.0, C, n, sB, D, ldd, sD, batch, st, skip);
  else
    return gemm_c128_tc(n, n, n, alpha, A, lda, sA, B, n, sB, 1.0, C, n, sB, D, ldd, sD, batch, st, skip);
}

size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// Whether the products run on operands split ahead of them (gemm_digits.cu)
// with the digits each step needs, rather than on gemm_f64_tc.cu with all of
// them: the passes that split cost some 20 us and 50 bytes a number, and pay
// from products of about 1 GFLOP with rows of 192 numbers on.  Measured, the
// two first products with their splits, whole against split: 432^3 x 3 120 and
// 115 us, 224^3 x 16 75 and 100, 1000^3 244 and 170, 224^3 x 256 800 and 690,
// complex 112^3 x 256 416 and 420, 512^3 x 64 1,620 and 1,080.
template <class T>
bool splits(int n, int batch) {
  const double f = sizeof(T) == 16 ? 2.0 : 1.0;
  return n * f >= 192.0 && 2.0 * n * (n * f) * (n * f) * batch >= 1e9;
}

// Bytes of the digits of one matrix: of A's rows (kept), of the second
// operand's columns, and of the rows of X (four digits and six).
struct DigitBytes {
  size_t a, b, x;
};
template <class T>
DigitBytes digit_bytes(int n) {
  const int f = sizeof(T) == 16 ? 2 : 1;
  return {digit_rows_bytes(n, n * f, 8), digit_cols_bytes(n * f, n * f, 8), digit_rows_bytes(n, n * f, 6)};
}

// Matrices at a time: about 2 GB of copies (one matrix always), and the digits
// of as many; with half of it the single-precision panels of 157 complex
// matrices of 256 were a third slower than those of 512.
int chunk_of(size_t es, int n, int batch) {
  const size_t per = 4 * es * (size_t)n * n, most = (size_t)2 << 30;
  const size_t c = most / per;
  return c < 1 ? 1 : c > (size_t)batch ? batch : c > 32768 ? 32768 : (int)c;
}

template <class T>
cudaError_t run(int n, const T* A, long long lda, long long sA, T* X, long long ldx, long long sX, int batch, int* info,
                unsigned char* base, size_t bytes, cudaStream_t st) {
  using L = typename Low<T>::type;
  const int cap = chunk_of(sizeof(T), n, batch), low_dt = DTypeOf<L>::value;
  const long long nn = (long long)n * n;
  unsigned char* w = base;
  auto take = [&](size_t b) {
    unsigned char* r = w;
    w += al256(b);
    return r;
  };
  T* P = (T*)take(sizeof(T) * (size_t)nn * cap);
  T* Q = (T*)take(sizeof(T) * (size_t)nn * cap);
  T* R = (T*)take(sizeof(T) * (size_t)nn * cap);
  L* l0 = (L*)take(sizeof(L) * (size_t)nn * cap);
  L* l1 = (L*)take(sizeof(L) * (size_t)nn * cap);
  L* l2 = (L*)take(sizeof(L) * (size_t)nn * cap);
  int* low_info = (int*)take(sizeof(int) * (size_t)cap);
  int* top = (int*)take(sizeof(int) * (size_t)cap * (n + 1));   // with the columns' spans behind it
  int* span = top + cap;
  int* skip = (int*)take(sizeof(int) * (size_t)cap);
  const size_t lowb = inverse_workspace_bytes(low_dt, n, cap);
  void* lows = take(lowb);
  constexpr bool CPLX = DTypeOf<T>::value == C128;
  const int f = CPLX ? 2 : 1, nr = n * f;   // the real views: n x nr times nr x nr
  const bool split = splits<T>(n, batch);
  unsigned char *da = nullptr, *db = nullptr, *dx = nullptr;
  int *ta = nullptr, *tb = nullptr, *tx = nullptr;
  if (split) {
    const DigitBytes d = digit_bytes<T>(n);
    da = take(d.a * cap);
    db = take(d.b * cap);
    dx = take(d.x * cap);
    ta = (int*)take(sizeof(int) * (size_t)n * cap);
    tb = (int*)take(sizeof(int) * (size_t)nr * cap);
    tx = (int*)take(sizeof(int) * (size_t)n * cap);
  }
  if ((size_t)(w - base) > bytes) return cudaErrorInvalidValue;
  const L one_ = one<L>(), zero_ = zero<L>();
  const int gr = (n + RF_NT / 32 - 1) / (RF_NT / 32);   // CTAs for the rows of one matrix
  // and for lower_kernel: four rows a warp (fewer flushes) where that fills the SMs
  // twice, else one (one matrix of 352 took 16 us with four)
  const int gl = (long long)(n / 32) * cap >= 304 ? (n + RF_NT / 8 - 1) / (RF_NT / 8) : gr;
  const int gx = (int)((nn + RF_NT * 4 - 1) / (RF_NT * 4) < 256 ? (nn + RF_NT * 4 - 1) / (RF_NT * 4) : 256);
  cudaError_t e;
#define RF_TRY(x)                              \
  do {                                         \
    if ((e = (x)) != cudaSuccess) return e;    \
  } while (0)
  for (int b0 = 0; b0 < batch; b0 += cap) {
    const int nb = batch - b0 < cap ? batch - b0 : cap;
    const T* Ab = A + (long long)b0 * sA;
    const long long total = nn * nb;
    const int gt = (int)((total + RF_NT * 4 - 1) / (RF_NT * 4) < 16384 ? (total + RF_NT * 4 - 1) / (RF_NT * 4) : 16384);
    RF_TRY(cudaMemsetAsync(top, 0, sizeof(int) * ((size_t)cap + (size_t)n * nb), st));
    note_launch();
    lower_kernel<T, L><<<dim3(gl, nb), RF_NT, 0, st>>>(n, Ab, lda, sA, l0, span);
    RF_TRY(inverse_batched<L>(n, l0, n, nn, l0, n, nn, nb, low_info, lows, lowb, st,
                              INV_TENSOR_MEMORY | INV_BLOCK_RECURSIVE));
    note_launch();
    raise_kernel<T, L><<<gt, RF_NT, 0, st>>>(total, l0, P);
    // D = X + X Y (contiguous X, Y) from the leading `digits` of both
    auto correct = [&](int digits, T* Xp, T* Y, T* D, long long ldd, long long sD, const int* sk) {
      RF_TRY(digit_rows(digits, n, nr, (const double*)Xp, nr, f * nn, tx, dx, nb, sk, st));
      RF_TRY(digit_cols(digits, CPLX, false, nr, nr, (double*)Y, nr, f * nn, tb, db, nb, sk, st));
      return digit_product(digits, digits, n, nr, nr, CPLX, false, dx, tx, db, tb, (const double*)Xp, nr, f * nn,
                           (double*)D, f * ldd, f * sD, nb, sk, st);
    };
    // R = -A X
    auto residual = [&](int digits, T* Xp, const int* sk) {
      RF_TRY(digit_cols(digits, CPLX, digits == 4, nr, nr, (double*)Xp, nr, f * nn, tb, db, nb, sk, st));
      return digit_product(8, digits, n, nr, nr, CPLX, true, da, ta, db, tb, nullptr, 0, 0, (double*)R, nr, f * nn, nb, sk,
                           st);
    };
    if (split)
      RF_TRY(digit_rows(8, n, nr, (const double*)Ab, f * lda, f * sA, ta, da, nb, nullptr, st));
    // first step: l0 = R, l1 = R + R^2, then l0 = R (R + R^2); P holds X0, Q gets X1
    RF_TRY(split ? residual(4, P, nullptr)
                 : digits_gemm<T>(n, -1.0, Ab, lda, sA, P, nn, nullptr, R, n, nn, nb, st, nullptr));
    note_launch();
    residual_kernel<T, L><<<dim3(gr, nb), RF_NT, 0, st>>>(n, R, l0, top, nullptr);
    note_launch();
    done_kernel<<<nb, 128, 0, st>>>(n, span, low_info, top, skip);
    RF_TRY(gemm_batched<L>(n, n, n, one_, l0, n, nn, l0, n, nn, one_, l0, n, nn, l1, n, nn, nb, st));
    RF_TRY(gemm_batched<L>(n, n, n, one_, l0, n, nn, l1, n, nn, zero_, nullptr, 0, 0, l2, n, nn, nb, st));
    note_launch();
    add_powers_kernel<T, L><<<gt, RF_NT, 0, st>>>(total, R, l2);
    RF_TRY(split ? correct(6, P, R, Q, n, nn, nullptr)
                 : digits_gemm<T>(n, 1.0, P, n, nn, R, nn, P, Q, n, nn, nb, st, nullptr));
    // second step, for the matrices that need it
    T* Xb = X + (long long)b0 * sX;
    RF_TRY(split ? residual(8, Q, skip) : digits_gemm<T>(n, -1.0, Ab, lda, sA, Q, nn, nullptr, R, n, nn, nb, st, skip));
    note_launch();
    residual_kernel<T, L><<<dim3(gr, nb), RF_NT, 0, st>>>(n, R, (L*)nullptr, top, skip);
    RF_TRY(split ? correct(4, Q, R, Xb, ldx, sX, skip)
                 : digits_gemm<T>(n, 1.0, Q, n, nn, R, nn, Q, Xb, ldx, sX, nb, st, skip));
    note_launch();
    keep_kernel<T><<<dim3(gx, nb), RF_NT, 0, st>>>(n, Q, Xb, ldx, sX, skip);
    note_launch();
    verdict_kernel<<<(nb + 255) / 256, 256, 0, st>>>(nb, low_info, top, skip, info + b0);
  }
#undef RF_TRY
  return cudaGetLastError();
}

}  // namespace

bool inverse_refined_takes(int dtype, int n) {
  return (dtype == F64 || dtype == C128) && n > 64 && f64_products_on_tensor_cores();
}

template <class T>
static size_t workspace_bytes(int n, int batch) {
  const size_t es = sizeof(T), nn = (size_t)n * n;
  const int cap = chunk_of(sizeof(T), n, batch), low_dt = es == 8 ? F32 : C64;
  size_t s = 3 * al256(es * nn * cap) + 3 * al256(es / 2 * nn * cap) + 2 * al256(sizeof(int) * (size_t)cap) +
             al256(sizeof(int) * (size_t)cap * (n + 1)) +
             al256(inverse_workspace_bytes(low_dt, n, cap)) + 512;
  if (splits<T>(n, batch)) {
    const DigitBytes d = digit_bytes<T>(n);
    const size_t nr = (size_t)n * (es / 8);
    s += al256(d.a * cap) + al256(d.b * cap) + al256(d.x * cap) + 2 * al256(sizeof(int) * n * cap) +
         al256(sizeof(int) * nr * cap);
  }
  return s;
}

size_t inverse_refined_workspace_bytes(int dtype, int n, int batch) {
  return dtype == F64 ? workspace_bytes<double>(n, batch) : workspace_bytes<c128>(n, batch);
}

template <class T>
cudaError_t inverse_refined(int n, const T* A, long long lda, long long sA, T* X, long long ldx, long long sX, int batch,
                            int* info, void* ws, size_t ws_bytes, cudaStream_t st) {
  if (batch <= 0) return cudaSuccess;
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
  const size_t lost = (size_t)(base - reinterpret_cast<unsigned char*>(ws));
  if (!ws || !info || ws_bytes < lost) return cudaErrorInvalidValue;
  ProfScope whole(KC_INVERSE, st, 2.0 * (DTypeOf<T>::value == C128 ? 4.0 : 1.0) * (double)n * n * n * batch);
  return run<T>(n, A, lda, sA, X, ldx, sX, batch, info, base, ws_bytes - lost, st);
}

template cudaError_t inverse_refined<double>(int, const double*, long long, long long, double*, long long, long long,
                                             int, int*, void*, size_t, cudaStream_t);
template cudaError_t inverse_refined<c128>(int, const c128*, long long, long long, c128*, long long, long long, int, int*,
                                           void*, size_t, cudaStream_t);

}  // namespace hps
