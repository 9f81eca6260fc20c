// Digit products of operands that are split once, ahead of the product.
//
// gemm_f64_tc.cu writes the digits of A once per 64 columns of D and those of
// B once per 128 rows, and its converting warps bound it (2,300 of the 3,300
// cycles of a stage of 16 steps at 1792^3, whose MMAs take 1,150).  For
// square products beyond a tile or two the digits are written to memory once
// by a pass of their own (digit_rows, digit_cols), as the very images of the
// shared-memory stages: a stage is one bulk copy per operand, and the product
// kernel only copies, multiplies and adds up.
//
// The callers choose how many digits each operand keeps and how many of the
// leading weights t + u are formed: an approximate inverse needs no more than
// four digits (it is rounded to them, and the residual is that of the rounded
// one), a correction of relative size r no more than its own leading ones.
//
// Measured, gemm_f64_tc.cu against (8, 8) (8, 4) (6, 6) (4, 4) digits, in us:
// 3072^3 2,690 and 1,440 1,055 1,045 724 (40 TFLOP/s with all 36 products),
// 512 x 512^3 complex 256 3,140 and 1,940 1,250 1,430 895, 1746 x 196^3 2,335
// and 1,515 1,045 1,190 833; splitting both operands into 8 digits 110, 795 and
// 680 (at the memory's rate).  A stage's MMAs read 136 KB of shared memory and
// the copies write 48 (1,450 cycles at 128 bytes a clock); 3072^3 takes 1,900 a
// stage, 1,300 without reading the accumulators: four warps a half read 128 x
// 32 x 8 of them every 8 stages, bound by the conversions to integers, and the
// ring lets the other half run ahead by four stages only.  Tried: 208 registers
// for the reading warps (setmaxnreg; 5% slower), both halves' chunks in step
// (1,550).
#include "hps_common.cuh"
#include "hps_internal.h"
#include "digits.cuh"

namespace hps {

namespace {

using namespace digits;
using tc::mbar_init;

constexpr int DG_BN = 64;                // columns of an output tile, two halves of 32
constexpr int DG_HN = 32;
constexpr int DG_APL = OZ_BM * 32;       // bytes of one digit plane of a stage of A
constexpr int DG_BPL = DG_HN * 32;       // and of half a stage of B
constexpr int DG_NT = 384;

template <int DA, int DB, int W>
struct DgCfg {
  static constexpr int ABYTES = DA * DG_APL, BBYTES = DB * 2 * DG_BPL, STAGE = ABYTES + BBYTES;
  static constexpr int NS = (216 * 1024) / STAGE < 8 ? (216 * 1024) / STAGE : 8;
  static constexpr size_t SMEM = (size_t)NS * STAGE + 1024;
  static constexpr int PAIRS = DA < DB ? DA : DB;           // most digit products in one accumulator and step
  static constexpr int CHUNK = 64 / PAIRS;                  // stages until |sum| <= 2^24 is used up
  static constexpr int HC = DG_HN * W;                      // accumulator columns of a half
  static constexpr int COLS = 2 * HC <= 256 ? 256 : 512;    // TMEM columns
};

struct DgArgs {
  int M, N, K;               // real sizes (complex: N and K doubled)
  int neg;                   // D = -A B + C
  int paired;                // columns 2j, 2j + 1 share their scale (complex)
  const unsigned char* A;    // images of the stages
  const int* ta;             // (batch, M) largest high words of the rows
  const unsigned char* B;
  const int* tb;             // (batch, N) of the columns
  const double* C;
  long long ldc, sC;
  double* D;
  long long ldd, sD;
  int batch, vec;
  const int* skip;
  int* err;
  const long long* limit;
};

// The exponent code of a row or column from the largest high word: 0x7ff with
// infinities and NaN; nothing but values below 2^-958 counts as zeros.
__device__ __forceinline__ int top_code(uint32_t top) {
  const int x = (int)(top >> 20);
  return x <= 64 ? 1024 : x;
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// One persistent CTA of 12 warps per SM.  A 128 x 64 tile of D is two halves
// of 32 columns, each with W accumulators (one per weight), an issuing warp
// and four reading warps of its own: while one half's accumulators are read
// (every CHUNK stages), the other's MMAs go on through the ring.
//   warps 0-3, 4-7  accumulators -> 96-bit sums -> D, one half each
//   warp 8          bulk copies of the stages (`full`, `empty`)
//   warps 9, 10     MMAs of a half: digit t of A meets the digits 0 .. W - 1 - t
//                   of B side by side, as one MMA into consecutive accumulators
// Every wait is bounded, as in gemm_oz_kernel.
template <int DA, int DB, int W>
__global__ void __launch_bounds__(DG_NT, 1) gemm_digits_kernel(const DgArgs p) {
  using Cfg = DgCfg<DA, DB, W>;
  constexpr int NS = Cfg::NS;
  extern __shared__ unsigned char dg_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(dg_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full[NS], empty[NS], accf[2], acce[2], fin[2];
  __shared__ uint32_t tmem_s;
  __shared__ int fail_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long limit = *(const volatile long long*)p.limit;
  if (tid == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 2);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&accf[i], 1);
      mbar_init(&acce[i], 4);
      mbar_init(&fin[i], 1);
    }
    fail_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 11) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)),
                 "r"(Cfg::COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_s;
  const int tiles_n = (p.N + DG_BN - 1) / DG_BN, tiles_m = (p.M + OZ_BM - 1) / OZ_BM;
  const long long per_b = (long long)tiles_m * tiles_n, n_units = per_b * p.batch;
  const int nk = (p.K + OZ_BK - 1) / OZ_BK;
  auto tile_from = [&](long long u) {
    if (p.skip)
      while (u < n_units && p.skip[u / per_b]) u += gridDim.x;
    return u;
  };
  const long long u0 = tile_from(blockIdx.x);
  bool ok = true;
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (ok) ok = (bool)__all_sync(0xffffffffu, tc::mbar_wait(bar, parity, limit));
  };

  if (warp < 8) {
    // ---------------- accumulators -> 96-bit sums -> D ----------------
    const int q = warp & 3, h = warp >> 2;
    const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(h * Cfg::HC);
    const int shift = h && nk > 2 * Cfg::CHUNK ? Cfg::CHUNK / 2 : 0;
    uint32_t s0[DG_HN], s1[DG_HN], s2[DG_HN];
    uint32_t ch = 0;
    for (long long u = u0; u < n_units; u = tile_from(u + gridDim.x)) {
      const long long b = u / per_b;
      const int r = (int)(u % per_b), m0 = (r / tiles_n) * OZ_BM, c0 = (r % tiles_n) * DG_BN + h * DG_HN;
      if (c0 >= p.N) continue;
#pragma unroll
      for (int j = 0; j < DG_HN; ++j) s0[j] = s1[j] = s2[j] = 0;
      for (int kt = -shift; kt < nk; kt += Cfg::CHUNK, ++ch) {
        wait(&accf[h], ch & 1);
        tc::fence_after();
        // steps of four columns and up to four weights, the next one's loads ahead
        constexpr int G = W > 4 ? 2 : 1;
        uint32_t v[2][4][4];
        auto load = [&](uint32_t (&x)[4][4], int i) {
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            const int w = W - 1 - 4 * (i % G) - l;
            if (w >= 0) tmem_ld4(tb + (uint32_t)(w * DG_HN + i / G * 4), x[l]);
          }
        };
        load(v[0], 0);
#pragma unroll
        for (int i = 0; i < DG_HN / 4 * G; ++i) {
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (i + 1 < DG_HN / 4 * G) load(v[(i + 1) & 1], i + 1);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int c = i / G * 4 + j;
            long long x = __float2int_rn(__uint_as_float(v[i & 1][0][j]));
#pragma unroll
            for (int l = 1; l < 4; ++l)
              if (W - 1 - 4 * (i % G) - l >= 0)
                asm("mad.wide.s32 %0, %1, %2, %0;"
                    : "+l"(x)
                    : "r"(__float2int_rn(__uint_as_float(v[i & 1][l][j]))), "r"(1 << (8 * l)));
            const uint32_t xl = (uint32_t)x, xh = (uint32_t)((unsigned long long)x >> 32);
            if (i % G == 0)
              asm("add.cc.u32 %0, %0, %3;\n addc.cc.u32 %1, %1, %4;\n addc.u32 %2, %2, %5;"
                  : "+r"(s0[c]), "+r"(s1[c]), "+r"(s2[c])
                  : "r"(xl), "r"(xh), "r"((uint32_t)((int)xh >> 31)));
            else   // the weights above the last four: 2^32
              asm("add.cc.u32 %0, %0, %2;\n addc.u32 %1, %1, %3;" : "+r"(s1[c]), "+r"(s2[c]) : "r"(xl), "r"(xh));
          }
        }
        tc::fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acce[h]);
        __syncwarp();
      }
      const int row = m0 + q * 32 + lane;
      if (!ok || row >= p.M) continue;
      const int re = top_code((uint32_t)p.ta[b * p.M + row]);
      const int* tb_ = p.tb + b * p.N;
      const double* Cr = p.C ? p.C + b * p.sC + (long long)row * p.ldc + c0 : nullptr;
      double* Dr = p.D + b * p.sD + (long long)row * p.ldd + c0;
#pragma unroll
      for (int g = 0; g < DG_HN; g += 4) {
        if (c0 + g >= p.N) break;
        double v[4];
        int ex[4];
        bool odd = re >= 0x7ff, bad = odd;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int n = c0 + g + j < p.N ? c0 + g + j : p.N - 1;
          uint32_t t = (uint32_t)tb_[n];
          if (p.paired) t = max(t, (uint32_t)tb_[n ^ 1]);
          const int ce = top_code(t);
          bad = bad || ce >= 0x7ff;
          // the last weight formed is W - 1: the unit is 2^(8 (8 - W)) that of eight
          ex[j] = re + ce - 2112 + 8 * (8 - W);
          v[j] = round_sum(s0[g + j], s1[g + j], s2[g + j], ex[j], odd);
        }
        if (odd || bad) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            v[j] = bad ? __longlong_as_double(0x7ff8000000000000ll)
                       : round_sum_any(s0[g + j], s1[g + j], s2[g + j], ex[j]);
        }
        if (p.neg) {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = -v[j];
        }
        if (c0 + g + 4 <= p.N && p.vec) {
          if (Cr) {
            const double2 x = *reinterpret_cast<const double2*>(Cr + g), y = *reinterpret_cast<const double2*>(Cr + g + 2);
            v[0] += x.x;
            v[1] += x.y;
            v[2] += y.x;
            v[3] += y.y;
          }
          *reinterpret_cast<double2*>(Dr + g) = make_double2(v[0], v[1]);
          *reinterpret_cast<double2*>(Dr + g + 2) = make_double2(v[2], v[3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (c0 + g + j < p.N) Dr[g + j] = Cr ? Cr[g + j] + v[j] : v[j];
        }
      }
    }
  } else if (warp == 8) {
    // ---------------- copies ----------------
    uint32_t it = 0;
    for (long long u = u0; u < n_units; u = tile_from(u + gridDim.x)) {
      const long long b = u / per_b;
      const int r = (int)(u % per_b), tm = r / tiles_n, tn = r % tiles_n;
      const unsigned char* a = p.A + (b * tiles_m + tm) * nk * (long long)Cfg::ABYTES;
      const unsigned char* bb = p.B + (b * tiles_n + tn) * nk * (long long)Cfg::BBYTES;
      const uint32_t nb = tn * DG_BN + DG_HN < p.N ? Cfg::BBYTES : Cfg::BBYTES / 2;
      for (int kt = 0; kt < nk; ++kt, ++it) {
        const int s = it % NS;
        if (it >= NS) wait(&empty[s], (it / NS - 1) & 1);
        if (!ok) break;
        if (lane == 0) {
          const uint32_t dst = smem_u32(smem + s * Cfg::STAGE);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&full[s])),
                       "r"((uint32_t)Cfg::ABYTES + nb)
                       : "memory");
          bulk_load(dst, a + (long long)kt * Cfg::ABYTES, Cfg::ABYTES, &full[s]);
          bulk_load(dst + Cfg::ABYTES, bb + (long long)kt * Cfg::BBYTES, nb, &full[s]);
        }
        __syncwarp();
      }
      if (!ok) break;
    }
    if (!ok) {   // a second bounded chance for the copies in flight
      for (int s = 0; s < NS; ++s)
        if (it > (uint32_t)s) tc::mbar_wait(&full[s], ((it - 1 - s) / NS) & 1, limit);
    }
  } else if (warp == 9 || warp == 10) {
    // ---------------- MMAs of one half ----------------
    const int h = warp - 9, shift = h && nk > 2 * Cfg::CHUNK ? Cfg::CHUNK / 2 : 0;
    uint32_t it = 0, ch = 0;
    for (long long u = u0; u < n_units; u = tile_from(u + gridDim.x)) {
      const bool active = (int)(u % per_b % tiles_n) * DG_BN + h * DG_HN < p.N;
      for (int kt = 0; kt < nk; ++kt, ++it) {
        const int s = it % NS;
        const int k = (kt + shift) % Cfg::CHUNK;
        const bool first = kt == 0 || k == 0, last = k == Cfg::CHUNK - 1 || kt == nk - 1;
        wait(&full[s], (it / NS) & 1);
        if (active) {
          if (first && ch > 0) wait(&acce[h], (ch - 1) & 1);
          tc::fence_after();
          if (ok && lane == 0) {
            const uint32_t a0 = desc_lo(smem_u32(smem + s * Cfg::STAGE));
            const uint32_t b0 = a0 + ((Cfg::ABYTES + h * DB * DG_BPL) >> 4);
            // the MMAs that reach an accumulator first overwrite it
#pragma unroll
            for (int o = 0; o < 2; ++o)
#pragma unroll
              for (int t = 0; t < (DA < W ? DA : W); ++t) {
                if ((t % DB == 0) != (o == 0)) continue;
                const int nw = DB < W - t ? DB : W - t;
                mma_f16(tmem + h * Cfg::HC + t * DG_HN, a0 + ((t * DG_APL) >> 4), b0, idesc_f16(nw * DG_HN),
                        (o == 0 && first) ? 0u : 1u);
              }
            tc::mma_commit(&empty[s]);
            if (last) tc::mma_commit(&accf[h]);
          }
          if (last) ++ch;
        } else if (ok && lane == 0) {
          mbar_arrive(&empty[s]);
        }
        __syncwarp();
      }
    }
    if (!ok && lane == 0) {   // and for the MMAs in flight
      tc::mma_commit(&fin[h]);
      tc::mbar_wait(&fin[h], 0, limit);
    }
    __syncwarp();
  }
  if (!ok) fail_s = 1;
  tc::fence_before();
  __syncthreads();
  if (fail_s && tid == 0) atomicExch(p.err, 1);
  if (warp == 11) {
    tc::fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::COLS) : "memory");
  }
}

// Largest high words (sign left out) of the rows and columns of (R x N)
// matrices: a CTA per 32 x 128 block, lane + 32 j the columns of a warp's four
// rows.
__global__ void __launch_bounds__(256) digit_tops_kernel(int R, int N, const double* __restrict__ X, long long ldx,
                                                         long long sX, int* rows, int* cols,
                                                         const int* __restrict__ skip) {
  const long long b = blockIdx.z;
  if (skip && skip[b]) return;
  __shared__ uint32_t part[8][128];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r0 = blockIdx.y * 32 + warp * 4, n0 = blockIdx.x * 128 + lane;
  uint32_t col[4] = {0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t row = 0;
    if (r0 + i < R) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n0 + 32 * j < N) {
          const uint32_t v = (uint32_t)__double2hiint(X[b * sX + (long long)(r0 + i) * ldx + n0 + 32 * j]) & 0x7fffffffu;
          row = max(row, v);
          col[j] = max(col[j], v);
        }
    }
    if (rows) {
      row = __reduce_max_sync(0xffffffffu, row);
      if (lane == 0 && row) atomicMax(rows + b * R + r0 + i, (int)row);
    }
  }
  if (!cols) return;
#pragma unroll
  for (int j = 0; j < 4; ++j) part[warp][lane + 32 * j] = col[j];
  __syncthreads();
  if (threadIdx.x < 128) {
    uint32_t m = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) m = max(m, part[w][threadIdx.x]);
    const int n = blockIdx.x * 128 + threadIdx.x;
    if (n < N && m) atomicMax(cols + b * N + n, (int)m);
  }
}

// The leading ND digits of eight values as ND 16-byte pieces, `plane` bytes apart.
template <int ND>
__device__ __forceinline__ void store_digits(const double (&v)[8], uint32_t emax20, unsigned char* d, int plane) {
  uint32_t x[16], one[4], off[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    sign_pair(__double2hiint(v[2 * i]), __double2hiint(v[2 * i + 1]), one[i], off[i]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint2 y = to_digits(__double2loint(v[2 * i + j]), __double2hiint(v[2 * i + j]), emax20);
      x[4 * i + 2 * j] = y.x, x[4 * i + 2 * j + 1] = y.y;
    }
  }
#pragma unroll
  for (int w = 0; w < ND / 2; ++w) {   // digits 2w, 2w + 1
    uint32_t z[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) z[i] = __byte_perm(x[4 * i + (w < 2)], x[4 * i + 2 + (w < 2)], (w & 1) ? 0x4051 : 0x6273);
    *reinterpret_cast<uint4*>(d + (2 * w) * plane) =
        make_uint4(f16_digits(z[0], 0x4140, one[0], off[0]), f16_digits(z[1], 0x4140, one[1], off[1]),
                   f16_digits(z[2], 0x4140, one[2], off[2]), f16_digits(z[3], 0x4140, one[3], off[3]));
    *reinterpret_cast<uint4*>(d + (2 * w + 1) * plane) =
        make_uint4(f16_digits(z[0], 0x4342, one[0], off[0]), f16_digits(z[1], 0x4342, one[1], off[1]),
                   f16_digits(z[2], 0x4342, one[2], off[2]), f16_digits(z[3], 0x4342, one[3], off[3]));
  }
}

// The value of the leading four digits of v (|v| < 2^(emax - 1022)), put
// together with integers: D 2^(emax - 1052), D < 2^31.
__device__ __forceinline__ double four_digits(double v, int emax) {
  const uint32_t D = to_digits(__double2loint(v), __double2hiint(v), (uint32_t)emax << 20).y - 0x80808080u;
  const int z = __clz(D), ex = emax + 2 - z;   // 2^(31 - z) leads
  if (D == 0 || ex <= 0) return 0.0;
  const uint32_t m = D << z;                   // the leading one at bit 31
  return __hiloint2double((int)((__double2hiint(v) & 0x80000000u) | ((uint32_t)ex << 20) | ((m >> 11) & 0xfffffu)),
                          (int)(m << 21));
}

// Stage images of A (M x K, rows of doubles): a CTA per 128 rows x 16 steps,
// two threads a row.  Rows beyond M are left as they are: they reach rows of
// the accumulators that are not read.
template <int ND>
__global__ void __launch_bounds__(256) digit_rows_kernel(int M, int K, const double* __restrict__ X, long long ldx,
                                                         long long sX, const int* __restrict__ top, unsigned char* out,
                                                         const int* __restrict__ skip) {
  const long long b = blockIdx.y;
  if (skip && skip[b]) return;
  const int nk = (K + OZ_BK - 1) / OZ_BK, tm = blockIdx.x / nk, kt = blockIdx.x % nk;
  const int r = threadIdx.x >> 1, c = threadIdx.x & 1, row = tm * OZ_BM + r, k0 = kt * OZ_BK + c * 8;
  if (row >= M) return;
  const double* x = X + b * sX + (long long)row * ldx + k0;
  double v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = k0 + i < K ? x[i] : 0.0;
  const long long tiles_m = (M + OZ_BM - 1) / OZ_BM;
  store_digits<ND>(v, (uint32_t)top_code((uint32_t)top[b * M + row]) << 20,
                   out + ((b * tiles_m + tm) * nk + kt) * (ND * DG_APL) + r * 32 + ((c ^ ((r >> 2) & 1)) << 4), DG_APL);
}

// Stage images of B (K x N): a CTA per 64 columns x 32 steps, two threads per
// column and stage.  CPLX: B is (K / 2 x N / 2) complex, and its real view has
// the rows 2k, 2k + 1 as (re, im) and (-im, re).  ROUND: what the digits hold
// is written back.
template <int ND, bool CPLX, bool ROUND>
__global__ void __launch_bounds__(256) digit_cols_kernel(int N, int K, double* X, long long ldx, long long sX,
                                                         const int* __restrict__ top, unsigned char* out,
                                                         const int* __restrict__ skip) {
  static_assert(!ROUND || ND == 4, "four_digits");
  const long long b = blockIdx.y;
  if (skip && skip[b]) return;
  const int nk = (K + OZ_BK - 1) / OZ_BK, nk2 = (nk + 1) / 2;
  const int tn = blockIdx.x / nk2, kt = (blockIdx.x % nk2) * 2 + (threadIdx.x >> 7);
  const int c = threadIdx.x & 1, j = (threadIdx.x >> 1) & 63, n = tn * DG_BN + j, k0 = kt * OZ_BK + c * 8;
  if (kt >= nk) return;
  const bool in = n < N;
  double* x = X + b * sX + (long long)(CPLX ? k0 >> 1 : k0) * ldx;
  uint32_t t = 0;
  double v[8];
  if (in) {
    t = (uint32_t)top[b * N + n];
    if (CPLX) t = max(t, (uint32_t)top[b * N + (n ^ 1)]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (CPLX) {
        // re where the row's and the column's parts agree, else im
        const double w = k0 + i < K ? x[(long long)(i >> 1) * ldx + (n & ~1) + ((i + n) & 1)] : 0.0;
        v[i] = (i & 1) && !(n & 1) ? -w : w;
      } else {
        v[i] = k0 + i < K ? x[(long long)i * ldx + n] : 0.0;
      }
    }
  }
  const int e = top_code(t);
  if (ROUND) {
    // a complex value stands at two places of the real view, in two lanes of
    // one warp: both read it first, then that of the even row writes
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (in && k0 + i < K && e < 0x7ff && !(CPLX && (i & 1)))
        x[(long long)(CPLX ? i >> 1 : i) * ldx + n] = four_digits(v[i], e);
  }
  if (!in) return;
  const long long tiles_n = (N + DG_BN - 1) / DG_BN;
  const int r = j & 31;
  store_digits<ND>(v, (uint32_t)e << 20,
                   out + ((b * tiles_n + tn) * nk + kt) * (ND * 2 * DG_BPL) + (j >> 5) * (ND * DG_BPL) + r * 32 +
                       ((c ^ ((r >> 2) & 1)) << 4),
                   DG_BPL);
}

template <int DA, int DB, int W>
cudaError_t launch_digits(DgArgs p, cudaStream_t st) {
  using Cfg = DgCfg<DA, DB, W>;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(gemm_digits_kernel<DA, DB, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM);
  if (e == cudaSuccess) e = tc_wait_state(&p.err, &p.limit);
  if (e != cudaSuccess) return e;
  const long long units = (long long)p.batch * ((p.M + OZ_BM - 1) / OZ_BM) * ((p.N + DG_BN - 1) / DG_BN);
  note_launch();
  gemm_digits_kernel<DA, DB, W><<<(unsigned)(units < sms ? units : sms), DG_NT, Cfg::SMEM, st>>>(p);
  return cudaGetLastError();
}

}  // namespace

size_t digit_rows_bytes(int M, int K, int digits) {
  return (size_t)((M + OZ_BM - 1) / OZ_BM) * ((K + OZ_BK - 1) / OZ_BK) * digits * DG_APL;
}

size_t digit_cols_bytes(int N, int K, int digits) {
  return (size_t)((N + DG_BN - 1) / DG_BN) * ((K + OZ_BK - 1) / OZ_BK) * digits * 2 * DG_BPL;
}

static cudaError_t digit_tops(int R, int N, const double* X, long long ldx, long long sX, int* rows, int* cols, int batch,
                              const int* skip, cudaStream_t st) {
  const cudaError_t e = cudaMemsetAsync(rows ? rows : cols, 0, sizeof(int) * (size_t)(rows ? R : N) * batch, st);
  if (e != cudaSuccess) return e;
  note_launch();
  digit_tops_kernel<<<dim3((N + 127) / 128, (R + 31) / 32, batch), 256, 0, st>>>(R, N, X, ldx, sX, rows, cols, skip);
  return cudaGetLastError();
}

cudaError_t digit_rows(int digits, int M, int K, const double* X, long long ldx, long long sX, int* top, void* out,
                       int batch, const int* skip, cudaStream_t st) {
  const cudaError_t e = digit_tops(M, K, X, ldx, sX, top, nullptr, batch, skip, st);
  if (e != cudaSuccess) return e;
  const dim3 g((unsigned)((M + OZ_BM - 1) / OZ_BM) * ((K + OZ_BK - 1) / OZ_BK), batch);
  auto go = [&](auto kernel) {
    note_launch();
    kernel<<<g, 256, 0, st>>>(M, K, X, ldx, sX, top, (unsigned char*)out, skip);
    return cudaGetLastError();
  };
  switch (digits) {
    case 8: return go(digit_rows_kernel<8>);
    case 6: return go(digit_rows_kernel<6>);
    case 4: return go(digit_rows_kernel<4>);
  }
  return cudaErrorInvalidValue;
}

cudaError_t digit_cols(int digits, bool cplx, bool round, int N, int K, double* X, long long ldx, long long sX, int* top,
                       void* out, int batch, const int* skip, cudaStream_t st) {
  if (round && digits != 4) return cudaErrorInvalidValue;
  const cudaError_t e = digit_tops(cplx ? K / 2 : K, N, X, ldx, sX, nullptr, top, batch, skip, st);
  if (e != cudaSuccess) return e;
  const dim3 g((unsigned)((N + DG_BN - 1) / DG_BN) * (((K + OZ_BK - 1) / OZ_BK + 1) / 2), batch);
  auto go = [&](auto kernel) {
    note_launch();
    kernel<<<g, 256, 0, st>>>(N, K, X, ldx, sX, top, (unsigned char*)out, skip);
    return cudaGetLastError();
  };
  if (round) return cplx ? go(digit_cols_kernel<4, true, true>) : go(digit_cols_kernel<4, false, true>);
  switch (digits) {
    case 8: return cplx ? go(digit_cols_kernel<8, true, false>) : go(digit_cols_kernel<8, false, false>);
    case 6: return cplx ? go(digit_cols_kernel<6, true, false>) : go(digit_cols_kernel<6, false, false>);
    case 4: return cplx ? go(digit_cols_kernel<4, true, false>) : go(digit_cols_kernel<4, false, false>);
  }
  return cudaErrorInvalidValue;
}

cudaError_t digit_product(int da, int db, int M, int N, int K, bool cplx, bool neg, const void* A, const int* ta,
                          const void* B, const int* tb, const double* C, long long ldc, long long sC, double* D,
                          long long ldd, long long sD, int batch, const int* skip, cudaStream_t st) {
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  DgArgs p{M, N, K, neg, cplx, (const unsigned char*)A, ta, (const unsigned char*)B, tb, C, ldc, sC, D, ldd, sD, batch, 0,
           skip, nullptr, nullptr};
  p.vec = al16(D) && ldd % 2 == 0 && (batch == 1 || sD % 2 == 0) &&
          (!C || (al16(C) && ldc % 2 == 0 && (batch == 1 || sC % 2 == 0)));
  ProfScope ps(KC_GEMM, st, 2.0 * M * (double)N * K * batch);
  if (da == 8 && db == 8) return launch_digits<8, 8, 8>(p, st);
  if (da == 8 && db == 4) return launch_digits<8, 4, 8>(p, st);
  if (da == 6 && db == 6) return launch_digits<6, 6, 6>(p, st);
  if (da == 4 && db == 4) return launch_digits<4, 4, 4>(p, st);
  return cudaErrorInvalidValue;
}

}  // namespace hps
