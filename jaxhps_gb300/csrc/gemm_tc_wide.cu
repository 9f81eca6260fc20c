// FP32 and complex64 batched products with wide N on the tensor cores: 128 x
// 128 tiles, TF32 hi + lo operands, three products (3xTF32, Ootomo & Yokota, as
// gemm_tf32x3_kernel, whose accuracy this kernel has), loads by TMA and every
// part of the work on its own warps.
//
// What bounds it: shared memory.  A K-tile of 32 moves 32 KB in (TMA), 32 KB
// through the converters and 64 KB of TF32 parts out of them, and 80 KB into
// the MMAs (A_hi against [B_hi | B_lo] as one product of 256 columns, A_lo
// against B_hi): about 1,660 cycles at 128 bytes a clock, where the MMAs take
// 770.  gemm_tf32x3_kernel, whose 8 warps load, convert and issue in turn with
// two tiles in flight, takes about 6,000.
//
// A raw ring of NR stages (A boxes 32 x 128 in the 128-byte-swizzled K-major
// layout, B boxes 128 x 32 row-major) decouples the loads from a ring of NS
// converted stages (A hi, A lo, B hi, B lo, K-major); two accumulators of 256
// TMEM columns let a tile's MMAs start while the tile before is written.
//   warp 0      producer: TMA loads (`rfull`, `rempty`)
//   warp 1      MMA issue (`cfull`, `cempty`, `accf`, `acce`)
//   warps 2-9   converters
//   warps 10-13 epilogue: the accumulator's halves added, alpha acc + beta C
// Every wait is bounded; a wait that runs out sets the failure flag and the
// CTA winds down as gemm_tma_kernel does.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "hps_common.cuh"
#include "hps_internal.h"
#include "tc_common.cuh"

namespace hps {

namespace {

using tc::mbar_init;
using tc::smem_u32;

constexpr int WD_B = 128;                       // tile rows and columns
constexpr int WD_K = 32;                        // K steps of a stage
constexpr int WD_NR = 3, WD_NS = 2;
constexpr int WD_CW = 8, WD_CT = WD_CW * 32;    // converters
constexpr int WD_NT = (2 + WD_CW + 4) * 32;
constexpr int WD_TILE = WD_B * WD_K * 4;        // 16 KB: one operand tile
constexpr int WD_RAW = 2 * WD_TILE;
constexpr int WD_STAGE = 4 * WD_TILE;
constexpr size_t WD_SMEM = (size_t)WD_NR * WD_RAW + (size_t)WD_NS * WD_STAGE + 1024;

__device__ __forceinline__ void arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void load_box(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// x = hi + lo: hi the nearest TF32 value (ties away from zero), lo = x - hi exactly.
__device__ __forceinline__ void split(float x, uint32_t& h, uint32_t& l) {
  h = (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u;
  l = __float_as_uint(x - __uint_as_float(h));
}
__device__ __forceinline__ void split4(float4 x, uint4& h, uint4& l) {
  split(x.x, h.x, l.x);
  split(x.y, h.y, l.y);
  split(x.z, h.z, l.z);
  split(x.w, h.w, l.w);
}

struct WideArgs {
  int M, N, K;   // real sizes (complex: N and K doubled)
  float alpha, beta;
  const float* C;
  long long ldc, sC;
  float* D;
  long long ldd, sD;
  int batch, a_batched, b_batched, vec_out;
  int* err;
  const long long* limit;
};

// CPLX: the real product of the interleaved views, as gemm_tf32x3_kernel: a
// K-tile of 32 real rows of B is 16 complex rows, each giving the rows
// (re, im, ...) and (-im, re, ...).
template <bool CPLX>
__global__ void __launch_bounds__(WD_NT, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const WideArgs p) {
  extern __shared__ unsigned char wd_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(wd_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* conv = smem + WD_NR * WD_RAW;
  __shared__ uint64_t rfull[WD_NR], rempty[WD_NR], cfull[WD_NS], cempty[WD_NS], accf[2], acce[2];
  __shared__ uint32_t armed[WD_NR], committed[WD_NS], acc_committed[2];
  __shared__ uint32_t tmem_s;
  __shared__ int fail_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long limit = *(const volatile long long*)p.limit;
  if (tid == 0) {
    for (int i = 0; i < WD_NR; ++i) {
      mbar_init(&rfull[i], 1);
      mbar_init(&rempty[i], WD_CW);
      armed[i] = 0;
    }
    for (int i = 0; i < WD_NS; ++i) {
      mbar_init(&cfull[i], WD_CW);
      mbar_init(&cempty[i], 1);
      committed[i] = 0;
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&accf[i], 1);
      mbar_init(&acce[i], 4);
      acc_committed[i] = 0;
    }
    fail_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_s;
  const int tiles_n = (p.N + WD_B - 1) / WD_B, tiles_m = (p.M + WD_B - 1) / WD_B;
  const long long per_b = (long long)tiles_m * tiles_n, n_units = per_b * p.batch;
  const int nk = (p.K + WD_K - 1) / WD_K;
  volatile int* fail = &fail_s;
  // a warp leaves its loop as a whole: every lane polls, the warp agrees
  auto failed = [&] { return (bool)__any_sync(0xffffffffu, *fail != 0); };
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(bar, parity, limit));
    if (!ok) *fail = 1;
    return ok;
  };
  // (batch, first row, first column) of a tile: column tiles of a row first
  auto place = [&](long long u, int& b, int& m0, int& n0) {
    b = (int)(u / per_b);
    const int r = (int)(u % per_b);
    m0 = (r / tiles_n) * WD_B;
    n0 = (r % tiles_n) * WD_B;
  };

  if (warp == 0) {
    // ---------------- producer ----------------
    constexpr uint32_t tx = WD_TILE + (CPLX ? WD_TILE / 2 : WD_TILE);
    uint32_t it = 0;
    int s = 0;
    bool ok = true;
    for (long long u = blockIdx.x; u < n_units && ok && !failed(); u += gridDim.x) {
      int b, m0, n0;
      place(u, b, m0, n0);
      for (int kt = 0; kt < nk && ok; ++kt, ++it) {
        if (it >= WD_NR) ok = wait(&rempty[s], (it / WD_NR - 1) & 1);
        if (ok && lane == 0) {
          unsigned char* st = smem + s * WD_RAW;
          expect_tx(&rfull[s], tx);
          armed[s] += 1;
          load_box(st, &tmA, kt * WD_K, m0, p.a_batched ? b : 0, &rfull[s]);
          load_box(st + WD_TILE, &tmB, n0, kt * (CPLX ? WD_K / 2 : WD_K), p.b_batched ? b : 0, &rfull[s]);
        }
        __syncwarp();
        s = s + 1 == WD_NR ? 0 : s + 1;
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issue ----------------
    constexpr uint32_t id256 = tc::idesc_tf32(WD_B, 2 * WD_B), id128 = tc::idesc_tf32(WD_B, WD_B);
    uint32_t it = 0, acc_it = 0;
    bool ok = true;
    for (long long u = blockIdx.x; u < n_units && ok && !failed(); u += gridDim.x, ++acc_it) {
      const int a = acc_it & 1;
      if (acc_it >= 2) ok = wait(&acce[a], ((acc_it >> 1) - 1) & 1);
      tc::fence_after();
      const uint32_t dt = tmem + (uint32_t)(a * 2 * WD_B);
      for (int kt = 0; kt < nk && ok; ++kt, ++it) {
        const int s = it % WD_NS;
        ok = wait(&cfull[s], (it / WD_NS) & 1);
        tc::fence_after();
        if (ok && lane == 0) {
          const uint32_t ah = smem_u32(conv + s * WD_STAGE), al = ah + WD_TILE, bh = al + WD_TILE;
          const int ks = min(WD_K / 8, (p.K - kt * WD_K + 7) / 8);
          for (int kk = 0; kk < ks; ++kk) {
            const uint32_t off = kk * 32;   // 8 TF32 = 32 bytes along K inside the swizzle row
            tc::mma_tf32(dt, tc::desc_sw128(ah + off), tc::desc_sw128(bh + off), id256, (kt > 0 || kk > 0) ? 1u : 0u);
            tc::mma_tf32(dt, tc::desc_sw128(al + off), tc::desc_sw128(bh + off), id128, 1u);
          }
          tc::mma_commit(&cempty[s]);
          committed[s] += 1;
          if (kt == nk - 1) {
            tc::mma_commit(&accf[a]);
            acc_committed[a] += 1;
          }
        }
        __syncwarp();
      }
    }
  } else if (warp < 2 + WD_CW) {
    // ---------------- converters ----------------
    const int ct = tid - 64;
    uint32_t it = 0;
    int rs = 0;
    bool ok = true;
    for (long long u = blockIdx.x; u < n_units && ok && !failed(); u += gridDim.x) {
      for (int kt = 0; kt < nk && ok; ++kt, ++it) {
        const int s = it % WD_NS;
        ok = wait(&rfull[rs], (it / WD_NR) & 1);
        if (ok && it >= WD_NS) ok = wait(&cempty[s], (it / WD_NS - 1) & 1);
        if (!ok) break;
        const unsigned char* ra = smem + rs * WD_RAW;
        unsigned char* st = conv + s * WD_STAGE;
        // A: chunk by chunk, the swizzle kept
#pragma unroll
        for (int i = 0; i < WD_TILE / 16 / WD_CT; ++i) {
          const int off = (ct + WD_CT * i) * 16;
          uint4 h, l;
          split4(*reinterpret_cast<const float4*>(ra + off), h, l);
          *reinterpret_cast<uint4*>(st + off) = h;
          *reinterpret_cast<uint4*>(st + WD_TILE + off) = l;
        }
        // B: row-major to K-major; an item is column n and four steps of K
        const float* rb = reinterpret_cast<const float*>(ra + WD_TILE);
#pragma unroll
        for (int i = 0; i < WD_B * WD_K / 4 / WD_CT; ++i) {
          const int f = ct + WD_CT * i, n = f % WD_B, k = (f / WD_B) * 4;
          float4 x;
          if constexpr (CPLX) {
            const float* q = rb + (k >> 1) * WD_B;
            const float y = q[n ^ 1], z = q[WD_B + (n ^ 1)];
            x = make_float4(q[n], (n & 1) ? y : -y, q[WD_B + n], (n & 1) ? z : -z);
          } else {
            const float* q = rb + k * WD_B + n;
            x = make_float4(q[0], q[WD_B], q[2 * WD_B], q[3 * WD_B]);
          }
          uint4 h, l;
          split4(x, h, l);
          const uint32_t o = 2 * WD_TILE + tc::sw128_off(n, k);
          *reinterpret_cast<uint4*>(st + o) = h;
          *reinterpret_cast<uint4*>(st + WD_TILE + o) = l;
        }
        // generic-proxy stores -> visible to the tensor core (async proxy)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          arrive(&cfull[s]);
          arrive(&rempty[rs]);
        }
        __syncwarp();
        rs = rs + 1 == WD_NR ? 0 : rs + 1;
      }
    }
  } else {
    // ---------------- epilogue ----------------
    const int q = warp & 3;
    uint32_t acc_it = 0;
    bool ok = true;
    for (long long u = blockIdx.x; u < n_units && ok && !failed(); u += gridDim.x, ++acc_it) {
      const int a = acc_it & 1;
      ok = wait(&accf[a], (acc_it >> 1) & 1);
      if (!ok) break;
      tc::fence_after();
      int b, m0, n0;
      place(u, b, m0, n0);
      const int row = m0 + q * 32 + lane;
      const float* Cr = p.C ? p.C + b * p.sC + (long long)row * p.ldc + n0 : nullptr;
      float* Dr = p.D + b * p.sD + (long long)row * p.ldd + n0;
      const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * 2 * WD_B);
      const int cols = min(WD_B, p.N - n0);
#pragma unroll 1
      for (int c = 0; c < WD_B; c += 32) {
        float v[32], w[32];
        tc::tmem_ld32(ta + c, v);
        tc::tmem_ld32(ta + WD_B + c, w);
        if (c + 32 == WD_B) {   // the last read: the accumulator is free
          tc::fence_before();
          __syncwarp();
          if (lane == 0) arrive(&acce[a]);
          __syncwarp();
        }
        if (row < p.M) {
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            if (c + j >= cols) break;
            float4 x = make_float4(p.alpha * (v[j] + w[j]), p.alpha * (v[j + 1] + w[j + 1]),
                                   p.alpha * (v[j + 2] + w[j + 2]), p.alpha * (v[j + 3] + w[j + 3]));
            if (p.vec_out && c + j + 4 <= cols) {
              if (Cr) {
                const float4 y = *reinterpret_cast<const float4*>(Cr + c + j);
                x.x = fmaf(p.beta, y.x, x.x);
                x.y = fmaf(p.beta, y.y, x.y);
                x.z = fmaf(p.beta, y.z, x.z);
                x.w = fmaf(p.beta, y.w, x.w);
              }
              *reinterpret_cast<float4*>(Dr + c + j) = x;
            } else {
              const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (c + j + i < cols) Dr[c + j + i] = Cr ? fmaf(p.beta, Cr[c + j + i], xs[i]) : xs[i];
            }
          }
        }
      }
    }
  }
  __syncthreads();
  if (fail_s && tid == 0) {
    atomicExch(p.err, 1);
    // a second bounded chance for the loads and MMAs in flight to finish
    // before the CTA leaves and frees the tensor memory they write
    for (int s = 0; s < WD_NR; ++s)
      if (armed[s]) tc::mbar_wait(&rfull[s], (armed[s] - 1) & 1, limit);
    for (int s = 0; s < WD_NS; ++s)
      if (committed[s]) tc::mbar_wait(&cempty[s], (committed[s] - 1) & 1, limit);
    for (int a = 0; a < 2; ++a)
      if (acc_committed[a]) tc::mbar_wait(&accf[a], (acc_committed[a] - 1) & 1, limit);
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

bool al16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; }

}  // namespace

// Real view (M, N, K real; complex: N and K doubled, strides in floats).
template <bool CPLX>
static cudaError_t gemm_wide(int M, int N, int K, float alpha, const float* A, long long lda, long long sA,
                             const float* B, long long ldb, long long sB, float beta, const float* C, long long ldc,
                             long long sC, float* D, long long ldd, long long sD, int batch, cudaStream_t st) {
  if (M <= 0 || N <= 0 || batch <= 0) return cudaSuccess;
  if (K <= 0 || !al16(A) || !al16(B) || lda % 4 || ldb % 4 || lda < K || ldb < N) return cudaErrorNotSupported;
  if (batch > 1 && ((sA != 0 && sA % 4) || (sB != 0 && sB % 4))) return cudaErrorNotSupported;
  const int ab = (batch > 1 && sA != 0) ? 1 : 0, bb = (batch > 1 && sB != 0) ? 1 : 0;
  CUtensorMap tmA, tmB;
  if (!tma_map_f32(&tmA, A, K, M, ab ? batch : 1, lda, sA, WD_K, WD_B, true) ||
      !tma_map_f32(&tmB, B, N, CPLX ? K / 2 : K, bb ? batch : 1, ldb, sB, WD_B, CPLX ? WD_K / 2 : WD_K, false))
    return cudaErrorNotSupported;
  WideArgs p{M, N, K, alpha, beta, C, ldc, sC, D, ldd, sD, batch, ab, bb, 0, nullptr, nullptr};
  p.vec_out = al16(D) && ldd % 4 == 0 && (batch == 1 || sD % 4 == 0) &&
              (!C || (al16(C) && ldc % 4 == 0 && (batch == 1 || sC % 4 == 0)));
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(gemm_wide_kernel<CPLX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WD_SMEM);
  if (e == cudaSuccess) e = tc_wait_state(&p.err, &p.limit);
  if (e != cudaSuccess) return e;
  const long long units = (long long)batch * ((M + WD_B - 1) / WD_B) * ((N + WD_B - 1) / WD_B);
  ProfScope ps(KC_GEMM, st, 2.0 * M * (double)N * K * batch);
  note_launch();
  gemm_wide_kernel<CPLX><<<(unsigned)(units < sms ? units : sms), WD_NT, WD_SMEM, st>>>(tmA, tmB, p);
  return cudaGetLastError();
}

cudaError_t gemm_wide_f32(int M, int N, int K, float alpha, const float* A, long long lda, long long sA, const float* B,
                          long long ldb, long long sB, float beta, const float* C, long long ldc, long long sC, float* D,
                          long long ldd, long long sD, int batch, cudaStream_t st) {
  return gemm_wide<false>(M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, D, ldd, sD, batch, st);
}

cudaError_t gemm_wide_c64(int M, int N, int K, float alpha, const c64* A, long long lda, long long sA, const c64* B,
                          long long ldb, long long sB, float beta, const c64* C, long long ldc, long long sC, c64* D,
                          long long ldd, long long sD, int batch, cudaStream_t st) {
  return gemm_wide<true>(M, 2 * N, 2 * K, alpha, reinterpret_cast<const float*>(A), 2 * lda, 2 * sA,
                         reinterpret_cast<const float*>(B), 2 * ldb, 2 * sB, beta, reinterpret_cast<const float*>(C),
                         2 * ldc, 2 * sC, reinterpret_cast<float*>(D), 2 * ldd, 2 * sD, batch, st);
}

}  // namespace hps
