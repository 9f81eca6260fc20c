// FP64 and complex128 batched products on the FP16 tensor cores:
// D = alpha * A @ B + beta * C with every product formed from 8-bit slices
// (the error-free splitting of Ozaki, Ogita, Oishi and Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication", 2012).
//
// What bounds the plain kernel: GB300 issues two FP64 multiply-adds per SM
// and clock (1.25 TFLOP/s in all) while kind::f16 MMAs run 2,048 times as
// many.  Here each row of A and each column of B is scaled by a power of two
// to 62-bit integers, written as eight balanced base-256 digits (-128..127,
// exact in FP16), and the 36 digit products of the eight leading weights
// t + u <= 7 are MMAs.  A product of digits is at most 2^14, so the 8 * 128
// products that meet in one FP32 accumulator over 128 steps of K stay within
// 2^24: every accumulator is an exact integer.  After each 128 steps the
// accumulators are added in 64-bit integers, and the sum is rounded to FP64
// once, at the end.  What is lost is the tail below 2^-62 of a row's or a
// column's largest entry and the digit products below the eighth weight
// (about 2^-60 of the largest product): the FP64 chain's own rounding is
// 2^-53 of its partial sums at every step.  An entry of D all of whose large
// factors meet small ones keeps the bound K 2^-56 max|a_i| max|b_j| only:
// callers bring rows of such operands to one scale first (leaf_dtn_impl,
// balance_rows, gje_balance_kernel), and hps_gemm_batched, which knows nothing
// of its operands, runs here only when asked to.
//
// Measured (FP64 chain before, digits): 4096 x (196 x 56 x 196) 21.6 -> 1.22 ms
// (14.5 TFLOP/s), 512 x (512 x 384 x 512) 82.7 -> 4.2 ms (24.5), 1792^3 10.7
// -> 0.54 ms, complex 1024 x (256 x 56 x 256) 27.6 -> 1.45 ms, 4096 x (196 x 8 x
// 196) 4.4 -> 0.86 ms (1.42, 4.8, 0.60, 1.58 and 0.94 without tensor maps).  The
// conversion bounds long products (about 24 integer operations an element on
// the half-rate ALU, A once per 64 columns: 20,000 cycles of a 196 x 56 x 196
// tile); with K = 64 and less the reading warps do: 14,700 cycles a tile to
// round its sums and write D, 7,700 to read the accumulators.
#include <cuda.h>

#include "hps_common.cuh"
#include "hps_internal.h"
#include "digits.cuh"

namespace hps {

namespace {

using namespace digits;
using tc::mbar_init;
using tc::smem_u32;

constexpr int OZ_SL = 8;                 // digits
constexpr int OZ_CHUNK = 8;              // stages summed in the FP32 accumulators (128 steps of K)
constexpr int OZ_DW = 8;                 // warps 0-7 read the accumulators
constexpr int OZ_CW = 8;                 // warps 8-15 convert A and B
constexpr int OZ_CT = OZ_CW * 32;
constexpr int OZ_MW = OZ_DW + OZ_CW;     // warp 16 issues the MMAs (17-19 fill its warpgroup)
constexpr int OZ_NT = (OZ_MW + 4) * 32;
constexpr int OZ_EB = 8;                 // tiles whose exponents are kept (up to NS + 3 are in use)
constexpr int OZ_APL = OZ_BM * 32;       // bytes of one digit plane of A

template <int BN, bool TMA = false>
struct OzCfg {
  static constexpr int BPL = BN * 32;                       // bytes of one digit plane of B
  static constexpr int STAGE = OZ_SL * (OZ_APL + BPL);      // digits of 16 steps of K
  static constexpr int RAW = (OZ_BM + BN) * OZ_BK * 8;      // the same as FP64
  static constexpr int NS = (TMA && BN > 16) ? 2 : 3;       // digit stages
  static constexpr int NR = (TMA || BN <= 16) ? 5 : 3;      // FP64 stages (NR - 1 in flight)
  static constexpr size_t SMEM = (size_t)NS * STAGE + (size_t)NR * RAW + 1024;
  static constexpr int COLS = OZ_SL * BN;                   // TMEM columns: one block of BN per weight
  static constexpr int CW = BN / 2;                         // output columns per reading thread
  static constexpr int KB = BN * OZ_BK / OZ_CT;             // B values per converting thread and stage
};

__device__ __forceinline__ void load_box(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// Asynchronous copies of 16 or 8 bytes; `in` false writes zeros and reads nothing.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(in ? 8 : 0) : "memory");
}

struct OzArgs {
  int M, N, K;              // real sizes (complex: N and K doubled)
  double alpha, beta;
  const double* A;
  long long lda, sA;
  const double* B;
  long long ldb, sB;
  const double* C;
  long long ldc, sC;
  double* D;
  long long ldd, sD;
  int batch, vec_a, vec_d;
  const int* skip;          // products of the batch that are left out, or null
  int* err;
  const long long* limit;
};

// Products of a batch whose operands are blocks of larger matrices (hps_internal.h),
// with the first of the group's tiles.
template <bool GROUP>
struct OzGroups {
  int n, tiles;
  GemmGroup g[GEMM_GROUPS];
  int t0[GEMM_GROUPS];
};
template <>
struct OzGroups<false> {};

// Tensor maps of A and B as FP32 pairs, and whether each has a batch.
template <bool TMA>
struct OzMaps {
  CUtensorMap a, b;
  int a_batched, b_batched;
};
template <>
struct OzMaps<false> {};

// One tile: its matrix of the batch, its first row and column (inside the
// group), and the group.
struct OzTile {
  long long b;
  int m0, n0, g;
};

// One entry of D whose row of A or column of B holds an infinity or a NaN:
// the multiply-add chain of gemm_kernel.
template <bool CPLX>
__device__ __noinline__ double plain_entry(const OzArgs& p, const double* A, const double* B, int m, int n,
                                           const GemmGroup* g) {
  const int segs = g ? g->segs : 1;
  const double* a0 = A + (long long)m * p.lda;
  if constexpr (CPLX) {
    c128 s = zero<c128>();
    for (int i = 0; i < segs; ++i) {
      const int k0 = g ? g->k0[i] : 0, K = g ? g->len[i] : p.K / 2;
      const c128* a = reinterpret_cast<const c128*>(a0) + k0;
      for (int k = 0; k < K; ++k)
        s = fma_(a[k], *reinterpret_cast<const c128*>(B + (long long)(k0 + k) * p.ldb + (n & ~1)), s);
    }
    s = mul(c128{p.alpha, 0.0}, s);
    return (n & 1) ? s.y : s.x;
  } else {
    double s = 0.0;
    for (int i = 0; i < segs; ++i) {
      const int k0 = g ? g->k0[i] : 0, K = g ? g->len[i] : p.K;
      for (int k = 0; k < K; ++k) s = fma(a0[k0 + k], B[(long long)(k0 + k) * p.ldb + n], s);
    }
    return p.alpha * s;
  }
}

// One persistent CTA of 20 warps per SM.  For each 128 x BN tile of D
//   * warps 8-15 stream the tile's rows of A and columns of B through a ring
//     of FP64 stages twice (cp.async, NR - 1 stages ahead, each warp only
//     what it uses itself): once for the largest exponents (`expo`), once to
//     write the eight FP16 digit planes of each into a ring of stages of 16
//     steps of K (`full`, `empty`);
//   * one lane of warp 16 issues the MMAs of a stage;
//   * warps 0-7 read the eight accumulators (one per weight) after every 128
//     steps, add them into 96-bit integers (`accf`, `acce`), and after the
//     tile's last ones round the sums and write D.
// The weights 0-3 and 4-7 are two halves of the tensor memory: the next
// chunk's MMAs start on the first half while the second is read.  A digit
// plane of A meets the planes of B with t + u <= 7 side by side, as MMAs of
// up to 256 columns into consecutive weights' accumulators: A's plane is read
// from shared memory once for all of them.
// Registers: 32 columns of 96-bit sums take 96 registers in each of the 256
// reading threads; the 640 x 96 registers of the launch are divided 144 / 80 / 24,
// 144 / 72 / 48 with a copying warp (TMA).
// Every wait is bounded: after one that runs out a warp goes through its loop
// without waiting (so that the named barrier is met by all) and the CTA frees
// its tensor memory.
// GROUP: the products of all groups at once, K running through a group's
// segments one after another (each one's last stage filled up with zeros).
// TMA: warp 17 brings the FP64 stages, a box of A (128 rows of 16, 128-byte
// swizzled) and one of B each (`rfull`, `rempty`; 16-byte aligned rows and
// matrices).  With each converting warp issuing its own cp.async of 16 and 8
// bytes, those took 700 cycles of every step, 18,000 of the 50,000 of a 196 x
// 56 x 196 tile; a bulk copy per row takes 9,000 a step.
template <int BN, bool CPLX, bool SKIP, bool GROUP, bool TMA>
__global__ void __launch_bounds__(OZ_NT, 1) gemm_oz_kernel(const OzArgs p, const __grid_constant__ OzGroups<GROUP> gs, const __grid_constant__ OzMaps<TMA> maps) {
  using Cfg = OzCfg<BN, TMA>;
  static_assert(!(TMA && GROUP), "segments end where their neighbours begin");
  constexpr int NS = Cfg::NS, NR = Cfg::NR, CW = Cfg::CW, KB = Cfg::KB;
  extern __shared__ unsigned char oz_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(oz_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full[NS], empty[NS], accf[2], acce[2], expo[OZ_EB], rfull[NR], rempty[NR];
  __shared__ uint32_t committed[NS], acc_committed[2];
  __shared__ short row_e[OZ_EB][OZ_BM], col_e[OZ_EB][BN];
  __shared__ uint2 col_part[2][OZ_CT];
  __shared__ uint32_t tmem_s;
  __shared__ int fail_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long limit = *(const volatile long long*)p.limit;
  if (tid == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(&full[i], OZ_CW);
      mbar_init(&empty[i], 1);
      committed[i] = 0;
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&accf[i], 1);
      mbar_init(&acce[i], OZ_DW);
      acc_committed[i] = 0;
    }
    for (int i = 0; i < OZ_EB; ++i) mbar_init(&expo[i], OZ_CW);
    for (int i = 0; i < NR; ++i) {
      mbar_init(&rfull[i], 1);
      mbar_init(&rempty[i], OZ_CW);
    }
    fail_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == OZ_MW) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)),
                 "r"(Cfg::COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_s;
  constexpr int F = CPLX ? 2 : 1;
  const int tiles_n = (p.N + BN - 1) / BN, tiles_m = (p.M + OZ_BM - 1) / OZ_BM;
  const int per_b = [&] {
    if constexpr (GROUP) return gs.tiles;
    else return tiles_m * tiles_n;
  }();
  const long long n_units = (long long)per_b * p.batch;
  auto tile_of = [&](long long u) {
    OzTile t;
    t.b = u / per_b;
    const int r = (int)(u - t.b * per_b);
    if constexpr (GROUP) {
      int g = 0;
      while (g + 1 < gs.n && r >= gs.t0[g + 1]) ++g;
      const int tn = (F * gs.g[g].n + BN - 1) / BN, i = r - gs.t0[g];
      t.g = g, t.m0 = (i / tn) * OZ_BM, t.n0 = (i % tn) * BN;
    } else {
      t.g = 0, t.m0 = (r / tiles_n) * OZ_BM, t.n0 = (r % tiles_n) * BN;
    }
    return t;
  };
  const int nk_all = (p.K + OZ_BK - 1) / OZ_BK;
  auto stages_of = [&](long long u) {
    if constexpr (GROUP) {
      const GemmGroup& g = gs.g[tile_of(u).g];
      int k = 0;
      for (int i = 0; i < g.segs; ++i) k += (F * g.len[i] + OZ_BK - 1) / OZ_BK;
      return k;
    } else {
      return nk_all;
    }
  };
  // sizes of a tile's product (real), and where its blocks begin (in doubles)
  auto rows_of = [&](const OzTile& t) {
    if constexpr (GROUP) return gs.g[t.g].m;
    else return p.M;
  };
  auto cols_of = [&](const OzTile& t) {
    if constexpr (GROUP) return F * gs.g[t.g].n;
    else return p.N;
  };
  auto row0_of = [&](const OzTile& t) {
    if constexpr (GROUP) return gs.g[t.g].m0;
    else return 0;
  };
  auto col0_of = [&](const OzTile& t) {
    if constexpr (GROUP) return F * gs.g[t.g].n0;
    else return 0;
  };
  // the first of the CTA's tiles u, u + gridDim.x, ... that is not left out
  auto tile_from = [&](long long u) {
    if constexpr (SKIP)
      while (u < n_units && p.skip[u / per_b]) u += gridDim.x;
    return u;
  };
  const long long u0 = tile_from(blockIdx.x);
  bool ok = true;
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (ok) ok = (bool)__all_sync(0xffffffffu, tc::mbar_wait(bar, parity, limit));
  };

  if (warp < OZ_DW) {
    // ---------------- accumulators -> 96-bit sums -> D ----------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
    const int q = warp & 3, cg = warp >> 2;   // TMEM lanes 32 q .., columns CW cg ..
    const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(cg * CW);
    uint32_t s0[CW], s1[CW], s2[CW];
    uint32_t ch = 0, tile = 0;
    for (long long u = u0; u < n_units; u = tile_from(u + gridDim.x), ++tile) {
      const int nk = stages_of(u);
#pragma unroll
      for (int j = 0; j < CW; ++j) s0[j] = s1[j] = s2[j] = 0;
      for (int kt = 0; kt < nk; kt += OZ_CHUNK, ++ch) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          wait(&accf[h], ch & 1);
          tc::fence_after();
#pragma unroll
          for (int c = 0; c < CW; c += 4) {
            uint32_t v[4][4];
#pragma unroll
            for (int l = 0; l < 4; ++l) tmem_ld4(tb + (uint32_t)((h * 4 + l) * BN + c), v[l]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              long long x = __float2int_rn(__uint_as_float(v[3][j]));
#pragma unroll
              for (int l = 0; l < 3; ++l)
                asm("mad.wide.s32 %0, %1, %2, %0;"
                    : "+l"(x)
                    : "r"(__float2int_rn(__uint_as_float(v[l][j]))), "r"(1 << (8 * (3 - l))));
              const uint32_t xl = (uint32_t)x, xh = (uint32_t)((unsigned long long)x >> 32);
              if (h == 0) {
                asm("add.cc.u32 %0, %0, %2;\n addc.u32 %1, %1, %3;" : "+r"(s1[c + j]), "+r"(s2[c + j]) : "r"(xl), "r"(xh));
              } else {
                asm("add.cc.u32 %0, %0, %3;\n addc.cc.u32 %1, %1, %4;\n addc.u32 %2, %2, %5;"
                    : "+r"(s0[c + j]), "+r"(s1[c + j]), "+r"(s2[c + j])
                    : "r"(xl), "r"(xh), "r"((uint32_t)((int)xh >> 31)));
              }
            }
          }
          tc::fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acce[h]);
          __syncwarp();
        }
      }
      const int eb = tile % OZ_EB;
      wait(&expo[eb], (tile / OZ_EB) & 1);
      const OzTile t = tile_of(u);
      const long long b = t.b;
      const int row = t.m0 + q * 32 + lane, c0 = t.n0 + cg * CW, N = cols_of(t);
      if (!ok || row >= rows_of(t) || c0 >= N) continue;
      const int re = row_e[eb][q * 32 + lane], r0 = row0_of(t) + row, n0 = col0_of(t) + c0;   // in the matrices
      const double* Cr = p.C ? p.C + b * p.sC + (long long)r0 * p.ldc + n0 : nullptr;
      double* Dr = p.D + b * p.sD + (long long)r0 * p.ldd + n0;
      const bool neg = p.alpha == -1.0;
#pragma unroll
      for (int g = 0; g < CW; g += 4) {
        if (c0 + g >= N) break;
        double v[4];
        bool odd = re >= 0x7ff;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int ce = col_e[eb][cg * CW + g + j];
          odd = odd || ce >= 0x7ff;
          v[j] = round_sum(s0[g + j], s1[g + j], s2[g + j], re + ce - 2112, odd);
        }
        if (odd || !(neg || p.alpha == 1.0)) {
          // results beyond the range as the chain gives them, too (a complex
          // one spreads an infinity to both of its parts)
          bool plain[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int ce = col_e[eb][cg * CW + g + j];
            plain[j] = re >= 0x7ff || ce >= 0x7ff;
            if (!plain[j]) {
              v[j] = p.alpha * round_sum_any(s0[g + j], s1[g + j], s2[g + j], re + ce - 2112);
              plain[j] = !isfinite(v[j]);
            }
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if ((plain[j] || (CPLX && plain[j ^ 1])) && c0 + g + j < N) {
              const GemmGroup* gp = nullptr;
              if constexpr (GROUP) gp = &gs.g[t.g];
              v[j] = plain_entry<CPLX>(p, p.A + b * p.sA, p.B + b * p.sB, r0, n0 + g + j, gp);
            }
        } else if (neg) {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = -v[j];
        }
        if (c0 + g + 4 <= N && p.vec_d) {
          if (Cr) {
            const double2 x = *reinterpret_cast<const double2*>(Cr + g), y = *reinterpret_cast<const double2*>(Cr + g + 2);
            v[0] = fma(p.beta, x.x, v[0]);
            v[1] = fma(p.beta, x.y, v[1]);
            v[2] = fma(p.beta, y.x, v[2]);
            v[3] = fma(p.beta, y.y, v[3]);
          }
          *reinterpret_cast<double2*>(Dr + g) = make_double2(v[0], v[1]);
          *reinterpret_cast<double2*>(Dr + g + 2) = make_double2(v[2], v[3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (c0 + g + j < N) Dr[g + j] = Cr ? fma(p.beta, Cr[g + j], v[j]) : v[j];
        }
      }
    }
  } else if (warp < OZ_MW) {
    // ---------------- FP64 -> exponents, digit planes ----------------
    if constexpr (TMA) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    const int ct = tid - OZ_DW * 32, cw = ct >> 5;
    const int ar = ct >> 1, ah = ct & 1;                // A: one row, steps 8 ah .. 8 ah + 7
    const int bn = ct % BN, bk = (ct / BN) * KB;        // B: one column, KB steps
    const uint32_t a_off = (uint32_t)(ar * 32 + ((ah ^ ((ar >> 2) & 1)) << 4));
    const uint32_t b_off = (uint32_t)(OZ_SL * OZ_APL + bn * 32 + (((bk >> 3) ^ ((bn >> 2) & 1)) << 4) + (bk & 7) * 2);
    // this warp's part of an FP64 stage: 16 rows of A (128 bytes each, 16-byte
    // pieces c at c ^ (row mod 8)), then KB x 32 values of B
    unsigned char* raw = smem + NS * Cfg::STAGE + cw * (16 * 128 + KB * 256);
    const uint32_t raw_s = smem_u32(raw);
    const int rr = ar & 15;

    // the stage that is copied next: a tile's stages twice
    long long lu = u0;
    int lslot = 0, lpass = 0, lseg = 0, lk = 0, lseg_len = 0;   // step inside the segment (all of K without groups)
    auto seg_len = [&] {
      if constexpr (GROUP) return lseg_len;
      else return p.K;
    };
    const double *lA = nullptr, *lB = nullptr;   // this lane's first piece of A, the thread's column of B, at the stage's first step
    int lrows = 0;                              // rows of this warp inside A
    bool lb_in = false;
    const int pr = p.vec_a ? lane >> 3 : lane >> 4, pc = p.vec_a ? lane & 7 : lane & 15;   // row and piece of a copy
    auto segment_ptrs = [&]() {
      const OzTile t = tile_of(lu);
      const int m = t.m0 + 16 * cw + pr, n = t.n0 + bn;
      lrows = rows_of(t) - m;
      lA = p.A + t.b * p.sA + (long long)(row0_of(t) + m) * p.lda + (p.vec_a ? 2 * pc : pc);
      lb_in = n < cols_of(t);
      lB = p.B + t.b * p.sB + (CPLX ? (long long)(bk >> 1) * p.ldb + (n & ~1) : (long long)bk * p.ldb + n) + col0_of(t);
      lk = 0;
      if constexpr (GROUP) {
        lseg_len = F * gs.g[t.g].len[lseg];
        lA += F * gs.g[t.g].k0[lseg];
        lB += (long long)gs.g[t.g].k0[lseg] * p.ldb;
      }
    };
    if (!TMA && lu < n_units) segment_ptrs();
    const double* safe = p.A;   // an address for copies that read nothing
    auto copy_stage = [&]() {
      if (lu < n_units) {
        const uint32_t dst = raw_s + lslot * Cfg::RAW;
        const int k0 = lk, lK = seg_len();
        const bool whole = k0 + OZ_BK <= lK;
        if (p.vec_a) {
          const uint32_t d = dst + pr * 128;
          if (whole) {
#pragma unroll
            for (int i = 0; i < 4; ++i)   // row pr + 4 i: its swizzle is pr ^ 4 (i & 1)
              cp_async16(d + i * 512 + ((pc ^ pr ^ (4 * (i & 1))) << 4), 4 * i < lrows ? lA + (long long)(4 * i) * p.lda : safe,
                         4 * i < lrows);
          } else {
            const int left = lK - k0 - 2 * pc;   // values of this piece inside the row
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t x = d + i * 512 + ((pc ^ pr ^ (4 * (i & 1))) << 4);
              const double* src = lA + (long long)(4 * i) * p.lda;
              const bool in = 4 * i < lrows;
              cp_async8(x, in && left > 0 ? src : safe, in && left > 0);
              cp_async8(x + 8, in && left > 1 ? src + 1 : safe, in && left > 1);
            }
          }
        } else {
          const bool kin = k0 + pc < lK;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const bool in = kin && 2 * i < lrows;
            cp_async8(dst + (2 * i + pr) * 128 + (((pc >> 1) ^ ((2 * i + pr) & 7)) << 4) + (pc & 1) * 8,
                      in ? lA + (long long)(2 * i) * p.lda : safe, in);
          }
        }
        const int left = lb_in ? lK - k0 - bk : 0;
#pragma unroll
        for (int i = 0; i < KB; ++i) {
          const double* src = CPLX ? lB + (long long)(KB > 1 ? i >> 1 : 0) * p.ldb + ((bk + i + bn) & 1) : lB + (long long)i * p.ldb;
          cp_async8(dst + 16 * 128 + i * 256 + lane * 8, i < left ? src : safe, i < left);
        }
        lslot = lslot + 1 == NR ? 0 : lslot + 1;
        lA += OZ_BK;
        lB += (long long)(CPLX ? OZ_BK / 2 : OZ_BK) * p.ldb;
        lk += OZ_BK;
        if (lk >= seg_len()) {
          bool end = true;
          if constexpr (GROUP) {
            end = ++lseg == gs.g[tile_of(lu).g].segs;
            if (end) lseg = 0;
          }
          if (end && ++lpass == 2) {
            lpass = 0;
            lu = tile_from(lu + gridDim.x);
          }
          if (lu < n_units) segment_ptrs();
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if constexpr (!TMA) {
#pragma unroll
      for (int i = 0; i < NR - 1; ++i) copy_stage();
    }
    int slot = 0;
    uint32_t round = 0;   // of the ring (TMA)
    // the next FP64 stage, and the copy into the slot read before it
    auto next_raw = [&]() -> const unsigned char* {
      if constexpr (TMA) {
        wait(&rfull[slot], round & 1);
        return smem + NS * Cfg::STAGE + slot * Cfg::RAW;
      }
      asm volatile("cp.async.wait_group %0;" ::"n"(NR - 2) : "memory");
      __syncwarp();   // the warp's copies are visible to all of its lanes, and all have read the slot refilled next
      const unsigned char* rw = raw + slot * Cfg::RAW;
      slot = slot + 1 == NR ? 0 : slot + 1;
      copy_stage();
      return rw;
    };
    // this warp has read the stage
    auto raw_done = [&]() {
      if constexpr (TMA) {
        // the lanes' loads, which may still be on their way, before the next box's
        // write (without this fence a few rows and columns per thousand short
        // tiles took their exponents from the box after)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&rempty[slot]);
        if (++slot == NR) slot = 0, ++round;
      }
    };
    // two of the thread's values of A and one of B
    auto raw_a = [&](const unsigned char* rw, int i) {
      const unsigned char* r = TMA ? rw + ar * 128 : rw + rr * 128;   // (ar mod 8 = rr mod 8)
      return *reinterpret_cast<const uint4*>(r + (((4 * ah + i) ^ (rr & 7)) << 4));
    };
    auto raw_b = [&](const unsigned char* rw, int i) {
      if constexpr (TMA) {
        const int k = bk + i;
        const unsigned char* b = rw + OZ_BM * 128;
        return CPLX ? *reinterpret_cast<const uint2*>(b + (k >> 1) * (BN * 8) + ((bn & ~1) + ((k + bn) & 1)) * 8)
                    : *reinterpret_cast<const uint2*>(b + k * (BN * 8) + bn * 8);
      }
      return *reinterpret_cast<const uint2*>(rw + 16 * 128 + i * 256 + lane * 8);
    };
    // 0x7ff for a row or column that cannot be scaled (infinities, NaN, or nothing but tiny values)
    auto code = [](uint32_t top, uint32_t low) {
      const int x = (int)(top >> 20);
      return (top | low) == 0 ? 1024 : x <= 64 ? 0x7ff : x;
    };

    uint32_t it = 0, tile = 0;
    for (long long u = u0; u < n_units; u = tile_from(u + gridDim.x), ++tile) {
      const int nk = stages_of(u);
      uint32_t ae, be;
      {
        uint32_t at = 0, al = 0, bt = 0, bl = 0;
        for (int kt = 0; kt < nk; ++kt) {
          const unsigned char* rw = next_raw();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 v = raw_a(rw, i);
            at = max(at, max(v.y & 0x7fffffffu, v.w & 0x7fffffffu));
            al |= v.x | v.z;
          }
#pragma unroll
          for (int i = 0; i < KB; ++i) {
            const uint2 v = raw_b(rw, i);
            bt = max(bt, v.y & 0x7fffffffu);
            bl |= v.x;
          }
          raw_done();
        }
        at = max(at, __shfl_xor_sync(0xffffffffu, at, 1));
        al |= __shfl_xor_sync(0xffffffffu, al, 1);
        if (CPLX) {   // the two columns of a complex one share their scale
          bt = max(bt, __shfl_xor_sync(0xffffffffu, bt, 1));
          bl |= __shfl_xor_sync(0xffffffffu, bl, 1);
        }
        col_part[tile & 1][ct] = make_uint2(bt, bl);
        asm volatile("bar.sync 1, %0;" ::"n"(OZ_CT) : "memory");
#pragma unroll
        for (int g = 1; g < OZ_CT / BN; ++g) {
          const uint2 v = col_part[tile & 1][(ct + g * BN) % OZ_CT];
          bt = max(bt, v.x);
          bl |= v.y;
        }
        const int ac = code(at, al), bc = code(bt, bl), e = tile % OZ_EB;
        if (ah == 0) row_e[e][ar] = (short)ac;
        if (ct < BN) col_e[e][bn] = (short)bc;
        __syncwarp();
        if (lane == 0) mbar_arrive(&expo[e]);
        ae = (uint32_t)ac << 20;
        be = (uint32_t)bc << 20;
      }
      for (int kt = 0; kt < nk; ++kt, ++it) {
        const int s = it % NS;
        const unsigned char* rw = next_raw();
        if (it >= NS) wait(&empty[s], (it / NS - 1) & 1);
        unsigned char* sb = smem + s * Cfg::STAGE;
        {
          uint32_t x[16], one[4], off[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 v = raw_a(rw, i);
            x[4 * i] = v.x, x[4 * i + 1] = v.y, x[4 * i + 2] = v.z, x[4 * i + 3] = v.w;
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) sign_pair(x[4 * i + 1], x[4 * i + 3], one[i], off[i]);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint2 y = to_digits(x[2 * i], x[2 * i + 1], ae);
            x[2 * i] = y.x, x[2 * i + 1] = y.y;
          }
          unsigned char* d = sb + a_off;
#pragma unroll
          for (int w = 0; w < 4; ++w) {   // digits 2w, 2w + 1
            uint32_t z[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              z[i] = __byte_perm(x[4 * i + (w < 2)], x[4 * i + 2 + (w < 2)], (w & 1) ? 0x4051 : 0x6273);
            *reinterpret_cast<uint4*>(d + (2 * w) * OZ_APL) =
                make_uint4(f16_digits(z[0], 0x4140, one[0], off[0]), f16_digits(z[1], 0x4140, one[1], off[1]),
                           f16_digits(z[2], 0x4140, one[2], off[2]), f16_digits(z[3], 0x4140, one[3], off[3]));
            *reinterpret_cast<uint4*>(d + (2 * w + 1) * OZ_APL) =
                make_uint4(f16_digits(z[0], 0x4342, one[0], off[0]), f16_digits(z[1], 0x4342, one[1], off[1]),
                           f16_digits(z[2], 0x4342, one[2], off[2]), f16_digits(z[3], 0x4342, one[3], off[3]));
          }
        }
        {
          constexpr int PB = (KB + 1) / 2;
          uint2 x[2 * PB];
          uint32_t one[PB], off[PB];
#pragma unroll
          for (int i = 0; i < KB; ++i) {
            x[i] = raw_b(rw, i);
            // real view of a complex column: rows 2k, 2k + 1 are (re, -im) or (im, re)
            if (CPLX && ((bk + i) & 1) && !(bn & 1)) x[i].y ^= 0x80000000u;
          }
          raw_done();
          if constexpr (KB == 1) x[1] = x[0];
#pragma unroll
          for (int i = 0; i < PB; ++i) sign_pair(x[2 * i].y, x[2 * i + 1].y, one[i], off[i]);
#pragma unroll
          for (int i = 0; i < 2 * PB; ++i) x[i] = to_digits(x[i].x, x[i].y, be);
          unsigned char* d = sb + b_off;
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            uint32_t d0[PB], d1[PB];
#pragma unroll
            for (int i = 0; i < PB; ++i) {
              const uint32_t z = __byte_perm(w < 2 ? x[2 * i].y : x[2 * i].x, w < 2 ? x[2 * i + 1].y : x[2 * i + 1].x,
                                             (w & 1) ? 0x4051 : 0x6273);
              d0[i] = f16_digits(z, 0x4140, one[i], off[i]);
              d1[i] = f16_digits(z, 0x4342, one[i], off[i]);
            }
            unsigned char* o = d + (2 * w) * Cfg::BPL;
            if constexpr (KB == 4) {
              *reinterpret_cast<uint2*>(o) = make_uint2(d0[0], d0[1]);
              *reinterpret_cast<uint2*>(o + Cfg::BPL) = make_uint2(d1[0], d1[1]);
            } else {
              static_assert(KB == 1 || KB == 4, "B split");
              *reinterpret_cast<unsigned short*>(o) = (unsigned short)d0[0];
              *reinterpret_cast<unsigned short*>(o + Cfg::BPL) = (unsigned short)d1[0];
            }
          }
        }
        // generic-proxy stores -> visible to the tensor core (async proxy)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[s]);
        __syncwarp();
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    // ---------------- MMA issuer ----------------
    if constexpr (TMA) asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
    if constexpr (TMA) {
      if (warp == OZ_MW + 1) {
        // ---------------- copies ----------------
        constexpr uint32_t BYTES = OZ_BM * 128 + (CPLX ? OZ_BK / 2 : OZ_BK) * BN * 8;
        int s = 0;
        uint32_t it = 0;
        for (long long u = u0; u < n_units && ok; u = tile_from(u + gridDim.x)) {
          const OzTile t = tile_of(u);
          const int za = maps.a_batched ? (int)t.b : 0, zb = maps.b_batched ? (int)t.b : 0;
          for (int k = 0; k < 2 * nk_all; ++k, ++it) {
            const int k0 = (k < nk_all ? k : k - nk_all) * OZ_BK;
            if (it >= NR) wait(&rempty[s], (it / NR - 1) & 1);
            if (!ok) break;
            if (lane == 0) {
              const uint32_t dst = smem_u32(smem + NS * Cfg::STAGE + s * Cfg::RAW);
              asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&rfull[s])), "r"(BYTES)
                           : "memory");
              load_box(dst, &maps.a, 2 * k0, t.m0, za, &rfull[s]);
              load_box(dst + OZ_BM * 128, &maps.b, 2 * t.n0, CPLX ? k0 / 2 : k0, zb, &rfull[s]);
            }
            __syncwarp();
            s = s + 1 == NR ? 0 : s + 1;
          }
        }
        if (!ok) {   // a second bounded chance for the copies in flight
          for (int i = 0; i < NR; ++i)
            if (it > (uint32_t)i) tc::mbar_wait(&rfull[i], ((it - 1 - i) / NR) & 1, limit);
        }
      }
    }
    if (warp == OZ_MW) {
      uint32_t it = 0, ch = 0;
      int s = 0;
      for (long long u = u0; u < n_units; u = tile_from(u + gridDim.x)) {
        const int nk = stages_of(u);
        for (int kt = 0; kt < nk; ++kt, ++it) {
          const bool first = kt % OZ_CHUNK == 0, last = kt % OZ_CHUNK == OZ_CHUNK - 1 || kt == nk - 1;
          wait(&full[s], (it / NS) & 1);
          const uint32_t a0 = desc_lo(smem_u32(smem + s * Cfg::STAGE)), b0 = a0 + ((OZ_SL * OZ_APL) >> 4);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (first && ch > 0) wait(&acce[h], (ch - 1) & 1);
            tc::fence_after();
            if (ok && lane == 0) {
#pragma unroll
              for (int t = 0; t < OZ_SL; ++t) {
                // weights w of this half with u = w - t >= 0
                const int w0 = h * 4 > t ? h * 4 : t, nw = h * 4 + 4 - w0;
                if (nw <= 0) continue;
                mma_f16(tmem + w0 * BN, a0 + ((t * OZ_APL) >> 4), b0 + (((w0 - t) * Cfg::BPL) >> 4), idesc_f16(nw * BN),
                        (t == 0 && first) ? 0u : 1u);
              }
              if (last) {
                tc::mma_commit(&accf[h]);
                acc_committed[h] += 1;
              }
              if (h == 1) {
                tc::mma_commit(&empty[s]);
                committed[s] += 1;
              }
            }
            __syncwarp();
          }
          if (last) ++ch;
          s = s + 1 == NS ? 0 : s + 1;
        }
      }
    }
  }
  if (!ok) fail_s = 1;
  __syncthreads();
  if (fail_s && tid == 0) {
    atomicExch(p.err, 1);
    // a second bounded chance for the MMAs in flight to finish before the
    // tensor memory they write is freed
    for (int s = 0; s < NS; ++s)
      if (committed[s]) tc::mbar_wait(&empty[s], (committed[s] - 1) & 1, limit);
    for (int a = 0; a < 2; ++a)
      if (acc_committed[a]) tc::mbar_wait(&accf[a], (acc_committed[a] - 1) & 1, limit);
  }
  tc::fence_before();
  __syncthreads();
  if (warp == OZ_MW) {
    tc::fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::COLS) : "memory");
  }
}

template <int BN, bool CPLX, bool SKIP, bool GROUP = false, bool TMA = false>
cudaError_t launch_oz(OzArgs p, cudaStream_t st, const OzGroups<GROUP>& gs = {}, const OzMaps<TMA>& maps = {}) {
  using Cfg = OzCfg<BN, TMA>;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(gemm_oz_kernel<BN, CPLX, SKIP, GROUP, TMA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM);
  if (e == cudaSuccess) e = tc_wait_state(&p.err, &p.limit);
  if (e != cudaSuccess) return e;
  long long units = (long long)p.batch * ((p.M + OZ_BM - 1) / OZ_BM) * ((p.N + BN - 1) / BN);
  if constexpr (GROUP) units = (long long)p.batch * gs.tiles;
  note_launch();
  gemm_oz_kernel<BN, CPLX, SKIP, GROUP, TMA><<<(unsigned)(units < sms ? units : sms), OZ_NT, Cfg::SMEM, st>>>(p, gs, maps);
  return cudaGetLastError();
}

}  // namespace

template <bool CPLX>
static cudaError_t gemm_oz(int M, int N, int K, double alpha, const double* A, long long lda, long long sA,
                           const double* B, long long ldb, long long sB, double beta, const double* C, long long ldc,
                           long long sC, double* D, long long ldd, long long sD, int batch, cudaStream_t st, const int* skip) {
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  OzArgs p{M, N, K, alpha, beta, A, lda, sA, B, ldb, sB, C, ldc, sC, D, ldd, sD, batch, 0, 0, skip, nullptr, nullptr};
  p.vec_a = al16(A) && lda % 2 == 0 && (batch == 1 || sA % 2 == 0);
  p.vec_d = al16(D) && ldd % 2 == 0 && (batch == 1 || sD % 2 == 0) &&
            (!C || (al16(C) && ldc % 2 == 0 && (batch == 1 || sC % 2 == 0)));
  ProfScope ps(KC_GEMM, st, 2.0 * M * (double)N * K * batch * (CPLX ? 2.0 : 1.0));
  if (skip) return launch_oz<64, CPLX, true>(p, st);
  // A tile per SM and more: the two tensor maps cost the host some 2 us a launch,
  // which the few tiles of a smaller product do not win back (256 leaves of 13^2
  // took 3.81 ms with maps everywhere, 3.78 without any).
  const long long tiles = (long long)batch * ((M + OZ_BM - 1) / OZ_BM) * ((N + 63) / 64);
  if (tiles >= 152 && p.vec_a && al16(B) && ldb % 2 == 0 && (batch == 1 || sB % 2 == 0)) {
    // FP64 numbers as FP32 pairs; boxes reach over the edges into zeros
    OzMaps<true> m;
    m.a_batched = batch > 1 && sA != 0;
    m.b_batched = batch > 1 && sB != 0;
    const int bn = N <= 16 ? 16 : 64;
    if (tma_map_f32(&m.a, reinterpret_cast<const float*>(A), 2ll * K, M, m.a_batched ? batch : 1, 2 * lda, 2 * sA, 2 * OZ_BK,
                    OZ_BM, true) &&
        tma_map_f32(&m.b, reinterpret_cast<const float*>(B), 2ll * N, CPLX ? K / 2 : K, m.b_batched ? batch : 1, 2 * ldb, 2 * sB,
                    2 * bn, CPLX ? OZ_BK / 2 : OZ_BK, false))
      return bn == 16 ? launch_oz<16, CPLX, false, false, true>(p, st, {}, m)
                      : launch_oz<64, CPLX, false, false, true>(p, st, {}, m);
  }
  if (N <= 16) return launch_oz<16, CPLX, false>(p, st);
  return launch_oz<64, CPLX, false>(p, st);
}

template <class T>
cudaError_t gemm_groups(const GemmGroup* groups, int n, double alpha, const T* A, long long lda, long long sA, const T* B,
                        long long ldb, long long sB, double beta, const T* C, long long ldc, long long sC, T* D,
                        long long ldd, long long sD, int batch, cudaStream_t st) {
  constexpr bool CPLX = DTypeOf<T>::value == C128;
  constexpr int F = CPLX ? 2 : 1;
  if (n < 1 || n > GEMM_GROUPS) return cudaErrorInvalidValue;
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  OzArgs p{0, 0, 0, alpha, beta, (const double*)A, F * lda, F * sA, (const double*)B, F * ldb, F * sB, (const double*)C,
           F * ldc, F * sC, (double*)D, F * ldd, F * sD, batch, 0, 0, nullptr, nullptr, nullptr};
  OzGroups<true> gs;
  gs.n = n;
  gs.tiles = 0;
  bool even_k = true, even_n = true;
  double flop = 0.0;
  for (int i = 0; i < n; ++i) {
    const GemmGroup& g = gs.g[i] = groups[i];
    gs.t0[i] = gs.tiles;
    gs.tiles += ((g.m + OZ_BM - 1) / OZ_BM) * ((F * g.n + 63) / 64);
    even_n = even_n && F * g.n0 % 2 == 0;
    for (int k = 0; k < g.segs; ++k) {
      even_k = even_k && F * g.k0[k] % 2 == 0;
      flop += 2.0 * F * F * g.m * (double)g.n * g.len[k] * batch;
    }
  }
  p.vec_a = even_k && al16(A) && p.lda % 2 == 0 && (batch == 1 || p.sA % 2 == 0);
  p.vec_d = even_n && al16(D) && p.ldd % 2 == 0 && (batch == 1 || p.sD % 2 == 0) &&
            (!C || (al16(C) && p.ldc % 2 == 0 && (batch == 1 || p.sC % 2 == 0)));
  ProfScope ps(KC_GEMM, st, flop);
  return launch_oz<64, CPLX, false, true>(p, st, gs);
}

template cudaError_t gemm_groups<double>(const GemmGroup*, int, double, const double*, long long, long long,
                                         const double*, long long, long long, double, const double*, long long, long long,
                                         double*, long long, long long, int, cudaStream_t);
template cudaError_t gemm_groups<c128>(const GemmGroup*, int, double, const c128*, long long, long long, const c128*,
                                       long long, long long, double, const c128*, long long, long long, c128*, long long,
                                       long long, int, cudaStream_t);

cudaError_t gemm_f64_tc(int M, int N, int K, double alpha, const double* A, long long lda, long long sA,
                        const double* B, long long ldb, long long sB, double beta, const double* C, long long ldc,
                        long long sC, double* D, long long ldd, long long sD, int batch, cudaStream_t st,
                        const int* skip) {
  return gemm_oz<false>(M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, D, ldd, sD, batch, st, skip);
}

// complex128 as the real product of the interleaved views, sizes (M, 2N, 2K).
cudaError_t gemm_c128_tc(int M, int N, int K, double alpha, const c128* A, long long lda, long long sA, const c128* B,
                         long long ldb, long long sB, double beta, const c128* C, long long ldc, long long sC, c128* D,
                         long long ldd, long long sD, int batch, cudaStream_t st, const int* skip) {
  return gemm_oz<true>(M, 2 * N, 2 * K, alpha, reinterpret_cast<const double*>(A), 2 * lda, 2 * sA,
                       reinterpret_cast<const double*>(B), 2 * ldb, 2 * sB, beta, reinterpret_cast<const double*>(C),
                       2 * ldc, 2 * sC, reinterpret_cast<double*>(D), 2 * ldd, 2 * sD, batch, st, skip);
}

}  // namespace hps
