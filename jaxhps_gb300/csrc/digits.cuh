// Helpers of the digit products (gemm_f64_tc.cu, gemm_digits.cu): FP64 values
// as balanced base-256 digits in FP16, their MMAs' descriptors, and exact
// integer sums rounded to FP64.
#pragma once

#include "tc_common.cuh"

namespace hps {
namespace digits {

using tc::smem_u32;

constexpr int OZ_BM = 128;   // rows of an output tile (TMEM lanes)
constexpr int OZ_BK = 16;    // K steps of a stage (one MMA): a digit row is 32 bytes

// K-major tile with 32-byte rows, 32-byte swizzle: 8-row groups 256 bytes
// apart; the 16-byte chunk c of row r lies at chunk c ^ ((r / 4) mod 2).
// Upper word: group stride, version bits, swizzle code 6; lower word: address.
constexpr uint32_t OZ_DESC_HI = (256u >> 4) | (1u << 14) | (6u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFF) >> 4) | (1u << 16); }

// D F32 (bits 4-5 = 1), A and B F16 (0), both K-major.
__host__ __device__ constexpr uint32_t idesc_f16(int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(OZ_BM >> 4) << 24);
}

__device__ __forceinline__ void mma_f16(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 da, db;\n setp.ne.b32 p, %4, 0;\n mov.b64 da, {%1, %5};\n mov.b64 db, {%2, %5};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n}\n" ::"r"(d),
      "r"(a), "r"(b), "r"(idesc), "r"(acc), "r"(OZ_DESC_HI)
      : "memory");
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// |x| (its two words) as floor(|x| * 2^(62 - E)) with |x| < 2^E, E = emax - 1022,
// plus 0x80 in every byte: byte 7 - t is digit t + 128.  emax > 64, so that a
// zero or subnormal x is shifted out.
__device__ __forceinline__ uint2 to_digits(uint32_t lo, uint32_t hi, uint32_t emax20) {
  const uint32_t mh = (hi & 0xfffffu) | 0x100000u;
  const uint32_t d = (emax20 - (hi & 0x7ff00000u)) >> 20;
  uint32_t yl, yh;
  asm("{\n .reg .b64 m;\n mov.b64 m, {%2, %3};\n shr.u64 m, m, %4;\n add.u64 m, m, 0x8080808080808080;\n"
      " mov.b64 {%0, %1}, m;\n}\n"
      : "=r"(yl), "=r"(yh)
      : "r"(lo << 9), "r"(__funnelshift_l(lo, mh, 9)), "r"(d));
  return make_uint2(yl, yh);
}

// Two elements' signs as FP16 factors +-1 and the offsets -+1152.
__device__ __forceinline__ void sign_pair(uint32_t hi0, uint32_t hi1, uint32_t& one, uint32_t& off) {
  const uint32_t p = __byte_perm(hi0, hi1, 0x7030) & 0x80008000u;
  one = p | 0x3C003C00u;
  off = p ^ 0xE480E480u;
}

// Two bytes of z as FP16 digits: (1024 + byte) * sign - 1152 * sign.
__device__ __forceinline__ uint32_t f16_digits(uint32_t z, uint32_t sel, uint32_t one, uint32_t off) {
  uint32_t h = __byte_perm(z, 0x64646464u, sel), r;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(h), "r"(one), "r"(off));
  return r;
}

// The 96-bit integer (s2, s1, s0) times 2^e, rounded to nearest even.  `odd`
// is set where the result's exponent is not that of a normal number.
__device__ __forceinline__ double round_sum(uint32_t s0, uint32_t s1, uint32_t s2, int e, bool& odd) {
  const uint32_t sg = (uint32_t)((int)s2 >> 31);
  // magnitude
  uint32_t m0, m1, m2;
  asm("sub.cc.u32 %0, %3, %6;\n subc.cc.u32 %1, %4, %6;\n subc.u32 %2, %5, %6;"
      : "=r"(m0), "=r"(m1), "=r"(m2)
      : "r"(s0 ^ sg), "r"(s1 ^ sg), "r"(s2 ^ sg), "r"(sg));
  // top bit to bit 95
  const bool t2 = m2 != 0, t1 = m1 != 0;
  const uint32_t a = t2 ? m2 : t1 ? m1 : m0, b = t2 ? m1 : t1 ? m0 : 0u, c = t2 ? m0 : 0u;
  const int z = __clz(a), w = t2 ? 95 : t1 ? 63 : 31;
  const uint32_t h = __funnelshift_l(b, a, z), l = __funnelshift_l(c, b, z), r = c << (z & 31);
  const int x = e + w - z;   // value in [2^x, 2^(x+1))
  // 53 bits of h:l; 11 dropped bits and the rest
  const uint32_t up = (((l & 0x7ffu) << 1) | (r ? 1u : 0u)) + ((l >> 11) & 1u) > 0x800u ? 1u : 0u;
  uint32_t ml = __funnelshift_r(l, h, 11), mh = (h >> 11) + ((uint32_t)(x + 1022) << 20);
  asm("add.cc.u32 %0, %0, %2;\n addc.u32 %1, %1, 0;" : "+r"(ml), "+r"(mh) : "r"(up));
  odd = odd || x < -1022 || x > 1022;
  const bool nz = a != 0;
  return __hiloint2double(nz ? (int)(mh | (sg & 0x80000000u)) : 0, nz ? (int)ml : 0);
}

// The same for results outside the normal range (and any other).
static __device__ __noinline__ double round_sum_any(uint32_t s0, uint32_t s1, uint32_t s2, int e) {
  bool odd = false;
  const double r = round_sum(s0, s1, s2, 0, odd);
  return scalbn(r, e);
}

}  // namespace digits
}  // namespace hps
