// oz_digits.cuh -- FP64 values as 64-bit fixed point, cut into FP16 digits for
// exact tensor-core products (the number format of oz_apply.cuh).
#pragma once
#include "common.cuh"

namespace tqr {
namespace oz {

constexpr int kD = 7;                  // digits
// 256 in every digit: x + kBias has the digits of x plus 256, without carries
constexpr unsigned long long kBias = 0x4020100804020100ull;
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: an integer |i| <= 2^22 is in the low bits of kMagic + i

__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                    uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

__device__ __forceinline__ void ldsm2(uint32_t addr, uint32_t (&r)[2]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm2t(uint32_t addr, uint32_t (&r)[2]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr) : "memory");
}

// x 2^s as an integer, rounded to nearest (RND) or towards zero; the caller
// sees to |x| 2^s < 2^62 (larger and non-finite values give garbage).
template <bool RND>
__device__ __forceinline__ long long to_fixed(double x, int s) {
  const uint32_t hi = __double2hiint(x), lo = __double2loint(x);
  unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 10;
  const int t = (1085 - s) - (int)((hi >> 20) & 0x7ff);   // m 2^-t is |x| 2^s; zeros and subnormals shift out
  if (RND) {
    // shr clamps the shift count, so a long shift gives zero
    asm("shr.u64 %0, %1, %2;" : "=l"(m) : "l"(m), "r"(t - 1));
    m = (m + 1) >> 1;
  } else {
    asm("shr.u64 %0, %1, %2;" : "=l"(m) : "l"(m), "r"(t));
  }
  const long long sg = (long long)((int)hi >> 31);
  return ((long long)m ^ sg) - sg;
}
// x 2^S biased by kBias, towards zero; out's top bit is set if some x was out
// of the digits' range (0.998 * 2^62 and up, infinities, NaN).
template <int S>
__device__ __forceinline__ unsigned long long to_biased(double x, uint32_t &out) {
  const uint32_t hi = __double2hiint(x), lo = __double2loint(x);
  const unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 10;
  const int t = (1085 - S) - (int)((hi & 0x7fffffffu) >> 20);
  const unsigned long long r = m >> min(max(t, 0), 63);  // 63 leaves nothing
  const uint32_t sg = (uint32_t)((int)hi >> 31);
  const unsigned long long y = (r ^ ((unsigned long long)sg << 32 | sg)) + ((kBias & 0xffffffff00000000ull) | ((uint32_t)kBias - sg));
  out |= (uint32_t)(y >> 32) | (uint32_t)t;              // t < 0: 2^63 and up
  return y;
}

// v 2^-s rounded to nearest even, |v| < 2^63, the result normal.  On the bits:
// a conversion instruction would take its warp 64 clocks.
__device__ __forceinline__ double from_fixed(long long v, int s) {
  const unsigned long long sg = (unsigned long long)(v >> 63), a = ((unsigned long long)v ^ sg) - sg;
  const int lz = __clzll((long long)a);
  const unsigned long long m = a << lz;                  // leading bit at 63
  const uint32_t rem = (uint32_t)m & 0x7ffu;
  unsigned long long q = m >> 11;
  q += rem + ((uint32_t)q & 1u) > 0x400u ? 1u : 0u;
  q += (unsigned long long)(unsigned int)(1023 + 62 - lz - s) << 52;   // q's bit 52 adds one to the exponent
  const uint32_t hi = (uint32_t)(q >> 32) | ((uint32_t)sg & 0x80000000u);
  return a == 0 ? 0.0 : __hiloint2double((int)hi, (int)(uint32_t)q);
}

// Digit J (0 = lowest) of two biased fixed-point values as an f16 pair.
template <int J>
__device__ __forceinline__ uint32_t digit(unsigned long long a, unsigned long long b) {
  const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32), bl = (uint32_t)b, bh = (uint32_t)(b >> 32);
  uint32_t w;
  // bytes J, J + 1 of each value hold the digit at bit J
  if (J == 0) w = __byte_perm(al, bl, 0x5410);
  if (J == 1) w = __byte_perm(al, bl, 0x6521) >> 1;
  if (J == 2) w = __byte_perm(al, bl, 0x7632) >> 2;
  if (J == 3) w = __byte_perm(__funnelshift_r(al, ah, 27), __funnelshift_r(bl, bh, 27), 0x5410);
  if (J == 4) w = __byte_perm(ah, bh, 0x5410) >> 4;
  if (J == 5) w = __byte_perm(ah, bh, 0x6521) >> 5;
  if (J == 6) w = __byte_perm(ah, bh, 0x7632) >> 6;
  w = (w & 0x01ff01ffu) | 0x64006400u;                // 1024 + digit + 256 in f16
  uint32_t r;
  asm("sub.f16x2 %0, %1, %2;" : "=r"(r) : "r"(w), "r"(0x65006500u));   // - 1280
  return r;
}

// |digit| of a pair of digits, -1 and 0 both zero: the highest digits of a
// number then give its magnitude, rounded down.
__device__ __forceinline__ uint32_t magnitude(uint32_t d) {
  uint32_t r;
  asm("add.f16x2 %0, %1, %2;" : "=r"(r) : "r"(d), "r"(0x38003800u));            // + 1/2
  r &= 0x7fff7fffu;
  asm("sub.f16x2 %0, %0, %1;" : "+r"(r) : "r"(0x38003800u));
  return r;
}

// The seven digits of a pair, highest first, through put(plane, word).
template <typename F>
__device__ __forceinline__ void digits(unsigned long long a, unsigned long long b, F &&put) {
  put(0, digit<6>(a, b));
  put(1, digit<5>(a, b));
  put(2, digit<4>(a, b));
  put(3, digit<3>(a, b));
  put(4, digit<2>(a, b));
  put(5, digit<1>(a, b));
  put(6, digit<0>(a, b));
}

template <typename F>
__device__ __forceinline__ void init_acc(F (&acc)[kD][4]) {
#pragma unroll
  for (int d = 0; d < kD; ++d)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[d][e] = d < 2 ? kMagic : 0.0f;
}

// sum_d acc[d][e] 2^(SH - 9 d), rounded once below the unit.  Diagonals 0 and
// 1 (|sum| <= 2^22) were accumulated on top of kMagic, so their integers are
// the low bits.  big collects acc[0] + 2^(62 - SH): while that stays in
// [0, 2^(63 - SH)) the value is below 2^63 in magnitude (the other diagonals
// add less than 2^62).
template <int SH>
__device__ __forceinline__ long long recon(const float (&acc)[kD][4], int e, uint32_t &big) {
  const int r0 = __float_as_int(acc[0][e]), r1 = __float_as_int(acc[1][e]);
  const int i2 = __float2int_rn(acc[2][e]), i3 = __float2int_rn(acc[3][e]), i4 = __float2int_rn(acc[4][e]);
  const int i5 = __float2int_rn(fmaf(acc[5][e], (float)(1 << (SH - 45)), acc[6][e] * (1.0f / (float)(1 << (54 - SH)))));
  constexpr uint32_t base = 0u - (0x4B400000u << (SH - 32)) - (0x4B400000u << (SH - 41));
  long long r = (long long)i5;
  r += (long long)i4 * (1ll << (SH - 36));
  r += (long long)i3 * (1ll << (SH - 27));
  r += (long long)i2 * (1ll << (SH - 18));
  const uint32_t hi = (uint32_t)r0 * (1u << (SH - 32)) + ((uint32_t)r1 * (1u << (SH - 41)) + base);
  big |= ((uint32_t)r0 - (0x4B400000u - (1u << (62 - SH)))) << (SH - 47);
  return r + (long long)((unsigned long long)hi << 32);
}
constexpr uint32_t kBig = 0xffff0000u;   // bits of big that mean an overflow


}  // namespace oz
}  // namespace tqr
