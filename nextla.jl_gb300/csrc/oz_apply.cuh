// oz_apply.cuh -- FP64 block-reflector apply on the tensor cores, exactly.
//
// GB300 executes two FP64 FMAs per clock and SM, on either FP64 pipe, but
// 1024 FP16 multiply-adds through mma.sync with FP32 accumulators.  The
// trailing update of apply_strip (W = A1 + V^T C, W = op(T) W, A1 -= W,
// C -= V W) is three products, so every operand is cut into seven 9-bit
// integer digits (error-free transformation in the manner of K. Ozaki,
// T. Ogita, S. Oishi, S. M. Rump, "Error-free transformations of matrix
// multiplication by using fast routines of matrix multiplication and its
// applications", Numer. Algorithms 59, 2012) and each product becomes 28 FP16
// products of digit planes, i + j <= 6.  A digit is in [-256, 255], so 32
// terms of up to 7 plane pairs sum to at most 7 * 2^21 < 2^24: every FP32
// accumulation is exact, whatever its order.
//
// Number format.  Column c of [A1; C] is held as 64-bit fixed point with its
// own power-of-two scale 2^s: s is the largest with ||column|| 2^s <= 2^60.9.
// An orthogonal update keeps that norm, |W| <= 2 ||column||, so nothing leaves
// the 62-bit range the digits cover; V (|v| < 1.99) is scaled by 2^61 and T
// (|t| < 3.99) by 2^60.  A strip that is not such an update (an infinity or NaN,
// exponents near the ends of the range, a V or T beyond those bounds, a sum
// that overflows) is detected before anything is written and the caller runs
// the DFMA path on it.  An element whose fixed-point value the update did not
// change is not written, so rows that no reflector touches keep their bits.
//
// Accuracy.  With c the column's root mean square over r rows, the unit of
// the fixed point is 2^-61 sqrt(r) c; the dropped digit products (i + j > 6)
// add about 2^2 units to W and to C, where the FP64 sums they replace round
// 256 and 32 times at 2^-53.  Against extended precision a 256-row tsmqr is
// 1.7e-16 off, normwise, with the FP64 loops 4.4e-16.
//
// That is by the column's norm (2^-58.7 of it, 256 rows); the FP64 loops round
// element i by its own size and that of sum_p |v_ip| |w_p|, which for a row
// much lighter than the others is far less.  So a group of eight columns goes
// to those loops if a row some block moved was light in all of them: neither
// the element, before or after, nor that sum at any block (by the highest
// digits: one more mma in 28) reached 2^-8.4 of the norm.  Rows of A1 take W itself; they and W are
// light below 2^-12.4 (A1 is the part above: rows lighter than those of C
// below it have no accuracy of their own to lose, which |V|^T |C| tells).
// Elements below 2^-40, but not zero, of [A1; C] or V are handed back at once.
// Root mean square row error, in roundings of the row's own size, split / FP64
// loops (k = 32, lower half of 256 rows scaled): equal rows 0.39 / 0.86, 2^-2
// 0.56 / 1.01, 2^-4 2.0 / 1.1; 2^-6 and lighter is handed back.  Cost: 8192^2
// 2.5 %.  A column that loses or gains a neighbour outside its group keeps its bits.
//
// Layout.  Warp w owns rows [32 w, 32 w + 32) of the strip in registers, as
// the accumulator fragment of (V W)^T: lane (g, t) = (lane / 4, lane % 4)
// holds columns g, g + 8 and rows 8 q + 2 t, 8 q + 2 t + 1, q = 0..3.  That
// is also the B fragment of V^T C, so C's digits go from registers to the
// tensor core without shared memory.  V's digits are warp-private too (the
// same 32 rows), one plane of 32 reflectors x 32 rows per digit in 64-byte
// rows whose 16-byte chunks are permuted by (row / 2) % 4: ldmatrix and
// ldmatrix.trans then serve both products conflict-free.  Only W crosses
// warps: 64-bit partial sums, then op(T) W on warps 0..3 (8 reflectors each),
// whose digits every warp reads as the A fragment of (V W)^T.
//
// What bounds it, per 32-reflector block of a 256-row, 16-column strip: 3584
// mma.sync (2 clk each on an SM) = 7.2 k clk, against 131 k clk of DFMAs.
#pragma once
#include "common.cuh"
#include "oz_digits.cuh"

namespace tqr {

template <typename R> struct ApplyArgs;

namespace oz {

constexpr int kCols = 16;              // strip columns
constexpr int kRowsMax = 512;          // region rows: 32 per warp, or two such chunks 256 apart
constexpr int kIbMax = 32;
constexpr int kKMax = 256;             // reflectors of a mode 1 apply (A1 rows kept until the end)
constexpr uint32_t kPlaneV = 32 * 64;  // one digit plane of 32 rows of V: 32 reflectors x 32 rows
constexpr uint32_t kWarpV = kD * kPlaneV;
constexpr uint32_t kPlaneW = 16 * 64;
constexpr int kLdWp = 36, kLdW1 = 40;
// Light or heavy (Accuracy): elements by the high word of their fixed point,
// sums of |v| |w| in units of the highest digits (2^-7, 2^54).  Rows of C:
// 2^-8.4 of the column's norm; W and A1: 2^-12.4.
constexpr uint32_t kHeavy = 3u << 18, kHeavyW = 3u << 14;
constexpr float kHeavySum = 24.0f, kHeavySumW = 1.0f;
// shared memory: V digits | T digits | W digits | W | partial W | reductions | flags | A1
constexpr size_t kOffT = 8 * (size_t)kWarpV;
constexpr size_t kOffW = kOffT + kD * (size_t)kPlaneV;
constexpr size_t kOffW1 = kOffW + (kD + 1) * (size_t)kPlaneW;   // and |W| by its highest digits
constexpr size_t kOffWp = kOffW1 + sizeof(long long) * kCols * kLdW1;
constexpr size_t kOffRed = kOffWp + sizeof(long long) * 8 * kCols * kLdWp;
constexpr size_t kOffSh = kOffRed + sizeof(uint32_t) * kCols * 9;
constexpr size_t kOffA1 = kOffSh + sizeof(uint32_t) * 32;
constexpr size_t kSmem = kOffA1 + sizeof(long long) * kCols * kKMax;
static_assert(kSmem <= TQR_SMEM_MAX, "one CTA's shared memory");

// Byte offset of 16-bit element (row, k), k even, in a plane of 64-byte rows.
__device__ __forceinline__ uint32_t plane_off(int row, int k) {
  return (uint32_t)row * 64u + (uint32_t)((((k >> 3) ^ (row >> 1)) & 3) << 4) + (uint32_t)((k & 7) * 2);
}

// Whether strip() takes a call: a property of the call, not of the strip, so
// that every driver of the same update takes the same path.  The lines are
// where the two paths cross.  One block of 32 reflectors on 16 columns costs
// strip() 23 us whatever the rows (10 us of them to bring the strip into
// fixed point and back); the DFMA loops take 64 us at 256 rows in a task graph,
// 29 us where a narrow stand-alone call spreads over one-column strips (23 at
// 192 rows, 19 at 128).  Four blocks: 45 us against 38 at 32 rows, 46 at 64,
// 101 at 256 (stand-alone, 16 columns).
__host__ __device__ inline bool covers(int mode, int L, int k, int ib) {
  return ib <= kIbMax && L <= kRowsMax && (mode == 0 || k <= kKMax) &&
         L * (ib < k ? ib : k) >= (k > ib ? 32 * 32 * 2 : 128 * 32);
}

// Rows r, r + 1 of reflectors p, p + 2, p + 4, p + 6 of a block at column i:
// the stored entries, with mode 0's unit diagonal and the zeros above it.
// whole: all of them are stored entries, 16-byte aligned.
__device__ __forceinline__ void load_v(const ApplyArgs<double> &a, const double *Vg, bool whole, int r, int p, int kb,
                                       int i, int Lr, bool tt, double (&v)[4][2]) {
  if (whole) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const double2 w = __ldcg(reinterpret_cast<const double2 *>(Vg + (size_t)(p + 2 * u) * a.ldv));
      v[u][0] = w.x; v[u][1] = w.y;
    }
  } else {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int pu = p + 2 * u;
      const int lo = a.mode == 0 ? i + pu + 1 : 0;
      const int hi = pu < kb ? (tt ? min(Lr, a.tt + i + pu + 1) : a.L) : 0;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        v[u][e] = (r + e >= lo && r + e < hi) ? __ldcg(Vg + e + (size_t)pu * a.ldv) : 0.0;
        if (a.mode == 0 && pu < kb && r + e == lo - 1) v[u][e] = 1.0;
      }
    }
  }
}

// Applies to the strip of columns [c0, c0 + nwl), nwl <= 16, over at most 256
// J rows.  reuse: V and T are those of the strip just done (0 returned, one
// block, J = 1), their digits still in place.  Returns which groups of eight
// columns (bit u: columns 8 u .. 8 u + 7) need the DFMA path; nothing of those
// has been written.  All threads get the same answer.
//
// Whatever depends on the columns' values is decided for such a group alone:
// strips are 8 or 16 columns wide and start at multiples of 8 in every driver,
// so a column's bits do not depend on the strip it is in.
template <int J>
__device__ __noinline__ int strip(const ApplyArgs<double> &a, int c0, int nwl, unsigned char *smem, bool reuse) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int L = a.L, ib = a.ib, k = a.k;
  unsigned char *const Vd = smem + (size_t)warp * kWarpV, *const Td = smem + kOffT, *const Wd = smem + kOffW;
  long long *const W1 = reinterpret_cast<long long *>(smem + kOffW1);
  long long *const Wp = reinterpret_cast<long long *>(smem + kOffWp);
  uint32_t *const red = reinterpret_cast<uint32_t *>(smem + kOffRed);   // [warp 0..7, A1][column]
  uint32_t *const shw = reinterpret_cast<uint32_t *>(smem + kOffSh);    // per warp and group: V^T C's share is scaled by 2^shw
  uint32_t *const light = shw + 16;                    // [block parity][group]: reflectors whose W is light
  uint32_t *const heavy = shw + 20;                    // [group]: those of them whose |V|^T |C| is not
  if (tid < 16) light[tid] = 0;
  long long *const A1s = reinterpret_cast<long long *>(smem + kOffA1);
  const bool tt = a.mode == 1 && a.tt >= 0;
  const int Lt = tt ? min(L, a.tt + k) : L;            // rows any reflector touches
  int bad = 0;                                         // bit u: group u
  uint32_t big[2] = {0, 0}, vout = 0;                  // vout: top bit set by a V or T out of range

  // ---- the strip, and A1's rows, from global memory ----
  double *const Cg = a.C + (size_t)c0 * a.c_cs;
  const bool vec = a.c_rs == 1 && ((uintptr_t)Cg & 15) == 0 && (a.c_cs & 1) == 0;
  // this lane's elements of a chunk: 16-byte loads, all in flight, where the
  // warp's 32 x 16 block is whole and aligned
  auto load_c = [&](int ch, double (&x)[2][4][2]) {
    const int r0 = 256 * ch + 32 * warp;
    if (vec && nwl == kCols && r0 + 32 <= Lt) {
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const double2 v = __ldcg(reinterpret_cast<const double2 *>(Cg + r0 + 8 * q + 2 * t + (size_t)(g + 8 * u) * a.c_cs));
          x[u][q][0] = v.x; x[u][q][1] = v.y;
        }
    } else {
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int c = g + 8 * u, r = r0 + 8 * q + 2 * t + e;
            x[u][q][e] = (c < nwl && r < Lt) ? __ldcg(Cg + (size_t)r * a.c_rs + (size_t)c * a.c_cs) : 0.0;
          }
    }
  };
  double x[J][2][4][2];
#pragma unroll
  for (int ch = 0; ch < J; ++ch) load_c(ch, x[ch]);
  // high word of |v|, nonzero for every nonzero v
  auto mag = [](double v) {
    return ((uint32_t)__double2hiint(v) & 0x7fffffffu) | (__double2loint(v) != 0 ? 1u : 0u);
  };
  const int ca = tid >> 4, la = tid & 15;              // A1: 16 threads a column
  double *const A1g = a.mode == 1 ? a.A1 + (size_t)(c0 + ca) * a.a_cs : nullptr;
  const int ka = a.mode == 1 && ca < nwl ? k : 0;
  double *const A1c = reinterpret_cast<double *>(A1s) + ca * kKMax;
  uint32_t m0 = 0, m1 = 0, ma = 0, l0 = ~0u, l1 = ~0u, lo = ~0u;   // largest; smallest but zero, less one, in this lane
#pragma unroll 8
  for (int r = la; r < ka; r += 16) {
    const double v = __ldcg(A1g + (size_t)r * a.a_rs);
    A1c[r] = v;
    ma = max(ma, mag(v));
    lo = min(lo, mag(v) - 1u);
  }
  // ---- column scales: largest exponent, then the norm ----
#pragma unroll
  for (int ch = 0; ch < J; ++ch)
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        m0 = max(m0, mag(x[ch][0][q][e]));
        m1 = max(m1, mag(x[ch][1][q][e]));
        l0 = min(l0, mag(x[ch][0][q][e]) - 1u);
        l1 = min(l1, mag(x[ch][1][q][e]) - 1u);
      }
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1) {
    m0 = max(m0, __shfl_xor_sync(0xffffffffu, m0, o));
    m1 = max(m1, __shfl_xor_sync(0xffffffffu, m1, o));
  }
#pragma unroll
  for (int o = 1; o <= 8; o <<= 1) ma = max(ma, __shfl_xor_sync(0xffffffffu, ma, o));
  if (t == 0) {
    red[warp * kCols + g] = m0;
    red[warp * kCols + g + 8] = m1;
  }
  if (la == 0) red[8 * kCols + ca] = ma;
  __syncthreads();
  auto col_exp = [&](int c) {
    uint32_t m = 0;
#pragma unroll
    for (int w = 0; w < 9; ++w) m = max(m, red[w * kCols + c]);
    const int e = m ? (int)(m >> 20) : 1023;           // any scale will do for a column of zeros
    bad |= ((m != 0) & ((e > 1900) | (e < 140))) << (c >> 3);   // far from the ends of the range only
    return e;
  };
  const int e0 = col_exp(g), e1 = col_exp(g + 8), ea = col_exp(ca);
  // |x| 2^(1022 - emax) < 1 as a float; tiny values go to zero
  auto rel = [](double v, int emax) {
    const int h = (int)((uint32_t)__double2hiint(v) & 0x7fffffffu) - ((emax - 126) << 20);
    return __int_as_float(max(h, 0) << 3);
  };
  float n0 = 0.0f, n1 = 0.0f, na = 0.0f;
#pragma unroll
  for (int ch = 0; ch < J; ++ch)
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float f0 = rel(x[ch][0][q][e], e0), f1 = rel(x[ch][1][q][e], e1);
        n0 = fmaf(f0, f0, n0);
        n1 = fmaf(f1, f1, n1);
      }
#pragma unroll 4
  for (int r = la; r < ka; r += 16) {
    const float f = rel(A1c[r], ea);
    na = fmaf(f, f, na);
  }
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1) {
    n0 += __shfl_xor_sync(0xffffffffu, n0, o);
    n1 += __shfl_xor_sync(0xffffffffu, n1, o);
  }
#pragma unroll
  for (int o = 1; o <= 8; o <<= 1) na += __shfl_xor_sync(0xffffffffu, na, o);
  __syncthreads();
  if (t == 0) {
    red[warp * kCols + g] = __float_as_uint(n0);
    red[warp * kCols + g + 8] = __float_as_uint(n1);
  }
  if (la == 0) red[8 * kCols + ca] = __float_as_uint(na);
  __syncthreads();
  // largest s with norm 2^s <= 2^60.9: norm^2 <= 3.48 * 4^h, s = 60 - h + 1022 - emax
  auto col_scale = [&](int c, int emax) {
    float n = 0.0f;
#pragma unroll
    for (int w = 0; w < 9; ++w) n += __uint_as_float(red[w * kCols + c]);
    const int ex = ((__float_as_int(n * (1.0f / 3.48f)) >> 23) & 0xff) - 127;   // floor(log2)
    return 60 - ((ex + 2) >> 1) + 1022 - emax;
  };
  const int s0 = col_scale(g, e0), s1 = col_scale(g + 8, e1), sa = col_scale(ca, ea);
  long long X[J][2][4][2];                             // biased by kBias
  uint32_t row[J];                                     // bit 8 u + 2 q + e: heavy element; + 16: element some block moved
  auto high = [](long long v) { return (uint32_t)abs((int)(uint32_t)(v >> 32)); };
  // high word of an FP64 magnitude of 1.5 * 2^e in fixed point
  auto level = [](int e, int s) { return ((uint32_t)(1023 + e - s) << 20) + 0x80000u; };
  // elements below 2^-40 of the norm, but not zero
  bad |= (int)(l0 < level(20, s0)) | (int)(l1 < level(20, s1)) << 1 | (int)(lo < level(20, sa)) << (ca >> 3);
  const uint32_t t0 = level(51, s0), t1 = level(51, s1);        // kHeavy
#pragma unroll
  for (int ch = 0; ch < J; ++ch) {
    row[ch] = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (mag(x[ch][u][q][e]) >= (u ? t1 : t0)) row[ch] |= 1u << (8 * u + 2 * q + e);
          X[ch][u][q][e] = to_fixed<true>(x[ch][u][q][e], u ? s1 : s0) + (long long)kBias;
        }
  }
#pragma unroll 2
  for (int r = la; r < ka; r += 16) A1s[ca * kKMax + r] = to_fixed<true>(A1c[r], sa);

  const int nblk = (k + ib - 1) / ib;
  const uint32_t vbase = saddr(Vd), wbase = saddr(Wd), tbase = saddr(Td);
  for (int b = 0; b < nblk; ++b) {
    const int i = a.fwd ? b * ib : (nblk - 1 - b) * ib;
    const int kb = min(ib, k - i);
    const int r0 = a.mode == 0 ? i : 0;
    const int Lr = tt ? min(L, a.tt + i + kb) : L;      // rows this block touches: [r0, Lr)
    const bool two = kb > 16;                           // second half of the 32 reflectors in use
    // whether this warp's chunk ch holds rows the block touches
    auto active = [&](int ch, int w) { return 256 * ch + 32 * w < Lr && 256 * ch + 32 * w + 32 > r0; };
    double tv[2][2];                                    // op(T)'s entries, loaded ahead of V's digits
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const int idx = tid + w * TQR_THREADS, p = idx >> 4, q = 2 * (idx & 15);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        // W2[p] = sum_q op(T)[p, q] W1[q]; op(T) = T^T reads T[q, p]
        const int row = a.transT ? q + e : p, col = a.transT ? p : q + e;
        tv[w][e] = (!reuse && row <= col && col < kb) ? __ldcg(a.T + ix(row, i + col, a.ldt)) : 0.0;
      }
    }
    // digits of 32 rows of V (chunk ch), four pairs of reflectors at a time
    auto v_chunk = [&](int ch) {
      const int rw = 256 * ch + 32 * warp, r = rw + 2 * (lane & 15);
      const double *const Vg = a.V + ix(r, i, a.ldv);
      const int np = two ? 32 : 16;                    // reflectors to fill
      const bool wholev = ((uintptr_t)Vg & 15) == 0 && (a.ldv & 1) == 0 && kb == np && rw + 32 <= Lr &&
                          (a.mode == 0 ? rw >= i + kb : !tt || rw + 32 <= a.tt + i + 1);
      constexpr int kStep = 8;                         // reflectors of a pass
      int p = lane >> 4;
      uint32_t least = ~0u;
      double v[4][2], n[4][2];
      load_v(a, Vg, wholev, r, p, kb, i, Lr, tt, v);
#pragma unroll 1
      for (; p < np; p += kStep) {
        if (p + kStep < np) load_v(a, Vg, wholev, r, p + kStep, kb, i, Lr, tt, n);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const unsigned long long y0 = to_biased<61>(v[u][0], vout);
          const unsigned long long y1 = to_biased<61>(v[u][1], vout);
          least = min(least, ((uint32_t)__double2hiint(v[u][0]) & 0x7fffffffu) - 1u);
          least = min(least, ((uint32_t)__double2hiint(v[u][1]) & 0x7fffffffu) - 1u);
          const uint32_t off = plane_off(p + 2 * u, 2 * (lane & 15));
          digits(y0, y1, [&](int d, uint32_t w) { *reinterpret_cast<uint32_t *>(Vd + d * kPlaneV + off) = w; });
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) { v[u][0] = n[u][0]; v[u][1] = n[u][1]; }
      }
      if (least < (1023u - 40u) << 20) vout |= 0x80000000u;       // an entry of V below 2^-40, but not zero
      __syncwarp();
    };
    if (!reuse && active(0, warp)) v_chunk(0);
    // ---- digits of op(T), pairs (q, q + 1) of one row p ----
    if (!reuse) {
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const int idx = tid + w * TQR_THREADS, p = idx >> 4, q = 2 * (idx & 15);
        const unsigned long long y0 = to_biased<60>(tv[w][0], vout);
        const unsigned long long y1 = to_biased<60>(tv[w][1], vout);
        const uint32_t off = plane_off(p, q);
        digits(y0, y1, [&](int d, uint32_t z) { *reinterpret_cast<uint32_t *>(Td + d * kPlaneV + off) = z; });
      }
    }
    // ---- this warp's share of V^T C, 16 reflectors x 8 columns at a time ----
    // a column's norm leaves its elements a few bits below the digits' range:
    // 4 C instead of C where no element of the warp and group reaches 2^59
    uint32_t mul[2];
    unsigned long long off4[2];                         // biased values: 4 (y - bias) + bias
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      uint32_t far = 0;
#pragma unroll
      for (int ch = 0; ch < J; ++ch)
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int e = 0; e < 2; ++e) far |= (uint32_t)(X[ch][u][q][e] >> 32) - (uint32_t)(kBias >> 32) + 0x08000000u;
      const bool up = __all_sync(0xffffffffu, far < 0x10000000u);
      mul[u] = up ? 4u : 1u;
      off4[u] = up ? 0ull - 3ull * kBias : 0ull;
      if (lane == 0) shw[2 * warp + u] = up ? 2u : 0u;
    }
    bool any = false;                                   // this warp's share has been started
#pragma unroll
    for (int ch = 0; ch < J; ++ch) {
      if (!active(ch, warp)) continue;
      if (ch > 0) v_chunk(ch);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        uint32_t cd[kD][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          unsigned long long y[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const unsigned long long v = (unsigned long long)X[ch][u][q][e];
            y[e] = (unsigned long long)(uint32_t)v * mul[u] + off4[u] + ((unsigned long long)((uint32_t)(v >> 32) * mul[u]) << 32);
          }
          digits(y[0], y[1], [&](int d, uint32_t w) { cd[d][q] = w; });
        }
#pragma unroll 1
        for (int mt = 0; mt < (two ? 2 : 1); ++mt) {
          float acc[kD][4];
          init_acc(acc);
          const int p = 16 * mt + (lane & 15);
#pragma unroll
          for (int d = 0; d < kD; ++d)
#pragma unroll
            for (int kt = 0; kt < 2; ++kt) {
              uint32_t av[4];
              ldsm4(vbase + d * kPlaneV + plane_off(p, 16 * kt + 8 * (lane >> 4)), av);
#pragma unroll
              for (int j = 0; j < kD - d; ++j)
                mma(acc[d + j], av[0], av[1], av[2], av[3], cd[j][2 * kt], cd[j][2 * kt + 1]);
            }
          long long *wp = Wp + ((size_t)warp * kCols + 8 * u + 2 * t) * kLdWp + 16 * mt + g;
          const long long z0 = recon<47>(acc, 0, big[u]), z1 = recon<47>(acc, 1, big[u]);
          const long long z2 = recon<47>(acc, 2, big[u]), z3 = recon<47>(acc, 3, big[u]);
          if (J == 1 || !any) {
            wp[0] = z0; wp[kLdWp] = z1; wp[8] = z2; wp[kLdWp + 8] = z3;
          } else {
            // two shares below 1.25 * 2^62 each: the sum's range is checked on the halves
            bad |= (int)(((uint64_t)((wp[0] >> 1) + (z0 >> 1) + (1ll << 62)) | (uint64_t)((wp[kLdWp] >> 1) + (z1 >> 1) + (1ll << 62)) |
                          (uint64_t)((wp[8] >> 1) + (z2 >> 1) + (1ll << 62)) | (uint64_t)((wp[kLdWp + 8] >> 1) + (z3 >> 1) + (1ll << 62))) >> 63) << u;
            wp[0] += z0; wp[kLdWp] += z1; wp[8] += z2; wp[kLdWp + 8] += z3;
          }
        }
      }
      any = true;
    }
    __syncthreads();
    // ---- W1 = A1 rows + the warps' shares ----
    if (tid < 2) {
      light[2 * ((b + 1) & 1) + tid] = 0;               // last read in the block before
      heavy[tid] = 0;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int q = tid & 31, c = (tid >> 5) + 8 * u;
      long long w = 0;
      if (q < kb) {
        int top = 0;
        if (a.mode == 1 && c < nwl) {
          w = A1s[c * kKMax + i + q];
          top = (int)(w >> 36);
        }
        const int wlo = J == 1 ? r0 >> 5 : 0, whi = J == 1 ? (Lr + 31) >> 5 : 8;
        for (int ww = wlo; ww < whi; ++ww) {
          if (J > 1 && !active(0, ww) && !active(1, ww)) continue;
          const uint32_t sh = shw[2 * ww + u];
          const long long v = (Wp[((size_t)ww * kCols + c) * kLdWp + q] + (long long)sh) >> sh;   // rounded
          w += v;
          top += (int)(v >> 36);
        }
        bad |= ((top > (1 << 26) - (1 << 18)) | (top < -(1 << 26) + (1 << 18))) << u;   // |w| < 0.996 * 2^62
      }
      W1[c * kLdW1 + q] = w + (long long)kBias;
    }
    __syncthreads();
    // ---- W2 = op(T) W1 (8 reflectors a warp), A1 -= W2, W2's digits ----
    if (warp < (two ? 4 : 2)) {
      float acc[kD][4];
      init_acc(acc);
#pragma unroll 1
      for (int kt = 0; kt < (two ? 2 : 1); ++kt) {
        uint32_t wa[kD][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const longlong2 v = *reinterpret_cast<const longlong2 *>(W1 + (g + 8 * (e & 1)) * kLdW1 + 16 * kt + 8 * (e >> 1) + 2 * t);
          digits((unsigned long long)v.x, (unsigned long long)v.y, [&](int d, uint32_t w) { wa[d][e] = w; });
        }
#pragma unroll
        for (int d = 0; d < kD; ++d) {
          uint32_t bt[2];
          ldsm2(tbase + d * kPlaneV + plane_off(8 * warp + (lane & 7), 16 * kt + 8 * ((lane >> 3) & 1)), bt);
#pragma unroll
          for (int j = 0; j < kD - d; ++j) mma(acc[d + j], wa[j][0], wa[j][1], wa[j][2], wa[j][3], bt[0], bt[1]);
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int c = g + 8 * u, p = 8 * warp + 2 * t;
        const long long w0 = recon<48>(acc, 2 * u, big[u]), w1 = recon<48>(acc, 2 * u + 1, big[u]);
        const longlong2 wv = *reinterpret_cast<const longlong2 *>(W1 + c * kLdW1 + p);
        uint32_t hn = 0;                                // bits 0, 1: W before or after T or A1's row heavy; 2, 3: not zero
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const long long v = (e ? wv.y : wv.x) - (long long)kBias, w2 = e ? w1 : w0;
          hn |= (uint32_t)(max(high(v), high(w2)) >= kHeavyW) << e | (uint32_t)(v != 0 || w2 != 0) << (e + 2);
        }
        if (a.mode == 1 && c < nwl) {
          long long *ap = A1s + c * kKMax + i + p;
          if (p < kb) {
            hn |= (uint32_t)(high(ap[0]) >= kHeavyW);
            ap[0] -= w0;
          }
          if (p + 1 < kb) {
            hn |= (uint32_t)(high(ap[1]) >= kHeavyW) << 1;
            ap[1] -= w1;
          }
        }
#pragma unroll
        for (int o = 4; o <= 16; o <<= 1) hn |= __shfl_xor_sync(0xffffffffu, hn, o);
        const uint32_t l = (hn >> 2) & ~hn & 3u;
        if (g == 0 && l) atomicOr(&light[2 * (b & 1) + u], l << p);
        const uint32_t off = plane_off(c, p);
        const unsigned long long y0 = (unsigned long long)w0 + kBias, y1 = (unsigned long long)w1 + kBias;
        bad |= (int)((uint32_t)((y0 | y1) >> 32) >> 31) << u;         // outside the digits' range
        digits(y0, y1, [&](int d, uint32_t w) {
          *reinterpret_cast<uint32_t *>(Wd + d * kPlaneW + off) = w;
          if (d == 0) *reinterpret_cast<uint32_t *>(Wd + kD * kPlaneW + off) = magnitude(w);
        });
      }
    }
    __syncthreads();
    // ---- light W: handed back unless |V|^T |C| over some warp's 32 rows (of the chunk whose digits are in place)
    // is heavy, which the FP64 loops would have rounded it by ----
    const uint32_t lw[2] = {light[2 * (b & 1)], light[2 * (b & 1) + 1]};
    if (lw[0] | lw[1]) {
      const int ch = J > 1 && active(J - 1, warp) ? J - 1 : 0;
      if (active(ch, warp)) {
#pragma unroll 1
        for (int um = 0; um < 4; ++um) {
          const int u = um >> 1, p = 16 * (um & 1) + (lane & 15);
          float am[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
          for (int kt = 0; kt < 2; ++kt) {
            uint32_t av[4], cm[2];
            ldsm4(vbase + plane_off(p, 16 * kt + 8 * (lane >> 4)), av);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              unsigned long long y[2];
#pragma unroll
              for (int e = 0; e < 2; ++e)
                y[e] = (unsigned long long)(J > 1 && ch ? (u ? X[J - 1][1][2 * kt + q][e] : X[J - 1][0][2 * kt + q][e])
                                                        : (u ? X[0][1][2 * kt + q][e] : X[0][0][2 * kt + q][e]));
              cm[q] = magnitude(digit<6>(y[0], y[1]));
            }
            mma(am, magnitude(av[0]), magnitude(av[1]), magnitude(av[2]), magnitude(av[3]), cm[0], cm[1]);
          }
          uint32_t h0 = __ballot_sync(0xffffffffu, fmaxf(am[0], am[1]) >= kHeavySumW);
          uint32_t h1 = __ballot_sync(0xffffffffu, fmaxf(am[2], am[3]) >= kHeavySumW);
          uint32_t m = 0;                               // a reflector's four lanes hold two columns each
#pragma unroll
          for (int r = 0; r < 8; ++r) m |= (uint32_t)((h0 >> (4 * r) & 15u) != 0) << r | (uint32_t)((h1 >> (4 * r) & 15u) != 0) << (r + 8);
          if (lane == 0 && m) atomicOr(&heavy[u], m << (16 * (um & 1)));
        }
      }
      __syncthreads();
      bad |= (int)((lw[0] & ~heavy[0]) != 0) | (int)((lw[1] & ~heavy[1]) != 0) << 1;
    }
    // ---- C -= V W2 on this warp's rows, 8 rows at a time; the last chunk's digits of V are in place ----
#pragma unroll
    for (int cj = 0; cj < J; ++cj) {
      const int ch = J - 1 - cj;
      if (!active(ch, warp)) continue;
      if (J > 1 && cj > 0 && active(J - 1, warp)) v_chunk(ch);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float acc[kD][4], am[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        init_acc(acc);
#pragma unroll 1
        for (int kt = 0; kt < (two ? 2 : 1); ++kt) {
          uint32_t wa[kD][4], wm[4];
          ldsm4(wbase + kD * kPlaneW + plane_off(lane & 15, 16 * kt + 8 * (lane >> 4)), wm);
#pragma unroll
          for (int d = 0; d < kD; ++d) ldsm4(wbase + d * kPlaneW + plane_off(lane & 15, 16 * kt + 8 * (lane >> 4)), wa[d]);
#pragma unroll
          for (int d = 0; d < kD; ++d) {
            uint32_t bv[2];
            ldsm2t(vbase + d * kPlaneV + plane_off(16 * kt + (lane & 15), 8 * q), bv);
#pragma unroll
            for (int j = 0; j < kD - d; ++j) mma(acc[d + j], wa[j][0], wa[j][1], wa[j][2], wa[j][3], bv[0], bv[1]);
            if (d == 0) mma(am, wm[0], wm[1], wm[2], wm[3], magnitude(bv[0]), magnitude(bv[1]));
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const long long dx = recon<47>(acc, 2 * u + e, big[u]);
            if (dx != 0) row[ch] |= 1u << (16 + 8 * u + 2 * q + e);
            if (am[2 * u + e] >= kHeavySum) row[ch] |= 1u << (8 * u + 2 * q + e);
            X[ch][u][q][e] -= dx;
            bad |= (int)((uint32_t)(X[ch][u][q][e] >> 32) >> 31) << u;   // left the biased range
          }
      }
      __syncwarp();
    }
  }
  bad |= (int)((big[0] & kBig) != 0) | (int)((big[1] & kBig) != 0) << 1 | (vout >> 31 ? 3 : 0);
  // rows that moved and were light throughout, in all of the group's columns
#pragma unroll
  for (int ch = 0; ch < J; ++ch) {
    uint32_t r = row[ch];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (high(X[ch][u][q][e] - (long long)kBias) >= kHeavy) r |= 1u << (8 * u + 2 * q + e);
#pragma unroll
    for (int o = 4; o <= 16; o <<= 1) r |= __shfl_xor_sync(0xffffffffu, r, o);
    r = r >> 16 & ~r;
    bad |= (int)((r & 0xffu) != 0) | (int)((r & 0xff00u) != 0) << 1;
  }
  const int all = nwl > 8 ? 3 : 1;                      // the strip's groups
  const int fail = ((__syncthreads_or(bad & 1) ? 1 : 0) | (__syncthreads_or(bad & 2) ? 2 : 0)) & all;
  if (fail == all) return fail;

  // ---- back to FP64: the elements whose value changed ----
#pragma unroll
  for (int ch = 0; ch < J; ++ch) {
    if (J > 1) load_c(ch, x[ch]);
    const int rw = 256 * ch + 32 * warp;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = g + 8 * u, r = rw + 8 * q + 2 * t, s = u ? s1 : s0;
        double *p = Cg + (size_t)r * a.c_rs + (size_t)c * a.c_cs;
        double y[2];
        bool moved[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const long long v = X[ch][u][q][e] - (long long)kBias;
          moved[e] = c < nwl && r + e < Lt && !((fail >> u) & 1) &&
                     (J == 1 ? ((row[ch] >> (16 + 8 * u + 2 * q + e)) & 1u) != 0 : v != to_fixed<true>(x[ch][u][q][e], s));
          y[e] = from_fixed(v, s);
        }
        if (vec && moved[0] && moved[1]) {
          *reinterpret_cast<double2 *>(p) = make_double2(y[0], y[1]);
        } else {
          if (moved[0]) p[0] = y[0];
          if (moved[1]) p[a.c_rs] = y[1];
        }
      }
  }
#pragma unroll 8
  for (int r = la; r < ((fail >> (ca >> 3)) & 1 ? 0 : ka); r += 16) {
    double *pe = A1g + (size_t)r * a.a_rs;
    const double o = __ldcg(pe);
    const long long v = A1s[ca * kKMax + r];
    if (v != to_fixed<true>(o, sa)) *pe = from_fixed(v, sa);
  }
  __syncthreads();
  return fail;
}

}  // namespace oz
}  // namespace tqr
