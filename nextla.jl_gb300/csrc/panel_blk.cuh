// panel_blk.cuh -- the column loop of a staged FP64 panel, eight columns at a
// time, with the rest of the block updated on the tensor cores.
//
// A column step of an ib = 32 panel spent 31 dot products and up to 31 column
// updates of 256 rows on the FP64 pipe (16 clocks of an SM per warp
// instruction): 14 k clocks a column.  Here a column meets only the columns of its own
// sub-block of eight; after eight columns their block reflector is applied
// to the columns right of them by two exact split products (oz_digits.cuh),
// and the Gram blocks V_a^T V_b that T needs are one more such product at the
// end.  Columns right of the sub-block are held in fixed point, in place,
// with the scale of their norm, which the reflectors preserve.
//
// Per column two block barriers: (1) S_j = x^T P_j for the sub-block's eight
// columns at once, the column's own norm among them (thread = column lane %
// 8, eight rows; two shuffles; eight warps' partials); (2) warp 0 forms the
// Householder scalars and d_j = -tau (row_j + scale S_j).  Then each thread
// scales and updates its own rows, which are its warp's rows of the next dot
// products.  While warp 0 is in the scalars (a square root and two divisions,
// the longest chain of a column), warp 1 forms the previous column of the
// sub-block's T.  With reflectors rounded to FP32 (round32) the dot products
// follow the rounding, a second round of barriers.
//
// Same result as columns_la_f64 up to rounding; the caller falls back to it
// (false is returned before anything is written) when a column's exponents are
// outside the fixed-point range, or a row is light: none of its elements
// reaches 2^-8 of its column's norm.  The FP64 loops round a row by its own
// size; the fixed point does by the column's, 2.5e-18 of it (256 rows), which
// for rows of 2^-8 is 2.2 times as much and grows as they get lighter (a row
// 2^-12 below forty others: 173 roundings of its own size against 2.2).  With
// reflectors rounded to FP32 the line is 2^-30.  Elements whose fixed point
// did not change keep their bits.
#pragma once
#include <new>

#include "common.cuh"
#include "oz_digits.cuh"

namespace tqr {

namespace blk {
constexpr int kW = 8;                                   // columns of a sub-block
constexpr int kMaxRows = 512;
// scratch: warp partials | sums and scalars | T and Gram of a sub-block | column
// scales | W digits | W | partial products (8 warps x 384)
constexpr size_t kPart = 0;                             // 64 doubles
constexpr size_t kSum = kPart + 64 * 8;                 // d[8], scal[4], tau[32]
constexpr size_t kT8 = kSum + 48 * 8;                   // 4 x 64
constexpr size_t kG8 = kT8 + 4 * 64 * 8;                // 64
constexpr size_t kScale = kG8 + 64 * 8;                 // 32 ints
constexpr size_t kWd = kScale + 32 * 4;                 // kD planes x 32 columns x 8 halves
constexpr size_t kW1 = kWd + oz::kD * 512;              // 32 x 8 doubles
constexpr size_t kWp = kW1 + 32 * 8 * 8;                // 8 x 384 int64 (then G, Y: 2 x 384 doubles)
constexpr size_t kOrig = kWp + 8 * 384 * 8;             // the caller's Orig, out of the registers' way
constexpr size_t kScratch = kOrig + 64;

// Panels the blocked loop takes; a property of the panel alone, so every
// driver of the same factorisation takes the same path.
__host__ __device__ inline bool covers(int m, int nc) { return m >= 64 && m <= kMaxRows && nc > kW && nc <= 32; }

__device__ __forceinline__ void mma8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(b0));
}

// V entry (row r, reflector of column col) as biased fixed point: the stored
// value, for geqr2 with the unit diagonal and zeros above it.
template <int FORM>
__device__ __forceinline__ unsigned long long v_fixed(const double *P, int ldp, int r, int col, int m, int kcol) {
  double v = (r < m && col < kcol) ? P[(size_t)col * ldp + r] : 0.0;
  if (FORM == 0 && col < kcol) v = r < col ? 0.0 : (r == col ? 1.0 : v);
  uint32_t out = 0;                                     // |v| <= 1
  return oz::to_biased<61>(v, out);
}

// householder() (common.cuh) with the square root and the two divisions as
// series from FP32 seeds: with y0 ~ v^(-1/2) and r = 1 - v y0^2, v^(-1/2) =
// y0 (1 - r)^(-1/2) = y0 (1 + r/2 + 3 r^2/8 + ...); with z0 ~ 1/d and q = 1 -
// d z0, 1/d = z0 (1 + q + q^2 + ...).  Seeds are good to 2^-22, so the first
// terms left out are below 2^-66.  Every FP64 instruction, a comparison or a
// conversion too, takes its warp 64 clocks whatever depends on it, so what can
// be done on the bits is: 13 of them here, 25 with the library's operations.
// The exponent arithmetic is for normal v with room on both sides; a column
// whose v is outside 2^-959 .. 2^941 (subnormal, infinite and NaN included)
// goes through householder() itself.  All lanes of the warp have the same one.
__device__ __forceinline__ bool is_zero(double v) {
  return ((__double2hiint(v) & 0x7fffffff) | __double2loint(v)) == 0;
}
__device__ __forceinline__ float to_float_12(double f) {      // f in [1, 4), truncated
  const uint32_t hi = __double2hiint(f), lo = __double2loint(f);
  return __uint_as_float((((hi << 3) | (lo >> 29)) & 0x007fffffu) | (hi >> 20 == 0x400u ? 0x40000000u : 0x3f800000u));
}
__device__ __forceinline__ double from_float(float x) {       // a normal number
  const uint32_t u = __float_as_uint(x);
  return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))), (int)(u << 29));
}
static __device__ __noinline__ bool householder_far(double alpha, double xnorm_sq, double &beta, double &tau, double &scale) {
  return householder(alpha, xnorm_sq, beta, tau, scale);
}
__device__ __forceinline__ bool householder_fast(double alpha, double xnorm_sq, double &beta, double &tau,
                                                 double &scale) {
  if (is_zero(xnorm_sq)) return false;
  const double v = fma(alpha, alpha, xnorm_sq);
  // v = f 4^e with f in [1, 4)
  const int hv = __double2hiint(v), e2 = ((hv >> 20) - 1023) >> 1;
  if ((uint32_t)(hv >> 20) - 64u > 1900u) return householder_far(alpha, xnorm_sq, beta, tau, scale);
  const double f = __hiloint2double(hv - (e2 << 21), __double2loint(v));
  const double y0 = from_float(rsqrtf(to_float_12(f)));
  const double h = f * y0, r = fma(-h, y0, 1.0);
  const double y = fma(y0 * r, fma(r, 0.375, 0.5), y0);
  const double n0 = f * y, hy = __hiloint2double(__double2hiint(y) - (1 << 20), __double2loint(y));
  const double n = fma(fma(-n0, n0, f), hy, n0);                      // one Newton step rounds the root
  const double nrm = __hiloint2double(__double2hiint(n) + (e2 << 20), __double2loint(n));
  const double inv = __hiloint2double(__double2hiint(y) - (e2 << 20), __double2loint(y));
  beta = -copysign(nrm, alpha);
  tau = fma(fabs(alpha), inv, 1.0);                                   // (beta - alpha) / beta
  const double d = alpha - beta;                                      // no cancellation: the signs agree
  const int hd = __double2hiint(d), ed = ((hd >> 20) & 0x7ff) - 1023;
  const double g = __hiloint2double((hd & 0x7fffffff) - (ed << 20), __double2loint(d));   // |d| = g 2^ed, g in [1, 2)
  const double z0 = from_float(__fdividef(1.0f, to_float_12(g)));
  const double q = fma(-g, z0, 1.0);
  const double z = fma(z0, fma(q, q, q), z0);
  scale = __hiloint2double((__double2hiint(z) - (ed << 20)) | (hd & 0x80000000), __double2loint(z));
  return true;
}

// Digits of eight reflectors (columns col0 + lane / 4) over 32 rows from r0,
// as A or B fragments: [plane][16-row step][half].
template <int FORM>
__device__ __forceinline__ void v_digits(const double *P, int ldp, int r0, int col0, int m, int kcol,
                                         uint32_t (&f)[oz::kD][2][2]) {
  const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
#pragma unroll
  for (int kt = 0; kt < 2; ++kt)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = r0 + 16 * kt + 8 * h + 2 * t;
      oz::digits(v_fixed<FORM>(P, ldp, r, col0 + g, m, kcol), v_fixed<FORM>(P, ldp, r + 1, col0 + g, m, kcol),
                 [&](int d, uint32_t w) { f[d][kt][h] = w; });
    }
}
}  // namespace blk

// FORM, P, rowb, Ts, tt, round32, zero_t_on_skip and tau as in columns_la_f64
// (panel_dev.cuh); scr: blk::kScratch bytes of shared memory, 16-byte aligned;
// orig(r, c): element (r, c) of P as the call found it.
template <int FORM, typename Orig>
__device__ __noinline__ bool columns_blk_f64(double *P, int ldp, double *rowb, int rs, double *Ts, int ldts, int m,
                                             int k, int nc, int tt, bool round32, bool zero_t_on_skip, double *tau,
                                             unsigned char *scr, const Orig &orig) {
  using namespace blk;
  constexpr int D = oz::kD;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  double *const part = reinterpret_cast<double *>(scr + kPart);
  double *const dS = reinterpret_cast<double *>(scr + kSum), *const scal = dS + 8, *const tauS = dS + 16;
  int *const has_s = reinterpret_cast<int *>(scal + 1);
  double *const T8 = reinterpret_cast<double *>(scr + kT8);
  double *const G8 = reinterpret_cast<double *>(scr + kG8);
  int *const sc2 = reinterpret_cast<int *>(scr + kScale);
  unsigned char *const Wd = scr + kWd;
  double *const W1 = reinterpret_cast<double *>(scr + kW1);
  long long *const Wp = reinterpret_cast<long long *>(scr + kWp);
  unsigned long long *const X = reinterpret_cast<unsigned long long *>(P);
  const int nch = (m + 255) >> 8;                       // 256-row chunks
  static_assert(sizeof(Orig) <= 64, "the caller's Orig in shared memory");
  if (k <= 0) return true;
  if (tid == 0) new (scr + kOrig) Orig(orig);

  // ---- column scales: eight threads a column ----
  {
    const int c = tid >> 3, e = tid & 7;
    const double *const pc = P + (size_t)c * ldp;
    const int nrow = FORM == 0 ? 0 : min(c + 1, nc);    // rows of the triangle above, kept in rowb
    uint32_t mx = 0;
    auto mag = [](double v) {
      return ((uint32_t)__double2hiint(v) & 0x7fffffffu) | (__double2loint(v) != 0 ? 1u : 0u);
    };
    if (c < nc) {
      for (int r = e; r < m; r += 8) mx = max(mx, mag(pc[r]));
      for (int r = e; r < nrow; r += 8) mx = max(mx, mag(rowb[(size_t)c * rs + r]));
    }
#pragma unroll
    for (int o = 1; o <= 4; o <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const int ex = mx ? (int)(mx >> 20) : 1023;
    float n2 = 0.0f;
    auto rel = [&](double v) {                          // |v| 2^(1022 - ex) < 1, tiny values to zero
      const int h = (int)((uint32_t)__double2hiint(v) & 0x7fffffffu) - ((ex - 126) << 20);
      return __int_as_float(max(h, 0) << 3);
    };
    if (c < nc) {
      for (int r = e; r < m; r += 8) { const float f = rel(pc[r]); n2 = fmaf(f, f, n2); }
      for (int r = e; r < nrow; r += 8) { const float f = rel(rowb[(size_t)c * rs + r]); n2 = fmaf(f, f, n2); }
    }
#pragma unroll
    for (int o = 1; o <= 4; o <<= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, o);
    // largest s with norm 2^s <= 2^60.9 (oz_apply.cuh)
    const int lg = ((__float_as_int(n2 * (1.0f / 3.48f)) >> 23) & 0xff) - 127;
    if (e == 0) sc2[c] = 60 - ((lg + 2) >> 1) + 1022 - ex;
    // the column loop's sums are of products of two entries: between 2^-400
    // and 2^498 (with the square of 544 rows' norm) none leaves the normal
    // range, residuals 2^-60 below the column included
    if (!__syncthreads_and(mx == 0 || (ex <= 1520 && ex >= 623))) return false;
  }
  // ---- rows much lighter than the columns, a thread a row ----
  {
    const int lim = 60 - (round32 ? 30 : 8);
    bool light = false;
    for (int r = tid; r < m; r += TQR_THREADS) {
      int top = -4096;                                  // largest exponent in the columns' scales
#pragma unroll 8
      for (int c = 0; c < nc; ++c) {
        const int h = __double2hiint(P[(size_t)c * ldp + r]) & 0x7fffffff;
        top = max(top, h ? (h >> 20) - 1023 + sc2[c] : -4096);
      }
      light |= top > -4096 && top < lim;
    }
    if (__syncthreads_or(light)) return false;
  }
  // ---- the columns right of the first sub-block to fixed point, in place ----
  for (int r = tid; r < m; r += TQR_THREADS)
    for (int c0 = kW; c0 < nc; c0 += kW) {
      double *const p = P + (size_t)c0 * ldp + r;
      double x[kW];
#pragma unroll
      for (int c = 0; c < kW; ++c)
        if (c0 + c < nc) x[c] = p[(size_t)c * ldp];
#pragma unroll
      for (int c = 0; c < kW; ++c)
        if (c0 + c < nc) p[(size_t)c * ldp] = __longlong_as_double(oz::to_fixed<true>(x[c], sc2[c0 + c]) + (long long)oz::kBias);
    }
  for (int x = tid; x < 4 * 64; x += TQR_THREADS) T8[x] = 0.0;
  __syncthreads();

  const int j8 = lane & 7;
  uint32_t big = 0;
  for (int j0 = 0; j0 < nc; j0 += kW) {
    const int w = min(kW, nc - j0);
    double *const T8s = T8 + (j0 / kW) * 64;            // T8s[q + 8 p]
    if (j0 > 0) {
      // a rolled loop, and orig's address from shared memory: eight loads in
      // flight here cost the strips of the same kernel their registers
      // (8192^2 189.6 ms against 172.1)
      const Orig &org = *reinterpret_cast<const Orig *>(scr + kOrig);
      for (int r = tid; r < m; r += TQR_THREADS) {
        double *p = P + (size_t)j0 * ldp + r;
#pragma unroll 2
        for (int c = 0; c < w; ++c, p += ldp) {
          const double o = org(r, j0 + c);
          const long long f = __double_as_longlong(*p) - (long long)oz::kBias;
          *p = f == oz::to_fixed<true>(o, sc2[j0 + c]) ? o : oz::from_fixed(f, sc2[j0 + c]);
        }
      }
    }
    __syncwarp();                                       // a thread's rows are its warp's rows

    auto dots = [&](int i, int lo) {                    // part[warp][j] = sum over the warp's rows >= lo
      const double *const xi = P + (size_t)i * ldp, *const pj = P + (size_t)(j0 + min(j8, w - 1)) * ldp;
      double a = 0.0;                                   // one chain: the pipe, not its latency, sets the pace
      for (int ch = 0; ch < nch; ++ch) {
        const int r = 256 * ch + 32 * warp + 8 * (lane >> 3);
        if (r >= lo && r + 8 <= m) {
#pragma unroll
          for (int e = 0; e < 8; ++e) a = fma(xi[r + e], pj[r + e], a);
        } else if (r + 8 > lo && r < m) {
          for (int e = max(0, lo - r); e < min(8, m - r); ++e) a = fma(xi[r + e], pj[r + e], a);
        }
      }
      a += __shfl_xor_sync(0xffffffffu, a, 8);
      a += __shfl_xor_sync(0xffffffffu, a, 16);
      if (lane < 8) part[warp * 8 + lane] = a;
    };
    auto total = [&]() {                                // S_j in every lane of its j (one warp)
      const int h = lane >> 3;
      double s = part[16 * h + j8] + part[16 * h + 8 + j8];
      s += __shfl_xor_sync(0xffffffffu, s, 8);
      s += __shfl_xor_sync(0xffffffffu, s, 16);
      return s;
    };
    // d_j = -tau (row_j + S_j) right of column c, the row updated; left of it
    // the Gram entry v_j^T v_c (warp 0, a lane a column)
    auto combine = [&](int c, double tv, double S) {
      const int i = j0 + c;
      if (lane >= w || lane == c) return;
      double *const row = rowb + (size_t)i + (size_t)(j0 + lane) * rs;
      const double r = lane > c || FORM == 0 ? *row : 0.0, s = r + S;
      if (lane > c) {
        const double d = -(tv * s);
        dS[lane] = d;
        *row = r + d;
      } else {
        G8[lane + 8 * c] = s;
      }
    };
    auto t_column = [&](int c) {                        // T8s[:, c] (one warp); a skipped column stays zero
      const double tv = tauS[j0 + c];
      if (lane < c) {
        double a = 0.0;
        for (int u = lane; u < c; ++u) a = fma(T8s[lane + 8 * u], G8[u + 8 * c], a);
        T8s[lane + 8 * c] = -(tv * a);
      } else if (lane == c) {
        T8s[c + 8 * c] = tv;
      }
      __syncwarp();
    };

    const int wk = min(w, k - j0);                      // columns of it that have a reflector step
    for (int c = 0; c < wk; ++c) {
      const int i = j0 + c, lo = FORM == 0 ? i + 1 : 0;
      double *const xi = P + (size_t)i * ldp;
      dots(i, lo);
      __syncthreads();
      if (warp == 0) {
        double S = total();
        const double nrm = __shfl_sync(0xffffffffu, S, c);
        double beta = 0.0, tv = 0.0, sc = 0.0;
        const bool has = householder_fast(rowb[(size_t)i + (size_t)i * rs], nrm, beta, tv, sc);
        if (!has) tv = 0.0;
        if (round32) tv = (double)(float)tv;
        __syncwarp();                                   // every lane has read the diagonal
        if (!round32 && has) combine(c, tv, sc * S);
        if (!has && lane < c) G8[lane + 8 * c] = 0.0;
        if (lane == c) {
          scal[0] = sc;
          *has_s = has;
          tauS[i] = tv;
          tau[i] = tv;
          if (has) rowb[(size_t)i + (size_t)i * rs] = beta;
        }
      } else if (warp == 1 && c > 0) {
        t_column(c - 1);
      }
      __syncthreads();
      if (!*has_s) continue;
      const double sc = scal[0];
      if (round32) {
        for (int r = tid; r < m; r += TQR_THREADS)
          if (r >= lo) xi[r] = (double)(float)(xi[r] * sc);
        __syncwarp();
        dots(i, lo);
        __syncthreads();
        if (warp == 0) combine(c, tauS[i], total());
        __syncthreads();
      }
      // rows of column i scaled, the sub-block's columns right of it updated
      for (int r = tid; r < m; r += TQR_THREADS) {
        if (r < lo) continue;
        double v = xi[r];
        if (!round32) {
          v *= sc;
          xi[r] = v;
        }
        double *pj = xi + ldp + r;
#pragma unroll 1
        for (int j = c + 1; j < w; ++j, pj += ldp) *pj = fma(v, dS[j], *pj);
      }
      __syncwarp();
    }
    __syncthreads();
    if (warp == 1 && wk > 0) t_column(wk - 1);
    const int cr = j0 + w, nr = nc - cr;                // columns right of the sub-block
    if (nr <= 0 || wk <= 0) {
      __syncthreads();
      continue;
    }
    const int kcol = j0 + wk;

    // ---- W = V^T X for the columns right of it: M = 16 columns, N = 8 reflectors ----
    for (int mt = 0; 16 * mt < nr; ++mt) {
      long long sum[4] = {0, 0, 0, 0};
      for (int ch = 0; ch < nch; ++ch) {
        const int r0 = 256 * ch + 32 * warp;
        if (r0 >= m) break;
        uint32_t vb[D][2][2];
        v_digits<FORM>(P, ldp, r0, j0, m, kcol, vb);
        float acc[D][4];
        oz::init_acc(acc);
#pragma unroll
        for (int kt = 0; kt < 2; ++kt) {
          uint32_t xa[D][4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int col = cr + 16 * mt + g + 8 * (e & 1), r = r0 + 16 * kt + 8 * (e >> 1) + 2 * t;
            const unsigned long long *const xp = X + (size_t)min(col, nc - 1) * ldp;
            const unsigned long long y0 = (col < nc && r < m) ? xp[r] : oz::kBias;
            const unsigned long long y1 = (col < nc && r + 1 < m) ? xp[r + 1] : oz::kBias;
            oz::digits(y0, y1, [&](int d, uint32_t z) { xa[d][e] = z; });
          }
#pragma unroll
          for (int d = 0; d < D; ++d)
#pragma unroll
            for (int j = 0; j < D - d; ++j)
              oz::mma(acc[d + j], xa[j][0], xa[j][1], xa[j][2], xa[j][3], vb[d][kt][0], vb[d][kt][1]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[e] += oz::recon<47>(acc, e, big);
      }
      // [warp][column][reflector]
      long long *const wp = Wp + warp * 256 + (16 * mt + g) * 8 + 2 * t;
      wp[0] = sum[0]; wp[1] = sum[1]; wp[64] = sum[2]; wp[65] = sum[3];
    }
    __syncthreads();
    // ---- W1 = row + V^T X as FP64, W2 = T^T W1, the rows, W2's digits ----
    {
      const int c = tid >> 3, p = tid & 7;
      const bool on = c < nr;
      if (on) {
        long long s = 0;
#pragma unroll
        for (int q = 0; q < TQR_WARPS; ++q) s += Wp[q * 256 + tid];
        double v = oz::from_fixed(s, sc2[cr + c]);
        if (FORM != 0 && p < wk) v += rowb[(size_t)(j0 + p) + (size_t)(cr + c) * rs];
        W1[tid] = v;
      }
      __syncthreads();
      double w2 = 0.0;
      if (on && p < wk) {
        double a0 = 0.0, a1 = 0.0;
#pragma unroll
        for (int q = 0; q < kW; q += 2) {
          // T8s is zero above its last column and below the diagonal
          a0 = fma(T8s[q + 8 * p], W1[c * 8 + q], a0);
          a1 = fma(T8s[q + 1 + 8 * p], W1[c * 8 + q + 1], a1);
        }
        w2 = a0 + a1;
        if (FORM != 0) rowb[(size_t)(j0 + p) + (size_t)(cr + c) * rs] -= w2;
      }
      const unsigned long long y = (unsigned long long)oz::to_fixed<true>(w2, on ? sc2[cr + c] : 0) + oz::kBias;
      const unsigned long long yn = __shfl_down_sync(0xffffffffu, y, 1);
      if ((p & 1) == 0)
        oz::digits(y, yn, [&](int d, uint32_t z) { *reinterpret_cast<uint32_t *>(Wd + d * 512 + c * 16 + p * 2) = z; });
    }
    __syncthreads();
    // ---- X -= V W2: M = 16 rows, N = 8 columns, K = 8 reflectors ----
    for (int ch = 0; ch < nch; ++ch) {
      const int r0 = 256 * ch + 32 * warp;
      if (r0 >= m) break;
#pragma unroll 1
      for (int mt = 0; mt < 2; ++mt) {
        uint32_t va[D][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = r0 + 16 * mt + 8 * h + g;
          oz::digits(v_fixed<FORM>(P, ldp, r, j0 + 2 * t, m, kcol), v_fixed<FORM>(P, ldp, r, j0 + 2 * t + 1, m, kcol),
                     [&](int d, uint32_t z) { va[d][h] = z; });
        }
#pragma unroll 1
        for (int nt = 0; 8 * nt < nr; ++nt) {
          float acc[D][4];
          oz::init_acc(acc);
          uint32_t wb[D];
#pragma unroll
          for (int d = 0; d < D; ++d)
            wb[d] = *reinterpret_cast<const uint32_t *>(Wd + d * 512 + (8 * nt + g) * 16 + t * 4);
#pragma unroll
          for (int d = 0; d < D; ++d)
#pragma unroll
            for (int j = 0; j < D - d; ++j) mma8(acc[d + j], va[d][0], va[d][1], wb[j]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int r = r0 + 16 * mt + g + 8 * (e >> 1), col = cr + 8 * nt + 2 * t + (e & 1);
            const long long dx = oz::recon<47>(acc, e, big);
            if (r < m && col < nc) X[(size_t)col * ldp + r] -= (unsigned long long)dx;
          }
        }
      }
    }
    __syncwarp();
  }

  // ---- Gram blocks (a, b), a < b, of the sub-blocks: block x = (0,1) (0,2) (1,2) (0,3) (1,3) (2,3) ----
  const int nsb = (nc + kW - 1) / kW;
  {
    for (int x = 0; x < 6 * 2; ++x) Wp[warp * 384 + 32 * x + lane] = 0;
    __syncwarp();
    for (int ch = 0; ch < nch; ++ch) {
      const int r0 = 256 * ch + 32 * warp;
      if (r0 >= m) break;
      uint32_t d0[D][2][2], d1[D][2][2], d2[D][2][2];
      v_digits<FORM>(P, ldp, r0, 0, m, k, d0);
      v_digits<FORM>(P, ldp, r0, kW, m, k, d1);
      // (reflector g of sub-blocks a0 and a1) x (reflectors 2 t, 2 t + 1 of b)
      auto gram = [&](const uint32_t (&a)[D][2][2], const uint32_t (&a1)[D][2][2], const uint32_t (&bb)[D][2][2],
                      int x0, int x1) {
        float acc[D][4];
        oz::init_acc(acc);
#pragma unroll
        for (int kt = 0; kt < 2; ++kt)
#pragma unroll
          for (int d = 0; d < D; ++d)
#pragma unroll
            for (int j = 0; j < D - d; ++j)
              oz::mma(acc[d + j], a[j][kt][0], a1[j][kt][0], a[j][kt][1], a1[j][kt][1], bb[d][kt][0], bb[d][kt][1]);
        long long *const wp = Wp + warp * 384 + g + 16 * t;        // block [p + 8 q]: row p of a, column q of b
        wp[64 * x0] += oz::recon<47>(acc, 0, big);
        wp[64 * x0 + 8] += oz::recon<47>(acc, 1, big);
        if (x1 >= 0) {
          wp[64 * x1] += oz::recon<47>(acc, 2, big);
          wp[64 * x1 + 8] += oz::recon<47>(acc, 3, big);
        }
      };
      gram(d0, d0, d1, 0, -1);
      if (nsb > 2) {
        v_digits<FORM>(P, ldp, r0, 2 * kW, m, k, d2);
        gram(d0, d1, d2, 1, 2);
      }
      if (nsb > 3) {
        uint32_t d3[D][2][2];
        v_digits<FORM>(P, ldp, r0, 3 * kW, m, k, d3);
        gram(d0, d1, d3, 3, 4);
        gram(d2, d2, d3, 5, -1);
      }
    }
  }
  __syncthreads();
  // T = [T_aa, -T_(0..a) G_(0..a),b T_bb]: first Y = G T_bb, then the block columns in turn
  double *const G = reinterpret_cast<double *>(Wp);     // a thread's sum goes where only it reads: warp 0's slots
  double *const Y = G + 384;
  for (int x = tid; x < 384; x += TQR_THREADS) {
    long long s = 0;
#pragma unroll
    for (int q = 0; q < TQR_WARPS; ++q) s += Wp[q * 384 + x];
    G[x] = oz::from_fixed(s, 61);
  }
  __syncthreads();
  double *const TT = Y + 384;                            // T with zero columns where there is no reflector, ld 33
  for (int x = tid; x < 384; x += TQR_THREADS) {
    const int b = x < 64 ? 1 : (x < 192 ? 2 : 3), p = x & 7, q = (x >> 3) & 7;
    const double *const Gx = G + (x & ~63) + p, *const Tx = T8 + b * 64 + 8 * q;   // T8 is zero below the diagonal
    double a0 = 0.0, a1 = 0.0;
#pragma unroll
    for (int u = 0; u < kW; u += 2) {
      a0 = fma(Gx[8 * u], Tx[u], a0);
      a1 = fma(Gx[8 * u + 8], Tx[u + 1], a1);
    }
    Y[x] = a0 + a1;
  }
  for (int x = tid; x < 4 * 64; x += TQR_THREADS) {
    const int b = x >> 6;
    TT[b * kW + (x & 7) + 33 * (b * kW + ((x >> 3) & 7))] = T8[x];
  }
  __syncthreads();
#pragma unroll
  for (int b = 1; b < 4; ++b) {
    // thread: row p < 8 b, column q of block column b; blocks (0, b) .. (b - 1, b) start at b (b - 1) / 2
    const int p = tid >> 3, q = tid & 7;
    if (b < nsb && p < b * kW) {
      double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int u = 0; u < b * kW; ++u) {
        const double tv = u >= p ? TT[p + 33 * u] : 0.0;
        a[u & 3] = fma(tv, Y[(b * (b - 1) / 2 + (u >> 3)) * 64 + (u & 7) + 8 * q], a[u & 3]);
      }
      TT[p + 33 * (b * kW + q)] = -((a[0] + a[1]) + (a[2] + a[3]));
    }
    __syncthreads();
  }
  // a column without a reflector keeps what T had (or gets zeros)
  for (int x = tid; x < 32 * 32; x += TQR_THREADS) {
    const int p = x & 31, q = x >> 5;
    if (p <= q && q < k && (zero_t_on_skip || tauS[q] != 0.0)) Ts[p + (size_t)q * ldts] = TT[p + 33 * q];
  }
  __syncthreads();
  (void)big;                                            // the reflectors are orthogonal: nothing overflows
  return true;
}

}  // namespace tqr
