// panel_reg.cuh -- FP32 panels in registers, a warp a set of columns.
//
// FP32 arithmetic is cheap on GB300 (128 FMAs per clock and SM, 4 clocks of
// latency); the FP32 column step (column_step, panel_dev.cuh) waited on five
// barriers a column and on the panel's trips through shared memory: 2.8 us.
// Here column j lives in warp j % 8, lane l holding its rows l, l + 32, ..., so a
// column's dot product with the reflector, its d and its update need no other
// warp; only the reflector itself goes through shared memory.  Column i's
// owner, once it has updated it for column i - 1, forms its norm and scalars
// and writes the scaled reflector: one barrier a column.  T's column i is
// formed during column i + 1 by a warp that is not the next owner.
//
// The sums are column_step's, term by term in its order, so the results are
// its bits: products of rows 32 apart run down one lane, lanes meet by the
// same exchanges (for geqr2, whose rows count from the diagonal, after a
// rotation of the lanes), warps' partial norms are added in order.
#pragma once
#include "common.cuh"

namespace tqr {

namespace reg {
constexpr int kMaxRows = 512, kMaxCols = 32;
// scratch (floats): reflector [2][512] | d [2][32] | tau, has reflector [4][2] (T's column reads them a step late)
constexpr int kV = 0, kD = 1024, kS = kD + 64;
constexpr size_t kScratch = sizeof(float) * (kS + 8);

__host__ __device__ inline bool covers(int m, int nc) { return m >= 1 && m <= kMaxRows && nc >= 1 && nc <= kMaxCols; }
}  // namespace reg

// FORM 0: geqr2 of the m x nc panel A.  1: tsqrt block [B; A] with B the
// triangle in shared memory (ld ldb).  2: ttqrt, column j of A holding rows
// [0, tt + j].  k reflectors; Ts (shared, ld ldts, may be null) receives T's
// columns that have a reflector (all with zero_t_on_skip).  CPW: columns a warp
// holds (8 CPW >= nc); RPL: rows a lane holds (32 RPL >= m).
template <int FORM, int CPW, int RPL>
__device__ __forceinline__ void columns_reg_nc(float *A, int lda, float *B, int ldb, float *Ts, int ldts, int m, int k,
                                               int nc, int tt, bool zero_t_on_skip, float *tau, float *scr) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr unsigned kAll = 0xffffffffu;
  float x[CPW][RPL];
#pragma unroll
  for (int u = 0; u < CPW; ++u)
#pragma unroll
    for (int t = 0; t < RPL; ++t) {
      const int c = 8 * u + warp, r = lane + 32 * t;
      x[u][t] = (r < m && c < nc && (FORM != 2 || r <= tt + c)) ? __ldcg(A + r + (size_t)c * lda) : 0.0f;
    }
  // sum over the lanes, lane l standing for row l - x0 of column_step's order
  auto lanes = [&](float a, int x0) {
    if (FORM == 0) a = __shfl_sync(kAll, a, (lane + x0) & 31);
    return warp_sum(a);
  };
  // T[0:i, i] from T's earlier columns and d (a warp, a lane a row)
  auto t_column = [&](int i) {
    const float *const d = scr + reg::kD + 32 * (i & 1), *const sc = scr + reg::kS + 2 * (i & 3);
    if (sc[1] == 0.0f) {
      if (zero_t_on_skip && lane <= i) Ts[lane + (size_t)i * ldts] = 0.0f;
      return;
    }
    if (lane < i) {
      float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
      const float *tp = Ts + lane;
      int q = lane;
      for (; q + 3 < i; q += 4) {
        a0 = fmaf(tp[(size_t)q * ldts], d[q], a0);
        a1 = fmaf(tp[(size_t)(q + 1) * ldts], d[q + 1], a1);
        a2 = fmaf(tp[(size_t)(q + 2) * ldts], d[q + 2], a2);
        a3 = fmaf(tp[(size_t)(q + 3) * ldts], d[q + 3], a3);
      }
      for (; q < i; ++q) a0 = fmaf(tp[(size_t)q * ldts], d[q], a0);
      Ts[lane + (size_t)i * ldts] = (a0 + a1) + (a2 + a3);
    } else if (lane == i) {
      Ts[i + (size_t)i * ldts] = sc[0];
    }
  };
#pragma unroll
  for (int u0 = 0; u0 < CPW; ++u0) {
#pragma unroll 1
    for (int w0 = 0; w0 < 8; ++w0) {
      const int i = 8 * u0 + w0, buf = i & 1, x0 = FORM == 0 ? i + 1 : 0;
      if (i >= k) break;
      float *const vs = scr + reg::kV + 512 * buf, *const ds = scr + reg::kD + 32 * buf, *const sS = scr + reg::kS + 2 * (i & 3);
      if (warp == w0) {
        // ---- the owner: norm, scalars, the scaled reflector ----
        const bool late = FORM == 0 && ((lane - x0) & 31) + x0 >= 32;   // this lane's first row below the diagonal is row lane + 32
        float part[8];
#pragma unroll
        for (int w = 0; w < 8; ++w) {
          float s = 0.0f;
#pragma unroll
          for (int t = w; t < RPL; t += 8) {
            const float a = x[u0][t], b = t + 1 < RPL ? x[u0][t + 1] : 0.0f, y = late ? b : a;
            s = fmaf(y, y, s);
          }
          part[w] = 32 * w < m ? lanes(s, x0) : 0.0f;
        }
        float nrm = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) nrm += part[w];
        const float alpha = FORM == 0 ? __shfl_sync(kAll, x[u0][0], i) : B[i + (size_t)i * ldb];
        float beta = 0.0f, tv = 0.0f, sc = 0.0f;
        const bool has = householder(alpha, nrm, beta, tv, sc);
        __syncwarp();                                     // every lane has read alpha
        if (has) {
#pragma unroll
          for (int t = 0; t < RPL; ++t) {
            const bool below = FORM != 0 || t > 0 || lane > i;
            const float v = x[u0][t] * sc;
            if (below) x[u0][t] = v;
            if (32 * t < m) vs[lane + 32 * t] = below ? v : 0.0f;
          }
          if (FORM == 0 && lane == i) x[u0][0] = beta;
          if (FORM != 0 && lane == 0) B[i + (size_t)i * ldb] = beta;
        }
        if (lane == 0) {
          sS[0] = tv;
          sS[1] = has ? 1.0f : 0.0f;
          tau[i] = has ? tv : 0.0f;
        }
      }
      __syncthreads();
      if (Ts && i > 0 && warp == ((w0 + 4) & 7)) t_column(i - 1);
      if (sS[1] == 0.0f) continue;
      const float tv = sS[0];
      float v[RPL];
#pragma unroll
      for (int t = 0; t < RPL; ++t) v[t] = 32 * t < m ? vs[lane + 32 * t] : 0.0f;
      const bool on0 = FORM != 0 || lane > i;             // row lane is one of the reflector's
      float a[CPW];
#pragma unroll
      for (int u = 0; u < CPW; ++u) {
        a[u] = on0 ? fmaf(v[0], x[u][0], 0.0f) : 0.0f;
#pragma unroll
        for (int t = 1; t < RPL; ++t)
          if (32 * t < m) a[u] = fmaf(v[t], x[u][t], a[u]);
      }
#pragma unroll
      for (int u = 0; u < CPW; ++u) a[u] = lanes(a[u], x0);
      // d of the warp's columns, side by side, then their updates
      float d[CPW], rv[CPW];
#pragma unroll
      for (int u = 0; u < CPW; ++u) {
        const int j = 8 * u + warp;
        rv[u] = FORM == 0 ? __shfl_sync(kAll, x[u][0], i) : (j > i && j < nc ? B[i + (size_t)j * ldb] : 0.0f);
      }
#pragma unroll
      for (int u = 0; u < CPW; ++u) {
        const int j = 8 * u + warp;
        const float s = FORM == 0 || j > i ? a[u] + rv[u] : a[u];
        d[u] = -(tv * s);
      }
      if (FORM != 0) __syncwarp();                        // every lane has the rows' entries
#pragma unroll
      for (int u = 0; u < CPW; ++u) {
        const int j = 8 * u + warp;
        if (lane == 0 && j != i && j < nc) {
          ds[j] = d[u];
          if (FORM != 0 && j > i) B[i + (size_t)j * ldb] = rv[u] + d[u];
        }
        if (j > i && j < nc) {
#pragma unroll
          for (int t = 1; t < RPL; ++t) x[u][t] = fmaf(v[t], d[u], x[u][t]);
          if (on0) x[u][0] = fmaf(v[0], d[u], x[u][0]);
          if (FORM == 0 && lane == i) x[u][0] += d[u];
        }
      }
    }
  }
  if (Ts && k > 0) {
    __syncthreads();
    if (warp == 0) t_column(k - 1);
  }
#pragma unroll
  for (int u = 0; u < CPW; ++u)
#pragma unroll
    for (int t = 0; t < RPL; ++t) {
      const int c = 8 * u + warp, r = lane + 32 * t;
      if (r < m && c < nc && (FORM != 2 || r <= tt + c)) A[r + (size_t)c * lda] = x[u][t];
    }
  __syncthreads();
}

// The instantiation for nc columns and m rows.
template <int FORM>
__device__ __noinline__ void columns_reg_f32(float *A, int lda, float *B, int ldb, float *Ts, int ldts, int m, int k,
                                             int nc, int tt, bool zero_t_on_skip, float *tau, float *scr) {
  if (m <= 256) {
    if (nc <= 16) columns_reg_nc<FORM, 2, 8>(A, lda, B, ldb, Ts, ldts, m, k, nc, tt, zero_t_on_skip, tau, scr);
    else columns_reg_nc<FORM, 4, 8>(A, lda, B, ldb, Ts, ldts, m, k, nc, tt, zero_t_on_skip, tau, scr);
  } else {
    if (nc <= 16) columns_reg_nc<FORM, 2, 16>(A, lda, B, ldb, Ts, ldts, m, k, nc, tt, zero_t_on_skip, tau, scr);
    else columns_reg_nc<FORM, 4, 16>(A, lda, B, ldb, Ts, ldts, m, k, nc, tt, zero_t_on_skip, tau, scr);
  }
}

}  // namespace tqr
