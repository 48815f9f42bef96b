// sapb_ldlt.cuh -- blocked LDL^T of a small symmetric positive definite matrix
// held in shared memory by one thread block (the per-world dense factor of
// the reference's BlockCholeskySolverBatched, sim/blocked_cholesky.py:414-604,
// as LDL^T: no square roots).
#pragma once

#include <cstdint>
#include <type_traits>

#include "sapb_device.cuh"

namespace sapb {

// Column-descending list of the lower triangle below row 0, each column
// followed by its nrhs right-hand-side rows: entries (i << 8 | j) for j = n-1
// .. 1, i = j .. n-1+nrhs.  The trailing triangle of columns > k is its first
// m(m+1)/2 + nrhs m entries, m = n-1-k.  n + nrhs <= 256.
__host__ __device__ constexpr int triangle_list_size(int n, int nrhs) {
  return n * (n - 1) / 2 + nrhs * (n - 1) + 1;
}
template <int NT>
__device__ __forceinline__ void build_triangle_list(uint16_t* tri, int n, int nrhs) {
#pragma unroll 1
  for (int j = n - 1 - (int)threadIdx.x; j >= 1; j -= NT) {
    const int m = n - 1 - j;
    const int off = m * (m + 1) / 2 + nrhs * m;
    for (int i = j; i < n + nrhs; ++i) tri[off + (i - j)] = (uint16_t)((i << 8) | j);
  }
}

// Pivot reciprocal of the factorization: Newton-Raphson steps from the
// hardware's approximation (two in FP64, one in FP32), without a range check.
// Of a pivot that is not positive and finite, or outside the approximation's
// range (subnormal, or beyond 2^126 in FP32 and 2^1022 in FP64), the result is
// no positive normal number: such pivots are kept away from it (the dense solve
// scales that world's H, WorldScale; the tree-blocked solve factors that block
// again with divisions) or reported like bad ones (the free motion's in FP64,
// whose velocity is then NaN).  A guard on each pivot is on the serial chain; a
// check of every block's reciprocals with divisions behind it cost 2 % of the
// dense solves and the free motion.
__device__ __forceinline__ double pivot_recip(double d) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
  x = fma(x, fma(-d, x, 1.0), x);
  return fma(x, fma(-d, x, 1.0), x);
}
__device__ __forceinline__ float pivot_recip(float d) {
  float x;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(d));
  return fmaf(x, fmaf(-d, x, 1.0f), x);
}

__device__ __forceinline__ bool positive_normal(double r) {
  return (unsigned)(__double2hiint(r) - 0x00100000) < 0x7fe00000u;
}
__device__ __forceinline__ bool positive_normal(float r) {
  return (unsigned)(__float_as_int(r) - 0x00800000) < 0x7f000000u;
}
template <bool DIVIDE, typename T>
__device__ __forceinline__ T pivot(T d) {
  return DIVIDE ? T(1) / d : pivot_recip(d);
}

// Values of S (the scaled panel) per row: B rounded up so that rows are
// 16-byte aligned.
template <typename T, int B>
__host__ __device__ constexpr int ldlt_panel_stride() {
  return sizeof(T) == 8 ? (B + 1) / 2 * 2 : (B + 3) / 4 * 4;
}

// The B values of a row of S, 16 bytes at a time.
template <typename T, int B>
__device__ __forceinline__ void load_panel_row(const T* Sj, T (&v)[B]) {
  constexpr int V = 16 / sizeof(T);
  using V16 = typename std::conditional<sizeof(T) == 8, double2, float4>::type;
#pragma unroll
  for (int c = 0; c < B; c += V) {
    const V16 q = *reinterpret_cast<const V16*>(Sj + c);
    const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
    for (int u = 0; u < V; ++u)
      if (c + u < B) v[c + u] = e[u];
  }
}

// In-place right-looking LDL^T of the lower triangle of H (row stride ldH;
// tri: the triangle list of build_triangle_list for n + tri_shift DOFs and
// NRHS right-hand sides): afterwards H_ik = L_ik d_k below the diagonal (L
// unit lower), d_k on it, dinv[k] = 1/d_k.  NRHS: H holds that many more rows
// from n on, right-hand sides b; they are carried through the panels like any
// other row and end as L^-1 b, so the forward substitution costs no pass of
// its own.  NS: n at compile time, or 0.
//
// B-column blocks, two barriers per block.  Panel: every thread that holds a
// row below the block eliminates it against the block's B x B diagonal block,
// which it factors in registers (its own copy: a shuffle costs more than the
// arithmetic).  Trailing triangle: every thread owns the same entries of the
// list throughout -- the prefix that is left only shrinks -- and with NS
// keeps them in registers until their column's panel is next; the panel is
// read as B-value rows, unscaled from H, divided by the pivots and negated
// from S.  A world's whole time here is latency: about 100 dependent
// instructions of one warp a panel.  The arithmetic is the right-looking
// recurrence on the stored form W_ik = L_ik d_k:
//   d_k = H_kk - sum_{e<k} W_ke^2 / d_e,  W_ik = H_ik - sum_{e<k} W_ie W_ke / d_e.
// H must be complete when called (barrier before); complete on return (NRHS:
// to warp 0; the last block's rows are its alone).
template <int NT, typename T, int B, int NRHS, int NS>
__device__ __forceinline__ void ldlt_blocked(T* H, int n, int ldH, T* dinv, T* S, const uint16_t* tri,
                                             int tri_shift = 0) {
  static_assert(B >= 1 && B <= 8, "block width");
  constexpr int kS = ldlt_panel_stride<T, B>();
  constexpr int kLeft = NS > B ? NS - B : 0;  // columns right of the first block
  constexpr int kRounds = NS > 0 ? (kLeft * (kLeft + 1) / 2 + NRHS * kLeft + NT - 1) / NT : 0;
  constexpr bool kWhole = NS > 0 && NS % B == 0;  // no partial block
  const int tid = threadIdx.x;
  const int rows = n + NRHS;
  T acc[kRounds > 0 ? kRounds : 1];
  int at[kRounds > 0 ? kRounds : 1];  // i << 8 | j, -1: no entry
  if constexpr (kRounds > 0) {
    const int left = n - B, cnt = left > 0 ? left * (left + 1) / 2 + NRHS * left : 0;
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const int e = tid + r * NT;
      at[r] = e < cnt ? (int)tri[e] - tri_shift * 257 : -1;
      acc[r] = e < cnt ? H[(at[r] >> 8) * ldH + (at[r] & 255)] : T(0);
    }
  }
#pragma unroll 1
  for (int K = 0; K < n; K += B) {
    const int bs = kWhole ? B : min(B, n - K);
    const int rest = n - K - bs, prow = rows - K - bs;
    T W[B][B], R[B];
    if ((tid & ~31) < (prow > 1 ? prow : 1)) {
      // the diagonal block (padding rows: identity)
      const T* Hd = H + K * ldH + K;
#pragma unroll
      for (int a = 0; a < B; ++a)
#pragma unroll
        for (int b = 0; b <= a; ++b) W[a][b] = a < bs ? Hd[a * ldH + b] : (a == b ? T(1) : T(0));
#pragma unroll
      for (int c = 0; c < B; ++c) {
        R[c] = pivot_recip(W[c][c]);
#pragma unroll
        for (int m = c + 1; m < B; ++m) {
          const T l = W[m][c] * R[c];
#pragma unroll
          for (int m2 = c + 1; m2 <= m; ++m2) W[m][m2] -= l * W[m2][c];
        }
      }
      auto eliminate = [&](int t) {
        const int i = K + bs + t;
        T* Hi = H + i * ldH + K;
        T v[B], q[B];
#pragma unroll
        for (int c = 0; c < B; ++c) v[c] = c < bs ? Hi[c] : T(0);
#pragma unroll
        for (int c = 0; c < B; ++c) {
          q[c] = -v[c] * R[c];
#pragma unroll
          for (int m = c + 1; m < B; ++m) v[m] += q[c] * W[m][c];
        }
        T* Si = S + (i < n ? i : n) * kS;  // (right-hand sides: a row past the others, not read)
#pragma unroll
        for (int c = 0; c < B; ++c)
          if (c < bs) {
            Hi[c] = v[c];
            Si[c] = q[c];
          }
      };
      if constexpr (NS > 0) {  // every row has its thread
        if (tid < prow) eliminate(tid);
      } else {
#pragma unroll 1
        for (int t = tid; t < prow; t += NT) eliminate(t);
      }
    }
    // The factored block goes back to H once every thread has read it: at
    // once when one warp holds all panel rows, else after the panel's barrier
    // (the trailing update never touches the diagonal block).  Every lane of
    // warp 0 holds the same values and stores them all: no selection by lane.
    const bool one_warp = prow <= 32;
    auto store_block = [&]() {
#pragma unroll
      for (int a = 0; a < B; ++a)
        if (a < bs) {
#pragma unroll
          for (int b = 0; b <= a; ++b) H[(K + a) * ldH + K + b] = W[a][b];
          dinv[K + a] = R[a];
        }
    };
    if (one_warp && tid < 32) {
      __syncwarp();
      store_block();
    }
    if (rest <= 0) {
      if (NRHS > 0) __syncwarp();
      else __syncthreads();
      break;
    }
    __syncthreads();
    if (!one_warp && tid < 32) store_block();
    // trailing update of entries (i, j), j >= K + bs: the first entries of
    // the column-descending list
    const int cnt = rest * (rest + 1) / 2 + NRHS * rest;
    const T* Hk = H + K;
    if constexpr (kRounds > 0) {
#pragma unroll
      for (int r = 0; r < kRounds; ++r) {
        if (r * NT < cnt) {
          const int e = tid + r * NT;
          const int i = at[r] >> 8, j = at[r] & 255;
          if (e < cnt) {
            const T* Hi = Hk + i * ldH;
            T sj[B];
            load_panel_row<T, B>(S + j * kS, sj);
#pragma unroll
            for (int c = 0; c < B; ++c) acc[r] += Hi[c] * sj[c];
            if (j < K + 2 * B) H[i * ldH + j] = acc[r];  // its column is next
          }
        }
      }
    } else {
#pragma unroll 2
      for (int e = tid; e < cnt; e += NT) {
        const int ij = tri[e] - tri_shift * 257;
        const int i = ij >> 8, j = ij & 255;
        T* h = H + i * ldH + j;
        const T* Hi = Hk + i * ldH;
        T sj[B];
        load_panel_row<T, B>(S + j * kS, sj);
        T v = *h;
#pragma unroll
        for (int c = 0; c < B; ++c) v += Hi[c] * sj[c];
        *h = v;
      }
    }
    __syncthreads();
  }
}

// z <- L^-T z by the calling warp: lanes hold z of rows lane and lane + 32
// (n <= 64) and their d0, d1 = 1/d.  From the last row on, x_k = z_k goes round
// by a shuffle: a chain of a shuffle and a fused multiply-add a row.
template <typename T>
__device__ __forceinline__ void ldlt_backward_lanes(const T* H, int n, int ldH, T d0, T d1, T& z0, T& z1) {
  const int lane = threadIdx.x & 31;
  const T* Hl = H + lane;
  int k = n - 1;
#pragma unroll 1
  for (; k >= 32; --k) {  // rows of the second slot
    const T w0 = Hl[k * ldH] * d0, w1 = lane + 32 < k ? Hl[k * ldH + 32] * d1 : T(0);
    const T xk = __shfl_sync(0xffffffffu, z1, k - 32);
    z1 -= w1 * xk;
    z0 -= w0 * xk;
  }
#pragma unroll 4
  for (; k > 0; --k) {
    const T w0 = lane < k ? Hl[k * ldH] * d0 : T(0);
    z0 -= w0 * __shfl_sync(0xffffffffu, z0, k);
  }
}

// x = L^-T D^-1 y by the calling warp alone, y = row `rhs` of the LDL^T that
// ldlt_blocked left in H (n <= 64).  Returns, to every lane, whether every
// pivot is positive and finite (by its reciprocal); if not, x is NaN.
template <typename T, int NS>
__device__ __forceinline__ bool ldlt_backward_warp(const T* H, int n, int ldH, const T* dinv, int rhs, double* x) {
  const int lane = threadIdx.x & 31;
  const T* y = H + rhs * ldH;
  const T d0 = lane < n ? dinv[lane] : T(1), d1 = lane + 32 < n ? dinv[lane + 32] : T(1);
  const bool ok = __all_sync(0xffffffffu, d0 > T(0) && d0 < T(INFINITY) && d1 > T(0) && d1 < T(INFINITY));
  T z0 = lane < n ? y[lane] * d0 : T(0), z1 = lane + 32 < n ? y[lane + 32] * d1 : T(0);
  ldlt_backward_lanes(H, n, ldH, d0, d1, z0, z1);
  const double nanv = __longlong_as_double(0x7ff8000000000000ULL);
  if (lane < n) x[lane] = ok ? double(z0) : nanv;
  if (lane + 32 < n) x[lane + 32] = ok ? double(z1) : nanv;
  return ok;
}

// x <- -A^-1 x (neg) or A^-1 x with the LDL^T that ldlt_blocked left in H
// and dinv, by the whole block: forward L z = b, zd = D^-1 z, backward
// L^T x = zd, over the same blocks as the factorization.  Per block every
// thread solves the small diagonal system in registers, then threads update
// the remaining rows (one row each); two barriers per block.  x (FP64 or T)
// holds the intermediate vectors; the arithmetic is in T.  A pivot that is
// not positive / finite makes x NaN.  x complete on entry (barrier before)
// and on return.
template <int NT, typename T, typename X>
__device__ void ldlt_solve_blocked(const T* H, int n, int ldH, const T* dinv, X* x, bool neg) {
  const int tid = threadIdx.x;
  constexpr int B = sizeof(T) == 4 ? 8 : 6;
  bool ok = true;
  for (int k = 0; k < n; ++k) ok = ok && dinv[k] > T(0) && dinv[k] < T(INFINITY);
  const T sgn = neg ? T(-1) : T(1);
  // forward
  for (int K = 0; K < n; K += B) {
    const int bs = min(B, n - K);
    T z[B], R[B];
#pragma unroll
    for (int a = 0; a < B; ++a) {
      R[a] = a < bs ? dinv[K + a] : T(0);
      T v = a < bs ? T(x[K + a]) : T(0);
      if (K == 0) v *= sgn;
#pragma unroll
      for (int e = 0; e < a; ++e)
        if (a < bs) v -= H[(size_t)(K + a) * ldH + K + e] * R[e] * z[e];
      z[a] = v;
    }
    __syncthreads();  // every thread has read the block's entries of x
    if (tid < bs) {
#pragma unroll
      for (int a = 0; a < B; ++a)
        if (a == tid) x[K + a] = X(z[a] * R[a]);
    }
    for (int i = K + bs + tid; i < n; i += NT) {
      T acc = T(x[i]);
      if (K == 0) acc *= sgn;
#pragma unroll
      for (int c = 0; c < B; ++c)
        if (c < bs) acc -= H[(size_t)i * ldH + K + c] * R[c] * z[c];
      x[i] = X(acc);
    }
    __syncthreads();
  }
  // backward
  const int last = ((n - 1) / B) * B;
  for (int K = last; K >= 0; K -= B) {
    const int bs = min(B, n - K);
    T xb[B];
#pragma unroll
    for (int a = B - 1; a >= 0; --a) {
      if (a >= bs) {
        xb[a] = T(0);
        continue;
      }
      T v = T(x[K + a]);
      const T ra = dinv[K + a];
#pragma unroll
      for (int c = a + 1; c < B; ++c)
        if (c < bs) v -= H[(size_t)(K + c) * ldH + K + a] * ra * xb[c];
      xb[a] = v;
    }
    __syncthreads();
    if (tid < bs) {
#pragma unroll
      for (int a = 0; a < B; ++a)
        if (a == tid) x[K + a] = X(xb[a]);
    }
    for (int i = tid; i < K; i += NT) {
      T acc = T(0);
#pragma unroll
      for (int c = 0; c < B; ++c)
        if (c < bs) acc += H[(size_t)(K + c) * ldH + i] * xb[c];
      x[i] = X(T(x[i]) - dinv[i] * acc);
    }
    __syncthreads();
  }
  if (!ok) {
    for (int i = tid; i < n; i += NT) x[i] = X(__longlong_as_double(0x7ff8000000000000ULL));
    __syncthreads();
  }
}

// x = A^-1 b (or -A^-1 b with neg) by the calling warp alone (all 32 lanes;
// no block barrier) with the LDL^T that ldlt_blocked left in H and dinv:
// lanes own rows lane and lane + 32 (n <= 64).  Forward, y_k / d_k goes round
// by a shuffle and each later row subtracts W_ik times it; backward as in
// ldlt_backward_lanes.  b is read before x is written (they may alias).  `ok`
// false (a pivot not positive / finite, ldlt_pivots_ok_warp) makes x NaN.
// (35 DOFs, forward and backward, alone on an SM: 8.7 k cycles with the
// pivots read per row and the owner of a row selected by branches.)
template <typename T>
__device__ __forceinline__ void ldlt_solve_warp(const T* H, int n, int ldH, const T* dinv, const double* b, double* x,
                                                bool neg, bool ok) {
  const int lane = threadIdx.x & 31;
  const T sg = neg ? T(-1) : T(1);
  const T d0 = lane < n ? dinv[lane] : T(1), d1 = lane + 32 < n ? dinv[lane + 32] : T(1);
  T h0 = lane < n ? sg * T(b[lane]) : T(0);
  T h1 = lane + 32 < n ? sg * T(b[lane + 32]) : T(0);
  const T* H0 = H + lane * ldH;
  const T* H1 = H + (lane + 32) * ldH;
  const bool two = n > 32;
#pragma unroll 4
  for (int k = 0; k < (two ? 32 : n); ++k) {
    const T w0 = lane > k && lane < n ? H0[k] : T(0);
    const T w1 = lane + 32 < n ? H1[k] : T(0);
    const T yk = __shfl_sync(0xffffffffu, h0 * d0, k);
    h0 -= w0 * yk;
    h1 -= w1 * yk;
  }
#pragma unroll 1
  for (int k = 32; k < n; ++k) {
    const T w1 = lane + 32 > k && lane + 32 < n ? H1[k] : T(0);
    h1 -= w1 * __shfl_sync(0xffffffffu, h1 * d1, k - 32);
  }
  T z0 = h0 * d0, z1 = h1 * d1;
  ldlt_backward_lanes(H, n, ldH, d0, d1, z0, z1);
  const double nanv = __longlong_as_double(0x7ff8000000000000ULL);
  __syncwarp();
  if (lane < n) x[lane] = ok ? double(z0) : nanv;
  if (lane + 32 < n) x[lane + 32] = ok ? double(z1) : nanv;
}

// Whether every pivot of a stored LDL^T is positive and finite by its
// reciprocal (the warp's lanes check two each), returned to every lane.
template <typename T>
__device__ __forceinline__ bool ldlt_pivots_ok_warp(const T* dinv, int n) {
  const int lane = threadIdx.x & 31;
  bool ok = true;
  for (int k = lane; k < n; k += 32) ok = ok && dinv[k] > T(0) && dinv[k] < T(INFINITY);
  return __all_sync(0xffffffffu, ok);
}

}  // namespace sapb
