// sapb_contact_solve.cuh -- fused SAP stage-2 Newton solve, one CTA per world.
//
// Restates SapContactSolve.solve (sim/contact_solve.py:6129-6285) as ONE
// persistent launch.  A CTA pulls a world index from a device counter, stages
// the world's contact Jacobian J in shared memory once, and runs prepare
// (:4285-4429), the Newton loop (:5474-5655) and the chosen line search
// (:2207-3175) on chip.  The dynamics matrix A is read through L1 (it is the
// only per-world array re-read from outside shared memory: twice a Newton
// iteration, for A dv and for the Hessian, from L1/L2).  Per line-search trial the kernel touches
// O(contacts + DOFs) data because the contact velocity along the search line
// is vc + alpha * (J dv) (vc is linear in v); the reference issues ~35
// launches per Newton iteration and re-reads A and J on every trial.
//
// Precision: the gradient, costs, line search, velocity update, the convergence
// test and the sums of the Hessian H = A + J^T G J + diag are FP64.  H is rounded
// once to HT (double, or float for the mixed path), in which its LDL^T
// factorization runs.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <type_traits>
#include <utility>

#include "sapb_device.cuh"
#include "sapb_internal.h"
#include "sapb_ldlt.cuh"
#include "sapb_linesearch.cuh"

namespace sapb {

struct SolveParams {
  sapb_contact_problem p;
  sapb_dof_terms dof;  // copy of *p.dof (has_pd/has_limits 0 if none)
  sapb_solve_options o;
  sapb_solve_outputs out;
  int32_t use_guess_flag_ptr_valid;
  int32_t* queue;      // work counter (zeroed before launch)
  // batches of per-world DOF counts in one launch per size class: this kernel
  // takes only its class (the runtime-size kernel the worlds of none)
  int32_t own_class_only;
};

// DOF counts with a specialised kernel: humanoid, quadruped, arm + box, one
// free body.
__host__ __device__ constexpr bool specialised_dofs(int n) { return n == 35 || n == 18 || n == 13 || n == 6; }

// Shared-memory layout of one world: the factorization's triangle list (of
// the kernel's largest world), the arrays sized by the world's DOFs alone --
// at compile-time offsets from one base in the specialised kernels, so that
// their addresses cost neither registers nor instructions -- then those sized
// by the contact slots.  ldJ and ldH odd: thread-per-row reads of J and column
// reads of H in the factorization are free of bank conflicts.
constexpr int kVecs = V_END;

__host__ __device__ constexpr size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct FixedLayout {
  int ps;  // one row of partial sums: up to eight chunks of n
  size_t off_scr, off_H, off_vec, off_flags, total;
};
// threads: of the CTA (the DOF products' partial sums hold one row per chunk)
__host__ __device__ constexpr FixedLayout fixed_layout(int n, int hsize, int threads) {
  FixedLayout L{};
  const size_t ld = n | 1;
  L.ps = n <= 8 || 8 * n > threads ? threads : 8 * n;
  size_t o = 0;
  L.off_scr = o;  // in turn: two rows of partial sums, the factorization's scaled panel
  const size_t sums = sizeof(double) * 2 * (size_t)L.ps, pan = (size_t)hsize * 8 * (n + 1);
  o = align_up(o + (sums > pan ? sums : pan), 16);
  L.off_H = o;  // n rows, then the right-hand side
  o = align_up(o + (size_t)hsize * (n + 1) * ld, 16);
  L.off_vec = o;
  o = align_up(o + sizeof(double) * (size_t)kVecs * ld, 16);
  L.off_flags = o;
  o = align_up(o + sizeof(int) * ld, 16);
  L.total = o;
  return L;
}

struct Layout {
  int n, C;
  size_t off_fixed, off_con, off_G, off_J, total;
};
__host__ __device__ inline Layout make_layout(int n, int C, int hsize, int threads = 128) {
  Layout L;
  L.n = n;
  L.C = C;
  const size_t Cc = C > 0 ? C : 1;
  size_t o = align_up(sizeof(uint16_t) * (size_t)triangle_list_size(n, 1), 16);  // the list, at 0
  L.off_fixed = o;
  // (a mixed batch's six-DOF worlds use their own fixed layout in this place)
  const size_t own = fixed_layout(n, hsize, threads).total, six = n > 6 ? fixed_layout(6, hsize, threads).total : 0;
  o += own > six ? own : six;
  L.off_con = o;
  o += sizeof(double) * C_END * Cc;
  L.off_G = o;  // (before the first evaluation: two staged impulse sets)
  o += sizeof(double) * 9 * Cc;
  L.off_J = o;
  L.total = align_up(o + sizeof(double) * (size_t)3 * C * (n | 1), 16);
  return L;
}

template <int NT, typename HT, int NS>
struct World {
  static constexpr int kCoefWarps = 1;  // warp 0 holds the line coefficients' shares
  int n_list, ps;   // DOFs of the triangle list; doubles in a row of partial sums
  const double* A;  // global, this world's [n][n]
  double* J;
  double* scr;      // scratch: partial sums or the scaled panel
  HT* H;
  double* G;        // [C][9]
  double* vec;
  double* con;
  int* flags;
  const uint16_t* tri;
  double* red;
  const double* scale;  // shared: the power of two that H and its right-hand sides carry (WorldScale)
  int* factor_ok;  // shared: whether the last Newton factorization's pivots were all positive and finite
  int n, count;
  // DOF count and leading dimensions: compile-time constants when NS > 0.
  __device__ __forceinline__ int dofs() const { return NS > 0 ? NS : n; }
  __device__ __forceinline__ int ldJ() const { return NS > 0 ? NS | 1 : n | 1; }
  __device__ __forceinline__ int ldH() const { return NS > 0 ? NS | 1 : n | 1; }
  // shift of the kernel's triangle list (built for L.n DOFs) to this world's n
  __device__ __forceinline__ int tri_shift() const { return n_list - dofs(); }
  __device__ __forceinline__ double* V(int k) const { return vec + k * ldJ(); }
  __device__ __forceinline__ double* cn(int c) const { return con + c * (int)C_END; }
  __device__ double* part(int which) const { return scr + which * ps; }
  __device__ ContactConst cc(int c) const {
    ContactConst x;
    x.rt = cn(c)[C_RT];
    x.rn = cn(c)[C_RN];
    x.rt_inv = cn(c)[C_RTINV];
    x.rn_inv = cn(c)[C_RNINV];
    x.vhat_n = cn(c)[C_VHAT];
    x.mu = cn(c)[C_MU];
    x.mu_hat = cn(c)[C_MUHAT];
    x.factor = cn(c)[C_FACTOR];
    return x;
  }
};

// The DOF products run on NT threads as (DOF i, chunk ch): thread t holds DOF
// t % n of chunk t / n, so consecutive threads read consecutive addresses and
// up to NT / n chunks of the summed index run side by side (35 DOFs: three
// chunks on 105 threads).
template <int NT, typename HT, int NS>
struct DofChunks {
  int i, ch, count;  // this thread's DOF and chunk (ch >= count: none), chunks
  __device__ __forceinline__ explicit DofChunks(const World<NT, HT, NS>& w) {
    const int n = w.dofs();
    count = NT / n < 8 ? NT / n : 8;
    ch = (int)threadIdx.x / n;
    i = (int)threadIdx.x - ch * n;
  }
  __device__ __forceinline__ bool active() const { return ch < count; }
};

// vc-type products: rows r < 3*count of J times x (length n, shared) into the
// contact slots `slot..slot+2`.  Two neighbouring threads per row, each half
// of the columns (20 contacts' rows are then one pass of 120 threads).
template <int NT, typename HT, int NS>
__device__ __forceinline__ void contact_rows_times(const World<NT, HT, NS>& w, const double* x, int slot) {
  const int n = w.dofs(), h = (n + 1) / 2;
  const int half = threadIdx.x & 1, j0 = half ? h : 0;
  const int items = 2 * 3 * w.count;
#pragma unroll 1
  for (int t0 = 0; t0 < items; t0 += NT) {
    const int t = t0 + (int)threadIdx.x, r = t >> 1;
    double s0 = 0.0, s1 = 0.0;
    if (t < items) {
      const double* row = w.J + r * w.ldJ() + j0;
      const double* xh = x + j0;
      int j = 0;
#pragma unroll 6
      for (; j + 1 < h - 1; j += 2) {
        s0 += row[j] * xh[j];
        s1 += row[j + 1] * xh[j + 1];
      }
      for (; j < h - (n & half); ++j) s0 += row[j] * xh[j];  // (odd n: the second half is one shorter)
      s0 += s1;
    }
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
    if (t < items && half == 0) {
      const int c = r / 3, k = r - 3 * c;
      w.cn(c)[slot + k] = s0;
    }
  }
}

// part(0) <- chunk sums of A x (x = V_DV), or of A (v - v*) with `residual`;
// part(1) <- chunk sums of A v* with `vstar_too`.
template <int NT, typename HT, int NS>
__device__ __forceinline__ void a_partials(const World<NT, HT, NS>& w, bool residual, bool vstar_too) {
  const DofChunks<NT, HT, NS> k(w);
  if (!k.active()) return;
  const int n = w.dofs();
  const int per = (n + k.count - 1) / k.count;
  const int j0 = k.ch * per, j1 = min(n, j0 + per);
  const double *x = w.V(residual ? V_V : V_DV), *vs = w.V(V_VSTAR);
  double a = 0.0, b = 0.0;
#pragma unroll 4
  for (int j = j0; j < j1; ++j) {
    const double aij = __ldg(w.A + (size_t)j * n + k.i);
    a += aij * (residual ? x[j] - vs[j] : x[j]);
    if (vstar_too) b += aij * vs[j];
  }
  w.part(0)[k.ch * n + k.i] = a;
  if (vstar_too) w.part(1)[k.ch * n + k.i] = b;
}

template <int NT, typename HT, int NS>
__device__ __forceinline__ double sum_partials(const World<NT, HT, NS>& w, int which, int i) {
  const int n = w.dofs(), nch = NT / n < 8 ? NT / n : 8;
  const double* p = w.part(which) + i;
  double s = p[0];
  for (int k = 1; k < nch; ++k) s += p[k * n];
  return s;
}

enum EvalStart { kEvalFull = 0, kEvalStep = 1, kEvalSame = 2 };

// vc and a_res, moved along line searches since they were formed, have to be
// formed again when v or v - v* has become small against what they went
// through.  Formed, their rounding errors are of the order of eps times
// |J| |v| and |A| |v - v*|; moved, they keep those of the largest v and v - v*
// on the way, and each step adds its own.  So the square of the largest size
// (in the norm of diag(A)) grows by half a step, and at sixteen times the
// present one -- a fourth of the size, or seven steps -- they are formed
// again: a start of the solution's size rarely gets there, one far from it (a
// poor guess or candidate) does so on its way in.  (From a guess 1e8 times too
// large the gradient at the returned velocity was 1e4 times the tolerance it
// was reported to meet when they were never formed again.)
constexpr double kSeenGrowth = 1.5, kSeenLimit = 16.0;

// Objective at the current v: contact impulses, costs and derivatives G,
// a_res = A(v - v*), J^T gamma, PD and limit terms, gradient (and its negative
// as the factorization's right-hand-side row).  Returns {cost, |g|^2, |p|^2,
// |jc|^2} (scaled, over participating DOFs), the momentum cost
// 1/2 (v - v*) a_res and whether the moved vc and a_res are too old
// (kSeenLimit) to every thread.  Restates _solver_update_active
// sim/contact_solve.py:4080-4136.
//
// kEvalFull forms vc = J v and a_res from V_V; kEvalStep moves v, vc and
// a_res by alpha times dv, J dv and A dv of the line search (all linear in v:
// a Newton step then reads neither A nor J here but for J^T gamma; kSeenLimit
// says when they are formed again); kEvalSame leaves them.  The first two warps hold the DOFs; of the others every second
// one projects the contacts for impulses and costs and the rest for the
// derivatives, side by side (the projection is a long dependent chain of few
// threads).
template <int NT, typename HT, int NS>
__device__ __forceinline__ void evaluate(const World<NT, HT, NS>& w, const SolveParams& P, double dt, int start,
                                         bool first, double alpha, double out4[4], double* mom,
                                         bool* too_old) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = NT / 32, kStride = 32 * (NW - 2) / 2;
  const int n = w.dofs();
  if (start == kEvalFull) {
    contact_rows_times<NT, HT, NS>(w, w.V(V_V), C_VC);
    a_partials<NT, HT, NS>(w, true, first);
    __syncthreads();
  }
  if (warp < 2) {
    if (tid < n) {
      if (start == kEvalFull) {
        w.V(V_ARES)[tid] = sum_partials<NT, HT, NS>(w, 0, tid);
        if (first) w.V(V_AVS)[tid] = sum_partials<NT, HT, NS>(w, 1, tid);
      } else if (start == kEvalStep) {
        w.V(V_V)[tid] += alpha * w.V(V_DV)[tid];
        w.V(V_ARES)[tid] += alpha * w.V(V_DP)[tid];
      }
    }
  } else {
    const bool derivs = warp & 1;
    double csum = 0.0;
#pragma unroll 1
    for (int c = 32 * ((warp - 2) >> 1) + lane; c < w.count; c += kStride) {
      double vc[3], g[3], cost, G[9];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        vc[k] = w.cn(c)[C_VC + k];
        if (start == kEvalStep) vc[k] += alpha * w.cn(c)[C_DVC + k];
      }
      if (derivs) {
        project_contact(w.cc(c), vc[0], vc[1], vc[2], g, &cost, G);
#pragma unroll
        for (int k = 0; k < 9; ++k) w.G[9 * c + k] = G[k];
      } else {
        project_contact(w.cc(c), vc[0], vc[1], vc[2], g, &cost, nullptr);
#pragma unroll
        for (int k = 0; k < 3; ++k) w.cn(c)[C_GAMMA + k] = g[k];
        csum += cost;
      }
    }
    if (!derivs) {
      csum = warp_sum<NT>(csum);
      if (lane == 0) w.red[kRedCost * NW + warp] = csum;
    }
  }
  __syncthreads();
  {  // J^T gamma over chunks of the contacts
    const DofChunks<NT, HT, NS> k(w);
    if (k.active()) {
      const int per = (w.count + k.count - 1) / k.count;
      const int c0 = k.ch * per, c1 = min(w.count, c0 + per);
      const int ld = w.ldJ();
      double g0 = 0.0, g1 = 0.0, g2 = 0.0;
      const double* Jc = w.J + 3 * c0 * ld + k.i;
#pragma unroll 2
      for (int c = c0; c < c1; ++c, Jc += 3 * ld) {
        g0 += Jc[0] * w.cn(c)[C_GAMMA + 0];
        g1 += Jc[ld] * w.cn(c)[C_GAMMA + 1];
        g2 += Jc[2 * ld] * w.cn(c)[C_GAMMA + 2];
      }
      w.part(0)[k.ch * n + k.i] = (g0 + g1) + g2;
    }
  }
  __syncthreads();
  if (warp == 0) {  // gradient and norms: two DOFs a lane
    double mterm = 0.0, extra = 0.0, g2 = 0.0, p2 = 0.0, j2 = 0.0;
    HT* rhs = w.H + n * w.ldH();
    const double scale = *w.scale;
#pragma unroll 1
    for (int i = lane; i < n; i += 32) {
      double imp = sum_partials<NT, HT, NS>(w, 0, i);
      const double a_res = w.V(V_ARES)[i], vi = w.V(V_V)[i];
      const double a_v = a_res + w.V(V_AVS)[i];
      mterm += 0.5 * (vi - w.V(V_VSTAR)[i]) * a_res;
      const int fl = w.flags[i];
      double pdg = 0.0, hd = 0.0;
      if (P.dof.has_pd && (fl & kFlagPd)) {
        const double gain = w.V(V_PDGAIN)[i], lim = w.V(V_PDLIM)[i];
        const double y = w.V(V_PDA)[i] - gain * vi;
        pdg = dt * clamp_limit(y, lim);
        hd += dt * gain * clamp_limit_derivative(y, lim);
        if (gain > 0.0) extra += (dt / gain) * clamp_limit_antiderivative(y, lim);
      }
      double lg = 0.0;
      if (P.dof.has_limits) {
        if (fl & kFlagLo) {
          const double g = w.V(V_LORINV)[i] * (w.V(V_LOVHAT)[i] - vi);
          if (g > 0.0) {
            lg += g;
            hd += w.V(V_LORINV)[i];
            extra += 0.5 * w.V(V_LOR)[i] * g * g;
          }
        }
        if (fl & kFlagUp) {
          const double g = w.V(V_UPRINV)[i] * (w.V(V_UPVHAT)[i] + vi);
          if (g > 0.0) {
            lg -= g;
            hd += w.V(V_UPRINV)[i];
            extra += 0.5 * w.V(V_UPR)[i] * g * g;
          }
        }
      }
      imp += pdg + lg;
      const double grad = a_res - imp;
      w.V(V_GRAD)[i] = grad;
      w.V(V_HDIAG)[i] = hd;
      rhs[i] = HT(-grad * scale);
      if (fl & kFlagPart) {
        const double s = w.V(V_DSCALE)[i];
        const double gs = s * grad, ps = s * a_v, js = s * imp;
        g2 += gs * gs;
        p2 += ps * ps;
        j2 += js * js;
      }
    }
    const double tot = warp_sum4(mterm, g2, p2, j2);
    double* r = w.red + kRedEval * NW;
    if ((lane & 7) == 0) r[lane >> 3] = tot;
    if (P.dof.has_pd || P.dof.has_limits) extra = warp_sum<NT>(extra);
    if (lane == 0) r[4] = extra;
  } else if (warp == 1) {  // the sizes of v and v - v*
    double sv = 0.0, sr = 0.0;
#pragma unroll 1
    for (int i = lane; i < n; i += 32) {
      const double vi = w.V(V_V)[i], ri = vi - w.V(V_VSTAR)[i], d = w.V(V_ADIAG)[i];
      sv += d * vi * vi;
      sr += d * ri * ri;
    }
    const double now = warp_sum4(sv, sr, 0.0, 0.0);
    double* r = w.red + kRedEval * NW;
    static_assert(8 <= (kRedSize - kRedEval) * NW, "the evaluation's sums");
    bool old = false;
    if (lane == 0 || lane == 8) {
      double* seen = r + 6 + (lane >> 3);
      const double m = start == kEvalFull ? now : (start == kEvalStep ? fmax(kSeenGrowth * *seen, now) : *seen);
      *seen = m;
      old = m > kSeenLimit * now;
    }
    old = __any_sync(0xffffffffu, old);
    if (lane == 0) r[5] = old ? 1.0 : 0.0;
  } else if (start == kEvalStep) {  // the moved contact velocities (their old ones are read)
#pragma unroll 1
    for (int q = tid - 64; q < 3 * w.count; q += NT - 64) {
      const int k = q / w.count, c = q - k * w.count;
      w.cn(c)[C_VC + k] += alpha * w.cn(c)[C_DVC + k];
    }
  }
  __syncthreads();
  const double* r = w.red + kRedEval * NW;
  double csum = 0.0;
#pragma unroll
  for (int q = 2; q < NW; q += 2) csum += w.red[kRedCost * NW + q];
  *mom = r[0];
  out4[0] = (csum + r[0]) + r[4];
  out4[1] = r[1];
  out4[2] = r[2];
  out4[3] = r[3];
  *too_old = r[5] != 0.0;
}

// H (lower triangle, HT) <- the lower triangle of the FP64 n x n matrix M in
// global memory, scaled: flat coalesced reads, four loads in flight per thread.
template <int NT, typename HT, int NS>
__device__ __forceinline__ void load_lower(const World<NT, HT, NS>& w, const double* M) {
  const int tid = threadIdx.x;
  const int n = w.dofs(), ldH = w.ldH();
  const int total = n * n;
  const double scale = *w.scale;
#pragma unroll 1
  for (int k0 = tid; k0 < total; k0 += 4 * NT) {
    double val[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = k0 + u * NT;
      val[u] = k < total ? __ldg(M + k) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = k0 + u * NT;
      if (k < total) {
        const int i = k / n, j = k - i * n;
        if (j <= i) w.H[(size_t)i * ldH + j] = HT(val[u] * scale);
      }
    }
  }
}

// One FP64 tensor-core product: c (8 x 8) += a (8 x 4) b (4 x 8).  Lane l
// holds a[l / 4][l % 4], b[l % 4][l / 4] and c[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void mma_f64(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

// The 8 x 8 blocks of H's lower triangle that a warp forms in one pass: Q0 of
// block column j0 and Q1 (0 or 1) of block column j1.
template <int Q0, int Q1>
struct HessBlocks {
  int i[Q0 + Q1], j0, j1;  // block rows (past the matrix: nothing to store)
};

// Adds J^T G J (k steps k0, k0 + dk, ...) to the accumulators of the warp's
// blocks.  The summed index is the contact row rho = 3 c + r, four rows a
// step: a = J^T, b = (G J)[rho] = sum_s G[3 rho + s] J[3 c + s] formed on the
// fly, once per block column.  Rows past 3 count enter with b = 0 (and a read
// from the last row); block rows and columns past n read the last column and
// are not stored.
template <int NT, typename HT, int NS, int Q0, int Q1>
__device__ __forceinline__ void hess_blocks(const World<NT, HT, NS>& w, const HessBlocks<Q0, Q1>& blk, int k0, int dk,
                                            double (&acc)[Q0 + Q1][2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, l4 = lane & 3;
  const int n = w.dofs(), ld = w.ldJ(), rows = 3 * w.count;
  int ca[Q0 + Q1];
#pragma unroll
  for (int q = 0; q < Q0 + Q1; ++q) ca[q] = min(8 * blk.i[q] + g, n - 1);
  const int c0 = min(8 * blk.j0 + g, n - 1), c1 = min(8 * blk.j1 + g, n - 1);
  const int steps = (rows + 3) / 4;
#pragma unroll 2
  for (int k = k0; k < steps; k += dk) {
    const int rho = 4 * k + l4;
    const bool live = rho < rows;
    const int rc = live ? rho : rows - 1;
    const double* Ja = w.J + rc * ld;
    const double* Jb = w.J + rc / 3 * 3 * ld;
    const double* Gr = w.G + 3 * rc;
    const double g0 = live ? Gr[0] : 0.0, g1 = live ? Gr[1] : 0.0, g2 = live ? Gr[2] : 0.0;
    const double b0 = g0 * Jb[c0] + g1 * Jb[ld + c0] + g2 * Jb[2 * ld + c0];
#pragma unroll
    for (int q = 0; q < Q0; ++q) mma_f64(acc[q][0], acc[q][1], Ja[ca[q]], b0);
    if (Q1 > 0) {
      const double b1 = g0 * Jb[c1] + g1 * Jb[ld + c1] + g2 * Jb[2 * ld + c1];
      mma_f64(acc[Q0 + Q1 - 1][0], acc[Q0 + Q1 - 1][1], Ja[ca[Q0 + Q1 - 1]], b1);
    }
  }
}

// H <- scale (A + J^T G J + diag) for the warp's blocks from its accumulators.
template <int NT, typename HT, int NS, int Q0, int Q1>
__device__ __forceinline__ void hess_store(const World<NT, HT, NS>& w, const HessBlocks<Q0, Q1>& blk,
                                           double diag_shift, const double (&acc)[Q0 + Q1][2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, l4 = lane & 3;
  const int n = w.dofs(), ldH = w.ldH();
  const double scale = *w.scale;
#pragma unroll
  for (int q = 0; q < Q0 + Q1; ++q) {
    const int i = 8 * blk.i[q] + g, j = 8 * (q < Q0 ? blk.j0 : blk.j1) + 2 * l4;
    if (i < n && j <= i) {
      const double* Ai = w.A + i * n + j;
      HT* Hi = w.H + i * ldH + j;
      const double hd = w.V(V_HDIAG)[i] + diag_shift;
      Hi[0] = HT((__ldg(Ai) + acc[q][0] + (i == j ? hd : 0.0)) * scale);
      if (j + 1 <= i) Hi[1] = HT((__ldg(Ai + 1) + acc[q][1] + (i == j + 1 ? hd : 0.0)) * scale);
    }
  }
}

template <int NT, typename HT, int NS, int Q0, int Q1>
__device__ __forceinline__ void hess_pass(const World<NT, HT, NS>& w, const HessBlocks<Q0, Q1>& blk,
                                          double diag_shift) {
  double acc[Q0 + Q1][2];
#pragma unroll
  for (int q = 0; q < Q0 + Q1; ++q) acc[q][0] = acc[q][1] = 0.0;
  hess_blocks<NT, HT, NS, Q0, Q1>(w, blk, 0, 1, acc);
  hess_store<NT, HT, NS, Q0, Q1>(w, blk, diag_shift, acc);
}

// H = A + J^T G J + diag(PD + limit + shift), lower triangle, from the
// derivatives G that evaluate() left: FP64 on the tensor cores
// (mma.m8n8k4), rounded once to HT.  Register tiles on the FP64 / FP32 cores
// took 11.6 k / 15.9 k cycles an iteration of 35 DOFs with three / four worlds
// per SM (20 contacts on average), the FP32 ones converting every element of
// J at the conversion unit's 16 a cycle.  Whole blocks per warp, so nothing is
// summed across warps, and the same code on every warp: the blocks are data.
// (A loop unrolled for each warp's blocks was 2000 instructions, which the
// instruction cache does not hold beside the rest of the Newton iteration.)
// 35 DOFs: 15 blocks as four warps' 3 + 1; up to 8 DOFs: the one block's
// contacts are split over the warps; else passes of one block pair.
template <int NT, typename HT, int NS>
__device__ __forceinline__ void assemble_hessian(const World<NT, HT, NS>& w, double diag_shift) {
  constexpr int NW = NT / 32;
  const int n = w.dofs(), nb = (n + 7) / 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (NS > 0 ? NS <= 8 : nb == 1) {
    double acc[1][2] = {{0.0, 0.0}};
    const HessBlocks<1, 0> blk{{0}, 0, 0};
    const int ks = min(NW, 2 * w.ps / 64);  // the scratch holds one block per warp
    double* p = w.scr;
    if (warp < ks) {
      hess_blocks<NT, HT, NS, 1, 0>(w, blk, warp, ks, acc);
      p[warp * 64 + 2 * lane] = acc[0][0];
      p[warp * 64 + 2 * lane + 1] = acc[0][1];
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        acc[0][u] = p[2 * lane + u];
        for (int q = 1; q < ks; ++q) acc[0][u] += p[q * 64 + 2 * lane + u];
      }
      hess_store<NT, HT, NS, 1, 0>(w, blk, diag_shift, acc);
    }
  } else if constexpr (NT == 128 && NS > 32 && NS <= 40) {
    // rows warp .. warp + 2 of column `warp`, and the blocks those leave:
    // (3, 0), (4, 1), (4, 0), (4, 4); warp 3's third row is past the matrix
    const HessBlocks<3, 1> blk{{warp, warp + 1, warp + 2, warp == 0 ? 3 : 4}, warp,
                               warp < 2 ? warp : (warp == 2 ? 0 : 4)};
    hess_pass<NT, HT, NS, 3, 1>(w, blk, diag_shift);
  } else {
    // block pairs (t, t + 1) in row order, (i, j) = row and column of block t
    const int nblk = nb * (nb + 1) / 2;
    auto row_of = [](int t) {
      int i = 0;
      while ((i + 1) * (i + 2) / 2 <= t) ++i;
      return i;
    };
#pragma unroll 1
    for (int t = 2 * warp; t < nblk; t += 2 * NW) {
      const int i0 = row_of(t), i1 = t + 1 < nblk ? row_of(t + 1) : nb;
      const HessBlocks<1, 1> blk{{i0, i1}, t - i0 * (i0 + 1) / 2, t + 1 < nblk ? t + 1 - i1 * (i1 + 1) / 2 : 0};
      hess_pass<NT, HT, NS, 1, 1>(w, blk, diag_shift);
    }
  }
  __syncthreads();
}

// Newton direction dv = -H^-1 grad: in-place LDL^T of the lower triangle of
// H (unit L stored below the diagonal unscaled as H_ik = L_ik d_k, D on the
// diagonal, 1/d_k in V_DINV) by the whole block with -grad carried as row n
// (its forward substitution is the factorization's own), then the backward
// substitution by warp 0.  Mathematically the Cholesky solve of the
// reference's BlockCholeskySolverBatched (sim/blocked_cholesky.py:414-604).
// A pivot that is not positive / finite makes dv NaN.
template <int NT, typename HT, int NS, int LB>
__device__ __forceinline__ void factor_and_solve(const World<NT, HT, NS>& w) {
  HT* dinv = reinterpret_cast<HT*>(w.V(V_DINV));
  ldlt_blocked<NT, HT, LB, 1, NS>(w.H, w.dofs(), w.ldH(), dinv, reinterpret_cast<HT*>(w.scr), w.tri, w.tri_shift());
  if ((threadIdx.x >> 5) == 0) {
    const bool ok = ldlt_backward_warp<HT, NS>(w.H, w.dofs(), w.ldH(), dinv, w.dofs(), w.V(V_DV));
    if (threadIdx.x == 0) *w.factor_ok = ok ? 1 : 0;
  }
  __syncthreads();
}

// out = -H^-1 rhs (vector slots) with the LDL^T in H and V_DINV, by warp
// `warp` alone (no block barrier).  A pivot that is not positive / finite
// makes out NaN.
template <int NT, typename HT, int NS>
__device__ void solve_warp(const World<NT, HT, NS>& w, int rhs_slot, int out_slot, int warp) {
  if ((threadIdx.x >> 5) == warp) {
    const HT* dinv = reinterpret_cast<const HT*>(w.V(V_DINV));
    const bool ok = ldlt_pivots_ok_warp<HT>(dinv, w.dofs());
    ldlt_solve_warp<HT>(w.H, w.dofs(), w.ldH(), dinv, w.V(rhs_slot), w.V(out_slot), true, ok);
  }
}

// Line coefficients (sim/contact_solve.py:2234-2263, 1657-1692): dp = A dv,
// dvc = J dv and warp 0's lanes' shares of {dell0, dell_a0, d2ell_a} (the
// line search sums them with its first trials).  One barrier: dvc and the
// partials are then published.
template <int NT, typename HT, int NS>
__device__ __forceinline__ void line_coefficients(const World<NT, HT, NS>& w, double (&cp)[3]) {
  contact_rows_times<NT, HT, NS>(w, w.V(V_DV), C_DVC);
  a_partials<NT, HT, NS>(w, false, false);
  __syncthreads();
  cp[0] = cp[1] = cp[2] = 0.0;
  if (threadIdx.x < 32) {
#pragma unroll 1
    for (int i = threadIdx.x; i < w.dofs(); i += 32) {
      const double acc = sum_partials<NT, HT, NS>(w, 0, i);
      const double dv = w.V(V_DV)[i];
      w.V(V_DP)[i] = acc;
      cp[0] += w.V(V_GRAD)[i] * dv;
      cp[1] += acc * (w.V(V_V)[i] - w.V(V_VSTAR)[i]);
      cp[2] += dv * acc;
    }
  }
}

// The powers of two by which a world's H is scaled, right-hand sides alike (so
// that directions are the same bits): 1, and where diag(A) comes near an end
// of the factor's type, away from it, so that pivots stay within pivot_recip's
// range.  (Always multiplied with: eight products a thread and iteration.)
template <typename HT>
struct WorldScale {
  static constexpr bool k64 = sizeof(HT) == 8;
  // 2^+-900 and 2^+-64, or 2^+-100 and 2^+-8
  static constexpr double kBig = k64 ? 8.452712498170644e270 : 1.2676506002282294e30;
  static constexpr double kUp = k64 ? 1.8446744073709552e19 : 256.0;
  static constexpr double kSmall = 1.0 / kBig, kDown = 1.0 / kUp;
};

constexpr int kMixed = -1;  // NS of the kernel that holds every size class's code
template <int NS> struct LdltBlocks { static constexpr int kCount = 1; static constexpr int kW[1] = {4}; };
template <> struct LdltBlocks<35> { static constexpr int kCount = 2; static constexpr int kW[2] = {5, 4}; };
template <> struct LdltBlocks<18> { static constexpr int kCount = 2; static constexpr int kW[2] = {6, 4}; };
template <> struct LdltBlocks<13> { static constexpr int kCount = 2; static constexpr int kW[2] = {4, 5}; };
template <> struct LdltBlocks<6> { static constexpr int kCount = 1; static constexpr int kW[1] = {6}; };

// One world of the persistent solve: stage its J and constants, the
// candidate starts, the Newton loop, the outputs.  NS: the world's DOF count
// at compile time (0: n_rt at run time); the arrays' slots (n_max DOFs) may
// hold more DOFs than the world has.
template <int NT, typename HT, int NS, int LSV, int LB>
__device__ __forceinline__ void solve_world(const SolveParams& P, const Layout& L, unsigned char* smem, double* red,
                                            unsigned long long& s_partmask, double& s_scale, int& s_factor_ok,
                                            const int e,
                                            const int n_max, const int n_rt, const bool use_guess) {
  const int tid = threadIdx.x;
  const int C = P.p.max_contacts;
  const int n = NS > 0 ? NS : n_rt;
  const FixedLayout F = fixed_layout(NS > 0 ? NS : n_max, (int)sizeof(HT), NT);
  unsigned char* fx = smem + L.off_fixed;
  World<NT, HT, NS> w{L.n,
                      F.ps,
                      P.p.dynamics_matrix + (size_t)e * n_max * n_max,
                      reinterpret_cast<double*>(smem + L.off_J),
                      reinterpret_cast<double*>(fx + F.off_scr),
                      reinterpret_cast<HT*>(fx + F.off_H),
                      reinterpret_cast<double*>(smem + L.off_G),
                      reinterpret_cast<double*>(fx + F.off_vec),
                      reinterpret_cast<double*>(smem + L.off_con),
                      reinterpret_cast<int*>(fx + F.off_flags),
                      reinterpret_cast<const uint16_t*>(smem),
                      red,
                      &s_scale,
                      &s_factor_ok,
                      n,
                      0};
  int count = P.p.contact_count[e];
  if (count > C) count = C;
  if (count < 0) count = 0;
  w.count = count;
  const double dt = P.p.dt[e];
  const size_t base = (size_t)e * n_max;

  // ---- stage J, per-contact constants and vectors -------------------------
  {
    const int rows = 3 * count;
    const double* Jg = P.p.jacobian + (size_t)e * C * 3 * n_max;
    const int ldj = w.ldJ();
    // Flat copy of the contiguous rows*n block by asynchronous 8-byte
    // copies (all in flight at once, completed before the barrier after the
    // per-DOF setup below; the rows land at stride ldj).
    const int total = rows * n;
#pragma unroll 4
    for (int k = tid; k < total; k += NT) {
      const int r = k / n, j = k - r * n;
      const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(w.J + (size_t)r * ldj + j));
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(Jg + k) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    // zero padding columns n..ldj-1
#pragma unroll 1
    for (int k = tid; k < rows * (ldj - n); k += NT) {
      const int r = k / (ldj - n), j = n + (k - r * (ldj - n));
      w.J[(size_t)r * ldj + j] = 0.0;
    }
#pragma unroll 1
    for (int c = tid; c < count; c += NT) {
      const size_t ci = (size_t)e * C + c;
      const double tau = P.p.tau_d ? P.p.tau_d[ci] : P.o.contact_tau_d;
      const ContactConst cc = make_contact_const(P.p.phi0[ci], P.p.w_eff[ci], P.p.mu[ci], P.p.stiffness[ci], tau,
                                                 P.o.contact_beta, P.o.contact_sigma, dt);
      w.cn(c)[C_RT] = cc.rt;
      w.cn(c)[C_RN] = cc.rn;
      w.cn(c)[C_RTINV] = cc.rt_inv;
      w.cn(c)[C_RNINV] = cc.rn_inv;
      w.cn(c)[C_VHAT] = cc.vhat_n;
      w.cn(c)[C_MU] = cc.mu;
      w.cn(c)[C_MUHAT] = cc.mu_hat;
      w.cn(c)[C_FACTOR] = cc.factor;
    }
#pragma unroll 1
    for (int i = tid; i < w.ldJ(); i += NT) {
      if (i < n) {
        w.V(V_VSTAR)[i] = P.p.v_star[base + i];
        double v = P.p.v0[base + i];
        if (P.p.v_guess) {
          if (use_guess) v = P.p.v_guess[base + i];
          P.p.v_guess[base + i] = v;
        }
        w.V(V_V)[i] = v;
        double d = __ldg(w.A + (size_t)i * n + i);
        if (d > 0.0 && d < WorldScale<HT>::kSmall) s_scale = WorldScale<HT>::kUp;  // (1 before; any thread)
        if (d < 1.0e-12 || !isfinite(d)) d = 1.0e-12;
        w.V(V_ADIAG)[i] = d;
        w.V(V_DSCALE)[i] = 1.0 / sqrt(d);
      } else {
        for (int k = 0; k < kVecs; ++k) w.V(k)[i] = 0.0;
      }
    }
  }
  // ---- PD and limit terms (sim/contact_solve.py:490-683) ------------------
#pragma unroll 1
  for (int i = tid; i < n; i += NT) {
    int fl = 0;
    const sapb_dof_terms& D = P.dof;
    // the per-DOF arrays: the solve's layout, or the model's global DOF order
    const size_t dof = D.world_dof_start ? (size_t)D.world_dof_start[e] + i : base + i;
    if (D.has_pd) {
      int coord = D.dof_coord_index[dof];
      if (coord >= D.joint_coord_count) coord = -1;
      int target = D.dof_target_index[dof];
      const int ndof = D.world_dof_start ? D.world_dof_start[P.p.num_envs] : P.p.num_envs * n_max;
      if (target < 0 || target >= ndof) target = (int)dof;
      if (D.joint_target_mode[target] != 0) {
        const double kp = (double)D.joint_target_ke[target], kd = (double)D.joint_target_kd[target];
        if (!(kp <= 0.0 && kd <= 0.0) && !(coord < 0 && kp > 0.0)) {
          double kpe, kde;
          effective_pd_gains(kp, kd, dt, 1.0 / w.V(V_ADIAG)[i], &kpe, &kde);
          const double gain = dt * kpe + kde;
          if (gain > 0.0) {
            double q0 = 0.0, qd = 0.0;
            if (coord >= 0) {
              q0 = D.joint_q[coord];
              qd = D.joint_target_pos ? (double)D.joint_target_pos[target] : 0.0;
            }
            const double vd = D.joint_target_vel ? (double)D.joint_target_vel[target] : 0.0;
            const double u0 = D.joint_act ? (double)D.joint_act[target] : 0.0;
            fl |= kFlagPd;
            w.V(V_PDA)[i] = kpe * (qd - q0) + kde * vd + u0;
            w.V(V_PDGAIN)[i] = gain;
            w.V(V_PDLIM)[i] = (double)D.joint_effort_limit[target];
          }
        }
      }
    }
    w.V(V_LOR)[i] = 1.0;
    w.V(V_UPR)[i] = 1.0;
    if (D.has_limits) {
      int coord = D.dof_coord_index[dof];
      if (coord >= D.joint_coord_count) coord = -1;
      const double ke = coord >= 0 ? D.joint_limit_ke[dof] : 0.0;
      if (coord >= 0 && D.limit_supported[dof] != 0 && ke > 0.0) {
        const double q0 = D.joint_q[coord];
        const double lower = D.joint_limit_lower[dof], upper = D.joint_limit_upper[dof];
        const double speed = fmax(fabs(P.p.v0[base + i]), fabs(w.V(V_VSTAR)[i]));
        const double window = kLimitWindow * dt * speed;
        const double kd = D.joint_limit_kd[dof];
        const double tau_d = kd > 0.0 ? kd / ke : 0.0;
        const double bf = kLimitBeta * kLimitBeta / (4.0 * kPi * kPi);
        const double r_nr = bf * fmax(1.0 / w.V(V_ADIAG)[i], 1.0e-12);
        const double r_soft = 1.0 / (dt * ke * (dt + tau_d));
        const double rr = fmax(r_nr, r_soft);
        if (isfinite(lower) && q0 - lower <= window) {
          fl |= kFlagLo;
          w.V(V_LOVHAT)[i] = -(q0 - lower) / (dt + tau_d);
          w.V(V_LOR)[i] = rr;
          w.V(V_LORINV)[i] = 1.0 / rr;
        }
        if (isfinite(upper) && upper - q0 <= window) {
          fl |= kFlagUp;
          w.V(V_UPVHAT)[i] = -(upper - q0) / (dt + tau_d);
          w.V(V_UPR)[i] = rr;
          w.V(V_UPRINV)[i] = 1.0 / rr;
        }
      }
    }
    w.flags[i] = fl;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");  // this thread's J copies
  __syncthreads();
  // ---- participating DOFs (sim/contact_solve.py:423-488) ------------------
  // A DOF takes part if a model term acts on it or a contact's body DOF
  // range or J column covers it.  The contacts mark their DOFs in a 64-bit
  // mask in parallel (n <= 60 here).
  if (tid == 0) s_partmask = 0ull;
  __syncthreads();
#pragma unroll 1
  for (int c = tid; c < count; c += NT) {
    const size_t ci = (size_t)e * C + c;
    unsigned long long mk = 0ull;
    if (P.p.body_dof_start) {
      const int bs[2] = {P.p.body0 ? P.p.body0[ci] : -1, P.p.body1 ? P.p.body1[ci] : -1};
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int b = bs[q];
        if (b < 0 || b >= P.p.num_bodies) continue;
        const int s = P.p.body_dof_start[b], m = P.p.body_dof_count[b];
        if (s < 0 || m <= 0 || s >= n) continue;
        const int hi = s + m < n ? s + m : n;
        mk |= ((1ull << (hi - s)) - 1ull) << s;
      }
    }
    const double* Jc = w.J + (size_t)(3 * c) * w.ldJ();
    if (mk != (1ull << n) - 1ull)
#pragma unroll 1
      for (int j = 0; j < n; ++j)
        if (Jc[j] != 0.0 || Jc[w.ldJ() + j] != 0.0 || Jc[2 * w.ldJ() + j] != 0.0) mk |= 1ull << j;
    atomicOr(&s_partmask, mk);
  }
  __syncthreads();
  int any_model_term = 0;
#pragma unroll 1
  for (int i = tid; i < n; i += NT) {
    const int model = (w.flags[i] & (kFlagPd | kFlagLo | kFlagUp)) ? 1 : 0;
    any_model_term |= model;
    if (model || ((s_partmask >> i) & 1ull)) w.flags[i] |= kFlagPart;
    if (w.V(V_ADIAG)[i] > WorldScale<HT>::kBig) s_scale = WorldScale<HT>::kDown;
  }
  const int model_terms = __syncthreads_or(any_model_term);
  const bool unconstrained = (count == 0) && !model_terms;
  // ---- input check: a NaN / Inf in A, J, the contact parameters, v* or
  // the start velocity leaves the world unsolved (SAPB_WORLD_NOT_FINITE)
  // (by the exponent bits; J as it lies, padding columns zero)
  bool bad = false;
  auto exponent_full = [](int hi) { return (hi & 0x7ff00000) == 0x7ff00000; };
#pragma unroll 5
  for (int k = tid; k < n * n; k += NT) bad |= exponent_full(__double2hiint(__ldg(w.A + k)));
  {
    const int* hi = reinterpret_cast<const int*>(w.J) + 1;
    const int tot = 3 * count * w.ldJ();
#pragma unroll 4
    for (int k = tid; k < tot; k += NT) bad |= exponent_full(hi[2 * k]);
  }
#pragma unroll 1
  for (int c = tid; c < count; c += NT) {
    const size_t ci = (size_t)e * C + c;
    if (!isfinite(P.p.phi0[ci]) || !isfinite(P.p.w_eff[ci]) || !isfinite(P.p.mu[ci]) ||
        !isfinite(P.p.stiffness[ci]) || (P.p.tau_d && !isfinite(P.p.tau_d[ci])))
      bad = true;
  }
#pragma unroll 1
  for (int i = tid; i < n; i += NT)
    if (!isfinite(w.V(V_VSTAR)[i]) || !isfinite(w.V(V_V)[i])) bad = true;
  const bool not_finite = __syncthreads_or(bad) != 0;

  int newton_iterations = 0, ls_total = 0, converged = 0, status = 0;
  double cost = 0.0, previous_cost = 0.0, alpha = 1.0, grad_norm = 0.0;
  int ws_accepted = 0;
  bool evaluated = false;
  if (not_finite) {
    status = SAPB_WORLD_NOT_FINITE;  // v stays the start velocity
  } else if (unconstrained) {
    converged = 1;
#pragma unroll 1
    for (int i = tid; i < n; i += NT) w.V(V_V)[i] = w.V(V_VSTAR)[i];
    __syncthreads();
  } else {
#pragma unroll 1
    for (int i = tid; i < n; i += NT)
      if (!(w.flags[i] & kFlagPart)) w.V(V_V)[i] = w.V(V_VSTAR)[i];
    __syncthreads();
    // Candidate starts (no counterpart in the reference): v_candidate_count
    // start velocities, then gamma0_count impulse sets with v_c = base +
    // A^-1 J^T gamma_c (base v* or gamma0_base), each taken on the
    // participating DOFs (v* on the others), A factored once in this
    // kernel's factor precision or read from the free motion's factor;
    // the start with the lowest cost among the plain start (unless skipped)
    // and the candidates is taken.  Its evaluation seeds iteration 0 when it
    // was the last one evaluated.  One loop evaluates the starts and the
    // Newton iterates alike, so the kernel holds one copy of the evaluation.
    const int KV = P.p.v_candidates ? (P.p.v_candidate_count > 1 ? P.p.v_candidate_count : 1) : 0;
    const int KG = P.p.gamma0 ? (P.p.gamma0_count > 1 ? P.p.gamma0_count : 1) : 0;
    int last_start = KV + KG;  // start 0: the plain one; 1 .. KV: velocities; then the impulse sets
    int start = -1;            // the start under trial; -1: Newton
    bool last_is_best = false, zero_sets = false;
    // the plain start competes unless the caller skips it; it stays the
    // fallback when no candidate's cost is finite
    double best_cost = 1.0e300;
    if (last_start > 0 && count > 0) {
#pragma unroll 1
      for (int i = tid; i < n; i += NT) w.V(V_SAVE)[i] = w.V(V_V)[i];
      start = P.o.skip_plain_start ? 1 : 0;
    }
    const double cost_min_alpha = LSV == SAPB_LS_MONOTONE_DECAY ? 0.0 : 0.5;
    int it = 0, from = kEvalFull;
    bool first = true;
    for (;;) {
      if (start > 0) {  // V(V_V) <- this start
        __syncthreads();
        if (start <= KV) {
          const double* vk = P.p.v_candidates + ((size_t)(start - 1) * P.p.num_envs + e) * n_max;
#pragma unroll 1
          for (int i = tid; i < n; i += NT)
            w.V(V_V)[i] = (w.flags[i] & kFlagPart) ? __ldg(vk + i) : w.V(V_VSTAR)[i];
        } else {
          const double* base_g = P.p.gamma0_base ? P.p.gamma0_base + (size_t)e * n_max : nullptr;
          const int kg = start - KV - 1;
          if (kg == 0) {
            // a world whose candidate impulses are all zero starts at the base
            int nz = 0;
#pragma unroll 1
            for (int q = tid; q < KG * 3 * count; q += NT) {
              const int kk = q / (3 * count), r = q - kk * 3 * count;
              if (__ldg(P.p.gamma0 + ((size_t)kk * P.p.num_envs + e) * C * 3 + r) != 0.0) nz = 1;
            }
            zero_sets = !__syncthreads_or(nz);
            if (zero_sets) {
              last_start = start;
            } else {
              HT* dinv = reinterpret_cast<HT*>(w.V(V_DINV));
              if (P.p.dynamics_factor) {
                // the free motion's LDL^T of A
                const double* Lg = P.p.dynamics_factor + (size_t)e * n_max * n_max;
                load_lower<NT, HT, NS>(w, Lg);
#pragma unroll 1
                for (int i = tid; i < n; i += NT) dinv[i] = fast_recip(HT(__ldg(Lg + (size_t)i * n + i) * s_scale));
              } else {
                load_lower<NT, HT, NS>(w, w.A);
                __syncthreads();
                ldlt_blocked<NT, HT, LB, 1, 0>(w.H, n, w.ldH(), dinv, reinterpret_cast<HT*>(w.scr), w.tri,
                                               w.tri_shift());  // the factor of A (row n rides along unread)
              }
            }
          }
          if (zero_sets) {
#pragma unroll 1
            for (int i = tid; i < n; i += NT)
              w.V(V_V)[i] = (w.flags[i] & kFlagPart) && base_g ? __ldg(base_g + i) : w.V(V_VSTAR)[i];
          } else {
            // Two sets at a time: stage their impulses in the place of G (the
            // next evaluation writes it), form J^T gamma for both (threads 0-63 set kg, 64-127
            // set kg+1) and solve both with the factor on warps 0 and 1.
            if (kg % 2 == 0) {
              const int ldj = w.ldJ();
              double* gs = w.G;
              const int nk = KG - kg < 2 ? KG - kg : 2;
              __syncthreads();
#pragma unroll 1
              for (int q = tid; q < nk * 3 * count; q += NT) {
                const int kk = q / (3 * count), r = q - kk * 3 * count;
                gs[q] = __ldg(P.p.gamma0 + ((size_t)(kg + kk) * P.p.num_envs + e) * C * 3 + r);
              }
              __syncthreads();
              {
                const int kk = tid >> 6, i = tid & 63;
                if (kk < nk && i < n) {
                  const double* g = gs + kk * 3 * count;
                  double acc = 0.0;
#pragma unroll 1
                  for (int c = 0; c < count; ++c) {
                    const double* Jc = w.J + (size_t)(3 * c) * ldj;
                    acc += Jc[i] * g[3 * c] + Jc[ldj + i] * g[3 * c + 1] + Jc[2 * ldj + i] * g[3 * c + 2];
                  }
                  w.V(kk == 0 ? V_GRAD : V_DP)[i] = -acc * *w.scale;  // the solves give -H^-1 rhs
                }
              }
              __syncthreads();
              solve_warp<NT, HT, NS>(w, V_GRAD, V_DV, 0);
              if (nk > 1) solve_warp<NT, HT, NS>(w, V_DP, V_DP, 1);  // in place
              __syncthreads();
            }
            const double* dvk = w.V(kg % 2 == 0 ? V_DV : V_DP);
#pragma unroll 1
            for (int i = tid; i < n; i += NT)
              w.V(V_V)[i] = (w.flags[i] & kFlagPart) ? (base_g ? __ldg(base_g + i) : w.V(V_VSTAR)[i]) + dvk[i]
                                                     : w.V(V_VSTAR)[i];
          }
        }
        __syncthreads();
      }
      double e4[4], mom;
      bool too_old;
      evaluate<NT, HT, NS>(w, P, dt, from, first, alpha, e4, &mom, &too_old);
      first = false;
      if (too_old) {
        from = kEvalFull;
        continue;
      }
      if (start >= 0) {
        if (start == 0) {
          best_cost = e4[0];
        } else {
          last_is_best = e4[0] < best_cost;
          if (last_is_best) {
            best_cost = e4[0];
            ws_accepted = start;
#pragma unroll 1
            for (int i = tid; i < n; i += NT) w.V(V_BEST)[i] = w.V(V_V)[i];
          }
        }
        if (start < last_start) {
          ++start;
          continue;
        }
        start = -1;
        if (!last_is_best) {
          __syncthreads();
          const int src = ws_accepted > 0 ? V_BEST : V_SAVE;
#pragma unroll 1
          for (int i = tid; i < n; i += NT) w.V(V_V)[i] = w.V(src)[i];
          __syncthreads();
          continue;
        }
      }
      evaluated = true;
      cost = e4[0];
      // convergence test (sim/contact_solve.py:2043-2087)
      const double gn = sqrt(fmax(e4[1], 0.0)), pn = sqrt(fmax(e4[2], 0.0)), jn = sqrt(fmax(e4[3], 0.0));
      grad_norm = gn;
      const double opt_tol = P.o.optimality_abs_tol + P.o.optimality_rel_tol * fmax(pn, jn);
      const bool opt = gn <= opt_tol;
      bool cost_ok = false;
      if (it > 0 && alpha > cost_min_alpha) {
        const double sc = 0.5 * (fabs(cost) + fabs(previous_cost));
        const double tol = P.o.cost_abs_tol + P.o.cost_rel_tol * sc;
        if (fabs(cost - previous_cost) < tol) cost_ok = true;
      }
      newton_iterations = it;
      if (opt || cost_ok) {
        converged = 1;
        break;
      }
      if (it >= P.o.max_iterations) break;
      converged = 0;
      // Newton direction
      assemble_hessian<NT, HT, NS>(w, P.o.diag_shift);
      factor_and_solve<NT, HT, NS, LB>(w);
      if (!*w.factor_ok) {  // H not SPD (uniform: published by the barrier above)
        status = SAPB_WORLD_NOT_SPD;
        converged = 0;
        break;
      }
      LsResult r;
      double cp[3];
      line_coefficients<NT, HT, NS>(w, cp);
      if constexpr (LSV == SAPB_LS_ARMIJO_DECAY)
        r = ls_armijo<NT, 1>(w, P, dt, cost, cp, mom);
      else if constexpr (LSV == SAPB_LS_EXACT_ROOT)
        r = ls_exact<NT>(w, P, dt, cost, cp, mom);
      else
        r = ls_monotone<NT, 1>(w, P, dt, cost, cp, mom);
      alpha = r.alpha;
      status = r.status;
      constexpr bool mono = LSV == SAPB_LS_MONOTONE_DECAY;
      if (r.accepted || mono) {
        ls_total += r.iterations;
        previous_cost = cost;
      }
      from = r.accepted ? kEvalStep : kEvalSame;
      ++it;
    }
  }
  // ---- outputs ------------------------------------------------------------
#pragma unroll 1
  for (int i = tid; i < n_max; i += NT) P.out.v[base + i] = i < n ? w.V(V_V)[i] : 0.0;
#pragma unroll 1
  for (int c = tid; c < C; c += NT) {
    const size_t ci = (size_t)e * C + c;
    const bool live = evaluated && c < count;
    if (P.out.contact_gamma) {
      P.out.contact_gamma[ci * 3 + 0] = live ? w.cn(c)[C_GAMMA + 0] : 0.0;
      P.out.contact_gamma[ci * 3 + 1] = live ? w.cn(c)[C_GAMMA + 1] : 0.0;
      P.out.contact_gamma[ci * 3 + 2] = live ? w.cn(c)[C_GAMMA + 2] : 0.0;
    }
    if (P.out.contact_mode) {
      int mode = SAPB_CONTACT_MODE_NONE;
      if (live) {
        double g[3], cst;
        mode = project_contact(w.cc(c), w.cn(c)[C_VC + 0], w.cn(c)[C_VC + 1], w.cn(c)[C_VC + 2], g, &cst, nullptr);
      }
      P.out.contact_mode[ci] = mode;
    }
  }
  if (tid == 0) {
    if (P.out.cost) P.out.cost[e] = evaluated ? cost : 0.0;
    if (P.out.newton_iterations) P.out.newton_iterations[e] = newton_iterations;
    if (P.out.line_search_iterations) P.out.line_search_iterations[e] = ls_total;
    if (P.out.converged) P.out.converged[e] = converged;
    if (P.out.status) P.out.status[e] = status;
    if (P.out.grad_norm) P.out.grad_norm[e] = grad_norm;
    if (P.out.warm_start_accepted) P.out.warm_start_accepted[e] = ws_accepted;
  }
  __syncthreads();
}

// LSV: the line search, fixed at compile time (SAPB_LS_ARMIJO_DECAY,
// SAPB_LS_EXACT_ROOT or SAPB_LS_MONOTONE_DECAY) so that one instantiation
// holds the code of one search only (smaller instruction footprint).  LB:
// the column-block width of the LDL^T factorization (a variant the
// autotuner chooses: the best width depends on the DOF count).
template <int NT, typename HT, int MINB, int NS, int LSV, int LB>
__global__ void __launch_bounds__(NT, MINB) contact_solve_kernel(const SolveParams P) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[kRedSize * (NT / 32)];
  __shared__ int s_next;
  __shared__ unsigned long long s_partmask;
  __shared__ double s_scale;
  __shared__ int s_factor_ok;
  const int tid = threadIdx.x;
  // n_max: the DOF slots of a world in the arrays; a world's own DOF count may
  // be smaller (dof_count), its arrays compact at the start of its slots
  const int n_max = P.p.dof_per_env, C = P.p.max_contacts;
  const Layout L = make_layout(NS > 0 ? NS : n_max, C, (int)sizeof(HT), NT);
  const bool use_guess = P.use_guess_flag_ptr_valid && P.p.v_guess_active[0] != 0;
  build_triangle_list<NT>(reinterpret_cast<uint16_t*>(smem), L.n, 1);
  // the DOFs of world e, and whether it is this launch's
  auto dofs_of = [&](int e) {
    if (!P.p.dof_count) return n_max;
    const int d = P.p.dof_count[e];
    return d < 1 ? 1 : (d > n_max ? n_max : d);
  };
  auto takes = [&](int d) { return !P.own_class_only || (NS > 0 ? d == NS : !specialised_dofs(d)); };

  if (tid == 0) s_next = atomicAdd(P.queue, 1);
  for (;;) {
    // Take the prefetched index, claim the next world and warm L2 with its A
    // and J (prefetch.global.L2 is a hint and has no alignment rule).
    __syncthreads();
    const int ticket = s_next;
    if (ticket >= P.p.num_envs) break;
    const int e = P.p.world_order ? P.p.world_order[ticket] : ticket;
    __syncthreads();
    if (tid == 0) {
      s_next = atomicAdd(P.queue, 1);
      s_scale = 1.0;
    }
    __syncthreads();
    if (e < 0 || e >= P.p.num_envs) continue;
    const int n_world = dofs_of(e);
    if (!takes(n_world)) continue;
    {
      const int nt = s_next;
      const int nx = nt < P.p.num_envs ? (P.p.world_order ? P.p.world_order[nt] : nt) : P.p.num_envs;
      if (nx >= 0 && nx < P.p.num_envs && takes(dofs_of(nx))) {
        const char* a0 = reinterpret_cast<const char*>(P.p.dynamics_matrix + (size_t)nx * n_max * n_max);
        const size_t abytes = sizeof(double) * (size_t)n_max * n_max;
        int cnt = P.p.contact_count[nx];
        cnt = cnt < 0 ? 0 : (cnt > C ? C : cnt);
        const char* j0 = reinterpret_cast<const char*>(P.p.jacobian + (size_t)nx * C * 3 * n_max);
        const size_t jbytes = sizeof(double) * (size_t)cnt * 3 * n_max;
        for (size_t off = (size_t)tid * 128; off < abytes; off += (size_t)NT * 128)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(a0 + off));
        for (size_t off = (size_t)tid * 128; off < jbytes; off += (size_t)NT * 128)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(j0 + off));
        if (P.p.v_candidates) {
          const int KV = P.p.v_candidate_count > 1 ? P.p.v_candidate_count : 1;
          const size_t vbytes = sizeof(double) * (size_t)n_max;
          for (int k = 0; k < KV; ++k) {
            const char* v0p =
                reinterpret_cast<const char*>(P.p.v_candidates + ((size_t)k * P.p.num_envs + nx) * n_max);
            for (size_t off = (size_t)tid * 128; off < vbytes; off += (size_t)NT * 128)
              asm volatile("prefetch.global.L2 [%0];" ::"l"(v0p + off));
          }
        }
        if (P.p.gamma0) {
          if (P.p.dynamics_factor) {
            const char* f0 = reinterpret_cast<const char*>(P.p.dynamics_factor + (size_t)nx * n_max * n_max);
            for (size_t off = (size_t)tid * 128; off < abytes; off += (size_t)NT * 128)
              asm volatile("prefetch.global.L2 [%0];" ::"l"(f0 + off));
          }
          const int K = P.p.gamma0_count > 1 ? P.p.gamma0_count : 1;
          const size_t gbytes = sizeof(double) * (size_t)cnt * 3;
          for (int k = 0; k < K; ++k) {
            const char* g0 = reinterpret_cast<const char*>(P.p.gamma0 + ((size_t)k * P.p.num_envs + nx) * C * 3);
            for (size_t off = (size_t)tid * 128; off < gbytes; off += (size_t)NT * 128)
              asm volatile("prefetch.global.L2 [%0];" ::"l"(g0 + off));
          }
        }
      }
    }

    if constexpr (NS == kMixed) {
      // each world's own DOF count: the specialised code of its size class
#define SAPB_CLASS(N)                                                                                              \
  case N:                                                                                                          \
    solve_world<NT, HT, N, LSV, LdltBlocks<N>::kW[0]>(P, L, smem, red, s_partmask, s_scale, s_factor_ok, e, n_max, N, use_guess); \
    break;
      switch (n_world) {
        SAPB_CLASS(35)
        SAPB_CLASS(18)
        SAPB_CLASS(13)
        SAPB_CLASS(6)
        default:
          solve_world<NT, HT, 0, LSV, LB>(P, L, smem, red, s_partmask, s_scale, s_factor_ok, e, n_max, n_world, use_guess);
      }
#undef SAPB_CLASS
    } else {
      solve_world<NT, HT, NS, LSV, LB>(P, L, smem, red, s_partmask, s_scale, s_factor_ok, e, n_max, n_world, use_guess);
    }
  }
}

template <int NT, typename HT, int MINB, int NS, int LSV, int LB>
cudaError_t launch_solve_ls(const SolveParams& P, cudaStream_t stream, int* blocks_out) {
  const Layout L = make_layout(NS > 0 ? NS : P.p.dof_per_env, P.p.max_contacts, (int)sizeof(HT), NT);
  auto kern = contact_solve_kernel<NT, HT, MINB, NS, LSV, LB>;
  cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.total);
  if (err != cudaSuccess) return err;
  int dev = 0;
  err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  int sms = 0;
  err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (err != cudaSuccess) return err;
  int per_sm = 0;
  err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, L.total);
  if (err != cudaSuccess) return err;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  if (blocks_out && P.p.num_envs == 0) {  // occupancy query only
    *blocks_out = per_sm;
    return cudaSuccess;
  }
  const int k = (P.o.ctas_per_sm > 0 && P.o.ctas_per_sm < per_sm) ? P.o.ctas_per_sm : per_sm;
  int blocks = sms * k;
  if (blocks > P.p.num_envs) blocks = P.p.num_envs;
  if (blocks < 1) blocks = 1;
  if (blocks_out) *blocks_out = blocks;
  kern<<<blocks, NT, L.total, stream>>>(P);
  return cudaGetLastError();
}

template <int NT, typename HT, int MINB, int NS, int LB>
static cudaError_t launch_solve(const SolveParams& P, cudaStream_t stream, int* blocks_out) {
  switch (P.o.line_search_variant) {
    case SAPB_LS_ARMIJO_DECAY:
      return launch_solve_ls<NT, HT, MINB, NS, SAPB_LS_ARMIJO_DECAY, LB>(P, stream, blocks_out);
    case SAPB_LS_EXACT_ROOT:
      return launch_solve_ls<NT, HT, MINB, NS, SAPB_LS_EXACT_ROOT, LB>(P, stream, blocks_out);
    default:
      return launch_solve_ls<NT, HT, MINB, NS, SAPB_LS_MONOTONE_DECAY, LB>(P, stream, blocks_out);
  }
}

// LDL^T block widths instantiated per DOF specialisation (the first is the
// default), from measurements on B200: 35 DOFs = 7 blocks of 5 is fastest
// in both precisions; wider blocks lengthen the serial diagonal chain and
// the register block, narrower ones add barriers.

// One Hessian precision of the kernels of one DOF specialisation NS (every
// line search, every LDL^T block width), instantiated in a translation unit
// of its own (sapb_solve_n*_f32.cu / _f64.cu) so they compile in parallel.
template <int NS, bool FP32>
cudaError_t launch_solve_np(const SolveParams& P, cudaStream_t stream, int* blocks_out) {
  using HT = typename std::conditional<FP32, float, double>::type;
  constexpr int MINB = FP32 ? 4 : 3;
  if constexpr (LdltBlocks<NS>::kCount > 1) {
    if (P.o.ldlt_block == LdltBlocks<NS>::kW[1])
      return launch_solve<128, HT, MINB, NS, LdltBlocks<NS>::kW[LdltBlocks<NS>::kCount > 1 ? 1 : 0]>(P, stream,
                                                                                                      blocks_out);
  }
  return launch_solve<128, HT, MINB, NS, LdltBlocks<NS>::kW[0]>(P, stream, blocks_out);  // the default (0 or unknown)
}

template <int NS>
inline cudaError_t launch_solve_ns(const SolveParams& P, bool fp32, cudaStream_t stream, int* blocks_out) {
  return fp32 ? launch_solve_np<NS, true>(P, stream, blocks_out) : launch_solve_np<NS, false>(P, stream, blocks_out);
}

// The runtime-size kernel with 256 threads (eight warps) per world, the
// default LDL^T width: on request (sapb_solve_options.threads_per_cta = 256), and
// by itself for worlds without a specialised kernel whose shared memory leaves
// one CTA per SM (solve_dispatch); instantiated in sapb_solve_nwide_f32.cu /
// _f64.cu.
template <bool FP32>
cudaError_t launch_solve_wide(const SolveParams& P, cudaStream_t stream, int* blocks_out) {
  using HT = typename std::conditional<FP32, float, double>::type;
  return launch_solve<256, HT, FP32 ? 2 : 1, 0, LdltBlocks<0>::kW[0]>(P, stream, blocks_out);
}
extern template cudaError_t launch_solve_wide<true>(const SolveParams&, cudaStream_t, int*);
extern template cudaError_t launch_solve_wide<false>(const SolveParams&, cudaStream_t, int*);

// The runtime-size kernels (128 and 256 threads) are the largest: each line
// search's kernel is instantiated in a translation unit of its own
// (sapb_solve_n{generic,mixed,wide}_f{32,64}_{armijo,exact,monotone}.cu).
#define SAPB_RUNTIME_SIZE_KERNELS(X, LSV)                                         \
  X(128, float, 4, 0, LSV, LdltBlocks<0>::kW[0])                                \
  X(128, double, 3, 0, LSV, LdltBlocks<0>::kW[0])                               \
  X(128, float, 4, kMixed, LSV, LdltBlocks<0>::kW[0])                           \
  X(128, double, 3, kMixed, LSV, LdltBlocks<0>::kW[0])                          \
  X(256, float, 2, 0, LSV, LdltBlocks<0>::kW[0])                                \
  X(256, double, 1, 0, LSV, LdltBlocks<0>::kW[0])
#define SAPB_EXTERN_LS(NT, HT, MINB, NS, LSV, LB) \
  extern template cudaError_t launch_solve_ls<NT, HT, MINB, NS, LSV, LB>(const SolveParams&, cudaStream_t, int*);
SAPB_RUNTIME_SIZE_KERNELS(SAPB_EXTERN_LS, SAPB_LS_ARMIJO_DECAY)
SAPB_RUNTIME_SIZE_KERNELS(SAPB_EXTERN_LS, SAPB_LS_EXACT_ROOT)
SAPB_RUNTIME_SIZE_KERNELS(SAPB_EXTERN_LS, SAPB_LS_MONOTONE_DECAY)
#undef SAPB_EXTERN_LS

#define SAPB_EXTERN_SOLVE(NS)                                                                  \
  extern template cudaError_t launch_solve_np<NS, true>(const SolveParams&, cudaStream_t, int*); \
  extern template cudaError_t launch_solve_np<NS, false>(const SolveParams&, cudaStream_t, int*);
SAPB_EXTERN_SOLVE(35)
SAPB_EXTERN_SOLVE(18)
SAPB_EXTERN_SOLVE(13)
SAPB_EXTERN_SOLVE(6)
SAPB_EXTERN_SOLVE(0)
SAPB_EXTERN_SOLVE(kMixed)
#undef SAPB_EXTERN_SOLVE

}  // namespace sapb

