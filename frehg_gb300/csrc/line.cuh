// Vertical line (column) preconditioner for the FP32 inner solve (not in reference).
//
// The scaled operator A~ = I + couplings is dominated by its vertical couplings (dz << dx, dy:
// the axis-2 transmissibility is (dx/dz)^2 = 400x the lateral one on 1 m x 1 m x 5 cm cells),
// which is what makes Jacobi-PCG slow.  M = blockdiag over columns of the tridiagonal part of A~
// (its axis-2 couplings and unit diagonal) is SPD whenever A~ is (principal submatrices), and
// M^-1 r is one Thomas solve per column.  Each thread owns one column; cells of a column are
// n0*n1 apart, so a warp's loads at one level are consecutive (coalesced).
//
// Factorisation (once per solve, FP64, stored FP32): M_col = L D L^T with unit lower
// bidiagonal L,
//   d_0 = 1,  l_k = a2_{k-1} / d_{k-1},  d_k = 1 - l_k a2_{k-1}      (l_0 = 0)
// Solve: y_k = r_k - l_k y_{k-1};  u_k = y_k / d_k;  z_k = u_k - l_{k+1} z_{k+1}.
// r . z = sum_k y_k^2 / d_k = sum_k y_k u_k comes out of the forward sweep, so the backward
// sweep needs neither r nor a reduction and can form the next search direction in place.
//
// PCG iteration, two kernels:
//   k32_dir_spmv(_v4) : p = z + beta p_old and w = A~ p in one pass (the neighbours' directions are
//                       formed again from z and p_old, so p goes from one buffer into the other),
//                       alpha = (r.z) / (p.w)
//   k32_line_step     : x += alpha p, r -= alpha w, z = M^-1 r with both sweeps, r.z, r.r, test, beta
#pragma once

#include "internal.h"
#include "reduce.cuh"

#include <algorithm>

namespace fg {

// The inner solve's tolerance in a refinement sweep whose true residual is rn (target: the
// refinement's own).  A sweep that can end the refinement aims at it: kSweepMargin below the
// target, which is looser than inner_rtol when the sweep before it just missed the target
// (LOOSE: for updates of an iterate only; other solves keep inner_rtol at least), and tighter
// when a few more iterations save a further sweep.  What one FP32 solve cannot reach (below
// kSweepReach) is left to the next sweep, and towards a tighter aim an inner solve that has met
// inner_rtol runs kSoftIterations more at most: the error the line solve leaves can be slow.
// On the 768x768x96 combined workload (line solve: one iteration reduces the residual by about
// 1e-6) a third sweep, 1.8 ms, was needed in 14 of 26 solves because the second ended 2 to 30
// times above the target; on 256x256x128 loam that sweep took 5 to 26 inner iterations for a
// factor 1e-4 where 2 was missing (two steps: 52.1 -> 46.5 ms; the combined workload 273 -> 266).
constexpr double kSweepMargin = 0.1;
constexpr double kSweepReach = 1e-7;
constexpr int kSoftIterations = 2;

template <bool LOOSE>
__device__ __forceinline__ void set_inner_tolerance(CgDevState* in, double inner_rtol, double rn,
                                                    double target) {
  const double aim = kSweepMargin * target / rn;
  in->soft_its = 0;
  in->ttol_soft = 0.0;
  in->ttol = inner_rtol * in->rnorm0;
  if (!(aim >= kSweepReach)) return;
  if (aim < inner_rtol) {
    in->ttol_soft = in->ttol;
    in->ttol = aim * in->rnorm0;
  } else if (LOOSE) {
    in->ttol = aim * in->rnorm0;
  }
}

// the inner stopping test on ||r|| = rn
__device__ __forceinline__ bool inner_converged(CgDevState* st, double rn) {
  if (rn <= st->ttol) return true;
  return rn <= st->ttol_soft && st->soft_its++ >= kSoftIterations;
}

__global__ void k_line_factor(const double* __restrict__ a2, float* __restrict__ lk,
                              float* __restrict__ dinv, int ncol, int nz) {
  const size_t sk = (size_t)ncol;
  for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < ncol;
       col += gridDim.x * blockDim.x) {
    size_t c = (size_t)col;
    double d = 1.0;
    lk[c] = 0.0f;
    dinv[c] = 1.0f;
    for (int k = 1; k < nz; ++k) {
      c += sk;
      const double a = a2[c - sk];
      const double l = a / d;
      d = 1.0 - l * a;
      // an SPD operator keeps d in (0, 1]; a non-positive pivot (an operator that is not
      // SPD) degrades that row to the Jacobi step instead of dividing by it
      if (!(d > 0.0)) d = 1.0;
      lk[c] = (float)l;
      dinv[c] = (float)(1.0 / d);
    }
  }
}

// The scalar end of k32_line_step (last block).  FIRST: the first application, z0 = M^-1 r0.
template <bool FIRST>
__device__ __forceinline__ void line_step_tail(CgDevState* st, double rzn, double rr) {
  if (FIRST) {
    st->beta = rzn;
    st->bcoef = 0.0;
    st->fresh = 0;
    if (!(rzn > 0.0)) st->status = rzn == 0.0 ? kConvergedAtol : kDivergedIndefinitePc;
    return;
  }
  const double rn = sqrt(rr);
  st->dp = rn;
  st->iter += 1;
  if (isnan(rn) || isnan(rzn)) {
    st->status = kDivergedNanOrInf;
  } else if (inner_converged(st, rn)) {
    st->status = kConvergedRtol;
  } else if (st->iter >= st->max_it) {
    st->status = kDivergedIts;
  } else if (!(rzn > 0.0)) {
    st->status = kDivergedIndefinitePc;
  } else {
    st->bcoef = rzn / st->beta;
    st->beta = rzn;
    st->its = st->iter + 1;
  }
}

// FIRST: z = M^-1 r.  Else the CG update x += alpha p, r -= alpha w, then z = M^-1 r.
// p0, p1: the direction's two buffers; iteration `iter` wrote p1 when iter is even.
// A block owns 32 neighbouring columns; its W warps split the levels, each thread
// holding its at most L levels of r, l, 1/d in registers, so that all of a column's loads are in
// flight at once (a march down the column with one thread has a few levels in flight and needs
// more columns than small grids have).  Both sweeps are affine recurrences: a warp runs its
// levels with a zero carry and the product of the factors, the warps' ends are combined through
// shared memory (W - 1 steps), and the carry's share is added.  36 B/cell.
// 768 x 768 x 96: 324 us, 0.93 of the copy peak (the two sweeps as marches with one thread per
// column were 318 + 157, and 28 of 36 bytes more); 256 x 256 x 128: 72 us against 69 + 40.  16
// warps: 8 with twice the levels fit fewer blocks (573 us), 32 lengthen the carry's chain (610).
template <bool FIRST, int W, int L>
__global__ void __launch_bounds__(32 * W, L > 8 ? 1 : 2) k32_line_step(
    float* x, float* r, const float* p0, const float* p1, const float* w, const float* lk,
    const float* dinv, float* z, int ncol, int nz, CgDevState* st, double* partials) {
  grid_begin();
  if (st->status || (FIRST && !st->fresh)) return;
  __shared__ float2 fwd[W][32], bwd[W][32];
  __shared__ float lfirst[W + 1][32];
  const float a = FIRST ? 0.0f : (float)st->a;
  const int iter = st->iter;
  const float* p = (iter & 1) ? p0 : p1;
  const bool xfirst = iter == 0;  // the first update writes x = alpha p (x is not initialised)
  const size_t sk = (size_t)ncol;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int len = (nz + W - 1) / W;  // levels per warp, <= L
  const int k0 = warp * len, nk = max(0, min(len, nz - k0));
  if (warp == 0) lfirst[W][lane] = 0.0f;
  Kahan32 rz, rr;
  const int groups = (ncol + 31) / 32;
  // FIRST: the next group's loads are issued before this group's sweeps (the update has its own
  // loads in flight then, and no registers to spare)
  float ny[FIRST ? L : 1], nl[FIRST ? L : 1], nd[FIRST ? L : 1];
  auto load = [&](int g, float* ry, float* rl, float* rd) {
    const int col = g * 32 + lane;
    const int n = col < ncol ? nk : 0;
    const size_t base = (size_t)min(col, ncol - 1) + sk * min(k0, nz - 1);
#pragma unroll
    for (int q = 0; q < L; ++q) {
      ry[q] = rl[q] = rd[q] = 0.0f;
      if (q < n) {
        const size_t c = base + sk * q;
        ry[q] = r[c];
        rl[q] = lk[c];
        rd[q] = dinv[c];
      }
    }
  };
  if (FIRST) load(blockIdx.x, ny, nl, nd);
  for (int g = blockIdx.x; g < groups; g += gridDim.x) {
    const int col = g * 32 + lane;
    const int n = col < ncol ? nk : 0;
    const size_t base = (size_t)min(col, ncol - 1) + sk * min(k0, nz - 1);
    float y[L], l[L], d[L];
    if (FIRST) {
#pragma unroll
      for (int q = 0; q < L; ++q) {
        y[q] = ny[FIRST ? q : 0];
        l[q] = nl[FIRST ? q : 0];
        d[q] = nd[FIRST ? q : 0];
      }
      if (g + (int)gridDim.x < groups) load(g + gridDim.x, ny, nl, nd);
    } else {
      load(g, y, l, d);
    }
    if (!FIRST) {
      // all loads before the first store: the compiler may not move them across it
      float pv[L], wv[L], xv[L];
#pragma unroll
      for (int q = 0; q < L; ++q) {
        pv[q] = wv[q] = xv[q] = 0.0f;
        if (q < n) {
          const size_t c = base + sk * q;
          pv[q] = p[c];
          wv[q] = w[c];
          if (!xfirst) xv[q] = x[c];
        }
      }
#pragma unroll
      for (int q = 0; q < L; ++q) {
        y[q] = fmaf(-a, wv[q], y[q]);
        if (q < n) {
          const size_t c = base + sk * q;
          x[c] = fmaf(a, pv[q], xv[q]);
          r[c] = y[q];
        }
      }
    }
#pragma unroll
    for (int q = 0; q < L; ++q) rr.add(y[q] * y[q]);
    // forward, zero carry: y_k = r_k - l_k y_{k-1}; the carry enters with the product of -l
    float prod = 1.0f;
#pragma unroll
    for (int q = 0; q < L; ++q) {
      if (q < n) {
        if (q > 0) y[q] = fmaf(-l[q], y[q - 1], y[q]);
        prod *= -l[q];
      }
    }
    float end = 0.0f;
#pragma unroll
    for (int q = 0; q < L; ++q)
      if (q == n - 1) end = y[q];
    fwd[warp][lane] = make_float2(end, n > 0 ? prod : 1.0f);
    lfirst[warp][lane] = l[0];
    __syncthreads();
    float carry = 0.0f;
    for (int v = 0; v < warp; ++v) carry = fmaf(fwd[v][lane].y, carry, fwd[v][lane].x);
#pragma unroll
    for (int q = 0; q < L; ++q) {
      if (q < n) {
        carry *= -l[q];
        const float yk = y[q] + carry;
        y[q] = yk * d[q];  // u
        rz.add(yk * y[q]);
      }
    }
    // backward: z_k = u_k - l_{k+1} z_{k+1}
    const float lnext = lfirst[warp + 1][lane];
    prod = 1.0f;
#pragma unroll
    for (int q = L - 1; q >= 0; --q) {
      if (q < n) {
        if (q + 1 < n) y[q] = fmaf(-l[min(q + 1, L - 1)], y[min(q + 1, L - 1)], y[q]);
        prod *= -(q + 1 < n ? l[min(q + 1, L - 1)] : lnext);
      }
    }
    bwd[warp][lane] = make_float2(y[0], n > 0 ? prod : 1.0f);
    __syncthreads();
    carry = 0.0f;
    for (int v = W - 1; v > warp; --v)
      carry = fmaf(bwd[v][lane].y, carry, bwd[v][lane].x);
#pragma unroll
    for (int q = L - 1; q >= 0; --q) {
      if (q < n) {
        carry *= -(q + 1 < n ? l[min(q + 1, L - 1)] : lnext);
        z[base + sk * q] = y[q] + carry;
      }
    }
  }
  double loc[2] = {rz.value(), rr.value()};
  double tot[2];
  if (!grid_sum<2>(loc, partials, &st->arrive[2], tot)) return;
  if (flat_tid() == 0) line_step_tail<FIRST>(st, tot[0], tot[1]);
}

// The same step with one thread per column, for columns longer than k32_line_step's registers
// hold (256 levels): the forward sweep leaves u in z, the backward sweep overwrites it.  Levels in
// groups, whose loads all come before the group's stores (the compiler may not move them across).
template <bool FIRST>
__global__ void __launch_bounds__(128) k32_line_step_long(
    float* x, float* r, const float* p0, const float* p1, const float* w, const float* lk,
    const float* dinv, float* z, int ncol, int nz, CgDevState* st, double* partials) {
  grid_begin();
  if (st->status || (FIRST && !st->fresh)) return;
  const float a = FIRST ? 0.0f : (float)st->a;
  const float* p = (st->iter & 1) ? p0 : p1;
  const bool xfirst = st->iter == 0;
  const size_t sk = (size_t)ncol;
  constexpr int U = 4;
  Kahan32 rz, rr;
  for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < ncol;
       col += gridDim.x * blockDim.x) {
    float y = 0.0f;
    size_t c = (size_t)col;
    for (int k = 0; k < nz; k += U) {
      float rv[U], lv[U], dv[U], pv[U], wv[U], xv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const size_t cu = c + sk * min(u, nz - 1 - k);
        rv[u] = r[cu];
        lv[u] = lk[cu];
        dv[u] = dinv[cu];
        pv[u] = FIRST ? 0.0f : p[cu];
        wv[u] = FIRST ? 0.0f : w[cu];
        xv[u] = FIRST || xfirst ? 0.0f : x[cu];
      }
#pragma unroll
      for (int u = 0; u < U; ++u, c += sk) {
        if (k + u >= nz) break;
        if (!FIRST) {
          x[c] = fmaf(a, pv[u], xv[u]);
          rv[u] = fmaf(-a, wv[u], rv[u]);
          r[c] = rv[u];
        }
        y = fmaf(-lv[u], y, rv[u]);
        const float uk = y * dv[u];
        z[c] = uk;
        rz.add(y * uk);
        rr.add(rv[u] * rv[u]);
      }
    }
    float zz = 0.0f, lnext = 0.0f;
    c = (size_t)col + sk * (nz - 1);
    for (int k = nz - 1; k >= 0; k -= U) {
      float uv[U], lv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const size_t cu = c - sk * min(u, k);
        uv[u] = z[cu];
        lv[u] = lk[cu];
      }
#pragma unroll
      for (int u = 0; u < U; ++u, c -= sk) {
        if (k - u < 0) break;
        zz = fmaf(-lnext, zz, uv[u]);
        lnext = lv[u];
        z[c] = zz;
      }
    }
  }
  double loc[2] = {rz.value(), rr.value()};
  double tot[2];
  if (!grid_sum<2>(loc, partials, &st->arrive[2], tot)) return;
  if (flat_tid() == 0) line_step_tail<FIRST>(st, tot[0], tot[1]);
}

// Launch of the step: the register form's level count per warp by the number of levels.
template <bool FIRST>
inline void launch_line_step(float* x, float* r, const float* p0, const float* p1, const float* w,
                             const float* lk, const float* dinv, float* z, int ncol, int nz,
                             CgDevState* dst, double* partials, cudaStream_t s) {
  const int groups = (ncol + 31) / 32;
  // the resident blocks (two per SM) walk the groups: a block's end costs a reduction on the FP64
  // pipe (about 3,000 clocks of it per block; one block per group took 0.5 ms instead of 0.2 on
  // 768 x 768 columns), and a third block per SM would wait for a second wave
#define FG_LINE_STEP(W, LEV)                                                              \
  launch_chained(k32_line_step<FIRST, W, LEV>, std::min(groups, (LEV > 8 ? 1 : 2) * kNumSMs), \
                 32 * W, 0, s, x, r, p0, p1, w, lk, dinv, z, ncol, nz, dst, partials)
  if (nz <= 32) FG_LINE_STEP(16, 2);
  else if (nz <= 64) FG_LINE_STEP(16, 4);
  else if (nz <= 96) FG_LINE_STEP(16, 6);
  else if (nz <= 128) FG_LINE_STEP(16, 8);
  else if (nz <= 256) FG_LINE_STEP(16, 16);
  else {
    const int lb = (ncol + 127) / 128;
    launch_chained(k32_line_step_long<FIRST>, lb < kMaxRedBlocks ? lb : kMaxRedBlocks, 128, 0, s, x,
                   r, p0, p1, w, lk, dinv, z, ncol, nz, dst, partials);
  }
#undef FG_LINE_STEP
}

// z (+)= M^-1 r for the flexible-CG path (u is scratch).
__global__ void __launch_bounds__(128) k32_line_apply(const float* __restrict__ r,
                                                      const float* __restrict__ lk,
                                                      const float* __restrict__ dinv,
                                                      float* __restrict__ u,
                                                      float* __restrict__ z, int ncol, int nz,
                                                      int accumulate) {
  const size_t sk = (size_t)ncol;
  for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < ncol;
       col += gridDim.x * blockDim.x) {
    float y = 0.0f;
    size_t c = (size_t)col;
    for (int k = 0; k < nz; ++k, c += sk) {
      y = fmaf(-lk[c], y, r[c]);
      u[c] = y * dinv[c];
    }
    float zz = 0.0f, lnext = 0.0f;
    for (int k = nz - 1; k >= 0; --k) {
      c -= sk;
      zz = fmaf(-lnext, zz, u[c]);
      lnext = lk[c];
      z[c] = accumulate ? z[c] + zz : zz;
    }
  }
}

}  // namespace fg
