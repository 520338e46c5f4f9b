// Mixed-precision Krylov path (not in reference): FP32 Jacobi-PCG under FP64 iterative
// refinement.
//
// The operator is the same unit-diagonal scaled stencil as the FP64 path (A~ = D^-1/2 A D^-1/2,
// b~ = D^-1/2 b); its couplings are rounded once to FP32.  Each refinement sweep
//   1. forms the true residual r~ = b~ - A~ x~ in FP64 (FP64 couplings; the float-float operator's
//      from exact FP32 products) and its unscaled norm ||b - A x|| = ||r~ / s||; stops when
//      ||b - A x|| <= ir_rtol * ||b||;
//   2. solves A~32 e = fp32(r~ 2^-k) with FP32 CG to a relative reduction inner_rtol (dot
//      products in FP32 with Kahan compensation per thread, combined in FP64 across
//      threads/blocks; 2^-k, a power of two near 1/||r~||, keeps FP32 away from underflow);
//   3. updates x~ += 2^k e in FP64.
// The FP32 inner iteration moves 56 B/cell (vs 120 B/cell in FP64) and leaves the FP64 pipe,
// the limiter of the FP64 path on GB300, idle.  Convergence is always to the FP64 true
// residual, so the inner precision changes the iteration count, not the accuracy.
#include "ff32.cuh"
#include "internal.h"
#include "krylov_kernels.cuh"
#include "line.cuh"
#include "reduce.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

namespace fg {

// A complete sweep: the refinement test on the new true residual and the next inner system, by the
// last block.  sum_rhs: the squares of the right-hand side r~ / 2^k' just written (2^k' next above
// the previous ||r~||), sum_true: of (r~ / s) / unscale.
template <bool LOOSE>
__device__ __forceinline__ void sweep_tail(CgDevState* ir, CgDevState* in, double sum_rhs,
                                           double sum_true, double unscale, double ir_rtol,
                                           double inner_rtol) {
  const double rn = sqrt(sum_true) * unscale;
  ir->sweep_its[min(ir->ir_its, 3)] = in->its;
  ir->ir_its += 1;
  ir->its += in->its;
  ir->ir_rnorm = rn;
  ir->dp = rn;
  const double rs0 = pow2d(pow2_above(ir->a));
  ir->a = sqrt(sum_rhs) * rs0;
  if (isnan(rn) || isinf(rn)) {
    ir->status = kDivergedNanOrInf;
  } else if (rn <= fmax(ir_rtol * ir->ir_bnorm, ir->atol) || sum_rhs == 0.0) {
    ir->status = rn < ir->atol ? kConvergedAtol : kConvergedRtol;
  }
  if (ir->status == 0) {
    // the inner CG state, as k_ir_scale sets it, for the right-hand side r~ / rs0
    ir->rscale = rs0;
    in->beta = sum_rhs;
    in->rnorm0 = sqrt(sum_rhs);
    set_inner_tolerance<LOOSE>(in, inner_rtol, rn, fmax(ir_rtol * ir->ir_bnorm, ir->atol));
    in->iter = 0;
    in->its = 0;
    in->dpi = 0.0;
    in->fresh = 1;
    in->status = 0;
  }
}

// r~ = s b - A~ x~ (FP64); sums of r~^2 (scale of the inner system),
// (r~/s)^2 = (sq r~)^2 for the true residual (sq = 1/s) and b^2 for ||b||.  The last block
// runs the refinement test.  The inner solution e needs no zeroing: the inner solve's first
// update writes it.
// FIRST (the first sweep, x~ = 0): r~ = s b without the stencil product, kept in rres for
// k_ir_scale (x~ is not read: the first k_ir_update writes it), and the b^2 sum that ||b||
// needs (with x~ = 0 the true residual is b itself).  Later sweeps write the next inner
// right-hand side themselves and form the stencil product in FP64: the residual is a
// difference of nearly equal terms, and the refinement converges only as far as this product
// is accurate (a float-float form, 2^-48, was both slower here and short of 1e-12 on
// ill-conditioned systems).
// The inner iterations and k_ir_update are launched ahead of the host's knowledge of the inner
// solve's state: as long as it runs (in->status == 0) this kernel returns at once.
template <bool FIRST>
__global__ void __launch_bounds__(256) k_ir_residual(
    const double* __restrict__ a0, const double* __restrict__ a1, const double* __restrict__ a2,
    const double* __restrict__ s, const double* __restrict__ sq, const double* __restrict__ b,
    double* __restrict__ x, double* __restrict__ rres, int n0, int n1, int n2, int planes,
    int tiles, CgDevState* ir, double* partials, double ir_rtol,
    float* __restrict__ rfo = nullptr, CgDevState* in = nullptr, double inner_rtol = 0.0) {
  if (ir->status || (!FIRST && in->status == 0)) return;
  const int t0 = (n0 + 31) / 32;
  const size_t s01 = (size_t)n0 * n1;
  double v[FIRST ? 3 : 2] = {};
  double unscale = 1.0;
  if constexpr (FIRST) {
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int i0 = (tile % t0) * 32 + threadIdx.x;
      const int i1 = (tile / t0) * 8 + threadIdx.y;
      if (i0 >= n0 || i1 >= n1) continue;
      const int kb = blockIdx.y * planes, ke = min(n2, kb + planes);
      size_t c = (size_t)i0 + (size_t)n0 * i1 + s01 * kb;
      for (int k = kb; k < ke; ++k, c += s01) {
        const double bc = b[c];
        const double r = s[c] * bc;
        rres[c] = r;
        v[0] = fma(r, r, v[0]);
        v[2] = fma(bc, bc, v[2]);
      }
    }
    v[1] = v[2];
  } else {
    // the sums of squares in FP32 (compensated), after scaling by the previous sweep's norms,
    // which keeps the terms far from the FP32 range limits: they only set the inner scale and
    // the stopping test, and the FP64 pipe stays with the stencil product
    // the right-hand side's scale a power of two (2^(k-1) <= previous ||r~|| < 2^k)
    const float sig0 = pow2f_of(-pow2_above(ir->a));
    const double rs1 = ir->ir_rnorm;
    const float sig1 = (float)(1.0 / rs1);
    Kahan32 k0, k1;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int i0 = (tile % t0) * 32 + threadIdx.x;
      const int i1 = (tile / t0) * 8 + threadIdx.y;
      if (i0 >= n0 || i1 >= n1) continue;
      const int kb = blockIdx.y * planes, ke = min(n2, kb + planes);
      size_t c = (size_t)i0 + (size_t)n0 * i1 + s01 * kb;
      for (int k = kb; k < ke; ++k, c += s01) {
        double ax = x[c];
        if (i0 > 0) ax = fma(a0[c - 1], x[c - 1], ax);
        if (i0 + 1 < n0) ax = fma(a0[c], x[c + 1], ax);
        if (i1 > 0) ax = fma(a1[c - n0], x[c - n0], ax);
        if (i1 + 1 < n1) ax = fma(a1[c], x[c + n0], ax);
        if (k > 0) ax = fma(a2[c - s01], x[c - s01], ax);
        if (k + 1 < n2) ax = fma(a2[c], x[c + s01], ax);
        const double r = fma(s[c], b[c], -ax);
        const float rf = ff_hi_of(r);
        const float sqc = ff_hi_of(sq[c]);  // sq r~ = r~ / s
        const float q0 = rf * sig0, q1 = rf * sqc * sig1;
        rfo[c] = q0;  // the next inner solve's right-hand side, r~ / rs0 (rs0 = 2^k)
        k0.add(q0 * q0);
        k1.add(q1 * q1);
      }
    }
    v[0] = k0.value();
    v[1] = k1.value();
    unscale = rs1;
  }
  double tot[FIRST ? 3 : 2];
  if (!grid_sum<FIRST ? 3 : 2>(v, partials, &ir->arrive[0], tot)) return;
  if (flat_tid() == 0) {
    if constexpr (FIRST) {
      const double rn = sqrt(tot[1]);
      ir->ir_bnorm = sqrt(tot[2]);
      ir->ir_rnorm = rn;
      ir->dp = rn;
      ir->a = sqrt(tot[0]);
      ir->first_a = ir->a;
      if (isnan(rn) || isinf(rn))
        ir->status = kDivergedNanOrInf;
      else if (rn <= fmax(ir_rtol * ir->ir_bnorm, ir->atol) || tot[0] == 0.0)
        ir->status = rn < ir->atol ? kConvergedAtol : kConvergedRtol;
    } else {
      sweep_tail<false>(ir, in, tot[0], tot[1], unscale, ir_rtol, inner_rtol);
    }
  }
}

// Inner right-hand side rf = fp32(r~ 2^-k), 2^(k-1) <= ||r~|| < 2^k: norm in [1/2, 1), so FP32
// products cannot underflow however small the refinement residual is.  The last block
// initialises the inner CG state.
__global__ void k_ir_scale(const double* __restrict__ rres, float* __restrict__ rf, size_t n,
                           CgDevState* ir, CgDevState* in, double* partials,
                           double inner_rtol) {
  if (ir->status) {  // the inner iterations launched ahead have nothing to do
    if (blockIdx.x == 0 && threadIdx.x == 0) in->status = kConvergedAtol;
    return;
  }
  // 2^-k with 2^(k-1) <= ||r~|| < 2^k: the right-hand side's norm in [1/2, 1), and the scale
  // a power of two (exact, and the refinement update forms rscale e without FP64 arithmetic)
  const int k = pow2_above(ir->a);
  const float sig = pow2f_of(-k);
  Kahan32 acc;
  // the FP32 right-hand side from the residual's leading 24 bits (integer split: GB300's
  // double->float conversion runs on the FP64 pipe); four cells per step, 16-byte accesses
  const size_t gid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const double2* r2 = reinterpret_cast<const double2*>(rres);
  float4* f4 = reinterpret_cast<float4*>(rf);
  for (size_t q = gid; q < n / 4; q += stride) {
    const double2 lo = r2[2 * q], hi = r2[2 * q + 1];
    const float4 v = make_float4(ff_hi_of(lo.x) * sig, ff_hi_of(lo.y) * sig,
                                 ff_hi_of(hi.x) * sig, ff_hi_of(hi.y) * sig);
    f4[q] = v;
    acc.add(v.x * v.x);
    acc.add(v.y * v.y);
    acc.add(v.z * v.z);
    acc.add(v.w * v.w);
  }
  for (size_t c = (n & ~(size_t)3) + gid; c < n; c += stride) {
    const float r32 = ff_hi_of(rres[c]) * sig;
    rf[c] = r32;
    acc.add(r32 * r32);
  }
  double loc[1] = {acc.value()};
  double tot[1];
  if (!grid_sum<1>(loc, partials, &in->arrive[0], tot)) return;
  if (flat_tid() == 0) {
    ir->rscale = pow2d(k);
    in->beta = tot[0];
    in->rnorm0 = sqrt(tot[0]);
    in->ttol = inner_rtol * in->rnorm0;
    in->iter = 0;
    in->its = 0;
    in->dpi = 0.0;
    in->fresh = 1;
    in->status = tot[0] == 0.0 ? kConvergedAtol : 0;
  }
}

__global__ void k32_p(const float* __restrict__ r, float* __restrict__ p, size_t n,
                      const CgDevState* st) {
  if (st->status) return;
  const float bc = (float)st->bcoef;
  const bool first = st->iter == 0;
  const size_t gid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const float4* r4 = reinterpret_cast<const float4*>(r);
  float4* p4 = reinterpret_cast<float4*>(p);
  for (size_t q = gid; q < n / 4; q += stride) {
    const float4 rv = r4[q];
    float4 pv;
    if (first) {
      pv = rv;
    } else {
      pv = p4[q];
      pv.x = fmaf(bc, pv.x, rv.x);
      pv.y = fmaf(bc, pv.y, rv.y);
      pv.z = fmaf(bc, pv.z, rv.z);
      pv.w = fmaf(bc, pv.w, rv.w);
    }
    p4[q] = pv;
  }
  if (gid < (n & 3)) {
    const size_t c = (n & ~(size_t)3) + gid;
    p[c] = first ? r[c] : fmaf(bc, p[c], r[c]);
  }
}

// p.w known: alpha, or the end of the inner solve (breakdown or NaN; the refinement decides)
__device__ __forceinline__ void spmv32_tail(CgDevState* st, double dpi) {
  st->its = st->iter + 1;
  if (!(dpi > 0.0)) {
    st->status = isnan(dpi) ? kDivergedNanOrInf : kDivergedIndefiniteMat;
    return;
  }
  st->dpi = dpi;
  st->a = st->beta / dpi;
}

__global__ void __launch_bounds__(256) k32_spmv(const float* __restrict__ a0,
                                                const float* __restrict__ a1,
                                                const float* __restrict__ a2,
                                                const float* __restrict__ p, float* __restrict__ w,
                                                int n0, int n1, int n2, int planes, int tiles,
                                                CgDevState* st, double* partials) {
  if (st->status) return;
  const int t0 = (n0 + 31) / 32;
  Kahan32 acc;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int i0 = (tile % t0) * 32 + threadIdx.x;
    const int i1 = (tile / t0) * 8 + threadIdx.y;
    if (i0 >= n0 || i1 >= n1) continue;
    const size_t s01 = (size_t)n0 * n1;
    const int kb = blockIdx.y * planes, ke = min(n2, kb + planes);
    size_t c = (size_t)i0 + (size_t)n0 * i1 + s01 * kb;
    float pm = 0.0f, am = 0.0f;
    if (kb > 0) {
      pm = p[c - s01];
      am = a2[c - s01];
    }
    float pc = p[c];
    for (int k = kb; k < ke; ++k) {
      const float pp = (k + 1 < n2) ? p[c + s01] : 0.0f;
      const float ac = a2[c];
      float v = pc;
      if (i0 > 0) v = fmaf(a0[c - 1], p[c - 1], v);
      if (i0 + 1 < n0) v = fmaf(a0[c], p[c + 1], v);
      if (i1 > 0) v = fmaf(a1[c - n0], p[c - n0], v);
      if (i1 + 1 < n1) v = fmaf(a1[c], p[c + n0], v);
      v = fmaf(am, pm, v);
      v = fmaf(ac, pp, v);
      w[c] = v;
      acc.add(pc * v);
      pm = pc;
      pc = pp;
      am = ac;
      c += s01;
    }
  }
  double loc[1] = {acc.value()};
  double tot[1];
  if (!grid_sum<1>(loc, partials, &st->arrive[1], tot)) return;
  if (flat_tid() == 0) spmv32_tail(st, tot[0]);
}

// Vectorised variant for n0 % 4 == 0: a thread owns 4 consecutive cells along axis 0 (16-byte
// loads of p and the couplings); the axis-0 neighbours across threads come from warp shuffles,
// the axis-2 neighbours roll in registers while the thread marches through its planes.
__device__ __forceinline__ float4 ld4(const float* a, size_t c) {
  return *reinterpret_cast<const float4*>(a + c);
}

// the unit-diagonal stencil product of four neighbouring cells: pl / pr (al) the cells beside
// them, PS / PN, pm / pp the rows and planes on either side
__device__ __forceinline__ float4 stencil4(float4 pc, float pl, float pr, float al, float4 A0,
                                           float4 PS, float4 AS, float4 PN, float4 A1, float4 pm,
                                           float4 am, float4 pp, float4 A2) {
  float4 v;
  v.x = pc.x;
  v.x = fmaf(al, pl, v.x);
  v.x = fmaf(A0.x, pc.y, v.x);
  v.y = fmaf(A0.x, pc.x, pc.y);
  v.y = fmaf(A0.y, pc.z, v.y);
  v.z = fmaf(A0.y, pc.y, pc.z);
  v.z = fmaf(A0.z, pc.w, v.z);
  v.w = fmaf(A0.z, pc.z, pc.w);
  v.w = fmaf(A0.w, pr, v.w);
  v.x = fmaf(AS.x, PS.x, v.x);
  v.y = fmaf(AS.y, PS.y, v.y);
  v.z = fmaf(AS.z, PS.z, v.z);
  v.w = fmaf(AS.w, PS.w, v.w);
  v.x = fmaf(A1.x, PN.x, v.x);
  v.y = fmaf(A1.y, PN.y, v.y);
  v.z = fmaf(A1.z, PN.z, v.z);
  v.w = fmaf(A1.w, PN.w, v.w);
  v.x = fmaf(am.x, pm.x, v.x);
  v.y = fmaf(am.y, pm.y, v.y);
  v.z = fmaf(am.z, pm.z, v.z);
  v.w = fmaf(am.w, pm.w, v.w);
  v.x = fmaf(A2.x, pp.x, v.x);
  v.y = fmaf(A2.y, pp.y, v.y);
  v.z = fmaf(A2.z, pp.z, v.z);
  v.w = fmaf(A2.w, pp.w, v.w);
  return v;
}

__global__ void __launch_bounds__(128) k32_spmv_v4(const float* __restrict__ a0,
                                                   const float* __restrict__ a1,
                                                   const float* __restrict__ a2,
                                                   const float* __restrict__ p,
                                                   float* __restrict__ w, int n0, int n1, int n2,
                                                   int planes, int tiles, CgDevState* st,
                                                   double* partials) {
  if (st->status) return;
  const int t0 = (n0 + 127) / 128;
  const int lane = threadIdx.x;
  const unsigned full = 0xffffffffu;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  Kahan32 acc;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int i0 = (tile % t0) * 128 + lane * 4;
    const int i1 = (tile / t0) * 4 + threadIdx.y;
    const bool act = i0 < n0 && i1 < n1;
    const size_t s01 = (size_t)n0 * n1;
    const int kb = blockIdx.y * planes, ke = min(n2, kb + planes);
    size_t c = act ? (size_t)i0 + (size_t)n0 * i1 + s01 * kb : 0;
    float4 pc = act ? ld4(p, c) : z4;
    float4 pm = z4, am = z4;
    if (act && kb > 0) {
      pm = ld4(p, c - s01);
      am = ld4(a2, c - s01);
    }
    for (int k = kb; k < ke; ++k) {
      const bool up = act && k + 1 < n2;
      const float4 pp = up ? ld4(p, c + s01) : z4;
      const float4 A0 = act ? ld4(a0, c) : z4;
      const float4 A1 = act ? ld4(a1, c) : z4;
      const float4 A2 = act ? ld4(a2, c) : z4;
      const bool hs = act && i1 > 0, hn = act && i1 + 1 < n1;
      const float4 PS = hs ? ld4(p, c - n0) : z4;
      const float4 AS = hs ? ld4(a1, c - n0) : z4;
      const float4 PN = hn ? ld4(p, c + n0) : z4;
      float pl = __shfl_up_sync(full, pc.w, 1);
      float al = __shfl_up_sync(full, A0.w, 1);
      float pr = __shfl_down_sync(full, pc.x, 1);
      if (lane == 0) {
        const bool l = act && i0 > 0;
        pl = l ? p[c - 1] : 0.f;
        al = l ? a0[c - 1] : 0.f;
      }
      if (lane == 31) pr = (act && i0 + 4 < n0) ? p[c + 4] : 0.f;
      const float4 v = stencil4(pc, pl, pr, al, A0, PS, AS, PN, A1, pm, am, pp, A2);
      if (act) {
        *reinterpret_cast<float4*>(w + c) = v;
        acc.add(pc.x * v.x);
        acc.add(pc.y * v.y);
        acc.add(pc.z * v.z);
        acc.add(pc.w * v.w);
      }
      pm = pc;
      pc = pp;
      am = A2;
      c += s01;
    }
  }
  double loc[1] = {acc.value()};
  double tot[1];
  if (!grid_sum<1>(loc, partials, &st->arrive[1], tot)) return;
  if (flat_tid() == 0) spmv32_tail(st, tot[0]);
}

// Line-PCG: p = z + bcoef p_old (p = z in iteration 0) and w = A~ p, p.w in one pass.  The
// direction goes from one buffer (iteration parity) into the other, since neighbouring blocks
// read p_old; the neighbours' new directions are formed from z and p_old again (two loads
// instead of one for each cell beside the tile's own, from L1 and L2).  28 B/cell, against 36
// for a direction pass and a product: 260 us at 768 x 768 x 96, 0.90 of the copy peak (the product
// alone was 210, the direction's pass 160).
// This form is for row lengths that are no multiple of 4: a thread owns four rows of a column and
// marches through its planes, so that loads stay coalesced along axis 0, a row's couplings and
// directions serve the rows on either side, and a level's loads are in flight together (203 x 149 x
// 96: 40 us an iteration with one row per thread, 32 so).
constexpr int kDirRows = 4;
template <bool FIRST>
__device__ __forceinline__ void dir_spmv_rows(
    const float* a0, const float* a1, const float* a2, const float* z, const float* po,
    float* __restrict__ pn, float* __restrict__ w, float bc, int n0, int n1, int n2, int planes,
    int tiles, Kahan32& acc) {
  constexpr int R = kDirRows;
  auto dir = [&](size_t c) { return FIRST ? z[c] : fmaf(bc, po[c], z[c]); };
  const int t0 = (n0 + 31) / 32, lane = threadIdx.x;
  const unsigned full = 0xffffffffu;
  const size_t s01 = (size_t)n0 * n1;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int i0 = (tile % t0) * 32 + lane;
    const int j0 = ((tile / t0) * blockDim.y + threadIdx.y) * R;
    const int nr = min(R, n1 - j0);  // the warp's rows
    if (nr <= 0) continue;
    const int kb = blockIdx.y * planes, ke = min(n2, kb + planes);
    // lanes past the row's end and rows past the last repeat the last ones (nothing is stored, and
    // the couplings towards them are zero)
    size_t c = (size_t)min(i0, n0 - 1) + (size_t)n0 * j0 + s01 * kb;
    int off[R];
#pragma unroll
    for (int r = 0; r < R; ++r) off[r] = n0 * min(r, nr - 1);
    const bool south = j0 > 0, north = j0 + nr < n1;
    const bool left = lane == 0 && i0 > 0, edge = left || (lane == 31 && i0 + 1 < n0);
    float pm[R], am[R], pc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      pm[r] = kb > 0 ? dir(c - s01 + off[r]) : 0.0f;
      am[r] = kb > 0 ? a2[c - s01 + off[r]] : 0.0f;
      pc[r] = dir(c + off[r]);
    }
    for (int k = kb; k < ke; ++k, c += s01) {
      float pp[R], A0[R], A1[R], A2[R], pe[R], ae[R];
      const size_t ce = left ? c - 1 : c + 1;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        pp[r] = k + 1 < n2 ? dir(c + s01 + off[r]) : 0.0f;
        A0[r] = a0[c + off[r]];
        A1[r] = a1[c + off[r]];
        A2[r] = a2[c + off[r]];
        pe[r] = edge ? dir(ce + off[r]) : 0.0f;
        ae[r] = left ? a0[c - 1 + off[r]] : 0.0f;
      }
      const float pS = south ? dir(c - n0) : 0.0f, AS = south ? a1[c - n0] : 0.0f;
      const float pN = north ? dir(c + (size_t)n0 * nr) : 0.0f;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float pl = __shfl_up_sync(full, pc[r], 1), al = __shfl_up_sync(full, A0[r], 1);
        float pr = __shfl_down_sync(full, pc[r], 1);
        if (lane == 0) {
          pl = pe[r];
          al = ae[r];
        }
        if (lane == 31) pr = pe[r];
        float v = fmaf(al, pl, pc[r]);
        v = fmaf(A0[r], pr, v);
        v = r == 0 ? fmaf(AS, pS, v) : fmaf(A1[r - 1], pc[r - 1], v);
        v = fmaf(A1[r], r + 1 < R && r + 1 < nr ? pc[r + 1] : pN, v);
        v = fmaf(am[r], pm[r], v);
        v = fmaf(A2[r], pp[r], v);
        if (r < nr && i0 < n0) {
          pn[c + off[r]] = pc[r];
          w[c + off[r]] = v;
          acc.add(pc[r] * v);
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        pm[r] = pc[r];
        pc[r] = pp[r];
        am[r] = A2[r];
      }
    }
  }
}

__global__ void __launch_bounds__(128) k32_dir_spmv(
    const float* a0, const float* a1, const float* a2, const float* z, float* p0, float* p1,
    float* w, int n0, int n1, int n2, int planes, int tiles, CgDevState* st, double* partials) {
  grid_begin();
  if (st->status) return;
  const bool odd = st->iter & 1;
  const float* po = odd ? p1 : p0;
  float* pn = odd ? p0 : p1;
  Kahan32 acc;
  if (st->iter == 0)
    dir_spmv_rows<true>(a0, a1, a2, z, po, pn, w, 0.0f, n0, n1, n2, planes, tiles, acc);
  else
    dir_spmv_rows<false>(a0, a1, a2, z, po, pn, w, (float)st->bcoef, n0, n1, n2, planes, tiles, acc);
  double loc[1] = {acc.value()};
  double tot[1];
  if (!grid_sum<1>(loc, partials, &st->arrive[1], tot)) return;
  if (flat_tid() == 0) spmv32_tail(st, tot[0]);
}

// n0 a multiple of 4: four cells per thread, 16-byte accesses
__global__ void __launch_bounds__(128) k32_dir_spmv_v4(
    const float* a0, const float* a1, const float* a2, const float* z, float* p0, float* p1,
    float* w, int n0, int n1, int n2, int planes, int tiles, CgDevState* st, double* partials) {
  grid_begin();
  if (st->status) return;
  const bool first = st->iter == 0, odd = st->iter & 1;
  const float bc = first ? 0.0f : (float)st->bcoef;
  const float* po = odd ? p1 : p0;
  float* pn = odd ? p0 : p1;
  auto dir4 = [&](size_t c) {
    float4 v = ld4(z, c);
    if (!first) {
      const float4 o = ld4(po, c);
      v.x = fmaf(bc, o.x, v.x);
      v.y = fmaf(bc, o.y, v.y);
      v.z = fmaf(bc, o.z, v.z);
      v.w = fmaf(bc, o.w, v.w);
    }
    return v;
  };
  auto dir = [&](size_t c) { return first ? z[c] : fmaf(bc, po[c], z[c]); };
  const int t0 = (n0 + 127) / 128;
  const int lane = threadIdx.x;
  const unsigned full = 0xffffffffu;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const size_t s01 = (size_t)n0 * n1;
  Kahan32 acc;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int i0 = (tile % t0) * 128 + lane * 4;
    const int i1 = (tile / t0) * 4 + threadIdx.y;
    const bool act = i0 < n0 && i1 < n1;
    const int kb = blockIdx.y * planes, ke = min(n2, kb + planes);
    size_t c = act ? (size_t)i0 + (size_t)n0 * i1 + s01 * kb : 0;
    float4 pc = act ? dir4(c) : z4;
    float4 pm = z4, am = z4;
    if (act && kb > 0) {
      pm = dir4(c - s01);
      am = ld4(a2, c - s01);
    }
    for (int k = kb; k < ke; ++k) {
      const bool up = act && k + 1 < n2;
      const float4 pp = up ? dir4(c + s01) : z4;
      const float4 A0 = act ? ld4(a0, c) : z4;
      const float4 A1 = act ? ld4(a1, c) : z4;
      const float4 A2 = act ? ld4(a2, c) : z4;
      const bool hs = act && i1 > 0, hn = act && i1 + 1 < n1;
      const float4 PS = hs ? dir4(c - n0) : z4;
      const float4 AS = hs ? ld4(a1, c - n0) : z4;
      const float4 PN = hn ? dir4(c + n0) : z4;
      float pl = __shfl_up_sync(full, pc.w, 1);
      float al = __shfl_up_sync(full, A0.w, 1);
      float pr = __shfl_down_sync(full, pc.x, 1);
      if (lane == 0) {
        const bool l = act && i0 > 0;
        pl = l ? dir(c - 1) : 0.f;
        al = l ? a0[c - 1] : 0.f;
      }
      if (lane == 31) pr = (act && i0 + 4 < n0) ? dir(c + 4) : 0.f;
      const float4 v = stencil4(pc, pl, pr, al, A0, PS, AS, PN, A1, pm, am, pp, A2);
      if (act) {
        *reinterpret_cast<float4*>(pn + c) = pc;
        *reinterpret_cast<float4*>(w + c) = v;
        acc.add(pc.x * v.x);
        acc.add(pc.y * v.y);
        acc.add(pc.z * v.z);
        acc.add(pc.w * v.w);
      }
      pm = pc;
      pc = pp;
      am = A2;
      c += s01;
    }
  }
  double loc[1] = {acc.value()};
  double tot[1];
  if (!grid_sum<1>(loc, partials, &st->arrive[1], tot)) return;
  if (flat_tid() == 0) spmv32_tail(st, tot[0]);
}

// launch geometry of k32_spmv_v4 and of the row form: (32 x 4) threads cover 128 x 4 cells of a
// plane, or 32 x 16
static StencilLaunch launch_v4(int n0, int n1, int n2, bool rows = false) {
  StencilLaunch L;
  L.block = dim3(32, 4, 1);
  const long tiles = rows ? (long)((n0 + 31) / 32) * ((n1 + 4 * kDirRows - 1) / (4 * kDirRows))
                          : (long)((n0 + 127) / 128) * ((n1 + 3) / 4);
  // one wave of eight 128-thread blocks per SM: each z chunk reads two more planes and each block
  // ends with a reduction on the FP64 pipe (line-PCG product at 256 x 256 x 128: 56 us, 65 with
  // four times the blocks; the same at 768 x 768 x 96)
  const long target = (long)kNumSMs * 8;
  long z = target / (tiles > 0 ? tiles : 1);
  if (z < 1) z = 1;
  if (z > n2) z = n2;
  int planes = (int)((n2 + z - 1) / z);
  z = (n2 + planes - 1) / planes;
  long gx = tiles;
  const long cap = kMaxRedBlocks / z;
  if (gx > cap) gx = cap;
  L.planes = planes;
  L.tiles = (int)tiles;
  L.grid = dim3((unsigned)gx, (unsigned)z, 1);
  return L;
}

__global__ void k32_update(float* __restrict__ e, float* __restrict__ r,
                           const float* __restrict__ p, const float* __restrict__ w, size_t n,
                           CgDevState* st, double* partials) {
  if (st->status) return;
  const float a = (float)st->a;
  // the first iteration writes e = a p (e is not initialised)
  const bool first = st->iter == 0;
  Kahan32 acc;
  const size_t gid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  float4* e4 = reinterpret_cast<float4*>(e);
  float4* r4 = reinterpret_cast<float4*>(r);
  const float4* p4 = reinterpret_cast<const float4*>(p);
  const float4* w4 = reinterpret_cast<const float4*>(w);
  for (size_t q = gid; q < n / 4; q += stride) {
    float4 ev = first ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : e4[q], rv = r4[q];
    const float4 pv = p4[q], wv = w4[q];
    ev.x = fmaf(a, pv.x, ev.x);
    ev.y = fmaf(a, pv.y, ev.y);
    ev.z = fmaf(a, pv.z, ev.z);
    ev.w = fmaf(a, pv.w, ev.w);
    rv.x = fmaf(-a, wv.x, rv.x);
    rv.y = fmaf(-a, wv.y, rv.y);
    rv.z = fmaf(-a, wv.z, rv.z);
    rv.w = fmaf(-a, wv.w, rv.w);
    e4[q] = ev;
    r4[q] = rv;
    acc.add(rv.x * rv.x);
    acc.add(rv.y * rv.y);
    acc.add(rv.z * rv.z);
    acc.add(rv.w * rv.w);
  }
  if (gid < (n & 3)) {
    const size_t c = (n & ~(size_t)3) + gid;
    e[c] = fmaf(a, p[c], first ? 0.0f : e[c]);
    const float rc = fmaf(-a, w[c], r[c]);
    r[c] = rc;
    acc.add(rc * rc);
  }
  double loc[1] = {acc.value()};
  double tot[1];
  if (!grid_sum<1>(loc, partials, &st->arrive[2], tot)) return;
  if (flat_tid() == 0) {
    const double rr = tot[0];
    const double rn = sqrt(rr);
    st->dp = rn;
    st->iter += 1;
    if (isnan(rn)) {
      st->status = kDivergedNanOrInf;
    } else if (inner_converged(st, rn)) {
      st->status = kConvergedRtol;
    } else if (st->iter >= st->max_it) {
      st->status = kDivergedIts;
    } else {
      st->bcoef = rr / st->beta;
      st->beta = rr;
      st->its = st->iter + 1;
    }
  }
}

// x~ += rscale e (the inner system was solved for the residual divided by rscale); the first
// sweep: x~ = rscale e (x~ was 0 and is not read).  The inner solve's first update writes e without
// reading it, so e holds nothing before it: an inner solve that stopped before its first
// iteration (in->iter == 0) contributes e = 0.  Four cells per step with 16-byte loads and
// stores (the buffers are whole cudaMalloc allocations: 256-byte aligned).
// rscale is a power of two 2^k: rscale e is formed by integer operations (f2d_scaled), which
// leaves the first sweep without FP64 instructions and the others with one addition per cell.
// Nothing is done while the inner solve runs or after the refinement has ended.
template <bool FIRST>
__device__ __forceinline__ void ir_update_cells(double* __restrict__ x,
                                                const float* __restrict__ e, size_t n, double rs,
                                                int scale) {
  const size_t gid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  if (rs != pow2d(scale)) {  // not a power of two (no path sets one): FP64 arithmetic
    for (size_t c = gid; c < n; c += stride)
      x[c] = FIRST ? rs * (double)e[c] : fma(rs, (double)e[c], x[c]);
    return;
  }
  auto step = [&](float ev, double xv) {
    const double v = f2d_scaled(ev, scale);
    return FIRST ? v : xv + v;
  };
  const float4* e4 = reinterpret_cast<const float4*>(e);
  double2* x2 = reinterpret_cast<double2*>(x);
  for (size_t q = gid; q < n / 4; q += stride) {
    const float4 ev = e4[q];
    double2 lo = make_double2(0.0, 0.0), hi = lo;
    if (!FIRST) {
      lo = x2[2 * q];
      hi = x2[2 * q + 1];
    }
    lo.x = step(ev.x, lo.x);
    lo.y = step(ev.y, lo.y);
    hi.x = step(ev.z, hi.x);
    hi.y = step(ev.w, hi.y);
    x2[2 * q] = lo;
    x2[2 * q + 1] = hi;
  }
  for (size_t c = (n & ~(size_t)3) + gid; c < n; c += stride) x[c] = step(e[c], FIRST ? 0.0 : x[c]);
}

__global__ void k_ir_update(double* __restrict__ x, const float* __restrict__ e, size_t n,
                            const CgDevState* ir, const CgDevState* in) {
  if (ir->status || in->status == 0) return;
  const bool first = ir->ir_its == 0;
  if (in->iter == 0) {
    if (first)
      for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
           c += (size_t)gridDim.x * blockDim.x)
        x[c] = 0.0;
    return;
  }
  const double rs = ir->rscale;
  const int scale = pow2_above(rs) - 1;  // rscale = 2^scale
  if (first)
    ir_update_cells<true>(x, e, n, rs, scale);
  else
    ir_update_cells<false>(x, e, n, rs, scale);
}

// x~ += 2^k e for the sweeps whose residual is updated (k_ir_sweep), not recomputed: e becomes the
// change that x~ really made, fl(x~ + 2^k e) - x~, so that the updated residual is that of the
// stored x~.  That change is a float, a multiple of ulp(x~) no longer than e's own 24 bits, but where
// the sum has a larger exponent than x~ and e: there one ulp of x~ is dropped (in few cells; half an
// ulp of the sum, as a recomputed residual's rounding is).  The first sweep's x~ = 2^k e is exact and
// written by k_ir_sweep.
__global__ void k_ir_update_exact(double* x, float* e, size_t n, const CgDevState* ir,
                                  const CgDevState* in) {
  grid_begin();
  if (ir->status || in->status == 0 || ir->ir_its == 0 || in->iter == 0) return;
  const int scale = pow2_above(ir->rscale) - 1;  // rscale = 2^scale
  const float back = pow2f_of(-scale);
  const size_t gid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  auto step = [&](float& ev, double& xv) {
    const double y = xv + f2d_scaled(ev, scale);
    ev = ff_hi_of(y - xv) * back;
    xv = y;
  };
  float4* e4 = reinterpret_cast<float4*>(e);
  double2* x2 = reinterpret_cast<double2*>(x);
  for (size_t q = gid; q < n / 4; q += stride) {
    float4 ev = e4[q];
    double2 lo = x2[2 * q], hi = x2[2 * q + 1];
    step(ev.x, lo.x);
    step(ev.y, lo.y);
    step(ev.z, hi.x);
    step(ev.w, hi.y);
    e4[q] = ev;
    x2[2 * q] = lo;
    x2[2 * q + 1] = hi;
  }
  for (size_t c = (n & ~(size_t)3) + gid; c < n; c += stride) step(e[c], x[c]);
}

__device__ __forceinline__ float scale_of(float d) { return rsqrtf(d == 0.0f ? 1.0f : d); }

// x 2^k as three floats h + m + l (24 + 24 + 5 bits of the significand, truncated in turn), by
// integer operations.  Below 2^-126: zero; beyond the float range, inf and NaN: NaN.
struct Float3 {
  float h, m, l;
};
__device__ __forceinline__ Float3 split3(double x, int k) {
  const int hx = __double2hiint(x), lx = __double2loint(x);
  const int fe = ((hx >> 20) & 0x7ff) - (1023 - 127) + k;  // the float's biased exponent
  const int sign = hx & (int)0x80000000;
  Float3 r;
  r.h = __int_as_float(sign | (fe << 23) | ((hx & 0x000fffff) << 3) | (int)((unsigned)lx >> 29));
  const float p2 = __int_as_float(sign | ((fe & 0xff) << 23));
  const unsigned low = (unsigned)lx & 0x1fffffffu;
  r.m = __fmul_rn(__fmul_rn(__uint2float_rn(low & ~31u), 0x1p-52f), p2);
  r.l = __fmul_rn(__fmul_rn(__uint2float_rn(low & 31u), 0x1p-52f), p2);
  if (fe < 1) r.h = r.m = r.l = 0.0f;
  if (fe > 254) r.h = __int_as_float(0x7fc00000);
  return r;
}

// An exact sum of floats in three levels (the extraction of S. M. Rump, T. Ogita, S. Oishi,
// "Accurate floating-point summation part I", SIAM J. Sci. Comput. 31(1), 2008): with 2^m above every term,
// s0 collects the terms' bits down to 2^(m-20), s1 (which the products' low parts enter) those
// down to 2^(m-39), both without rounding for up to 16 and 32 terms, s2 the rest: the sum is within
// about 2^(m-57), where FP64's partial sums round at 2^(m-54).
struct ExactSum {
  float g0, g1, s0, s1, s2;
  // m: the largest magnitude of the terms
  __device__ __forceinline__ explicit ExactSum(float m) {
    const int e = max(__float_as_int(m), 0x12000000) & 0x7f800000;  // 2^-91 at least
    g0 = __int_as_float(e + (5 << 23));
    g1 = __int_as_float(e - (14 << 23));
    s0 = s1 = s2 = 0.0f;
  }
  __device__ __forceinline__ void low(float x) {
    const float h = __fsub_rn(__fadd_rn(g1, x), g1);
    s1 = __fadd_rn(s1, h);
    s2 = __fadd_rn(s2, __fsub_rn(x, h));
  }
  __device__ __forceinline__ void add(float x) {
    const float h = __fsub_rn(__fadd_rn(g0, x), g0);
    s0 = __fadd_rn(s0, h);
    low(__fsub_rn(x, h));
  }
  __device__ __forceinline__ ff value() const {
    const ff t = two_sum(s0, s1);
    return fast_two_sum(t.h, __fadd_rn(t.l, s2));
  }
};

// The refinement residual of the float-float operator (a = hi + lo exactly), updated instead of
// recomputed: r~ - A~ (2^k e), or s b - A~ (2^k e) in the first sweep, from exact FP32 products summed
// in ExactSum, so that it stays the true residual of x~ to 2^-48 of itself and 2^-57 of its terms
// (the FP64 stencil product rounds at 2^-53 of them) while the FP64 pipe, which bound that product
// at 690 us for 56.6M cells, has nothing to do.  The low couplings' products enter with their own
// rounding errors: without those it was off by 1.7e-16 of its terms at 40 x 40 x 100, 5e-19 so.
// With the x~ update: 690 + 155 -> 613 + 132 us for 56.6M cells, 62 + 14 -> 55 + 12 for 2.9M, bound by
// its 392 instructions per warp and cell.  r~ is kept as float pairs in units of the inner system's
// scale; the leading floats are the next right-hand side.  The first sweep also writes x~ = 2^k e.
struct SweepArgs {
  const float *h0, *h1, *h2, *l0, *l1, *l2;  // A~
  const float *dg, *e;                       // the diagonal (scale factors), the correction
  const double* b;
  double* x;
  float2* r;
  float* rf;
};

template <bool FIRST>
__device__ __forceinline__ void sweep_cells(const SweepArgs& a, int n0, int n1, int n2, int planes,
                                            int tiles, int scale, bool moved, float to_next,
                                            float to_true, Kahan32& k0, Kahan32& k1) {
  const int t0 = (n0 + 31) / 32;
  const size_t s01 = (size_t)n0 * n1;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int i0 = (tile % t0) * 32 + threadIdx.x;
    const int i1 = (tile / t0) * 8 + threadIdx.y;
    if (i0 >= n0 || i1 >= n1) continue;
    const bool xm = i0 > 0, xp = i0 + 1 < n0, ym = i1 > 0, yp = i1 + 1 < n1;
    const int kb = blockIdx.y * planes, ke = min(n2, kb + planes);
    size_t c = (size_t)i0 + (size_t)n0 * i1 + s01 * kb;
    auto ev = [&](bool in, size_t at) { return in && moved ? a.e[at] : 0.0f; };
    float eu = ev(kb > 0 && kb < ke, c - s01), ec = ev(kb < ke, c);
    float hu = kb > 0 && kb < ke ? a.h2[c - s01] : 0.0f;
    float lu = kb > 0 && kb < ke ? a.l2[c - s01] : 0.0f;
    for (int k = kb; k < ke; ++k, c += s01) {
      const bool zp = k + 1 < n2;
      const float ed = ev(zp, c + s01);
      const float en[6] = {ev(xm, c - 1), ev(xp, c + 1), ev(ym, c - n0), ev(yp, c + n0), eu, ed};
      const float h2 = a.h2[c], l2 = a.l2[c];
      const float ah[6] = {xm ? a.h0[c - 1] : 0.0f, a.h0[c], ym ? a.h1[c - n0] : 0.0f, a.h1[c],
                           hu, h2};
      const float al[6] = {xm ? a.l0[c - 1] : 0.0f, a.l0[c], ym ? a.l1[c - n0] : 0.0f, a.l1[c],
                           lu, l2};
      const float sc = scale_of(a.dg[c]);
      Float3 bs;
      float2 r;
      if (FIRST) {
        bs = split3(a.b[c], -scale);
        r.x = __fmul_rn(sc, bs.h);
        r.y = __fmaf_rn(sc, bs.h, -r.x);
      } else {
        r = a.r[c];
      }
      float p[6], m = fmaxf(fabsf(r.x), fabsf(ec));
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        p[q] = __fmul_rn(-ah[q], en[q]);
        m = fmaxf(m, fabsf(p[q]));
      }
      ExactSum sum(m);
      sum.add(r.x);
      sum.low(r.y);
      if (FIRST) {
        const float pm = __fmul_rn(sc, bs.m);
        sum.low(pm);
        sum.s2 = __fadd_rn(sum.s2, __fmaf_rn(sc, bs.l, __fmaf_rn(sc, bs.m, -pm)));
      }
      sum.add(-ec);
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        sum.add(p[q]);
        sum.low(__fmaf_rn(-ah[q], en[q], -p[q]));
        const float pl = __fmul_rn(-al[q], en[q]);
        sum.low(pl);
        sum.s2 = __fadd_rn(sum.s2, __fmaf_rn(-al[q], en[q], -pl));
      }
      const ff v = sum.value();
      const float q0 = v.h * to_next;
      a.rf[c] = q0;
      a.r[c] = make_float2(q0, v.l * to_next);
      const float q1 = v.h * __frcp_rn(sc) * to_true;  // r~ / s
      k0.add(q0 * q0);
      k1.add(q1 * q1);
      if (FIRST) a.x[c] = f2d_scaled(ec, scale);
      eu = ec;
      ec = ed;
      hu = h2;
      lu = l2;
    }
  }
}

__global__ void __launch_bounds__(256, 4) k_ir_sweep(SweepArgs a, int n0, int n1, int n2,
                                                     int planes, int tiles, CgDevState* ir,
                                                     CgDevState* in, double* partials,
                                                     double ir_rtol, double inner_rtol) {
  grid_begin();
  if (ir->status || in->status == 0) return;
  const int scale = pow2_above(ir->rscale) - 1;  // rscale = 2^scale
  const int next = pow2_above(ir->a);            // the next inner system's
  const int tru = pow2_above(ir->ir_rnorm);
  const bool moved = in->iter > 0;  // else e was not written: no correction
  const float to_next = pow2f_of(min(max(scale - next, -120), 120));
  const float to_true = pow2f_of(min(max(scale - tru, -120), 120));
  Kahan32 k0, k1;
  if (ir->ir_its == 0)
    sweep_cells<true>(a, n0, n1, n2, planes, tiles, scale, moved, to_next, to_true, k0, k1);
  else
    sweep_cells<false>(a, n0, n1, n2, planes, tiles, scale, moved, to_next, to_true, k0, k1);
  double v[2] = {k0.value(), k1.value()};
  double tot[2];
  if (!grid_sum<2>(v, partials, &ir->arrive[0], tot)) return;
  if (flat_tid() == 0)
    sweep_tail<true>(ir, in, tot[0], tot[1], pow2d(tru), ir_rtol, inner_rtol);
}

__global__ void k_to_f32(const double* __restrict__ a0, const double* __restrict__ a1,
                         const double* __restrict__ a2, float* __restrict__ f0,
                         float* __restrict__ f1, float* __restrict__ f2, size_t n) {
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x) {
    f0[c] = (float)a0[c];
    f1[c] = (float)a1[c];
    f2[c] = (float)a2[c];
  }
}

__global__ void k_zero64(double* __restrict__ x, size_t n) {
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x)
    x[c] = 0.0;
}

// ---- flexible CG (FCG(1), Notay 2000) with a nonlinear preconditioner z = M(r) ----------
//   beta = -(z . A p_prev) / (p_prev . A p_prev);  p = z + beta p_prev;  alpha = (p . r)/(p . A p)
// k_fcg_beta forms beta from z . w_prev (w_prev = A p_prev still holds the previous SpMV);
// k_fcg_p forms p and p . r, stored as st->beta so that k32_spmv* yields alpha = (p.r)/(p.Ap).
__global__ void k_fcg_beta(const float* __restrict__ z, const float* __restrict__ w, size_t n,
                           CgDevState* st, double* partials) {
  if (st->status) return;
  Kahan32 acc;
  if (st->iter > 0)
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
         c += (size_t)gridDim.x * blockDim.x)
      acc.add(z[c] * w[c]);
  double loc[1] = {acc.value()};
  double tot[1];
  if (!grid_sum<1>(loc, partials, &st->arrive[3], tot)) return;
  if (flat_tid() == 0) st->bcoef = st->iter > 0 ? -tot[0] / st->dpi : 0.0;
}

__global__ void k_fcg_p(const float* __restrict__ z, float* __restrict__ p,
                        const float* __restrict__ r, size_t n, CgDevState* st, double* partials) {
  if (st->status) return;
  const float bc = (float)st->bcoef;
  const bool first = st->iter == 0;
  Kahan32 acc;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x) {
    const float pv = first ? z[c] : fmaf(bc, p[c], z[c]);
    p[c] = pv;
    acc.add(pv * r[c]);
  }
  double loc[1] = {acc.value()};
  double tot[1];
  if (!grid_sum<1>(loc, partials, &st->arrive[4], tot)) return;
  if (flat_tid() == 0) st->beta = tot[0];
}

// z += r: the network supplies the correction on top of the (unit-diagonal) Jacobi step
__global__ void k_add_f32(float* __restrict__ z, const float* __restrict__ r, size_t n) {
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x)
    z[c] += r[c];
}

// ------------------------------------------------------------------------------------------

int KrylovSolver::ensure32(size_t n) {
  if (n <= cap32 && xf) return FREHG_OK;
  cudaFree(xf);
  cudaFree(rf);
  cudaFree(pf);
  cudaFree(wf);
  xf = rf = pf = wf = nullptr;
  if (g32) {
    cudaGraphExecDestroy(g32);
    g32 = nullptr;
  }
  FG_CUDA(cudaMalloc(&xf, n * sizeof(float)));
  FG_CUDA(cudaMalloc(&rf, n * sizeof(float)));
  FG_CUDA(cudaMalloc(&pf, n * sizeof(float)));
  FG_CUDA(cudaMalloc(&wf, n * sizeof(float)));
  cudaFree(rres);
  rres = nullptr;
  FG_CUDA(cudaMalloc(&rres, n * sizeof(double)));
  FG_TRY(op32.alloc(n));
  if (!dst32) {
    FG_CUDA(cudaMalloc(&dst32, sizeof(CgDevState)));
    FG_CUDA(cudaMemset(dst32, 0, sizeof(CgDevState)));
    FG_TRY(alloc_mapped(reinterpret_cast<void**>(&hst32), sizeof(CgDevState)));
  }
  cap32 = n;
  return FREHG_OK;
}

// Scaling of a fresh operator for the mixed path in two passes (solves whose result is the
// solution itself): s = D^-1/2 with sq = D^1/2 in FP64 (d s^2 = 1 to rounding, as the
// refinement residual's unit diagonal assumes), then one pass per column that scales the
// couplings in place (FP64, for the refinement residual), writes their FP32 copies (leading 24
// bits, without a double->float conversion: GB300 runs those on the FP64 pipe) and, with the
// line preconditioner, the column factors
//   l_k = v2_{k-1} / d_{k-1},  d_k = 1 - l_k v2_{k-1}   (d_0 = 1)
// in float-float, stored as floats.  The float-float path's update solves take k_prep_ff.
__global__ void k_diag_rsqrt_sq(double* __restrict__ s, double* __restrict__ sq, size_t n) {
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x) {
    const double d = s[c];
    const double dd = d == 0.0 ? 1.0 : d;  // PCJacobi replaces a zero diagonal entry by 1
    const double r = rsqrt(dd);
    s[c] = r;
    sq[c] = dd * r;
  }
}

__device__ __forceinline__ ff scaled_coupling64(double* a, size_t c, double sc, double sn) {
  const double v = a[c] * sc * sn;
  a[c] = v;
  return ff_make(ff_hi_of(v));
}

// the float-float path's scale factors are floats, and so are the couplings the float-float
// Picard assembly writes: a s_c s_n = a (p_h + p_l) with p = s_c s_n exact, one float-float by
// float product; the pair is the operator that k_ir_sweep's residual uses
__device__ __forceinline__ ff scaled_coupling_f(float af, float sc, float sn) {
  return ff_mul_f(two_prod(sc, sn), af);
}

__global__ void __launch_bounds__(128) k_scale_mixed(double* __restrict__ a0,
                                                     double* __restrict__ a1,
                                                     double* __restrict__ a2,
                                                     const double* __restrict__ s,
                                                     float* __restrict__ f0,
                                                     float* __restrict__ f1,
                                                     float* __restrict__ f2,
                                                     float* __restrict__ lk,
                                                     float* __restrict__ dinv, int n0, int n1,
                                                     int n2, int line) {
  const int ncol = n0 * n1;
  const size_t sk = (size_t)ncol;
  const ff zero = ff_make(0.0f);
  for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < ncol;
       col += gridDim.x * blockDim.x) {
    const int i0 = col % n0, i1 = col / n0;
    ff inv_d = ff_make(1.0f), aprev = zero;
    size_t c = (size_t)col;
    double sc = s[c];
    for (int k = 0; k < n2; ++k, c += sk) {
      const double sb = (k + 1 < n2) ? s[c + sk] : 0.0;
      ff v0 = zero, v1 = zero, v2 = zero;
      if (i0 + 1 < n0) v0 = scaled_coupling64(a0, c, sc, s[c + 1]);
      else a0[c] = 0.0;
      if (i1 + 1 < n1) v1 = scaled_coupling64(a1, c, sc, s[c + n0]);
      else a1[c] = 0.0;
      if (k + 1 < n2) v2 = scaled_coupling64(a2, c, sc, sb);
      else a2[c] = 0.0;
      f0[c] = v0.h;
      f1[c] = v1.h;
      f2[c] = v2.h;
      if (line) {
        ff l = zero;
        if (k > 0) {
          l = ff_mul(aprev, inv_d);
          ff d = ff_add_f(ff_neg(ff_mul(l, aprev)), 1.0f);
          if (!(d.h > 1e-30f)) d = ff_make(1.0f);  // not SPD: that row falls back to Jacobi
          inv_d = ff_div(ff_make(1.0f), d);
        }
        lk[c] = l.h;
        dinv[c] = inv_d.h;
        aprev = v2;
      }
      sc = sb;
    }
  }
}

// The float-float path's preparation in one pass per column (update solves, ff_operator): the
// scale factors s = D^-1/2 rounded to FP32 (a similarity transform: any s applied consistently
// gives the same solution, and FP32 s make s_c s_n an exact float product; d s^2 is then 1 only
// to FP32 precision while the refinement takes it as 1, which perturbs the update, not the
// iterate's fixed point), formed from the diagonal by each thread for itself and its neighbours
// (the same rounding everywhere, so the diagonal stays in place) and written to s_out; the
// scaled couplings a s_c s_n in float-float and their FP32 copies; the line factors as in
// k_scale_mixed; and the first refinement sweep (x~ = 0): the inner right-hand side
// fp32(s b) 2^-e with its CG state (k_ir_scale's job) and the norms ||s b||, ||b|| and the
// stopping test (k_ir_residual<true>'s), all in FP32 arithmetic: the scale 2^-e comes from the
// previous solve's first residual, which keeps the scaled values and their squares far from
// the FP32 range limits (a power of two changes no rounding).  When a scaled sum of squares
// leaves [2^-60, 2^60] (the first solve, a jump in scale) the last block sets
// the status kRescaleRhs and the host runs k_ir_residual<true> and k_ir_scale instead (FP64).  The
// kernel has no FP64 arithmetic: GB300's FP64 pipe would bound it.
// This replaces k_diag_rsqrt_sq, k_scale_mixed, the first k_ir_residual and k_ir_scale: the
// diagonal, the couplings and b are read once.  The assembly wrote
// the diagonal (dg) and the unscaled couplings (f0-f2) as floats; f0-f2 are overwritten in
// place by the scaled couplings' leading floats, and their low floats go to l0-l2, where the FP64
// couplings of other operators are.
// One cell of the preparation: scale factors sc (its own), sx, sy, sz (the +1 neighbours'), the
// unscaled couplings e0-e2 (0 towards absent neighbours); writes the scaled operator, s and the
// first right-hand side and returns the scaled axis-2 coupling.
struct PrepOut {
  double* s;
  float *f0, *f1, *f2, *l0, *l1, *l2, *rf;  // the couplings' leading and low floats
};
__device__ __forceinline__ ff prep_cell(const PrepOut& o, size_t c, float e0, float e1, float e2,
                                        float sc, float sx, float sy, float sz, bool hx, bool hy,
                                        bool hz, double bc, float sig, Kahan32& kq, Kahan32& kb) {
  const ff zero = ff_make(0.0f);
  o.s[c] = f2d_scaled(sc, 0);
  ff v0 = zero, v1 = zero, v2 = zero;
  if (hx) v0 = scaled_coupling_f(e0, sc, sx);
  if (hy) v1 = scaled_coupling_f(e1, sc, sy);
  if (hz) v2 = scaled_coupling_f(e2, sc, sz);
  o.f0[c] = v0.h;
  o.f1[c] = v1.h;
  o.f2[c] = v2.h;
  o.l0[c] = v0.l;
  o.l1[c] = v1.l;
  o.l2[c] = v2.l;
  // first sweep: x~ = 0 (the first k_ir_sweep writes x~ without reading it), r~ = s b,
  // kept only as its FP32 form r~ 2^-e (the inner right-hand side), with the sums of
  // squares of r~ 2^-e and b 2^-e (with x~ = 0 the true residual is b) compensated in FP32
  const float qb = ff_hi_of(bc) * sig;
  const float q = sc * qb;
  o.rf[c] = q;
  kq.add(q * q);
  kb.add(qb * qb);
  return v2;
}

// the line factors of level k > 0: l = aprev / d_{k-1}, inv_d = 1 / d_k
__device__ __forceinline__ ff prep_factor(ff aprev, ff& inv_d) {
  const ff l = ff_mul(aprev, inv_d);
  ff d = ff_add_f(ff_neg(ff_mul(l, aprev)), 1.0f);
  if (!(d.h > 1e-30f)) d = ff_make(1.0f);  // not SPD: that row falls back to Jacobi
  inv_d = ff_div(ff_make(1.0f), d);
  return l;
}

// The scalar end of the preparation (last block): norms, test and the first inner system.
__device__ __forceinline__ void prep_tail(CgDevState* ir, CgDevState* in, const double (&tot)[2],
                                          int sig_exp, double ir_rtol, double inner_rtol) {
  if (!(tot[0] >= 0x1p-60 && tot[0] <= 0x1p60 && tot[1] >= 0x1p-60 && tot[1] <= 0x1p60)) {
    // the scaled sums left the FP32 margin (or are 0, inf, NaN): the host recomputes this
    // sweep's residual, norms and test in FP64 (k_ir_residual<true>, k_ir_scale)
    ir->status = kRescaleRhs;
    in->status = kConvergedAtol;  // the inner iterations launched ahead have nothing to do
    return;
  }
  const double inv_sig = pow2d(sig_exp);
  const double rn = sqrt(tot[1]) * inv_sig;
  ir->ir_bnorm = rn;
  ir->ir_rnorm = rn;
  ir->dp = rn;
  ir->a = sqrt(tot[0]) * inv_sig;
  ir->first_a = ir->a;
  if (rn <= fmax(ir_rtol * ir->ir_bnorm, ir->atol))
    ir->status = rn < ir->atol ? kConvergedAtol : kConvergedRtol;
  if (ir->status == 0) {
    ir->rscale = inv_sig;
    in->beta = tot[0];
    in->rnorm0 = sqrt(tot[0]);
    in->ttol = inner_rtol * in->rnorm0;
    in->iter = 0;
    in->its = 0;
    in->dpi = 0.0;
    in->fresh = 1;
    in->status = 0;
  } else {
    in->status = kConvergedAtol;
  }
}

__global__ void __launch_bounds__(128) k_prep_ff(
    PrepOut o, const float* dg, const double* b, float* lk, float* dinv, int n0, int n1, int n2,
    int line, CgDevState* ir, double* partials, double ir_rtol, CgDevState* in, int sig_exp,
    double inner_rtol) {
  grid_begin();
  const int ncol = n0 * n1;
  const size_t sk = (size_t)ncol;
  const float sig = pow2f_of(-sig_exp);
  Kahan32 kq, kb;
  for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < ncol;
       col += gridDim.x * blockDim.x) {
    const int i0 = col % n0, i1 = col / n0;
    const bool hx = i0 + 1 < n0, hy = i1 + 1 < n1;
    ff inv_d = ff_make(1.0f), aprev = ff_make(0.0f);
    size_t c = (size_t)col;
    // level k's inputs are loaded one level ahead (two levels of loads in flight per thread)
    float sc = scale_of(dg[c]);
    float q0 = o.f0[c], q1 = o.f1[c], q2 = o.f2[c];
    float dx = hx ? dg[c + 1] : 1.0f, dy = hy ? dg[c + n0] : 1.0f;
    float dz = n2 > 1 ? dg[c + sk] : 1.0f;
    double bq = b[c];
    for (int k = 0; k < n2; ++k, c += sk) {
      const float e0 = q0, e1 = q1, e2 = q2, ex = dx, ey = dy, ez = dz;
      const double bc = bq;
      const bool hz = k + 1 < n2;
      if (hz) {
        const size_t cn = c + sk;
        q0 = o.f0[cn];
        q1 = o.f1[cn];
        q2 = o.f2[cn];
        dx = hx ? dg[cn + 1] : 1.0f;
        dy = hy ? dg[cn + n0] : 1.0f;
        dz = k + 2 < n2 ? dg[cn + sk] : 1.0f;
        bq = b[cn];
      }
      const float sb = hz ? scale_of(ez) : 0.0f;
      const ff v2 = prep_cell(o, c, e0, e1, e2, sc, scale_of(ex), scale_of(ey), sb, hx, hy, hz, bc,
                              sig, kq, kb);
      if (line) {
        ff l = ff_make(0.0f);
        if (k > 0) l = prep_factor(aprev, inv_d);
        lk[c] = l.h;
        dinv[c] = inv_d.h;
        aprev = v2;
      }
      sc = sb;
    }
  }
  double v[2] = {kq.value(), kb.value()};
  double tot[2];
  if (!grid_sum<2>(v, partials, &ir->arrive[0], tot)) return;
  if (flat_tid() == 0) prep_tail(ir, in, tot, sig_exp, ir_rtol, inner_rtol);
}

// The same preparation for grids whose columns are too few for a march with one thread each to keep
// the loads in flight (a microsecond per level): a block owns 32 columns, its eight warps take the
// cells' part level by level in any order, and only the line factors, which need the level above,
// are left to one warp, from shared memory.  March / split: 40 x 40 x 100 107 / 35 us, 200 x 200 x
// 96 120 / 75, 256 x 256 x 96 129 / 111, 256 x 256 x 128 208 / 202; 300 x 300 x 96 141 / 152, 400 x
// 400 x 96 200 / 232, 600 x 600 x 96 412 / 497, 768 x 768 x 96 846 / 1400, where the march's loads
// already fill the memory pipe and this form's barrier between its two parts empties it.
constexpr int kPrepWarps = 8;
constexpr int kPrepLevels = 190;         // 48 KB of scaled couplings beside the sums' 4 KB
constexpr int kPrepSplitGroups = 2048;   // 65,536 columns (the forms cross at about 80,000)
__global__ void __launch_bounds__(32 * kPrepWarps) k_prep_ff_split(
    PrepOut o, const float* dg, const double* b, float* lk, float* dinv, int n0, int n1, int n2,
    int line, CgDevState* ir, double* partials, double ir_rtol, CgDevState* in, int sig_exp,
    double inner_rtol) {
  grid_begin();
  extern __shared__ float2 prep_sh[];  // [n2][32]
  const int ncol = n0 * n1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t sk = (size_t)ncol;
  const float sig = pow2f_of(-sig_exp);
  Kahan32 kq, kb;
  const int groups = (ncol + 31) / 32;
  for (int g = blockIdx.x; g < groups; g += gridDim.x) {
    const int col = g * 32 + lane;
    const bool act = col < ncol;
    const int i0 = col % n0, i1 = col / n0;
    const bool hx = act && i0 + 1 < n0, hy = act && i1 + 1 < n1;
    __syncthreads();  // the previous group's factors have been read
#pragma unroll 4
    for (int k = warp; k < n2; k += kPrepWarps) {
      if (act) {
        const size_t c = (size_t)col + sk * k;
        const bool hz = k + 1 < n2;
        const float sc = scale_of(dg[c]);
        const float sx = scale_of(hx ? dg[c + 1] : 1.0f), sy = scale_of(hy ? dg[c + n0] : 1.0f);
        const float sz = scale_of(hz ? dg[c + sk] : 1.0f);
        const ff v2 = prep_cell(o, c, o.f0[c], o.f1[c], o.f2[c], sc, sx, sy, sz, hx, hy, hz, b[c],
                                sig, kq, kb);
        prep_sh[k * 32 + lane] = make_float2(v2.h, v2.l);
      }
    }
    __syncthreads();
    if (line && warp == 0 && act) {
      ff inv_d = ff_make(1.0f);
      size_t c = (size_t)col;
      lk[c] = 0.0f;
      dinv[c] = 1.0f;
#pragma unroll 2
      for (int k = 1; k < n2; ++k) {
        c += sk;
        const float2 v = prep_sh[(k - 1) * 32 + lane];
        const ff l = prep_factor(ff_make(v.x, v.y), inv_d);
        lk[c] = l.h;
        dinv[c] = inv_d.h;
      }
    }
  }
  double v[2] = {kq.value(), kb.value()};
  double tot[2];
  if (!grid_sum<2>(v, partials, &ir->arrive[0], tot)) return;
  if (flat_tid() == 0) prep_tail(ir, in, tot, sig_exp, ir_rtol, inner_rtol);
}

// sq = 1 / s for an operator scaled earlier (s already holds D^-1/2)
__global__ void k_inv64(const double* __restrict__ s, double* __restrict__ sq, size_t n) {
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x)
    sq[c] = 1.0 / s[c];
}

// the float-float operator's low floats lie where the FP64 couplings do otherwise
static float* low32(double* a) { return reinterpret_cast<float*>(a); }

int KrylovSolver::prep_mixed(Stencil64& A, cudaStream_t st, bool line,
                             const frehg_solver_config& cfg) {
  const size_t n = A.n;
  FG_TRY(ensure32(n));
  if (line) FG_TRY(ensure_line(n));
  const int nb = reduction_blocks(n, 256, 4);
  const double dn = (double)n;
  const int ncol = A.n0 * A.n1;
  const int lb = (int)std::min<long>((ncol + 127) / 128, kMaxRedBlocks);
  first_done = false;
  if (A.f32_entries && (A.scaled || !ff_operator)) {
    set_error("FP32-form operator outside the float-float preparation");
    return FREHG_ERR_STATE;
  }
  if (!A.scaled) {
    if (ff_operator) {
      if (!A.f32_entries) {
        set_error("the float-float preparation needs the assembly's FP32-form operator");
        return FREHG_ERR_STATE;
      }
      // the refinement state, then one pass: scale factors, scaled operator, FP32 copy, line
      // factors and the first sweep's residual
      CgDevState ir0, in0;
      memset(&ir0, 0, sizeof(ir0));
      memset(&in0, 0, sizeof(in0));
      ir0.atol = cfg.atol;
      in0.max_it = cfg.max_it;
      FG_TRY(set_states(dst, ir0, dst32, in0, st));
      // the first inner right-hand side's scale: 2^-e with 2^(e-1) <= the previous solve's
      // first residual norm < 2^e
      const int sig_exp = pow2_above(first_rnorm[rnorm_slot & 1]);
      const int groups = (ncol + 31) / 32;
      const bool split = groups <= kPrepSplitGroups && A.n2 <= kPrepLevels;
      const size_t split_sh = (size_t)A.n2 * 32 * sizeof(float2);
      if (split && split_sh > 40 * 1024)
        FG_CUDA(cudaFuncSetAttribute(k_prep_ff_split, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)split_sh));
      FG_LAUNCH(prof, st, "k_prep_ff",
                (4.0 + 12.0 + 8.0 + 12.0 + 12.0 + 8.0 + 4.0 + (line ? 8.0 : 0.0)) * dn,
                {
                  const PrepOut o = {r, op32.a0, op32.a1, op32.a2, low32(A.a0), low32(A.a1),
                                     low32(A.a2), rf};
                  const float* dg = reinterpret_cast<const float*>(A.s);
                  if (split)
                    launch_chained(k_prep_ff_split, std::min(groups, 6 * kNumSMs), 32 * kPrepWarps,
                                   split_sh, st, o, dg, A.b, lkf, dinvf, A.n0, A.n1, A.n2,
                                   line ? 1 : 0, dst, partials, cfg.ir_rtol, dst32, sig_exp,
                                   cfg.inner_rtol);
                  else
                    launch_chained(k_prep_ff, lb, 128, 0, st, o, dg, A.b, lkf, dinvf, A.n0, A.n1,
                                   A.n2, line ? 1 : 0, dst, partials, cfg.ir_rtol, dst32, sig_exp,
                                   cfg.inner_rtol);
                });
      FG_CUDA(cudaGetLastError());
      A.scaled = true;
      A.s_in_r = true;
      A.f32_entries = false;
      first_done = true;
      ff_line = line;
      return FREHG_OK;
    }
    FG_LAUNCH(prof, st, "k_diag_rsqrt_sq", 24.0 * dn,
              k_diag_rsqrt_sq<<<nb, 256, 0, st>>>(A.s, r, n));
    FG_LAUNCH(prof, st, "k_scale_mixed", (56.0 + 12.0 + (line ? 8.0 : 0.0)) * dn,
              k_scale_mixed<<<lb, 128, 0, st>>>(A.a0, A.a1, A.a2, A.s, op32.a0, op32.a1,
                                                op32.a2, lkf, dinvf, A.n0, A.n1, A.n2,
                                                line ? 1 : 0));
    FG_CUDA(cudaGetLastError());
    A.scaled = true;
    return FREHG_OK;
  }
  // an operator scaled by an earlier solve.  The float-float preparation's scale factors, operator
  // and line factors are still in place; factors it did not make cannot be made now (A.a2 holds the
  // couplings' low floats)
  if (A.s_in_r) {
    if (!line || ff_line) return FREHG_OK;
    set_error("operator prepared for another preconditioner of the float-float solve; "
              "reassemble it");
    return FREHG_ERR_STATE;
  }
  // else derive sq, the FP32 copy and the factors from it
  FG_LAUNCH(prof, st, "k_inv64", 16.0 * dn, k_inv64<<<nb, 256, 0, st>>>(A.s, r, n));
  FG_LAUNCH(prof, st, "k_to_f32", 36.0 * dn,
            k_to_f32<<<nb, 256, 0, st>>>(A.a0, A.a1, A.a2, op32.a0, op32.a1, op32.a2, n));
  if (line)
    FG_LAUNCH(prof, st, "k_line_factor", 16.0 * dn,
              k_line_factor<<<lb, 128, 0, st>>>(A.a2, lkf, dinvf, ncol, A.n2));
  FG_CUDA(cudaGetLastError());
  return FREHG_OK;
}

int KrylovSolver::ensure_line(size_t n) {
  if (lkf && n <= cap_line) return FREHG_OK;
  cudaFree(lkf);
  cudaFree(dinvf);
  cudaFree(uf);
  cudaFree(pf2);
  lkf = dinvf = uf = pf2 = nullptr;
  FG_CUDA(cudaMalloc(&lkf, n * sizeof(float)));
  FG_CUDA(cudaMalloc(&dinvf, n * sizeof(float)));
  FG_CUDA(cudaMalloc(&uf, n * sizeof(float)));
  FG_CUDA(cudaMalloc(&pf2, n * sizeof(float)));
  cap_line = n;
  return FREHG_OK;
}

int KrylovSolver::solve_mixed(Stencil64& A, double* x_out, const frehg_solver_config& cfg,
                              cudaStream_t st, CgResult* res) {
  const size_t n = A.n;
  FG_TRY(ensure32(n));
  const int nb = reduction_blocks(n, 256, 4);
  const double dn = (double)n;
  const StencilLaunch L = stencil_launch(A.n0, A.n1, A.n2);
  const bool vec4 = (A.n0 % 4) == 0 && getenv("FREHG_NO_VEC4") == nullptr;
  const StencilLaunch L4 = launch_v4(A.n0, A.n1, A.n2);
  const StencilLaunch LR = launch_v4(A.n0, A.n1, A.n2, true);
  FG_CUDA(cudaGetLastError());
  // inner preconditioner: Jacobi (unit diagonal, z = r) or vertical lines
  const bool line = !strcmp(cfg.pc_type, "line");
  const int ncol = A.n0 * A.n1, nzl = A.n2;
  // prep_mixed may have formed the first sweep's residual and its state already
  const bool first_done_here = first_done;
  first_done = false;
  if (!first_done_here) {
    CgDevState ir0, in0;
    memset(&ir0, 0, sizeof(ir0));
    memset(&in0, 0, sizeof(in0));
    ir0.atol = cfg.atol;
    in0.max_it = cfg.max_it;
    FG_TRY(set_states(dst, ir0, dst32, in0, st));
  }
  // where the scale factors are: A.s, or r (as floats) after the float-float preparation
  const double* sv = A.s_in_r ? r : A.s;
  const char* spmv_name = vec4 ? "k32_spmv_v4" : "k32_spmv";
  const char* dir_name = vec4 ? "k32_dir_spmv_v4" : "k32_dir_spmv";

  auto spmv32 = [&](cudaStream_t s) {
    if (vec4)
      k32_spmv_v4<<<L4.grid, L4.block, 0, s>>>(op32.a0, op32.a1, op32.a2, pf, wf, A.n0, A.n1,
                                                A.n2, L4.planes, L4.tiles, dst32, partials);
    else
      k32_spmv<<<L.grid, L.block, 0, s>>>(op32.a0, op32.a1, op32.a2, pf, wf, A.n0, A.n1, A.n2,
                                          L.planes, L.tiles, dst32, partials);
  };
  // one inner iteration; returns at once on the device when the inner solve has ended
  auto iteration = [&](cudaStream_t s, Profiler* pr) {
    if (line) {
      FG_LAUNCH(pr, s, dir_name, 28.0 * dn, {
        if (vec4)
          launch_chained(k32_dir_spmv_v4, L4.grid, L4.block, 0, s, op32.a0, op32.a1, op32.a2, uf,
                         pf, pf2, wf, A.n0, A.n1, A.n2, L4.planes, L4.tiles, dst32, partials);
        else
          launch_chained(k32_dir_spmv, LR.grid, LR.block, 0, s, op32.a0, op32.a1, op32.a2, uf, pf,
                         pf2, wf, A.n0, A.n1, A.n2, LR.planes, LR.tiles, dst32, partials);
      });
      FG_LAUNCH(pr, s, "k32_line_step", 36.0 * dn,
                launch_line_step<false>(xf, rf, pf, pf2, wf, lkf, dinvf, uf, ncol, nzl, dst32,
                                        partials, s));
    } else {
      FG_LAUNCH(pr, s, "k32_p", 12.0 * dn, k32_p<<<nb, 256, 0, s>>>(rf, pf, n, dst32));
      FG_LAUNCH(pr, s, spmv_name, 20.0 * dn, spmv32(s));
      FG_LAUNCH(pr, s, "k32_update", 24.0 * dn,
                k32_update<<<nb, 256, 0, s>>>(xf, rf, pf, wf, n, dst32, partials));
    }
  };
  // Jacobi: long inner solves, captured in chunks (the line solves' few iterations are launched
  // one by one)
  const int chunk = 32;
  const bool graphs = !line && !(prof && prof->on);
  const long shape_key = (long)A.n0 * 1000003L + A.n1;
  if (graphs && (!g32 || g32_key != (const void*)op32.a0 || g_stream32 != st || g_n32 != n ||
                 g32_shape != shape_key)) {
    if (g32) cudaGraphExecDestroy(g32);
    g32 = nullptr;
    cudaStream_t cap_st;
    FG_CUDA(cudaStreamCreateWithFlags(&cap_st, cudaStreamNonBlocking));
    cudaGraph_t graph;
    FG_CUDA(cudaStreamBeginCapture(cap_st, cudaStreamCaptureModeThreadLocal));
    for (int q = 0; q < chunk; ++q) iteration(cap_st, nullptr);
    cudaError_t e = cudaStreamEndCapture(cap_st, &graph);
    cudaStreamDestroy(cap_st);
    if (e != cudaSuccess) {
      set_error("graph capture failed: %s", cudaGetErrorString(e));
      return FREHG_ERR_CUDA;
    }
    e = cudaGraphInstantiate(&g32, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
      set_error("graph instantiate failed: %s", cudaGetErrorString(e));
      return FREHG_ERR_CUDA;
    }
    g32_key = op32.a0;
    g_stream32 = st;
    g_n32 = n;
    g32_shape = shape_key;
  }

  // both states at the host
  auto fetch = [&]() -> int {
    FG_CUDA(cudaGetLastError());
    FG_TRY(fetch_small2(hst, dst, hst32, dst32, sizeof(CgDevState), st));
    FG_CUDA(cudaStreamSynchronize(st));
    if (prof && prof->on) FG_TRY(prof->flush());
    return FREHG_OK;
  };
  // the first sweep's residual, norms and test in FP64, and its right-hand side
  auto first_residual = [&]() {
    FG_LAUNCH(prof, st, "k_ir_residual0", 24.0 * dn,
              k_ir_residual<true><<<L.grid, L.block, 0, st>>>(
                  A.a0, A.a1, A.a2, sv, r, A.b, x, rres, A.n0, A.n1, A.n2, L.planes, L.tiles,
                  dst, partials, cfg.ir_rtol));
    FG_LAUNCH(prof, st, "k_ir_scale", 12.0 * dn,
              k_ir_scale<<<nb, 256, 0, st>>>(rres, rf, n, dst, dst32, partials, cfg.inner_rtol));
  };
  // the inner solve's start: z0 = M^-1 r0 and r0.z0
  auto line_first = [&]() {
    if (line)
      FG_LAUNCH(prof, st, "k32_line_first", 16.0 * dn,
                launch_line_step<true>(xf, rf, pf, pf2, wf, lkf, dinvf, uf, ncol, nzl, dst32,
                                       partials, st));
  };
  // x~ += 2^k e and the next true residual with the next inner system (both return at once on the
  // device while the inner solve still runs)
  auto sweep_end = [&]() {
    if (A.s_in_r) {
      const SweepArgs sa = {op32.a0, op32.a1, op32.a2, low32(A.a0), low32(A.a1), low32(A.a2),
                            reinterpret_cast<const float*>(A.s), xf, A.b, x,
                            reinterpret_cast<float2*>(rres), rf};
      FG_LAUNCH(prof, st, "k_ir_update", 24.0 * dn,
                launch_chained(k_ir_update_exact, nb, 256, 0, st, x, xf, n, dst, dst32));
      FG_LAUNCH(prof, st, "k_ir_sweep", 56.0 * dn,
                launch_chained(k_ir_sweep, L.grid, L.block, 0, st, sa, A.n0, A.n1, A.n2, L.planes,
                               L.tiles, dst, dst32, partials, cfg.ir_rtol, cfg.inner_rtol));
    } else {
      FG_LAUNCH(prof, st, "k_ir_update", 20.0 * dn,
                k_ir_update<<<nb, 256, 0, st>>>(x, xf, n, dst, dst32));
      FG_LAUNCH(prof, st, "k_ir_residual", 52.0 * dn,
                k_ir_residual<false><<<L.grid, L.block, 0, st>>>(
                    A.a0, A.a1, A.a2, A.s, r, A.b, x, rres, A.n0, A.n1, A.n2, L.planes, L.tiles, dst,
                    partials, cfg.ir_rtol, rf, dst32, cfg.inner_rtol));
    }
  };

  // Rounds of: the inner solve's start (on a new sweep), some inner iterations, the sweep's end,
  // and one read-back of both states.  The host launches ahead of what it knows: every kernel
  // returns at once when it has nothing to do, and what a round did is read off the states after
  // it.  The iterations launched are those that recent sweeps took (spec32: first sweeps, later
  // ones); a sweep that takes more goes on in the next round.
  const int max_sweeps = 60;
  bool fcg_fallback = false;
  const bool dbg = getenv("FREHG_DEBUG_IR") != nullptr;
  if (!first_done_here) first_residual();
  if (net.net != nullptr) FG_TRY(fetch());  // the network's loop is host-driven
  int sweeps = 0;     // complete sweeps
  int round = 0;      // rounds of the current sweep
  int total = 0;      // inner iterations
  // a sweep's start (on its first round) and some inner iterations; the number launched
  auto launch_sweep = [&](int sweep, int rnd) {
    if (rnd == 0) line_first();
    const int spec = spec32[sweep > 0];
    if (graphs && (rnd > 0 || spec > 8)) {
      cudaGraphLaunch(g32, st);
      if (prof) prof->launches += 3 * chunk;
      return chunk;
    }
    // An idle iteration costs 5 to 8 us, another round about 25 (two idle launches, the read-back).
    // Sweeps that run over their prediction do so by one iteration mostly (2, then more); the few
    // long ones vary between 1 and 27 from solve to solve, so they go on in eights.
    const int its = rnd == 0 ? std::max(1, std::min(spec, 8))
                             : (spec > 8 ? 8 : 2 << std::min(rnd - 1, 2));
    for (int q = 0; q < its; ++q) iteration(st, prof);
    return its;
  };
  for (;;) {
    int launched = 0, ends = 1;
    // a sweep that starts with the network's budget (twice the reference solve's inner
    // iterations) spent runs without it, as do the later ones
    if (net.net != nullptr && !fcg_fallback && net.max_inner > 0 && total >= net.max_inner)
      fcg_fallback = true;
    if (net.net != nullptr && !fcg_fallback && hst->status == 0) {
      if (!zf) FG_CUDA(cudaMalloc(&zf, cap32 * sizeof(float)));
      const int lb = (int)std::min<long>((ncol + 127) / 128, kMaxRedBlocks);
      const int check = 4;
      for (int it = 0; it < cfg.max_it && hst32->status == 0; ++it) {
        FG_TRY(unet_apply(net.net, A.n0, A.n1, A.n2, rf, net.lnk, net.cap, zf, st));
        if (line)
          FG_LAUNCH(prof, st, "k32_line_apply", 32.0 * dn,
                    k32_line_apply<<<lb, 128, 0, st>>>(rf, lkf, dinvf, uf, zf, ncol, nzl, 1));
        else
          FG_LAUNCH(prof, st, "k_add_f32", 12.0 * dn, k_add_f32<<<nb, 256, 0, st>>>(zf, rf, n));
        FG_LAUNCH(prof, st, "k_fcg_beta", 8.0 * dn,
                  k_fcg_beta<<<nb, 256, 0, st>>>(zf, wf, n, dst32, partials));
        FG_LAUNCH(prof, st, "k_fcg_p", 16.0 * dn,
                  k_fcg_p<<<nb, 256, 0, st>>>(zf, pf, rf, n, dst32, partials));
        FG_LAUNCH(prof, st, spmv_name, 20.0 * dn, spmv32(st));
        FG_LAUNCH(prof, st, "k32_update", 24.0 * dn,
                  k32_update<<<nb, 256, 0, st>>>(xf, rf, pf, wf, n, dst32, partials));
        FG_CUDA(cudaGetLastError());
        if ((it + 1) % check == 0) {
          FG_TRY(fetch());
          if (net.max_inner > 0 && total + hst32->its > net.max_inner) {
            fcg_fallback = true;  // too slow: plain CG from the next sweep on (the iterate is kept)
            break;
          }
        }
      }
      if (fcg_fallback && hst32->status == 0) {  // this sweep's inner solve ends here
        const int stop = kDivergedIts;
        FG_CUDA(cudaMemcpyAsync(&dst32->status, &stop, sizeof(int), cudaMemcpyHostToDevice, st));
      }
    } else {
      launched = launch_sweep(sweeps, round);
      // where the last solve took a second sweep, it is launched behind the first without a
      // read-back between them (7 us of a sweep's 70 at 40 x 40 x 100)
      if (line && net.net == nullptr && sweeps == 0 && round == 0 && two_sweeps) {
        sweep_end();
        launched += launch_sweep(1, 0);
        ends = 2;
      }
    }
    sweep_end();
    FG_TRY(fetch());
    if (hst->status == kRescaleRhs) {
      // the preparation could not scale its right-hand side: FP64, and the sweep again
      const int zero = 0;
      FG_CUDA(cudaMemcpyAsync(&dst->status, &zero, sizeof(int), cudaMemcpyHostToDevice, st));
      first_residual();
      if (net.net != nullptr) FG_TRY(fetch());
      continue;
    }
    if (hst->first_a > 0.0 && std::isfinite(hst->first_a))
      first_rnorm[rnorm_slot & 1] = hst->first_a;
    const int done = hst->its + (hst->status == 0 ? hst32->its : 0) - total;
    if (prof && prof->on && launched > 0) {
      const int64_t idle = std::max(0, launched - std::max(0, done));
      if (line) {
        prof->idle(dir_name, idle);
        prof->idle("k32_line_step", idle);
      } else {
        prof->idle("k32_p", idle);
        prof->idle(spmv_name, idle);
        prof->idle("k32_update", idle);
      }
      if (const int idle_ends = ends - (hst->ir_its - sweeps); idle_ends > 0) {
        prof->idle("k_ir_update", idle_ends);
        prof->idle(A.s_in_r ? "k_ir_sweep" : "k_ir_residual", idle_ends);
      }
    }
    if (dbg)
      fprintf(stderr,
              "ir sweep %d round %d: launched %d done %d; true |r| %.3e / |b| %.3e status %d\n", sweeps, round, launched, done, hst->ir_rnorm, hst->ir_bnorm, hst->status);
    total += done;
    ++round;
    for (; sweeps < hst->ir_its; ++sweeps, round = hst32->its > 0 ? 1 : 0)
      if (launched > 0)
        spec32[sweeps > 0] =
            std::max(hst->sweep_its[std::min(sweeps, 3)], spec32[sweeps > 0] - 1);
    if (hst->status != 0 || sweeps >= max_sweeps) break;
  }
  two_sweeps = sweeps > 1;
  // stopped before the first update: x~ = 0
  if (sweeps == 0)
    FG_LAUNCH(prof, st, "k_zero64", 8.0 * dn, k_zero64<<<nb, 256, 0, st>>>(x, n));
  FG_TRY(finish64(A, x_out, st, res, nb));
  res->its = total;
  res->inner_its = total;
  res->ir_its = sweeps;
  res->fallback = fcg_fallback ? 1 : 0;
  res->rnorm = hst->ir_rnorm;
  res->reason = hst->status;
  if (hst->status <= 0) {
    set_error("mixed-precision refinement stopped after %d sweeps: true residual %g vs %g * %g "
              "(reason %d)", sweeps, hst->ir_rnorm, cfg.ir_rtol, hst->ir_bnorm, hst->status);
    return hst->status == kDivergedNanOrInf ? FREHG_ERR_NONFINITE : FREHG_ERR_NOT_CONVERGED;
  }
  return FREHG_OK;
}

}  // namespace fg
