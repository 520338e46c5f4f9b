// Krylov solver on the GPU: Jacobi-preconditioned CG for a 7-point SPD stencil.
//
// Replaces the PETSc KSP solve behind PetscLinearSolver::solve
// (src/linear/backends/PetscLinearSolver.cpp:200-220): KSPSolve_CG with the preconditioned
// residual norm, zero initial guess and KSPConvergedDefault (converged when
// ||B r|| <= max(rtol*||B b||, atol); divergence when ||B r|| >= 1e4*||B b||, NaN/Inf,
// indefinite matrix or preconditioner, or max_it).
//
// GB300 design:
//  * The operator is scaled once per solve to unit diagonal: A~ = D^-1/2 A D^-1/2.  CG on A~
//    is Jacobi-PCG on A (x~ = D^1/2 x, r~ = D^-1/2 r, beta = r.z = r~.r~, p'Ap = p~'A~p~,
//    ||B r|| = ||s r~|| with s = D^-1/2), so the diagonal is never stored or multiplied and
//    no divisions remain in the loop.
//  * Three phases per iteration (p-update, stencil SpMV + p.w, update + two norms).  By default
//    the whole loop is one cooperative launch with its vectors in registers (k_cg_solve, up to
//    622,592 unknowns).  Larger systems, and on request or under profiling all, run iterations as
//    one cooperative launch each (k_cg_iter, the phases separated by two bounded grid barriers;
//    by default up to kFusedAutoCells unknowns) or as three kernels; the last reduction ends in the
//    last-arriving block, which also runs the scalar part of the algorithm (beta, stopping
//    test) on the device.  Launches of a converged solve return at once, so
//    iterations are captured in a CUDA graph of `chunk` iterations and the host only reads
//    the status between chunks.  Reductions are deterministic (fixed block partition, fixed
//    summation tree).
//  * FP64 is 1/64 of the FP32 rate on GB300, so the kernels are arranged to keep the FP64
//    instruction count per cell low (13 FMA-class ops per iteration) as well as the bytes.
#include "internal.h"
#include "reduce.cuh"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>

namespace fg {

// KSPConvergedDefault
__device__ __forceinline__ int converged_test(CgDevState* s, double rnorm) {
  if (isnan(rnorm) || isinf(rnorm)) return kDivergedNanOrInf;
  if (rnorm <= s->ttol) return rnorm < s->atol ? kConvergedAtol : kConvergedRtol;
  if (s->divtol > 0.0 && rnorm >= s->divtol * s->rnorm0) return kDivergedDtol;
  return 0;
}

// ------------------------------------------------------------------------------------------
// geometry helpers

StencilLaunch stencil_launch(int n0, int n1, int n2) {
  StencilLaunch L;
  L.block = dim3(32, 8, 1);
  const int t0 = (n0 + 31) / 32, t1 = (n1 + 7) / 8;
  const long tiles = (long)t0 * t1;
  // about two waves of 8 resident (32 x 8)-thread blocks per SM, fewer on small grids: 8 cells per
  // thread, down to two blocks per SM, since each block's sums and its uneven share cost the FP64
  // pipe more than the cells do (FP64 assembly of 101 x 77 x 53: 159 us with 1 to 2 cells per
  // thread, 106 with 8).  Whole passes with 4 / 8 / 16 cells per thread: FP64 Picard of 101 x 77 x 53
  // 8.44 / 7.74 / 7.75 ms, PCA of 120 x 110 x 90 3.87 / 3.82 / 3.88 and of 90 x 75 x 60 1.85 / 1.79 /
  // 1.80, float-float Picard of 203 x 149 x 96 11.7 / 11.4 / 12.0; of 100 x 90 x 96, where 4 is the
  // best, 5.02 / 5.19 / 5.49; 40 x 40 x 100 and 256 x 256 x 128 the same.  The launch shape, and with
  // it the summation tree of the reductions, depends on the grid sizes only
  const long want = (long)n0 * n1 * n2 / 2048;
  const long target = std::min((long)kNumSMs * 8 * 2, std::max((long)kNumSMs * 2, want));
  long z = target / (tiles > 0 ? tiles : 1);
  if (z < 1) z = 1;
  if (z > n2) z = n2;
  int planes = (int)((n2 + z - 1) / z);
  z = (n2 + planes - 1) / planes;
  // blocks stride over tiles when there are more tiles than reduction partial slots
  long gx = tiles;
  const long cap = kMaxRedBlocks / z;
  if (gx > cap) gx = cap;
  L.planes = planes;
  L.tiles = (int)tiles;
  L.grid = dim3((unsigned)gx, (unsigned)z, 1);
  return L;
}

namespace {
__global__ void k_fetch_words(const unsigned* src, unsigned* dst, int words) {
  grid_begin();
  for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
}
}  // namespace

int alloc_mapped(void** host, size_t bytes) {
  FG_CUDA(cudaHostAlloc(host, bytes, cudaHostAllocMapped));
  return FREHG_OK;
}

int fetch_small(void* host_mapped, const void* dev, size_t bytes, cudaStream_t st) {
  void* d = nullptr;
  FG_CUDA(cudaHostGetDevicePointer(&d, host_mapped, 0));
  launch_chained(k_fetch_words, 1, 32, 0, st, static_cast<const unsigned*>(dev),
                 static_cast<unsigned*>(d), (int)(bytes / 4));
  FG_CUDA(cudaGetLastError());
  return FREHG_OK;
}

namespace {
__global__ void k_fetch_words2(const unsigned* src, unsigned* dst, const unsigned* src2,
                               unsigned* dst2, int words) {
  grid_begin();
  for (int i = threadIdx.x; i < words; i += blockDim.x) {
    dst[i] = src[i];
    dst2[i] = src2[i];
  }
}
}  // namespace

int fetch_small2(void* host_mapped, const void* dev, void* host_mapped2, const void* dev2,
                 size_t bytes, cudaStream_t st) {
  void *d = nullptr, *d2 = nullptr;
  FG_CUDA(cudaHostGetDevicePointer(&d, host_mapped, 0));
  FG_CUDA(cudaHostGetDevicePointer(&d2, host_mapped2, 0));
  launch_chained(k_fetch_words2, 1, 32, 0, st, static_cast<const unsigned*>(dev),
                 static_cast<unsigned*>(d), static_cast<const unsigned*>(dev2),
                 static_cast<unsigned*>(d2), (int)(bytes / 4));
  FG_CUDA(cudaGetLastError());
  return FREHG_OK;
}

namespace {
__global__ void k_set_states(CgDevState* a, CgDevState va, CgDevState* b, CgDevState vb) {
  grid_begin();
  *a = va;
  if (b) *b = vb;
}
}  // namespace

int set_states(CgDevState* a, const CgDevState& va, CgDevState* b, const CgDevState& vb,
               cudaStream_t st) {
  FG_CUDA(launch_chained(k_set_states, 1, 1, 0, st, a, va, b, vb));
  return FREHG_OK;
}

int reduction_blocks(size_t n, int threads, int per_thread) {
  size_t b = (n + (size_t)threads * per_thread - 1) / ((size_t)threads * per_thread);
  if (b < 1) b = 1;
  if (b > (size_t)kNumSMs * 8) b = (size_t)kNumSMs * 8;
  return (int)b;
}

// ------------------------------------------------------------------------------------------
// operator scaling

__global__ void k_diag_rsqrt(double* s, size_t n) {
  grid_begin();
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x) {
    double d = s[c];
    if (d == 0.0) d = 1.0;  // PCJacobi replaces a zero diagonal entry by 1
    s[c] = rsqrt(d);        // NaN for d < 0: the solve then stops with DIVERGED_NANORINF
  }
}

__global__ void k_scale_offdiag(double* a0, double* a1, double* a2, const double* s, int n0, int n1,
                                int n2, int planes, int tiles) {
  grid_begin();
  const int t0 = (n0 + 31) / 32;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int i0 = (tile % t0) * 32 + threadIdx.x;
    const int i1 = (tile / t0) * 8 + threadIdx.y;
    if (i0 >= n0 || i1 >= n1) continue;
    const size_t s01 = (size_t)n0 * n1;
    const int kb = blockIdx.y * planes;
    const int ke = min(n2, kb + planes);
    for (int k = kb; k < ke; ++k) {
      const size_t c = (size_t)i0 + (size_t)n0 * i1 + s01 * k;
      const double sc = s[c];
      if (i0 + 1 < n0) a0[c] *= sc * s[c + 1]; else a0[c] = 0.0;
      if (i1 + 1 < n1) a1[c] *= sc * s[c + n0]; else a1[c] = 0.0;
      if (k + 1 < n2) a2[c] *= sc * s[c + s01]; else a2[c] = 0.0;
    }
  }
}

// ------------------------------------------------------------------------------------------
// FP64 CG kernels

// r~ = s b, x~ = 0; ||B b|| and beta = r~.r~; iteration-0 stopping test.
__global__ void k_cg_init(const double* s, const double* b, double* x, double* r, size_t n,
                          CgDevState* st, double* partials) {
  grid_begin();
  double v[2] = {0.0, 0.0};
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x) {
    const double sc = s[c];
    const double rc = sc * b[c];
    r[c] = rc;
    x[c] = 0.0;
    v[0] = fma(rc, rc, v[0]);
    const double z = sc * rc;
    v[1] = fma(z, z, v[1]);
  }
  double tot[2];
  if (!grid_sum<2>(v, partials, &st->arrive[0], tot)) return;
  if (flat_tid() == 0) {
    const double dp = sqrt(tot[1]);
    st->dp = dp;
    st->rnorm0 = dp;
    st->ttol = fmax(st->rtol * dp, st->atol);
    st->its = 0;
    st->iter = 0;
    st->dpi = 0.0;
    st->beta = tot[0];
    st->status = converged_test(st, dp);
    if (!st->status && st->beta == 0.0) {  // loop top of iteration 0
      st->its = 1;
      st->status = kConvergedAtol;
    }
  }
}

// p = r~ (first iteration) or p = r~ + bcoef p   (16-byte vector accesses)
__global__ void k_cg_p(const double* __restrict__ r, double* __restrict__ p, size_t n,
                       const CgDevState* st) {
  if (st->status) return;
  const double bc = st->bcoef;
  const bool first = st->iter == 0;
  const size_t gid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const double2* r2 = reinterpret_cast<const double2*>(r);
  double2* p2 = reinterpret_cast<double2*>(p);
  for (size_t q = gid; q < n / 2; q += stride) {
    const double2 rv = r2[q];
    double2 pv;
    if (first) {
      pv = rv;
    } else {
      pv = p2[q];
      pv.x = fma(bc, pv.x, rv.x);
      pv.y = fma(bc, pv.y, rv.y);
    }
    p2[q] = pv;
  }
  if ((n & 1) && gid == 0) p[n - 1] = first ? r[n - 1] : fma(bc, p[n - 1], r[n - 1]);
}

// w = A~ p (unit diagonal) and p.w; the last block forms alpha.
template <typename T, typename Acc>
__device__ __forceinline__ Acc spmv_cell(const T* __restrict__ p, const T* __restrict__ a0,
                                         const T* __restrict__ a1, size_t c, int i0, int i1,
                                         int n0, int n1, T pc) {
  Acc v = (Acc)pc;
  if (i0 > 0) v = fma((Acc)a0[c - 1], (Acc)p[c - 1], v);
  if (i0 + 1 < n0) v = fma((Acc)a0[c], (Acc)p[c + 1], v);
  if (i1 > 0) v = fma((Acc)a1[c - n0], (Acc)p[c - n0], v);
  if (i1 + 1 < n1) v = fma((Acc)a1[c], (Acc)p[c + n0], v);
  return v;
}

// p.w known: the iteration's alpha, or the end of the solve
__device__ __forceinline__ void cg_alpha(CgDevState* st, double dpi) {
  st->its = st->iter + 1;
  if (dpi == 0.0 || (st->iter > 0 && ((dpi > 0.0) != (st->dpi > 0.0))) || isnan(dpi)) {
    st->status = isnan(dpi) ? kDivergedNanOrInf : kDivergedIndefiniteMat;
    return;
  }
  st->dpiold = st->dpi;
  st->dpi = dpi;
  st->a = st->beta / dpi;
}

__global__ void __launch_bounds__(256) k_cg_spmv(const double* __restrict__ a0,
                                                 const double* __restrict__ a1,
                                                 const double* __restrict__ a2,
                                                 const double* __restrict__ p,
                                                 double* __restrict__ w, int n0, int n1, int n2,
                                                 int planes, int tiles, CgDevState* st,
                                                 double* partials) {
  if (st->status) return;
  const int t0 = (n0 + 31) / 32;
  double acc[1] = {0.0};
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int i0 = (tile % t0) * 32 + threadIdx.x;
    const int i1 = (tile / t0) * 8 + threadIdx.y;
    if (i0 >= n0 || i1 >= n1) continue;
    const size_t s01 = (size_t)n0 * n1;
    const int kb = blockIdx.y * planes;
    const int ke = min(n2, kb + planes);
    size_t c = (size_t)i0 + (size_t)n0 * i1 + s01 * kb;
    double pm = 0.0, am = 0.0;
    if (kb > 0) {
      pm = p[c - s01];
      am = a2[c - s01];
    }
    double pc = p[c];
    for (int k = kb; k < ke; ++k) {
      const double pp = (k + 1 < n2) ? p[c + s01] : 0.0;
      const double ac = a2[c];
      double v = spmv_cell<double, double>(p, a0, a1, c, i0, i1, n0, n1, pc);
      v = fma(am, pm, v);
      v = fma(ac, pp, v);
      w[c] = v;
      acc[0] = fma(pc, v, acc[0]);
      pm = pc;
      pc = pp;
      am = ac;
      c += s01;
    }
  }
  double tot[1];
  if (!grid_sum<1>(acc, partials, &st->arrive[1], tot)) return;
  if (flat_tid() == 0) cg_alpha(st, tot[0]);
}

// The scalar end of an iteration (last block): ||B r|| = sqrt(tot[1]) and the stopping test,
// beta = r~.r~ = tot[0] and the next direction's coefficient.
__device__ __forceinline__ void cg_update_tail(CgDevState* st, const double (&tot)[2]) {
  const double dp = sqrt(tot[1]);
  st->dp = dp;
  const int reason = converged_test(st, dp);
  if (reason) {
    st->status = reason;
    return;
  }
  st->betaold = st->beta;
  st->beta = tot[0];
  st->iter += 1;
  if (st->iter >= st->max_it) {
    st->status = kDivergedIts;
    return;
  }
  st->its = st->iter + 1;
  if (st->beta == 0.0) {
    st->status = kConvergedAtol;
    return;
  }
  st->bcoef = st->beta / st->betaold;
  if (st->bcoef < 0.0) st->status = kDivergedIndefinitePc;
}

// x~ += a p, r~ -= a w, then ||B r|| and beta = r~.r~; the last block runs the stopping test
// and prepares the next iteration's beta ratio.
__global__ void k_cg_update(double* __restrict__ x, double* __restrict__ r,
                            const double* __restrict__ p, const double* __restrict__ w,
                            const double* __restrict__ s, size_t n, CgDevState* st,
                            double* partials) {
  if (st->status) return;
  const double a = st->a;
  double v[2] = {0.0, 0.0};
  const size_t gid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  double2* x2 = reinterpret_cast<double2*>(x);
  double2* r2 = reinterpret_cast<double2*>(r);
  const double2* p2 = reinterpret_cast<const double2*>(p);
  const double2* w2 = reinterpret_cast<const double2*>(w);
  const double2* s2 = reinterpret_cast<const double2*>(s);
  for (size_t q = gid; q < n / 2; q += stride) {
    double2 xv = x2[q], rv = r2[q];
    const double2 pv = p2[q], wv = w2[q], sv = s2[q];
    xv.x = fma(a, pv.x, xv.x);
    xv.y = fma(a, pv.y, xv.y);
    rv.x = fma(-a, wv.x, rv.x);
    rv.y = fma(-a, wv.y, rv.y);
    x2[q] = xv;
    r2[q] = rv;
    v[0] = fma(rv.x, rv.x, v[0]);
    v[0] = fma(rv.y, rv.y, v[0]);
    const double zx = sv.x * rv.x, zy = sv.y * rv.y;
    v[1] = fma(zx, zx, v[1]);
    v[1] = fma(zy, zy, v[1]);
  }
  if ((n & 1) && gid == 0) {
    const size_t c = n - 1;
    x[c] = fma(a, p[c], x[c]);
    const double rc = fma(-a, w[c], r[c]);
    r[c] = rc;
    v[0] = fma(rc, rc, v[0]);
    const double z = s[c] * rc;
    v[1] = fma(z, z, v[1]);
  }
  double tot[2];
  if (!grid_sum<2>(v, partials, &st->arrive[2], tot)) return;
  if (flat_tid() == 0) cg_update_tail(st, tot);
}

// One Jacobi-PCG iteration (KSPSolve_CG's loop body) in one cooperative launch, all blocks
// resident: the direction p = r~ + bcoef p (p = r~ in iteration 0), a grid barrier, w = A~ p
// with the block partials of p.w, a grid barrier after which every block sums the same
// partials in the same order and forms alpha itself, then x~ += alpha p, r~ -= alpha w and the
// two norms, reduced by the last block to arrive, which runs the stopping test (cg_update_tail).
// The arithmetic per cell is that of k_cg_p, k_cg_spmv and k_cg_update.  Work units (a
// 32 x 8-column tile over a chunk of `planes` planes) are dealt round-robin to the blocks, the
// same units to the same block in all three phases, so the only values a block reads that
// another block wrote in this launch are the neighbours' directions of the stencil product;
// every direction read goes through L2 (ld.global.cg), since L1 is not coherent within a
// launch.  The iteration's scalars are read once at the start, before the first barrier, so
// that block 0 may update them after the second.
__global__ void __launch_bounds__(256) k_cg_iter(const double* __restrict__ a0,
                                                 const double* __restrict__ a1,
                                                 const double* __restrict__ a2,
                                                 const double* __restrict__ s,
                                                 double* __restrict__ x, double* __restrict__ r,
                                                 double* __restrict__ p, double* __restrict__ w,
                                                 int n0, int n1, int n2, int planes, int tiles,
                                                 CgDevState* st, double* partials) {
  if (st->status) return;
  const double bc = st->bcoef, beta = st->beta, dpi_prev = st->dpi;
  const int iter = st->iter;
  const int t0 = (n0 + 31) / 32;
  const size_t s01 = (size_t)n0 * n1;
  const int units = tiles * ((n2 + planes - 1) / planes);
  const int nb = flat_nblocks(), bid = flat_bid();
  // 1. direction
  for (int u = bid; u < units; u += nb) {
    const int tile = u % tiles, kb = (u / tiles) * planes, ke = min(n2, kb + planes);
    const int i0 = (tile % t0) * 32 + threadIdx.x;
    const int i1 = (tile / t0) * 8 + threadIdx.y;
    if (i0 >= n0 || i1 >= n1) continue;
    size_t c = (size_t)i0 + (size_t)n0 * i1 + s01 * kb;
    for (int k = kb; k < ke; ++k, c += s01) {
      const double rc = r[c];
      p[c] = iter == 0 ? rc : fma(bc, __ldcg(p + c), rc);
    }
  }
  if (!grid_barrier(&st->bar_count, &st->bar_gen, &st->bar_timeout)) {
    if (flat_tid() == 0) atomicExch(&st->status, (int)kGridBarrierTimeout);
    return;
  }
  // 2. stencil product and p.w
  double acc[1] = {0.0};
  for (int u = bid; u < units; u += nb) {
    const int tile = u % tiles, kb = (u / tiles) * planes, ke = min(n2, kb + planes);
    const int i0 = (tile % t0) * 32 + threadIdx.x;
    const int i1 = (tile / t0) * 8 + threadIdx.y;
    if (i0 >= n0 || i1 >= n1) continue;
    size_t c = (size_t)i0 + (size_t)n0 * i1 + s01 * kb;
    double pm = 0.0, am = 0.0;
    if (kb > 0) {
      pm = __ldcg(p + c - s01);
      am = a2[c - s01];
    }
    double pc = __ldcg(p + c);
    for (int k = kb; k < ke; ++k) {
      const double pp = (k + 1 < n2) ? __ldcg(p + c + s01) : 0.0;
      const double ac = a2[c];
      double v = pc;
      if (i0 > 0) v = fma(a0[c - 1], __ldcg(p + c - 1), v);
      if (i0 + 1 < n0) v = fma(a0[c], __ldcg(p + c + 1), v);
      if (i1 > 0) v = fma(a1[c - n0], __ldcg(p + c - n0), v);
      if (i1 + 1 < n1) v = fma(a1[c], __ldcg(p + c + n0), v);
      v = fma(am, pm, v);
      v = fma(ac, pp, v);
      w[c] = v;
      acc[0] = fma(pc, v, acc[0]);
      pm = pc;
      pc = pp;
      am = ac;
      c += s01;
    }
  }
  __shared__ double sh[256];
  __shared__ double dpi_sh;
  double* pw = partials + 3 * (size_t)kMaxRedBlocks;
  block_sum<1>(acc, sh);
  if (flat_tid() == 0) pw[bid] = acc[0];
  if (!grid_barrier(&st->bar_count, &st->bar_gen, &st->bar_timeout)) {
    if (flat_tid() == 0) atomicExch(&st->status, (int)kGridBarrierTimeout);
    return;
  }
  double t[1] = {0.0};
  for (int b = flat_tid(); b < nb; b += flat_nthreads()) t[0] += __ldcg(&pw[b]);
  block_sum<1>(t, sh);
  if (flat_tid() == 0) dpi_sh = t[0];
  __syncthreads();
  const double dpi = dpi_sh;
  const bool lead = bid == 0 && flat_tid() == 0;
  if (dpi == 0.0 || (iter > 0 && ((dpi > 0.0) != (dpi_prev > 0.0))) || isnan(dpi)) {
    if (lead) {
      st->its = iter + 1;
      st->status = isnan(dpi) ? kDivergedNanOrInf : kDivergedIndefiniteMat;
    }
    return;
  }
  const double a = beta / dpi;
  if (lead) {
    st->its = iter + 1;
    st->dpiold = dpi_prev;
    st->dpi = dpi;
    st->a = a;
  }
  // 3. update and norms
  double v[2] = {0.0, 0.0};
  for (int u = bid; u < units; u += nb) {
    const int tile = u % tiles, kb = (u / tiles) * planes, ke = min(n2, kb + planes);
    const int i0 = (tile % t0) * 32 + threadIdx.x;
    const int i1 = (tile / t0) * 8 + threadIdx.y;
    if (i0 >= n0 || i1 >= n1) continue;
    size_t c = (size_t)i0 + (size_t)n0 * i1 + s01 * kb;
    for (int k = kb; k < ke; ++k, c += s01) {
      x[c] = fma(a, __ldcg(p + c), x[c]);
      const double rc = fma(-a, w[c], r[c]);
      r[c] = rc;
      v[0] = fma(rc, rc, v[0]);
      const double z = s[c] * rc;
      v[1] = fma(z, z, v[1]);
    }
  }
  double tot[2];
  if (!grid_sum<2>(v, partials, &st->arrive[2], tot)) return;
  if (flat_tid() == 0) cg_update_tail(st, tot);
}

// The whole loop of a solve in one cooperative launch: every block owns blockDim x K consecutive
// cells, each thread K of them, whose x, r, p and w stay in its registers; the operator comes
// from L1 (32 bytes a cell, read-only: it stays there for the block's cells), and the neighbours'
// values go through the L2.  A reduction ends in every block: after its barrier each sums the
// same partials in the same order and runs the same scalar steps, so nothing is waited for
// twice.  Same arithmetic per cell as the three kernels; an absent neighbour's product is with
// the zero coupling that the operator holds there.
//   REDIR: two grid-wide exchanges an iteration (p.w; the norms, behind which r is there): the
//   neighbours' directions are formed from r and the previous directions, six more FP64
//   instructions per cell.  Else the directions are written and the blocks that own neighbouring
//   cells waited for.
// An exchange between a few blocks is one trip through the L2: each block writes its partial sum
// and the exchange's number as one 16-byte word, and a warp of each block reads all blocks' words
// until they carry that number (numbers are never reused: the solver counts its solves).  With
// many blocks the readers hold up the writers (32,768 cells, 128 blocks: 14.2 us an iteration),
// and a counter with one reader per block comes first (9.7).
// The FP64 unit of an SM (19 clocks per warp instruction, 64 and more in a chain) sets the
// shape: few warps per block (a reduction costs each of them five steps), as many cells per thread
// as fill the SMs evenly, no square root and no FP64 comparison in the loop (the norms' squares
// are compared as integers), and the division for beta done ahead by another warp.
// A solve with 73 to 96 iterations, this / three kernels in graph chunks: 512 cells 0.51 / 1.3 ms,
// 4,096 0.80 / 1.7, 32,768 1.03 / 1.86, 160,000 1.65 / 2.56, 412,000 2.1 / 3.6, 524,288 2.3 / 4.0.
constexpr int kSolveThreads = 512;  // at most
constexpr int kSolveCells = 8;      // per thread, at most
constexpr int kSolveBlocks = 160;   // at most (five words per lane)
constexpr int kSolveWordBlocks = 16;  // blocks that exchange without the counter, at most
constexpr long kSolvePolls = 1L << 22;

// all blocks have arrived: a count that only grows within a launch (bar_count, zero before it)
__device__ __forceinline__ bool solve_arrive_wait(CgDevState* st, unsigned target, long polls) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&st->bar_count) : "memory");
  unsigned v = 0;
  for (long q = 0; v < target; ++q) {
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&st->bar_count) : "memory");
    if (q >= polls) {
      atomicExch(&st->bar_timeout, 1);
      return false;
    }
  }
  return true;
}

struct alignas(16) SolveWord {
  double v;
  unsigned long long epoch;
};

__device__ __forceinline__ void word_put(SolveWord* p, double v, unsigned long long epoch) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}"
               ::"l"(p), "l"(__double_as_longlong(v)), "l"(epoch)
               : "memory");
}

__device__ __forceinline__ bool word_get(const SolveWord* p, unsigned long long epoch, double* v) {
  unsigned long long lo, hi;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  *v = __longlong_as_double((long long)lo);
  return hi == epoch;
}

// words w[b], b = first + lane + 32 j up to last, until all carry `epoch` (one warp); the sum of
// this lane's, in order of b.  *ok false when the wait ran out.
__device__ __forceinline__ double words_wait(const SolveWord* w, int first, int last,
                                             unsigned long long epoch, bool* ok, CgDevState* st,
                                             long polls) {
  const int lane = threadIdx.x & 31;
  double v[kSolveBlocks / 32];
  for (long q = 0;; ++q) {
    bool have = true;
#pragma unroll
    for (int j = 0; j < kSolveBlocks / 32; ++j) {
      v[j] = 0.0;
      const int b = first + lane + 32 * j;
      if (b <= last && !word_get(w + b, epoch, &v[j])) have = false;
    }
    if (__all_sync(0xffffffffu, have)) break;
    if (q >= polls) {
      *ok = false;
      if (lane == 0) atomicExch(&st->bar_timeout, 1);
      break;
    }
  }
  double t = v[0];
#pragma unroll
  for (int j = 1; j < kSolveBlocks / 32; ++j)
    if (32 * j <= last - first) t += v[j];
  return t;
}

// the block's copy of the solve's scalars
struct SolveScalars {
  double bcoef, a, beta, inv_beta, dpi, dp0, zz;  // dp0: ||B b||
  double ttol, ttol2, atol, atol2, div, div2;
  int iter, its, max_it, status, squares, ok;
};

// grid totals of NV values, in sh[16 q]: value q by warp q.  RELEASE: what the block wrote
// before is visible to the other blocks behind it.  Blocks of eight warps and more add up through
// shared memory, two warps to a value: 12 FP64 instructions in each of those instead of five
// in every warp, of which the SM's FP64 unit takes 19 clocks each (an iteration with 160,000 unknowns
// 17.0 -> 15.6 us, with 412,000 21.4 -> 20.9).
template <int NV, bool RELEASE>
__device__ __forceinline__ bool solve_sum(double (&v)[NV], SolveWord* words, CgDevState* st,
                                          unsigned long long epoch, unsigned target, double* sh,
                                          double* buf, int* ok_sh, long polls) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  int parts = warps;
  if (warps >= 8) {
    parts = 2;
#pragma unroll
    for (int q = 0; q < NV; ++q) buf[q * kSolveThreads + threadIdx.x] = v[q];
    __syncthreads();
    if (warp < 2 * NV) {
      const double* p = buf + (warp >> 1) * kSolveThreads + (warp & 1) * 32 + lane;
      double a = p[0], b = p[64];  // two chains
      for (int i = 128; i < (int)blockDim.x - (warp & 1) * 32; i += 128) {
        a += p[i];
        if (i + 64 < (int)blockDim.x - (warp & 1) * 32) b += p[i + 64];
      }
      a = warp_sum(a + b);
      if (lane == 0) sh[(warp >> 1) * 16 + (warp & 1)] = a;
    }
  } else {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      v[q] = warp_sum(v[q]);
      if (lane == 0) sh[q * 16 + warp] = v[q];
    }
  }
  __syncthreads();
  const bool counter = gridDim.x > kSolveWordBlocks;
  double t = 0.0;
  if (warp < NV) {
    // the block's parts, at most 8
    t = lane < parts ? sh[warp * 16 + lane] : 0.0;
    for (int o = 4; o > 0; o >>= 1)
      if (o < parts) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (gridDim.x > 1 && lane == 0) {
      if (RELEASE && !counter) __threadfence();
      word_put(words + warp * kSolveBlocks + blockIdx.x, t, epoch);
    }
  }
  if (counter) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      if (!solve_arrive_wait(st, target, polls)) *ok_sh = 0;
    }
    __syncthreads();
  }
  if (warp < NV) {
    if (gridDim.x > 1) {
      bool ok = true;
      t = warp_sum(words_wait(words + warp * kSolveBlocks, 0, (int)gridDim.x - 1, epoch, &ok, st,
                              polls));
      if (RELEASE) __threadfence();
      if (!ok) *ok_sh = 0;
    }
    if (lane == 0) sh[warp * 16] = t;
  }
  __syncthreads();
  return *ok_sh != 0;
}

// cg_alpha and cg_update_tail on the block's scalars; non-negative doubles order like their bits
__device__ __forceinline__ long long solve_bits(double v) { return __double_as_longlong(v); }

__device__ __forceinline__ void solve_alpha(SolveScalars& s, double dpi) {
  s.its = s.iter + 1;
  const long long b = solve_bits(dpi) & 0x7fffffffffffffffll;
  if (b == 0 || (s.iter > 0 && (solve_bits(dpi) < 0) != (solve_bits(s.dpi) < 0)) ||
      b > 0x7ff0000000000000ll) {
    s.status = b > 0x7ff0000000000000ll ? kDivergedNanOrInf : kDivergedIndefiniteMat;
    return;
  }
  s.dpi = dpi;
  s.a = s.beta / dpi;
}

__device__ __forceinline__ void solve_tail(SolveScalars& s, double rr, double zz) {
  s.zz = zz;
  const long long bz = solve_bits(zz);
  if ((bz & 0x7fffffffffffffffll) >= 0x7ff0000000000000ll) {
    s.status = kDivergedNanOrInf;
    return;
  }
  bool done, small, far;
  if (s.squares) {
    done = bz <= solve_bits(s.ttol2);
    small = bz < solve_bits(s.atol2);
    far = bz >= solve_bits(s.div2);
  } else {  // tolerances whose squares leave the normal range
    const double dp = sqrt(zz);
    done = dp <= s.ttol;
    small = dp < s.atol;
    far = dp >= s.div;
  }
  if (done) {
    s.status = small ? kConvergedAtol : kConvergedRtol;
    return;
  }
  if (s.div > 0.0 && far) {
    s.status = kDivergedDtol;
    return;
  }
  s.beta = rr;
  s.iter += 1;
  if (s.iter >= s.max_it) {
    s.status = kDivergedIts;
    return;
  }
  s.its = s.iter + 1;
  if (solve_bits(rr) == 0) {
    s.status = kConvergedAtol;
    return;
  }
  s.bcoef = rr * s.inv_beta;
  if (solve_bits(s.bcoef) < 0) s.status = kDivergedIndefinitePc;
}

template <int K, bool REDIR>
__global__ void __launch_bounds__(kSolveThreads, 1) k_cg_solve(
    const double* __restrict__ a0, const double* __restrict__ a1, const double* __restrict__ a2,
    const double* __restrict__ s, double* __restrict__ x_out, double* r_io, double* p0, double* p1,
    unsigned n, unsigned s1, unsigned s2, CgDevState* st, SolveWord* words,
    unsigned long long epoch, int absent, long polls) {
  if ((int)blockIdx.x == absent) return;  // (a self-check of the waits)
  __shared__ SolveScalars ss;
  __shared__ double sh[32], buf[2 * kSolveThreads];
  if (threadIdx.x == 0) {
    ss.status = st->status;
    ss.beta = st->beta;
    ss.bcoef = ss.dpi = ss.a = 0.0;
    ss.dp0 = st->rnorm0;
    ss.zz = st->rnorm0 * st->rnorm0;
    ss.ttol = st->ttol;
    ss.ttol2 = ss.ttol * ss.ttol;
    ss.atol = st->atol;
    ss.atol2 = ss.atol * ss.atol;
    ss.div = st->divtol > 0.0 ? st->divtol * st->rnorm0 : 0.0;
    ss.div2 = ss.div * ss.div;
    ss.iter = ss.its = 0;
    ss.max_it = st->max_it;
    ss.squares = ss.ttol > 1e-140 && ss.atol >= 0.0 && ss.div < 1e150;
    ss.ok = 1;
  }
  __syncthreads();
  if (ss.status) return;
  const unsigned nt = blockDim.x;
  const unsigned c0 = blockIdx.x * (K * nt) + threadIdx.x;
  double x[K], r[K], p[K], w[K];
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const unsigned c = c0 + q * nt;
    x[q] = p[q] = w[q] = 0.0;
    r[q] = c < n ? __ldcg(r_io + c) : 0.0;
  }
  const int reach = (int)((s2 + K * nt - 1) / (K * nt));  // blocks on either side with neighbours
  unsigned target = 0;
  bool ok = true;
  for (;;) {
    const double bc = ss.bcoef;
    const bool first = ss.iter == 0;
    const double* po = (ss.iter & 1) ? p0 : p1;
    double* pn = (ss.iter & 1) ? p1 : p0;
    if (threadIdx.x == nt - 1) ss.inv_beta = 1.0 / ss.beta;  // read behind the norms' exchange
#pragma unroll
    for (int q = 0; q < K; ++q) {
      const unsigned c = c0 + q * nt;
      p[q] = first ? r[q] : fma(bc, p[q], r[q]);
      if (c < n) __stcg(pn + c, p[q]);
    }
    if (!REDIR) {
      ++epoch;
      __syncthreads();
      if (threadIdx.x < 32 && gridDim.x > 1) {
        bool there = true;
        if (threadIdx.x == 0) {
          __threadfence();
          word_put(words + 3 * kSolveBlocks + blockIdx.x, 0.0, epoch);
        }
        const int b = (int)blockIdx.x;
        words_wait(words + 3 * kSolveBlocks, max(0, b - reach), min((int)gridDim.x - 1, b + reach),
                   epoch, &there, st, polls);
        __threadfence();
        if (!there) ss.ok = 0;
      }
      __syncthreads();
      if (!(ok = ss.ok != 0)) break;
    }
    auto dir = [&](unsigned c) {
      if (!REDIR) return __ldcg(pn + c);
      const double rc = __ldcg(r_io + c);
      return first ? rc : fma(bc, __ldcg(po + c), rc);
    };
    double acc[1] = {0.0};
#pragma unroll
    for (int q = 0; q < K; ++q) {
      const unsigned c = c0 + q * nt;
      if (c < n) {
        double v = p[q];
        if (c >= 1) v = fma(a0[c - 1], dir(c - 1), v);
        if (c + 1 < n) v = fma(a0[c], dir(c + 1), v);
        if (c >= s1) v = fma(a1[c - s1], dir(c - s1), v);
        if (c + s1 < n) v = fma(a1[c], dir(c + s1), v);
        if (c >= s2) v = fma(a2[c - s2], dir(c - s2), v);
        if (c + s2 < n) v = fma(a2[c], dir(c + s2), v);
        w[q] = v;
        acc[0] = fma(p[q], v, acc[0]);
      }
    }
    if (!(ok = solve_sum<1, false>(acc, words + 2 * kSolveBlocks, st, ++epoch, target += gridDim.x,
                                   sh, buf, &ss.ok, polls)))
      break;
    if (threadIdx.x == 0) solve_alpha(ss, sh[0]);
    __syncthreads();
    if (ss.status) break;
    const double a = ss.a;
    double v[2] = {0.0, 0.0};
#pragma unroll
    for (int q = 0; q < K; ++q) {
      const unsigned c = c0 + q * nt;
      if (c < n) {
        x[q] = fma(a, p[q], x[q]);
        r[q] = fma(-a, w[q], r[q]);
        if (REDIR) __stcg(r_io + c, r[q]);
        v[0] = fma(r[q], r[q], v[0]);
        const double z = s[c] * r[q];
        v[1] = fma(z, z, v[1]);
      }
    }
    if (!(ok = solve_sum<2, REDIR>(v, words, st, ++epoch, target += gridDim.x, sh, buf, &ss.ok,
                                   polls)))
      break;
    if (threadIdx.x == 0) solve_tail(ss, sh[0], sh[16]);
    __syncthreads();
    if (ss.status) break;
  }
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const unsigned c = c0 + q * nt;
    if (c < n) x_out[c] = x[q];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->its = ss.its;
    st->iter = ss.iter;
    st->dp = sqrt(ss.zz);
    st->status = ok ? ss.status : (int)kGridBarrierTimeout;
  }
}

__global__ void k_unscale(const double* s, const double* xs, double* x, size_t n) {
  grid_begin();
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x)
    x[c] = s[c] * xs[c];
}

// ------------------------------------------------------------------------------------------
// host side

int Stencil64::alloc(int n0_, int n1_, int n2_) {
  release();
  n0 = n0_;
  n1 = n1_;
  n2 = n2_;
  n = (size_t)n0 * n1 * n2;
  FG_CUDA(cudaMalloc(&a0, n * sizeof(double)));
  FG_CUDA(cudaMalloc(&a1, n * sizeof(double)));
  FG_CUDA(cudaMalloc(&a2, n * sizeof(double)));
  FG_CUDA(cudaMalloc(&s, n * sizeof(double)));
  FG_CUDA(cudaMalloc(&b, n * sizeof(double)));
  scaled = false;
  s_in_r = false;
  return FREHG_OK;
}

void Stencil64::release() {
  cudaFree(a0);
  cudaFree(a1);
  cudaFree(a2);
  cudaFree(s);
  cudaFree(b);
  a0 = a1 = a2 = s = b = nullptr;
  n = 0;
}

int Stencil32::alloc(size_t n_) {
  release();
  n = n_;
  FG_CUDA(cudaMalloc(&a0, n * sizeof(float)));
  FG_CUDA(cudaMalloc(&a1, n * sizeof(float)));
  FG_CUDA(cudaMalloc(&a2, n * sizeof(float)));
  return FREHG_OK;
}

void Stencil32::release() {
  cudaFree(a0);
  cudaFree(a1);
  cudaFree(a2);
  a0 = a1 = a2 = nullptr;
  n = 0;
}

KrylovSolver::~KrylovSolver() {
  if (g64) cudaGraphExecDestroy(g64);
  if (g32) cudaGraphExecDestroy(g32);
  if (gsor) cudaGraphExecDestroy(gsor);
  cudaFree(invd);
  cudaFree(zs);
  cudaFree(sor_slots);
  cudaFree(x);
  cudaFree(r);
  cudaFree(p);
  cudaFree(w);
  cudaFree(partials);
  cudaFree(solve_words);
  cudaFree(dst);
  cudaFreeHost(hst);
  cudaFree(xf);
  cudaFree(rf);
  cudaFree(pf);
  cudaFree(wf);
  cudaFree(rres);
  cudaFree(dst32);
  cudaFreeHost(hst32);
  cudaFree(zf);
  cudaFree(lkf);
  cudaFree(dinvf);
  cudaFree(uf);
  cudaFree(pf2);
  op32.release();
}

int KrylovSolver::ensure(size_t n) {
  if (n <= cap && x) return FREHG_OK;
  cudaFree(x);
  cudaFree(r);
  cudaFree(p);
  cudaFree(w);
  x = r = p = w = nullptr;
  for (cudaGraphExec_t* g : {&g64, &gsor}) {
    if (*g) cudaGraphExecDestroy(*g);
    *g = nullptr;
  }
  FG_CUDA(cudaMalloc(&x, n * sizeof(double)));
  FG_CUDA(cudaMalloc(&r, n * sizeof(double)));
  FG_CUDA(cudaMalloc(&p, n * sizeof(double)));
  FG_CUDA(cudaMalloc(&w, n * sizeof(double)));
  if (!partials) FG_CUDA(cudaMalloc(&partials, 4 * kMaxRedBlocks * sizeof(double)));
  if (!dst) {
    FG_CUDA(cudaMalloc(&dst, sizeof(CgDevState)));
    FG_CUDA(cudaMemset(dst, 0, sizeof(CgDevState)));
    FG_TRY(alloc_mapped(reinterpret_cast<void**>(&hst), sizeof(CgDevState)));
    FG_CUDA(cudaMalloc(&solve_words, 4 * kSolveBlocks * sizeof(SolveWord)));
    FG_CUDA(cudaMemset(solve_words, 0, 4 * kSolveBlocks * sizeof(SolveWord)));
    // (the solves run on streams that do not wait for the legacy one)
    FG_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
  }
  cap = n;
  return FREHG_OK;
}

int KrylovSolver::scale(Stencil64& A, cudaStream_t st) {
  if (A.scaled && A.s_in_r) {
    set_error("operator prepared for the float-float mixed-precision solve; reassemble it");
    return FREHG_ERR_STATE;
  }
  if (A.scaled) return FREHG_OK;
  if (A.f32_entries) {
    set_error("operator assembled in FP32 form for the mixed-precision solve (precision 1)");
    return FREHG_ERR_STATE;
  }
  const int nb = reduction_blocks(A.n, 256, 4);
  const double n = (double)A.n;
  FG_LAUNCH(prof, st, "k_diag_rsqrt", 16.0 * n, launch_chained(k_diag_rsqrt, nb, 256, 0, st, A.s,
                                                               A.n));
  FG_CUDA(cudaGetLastError());
  const StencilLaunch L = stencil_launch(A.n0, A.n1, A.n2);
  FG_LAUNCH(prof, st, "k_scale_offdiag", 56.0 * n,
            launch_chained(k_scale_offdiag, L.grid, L.block, 0, st, A.a0, A.a1, A.a2, A.s, A.n0,
                           A.n1, A.n2, L.planes, L.tiles));
  FG_CUDA(cudaGetLastError());
  A.scaled = true;
  return FREHG_OK;
}

// Run a captured chunk graph until the device status leaves "running" or max_it is reached.
int KrylovSolver::run_chunks(cudaGraphExec_t g, cudaStream_t st, int max_it, int chunk,
                            int launches_per_it) {
  const int max_launch = max_it / chunk + 2;
  for (int q = 0; q < max_launch; ++q) {
    FG_CUDA(cudaGraphLaunch(g, st));
    if (prof) prof->launches += (int64_t)launches_per_it * chunk;
    FG_TRY(fetch_small(hst, dst, sizeof(CgDevState), st));
    FG_CUDA(cudaStreamSynchronize(st));
    if (hst->status != 0) return FREHG_OK;
  }
  set_error("Krylov loop: device status still running after %d chunk launches", max_launch);
  return FREHG_ERR_STATE;
}

int KrylovSolver::solve(Stencil64& A, double* x_out, const frehg_solver_config& cfg,
                        cudaStream_t st, CgResult* res) {
  FG_TRY(ensure(A.n));
  if (!strcmp(cfg.pc_type, "sor")) {
    if (cfg.precision != 0) {
      set_error("pc_type 'sor' runs in FP64 (precision 0)");
      return FREHG_ERR_UNSUPPORTED;
    }
    if (keep_scaled) {
      set_error("pc_type 'sor' returns the unscaled solution");
      return FREHG_ERR_STATE;
    }
    return solve_sor(A, x_out, cfg, st, res);
  }
  if (cfg.precision == 1) {
    FG_TRY(prep_mixed(A, st, !strcmp(cfg.pc_type, "line"), cfg));
    return solve_mixed(A, x_out, cfg, st, res);
  }
  FG_TRY(scale(A, st));
  if (strcmp(cfg.pc_type, "jacobi") != 0) {
    set_error("pc_type '%s' needs the mixed-precision solve (precision 1)", cfg.pc_type);
    return FREHG_ERR_UNSUPPORTED;
  }
  return solve64(A, x_out, cfg, st, res);
}

// Self-check of the grid barrier: every block but skip_block waits at one barrier with a
// bound of `polls` polls; with a block that never arrives the others' waits run out and set
// *timeout, and the kernel returns normally.
__global__ void k_barrier_check(unsigned int* count, unsigned int* gen, int* timeout,
                                int skip_block, long polls) {
  if ((int)blockIdx.x == skip_block) return;
  grid_barrier(count, gen, timeout, polls);
}

// Launch shape of k_cg_iter: the stencil tiles over at most the blocks the device holds at
// once (a cooperative launch may not exceed them).  False where the device has no cooperative
// launch or the shape does not fit.
static bool cg_iter_launch(int n0, int n1, int n2, StencilLaunch* L) {
  int dev = 0, coop = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cg_iter, 256, 0) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (!coop || per_sm < 1 || sms < 1) return false;
  const long resident = std::min<long>((long)per_sm * sms, kMaxRedBlocks);
  const long t0 = (n0 + 31) / 32, t1 = (n1 + 7) / 8, tiles = t0 * t1;
  // plane chunks short enough for about 16 work units per block (the blocks' shares then
  // differ by at most a sixteenth), long enough to keep the stencil's march along axis 2
  long planes = (tiles * n2 + 16 * resident - 1) / (16 * resident);
  planes = std::max<long>(1, std::min<long>(planes, n2));
  const long units = tiles * ((n2 + planes - 1) / planes);
  if (units > (long)INT32_MAX - resident) return false;
  // as few blocks as give every block the same number of units (small systems: fewer blocks
  // to wait for at the grid barriers)
  const long per_block = (units + resident - 1) / resident;
  const long blocks = (units + per_block - 1) / per_block;
  L->block = dim3(32, 8, 1);
  L->grid = dim3((unsigned)blocks, 1, 1);
  L->planes = (int)planes;
  L->tiles = (int)tiles;
  return true;
}

static cudaError_t launch_cg_iter(const StencilLaunch& L, cudaStream_t st, const Stencil64& A,
                                  double* x, double* r, double* p, double* w, CgDevState* dst,
                                  double* partials) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = L.grid;
  cfg.blockDim = L.block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_cg_iter, (const double*)A.a0, (const double*)A.a1,
                            (const double*)A.a2, (const double*)A.s, x, r, p, w, A.n0, A.n1,
                            A.n2, L.planes, L.tiles, dst, partials);
}

// Launch shape of k_cg_solve: cells per thread, threads and blocks.  False where the system is too
// large (more than 512 x 8 cells per SM) or cooperative launches are absent.
struct SolveShape {
  int cells, threads, blocks;
  bool redir;
};

static bool solve_shape(size_t n, SolveShape* sh) {
  int dev = 0, coop = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  sms = std::min(sms, kSolveBlocks);
  if (!coop || sms < 1 || n > (size_t)sms * kSolveThreads * kSolveCells) return false;
  // least FP64 work of the fullest SM: 13 instructions per warp and cell, and the reductions'
  // (15 per warp, 36 in all from eight warps on); at least 4 warps (one per scheduler)
  const size_t per_sm = (n + sms - 1) / sms;
  long best = LONG_MAX;
  for (int k = 1; k <= kSolveCells; ++k) {
    const long warps = std::max<long>(4, (long)((per_sm + 32 * k - 1) / (32 * k)));
    if (warps * 32 > kSolveThreads) continue;
    const long cost = warps * 13 * k + (warps < 8 ? 15 * warps : 36);
    if (cost < best) {
      best = cost;
      sh->cells = k;
      sh->threads = (int)warps * 32;
    }
  }
  const size_t per = (size_t)sh->cells * sh->threads;
  sh->blocks = (int)((n + per - 1) / per);
  // the wait for the neighbouring blocks costs about 1,500 clocks, forming their directions
  // 6 x 19 per warp and cell
  sh->redir = sh->blocks > 1 && sh->cells <= 3 && 6 * 19 * sh->cells * (sh->threads / 32) < 1500;
  return true;
}

static cudaError_t launch_cg_solve(const SolveShape& sh, cudaStream_t st, const Stencil64& A,
                                   double* x, double* r, double* p, double* p2, CgDevState* dst,
                                   void* words, unsigned long long epoch, long check_polls) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)sh.blocks);
  cfg.blockDim = dim3((unsigned)sh.threads);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = sh.blocks > 1 ? 1 : 0;
  auto go = [&](auto kernel) {
    return cudaLaunchKernelEx(&cfg, kernel, (const double*)A.a0, (const double*)A.a1,
                              (const double*)A.a2, (const double*)A.s, x, r, p, p2, (unsigned)A.n,
                              (unsigned)A.n0, (unsigned)(A.n0 * A.n1), dst,
                              static_cast<SolveWord*>(words), epoch,
                              check_polls && sh.blocks > 1 ? sh.blocks - 1 : -1,
                              check_polls ? check_polls : kSolvePolls);
  };
  switch (sh.cells) {  // (redir: at most three, solve_shape)
    case 1: return sh.redir ? go(k_cg_solve<1, true>) : go(k_cg_solve<1, false>);
    case 2: return sh.redir ? go(k_cg_solve<2, true>) : go(k_cg_solve<2, false>);
    case 3: return sh.redir ? go(k_cg_solve<3, true>) : go(k_cg_solve<3, false>);
    case 4: return go(k_cg_solve<4, false>);
    case 5: return go(k_cg_solve<5, false>);
    case 6: return go(k_cg_solve<6, false>);
    case 7: return go(k_cg_solve<7, false>);
    default: return go(k_cg_solve<8, false>);
  }
}

static int chunk_for(size_t n) {
  if (n >= (size_t)4 << 20) return 16;
  if (n >= (size_t)1 << 18) return 32;
  return 64;
}

int KrylovSolver::solve64(Stencil64& A, double* x_out, const frehg_solver_config& cfg,
                          cudaStream_t st, CgResult* res) {
  const size_t n = A.n;
  // stopping parameters
  CgDevState init;
  memset(&init, 0, sizeof(init));
  init.rtol = cfg.rtol;
  init.atol = cfg.atol;
  init.divtol = 1.0e4;
  init.max_it = cfg.max_it;
  FG_TRY(set_states(dst, init, nullptr, init, st));
  const int nb = reduction_blocks(n, 256, 4);
  const double dn = (double)n;
  FG_LAUNCH(prof, st, "k_cg_init", 32.0 * dn,
            launch_chained(k_cg_init, nb, 256, 0, st, A.s, A.b, x, r, n, dst, partials));
  FG_CUDA(cudaGetLastError());

  // by default the whole loop in one launch, where the system fits (and no per-kernel times are
  // asked for)
  if (fused64 < 0 && !coop_failed && !(prof && prof->on)) {
    SolveShape sh;
    if (solve_shape(n, &sh)) {
      const cudaError_t e = launch_cg_solve(sh, st, A, x, r, p, w, dst, solve_words,
                                            ++solve_count << 32, check_polls);
      if (e == cudaSuccess) {
        if (prof) prof->launches += 1;
        FG_TRY(fetch_small(hst, dst, sizeof(CgDevState), st));
        FG_CUDA(cudaStreamSynchronize(st));
        return finish64(A, x_out, st, res, nb);
      }
      // the cooperative launch was refused (e.g. under MPS): three kernels from now on
      cudaGetLastError();
      coop_failed = true;
    }
  }
  const int chunk = chunk_for(n);
  const StencilLaunch L = stencil_launch(A.n0, A.n1, A.n2);
  StencilLaunch LF;
  const bool want = !coop_failed && (fused64 > 0 || (fused64 < 0 && n <= kFusedAutoCells));
  const int form = want && cg_iter_launch(A.n0, A.n1, A.n2, &LF) ? 1 : 0;
  if (prof && prof->on) {
    // profiled path: the same kernels launched one by one between CUDA events
    FG_TRY(fetch_small(hst, dst, sizeof(CgDevState), st));
    FG_CUDA(cudaStreamSynchronize(st));
    for (int q = 0; q < cfg.max_it / chunk + 2 && hst->status == 0; ++q) {
      for (int it = 0; it < chunk; ++it) {
        if (form) {
          FG_LAUNCH(prof, st, "k_cg_iter", 120.0 * dn,
                    FG_CUDA(launch_cg_iter(LF, st, A, x, r, p, w, dst, partials)));
          continue;
        }
        FG_LAUNCH(prof, st, "k_cg_p", 24.0 * dn, k_cg_p<<<nb, 256, 0, st>>>(r, p, n, dst));
        FG_LAUNCH(prof, st, "k_cg_spmv", 40.0 * dn,
                  k_cg_spmv<<<L.grid, L.block, 0, st>>>(A.a0, A.a1, A.a2, p, w, A.n0, A.n1, A.n2,
                                                        L.planes, L.tiles, dst, partials));
        FG_LAUNCH(prof, st, "k_cg_update", 56.0 * dn,
                  k_cg_update<<<nb, 256, 0, st>>>(x, r, p, w, A.s, n, dst, partials));
      }
      FG_CUDA(cudaGetLastError());
      FG_TRY(fetch_small(hst, dst, sizeof(CgDevState), st));
      FG_CUDA(cudaStreamSynchronize(st));
      FG_TRY(prof->flush());
    }
    return finish64(A, x_out, st, res, nb);
  }
  const GraphKey key(A, form, st);
  if (!g64 || !(g64_key == key)) {
    if (g64) cudaGraphExecDestroy(g64);
    g64 = nullptr;
    cudaStream_t cap_st;
    FG_CUDA(cudaStreamCreateWithFlags(&cap_st, cudaStreamNonBlocking));
    cudaGraph_t graph;
    FG_CUDA(cudaStreamBeginCapture(cap_st, cudaStreamCaptureModeThreadLocal));
    cudaError_t le = cudaSuccess;
    for (int q = 0; q < chunk; ++q) {
      if (form) {
        const cudaError_t e1 = launch_cg_iter(LF, cap_st, A, x, r, p, w, dst, partials);
        if (le == cudaSuccess) le = e1;
        continue;
      }
      k_cg_p<<<nb, 256, 0, cap_st>>>(r, p, n, dst);
      k_cg_spmv<<<L.grid, L.block, 0, cap_st>>>(A.a0, A.a1, A.a2, p, w, A.n0, A.n1, A.n2,
                                                L.planes, L.tiles, dst, partials);
      k_cg_update<<<nb, 256, 0, cap_st>>>(x, r, p, w, A.s, n, dst, partials);
    }
    cudaError_t e = cudaStreamEndCapture(cap_st, &graph);
    cudaStreamDestroy(cap_st);
    if (le != cudaSuccess) {
      // the cooperative launch was refused (e.g. under MPS): three kernels from now on
      if (e == cudaSuccess) cudaGraphDestroy(graph);
      cudaGetLastError();
      coop_failed = true;
      return solve64(A, x_out, cfg, st, res);
    }
    if (e != cudaSuccess) {
      set_error("graph capture failed: %s", cudaGetErrorString(e));
      return FREHG_ERR_CUDA;
    }
    e = cudaGraphInstantiate(&g64, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
      set_error("graph instantiate failed: %s", cudaGetErrorString(e));
      return FREHG_ERR_CUDA;
    }
    g64_key = key;
  }
  // iteration 0 may already have converged
  FG_TRY(fetch_small(hst, dst, sizeof(CgDevState), st));
  FG_CUDA(cudaStreamSynchronize(st));
  if (hst->status == 0) FG_TRY(run_chunks(g64, st, cfg.max_it, chunk, form ? 1 : 3));
  return finish64(A, x_out, st, res, nb);
}

int KrylovSolver::finish64(Stencil64& A, double* x_out, cudaStream_t st, CgResult* res, int nb) {
  if (!keep_scaled) {
    FG_LAUNCH(prof, st, "k_unscale", 24.0 * (double)A.n,
              launch_chained(k_unscale, nb, 256, 0, st, scale_vector(A), x, x_out, A.n));
    FG_CUDA(cudaGetLastError());
  }
  res->its = hst->its;
  res->reason = hst->status;
  res->rnorm = hst->dp;
  res->inner_its = hst->its;
  res->ir_its = 0;
  if (hst->bar_timeout || hst->status == kGridBarrierTimeout) {
    set_error("Krylov loop: a grid barrier of the one-launch CG iteration timed out after %d "
              "iterations", hst->its);
    return FREHG_ERR_CUDA;
  }
  if (hst->status < 0) {
    set_error("KSP diverged (reason %d) after %d iterations, residual norm %g", hst->status,
              hst->its, hst->dp);
    return hst->status == kDivergedNanOrInf ? FREHG_ERR_NONFINITE : FREHG_ERR_NOT_CONVERGED;
  }
  return FREHG_OK;
}

}  // namespace fg

extern "C" int frehg_check_grid_barrier(int skip_block, long long polls, int* timed_out) {
  using namespace fg;
  clear_error();
  FG_ARG(timed_out && polls > 0 && skip_block >= -1 && skip_block < 2,
         "timed_out required, polls > 0, skip_block in {-1, 0, 1}");
  int dev = 0, coop = 0;
  FG_CUDA(cudaGetDevice(&dev));
  FG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  if (!coop) {
    set_error("the device has no cooperative launch");
    return FREHG_ERR_UNSUPPORTED;
  }
  unsigned int* w = nullptr;  // count, generation, timeout flag
  FG_CUDA(cudaMalloc(&w, 3 * sizeof(unsigned int)));
  cudaError_t e = cudaMemset(w, 0, 3 * sizeof(unsigned int));
  if (e == cudaSuccess) {
    unsigned int* count = w;
    unsigned int* gen = w + 1;
    int* flag = reinterpret_cast<int*>(w + 2);
    long npolls = (long)polls;
    void* args[] = {&count, &gen, &flag, &skip_block, &npolls};
    e = cudaLaunchCooperativeKernel((const void*)k_barrier_check, dim3(2), dim3(32), args, 0,
                                    nullptr);
  }
  int host_flag = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&host_flag, w + 2, sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(w);
  if (e != cudaSuccess) {
    set_error("grid barrier check: %s", cudaGetErrorString(e));
    return FREHG_ERR_CUDA;
  }
  *timed_out = host_flag;
  return FREHG_OK;
}
