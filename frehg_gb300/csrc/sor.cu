// PCSOR on the GPU: CG preconditioned by PETSc's local symmetric SOR sweep (omega = 1, one
// sweep, zero initial guess), the groundwater default of the reference
// (groundwater.solver.pc_type = "sor", src/driver/Orchestrator.cpp:489, applied by
// PCSetType / KSPSolve in src/linear/backends/PetscLinearSolver.cpp:193,204).
//
// M^-1 r = (D+U)^-1 D (D+L)^-1 r in the owned row order of Decomp3D on one rank
// (row = (j*nx + i)*nz + k, DomainDecomposition.cpp:109-119):
//   forward   y_c = (r_c - a_S y_S - a_W y_W - a_Up y_Up) / d_c     (lower neighbours)
//   backward  z_c = (d_c y_c - a_Down z_Down - a_E z_E - a_N z_N) / d_c
// with 1/d formed once as PETSc's MatSOR does (a zero diagonal entry taken as 1), the product
// d y formed as y / (1/d), and the neighbour terms in the reference's column order.
//
// Evaluation, larger systems of three axes.  With v = D y the two sweeps need one fused multiply-add
// per neighbour and cell:
//   v_c = r_c - sum e_m v_m        (m the lower neighbours, e_m = a_m / d_m at the neighbour)
//   z_c = v_c / d_c - sum e_c z_u  (u the upper neighbours, e_c = a_c / d_c at the cell)
// with the same e = a / d for both, formed once per solve (a zero diagonal entry taken as 1, as
// MatSOR does).  This is the same preconditioner as the product / difference / scaling sequence
// of MatSOR to rounding; on GB300 a warp issues one FP64 instruction per 64 clocks however few of
// its lanes are active, so the dependent FP64 instructions per cell are what the sweeps cost
// (three instead of seven, and no division).  A line of cells (a soil column) takes the same form.
// Evaluation, systems of two axes (sections) and of up to kSorSolveCells.  MatSOR's products,
// differences and scalings, each rounded and in its order, and the sums in the order of sor_sum: the
// results are those of the sequential form (a launch per hyperplane) to the bit.  The one long solve of
// a dry section under recharge (23 iterations at 50 x 30, 38 at 100 x 60; its others take one or two)
// ends within its own rounding noise (3 % of the residual) of the tolerance: with another rounding it
// stopped an iteration earlier or later in one of four runs of 50 x 30, and heads of -500 m moved by up
// to 1.5e-6 m.  It costs 5 FP64 instructions a step instead of 2 (47 us an application of 50 x 30, 29
// before; 115 us of 100 x 60, 77 before).  Larger systems of three axes keep the fused form: their
// runs agree with the sequential form to 1e-14 (ponded loam) and 2e-10 (dry sections a few cells
// thick) with equal iteration counts, closer than rtol 1e-10 determines those, and rounding every
// operation takes 1.23 times as long on 90 x 75 x 60.
//
// Schedule.  A cell depends only on its lower (backward: upper) neighbours, so the sequential
// order is a wavefront.  One warp owns a tile of 32 lines (lines run along the longest axis, the
// tile spans the other two): in step t, lane (l1, l2) takes the cell at position t - l1 - l2 of
// its line.  Neighbours inside the tile are the values two lanes computed one step earlier (warp
// shuffles), the line's own previous value is a register, and the values of the neighbouring
// tiles are read from memory, where the value itself is the signal that it is there: before a
// sweep the array holds kSorWait (a NaN that no arithmetic produces), a reader repeats its load
// until that is gone (bounded).  The loads run a group of steps ahead of their use.  No barrier, no
// fence and no flag: a handover costs one trip through the L2.
//   n <= kSorSolveCells: the whole CG solve in one block with its vectors in shared memory.
//   larger: one cooperative launch (all tiles' blocks resident) per preconditioner application
//   and the CG kernels around it, captured as graphs.
// Measured on GB300, one application (both sweeps): 405,000 cells (90 x 75 x 60) 244 us against
// 1.1 ms for a launch per hyperplane; 4,096 cells 45 us; a whole solve of a 100-cell column (four
// applications, three iterations) 30 us, of a 50 x 30 section 150 us in the mean of twenty (3.2
// applications), where one block with a barrier and an L2 round trip per hyperplane took 168 and 228 us
// for each application.  A step costs about 85 clocks per dependent FP64 instruction, a handover to the next
// tile about 10,000 clocks (the tile's skew, a group of steps and the trip through the L2).
#include "internal.h"
#include "reduce.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace fg {

namespace {

// a quiet NaN with a payload: FP64 arithmetic on the device returns the canonical NaN, never this
constexpr unsigned long long kSorWait = 0x7ff85eed5eed5eedull;
constexpr long kSorPolls = 1L << 22;  // polls of one value before a sweep gives up (seconds)
// largest system solved in one block: eight shared arrays of FP64 (64 bytes a cell, 227 KB)
constexpr int kSorSolveCells = 3600;
constexpr int kSorSolveThreads = 256;
// threads of a sweeping block
__host__ __device__ constexpr int sor_sweep_threads(bool rounded) { return rounded ? 128 : 32; }

struct SorGeom {
  // line axis, then the two tile axes: extents and strides
  int n[3];
  long s[3];
  int ax[3];     // which axis of the operator each is
  int t1, t2;    // lines of a tile along the two tile axes (t1 t2 = 32)
  int nb1, nb2;  // tiles along them
  int steps;     // steps of a full tile
  int axes;      // tile axes of more than one cell (one: the first)
  int ord[3];    // this geometry's axes in the column order of the reference's rows (forward)
};

SorGeom sor_geom(const Stencil64& A) {
  const int n[3] = {A.n0, A.n1, A.n2};
  const long st[3] = {1, A.n0, (long)A.n0 * A.n1};
  int la = 0;
  for (int q = 1; q < 3; ++q)
    if (n[q] > n[la]) la = q;
  int x1 = la == 0 ? 1 : 0, x2 = la == 2 ? 1 : 2;
  if (n[x1] == 1) std::swap(x1, x2);  // an axis of one cell last
  SorGeom g;
  const int ord[3] = {la, x1, x2};
  for (int q = 0; q < 3; ++q) {
    g.n[q] = n[ord[q]];
    g.s[q] = st[ord[q]];
    g.ax[q] = ord[q];
  }
  // 8 x 4 lines; along an axis with fewer than that, as many as it has (rounded up to a power of
  // two), and the others along its partner
  g.axes = (g.n[1] > 1) + (g.n[2] > 1);
  for (int q = 0; q < 3; ++q)
    for (int m = 0; m < 3; ++m)
      if (A.ref_order[q] == ord[m]) g.ord[q] = m;
  g.t2 = 4;
  while (g.t2 > 1 && g.t2 / 2 >= g.n[2]) g.t2 /= 2;
  g.t1 = 32 / g.t2;
  while (g.t1 > 8 && g.t2 < g.n[2] && g.t1 / 2 >= g.n[1]) {
    g.t1 /= 2;
    g.t2 *= 2;
  }
  while (g.t1 > 1 && g.t1 / 2 >= g.n[1] && g.t2 < g.n[2]) {
    g.t1 /= 2;
    g.t2 *= 2;
  }
  g.nb1 = (g.n[1] + g.t1 - 1) / g.t1;
  g.nb2 = (g.n[2] + g.t2 - 1) / g.t2;
  g.steps = g.n[0] + g.t1 + g.t2 - 2;
  return g;
}

__device__ __forceinline__ double sor_peek(const double* p) {
  return *reinterpret_cast<const volatile double*>(p);
}

__device__ __forceinline__ bool sor_missing(double v) {
  return __double2hiint(v) == (int)(kSorWait >> 32);
}

// The lane's line of a tile.  Loads of a lane outside its line (before its first and after its
// last step) go to the line's end cells and are not used.
struct SorLane {
  int l1, l2;       // position in the tile
  int x1, x2;       // the tile's extent (less than t1, t2 in the last tiles)
  bool line;        // the lane has a line
  int i1, i2;
  __device__ __forceinline__ SorLane(const SorGeom& g, int b1, int b2) {
    const int lane = threadIdx.x & 31;
    l1 = lane % g.t1;
    l2 = lane / g.t1;
    x1 = min(g.t1, g.n[1] - b1 * g.t1);
    x2 = min(g.t2, g.n[2] - b2 * g.t2);
    line = l1 < x1 && l2 < x2;
    i1 = b1 * g.t1 + (line ? l1 : 0);
    i2 = b2 * g.t2 + (line ? l2 : 0);
  }
};

// The operands of N consecutive steps of one lane: start value, couplings (global form: over d)
// with the neighbours one step back along the line and the two tile axes, 1 / d, and the values
// of neighbouring tiles.
template <int N>
struct SorSet {
  double a[N], c0[N], c1[N], c2[N], w[N], f1[N], f2[N];
};

// One tile of one sweep by one warp.  In step q the lane takes position q - l1 - l2 of its line,
// backward from the far ends in the reverse of the forward steps.  P loads the operands of a
// step, tells where the neighbouring tiles' values are and takes the result.  Operands are loaded
// a group of steps ahead into the other of two register sets; a group starts when the
// neighbouring tiles' values it needs are there, so a wait costs a trip to the L2 per group and
// not per step.  AXES: tile axes of more than one cell (one: the first); the products of the
// others are left out.  Returns false when a wait ran out.
template <bool FWD, int AXES, class P>
__device__ __forceinline__ bool sor_tile(const SorGeom& g, const SorLane& L, const P& ops,
                                         int* abort_word, long polls) {
  constexpr int N = P::kGroup;
  const int lane = threadIdx.x & 31;
  const int steps = g.n[0] + L.x1 + L.x2 - 2;
  const bool edge1 = FWD ? L.l1 == 0 : L.l1 == L.x1 - 1;
  const bool edge2 = FWD ? L.l2 == 0 : L.l2 == L.x2 - 1;
  const bool far1 = AXES > 0 && L.line && edge1 && (FWD ? L.i1 > 0 : L.i1 + 1 < g.n[1]);
  const bool far2 = AXES > 1 && L.line && edge2 && (FWD ? L.i2 > 0 : L.i2 + 1 < g.n[2]);
  const bool any_far = AXES > 0 && __any_sync(0xffffffffu, far1 || far2);
  const int from1 = (FWD ? lane - 1 : lane + 1) & 31, from2 = (FWD ? lane - g.t1 : lane + g.t1) & 31;
  // position of step 0, and per step; a lane without a line has no position in [0, len)
  const int len = g.n[0], start = (FWD ? 0 : steps - 1) - L.l1 - L.l2;
  const unsigned len_on = L.line ? (unsigned)len : 0u;
  auto at = [&](int q) { return FWD ? start + q : start - q; };
  auto clamp = [&](int i0) { return min(max(i0, 0), len - 1); };
  auto fetch = [&](int q0, SorSet<N>& S) {
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int i0 = at(q0 + u), ic = clamp(i0);
      ops.template load<FWD, AXES>(min(q0 + u, steps - 1), steps, ic, S.a[u], S.c0[u], S.c1[u],
                                   S.c2[u], S.w[u]);
      if (any_far) {
        S.f1[u] = far1 && (unsigned)i0 < len_on ? sor_peek(ops.template near1<FWD>(ic)) : 0.0;
        if (AXES > 1)
          S.f2[u] = far2 && (unsigned)i0 < len_on ? sor_peek(ops.template near2<FWD>(ic)) : 0.0;
      } else {
        S.f1[u] = 0.0;
        S.f2[u] = 0.0;
      }
    }
  };
  auto missing = [&](const SorSet<N>& S) {
    bool m = false;
#pragma unroll
    for (int u = 0; u < N; ++u) {
      m = m || sor_missing(S.f1[u]);
      if (AXES > 1) m = m || sor_missing(S.f2[u]);
    }
    return m;
  };
  bool ok = true;
  double v = 0.0;
  // the set's loads are complete and the neighbouring tiles' values there
  auto arrive = [&](int q0, SorSet<N>& S) {
    // a use of every operand: the next set's loads are issued only behind it.  A load's
    // completion is tracked by one of a few counters; with both sets' loads outstanding on the
    // same ones, the first use of this set would wait for the next set's as well, a trip to the L2
    // per group (222 against 238 ns a step).
    int t = 0;
#pragma unroll
    for (int u = 0; P::kGlobal && u < N; ++u) {
      t ^= __double2loint(S.a[u]) ^ __double2loint(S.c0[u]);
      if (P::kRounded) t ^= __double2loint(S.w[u]);
      if (AXES > 0) t ^= __double2loint(S.c1[u]);
      if (AXES > 1) t ^= __double2loint(S.c2[u]);
    }
    if (P::kGlobal && t == 0x5eed5eed) __nanosleep(0);
    if (any_far) {
      for (long k = 0; ok && __any_sync(0xffffffffu, missing(S)); ++k) {
#pragma unroll
        for (int u = 0; u < N; ++u) {
          const int ic = clamp(at(q0 + u));
          if (sor_missing(S.f1[u])) S.f1[u] = sor_peek(ops.template near1<FWD>(ic));
          if (AXES > 1 && sor_missing(S.f2[u])) S.f2[u] = sor_peek(ops.template near2<FWD>(ic));
        }
        // (warp-uniform: every lane sees the same k, and the abort word is voted on)
        if (k > polls ||
            ((k & 1023) == 1023 &&
             __any_sync(0xffffffffu, *reinterpret_cast<volatile int*>(abort_word) != 0)))
          ok = false;
      }
    }
  };
  auto compute = [&](int q0, SorSet<N>& S) {
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int i0 = at(q0 + u);
      double x = !P::kRounded && !FWD ? S.w[u] * S.a[u] : S.a[u];
      // the line's first cell has no coupling back: v is still 0 there
      if (P::kRounded) {
        // every operation rounded, the neighbours in the column order of the reference's rows
        const double y1 = AXES > 0 ? __shfl_sync(0xffffffffu, v, from1) : 0.0;
        const double y2 = AXES > 1 ? __shfl_sync(0xffffffffu, v, from2) : 0.0;
        const double p0 = __dmul_rn(S.c0[u], v);
        const double p1 = AXES > 0 ? __dmul_rn(S.c1[u], edge1 ? S.f1[u] : y1) : 0.0;
        const double p2 = AXES > 1 ? __dmul_rn(S.c2[u], edge2 ? S.f2[u] : y2) : 0.0;
        if (AXES < 2) {
          constexpr bool kLineFirst = P::kLineFirst == FWD;
          x = __dsub_rn(__dsub_rn(x, kLineFirst ? p0 : p1), kLineFirst ? p1 : p0);
        } else {
          const int first = FWD ? g.ord[0] : g.ord[2], last = FWD ? g.ord[2] : g.ord[0];
          x = __dsub_rn(x, first == 0 ? p0 : (first == 1 ? p1 : p2));
          x = __dsub_rn(x, g.ord[1] == 0 ? p0 : (g.ord[1] == 1 ? p1 : p2));
          x = __dsub_rn(x, last == 0 ? p0 : (last == 1 ? p1 : p2));
        }
        x = __dmul_rn(x, S.w[u]);
      } else {
        x = fma(-S.c0[u], v, x);
        if (AXES > 0) {
          const double y = __shfl_sync(0xffffffffu, v, from1);
          x = fma(-S.c1[u], edge1 ? S.f1[u] : y, x);
        }
        if (AXES > 1) {
          const double y = __shfl_sync(0xffffffffu, v, from2);
          x = fma(-S.c2[u], edge2 ? S.f2[u] : y, x);
        }
      }
      const bool on = (unsigned)i0 < len_on;
      v = on ? x : v;
      if (on) ops.template store<FWD>(q0 + u, i0, x);
    }
  };
  SorSet<N> A, B;
  fetch(0, A);
  for (int q0 = 0; q0 < steps && ok; q0 += 2 * N) {
    arrive(q0, A);
    fetch(q0 + N, B);
    compute(q0, A);
    arrive(q0 + N, B);
    fetch(q0 + 2 * N, A);
    compute(q0 + N, B);
  }
  return ok;
}

// the vectors in shared memory in cell order: src r (forward) or d y, out y or z, e the couplings
template <bool LINE_FIRST>
struct SorShared {
  static constexpr bool kGlobal = false, kRounded = true, kLineFirst = LINE_FIRST;
  static constexpr int kGroup = 2;  // 8 % faster than 4 on a 100-cell column
  const double *src, *invd, *e0, *e1, *e2;  // e shifted to the neighbour's (forward)
  double* out;
  int first, s0, o1, o2;
  __device__ __forceinline__ SorShared(bool fwd, const SorGeom& g, const SorLane& L,
                                       const double* src_, const double* invd_, const double* e0_,
                                       const double* e1_, const double* e2_, double* out_)
      : src(src_), invd(invd_), e0(e0_), e1(e1_), e2(e2_), out(out_) {
    s0 = (int)g.s[0];
    o1 = fwd ? -(int)g.s[1] : (int)g.s[1];
    o2 = fwd ? -(int)g.s[2] : (int)g.s[2];
    first = L.i1 * (int)g.s[1] + L.i2 * (int)g.s[2];
    if (fwd && L.i1 > 0) e1 += o1;
    if (fwd && L.i2 > 0) e2 += o2;
  }
  template <bool FWD, int AXES>
  __device__ __forceinline__ void load(int, int, int ic, double& a, double& c0, double& c1,
                                       double& c2, double& w) const {
    const int c = first + s0 * ic;
    a = src[c];
    w = invd[c];
    c0 = e0[FWD ? c - (ic > 0 ? s0 : 0) : c];
    if (AXES > 0) c1 = e1[c];
    if (AXES > 1) c2 = e2[c];
  }
  template <bool FWD>
  __device__ __forceinline__ const double* near1(int ic) const { return out + (first + s0 * ic + o1); }
  template <bool FWD>
  __device__ __forceinline__ const double* near2(int ic) const { return out + (first + s0 * ic + o2); }
  template <bool FWD>
  __device__ __forceinline__ void store(int, int i0, double x) const {
    *reinterpret_cast<volatile double*>(out + (first + s0 * i0)) = x;
  }
};

// Larger systems keep the sweeps' operands in the order the warps take them ("slots"):
// slot = (tile * steps + t) * 32 + lane, so a step's loads are consecutive.
// ROUNDED: the couplings as they are, not over d.
struct SorSlots {
  double2* f01;  // forward: couplings over d with the line's previous cell and along tile axis 1
  double* f2;    // and along tile axis 2 (0 where there is no neighbour)
  double2* e01;  // backward, the same
  double2* e2d;  // backward: along tile axis 2, and 1 / d
  double* v;     // forward values
  double* u;     // ROUNDED: those times d, the backward sweep's right-hand side
};

// The far neighbours' values: forward in the slot array (the last lane of the tile before took
// the same position t1 - 1 or t2 - 1 steps later), backward in z.
template <bool ROUNDED, bool LINE_FIRST>
struct SorGlobal {
  static constexpr bool kGlobal = true, kRounded = ROUNDED, kLineFirst = LINE_FIRST;
  static constexpr int kGroup = 4;  // 2: 20 % slower, the loads' latency shows
  const SorSlots& S;
  const double* r;
  double* z;
  long first, s0, s1, s2;
  size_t slot0;
  const double *p1, *p2;
  __device__ __forceinline__ SorGlobal(const SorSlots& S_, const SorGeom& g, const SorLane& L,
                                       int tile, const double* r_, double* z_)
      : S(S_), r(r_), z(z_) {
    s0 = g.s[0];
    s1 = g.s[1];
    s2 = g.s[2];
    first = (long)L.i1 * s1 + (long)L.i2 * s2;
    slot0 = (size_t)tile * g.steps * 32 + (threadIdx.x & 31);
    p1 = S.v + ((size_t)(tile - 1) * g.steps + (g.t1 - 1) + L.l2) * 32 + (g.t1 - 1) + g.t1 * L.l2;
    p2 = S.v + ((size_t)(tile - g.nb1) * g.steps + (g.t2 - 1) + L.l1) * 32 + L.l1 +
         g.t1 * (g.t2 - 1);
  }
  template <bool FWD, int AXES>
  __device__ __forceinline__ void load(int q, int steps, int ic, double& a, double& c0, double& c1,
                                       double& c2, double& w) const {
    const size_t slot = slot0 + (size_t)(FWD ? q : steps - 1 - q) * 32;
    if (FWD) {
      a = __ldg(r + first + s0 * ic);
      const double2 f = __ldg(S.f01 + slot);
      c0 = f.x;
      c1 = f.y;
      if (AXES > 1) c2 = __ldg(S.f2 + slot);
      if (ROUNDED) w = __ldg(&S.e2d[slot].y);
    } else {
      a = ROUNDED ? S.u[slot] : S.v[slot];
      const double2 e = __ldg(S.e01 + slot), d = __ldg(S.e2d + slot);
      c0 = e.x;
      c1 = e.y;
      c2 = d.x;
      w = d.y;
    }
  }
  template <bool FWD>
  __device__ __forceinline__ const double* near1(int ic) const {
    return FWD ? p1 + 32L * ic : z + (first + s0 * ic + s1);
  }
  template <bool FWD>
  __device__ __forceinline__ const double* near2(int ic) const {
    return FWD ? p2 + 32L * ic : z + (first + s0 * ic + s2);
  }
  template <bool FWD>
  __device__ __forceinline__ void store(int q, int i0, double x) const {
    double* o = FWD ? S.v + slot0 + (size_t)q * 32 : z + first + s0 * i0;
    *reinterpret_cast<volatile double*>(o) = x;
  }
};

// y / (1/d), rounded as a division: the product with d and one correction by its exact remainder
// (Markstein's theorem, IBM J. Res. Dev. 34, 1990).  A division here is a tenth of an application.
__device__ __forceinline__ double sor_undo(double y, double invd, double d) {
  const double dc = d == 0.0 ? 1.0 : d, q = y * dc;
  return fma(fma(-q, invd, y), dc, q);
}

// Both sweeps over all tiles, one warp per block, every block resident (cooperative launch).  A
// block's tiles are in row order forward and in the reverse order backward, so each tile comes
// after the tiles it reads from wherever they run.
// ROUNDED: three more warps wait while the first one sweeps; between the sweeps all four form d y
// of the block's tiles, which in the sweep would lengthen the one warp's instruction stream by half.
template <int AXES, bool ROUNDED, bool LINE_FIRST>
__global__ void __launch_bounds__(sor_sweep_threads(ROUNDED))
    k_sor_sweeps(SorGeom g, SorSlots S, const double* __restrict__ r, const double* __restrict__ d,
                 const double* __restrict__ invd, double* z, CgDevState* st, int absent,
                 long polls) {
  if (st->status || (int)blockIdx.x == absent) return;  // (absent: a self-check of the waits)
  using Ops = SorGlobal<ROUNDED, LINE_FIRST>;
  const int tiles = g.nb1 * g.nb2;
  const bool sweeps = threadIdx.x < 32;
  bool ok = true;
  int last = -1;
  for (int b = blockIdx.x; b < tiles && ok; b += gridDim.x) {
    const SorLane L(g, b % g.nb1, b / g.nb1);
    if (sweeps) ok = sor_tile<true, AXES>(g, L, Ops(S, g, L, b, r, z), &st->bar_timeout, polls);
    last = b;
  }
  if (ROUNDED) {
    __syncthreads();
    for (int b = blockIdx.x; b < tiles; b += gridDim.x) {
      const SorLane L(g, b % g.nb1, b / g.nb1);
      for (int t = threadIdx.x >> 5; t < g.steps; t += sor_sweep_threads(ROUNDED) / 32) {
        const size_t slot = ((size_t)b * g.steps + t) * 32 + (threadIdx.x & 31);
        const int i0 = t - L.l1 - L.l2;
        if (!L.line || i0 < 0 || i0 >= g.n[0]) continue;
        const size_t c = (size_t)i0 * g.s[0] + (size_t)L.i1 * g.s[1] + (size_t)L.i2 * g.s[2];
        S.u[slot] = sor_undo(S.v[slot], invd[c], d[c]);
      }
    }
    __syncthreads();
  }
  __syncwarp();
  for (int b = last; sweeps && b >= 0 && ok; b -= gridDim.x) {
    const SorLane L(g, b % g.nb1, b / g.nb1);
    ok = sor_tile<false, AXES>(g, L, Ops(S, g, L, b, r, z), &st->bar_timeout, polls);
  }
  if (!ok && threadIdx.x == 0) {
    atomicExch(&st->bar_timeout, 1);
    atomicExch(&st->status, (int)kGridBarrierTimeout);
  }
}

__device__ __forceinline__ double sor_wait_value() {
  return __longlong_as_double((long long)kSorWait);
}

// 1/d (a zero diagonal entry replaced by 1, MatSOR / PCJacobi), x = 0, r = b, and z set to "not
// there yet"
__global__ void k_sor_prep(const double* d, const double* b, double* invd, double* x, double* r,
                           double* z, size_t n) {
  grid_begin();
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x) {
    const double dc = d[c];
    invd[c] = 1.0 / (dc == 0.0 ? 1.0 : dc);
    x[c] = 0.0;
    r[c] = b[c];
    z[c] = sor_wait_value();
  }
}

// the sweeps' operands in slot order, and v set to "not there yet"; a0, a1, a2 in the order of the
// geometry's axes
template <bool ROUNDED>
__global__ void k_sor_slots(SorGeom g, SorSlots S, const double* a0, const double* a1,
                            const double* a2, const double* invd, size_t slots) {
  grid_begin();
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < slots;
       e += (size_t)gridDim.x * blockDim.x) {
    const int lane = (int)(e & 31);
    const unsigned row = (unsigned)(e >> 5), tile = row / (unsigned)g.steps;
    const int t = (int)(row - tile * (unsigned)g.steps);
    const int b1 = (int)(tile % (unsigned)g.nb1), b2 = (int)(tile / (unsigned)g.nb1);
    const int l1 = lane % g.t1, l2 = lane / g.t1;
    const int i0 = t - l1 - l2, i1 = b1 * g.t1 + l1, i2 = b2 * g.t2 + l2;
    double2 f = make_double2(0.0, 0.0), h = f, w = f;
    double f2 = 0.0;
    if (i0 >= 0 && i0 < g.n[0] && i1 < g.n[1] && i2 < g.n[2]) {
      const size_t c = (size_t)i0 * g.s[0] + (size_t)i1 * g.s[1] + (size_t)i2 * g.s[2];
      const double id = invd[c];
      auto over_d = [&](const double* a, size_t m) { return ROUNDED ? a[m] : a[m] * invd[m]; };
      if (i0 > 0) f.x = over_d(a0, c - g.s[0]);
      if (i1 > 0) f.y = over_d(a1, c - g.s[1]);
      if (i2 > 0) f2 = over_d(a2, c - g.s[2]);
      if (i0 + 1 < g.n[0]) h.x = over_d(a0, c);
      if (i1 + 1 < g.n[1]) h.y = over_d(a1, c);
      if (i2 + 1 < g.n[2]) w.x = over_d(a2, c);
      w.y = id;
    }
    S.f01[e] = f;
    S.f2[e] = f2;
    S.e01[e] = h;
    S.e2d[e] = w;
    S.v[e] = sor_wait_value();
  }
}

__device__ __forceinline__ int sor_converged(CgDevState* s, double rnorm) {
  if (isnan(rnorm) || isinf(rnorm)) return kDivergedNanOrInf;
  if (rnorm <= s->ttol) return rnorm < s->atol ? kConvergedAtol : kConvergedRtol;
  if (s->divtol > 0.0 && rnorm >= s->divtol * s->rnorm0) return kDivergedDtol;
  return 0;
}

// KSPSolve_CG's scalar steps after a preconditioner application (||z||^2 = zz, z.r = zr): the
// stopping test and the next direction's coefficient; INIT: before the first iteration.
// QUOTIENT false: the caller forms bcoef = beta / betaold itself
template <bool INIT, bool QUOTIENT = true>
__device__ __forceinline__ void sor_scalars(CgDevState* st, double zz, double zr) {
  const double dp = sqrt(zz);
  st->dp = dp;
  if (INIT) {
    st->rnorm0 = dp;
    st->ttol = fmax(st->rtol * dp, st->atol);
    st->its = 0;
    st->iter = 0;
    st->dpi = 0.0;
    st->status = sor_converged(st, dp);
    if (st->status) return;
    st->beta = zr;
    st->its = 1;
    if (st->beta == 0.0) st->status = kConvergedAtol;
    return;
  }
  const int reason = sor_converged(st, dp);
  if (reason) {
    st->status = reason;
    return;
  }
  st->betaold = st->beta;
  st->beta = zr;
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
  if (!QUOTIENT) return;
  st->bcoef = st->beta / st->betaold;
  if (st->bcoef < 0.0) st->status = kDivergedIndefinitePc;
}

// p.w known: the iteration's alpha, or the end of the solve
__device__ __forceinline__ void sor_alpha(CgDevState* st, double dpi) {
  st->its = st->iter + 1;
  if (dpi == 0.0 || (st->iter > 0 && ((dpi > 0.0) != (st->dpi > 0.0))) || isnan(dpi)) {
    st->status = isnan(dpi) ? kDivergedNanOrInf : kDivergedIndefiniteMat;
    return;
  }
  st->dpiold = st->dpi;
  st->dpi = dpi;
  st->a = st->beta / dpi;
}

// ||z|| and beta = z.r after a preconditioner application; the last block runs
// KSPSolve_CG's scalar steps (stopping test, beta ratio) as in the Jacobi path.
template <bool INIT, bool ROUNDED>
__global__ void k_sor_dots(const double* __restrict__ z, const double* __restrict__ r, size_t n,
                           CgDevState* st, double* partials) {
  if (st->status) return;
  double v[2] = {0.0, 0.0};
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x) {
    const double zc = z[c];
    v[0] = fma(zc, zc, v[0]);
    v[1] = fma(zc, r[c], v[1]);
  }
  double tot[2];
  if (!grid_sum<2, ROUNDED>(v, partials, &st->arrive[3], tot)) return;
  if (flat_tid() == 0) sor_scalars<INIT>(st, tot[0], tot[1]);
}

// p = z (first iteration) or z + (beta/betaold) p
__global__ void k_sor_p(const double* __restrict__ z, double* __restrict__ p, size_t n,
                        const CgDevState* st) {
  if (st->status) return;
  const double bc = st->bcoef;
  const bool first = st->iter == 0;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x)
    p[c] = first ? z[c] : fma(bc, p[c], z[c]);
}

// w = A p with the diagonal, p.w, alpha = beta / p.w
template <bool ROUNDED>
__global__ void __launch_bounds__(256) k_sor_spmv(const double* __restrict__ d,
                                                  const double* __restrict__ a0,
                                                  const double* __restrict__ a1,
                                                  const double* __restrict__ a2,
                                                  const double* __restrict__ p,
                                                  double* __restrict__ w, int n0, int n1, int n2,
                                                  CgDevState* st, double* partials) {
  if (st->status) return;
  const size_t s1 = (size_t)n0, s2 = (size_t)n0 * n1, n = s2 * n2;
  double acc[1] = {0.0};
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x) {
    const unsigned line = (unsigned)c / (unsigned)n0;  // fewer than 2^31 cells
    const int i0 = (int)((unsigned)c - line * (unsigned)n0);
    const int i2 = (int)(line / (unsigned)n1), i1 = (int)(line - (unsigned)i2 * (unsigned)n1);
    const double pc = p[c];
    double v = d[c] * pc;
    if (i0 > 0) v = fma(a0[c - 1], p[c - 1], v);
    if (i0 + 1 < n0) v = fma(a0[c], p[c + 1], v);
    if (i1 > 0) v = fma(a1[c - s1], p[c - s1], v);
    if (i1 + 1 < n1) v = fma(a1[c], p[c + s1], v);
    if (i2 > 0) v = fma(a2[c - s2], p[c - s2], v);
    if (i2 + 1 < n2) v = fma(a2[c], p[c + s2], v);
    w[c] = v;
    acc[0] = fma(pc, v, acc[0]);
  }
  double tot[1];
  if (!grid_sum<1, ROUNDED>(acc, partials, &st->arrive[1], tot)) return;
  if (flat_tid() == 0) sor_alpha(st, tot[0]);
}

// x += a p, r -= a w, and the sweeps' arrays set to "not there yet"
__global__ void k_sor_update(double* __restrict__ x, double* __restrict__ r,
                             const double* __restrict__ p, const double* __restrict__ w,
                             double* __restrict__ v, size_t slots, double* __restrict__ z,
                             size_t n, const CgDevState* st) {
  if (st->status) return;
  const double a = st->a;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x) {
    x[c] = fma(a, p[c], x[c]);
    r[c] = fma(-a, w[c], r[c]);
    z[c] = sor_wait_value();
  }
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < slots;
       c += (size_t)gridDim.x * blockDim.x)
    v[c] = sor_wait_value();
}

// The sweeps of a system that is one line of cells (a soil column), by one warp: first-order linear
// recurrences, solved as a scan.  A lane takes a chunk of consecutive cells; per sweep it solves the
// chunk from zero, the chunks' ends are combined over the lanes in five steps, and every cell gets its
// share of what enters its chunk.  The recurrence's factors do not change during a solve, so their
// products (within chunks: `pf`, `pb`; over lanes: registers) are formed once.  2 n / 32 + 5
// dependent FP64 instructions a sweep (64 to 85 clocks each) instead of n: the solve of a column of
// 100 cells takes 30 us, 58 in order.
struct LineScan {
  int lo, hi;  // the lane's cells
  double f[5], b[5];
  double *pf, *pb;
  const double* e;  // coupling c to c + 1 over the diagonal of c
  int n;

  // products of the chunk's factors before step s over lanes, then combined with the neighbour's
  __device__ __forceinline__ static void steps(double (&out)[5], double a, bool up, int lane) {
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      out[q] = a;
      const double t = up ? __shfl_up_sync(0xffffffffu, a, 1 << q)
                          : __shfl_down_sync(0xffffffffu, a, 1 << q);
      if (up ? lane >= (1 << q) : lane + (1 << q) < 32) a *= t;
    }
  }

  __device__ __forceinline__ LineScan(const double* e_, double* pf_, double* pb_, int n_)
      : pf(pf_), pb(pb_), e(e_), n(n_) {
    const int lane = threadIdx.x & 31, m = (n + 31) / 32;
    lo = min(n, lane * m);
    hi = min(n, lo + m);
    double a = 1.0;
    for (int c = lo; c < hi; ++c) pf[c] = a = c ? a * -e[c - 1] : 0.0;
    steps(f, a, true, lane);
    a = 1.0;
    for (int c = hi - 1; c >= lo; --c) pb[c] = a = c + 1 < n ? a * -e[c] : 0.0;
    steps(b, a, false, lane);
  }

  // v_c = r_c - e_{c-1} v_{c-1}
  __device__ __forceinline__ void forward(const double* r, double* v) const {
    const int lane = threadIdx.x & 31;
    double y = 0.0;
    for (int c = lo; c < hi; ++c) {
      y = c > lo ? fma(-e[c - 1], y, r[c]) : r[c];
      v[c] = y;
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const double t = __shfl_up_sync(0xffffffffu, y, 1 << q);
      if (lane >= (1 << q)) y = fma(f[q], t, y);
    }
    const double in = __shfl_up_sync(0xffffffffu, y, 1);
    if (lane)
      for (int c = lo; c < hi; ++c) v[c] = fma(pf[c], in, v[c]);
  }

  // z_c = v_c - e_c z_{c+1}
  __device__ __forceinline__ void backward(const double* v, double* z) const {
    const int lane = threadIdx.x & 31;
    double y = 0.0;
    for (int c = hi - 1; c >= lo; --c) {
      y = c + 1 < hi ? fma(-e[c], y, v[c]) : v[c];
      z[c] = y;
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const double t = __shfl_down_sync(0xffffffffu, y, 1 << q);
      if (lane + (1 << q) < 32) y = fma(b[q], t, y);
    }
    const double in = __shfl_down_sync(0xffffffffu, y, 1);
    if (lane < 31)
      for (int c = lo; c < hi; ++c) z[c] = fma(pb[c], in, z[c]);
  }
};

// Sums of NV values over a block of at most 256 threads, in the order of `nb` such blocks with four
// cells a thread whose warps add by butterflies: acc[q][b] are thread t's cells t + 256 b +
// 256 nb k, k = 0, 1, ...  Within a warp the sums of different (q, b) share the butterfly's steps
// (each step halves the lanes of a sum and the sums of a lane: 9 FP64 instructions for eight sums,
// not 40); the warps' sums are added by one warp per value.  Valid in every thread; sh[NV * 32].
constexpr int kSorParts = (kSorSolveCells + 1023) / 1024;
template <int NV>
__device__ __forceinline__ void sor_sum(double (&acc)[NV * kSorParts], double (&tot)[NV],
                                        double* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = blockDim.x >> 5;
  constexpr int M = NV * kSorParts;  // 4 or 8
  int have = M;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
    if (have > 1) {
      have >>= 1;
#pragma unroll
      for (int i = 0; i < M / 2; ++i)
        if (i < have) {
          const double mine = up ? acc[i + have] : acc[i], theirs = up ? acc[i] : acc[i + have];
          acc[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, o);
        }
    } else {
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
    }
  }
  // the sum a lane holds: the halves taken, from the highest lane bit
  constexpr int kShare = 32 / M;
  const int which = lane / kShare;
  if (lane % kShare == 0) sh[which * 8 + warp] = acc[0];
  if (warp == 0)
    for (int w = warps; w < 8; ++w)
      if (lane % kShare == 0) sh[which * 8 + w] = 0.0;
  __syncthreads();
  if (warp < NV) {
    double t = sh[warp * 32 + lane];
    t += __shfl_xor_sync(0xffffffffu, t, 4);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    t += __shfl_xor_sync(0xffffffffu, t, 16);
    t += __shfl_xor_sync(0xffffffffu, t, 8);
    __syncwarp();
    if (lane == 0) sh[warp * 32] = t;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; ++q) tot[q] = sh[q * 32];
}

// The whole solve of a small system in one block: the same iteration with every vector that the
// sweeps or the neighbours read in shared memory (the couplings, of a line over d; 1/d, r, v, z, p),
// the operator and x in global memory (each thread its own cells).  w = A p lives where v does (v is
// written by the next sweep).  x_out receives the solution of a converged solve.
template <int AXES, bool LINE_FIRST = true>
__global__ void __launch_bounds__(kSorSolveThreads) k_sor_solve(
    SorGeom g, const double* d, const double* a0, const double* a1, const double* a2,
    const double* b, double* x, double* x_out, int n0, int n1, int n2, double rtol, double atol,
    double divtol, int max_it, CgDevState* dst, int absent, long polls) {
  grid_begin();
  extern __shared__ double sor_sh[];
  __shared__ CgDevState st;
  __shared__ double quot;  // beta / the last beta, by warp 1 while thread 0 tests the norm
  double beta = 0.0;       // (thread 32's)
  __shared__ double red[64];
  const int n = n0 * n1 * n2, tid = threadIdx.x, warp = tid >> 5;
  const int nt = blockDim.x, warps = nt >> 5;
  const int parts = (n + 1023) / 1024;  // (one where the block has fewer than 256 threads)
  double *e0 = sor_sh, *e1 = e0 + n, *e2 = e1 + n, *invd = e2 + n, *r = invd + n, *v = r + n,
         *z = v + n, *p = z + n;
  // the couplings in the order of the geometry's axes
  const double *g0 = sor_sh + g.ax[0] * n, *g1 = sor_sh + g.ax[1] * n, *g2 = sor_sh + g.ax[2] * n;
  if (tid == 0) {
    st.rtol = rtol;
    st.atol = atol;
    st.divtol = divtol;
    st.max_it = max_it;
    st.status = 0;
    st.bar_timeout = 0;
    st.bcoef = st.beta = st.betaold = st.dp = st.dpiold = 0.0;
  }
  for (int c = tid; c < n; c += nt) {
    const double dc = d[c];
    const double id = 1.0 / (dc == 0.0 ? 1.0 : dc);
    invd[c] = id;
    e0[c] = AXES ? a0[c] : a0[c] * id;
    e1[c] = AXES ? a1[c] : a1[c] * id;
    e2[c] = AXES ? a2[c] : a2[c] * id;
    r[c] = b[c];
    v[c] = sor_wait_value();
    z[c] = sor_wait_value();
  }
  for (int c = tid; c < n; c += nt) x[c] = 0.0;
  __syncthreads();
  const int tiles = AXES == 0 ? 0 : g.nb1 * g.nb2;
  // one line: its sweeps by warp 0, the products in the arrays of the axes without couplings
  LineScan line(g0, sor_sh + g.ax[1] * n, sor_sh + g.ax[2] * n, AXES == 0 && warp == 0 ? n : 0);
  // z = M r and (z.z, z.r) into the scalar steps; block-uniform
  auto apply = [&](bool init) {
    bool ok = true;
    if (AXES == 0 && warp == 0) line.forward(r, v);
    for (int t = warp; t < tiles && ok; t += warps) {
      if (t == absent) continue;  // (a self-check of the waits)
      const SorLane L(g, t % g.nb1, t / g.nb1);
      const SorShared<LINE_FIRST> ops(true, g, L, r, invd, g0, g1, g2, v);
      ok = sor_tile<true, AXES>(g, L, ops, &st.bar_timeout, polls);
    }
    if (!ok) atomicExch(&st.bar_timeout, 1);
    __syncthreads();
    // d y (a line: v / d) by all threads: in the sweep it would lengthen the chain
    for (int c = tid; c < n; c += nt)
      v[c] = AXES ? sor_undo(v[c], invd[c], d[c]) : v[c] * invd[c];
    __syncthreads();
    if (AXES == 0 && warp == 0) line.backward(v, z);
    for (int t = warp + (tiles - 1 - warp) / warps * warps; warp < tiles && t >= 0 && ok;
         t -= warps) {
      const SorLane L(g, t % g.nb1, t / g.nb1);
      const SorShared<LINE_FIRST> ops(false, g, L, v, invd, g0, g1, g2, z);
      ok = sor_tile<false, AXES>(g, L, ops, &st.bar_timeout, polls);
    }
    if (!ok) atomicExch(&st.bar_timeout, 1);
    __syncthreads();
    double part[2 * kSorParts] = {}, s[2];
#pragma unroll
    for (int q = 0; q < kSorParts; ++q)
      for (int c = tid + q * nt; q < parts && c < n; c += nt * parts) {
        part[q] = fma(z[c], z[c], part[q]);
        part[kSorParts + q] = fma(z[c], r[c], part[kSorParts + q]);
      }
    sor_sum<2>(part, s, red);
    if (tid == 0) {
      if (st.bar_timeout)
        st.status = kGridBarrierTimeout;
      else if (init)
        sor_scalars<true, false>(&st, s[0], s[1]);
      else
        sor_scalars<false, false>(&st, s[0], s[1]);
    }
    if (tid == 32) {
      quot = init ? 0.0 : s[1] / beta;
      beta = s[1];
    }
    __syncthreads();
    if (st.status == 0 && quot < 0.0) {
      __syncthreads();
      if (tid == 0) st.status = kDivergedIndefinitePc;
      __syncthreads();
    }
  };
  apply(true);
  const int s1 = n0, s2 = n0 * n1;
  while (st.status == 0) {
    const double bc = quot;
    const bool first = st.iter == 0;
    for (int c = tid; c < n; c += nt) p[c] = first ? z[c] : fma(bc, p[c], z[c]);
    __syncthreads();
    double acc[kSorParts] = {}, pw[1];
    double* w = v;
#pragma unroll
    for (int k = 0; k < kSorParts; ++k)
      for (int c = tid + k * nt; k < parts && c < n; c += nt * parts) {
        const int i0 = c % n0, q = c / n0, i1 = q % n1, i2 = q / n1;
        const double pc = p[c];
        double y = d[c] * pc;
        if (i0 > 0) y = fma(a0[c - 1], p[c - 1], y);
        if (i0 + 1 < n0) y = fma(a0[c], p[c + 1], y);
        if (i1 > 0) y = fma(a1[c - s1], p[c - s1], y);
        if (i1 + 1 < n1) y = fma(a1[c], p[c + s1], y);
        if (i2 > 0) y = fma(a2[c - s2], p[c - s2], y);
        if (i2 + 1 < n2) y = fma(a2[c], p[c + s2], y);
        w[c] = y;
        acc[k] = fma(pc, y, acc[k]);
      }
    sor_sum<1>(acc, pw, red);
    if (tid == 0) sor_alpha(&st, pw[0]);
    __syncthreads();
    if (st.status) break;
    const double a = st.a;
    for (int c = tid; c < n; c += nt) {
      x[c] = fma(a, p[c], x[c]);
      r[c] = fma(-a, w[c], r[c]);
      v[c] = sor_wait_value();
      z[c] = sor_wait_value();
    }
    __syncthreads();
    apply(false);
  }
  if (st.status > 0 && x_out != x)
    for (int c = tid; c < n; c += nt) x_out[c] = x[c];
  if (tid == 0) {
    dst->its = st.its;
    dst->iter = st.iter;
    dst->status = st.status;
    dst->dp = st.dp;
    dst->bar_timeout = st.bar_timeout;
  }
}

// blocks of a cooperative k_sor_sweeps launch: one per tile, at most what the device holds at once
// (0: no cooperative launch)
int sor_sweep_blocks(const SorGeom& g, const void* kernel, int threads) {
  int dev = 0, coop = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (!coop) return 0;
  return (int)std::min<long>((long)g.nb1 * g.nb2, (long)per_sm * sms);
}

}  // namespace

int KrylovSolver::ensure_sor(size_t n, size_t slot_doubles) {
  if (gsor && (n > cap_sor || slot_doubles > cap_slots)) {
    cudaGraphExecDestroy(gsor);
    gsor = nullptr;
  }
  if (n > cap_sor || !invd) {
    cudaFree(invd);
    cudaFree(zs);
    invd = zs = nullptr;
    cap_sor = 0;
    FG_CUDA(cudaMalloc(&invd, n * sizeof(double)));
    FG_CUDA(cudaMalloc(&zs, n * sizeof(double)));
    cap_sor = n;
  }
  if (slot_doubles > cap_slots || !sor_slots) {
    cudaFree(sor_slots);
    sor_slots = nullptr;
    cap_slots = 0;
    FG_CUDA(cudaMalloc(&sor_slots, slot_doubles * sizeof(double)));
    cap_slots = slot_doubles;
  }
  return FREHG_OK;
}

int KrylovSolver::solve_sor(Stencil64& A, double* x_out, const frehg_solver_config& cfg,
                            cudaStream_t st, CgResult* res) {
  if (A.scaled || A.f32_entries) {
    set_error("pc_type 'sor' needs the unscaled FP64 operator; reassemble the system");
    return FREHG_ERR_STATE;
  }
  const size_t n = A.n;
  const SorGeom g = sor_geom(A);
  const double dn = (double)n;
  // two axes: the order of their terms known to the compiler (161 -> 150 us on a 50 x 30 section: a
  // selection per term is as long as half an FP64 instruction in the chain)
  const bool line_first = g.ord[0] == 0 || (g.ord[1] == 0 && g.ord[0] == 2);
  const long polls = check_polls ? check_polls : kSorPolls;
  auto finish = [&]() -> int {
    res->its = hst->its;
    res->reason = hst->status;
    res->rnorm = hst->dp;
    res->inner_its = hst->its;
    res->ir_its = 0;
    if (hst->bar_timeout || hst->status == kGridBarrierTimeout) {
      set_error("SOR sweep: a bounded wait for a neighbouring tile ran out after %d iterations",
                hst->its);
      return FREHG_ERR_CUDA;
    }
    if (hst->status < 0) {
      set_error("KSP diverged (reason %d) after %d iterations, residual norm %g", hst->status,
                hst->its, hst->dp);
      return hst->status == kDivergedNanOrInf ? FREHG_ERR_NONFINITE : FREHG_ERR_NOT_CONVERGED;
    }
    return FREHG_OK;
  };
  if (n <= (size_t)kSorSolveCells) {
    const int smem = 8 * (int)n * (int)sizeof(double);
    // no more warps than cells need: each takes part in every sum on the FP64 unit
    const int threads = std::min(kSorSolveThreads, std::max(64, ((int)n + 31) / 32 * 32));
    // on every solve: the attribute belongs to the current device, and the call is cheap
    auto kernel = g.axes == 2   ? k_sor_solve<2>
                  : g.axes == 1 ? (line_first ? k_sor_solve<1, true> : k_sor_solve<1, false>)
                                : k_sor_solve<0>;
    const int absent = check_polls && g.axes > 0 && g.nb1 * g.nb2 > 1 ? 0 : -1;
    FG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 8 * kSorSolveCells * (int)sizeof(double)));
    FG_LAUNCH(prof, st, "k_sor_solve", 48.0 * dn,
              launch_chained(kernel, 1, threads, smem, st, g, A.s, A.a0, A.a1, A.a2, A.b, x,
                             x_out ? x_out : x, A.n0, A.n1, A.n2, cfg.rtol, cfg.atol, 1.0e4,
                             cfg.max_it, dst, absent, polls));
    FG_CUDA(cudaGetLastError());
    FG_TRY(fetch_small(hst, dst, sizeof(CgDevState), st));
    FG_CUDA(cudaStreamSynchronize(st));
    if (prof && prof->on) FG_TRY(prof->flush());
    return finish();
  }
  const size_t slots = (size_t)g.nb1 * g.nb2 * g.steps * 32;
  const bool rounded = g.axes == 1;
  FG_TRY(ensure_sor(n, slots * (rounded ? 9 : 8)));
  SorSlots S;
  S.f01 = reinterpret_cast<double2*>(sor_slots);
  S.e01 = S.f01 + slots;
  S.e2d = S.e01 + slots;
  S.f2 = reinterpret_cast<double*>(S.e2d + slots);
  S.v = S.f2 + slots;
  S.u = rounded ? S.v + slots : nullptr;
  // one block (all tiles in order, nothing to wait for) where the device refuses cooperative
  // launches
  auto kernel = g.axes == 2   ? k_sor_sweeps<2, false, true>
                : g.axes == 1 ? (line_first ? k_sor_sweeps<1, true, true>
                                            : k_sor_sweeps<1, true, false>)
                              : k_sor_sweeps<0, false, true>;
  const int sweep_threads = sor_sweep_threads(rounded);
  const int sweep_blocks =
      coop_failed ? 1 : std::max(1, sor_sweep_blocks(g, (const void*)kernel, sweep_threads));
  const int absent = check_polls && sweep_blocks > 1 ? 0 : -1;
  CgDevState init;
  memset(&init, 0, sizeof(init));
  init.rtol = cfg.rtol;
  init.atol = cfg.atol;
  init.divtol = 1.0e4;
  init.max_it = cfg.max_it;
  FG_TRY(set_states(dst, init, nullptr, init, st));
  const int nb = reduction_blocks(n, 256, 4);
  double* xs = x;  // the graph keeps fixed pointers; x_out receives a copy
  auto dots_first = rounded ? k_sor_dots<true, true> : k_sor_dots<true, false>;
  auto dots = rounded ? k_sor_dots<false, true> : k_sor_dots<false, false>;
  auto spmv = rounded ? k_sor_spmv<true> : k_sor_spmv<false>;
  auto sweeps = [&](cudaStream_t s) -> cudaError_t {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)sweep_blocks);
    lc.blockDim = dim3((unsigned)sweep_threads);
    lc.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    lc.attrs = at;
    lc.numAttrs = sweep_blocks > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&lc, kernel, g, S, (const double*)r, (const double*)A.s,
                              (const double*)invd, zs, dst, absent, polls);
  };
  FG_LAUNCH(prof, st, "k_sor_prep", 48.0 * dn,
            launch_chained(k_sor_prep, nb, 256, 0, st, A.s, A.b, invd, xs, r, zs, n));
  const double* ax[3] = {A.a0, A.a1, A.a2};
  FG_LAUNCH(prof, st, "k_sor_slots", 32.0 * dn + 64.0 * (double)slots,
            launch_chained(rounded ? k_sor_slots<true> : k_sor_slots<false>,
                           reduction_blocks(slots, 256, 1), 256, 0, st, g, S, ax[g.ax[0]], ax[g.ax[1]],
                           ax[g.ax[2]], invd, slots));
  cudaError_t le = cudaSuccess;
  const double sweep_bytes = 16.0 * dn + (rounded ? 96.0 : 72.0) * (double)slots;
  FG_LAUNCH(prof, st, "k_sor_sweeps", sweep_bytes, le = sweeps(st));
  if (le != cudaSuccess && sweep_blocks > 1) {
    cudaGetLastError();
    coop_failed = true;
    return solve_sor(A, x_out, cfg, st, res);
  }
  FG_CUDA(le);
  FG_LAUNCH(prof, st, "k_sor_dots", 16.0 * dn,
            dots_first<<<nb, 256, 0, st>>>(zs, r, n, dst, partials));
  FG_CUDA(cudaGetLastError());

  // one iteration: p, w = A p (alpha), x/r update, z = M r, norms and beta
  auto iteration = [&](cudaStream_t s, Profiler* pr) -> int {
    FG_LAUNCH(pr, s, "k_sor_p", 24.0 * dn, k_sor_p<<<nb, 256, 0, s>>>(zs, p, n, dst));
    FG_LAUNCH(pr, s, "k_sor_spmv", 48.0 * dn,
              spmv<<<nb, 256, 0, s>>>(A.s, A.a0, A.a1, A.a2, p, w, A.n0, A.n1, A.n2, dst,
                                            partials));
    FG_LAUNCH(pr, s, "k_sor_update", 56.0 * dn + 8.0 * (double)slots,
              k_sor_update<<<nb, 256, 0, s>>>(xs, r, p, w, S.v, slots, zs, n, dst));
    FG_LAUNCH(pr, s, "k_sor_sweeps", sweep_bytes, FG_CUDA(sweeps(s)));
    FG_LAUNCH(pr, s, "k_sor_dots", 16.0 * dn,
              dots<<<nb, 256, 0, s>>>(zs, r, n, dst, partials));
    return FREHG_OK;
  };
  // iterations between two reads of the status: few, as a solve takes from 1 to a few tens of
  // iterations and an idle one costs five launches (about 6 us)
  const int per_it = 5, chunk = 4;

  FG_TRY(fetch_small(hst, dst, sizeof(CgDevState), st));
  FG_CUDA(cudaStreamSynchronize(st));
  if (prof && prof->on) {
    FG_TRY(prof->flush());
    for (int q = 0; q < cfg.max_it + 1 && hst->status == 0; ++q) {
      FG_TRY(iteration(st, prof));
      FG_CUDA(cudaGetLastError());
      FG_TRY(fetch_small(hst, dst, sizeof(CgDevState), st));
      FG_CUDA(cudaStreamSynchronize(st));
      FG_TRY(prof->flush());
    }
  } else if (hst->status == 0) {
    const GraphKey key(A, sweep_blocks, st);
    if (!gsor || !(gsor_key == key)) {
      if (gsor) cudaGraphExecDestroy(gsor);
      gsor = nullptr;
      cudaStream_t cap_st;
      FG_CUDA(cudaStreamCreateWithFlags(&cap_st, cudaStreamNonBlocking));
      cudaGraph_t graph;
      FG_CUDA(cudaStreamBeginCapture(cap_st, cudaStreamCaptureModeThreadLocal));
      int rc = FREHG_OK;
      for (int q = 0; q < chunk && rc == FREHG_OK; ++q) rc = iteration(cap_st, nullptr);
      cudaError_t e = cudaStreamEndCapture(cap_st, &graph);
      cudaStreamDestroy(cap_st);
      if (rc != FREHG_OK || e != cudaSuccess) {
        if (rc == FREHG_OK) set_error("SOR graph capture failed: %s", cudaGetErrorString(e));
        else if (e == cudaSuccess) cudaGraphDestroy(graph);
        cudaGetLastError();
        return FREHG_ERR_CUDA;
      }
      e = cudaGraphInstantiate(&gsor, graph, 0);
      cudaGraphDestroy(graph);
      if (e != cudaSuccess) {
        set_error("SOR graph instantiate failed: %s", cudaGetErrorString(e));
        return FREHG_ERR_CUDA;
      }
      gsor_key = key;
    }
    const int max_launch = cfg.max_it / chunk + 2;
    int q = 0;
    for (; q < max_launch; ++q) {
      FG_CUDA(cudaGraphLaunch(gsor, st));
      if (prof) prof->launches += (int64_t)per_it * chunk;
      FG_TRY(fetch_small(hst, dst, sizeof(CgDevState), st));
      FG_CUDA(cudaStreamSynchronize(st));
      if (hst->status != 0) break;
    }
    if (q == max_launch) {
      set_error("SOR Krylov loop: device status still running after %d chunk launches",
                max_launch);
      return FREHG_ERR_STATE;
    }
  }
  FG_TRY(finish());
  if (x_out && x_out != x)
    FG_CUDA(cudaMemcpyAsync(x_out, x, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
  return FREHG_OK;
}

}  // namespace fg
