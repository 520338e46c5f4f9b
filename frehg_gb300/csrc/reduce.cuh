// Deterministic block / grid reductions shared by the kernels (last-arriving-block pattern:
// no grid barrier, no spin-wait), and the bounded grid barrier of cooperative launches.
#pragma once

#include "ff32.cuh"
#include "internal.h"

namespace fg {

// per-thread compensated FP32 sum (Kahan); the FP32 Krylov kernels combine these in FP64
struct Kahan32 {
  float s = 0.0f, c = 0.0f;
  __device__ __forceinline__ void add(float x) {
    const float y = x - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  // the sum as a double by integer operations (each FP64 instruction of a block's threads costs
  // the SM's FP64 unit 19 clocks per warp)
  __device__ __forceinline__ double value() const { return ff_to_double_nb(fast_two_sum(s, -c)); }
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ int flat_tid() { return threadIdx.x + threadIdx.y * blockDim.x; }
__device__ __forceinline__ int flat_nthreads() { return blockDim.x * blockDim.y; }
__device__ __forceinline__ int flat_bid() { return blockIdx.x + blockIdx.y * gridDim.x; }
__device__ __forceinline__ int flat_nblocks() { return gridDim.x * gridDim.y; }

// The first statement of a kernel that launch_chained() starts: the next launch may be placed, and
// everything the stream did before is complete and visible.
__device__ __forceinline__ void grid_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Sum NV values over the block; the result is valid in every thread.  Uses sh[NV * CAP]; a
// __syncthreads has to come between this and the next use of sh.
// The threads' values (folded by shuffles to CAP at most) go through shared memory to one warp
// per value: 13 FP64 instructions per value and block of 256 threads, where shuffles in every
// warp take 45 (the SM's one FP64 unit serves a warp instruction in 19 clocks, so the reductions at
// the ends of the blocks cost more than many of the kernels' own work on small grids: the FP64
// residual of 40 x 40 x 100 took 26.8 us with shuffles in every warp, 18.1 so).
template <int NV, int CAP = 256>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* sh) {
  const int tid = flat_tid(), lane = tid & 31, wid = tid >> 5;
  const int nw = flat_nthreads() >> 5;
  int width = 32;
  for (; nw * width > CAP; width >>= 1) {
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], width >> 1);
  }
  if (lane < width) {
#pragma unroll
    for (int q = 0; q < NV; ++q) sh[q * CAP + wid * width + lane] = v[q];
  }
  __syncthreads();
  const int count = nw * width;
  for (int q = wid; q < NV; q += nw) {
    double t = lane < count ? sh[q * CAP + lane] : 0.0;
    for (int i = lane + 32; i < count; i += 32) t += sh[q * CAP + i];
    t = warp_sum(t);
    if (lane == 0) sh[q * CAP] = t;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; ++q) v[q] = sh[q * CAP];
}

// The same by butterflies in every warp and one over the warps' sums; valid in thread 0.
template <int NV, int CAP = 256>
__device__ __forceinline__ void block_sum_butterfly(double (&v)[NV], double* sh) {
  const int tid = flat_tid(), lane = tid & 31, wid = tid >> 5, nw = flat_nthreads() >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    v[q] = warp_sum(v[q]);
    if (lane == 0) sh[q * CAP + wid] = v[q];
  }
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = warp_sum(lane < nw ? sh[q * CAP + lane] : 0.0);
  }
}

// Grid-wide sum through per-block partials; returns true in every thread of the last block
// to arrive, where tot[] (valid in thread 0) holds the deterministic grid total.
// BUTTERFLY: the blocks' sums in the order of butterflies.
template <int NV, bool BUTTERFLY = false>
__device__ __forceinline__ bool grid_sum(double (&v)[NV], double* partials, unsigned int* arrive,
                         double (&tot)[NV]) {
  __shared__ double sh[NV * 256];
  __shared__ unsigned int ticket;
  const int tid = flat_tid(), bid = flat_bid(), nb = flat_nblocks();
  if (BUTTERFLY)
    block_sum_butterfly<NV>(v, sh);
  else
    block_sum<NV>(v, sh);
  if (tid == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) partials[q * kMaxRedBlocks + bid] = v[q];
    __threadfence();
    ticket = atomicAdd(arrive, 1u);
  }
  __syncthreads();
  if (ticket != (unsigned)(nb - 1)) return false;
  __threadfence();
  double acc[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    acc[q] = 0.0;
    for (int b = tid; b < nb; b += flat_nthreads()) acc[q] += __ldcg(&partials[q * kMaxRedBlocks + b]);
  }
  if (BUTTERFLY)
    block_sum_butterfly<NV>(acc, sh);
  else
    block_sum<NV>(acc, sh);
#pragma unroll
  for (int q = 0; q < NV; ++q) tot[q] = acc[q];
  if (tid == 0) *arrive = 0u;
  return true;
}

// Grid barrier for cooperative launches (every block resident at once): an arrival counter
// and a generation word in device memory, both 0 before the first use; the last block to
// arrive resets the counter and advances the generation, so consecutive barriers and launches
// reuse them.  The wait is bounded (kGridBarrierPolls polls, about two seconds); a block whose
// wait runs out sets *timeout and gets false, and the caller stops (its launch then reports
// the timeout instead of a result).
constexpr long kGridBarrierPolls = 1L << 24;
__device__ __forceinline__ bool grid_barrier(unsigned int* count, unsigned int* gen,
                                             int* timeout, long max_polls = kGridBarrierPolls) {
  __shared__ int ok;
  __syncthreads();
  if (flat_tid() == 0) {
    volatile unsigned int* vgen = gen;
    const unsigned int g = *vgen;
    __threadfence();
    int good = 1;
    if (atomicAdd(count, 1u) + 1u == (unsigned int)flat_nblocks()) {
      atomicExch(count, 0u);
      __threadfence();
      atomicAdd(gen, 1u);
    } else {
      for (long q = 0; *vgen == g; ++q) {
        if (q >= max_polls) {
          good = 0;
          atomicExch(timeout, 1);
          break;
        }
        if (q >= 256) __nanosleep(100);  // poll at once first: most waits are short
      }
      __threadfence();
    }
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// Grid-wide max through per-block partials (NaN-ignoring, as std::max/std::min with a NaN
// second argument keep the first).  Same last-block contract as grid_sum.
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ bool grid_max(double v, double* partials, unsigned int* arrive, double* tot) {
  __shared__ double sh[32];
  __shared__ unsigned int ticket;
  const int tid = flat_tid(), lane = tid & 31, wid = tid >> 5, nw = flat_nthreads() >> 5;
  const int bid = flat_bid(), nb = flat_nblocks();
  v = warp_max(v);
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (wid == 0) {
    double t = lane < nw ? sh[lane] : -INFINITY;
    t = warp_max(t);
    if (lane == 0) {
      partials[bid] = t;
      __threadfence();
      ticket = atomicAdd(arrive, 1u);
    }
  }
  __syncthreads();
  if (ticket != (unsigned)(nb - 1)) return false;
  __threadfence();
  double acc = -INFINITY;
  for (int b = tid; b < nb; b += flat_nthreads()) acc = fmax(acc, __ldcg(&partials[b]));
  acc = warp_max(acc);
  __syncthreads();
  if (lane == 0) sh[wid] = acc;
  __syncthreads();
  if (tid == 0) {
    double t = -INFINITY;
    for (int q = 0; q < nw; ++q) t = fmax(t, sh[q]);
    *tot = t;
    *arrive = 0u;
  }
  return true;
}

}  // namespace fg
