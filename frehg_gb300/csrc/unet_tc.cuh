// The U-Net's 3x3x3 convolutions on the fifth-generation tensor cores (tcgen05, accumulators in
// tensor memory).  Not in reference.
//
// Implicit GEMM per tile of 8 x 16 pixels (x, y) of one z plane: D[128 x COUT] (FP32, in TMEM;
// row r = 8 py + px) = sum over the 27 taps and the input channels of A[128 x 16] . B[16 x COUT],
// tcgen05.mma.cta_group::1.kind::f16 (BF16 operands, FP32 accumulation, M = 128, K = 16).
// An MMA of M = 128 takes 32 + N / 4 clocks up to N = 96 (shared-memory reads: 4 KB of A, 32 N bytes
// of B) and N / 2 above (measured, whatever the alignment of A), so the three dz taps are stacked
// along N: the weights sit as [t9][chunk][rb COUT + o][8] with row block rb = 2 - dz, and one group
// of MMAs per INPUT plane z' (9 taps x CIN/16 slices, N = 3 COUT) adds W(dz=2) In(z') to out(z'-1),
// W(1) In(z') to out(z') and W(0) In(z') to out(z'+1): a third of the MMAs of one group per output
// plane over three input planes, and each input plane is read once per tile.
// Operands sit in shared memory in the no-swizzle K-major core-matrix layout, which the
// channels-last activations reach by splitting the channels into 8-channel chunks:
//   ring slots  [chunk of 2][hy][hx][8]: 16 channels of the 10 x 18 pixels x0-1 .. x0+8,
//               y0-1 .. y0+16 of a plane, zero outside the grid; a tap (dx, dy) is the view starting
//               at pixel (dx, dy), its M-adjacent core matrices one patch row (160 bytes) apart, its
//               K-adjacent ones one chunk (2880 bytes);
//   weights     N-adjacent core matrices 128 bytes apart, K-adjacent ones 3 COUT x 16 bytes; all 27
//               taps stay resident.
// The accumulators of consecutive output planes lie side by side in all 512 tensor-memory columns,
// used as a ring (two MMAs instead of one where the three planes' columns wrap round); the epilogue
// leaves each zeroed, so every MMA accumulates.
// One block per SM; its warps work in parallel through mbarriers: eight copy planes into a ring of
// patches (16-byte cp.async), one issues MMAs, one runs ahead with that warp's waits, eight read
// finished accumulators (tcgen05.ld 32x32b), free them, add the bias, apply the ReLU and store BF16.
// A block walks z columns of zc output planes (which cost zc + 2 input planes; conv_column chooses
// zc so that the last blocks do not work alone).  The order of the sums is (dz, t9, channel slice)
// for every output, whatever the columns.
// Bound by shared memory: the MMAs' reads (44 clocks of the 61 that an MMA of 48 -> 16 takes) and
// the copies, which pass through L1.  (Copies past L1 are slower but for 96 channels, 16 copy warps
// no faster.)  The decoder convolutions read the upsampled half of their input from the coarse
// field, as the stored concatenation took 170 us more in all at 256 x 256 x 128.  There, against one
// MMA group per output plane and per-plane barriers of one warpgroup: 16 -> 16 305 -> 153 us,
// 48 -> 16 617 -> 372; 128 x 128 x 64: 96 -> 32 628 -> 200, 32 -> 32 96 -> 61; 64 x 64 x 32:
// 64 -> 64 112 -> 33.
//
// Every wait is bounded: a wait that runs out records an error word, the block's other waits see
// the abort word and return, and the MMAs in flight finish (bounded) before the tensor memory is
// freed.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>
#include <type_traits>

namespace fg {
namespace unet {

constexpr int kTcM = 128;                       // pixels per tile (the MMA's M)
constexpr int kTcTX = 8, kTcTY = 16;             // the tile: 8 x 16 pixels, row r = 8 py + px
constexpr int kTcHX = kTcTX + 2, kTcHY = kTcTY + 2;  // with the halo
constexpr int kTcHP = kTcHX * kTcHY;             // 180 staged pixels per plane
constexpr long kTcSpin = 1L << 22;
constexpr uint32_t kTcStop = 0xffffffffu;

// tiles of an nx x ny plane
__host__ __device__ inline int tc_tiles_x(int nx) { return (nx + kTcTX - 1) / kTcTX; }
__host__ __device__ inline int tc_tiles_y(int ny) { return (ny + kTcTY - 1) / kTcTY; }

__device__ __forceinline__ uint32_t tc_smem(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor: start, leading (K) and stride (M / N) byte offsets, no swizzle
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of the fifth-generation tensor cores
  return d;                // base offset 0, absolute leading offset, layout: no swizzle
}

// instruction descriptor of kind::f16: D FP32, A and B BF16, both K-major, M = 128, N = n
__host__ __device__ constexpr uint32_t tc_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(kTcM >> 4) << 24);
}

// 16-byte copy global -> shared with zero fill past `bytes`, through L1: a thread's chunks of one
// pixel share 32-byte sectors, which L1 then serves once
__device__ __forceinline__ void tc_cp16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(tc_smem(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void tc_bar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_smem(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void tc_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem(bar)) : "memory");
}

// this thread's copies so far arrive on the barrier when they have landed
__device__ __forceinline__ void tc_arrive_copies(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc_smem(bar)) : "memory");
}

// whether the phase is complete (TRY: after waiting for it for a time that the hardware limits)
template <bool TRY = false>
__device__ __forceinline__ bool tc_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  if (TRY)
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(tc_smem(bar)), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(tc_smem(bar)), "r"(parity)
        : "memory");
  return ok != 0;
}

// 1: the phase is complete; 0: the wait ran out; -1: *stop was set meanwhile
__device__ __forceinline__ int tc_wait(uint64_t* bar, uint32_t parity, const volatile int* stop) {
  for (long q = 0; q < kTcSpin; ++q) {
    if (tc_test<true>(bar, parity)) return 1;
    if (stop && *stop) return -1;
  }
  return 0;
}

__device__ __forceinline__ float2 tc_bf16x2(uint32_t v) {
  return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&v));
}

// the published count of ready planes once it exceeds p (kTcStop: the block stops)
__device__ __forceinline__ uint32_t tc_ready(const uint32_t* word, uint32_t p) {
  for (long q = 0; q < 16 * kTcSpin; ++q) {
    uint32_t r;
    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(r) : "r"(tc_smem(word)) : "memory");
    if (r > p) return r;
  }
  return kTcStop;
}

// true in one lane of a converged warp
__device__ __forceinline__ bool tc_elect() {
  uint32_t p;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}"
               : "=r"(p));
  return p != 0;
}

// D (tensor memory) += A B of one M128 x N x K16 product
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.eq.u32 p, 0, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc)
      : "memory");
}

// *bar completes when every MMA issued so far has
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          tc_smem(bar))
      : "memory");
}

// zero 16 tensor-memory columns of the warp's lanes
__device__ __forceinline__ void tc_zero16(uint32_t taddr) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,"
      "%1};" ::"r"(taddr),
      "r"(0u)
      : "memory");
}

// A descriptor advanced by a byte offset (a multiple of 16): the start address is the low
// 14-bit field in 16-byte units, and shared-memory addresses stay below 2^18 bytes, so the sum
// does not carry out of the field.
__device__ __forceinline__ uint64_t tc_desc_at(uint64_t d, uint32_t bytes) {
  return d + (uint64_t)(bytes >> 4);
}

// Shape of the convolution CIN -> NB output channels (of COUT, in COUT / NB parts that blocks of
// their own compute, where the weights of all COUT do not fit or 3 COUT exceeds the MMA's N of 256).
template <int CIN, int NB>
struct TcShape {
  static_assert(CIN % 16 == 0 && NB % 16 == 0 && 3 * NB <= 256, "channel counts");
  static constexpr int KC = CIN / 16;                  // 16-channel slices of a plane
  static constexpr int N3 = 3 * NB;                    // the stacked N
  static constexpr int PLANE = kTcHP * 16;             // eight channels of a patch
  static constexpr int SLOT = 2 * PLANE;               // one slice of a plane's patch
  static constexpr int WTS = 27 * CIN * NB * 2;        // all taps, [t9][chunk][rb NB + o][8]
  static constexpr int LIMIT = 230400;                 // of the 227 KB a block can have
  static constexpr int FIT = (LIMIT - WTS) / SLOT;
  static constexpr int PLANES = (FIT < 30 ? FIT : 30) / KC;  // whole planes in the ring
  static constexpr int SMEM = WTS + PLANES * KC * SLOT + 128;  // + alignment slack
  static constexpr int R = 512 / NB;                   // accumulators in tensor memory
  static constexpr int COPY_WARPS = KC == 1 ? 2 : KC <= 3 ? 4 : 8;  // that copy a plane together
  static_assert(PLANES >= 2 && R >= 4, "ring");
};

// warps 0-7 epilogue (two groups of four, one per output plane in turn), 8-15 copies, 16 MMAs,
// 17 the MMAs' waits
constexpr int kTcCopyWarps = 8, kTcCopy0 = 8, kTcMma = kTcCopy0 + kTcCopyWarps;
constexpr int kTcThreads = 32 * (kTcMma + 2);
constexpr int kTcDone = 64;  // barriers of finished input planes, more than the roles can be apart

// What else the epilogue does with a layer's output (at 256 x 256 x 128 the pooling in a pass of its own
// took 53 us, here 36; the output layer 50, here 2).
enum TcEpilogue { kTcPlain, kTcPool, kTcOut };
struct TcExtra {
  __nv_bfloat16* pooled = nullptr;  // kTcPool: the 2x2x2 means (COUT channels), zc and nz even
  const float* wo = nullptr;        // kTcOut: y = (w_o . out + b_o) scale, COUT = 16
  const float* scale = nullptr;     // (1 where null)
  float* y = nullptr;
};

// UP > 0: the first UP input channels are the nearest 2x upsampling of the coarse field `coarse` (UP
// channels), read where it lies; `in` holds the others.
template <int CIN, int COUT, int NB, int UP, int EPI>
__global__ void __launch_bounds__(kTcThreads, 1)
    k_conv3_tc(const __nv_bfloat16* __restrict__ in, int in_stride, int in_off,
               const __nv_bfloat16* __restrict__ coarse,
               const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias,
               __nv_bfloat16* __restrict__ out, int out_stride, int out_off, int nx, int ny, int nz,
               int zc, int relu, TcExtra extra, int* err) {
  using S = TcShape<CIN, NB>;
  constexpr int PARTS = COUT / NB;
  extern __shared__ __align__(128) unsigned char tc_dyn[];
  unsigned char* wts = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(tc_dyn) + 127) & ~static_cast<uintptr_t>(127));
  unsigned char* ring = wts + S::WTS;
  __shared__ __align__(8) uint64_t full[S::PLANES];     // a plane's slices have landed
  __shared__ __align__(8) uint64_t acc_empty[S::R];     // an accumulator is read and zero again
  __shared__ __align__(8) uint64_t done[kTcDone + 1];   // the MMAs of an input plane (last: all)
  __shared__ uint32_t ready_word;  // input planes whose slices and accumulators are ready
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  __shared__ float bias_s[NB], wo_s[EPI == kTcOut ? NB + 1 : 1];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform to the compiler, too
  const int part = blockIdx.x % PARTS, o0 = part * NB;

  if (warp == kTcMma) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     tc_smem(&tmem_slot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int q = 0; q < S::PLANES; ++q) tc_bar_init(&full[q], 32 * S::COPY_WARPS);
    for (int q = 0; q < S::R; ++q) tc_bar_init(&acc_empty[q], 4);
    for (int q = 0; q <= kTcDone; ++q) tc_bar_init(&done[q], 1);
    ready_word = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_word = 0;
  }
  if (tid < NB) bias_s[tid] = bias ? bias[o0 + tid] : 0.f;
  if (EPI == kTcOut && tid <= NB) wo_s[tid] = extra.wo[tid];
  // all 27 taps of the weights, once per block, the dz taps stacked along N
  for (int q = tid; q < 9 * 2 * S::KC * S::N3; q += kTcThreads) {
    const int c = q % (2 * S::KC), orow = (q / (2 * S::KC)) % S::N3, t9 = q / (S::N3 * 2 * S::KC);
    const int rb = orow / NB, o = orow % NB, tap = (2 - rb) * 9 + t9;
    tc_cp16(wts + ((t9 * 2 * S::KC + c) * S::N3 + orow) * 16,
            W + ((size_t)tap * COUT + o0 + o) * CIN + 8 * c, 16);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  // the copies are generic-proxy writes the tensor cores read through the async proxy
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  volatile int* abort_flag = &abort_word;
  // a bounded wait; where it runs out (or another role's has) the block stops issuing work
  auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
    const int r = tc_wait(bar, parity, abort_flag);
    if (r == 0) {
      *abort_flag = 1;
      atomicExch(err, 1);
    }
    return r == 1;
  };

  const int xt = tc_tiles_x(nx), yt = tc_tiles_y(ny);
  const int zcols = (nz + zc - 1) / zc;
  const long items = (long)xt * yt * zcols;
  const long first = blockIdx.x / PARTS, step = gridDim.x / PARTS;
  // the input planes of the whole block are counted: plane p's MMAs complete done[p % kTcDone]
  auto wait_done = [&](uint32_t p) {
    return wait(&done[p % kTcDone], (p / kTcDone) & 1u);
  };

  if (warp < kTcCopy0) {
    // ---- epilogue: warp w reads lanes 32 (w % 4) .. (its 32 pixels) of each finished accumulator
    const int wr = warp & 3;
    const uint32_t lane_base = tmem + ((uint32_t)(wr * 32) << 16);
    if (warp < 4) {
      for (int c0 = 0; c0 < S::R * NB; c0 += 16) tc_zero16(lane_base + (uint32_t)c0);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        for (int q = 0; q < S::R; ++q) tc_arrive(&acc_empty[q]);
    }
    const int px0 = (wr * 32 + lane) & 7, py0 = (wr * 32 + lane) >> 3;
    uint32_t v = 0, pb = 0;  // accumulators and input planes of the columns before
    const float yscale = EPI == kTcOut && extra.scale ? *extra.scale : 1.f;
    bool ok = true;
    for (long item = first; item < items && ok; item += step) {
      const int px = (int)(item % xt) * kTcTX + px0;
      const long rest = item / xt;
      const int py = (int)(rest % yt) * kTcTY + py0;
      const int zb = (int)(rest / yt) * zc, ze = min(nz, zb + zc);
      const int z0 = max(zb - 1, 0), z1 = min(ze, nz - 1);
      __nv_bfloat16* dst = out + ((size_t)px + (size_t)nx * ((size_t)py + (size_t)ny * zb)) *
                                     out_stride + out_off + o0;
      float pool[EPI == kTcPool ? NB : 1];  // of the plane pair that this warp's group takes
      for (int z = zb; z < ze; ++z, ++v, dst += (size_t)nx * ny * out_stride) {
        if ((int)((EPI == kTcPool ? v >> 1 : v) & 1u) != warp >> 2) continue;
        const uint32_t slot = v % S::R;
        // complete with the input plane below it (the last plane of the grid with its own)
        ok = wait_done(pb + (uint32_t)(min(z + 1, z1) - z0));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t r[NB];
#pragma unroll
        for (int cb = 0; cb < NB; cb += 16) {
          uint32_t* q = r + cb;
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
              "%13,%14,%15}, [%16];"
              : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]),
                "=r"(q[6]), "=r"(q[7]), "=r"(q[8]), "=r"(q[9]), "=r"(q[10]), "=r"(q[11]),
                "=r"(q[12]), "=r"(q[13]), "=r"(q[14]), "=r"(q[15])
              : "r"(lane_base + slot * NB + (uint32_t)cb));
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int cb = 0; cb < NB; cb += 16) tc_zero16(lane_base + slot * NB + (uint32_t)cb);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) tc_arrive(&acc_empty[slot]);
        const bool in_grid = px < nx && py < ny;
        uint32_t packed[NB / 2];
#pragma unroll
        for (int q = 0; q < NB / 2; ++q) {
          float v0 = __uint_as_float(r[2 * q]) + bias_s[2 * q];
          float v1 = __uint_as_float(r[2 * q + 1]) + bias_s[2 * q + 1];
          if (relu) {
            v0 = fmaxf(v0, 0.f);
            v1 = fmaxf(v1, 0.f);
          }
          __nv_bfloat162 h = __floats2bfloat162_rn(v0, v1);
          packed[q] = *reinterpret_cast<uint32_t*>(&h);
        }
        if (in_grid && (EPI != kTcOut || out != nullptr)) {
#pragma unroll
          for (int q = 0; q < NB / 8; ++q)
            reinterpret_cast<uint4*>(dst)[q] = make_uint4(packed[4 * q], packed[4 * q + 1],
                                                          packed[4 * q + 2], packed[4 * q + 3]);
        }
        if constexpr (EPI == kTcOut) {
          float t = wo_s[NB];
#pragma unroll
          for (int q = 0; q < NB / 2; ++q) {
            const float2 f = tc_bf16x2(packed[q]);
            t = fmaf(wo_s[2 * q], f.x, t);
            t = fmaf(wo_s[2 * q + 1], f.y, t);
          }
          if (in_grid) extra.y[(size_t)px + (size_t)nx * ((size_t)py + (size_t)ny * z)] = t * yscale;
        }
        if constexpr (EPI == kTcPool) {
          // the pixels right, below and below right are lanes + 1, + 8, + 9 (four rows of eight)
#pragma unroll
          for (int q = 0; q < NB / 2; ++q) {
            float2 t = z & 1 ? make_float2(pool[2 * q], pool[2 * q + 1]) : make_float2(0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int off = u == 0 ? 0 : u == 1 ? 1 : u == 2 ? 8 : 9;
              const float2 f =
                  tc_bf16x2(off ? __shfl_down_sync(0xffffffffu, packed[q], off) : packed[q]);
              t.x += f.x;
              t.y += f.y;
            }
            pool[2 * q] = t.x;
            pool[2 * q + 1] = t.y;
          }
          if ((z & 1) && in_grid && !(px & 1) && !(py & 1)) {
            const size_t c = (size_t)(px >> 1) +
                             (size_t)(nx >> 1) * ((size_t)(py >> 1) + (size_t)(ny >> 1) * (z >> 1));
            uint4* pd = reinterpret_cast<uint4*>(extra.pooled + c * COUT + o0);
#pragma unroll
            for (int q = 0; q < NB / 8; ++q) {
              uint32_t w4[4];
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                __nv_bfloat162 h = __floats2bfloat162_rn(0.125f * pool[8 * q + 2 * u],
                                                         0.125f * pool[8 * q + 2 * u + 1]);
                w4[u] = *reinterpret_cast<uint32_t*>(&h);
              }
              pd[q] = make_uint4(w4[0], w4[1], w4[2], w4[3]);
            }
          }
        }
      }
      pb += (uint32_t)(z1 - z0 + 1);
    }
  } else if (warp < kTcMma) {
    // ---- copies: a plane's 16-byte pieces in memory order (a pixel's channels, then the next
    // pixel's) over the lanes of a group of copy warps, so that an instruction's pieces share lines;
    // the groups take the planes in turn (about six pieces per lane and plane).  The
    // copies signal the plane's barrier themselves when they have landed, so that all free slots of
    // the ring are being filled at any time; the warp that sees the barrier complete fences them
    // against the tensor cores' reads (a fence here would wait for the warp's copies in flight).
    constexpr int CH = 2 * S::KC, N = kTcHP * CH, LANES = 32 * S::COPY_WARPS;
    constexpr uint32_t GROUPS = kTcCopyWarps / S::COPY_WARPS;
    constexpr int PIECES = (N + LANES - 1) / LANES;
    const int t = (tid - 32 * kTcCopy0) % LANES;
    const uint32_t group = (uint32_t)(warp - kTcCopy0) / S::COPY_WARPS;
    uint32_t p = 0;
    bool ok = true;
    for (long item = first; item < items && ok; item += step) {
      const int x0 = (int)(item % xt) * kTcTX - 1;
      const long rest = item / xt;
      const int y0 = (int)(rest % yt) * kTcTY - 1;
      const int zb = (int)(rest / yt) * zc, ze = min(nz, zb + zc);
      const int z0 = max(zb - 1, 0), z1 = min(ze, nz - 1);
      // the lane's pixels in the plane (of the coarse field for its channels), -1 outside the grid
      int pix[PIECES];
#pragma unroll
      for (int q = 0; q < PIECES; ++q) {
        const int h = (t + q * LANES) / CH, xx = x0 + h % kTcHX, yy = y0 + h / kTcHX;
        const bool in_grid = h < kTcHP && xx >= 0 && xx < nx && yy >= 0 && yy < ny;
        const bool up = UP > 0 && (t + q * LANES) % CH < UP / 8;
        pix[q] = !in_grid ? -1 : up ? (xx >> 1) + (nx >> 1) * (yy >> 1) : xx + nx * yy;
      }
      for (int z = z0; z <= z1; ++z, ++p) {
        if (p % GROUPS != group) continue;
        const uint32_t slot = p % S::PLANES;
        if (p >= S::PLANES) {
          ok = wait_done(p - S::PLANES);  // the slot's last readers
          if (!ok) break;
        }
        const __nv_bfloat16* src = in + (size_t)nx * ny * z * in_stride + in_off - UP;
        const __nv_bfloat16* csrc =
            UP > 0 ? coarse + (size_t)(nx >> 1) * (ny >> 1) * (z >> 1) * UP : nullptr;
        unsigned char* d = ring + slot * (uint32_t)(S::KC * S::SLOT);
#pragma unroll
        for (int q = 0; q < PIECES; ++q) {
          const int e = t + q * LANES, h = e / CH, c = e % CH;
          const bool up = UP > 0 && c < UP / 8;
          if (e < N)
            tc_cp16(d + c * S::PLANE + h * 16,
                    pix[q] < 0 ? in
                               : (up ? csrc + (size_t)pix[q] * UP
                                     : src + (size_t)pix[q] * in_stride) + 8 * c,
                    pix[q] < 0 ? 0 : 16);
        }
        tc_arrive_copies(&full[slot]);
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp == kTcMma) {
    // ---- MMAs: the whole warp runs the loop, so that the descriptors are warp-uniform values
    // (the instruction's operands are uniform registers); an elected lane issues
    const uint32_t wts_s = tc_smem(wts), ring_s = tc_smem(ring);
    const bool leader = tc_elect();
    const uint64_t a_ring = tc_desc(ring_s, S::PLANE, kTcHX * 16);
    const uint64_t b_all = tc_desc(wts_s, S::N3 * 16, 128);
    constexpr uint32_t i3 = tc_idesc(S::N3);
    uint32_t ready = 0, p = 0;        // input planes known to be ready, and done
    uint32_t slot = 0, bar = 0;       // p % PLANES, p % kTcDone
    uint32_t s0 = 0;                  // accumulator of the plane's first output plane
    for (long item = first; item < items && ready != kTcStop; item += step) {
      const int zb = (int)(item / ((long)xt * yt)) * zc, ze = min(nz, zb + zc);
      const int z0 = max(zb - 1, 0), z1 = min(ze, nz - 1);
      for (int zp = z0; zp <= z1; ++zp) {
        const uint64_t a0 = tc_desc_at(a_ring, slot * (uint32_t)(S::KC * S::SLOT));
        const uint32_t d0 = tmem + s0 * NB;
        // one or two MMAs for each tap and slice
        auto taps = [&](uint64_t b1, uint32_t i1, auto split, uint64_t b2, uint32_t i2) {
          if (leader) {
#pragma unroll
            for (int t9 = 0; t9 < 9; ++t9) {
#pragma unroll
              for (int kc = 0; kc < S::KC; ++kc) {
                const uint64_t a = tc_desc_at(a0, kc * S::SLOT + (t9 / 3 * kTcHX + t9 % 3) * 16);
                const uint32_t bo = (uint32_t)((t9 * S::KC + kc) * 2 * S::N3 * 16);
                tc_mma(d0, a, tc_desc_at(b1, bo), i1);
                if (split) tc_mma(tmem, a, tc_desc_at(b2, bo), i2);
              }
            }
            tc_commit(&done[bar]);
          }
        };
        if (ready <= p) ready = __shfl_sync(0xffffffffu, tc_ready(&ready_word, p), 0);
        if (ready == kTcStop) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (zp > zb && zp < ze - 1 && s0 + 3 <= S::R) {
          taps(b_all, i3, std::false_type{}, b_all, i3);
          s0 = s0 + 1 == S::R ? 0 : s0 + 1;
        } else {
          // output planes lo .. hi, which this input plane adds to; their accumulators are adjacent
          // but where the ring of accumulators starts again
          const int lo = max(zb, zp - 1), hi = min(ze - 1, zp + 1), count = hi - lo + 1;
          const int c1 = min(count, (int)(S::R - s0)), c2 = count - c1;
          const uint64_t b1 = tc_desc_at(b_all, (uint32_t)((lo - (zp - 1)) * NB * 16));
          if (c2)
            taps(b1, tc_idesc(NB * c1), std::true_type{},
                 tc_desc_at(b1, (uint32_t)(c1 * NB * 16)), tc_idesc(NB * c2));
          else
            taps(b1, tc_idesc(NB * c1), std::false_type{}, b1, i3);
          // the next plane's first output plane; after a column, the next column's
          const int next = zp == z1 ? ze : max(zb, zp);
          s0 = (s0 + (uint32_t)(next - lo)) % S::R;
        }
        ++p;
        slot = slot + 1 == S::PLANES ? 0 : slot + 1;
        bar = (bar + 1) % kTcDone;
      }
    }
    // every MMA has finished before the tensor memory is freed, also after a wait that ran out
    if (leader) {
      tc_commit(&done[kTcDone]);
      (void)tc_wait(&done[kTcDone], 0u, nullptr);
    }
    __syncwarp();
  } else {
    // ---- the MMAs' waits: a wait's latency (about 350 clocks, ready or not) in the issuing warp
    // would leave the tensor cores idle between planes.  Here half the lanes test the next 16 planes
    // and half the next 16 accumulators at once (a barrier's next phase only: the one before is
    // known to be complete), and the issuing warp reads one counter when the planes it knows of
    // are used up.
    constexpr int NF = S::PLANES < 16 ? S::PLANES : 16, NA = S::R < 16 ? S::R : 16;
    uint32_t p = 0, vb = 0;          // planes published; accumulators of the columns before
    uint32_t landed = 0, accs = 0;   // that are known to be ready
    bool ok = true;
    for (long item = first; item < items && ok; item += step) {
      const int zb = (int)(item / ((long)xt * yt)) * zc, ze = min(nz, zb + zc);
      const int z0 = max(zb - 1, 0), z1 = min(ze, nz - 1);
      for (int zp = z0; zp <= z1 && ok; ++zp, ++p) {
        const uint32_t need_acc = vb + (uint32_t)(min(ze - 1, zp + 1) - zb + 1);
        for (long q = 0; landed <= p || accs < need_acc; ++q) {
          const uint32_t n = lane < 16 ? landed + lane : accs + (uint32_t)(lane - 16);
          const bool t = lane < 16 ? lane < NF && tc_test(&full[n % S::PLANES], (n / S::PLANES) & 1u)
                                   : lane - 16 < NA &&
                                         tc_test(&acc_empty[n % S::R], (n / S::R) & 1u);
          const uint32_t m = ~__ballot_sync(0xffffffffu, t);
          landed += (uint32_t)__ffs(m & 0xffffu | 0x10000u) - 1;
          accs += (uint32_t)__ffs(m >> 16 | 0x10000u) - 1;
          if (__any_sync(0xffffffffu, *abort_flag || q >= kTcSpin)) {
            ok = false;
            break;
          }
        }
        // the copies are generic-proxy writes the tensor cores read through the async proxy
        __syncwarp();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0)
          asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(tc_smem(&ready_word)),
                       "r"(ok ? p + 1 : kTcStop)
                       : "memory");
      }
      vb += (uint32_t)(ze - zb);
    }
    if (!ok && lane == 0 && !*abort_flag) {
      *abort_flag = 1;
      atomicExch(err, 1);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kTcMma)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512)
                 : "memory");
}

}  // namespace unet
}  // namespace fg
