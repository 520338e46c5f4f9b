// Weight gradients of the U-Net's 3x3x3 convolutions.  Not in reference.
//
//   dW[t][o][i] = sum over pixels p of g[p][o] in[p + off(t)][i]      (zero outside the grid)
//
// For every tap a small matrix product whose long dimension is the pixels: M = output channels,
// N = input channels (both 16 to 96), K = pixels, on the warp-level mma.m16n8k16 (BF16 operands,
// FP32 accumulators).  (tcgen05 has 64 or 128 rows of M, three quarters empty for 16 output
// channels; with (tap, input channel) along M they would be full, a form not written yet.)  One warp owns the nine taps of one dz for 16
// input channels and 16 or 32 output channels, 72 or 144 accumulators that stay in registers
// over all of the block's pixels.  Both operands lie channels-last, that is with the pixel (K)
// outermost, and reach the fragments by transposing ldmatrix loads; a tap is the same patch read
// from a shifted pixel, so nothing is copied per tap.
//
// A block walks z columns of 16 x 16-pixel tiles: a ring of four input planes (18 x 18 pixels
// with the halo, 16 channels, [chunk of 8][pixel][16 bytes]: eight consecutive pixels of a
// chunk are 128 consecutive bytes, free of bank conflicts) and two planes of g; the next
// plane's cp.async copies run during this plane's products, one barrier per plane.
//
// Measured at 128 x 128 x 64: 16 -> 16 channels 59 us (122 GMAC/ms; an FP32 form with one thread
// per weight and pixels staged as floats took 3,340 us), 48 -> 16 156 us (10,120), 96 -> 32 on the
// half-size grid 97 us (3,350).  Bound by the transposing loads and products of the warps
// resident (18 per SM), not by memory: 64 bytes per pixel are 10 us.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

#include "unet_tc.cuh"

namespace fg {
namespace unet {

constexpr int kDwT = 16;               // the tile: 16 x 16 pixels of a plane
constexpr int kDwH = kDwT + 2;         // with the halo
constexpr int kDwPix = kDwT * kDwT;    // pixels of g per plane
constexpr int kDwHPix = kDwH * kDwH;   // staged input pixels per plane
constexpr int kDwThreads = 192;        // six warps: three dz times two row or channel groups

template <int COUT>
struct DwShape {
  static_assert(COUT % 16 == 0 && COUT <= 64, "output channels");
  static constexpr int MT = COUT == 16 ? 1 : 2;       // 16-channel row blocks per warp
  static constexpr int MG = COUT / (16 * MT);         // channel groups over warps
  static constexpr int RG = 2 / MG;                   // row groups over warps
  static constexpr int INP = 2 * kDwHPix * 16;        // one input plane, 16 channels
  static constexpr int GP = (COUT / 8) * kDwPix * 16; // one plane of g
  static constexpr int SMEM = 4 * INP + 2 * GP;
  static constexpr int BLOCKS = COUT == 16 ? 3 : 2;   // resident blocks per SM aimed at
};

__device__ __forceinline__ void dw_ldsm_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

__device__ __forceinline__ void dw_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                       uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// blockIdx.y: the group of 16 input channels; blocks of one group stride over the work items
// (an x/y tile times a z column of zc planes).  dW is added to (FP32 atomics, one per
// accumulator and block).  UP > 0: the first UP input channels are the nearest 2x upsampling of
// `coarse` (UP channels); `in` holds the others.
template <int CIN, int COUT, int UP>
__global__ void __launch_bounds__(kDwThreads, DwShape<COUT>::BLOCKS) k_conv3_dw(
    const __nv_bfloat16* __restrict__ in, int in_stride, int in_off,
    const __nv_bfloat16* __restrict__ coarse, const __nv_bfloat16* __restrict__ gout, int g_stride,
    int g_off, float* __restrict__ dW, int nx, int ny, int nz, int zc) {
  using S = DwShape<COUT>;
  extern __shared__ __align__(128) unsigned char dw_smem[];
  unsigned char* gbuf = dw_smem + 4 * S::INP;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int dz = warp % 3, grp = warp / 3;
  const int mg = S::MG == 2 ? grp : 0, rg = S::RG == 2 ? grp : 0;
  const int ic = blockIdx.y * 16;
  const uint32_t in_s = tc_smem(dw_smem), g_s = tc_smem(gbuf);
  const int j = lane >> 3, l8 = lane & 7;  // ldmatrix: matrix and row this lane addresses
  // A (g): matrices (k 0-7, m 0-7), (k 0-7, m 8-15), (k 8-15, m 0-7), (k 8-15, m 8-15)
  const uint32_t a_lane = (uint32_t)(((mg * S::MT * 2 + (j & 1)) * kDwPix + (j >> 1) * 8 + l8) * 16);
  // B (in): matrices (k 0-7, n 0-7), (k 8-15, n 0-7), (k 0-7, n 8-15), (k 8-15, n 8-15)
  const uint32_t b_lane = (uint32_t)(((j >> 1) * kDwHPix + (j & 1) * 8 + l8) * 16);

  float acc[S::MT][9][2][4];
#pragma unroll
  for (int m = 0; m < S::MT; ++m)
#pragma unroll
    for (int t = 0; t < 9; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[m][t][h][q] = 0.f;

  const int xt = (nx + kDwT - 1) / kDwT, yt = (ny + kDwT - 1) / kDwT;
  const int zt = (nz + zc - 1) / zc;
  const long items = (long)xt * yt * zt;
  for (long item = blockIdx.x; item < items; item += gridDim.x) {
    const int x0 = (int)(item % xt) * kDwT;
    const long rest = item / xt;
    const int y0 = (int)(rest % yt) * kDwT;
    const int zb = (int)(rest / yt) * zc, ze = min(nz, zb + zc);
    // input plane zz (16 channels, with the halo) into its ring slot, zero outside the grid
    auto load_in = [&](int zz) {
      unsigned char* dst = dw_smem + (zz & 3) * S::INP;
      const bool zok = zz >= 0 && zz < nz;
      for (int p = tid; p < kDwHPix; p += kDwThreads) {
        const int xx = x0 + p % kDwH - 1, yy = y0 + p / kDwH - 1;
        const bool ok = zok && xx >= 0 && xx < nx && yy >= 0 && yy < ny;
        const __nv_bfloat16* src = in;
        if (ok && UP > 0 && ic < UP)
          src = coarse + ((size_t)(xx >> 1) +
                          (size_t)(nx >> 1) * ((size_t)(yy >> 1) + (size_t)(ny >> 1) * (zz >> 1))) *
                             UP + ic;
        else if (ok)
          src = in + ((size_t)xx + (size_t)nx * ((size_t)yy + (size_t)ny * zz)) * in_stride + in_off +
                ic - UP;
        tc_cp16(dst + p * 16, src, ok ? 16 : 0);
        tc_cp16(dst + (kDwHPix + p) * 16, ok ? src + 8 : in, ok ? 16 : 0);
      }
    };
    auto load_g = [&](int z) {
      unsigned char* dst = gbuf + (z & 1) * S::GP;
      for (int p = tid; p < kDwPix; p += kDwThreads) {
        const int xx = x0 + p % kDwT, yy = y0 + p / kDwT;
        const bool ok = xx < nx && yy < ny;
        const __nv_bfloat16* src =
            ok ? gout + ((size_t)xx + (size_t)nx * ((size_t)yy + (size_t)ny * z)) * g_stride + g_off
               : gout;
#pragma unroll
        for (int c = 0; c < COUT / 8; ++c)
          tc_cp16(dst + (c * kDwPix + p) * 16, ok ? src + 8 * c : gout, ok ? 16 : 0);
      }
    };
    __syncthreads();  // the previous item's last products have read the slots
    load_in(zb - 1);
    load_in(zb);
    load_in(zb + 1);
    load_g(zb);
    for (int z = zb; z < ze; ++z) {
      // planes z-1, z, z+1 and g(z) have landed; every warp is done with plane z-1's products,
      // the last readers of input plane z-2 and of g(z-1), whose slots the next copies take
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      if (z + 1 < ze) {
        load_in(z + 2);
        load_g(z + 1);
      }
      const uint32_t a0 = g_s + (uint32_t)((z & 1) * S::GP) + a_lane;
      const uint32_t b0 = in_s + (uint32_t)(((z + dz - 1) & 3) * S::INP) + b_lane;
#pragma unroll 1
      for (int r = rg * (kDwT / S::RG); r < (rg + 1) * (kDwT / S::RG); ++r) {
        uint32_t a[S::MT][4];
#pragma unroll
        for (int m = 0; m < S::MT; ++m)
          dw_ldsm_t(a[m], a0 + (uint32_t)((m * 2 * kDwPix + r * kDwT) * 16));
#pragma unroll
        for (int t = 0; t < 9; ++t) {
          uint32_t b[4];
          dw_ldsm_t(b, b0 + (uint32_t)(((r + t / 3) * kDwH + t % 3) * 16));
#pragma unroll
          for (int m = 0; m < S::MT; ++m) {
            dw_mma(acc[m][t][0], a[m], b[0], b[1]);
            dw_mma(acc[m][t][1], a[m], b[2], b[3]);
          }
        }
      }
    }
  }
  // fragment row g = lane / 4 (and + 8), columns 2 (lane % 4) and the next
#pragma unroll
  for (int m = 0; m < S::MT; ++m)
#pragma unroll
    for (int t = 0; t < 9; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int o = (mg * S::MT + m) * 16 + (lane >> 2), i = ic + h * 8 + 2 * (lane & 3);
        float* d = dW + ((size_t)(dz * 9 + t) * COUT + o) * CIN + i;
        atomicAdd(reinterpret_cast<float2*>(d), make_float2(acc[m][t][h][0], acc[m][t][h][1]));
        atomicAdd(reinterpret_cast<float2*>(d + 8 * CIN),
                  make_float2(acc[m][t][h][2], acc[m][t][h][3]));
      }
}

}  // namespace unet
}  // namespace fg
