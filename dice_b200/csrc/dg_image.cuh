// dg_image.cuh -- image preparation: the Gaussian pre-filter and the gradients.
//
// Both are stencils whose every float product and sum is rounded on its own,
// in the reference's order, so their cost is the rounded operations (a
// multiply and an add per tap, no fused form): 98 per pixel for a 7 x 7
// filter, about 115 for smoothed gradients, against 8 and 12 bytes of DRAM
// traffic.  What has to be kept small is everything beside them: a CTA stages
// its input tile (with the halo) in shared memory once, a thread takes a
// column of several output rows, so that a tile value is read once for all
// the rows it contributes to, and the operations run two at a time (packed
// float pairs), which leaves the issue slots to the rest.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "dg_device.cuh"

namespace dg {

// ---------------------------------------------------------------------------
// Image_::gauss_filter (DICe_Image.cpp:1194-1230): the sum runs x offset
// outer, y offset inner; pixels within M/2 + 1 of an edge keep their value.
// The M x M weights travel by value in the parameter bank (uniform reads).
//
// A thread sums P rows of columns x and x + 32 as packed pairs (the tile holds
// the two columns' values side by side): for each x offset it reads the
// M + P - 1 pairs its rows need, 14 shared loads for 112 products at M = 7 and
// P = 8, where a row of one column per thread took 49 loads for 49.  The x
// offsets are a rolled loop, which keeps the code within the instruction
// cache.  P = 8 amortises the loads of large images; small ones want CTAs
// for every SM (P = 2).  4096^2, M = 7: 80 us, 0.55 of the rounded operations'
// rate (one column per thread, scalar operations: 105 us).
// ---------------------------------------------------------------------------
struct GaussWeights {
  f32x2 c[13 * 13];   // each weight twice
};

constexpr int kGaussBX = 32, kGaussBY = 8;   // threads; a tile is 64 columns by 8 P rows

template <int M, int P>
__global__ void __launch_bounds__(kGaussBX* kGaussBY)
gauss_filter_kernel(int w, int h, const __grid_constant__ GaussWeights wt, f32x2 minus_zero,
                    const float* __restrict__ in, float* __restrict__ out) {
  constexpr int R = M / 2;              // taps reach R pixels either side
  constexpr int half = M / 2 + 1;       // the reference's interior test
  constexpr int TW = kGaussBX + 2 * R, TH = kGaussBY * P + 2 * R;
  __shared__ float2 tile[TH * TW];
  const int x0 = blockIdx.x * 2 * kGaussBX - R, y0 = blockIdx.y * kGaussBY * P - R;
  if (x0 >= 0 && y0 >= 0 && x0 + TW + kGaussBX <= w && y0 + TH <= h) {
    // 32 of the TW pairs of a row per warp, then the 2 R that are left over
    // of all rows, spread over the CTA (a second, nearly empty load per row
    // cost as much as the first)
    const float* src = in + (size_t)(y0 + threadIdx.y) * w + x0 + threadIdx.x;
    for (int ty = threadIdx.y; ty < TH; ty += kGaussBY) {
      tile[ty * TW + threadIdx.x] = make_float2(__ldg(src), __ldg(src + kGaussBX));
      src += (size_t)kGaussBY * w;
    }
    for (int k = threadIdx.y * kGaussBX + threadIdx.x; k < TH * 2 * R; k += kGaussBX * kGaussBY) {
      const int ty = k / (2 * R), tx = kGaussBX + k - ty * 2 * R;
      const float* q = in + (size_t)(y0 + ty) * w + x0 + tx;
      tile[ty * TW + tx] = make_float2(__ldg(q), __ldg(q + kGaussBX));
    }
  } else {
    for (int k = threadIdx.y * kGaussBX + threadIdx.x; k < TH * TW; k += kGaussBX * kGaussBY) {
      const int ty = k / TW, tx = k - ty * TW;
      const int ga = x0 + tx, gb = ga + kGaussBX, gy = y0 + ty;
      const bool row = gy >= 0 && gy < h;
      const float* src = in + (size_t)(row ? gy : 0) * w;
      tile[k] = make_float2(row && ga >= 0 && ga < w ? __ldg(src + ga) : 0.0f,
                            row && gb >= 0 && gb < w ? __ldg(src + gb) : 0.0f);
    }
  }
  __syncthreads();
  const int ya = threadIdx.y * P;   // the thread's first row in the tile's output
  const float2* col = tile + ya * TW + threadIdx.x;
  f32x2 v[P];
#pragma unroll
  for (int p = 0; p < P; ++p) v[p] = f2_pack(0.0f, 0.0f);
#pragma unroll 1
  for (int i = 0; i < M; ++i) {
    f32x2 t[P + M - 1];
#pragma unroll
    for (int r = 0; r < P + M - 1; ++r) t[r] = *reinterpret_cast<const f32x2*>(col + r * TW + i);
#pragma unroll
    for (int j = 0; j < M; ++j) {
      const f32x2 c = wt.c[i * M + j];
#pragma unroll
      for (int p = 0; p < P; ++p) v[p] = f2_add(v[p], f2_mul(c, t[p + j], minus_zero));
    }
  }
  const int x = blockIdx.x * 2 * kGaussBX + threadIdx.x;
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const int y = blockIdx.y * kGaussBY * P + ya + p;
    if (y >= h) break;
    float a, b;
    f2_unpack(v[p], a, b);
    const float2 keep = col[(p + R) * TW + R];
    const bool rows = y >= half && y < h - half;
    const int xb = x + kGaussBX;
    if (x < w) out[(size_t)y * w + x] = rows && x >= half && x < w - half ? a : keep.x;
    if (xb < w) out[(size_t)y * w + xb] = rows && xb >= half && xb < w - half ? b : keep.y;
  }
}

// ---------------------------------------------------------------------------
// Image_::compute_gradients (DICe_Image.cpp:1015-1093): finite differences
// with c1 = 1/12, c2 = -8/12 stored as float (:214-215), one-sided within two
// pixels of the border.  A row of 256 pixels per CTA: bound by DRAM on large
// images, by the launch on small ones (a tile in shared memory gained nothing
// at 4096^2 and lost 5 us at 512^2).
// ---------------------------------------------------------------------------
__global__ void gradient_fd_kernel(int w, int h, const float* __restrict__ I, float* __restrict__ gx,
                                   float* __restrict__ gy) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  if (x >= w || y >= h) return;
  const float c1 = (float)(1.0 / 12.0), c2 = (float)(-8.0 / 12.0);
  const size_t i = (size_t)y * w + x;
  float a, b;
  if (x < 2) a = __fsub_rn(I[i + 1], I[i]);
  else if (x >= w - 2) a = __fsub_rn(I[i], I[i - 1]);
  else a = __fsub_rn(__fsub_rn(__fadd_rn(__fmul_rn(c1, I[i - 2]), __fmul_rn(c2, I[i - 1])),
                               __fmul_rn(c2, I[i + 1])),
                     __fmul_rn(c1, I[i + 2]));
  if (y < 2) b = __fsub_rn(I[i + w], I[i]);
  else if (y >= h - 2) b = __fsub_rn(I[i], I[i - w]);
  else b = __fsub_rn(__fsub_rn(__fadd_rn(__fmul_rn(c1, I[i - 2 * (size_t)w]), __fmul_rn(c2, I[i - w])),
                               __fmul_rn(c2, I[i + w])),
                     __fmul_rn(c1, I[i + 2 * (size_t)w]));
  gx[i] = a;
  gy[i] = b;
}

// The differences followed by smooth_gradients_convolution_5_point
// (:1034-1060): the outer product of (1,4,6,4,1)/16, rows outer, on the
// interior, borders copied.  One launch: the differences of the tile and its
// halo stay in shared memory (as two kernels they crossed DRAM twice, through
// 134 MB of planes allocated and freed for each call at 4096^2).  A thread
// smooths eight rows of a column, both differences as one packed pair: a pair
// read once enters up to five rows of sums with three distinct products.
// 4096^2: 95 us, 512^2: 10.5 us (tiles with flat index loops and no shared
// products: 139 and 10.6; a warp walking down a strip without CTA barriers:
// 129 and 16.7).
constexpr int kSmoothB = 32, kSmoothBY = 4, kSmoothP = kSmoothB / kSmoothBY;   // 32 x 32 tile, 32 x 4 threads
struct SmoothWeights {
  f32x2 k[3][3];   // products of 1/16, 4/16, 6/16 (exact), each twice
};

template <bool EDGE>
__device__ __forceinline__ f32x2 tile_difference(const float* q, int S, int x, int y, int w, int h) {
  const float c1 = (float)(1.0 / 12.0), c2 = (float)(-8.0 / 12.0);
  float a, b;
  if (EDGE && x < 2) a = __fsub_rn(q[1], q[0]);
  else if (EDGE && x >= w - 2) a = __fsub_rn(q[0], q[-1]);
  else a = __fsub_rn(__fsub_rn(__fadd_rn(__fmul_rn(c1, q[-2]), __fmul_rn(c2, q[-1])), __fmul_rn(c2, q[1])),
                     __fmul_rn(c1, q[2]));
  if (EDGE && y < 2) b = __fsub_rn(q[S], q[0]);
  else if (EDGE && y >= h - 2) b = __fsub_rn(q[0], q[-S]);
  else b = __fsub_rn(__fsub_rn(__fadd_rn(__fmul_rn(c1, q[-2 * S]), __fmul_rn(c2, q[-S])), __fmul_rn(c2, q[S])),
                     __fmul_rn(c1, q[2 * S]));
  return f2_pack(a, b);
}

__global__ void __launch_bounds__(kSmoothB* kSmoothBY)
gradient_smooth_kernel(int w, int h, const __grid_constant__ SmoothWeights wt, f32x2 minus_zero,
                       const float* __restrict__ I, float* __restrict__ gx, float* __restrict__ gy) {
  constexpr int S = kSmoothB + 8;   // the image tile, four pixels of halo
  constexpr int D = kSmoothB + 4;   // the differences' tile, two of halo
  constexpr int NT = kSmoothB * kSmoothBY;
  __shared__ float img[S * S];
  __shared__ f32x2 dif[D * D];
  const int bx = blockIdx.x * kSmoothB, by = blockIdx.y * kSmoothB;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kSmoothB + tx;
  // every pixel read lies inside the image, every difference two or more from its border
  const bool inside = bx >= 4 && by >= 4 && bx + kSmoothB + 4 <= w && by + kSmoothB + 4 <= h;
  if (inside) {
    // 32 columns of each row per warp, then the columns left over of all rows
    const float* src = I + (size_t)(by - 4) * w + bx - 4;
#pragma unroll
    for (int r = 0; r < S / kSmoothBY; ++r)
      img[(ty + r * kSmoothBY) * S + tx] = __ldg(src + (size_t)(ty + r * kSmoothBY) * w + tx);
    for (int k = tid; k < S * (S - kSmoothB); k += NT) {
      const int y = k / (S - kSmoothB), x = kSmoothB + k % (S - kSmoothB);
      img[y * S + x] = __ldg(src + (size_t)y * w + x);
    }
    __syncthreads();
    constexpr int RD = D / kSmoothBY;   // rows of differences per thread
    const float* q = img + (ty * RD + 2) * S + tx + 2;
#pragma unroll
    for (int r = 0; r < RD; ++r)
      dif[(ty * RD + r) * D + tx] = tile_difference<false>(q + r * S, S, 0, 0, w, h);
    for (int k = tid; k < D * (D - kSmoothB); k += NT) {
      const int y = k / (D - kSmoothB), x = kSmoothB + k % (D - kSmoothB);
      dif[y * D + x] = tile_difference<false>(img + (y + 2) * S + x + 2, S, 0, 0, w, h);
    }
  } else {
    for (int k = tid; k < S * S; k += NT) {
      const int x = bx - 4 + k % S, y = by - 4 + k / S;
      img[k] = (x >= 0 && x < w && y >= 0 && y < h) ? __ldg(I + (size_t)y * w + x) : 0.0f;
    }
    __syncthreads();
    for (int k = tid; k < D * D; k += NT) {
      const int dx = k % D, dy = k / D, x = bx - 2 + dx, y = by - 2 + dy;
      dif[k] = (x >= 0 && x < w && y >= 0 && y < h)
                   ? tile_difference<true>(img + (dy + 2) * S + dx + 2, S, x, y, w, h) : 0ull;
    }
  }
  __syncthreads();
  const int x = bx + tx, ya = ty * kSmoothP;
  const f32x2* col = dif + ya * D + tx;
  f32x2 sum[kSmoothP];
#pragma unroll
  for (int p = 0; p < kSmoothP; ++p) sum[p] = f2_pack(0.0f, 0.0f);
#pragma unroll
  for (int r = 0; r < kSmoothP + 4; ++r) {
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      const f32x2 t = col[r * D + b];
      f32x2 m[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) m[k] = f2_mul(wt.k[k][b < 3 ? b : 4 - b], t, minus_zero);
#pragma unroll
      for (int p = 0; p < kSmoothP; ++p) {
        const int a = r - p;   // row a of the five of output row p
        if (a >= 0 && a < 5) sum[p] = f2_add(sum[p], m[a < 3 ? a : 4 - a]);
      }
    }
  }
  if (x >= w) return;
#pragma unroll
  for (int p = 0; p < kSmoothP; ++p) {
    const int y = by + ya + p;
    if (y >= h) break;
    f32x2 g = sum[p];
    if (!inside && (x < 2 || x >= w - 2 || y < 2 || y >= h - 2)) g = dif[(ya + p + 2) * D + tx + 2];
    float a, b;
    f2_unpack(g, a, b);
    const size_t i = (size_t)y * w + x;
    gx[i] = a;
    gy[i] = b;
  }
}

// (I, Gx, Gy) -> interleaved float4 (the layout the frame kernel gathers from)
__global__ void pack_kernel(size_t n, const float* __restrict__ I, const float* __restrict__ gx,
                            const float* __restrict__ gy, float4* __restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = make_float4(I[i], gx[i], gy[i], 0.0f);
}

}  // namespace dg
