// Headless point rasteriser: the reference's draw pass
// (assets/shaders/draw.wgsl:18-40: one instanced quad of half-size 0.4 world
// units per particle, white on black; MSAA 4, runners/bevy/src/render/
// pipeline.rs:52-56) as CUDA kernels writing an 8-bit framebuffer instead of
// a swapchain image.
//
// Mapping (the vertex shader's NDC transform, y up in the world, row 0 at the
// top of the image): a world point (x, y) lands on pixel coordinates
//   X = x * sx,  Y = height_px - y * sy,  sx = width_px / W, sy = height_px / H.
// A particle covers the axis-aligned square [X - hx, X + hx) x [Y - hy, Y + hy)
// with hx = 0.4 * sx, hy = 0.4 * sy; a sample is covered when it lies in that
// half-open square (the top-left fill rule of an axis-aligned quad).  Each
// pixel has the four standard MSAA sample positions.  As in a multisampled
// colour target, a sample is white once any quad covers it, so a pixel's
// value is the resolve of the union of its covered samples:
// 255 * popcount(mask) / 4, rounded down, where the 4-bit mask is OR-ed over
// every particle that touches the pixel.
#include <stdint.h>

#include "wrach_internal.cuh"
#include "wrach_kernels.h"

namespace wrach {

namespace {

// standard 4x sample positions inside a pixel
__constant__ float kSampleX[4] = {0.375f, 0.875f, 0.125f, 0.625f};
__constant__ float kSampleY[4] = {0.125f, 0.375f, 0.625f, 0.875f};

// The samples of pixel column px whose x lies in [x0, x1) (or of a row's y).
__device__ __forceinline__ uint32_t samples_in(const float (&offset)[4], int px, float x0,
                                               float x1) {
  uint32_t m = 0;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const float at = __fadd_rn((float)px, offset[s]);
    m |= at >= x0 && at < x1 ? 1u << s : 0u;
  }
  return m;
}

// The coverage is kept 4 bits per pixel, 8 pixels of a row per word.  A
// sample is covered when its column's and its row's tests both hold, so the
// two are taken apart, and pixels of a word share one atomic.  Squares of at
// most 2 x 2 pixels (a window at the world's own scale) take no loops.  1M
// particles at 1920x1080: 15.7 us with a word and an atomic per pixel and 16
// tests for each, 9.2 us now, and the resolve reads an eighth (5.7 -> 2.4 us);
// what bounds it are the tests, not the atomics (collecting a block's words
// in shared memory first took longer).
__global__ void __launch_bounds__(256)
k_raster(const float2* __restrict__ pos, uint32_t n, float sx, float sy, uint32_t width_px,
         uint32_t height_px, uint32_t row_words, uint32_t* __restrict__ cover) {
  begin_after();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float2 p = pos[i];
  const float X = __fmul_rn(p.x, sx);
  const float Y = __fsub_rn((float)height_px, __fmul_rn(p.y, sy));
  const float hx = __fmul_rn(0.4f, sx), hy = __fmul_rn(0.4f, sy);
  const float x0 = __fsub_rn(X, hx), x1 = __fadd_rn(X, hx);
  const float y0 = __fsub_rn(Y, hy), y1 = __fadd_rn(Y, hy);
  if (!(x1 > 0.0f) || !(y1 > 0.0f) || !(x0 < (float)width_px) || !(y0 < (float)height_px)) return;
  const int px0 = max((int)floorf(x0), 0), px1 = min((int)floorf(x1), (int)width_px - 1);
  const int py0 = max((int)floorf(y0), 0), py1 = min((int)floorf(y1), (int)height_px - 1);
  uint32_t* row = cover + (size_t)py0 * row_words + (px0 >> 3);
  if (px1 - px0 <= 1 && py1 - py0 <= 1) {
    const uint32_t shift = 4u * (px0 & 7);
    uint32_t columns = samples_in(kSampleX, px0, x0, x1);
    if (px1 > px0) columns |= samples_in(kSampleX, px1, x0, x1) << 4;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if (py0 + r > py1) break;
      const uint32_t m = columns & (samples_in(kSampleY, py0 + r, y0, y1) * 0x11u);
      const uint32_t here = m << shift, next = shift == 28u ? m >> 4 : 0u;
      if (here) atomicOr(row, here);
      if (next) atomicOr(row + 1, next);
      row += row_words;
    }
    return;
  }
  for (int w = px0 >> 3; w <= px1 >> 3; ++w, ++row) {
    uint32_t columns = 0;
    for (int px = max(px0, 8 * w); px <= min(px1, 8 * w + 7); ++px)
      columns |= samples_in(kSampleX, px, x0, x1) << (4 * (px & 7));
    for (int py = py0; py <= py1; ++py) {
      const uint32_t m = columns & (samples_in(kSampleY, py, y0, y1) * 0x11111111u);
      if (m) atomicOr(row + (size_t)(py - py0) * row_words, m);
    }
  }
}

// 8 pixels per thread; leaves the coverage zero for the next frame.
__global__ void __launch_bounds__(256)
k_resolve(uint32_t* __restrict__ cover, uint32_t width_px, uint32_t height_px, uint32_t row_words,
          uint8_t* __restrict__ image) {
  begin_after();
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)row_words * height_px) return;
  const uint32_t mask = cover[i];
  if (mask) cover[i] = 0u;
  const uint32_t py = (uint32_t)(i / row_words), px = (uint32_t)(i % row_words) * 8u;
  uint64_t out = 0;
#pragma unroll
  for (uint32_t k = 0; k < 8; ++k)
    out |= (uint64_t)(255u * (uint32_t)__popc((mask >> (4 * k)) & 15u) / 4u) << (8 * k);
  uint8_t* dst = image + (size_t)py * width_px + px;
  if (width_px % 8 == 0) {
    *reinterpret_cast<uint64_t*>(dst) = out;
  } else {
    for (uint32_t k = 0; k < 8 && px + k < width_px; ++k) dst[k] = (uint8_t)(out >> (8 * k));
  }
}

}  // namespace

size_t render_words(uint32_t width_px, uint32_t height_px) {
  return (size_t)((width_px + 7) / 8) * height_px;
}

cudaError_t launch_render(const float2* pos, uint32_t n, float world_w, float world_h,
                          uint32_t width_px, uint32_t height_px, uint32_t* cover,
                          uint8_t* image, cudaStream_t st) {
  const uint32_t row_words = (width_px + 7) / 8;
  const float sx = (float)width_px / world_w, sy = (float)height_px / world_h;
  if (n) {
    const cudaError_t e = launch_after(k_raster, (n + 255) / 256, 256, st, pos, n, sx, sy, width_px,
                                       height_px, row_words, cover);
    if (e != cudaSuccess) return e;
  }
  return launch_after(k_resolve, (uint32_t)((render_words(width_px, height_px) + 255) / 256), 256, st,
                      cover, width_px, height_px, row_words, image);
}

}  // namespace wrach
