// The learned solver surrogate: a per-particle MLP that predicts the
// position correction of the first K-1 Jacobi iterations of the extended
// solve from the particle's k nearest neighbours.
//
//   features  knn_row: the 12 nearest taking-part particles within the 3x3
//             cells around the particle -- the candidates its Jacobi
//             iterations scan (squared distance, ties by index) -- each as
//             (dx, dy, dvx, dvy) relative to the particle, then the
//             particle's own velocity; 50 values padded to 64, BF16.
//   network   64 -> 64 -> 64 -> 2 (padded to 8), GELU (tanh form) after the
//             two hidden layers (inference evaluates it on packed FP16 pairs,
//             gelu.cuh); BF16 weights, FP32 accumulation, on the
//             tensor cores with mma.sync m16n8k16 (one warp per 16 rows; the
//             accumulator fragment of one layer is the A fragment of the
//             next, so the layers chain in registers).
//   training  k_mlp_backward recomputes the forward pass of its rows and
//             accumulates the gradients of 0.5 * mean squared error into
//             FP32 buffers; k_adam updates FP32 master weights and refreshes
//             their BF16 copies.
#include <cuda_bf16.h>
#include <stdint.h>

#include "gelu.cuh"
#include "wrach_internal.cuh"
#include "wrach_kernels.h"

namespace wrach {

namespace {

constexpr uint32_t kIn = kMlpIn, kHid = kMlpHidden, kOutPad = kMlpOutPad;

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, "
      "{%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// GELU in its tanh form, 0.5 x (1 + tanh(c (x + a x^3))), c = sqrt(2/pi),
// a = 0.044715 (Hendrycks & Gimpel, 2016), with the hardware tanh
// (tanh.approx.f32, relative error about 2^-11, below the BF16 rounding the
// activations then get).
constexpr float kGeluC = 0.7978845608028654f, kGeluA = 0.044715f;

__device__ __forceinline__ float tanh_hw(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Returns GELU(x) and turns x into the derivative there,
// 0.5 (1 + t) + 0.5 x (1 - t^2) c (1 + 3 a x^2).
__device__ __forceinline__ float gelu_and_grad(float& x) {
  const float x2 = x * x, h = 0.5f * x;
  const float t = tanh_hw(kGeluC * x * (1.0f + kGeluA * x2));
  x = 0.5f * (1.0f + t) + h * (1.0f - t * t) * kGeluC * (1.0f + 3.0f * kGeluA * x2);
  return h * (1.0f + t);
}
// GELU for the loss, to some FP32 ulps: 0.5 (1 + tanh(u)) = 1 / (1 + exp(-2 u)).
__device__ __forceinline__ float gelu_full(float x) {
  return __fdividef(x, 1.0f + __expf(-2.0f * kGeluC * x * (1.0f + kGeluA * x * x)));
}

// Shared-memory copy of the network for the forward pass: the weights as
// BF16 in the [out][in] layout (the B operand, k = in contiguous) and the
// biases in FP32.  Each row of 64 BF16 (32 words) is padded to kRow = 36
// words, so that the B-fragment loads of a warp (rows g = 0..7, words t =
// 0..3) fall in 32 distinct banks: (36 g + t) mod 32 = 4 g + t.
constexpr uint32_t kRow = kIn / 2 + 4;
static_assert(kIn == kHid, "one padded row length serves every layer");
struct alignas(16) SmemNet {
  uint32_t w1t[kHid * kRow], w2t[kHid * kRow], w3t[kOutPad * kRow];
  float b1[kHid], b2[kHid], b3[kOutPad];
};
// The [in][out] copies the backward pass multiplies the gradients by.
struct alignas(16) SmemNetT {
  uint32_t w2[kHid * kRow], w3[kHid * kOutPad / 2];
};

// 16 bytes from global to shared memory without a register between (zeros when
// not `real`); copies_wait ends the thread's own copies.
__device__ __forceinline__ void copy16(void* dst, const void* src, bool real = true) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(real ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// rows x 64 BF16 from a packed global array into padded shared rows, 16
// bytes at a time (both sides are 16-byte aligned: kRow words are 144 bytes)
__device__ __forceinline__ void load_rows(uint32_t* dst, const uint16_t* src, uint32_t rows) {
  for (uint32_t i = threadIdx.x; i < rows * (kIn / 8); i += blockDim.x)
    copy16(dst + (i / (kIn / 8)) * kRow + (i % (kIn / 8)) * 4, src + 8 * i);
}
// `words` (a multiple of 4) packed on both sides.
__device__ __forceinline__ void load_words(void* dst, const void* src, uint32_t words) {
  for (uint32_t i = threadIdx.x; i < words / 4; i += blockDim.x)
    copy16(static_cast<uint4*>(dst) + i, static_cast<const uint4*>(src) + i);
}

// The network's copies start; load_net also waits for them.
__device__ __forceinline__ void start_net(const MlpDev& m, SmemNet& s, SmemNetT* st) {
  load_rows(s.w1t, m.w1t, kHid);
  load_rows(s.w2t, m.w2t, kHid);
  load_rows(s.w3t, m.w3t, kOutPad);
  if (st) {
    load_rows(st->w2, m.w2, kHid);
    load_words(st->w3, m.w3, kHid * kOutPad / 2);
  }
  load_words(s.b1, m.b1, kHid);
  load_words(s.b2, m.b2, kHid);
  load_words(s.b3, m.b3, kOutPad);
}
__device__ __forceinline__ void load_net(const MlpDev& m, SmemNet& s) {
  start_net(m, s, nullptr);
  copies_wait();
  __syncthreads();
}

// B fragment of a weight matrix stored [n][k] in padded rows: k-tile kk,
// n-tile nt.
__device__ __forceinline__ void bfrag(const uint32_t* wt, uint32_t kk, uint32_t nt,
                                      uint32_t lane, uint32_t& b0, uint32_t& b1) {
  const uint32_t g = lane >> 2, t = lane & 3;
  const uint32_t row = (nt * 8 + g) * kRow;
  b0 = wt[row + kk * 8 + t];
  b1 = wt[row + kk * 8 + 4 + t];
}

// Forward pass of one 16-row tile held by a warp, for training.  `ax` is the A
// fragment of the input (4 k-tiles).  Writes the A fragments h1, h2 of the
// activations, the GELU's derivatives z1, z2 at the pre-activations (C
// layout, 8 n-tiles) and the output y (one n-tile).
//
// LOSS: the outputs for the loss, yl, by activations of their own from the same
// weight fragments.  An activation that is rounded to the other BF16 neighbour
// shifts the loss, and the hardware tanh (and, less, sums that the tensor cores
// round towards zero along a chain) does that to many: here each product of 16
// inputs starts from zero, the four are added to nearest and the GELU is
// gelu_full.  Root mean square error of the loss against 64 bits over 50 batches
// of 1,000 and 16,384 and 20 of 65,536 rows, as the gradients' activations have
// it 9.7e-6, 2.4e-6 and 1.5e-6, this way 1.0e-6, 4.7e-7 and 2.9e-7; the batches'
// times 27.1, 33.5 and 45.8 us without, 29.3, 35.2 and 52.7 with it, so that it is
// done only for a loss that is read.  (A pass of its own: 29.5, 35.2 and 54.5;
// with exact sums of the four and an FP32-exact GELU 9.9e-7, 3.6e-7 and 2.2e-7
// in 34.5, 40.0 and 74.3 us.)
template <bool LOSS>
__device__ __forceinline__ void hidden_layer(const uint32_t* wt, const float* b, uint32_t lane,
                                             const uint32_t (&in)[4][4],
                                             const uint32_t (&inl)[4][4], float (&z)[8][4],
                                             uint32_t (&h)[4][4], uint32_t (&hl)[4][4]) {
  const uint32_t t = lane & 3;
#pragma unroll
  for (uint32_t nt = 0; nt < 8; ++nt) {
    const float bl = b[nt * 8 + 2 * t], bh = b[nt * 8 + 2 * t + 1];
    z[nt][0] = bl; z[nt][1] = bh; z[nt][2] = bl; z[nt][3] = bh;
    float p[4][4] = {};
#pragma unroll
    for (uint32_t kk = 0; kk < 4; ++kk) {
      uint32_t b0, b1;
      bfrag(wt, kk, nt, lane, b0, b1);
      mma_bf16(z[nt], in[kk], b0, b1);
      if (LOSS) mma_bf16(p[kk], inl[kk], b0, b1);
    }
    if (LOSS) {
      float g[4];
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q)
        g[q] = gelu_full((p[0][q] + p[1][q]) + (p[2][q] + p[3][q]) + (q & 1 ? bh : bl));
      hl[nt / 2][2 * (nt & 1)] = pack_bf16(g[0], g[1]);
      hl[nt / 2][2 * (nt & 1) + 1] = pack_bf16(g[2], g[3]);
    }
  }
#pragma unroll
  for (uint32_t nt = 0; nt < 8; ++nt) {
    const float g0 = gelu_and_grad(z[nt][0]), g1 = gelu_and_grad(z[nt][1]);
    const float g2 = gelu_and_grad(z[nt][2]), g3 = gelu_and_grad(z[nt][3]);
    h[nt / 2][2 * (nt & 1)] = pack_bf16(g0, g1);
    h[nt / 2][2 * (nt & 1) + 1] = pack_bf16(g2, g3);
  }
}
template <bool LOSS>
__device__ __forceinline__ void mlp_tile_forward(const SmemNet& s, uint32_t lane,
                                                 const uint32_t (&ax)[4][4],
                                                 float (&z1)[8][4], uint32_t (&h1)[4][4],
                                                 float (&z2)[8][4], uint32_t (&h2)[4][4],
                                                 float (&y)[4], float (&yl)[4]) {
  const uint32_t t = lane & 3;
  uint32_t l1[4][4], l2[4][4];
  hidden_layer<LOSS>(s.w1t, s.b1, lane, ax, ax, z1, h1, l1);
  hidden_layer<LOSS>(s.w2t, s.b2, lane, h1, l1, z2, h2, l2);
  const float bl = s.b3[2 * t], bh = s.b3[2 * t + 1];
  y[0] = bl; y[1] = bh; y[2] = bl; y[3] = bh;
  float p[4][4] = {};
#pragma unroll
  for (uint32_t kk = 0; kk < 4; ++kk) {
    uint32_t b0, b1;
    bfrag(s.w3t, kk, 0, lane, b0, b1);
    mma_bf16(y, h2[kk], b0, b1);
    if (LOSS) mma_bf16(p[kk], l2[kk], b0, b1);
  }
  if (LOSS) {
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q)
      yl[q] = (p[0][q] + p[1][q]) + (p[2][q] + p[3][q]) + (q & 1 ? bh : bl);
  }
}

// A shared-memory word read that the compiler keeps in place (it would
// otherwise hoist the loop-invariant weight fragments of a persistent loop
// into registers and lose occupancy).
__device__ __forceinline__ uint32_t lds_keep(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];"
               : "=r"(v)
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
  return v;
}

// The forward pass of TILES 16-row tiles for inference only: the same products
// in the same order as mlp_tile_forward, computed two n-tiles at a time so
// that no pre-activation array stays live, with the GELU on packed FP16 pairs
// (gelu2_bf16; the training pass keeps the FP32 GELU and its derivative).
// Each weight fragment read from shared memory serves all TILES tiles: with
// one tile the 17 KB of fragments per 16 rows bound the kernels by shared
// memory's bandwidth.
template <uint32_t TILES>
__device__ __forceinline__ void infer_layer(const uint32_t* wt, const float* b, uint32_t lane,
                                            const uint32_t (&in)[TILES][4][4],
                                            uint32_t (&out)[TILES][4][4]) {
  const uint32_t g = lane >> 2, t = lane & 3;
#pragma unroll
  for (uint32_t kq = 0; kq < 4; ++kq) {
    float z[TILES][2][4];
#pragma unroll
    for (uint32_t u = 0; u < 2; ++u) {
      const uint32_t nt = 2 * kq + u;
      const float bl = b[nt * 8 + 2 * t], bh = b[nt * 8 + 2 * t + 1];
#pragma unroll
      for (uint32_t r = 0; r < TILES; ++r) {
        z[r][u][0] = bl; z[r][u][1] = bh; z[r][u][2] = bl; z[r][u][3] = bh;
      }
      const uint32_t* row = wt + (nt * 8 + g) * kRow + t;
#pragma unroll
      for (uint32_t kk = 0; kk < 4; ++kk) {
        const uint32_t b0 = lds_keep(row + kk * 8), b1 = lds_keep(row + kk * 8 + 4);
#pragma unroll
        for (uint32_t r = 0; r < TILES; ++r) mma_bf16(z[r][u], in[r][kk], b0, b1);
      }
    }
#pragma unroll
    for (uint32_t r = 0; r < TILES; ++r) {
      out[r][kq][0] = gelu2_bf16(z[r][0][0], z[r][0][1]);
      out[r][kq][1] = gelu2_bf16(z[r][0][2], z[r][0][3]);
      out[r][kq][2] = gelu2_bf16(z[r][1][0], z[r][1][1]);
      out[r][kq][3] = gelu2_bf16(z[r][1][2], z[r][1][3]);
    }
  }
}

template <uint32_t TILES>
__device__ __forceinline__ void mlp_infer(const SmemNet& s, uint32_t lane,
                                          const uint32_t (&ax)[TILES][4][4],
                                          float (&y)[TILES][4]) {
  const uint32_t g = lane >> 2, t = lane & 3;
  uint32_t h1[TILES][4][4], h2[TILES][4][4];
  infer_layer<TILES>(s.w1t, s.b1, lane, ax, h1);
  infer_layer<TILES>(s.w2t, s.b2, lane, h1, h2);
  const float bl = s.b3[2 * t], bh = s.b3[2 * t + 1];
#pragma unroll
  for (uint32_t r = 0; r < TILES; ++r) {
    y[r][0] = bl; y[r][1] = bh; y[r][2] = bl; y[r][3] = bh;
  }
  const uint32_t* row = s.w3t + g * kRow + t;
#pragma unroll
  for (uint32_t kk = 0; kk < 4; ++kk) {
    const uint32_t b0 = lds_keep(row + kk * 8), b1 = lds_keep(row + kk * 8 + 4);
#pragma unroll
    for (uint32_t r = 0; r < TILES; ++r) mma_bf16(y[r], h2[r][kk], b0, b1);
  }
}

// A fragment (4 k-tiles) of 16 rows of X (BF16 [rows][64]); rows past n read
// as zero.
__device__ __forceinline__ void load_x_tile(const uint16_t* x, uint32_t row0, uint32_t n,
                                            uint32_t lane, uint32_t (&ax)[4][4]) {
  const uint32_t g = lane >> 2, t = lane & 3;
  const uint32_t r0 = row0 + g, r1 = row0 + g + 8;
  const uint32_t* p0 = reinterpret_cast<const uint32_t*>(x + (size_t)r0 * kIn);
  const uint32_t* p1 = reinterpret_cast<const uint32_t*>(x + (size_t)r1 * kIn);
#pragma unroll
  for (uint32_t kk = 0; kk < 4; ++kk) {
    ax[kk][0] = r0 < n ? p0[kk * 8 + t] : 0u;
    ax[kk][1] = r1 < n ? p1[kk * 8 + t] : 0u;
    ax[kk][2] = r0 < n ? p0[kk * 8 + 4 + t] : 0u;
    ax[kk][3] = r1 < n ? p1[kk * 8 + 4 + t] : 0u;
  }
}

__global__ void __launch_bounds__(128) k_mlp_forward(MlpDev m, const uint16_t* __restrict__ x,
                                                     uint32_t n, float2* __restrict__ y) {
  __shared__ SmemNet s;
  load_net(m, s);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t g = lane >> 2, t = lane & 3;
  constexpr uint32_t kTiles = 2;
  const uint32_t groups = (n + 16 * kTiles - 1) / (16 * kTiles);
  for (uint32_t group = blockIdx.x * 4 + warp; group < groups; group += gridDim.x * 4) {
    uint32_t ax[kTiles][4][4];
    float out[kTiles][4];
#pragma unroll
    for (uint32_t r = 0; r < kTiles; ++r)
      load_x_tile(x, (group * kTiles + r) * 16, n, lane, ax[r]);
    mlp_infer<kTiles>(s, lane, ax, out);
    if (t == 0) {
#pragma unroll
      for (uint32_t r = 0; r < kTiles; ++r) {
        const uint32_t r0 = (group * kTiles + r) * 16 + g, r1 = r0 + 8;
        if (r0 < n) y[r0] = make_float2(out[r][0], out[r][1]);
        if (r1 < n) y[r1] = make_float2(out[r][2], out[r][3]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Training
// ---------------------------------------------------------------------------

// A block of 8 warps takes tiles of 128 rows.  First each warp runs 16 of the
// rows forward and backward and leaves their activations and gradients in
// shared memory as BF16, [row][feature] in padded rows.  Then the warps share
// out the weight gradients X^T dZ1, H1^T dZ2 and H2^T dY, contractions over
// the tile's rows: warp w owns input features 16 (w mod 4) .. + 15 and one
// half of the outputs of each product, and adds them to sums in its registers
// over all of the block's tiles (the transposed operands come from
// ldmatrix.trans).  What it waits for is latency (of the weights' loads, the
// two layers and the final sums into global memory): 16,384 rows are 128
// blocks of one tile.  Before, each warp added every 16-row product into
// shared memory with atomics, 272 of them a tile, and 4 warps filled an SM's
// shared memory: 61 us then, 15 us now, 17 with the loss (16,384 rows).
constexpr uint32_t kTrainRows = 128, kTrainThreads = 256;

struct SmemTile {
  uint32_t x[kTrainRows * kRow], h1[kTrainRows * kRow], h2[kTrainRows * kRow];
  uint32_t dz1[kTrainRows * kRow], dz2[kTrainRows * kRow];
  uint32_t dy[kTrainRows * kOutPad / 2];
};
struct SmemTrain {
  SmemNet net;
  SmemNetT t;
  SmemTile tile;
};
static_assert(sizeof(SmemNet) % 16 == 0 && sizeof(SmemNetT) % 16 == 0, "16-byte rows");

// Four (two) 8x8 BF16 matrices from shared memory; lane l gives the address of
// row l mod 8 of matrix l / 8.
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm2t(uint32_t& r0, uint32_t& r1, const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(r0), "=r"(r1)
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

// A fragments of 16 rows (4 k-tiles) into padded rows, row0 the first.
__device__ __forceinline__ void store_a(uint32_t* dst, uint32_t row0, uint32_t lane,
                                        const uint32_t (&a)[4][4]) {
  const uint32_t g = lane >> 2, t = lane & 3;
  uint32_t* p0 = dst + (row0 + g) * kRow + t;
  uint32_t* p1 = p0 + 8 * kRow;
#pragma unroll
  for (uint32_t kk = 0; kk < 4; ++kk) {
    p0[kk * 8] = a[kk][0];
    p1[kk * 8] = a[kk][1];
    p0[kk * 8 + 4] = a[kk][2];
    p1[kk * 8 + 4] = a[kk][3];
  }
}

// A C-layout tile (8 n-tiles of 16x8) as the A fragment of the next product.
__device__ __forceinline__ void to_a(uint32_t (&a)[4][4], const float (&c)[8][4]) {
#pragma unroll
  for (uint32_t kk = 0; kk < 4; ++kk) {
    a[kk][0] = pack_bf16(c[2 * kk][0], c[2 * kk][1]);
    a[kk][1] = pack_bf16(c[2 * kk][2], c[2 * kk][3]);
    a[kk][2] = pack_bf16(c[2 * kk + 1][0], c[2 * kk + 1][1]);
    a[kk][3] = pack_bf16(c[2 * kk + 1][2], c[2 * kk + 1][3]);
  }
}

// sum (4 n-tiles from column n0) += AT^T BT over the tile's rows, AT the
// columns m0 .. m0 + 15 of `at`.  The product of a tile's 128 rows starts from
// zero and is added to nearest: sums that stayed in the tensor cores'
// accumulators over all of a block's tiles were rounded towards zero at every
// 16 rows (2M rows, 108 tiles a block: 1.5e-5 of the gradients' norm, 2.2e-7 now).
__device__ __forceinline__ void rows_product(float (&sum)[4][4], const uint32_t* at,
                                             const uint32_t* bt, uint32_t m0, uint32_t n0,
                                             uint32_t lane) {
  const uint32_t mi = lane >> 3, r = lane & 7;
  // A: matrices (k 0-7, m 0-7), (k 0-7, m 8-15), (k 8-15, m 0-7), (k 8-15, m 8-15)
  const uint32_t* pa = at + ((mi >> 1) * 8 + r) * kRow + (m0 + (mi & 1) * 8) / 2;
  // B: matrices (k 0-7, n 0-7), (k 8-15, n 0-7), (k 0-7, n 8-15), (k 8-15, n 8-15)
  const uint32_t* pb = bt + ((mi & 1) * 8 + r) * kRow + (n0 + (mi >> 1) * 8) / 2;
  float acc[4][4] = {};
#pragma unroll
  for (uint32_t ks = 0; ks < kTrainRows / 16; ++ks) {
    uint32_t a[4], b[4], c[4];
    ldsm4t(a, pa + ks * 16 * kRow);
    ldsm4t(b, pb + ks * 16 * kRow);
    ldsm4t(c, pb + ks * 16 * kRow + 8);
    mma_bf16(acc[0], a, b[0], b[1]);
    mma_bf16(acc[1], a, b[2], b[3]);
    mma_bf16(acc[2], a, c[0], c[1]);
    mma_bf16(acc[3], a, c[2], c[3]);
  }
#pragma unroll
  for (uint32_t u = 0; u < 4; ++u)
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) sum[u][q] += acc[u][q];
}

// A 16x8 tile of sums (C layout) into the row-major matrix w of `ld` columns.
__device__ __forceinline__ void add_tile(float* w, uint32_t ld, uint32_t m0, uint32_t n0,
                                         const float (&c)[4], uint32_t lane) {
  const uint32_t g = lane >> 2, t = lane & 3;
  float* p = w + (m0 + g) * ld + n0 + 2 * t;
  atomicAdd(reinterpret_cast<float2*>(p), make_float2(c[0], c[1]));
  atomicAdd(reinterpret_cast<float2*>(p + 8 * ld), make_float2(c[2], c[3]));
}

// The loss, a 64-bit sum behind the gradients: with 32 bits it turned with the
// order of the warps' shares by up to 2e-6 of itself.
__device__ __forceinline__ double* loss_of(float* grad) {
  return reinterpret_cast<double*>(grad + kMlpParams);
}
static_assert(kMlpParams % 2 == 0, "the loss is 8-byte aligned");
__device__ __forceinline__ double half_square(float e0, float e1) {
  return 0.5 * ((double)e0 * e0 + (double)e1 * e1);
}

// Gradients of L = 0.5 * sum over rows and the 2 outputs of (y - target)^2 /
// `scale_rows` with respect to every parameter, added into `grad` (FP32,
// the MlpDev parameter order: w1 [in][out], b1, w2, b2, w3 [in][8], b3).
// LOSS: also adds the loss into the 64-bit sum behind them.
template <bool LOSS>
__global__ void __launch_bounds__(kTrainThreads, 1)
k_mlp_backward(MlpDev m, const uint16_t* __restrict__ x, const float2* __restrict__ target,
               uint32_t n, float inv_rows, float* __restrict__ grad) {
  extern __shared__ __align__(16) uint8_t dyn[];
  begin_after();
  SmemTrain& sm = *reinterpret_cast<SmemTrain*>(dyn);
  SmemTile& st = sm.tile;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t g = lane >> 2, t = lane & 3;
  const uint32_t row0 = warp * 16, m0 = (warp & 3) * 16, n0 = (warp >> 2) * 32;
  float sum1[4][4] = {}, sum2[4][4] = {}, sum3[4] = {};
  float sb1[8][2] = {}, sb2[8][2] = {}, sb3[2] = {};
  double lsum = 0.0;
  const uint32_t tiles = (n + kTrainRows - 1) / kTrainRows;
  // a caller's rows may start at any 4-byte boundary
  const bool x16 = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    // the tile's features (rows past n are zero) and, with the first, the
    // network: all copies are in flight together (16,384 rows' gradients 34.2
    // us with each array's loads ahead of its stores, 32.7 now; 1,000 rows 28.0
    // and 26.3)
    const uint32_t base = tile * kTrainRows;
#pragma unroll
    for (uint32_t i = threadIdx.x; i < kTrainRows * (kIn / 8); i += kTrainThreads) {
      const uint32_t r = i / (kIn / 8), c = i % (kIn / 8);
      const bool real = base + r < n;
      const uint16_t* p = x + (real ? (size_t)(base + r) * kIn + c * 8 : 0);
      uint32_t* to = st.x + r * kRow + c * 4;
      if (x16) {
        copy16(to, p, real);
      } else {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
        *reinterpret_cast<uint4*>(to) =
            real ? make_uint4(w[0], w[1], w[2], w[3]) : make_uint4(0, 0, 0, 0);
      }
    }
    if (tile == blockIdx.x) start_net(m, sm.net, &sm.t);
    const uint32_t r0 = base + row0 + g, r1 = r0 + 8;
    float2 tg0 = make_float2(0.f, 0.f), tg1 = tg0;
    if (t == 0 && r0 < n) tg0 = target[r0];
    if (t == 0 && r1 < n) tg1 = target[r1];
    copies_wait();
    __syncthreads();

    uint32_t a[4][4], h1[4][4], h2[4][4];
    float z1[8][4], z2[8][4], y[4];
#pragma unroll
    for (uint32_t kk = 0; kk < 4; ++kk)
      ldsm4(a[kk], st.x + (row0 + (lane & 15)) * kRow + kk * 8 + (lane >> 4) * 4);
    float yl[4];
    mlp_tile_forward<LOSS>(sm.net, lane, a, z1, h1, z2, h2, y, yl);
    if (LOSS && t == 0) {
      if (r0 < n) lsum += half_square(yl[0] - tg0.x, yl[1] - tg0.y);
      if (r1 < n) lsum += half_square(yl[2] - tg1.x, yl[3] - tg1.y);
    }
    store_a(st.h1, row0, lane, h1);
    store_a(st.h2, row0, lane, h2);
    // dY (C layout, one n-tile; only columns 0 and 1 are real outputs)
    float dy[4] = {0.f, 0.f, 0.f, 0.f};
    if (t == 0) {
      if (r0 < n) {
        const float e0 = y[0] - tg0.x, e1 = y[1] - tg0.y;
        dy[0] = e0 * inv_rows;
        dy[1] = e1 * inv_rows;
      }
      if (r1 < n) {
        const float e0 = y[2] - tg1.x, e1 = y[3] - tg1.y;
        dy[2] = e0 * inv_rows;
        dy[3] = e1 * inv_rows;
      }
    }
    sb3[0] += dy[0] + dy[2];
    sb3[1] += dy[1] + dy[3];
    // dH2 = dY W3^T  (K = 8 outputs padded to 16 with zeros)
    const uint32_t ady[4] = {pack_bf16(dy[0], dy[1]), pack_bf16(dy[2], dy[3]), 0u, 0u};
    st.dy[(row0 + g) * (kOutPad / 2) + t] = ady[0];
    st.dy[(row0 + g + 8) * (kOutPad / 2) + t] = ady[1];
#pragma unroll
    for (uint32_t nt = 0; nt < 8; ++nt) {
      float d[4] = {0.f, 0.f, 0.f, 0.f};
      // B(k = out, n = in) = W3[in][out]; W3 stored [in][8]
      mma_bf16(d, ady, sm.t.w3[(nt * 8 + g) * (kOutPad / 2) + t], 0u);
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) z2[nt][q] = d[q] * z2[nt][q];
      sb2[nt][0] += z2[nt][0] + z2[nt][2];
      sb2[nt][1] += z2[nt][1] + z2[nt][3];
    }
    // dH1 = dZ2 W2^T
    to_a(a, z2);
    store_a(st.dz2, row0, lane, a);
#pragma unroll
    for (uint32_t nt = 0; nt < 8; ++nt) {
      float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (uint32_t kk = 0; kk < 4; ++kk) {
        uint32_t b0, b1;
        bfrag(sm.t.w2, kk, nt, lane, b0, b1);  // W2 [in][out]: B(k=out, n=in)
        mma_bf16(d, a[kk], b0, b1);
      }
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) z1[nt][q] = d[q] * z1[nt][q];
      sb1[nt][0] += z1[nt][0] + z1[nt][2];
      sb1[nt][1] += z1[nt][1] + z1[nt][3];
    }
    to_a(a, z1);
    store_a(st.dz1, row0, lane, a);
    __syncthreads();
    // the weight gradients' products over the tile's rows
    rows_product(sum1, st.x, st.dz1, m0, n0, lane);
    rows_product(sum2, st.h1, st.dz2, m0, n0, lane);
    if (n0 == 0) {
      const uint32_t mi = lane >> 3, r = lane & 7;
      float acc[4] = {};
#pragma unroll
      for (uint32_t ks = 0; ks < kTrainRows / 16; ++ks) {
        uint32_t b[4], b0, b1;
        ldsm4t(b, st.h2 + (ks * 16 + (mi >> 1) * 8 + r) * kRow + (m0 + (mi & 1) * 8) / 2);
        ldsm2t(b0, b1, st.dy + (ks * 16 + (mi & 1) * 8 + r) * (kOutPad / 2));
        mma_bf16(acc, b, b0, b1);
      }
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) sum3[q] += acc[q];
    }
    __syncthreads();
  }
  // the block's sums into global memory
  const uint32_t o_b1 = kIn * kHid, o_w2 = o_b1 + kHid, o_b2 = o_w2 + kHid * kHid;
  const uint32_t o_w3 = o_b2 + kHid, o_b3 = o_w3 + kHid * kOutPad;
#pragma unroll
  for (uint32_t u = 0; u < 4; ++u) {
    add_tile(grad, kHid, m0, n0 + u * 8, sum1[u], lane);
    add_tile(grad + o_w2, kHid, m0, n0 + u * 8, sum2[u], lane);
  }
  if (n0 == 0) add_tile(grad + o_w3, kOutPad, m0, 0, sum3, lane);
  // bias gradients: the columns' sums over the rows a warp's lanes hold
#pragma unroll
  for (uint32_t o = 4; o < 32; o <<= 1) {
#pragma unroll
    for (uint32_t nt = 0; nt < 8; ++nt)
#pragma unroll
      for (uint32_t u = 0; u < 2; ++u) {
        sb1[nt][u] += __shfl_xor_sync(0xffffffffu, sb1[nt][u], o);
        sb2[nt][u] += __shfl_xor_sync(0xffffffffu, sb2[nt][u], o);
      }
#pragma unroll
    for (uint32_t u = 0; u < 2; ++u) sb3[u] += __shfl_xor_sync(0xffffffffu, sb3[u], o);
    if (LOSS) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  }
  if (g == 0) {
#pragma unroll
    for (uint32_t nt = 0; nt < 8; ++nt) {
      atomicAdd(reinterpret_cast<float2*>(grad + o_b1 + nt * 8 + 2 * t),
                make_float2(sb1[nt][0], sb1[nt][1]));
      atomicAdd(reinterpret_cast<float2*>(grad + o_b2 + nt * 8 + 2 * t),
                make_float2(sb2[nt][0], sb2[nt][1]));
    }
  }
  if (lane == 0) {
    atomicAdd(reinterpret_cast<float2*>(grad + o_b3), make_float2(sb3[0], sb3[1]));
    if (LOSS) atomicAdd(loss_of(grad), lsum * (double)inv_rows);
  }
}

// A batch's sums end with the launch that reads them: it leaves zeros for the
// next batch's, so that no clear stands between two batches (16,384 rows, with
// a copy to the host and its gap replaced by k_take_gradients: 44 -> 34 us).
// Behind the gradients lie the loss and the last batch's loss, which stays.
__device__ __forceinline__ float take_sum(float* grad, uint32_t i, uint32_t nparams) {
  if (i == nparams) {
    const float loss = (float)*loss_of(grad);
    *loss_of(grad) = 0.0;
    grad[nparams + 2] = loss;
    return loss;
  }
  const float g = grad[i];
  grad[i] = 0.f;
  return g;
}

// The gradients and the loss to pinned host memory.
__global__ void __launch_bounds__(256) k_take_gradients(float* __restrict__ grad,
                                                        float* __restrict__ out,
                                                        uint32_t nparams) {
  begin_after();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i <= nparams) out[i] = take_sum(grad, i, nparams);
}

// Adam on the FP32 master parameters (the order above), then the BF16
// copies in both layouts.
__global__ void k_adam(MlpDev m, float* __restrict__ grad, float* __restrict__ mom1,
                       float* __restrict__ mom2, float lr, float b1, float b2, float eps,
                       float bc1, float bc2, uint32_t nparams) {
  begin_after();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > nparams) return;
  const float gr = take_sum(grad, i, nparams);
  if (i == nparams) return;
  const float a = b1 * mom1[i] + (1.f - b1) * gr;
  const float b = b2 * mom2[i] + (1.f - b2) * gr * gr;
  mom1[i] = a;
  mom2[i] = b;
  const float step = lr * (a / bc1) / (sqrtf(b / bc2) + eps);
  float* p = m.params;
  const float v = p[i] - step;
  p[i] = v;
  const __nv_bfloat16 h = __float2bfloat16_rn(v);
  // parameter order: w1 [in][hid], b1, w2 [hid][hid], b2, w3 [hid][8], b3
  const uint32_t o_b1 = kIn * kHid, o_w2 = o_b1 + kHid, o_b2 = o_w2 + kHid * kHid;
  const uint32_t o_w3 = o_b2 + kHid, o_b3 = o_w3 + kHid * kOutPad;
  __nv_bfloat16* w1 = reinterpret_cast<__nv_bfloat16*>(m.w1);
  __nv_bfloat16* w1t = reinterpret_cast<__nv_bfloat16*>(m.w1t);
  __nv_bfloat16* w2 = reinterpret_cast<__nv_bfloat16*>(m.w2);
  __nv_bfloat16* w2t = reinterpret_cast<__nv_bfloat16*>(m.w2t);
  __nv_bfloat16* w3 = reinterpret_cast<__nv_bfloat16*>(m.w3);
  __nv_bfloat16* w3t = reinterpret_cast<__nv_bfloat16*>(m.w3t);
  if (i < o_b1) {
    const uint32_t r = i / kHid, c = i % kHid;  // in, out
    w1[i] = h;
    w1t[c * kIn + r] = h;
  } else if (i < o_w2) {
    m.b1[i - o_b1] = v;
  } else if (i < o_b2) {
    const uint32_t j = i - o_w2, r = j / kHid, c = j % kHid;
    w2[j] = h;
    w2t[c * kHid + r] = h;
  } else if (i < o_w3) {
    m.b2[i - o_b2] = v;
  } else if (i < o_b3) {
    const uint32_t j = i - o_w3, r = j / kOutPad, c = j % kOutPad;
    w3[j] = h;
    w3t[c * kHid + r] = h;
  } else {
    m.b3[i - o_b3] = v;
  }
}

// ---------------------------------------------------------------------------
// Features
// ---------------------------------------------------------------------------

constexpr uint32_t kK = kKnn, kBatch = 4;
static_assert(kK % kBatch == 0, "whole batches");

// 32 words of a feature row, from registers: 16 bytes at a time into shared
// memory, where 8 lanes' rows (144 bytes apart) then cover all banks, and 4
// into a caller's global buffer, which may start anywhere.
template <bool SHARED>
__device__ __forceinline__ void set_row(uint32_t* row, const uint32_t (&w)[kIn / 2]) {
  if (SHARED) {
#pragma unroll
    for (uint32_t k = 0; k < kIn / 8; ++k)
      reinterpret_cast<uint4*>(row)[k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
  } else {
#pragma unroll
    for (uint32_t k = 0; k < kIn / 2; ++k) row[k] = w[k];
  }
}

template <bool SHARED>
__device__ __forceinline__ void zero_row(uint32_t* row) {
  const uint32_t w[kIn / 2] = {};
  set_row<SHARED>(row, w);
}

// Features of the taking-part particle of compacted index t (cell c) into
// `row` (32 words): the 12 nearest taking-part particles in the 3x3 cells
// around its cell -- the candidates of its Jacobi iterations, one contiguous
// compacted range per neighbour row -- by binary32 squared distance (each
// product and sum rounded on its own), ties by index; each as (dx, dy, dvx,
// dvy) relative to the particle; then the own velocity; zero padding to 64.
// A candidate at a NaN or infinite distance is left out.  Positions and
// velocities are the frame's binned state, compacted (tpp, tpv).
//
// With at most 12 candidates (sparse frames: 4.2 of them on average) all are
// listed, and each one's place is the number of nearer ones, counted pair by
// pair; more are inserted into an ascending list, which moves 12 entries per
// candidate.
template <bool SHARED>
__device__ __forceinline__ void knn_row(const WorldDev& w, const CellTable& table,
                                        const float2* __restrict__ tpp,
                                        const float2* __restrict__ tpv, uint32_t c, uint32_t t,
                                        uint32_t* row) {
  uint32_t rs[3], re[3];
  neighbour_rows(w, table, c, rs, re);
  const float2 pi = tpp[t], vi = tpv[t];
  uint32_t out[kIn / 2] = {};
  out[2 * kK] = pack_bf16(vi.x, vi.y);
  const uint32_t b0 = re[0] - rs[0], b1 = b0 + t - rs[1], b2 = b0 + re[1] - rs[1] - 1u;
  const uint32_t others = b2 + re[2] - rs[2];
  if (others <= kK) {
    // candidate m is t's m-th in index order: first row, middle row before
    // and after t, last row
    const uint32_t o0 = rs[0], o1 = rs[1] - b0, o2 = o1 + 1u, o3 = rs[2] - b2;
    set_row<SHARED>(row, out);
    float d[kK];
    uint32_t place[kK], dp[kK], dv[kK];
#pragma unroll
    for (uint32_t m0 = 0; m0 < kK; m0 += kBatch) {
      // a batch's loads go out together (past the last candidate: t itself)
      float2 p[kBatch], v[kBatch];
      if (m0 < others) {
#pragma unroll
        for (uint32_t u = 0; u < kBatch; ++u) {
          const uint32_t m = m0 + u;
          const uint32_t j = m < others ? m + (m < b0 ? o0 : m < b1 ? o1 : m < b2 ? o2 : o3) : t;
          p[u] = tpp[j];
          v[u] = tpv[j];
        }
      }
#pragma unroll
      for (uint32_t u = 0; u < kBatch; ++u) {
        const uint32_t m = m0 + u;
        d[m] = INFINITY;
        place[m] = 0u;
        if (m0 < others) {
          const float dx = __fsub_rn(p[u].x, pi.x), dy = __fsub_rn(p[u].y, pi.y);
          const float s = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
          dp[m] = pack_bf16(dx, dy);
          dv[m] = pack_bf16(__fsub_rn(v[u].x, vi.x), __fsub_rn(v[u].y, vi.y));
          if (m < others && s < INFINITY) d[m] = s;
          // a tie keeps the earlier one nearer
#pragma unroll
          for (uint32_t k = 0; k < m; ++k) {
            if (d[m] < d[k]) ++place[k];
            else ++place[m];
          }
        }
      }
    }
#pragma unroll
    for (uint32_t m = 0; m < kK; ++m)
      if (d[m] < INFINITY) {
        row[2 * place[m]] = dp[m];
        row[2 * place[m] + 1] = dv[m];
      }
    return;
  }
  float bd[kK];
  uint32_t bj[kK];
#pragma unroll
  for (uint32_t k = 0; k < kK; ++k) {
    bd[k] = INFINITY;
    bj[k] = 0xFFFFFFFFu;
  }
  // the candidates come in ascending index order (rows bottom-up, compacted
  // order inside a row), so a tie in distance keeps the one already listed;
  // each is inserted into the ascending list: every comparison against the
  // old list first, then the shift
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    for (uint32_t j = rs[r]; j < re[r]; ++j) {
      if (j == t) continue;
      const float2 pj = tpp[j];
      const float dx = __fsub_rn(pj.x, pi.x), dy = __fsub_rn(pj.y, pi.y);
      const float d = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
      if (!(d < bd[kK - 1])) continue;
      bool lt[kK];
#pragma unroll
      for (uint32_t k = 0; k < kK; ++k) lt[k] = d < bd[k];
#pragma unroll
      for (uint32_t k = kK - 1; k > 0; --k) {
        bd[k] = lt[k - 1] ? bd[k - 1] : (lt[k] ? d : bd[k]);
        bj[k] = lt[k - 1] ? bj[k - 1] : (lt[k] ? j : bj[k]);
      }
      bd[0] = lt[0] ? d : bd[0];
      bj[0] = lt[0] ? j : bj[0];
    }
  }
#pragma unroll
  for (uint32_t k = 0; k < kK; ++k) {
    if (bj[k] != 0xFFFFFFFFu) {
      const float2 pj = tpp[bj[k]], vj = tpv[bj[k]];
      out[2 * k] = pack_bf16(__fsub_rn(pj.x, pi.x), __fsub_rn(pj.y, pi.y));
      out[2 * k + 1] = pack_bf16(__fsub_rn(vj.x, vi.x), __fsub_rn(vj.y, vi.y));
    }
  }
  set_row<SHARED>(row, out);
}

__global__ void k_compact_velocities(uint32_t n, const uint32_t* __restrict__ tp_of,
                                     const float2* __restrict__ vel,
                                     float2* __restrict__ tp_vel) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && tp_of[i] != kNoTp) tp_vel[tp_of[i]] = vel[i];
}

// Features of the binned frame into x (BF16 [n][64]), one thread per frame
// particle; a particle that does not take part (past the capacity of its
// cell) gets all zeros.
__global__ void __launch_bounds__(256)
k_knn_features(const WorldDev* __restrict__ worlds, int nworlds, uint32_t n,
               const uint32_t* __restrict__ tp_of, const CellTable table,
               const uint32_t* __restrict__ cell_of, const float2* __restrict__ tpp,
               const float2* __restrict__ tpv, uint16_t* __restrict__ x) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t* row = reinterpret_cast<uint32_t*>(x + (size_t)i * kIn);
  const uint32_t c = cell_of[i];
  const uint32_t t = tp_of[i];
  if (t == kNoTp) {
    zero_row<false>(row);
    return;
  }
  knn_row<false>(worlds[world_of_cell(worlds, nworlds, c)], table, tpp, tpv, c, t, row);
}

// Training samples of the binned frame: the features of the taking-part
// particles t = phase + k * stride, k = 0, 1, ..., into rows k of x (at most
// `rows`), and their targets q_t - p_t from the compacted iterate q (the
// plain solver's first iterations) into target.
__global__ void __launch_bounds__(256)
k_samples(const WorldDev* __restrict__ worlds, int nworlds, uint32_t ncells,
          const CellTable table, const uint32_t* __restrict__ tp_cell,
          const float2* __restrict__ tpp, const float2* __restrict__ tpv,
          const float2* __restrict__ q, uint32_t stride, uint32_t phase, uint32_t rows,
          uint16_t* __restrict__ x, float2* __restrict__ target) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t t = phase + k * stride;
  if (k >= rows || t >= table.taking(ncells)) return;
  const uint32_t c = tp_cell[t];
  knn_row<false>(worlds[world_of_cell(worlds, nworlds, c)], table, tpp, tpv, c, t,
                 reinterpret_cast<uint32_t*>(x + (size_t)k * kIn));
  const float2 p = tpp[t], v = q[t];
  target[k] = make_float2(v.x - p.x, v.y - p.y);
}

// The surrogate correction of a frame in one pass over its taking-part
// particles (compacted): per tile of 256 of them, the features go to shared
// memory (padded rows, so the A-fragment loads are conflict-free like the
// weights'), each warp runs the network on 32 of the rows, and the
// correction is applied on the spot: the compacted iterate q_t = p_t +
// correction.  `corr` (optional) receives the correction at the frame index
// of each taking-part particle.  Persistent: the network is loaded once per
// block, and a warp waits for none of the others afterwards (its rows are its
// own lanes').  1M lattice: 130 us with one 16-row tile at a time, 4-byte row
// stores (8 lanes to a bank) and every candidate inserted, 95 us now; it
// issues 57% of the time and waits for the candidates' loads and the products
// for the rest, with 4 warps a scheduler (128 registers; 3 blocks an SM spill:
// 118).
constexpr uint32_t kFuseThreads = 256;

__global__ void __launch_bounds__(kFuseThreads, 2)
k_surrogate_correct(MlpDev m, const WorldDev* __restrict__ worlds, int nworlds,
                    uint32_t ncells, const CellTable table, const uint32_t* __restrict__ tp_cell,
                    const float2* __restrict__ tpp, const float2* __restrict__ tpv,
                    float2* __restrict__ q, float2* __restrict__ corr) {
  extern __shared__ __align__(16) uint8_t dyn[];
  SmemNet& s = *reinterpret_cast<SmemNet*>(dyn);
  uint32_t* sx = reinterpret_cast<uint32_t*>(dyn + sizeof(SmemNet));  // [256][kRow]
  load_net(m, s);
  const uint32_t ntp = table.taking(ncells);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t g = lane >> 2, t4 = lane & 3;
  for (uint32_t base = blockIdx.x * kFuseThreads; base < ntp; base += gridDim.x * kFuseThreads) {
    const uint32_t t = base + threadIdx.x;
    uint32_t* row = sx + threadIdx.x * kRow;
    if (t < ntp) {
      const uint32_t c = tp_cell[t];
      knn_row<true>(worlds[world_of_cell(worlds, nworlds, c)], table, tpp, tpv, c, t, row);
    } else {
      zero_row<true>(row);
    }
    __syncwarp();  // a warp's 32 rows are its own lanes'
    uint32_t ax[2][4][4];
    float out[2][4];
#pragma unroll
    for (uint32_t rt = 0; rt < 2; ++rt) {
      const uint32_t* p0 = sx + (warp * 32 + rt * 16 + g) * kRow;
      const uint32_t* p1 = p0 + 8 * kRow;
#pragma unroll
      for (uint32_t kk = 0; kk < 4; ++kk) {
        ax[rt][kk][0] = p0[kk * 8 + t4];
        ax[rt][kk][1] = p1[kk * 8 + t4];
        ax[rt][kk][2] = p0[kk * 8 + 4 + t4];
        ax[rt][kk][3] = p1[kk * 8 + 4 + t4];
      }
    }
    mlp_infer<2>(s, lane, ax, out);
    if (t4 == 0) {
#pragma unroll
      for (uint32_t rt = 0; rt < 2; ++rt) {
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
          const uint32_t idx = base + warp * 32 + rt * 16 + g + 8 * h;
          if (idx < ntp) {
            const float cxv = out[rt][2 * h], cyv = out[rt][2 * h + 1];
            const float2 p = tpp[idx];
            q[idx] = make_float2(__fadd_rn(p.x, cxv), __fadd_rn(p.y, cyv));
            if (corr) {
              const uint32_t c = tp_cell[idx];
              corr[table.start(c) + (idx - table.taking(c))] = make_float2(cxv, cyv);
            }
          }
        }
      }
    }
    __syncwarp();
  }
}

size_t correct_smem() { return sizeof(SmemNet) + (size_t)kFuseThreads * kRow * 4; }

// target = q - p, the first K-1 iterations' correction of frame particle i
// (q compacted: zero for a particle that takes no part)
__global__ void k_target(uint32_t n, const uint32_t* __restrict__ tp_of,
                         const float2* __restrict__ pos, const float2* __restrict__ q,
                         float2* __restrict__ target) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t t = tp_of[i];
  if (t == kNoTp) {
    target[i] = make_float2(0.f, 0.f);
    return;
  }
  const float2 p = pos[i], v = q[t];
  target[i] = make_float2(v.x - p.x, v.y - p.y);
}

// Sums of a block: 5 values per thread (sum, max, sum, sum, sum order in
// `v`), reduced over the block and written to part[blockIdx.x * 8 + k].
__device__ __forceinline__ void block_partials(float (&v)[5], float* __restrict__ part) {
  __shared__ float red[32][5];
#pragma unroll
  for (uint32_t o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const float u = __shfl_xor_sync(0xffffffffu, v[k], o);
      v[k] = k == 1 ? fmaxf(v[k], u) : v[k] + u;
    }
  }
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < 5; ++k) red[warp][k] = v[k];
  __syncthreads();
  if (threadIdx.x < 5) {
    float acc = red[0][threadIdx.x];
    for (uint32_t w = 1; w < nw; ++w)
      acc = threadIdx.x == 1 ? fmaxf(acc, red[w][threadIdx.x]) : acc + red[w][threadIdx.x];
    part[blockIdx.x * 8 + threadIdx.x] = acc;
  }
}

// Frame metrics (report only): per taking-part particle the deepest overlap
// with a taking-part neighbour of the 3x3 cells, max(0, max_j (min_d -
// |p_j - p_i|)); per block: [0] sum of overlaps, [1] max overlap, [2] number
// of taking-part particles, [3] kinetic energy, [4] 0.
__global__ void __launch_bounds__(256)
k_penetration(const WorldDev* __restrict__ worlds, int nworlds, PhysDev ph, uint32_t n,
              const CellTable table, const uint32_t* __restrict__ cell_of,
              const float2* __restrict__ pos, const float2* __restrict__ vel,
              float* __restrict__ part) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  float pen = 0.f, ke = 0.f, cnt = 0.f;
  if (i < n) {
    const float2 v = vel[i];
    ke = __fmul_rn(0.5f, __fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y)));
    const uint32_t c = cell_of[i];
    if (i - table.start(c) < ph.cap) {
      cnt = 1.f;
      const WorldDev w = worlds[world_of_cell(worlds, nworlds, c)];
      uint32_t cx, cy;
      cell_xy(w, c - w.cell_off, cx, cy);
      const float2 pi = pos[i];
      const int y0 = max((int)cy - 1, 0), y1 = min((int)cy + 1, (int)w.gy - 1);
      const int x0 = max((int)cx - 1, 0), x1 = min((int)cx + 1, (int)w.gx - 1);
      for (int ny = y0; ny <= y1; ++ny) {
        const uint32_t rb = w.cell_off + (uint32_t)ny * w.gx;
        for (int nx = x0; nx <= x1; ++nx) {
          uint32_t js, je;
          table.span(rb + nx, js, je);
          je = min(je, js + ph.cap);
          for (uint32_t j = js; j < je; ++j) {
            if (j == i) continue;
            const float2 pj = pos[j];
            const float dx = __fsub_rn(pj.x, pi.x), dy = __fsub_rn(pj.y, pi.y);
            const float s2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
            if (s2 >= ph.skip_d2) continue;  // no overlap
            pen = fmaxf(pen, __fsub_rn(ph.min_d, __fsqrt_rn(s2)));
          }
        }
      }
    }
  }
  float v[5] = {pen, pen, cnt, ke, 0.f};
  block_partials(v, part);
}

// Deterministic sum of per-block partials: out[k] for k in 0..4 (out[1] the
// max), one block of 256 threads.
__global__ void __launch_bounds__(256)
k_reduce_partials(const float* __restrict__ part, uint32_t nparts, float* __restrict__ out) {
  float v[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  // unrolled, so that the loads of several partials are in flight at once
#pragma unroll 4
  for (uint32_t b = threadIdx.x; b < nparts; b += blockDim.x) {
#pragma unroll
    for (int k = 0; k < 5; ++k) v[k] = k == 1 ? fmaxf(v[k], part[b * 8 + k]) : v[k] + part[b * 8 + k];
  }
  block_partials(v, out - blockIdx.x * 8);
}

// The fallback gate of a surrogate frame, one block.  The partials come from
// the final Jacobi iteration ([0] sum and [1] max of the deepest overlap
// before that iteration, [2] taking-part count, [3] kinetic energy of the
// output, [4] kinetic energy the plain frame has); `mode`:
//   0  after the surrogate correction and the last plain iteration: the frame
//      falls back when its mean overlap exceeds the latest plain frame's by
//      more than `tol`, or its kinetic energy deviates from the plain value
//      by more than `max_drift` (relative); NaN falls back too;
//   1  after the (gated) fallback solve: when the frame fell back, its plain
//      metrics become the reference;
//   2  after a plain calibration frame: its metrics become the reference.
__global__ void __launch_bounds__(1024)
k_gate(const float* __restrict__ part, uint32_t nparts, GateState* __restrict__ gs, int mode) {
  if (mode == 1 && gs->fallback == 0u) return;
  float v[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  // unrolled, so that the loads of several partials are in flight at once
#pragma unroll 8
  for (uint32_t b = threadIdx.x; b < nparts; b += blockDim.x) {
    const float4 p = reinterpret_cast<const float4*>(part)[b * 2];
    const float last = part[b * 8 + 4];
    v[0] += p.x;
    v[1] = fmaxf(v[1], p.y);
    v[2] += p.z;
    v[3] += p.w;
    v[4] += last;
  }
  __shared__ float tot[8];
  block_partials(v, tot - blockIdx.x * 8);
  __syncthreads();
  if (threadIdx.x != 0) return;
  const float mean = tot[2] > 0.f ? tot[0] / tot[2] : 0.f;
  const float drift = tot[4] > 0.f ? fabsf(tot[3] - tot[4]) / tot[4] : 0.f;
  if (mode == 0) {
    const bool ok = mean <= gs->pen_ref + gs->tol && drift <= gs->max_drift;
    gs->fallback = ok ? 0u : 1u;
    gs->frames += 1;
    gs->drift_max = fmaxf(gs->drift_max, drift);
    if (ok) {
      gs->pen_sum += mean;
      gs->pen_max = fmaxf(gs->pen_max, tot[1]);
    } else {
      gs->fallbacks += 1;
    }
  } else {
    gs->pen_ref = mean;
    gs->pen_sum += mean;
    gs->pen_max = fmaxf(gs->pen_max, tot[1]);
    if (mode == 2) {
      gs->frames += 1;
      gs->calibrations += 1;
    }
  }
}

// Squared errors of the correction against the target, and of zero against
// the target, over taking-part particles: out[0] += |corr - t|^2,
// out[1] += |t|^2, out[2] += count.
__global__ void k_errors(uint32_t n, const uint32_t* __restrict__ tp_of,
                         const float2* __restrict__ corr, const float2* __restrict__ target,
                         float* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  float e = 0.f, z = 0.f, c = 0.f;
  if (i < n && tp_of[i] != kNoTp) {
    const float2 a = corr[i], t = target[i];
    e = (a.x - t.x) * (a.x - t.x) + (a.y - t.y) * (a.y - t.y);
    z = t.x * t.x + t.y * t.y;
    c = 1.f;
  }
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    e += __shfl_xor_sync(0xffffffffu, e, o);
    z += __shfl_xor_sync(0xffffffffu, z, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&out[0], e);
    atomicAdd(&out[1], z);
    atomicAdd(&out[2], c);
  }
}

}  // namespace

cudaError_t launch_errors(const SolveArgs& a, const float2* corr, const float2* target, float* out,
                          cudaStream_t st) {
  if (a.n == 0) return cudaSuccess;
  k_errors<<<(a.n + 255) / 256, 256, 0, st>>>(a.n, a.tp_of, corr, target, out);
  return cudaGetLastError();
}

cudaError_t launch_compact_velocities(uint32_t n, const uint32_t* tp_of, const float2* vel,
                                      float2* tp_vel, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_compact_velocities<<<(n + 255) / 256, 256, 0, st>>>(n, tp_of, vel, tp_vel);
  return cudaGetLastError();
}

cudaError_t launch_knn_features(const SolveArgs& a, uint16_t* x, cudaStream_t st) {
  if (a.n == 0) return cudaSuccess;
  k_knn_features<<<(a.n + 255) / 256, 256, 0, st>>>(a.worlds, a.nworlds, a.n, a.tp_of, a.table,
                                                    a.cell_of, a.tp_pos, a.tp_vel, x);
  return cudaGetLastError();
}

cudaError_t launch_samples(const SolveArgs& a, const float2* q, uint32_t stride, uint32_t phase,
                           uint32_t rows, uint16_t* x, float2* target, cudaStream_t st) {
  if (rows == 0) return cudaSuccess;
  k_samples<<<(rows + 255) / 256, 256, 0, st>>>(a.worlds, a.nworlds, a.ncells, a.table, a.tp_cell,
                                                a.tp_pos, a.tp_vel, q, stride, phase, rows, x,
                                                target);
  return cudaGetLastError();
}

int surrogate_correct_blocks(int device) {
  const size_t smem = correct_smem();
  if (cudaFuncSetAttribute(k_surrogate_correct, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) != cudaSuccess)
    return 0;
  // persistent: one wave of co-resident blocks
  int sms = 0, per_sm = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_surrogate_correct, kFuseThreads,
                                                    smem) != cudaSuccess)
    return 0;
  return sms * (per_sm > 0 ? per_sm : 1);
}

cudaError_t launch_surrogate_correct(const MlpDev& m, const SolveArgs& a, float2* q, float2* corr,
                                     int blocks, cudaStream_t st) {
  if (a.n == 0) return cudaSuccess;
  const int need = (int)((a.n + kFuseThreads - 1) / kFuseThreads);
  k_surrogate_correct<<<need < blocks ? need : blocks, kFuseThreads, correct_smem(), st>>>(
      m, a.worlds, a.nworlds, a.ncells, a.table, a.tp_cell, a.tp_pos, a.tp_vel, q,
      corr);
  return cudaGetLastError();
}

cudaError_t launch_gate(const float* part, uint32_t nparts, GateState* gs, int mode,
                        cudaStream_t st) {
  k_gate<<<1, 1024, 0, st>>>(part, nparts, gs, mode);
  return cudaGetLastError();
}

cudaError_t launch_mlp_forward(const MlpDev& m, const uint16_t* x, uint32_t n, float2* y,
                               int blocks, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const int need = (int)((n + 63) / 64);
  k_mlp_forward<<<need < blocks ? need : blocks, 128, 0, st>>>(m, x, n, y);
  return cudaGetLastError();
}

bool train_setup() {
  for (auto k : {k_mlp_backward<false>, k_mlp_backward<true>})
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(SmemTrain)) != cudaSuccess)
      return false;
  return true;
}

cudaError_t launch_mlp_backward(const MlpDev& m, const uint16_t* x, const float2* target,
                                uint32_t n, float inv_rows, float* grad, bool want_loss, int sms,
                                cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const uint32_t tiles = (n + kTrainRows - 1) / kTrainRows, most = sms > 0 ? sms : 1;
  return launch_after_with(sizeof(SmemTrain), want_loss ? k_mlp_backward<true> : k_mlp_backward<false>,
                           tiles < most ? tiles : most, kTrainThreads, st, m, x, target, n, inv_rows,
                           grad);
}

cudaError_t launch_take_gradients(float* grad, float* out, cudaStream_t st) {
  return launch_after(k_take_gradients, kMlpParams / 256 + 1, 256, st, grad, out,
                      (uint32_t)kMlpParams);
}

cudaError_t launch_adam(const MlpDev& m, float* grad, float* mom1, float* mom2, float lr,
                        uint32_t step, cudaStream_t st) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
  return launch_after(k_adam, kMlpParams / 256 + 1, 256, st, m, grad, mom1, mom2, lr, b1, b2, eps,
                      bc1, bc2, (uint32_t)kMlpParams);
}

cudaError_t launch_target(const SolveArgs& a, uint32_t n, const float2* q, float2* target,
                          cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_target<<<(n + 255) / 256, 256, 0, st>>>(n, a.tp_of, a.pos, q, target);
  return cudaGetLastError();
}

cudaError_t launch_penetration(const SolveArgs& a, const float2* pos, const float2* vel,
                               float* part, float* out, cudaStream_t st) {
  const uint32_t blocks = (a.n + 255) / 256;
  if (blocks) {
    k_penetration<<<blocks, 256, 0, st>>>(a.worlds, a.nworlds, a.ph, a.n, a.table, a.cell_of,
                                          pos, vel, part);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  k_reduce_partials<<<1, 256, 0, st>>>(part, blocks, out);
  return cudaGetLastError();
}

}  // namespace wrach
