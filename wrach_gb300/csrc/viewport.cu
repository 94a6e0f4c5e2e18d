// Viewport streaming: the device side of writing a world's frame back into
// its particle store (the reference's `ParticleStore::update_from_gpu`,
// runners/bevy/src/particle_store.rs:71-85, a TODO there).  The store keeps
// the particles it holds outside the viewport, in store order; the frame's
// particles are appended after them.  Per tile of 1024 store items one bit an
// item and a count, one block scans the counts, then one launch moves the
// kept items and, from the device's own count of them, appends the frame's.
//
// Bound by memory (16 bytes read and written per item) and by its three
// launches.  The host waits for the count alone, while the store is rebuilt.
// With 32-bit keys read twice, and the frame copied by the host once it knew
// the count, moving the viewport of a 1M-particle world, one frame and its
// readback took 373 us; 296 now, with the re-packing that follows.
#include "wrach_internal.cuh"
#include "wrach_kernels.h"

namespace wrach {

namespace {

constexpr uint32_t kThreads = 256, kPer = 4, kTile = kThreads * kPer;
constexpr uint32_t kWarps = kThreads / 32, kTileWords = kTile / 32;
constexpr uint32_t kNoCell = 0xFFFFFFFFu;
static_assert(kTileWords == 32, "a tile's words are one per lane");

// Exclusive scan of one value per thread over the block; *total receives
// the sum.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t warp_sum[32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sum[warp] = x;
  __syncthreads();
  uint32_t before = 0, all = 0;
  for (uint32_t w = 0; w < nw; ++w) {
    before += w < warp ? warp_sum[w] : 0u;
    all += warp_sum[w];
  }
  __syncthreads();
  *total = all;
  return before + x - v;
}

// outside: bit i % 32 of word i / 32 is set when store item i lies outside the
// viewport; tile_sums: the tiles' numbers of them.
__global__ void __launch_bounds__(kThreads) k_outside(const StoreRebuild r) {
  __shared__ uint32_t warp_sum[kWarps];
  begin_after();
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t i0 = blockIdx.x * kTile + threadIdx.x;
  const WorldDev w = r.worlds[r.target];
  float2 p[kPer];
#pragma unroll
  for (uint32_t u = 0; u < kPer; ++u)
    p[u] = i0 + u * kThreads < r.n ? r.pos[i0 + u * kThreads] : make_float2(0.f, 0.f);
  uint32_t sum = 0;
#pragma unroll
  for (uint32_t u = 0; u < kPer; ++u) {
    const bool out = i0 + u * kThreads < r.n && upload_key(w, p[u], kNoCell) == kNoCell;
    const uint32_t bits = __ballot_sync(0xffffffffu, out);
    if (lane == 0) r.outside[blockIdx.x * kTileWords + u * kWarps + warp] = bits;
    sum += __popc(bits);
  }
  if (lane == 0) warp_sum[warp] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t total = 0;
#pragma unroll
    for (uint32_t k = 0; k < kWarps; ++k) total += warp_sum[k];
    r.tile_sums[blockIdx.x] = total;
  }
}

// One block: tile_sums becomes its exclusive scan.
__global__ void __launch_bounds__(1024) k_outside_scan(const StoreRebuild r, uint32_t ntiles) {
  begin_after();
  uint32_t carry = 0;
  for (uint32_t b0 = 0; b0 < ntiles; b0 += blockDim.x) {
    const uint32_t b = b0 + threadIdx.x;
    const uint32_t v = b < ntiles ? r.tile_sums[b] : 0u;
    uint32_t total;
    const uint32_t ex = block_scan(v, &total);
    if (b < ntiles) r.tile_sums[b] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) {
    *r.kept = carry;
    *r.kept_host = carry;
    if (r.moves) r.worlds[r.target] = r.moved;
  }
}

// Blocks below ntiles move a tile's kept items, the others 1024 of the frame's.
__global__ void __launch_bounds__(kThreads) k_rebuild(const StoreRebuild r, uint32_t ntiles) {
  begin_after();
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (blockIdx.x < ntiles) {
    // lane k: word k of the tile, and the kept items before it
    const uint32_t word = r.outside[blockIdx.x * kTileWords + lane];
    uint32_t before = __popc(word);
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += y;
    }
    before += r.tile_sums[blockIdx.x] - __popc(word);
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u) {
      const uint32_t k = u * kWarps + warp;
      const uint32_t bits = __shfl_sync(0xffffffffu, word, k);
      const uint32_t d = __shfl_sync(0xffffffffu, before, k) + __popc(bits & ((1u << lane) - 1u));
      if (bits >> lane & 1u) {
        const uint32_t i = blockIdx.x * kTile + u * kThreads + threadIdx.x;
        r.dst_pos[d] = r.pos[i];
        r.dst_vel[d] = r.vel[i];
      }
    }
    return;
  }
  const uint32_t j0 = (blockIdx.x - ntiles) * kTile + threadIdx.x;
  const size_t kept = *r.kept;
#pragma unroll
  for (uint32_t u = 0; u < kPer; ++u) {
    const uint32_t j = j0 + u * kThreads;
    if (j < r.nf) {
      r.dst_pos[kept + j] = r.frame_pos[j];
      r.dst_vel[kept + j] = r.frame_vel[j];
    }
  }
}

}  // namespace

uint32_t store_tiles(uint32_t n) { return (n + kTile - 1) / kTile; }

cudaError_t launch_outside(const StoreRebuild& r, cudaStream_t st) {
  const uint32_t ntiles = store_tiles(r.n);
  if (ntiles) {
    const cudaError_t e = launch_after(k_outside, ntiles, kThreads, st, r);
    if (e != cudaSuccess) return e;
  }
  return launch_after(k_outside_scan, 1, 1024, st, r, ntiles);
}

cudaError_t launch_rebuild(const StoreRebuild& r, cudaStream_t st) {
  const uint32_t ntiles = store_tiles(r.n), blocks = ntiles + store_tiles(r.nf);
  return blocks ? launch_after(k_rebuild, blocks, kThreads, st, r, ntiles) : cudaSuccess;
}

}  // namespace wrach
