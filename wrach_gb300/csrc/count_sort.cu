// Rebin as a stable counting sort over the cells: the count, scan and pack
// passes of a frame (assets/shaders/particles_per_cell.wgsl, prefix_sum.wgsl,
// pack_new_particle_data.wgsl; dispatched by runners/bevy/src/compute/
// builder.rs:86-89) as a chain of short launches.
//
//   count    (warp_ticket, in the launch that computes the keys: a frame's
//            last solve launch, an upload's keys) per warp, the particles of
//            one cell (__match_any_sync) take one atomic on the cell's
//            counter; each particle's ticket (its slot inside the cell,
//            arrival order) is the returned base plus its rank among the
//            warp's particles of that cell; per warp one more atomic adds the
//            particles of each tile of 2048 cells to the tile's sum
//   scan     exclusive scan of the per-cell counts, one block per tile of
//            2048 cells; a tile's prefix is the sum of the earlier tiles'
//            sums (already final, so no block waits): each block adds them
//            up itself, or, past kPrefixTiles tiles (where that sum grows
//            with the square of the grid), a launch first turns runs of tile
//            sums into their prefixes; it writes the cell table
//            (CellTable: starts, and the starts among the taking-part
//            particles from the counts capped at the cell capacity) and
//            lists the cells of more than kSmallCell particles
//            (the pass that takes the tickets empties that list first); the
//            place steps clear the counts of the non-empty cells afterwards
//   scatter  source index and cell of every particle to table start + ticket
//            (arrival order inside a cell)
//   place    the stable order: inside a cell, a particle's rank is the number
//            of the cell's particles with a smaller source index; then the
//            gather of positions, velocities and cells into that slot, and of
//            the taking-part particles' positions, cells and (for the learned
//            surrogate) velocities into the compacted arrays.  Cells of up
//            to kSmallCell particles are ranked by one thread per slot
//   large    (with place, in blocks of their own) one block per listed cell:
//            up to kBigCell particles ranked by a bitmap of their source
//            indices (or a bitonic sort) in shared memory, more than that a
//            block-wide LSD radix sort of them in global memory; then the
//            gather.  It writes other slots than place, so the two may run at
//            the same time
//
// The result is the stable order (a cell's particles keep their source
// order), the order of the oracle's counting sort and of rebin.cu's radix
// sort.
#include "wrach_internal.cuh"
#include "wrach_kernels.h"

namespace wrach {

namespace {

constexpr uint32_t kScanThreads = 256, kScanPer = 8;
static_assert(kScanPer == 8, "a scan thread takes 4 cells of each half tile");
// Without taking-part particles (reference physics) a grouped table's records
// count up to this many particles of a cell; cells with more are wide.
constexpr uint32_t kPlainCap = 31;
static_assert(kDenseCells / kCountScanTile >= 2048, "grouped tables' tiles are prefixed");
static_assert(kGroup * kPlainCap < 256 && kPlainCap < kSmallCell && kMaxCellCapacity < kSmallCell,
              "a record's bytes; large cells are wide");

// The new cell table; GROUPED as a constant, so that a dense table's lookups
// are plain loads.
template <bool GROUPED>
__device__ __forceinline__ CellTable new_table(const RebinArgs& a) {
  return CellTable{GROUPED ? a.groups_new : nullptr, a.cs_new, a.ct_new};
}
constexpr uint32_t kScanTile = kScanThreads * kScanPer;
static_assert(kScanTile == kCountScanTile, "tile size shared with the tickets' tile sums");

// Gives back the tickets of n particles: their cells' counters and all tile
// sums are zero again.  Returns at once when *run_if reads 0.
__global__ void __launch_bounds__(256)
k_cs_untake(const uint32_t* __restrict__ run_if, const uint32_t* __restrict__ keys, uint32_t n,
            CountDev c, uint32_t ntiles) {
  if (*run_if == 0u) return;
  const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  for (uint32_t i = i0; i < n; i += stride)
    if (keys[i] < c.ncells) c.counts[keys[i]] = 0u;
  for (uint32_t t = i0; t < ntiles; t += stride) {
    c.tile_sums[t] = 0u;
    if (c.tile_sums_cap) c.tile_sums_cap[t] = 0u;
  }
}

// Scans: one block per tile of 2048 cells.  The tile's prefix is the sum of the
// earlier tiles' counts, which the tickets' pass has already totalled, so no
// block waits for another.  Past this many tiles of the table,
// k_cs_tile_prefix first turns the tile sums into prefixes, one block per kRun
// tiles: a tile's sum becomes that of the run's earlier tiles, and the run's
// own sum goes behind the tile sums.  A scan block then adds up the earlier
// runs instead of the earlier tiles (one block that scanned all tiles by
// itself took 134 us for the 44,775 tiles of 92M cells; 2.5 us now).  1,013
// tiles are still better summed by each block (a frame 103.9 us, 105.8 with
// the launch).
constexpr uint32_t kPrefixTiles = 2048, kRun = 256;

__global__ void __launch_bounds__(kRun) k_cs_tile_prefix(RebinArgs a, uint32_t ntiles) {
  begin_after();
  __shared__ uint32_t ws[kRun / 32], wc[kRun / 32];
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t i = blockIdx.x * kRun + t;
  const uint32_t s = i < ntiles ? a.tile_sums[i] : 0u;
  const uint32_t c = i < ntiles && a.tp_cap ? a.tile_sums_cap[i] : 0u;
  uint32_t x = s, y = c;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, x, o), v = __shfl_up_sync(0xffffffffu, y, o);
    if (lane >= o) {
      x += u;
      y += v;
    }
  }
  if (lane == 31) {
    ws[warp] = x;
    wc[warp] = y;
  }
  __syncthreads();
  for (uint32_t w = 0; w < warp; ++w) {
    x += ws[w];
    y += wc[w];
  }
  if (i < ntiles) {
    a.tile_sums[i] = x - s;
    if (a.tp_cap) a.tile_sums_cap[i] = y - c;
  }
  if (t == kRun - 1) {
    a.tile_sums[ntiles + blockIdx.x] = x;
    if (a.tp_cap) a.tile_sums_cap[ntiles + blockIdx.x] = y;
  }
}

// The particles (sums: tile_sums or tile_sums_cap) before a tile; the warp's
// lanes call it together.
__device__ __forceinline__ uint32_t before_tile(const uint32_t* sums, uint32_t tile,
                                                uint32_t ntiles) {
  uint32_t s = 0;
  for (uint32_t r = threadIdx.x & 31; r < tile / kRun; r += 32) s += sums[ntiles + r];
  return __reduce_add_sync(0xffffffffu, s) + sums[tile];
}

// The large cells' work list (at most n / (kSmallCell + 1) cells qualify, and
// big_cap is larger).
__device__ __forceinline__ void list_large(const RebinArgs& a, uint32_t cell) {
  const uint32_t w = atomicAdd(&a.ctrl->big_count, 1u);
  if (w < a.big_cap) a.big_list[w] = cell;
}

// A thread takes four cells of either half of the tile, so that a warp's 16-byte
// loads and stores are contiguous: with eight cells in a row per thread every
// sector moved in two halves, and each count crossed from L2 twice (2.1M cells
// 8.2 -> 6.1 us, 8.4M 24.6 -> 20.5; a frame of 262,144 particles 52.8 -> 49.0).
__global__ void __launch_bounds__(kScanThreads) k_cs_scan(RebinArgs a) {
  begin_after();
  __shared__ uint4 sums[kScanThreads / 32];
  __shared__ uint2 earlier[kScanThreads / 32];
  constexpr uint32_t kHalf = kScanTile / 2;
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t tile = blockIdx.x, n = a.ncells;
  if (tile == 0 && t == 0 && !a.force_general) a.ctrl->frames += 1;
  const uint32_t c0 = tile * kScanTile + t * 4;
  uint32_t v[2][4];
#pragma unroll
  for (uint32_t h = 0; h < 2; ++h) {
    const uint32_t c = c0 + h * kHalf;
    if (c + 4 <= n) {
      const uint4 q = *reinterpret_cast<const uint4*>(a.counts + c);
      v[h][0] = q.x; v[h][1] = q.y; v[h][2] = q.z; v[h][3] = q.w;
    } else {
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) v[h][u] = c + u < n ? a.counts[c + u] : 0u;
    }
  }
  // the capped counts (the taking-part particles) when the capped table is wanted
  const uint32_t cap = a.tp_cap;
  // the earlier tiles' totals: the tickets' pass has them ready.  Their sum
  // goes through the same barrier as the block's own scans below
  uint32_t pre = 0, cpre = 0;
  if (!a.prefixed_tiles) {
    for (uint32_t u = t; u < tile; u += kScanThreads) {
      pre += a.tile_sums[u];
      if (cap) cpre += a.tile_sums_cap[u];
    }
    pre = __reduce_add_sync(0xffffffffu, pre);
    if (cap) cpre = __reduce_add_sync(0xffffffffu, cpre);
  } else if (warp == 0) {
    pre = before_tile(a.tile_sums, tile, a.prefixed_tiles);
    if (cap) cpre = before_tile(a.tile_sums_cap, tile, a.prefixed_tiles);
  }
  uint32_t x[2], cx[2];
#pragma unroll
  for (uint32_t h = 0; h < 2; ++h) {
    x[h] = v[h][0] + v[h][1] + v[h][2] + v[h][3];
    cx[h] = min(v[h][0], cap) + min(v[h][1], cap) + min(v[h][2], cap) + min(v[h][3], cap);
  }
  const uint32_t own[2] = {x[0], x[1]}, cown[2] = {cx[0], cx[1]};
  // block-wide exclusive scans of the per-thread sums
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x[h], o);
      const uint32_t cy = __shfl_up_sync(0xffffffffu, cx[h], o);
      if (lane >= o) {
        x[h] += y;
        cx[h] += cy;
      }
    }
  }
  if (lane == 31) {
    sums[warp] = make_uint4(x[0], cx[0], x[1], cx[1]);
    earlier[warp] = make_uint2(pre, cpre);
  }
  __syncthreads();
  uint32_t run[2] = {0u, 0u}, crun[2] = {0u, 0u}, first = 0, cfirst = 0, total = 0, ctotal = 0;
  uint32_t prefix = 0, cprefix = 0;
#pragma unroll
  for (uint32_t w = 0; w < kScanThreads / 32; ++w) {
    const uint4 s = sums[w];
    const uint2 e = earlier[w];
    run[0] += w < warp ? s.x : 0u;
    crun[0] += w < warp ? s.y : 0u;
    run[1] += w < warp ? s.z : 0u;
    crun[1] += w < warp ? s.w : 0u;
    first += s.x;
    cfirst += s.y;
    total += s.x + s.z;
    ctotal += s.y + s.w;
    prefix += e.x;
    cprefix += e.y;
  }
  run[0] += prefix + x[0] - own[0];
  crun[0] += cprefix + cx[0] - cown[0];
  run[1] += prefix + first + x[1] - own[1];
  crun[1] += cprefix + cfirst + cx[1] - cown[1];
#pragma unroll
  for (uint32_t h = 0; h < 2; ++h) {
    const uint32_t c = c0 + h * kHalf;
    uint32_t at[4], cat[4];
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
      if (v[h][u] > kSmallCell) list_large(a, c + u);
      at[u] = run[h];
      cat[u] = crun[h];
      run[h] += v[h][u];
      crun[h] += min(v[h][u], cap);
    }
    if (c + 4 <= n) {
      *reinterpret_cast<uint4*>(a.cs_new + c) = make_uint4(at[0], at[1], at[2], at[3]);
      if (cap) *reinterpret_cast<uint4*>(a.ct_new + c) = make_uint4(cat[0], cat[1], cat[2], cat[3]);
    } else {
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) {
        if (c + u >= n) break;
        a.cs_new[c + u] = at[u];
        if (cap) a.ct_new[c + u] = cat[u];
      }
    }
  }
  if (t == 0 && (tile + 1) * kScanTile >= n) {
    if (cap) a.ct_new[n] = cprefix + ctotal;
    a.cs_new[n] = prefix + total;
    if (a.total_out) *a.total_out = prefix + total;
  }
}

// The same for a grouped table: a thread takes 16 cells, two records.  It
// reads 4 bytes per cell and writes 2 where the dense scan writes 8 (92M
// cells: 181 us dense, 82 us).
constexpr uint32_t kGroupThreads = kScanTile / (2 * kGroup);

__global__ void __launch_bounds__(kGroupThreads) k_cs_scan_groups(RebinArgs a) {
  begin_after();
  __shared__ uint32_t warp_sum[kGroupThreads / 32], warp_cap[kGroupThreads / 32];
  constexpr uint32_t per = 2 * kGroup;
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t tile = blockIdx.x, n = a.ncells;
  if (tile == 0 && t == 0 && !a.force_general) a.ctrl->frames += 1;
  const uint32_t c0 = tile * kScanTile + t * per;
  uint32_t v[per];
  if (c0 + per <= n) {
    const uint4* src = reinterpret_cast<const uint4*>(a.counts + c0);
#pragma unroll
    for (uint32_t u = 0; u < per / 4; ++u) {
      const uint4 q = src[u];
      v[4 * u] = q.x; v[4 * u + 1] = q.y; v[4 * u + 2] = q.z; v[4 * u + 3] = q.w;
    }
  } else {
#pragma unroll
    for (uint32_t u = 0; u < per; ++u) v[u] = c0 + u < n ? a.counts[c0 + u] : 0u;
  }
  const uint32_t prefix = before_tile(a.tile_sums, tile, a.prefixed_tiles);
  const uint32_t cprefix = a.tp_cap ? before_tile(a.tile_sums_cap, tile, a.prefixed_tiles) : 0u;
  // the capped counts: the taking-part particles (extended physics)
  const uint32_t cap = a.tp_cap ? a.tp_cap : kPlainCap;
  uint32_t sum[2], csum[2], low[2], high[2];
  bool wide[2];
#pragma unroll
  for (uint32_t h = 0; h < 2; ++h) {
    sum[h] = csum[h] = low[h] = high[h] = 0u;
    wide[h] = false;
#pragma unroll
    for (uint32_t u = 0; u < kGroup; ++u) {
      const uint32_t x = v[h * kGroup + u];
      if (u < 4) low[h] |= csum[h] << (8 * u);
      else high[h] |= csum[h] << (8 * (u - 4));
      sum[h] += x;
      csum[h] += min(x, cap);
      wide[h] = wide[h] || x > cap;
    }
  }
  uint32_t x = sum[0] + sum[1], cx = csum[0] + csum[1];
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    const uint32_t cy = __shfl_up_sync(0xffffffffu, cx, o);
    if (lane >= o) {
      x += y;
      cx += cy;
    }
  }
  if (lane == 31) {
    warp_sum[warp] = x;
    warp_cap[warp] = cx;
  }
  __syncthreads();
  uint32_t run = prefix + x - sum[0] - sum[1], crun = cprefix + cx - csum[0] - csum[1];
#pragma unroll
  for (uint32_t w = 0; w < kGroupThreads / 32 - 1; ++w) {
    run += w < warp ? warp_sum[w] : 0u;
    crun += w < warp ? warp_cap[w] : 0u;
  }
#pragma unroll
  for (uint32_t h = 0; h < 2; ++h) {
    // the record past the last cell holds the totals
    const uint32_t c = c0 + h * kGroup;
    if (c <= n)
      a.groups_new[c / kGroup] = make_uint4(run, crun | (wide[h] ? kWide : 0u), low[h], high[h]);
    if (wide[h]) {
      uint32_t at = run;
#pragma unroll
      for (uint32_t u = 0; u < kGroup; ++u) {
        const uint32_t k = v[h * kGroup + u];
        if (c + u <= n) a.cs_new[c + u] = at;
        at += k;
        if (k > kSmallCell) list_large(a, c + u);
      }
    }
    run += sum[h];
    crun += csum[h];
  }
  if (t == kGroupThreads - 1 && (tile + 1) * kScanTile == n)
    a.groups_new[n / kGroup] = make_uint4(run, crun, 0u, 0u);
  if (a.total_out && t == kGroupThreads - 1 && tile == gridDim.x - 1) *a.total_out = run;
}

// Bound by its chain of loads: the key and the ticket together, then the cell's
// span.  The span also tells the large cells apart, whose slots the next launch
// then leaves at their first load (4M particles in 256 worlds, this and the
// place step's loads side by side: 391 -> 387 us a frame).
template <bool GROUPED>
__global__ void __launch_bounds__(256) k_cs_scatter(RebinArgs a, uint32_t ntiles) {
  begin_after();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  // the scan has read the tile sums: clear them for the next rebin
  for (uint32_t u = i; u < ntiles; u += gridDim.x * blockDim.x) {
    a.tile_sums[u] = 0u;
    if (a.tp_cap) a.tile_sums_cap[u] = 0u;
  }
  if (i >= a.n) return;
  const uint32_t k = a.keys[i], ticket = a.ticket[i];
  if (k >= a.ncells) return;
  uint32_t s0, s1;
  new_table<GROUPED>(a).span(k, s0, s1);
  const uint32_t dst = s0 + ticket;
  if (dst < a.n) {  // (always: the tickets number what the scan counted)
    a.idx_tmp[dst] = i;
    // a large cell's slots are not place_slot's
    a.cell_tmp[dst] = s1 - s0 > kSmallCell ? a.ncells : k;
  }
}

// The particle of source index `src` into `slot`, rank `rank` inside its
// cell; a taking-part one (rank < tp_cap) also into the compacted arrays.
template <bool GROUPED>
__device__ __forceinline__ void place_one(const RebinArgs& a, uint32_t slot, uint32_t rank,
                                          uint32_t src, uint32_t cell, uint32_t& overflow) {
  if (slot < a.dst_capacity && src < a.n) {
    const float2 p = a.pos_src[src], v = a.vel_src[src];
    a.pos_dst[slot] = p;
    a.vel_dst[slot] = v;
    a.cell_dst[slot] = cell;
    if (a.tp_cap) {
      const uint32_t t = rank < a.tp_cap ? new_table<GROUPED>(a).taking(cell) + rank : kNoTp;
      a.tp_of[slot] = t;
      if (t < a.dst_capacity) {
        a.tp_pos[t] = p;
        if (a.tp_vel) a.tp_vel[t] = v;
        a.tp_cell[t] = cell;
      }
    }
  } else {
    ++overflow;
  }
}

__device__ __forceinline__ void add_overflow(const RebinArgs& a, uint32_t overflow) {
  const uint32_t wo = __reduce_add_sync(0xffffffffu, overflow);
  if ((threadIdx.x & 31) == 0 && wo) atomicAdd(&a.ctrl->overflow, wo);
}

// The small cells: one thread per slot q.
template <bool GROUPED>
__device__ __forceinline__ void place_slot(const RebinArgs& a, uint32_t q) {
  const CellTable table = new_table<GROUPED>(a);
  const uint32_t total = table.start(a.ncells);
  uint32_t overflow = 0;
  const bool in = q < total && q < a.n;
  const uint32_t k = in ? a.cell_tmp[q] : a.ncells, me = in ? a.idx_tmp[q] : a.n;
  if (k < a.ncells) {
    uint32_t c0, c1;
    table.span(k, c0, c1);
    const uint32_t s1 = min(c1, min(total, a.n));
    // the particle's data and its cell's compacted start do not depend on
    // its rank: their loads go out with the cell's span
    const bool src_ok = me < a.n;
    const float2 p = src_ok ? a.pos_src[me] : make_float2(0.f, 0.f);
    const float2 v = src_ok ? a.vel_src[me] : make_float2(0.f, 0.f);
    const uint32_t tp0 = a.tp_cap ? table.taking(k) : 0u;
    uint32_t rank = 0;
    for (uint32_t m = c0; m < s1; ++m) rank += a.idx_tmp[m] < me ? 1u : 0u;
    const uint32_t slot = c0 + rank;
    if (slot < a.dst_capacity && src_ok) {
      a.pos_dst[slot] = p;
      a.vel_dst[slot] = v;
      a.cell_dst[slot] = k;
      if (a.tp_cap) {
        const uint32_t t = rank < a.tp_cap ? tp0 + rank : kNoTp;
        a.tp_of[slot] = t;
        if (t < a.dst_capacity) {
          a.tp_pos[t] = p;
          if (a.tp_vel) a.tp_vel[t] = v;
          a.tp_cell[t] = k;
        }
      }
    } else {
      ++overflow;
    }
    // the scan has read the cell's count: zero for the next rebin (only
    // non-empty cells were counted)
    if (rank == 0) a.counts[k] = 0u;
  }
  add_overflow(a, overflow);
}

constexpr uint32_t kBigThreads = 256;
static_assert(kBigThreads == 256, "one radix digit per thread");

// Stable block-wide LSD radix sort (8-bit digits) of the m values src[0..m)
// into src or alt (returned), in chunks of 256 values: inside a chunk a
// value's slot is its digit's running offset, plus the counts of its digit
// in the chunk's earlier warps, plus its rank among its warp's equal digits.
struct RadixScratch {
  uint32_t hist[256], wcnt[kBigThreads / 32][256];
};
__device__ uint32_t* block_radix_sort(RadixScratch& R, uint32_t* src, uint32_t* alt, uint32_t m,
                                      uint32_t key_bits) {
  auto& hist = R.hist;
  auto& wcnt = R.wcnt;
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t lanemask_lt = (1u << lane) - 1u;
  for (uint32_t shift = 0; shift < key_bits; shift += 8) {
    hist[t] = 0u;
    __syncthreads();
    for (uint32_t r = t; r < m; r += kBigThreads) atomicAdd(&hist[(src[r] >> shift) & 255u], 1u);
    __syncthreads();
    // exclusive scan of the 256 digit counts (thread t owns digit t)
    uint32_t cnt = hist[t], x = cnt;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wcnt[0][warp] = x;
    __syncthreads();
    uint32_t before = 0;
    for (uint32_t w = 0; w < warp; ++w) before += wcnt[0][w];
    __syncthreads();
    uint32_t base = before + x - cnt;  // digit t's running offset
    for (uint32_t c0 = 0; c0 < m; c0 += kBigThreads) {
      const uint32_t r = c0 + t;
      const bool valid = r < m;
      const uint32_t v = valid ? src[r] : 0u;
      const uint32_t d = valid ? (v >> shift) & 255u : 256u;
      const uint32_t peers = __match_any_sync(0xffffffffu, d);
#pragma unroll
      for (uint32_t w = 0; w < kBigThreads / 32; ++w) wcnt[w][t] = 0u;
      __syncthreads();
      if (valid && (peers & lanemask_lt) == 0u) wcnt[warp][d] = __popc(peers);
      __syncthreads();
      uint32_t acc = 0;
#pragma unroll
      for (uint32_t w = 0; w < kBigThreads / 32; ++w) {
        const uint32_t c = wcnt[w][t];
        wcnt[w][t] = acc;
        acc += c;
      }
      hist[t] = base;
      __syncthreads();
      if (valid) alt[hist[d] + wcnt[warp][d] + __popc(peers & lanemask_lt)] = v;
      __syncthreads();
      base += acc;
    }
    uint32_t* tmp = src;
    src = alt;
    alt = tmp;
    __syncthreads();
  }
  return src;
}

// The ranks of a large cell's source indices from a bitmap.  A pile's
// particles come from its own cell and those around it, so their sources lie
// in few pages of kPageBits indices, one word of bits per 32: the rank of an
// index is the number of bits before its own.  Seven barriers for a cell of
// any size, where the bitonic sort takes 45 for 512 indices (the collapsed 1M
// lattice: 33 us sorting, 16 us now; 4M particles: 122 and 49 us).  Cells whose indices lie in more than
// kPages pages (uploads in any order) are sorted.
constexpr uint32_t kPages = 32, kPageBits = 1024, kPageWords = kPageBits / 32;
constexpr uint32_t kNoPage = 0xFFFFFFFFu;

struct PageRanks {
  uint32_t bits[kPages * kPageWords];
  uint16_t before[kPages * kPageWords];  // indices in the words before
  uint32_t page[kPages];                 // hash table of the pages present
  uint32_t place[kPages];                // first word of a slot's page, in page order
  uint32_t warp_sum[kBigThreads / 32];
  uint32_t full;
};
static_assert(kPages == 32 && kBigCell < 65536, "one lane per page; ranks fit 16 bits");

__device__ __forceinline__ uint32_t page_word(const PageRanks& P, uint32_t idx) {
  const uint32_t page = idx / kPageBits;
  uint32_t h = page % kPages;
  for (uint32_t tries = 1; P.page[h] != page && tries < kPages; ++tries) h = (h + 1) % kPages;
  return P.place[h] + (idx / 32) % kPageWords;
}

// Fills P for the s indices of `src`; false (for the whole block) when their
// pages do not fit.
__device__ bool page_ranks(PageRanks& P, const uint32_t* src, uint32_t s) {
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (uint32_t w = t; w < kPages * kPageWords; w += kBigThreads) P.bits[w] = 0u;
  if (t < kPages) P.page[t] = kNoPage;
  if (t == 0) P.full = 0u;
  __syncthreads();
  for (uint32_t r0 = 0; r0 < s; r0 += kBigThreads) {
    const uint32_t r = r0 + t;
    const uint32_t page = r < s ? src[r] / kPageBits : kNoPage;
    const uint32_t peers = __match_any_sync(0xffffffffu, page);
    if (page != kNoPage && lane == (uint32_t)(__ffs(peers) - 1)) {
      uint32_t h = page % kPages, tries = 0;
      for (; tries < kPages; ++tries) {
        const uint32_t old = atomicCAS(&P.page[h], kNoPage, page);
        if (old == kNoPage || old == page) break;
        h = (h + 1) % kPages;
      }
      if (tries == kPages) P.full = 1u;
    }
  }
  __syncthreads();
  if (P.full) return false;
  if (warp == 0) {
    const uint32_t mine = P.page[lane];
    uint32_t rank = 0;
#pragma unroll
    for (uint32_t o = 1; o < kPages; ++o)
      rank += __shfl_sync(0xffffffffu, mine, (lane + o) & 31u) < mine ? 1u : 0u;
    P.place[lane] = (mine == kNoPage ? 0u : rank) * kPageWords;
  }
  __syncthreads();
  for (uint32_t r = t; r < s; r += kBigThreads) {
    const uint32_t idx = src[r];
    atomicOr(&P.bits[page_word(P, idx)], 1u << (idx & 31u));
  }
  __syncthreads();
  constexpr uint32_t per = kPages * kPageWords / kBigThreads;
  uint32_t sum = 0;
#pragma unroll
  for (uint32_t u = 0; u < per; ++u) sum += __popc(P.bits[t * per + u]);
  uint32_t x = sum;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) P.warp_sum[warp] = x;
  __syncthreads();
  x -= sum;
  for (uint32_t w = 0; w < warp; ++w) x += P.warp_sum[w];
#pragma unroll
  for (uint32_t u = 0; u < per; ++u) {
    P.before[t * per + u] = (uint16_t)x;
    x += __popc(P.bits[t * per + u]);
  }
  __syncthreads();
  return true;
}

// One block per listed cell (looping over the list): up to kBigCell source
// indices ranked by the bitmap above or, when their pages do not fit, sorted
// in shared memory (bitonic, padded to a power of two, one compare-exchange
// per pair index and stage); larger cells by the block-wide radix sort in
// global memory; then the gather.
union BigScratch {
  uint32_t sv[kBigCell];
  PageRanks pages;
  RadixScratch radix;
};

// The large cells, by blocks block, block + blocks, ... of `blocks`.
template <bool GROUPED>
__device__ __forceinline__ void place_large(const RebinArgs& a, BigScratch& sh, uint32_t block,
                                            uint32_t blocks) {
  uint32_t* sv = sh.sv;
  const uint32_t nb = min(a.ctrl->big_count, a.big_cap);
  const CellTable table = new_table<GROUPED>(a);
  uint32_t overflow = 0;
  const uint32_t key_bits = a.n > 1 ? 32u - __clz(a.n - 1) : 1u;
  for (uint32_t w = block; w < nb; w += blocks) {
    const uint32_t k = a.big_list[w];
    uint32_t s0, s1;
    table.span(k, s0, s1);
    s1 = min(s1, a.n);
    if (threadIdx.x == 0) a.counts[k] = 0u;  // read by the scan; zero for the next rebin
    const uint32_t s = s1 > s0 ? s1 - s0 : 0u;
    if (s > kBigCell) {
      const uint32_t* sorted = block_radix_sort(sh.radix, a.idx_tmp + s0, a.idx_alt + s0, s, key_bits);
      for (uint32_t r = threadIdx.x; r < s; r += kBigThreads) place_one<GROUPED>(a, s0 + r, r, sorted[r], k, overflow);
      if (threadIdx.x == 0) atomicAdd(&a.ctrl->huge_cells, 1u);
      __syncthreads();
      continue;
    }
    if (page_ranks(sh.pages, a.idx_tmp + s0, s)) {
      for (uint32_t r = threadIdx.x; r < s; r += kBigThreads) {
        const uint32_t idx = a.idx_tmp[s0 + r], at = page_word(sh.pages, idx);
        const uint32_t rank =
            sh.pages.before[at] + __popc(sh.pages.bits[at] & ((1u << (idx & 31u)) - 1u));
        place_one<GROUPED>(a, s0 + rank, rank, idx, k, overflow);
      }
      __syncthreads();
      continue;
    }
    __syncthreads();  // the sort reuses the ranks' memory
    uint32_t P = 1;
    while (P < s) P <<= 1;
    for (uint32_t r = threadIdx.x; r < P; r += kBigThreads)
      sv[r] = r < s ? a.idx_tmp[s0 + r] : 0xFFFFFFFFu;
    __syncthreads();
    for (uint32_t len = 2; len <= P; len <<= 1) {
      for (uint32_t j = len >> 1; j > 0; j >>= 1) {
        for (uint32_t pi = threadIdx.x; pi < P / 2; pi += kBigThreads) {
          // j is a power of two: r = 2 j floor(pi / j) + pi mod j
          const uint32_t r = ((pi & ~(j - 1u)) << 1) | (pi & (j - 1u)), o = r + j;
          const uint32_t x = sv[r], y = sv[o];
          if ((x > y) == ((r & len) == 0)) {
            sv[r] = y;
            sv[o] = x;
          }
        }
        __syncthreads();
      }
    }
    for (uint32_t r = threadIdx.x; r < s; r += kBigThreads) place_one<GROUPED>(a, s0 + r, r, sv[r], k, overflow);
    __syncthreads();
  }
  add_overflow(a, overflow);
}

// The place steps: the first big_blocks blocks take the large cells, which
// last longest, the others the small ones' slots.  In one launch the two run
// side by side without a second stream's fork and join, and its blocks wait
// their turn behind the scatter's (on a stream of their own the large cells'
// blocks came after those of a place launch that overlaps the scatter: the
// collapsed 1M lattice 101 -> 107 us).  Eight blocks per SM (kBigBlocksPerSm), so
// at most 32 registers.
template <bool GROUPED>
__global__ void __launch_bounds__(kBigThreads, 8) k_cs_place(RebinArgs a, uint32_t big_blocks) {
  __shared__ BigScratch sh;
  begin_after();
  // an upload that is refused leaves the frame as it is
  if (a.fits_only && new_table<GROUPED>(a).start(a.ncells) > a.dst_capacity) return;
  if (blockIdx.x < big_blocks)
    place_large<GROUPED>(a, sh, blockIdx.x, big_blocks);
  else
    place_slot<GROUPED>(a, (blockIdx.x - big_blocks) * kBigThreads + threadIdx.x);
}

}  // namespace

cudaError_t launch_untake(const uint32_t* run_if, const uint32_t* keys, uint32_t n,
                          const CountDev& c, int sms, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const uint32_t need = (n + 255) / 256, few = (uint32_t)(sms > 0 ? sms : 1) * 4u;
  k_cs_untake<<<need < few ? need : few, 256, 0, st>>>(run_if, keys, n, c,
                                                       (c.ncells + kScanTile - 1) / kScanTile);
  return cudaGetLastError();
}

cudaError_t launch_count_sort_step(const RebinArgs& a, int step, uint32_t big_blocks,
                                   cudaStream_t st, bool* launched) {
  const uint32_t ntiles = (a.ncells + kScanTile - 1) / kScanTile;
  const uint32_t nblk = (a.n + 255) / 256;
  *launched = true;
  if (step == kScan) {
    RebinArgs b = a;
    b.prefixed_tiles = ntiles > kPrefixTiles ? ntiles : 0u;
    if (b.prefixed_tiles) {
      const cudaError_t e =
          launch_after(k_cs_tile_prefix, (ntiles + kRun - 1) / kRun, kRun, st, b, ntiles);
      if (e != cudaSuccess) return e;
    }
    return a.groups_new ? launch_after(k_cs_scan_groups, ntiles, kGroupThreads, st, b)
                        : launch_after(k_cs_scan, ntiles ? ntiles : 1u, kScanThreads, st, b);
  } else if (!nblk) {
    *launched = false;
    return cudaSuccess;
  } else if (step == kScatter) {
    return launch_after(a.groups_new ? k_cs_scatter<true> : k_cs_scatter<false>, nblk, 256, st, a,
                        ntiles);
  } else {
    // at most n / (kSmallCell + 1) cells are large
    const uint32_t large = min(big_blocks ? big_blocks : 1u, a.n / (kSmallCell + 1) + 1);
    const uint32_t big = step == kPlaceSmall ? 0u : large;
    const uint32_t small = step == kPlaceLarge ? 0u : nblk;
    return launch_after(a.groups_new ? k_cs_place<true> : k_cs_place<false>, big + small,
                        kBigThreads, st, a, big);
  }
  return cudaGetLastError();
}

uint32_t count_sort_launches(uint32_t n, uint32_t ncells) {
  const uint32_t ntiles = (ncells + kScanTile - 1) / kScanTile;
  return (n ? 3u : 1u) + (ntiles > kPrefixTiles ? 1u : 0u);
}

}  // namespace wrach
