// Solve kernels: the collision/constraint pass plus the fused
// integrate + boundary + velocity-clamp epilogue, which also emits each
// particle's next cell key for the rebin.
//
// Reference-mode kernel: one lane per particle, the sequential sweep of
// World::physics_for_cell (shaders/physics/src/cell.rs:52-95) as a wavefront.
// Extended-mode kernels: one thread per taking-part particle (compacted), a
// Jacobi iteration over the particle's 3x3 cell neighbourhood; the last
// iteration one thread per particle.
#include <algorithm>

#include "wrach_internal.cuh"
#include "wrach_kernels.h"

namespace wrach {

namespace {

// The worlds as a kernel's argument.  With one world (ONE) its settings come
// with the launch, in the constant bank: no loads ahead of the first use and no
// registers held.
template <bool ONE>
struct Worlds;
template <>
struct Worlds<true> {
  WorldDev w;
  __device__ __forceinline__ const WorldDev& of(uint32_t) const { return w; }
};
template <>
struct Worlds<false> {
  const WorldDev* all;
  int n;
  __device__ __forceinline__ const WorldDev& of(uint32_t c) const {
    return all[world_of_cell(all, n, c)];
  }
};

// Next cell of a solved particle (assets/shaders/particles_per_cell.wgsl:
// 14-27), the key the rebin sorts by.
__device__ __forceinline__ uint32_t next_key(const WorldDev& w, float px,
                                             float py, uint32_t& flags) {
  const uint32_t ncx = axis_cell(px, w.ax, w.cs, w.gx, flags);
  const uint32_t ncy = axis_cell(py, w.ay, w.cs, w.gy, flags);
  return w.cell_off + ncy * w.gx + ncx;
}

__device__ __forceinline__ void publish_flags(Ctrl* ctrl, uint32_t flags) {
  const uint32_t wf = warp_or_u32(flags);
  if ((threadIdx.x & 31) == 0 && wf) atomicOr(&ctrl->flags, wf);
}

// Reference mode, one lane per particle.
//  - Particles::new: the first m = min(count, capacity) particles of a cell
//    (shaders/physics/src/particles.rs:31-59)
//  - Particles::pairs / push_close_particles_apart: Gauss-Seidel over i < j
//    (particles.rs:62-93)
//  - Particles::finish: integrate, boundaries, clamp, write (particles.rs:
//    96-107, particle.rs:40-106)
//  - handle_overflown_particles: the rest only integrate (cell.rs:79-95)
// and the rebin's tickets.
//
// A cell's m particles sit in m neighbouring lanes of one warp, and the sweep
// over its pairs runs as a wavefront: turn t takes the pairs i + j = t, which
// have no particle in common, and a pair's turn comes after every pair of the
// sweep that changes one of its two particles before it.  So 2 m - 3 turns
// serve m (m - 1) / 2 pairs, with a particle's position in its lane's
// registers (one thread per cell held them in indexed arrays, in local
// memory, and swept them one by one).  A pair's two lanes both compute its
// push, from the same difference as the reference: p_i - (p_j - p_i) f and
// p_j + (p_j - p_i) f (with the other difference, two coordinates of -0 would
// both stay -0, where the reference's j becomes +0).
//
// Warp w covers the particles [W w, W w + 32), W = 33 - capacity: it solves
// the cells that start in its first W particles (all their m particles are in
// its lanes), and integrates the particles past a cell's capacity among its
// first W.  1M particles, cell size 1: 36 us and a separate ticket launch of
// 14 us before, 21 us with the tickets now.
template <bool ONE>
__global__ void __launch_bounds__(512, 3)
k_solve_reference(const __grid_constant__ Worlds<ONE> worlds, PhysDev ph, uint32_t n,
                  const CellTable table, const uint32_t* __restrict__ cell_of,
                  const float2* __restrict__ pin, const float2* __restrict__ vin,
                  float2* __restrict__ pout, float2* __restrict__ vout,
                  uint32_t* __restrict__ keys, Ctrl* ctrl, CountDev count) {
  begin_after();
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (blockIdx.x == 0 && threadIdx.x == 0) ctrl->big_count = 0u;  // listed afresh by the scan
  const uint32_t own = 33u - ph.cap, first = warp * own, i = first + lane;
  if (first >= n) return;
  uint32_t flags = 0, key = count.ncells, rank = 0, m = 0;
  float px = 0.f, py = 0.f;
  float2 v = make_float2(0.f, 0.f);
  bool mine = i < n;
  const uint32_t c = mine ? cell_of[i] : 0u;
  const WorldDev& w = worlds.of(c);
  if (mine) {
    uint32_t s, e;
    table.span(c, s, e);
    rank = i - s;
    m = min(e - s, ph.cap);
    mine = rank < m ? s >= first && s - first < own : lane < own;
    if (mine) {
      const float2 p = pin[i];
      v = vin[i];
      px = p.x;
      py = p.y;
      // the counters that the ticket will most likely touch
      prefetch_l2(count.counts + c);
      prefetch_l2(count.counts + (c >= w.gx ? c - w.gx : c));
      prefetch_l2(count.counts + min(c + w.gx, count.ncells - 1));
    }
  }
  if (!mine || rank >= m) m = 0;
  const uint32_t most = __reduce_max_sync(0xffffffffu, m);
  for (uint32_t t = 1; t + 3 <= 2 * most; ++t) {
    const uint32_t other = t - rank;  // wraps past m when t < rank
    const bool pair = other < m && other != rank;
    const uint32_t from = (lane + other - rank) & 31u;
    const float qx = __shfl_sync(0xffffffffu, px, from), qy = __shfl_sync(0xffffffffu, py, from);
    const bool second = rank > other;
    const float dx = second ? __fsub_rn(px, qx) : __fsub_rn(qx, px);
    const float dy = second ? __fsub_rn(py, qy) : __fsub_rn(qy, py);
    float f;
    if (pair && push_factor(dx, dy, ph.min_d, ph.skip_d2, f)) {
      const float mx = __fmul_rn(dx, f), my = __fmul_rn(dy, f);
      px = __fadd_rn(px, second ? mx : -mx);
      py = __fadd_rn(py, second ? my : -my);
    }
  }
  if (mine) {
    px = __fadd_rn(px, v.x);
    py = __fadd_rn(py, v.y);
    enforce_limits(w, ph.vmax, px, py, v.x, v.y);
    pout[i] = make_float2(px, py);
    vout[i] = v;
    key = next_key(w, px, py, flags);
    keys[i] = key;
  }
  const uint32_t tk = warp_ticket(key, count.ncells, count.counts, count.tile_sums,
                                  count.tile_shift, count.cap, count.tile_sums_cap);
  if (mine) count.ticket[i] = tk;
  publish_flags(ctrl, flags);
}

// Extended mode (3x3 cells, Jacobi iterations, gravity).  As in the
// reference (cell.rs:29-30, 79-95) only the first `cap` particles of a cell
// take part in the pushes, as pushed particles and as neighbours; the rest of
// an over-full cell keep their position.  The neighbour order is fixed (the
// 3x3 cells in row-major order, table order inside a cell), so each
// particle's push sum is deterministic.
//
// The iterations run over the compacted taking-part particles: there a
// neighbour row of the 3x3 search is one contiguous range [taking(row + x0),
// taking(row + x1 + 1)) whatever the cells' occupancy, and the particles that
// take no part cost nothing.

// The candidates of one particle: the compacted starts of its three
// neighbour rows, and packed their lengths (6 bits each, at most 3 * 16) and
// the particle's own place in the middle row (6 bits).
struct Rows {
  uint32_t s0, s1, s2, len;
  __device__ uint32_t start(int r) const { return r == 0 ? s0 : r == 1 ? s1 : s2; }
  __device__ uint32_t length(int r) const { return (len >> (6 * r)) & 63u; }
  __device__ uint32_t particle() const { return s1 + (len >> 18); }
};
static_assert(3 * kMaxCellCapacity < 64, "row lengths fit 6 bits");

// The rows of the compacted particle t of cell c.
__device__ __forceinline__ Rows tp_rows(const WorldDev& w, const CellTable& table, uint32_t c,
                                        uint32_t t) {
  uint32_t rs[3], re[3];
  neighbour_rows(w, table, c, rs, re);
  return Rows{rs[0], rs[1], rs[2],
              (re[0] - rs[0]) | ((re[1] - rs[1]) << 6) | ((re[2] - rs[2]) << 12) |
                  ((t - rs[1]) << 18)};
}

// Candidates are read two per 16-byte load from an even index, kStep per
// step: a row's marks have one bit per index from its start rounded down to
// even, and up to kStep - 1 indices past its end are read (and unmarked).
constexpr uint32_t kStep = 4;
static_assert(kStep - 1 <= kRowPad, "the iterates are padded for the last step");

// One step of a row: the candidates c[0 .. kStep - 1] within reach of the
// particle at qi2 (a NaN distance counts, as in the reference's test).
struct RowStep {
  ulonglong2 c[kStep / 2];
  __device__ __forceinline__ void load(const f32x2* __restrict__ p) {
#pragma unroll
    for (uint32_t u = 0; u < kStep / 2; ++u) c[u] = reinterpret_cast<const ulonglong2*>(p)[u];
  }
  __device__ __forceinline__ uint32_t marks(const PhysDev& ph, f32x2 qi2) const {
    uint32_t in = 0;
#pragma unroll
    for (uint32_t u = 0; u < kStep / 2; ++u) {
      if (!(f2_len2(f2_sub(c[u].x, qi2)) >= ph.skip_d2)) in |= 1u << (2 * u);
      if (!(f2_len2(f2_sub(c[u].y, qi2)) >= ph.skip_d2)) in |= 2u << (2 * u);
    }
    return in;
  }
};

// The marks of the three rows' candidates.  Mask holds the bits of a row:
// 3 * cap + 1.  The rows' first steps are loaded together; few rows of sparse
// frames need a second.  FEW: the further steps of the three rows side by
// side, two of each at a time, for grids so small that a scheduler has a warp
// or two and every wait for a load shows.
template <typename Mask>
struct Marks {
  Mask m[3];
};
template <typename Mask, bool FEW>
__device__ __forceinline__ Marks<Mask> all_marks(const PhysDev& ph, const f32x2* __restrict__ q,
                                                 f32x2 qi2, const Rows& R) {
  Marks<Mask> M;
  RowStep first[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) first[r].load(q + (R.start(r) & ~1u));
#pragma unroll
  for (int r = 0; r < 3; ++r) M.m[r] = first[r].marks(ph, qi2);
  if constexpr (FEW) {
    uint32_t end[3], most = 0;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      end[r] = (R.start(r) & 1u) + R.length(r);
      most = max(most, end[r]);
    }
    for (uint32_t k0 = kStep; k0 < most; k0 += 2 * kStep) {
      RowStep more[3][2];
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (uint32_t k = k0; k < k0 + 2 * kStep; k += kStep)
          if (k < end[r]) more[r][(k - k0) / kStep].load(q + ((R.start(r) & ~1u) + k));
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (uint32_t k = k0; k < k0 + 2 * kStep; k += kStep)
          if (k < end[r]) M.m[r] |= (Mask)more[r][(k - k0) / kStep].marks(ph, qi2) << k;
    }
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const uint32_t s = R.start(r), n = R.length(r), odd = s & 1u;
    if constexpr (!FEW) {
      for (uint32_t k = kStep; k < odd + n; k += kStep) {
        RowStep more;
        more.load(q + (s - odd + k));
        M.m[r] |= (Mask)more.marks(ph, qi2) << k;
      }
    }
    // the row alone, without the particle itself
    M.m[r] &= (((Mask)1 << n) - 1) << odd;
    if (r == 1) M.m[r] &= ~((Mask)1 << (R.particle() - (s - odd)));
  }
  return M;
}

__device__ __forceinline__ uint32_t low_bit(uint32_t m) { return __ffs((int)m) - 1; }
__device__ __forceinline__ uint32_t low_bit(uint64_t m) { return __ffsll((long long)m) - 1; }

// The marked candidates in order, one after the other: `cur` holds the marks
// left of the row at `base`, and is empty only when no marks are left.
template <typename Mask>
struct MarkWalk {
  Mask cur, next1, next2;
  uint32_t base, base1, base2;
  __device__ __forceinline__ MarkWalk(const Rows& R, const Marks<Mask>& M)
      : cur(M.m[0]), next1(M.m[1]), next2(M.m[2]), base(R.s0 & ~1u), base1(R.s1 & ~1u),
        base2(R.s2 & ~1u) {
    if (!next1) advance1();
    if (!cur) advance();
  }
  __device__ __forceinline__ void advance1() {
    next1 = next2;
    base1 = base2;
    next2 = 0;
  }
  __device__ __forceinline__ void advance() {
    cur = next1;
    base = base1;
    advance1();
  }
  __device__ __forceinline__ uint32_t take() {
    const uint32_t j = base + low_bit(cur);
    cur &= cur - 1;
    if (!cur) advance();
    return j;
  }
};

// The reference's push by the marked candidates, in candidate order, summed
// into (ax, ay), in one loop over the three rows' marks, so that a lane moves
// on to its next row without waiting for the warp's other lanes to finish the
// current one.  Two marks a turn: their factors are paired arithmetic, and the
// loop's own instructions serve both (4M particles in dense clusters, frame
// 8: the three iterations 203, 176 and 227 us with one mark a turn and the
// general square root and division, 181, 157 and 135 us now).  FEW: four a
// turn, whose chains of arithmetic run side by side.  METRICS: pen = the
// deepest overlap min_d - distance with a pushing neighbour.
template <typename Mask, bool METRICS, bool FEW>
__device__ __forceinline__ void push_marked(const PhysDev& ph, const f32x2* __restrict__ q,
                                            f32x2 qi2, const Rows& R, const Marks<Mask>& M,
                                            float& ax, float& ay, float& pen) {
  MarkWalk<Mask> walk(R, M);
  constexpr int turn = FEW ? 4 : 2;
  while (walk.cur) {
    uint32_t j[turn];
    int many = 1;
    j[0] = walk.take();
#pragma unroll
    for (int u = 1; u < turn; ++u) {
      j[u] = j[0];
      if (walk.cur) {
        j[u] = walk.take();
        ++many;
      }
    }
    f32x2 d[turn];
    float s[turn], f[turn], e[turn];
#pragma unroll
    for (int u = 0; u < turn; ++u) d[u] = f2_sub(q[j[u]], qi2);
#pragma unroll
    for (int u = 0; u < turn; ++u) s[u] = f2_len2(d[u]);
    push_factors_near<turn>(s, ph, f, e);
#pragma unroll
    for (int u = 0; u < turn; ++u) {
      if (u == 0 || u < many) {
        if (METRICS) pen = fmaxf(pen, __fsub_rn(ph.min_d, e[u]));
        // scalar: a paired multiply feeding a paired add may be fused
        ax = __fadd_rn(ax, __fmul_rn(f2_x(d[u]), f[u]));
        ay = __fadd_rn(ay, __fmul_rn(f2_y(d[u]), f[u]));
      }
    }
  }
}

// An iteration's push by all candidates in reach.  Where the cell capacity
// allows rows of more marks than 32 bits, most warps have none: they take the
// 32-bit walk (300,000 particles, capacity 16, six passes: 67.7 us a frame
// with 64-bit marks throughout, 63.2 now; at 5 a cell 94.7 and 87.9; with all
// cells past 10, where nearly no warp does, 139.7 and 141.0).  The last pass
// keeps its one walk: it gains nothing from a second.
template <typename Mask, bool FEW>
__device__ __forceinline__ void push_all(const PhysDev& ph, const f32x2* __restrict__ q, f32x2 qi2,
                                         const Rows& R, float& ax, float& ay) {
  float pen = 0.f;
  if constexpr (sizeof(Mask) > 4) {
    // no length has bit 5: 31 candidates and an odd start are 32 marks
    if (!__any_sync(__activemask(), (R.len & 0x20820u) != 0u)) {
      push_marked<uint32_t, false, FEW>(ph, q, qi2, R, all_marks<uint32_t, FEW>(ph, q, qi2, R), ax,
                                        ay, pen);
      return;
    }
  }
  push_marked<Mask, false, FEW>(ph, q, qi2, R, all_marks<Mask, FEW>(ph, q, qi2, R), ax, ay, pen);
}

// One Jacobi iteration but the last, one thread per compacted (taking-part)
// particle: q' = q - push sum, over the compacted count (a
// grid-stride loop; the plain frames' grid covers every particle of the
// frame, so each thread takes one or none).  A launch whose `run_if` flag
// reads 0 returns at once.
// ROWS 0: the neighbour rows from the cell table; 1: also written to
// `rows`; 2: read from `rows` (the cell and its world are then not needed).
// At most 42 registers (three blocks of 512): the loads' latency needs the
// warps.  On the 1M lattice an iteration issues about 60% of the time and
// waits for its gathers through L1 for the rest.
template <typename Mask, int ROWS, bool ONE, bool FEW>
__global__ void __launch_bounds__(512, FEW ? 1 : 3)
k_jacobi_tp(const __grid_constant__ Worlds<ONE> worlds, PhysDev ph, uint32_t ncells,
            const CellTable table, const uint32_t* __restrict__ tp_cell,
            const float2* __restrict__ qin, float2* __restrict__ qout,
            const uint32_t* __restrict__ run_if, uint4* __restrict__ rows) {
  // the table is older than the kernel before (RebinOrder): blocks without a
  // particle (on a piled-up floor, most) end at once; block 0 always has one
  const uint32_t ntp = table.taking(ncells);
  if (blockIdx.x * blockDim.x >= ntp && blockIdx.x != 0) return;
  begin_after();
  if (run_if && *run_if == 0u) return;
  const f32x2* __restrict__ q = reinterpret_cast<const f32x2*>(qin);
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < ntp; t += gridDim.x * blockDim.x) {
    Rows R;
    if (ROWS == 2) {
      const uint4 u = rows[t];
      R = Rows{u.x, u.y, u.z, u.w};
    } else {
      const uint32_t c = tp_cell[t];
      R = tp_rows(worlds.of(c), table, c, t);
      if (ROWS == 1) rows[t] = make_uint4(R.s0, R.s1, R.s2, R.len);
    }
    const f32x2 qi2 = q[t];
    float ax = 0.f, ay = 0.f;
    push_all<Mask, FEW>(ph, q, qi2, R, ax, ay);
    qout[t] = make_float2(__fsub_rn(f2_x(qi2), ax), __fsub_rn(f2_y(qi2), ay));
  }
}

// The last iteration, one thread per frame particle (a grid-stride loop
// over whole blocks of particles; the plain frames' grid covers them all):
// the push (taking-part particles, from the compacted iterate q; ROWS 2: by
// the neighbour rows that the iterations wrote, 0: from the cell table),
// then gravity, integration, boundaries, the velocity clamp and the key
// emission, and the rebin's tickets.  METRICS also writes the block's sums
// for the surrogate's fallback gate to part[blockIdx.x * 8 + k]: [0] sum and
// [1] max over taking-part particles of the deepest overlap max(0, min_d -
// distance) with a pushing neighbour (measured on the pass's input), [2] the
// number of taking-part particles, [3] the kinetic energy of the output and
// [4] the kinetic energy a plain frame gives (gravity, the clamp and wall
// reflections only change the velocity).  A launch whose `run_if` flag reads
// 0 returns at once.
// Three blocks of 512 an SM with METRICS too: with 64 registers and two blocks a
// surrogate frame of the 1M lattice takes 193.0 us, with 40 registers 189.2.
template <typename Mask, int ROWS, bool METRICS, bool ONE, bool FEW>
__global__ void __launch_bounds__(512, FEW ? 1 : 3)
k_jacobi_final(const __grid_constant__ Worlds<ONE> worlds, PhysDev ph, uint32_t n,
               int do_push, const CellTable table, const uint32_t* __restrict__ tp_of,
               const uint32_t* __restrict__ cell_of, const uint4* __restrict__ rows,
               const float2* __restrict__ pin, const float2* __restrict__ qtp,
               float2* __restrict__ pout, const float2* __restrict__ vin,
               float2* __restrict__ vout, uint32_t* __restrict__ keys, Ctrl* ctrl,
               const uint32_t* __restrict__ run_if, float* __restrict__ part, CountDev count) {
  begin_after();
  if (run_if && *run_if == 0u) return;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // taking the tickets: the rebin's scan lists its large cells afresh
  if (count.ticket && blockIdx.x == 0 && threadIdx.x == 0) ctrl->big_count = 0u;
  uint32_t flags = 0;
  float pen = 0.f, taking = 0.f, ke = 0.f, ke_plain = 0.f;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    const bool live = i < n;
    uint32_t key = count.ncells;  // no cell
    if (live) {
      const uint32_t t = tp_of[i], c = cell_of[i];
      const WorldDev& w = worlds.of(c);
      // the velocity and, for the tickets' atomics, the counters of the
      // particle's cell and of the cells above and below it (its next cell
      // is almost always among their lines) are fetched before the push
      const float2 v = vin[i];
      if (count.ticket) {
        prefetch_l2(count.counts + c);
        prefetch_l2(count.counts + (c >= w.gx ? c - w.gx : c));
        prefetch_l2(count.counts + min(c + w.gx, count.ncells - 1));
      }
      float qx, qy;
      if (t != kNoTp) {
        if (METRICS) taking = __fadd_rn(taking, 1.f);
        const f32x2* __restrict__ q = reinterpret_cast<const f32x2*>(qtp);
        const f32x2 qi2 = q[t];
        float ax = 0.f, ay = 0.f;
        if (do_push) {
          Rows R;
          if (ROWS == 2) {
            const uint4 u = rows[t];
            R = Rows{u.x, u.y, u.z, u.w};
          } else {
            R = tp_rows(w, table, c, t);
          }
          push_marked<Mask, METRICS, FEW>(ph, q, qi2, R, all_marks<Mask, FEW>(ph, q, qi2, R), ax, ay,
                                          pen);
        }
        qx = __fsub_rn(f2_x(qi2), ax);
        qy = __fsub_rn(f2_y(qi2), ay);
      } else {
        const float2 p = pin[i];
        qx = p.x;
        qy = p.y;
      }
      float ux = v.x, uy = __fsub_rn(v.y, ph.gravity);
      float px = __fadd_rn(qx, ux), py = __fadd_rn(qy, uy);
      enforce_limits(w, ph.vmax, px, py, ux, uy);
      pout[i] = make_float2(px, py);
      vout[i] = make_float2(ux, uy);
      key = next_key(w, px, py, flags);
      keys[i] = key;
      if (METRICS) {
        ke = __fadd_rn(ke, __fmul_rn(0.5f, __fadd_rn(__fmul_rn(ux, ux), __fmul_rn(uy, uy))));
        const float cx = fminf(fmaxf(v.x, -ph.vmax), ph.vmax);
        const float cy = fminf(fmaxf(__fsub_rn(v.y, ph.gravity), -ph.vmax), ph.vmax);
        ke_plain = __fadd_rn(ke_plain,
                             __fmul_rn(0.5f, __fadd_rn(__fmul_rn(cx, cx), __fmul_rn(cy, cy))));
      }
    }
    if (count.ticket) {
      // the rebin's tickets (every lane of the warp takes part)
      const uint32_t tk = warp_ticket(key, count.ncells, count.counts, count.tile_sums,
                                      count.tile_shift, count.cap, count.tile_sums_cap);
      if (live) count.ticket[i] = tk;
    }
  }
  publish_flags(ctrl, flags);
  if (METRICS) {
    // warp sums, then one thread sums the block's warps in a fixed order
    __shared__ float red[16][5];
    float v[5] = {pen, pen, taking, ke, ke_plain};
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const float u = __shfl_xor_sync(0xffffffffu, v[k], o);
        v[k] = k == 1 ? fmaxf(v[k], u) : __fadd_rn(v[k], u);
      }
    }
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < 5; ++k) red[warp][k] = v[k];
    __syncthreads();
    if (threadIdx.x < 5) {
      const uint32_t nw = (blockDim.x + 31) >> 5;
      float acc = red[0][threadIdx.x];
      for (uint32_t wi = 1; wi < nw; ++wi)
        acc = threadIdx.x == 1 ? fmaxf(acc, red[wi][threadIdx.x]) : __fadd_rn(acc, red[wi][threadIdx.x]);
      part[blockIdx.x * 8 + threadIdx.x] = acc;
    }
  }
}

// Every squared distance that the short push factor serves, two at a time,
// against the general square root and division: counts[0] += compared,
// counts[1] += of them, root or factor with other bits.
__global__ void __launch_bounds__(256) k_push_check(PhysDev ph, uint32_t first, uint32_t end,
                                                    unsigned long long* __restrict__ counts) {
  unsigned long long compared = 0, wrong = 0;
  const uint64_t stride = 2ull * gridDim.x * blockDim.x;
  for (uint64_t i = first + 2ull * (blockIdx.x * blockDim.x + threadIdx.x); i < end; i += stride) {
    const float s[2] = {__uint_as_float((uint32_t)i), __uint_as_float((uint32_t)i + 1u)};
    float f[2], d[2];
    push_factors_plain(s[0], s[1], ph, f[0], f[1], d[0], d[1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (i + u >= end || push_special(s[u], d[u], ph)) continue;
      float dist;
      const float want = push_factor_general(s[u], ph, dist);
      ++compared;
      wrong += __float_as_uint(want) != __float_as_uint(f[u]) ||
               __float_as_uint(dist) != __float_as_uint(d[u]);
    }
  }
  atomicAdd(&counts[0], compared);
  if (wrong) atomicAdd(&counts[1], wrong);
}

}  // namespace

cudaError_t launch_push_check(const PhysDev& ph, uint32_t first, uint32_t end, int sms,
                              unsigned long long* counts, cudaStream_t st) {
  if (first >= end) return cudaSuccess;
  k_push_check<<<(sms > 0 ? sms : 1) * 8, 256, 0, st>>>(ph, first, end, counts);
  return cudaGetLastError();
}

cudaError_t launch_solve_reference(const SolveArgs& a, cudaStream_t st) {
  if (a.n == 0) return cudaSuccess;
  const uint32_t threads = a.block ? a.block : 128;
  const uint32_t own = (33u - a.ph.cap) * (threads / 32);
  const uint32_t blocks = (a.n + own - 1) / own;
  if (a.nworlds == 1)
    return launch_after(k_solve_reference<true>, blocks, threads, st, Worlds<true>{a.world}, a.ph,
                        a.n, a.table, a.cell_of, a.pos, a.vel, a.pos_out, a.vel_out, a.keys,
                        a.ctrl, a.count);
  return launch_after(k_solve_reference<false>, blocks, threads, st,
                      Worlds<false>{a.worlds, a.nworlds}, a.ph, a.n, a.table, a.cell_of, a.pos,
                      a.vel, a.pos_out, a.vel_out, a.keys, a.ctrl, a.count);
}

uint32_t solve_blocks(const SolveArgs& a) {
  const uint32_t threads = a.block ? a.block : 128;
  const uint32_t per = a.per_thread ? a.per_thread : 1u;
  const uint32_t blocks = (a.n + threads * per - 1) / (threads * per);
  // a launch that usually returns at once (the surrogate's fallback) strides
  // over the frame with a few blocks per SM, so that skipping it is cheap
  const uint32_t few = (uint32_t)(a.sms > 0 ? a.sms : 1) * (1024u / threads);
  return a.run_if && blocks > few ? few : blocks;
}

// A row's marks fit 32 bits: its candidates and one more for an odd start.
static bool narrow_marks(const PhysDev& ph) { return 3 * ph.cap + 1 <= 32; }

template <typename Mask, int ROWS, bool FEW>
static cudaError_t launch_iteration(const SolveArgs& a, uint32_t blocks, uint32_t threads,
                                    const float2* qin, float2* qout, cudaStream_t st) {
  if constexpr (ROWS != 2) {
    if (a.nworlds != 1)
      return launch_after(k_jacobi_tp<Mask, ROWS, false, FEW>, blocks, threads, st,
                          Worlds<false>{a.worlds, a.nworlds}, a.ph, a.ncells, a.table, a.tp_cell,
                          qin, qout, a.run_if, a.rows);
  }
  // the rows read back need no world
  return launch_after(k_jacobi_tp<Mask, ROWS, true, FEW>, blocks, threads, st, Worlds<true>{a.world},
                      a.ph, a.ncells, a.table, a.tp_cell, qin, qout, a.run_if, a.rows);
}

// Up to two blocks of 128 per SM, the kernels with more loads and pushes in
// flight per thread (their 108 registers leave 16 warps an SM): 16,384
// particles piled up, 35.0 -> 31.0 us a frame, 32,768 39.0 -> 34.8, spread out
// 20.7 and 24.0 either way.  From 2,000 to 38,900 particles (the rule's end on
// 152 SMs), 0.06 and 0.48 of them per px^2 and two to six iterations, frames take
// 0 to 13% less spread out and 0 to 16% less piled up.  65,536 42.8 -> 40.2, but
// spread out 26.8 -> 28.3, and 262,144 52 -> 62.
static bool few_particles(const SolveArgs& a) {
  return narrow_marks(a.ph) && !a.part && a.n <= (uint32_t)(a.sms > 0 ? a.sms : 1) * 256u;
}

template <typename Mask, bool FEW>
static cudaError_t launch_iteration(const SolveArgs& a, uint32_t blocks, uint32_t threads,
                                    const float2* qin, float2* qout, cudaStream_t st) {
  const int mode = a.rows ? a.rows_mode : 0;
  if (mode == 1) return launch_iteration<Mask, 1, FEW>(a, blocks, threads, qin, qout, st);
  if (mode == 2) return launch_iteration<Mask, 2, FEW>(a, blocks, threads, qin, qout, st);
  return launch_iteration<Mask, 0, FEW>(a, blocks, threads, qin, qout, st);
}

cudaError_t launch_jacobi_iteration(const SolveArgs& a, const float2* qin, float2* qout,
                                    cudaStream_t st) {
  if (a.n == 0) return cudaSuccess;
  const uint32_t threads = a.block ? a.block : 128;
  // The taking-part particles are few once the floor has piled up, and a
  // block without one still costs its launch: past 9 waves of blocks (108 of
  // 128 threads per SM) the blocks stride instead.  4M particles, 31,250 blocks:
  // 771 -> 765 us spread out, 326 -> 304 us piled up; with 54 per SM 786 and 295.
  // It begins to act at 2.1M on 152 SMs, and from there to 4M frames take 0 to 2%
  // less spread out and 0.5 to 7% less piled up (2.6M: 254 -> 251, 222 -> 216).
  const uint32_t most = (uint32_t)(a.sms > 0 ? a.sms : 1) * (13824u / threads);
  const uint32_t blocks = std::min(solve_blocks(a), most);
  if (few_particles(a)) return launch_iteration<uint32_t, true>(a, blocks, threads, qin, qout, st);
  return narrow_marks(a.ph) ? launch_iteration<uint32_t, false>(a, blocks, threads, qin, qout, st)
                            : launch_iteration<uint64_t, false>(a, blocks, threads, qin, qout, st);
}

template <typename Mask, int ROWS, bool METRICS, bool FEW>
static cudaError_t launch_final(const SolveArgs& a, uint32_t blocks, uint32_t threads,
                                const float2* qtp, int do_push, cudaStream_t st) {
  if (a.nworlds == 1)
    return launch_after(k_jacobi_final<Mask, ROWS, METRICS, true, FEW>, blocks, threads, st,
                        Worlds<true>{a.world}, a.ph, a.n, do_push, a.table, a.tp_of, a.cell_of,
                        a.rows, a.pos, qtp, a.pos_out, a.vel, a.vel_out, a.keys, a.ctrl, a.run_if,
                        a.part, a.count);
  return launch_after(k_jacobi_final<Mask, ROWS, METRICS, false, FEW>, blocks, threads, st,
                      Worlds<false>{a.worlds, a.nworlds}, a.ph, a.n, do_push, a.table, a.tp_of,
                      a.cell_of, a.rows, a.pos, qtp, a.pos_out, a.vel, a.vel_out, a.keys, a.ctrl,
                      a.run_if, a.part, a.count);
}

template <typename Mask>
static cudaError_t launch_final(const SolveArgs& a, uint32_t blocks, uint32_t threads,
                                const float2* qtp, int do_push, cudaStream_t st) {
  const bool rows = a.rows && a.rows_mode == 2;
  if (a.part)
    return rows ? launch_final<Mask, 2, true, false>(a, blocks, threads, qtp, do_push, st)
                : launch_final<Mask, 0, true, false>(a, blocks, threads, qtp, do_push, st);
  if constexpr (sizeof(Mask) == 4) {
    if (few_particles(a))
      return rows ? launch_final<Mask, 2, false, true>(a, blocks, threads, qtp, do_push, st)
                  : launch_final<Mask, 0, false, true>(a, blocks, threads, qtp, do_push, st);
  }
  return rows ? launch_final<Mask, 2, false, false>(a, blocks, threads, qtp, do_push, st)
              : launch_final<Mask, 0, false, false>(a, blocks, threads, qtp, do_push, st);
}

cudaError_t launch_jacobi_final(const SolveArgs& a, const float2* qtp, int do_push,
                                cudaStream_t st) {
  if (a.n == 0) return cudaSuccess;
  const uint32_t threads = a.block ? a.block : 128;
  const uint32_t blocks = solve_blocks(a);
  return narrow_marks(a.ph) ? launch_final<uint32_t>(a, blocks, threads, qtp, do_push, st)
                            : launch_final<uint64_t>(a, blocks, threads, qtp, do_push, st);
}

}  // namespace wrach
