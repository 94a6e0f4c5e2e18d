// The C ABI (include/wrach.h): context lifetime, uploads, the frame loop,
// viewport streaming and readback.  Host orchestration of the kernels in
// solve.cu, count_sort.cu, rebin.cu and viewport.cu; the learned surrogate's
// entry points are in surrogate_host.cu.
//
// Device layout of a context (all worlds concatenated; world w owns the
// global cells [cell_off_w, cell_off_w + gx_w * gy_w) and, in the frame, the
// particles [start(cell_off_w), start(cell_off_w + cells_w))):
//   pos, vel          binned state, float2 x capacity        (cell order)
//   pos_o, vel_o      solve output, float2 x capacity        (same order)
//   q1, q2            extended-mode Jacobi iterates
//   rows              the iterations' neighbour-row ranges per compacted particle
//   cell_of[2]        cell of each binned particle (u32)
//   cs[2], ct[2] or groups[2]
//                     the cell table (CellTable; ping-pong per frame)
//   tp_pos[2], tp_cell[2], tp_of[2]; tp_vel[2] with a surrogate
//                     extended physics: the taking-part particles' positions,
//                     cells and velocities, compacted in cell order, and each
//                     frame particle's place among them
//   keys              next cell of each solve output (u32)
//   kA kB iA iB       rebin scratch (tickets, slot cells, slot sources, sort ping-pong)
//   tile_sums         rebin: particles per tile of 2048 cells (zero between frames)
//   ctrl              counters and sticky flags
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "context_internal.h"

using wrach::Ctrl;
using wrach::PhysDev;
using wrach::WorldDev;
using namespace wrach::host;

namespace {

// Rust's saturating `f32 as i32` (NaN -> 0).
int32_t sat_i32(float f) {
  if (f != f) return 0;
  if (f >= 2147483648.0f) return INT32_MAX;
  if (f <= -2147483648.0f) return INT32_MIN;
  return (int32_t)f;
}

// SpatialBin::get_cell_coord (runners/bevy/src/spatial_bin.rs:48-64).
int32_t cell_coord(float x, uint32_t cs) {
  volatile float d = (float)cs;  // keep the binary32 division
  float q = std::trunc(x / d);
  if (std::fmod(x, (float)d) < 0.0f) q = q - 1.0f;
  return sat_i32(q);
}

// The device's view of `bytes` of host memory at p when all of them lie in one
// pinned allocation that kernels may write to, or null: pageable memory, and
// pinned memory with other flags than portable and mapped (write-combined,
// read-only or I/O memory), go through the copy engine.
uint32_t* device_view(void* p, size_t bytes) {
  if (!p || (uintptr_t)p % 4) return nullptr;
  using GetAttribute = CUresult (*)(void*, CUpointer_attribute, CUdeviceptr);
  static const GetAttribute get = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &f, 12000, cudaEnableDefault,
                                         &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<GetAttribute>(f);
  }();
  cudaPointerAttributes at;
  unsigned flags = 0;
  CUdeviceptr start = 0;
  size_t size = 0;
  if (!get || cudaPointerGetAttributes(&at, p) != cudaSuccess || at.type != cudaMemoryTypeHost ||
      !at.devicePointer || cudaHostGetFlags(&flags, p) != cudaSuccess ||
      (flags & ~(cudaHostAllocPortable | cudaHostAllocMapped)) != 0) {
    cudaGetLastError();
    return nullptr;
  }
  const CUdeviceptr q = (CUdeviceptr)(uintptr_t)p;
  if (get(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, q) != CUDA_SUCCESS ||
      get(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, q) != CUDA_SUCCESS || q < start ||
      q + bytes > start + size)
    return nullptr;
  return static_cast<uint32_t*>(at.devicePointer);
}

__global__ void k_gather_starts(const wrach::CellTable table,
                                const uint32_t* __restrict__ cells, uint32_t n,
                                uint32_t* __restrict__ out) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = table.start(cells[i]);
}

// The smallest binary32 s with sqrt_rn(s) > min_d.  Correctly rounded
// square roots are monotonic, so for every s: s >= skip_threshold(min_d)
// exactly when sqrtf(s) > min_d.
float skip_threshold(float min_d) {
  volatile float s = min_d * min_d;
  while (s > 0.0f && std::sqrt((float)std::nextafter((float)s, 0.0f)) > min_d)
    s = std::nextafter((float)s, 0.0f);
  while (!(std::sqrt((float)s) > min_d)) s = std::nextafter((float)s, INFINITY);
  return s;
}

// The push factor's constants for a minimum distance.  Far from the ends of the
// exponent range every intermediate value of the short push factor is normal;
// other distances take the general code.
void set_push(PhysDev& ph, float min_d) {
  ph.min_d = min_d;
  ph.skip_d2 = skip_threshold(min_d);
  ph.slow_below = min_d >= 0x1p-20f && min_d <= 0x1p20f ? 0x1p-60f : INFINITY;
}

uint32_t bits_for(uint32_t v) {
  uint32_t b = 0;
  while (b < 32 && (v >> b) != 0) ++b;
  return b;
}

}  // namespace


namespace {

void release(WrachContext* ctx) {
  drop_graphs(ctx);
  {
    void* sp[] = {ctx->sur.params, ctx->sur.grad, ctx->sur.mom1, ctx->sur.mom2,
                  ctx->sur.metrics, ctx->sur.bf16, ctx->sur.x, ctx->sur.corr, ctx->sur.tx,
                  ctx->sur.tt, ctx->sur.part, ctx->sur.gate};
    for (void* p : sp) dfree(p);
  }
  void* ptrs[] = {ctx->worlds_d, ctx->pos, ctx->vel, ctx->pos_o, ctx->vel_o,
                  ctx->q1, ctx->q2, ctx->rows, ctx->cell_of[0], ctx->cell_of[1],
                  ctx->cs[0], ctx->cs[1], ctx->keys, ctx->kA, ctx->kB,
                  ctx->iA, ctx->iB, ctx->tile_sums, ctx->ctrl, ctx->big_list,
                  ctx->groups[0], ctx->groups[1], ctx->ct[0], ctx->ct[1], ctx->tp_pos[0], ctx->tp_pos[1], ctx->tp_cell[0],
                  ctx->tp_cell[1], ctx->tp_of[0], ctx->tp_of[1], ctx->tile_sums_cap, ctx->tp_vel[0], ctx->tp_vel[1],
                  ctx->stage_pos, ctx->stage_vel, ctx->table_tmp, ctx->counts, ctx->render_cover, ctx->render_image,
                  ctx->gather_idx, ctx->gather_out, ctx->compact_sums};
  for (void* p : ptrs) dfree(p);
  for (auto& s : ctx->stores) {
    dfree(s.pos);
    dfree(s.vel);
  }
  if (ctx->gather_h) cudaFreeHost(ctx->gather_h);
  if (ctx->sur.grad_h) cudaFreeHost(ctx->sur.grad_h);
  if (ctx->fork_ev) cudaEventDestroy(ctx->fork_ev);
  if (ctx->join_ev) cudaEventDestroy(ctx->join_ev);
  if (ctx->counts_ev) cudaEventDestroy(ctx->counts_ev);
  if (ctx->aux) cudaStreamDestroy(ctx->aux);
  if (ctx->stream) cudaStreamDestroy(ctx->stream);
}

// The buffers below may still be in use by work queued on the context's
// streams (a frame, or the last steps of an upload), so a reallocation waits
// for that work before freeing them.
int ensure_stage(WrachContext* ctx, size_t need) {
  if (need <= ctx->stage_cap) return WRACH_OK;
  size_t cap = std::max(need, ctx->stage_cap * 2);
  CK(cudaStreamSynchronize(ctx->stream));
  CK(cudaStreamSynchronize(ctx->aux));
  ctx->stage_cap = 0;  // until both are there
  dfree(ctx->stage_pos);
  dfree(ctx->stage_vel);
  ctx->stage_pos = ctx->stage_vel = nullptr;
  CK(dalloc(ctx, &ctx->stage_pos, cap));
  CK(dalloc(ctx, &ctx->stage_vel, cap));
  ctx->stage_cap = cap;
  return WRACH_OK;
}

// Particles of one sort: their number is a 32-bit count.
constexpr size_t kMaxStore = 0xFFFFFFF0u;

int ensure_store(WrachContext* ctx, Store& s, size_t need) {
  if (need <= s.cap) return WRACH_OK;
  size_t cap = std::max<size_t>(need, (size_t)s.cap * 2);
  if (cap > kMaxStore) return fail(ctx, WRACH_ERR_CAPACITY, "store too large");
  float2 *np = nullptr, *nv = nullptr;
  CK(dalloc(ctx, &np, cap));
  const cudaError_t e = dalloc(ctx, &nv, cap);
  if (e != cudaSuccess) {
    dfree(np);
    CK(e);
  }
  if (s.n) {
    CK(cudaMemcpyAsync(np, s.pos, s.n * sizeof(float2), cudaMemcpyDeviceToDevice, ctx->stream));
    CK(cudaMemcpyAsync(nv, s.vel, s.n * sizeof(float2), cudaMemcpyDeviceToDevice, ctx->stream));
  }
  CK(cudaStreamSynchronize(ctx->stream));
  CK(cudaStreamSynchronize(ctx->aux));
  dfree(s.pos);
  dfree(s.vel);
  s.pos = np;
  s.vel = nv;
  s.cap = (uint32_t)cap;
  return WRACH_OK;
}

}  // namespace

namespace wrach {
namespace host {

void drop_graphs(WrachContext* ctx) {
  for (auto& g : ctx->graph)
    if (g) {
      cudaGraphExecDestroy(g);
      g = nullptr;
    }
  for (auto& row : ctx->sur.graph)
    for (auto& g : row)
      if (g) {
        cudaGraphExecDestroy(g);
        g = nullptr;
      }
}

int ensure_sort_capacity(WrachContext* ctx, size_t need) {
  if (need <= ctx->sort_cap) return WRACH_OK;
  size_t cap = std::max(need, ctx->sort_cap * 2);
  CK(cudaStreamSynchronize(ctx->stream));
  CK(cudaStreamSynchronize(ctx->aux));
  drop_graphs(ctx);
  ctx->sort_cap = 0;  // until all of them are there
  uint32_t** bufs[] = {&ctx->keys, &ctx->kA, &ctx->kB, &ctx->iA, &ctx->iB, &ctx->big_list};
  for (auto b : bufs) {
    dfree(*b);
    *b = nullptr;
  }
  // at most cap / (kSmallCell + 1) cells can be larger than kSmallCell
  ctx->big_cap = (uint32_t)(cap / (wrach::kSmallCell + 1) + 2);
  for (auto b : bufs) CK(dalloc(ctx, b, b == &ctx->big_list ? ctx->big_cap : cap));
  ctx->sort_cap = cap;
  return WRACH_OK;
}

int fail(WrachContext* c, int code, const std::string& msg) {
  if (c) c->err = msg;
  return code;
}

void dfree(void* p) {
  if (p) cudaFree(p);
}

wrach::SolveArgs solve_args(WrachContext* ctx) {
  wrach::SolveArgs a{};
  a.worlds = ctx->worlds_d;
  a.nworlds = (int)ctx->nworlds;
  a.world = ctx->worlds_h[0];
  a.ph = ctx->ph;
  a.ncells = ctx->ncells;
  a.n = ctx->n;
  a.table = ctx->table(ctx->cur);
  a.cell_of = ctx->cell_of[ctx->cur];
  a.pos = ctx->pos;
  a.vel = ctx->vel;
  a.pos_out = ctx->pos_o;
  a.vel_out = ctx->vel_o;
  a.keys = ctx->keys;
  a.ctrl = ctx->ctrl;
  a.block = ctx->cfg.solve_block;
  a.per_thread = ctx->cfg.solve_per_thread;
  a.tp_cell = ctx->tp_cell[ctx->cur];
  a.tp_of = ctx->tp_of[ctx->cur];
  a.tp_pos = ctx->tp_pos[ctx->cur];
  a.tp_vel = ctx->tp_vel[ctx->cur];
  a.sms = ctx->sms;
  a.rows = ctx->rows;
  return a;
}

wrach::CountDev ticket_args(WrachContext* ctx) {
  return wrach::CountDev{ctx->counts, ctx->tile_sums, ctx->kA, ctx->ncells, wrach::kCountScanShift,
                         ctx->ph.cap, ctx->tile_sums_cap};
}

wrach::RebinArgs rebin_args(WrachContext* ctx) {
  wrach::RebinArgs r{};
  r.worlds = ctx->worlds_d;
  r.nworlds = (int)ctx->nworlds;
  r.ncells = ctx->ncells;
  r.tile_sums = ctx->tile_sums;
  r.kA = ctx->kA;
  r.kB = ctx->kB;
  r.iA = ctx->iA;
  r.iB = ctx->iB;
  r.keys = ctx->keys;
  r.counts = ctx->counts;
  r.ctrl = ctx->ctrl;
  r.ticket = ctx->kA;
  r.idx_tmp = ctx->iA;
  r.cell_tmp = ctx->kB;
  r.idx_alt = ctx->iB;
  r.big_list = ctx->big_list;
  r.big_cap = ctx->big_cap;
  // every rebin writes the next table parity; extended physics also the
  // compacted taking-part particles
  r.cs_new = ctx->cs[ctx->cur ^ 1];
  r.groups_new = ctx->groups[ctx->cur ^ 1];
  r.ct_new = ctx->ct[ctx->cur ^ 1];
  if (ctx->ph.mode == WRACH_MODE_EXTENDED) {
    r.tp_cap = ctx->ph.cap;
    r.tile_sums_cap = ctx->tile_sums_cap;
    r.tp_pos = ctx->tp_pos[ctx->cur ^ 1];
    r.tp_vel = ctx->tp_vel[ctx->cur ^ 1];
    r.tp_cell = ctx->tp_cell[ctx->cur ^ 1];
    r.tp_of = ctx->tp_of[ctx->cur ^ 1];
  }
  return r;
}

}  // namespace host
}  // namespace wrach

namespace {

void mark(WrachContext* ctx) {
  if (ctx->event_hook) cudaEventRecord(ctx->event_hook[ctx->event_count++], ctx->stream);
}

// One frame: solve (1 or `iterations` launches) then the rebin launch.
int enqueue_frame(WrachContext* ctx) {
  wrach::SolveArgs a = solve_args(ctx);
  cudaStream_t st = ctx->stream;
  mark(ctx);
  // the last solve launch takes the rebin's tickets (it computes the keys)
  wrach::SolveArgs fin = a;
  fin.count = ticket_args(ctx);
  if (ctx->ph.mode == WRACH_MODE_REFERENCE) {
    CK(wrach::launch_solve_reference(fin, st));
    mark(ctx);
    ctx->launches += ctx->n ? 1 : 0;
  } else {
    const uint32_t K = ctx->ph.iterations;
    const float2* q = nullptr;
    CK(enqueue_iterations(ctx, a, K > 0 ? K - 1 : 0, st, &q, [&]() { mark(ctx); }));
    fin.rows_mode = K > 1 ? 2 : 0;
    CK(wrach::launch_jacobi_final(fin, q, K > 0 ? 1 : 0, st));
    mark(ctx);
    ctx->launches += ctx->n ? std::max<uint32_t>(K, 1) : 0u;
  }
  CK(enqueue_rebin(ctx, ctx->event_hook != nullptr, [&]() { mark(ctx); }));
  return WRACH_OK;
}

// Steps wrach_profile_frame times in one frame: each solve launch, then the
// scan and the scatter and place steps (an empty frame's solve launches
// nothing, but still marks its steps).
uint32_t frame_steps(const WrachContext* ctx) {
  return std::max<uint32_t>(ctx->ph.iterations, 1) + (ctx->n ? 4u : 1u);
}

// Kernel launches of one frame.
uint32_t frame_launches(const WrachContext* ctx) {
  return (ctx->n ? std::max<uint32_t>(ctx->ph.iterations, 1) : 0u) +
         wrach::count_sort_launches(ctx->n, ctx->ncells);
}

// One frame captured as a CUDA graph, instantiated once per table parity
// (the frame reads cs[parity] and writes cs[parity ^ 1]) and particle count.
int build_graph(WrachContext* ctx) {
  const int parity = ctx->cur;
  const uint64_t launches = ctx->launches;
  cudaGraph_t g = nullptr;
  if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    ctx->graph_ok = false;
    return WRACH_OK;
  }
  int rc = enqueue_frame(ctx);
  cudaError_t e = cudaStreamEndCapture(ctx->stream, &g);
  ctx->cur = parity;
  ctx->launches = launches;
  if (rc != WRACH_OK || e != cudaSuccess || !g) {
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    ctx->graph_ok = false;
    ctx->err.clear();
    return WRACH_OK;
  }
  cudaGraphExec_t exec = nullptr;
  e = cudaGraphInstantiate(&exec, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) {
    cudaGetLastError();
    ctx->graph_ok = false;
    return WRACH_OK;
  }
  ctx->graph[parity] = exec;
  ctx->graph_n[parity] = ctx->n;
  return WRACH_OK;
}

int world_settings_init(WorldDev& w, float width, float height, float ax,
                        float ay, uint32_t cs) {
  std::memset(&w, 0, sizeof(w));
  w.dim_x = width;
  w.dim_y = height;
  w.ax = ax;
  w.ay = ay;
  w.cs = cs;
  volatile float x1 = ax + width, y1 = ay + height;
  w.x1 = x1;
  w.y1 = y1;
  const int32_t blx = cell_coord(ax, cs), bly = cell_coord(ay, cs);
  const int32_t trx = cell_coord(x1, cs), try_ = cell_coord(y1, cs);
  if (trx < blx || try_ < bly) return 1;
  const int64_t gx = (int64_t)trx - blx + 1, gy = (int64_t)try_ - bly + 1;
  if (gx * gy > 0x7FFFFFFFll) return 1;
  w.gx = (uint32_t)gx;
  w.gy = (uint32_t)gy;
  w.blx = blx;
  w.bly = bly;
  // x / gx for every x < 2^31 as (x * m) >> (31 + l), l = ceil(log2 gx),
  // m = floor(2^(31 + l) / gx) + 1 < 2^32 (Granlund & Montgomery, 1994)
  uint32_t l = 0;
  while ((1ull << l) < w.gx) ++l;
  w.div_m = (uint32_t)((1ull << (31 + l)) / w.gx + 1);
  w.div_s = 31 + l;
  return 0;
}

int create_impl(const WrachConfig* config, uint32_t nworlds, const float* dims,
                WrachContext** out) {
  if (!config || !out || nworlds == 0) return WRACH_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  WrachContext* ctx = new (std::nothrow) WrachContext();
  if (!ctx) return WRACH_ERR_OUT_OF_MEMORY;
  ctx->cfg = *config;
  const WrachConfig& c = ctx->cfg;
  auto bad = [&](const char* m) {
    int rc = fail(ctx, WRACH_ERR_INVALID_ARGUMENT, m);
    delete ctx;
    return rc;
  };
  if (c.cell_size == 0) return bad("cell_size must be positive");
  if (c.mode != WRACH_MODE_REFERENCE && c.mode != WRACH_MODE_EXTENDED) return bad("unknown mode");
  if (c.cell_capacity == 0 || c.cell_capacity > wrach::kMaxCellCapacity)
    return bad("cell_capacity must be in 1..16");
  if (!(c.min_distance > 0.0f) || !(c.max_velocity >= 0.0f)) return bad("bad physics constants");
  if (c.iterations > 64) return bad("iterations must be at most 64");
  if (c.solve_block && (c.solve_block > 512 || c.solve_block % 32))
    return bad("solve_block must be a multiple of 32 up to 512");
  if (c.solve_per_thread > 64) return bad("solve_per_thread must be at most 64");

  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    int rc = fail(ctx, WRACH_ERR_UNSUPPORTED, "no CUDA device");
    delete ctx;
    return rc;
  }
  if (c.device < 0 || c.device >= ndev) return bad("device ordinal out of range");
  ctx->device = c.device;
  DeviceGuard guard(ctx->device);
  cudaDeviceProp prop{};
  if (cudaGetDeviceProperties(&prop, ctx->device) != cudaSuccess ||
      !(prop.major == 10 && prop.minor == 3)) {
    int rc = fail(ctx, WRACH_ERR_UNSUPPORTED,
                  std::string("this build targets sm_103a; device is ") + prop.name);
    delete ctx;
    return rc;
  }

  ctx->ph.mode = c.mode;
  ctx->ph.iterations = c.mode == WRACH_MODE_REFERENCE ? 1u : c.iterations;
  ctx->ph.gravity = c.mode == WRACH_MODE_REFERENCE ? 0.0f : c.gravity;
  set_push(ctx->ph, c.min_distance);
  ctx->ph.vmax = c.max_velocity;
  ctx->ph.cap = c.cell_capacity;

  ctx->nworlds = nworlds;
  ctx->worlds_h.resize(nworlds);
  ctx->cap_h.resize(nworlds);
  ctx->n_h.assign(nworlds, 0);
  ctx->poff_h.assign(nworlds, 0);
  ctx->stores.resize(nworlds);
  uint64_t cells = 0, cap = 0;
  for (uint32_t w = 0; w < nworlds; ++w) {
    const float wd = dims ? dims[2 * w] : c.width;
    const float ht = dims ? dims[2 * w + 1] : c.height;
    if (!(wd >= 0.0f) || !(ht >= 0.0f)) return bad("world dimensions must be non-negative");
    if (world_settings_init(ctx->worlds_h[w], wd, ht, c.anchor_x, c.anchor_y, c.cell_size))
      return bad("grid too large");
    WorldDev& wd_ = ctx->worlds_h[w];
    wd_.cell_off = (uint32_t)cells;
    const uint64_t wc = (uint64_t)wd_.gx * wd_.gy;
    cells += wc;
    ctx->max_world_cells = std::max<uint32_t>(ctx->max_world_cells, (uint32_t)wc);
    const uint32_t wcap = c.capacity ? c.capacity
                                     : wrach_max_particles_per_frame((uint32_t)wc, c.cell_size);
    ctx->cap_h[w] = wcap;
    cap += wcap;
    // keys carry a flag in bit 31, so cell indices stay below 2^31
    if (cells > 0x7FFFFFF0ull || cap > 0x7FFFFFFFull) return bad("grid or capacity too large");
  }
  ctx->ncells = (uint32_t)cells;
  ctx->total_cap = (uint32_t)cap;

  auto oom = [&](cudaError_t e) {
    int rc = fail(ctx, e == cudaErrorMemoryAllocation ? WRACH_ERR_OUT_OF_MEMORY : WRACH_ERR_CUDA,
                  std::string("allocation: ") + cudaGetErrorString(e));
    cudaGetLastError();
    release(ctx);
    delete ctx;
    return rc;
  };
  cudaError_t e;
  if ((e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking)) != cudaSuccess) return oom(e);
  if ((e = cudaStreamCreateWithFlags(&ctx->aux, cudaStreamNonBlocking)) != cudaSuccess) return oom(e);
  if ((e = cudaEventCreateWithFlags(&ctx->fork_ev, cudaEventDisableTiming)) != cudaSuccess) return oom(e);
  if ((e = cudaEventCreateWithFlags(&ctx->join_ev, cudaEventDisableTiming)) != cudaSuccess) return oom(e);
  if ((e = cudaEventCreateWithFlags(&ctx->counts_ev, cudaEventDisableTiming)) != cudaSuccess) return oom(e);
  const size_t tc = ctx->total_cap;
  // the worlds, then (batches) the first world of each tile of cells
  const size_t tiles_words = nworlds > 1 ? (size_t)wrach::world_tiles(ctx->ncells) + 2 : 0;
  const size_t worlds_words = (nworlds * sizeof(WorldDev) + 3) / 4 + tiles_words;
  {
    uint32_t* raw = nullptr;
    if ((e = dalloc(&raw, worlds_words)) != cudaSuccess) return oom(e);
    ctx->worlds_d = reinterpret_cast<WorldDev*>(raw);
  }
  if ((e = dalloc(&ctx->pos, tc)) != cudaSuccess) return oom(e);
  if ((e = dalloc(&ctx->vel, tc)) != cudaSuccess) return oom(e);
  if ((e = dalloc(&ctx->pos_o, tc)) != cudaSuccess) return oom(e);
  if ((e = dalloc(&ctx->vel_o, tc)) != cudaSuccess) return oom(e);
  if (c.mode == WRACH_MODE_EXTENDED && ctx->ph.iterations >= 2) {
    if ((e = dalloc(&ctx->q1, tc + wrach::kRowPad)) != cudaSuccess) return oom(e);
    if ((e = dalloc(&ctx->q2, tc + wrach::kRowPad)) != cudaSuccess) return oom(e);
  }
  if (c.mode == WRACH_MODE_EXTENDED && ctx->ph.iterations >= 2)
    if ((e = dalloc(&ctx->rows, tc)) != cudaSuccess) return oom(e);
  if (c.mode == WRACH_MODE_EXTENDED) {
    for (int i = 0; i < 2; ++i) {
      if ((e = dalloc(&ctx->tp_pos[i], tc + wrach::kRowPad)) != cudaSuccess) return oom(e);
      if ((e = dalloc(&ctx->tp_cell[i], tc)) != cudaSuccess) return oom(e);
      if ((e = dalloc(&ctx->tp_of[i], tc)) != cudaSuccess) return oom(e);
    }
  }
  for (int i = 0; i < 2; ++i) {
    if ((e = dalloc(&ctx->cell_of[i], tc)) != cudaSuccess) return oom(e);
    if (ctx->ncells > wrach::kDenseCells) {
      const size_t ngroups = ctx->ncells / wrach::kGroup + 1;
      if ((e = dalloc(&ctx->groups[i], ngroups)) != cudaSuccess) return oom(e);
      if ((e = cudaMemset(ctx->groups[i], 0, ngroups * sizeof(uint4))) != cudaSuccess) return oom(e);
    } else if (c.mode == WRACH_MODE_EXTENDED) {
      if ((e = dalloc(&ctx->ct[i], (size_t)ctx->ncells + 1)) != cudaSuccess) return oom(e);
      if ((e = cudaMemset(ctx->ct[i], 0, ((size_t)ctx->ncells + 1) * 4)) != cudaSuccess) return oom(e);
    }
    if ((e = dalloc(&ctx->cs[i], (size_t)ctx->ncells + 1)) != cudaSuccess) return oom(e);
    if ((e = cudaMemset(ctx->cs[i], 0, ((size_t)ctx->ncells + 1) * 4)) != cudaSuccess) return oom(e);
  }
  // one sum per tile of kTileCells cells of the table
  ctx->ntiles = (ctx->ncells + wrach::kTileCells - 1) / wrach::kTileCells;
  if ((e = dalloc(&ctx->tile_sums, ctx->ntiles)) != cudaSuccess) return oom(e);
  // the counting sort's tile sums reuse the table tile sums (kTileCells <= 2048)
  static_assert(wrach::kTileCells <= wrach::kCountScanTile, "tile sums buffer large enough");
  if ((e = cudaMemset(ctx->tile_sums, 0, (size_t)ctx->ntiles * 4)) != cudaSuccess) return oom(e);
  if (c.mode == WRACH_MODE_EXTENDED) {
    if ((e = dalloc(&ctx->tile_sums_cap, ctx->ntiles)) != cudaSuccess) return oom(e);
    if ((e = cudaMemset(ctx->tile_sums_cap, 0, (size_t)ctx->ntiles * 4)) != cudaSuccess) return oom(e);
  }
  if ((e = cudaDeviceGetAttribute(&ctx->sms, cudaDevAttrMultiProcessorCount, ctx->device)) != cudaSuccess)
    return oom(e);
  ctx->big_blocks = c.rebin_blocks ? c.rebin_blocks : wrach::kBigBlocksPerSm * (uint32_t)ctx->sms;
  if ((e = dalloc(&ctx->ctrl, 1)) != cudaSuccess) return oom(e);
  if ((e = cudaMemset(ctx->ctrl, 0, sizeof(Ctrl))) != cudaSuccess) return oom(e);
  if ((e = dalloc(&ctx->table_tmp, (size_t)ctx->max_world_cells + 2)) != cudaSuccess) return oom(e);
  if ((e = dalloc(&ctx->counts, (size_t)ctx->ncells + 1)) != cudaSuccess) return oom(e);
  if ((e = cudaMemset(ctx->counts, 0, ((size_t)ctx->ncells + 1) * 4)) != cudaSuccess) return oom(e);
  if ((e = dalloc(&ctx->gather_idx, nworlds + 1)) != cudaSuccess) return oom(e);
  if ((e = dalloc(&ctx->gather_out, nworlds + 1)) != cudaSuccess) return oom(e);
  if ((e = cudaMallocHost(reinterpret_cast<void**>(&ctx->gather_h), (nworlds + 1) * sizeof(uint32_t))) !=
      cudaSuccess)
    return oom(e);
  {
    std::vector<uint32_t> idx(nworlds + 1);
    for (uint32_t w = 0; w < nworlds; ++w) idx[w] = ctx->worlds_h[w].cell_off;
    idx[nworlds] = ctx->ncells;
    if ((e = cudaMemcpy(ctx->gather_idx, idx.data(), idx.size() * 4, cudaMemcpyHostToDevice)) != cudaSuccess) return oom(e);
  }
  if ((e = cudaMemcpy(ctx->worlds_d, ctx->worlds_h.data(), nworlds * sizeof(WorldDev),
                      cudaMemcpyHostToDevice)) != cudaSuccess)
    return oom(e);
  if (tiles_words) {
    static_assert(sizeof(WorldDev) % 4 == 0, "the tile table follows the worlds word-aligned");
    std::vector<uint32_t> first(tiles_words);
    uint32_t wi = 0;
    for (size_t t = 0; t < tiles_words; ++t) {
      const uint64_t c = std::min<uint64_t>((uint64_t)t << wrach::kWorldTileShift, ctx->ncells - 1);
      while (wi + 1 < nworlds && ctx->worlds_h[wi + 1].cell_off <= c) ++wi;
      first[t] = wi;
    }
    first[tiles_words - 2] = first[tiles_words - 1] = nworlds - 1;
    if ((e = cudaMemcpy(reinterpret_cast<uint32_t*>(ctx->worlds_d + nworlds), first.data(),
                        tiles_words * 4, cudaMemcpyHostToDevice)) != cudaSuccess)
      return oom(e);
  }
  if (ensure_sort_capacity(ctx, tc) != WRACH_OK) {
    int rc = WRACH_ERR_OUT_OF_MEMORY;
    release(ctx);
    delete ctx;
    return rc;
  }
  *out = ctx;
  return WRACH_OK;
}

// The particles of the other worlds' frames, which a re-pack of one world
// sorts again; with one world there are none.
uint32_t kept_particles(const WrachContext* ctx) { return ctx->nworlds > 1 ? ctx->n : 0u; }

// The n particles staged behind the first `at` places become the store `s`.
// With one world (at = 0) its buffers serve the next staging; with more the
// staging buffers are larger than any world's store, which has room for n.
int take_staged(WrachContext* ctx, Store& s, uint32_t at, uint32_t n) {
  if (ctx->nworlds == 1) {
    std::swap(s.pos, ctx->stage_pos);
    std::swap(s.vel, ctx->stage_vel);
    const size_t cap = s.cap;
    s.cap = (uint32_t)std::min(ctx->stage_cap, kMaxStore);
    ctx->stage_cap = cap;
  } else if (n) {
    CK(cudaMemcpyAsync(s.pos, ctx->stage_pos + at, (size_t)n * sizeof(float2), cudaMemcpyDeviceToDevice, ctx->stream));
    CK(cudaMemcpyAsync(s.vel, ctx->stage_vel + at, (size_t)n * sizeof(float2), cudaMemcpyDeviceToDevice, ctx->stream));
  }
  s.n = n;
  return WRACH_OK;
}

// Packs the frame of `world` from n_new particles: its store's or, `staged`,
// those in the staging buffers behind the kept ones, which then become the
// store.  The caller has made room in the store (of several worlds), the staging
// buffers (kept and new) and the sort's scratch.  Frame, table, counters and
// store stay as they are when the frame's capacity is exceeded.  vel_aside: the
// new velocities are on their way on the second stream.
int repack(WrachContext* ctx, uint32_t world, uint32_t n_new, bool staged, bool vel_aside) {
  Store& s = ctx->stores[world];
  const uint32_t n_keep = kept_particles(ctx), nsrc = n_keep + n_new;
  // The sort places straight into the frame buffers.  One world's place steps
  // follow the scan at once (they place nothing when the frame's capacity is
  // exceeded, which the host then reports), and its velocities are copied
  // while the positions' keys are counted, scanned and scattered (only the
  // place steps read them).  Of several worlds each has its own capacity: their
  // place steps wait for the counts.
  const bool direct = ctx->nworlds == 1;
  // the sort's source: [kept frame particles, new particles]; without kept
  // particles the store itself
  const bool from_stage = staged || n_keep;
  const float2* src_pos = from_stage ? ctx->stage_pos : s.pos;
  const float2* src_vel = from_stage ? ctx->stage_vel : s.vel;
  if (n_keep) {
    CK(cudaMemcpyAsync(ctx->stage_pos, ctx->pos, n_keep * sizeof(float2), cudaMemcpyDeviceToDevice, ctx->stream));
    CK(cudaMemcpyAsync(ctx->stage_vel, ctx->vel, n_keep * sizeof(float2), cudaMemcpyDeviceToDevice, ctx->stream));
    if (n_new && !staged) {
      CK(cudaMemcpyAsync(ctx->stage_pos + n_keep, s.pos, n_new * sizeof(float2), cudaMemcpyDeviceToDevice, ctx->stream));
      CK(cudaMemcpyAsync(ctx->stage_vel + n_keep, s.vel, n_new * sizeof(float2), cudaMemcpyDeviceToDevice, ctx->stream));
    }
  }
  CK(wrach::launch_upload_keys(ctx->worlds_d, (int)ctx->nworlds, ctx->ncells, world,
                               ctx->worlds_h[world], n_keep, ctx->cell_of[ctx->cur], n_new,
                               src_pos + n_keep, ctx->keys, ctx->ctrl, ticket_args(ctx),
                               ctx->stream));
  ctx->launches += nsrc ? 1 : 0;
  wrach::RebinArgs r = rebin_args(ctx);
  r.n = nsrc;
  r.dst_capacity = ctx->total_cap;
  r.pos_src = src_pos;
  r.vel_src = src_vel;
  r.pos_dst = ctx->pos;
  r.vel_dst = ctx->vel;
  r.cell_dst = ctx->cell_of[ctx->cur ^ 1];
  r.force_general = 1;
  // per-world counts from the new table, written to the host ahead of the
  // place steps: one world's by the scan itself
  const uint32_t nw = ctx->nworlds;
  if (direct) {
    r.fits_only = 1;
    r.total_out = ctx->gather_h + 1;
  }
  bool launched;
  CK(wrach::launch_count_sort_step(r, wrach::kScan, ctx->big_blocks, ctx->stream, &launched));
  if (!direct) {
    k_gather_starts<<<(nw + 1 + 255) / 256, 256, 0, ctx->stream>>>(
        ctx->table(ctx->cur ^ 1), ctx->gather_idx, nw + 1, ctx->gather_h);
    CK(cudaGetLastError());
    ctx->launches += 1;
  }
  CK(cudaEventRecord(ctx->counts_ev, ctx->stream));
  ctx->launches += wrach::count_sort_launches(r.n, ctx->ncells);
  auto place = [&]() {
    CK(wrach::launch_count_sort_step(r, wrach::kScatter, ctx->big_blocks, ctx->stream, &launched));
    // the place step is the first to read the velocities (the order is RebinOrder's)
    if (vel_aside) CK(cudaStreamWaitEvent(ctx->stream, ctx->join_ev, 0));
    CK(wrach::launch_count_sort_step(r, wrach::kPlace, ctx->big_blocks, ctx->stream, &launched));
    return (int)WRACH_OK;
  };
  int rc;
  if (direct && (rc = place())) return rc;
  // the call returns once the counts are known and the source arrays have
  // been read; the place steps may still be running, ahead of whatever the
  // caller enqueues next on the context's stream
  CK(cudaEventSynchronize(ctx->counts_ev));
  if (vel_aside) CK(cudaEventSynchronize(ctx->join_ev));
  if (direct) ctx->gather_h[0] = 0u;
  const std::vector<uint32_t> starts(ctx->gather_h, ctx->gather_h + nw + 1);
  for (uint32_t w = 0; w < nw; ++w) {
    const uint32_t cnt = starts[w + 1] - starts[w];
    if (cnt > ctx->cap_h[w]) {
      // nothing is placed; the counters are left as the place steps leave them
      CK(cudaMemsetAsync(ctx->counts, 0, ((size_t)ctx->ncells + 1) * 4, ctx->stream));
      CK(cudaMemsetAsync(ctx->tile_sums, 0, (size_t)ctx->ntiles * 4, ctx->stream));
      if (ctx->tile_sums_cap)
        CK(cudaMemsetAsync(ctx->tile_sums_cap, 0, (size_t)ctx->ntiles * 4, ctx->stream));
      return fail(ctx, WRACH_ERR_CAPACITY,
                  "world " + std::to_string(w) + ": " + std::to_string(cnt) +
                      " particles in the frame exceed its capacity " + std::to_string(ctx->cap_h[w]));
    }
  }
  if (!direct && (rc = place())) return rc;
  if (staged && (rc = take_staged(ctx, s, n_keep, n_new))) return rc;
  s.n = n_new;
  ctx->cur ^= 1;
  ctx->n = starts[nw];
  for (uint32_t w = 0; w < nw; ++w) {
    ctx->n_h[w] = starts[w + 1] - starts[w];
    ctx->poff_h[w] = starts[w];
  }
  ctx->graph_ok = true;
  return WRACH_OK;
}

int upload_impl(WrachContext* ctx, uint32_t world, const float* pos,
                const float* vel, uint32_t n_add, cudaMemcpyKind kind,
                bool replace) {
  if (!ctx) return WRACH_ERR_INVALID_ARGUMENT;
  if (world >= ctx->nworlds) return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "world out of range");
  if (n_add && (!pos || !vel)) return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "null particle arrays");
  DeviceGuard guard(ctx->device);
  Store& s = ctx->stores[world];
  const uint32_t n_keep = kept_particles(ctx);
  const size_t n_new = (size_t)(replace ? 0u : s.n) + n_add, nsrc = n_keep + n_new;
  if (nsrc > kMaxStore) return fail(ctx, WRACH_ERR_CAPACITY, "too many particles");
  // A replacing upload is staged, any other goes behind the store's particles:
  // the store keeps what it holds until the frame is known to fit.
  const bool one = ctx->nworlds == 1;
  int rc;
  if ((rc = ensure_stage(ctx, nsrc))) return rc;
  if (!(one && replace) && (rc = ensure_store(ctx, s, n_new))) return rc;
  if ((rc = ensure_sort_capacity(ctx, nsrc))) return rc;
  const bool vel_aside = one && n_add;
  if (n_add) {
    float2* to_pos = replace ? ctx->stage_pos + n_keep : s.pos + s.n;
    float2* to_vel = replace ? ctx->stage_vel + n_keep : s.vel + s.n;
    CK(cudaMemcpyAsync(to_pos, pos, (size_t)n_add * sizeof(float2), kind, ctx->stream));
    if (vel_aside) {
      CK(cudaEventRecord(ctx->fork_ev, ctx->stream));
      CK(cudaStreamWaitEvent(ctx->aux, ctx->fork_ev, 0));
    }
    cudaStream_t st = vel_aside ? ctx->aux : ctx->stream;
    CK(cudaMemcpyAsync(to_vel, vel, (size_t)n_add * sizeof(float2), kind, st));
    if (vel_aside) CK(cudaEventRecord(ctx->join_ev, ctx->aux));
  }
  return repack(ctx, world, (uint32_t)n_new, replace, vel_aside);
}

// ---------------------------------------------------------------------------
// Viewport streaming
// ---------------------------------------------------------------------------

// The world's store as it becomes, staged behind the first `at` places: its
// particles outside the viewport (store order), then the world's frame
// particles (frame order) -- per cell the reference's write-back of the GPU's
// particles into its store (particle_store.rs:71-85, a TODO there).  *count is
// its size, for which the store of a batch has room then.  With `moved` the
// world's settings on the device become those, for the re-packing that follows
// (a copy from the host would stand between the two).
int rebuild_store(WrachContext* ctx, uint32_t world, uint32_t at, const WorldDev* moved,
                  uint32_t* count) {
  Store& s = ctx->stores[world];
  const uint32_t nf = ctx->n_h[world], off = ctx->poff_h[world];
  int rc;
  const uint32_t ntiles = wrach::store_tiles(s.n);
  if ((rc = ensure_sort_capacity(ctx, std::max((size_t)s.n + 1, (size_t)ntiles * 32)))) return rc;
  if ((rc = ensure_stage(ctx, (size_t)at + s.n + nf))) return rc;
  if (ntiles + 1 > ctx->compact_cap) {
    dfree(ctx->compact_sums);
    ctx->compact_sums = nullptr;
    ctx->compact_cap = 0;
    CK(dalloc(&ctx->compact_sums, (size_t)ntiles + 1));
    ctx->compact_cap = (size_t)ntiles + 1;
  }
  wrach::StoreRebuild r{};
  r.worlds = ctx->worlds_d;
  r.moves = moved != nullptr;
  if (moved) r.moved = *moved;
  r.target = world;
  r.n = s.n;
  r.nf = nf;
  r.pos = s.pos;
  r.vel = s.vel;
  r.frame_pos = ctx->pos + off;
  r.frame_vel = ctx->vel + off;
  r.dst_pos = ctx->stage_pos + at;
  r.dst_vel = ctx->stage_vel + at;
  r.outside = ctx->keys;
  r.tile_sums = ctx->compact_sums;
  r.kept = ctx->compact_sums + ntiles;
  r.kept_host = ctx->gather_h;
  CK(wrach::launch_outside(r, ctx->stream));
  CK(cudaEventRecord(ctx->counts_ev, ctx->stream));
  CK(wrach::launch_rebuild(r, ctx->stream));
  ctx->launches += (ntiles ? 2 : 1) + (s.n + nf ? 1 : 0);
  // the store is rebuilt while the host learns its size
  CK(cudaEventSynchronize(ctx->counts_ev));
  const size_t size = (size_t)ctx->gather_h[0] + nf;
  if (at + size > kMaxStore) return fail(ctx, WRACH_ERR_CAPACITY, "store too large");
  if (ctx->nworlds > 1 && (rc = ensure_store(ctx, s, size))) return rc;
  *count = (uint32_t)size;
  return WRACH_OK;
}

}  // namespace

extern "C" {

int wrach_config_default(WrachConfig* c) {
  if (!c) return WRACH_ERR_INVALID_ARGUMENT;
  std::memset(c, 0, sizeof(*c));
  c->width = 480.0f;
  c->height = 352.0f;
  c->cell_size = 3;
  c->mode = WRACH_MODE_REFERENCE;
  c->iterations = 4;
  c->gravity = 0.0f;
  c->min_distance = 1.0f;
  c->max_velocity = 1.0f;
  c->cell_capacity = 9;
  c->capacity = 0;
  c->device = 0;
  return WRACH_OK;
}

uint32_t wrach_max_particles_per_frame(uint32_t cells, uint32_t cell_size) {
  const uint32_t cs2 = (uint32_t)(uint16_t)(cell_size * cell_size);
  const uint32_t normal = cells * cs2;
  const uint32_t one_percent = (normal + 99u) / 100u;
  return normal + 10u * one_percent;
}

int wrach_create(const WrachConfig* config, WrachContext** out) {
  return create_impl(config, 1, nullptr, out);
}

int wrach_create_batch(const WrachConfig* config, uint32_t nworlds, const float* dims,
                       WrachContext** out) {
  if (!dims) return WRACH_ERR_INVALID_ARGUMENT;
  return create_impl(config, nworlds, dims, out);
}

int wrach_destroy(WrachContext* ctx) {
  if (!ctx) return WRACH_ERR_INVALID_ARGUMENT;
  {
    DeviceGuard guard(ctx->device);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    // an upload's copy on `aux` is joined into `stream`, unless its enqueue
    // failed between the fork and the join
    if (ctx->aux) cudaStreamSynchronize(ctx->aux);
    release(ctx);
  }
  delete ctx;
  return WRACH_OK;
}

int wrach_add_particles(WrachContext* ctx, uint32_t world, const float* pos, const float* vel,
                        uint32_t n) {
  return upload_impl(ctx, world, pos, vel, n, cudaMemcpyHostToDevice, false);
}

int wrach_set_particles(WrachContext* ctx, uint32_t world, const float* pos, const float* vel,
                        uint32_t n) {
  return upload_impl(ctx, world, pos, vel, n, cudaMemcpyHostToDevice, true);
}

int wrach_add_particles_device(WrachContext* ctx, uint32_t world, const float* d_pos,
                               const float* d_vel, uint32_t n) {
  return upload_impl(ctx, world, d_pos, d_vel, n, cudaMemcpyDeviceToDevice, false);
}

int wrach_step(WrachContext* ctx, uint32_t nsteps) {
  if (!ctx) return WRACH_ERR_INVALID_ARGUMENT;
  DeviceGuard guard(ctx->device);
  if (int rc = ensure_sort_capacity(ctx, ctx->total_cap)) return rc;
  for (uint32_t s = 0; s < nsteps; ++s) {
    // a graph holds the particle count (grid sizes) it was captured with;
    // buffer reallocations drop the graphs.  Capturing one takes about as long
    // as a 1M-particle frame, so the first frame of a new count, or of a single
    // world's new viewport, runs eagerly.
    cudaGraphExec_t& graph = ctx->graph[ctx->cur];
    const bool again = ctx->last_n == ctx->n;
    ctx->last_n = ctx->n;
    if (ctx->graph_ok && again && (!graph || ctx->graph_n[ctx->cur] != ctx->n)) {
      if (graph) cudaGraphExecDestroy(graph);
      graph = nullptr;
      int rc = build_graph(ctx);
      if (rc) return rc;
    }
    if (ctx->graph_ok && graph && ctx->graph_n[ctx->cur] == ctx->n) {
      CK(cudaGraphLaunch(graph, ctx->stream));
      ctx->launches += frame_launches(ctx);
      ctx->cur ^= 1;
    } else {
      int rc = enqueue_frame(ctx);
      if (rc) return rc;
    }
  }
  return WRACH_OK;
}

int wrach_profile_frame(WrachContext* ctx, float* ms, uint32_t cap, uint32_t* count) {
  if (!ctx || !count) return WRACH_ERR_INVALID_ARGUMENT;
  DeviceGuard guard(ctx->device);
  const uint32_t nl = frame_steps(ctx);
  *count = nl;
  if (!ms || cap < nl) return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "profile buffer too small");
  int rc = ensure_sort_capacity(ctx, ctx->total_cap);
  if (rc) return rc;
  std::vector<cudaEvent_t> ev(nl + 1);
  for (auto& e : ev) CK(cudaEventCreate(&e));
  ctx->event_hook = ev.data();
  ctx->event_count = 0;
  rc = enqueue_frame(ctx);
  ctx->event_hook = nullptr;
  if (rc == WRACH_OK) {
    CK(cudaStreamSynchronize(ctx->stream));
    for (uint32_t i = 0; i < nl; ++i) CK(cudaEventElapsedTime(&ms[i], ev[i], ev[i + 1]));
  }
  for (auto& e : ev) cudaEventDestroy(e);
  return rc;
}

int wrach_read(WrachContext* ctx, uint32_t world, float* positions, float* velocities,
               uint32_t* indices, uint32_t capacity) {
  if (!ctx) return WRACH_ERR_INVALID_ARGUMENT;
  if (world >= ctx->nworlds) return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "world out of range");
  DeviceGuard guard(ctx->device);
  const uint32_t n = ctx->n_h[world], off = ctx->poff_h[world];
  if ((positions || velocities) && capacity < ctx->cap_h[world])
    return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "capacity smaller than the world's frame capacity");
  if (n == 0) positions = velocities = nullptr;
  const WorldDev& w = ctx->worlds_h[world];
  const uint32_t cells = w.gx * w.gy;
  // a dense table's starts are the reference's table from its second entry on
  const bool whole = ctx->nworlds == 1 && !ctx->groups[0];
  wrach::WorldRead r{};
  r.pos = reinterpret_cast<const uint32_t*>(ctx->pos + off);
  r.vel = reinterpret_cast<const uint32_t*>(ctx->vel + off);
  r.n = n;
  r.table = ctx->table(ctx->cur);
  r.cell_off = w.cell_off;
  r.cells = cells;
  // Two arrays or more in the host's pinned memory are written by one launch:
  // three copies of 1/3 MB each take 17.0 us, one of 1 MB 13.7 and the launch
  // 14.1.  For one array alone the copy engine's start is the cheaper one,
  // except for a table that a launch has to lay out anyway.
  if (!!positions + !!velocities + !!indices >= 2 || (indices && !whole)) {
    r.pos_out = device_view(positions, (size_t)n * 8);
    r.vel_out = device_view(velocities, (size_t)n * 8);
    r.table_out = device_view(indices, ((size_t)cells + 2) * 4);
  }
  const bool table_mapped = r.table_out != nullptr;
  if (indices && !table_mapped && !whole) r.table_out = ctx->table_tmp;
  if (r.pos_out || r.vel_out || r.table_out) {
    CK(wrach::launch_read_world(r, ctx->sms, ctx->stream));
    ctx->launches += 1;
  }
  if (positions && !r.pos_out)
    CK(cudaMemcpyAsync(positions, ctx->pos + off, (size_t)n * 8, cudaMemcpyDeviceToHost, ctx->stream));
  if (velocities && !r.vel_out)
    CK(cudaMemcpyAsync(velocities, ctx->vel + off, (size_t)n * 8, cudaMemcpyDeviceToHost, ctx->stream));
  if (indices && !table_mapped) {
    if (whole)
      CK(cudaMemcpyAsync(indices + 1, ctx->cs[ctx->cur], ((size_t)cells + 1) * 4,
                         cudaMemcpyDeviceToHost, ctx->stream));
    else
      CK(cudaMemcpyAsync(indices, ctx->table_tmp, ((size_t)cells + 2) * 4, cudaMemcpyDeviceToHost,
                         ctx->stream));
  }
  CK(cudaStreamSynchronize(ctx->stream));
  if (indices && !table_mapped && whole) indices[0] = 0;
  return WRACH_OK;
}

int wrach_tick(WrachContext* ctx, uint32_t world, float* positions, float* velocities,
               uint32_t* indices, uint32_t capacity) {
  int rc = wrach_step(ctx, 1);
  if (rc) return rc;
  return wrach_read(ctx, world, positions, velocities, indices, capacity);
}

int wrach_get_settings(WrachContext* ctx, uint32_t world, WrachWorldSettings* out) {
  if (!ctx || !out || world >= ctx->nworlds) return WRACH_ERR_INVALID_ARGUMENT;
  const WorldDev& w = ctx->worlds_h[world];
  out->view_dimensions[0] = w.dim_x;
  out->view_dimensions[1] = w.dim_y;
  out->view_anchor[0] = w.ax;
  out->view_anchor[1] = w.ay;
  out->grid_dimensions[0] = w.gx;
  out->grid_dimensions[1] = w.gy;
  out->cell_size = w.cs;
  out->particles_in_frame_count = ctx->n_h[world];
  return WRACH_OK;
}

int wrach_read_keys(WrachContext* ctx, uint32_t world, uint32_t* keys, uint32_t capacity) {
  if (!ctx) return WRACH_ERR_INVALID_ARGUMENT;
  if (world >= ctx->nworlds) return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "world out of range");
  const uint32_t n = ctx->n_h[world], off = ctx->poff_h[world];
  if (n && (!keys || capacity < n)) return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "key buffer too small");
  DeviceGuard guard(ctx->device);
  if (n) {
    // the keys land in the scratch the sort uses between frames
    int rc = ensure_sort_capacity(ctx, (size_t)n);
    if (rc) return rc;
    CK(wrach::launch_local_keys(ctx->cell_of[ctx->cur] + off, n, ctx->worlds_h[world].cell_off,
                                ctx->iB, ctx->stream));
    ctx->launches += 1;
    CK(cudaMemcpyAsync(keys, ctx->iB, (size_t)n * 4, cudaMemcpyDeviceToHost, ctx->stream));
  }
  CK(cudaStreamSynchronize(ctx->stream));
  return WRACH_OK;
}

int wrach_write_back(WrachContext* ctx, uint32_t world) {
  if (!ctx) return WRACH_ERR_INVALID_ARGUMENT;
  if (world >= ctx->nworlds) return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "world out of range");
  DeviceGuard guard(ctx->device);
  uint32_t count = 0;
  int rc = rebuild_store(ctx, world, 0, nullptr, &count);
  if (rc || (rc = take_staged(ctx, ctx->stores[world], 0, count))) return rc;
  CK(cudaStreamSynchronize(ctx->stream));
  return WRACH_OK;
}

int wrach_set_viewport(WrachContext* ctx, uint32_t world, float anchor_x, float anchor_y) {
  if (!ctx) return WRACH_ERR_INVALID_ARGUMENT;
  if (world >= ctx->nworlds) return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "world out of range");
  DeviceGuard guard(ctx->device);
  const WorldDev old = ctx->worlds_h[world];
  WorldDev w;
  if (world_settings_init(w, old.dim_x, old.dim_y, anchor_x, anchor_y, old.cs) || w.gx != old.gx ||
      w.gy != old.gy)
    return fail(ctx, WRACH_ERR_INVALID_ARGUMENT,
                "the viewport at this anchor has a different grid size; move it by whole cells "
                "or use a size that is a multiple of the cell size");
  w.cell_off = old.cell_off;
  // the rebuilt store is staged and the frame packed from it under the new
  // viewport; both are taken when the frame fits
  uint32_t count = 0;
  const uint32_t n_keep = kept_particles(ctx);
  int rc = rebuild_store(ctx, world, n_keep, &w, &count);
  if (!rc) {
    ctx->worlds_h[world] = w;
    rc = ensure_sort_capacity(ctx, (size_t)n_keep + count);
    if (!rc) rc = repack(ctx, world, count, true, false);
  }
  if (rc) {
    // refused: host and device keep the viewport
    ctx->worlds_h[world] = old;
    cudaMemcpyAsync(ctx->worlds_d + world, &old, sizeof(WorldDev), cudaMemcpyHostToDevice, ctx->stream);
    return rc;
  }
  if (ctx->nworlds == 1) {
    // its settings are among its launches' arguments; a batch's launches read
    // them from the device and are captured no more often than its counts change
    drop_graphs(ctx);
    ctx->last_n = 0xFFFFFFFFu;
  }
  return WRACH_OK;
}

int wrach_selftest_wait(WrachContext* ctx, uint32_t limit_us, uint32_t* timed_out,
                        uint32_t* waited_us) {
  if (!ctx || !timed_out || !waited_us) return WRACH_ERR_INVALID_ARGUMENT;
  if (limit_us > 1000000u) return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "limit above 1 s");
  DeviceGuard guard(ctx->device);
  CK(wrach::launch_wait_probe(&ctx->ctrl->never_set, 0u, (uint64_t)limit_us * 1000u,
                              ctx->gather_out, ctx->stream));
  ctx->launches += 1;
  uint32_t h[2];
  CK(cudaMemcpyAsync(h, ctx->gather_out, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  *timed_out = h[0];
  *waited_us = h[1];
  return WRACH_OK;
}

int wrach_selftest_push(WrachContext* ctx, float min_distance, uint64_t* compared,
                        uint64_t* wrong) {
  if (!ctx || !compared || !wrong) return WRACH_ERR_INVALID_ARGUMENT;
  if (!(min_distance > 0.0f) || std::isinf(min_distance))
    return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "bad minimum distance");
  DeviceGuard guard(ctx->device);
  PhysDev ph{};
  set_push(ph, min_distance);
  // positive binary32 values order like their bits
  uint32_t first, end;
  std::memcpy(&first, &ph.slow_below, 4);
  std::memcpy(&end, &ph.skip_d2, 4);
  unsigned long long *d = nullptr, h[2] = {0, 0};
  CK(dalloc(&d, 2));
  cudaError_t e = cudaMemsetAsync(d, 0, sizeof(h), ctx->stream);
  if (e == cudaSuccess) e = wrach::launch_push_check(ph, first, end, ctx->sms, d, ctx->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  dfree(d);
  CK(e);
  ctx->launches += first < end ? 1 : 0;
  *compared = h[0];
  *wrong = h[1];
  return WRACH_OK;
}

int wrach_selftest_alloc(WrachContext* ctx, uint32_t nth) {
  if (!ctx) return WRACH_ERR_INVALID_ARGUMENT;
  ctx->fail_alloc = nth;
  return WRACH_OK;
}

int wrach_store_size(WrachContext* ctx, uint32_t world, uint32_t* count) {
  if (!ctx || !count || world >= ctx->nworlds) return WRACH_ERR_INVALID_ARGUMENT;
  *count = ctx->stores[world].n;
  return WRACH_OK;
}

int wrach_read_store(WrachContext* ctx, uint32_t world, float* positions, float* velocities,
                     uint32_t capacity) {
  if (!ctx || world >= ctx->nworlds) return WRACH_ERR_INVALID_ARGUMENT;
  const Store& s = ctx->stores[world];
  if (capacity < s.n) return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "capacity smaller than the store");
  DeviceGuard guard(ctx->device);
  if (positions && s.n)
    CK(cudaMemcpyAsync(positions, s.pos, (size_t)s.n * 8, cudaMemcpyDeviceToHost, ctx->stream));
  if (velocities && s.n)
    CK(cudaMemcpyAsync(velocities, s.vel, (size_t)s.n * 8, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  return WRACH_OK;
}

uint32_t wrach_capacity(WrachContext* ctx, uint32_t world) {
  if (!ctx || world >= ctx->nworlds) return 0;
  return ctx->cap_h[world];
}

uint32_t wrach_num_worlds(WrachContext* ctx) { return ctx ? ctx->nworlds : 0; }

int wrach_render(WrachContext* ctx, uint32_t world, uint32_t width_px, uint32_t height_px,
                 uint8_t* image) {
  if (!ctx || !image || !width_px || !height_px) return WRACH_ERR_INVALID_ARGUMENT;
  if (world >= ctx->nworlds) return fail(ctx, WRACH_ERR_INVALID_ARGUMENT, "world out of range");
  DeviceGuard guard(ctx->device);
  const size_t npix = (size_t)width_px * height_px;
  const size_t words = wrach::render_words(width_px, height_px);
  // a narrow image takes more words per pixel than a wide one
  if (npix > ctx->render_cap || words > ctx->cover_cap) {
    const size_t pixels = std::max(npix, ctx->render_cap), cover = std::max(words, ctx->cover_cap);
    dfree(ctx->render_cover);
    dfree(ctx->render_image);
    ctx->render_cover = nullptr;
    ctx->render_image = nullptr;
    ctx->render_cap = ctx->cover_cap = 0;
    CK(dalloc(&ctx->render_cover, cover));
    CK(dalloc(&ctx->render_image, pixels));
    CK(cudaMemsetAsync(ctx->render_cover, 0, cover * sizeof(uint32_t), ctx->stream));
    ctx->render_cap = pixels;
    ctx->cover_cap = cover;
  }
  const WorldDev& w = ctx->worlds_h[world];
  CK(wrach::launch_render(ctx->pos + ctx->poff_h[world], ctx->n_h[world], w.dim_x, w.dim_y, width_px,
                          height_px, ctx->render_cover, ctx->render_image, ctx->stream));
  ctx->launches += ctx->n_h[world] ? 2 : 1;
  CK(cudaMemcpyAsync(image, ctx->render_image, npix, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  return WRACH_OK;
}

int wrach_sync(WrachContext* ctx) {
  if (!ctx) return WRACH_ERR_INVALID_ARGUMENT;
  DeviceGuard guard(ctx->device);
  CK(cudaStreamSynchronize(ctx->stream));
  return WRACH_OK;
}

int wrach_flags(WrachContext* ctx, uint32_t* flags) {
  if (!ctx || !flags) return WRACH_ERR_INVALID_ARGUMENT;
  DeviceGuard guard(ctx->device);
  Ctrl h{};
  CK(cudaMemcpyAsync(&h, ctx->ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  *flags = h.flags;
  return WRACH_OK;
}

int wrach_stats(WrachContext* ctx, WrachStats* out) {
  if (!ctx || !out) return WRACH_ERR_INVALID_ARGUMENT;
  DeviceGuard guard(ctx->device);
  Ctrl h{};
  CK(cudaMemcpyAsync(&h, ctx->ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  std::memset(out, 0, sizeof(*out));
  out->flags = h.flags;
  out->frames = h.frames;
  out->overflow = h.overflow;
  out->rebin_blocks = ctx->big_blocks;
  out->tiles = ctx->ntiles;
  out->particles = ctx->n;
  out->cells = ctx->ncells;
  out->huge_cells = h.huge_cells;
  return WRACH_OK;
}

const char* wrach_last_error(WrachContext* ctx) { return ctx ? ctx->err.c_str() : "null context"; }

uint64_t wrach_kernel_launches(WrachContext* ctx) { return ctx ? ctx->launches : 0; }

void* wrach_stream(WrachContext* ctx) { return ctx ? (void*)ctx->stream : nullptr; }

}  // extern "C"
