// C-ABI implementation of the B200 vortex-particle backend (include/pawan_gpu.h).
//
// Device memory of a context (cap = total particle slots of all wakes):
//   x0     [6][cap] FP64   state at the step start (x, y, z, alpha_x, alpha_y, alpha_z), SoA
//   acc    [6][cap] FP64   RK accumulator
//   rates  [6][cap] FP64   rates of the last evaluation
//   sig, vol [cap]  FP64   smoothing radius, volume
//   P, Q   [cap]    float4 (FP32C) or double4 (FP64) source records (x, y, z, sigma^2/2), (alpha, vol)
//   partial [nch][6][cap] FP64 per-chunk partial rates written by the pair kernel
//   stage  [8][cap] FP64   staging for host row-major <-> SoA transfers
// Systems occupy contiguous slot ranges; inside a system its wakes are laid out
// in the order they were added.
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdint>
#include <map>
#include <mutex>
#include <numeric>
#include <string>
#include <thread>
#include <tuple>
#include <vector>

#include "../../include/pawan_gpu.h"
#include "kernels.cuh"
#include "treeeval.cuh"

#include <cub/cub.cuh>

using namespace pgpu;

namespace {

constexpr int kCG = kPairCG;
static_assert(kDiagFields == PGPU_DIAG_FIELDS, "the diagnostic field layout of the header");

struct Shape { int block, tpt; };
// Compiled pair-kernel shapes (the autotuner chooses among these).
constexpr Shape kShapes[] = {{128, 1}, {128, 2}, {256, 1}, {256, 2}, {64, 2}, {128, 4}};
constexpr int kNumShapes = sizeof(kShapes) / sizeof(kShapes[0]);

template <typename T> using PairFn = void (*)(PairArgs<T>);

template <typename T, int KER, bool SPLIT = false> PairFn<T> pair_fn_k(int s) {
  switch (s) {
    case 0: return pair_kernel<T, 128, 1, kCG, KER, SPLIT>;
    case 1: return pair_kernel<T, 128, 2, kCG, KER, SPLIT>;
    case 2: return pair_kernel<T, 256, 1, kCG, KER, SPLIT>;
    case 3: return pair_kernel<T, 256, 2, kCG, KER, SPLIT>;
    case 4: return pair_kernel<T, 64, 2, kCG, KER, SPLIT>;
    default: return pair_kernel<T, 128, 4, kCG, KER, SPLIT>;
  }
}
// Pair kernel of shape s for regularisation kernel `ker` (PGPU_KERNEL_*);
// split: the FP32C Gaussian body with split positions.
template <typename T> PairFn<T> pair_fn(int s, int ker, bool split) {
  if (ker == PGPU_KERNEL_HIGHORDER) return pair_fn_k<T, kHighOrder>(s);
  if constexpr (sizeof(T) == 4) {
    if (split) return pair_fn_k<T, kGaussian, true>(s);
  }
  return pair_fn_k<T, kGaussian>(s);
}

// Variants of the slices kernel (pair_slices.cuh): 32-source slices of one
// source per lane, with or without split positions, and 64-source ones.
constexpr int kSliceLen[] = {32, 64};
constexpr int kNumSlices = 2;
PairFn<float> slices_fn(int v, int ker, bool split) {
  if (ker == PGPU_KERNEL_HIGHORDER)
    return v == 0 ? pair_slices_kernel<1, false, kHighOrder> : pair_slices_kernel<2, false, kHighOrder>;
  if (split) return pair_slices_kernel<1, true>;
  return v == 0 ? pair_slices_kernel<1, false> : pair_slices_kernel<2, false>;
}

// The same row list in FP64 (pair_slices64.cuh), with its dynamic shared memory.
PairFn<double> slices64_fn(int v, int ker) {
  if (ker == PGPU_KERNEL_HIGHORDER)
    return v == 0 ? pair_slices64_kernel<1, kHighOrder> : pair_slices64_kernel<2, kHighOrder>;
  return v == 0 ? pair_slices64_kernel<1, kGaussian> : pair_slices64_kernel<2, kGaussian>;
}
size_t slices64_bytes(int v) { return v == 0 ? slices64_smem<1>() : slices64_smem<2>(); }

struct WakeRec {
  int sys;
  int64_t cap, n, off;
};
struct SysRec {
  std::vector<int> wakes;
  int64_t off = 0, cap = 0;
  double zc = 0.0;  // last reported Zc (PAWAN keeps _Zc across calls)
  int64_t t_first = 0, t_count = -1;  // owned targets (pgpu_set_target_range); count < 0: all
};

}  // namespace

struct SurrogateState;

struct pgpu_ctx {
  pgpu_config cfg;
  cudaStream_t st = nullptr;
  int sms = 0;
  std::vector<WakeRec> wakes;
  std::vector<SysRec> sys;
  bool frozen = false;
  int64_t cap = 0;
  double *x0 = nullptr, *acc = nullptr, *rates = nullptr, *sig = nullptr, *vol = nullptr;
  double *partial = nullptr, *stage = nullptr;
  void *P = nullptr, *Q = nullptr;
  int64_t *d_sysoff = nullptr, *d_sysn = nullptr, *d_syst = nullptr;
  PlanEntry *d_plan = nullptr, *d_plan_diag = nullptr, *d_plan_field = nullptr;
  double *d_field = nullptr;  // [3][cap] vorticity field, allocated by pgpu_influence
  unsigned long long *d_merge = nullptr;  // merge candidate keys (pgpu_merge): d_merge_cap, a counter, d_merge_cap sorted
  int64_t d_merge_cap = 0;
  void *d_merge_tmp = nullptr;  // radix-sort space of the candidate keys
  size_t d_merge_tmp_bytes = 0;
  unsigned int *d_counters = nullptr;
  unsigned long long *d_nfull = nullptr;
  float4 *d_box = nullptr;  // FP32 source boxes per kBoxGran slots (box_kernel), FP32C Gaussian contexts
  float4 *d_L = nullptr;    // [cap] split-position residuals (pgpu_config.split_positions)
  int64_t pairs_acc = 0, selfs_acc = 0;  // ordered pairs and self pairs of the pair launches so far
  // Pinned host memory of the context, mapped: the non-finite flag the kernels
  // set (h_flag), then a ring of io_bytes for small transfers (io_take), so
  // that a call on a few thousand particles queues kernels and no copies.
  unsigned char *h_io = nullptr;
  size_t io_bytes = 0, io_pos = 0;
  int *h_flag = nullptr;
  int diag_blocks = 0;
  int shape = 2;  // (256, 1) before autotuning: the high-order kernel's default (pgpu_create picks the Gaussian's)
  // Shapes per system chosen by pgpu_autotune_classes (empty: `shape` for
  // every system).  Each distinct shape in `groups` (ascending) is one pair
  // launch per evaluation over the systems that use it, with its own plan at
  // d_plan + g (nsys + 1).
  std::vector<int> sys_shape;
  std::vector<int> groups;
  int grid[kNumShapes] = {0};
  // no shape was asked for or tuned: small FP32C Gaussian systems may take
  // the slices kernel (choose_slices); slices is its variant, -1 for none
  bool auto_shape = true;
  bool shape_asked = false;  // the configuration names a shape
  int slices = -1;
  int grid_slices[kNumSlices] = {0};
  int nch = 1;
  bool plan_dirty = true;
  bool timing = true;
  bool capturing = false;
  cudaEvent_t ev[8][2] = {};
  // Capture of a step's graph: the event records are nodes on a side branch
  // (record_time), created with the first captured step.
  cudaStream_t st_side = nullptr;
  cudaEvent_t ev_side = nullptr;
  bool side_used = false;
  double pair_ms = 0.0;
  int64_t pair_launches = 0;
  int64_t launches = 0;
  // (scheme, dt, launch layout, nch, timing, first event slot)
  std::map<std::tuple<int, double, int, int, bool, int>, cudaGraphExec_t> graphs;
  std::vector<cudaGraph_t> graph_defs;
  // last error message: a fixed buffer under a mutex, since pgpu_snapshot_wait
  // may fail on a writer thread while the owning thread queues work
  char err[512] = {0};
  std::mutex err_mu;
  SurrogateState *sur = nullptr;  // far-field surrogate of the single system, when enabled
  // State snapshots (pgpu_snapshot_begin / _wait): per slot a device buffer,
  // a pinned host buffer, the gather's and the copy's events, and the wake
  // rows the snapshot holds.
  cudaStream_t st_copy = nullptr;
  double *d_snap[2] = {nullptr, nullptr};
  double *h_snap[2] = {nullptr, nullptr};
  cudaEvent_t snap_gathered[2] = {nullptr, nullptr};
  cudaEvent_t snap_copied[2] = {nullptr, nullptr};
  bool snap_begun[2] = {false, false};
  std::vector<int64_t> snap_off[2], snap_n[2];
};

namespace {

// NVTX range over an entry point (header-only NVTX3: a no-op unless a
// profiler is attached), so profiler timelines show the library's phases.
struct NvtxRange {
  explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
};

// Makes a context's (or network's) device current for one entry point that
// works on the device, and restores the caller's device on return, so that
// contexts on different GPUs can be driven from one host thread.  pgpu_create
// leaves the new context's device current (as cudaSetDevice would), so a
// thread that creates a context and then uses it never switches: it calls
// nothing but cudaGetDevice.  Host-only calls and pgpu_snapshot_wait (which
// writer threads call; events need no current device) do not switch.
struct DeviceScope {
  int prev = -1;
  explicit DeviceScope(int dev) {
    int cur = -1;
    if (cudaGetDevice(&cur) == cudaSuccess && cur != dev && cudaSetDevice(dev) == cudaSuccess) prev = cur;
  }
  ~DeviceScope() {
    if (prev >= 0) cudaSetDevice(prev);
  }
  DeviceScope(const DeviceScope &) = delete;
  DeviceScope &operator=(const DeviceScope &) = delete;
};

int fail(pgpu_ctx *c, int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (c) {
    std::lock_guard<std::mutex> lock(c->err_mu);
    memcpy(c->err, buf, sizeof(buf));
  }
  return code;
}

// On failure the per-thread last error is reset (cudaGetLastError), so a
// non-sticky error such as a failed allocation is reported once, by the call
// that met it, and not again by the next healthy launch.
#define CK(call)                                                                                    \
  do {                                                                                              \
    cudaError_t e_ = (call);                                                                        \
    if (e_ != cudaSuccess) {                                                                        \
      cudaGetLastError();                                                                           \
      return fail(c, PGPU_ECUDA, "%s failed: %s", #call, cudaGetErrorString(e_));                   \
    }                                                                                               \
  } while (0)

// Why the calling thread's last pgpu_create failed ("" after a success);
// pgpu_last_error(NULL) returns it.
thread_local char g_create_err[512] = "";

// Releases what pgpu_create made before it failed, and records why.
int create_fail(pgpu_ctx *c, int code, const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_create_err, sizeof(g_create_err), fmt, ap);
  va_end(ap);
  if (c) {
    for (auto &pair : c->ev)
      for (cudaEvent_t e : pair)
        if (e) cudaEventDestroy(e);
    if (c->st) cudaStreamDestroy(c->st);
    delete c;
  }
  return code;
}

bool fp64(const pgpu_ctx *c) { return c->cfg.precision == PGPU_FP64; }
// The FP32C Gaussian pair kernel tests whole source tiles against boxes
// precomputed per kBoxGran slots (box_kernel) before each launch.
bool uses_boxes(const pgpu_ctx *c) { return !fp64(c) && c->cfg.kernel == PGPU_KERNEL_GAUSSIAN; }
// Split positions: FP32C Gaussian contexts with pgpu_config.split_positions.
bool uses_split(const pgpu_ctx *c) { return uses_boxes(c) && c->cfg.split_positions != 0; }
// Boxes cover every slot plus one largest tile (256 slots) past the last:
// the last tile of the last system may end beyond `cap`, and those blocks
// hold empty boxes.
int64_t box_blocks(const pgpu_ctx *c) { return (c->cap + kBoxGran - 1) / kBoxGran + 256 / kBoxGran; }
size_t rec_bytes(const pgpu_ctx *c) { return fp64(c) ? sizeof(double4) : sizeof(float4); }

int64_t sys_n(const pgpu_ctx *c, int s) {
  const SysRec &S = c->sys[s];
  if (S.wakes.empty()) return 0;
  const WakeRec &L = c->wakes[S.wakes.back()];
  return (L.off - S.off) + L.n;
}

int check_contiguous(pgpu_ctx *c) {
  for (size_t s = 0; s < c->sys.size(); ++s) {
    const SysRec &S = c->sys[s];
    for (size_t k = 0; k + 1 < S.wakes.size(); ++k) {
      const WakeRec &W = c->wakes[S.wakes[k]];
      if (W.n != W.cap)
        return fail(c, PGPU_EINVAL,
                    "wake %d of system %zu holds %lld of %lld particles; every wake but the last of a system must be full",
                    S.wakes[k], s, (long long)W.n, (long long)W.cap);
    }
  }
  return PGPU_OK;
}

template <typename T> int occupancy(pgpu_ctx *c, int s) {
  int nb = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, pair_fn<T>(s, c->cfg.kernel, uses_split(c)), kShapes[s].block, 0);
  if (e != cudaSuccess || nb < 1) nb = 1;
  return nb * c->sms;
}

// Largest ring of pinned memory for small transfers (pinning 2 MB takes 2 ms of
// the first upload, 512 kB a quarter of that), and the largest transfers that
// go through it, in pieces of half a ring.  Larger ones take the driver's
// own staging of pageable copies.  An upload waits for the stream wherever the
// ring turns, so it takes the ring only once round: 5000 rows 44 us by the ring
// and 75 us staged, 10,000 rows 62 and 60, 30,000 rows 198 and 145, 65,536 rows
// 418 and 244.  Downloads: 30,000 rows 200 and 296 us, 65,536 rows 495 and 563.
constexpr size_t kIoMax = 512 << 10;
constexpr int64_t kIoUploadMax = 8192;
constexpr int64_t kIoRowsMax = 65536;

// `bytes` of the context's pinned ring for work on its stream, nullptr if it is
// larger than the ring.  When the ring is used up, waits for the stream, whose
// work no longer needs any of it then.
unsigned char *io_take(pgpu_ctx *c, size_t bytes) {
  bytes = (bytes + 63) / 64 * 64;
  if (bytes > c->io_bytes) return nullptr;
  if (c->io_pos + bytes > c->io_bytes) {
    if (cudaStreamSynchronize(c->st) != cudaSuccess) return nullptr;  // the next call on the stream reports it
    c->io_pos = 0;
  }
  unsigned char *p = c->h_io + 64 + c->io_pos;
  c->io_pos += bytes;
  return p;
}

// Rows of a piece: half a ring of the 8 doubles an uploaded row takes.
int64_t io_rows(const pgpu_ctx *c) { return std::max<int64_t>(1, (int64_t)(c->io_bytes / 128)); }

// Queues a copy of host data to the device through the ring; data too large
// for it is copied at once (the stream is waited for).
cudaError_t put_data(pgpu_ctx *c, void *dst, const void *src, size_t bytes) {
  unsigned char *h = io_take(c, bytes);
  if (h) memcpy(h, src, bytes);
  const cudaError_t e = cudaMemcpyAsync(dst, h ? h : src, bytes, cudaMemcpyHostToDevice, c->st);
  return e != cudaSuccess || h ? e : cudaStreamSynchronize(c->st);
}

// Freeze the slot layout and allocate device memory (first upload).
int freeze(pgpu_ctx *c) {
  if (c->frozen) return PGPU_OK;
  if (c->wakes.empty()) return fail(c, PGPU_EINVAL, "no wakes were added");
  int64_t off = 0;
  for (auto &S : c->sys) {
    // systems start at multiples of kBoxGran slots, so every source tile of
    // the pair kernel is a run of whole precomputed boxes
    off = (off + kBoxGran - 1) / kBoxGran * kBoxGran;
    S.off = off;
    for (int w : S.wakes) {
      c->wakes[w].off = off;
      off += c->wakes[w].cap;
    }
    S.cap = off - S.off;
  }
  c->cap = std::max<int64_t>(off, 1);
  const int64_t cap = c->cap;
  auto alloc = [&](void **p, size_t bytes) -> int {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {
      cudaGetLastError();  // a failed allocation must not surface again at the next launch
      return fail(c, PGPU_ENOMEM, "cudaMalloc(%zu) failed: %s", bytes, cudaGetErrorString(e));
    }
    return PGPU_OK;
  };
  int r;
  if ((r = alloc((void **)&c->x0, 6 * cap * sizeof(double)))) return r;
  if ((r = alloc((void **)&c->acc, 6 * cap * sizeof(double)))) return r;
  if ((r = alloc((void **)&c->rates, 6 * cap * sizeof(double)))) return r;
  if ((r = alloc((void **)&c->sig, cap * sizeof(double)))) return r;
  if ((r = alloc((void **)&c->vol, cap * sizeof(double)))) return r;
  if ((r = alloc((void **)&c->stage, 8 * cap * sizeof(double)))) return r;
  if ((r = alloc((void **)&c->partial, (size_t)kMaxChunks * 6 * cap * sizeof(double)))) return r;
  if ((r = alloc(&c->P, cap * rec_bytes(c)))) return r;
  if ((r = alloc(&c->Q, cap * rec_bytes(c)))) return r;
  const size_t ns = c->sys.size();
  if ((r = alloc((void **)&c->d_sysoff, (ns + 1) * sizeof(int64_t)))) return r;
  if ((r = alloc((void **)&c->d_sysn, ns * sizeof(int64_t)))) return r;
  if ((r = alloc((void **)&c->d_syst, 2 * ns * sizeof(int64_t)))) return r;
  if ((r = alloc((void **)&c->d_plan, (size_t)kNumShapes * (ns + 1) * sizeof(PlanEntry)))) return r;
  if ((r = alloc((void **)&c->d_plan_diag, 2 * sizeof(PlanEntry)))) return r;
  if ((r = alloc((void **)&c->d_plan_field, (ns + 1) * sizeof(PlanEntry)))) return r;
  if ((r = alloc((void **)&c->d_counters, 4 * sizeof(unsigned int)))) return r;
  if ((r = alloc((void **)&c->d_nfull, sizeof(unsigned long long)))) return r;
  if (uses_boxes(c) && (r = alloc((void **)&c->d_box, 2 * box_blocks(c) * sizeof(float4)))) return r;
  if (uses_split(c)) {
    if ((r = alloc((void **)&c->d_L, cap * sizeof(float4)))) return r;
    CK(cudaMemsetAsync(c->d_L, 0, cap * sizeof(float4), c->st));
  }
  // at least the sums of one diagnostics call and a small work plan
  c->io_bytes = std::min<size_t>(std::max<size_t>(8 * cap * sizeof(double), 64 << 10), kIoMax);
  {
    const cudaError_t e = cudaHostAlloc((void **)&c->h_io, 64 + c->io_bytes, cudaHostAllocMapped);
    if (e != cudaSuccess) {
      cudaGetLastError();
      c->h_io = nullptr;
      return fail(c, PGPU_ENOMEM, "pinned transfer buffer of %zu bytes: %s", c->io_bytes, cudaGetErrorString(e));
    }
    c->h_flag = reinterpret_cast<int *>(c->h_io);
    *c->h_flag = 0;
  }
  c->diag_blocks = 2 * c->sms;
  CK(cudaMemsetAsync(c->x0, 0, 6 * cap * sizeof(double), c->st));
  CK(cudaMemsetAsync(c->acc, 0, 6 * cap * sizeof(double), c->st));
  CK(cudaMemsetAsync(c->rates, 0, 6 * cap * sizeof(double), c->st));
  CK(cudaMemsetAsync(c->sig, 0, cap * sizeof(double), c->st));
  CK(cudaMemsetAsync(c->vol, 0, cap * sizeof(double), c->st));
  CK(cudaMemsetAsync(c->partial, 0, (size_t)kMaxChunks * 6 * cap * sizeof(double), c->st));
  CK(cudaMemsetAsync(c->d_counters, 0, 4 * sizeof(unsigned int), c->st));
  CK(cudaMemsetAsync(c->d_nfull, 0, sizeof(unsigned long long), c->st));
  for (int s = 0; s < kNumShapes; ++s) c->grid[s] = fp64(c) ? occupancy<double>(c, s) : occupancy<float>(c, s);
  for (int v = 0; v < kNumSlices; ++v) {
    int nb = 0;
    cudaError_t e;
    if (fp64(c)) {
      const PairFn<double> fn = slices64_fn(v, c->cfg.kernel);
      CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)slices64_bytes(v)));
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, 32 * kSliceWarps, slices64_bytes(v));
    } else {
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, slices_fn(v, c->cfg.kernel, uses_split(c)),
                                                        32 * kSliceWarps, 0);
    }
    if (e != cudaSuccess || nb < 1) nb = 1;
    c->grid_slices[v] = nb * c->sms;
  }
  c->frozen = true;
  c->plan_dirty = true;
  return PGPU_OK;
}

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Owned targets [first, first + count) of system s (all of them unless
// pgpu_set_target_range restricted it), clamped to its particles.
std::pair<int64_t, int64_t> owned(const pgpu_ctx *c, int s) {
  const int64_t n = sys_n(c, s);
  const SysRec &S = c->sys[s];
  if (S.t_count < 0) return {0, n};
  const int64_t lo = std::min(S.t_first, n);
  return {lo, std::min(S.t_count, n - lo)};
}

bool restricted(const pgpu_ctx *c) {
  for (const SysRec &S : c->sys)
    if (S.t_count >= 0) return true;
  return false;
}

// Work list: systems by decreasing work, tiles of the owned targets x source
// chunks each.
std::vector<PlanEntry> build_plan(const pgpu_ctx *c, const std::vector<int> &systems, int shape, int nch) {
  const int64_t TT = (int64_t)kShapes[shape].block * kShapes[shape].tpt;
  const int64_t TILE = kShapes[shape].block;
  std::vector<std::pair<int64_t, int>> order;
  for (int s : systems) {
    const int64_t tn = owned(c, s).second;
    order.push_back({tn * sys_n(c, s), s});
  }
  std::stable_sort(order.begin(), order.end(), [](auto &a, auto &b) { return a.first > b.first; });
  std::vector<PlanEntry> plan;
  int64_t item = 0;
  for (auto &o : order) {
    const int64_t n = sys_n(c, o.second);
    const auto t = owned(c, o.second);
    if (n <= 0 || t.second <= 0) continue;
    PlanEntry e;
    e.off = c->sys[o.second].off;
    e.n = n;
    e.item_start = item;
    e.tiles = ceil_div(t.second, TT);
    e.chunk = ceil_div(ceil_div(n, nch), TILE) * TILE;
    e.toff = t.first;
    e.tn = t.second;
    e.mult = 0;
    item += e.tiles * nch;
    plan.push_back(e);
  }
  PlanEntry sentinel{};
  sentinel.item_start = item;
  plan.push_back(sentinel);
  return plan;
}

// Source chunks per system for one pair launch of `shape` over `systems`:
// enough work items for >= 24 per resident CTA, which keeps the tail of the
// persistent launch below ~2%.
int choose_nch_for(const pgpu_ctx *c, int shape, const std::vector<int> &systems) {
  if (c->cfg.chunks > 0) return std::min(c->cfg.chunks, kMaxChunks);
  const int64_t TT = (int64_t)kShapes[shape].block * kShapes[shape].tpt;
  int64_t tiles = 0;
  for (int s : systems) tiles += ceil_div(owned(c, s).second, TT);
  if (tiles <= 0) return 1;
  const int64_t want = 24LL * c->grid[shape];
  return (int)std::max<int64_t>(1, std::min<int64_t>(kMaxChunks, ceil_div(want, tiles)));
}

std::vector<int> all_systems(const pgpu_ctx *c) {
  std::vector<int> all(c->sys.size());
  for (size_t s = 0; s < all.size(); ++s) all[s] = (int)s;
  return all;
}

int choose_nch(const pgpu_ctx *c, int shape) { return choose_nch_for(c, shape, all_systems(c)); }

// Systems that launch with the g-th group's shape.
std::vector<int> group_systems(const pgpu_ctx *c, int g) {
  std::vector<int> out;
  for (size_t s = 0; s < c->sys.size(); ++s)
    if (c->sys_shape[s] == c->groups[g]) out.push_back((int)s);
  return out;
}

// Graph key part that fixes the launch sequence of one evaluation: the single
// shape, or the set of group shapes.
int launch_layout(const pgpu_ctx *c) {
  if (c->slices >= 0) return 2000 + c->slices;
  if (c->groups.empty()) return c->shape;
  int mask = 0;
  for (int g : c->groups) mask |= 1 << g;
  return 1000 + mask;
}

// Work list of the slices kernel: systems added one by one, then closed for a
// grid of `grid` CTAs with an equal run of rows each; nch is the number of
// partials a tile's rows can be split over.
struct SlicesPlan {
  std::vector<PlanEntry> plan;
  int64_t rows = 0, rps_max = 1;
  int nch = 1;
  void add(int variant, int64_t off, int64_t n, int64_t toff, int64_t tn) {
    if (n <= 0 || tn <= 0) return;
    PlanEntry e;
    e.off = off;
    e.n = n;
    e.item_start = rows;
    e.tiles = ceil_div(tn, 32);
    e.chunk = ceil_div(n, (int64_t)kSliceLen[variant] * kSliceWarps);
    e.toff = toff;
    e.tn = tn;
    // a step near the golden section of the rows, coprime to their number,
    // scatters any run of rows over the system
    e.mult = std::max<int64_t>(1, (int64_t)(0.618 * (double)e.chunk));
    while (std::gcd(e.mult, e.chunk) != 1) ++e.mult;
    e.mult %= e.chunk;
    rows += e.tiles * e.chunk;
    rps_max = std::max(rps_max, e.chunk);
    plan.push_back(e);
  }
  void close(int grid, size_t entries) {
    PlanEntry sentinel{};
    sentinel.item_start = rows;
    // at most kMaxChunks partials per tile: a tile's rows start anywhere in a CTA's run
    sentinel.chunk = std::max<int64_t>(1, std::max(ceil_div(rows, grid), ceil_div(rps_max, kMaxChunks - 1)));
    nch = 1;
    for (const PlanEntry &e : plan)
      nch = std::max(nch, (int)std::min(e.chunk, ceil_div(e.chunk, sentinel.chunk) + 1));
    plan.resize(entries, sentinel);
  }
};

// The systems' owned targets or all of them.
SlicesPlan build_slices_plan(const pgpu_ctx *c, const std::vector<int> &systems, int variant, int grid,
                             bool own_targets) {
  SlicesPlan p;
  for (int s : systems) {
    const int64_t n = sys_n(c, s);
    const auto t = own_targets ? owned(c, s) : std::make_pair<int64_t, int64_t>(0, sys_n(c, s));
    p.add(variant, c->sys[s].off, n, t.first, t.second);
  }
  p.close(grid, c->sys.size() + 1);
  return p;
}

// Whether the closed-form pairs that 32-source slices save outweigh the tiles'
// two targets per staged source, from box tests at 128 positions spread over
// the context's pairs.  F and f are the shares of closed-form pairs in tiles
// and in slices; slices against tiles, in ms: F - f = 0.01 (1M ring of 1000 per
// section) 1409 / 1083; 0.14 (rotor wake of 600,000) 491 / 516; 0.27 (of 200,000)
// 58.6 / 74.5.  They meet at about 1/8.
int rows_pay(pgpu_ctx *c, double pairs, bool *pay) {
  constexpr int kSamples = 128;
  NearSample smp[kSamples];
  double before = 0.0;
  int k = 0;
  for (int s = 0; s < (int)c->sys.size(); ++s) {
    const int64_t n = sys_n(c, s);
    const auto t = owned(c, s);
    const double p = (double)t.second * (double)n;
    for (; k < kSamples && (k + 0.5) / kSamples * pairs < before + p; ++k) {
      const int64_t i = std::min<int64_t>(t.second - 1, (int64_t)(((k + 0.5) / kSamples * pairs - before) / n));
      smp[k] = {c->sys[s].off, n, c->sys[s].off + t.first + i};
    }
    before += p;
  }
  *pay = false;
  if (k == 0) return PGPU_OK;
  NearSample *in = reinterpret_cast<NearSample *>(io_take(c, sizeof(smp)));
  int4 *out = in ? reinterpret_cast<int4 *>(io_take(c, kSamples * sizeof(int4))) : nullptr;
  if (!out) return fail(c, PGPU_ECUDA, "waiting for the pinned transfer buffer failed");
  memcpy(in, smp, k * sizeof(NearSample));
  near_share_kernel<<<k, 256, 0, c->st>>>(static_cast<const float4 *>(c->P), in, 512, out);
  CK(cudaGetLastError());
  c->launches++;
  CK(cudaStreamSynchronize(c->st));
  double gain = 0.0;  // sum of F - f
  for (int j = 0; j < k; ++j) gain += (out[j].y - 0.25 * out[j].x) / out[j].z;
  *pay = gain > k / 8.0;
  return PGPU_OK;
}

// Slice length of the row list: 32 sources (0) or 64 (1).  Longer slices share
// the box and the fold among more pairs, shorter ones find more far pairs and
// keep all eight warps of a row busy in systems of a few hundred particles.
// Times per evaluation, 32-source / 64-source, in us:
//   one Gaussian ring  5000: 55 / 61;  8000: 110 / 106;  20,000: 575 / 541
//   FP64  10,000: 562 / 583;  7 systems of 6000: 1310 / 1323;  781 of 512: 1435 / 1856
//   high-order  781 of 512: 507 / 485, FP64 913 / 907;  1562 of 256: 302 / 315, 520 / 619
// A wake of several systems has pairs / targets sources on average.
int slice_variant(double pairs, double targets, int kernel) {
  return pairs >= 4.5e7 && pairs >= (kernel == PGPU_KERNEL_HIGHORDER ? 512.0 : 4000.0) * targets ? 1 : 0;
}

// Variant of the slices kernel for the context's next evaluations, -1 for the
// CTA-wide tiles of pair_kernel.  A shape or chunk count that was asked for, and
// a tuned shape, keep the tiles.  Times per evaluation, CTA-wide 128 x 2 tiles
// / 32-source / 64-source slices, in us:
//   Gaussian rings (sigma = 0.02)  5000: 127 / 55 / 61;  8000: 184 / 110 / 106;
//     20,000: 658 / 575 / 541;  40,000: 2103 / 2228 / 2065;  60,000: 4388 / 4982 / 4593
//   station rings (sigma = 0.1)  1000: 53 / 17 / 19;  5000: 167 / 62 / 66;
//     20,000: 850 / 687 / 658;  40,000: 2856 / 2701 / 2541
//   rotor wakes, split positions  4800: 168 / 58 / 72;  24,000: 1308 / 931 / 949;
//     200,000: 76,306 / 58,493 / 58,840
// The CTA-wide tiles need about 24 items per CTA to fill the device and gain
// two targets per staged source; the slices' finer boxes find more far pairs.
// So FP32C Gaussian contexts take slices while all systems together have fewer
// than 48,000 targets (16 rings of 2000-40,000, 169,125 in all: 4.4 ms in tiles).
// Beyond, contexts with split positions, which are meant for dense filaments,
// keep 32-source slices where the finer boxes pay (rows_pay).
// The high-order kernel's full terms for every pair take the slices at any size
// (1000 particles: 14 against 52 us in 256 x 1 tiles; 60,000: 6.7 against 8.9 ms
// per call; FP64 60,001: 12.5 against 14.2 ms, 400,000: 553 against 610 ms), and
// so does the Gaussian kernel in FP64 (5000 particles: 158 against 301 us in 128
// x 1 tiles; 60,001: 10.7 against 12.0 ms; 1M: 2914 against 3065 ms), except for
// systems of 33 to 256 particles with more than 150,000 targets in all, which
// leave warps of a row idle (2000 of 100: 627 us in rows, 400 in tiles; 1000 of
// 200: 603 and 531; but 781 of 129: 327 and 358; 16,000 of 25: 1081 and 1351).
int choose_slices(pgpu_ctx *c, int *variant) {
  *variant = -1;
  if (!c->auto_shape || c->cfg.chunks > 0 || c->sur) return PGPU_OK;
  double pairs = 0.0, targets = 0.0;
  for (int s = 0; s < (int)c->sys.size(); ++s) {
    const double tn = (double)owned(c, s).second;
    pairs += tn * (double)sys_n(c, s);
    targets += tn;
  }
  if (targets > 48000.0 && c->cfg.kernel == PGPU_KERNEL_GAUSSIAN && !fp64(c)) {
    bool pay = false;
    if (uses_split(c))
      if (int r = rows_pay(c, pairs, &pay)) return r;
    if (!pay) return PGPU_OK;
  }
  if (fp64(c) && c->cfg.kernel == PGPU_KERNEL_GAUSSIAN && targets > 150000.0 && pairs > 32.0 * targets &&
      pairs <= 256.0 * targets)
    return PGPU_OK;
  *variant = uses_split(c) ? 0 : slice_variant(pairs, targets, c->cfg.kernel);
  return PGPU_OK;
}

int upload_plan(pgpu_ctx *c) {
  if (!c->plan_dirty) return PGPU_OK;
  int r = check_contiguous(c);
  if (r) return r;
  const size_t ns = c->sys.size();
  c->groups.clear();
  if (!c->sur && c->sys_shape.size() == ns) {
    for (int sh : c->sys_shape)
      if (std::find(c->groups.begin(), c->groups.end(), sh) == c->groups.end()) c->groups.push_back(sh);
    std::sort(c->groups.begin(), c->groups.end());
    if (c->groups.size() == 1) {  // one shape after all: the single-launch path
      c->shape = c->groups[0];
      c->groups.clear();
    }
  }
  std::vector<PlanEntry> plan;
  c->slices = -1;
  if (c->groups.empty() && (r = choose_slices(c, &c->slices))) return r;
  if (c->slices >= 0) {
    SlicesPlan p = build_slices_plan(c, all_systems(c), c->slices, c->grid_slices[c->slices], true);
    plan = std::move(p.plan);
    c->nch = p.nch;
  } else if (c->groups.empty()) {
    // the surrogate writes one chunk of rates per evaluation
    c->nch = c->sur ? 1 : choose_nch(c, c->shape);
    plan = build_plan(c, all_systems(c), c->shape, c->nch);
    // Unused tail entries keep the sentinel item_start so the device search is bounded.
    plan.resize(ns + 1, plan.back());
  } else {
    // one chunk count for every group (the stage kernel sums nch chunks of
    // every particle): the largest any group's launch wants
    c->nch = 1;
    for (size_t g = 0; g < c->groups.size(); ++g)
      c->nch = std::max(c->nch, choose_nch_for(c, c->groups[g], group_systems(c, (int)g)));
    for (size_t g = 0; g < c->groups.size(); ++g) {
      std::vector<PlanEntry> p = build_plan(c, group_systems(c, (int)g), c->groups[g], c->nch);
      p.resize(ns + 1, p.back());
      plan.insert(plan.end(), p.begin(), p.end());
    }
  }
  std::vector<int64_t> off(c->sys.size() + 1), n(c->sys.size());
  for (size_t s = 0; s < c->sys.size(); ++s) { off[s] = c->sys[s].off; n[s] = sys_n(c, (int)s); }
  off[c->sys.size()] = c->cap;
  std::vector<int64_t> t(2 * c->sys.size());
  for (size_t k = 0; k < c->sys.size(); ++k) {
    // an unrestricted system owns every slot, including particles appended later
    const auto o = owned(c, (int)k);
    t[2 * k] = c->sys[k].t_count < 0 ? 0 : o.first;
    t[2 * k + 1] = c->sys[k].t_count < 0 ? INT64_MAX : o.first + o.second;
  }
  CK(put_data(c, c->d_plan, plan.data(), plan.size() * sizeof(PlanEntry)));
  CK(put_data(c, c->d_sysoff, off.data(), off.size() * sizeof(int64_t)));
  CK(put_data(c, c->d_sysn, n.data(), n.size() * sizeof(int64_t)));
  CK(put_data(c, c->d_syst, t.data(), t.size() * sizeof(int64_t)));
  c->plan_dirty = false;
  return PGPU_OK;
}

void account_pairs(pgpu_ctx *c, int launches) {
  for (size_t s = 0; s < c->sys.size(); ++s) {
    const int64_t n = sys_n(c, (int)s), tn = owned(c, (int)s).second;
    c->pairs_acc += launches * tn * (n > 0 ? n - 1 : 0);
    c->selfs_acc += launches * tn;
  }
}

int launch_boxes(pgpu_ctx *c) {
  const int64_t nb = box_blocks(c);
  const int grid = (int)std::min<int64_t>(ceil_div(nb, 8), 16LL * c->sms);  // 8 warps per CTA, one per block
  box_kernel<<<grid, 256, 0, c->st>>>(static_cast<const float4 *>(c->P), c->d_sysoff, c->d_sysn, (int)c->sys.size(),
                                      c->cap, nb, c->d_box);
  CK(cudaGetLastError());
  c->launches++;
  return PGPU_OK;
}

// Kernel launches of one rate evaluation by the direct sum.
int64_t eval_launches(const pgpu_ctx *c) {
  return (int64_t)std::max<size_t>(1, c->groups.size()) + (uses_boxes(c) && c->slices < 0 ? 1 : 0);
}

// Start (which = 0) or end event of a pair launch.  In a captured step the
// record is a timestamp node of the graph (external), on a branch of its own
// beside the kernels: in line with them, the eight records of an RK4 step
// kept the next kernel waiting for a few us each (1000 particles: 81 us per
// step with the branch, 107 us without it, 71 us with no records at all).
// Nothing orders the start record before the pair kernel then: both follow the
// previous stage kernel.  Readings in us, branch / records that bracket the
// launch / ncu's duration of the kernel alone, with cold caches: 25 particles
// 7.1 / 11.2 / 8.5, 1000: 11.2 / 15.6 / 12.2, 5000: 54.8 / 59.6 / 57.7, 20,000:
// 657 / 661.  A kernel that waits for the start record too reads as the
// bracketed launch and costs the 1000-particle step 22 us.
int record_time(pgpu_ctx *c, int slot, int which) {
  if (!c->timing || slot < 0) return PGPU_OK;
  if (!c->capturing) {
    CK(cudaEventRecord(c->ev[slot][which], c->st));
    return PGPU_OK;
  }
  CK(cudaEventRecord(c->ev_side, c->st));
  CK(cudaStreamWaitEvent(c->st_side, c->ev_side, 0));
  CK(cudaEventRecordWithFlags(c->ev[slot][which], c->st_side, cudaEventRecordExternal));
  c->side_used = true;
  return PGPU_OK;
}

// Joins the side branch of a captured step.
int join_side(pgpu_ctx *c) {
  if (!c->side_used) return PGPU_OK;
  c->side_used = false;
  CK(cudaEventRecord(c->ev_side, c->st_side));
  CK(cudaStreamWaitEvent(c->st, c->ev_side, 0));
  return PGPU_OK;
}

// One launch of the row list `a` of slices variant v.
template <typename T> int launch_rows(pgpu_ctx *c, int v, const PairArgs<T> &a) {
  if constexpr (sizeof(T) == 4) {
    slices_fn(v, c->cfg.kernel, uses_split(c))<<<c->grid_slices[v], 32 * kSliceWarps, 0, c->st>>>(a);
  } else {
    slices64_fn(v, c->cfg.kernel)<<<c->grid_slices[v], 32 * kSliceWarps, slices64_bytes(v), c->st>>>(a);
  }
  CK(cudaGetLastError());
  c->launches++;
  return PGPU_OK;
}

template <typename T> int launch_pair(pgpu_ctx *c, int slot) {
  PairArgs<T> a;
  a.P = static_cast<const v4_t<T> *>(c->P);
  a.Q = static_cast<const v4_t<T> *>(c->Q);
  a.partial = c->partial;
  a.plan = c->d_plan;
  a.nsys = (int)c->sys.size();
  a.nch = c->nch;
  a.cap = c->cap;
  a.nu2 = (T)(2.0 * c->cfg.nu);
  a.counters = c->d_counters;
  a.nfull = c->d_nfull;
  if (uses_boxes(c) && c->slices < 0) {
    // source boxes of the current records, ahead of (and outside the timing of) the pair launch
    int r = launch_boxes(c);
    if (r) return r;
    a.box = c->d_box;
  }
  a.L = c->d_L;
  if (int r = record_time(c, slot, 0)) return r;
  if (c->slices >= 0) {
    if (int r = launch_rows(c, c->slices, a)) return r;
  } else if (c->groups.empty()) {
    pair_fn<T>(c->shape, c->cfg.kernel, uses_split(c))<<<c->grid[c->shape], kShapes[c->shape].block, 0, c->st>>>(a);
    CK(cudaGetLastError());
    c->launches++;
  } else {
    // one launch per group shape, each over its own plan; the launches share
    // the work counters, which each resets when its last CTA leaves
    for (size_t g = 0; g < c->groups.size(); ++g) {
      const int sh = c->groups[g];
      a.plan = c->d_plan + g * (c->sys.size() + 1);
      pair_fn<T>(sh, c->cfg.kernel, uses_split(c))<<<c->grid[sh], kShapes[sh].block, 0, c->st>>>(a);
      CK(cudaGetLastError());
      c->launches++;
    }
  }
  if (int r = record_time(c, slot, 1)) return r;
  if (!c->capturing) account_pairs(c, 1);
  return PGPU_OK;
}

int launch_stage(pgpu_ctx *c, int scheme, int stage, double dt) {
  StageArgs s;
  s.x0 = c->x0; s.acc = c->acc; s.rates = c->rates; s.sig = c->sig; s.vol = c->vol; s.L = c->d_L;
  s.partial = c->partial; s.P = c->P; s.Q = c->Q;
  s.sys_off = c->d_sysoff; s.sys_n = c->d_sysn; s.sys_t = c->d_syst; s.nsys = (int)c->sys.size();
  s.nch = c->nch; s.cap = c->cap; s.scheme = scheme; s.stage = stage; s.dt = dt;
  for (int m = 0; m < 3; ++m) s.vinf[m] = c->cfg.vinf[m];
  s.flag = c->h_flag;
  const int grid = (int)std::min<int64_t>(ceil_div(c->cap, kStageParticles), 10LL * c->sms);
  if (fp64(c)) stage_kernel<double><<<grid, kStageBlock, 0, c->st>>>(s);
  else stage_kernel<float><<<grid, kStageBlock, 0, c->st>>>(s);
  CK(cudaGetLastError());
  c->launches++;
  return PGPU_OK;
}

int launch_pack(pgpu_ctx *c, int64_t lo, int64_t hi) {
  if (hi <= lo) return PGPU_OK;
  const int block = 256;
  const int grid = (int)std::min<int64_t>(ceil_div(hi - lo, block), 16LL * c->sms);
  if (fp64(c)) pack_kernel<double><<<grid, block, 0, c->st>>>(c->x0, c->sig, c->vol, c->P, c->Q, nullptr, lo, hi, c->cap);
  else pack_kernel<float><<<grid, block, 0, c->st>>>(c->x0, c->sig, c->vol, c->P, c->Q, c->d_L, lo, hi, c->cap);
  CK(cudaGetLastError());
  c->launches++;
  return PGPU_OK;
}

int surrogate_eval(pgpu_ctx *c);
void surrogate_free(pgpu_ctx *c);
int surrogate_pick_targets(pgpu_ctx *c, SurrogateState *s);

int launch_eval(pgpu_ctx *c, int slot) {
  if (c->sur) return surrogate_eval(c);
  return fp64(c) ? launch_pair<double>(c, slot) : launch_pair<float>(c, slot);
}

// Reads the pair-kernel times of event slots [base, base + nslots), waiting for
// the last of them.
int collect_timing(pgpu_ctx *c, int nslots, int base = 0) {
  if (!c->timing || c->sur) return PGPU_OK;  // surrogate evaluations keep their own phase times
  CK(cudaEventSynchronize(c->ev[base + nslots - 1][1]));
  for (int k = base; k < base + nslots; ++k) {
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, c->ev[k][0], c->ev[k][1]));
    c->pair_ms += ms;
    c->pair_launches++;
  }
  return PGPU_OK;
}

int stages_of(int scheme) { return scheme == PGPU_RK4 ? 4 : scheme == PGPU_RK3 ? 3 : 1; }

int record_step(pgpu_ctx *c, int scheme, double dt, int base = 0) {
  const int ns = stages_of(scheme);
  for (int k = 0; k < ns; ++k) {
    int r = launch_eval(c, base + k);
    if (r) return r;
    if ((r = launch_stage(c, scheme, k, dt))) return r;
  }
  return PGPU_OK;
}

int wake_ok(pgpu_ctx *c, int32_t wake) {
  if (!c) return PGPU_EINVAL;
  if (wake < 0 || wake >= (int32_t)c->wakes.size()) return fail(c, PGPU_EINVAL, "invalid wake id %d", wake);
  return PGPU_OK;
}

int upload_rows(pgpu_ctx *c, const WakeRec &W, int64_t first, int64_t m, const double *pos, const double *alpha,
                const double *sigma, const double *vol) {
  if (m <= 0) return PGPU_OK;
  if (!pos || !alpha || !sigma || !vol) return fail(c, PGPU_EINVAL, "null particle array");
  auto fn = fp64(c) ? upload_kernel<double> : upload_kernel<float>;
  auto launch = [&](const double *rows, int64_t at, int64_t k) -> int {
    const int grid = (int)std::min<int64_t>(ceil_div(k, kIoRows), 8LL * c->sms);
    fn<<<grid, kIoRows, 0, c->st>>>(rows, k, W.off + first + at, c->cap, c->x0, c->sig, c->vol, c->P, c->Q, c->d_L);
    CK(cudaGetLastError());
    c->launches++;
    return PGPU_OK;
  };
  if (m <= kIoUploadMax) {
    const int64_t piece = io_rows(c);
    for (int64_t at = 0; at < m; at += piece) {
      const int64_t k = std::min(piece, m - at);
      double *h = reinterpret_cast<double *>(io_take(c, 8 * k * sizeof(double)));
      if (!h) return fail(c, PGPU_ECUDA, "waiting for the pinned transfer buffer failed");
      memcpy(h, pos + 3 * at, 3 * k * sizeof(double));
      memcpy(h + 3 * k, alpha + 3 * at, 3 * k * sizeof(double));
      memcpy(h + 6 * k, sigma + at, k * sizeof(double));
      memcpy(h + 7 * k, vol + at, k * sizeof(double));
      if (int r = launch(h, at, k)) return r;
    }
    return PGPU_OK;
  }
  CK(cudaMemcpyAsync(c->stage, pos, 3 * m * sizeof(double), cudaMemcpyHostToDevice, c->st));
  CK(cudaMemcpyAsync(c->stage + 3 * m, alpha, 3 * m * sizeof(double), cudaMemcpyHostToDevice, c->st));
  CK(cudaMemcpyAsync(c->stage + 6 * m, sigma, m * sizeof(double), cudaMemcpyHostToDevice, c->st));
  CK(cudaMemcpyAsync(c->stage + 7 * m, vol, m * sizeof(double), cudaMemcpyHostToDevice, c->st));
  return launch(c->stage, 0, m);
}

}  // namespace

extern "C" {

void pgpu_config_default(pgpu_config *cfg) {
  memset(cfg, 0, sizeof(*cfg));
  cfg->precision = PGPU_FP32C;
  cfg->device = 0;
  cfg->nu = 1.56e-5;
  cfg->use_graphs = 1;
}

const char *pgpu_version(void) { return "pawan_b200 0.1 (sm_100a)"; }

int pgpu_create(pgpu_ctx **out, const pgpu_config *cfg) {
  if (!out) return create_fail(nullptr, PGPU_EINVAL, "no output pointer for the context");
  *out = nullptr;
  pgpu_ctx *c = new pgpu_ctx;
  if (cfg) c->cfg = *cfg;
  else pgpu_config_default(&c->cfg);
  if (c->cfg.precision != PGPU_FP32C && c->cfg.precision != PGPU_FP64)
    return create_fail(c, PGPU_EINVAL, "unknown precision %d", c->cfg.precision);
  if (c->cfg.kernel != PGPU_KERNEL_GAUSSIAN && c->cfg.kernel != PGPU_KERNEL_HIGHORDER)
    return create_fail(c, PGPU_EINVAL, "unknown regularisation kernel %d", c->cfg.kernel);
  if (c->cfg.block > 0 || c->cfg.tpt > 0) {
    int found = -1;
    for (int s = 0; s < kNumShapes; ++s)
      if ((c->cfg.block <= 0 || kShapes[s].block == c->cfg.block) && (c->cfg.tpt <= 0 || kShapes[s].tpt == c->cfg.tpt)) {
        found = s;
        break;
      }
    if (found < 0)
      return create_fail(c, PGPU_EINVAL, "no compiled pair-kernel shape with block %d and %d targets per thread",
                         c->cfg.block, c->cfg.tpt);
    c->shape = found;
    c->auto_shape = false;
    c->shape_asked = true;
  } else if (c->cfg.kernel == PGPU_KERNEL_GAUSSIAN) {
    // untuned defaults: the fastest Gaussian shapes on the 1M ring, FP32C
    // 128 x 2 (1075 ms per evaluation against 1163 ms for 256 x 1) and FP64
    // 128 x 1 (3.09 s against 3.22 s)
    c->shape = c->cfg.precision == PGPU_FP32C ? 1 : 0;
  }
  cudaError_t e = cudaSetDevice(c->cfg.device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, c->cfg.device);
  for (int k = 0; k < 8 && e == cudaSuccess; ++k) {
    e = cudaEventCreate(&c->ev[k][0]);
    if (e == cudaSuccess) e = cudaEventCreate(&c->ev[k][1]);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return create_fail(c, PGPU_ECUDA, "device %d: %s", c->cfg.device, cudaGetErrorString(e));
  }
  g_create_err[0] = '\0';
  *out = c;
  return PGPU_OK;
}

int pgpu_destroy(pgpu_ctx *c) {
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  cudaStreamSynchronize(c->st);
  surrogate_free(c);
  for (auto &g : c->graphs) cudaGraphExecDestroy(g.second);
  for (auto g : c->graph_defs) cudaGraphDestroy(g);
  void *ptrs[] = {c->x0, c->acc, c->rates, c->sig, c->vol, c->partial, c->stage, c->P, c->Q,
                  c->d_sysoff, c->d_sysn, c->d_syst, c->d_plan, c->d_plan_diag, c->d_plan_field, c->d_field,
                  c->d_counters, c->d_nfull, c->d_merge, c->d_merge_tmp, c->d_box, c->d_L};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  for (int k = 0; k < 8; ++k) { cudaEventDestroy(c->ev[k][0]); cudaEventDestroy(c->ev[k][1]); }
  if (c->h_io) cudaFreeHost(c->h_io);
  if (c->st_side) cudaStreamDestroy(c->st_side);
  if (c->ev_side) cudaEventDestroy(c->ev_side);
  if (c->st_copy) cudaStreamSynchronize(c->st_copy);
  for (int s = 0; s < 2; ++s) {
    if (c->d_snap[s]) cudaFree(c->d_snap[s]);
    if (c->h_snap[s]) cudaFreeHost(c->h_snap[s]);
    if (c->snap_gathered[s]) cudaEventDestroy(c->snap_gathered[s]);
    if (c->snap_copied[s]) cudaEventDestroy(c->snap_copied[s]);
  }
  if (c->st_copy) cudaStreamDestroy(c->st_copy);
  cudaStreamDestroy(c->st);
  delete c;
  return PGPU_OK;
}

int pgpu_add_wake(pgpu_ctx *c, int32_t system, int64_t capacity, int32_t *wake_id) {
  if (!c) return PGPU_EINVAL;
  if (c->frozen) return fail(c, PGPU_EINVAL, "wakes must be added before the first particle upload");
  if (system < 0 || system > 1 << 20) return fail(c, PGPU_EINVAL, "invalid system id %d", system);
  if (capacity < 0 || capacity > (int64_t)1 << 31) return fail(c, PGPU_EINVAL, "invalid capacity %lld", (long long)capacity);
  if ((int)c->sys.size() <= system) c->sys.resize(system + 1);
  WakeRec w{system, capacity, 0, 0};
  c->wakes.push_back(w);
  c->sys[system].wakes.push_back((int)c->wakes.size() - 1);
  if (wake_id) *wake_id = (int32_t)c->wakes.size() - 1;
  return PGPU_OK;
}

int pgpu_set_particles(pgpu_ctx *c, int32_t wake, int64_t n, const double *pos, const double *alpha,
                       const double *sigma, const double *vol) {
  int r = wake_ok(c, wake);
  if (r) return r;
  DeviceScope device_scope(c->cfg.device);
  if ((r = freeze(c))) return r;
  WakeRec &W = c->wakes[wake];
  if (n < 0 || n > W.cap) return fail(c, PGPU_EINVAL, "n=%lld exceeds the capacity %lld of wake %d", (long long)n, (long long)W.cap, wake);
  if ((r = upload_rows(c, W, 0, n, pos, alpha, sigma, vol))) return r;
  if (W.n != n) c->plan_dirty = true;  // the work list depends on the sizes alone
  W.n = n;
  return PGPU_OK;
}

int pgpu_append_particles(pgpu_ctx *c, int32_t wake, int64_t m, const double *pos, const double *alpha,
                          const double *sigma, const double *vol) {
  int r = wake_ok(c, wake);
  if (r) return r;
  DeviceScope device_scope(c->cfg.device);
  if ((r = freeze(c))) return r;
  WakeRec &W = c->wakes[wake];
  if (c->sys[W.sys].wakes.back() != wake) return fail(c, PGPU_EINVAL, "only the last wake of a system can grow");
  if (m < 0 || W.n + m > W.cap) return fail(c, PGPU_EINVAL, "appending %lld particles exceeds the capacity of wake %d", (long long)m, wake);
  if ((r = upload_rows(c, W, W.n, m, pos, alpha, sigma, vol))) return r;
  // Appended particles start a step with a zero RK accumulator.
  W.n += m;
  c->plan_dirty = true;
  return PGPU_OK;
}

int pgpu_get_num_particles(pgpu_ctx *c, int32_t wake, int64_t *n) {
  int r = wake_ok(c, wake);
  if (r) return r;
  if (n) *n = c->wakes[wake].n;
  return PGPU_OK;
}

// Components 0..2 of the wake's rows to a and, unless b is null, 3..5 to b.
static int download_rows(pgpu_ctx *c, const double *src, const WakeRec &W, double *a, double *b) {
  if (W.n == 0) return PGPU_OK;
  const int parts = b ? 2 : 1;
  auto launch = [&](int64_t at, int64_t k, double *dst) -> int {
    const int grid = (int)std::min<int64_t>(ceil_div(k, kIoRows), 8LL * c->sms);
    gather_kernel<<<grid, kIoRows, 0, c->st>>>(src, k, W.off + at, c->cap, parts, dst);
    CK(cudaGetLastError());
    c->launches++;
    return PGPU_OK;
  };
  if (W.n > kIoRowsMax) {
    if (int r = launch(0, W.n, c->stage)) return r;
    CK(cudaMemcpyAsync(a, c->stage, 3 * W.n * sizeof(double), cudaMemcpyDeviceToHost, c->st));
    if (b) CK(cudaMemcpyAsync(b, c->stage + 3 * W.n, 3 * W.n * sizeof(double), cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
    return PGPU_OK;
  }
  // two pieces in the ring at a time, then on to the caller's arrays
  const int64_t piece = io_rows(c);
  for (int64_t at = 0; at < W.n; at += 2 * piece) {
    double *h[2] = {nullptr, nullptr};
    for (int q = 0; q < 2; ++q) {
      const int64_t lo = at + q * piece, k = std::min(piece, W.n - lo);
      if (k <= 0) break;
      h[q] = reinterpret_cast<double *>(io_take(c, 3 * parts * k * sizeof(double)));
      if (!h[q]) return fail(c, PGPU_ECUDA, "waiting for the pinned transfer buffer failed");
      if (q == 1 && h[1] <= h[0]) {  // the ring started over and the first piece has landed: take it out first
        memcpy(a + 3 * at, h[0], 3 * piece * sizeof(double));
        if (b) memcpy(b + 3 * at, h[0] + 3 * piece, 3 * piece * sizeof(double));
        h[0] = nullptr;
      }
      if (int r = launch(lo, k, h[q])) return r;
    }
    CK(cudaStreamSynchronize(c->st));
    for (int q = 0; q < 2; ++q) {
      const int64_t lo = at + q * piece, k = std::min(piece, W.n - lo);
      if (!h[q]) continue;
      memcpy(a + 3 * lo, h[q], 3 * k * sizeof(double));
      if (b) memcpy(b + 3 * lo, h[q] + 3 * k, 3 * k * sizeof(double));
    }
    c->io_pos = 0;  // the stream is idle: nothing needs the ring any more
  }
  return PGPU_OK;
}

int pgpu_get_state(pgpu_ctx *c, int32_t wake, double *pos, double *alpha) {
  int r = wake_ok(c, wake);
  if (r) return r;
  DeviceScope device_scope(c->cfg.device);
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  if (!pos || !alpha) return fail(c, PGPU_EINVAL, "null output array");
  return download_rows(c, c->x0, c->wakes[wake], pos, alpha);
}

int pgpu_get_rates(pgpu_ctx *c, int32_t wake, double *vel, double *dalpha) {
  int r = wake_ok(c, wake);
  if (r) return r;
  DeviceScope device_scope(c->cfg.device);
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  if (!vel || !dalpha) return fail(c, PGPU_EINVAL, "null output array");
  return download_rows(c, c->rates, c->wakes[wake], vel, dalpha);
}

static int flat_io(pgpu_ctx *c, double *flat, const int64_t *maxn, int32_t nwakes, int dir, const double *soa_src) {
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  if (!flat || !maxn || nwakes != (int32_t)c->wakes.size()) return fail(c, PGPU_EINVAL, "flat state needs one capacity per wake");
  int64_t off = 0;
  for (int w = 0; w < nwakes; ++w) {
    const WakeRec &W = c->wakes[w];
    if (maxn[w] < W.n) return fail(c, PGPU_EINVAL, "maxn[%d] is smaller than the wake size", w);
    const int64_t sz = 6 * maxn[w];
    if (W.n > 0) {
      const int grid = (int)std::min<int64_t>(ceil_div(W.n, 256), 16LL * c->sms);
      if (dir == 0) {
        CK(cudaMemcpyAsync(c->stage, flat + off, 3 * W.n * sizeof(double), cudaMemcpyHostToDevice, c->st));
        CK(cudaMemcpyAsync(c->stage + 3 * W.n, flat + off + 3 * maxn[w], 3 * W.n * sizeof(double), cudaMemcpyHostToDevice, c->st));
        flat_kernel<<<grid, 256, 0, c->st>>>(c->stage, W.n, W.n, W.off, c->cap, c->x0, 0);
        CK(cudaGetLastError());
        c->launches++;
        int r = launch_pack(c, W.off, W.off + W.n);
        if (r) return r;
        CK(cudaStreamSynchronize(c->st));
      } else {
        flat_kernel<<<grid, 256, 0, c->st>>>(c->stage, W.n, W.n, W.off, c->cap, const_cast<double *>(soa_src), 1);
        CK(cudaGetLastError());
        c->launches++;
        CK(cudaMemcpyAsync(flat + off, c->stage, 3 * W.n * sizeof(double), cudaMemcpyDeviceToHost, c->st));
        CK(cudaMemcpyAsync(flat + off + 3 * maxn[w], c->stage + 3 * W.n, 3 * W.n * sizeof(double), cudaMemcpyDeviceToHost, c->st));
        CK(cudaStreamSynchronize(c->st));
      }
    }
    off += sz;
  }
  return PGPU_OK;
}

int pgpu_set_states_flat(pgpu_ctx *c, const double *state, const int64_t *maxn, int32_t nwakes) {
  return flat_io(c, const_cast<double *>(state), maxn, nwakes, 0, nullptr);
}
int pgpu_get_states_flat(pgpu_ctx *c, double *state, const int64_t *maxn, int32_t nwakes) {
  return flat_io(c, state, maxn, nwakes, 1, c ? c->x0 : nullptr);
}
int pgpu_get_rates_flat(pgpu_ctx *c, double *rate, const int64_t *maxn, int32_t nwakes) {
  return flat_io(c, rate, maxn, nwakes, 1, c ? c->rates : nullptr);
}

int pgpu_solve(pgpu_ctx *c) {
  NvtxRange nvtx("pgpu_solve");
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  int r = upload_plan(c);
  if (r) return r;
  if ((r = launch_eval(c, 0))) return r;
  if ((r = launch_stage(c, -1, 0, 0.0))) return r;
  return collect_timing(c, 1);
}

int pgpu_set_target_range(pgpu_ctx *c, int32_t system, int64_t first, int64_t count) {
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  if (system < 0 || system >= (int32_t)c->sys.size()) return fail(c, PGPU_EINVAL, "invalid system id %d", system);
  if (uses_split(c) && count >= 0)
    return fail(c, PGPU_EINVAL, "split positions are not exchanged between contexts: use one context per system");
  if (count >= 0 && first < 0) return fail(c, PGPU_EINVAL, "negative first target %lld", (long long)first);
  SysRec &S = c->sys[system];
  S.t_first = count < 0 ? 0 : first;
  S.t_count = count < 0 ? -1 : count;
  c->plan_dirty = true;
  // the surrogate's sampled check draws from the owned targets
  if (c->sur) return surrogate_pick_targets(c, c->sur);
  return PGPU_OK;
}

int pgpu_stage(pgpu_ctx *c, int scheme, int stage, double dt) {
  NvtxRange nvtx("pgpu_stage");
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  if (scheme != PGPU_EULER && scheme != PGPU_RK3 && scheme != PGPU_RK4) return fail(c, PGPU_EINVAL, "unknown scheme %d", scheme);
  if (stage < 0 || stage >= stages_of(scheme)) return fail(c, PGPU_EINVAL, "stage %d out of range for scheme %d", stage, scheme);
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  int r = upload_plan(c);
  if (r) return r;
  if ((r = launch_eval(c, 0))) return r;
  if ((r = launch_stage(c, scheme, stage, dt))) return r;
  return collect_timing(c, 1);
}

int pgpu_records(pgpu_ctx *c, int32_t system, void **P, void **Q) {
  if (!c || !P || !Q) return PGPU_EINVAL;
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  if (system < 0 || system >= (int32_t)c->sys.size()) return fail(c, PGPU_EINVAL, "invalid system id %d", system);
  const size_t rb = rec_bytes(c);
  *P = static_cast<char *>(c->P) + (size_t)c->sys[system].off * rb;
  *Q = static_cast<char *>(c->Q) + (size_t)c->sys[system].off * rb;
  return PGPU_OK;
}

int pgpu_step(pgpu_ctx *c, int scheme, double dt, int32_t nsteps) {
  NvtxRange nvtx("pgpu_step");
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  if (scheme != PGPU_EULER && scheme != PGPU_RK3 && scheme != PGPU_RK4) return fail(c, PGPU_EINVAL, "unknown scheme %d", scheme);
  if (nsteps < 0) return fail(c, PGPU_EINVAL, "negative step count");
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  if (restricted(c))
    return fail(c, PGPU_EINVAL, "a context with target ranges steps stage by stage (pgpu_stage), with the source "
                                "records of the other targets exchanged between stages");
  int r = upload_plan(c);
  if (r) return r;
  const int ns = stages_of(scheme);
  if (!c->cfg.use_graphs || c->sur) {  // the surrogate's tree build synchronises with the host
    for (int i = 0; i < nsteps; ++i) {
      if ((r = record_step(c, scheme, dt))) return r;
      if ((r = collect_timing(c, ns))) return r;
    }
    return PGPU_OK;
  }
  // With timing on, the steps of a call alternate between two graphs with
  // their own event slots, so that a step's times are read while the next one
  // runs (5000 particles: the device would idle 15 us between steps).
  auto graph = [&](int base, cudaGraphExec_t *out) -> int {
    auto key = std::make_tuple(scheme, dt, launch_layout(c), c->nch, c->timing, base);
    auto it = c->graphs.find(key);
    if (it == c->graphs.end()) {
      cudaGraph_t g;
      if (c->timing && !c->st_side) {
        CK(cudaStreamCreateWithFlags(&c->st_side, cudaStreamNonBlocking));
        CK(cudaEventCreateWithFlags(&c->ev_side, cudaEventDisableTiming));
      }
      c->side_used = false;
      CK(cudaStreamBeginCapture(c->st, cudaStreamCaptureModeThreadLocal));
      const int64_t before = c->launches;
      c->capturing = true;
      int rr = record_step(c, scheme, dt, base);
      if (!rr) rr = join_side(c);
      c->capturing = false;
      cudaError_t e = cudaStreamEndCapture(c->st, &g);
      if (rr) return rr;
      if (e != cudaSuccess) return fail(c, PGPU_ECUDA, "stream capture failed: %s", cudaGetErrorString(e));
      c->launches = before;  // counted at replay
      cudaGraphExec_t ex;
      CK(cudaGraphInstantiate(&ex, g, 0));
      c->graph_defs.push_back(g);
      it = c->graphs.emplace(key, ex).first;
    }
    *out = it->second;
    return PGPU_OK;
  };
  for (int i = 0; i < nsteps; ++i) {
    cudaGraphExec_t ex;
    const int base = c->timing && (i & 1) ? 4 : 0;
    if ((r = graph(base, &ex))) return r;
    CK(cudaGraphLaunch(ex, c->st));
    c->launches += (1 + eval_launches(c)) * ns;
    account_pairs(c, ns);
    if (i > 0 && (r = collect_timing(c, ns, 4 - base))) return r;
  }
  return nsteps > 0 ? collect_timing(c, ns, c->timing && ((nsteps - 1) & 1) ? 4 : 0) : PGPU_OK;
}

int pgpu_diagnose_partial(pgpu_ctx *c, int32_t system, double *fields) {
  NvtxRange nvtx("pgpu_diagnose_partial");
  if (!c || !fields) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  if (system < 0 || system >= (int32_t)c->sys.size()) return fail(c, PGPU_EINVAL, "invalid system id %d", system);
  int r = check_contiguous(c);
  if (r) return r;
  const int shape = 2;  // 256-thread tiles for the diagnostic pair sums
  const int block = 256;
  const auto own = owned(c, system);
  const int64_t row_lo = c->sys[system].off + own.first, row_hi = row_lo + own.second;
  // about 72 items per SM, as far as kMaxChunks allows: each row tile sums only
  // the sources above it, so an item is anything from full to empty (100,000
  // particles: 7.6 ms per call, 8.1 ms with 8 items per SM)
  const int nch = (int)std::max<int64_t>(
      1, std::min<int64_t>(kMaxChunks, ceil_div(72LL * c->sms, std::max<int64_t>(1, ceil_div(own.second, block)))));
  // rows: the owned targets (all of them without a target range); each
  // unordered pair is summed from its lower index, so the ranks' row ranges
  // together cover every pair once
  std::vector<PlanEntry> plan = build_plan(c, {system}, shape, nch);
  CK(put_data(c, c->d_plan_diag, plan.data(), plan.size() * sizeof(PlanEntry)));
  const bool quad = plan.size() > 1;
  if (quad) {
    int grid = 0;
    const bool ho = c->cfg.kernel == PGPU_KERNEL_HIGHORDER;
    if (fp64(c)) {
      DiagArgs<double> a{static_cast<const double4 *>(c->P), static_cast<const double4 *>(c->Q), c->partial,
                         c->d_plan_diag, 1, nch, c->cap, c->d_counters};
      auto fn = ho ? diag_pair_kernel<double, 256, kHighOrder> : diag_pair_kernel<double, 256, kGaussian>;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&grid, fn, block, 0);
      fn<<<std::max(1, grid) * c->sms, block, 0, c->st>>>(a);
    } else {
      DiagArgs<float> a{static_cast<const float4 *>(c->P), static_cast<const float4 *>(c->Q), c->partial,
                        c->d_plan_diag, 1, nch, c->cap, c->d_counters};
      auto fn = ho ? diag_pair_kernel<float, 256, kHighOrder> : diag_pair_kernel<float, 256, kGaussian>;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&grid, fn, block, 0);
      fn<<<std::max(1, grid) * c->sms, block, 0, c->st>>>(a);
    }
    CK(cudaGetLastError());
    c->launches++;
  }
  const std::vector<int> &ws = c->sys[system].wakes;
  for (size_t k = 0; k < ws.size(); ++k) {
    const WakeRec &W = c->wakes[ws[k]];
    double *g = fields + k * PGPU_DIAG_FIELDS;
    for (int m = 0; m < PGPU_DIAG_FIELDS; ++m) g[m] = 0.0;
    const int64_t lo = std::max(W.off, row_lo), hi = std::min(W.off + W.n, row_hi);
    if (hi <= lo) continue;
    const int grid = (int)std::min<int64_t>(ceil_div(hi - lo, 256), c->diag_blocks);
    // the CTAs' sums go straight to the pinned ring (at most 296 x 23 values)
    const size_t bytes = (size_t)grid * kDiagFields * sizeof(double);
    double *h = reinterpret_cast<double *>(io_take(c, bytes));
    if (!h) return fail(c, PGPU_ECUDA, "no pinned memory for the diagnostic sums");
    diag_wake_kernel<<<grid, 256, 0, c->st>>>(c->x0, c->sig, c->partial, nch, c->cap, lo, hi, quad ? 1 : 0,
                                              c->cfg.kernel, h);
    CK(cudaGetLastError());
    c->launches++;
    CK(cudaStreamSynchronize(c->st));
    // per-CTA partials summed in CTA order: deterministic
    for (int b = 0; b < grid; ++b)
      for (int m = 0; m < kDiagFields; ++m) g[m] += h[(size_t)b * kDiagFields + m];
  }
  return PGPU_OK;
}

int pgpu_diagnose_combine(const double *fields, int32_t nwakes, double zc_prev, double *out, double *vbi,
                          double *zc_out) {
  if (!fields || !out || nwakes < 0) return PGPU_EINVAL;
  double f[PGPU_DIAG_FIELDS] = {0};
  double zc = zc_prev;
  for (int k = 0; k < nwakes; ++k) {
    const double *g = fields + (size_t)k * PGPU_DIAG_FIELDS;
    for (int m = 0; m < PGPU_DIAG_FIELDS; ++m) f[m] += g[m];
    // PAWAN's Zc: the last wake with non-zero weight wins (interaction.cpp:135-157)
    if (g[10] != 0.0) zc = g[9] / g[10];
  }
  for (int m = 0; m < 3; ++m) {
    out[m] = f[m];
    out[3 + m] = 0.5 * f[3 + m];
    out[6 + m] = f[6 + m] / 3.0;
  }
  out[9] = f[14];
  out[10] = f[21] + f[19];
  out[11] = f[22] + f[20];
  out[12] = f[17] + f[15];
  out[13] = f[18] + f[16];
  out[14] = zc;
  if (vbi)
    for (int m = 0; m < 3; ++m) vbi[m] = f[11 + m];
  if (zc_out) *zc_out = zc;
  return PGPU_OK;
}

int pgpu_diagnose(pgpu_ctx *c, int32_t system, double *out, double *vbi) {
  NvtxRange nvtx("pgpu_diagnose");
  if (!c || !out) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  if (restricted(c))
    return fail(c, PGPU_EINVAL, "with target ranges each context holds a part of the diagnostics: sum "
                                "pgpu_diagnose_partial over the contexts and finish with pgpu_diagnose_combine");
  if (system < 0 || system >= (int32_t)c->sys.size()) return fail(c, PGPU_EINVAL, "invalid system id %d", system);
  std::vector<double> fields(c->sys[system].wakes.size() * PGPU_DIAG_FIELDS);
  int r = pgpu_diagnose_partial(c, system, fields.data());
  if (r) return r;
  double zc = c->sys[system].zc;
  pgpu_diagnose_combine(fields.data(), (int32_t)c->sys[system].wakes.size(), zc, out, vbi, &zc);
  c->sys[system].zc = zc;
  return PGPU_OK;
}

// Whether the lanes of a probe call hold points instead of particles: from the
// point counts on at which the points fill the device.  Gaussian pairs take the
// far limit by warps, and 32 particles in a row are together where 32 points
// need not be, so only wakes of a few hundred particles gain there.  Whole
// calls, lanes over particles / points, in us:
//   Gaussian, 30,000 points  100 particles: 747 / 733;  200: 761 / 802
//     100,000 points  25: 1272 / 1075;  400: 1422 / 1387;  1000: 1563 / 1902
//     1M points  25: 8376 / 7068;  400: 9573 / 8427;  5000: 27,427 / 37,490
//   high-order, 30,000 points  1000: 816 / 853;  5000: 1182 / 1457
//     60,000 points  100: 918 / 846;  5000: 1868 / 1805;  20,000: 4826 / 4468
//     1M points  100: 8006 / 7431;  20,000: 72,202 / 47,387
static bool probe_by_points(const pgpu_ctx *c, int64_t n, int64_t npts) {
  if (c->cfg.kernel == PGPU_KERNEL_HIGHORDER) return npts >= 60000;
  return npts >= 30000 && n <= (npts >= 100000 ? 400 : 128);
}

int pgpu_probe(pgpu_ctx *c, int32_t system, int64_t npts, const double *pts, double *vel) {
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  if (system < 0 || system >= (int32_t)c->sys.size()) return fail(c, PGPU_EINVAL, "invalid system id %d", system);
  if (npts < 0 || (npts > 0 && (!pts || !vel))) return fail(c, PGPU_EINVAL, "bad probe arrays");
  if (npts == 0) return PGPU_OK;
  const int64_t lo = c->sys[system].off, hi = lo + sys_n(c, system);
  // Particle chunks: about eight CTAs per SM in all, of at least one particle
  // per thread, and at most 512 chunks, so that the reduction stays a small
  // part (400 points: 11 chunks of 100 point tiles).
  const int64_t tiles = ceil_div(npts, kProbePoints);
  int64_t chunks = std::min<int64_t>(std::max<int64_t>(1, 8LL * c->sms / tiles), 512);
  chunks = std::max<int64_t>(1, std::min(chunks, ceil_div(hi - lo, kProbeBlock)));
  const int64_t per = ceil_div(std::max<int64_t>(hi - lo, 1), chunks);
  // points, velocities and per-chunk sums: in the context's transfer staging
  // (free between calls, ordered on its stream) where they fit, as for a few
  // hundred points of any wake, else in an allocation of this call
  const bool by_points = probe_by_points(c, hi - lo, npts);
  const int64_t need = (6 + (by_points ? 0 : 3 * chunks)) * npts;
  const bool own = need > 8 * c->cap;
  double *d = c->stage;
  if (own) CK(cudaMallocAsync((void **)&d, need * sizeof(double), c->st));
  double *d_vel = d + 3 * npts, *d_part = d + 6 * npts;
  CK(put_data(c, d, pts, 3 * npts * sizeof(double)));
  // the velocities come back through the ring where they fit
  double *h_vel = reinterpret_cast<double *>(io_take(c, 3 * npts * sizeof(double)));
  if (h_vel) d_vel = h_vel;
  const bool ho = c->cfg.kernel == PGPU_KERNEL_HIGHORDER;
  if (hi > lo && by_points) {
    auto fn = ho ? probe_points_kernel<kHighOrder> : probe_points_kernel<kGaussian>;
    fn<<<(unsigned)ceil_div(npts, kProbeBlock), kProbeBlock, 0, c->st>>>(c->x0, c->sig, c->cap, lo, hi, d, npts, d_vel);
    CK(cudaGetLastError());
    c->launches++;
  } else if (hi > lo) {
    auto fn = ho ? probe_kernel<kHighOrder> : probe_kernel<kGaussian>;
    fn<<<dim3((unsigned)tiles, (unsigned)chunks), kProbeBlock, 0, c->st>>>(c->x0, c->sig, c->cap, lo, hi, per, d, npts,
                                                                           d_part);
    CK(cudaGetLastError());
    const int rg = (int)std::min<int64_t>(ceil_div(3 * npts, 128), 16LL * c->sms);
    probe_reduce_kernel<<<rg, 128, 0, c->st>>>(d_part, (int)chunks, 3 * npts, d_vel);
    CK(cudaGetLastError());
    c->launches += 2;
  } else {
    CK(cudaMemsetAsync(d_vel, 0, 3 * npts * sizeof(double), c->st));
  }
  if (!h_vel) CK(cudaMemcpyAsync(vel, d_vel, 3 * npts * sizeof(double), cudaMemcpyDeviceToHost, c->st));
  if (own) CK(cudaFreeAsync(d, c->st));
  CK(cudaStreamSynchronize(c->st));
  if (h_vel) memcpy(vel, h_vel, 3 * npts * sizeof(double));
  c->io_pos = 0;  // the stream is idle
  return PGPU_OK;
}

int pgpu_sync(pgpu_ctx *c) {
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  CK(cudaStreamSynchronize(c->st));
  if (c->frozen) {
    if (*static_cast<volatile int *>(c->h_flag)) {
      *c->h_flag = 0;
      return fail(c, PGPU_ENUMERIC, "a time step produced a non-finite particle state");
    }
  }
  return PGPU_OK;
}

int pgpu_influence(pgpu_ctx *c) {
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  NvtxRange nvtx("pgpu_influence");
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  int r = check_contiguous(c);
  if (r) return r;
  if (!c->d_field) {
    const cudaError_t e = cudaMalloc((void **)&c->d_field, 3 * (size_t)c->cap * sizeof(double));
    if (e != cudaSuccess) {
      cudaGetLastError();
      c->d_field = nullptr;
      return fail(c, PGPU_ENOMEM, "cudaMalloc of the vorticity field failed: %s", cudaGetErrorString(e));
    }
  }
  // every particle of every system is a target; slice length as choose_slices
  double pairs = 0.0, targets = 0.0;
  for (size_t k = 0; k < c->sys.size(); ++k) {
    pairs += (double)sys_n(c, (int)k) * (double)sys_n(c, (int)k);
    targets += (double)sys_n(c, (int)k);
  }
  const int v = slice_variant(pairs, targets, c->cfg.kernel);
  const bool ho = c->cfg.kernel == PGPU_KERNEL_HIGHORDER;
  auto fn = v == 0 ? (ho ? field_kernel<1, kHighOrder> : field_kernel<1, kGaussian>)
                   : (ho ? field_kernel<2, kHighOrder> : field_kernel<2, kGaussian>);
  int nb = 0;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, 32 * kSliceWarps, 0));
  const int grid = std::max(1, nb) * c->sms;
  const SlicesPlan p = build_slices_plan(c, all_systems(c), v, grid, false);
  const int nch = p.nch;
  CK(put_data(c, c->d_plan_field, p.plan.data(), p.plan.size() * sizeof(PlanEntry)));
  if (p.rows > 0) {
    FieldArgs a{c->x0, c->sig, c->partial, c->d_plan_field, (int)c->sys.size(), nch, c->cap};
    fn<<<grid, 32 * kSliceWarps, 0, c->st>>>(a);
    CK(cudaGetLastError());
    c->launches++;
  }
  const int rg = (int)std::min<int64_t>(ceil_div(c->cap, 256), 16LL * c->sms);
  field_reduce_kernel<<<rg, 256, 0, c->st>>>(c->partial, nch, c->cap, c->d_field);
  CK(cudaGetLastError());
  c->launches++;
  return PGPU_OK;
}

int pgpu_get_vorticity_field(pgpu_ctx *c, int32_t wake, double *field) {
  int r = wake_ok(c, wake);
  if (r) return r;
  DeviceScope device_scope(c->cfg.device);
  if (!field) return fail(c, PGPU_EINVAL, "null output array");
  if (!c->d_field) return fail(c, PGPU_EINVAL, "no vorticity field was computed (pgpu_influence)");
  const WakeRec &W = c->wakes[wake];
  return download_rows(c, c->d_field, W, field, nullptr);
}

int pgpu_set_timing(pgpu_ctx *c, int on) {
  if (!c) return PGPU_EINVAL;
  c->timing = on != 0;
  return PGPU_OK;
}

int pgpu_sync_timeout(pgpu_ctx *c, double seconds) {
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  NvtxRange nvtx("pgpu_sync_timeout");
  const auto t0 = std::chrono::steady_clock::now();
  for (;;) {
    const cudaError_t e = cudaStreamQuery(c->st);
    if (e == cudaSuccess) break;
    if (e != cudaErrorNotReady) return fail(c, PGPU_ECUDA, "cudaStreamQuery failed: %s", cudaGetErrorString(e));
    const double waited = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (waited > seconds)
      return fail(c, PGPU_ETIMEOUT, "the queued work did not finish within %.3f s (it keeps running)", seconds);
    std::this_thread::sleep_for(std::chrono::microseconds(100));
  }
  return pgpu_sync(c);
}

int pgpu_snapshot_begin(pgpu_ctx *c, int32_t slot) {
  NvtxRange nvtx("pgpu_snapshot_begin");
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  if (slot != 0 && slot != 1) return fail(c, PGPU_EINVAL, "snapshot slot %d is not 0 or 1", slot);
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  if (c->capturing) return fail(c, PGPU_EINVAL, "a snapshot cannot be taken during graph capture");
  const size_t bytes = 6 * (size_t)c->cap * sizeof(double);
  if (!c->st_copy) CK(cudaStreamCreateWithFlags(&c->st_copy, cudaStreamNonBlocking));
  if (!c->d_snap[slot]) {
    if (cudaMalloc(&c->d_snap[slot], std::max<size_t>(bytes, 64)) != cudaSuccess) {
      cudaGetLastError();
      c->d_snap[slot] = nullptr;
      return fail(c, PGPU_ENOMEM, "snapshot buffer of %zu bytes", bytes);
    }
    if (cudaHostAlloc(reinterpret_cast<void **>(&c->h_snap[slot]), std::max<size_t>(bytes, 64), cudaHostAllocDefault) !=
        cudaSuccess) {
      cudaGetLastError();
      c->h_snap[slot] = nullptr;
      cudaFree(c->d_snap[slot]);
      c->d_snap[slot] = nullptr;
      return fail(c, PGPU_ENOMEM, "pinned snapshot buffer of %zu bytes", bytes);
    }
  }
  if (!c->snap_gathered[slot]) CK(cudaEventCreateWithFlags(&c->snap_gathered[slot], cudaEventDisableTiming));
  if (!c->snap_copied[slot]) CK(cudaEventCreateWithFlags(&c->snap_copied[slot], cudaEventDisableTiming));
  // the gather must not overwrite the slot while its previous copy reads it
  if (c->snap_begun[slot]) CK(cudaStreamWaitEvent(c->st, c->snap_copied[slot], 0));
  c->snap_begun[slot] = false;  // until this snapshot is fully queued
  auto &offs = c->snap_off[slot];
  auto &ns = c->snap_n[slot];
  offs.assign(c->wakes.size(), 0);
  ns.assign(c->wakes.size(), 0);
  int64_t total = 0;
  for (size_t w = 0; w < c->wakes.size(); ++w) {
    const WakeRec &W = c->wakes[w];
    offs[w] = total;
    ns[w] = W.n;
    if (W.n > 0) {
      const int grid = (int)std::min<int64_t>(ceil_div(W.n, kIoRows), 8LL * c->sms);
      gather_kernel<<<grid, kIoRows, 0, c->st>>>(c->x0, W.n, W.off, c->cap, 2, c->d_snap[slot] + 6 * total);
      CK(cudaGetLastError());
      c->launches++;
    }
    total += W.n;
  }
  CK(cudaEventRecord(c->snap_gathered[slot], c->st));
  CK(cudaStreamWaitEvent(c->st_copy, c->snap_gathered[slot], 0));
  if (total > 0)
    CK(cudaMemcpyAsync(c->h_snap[slot], c->d_snap[slot], 6 * (size_t)total * sizeof(double), cudaMemcpyDeviceToHost,
                       c->st_copy));
  CK(cudaEventRecord(c->snap_copied[slot], c->st_copy));
  c->snap_begun[slot] = true;
  return PGPU_OK;
}

int pgpu_snapshot_wait(pgpu_ctx *c, int32_t slot, double seconds, const double **state, int64_t *off, int64_t *n,
                       int32_t nwakes) {
  NvtxRange nvtx("pgpu_snapshot_wait");
  if (!c) return PGPU_EINVAL;
  if (slot != 0 && slot != 1) return fail(c, PGPU_EINVAL, "snapshot slot %d is not 0 or 1", slot);
  if (!c->snap_begun[slot]) return fail(c, PGPU_EINVAL, "no snapshot was begun in slot %d", slot);
  if (seconds > 0) {
    const auto t0 = std::chrono::steady_clock::now();
    for (;;) {
      const cudaError_t e = cudaEventQuery(c->snap_copied[slot]);
      if (e == cudaSuccess) break;
      if (e != cudaErrorNotReady) return fail(c, PGPU_ECUDA, "cudaEventQuery failed: %s", cudaGetErrorString(e));
      const double waited = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
      if (waited > seconds)
        return fail(c, PGPU_ETIMEOUT, "snapshot %d did not land within %.3f s (the copy keeps running)", slot, seconds);
      std::this_thread::sleep_for(std::chrono::microseconds(50));
    }
  } else {
    CK(cudaEventSynchronize(c->snap_copied[slot]));
  }
  if (state) *state = c->h_snap[slot];
  const int32_t m = std::min<int32_t>(std::max(nwakes, 0), (int32_t)c->snap_off[slot].size());
  for (int32_t w = 0; w < m; ++w) {
    if (off) off[w] = c->snap_off[slot][w];
    if (n) n[w] = c->snap_n[slot][w];
  }
  return PGPU_OK;
}

int pgpu_pair_kernel_time(pgpu_ctx *c, double *ms, int64_t *launches) {
  if (!c) return PGPU_EINVAL;
  if (ms) *ms = c->pair_ms;
  if (launches) *launches = c->pair_launches;
  c->pair_ms = 0.0;
  c->pair_launches = 0;
  return PGPU_OK;
}

int64_t pgpu_launch_count(pgpu_ctx *c) { return c ? c->launches : -1; }

int pgpu_pair_counts(pgpu_ctx *c, int64_t *pairs, int64_t *full_pairs) {
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  int64_t full = c->pairs_acc;
  // the Gaussian kernel has a far regime in both precisions (and counts its
  // full-formula pairs); the high-order kernel evaluates every pair in full
  if (c->frozen && c->cfg.kernel == PGPU_KERNEL_GAUSSIAN) {
    unsigned long long nf = 0;
    CK(cudaStreamSynchronize(c->st));
    CK(cudaMemcpy(&nf, c->d_nfull, sizeof(nf), cudaMemcpyDeviceToHost));
    CK(cudaMemset(c->d_nfull, 0, sizeof(nf)));
    full = (int64_t)nf - c->selfs_acc;
  }
  if (pairs) *pairs = c->pairs_acc;
  if (full_pairs) *full_pairs = full;
  c->pairs_acc = 0;
  c->selfs_acc = 0;
  return PGPU_OK;
}

int pgpu_kernel_shapes(int *block, int *tpt, int max) {
  for (int s = 0; s < kNumShapes && s < max; ++s) {
    if (block) block[s] = kShapes[s].block;
    if (tpt) tpt[s] = kShapes[s].tpt;
  }
  return kNumShapes;
}

// Times every shape and, where the context was not asked for one, its own choice
// of the row list, leaving the faster in place.
static int autotune(pgpu_ctx *c, int reps, double *ms_per_launch) {
  double best = 1e300;
  int best_s = c->shape;
  int64_t nl;
  int r;
  auto time = [&](double *ms) -> int {
    for (int k = 0; k <= reps; ++k) {
      int e = launch_eval(c, 0);
      if (!e) e = collect_timing(c, 1);
      if (e) return e;
      if (k == 0) pgpu_pair_kernel_time(c, nullptr, nullptr);  // warm-up
    }
    pgpu_pair_kernel_time(c, ms, &nl);
    *ms /= reps;
    return PGPU_OK;
  };
  c->auto_shape = false;
  for (int s = 0; s < kNumShapes; ++s) {
    c->shape = s;
    c->plan_dirty = true;
    double ms;
    if ((r = upload_plan(c))) return r;
    if ((r = time(&ms))) return r;
    if (ms_per_launch) ms_per_launch[s] = ms;
    if (ms < best) { best = ms; best_s = s; }
  }
  c->shape = best_s;
  if (!c->shape_asked) {
    c->auto_shape = true;
    c->plan_dirty = true;
    if ((r = upload_plan(c))) return r;
    double ms = 1e300;
    if (c->slices >= 0 && (r = time(&ms))) return r;
    c->auto_shape = ms <= best;
  }
  c->plan_dirty = true;
  return upload_plan(c);
}

int pgpu_autotune(pgpu_ctx *c, int reps, int *block, int *tpt, double *ms_per_launch) {
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  if (reps < 1) reps = 1;
  int r;
  if (c->sur) {
    // the surrogate's evaluations do not use the shape: nothing to choose
    if ((r = upload_plan(c))) return r;
    for (int s = 0; s < kNumShapes && ms_per_launch; ++s) ms_per_launch[s] = 0.0;
  } else {
    const int shape = c->shape;
    const bool auto_shape = c->auto_shape;
    const std::vector<int> sys_shape = c->sys_shape;
    c->sys_shape.clear();  // one shape for every system from here on
    pgpu_pair_kernel_time(c, nullptr, nullptr);
    if ((r = autotune(c, reps, ms_per_launch))) {
      c->shape = shape;
      c->auto_shape = auto_shape;
      c->sys_shape = sys_shape;
      c->plan_dirty = true;
      return r;
    }
  }
  // The partial buffer now holds the last candidate's chunks: recompute the
  // rates of the current state with the chosen shape.
  if ((r = pgpu_solve(c))) return r;
  pgpu_pair_kernel_time(c, nullptr, nullptr);
  if (block) *block = kShapes[c->shape].block;
  if (tpt) *tpt = kShapes[c->shape].tpt;
  return PGPU_OK;
}

}  // extern "C"

namespace {

// Size class of a system of n particles: class 0 holds n < 4096, class k >= 1
// holds [1024 4^k, 1024 4^(k+1)).
int size_class(int64_t n) {
  int k = 0;
  for (int64_t hi = 4096; n >= hi && k < 30; hi *= 4) ++k;
  return k;
}
int64_t class_lo(int k) { return k == 0 ? 0 : (int64_t)1024 << (2 * k); }
int64_t class_hi(int k) { return (int64_t)1024 << (2 * (k + 1)); }

// Device time of one pair launch of `shape` (kNumShapes + v: the row list of
// slices variant v) over `systems` (their own plan and chunk count), mean of
// `reps` launches after one untimed.
template <typename T> int time_subset(pgpu_ctx *c, const std::vector<int> &systems, int shape, int reps, double *ms) {
  int r = upload_plan(c);  // system sizes on the device, for the source boxes
  if (r) return r;
  const int rows = shape - kNumShapes;
  int nch;
  std::vector<PlanEntry> plan;
  if (rows >= 0) {
    SlicesPlan p = build_slices_plan(c, systems, rows, c->grid_slices[rows], true);
    plan = std::move(p.plan);
    nch = p.nch;
  } else {
    nch = choose_nch_for(c, shape, systems);
    plan = build_plan(c, systems, shape, nch);
    plan.resize(c->sys.size() + 1, plan.back());
  }
  // d_plan now holds this subset's plan: the next evaluation rebuilds the
  // context's own, also when the tuning stops early on an error
  c->plan_dirty = true;
  CK(cudaMemcpyAsync(c->d_plan, plan.data(), plan.size() * sizeof(PlanEntry), cudaMemcpyHostToDevice, c->st));
  CK(cudaStreamSynchronize(c->st));
  PairArgs<T> a;
  a.P = static_cast<const v4_t<T> *>(c->P);
  a.Q = static_cast<const v4_t<T> *>(c->Q);
  a.partial = c->partial;
  a.plan = c->d_plan;
  a.nsys = (int)c->sys.size();
  a.nch = nch;
  a.cap = c->cap;
  a.nu2 = (T)(2.0 * c->cfg.nu);
  a.counters = c->d_counters;
  a.nfull = c->d_nfull;
  if (uses_boxes(c) && rows < 0) {
    if ((r = launch_boxes(c))) return r;
    a.box = c->d_box;
  }
  a.L = c->d_L;
  float total = 0.f;
  for (int k = 0; k <= reps; ++k) {
    CK(cudaEventRecord(c->ev[0][0], c->st));
    if (rows >= 0) {
      if ((r = launch_rows(c, rows, a))) return r;
    } else {
      pair_fn<T>(shape, c->cfg.kernel, uses_split(c))<<<c->grid[shape], kShapes[shape].block, 0, c->st>>>(a);
      CK(cudaGetLastError());
      c->launches++;
    }
    CK(cudaEventRecord(c->ev[0][1], c->st));
    CK(cudaEventSynchronize(c->ev[0][1]));
    float t = 0.f;
    CK(cudaEventElapsedTime(&t, c->ev[0][0], c->ev[0][1]));
    if (k > 0) total += t;
  }
  *ms = total / reps;
  return PGPU_OK;
}

std::string json_str(const std::string &line, const char *key) {
  const std::string k = std::string("\"") + key + "\": \"";
  const size_t p = line.find(k);
  if (p == std::string::npos) return "";
  const size_t e = line.find('"', p + k.size());
  return e == std::string::npos ? "" : line.substr(p + k.size(), e - p - k.size());
}

bool json_num(const std::string &line, const char *key, double *v) {
  const std::string k = std::string("\"") + key + "\": ";
  const size_t p = line.find(k);
  if (p == std::string::npos) return false;
  char *end = nullptr;
  *v = strtod(line.c_str() + p + k.size(), &end);
  return end != line.c_str() + p + k.size();
}

// Times of every shape for one cached class ("ms": [..] of the line).
bool json_ms(const std::string &line, double *ms, int n) {
  const size_t p = line.find("\"ms\": [");
  if (p == std::string::npos) return false;
  const char *q = line.c_str() + p + 7;
  for (int i = 0; i < n; ++i) {
    char *end = nullptr;
    ms[i] = strtod(q, &end);
    if (end == q) return false;
    q = end;
    while (*q == ',' || *q == ' ') ++q;
  }
  return true;
}

}  // namespace

extern "C" {

int pgpu_autotune_classes(pgpu_ctx *c, int reps, const char *cache_path, pgpu_tune_class *classes, int max_classes,
                          int *nclasses, int *per_class) {
  NvtxRange nvtx("pgpu_autotune_classes");
  if (!c) return PGPU_EINVAL;
  DeviceScope device_scope(c->cfg.device);
  if (!c->frozen) return fail(c, PGPU_EINVAL, "no particles were uploaded");
  if (c->sur) return fail(c, PGPU_EINVAL, "the surrogate evaluates one system; use pgpu_autotune");
  if (reps < 1) reps = 1;
  int r = check_contiguous(c);
  if (r) return r;
  // systems by size class
  std::map<int, std::vector<int>> cls;
  for (size_t s = 0; s < c->sys.size(); ++s)
    if (owned(c, (int)s).second > 0) cls[size_class(sys_n(c, (int)s))].push_back((int)s);
  if (cls.empty()) return fail(c, PGPU_EINVAL, "no system has particles");
  cudaDeviceProp prop;
  CK(cudaGetDeviceProperties(&prop, c->cfg.device));
  const std::string gpu = prop.name;
  const std::string prec = fp64(c) ? "fp64" : "fp32c";
  const std::string ker = c->cfg.kernel == PGPU_KERNEL_HIGHORDER ? "highorder" : "gaussian";
  // the context's own choice of the row list for these systems, if it makes one
  int rows = -1;
  if (!c->shape_asked) {
    const bool auto_shape = c->auto_shape;
    c->auto_shape = true;
    r = choose_slices(c, &rows);
    c->auto_shape = auto_shape;
    if (r) return r;
  }
  // cached times: the last matching line of the file wins; the row list's time
  // is an entry of its own after the shapes', negative where it is not known
  std::map<int, std::vector<double>> cached;
  if (cache_path && *cache_path) {
    if (FILE *f = fopen(cache_path, "r")) {
      char buf[2048];
      while (fgets(buf, sizeof(buf), f)) {
        const std::string line(buf);
        double k = -1;
        std::vector<double> ms(kNumShapes + 1, -1.0);
        if (json_str(line, "gpu") == gpu && json_str(line, "precision") == prec && json_str(line, "kernel") == ker &&
            json_num(line, "class", &k) && json_ms(line, ms.data(), kNumShapes)) {
          double v = -1;
          if (rows >= 0 && json_num(line, "row_sources", &v) && (int)v == kSliceLen[rows])
            json_num(line, "rows_ms", &ms[kNumShapes]);
          cached[(int)k] = ms;
        }
      }
      fclose(f);
    }
  }
  double ms_acc;
  int64_t nl;
  pgpu_pair_kernel_time(c, &ms_acc, &nl);
  std::vector<int> keys;
  std::vector<std::vector<double>> tms;
  std::vector<int> from_cache;
  for (auto &kv : cls) {
    keys.push_back(kv.first);
    auto it = cached.find(kv.first);
    from_cache.push_back(it != cached.end());
    std::vector<double> ms = from_cache.back() ? it->second : std::vector<double>(kNumShapes + 1, -1.0);
    for (int sh = from_cache.back() ? kNumShapes : 0; sh < kNumShapes + (rows >= 0); ++sh) {
      if (sh == kNumShapes && ms[sh] >= 0.0) break;  // known from the cache
      const int k = sh < kNumShapes ? sh : kNumShapes + rows;
      r = fp64(c) ? time_subset<double>(c, kv.second, k, reps, &ms[sh]) : time_subset<float>(c, kv.second, k, reps, &ms[sh]);
      if (r) return r;
    }
    tms.push_back(ms);
  }
  // fastest shape per class, and the one shape with the least total time
  const size_t K = keys.size();
  std::vector<int> best(K);
  for (size_t i = 0; i < K; ++i)
    best[i] = (int)(std::min_element(tms[i].begin(), tms[i].begin() + kNumShapes) - tms[i].begin());
  int single = 0;
  double single_t = 1e300;
  for (int sh = 0; sh < kNumShapes; ++sh) {
    double t = 0.0;
    for (size_t i = 0; i < K; ++i) t += tms[i][sh];
    if (t < single_t) { single_t = t; single = sh; }
  }
  // one launch per class shape only if the single shape loses more than 2%
  // on some class
  bool split = false;
  for (size_t i = 0; i < K; ++i)
    if (tms[i][single] > 1.02 * tms[i][best[i]]) split = true;
  // the row list stays where it beats the chosen shapes over all classes
  double rows_t = 0.0, shapes_t = 0.0;
  for (size_t i = 0; i < K; ++i) {
    rows_t += tms[i][kNumShapes];
    shapes_t += tms[i][split ? best[i] : single];
  }
  c->auto_shape = rows >= 0 && rows_t <= shapes_t;
  if (c->auto_shape) split = false;
  if (split) {
    c->sys_shape.assign(c->sys.size(), single);
    for (size_t i = 0; i < K; ++i)
      for (int s : cls[keys[i]]) c->sys_shape[s] = best[i];
  } else {
    c->sys_shape.clear();
    c->shape = single;
  }
  bool cache_failed = false;
  if (cache_path && *cache_path) {
    if (FILE *f = fopen(cache_path, "a")) {
      for (size_t i = 0; i < K; ++i) {
        if (from_cache[i]) continue;
        fprintf(f, "{\"gpu\": \"%s\", \"precision\": \"%s\", \"kernel\": \"%s\", \"class\": %d, \"nmin\": %lld, "
                   "\"nmax\": %lld, \"block\": %d, \"tpt\": %d, \"ms\": [",
                gpu.c_str(), prec.c_str(), ker.c_str(), keys[i], (long long)class_lo(keys[i]),
                (long long)class_hi(keys[i]), kShapes[best[i]].block, kShapes[best[i]].tpt);
        for (int sh = 0; sh < kNumShapes; ++sh) fprintf(f, "%s%.6g", sh ? ", " : "", tms[i][sh]);
        fprintf(f, "]");
        if (rows >= 0) fprintf(f, ", \"row_sources\": %d, \"rows_ms\": %.6g", kSliceLen[rows], tms[i][kNumShapes]);
        fprintf(f, "}\n");
      }
      fclose(f);
    } else {
      cache_failed = true;  // reported after the chosen launches are in place
    }
  }
  if (nclasses) *nclasses = (int)K;
  if (per_class) *per_class = split ? 1 : 0;
  for (size_t i = 0; i < K && classes && (int)i < max_classes; ++i) {
    pgpu_tune_class &o = classes[i];
    memset(&o, 0, sizeof(o));
    o.size_class = keys[i];
    o.nmin = class_lo(keys[i]);
    o.nmax = class_hi(keys[i]);
    o.systems = (int32_t)cls[keys[i]].size();
    o.block = kShapes[best[i]].block;
    o.tpt = kShapes[best[i]].tpt;
    o.from_cache = from_cache[i];
    for (int sh = 0; sh < kNumShapes && sh < 8; ++sh) o.ms[sh] = tms[i][sh];
    o.single_block = kShapes[single].block;
    o.single_tpt = kShapes[single].tpt;
  }
  // recompute the rates of the current state with the chosen launches (the
  // partial buffer holds the last candidate's chunks)
  c->plan_dirty = true;
  if ((r = upload_plan(c))) return r;
  if ((r = pgpu_solve(c))) return r;
  pgpu_pair_kernel_time(c, nullptr, nullptr);
  if (cache_failed) return fail(c, PGPU_EINVAL, "cannot append to the autotune cache %s", cache_path);
  return PGPU_OK;
}

int pgpu_get_stream(pgpu_ctx *c, void **stream) {
  if (!c || !stream) return PGPU_EINVAL;
  *stream = (void *)c->st;
  return PGPU_OK;
}

int pgpu_fp32_peaks(int device, double *ffma_tflops, double *ffma2_tflops) {
  pgpu_ctx *c = nullptr;  // for CK's error path
  CK(cudaSetDevice(device));
  int sms = 0;
  CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  float *out = nullptr;
  cudaStream_t st;
  CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  CK(cudaMallocAsync((void **)&out, sizeof(float), st));
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  const int block = 256, grid = sms * 8, iters = 1 << 14;
  // both loops do kFfmaChains FMAs per thread per iteration
  const double flops = 2.0 * kFfmaChains * (double)iters * grid * block;
  for (int packed = 0; packed < 2; ++packed) {
    auto run = [&]() {
      if (packed) ffma2_peak_kernel<<<grid, block, 0, st>>>(out, iters, 0.999f, 1e-3f);
      else ffma_peak_kernel<<<grid, block, 0, st>>>(out, iters, 0.999f, 1e-3f);
    };
    run();  // warm-up
    CK(cudaEventRecord(e0, st));
    run();
    CK(cudaEventRecord(e1, st));
    CK(cudaEventSynchronize(e1));
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, e0, e1));
    double *dst = packed ? ffma2_tflops : ffma_tflops;
    if (dst) *dst = flops / (ms * 1e-3) / 1e12;
  }
  cudaFreeAsync(out, st);
  cudaStreamSynchronize(st);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(st);
  return PGPU_OK;
}

int pgpu_fp64_peak(int device, double *tflops) {
  pgpu_ctx *c = nullptr;  // for CK's error path
  CK(cudaSetDevice(device));
  int sms = 0;
  CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  float *out = nullptr;
  cudaStream_t st;
  CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  CK(cudaMallocAsync((void **)&out, sizeof(float), st));
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  const int block = 256, grid = sms * 8, iters = 1 << 12;
  const double flops = 2.0 * kFfmaChains * (double)iters * grid * block;
  dfma_peak_kernel<<<grid, block, 0, st>>>(out, iters, 0.999, 1e-3);  // warm-up
  CK(cudaEventRecord(e0, st));
  dfma_peak_kernel<<<grid, block, 0, st>>>(out, iters, 0.999, 1e-3);
  CK(cudaEventRecord(e1, st));
  CK(cudaEventSynchronize(e1));
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, e0, e1));
  if (tflops) *tflops = flops / (ms * 1e-3) / 1e12;
  cudaFreeAsync(out, st);
  cudaStreamSynchronize(st);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(st);
  return PGPU_OK;
}

int pgpu_fp32_peak(int device, double *tflops, double *ms_out) {
  double f1 = 0.0, f2 = 0.0;
  const int r = pgpu_fp32_peaks(device, &f1, &f2);
  if (r) return r;
  if (tflops) *tflops = f1 > f2 ? f1 : f2;
  if (ms_out) *ms_out = 0.0;
  return PGPU_OK;
}

const char *pgpu_last_error(pgpu_ctx *c) { return c ? c->err : g_create_err; }

}  // extern "C"

#include "mlp_host.inc"
#include "surrogate_host.inc"
#include "merge_host.inc"
