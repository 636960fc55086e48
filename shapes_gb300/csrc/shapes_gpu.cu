/*
 * Host runtime behind include/shapes_gpu.h: one handle = a batch of
 * independent worlds resident on the device as structure-of-arrays, stepped by
 * the kernels of step_kernels.cuh on the handle's own CUDA stream.
 *
 * Buffers whose size depends on the step (pairs, contacts, solver updates) are
 * sized generously up front.  Kernels never write past a capacity: they raise a
 * sticky overflow flag instead, and the host then restores the state saved at
 * the start of the call, doubles the capacities and runs the call again, so a
 * call either completes exactly or returns an error with the state untouched.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <new>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

#include "../../include/shapes_gpu.h"
#include "step_kernels.cuh"
#include "large_world.cuh"
#include "learned.cuh"
#include "mlp.h"

using shapes::Con;
using shapes::Dev;

/* Text of the last CUDA error on this thread (shared with the MLP unit). */
thread_local std::string g_last_error;

namespace {

struct CudaError {
  cudaError_t err;
};

inline void ck(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    g_last_error = std::string(what) + ": " + cudaGetErrorString(e);
    throw CudaError{e};
  }
}

constexpr int kSMs = 152;

template <typename T>
T* dalloc(size_t n, const char* what) {
  void* p = nullptr;
  ck(cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T)), what);
  return static_cast<T*>(p);
}

inline void dfree(void* p) {
  if (p) cudaFree(p);
}

inline int grid_for(long long n, int threads) {
  long long blocks = (n + threads - 1) / threads;
  long long cap = (long long)kSMs * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

/* Launches a kernel that begins with chained_entry(): its blocks may take their
 * places while the kernel before it in the stream (or in the captured graph)
 * still runs, and wait there.  A step of a small or middling batch is 9 to 14 such
 * kernels; chained, one of 401 boxes took 306 us in place of 323.  Not `chain`: an
 * ordinary launch, for handles that step at the same time, where the waiting
 * blocks would hold places that the other streams can use (eight handles of 128
 * worlds: 1.40 ms in place of 1.37). */
template <class... P, class... A>
inline void launch_chained(bool chain, void (*kernel)(P...), unsigned grid, unsigned threads, size_t smem,
                           cudaStream_t stream, A... args) {
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = stream;
  c.attrs = &early;
  c.numAttrs = chain ? 1 : 0;
  cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...); /* an error stays for the caller's cudaGetLastError */
}

/* Small batches spread over more blocks of fewer bodies. */
inline void launch_pose(bool chain, cudaStream_t stream, int n, const Dev& d, double dt, int advance,
                        const uint8_t* only = nullptr) {
  const int per_block = n >= 2 * kSMs * shapes::kPoseThreads ? shapes::kPoseThreads : 32;
  launch_chained(chain, shapes::k_integrate_pose, grid_for(n, per_block), shapes::kPoseThreads, 0, stream, d, dt,
                 advance, per_block, only);
}

/* Handles that some thread's call has at work on a device at this moment: their
 * launches share its SMs, whichever call they came through (eight handles of 128
 * worlds that each took the GPU for their own, stepped from eight threads: 1.91 ms
 * a step in place of 1.28).  Only launch shapes follow it, no result does. */
constexpr int kMaxDevices = 64;
std::atomic<int> g_at_work[kMaxDevices];

class AtWork {
 public:
  explicit AtWork(int device) {
    devices_.reserve(1);
    add(device);
  }
  template <class Batch>
  AtWork(Batch* const* bs, int n) {
    devices_.reserve(n); /* the only throw, before anything is counted */
    for (int k = 0; k < n; ++k) add(bs[k]->device);
  }
  AtWork(const AtWork&) = delete;
  ~AtWork() {
    for (const int d : devices_) g_at_work[d].fetch_sub(1, std::memory_order_relaxed);
  }
  static int on(int device) {
    return known(device) ? std::max(1, g_at_work[device].load(std::memory_order_relaxed)) : 1;
  }

 private:
  static bool known(int device) { return device >= 0 && device < kMaxDevices; }
  void add(int device) {
    if (!known(device)) return;
    devices_.push_back(device);
    g_at_work[device].fetch_add(1, std::memory_order_relaxed);
  }
  std::vector<int> devices_;
};

}  // namespace

struct shapes_batch {
  int device = 0;
  cudaStream_t stream = nullptr;
  int32_t W = 0, N = 0, V = 0;
  std::vector<int32_t> h_world_body_off;
  std::vector<int32_t> h_body_world;

  /* topology */
  int32_t* world_body_off = nullptr;
  int32_t* body_world = nullptr;
  int32_t* vert_off = nullptr;
  double* lx = nullptr;
  double* ly = nullptr;
  double* radius = nullptr; /* [N] circle radii (0 for hulls); null when there is no circle */
  int32_t* emin = nullptr;
  int32_t* emax = nullptr;
  /* state */
  double* body[10] = {nullptr};
  double* body_stage[10] = {nullptr}; /* set_bodies uploads here, validated, then swapped in */
  double* wx = nullptr;
  double* wy = nullptr;
  double* nx = nullptr;
  double* ny = nullptr;
  float4* vf = nullptr; /* [V] posed vertices and normals in binary32 (narrowphase filter) */
  float2* ef = nullptr; /* [V] self extents of each edge in binary32 */
  double* box = nullptr;
  uint64_t* boxk = nullptr;
  uint8_t* flags = nullptr;
  uint8_t* body_changed = nullptr; /* [N] scratch of set_bodies: pose inputs changed */
  int32_t* export_keys = nullptr;  /* staging of get_contacts for pageable caller arrays */
  double* export_vals = nullptr;
  int64_t export_cap = 0;
  /* broadphase / narrowphase */
  int32_t pair_cap = 0, contact_cap = 0;
  int64_t item_cap = 0;
  int32_t* row_cnt = nullptr;
  int32_t* row_hits = nullptr;
  int32_t* row_off = nullptr;
  /* grid broadphase */
  int32_t grid_min_bodies = 64;
  bool any_grid = false;
  int32_t n_buckets = 0;
  int32_t* grid_T = nullptr;
  int32_t* grid_base = nullptr;
  double* grid_inv_s = nullptr;
  double* grid_lim = nullptr;
  int32_t* bucket_cnt = nullptr;
  int32_t* bucket_off = nullptr;
  int4* grid_ent = nullptr;
  int2* cell = nullptr;
  uint8_t* row_mode = nullptr;
  int32_t* large_cnt = nullptr;
  int32_t* large_ids = nullptr;
  double* metric_part = nullptr; /* [kMetricParts] partial metrics of one large world */
  /* incremental grid pairs (fat boxes and adjacency lists) */
  bool incremental = true;
  int32_t nbr_cap = 24;
  uint64_t* fatk = nullptr;
  int32_t* nbr = nullptr;
  int32_t* nbr_cnt = nullptr;
  uint8_t* moved = nullptr;
  int32_t* inc_state = nullptr;
  int32_t* inc_rebuild = nullptr;
  int32_t* inc_moved = nullptr;
  int32_t* inc_frames = nullptr;
  double* inc_margin = nullptr;
  int32_t* pair_a = nullptr;
  int32_t* pair_b = nullptr;
  int32_t* slot_cnt = nullptr;
  int32_t* slot_off = nullptr;
  int32_t* slot_feat = nullptr;
  double* slot_val = nullptr;
  int32_t* np_perm = nullptr;
  int32_t* ext_chunk = nullptr;      /* extent reduction: chunk body ranges, per-world chunk offsets, partials */
  int32_t* ext_chunk_off = nullptr;
  double* ext_part_sum = nullptr;
  int32_t* ext_part_cnt = nullptr;
  int32_t* ext_done = nullptr;
  int32_t n_ext_chunks = 0;
  /* sweep and prune for the small bodies of large grid worlds (incremental pairs off) */
  int32_t sap_min_bodies = 0; /* 0: off */
  int32_t np_lanes = 1;       /* lanes per pair in the narrowphase (1: k_narrowphase) */
  long long poll_limit = 0; /* polls of a wait in a solve before it gives up; 0: each kernel's own limit */
  int poll_limit_or(long long own) const {
    return (int)std::min<long long>(poll_limit > 0 ? poll_limit : own, INT32_MAX);
  }
  bool any_sap = false;
  int32_t n_sap_buckets = 0;
  uint8_t* world_sap = nullptr;
  int32_t *sap_base = nullptr, *sap_cnt = nullptr, *sap_off = nullptr, *sap_ids = nullptr, *sap_qs = nullptr;
  int32_t *sap_cursor = nullptr, *sap_end = nullptr;
  uint64_t* sap_range = nullptr;

  /* Tile sums every scan of a step needs: the longest scanned array is the
   * bodies, the contact slots, the grid buckets or the sweep buckets. */
  int32_t scan_tiles_needed() const {
    const int64_t scan_n =
        std::max<int64_t>(std::max<int64_t>(std::max<int64_t>(N, contact_cap), n_buckets), n_sap_buckets) + 1;
    return (int32_t)((scan_n + shapes::kScanTile - 1) / shapes::kScanTile) + 1;
  }

  void free_scan() {
    dfree(scan_state.tile);
    dfree(scan_state.ctl);
    scan_state = {nullptr, nullptr, 0};
  }
  void alloc_scan() {
    free_scan();
    tile_cap = scan_tiles_needed();
    scan_state.tile = dalloc<unsigned long long>(tile_cap, "cudaMalloc scan");
    scan_state.ctl = dalloc<uint32_t>(3, "cudaMalloc scan");
    scan_state.tiles = tile_cap;
    ck(cudaMemsetAsync(scan_state.tile, 0, sizeof(unsigned long long) * tile_cap, stream), "memset");
    ck(cudaMemsetAsync(scan_state.ctl, 0, 3 * sizeof(uint32_t), stream), "memset");
  }

  void free_sap() {
    dfree(world_sap); dfree(sap_base); dfree(sap_cnt); dfree(sap_off); dfree(sap_ids); dfree(sap_qs);
    dfree(sap_cursor); dfree(sap_end); dfree(sap_range);
    world_sap = nullptr;
    sap_base = sap_cnt = sap_off = sap_ids = sap_qs = sap_cursor = sap_end = nullptr;
    sap_range = nullptr;
    any_sap = false;
    n_sap_buckets = 0;
  }

  /* Marks the grid worlds of at least sap_min_bodies bodies and sizes their
   * buckets (kSapBuckets per world). */
  void setup_sap() {
    free_sap();
    if (sap_min_bodies <= 0) return;
    std::vector<uint8_t> flag(W, 0);
    std::vector<int32_t> base(W, 0);
    int64_t nb = 0;
    for (int w = 0; w < W; ++w) {
      const int32_t n = h_world_body_off[w + 1] - h_world_body_off[w];
      if (n >= grid_min_bodies && n >= sap_min_bodies) {
        flag[w] = 1;
        base[w] = (int32_t)nb;
        nb += shapes::kSapBuckets;
      }
    }
    if (nb == 0) return;
    if (nb > INT32_MAX / 2) throw CudaError{cudaErrorMemoryAllocation};
    any_sap = true;
    n_sap_buckets = (int32_t)nb;
    world_sap = dalloc<uint8_t>(W, "cudaMalloc sweep");
    sap_base = dalloc<int32_t>(W, "cudaMalloc sweep");
    sap_cnt = dalloc<int32_t>((size_t)nb + 1, "cudaMalloc sweep");
    sap_off = dalloc<int32_t>((size_t)nb + 1, "cudaMalloc sweep");
    sap_ids = dalloc<int32_t>(std::max<int32_t>(N, 1), "cudaMalloc sweep");
    sap_qs = dalloc<int32_t>(std::max<int32_t>(N, 1), "cudaMalloc sweep");
    sap_cursor = dalloc<int32_t>(std::max<int32_t>(N, 1), "cudaMalloc sweep");
    sap_end = dalloc<int32_t>(W, "cudaMalloc sweep");
    sap_range = dalloc<uint64_t>(2 * (size_t)W, "cudaMalloc sweep");
    ck(cudaMemsetAsync(sap_cnt, 0, sizeof(int32_t) * ((size_t)nb + 1), stream), "memset");
    ck(cudaMemcpy(world_sap, flag.data(), W, cudaMemcpyHostToDevice), "upload sweep");
    ck(cudaMemcpy(sap_base, base.data(), sizeof(int32_t) * W, cudaMemcpyHostToDevice), "upload sweep");
    if (scan_state.tile && tile_cap < scan_tiles_needed()) alloc_scan(); /* the sweep buckets' scan is the longest */
  }
  int32_t* np_cls = nullptr; /* [2 * kNpClasses + 1] */
  int32_t* world_pair_off = nullptr;
  /* contacts: ping-pong between two buffers, the cache of step s is the
   * contact keys + Lagrangians of step s */
  uint64_t* c_key[2] = {nullptr, nullptr};
  double* lam[2] = {nullptr, nullptr};
  int32_t* cwo[2] = {nullptr, nullptr};
  int cache_buf = 0;   /* buffer holding the current cache */
  int results_buf = 0; /* buffer holding the last pairs/contacts results */
  bool have_results = false;
  int32_t* c_ga = nullptr;
  int32_t* c_slot = nullptr; /* [contact_cap] slot of each contact */
  int32_t* c_gb = nullptr;
  uint8_t* c_flip = nullptr;
  uint8_t* c_hit = nullptr;
  double* c_val = nullptr;
  Con* con = nullptr;
  /* scheduler */
  int4* sched_info = nullptr; /* lists of solver groups too large for shared memory (frontier.cuh) */
  int32_t* sched_list = nullptr;
  int32_t* sched_arr = nullptr;
  int32_t* sched_body = nullptr;
  uint32_t* sched_cur = nullptr;
  int4* gdesc = nullptr;
  long long* phase_clock = nullptr; /* [8 * G], allocated while profiling */
  int32_t phase_clock_groups = 0;
  int32_t* world_levels = nullptr;
  int32_t* group_world_off = nullptr;
  int32_t* group_worlds = nullptr;
  std::vector<int32_t> h_group_world_off;
  std::vector<int32_t> h_group_worlds;
  int32_t grouped_iterations = -1;
  /* worlds solved by the large-world paths (not packed into warp groups) */
  int32_t large_world_bodies = SHAPES_LARGE_WORLD_BODIES;
  std::vector<int32_t> large_worlds;
  int32_t lw_nb_max = 0;
  int32_t* lw_bcnt = nullptr;
  int32_t* lw_bstart = nullptr;
  int32_t* lw_bh = nullptr;
  int32_t* lw_bn = nullptr;
  ulonglong2* lw_vel = nullptr; /* ordered path: velocities and Lagrangians with their counts */
  ulonglong2* lw_lag = nullptr;
  int32_t* lw_refs = nullptr;
  int32_t* lw_rank = nullptr;
  int32_t* lw_hrank = nullptr;
  int32_t* lw_hitflag = nullptr;
  int32_t* lw_rowflag = nullptr; /* ordered path by rows: row starts (flag, scanned, list) */
  int32_t* lw_rowoff = nullptr;
  int32_t* lw_row_start = nullptr;
  int4* lw_side = nullptr;
  int32_t* lw_color = nullptr;
  int32_t* lw_color_cnt = nullptr;
  unsigned long long* lw_ctl = nullptr; /* 8 per large world */
  int32_t worlds_per_group_override = 0;
  int32_t target_group_bodies = 0;
  int32_t solve_threads = 32;
  int32_t group_warps = 1;       /* solver warps of each group, when the caller chose them */
  bool group_warps_auto = true;  /* until then launch_groups chooses */
  int32_t group_max_bodies = 0;  /* bodies of the largest group */
  int32_t handles_in_flight = 1; /* handles at work on this device, when the step was enqueued (AtWork) */
  bool chain() const { return handles_in_flight <= 1; }
  bool parallel_levels = true; /* kept for the caller, see shapes_batch_set_parallel_levels */
  bool spread_heavy = false;   /* heaviest groups first, one per SM, then lightest first */
  int num_sms() {
    if (sm_count <= 0) {
      int dev = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
      if (sm_count <= 0) sm_count = 1;
    }
    return sm_count;
  }
  int sm_count = 0;
  std::vector<int32_t> world_order; /* packing order of the worlds; empty = by body count */
  /* scans */
  shapes::ScanState scan_state{nullptr, nullptr, 0};
  int32_t tile_cap = 0;
  unsigned long long* counters = nullptr;
  double* world_residual = nullptr;
  double* world_depth = nullptr;
  bool residual_valid = false;
  /* world mutation: filled slots (device copy allocated on the first delete)
   * and each world's stack of empty slots (world-local slot ids) */
  uint8_t* active = nullptr;
  std::vector<uint8_t> h_active;
  std::vector<int32_t> h_vert_off;
  std::vector<double> h_radius; /* [N] circle radii, 0 for hulls */
  std::vector<std::vector<int32_t>> h_empties;
  /* learned warm start */
  const shapes_mlp* mlp_model = nullptr;
  uint8_t* learned_mask = nullptr; /* [W] */
  double* judge_res = nullptr;     /* [W] */
  double* judge_depth = nullptr;   /* [W] */
  bool judge_set = false;
  int32_t miss_cap = 0;            /* contact capacity the row buffers were sized for */
  int32_t* miss_flag = nullptr;
  int32_t* miss_off = nullptr;
  int32_t* miss_ids = nullptr;
  int32_t* miss_n = nullptr;
  float* mfeat = nullptr;
  /* training samples */
  float* ds_feat = nullptr;
  float* ds_tgt = nullptr;
  int64_t ds_cap = 0;
  unsigned long long* ds_count = nullptr;
  unsigned long long* snap_ds_count = nullptr;
  uint8_t* snap_mask = nullptr;
  /* snapshot for retries */
  double* snap_body[6] = {nullptr};
  uint64_t* snap_key = nullptr;
  double* snap_lam = nullptr;
  int32_t* snap_cwo = nullptr;
  int32_t snap_cap = 0;

  shapes_stats stats{};

  /* What the number of handles that share the GPU decides about a step's
   * launches (solve_shape); the rest of them follows from the configuration and
   * from what bumps graph_epoch. */
  struct SolveShape {
    bool chained;
    int warps, smem, split_limit;
    bool operator==(const SolveShape& o) const {
      return chained == o.chained && warps == o.warps && smem == o.smem && split_limit == o.split_limit;
    }
  };

  /* CUDA graphs: captured steps, replayed while the configuration and every
   * buffer the step touches stay the same.  Anything that reallocates a buffer,
   * regroups the solver or changes which kernels a step launches bumps
   * graph_epoch.  Per write buffer the kStepGraphs used last are kept, one for
   * each configuration and shape, so that a handle stepped now alone, now beside
   * others captures once for each: five shapes can occur (alone; beside others
   * with one, two, three or more groups to an SM). */
  static constexpr int kStepGraphs = 6;
  bool graphs_enabled = true;
  uint64_t graph_epoch = 1;
  struct StepGraph {
    cudaGraphExec_t exec = nullptr;
    uint64_t epoch = 0, used = 0;
    shapes_config cfg{};
    SolveShape shape{};
  };
  StepGraph graph[2][kStepGraphs];
  uint64_t graph_clock = 0;
  int64_t graph_captures = 0;

  void invalidate_graphs() { ++graph_epoch; }

  void drop_graph(StepGraph& g) {
    if (g.exec) cudaGraphExecDestroy(g.exec);
    g.exec = nullptr;
  }
  void drop_graphs() {
    for (auto& of_buffer : graph)
      for (auto& g : of_buffer) drop_graph(g);
  }

  /* One solver step writing buffer wb: replayed from its graph, captured on
   * first use (or after an invalidation).  Profiling records events between
   * stages, so profiled steps are launched directly. */
  void launch_step(const shapes_config& cfg, int wb) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (graphs_enabled && !profiling && stream != cudaStreamLegacy && stream != cudaStreamPerThread)
      ck(cudaStreamIsCapturing(stream, &cap), "cudaStreamIsCapturing");
    if (!graphs_enabled || profiling || stream == cudaStreamLegacy || stream == cudaStreamPerThread ||
        cap != cudaStreamCaptureStatusNone) { /* a caller's own capture takes the kernels as they are */
      enqueue_step(cfg, true, wb);
      return;
    }
    const SolveShape shape = solve_shape();
    StepGraph* hit = nullptr;
    StepGraph* oldest = &graph[wb][0];
    for (auto& g : graph[wb]) {
      if (g.exec && g.epoch != graph_epoch) drop_graph(g);
      if (g.exec && g.shape == shape && std::memcmp(&g.cfg, &cfg, sizeof cfg) == 0) hit = &g;
      if (oldest->exec && (!g.exec || g.used < oldest->used)) oldest = &g;
    }
    StepGraph& g = hit ? *hit : *oldest;
    if (!hit) {
      drop_graph(g);
      cudaGraph_t gr = nullptr;
      ck(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture");
      try {
        enqueue_step(cfg, true, wb);
      } catch (...) {
        cudaStreamEndCapture(stream, &gr);
        if (gr) cudaGraphDestroy(gr);
        throw;
      }
      ck(cudaStreamEndCapture(stream, &gr), "cudaStreamEndCapture");
      const cudaError_t e = cudaGraphInstantiate(&g.exec, gr, 0);
      cudaGraphDestroy(gr);
      ck(e, "cudaGraphInstantiate");
      g.epoch = graph_epoch;
      g.cfg = cfg;
      g.shape = shape;
      ++graph_captures;
    }
    g.used = ++graph_clock;
    ck(cudaGraphLaunch(g.exec, stream), "cudaGraphLaunch");
  }

  /* caller stream + per-stage profiling */
  cudaStream_t own_stream = nullptr;
  bool profiling = false;
  std::vector<cudaEvent_t> ev_pool;
  std::vector<int> ev_stage; /* stage of each recorded (start, end) pair */
  size_t ev_used = 0;
  double prof_ms[SHAPES_STAGE_COUNT] = {0};
  int64_t prof_launches[SHAPES_STAGE_COUNT] = {0};

  cudaEvent_t next_event() {
    if (ev_used == ev_pool.size()) {
      cudaEvent_t e;
      ck(cudaEventCreate(&e), "cudaEventCreate");
      ev_pool.push_back(e);
    }
    return ev_pool[ev_used++];
  }

  /* Brackets `launches` kernel launches of stage `st` issued by f(). */
  template <typename F>
  void stage(int st, int launches, F&& f) {
    if (!profiling) {
      f();
      return;
    }
    ck(cudaEventRecord(next_event(), stream), "cudaEventRecord");
    f();
    ck(cudaEventRecord(next_event(), stream), "cudaEventRecord");
    ev_stage.push_back(st);
    prof_launches[st] += launches;
  }

  /* Accumulates the recorded stage times (stream already synchronized). */
  void collect_profile() {
    for (size_t k = 0; k < ev_stage.size(); ++k) {
      float ms = 0.f;
      ck(cudaEventElapsedTime(&ms, ev_pool[2 * k], ev_pool[2 * k + 1]), "cudaEventElapsedTime");
      prof_ms[ev_stage[k]] += ms;
    }
    ev_stage.clear();
    ev_used = 0;
  }

  Dev view(int write_buf) const {
    Dev d{};
    d.n_worlds = W;
    d.n_bodies = N;
    d.n_verts = V;
    d.pair_cap = pair_cap;
    d.contact_cap = contact_cap;
    d.item_cap = (int32_t)std::min<int64_t>(item_cap, INT32_MAX);
    d.world_body_off = world_body_off;
    d.body_world = body_world;
    d.vert_off = vert_off;
    d.ext_chunk = ext_chunk;
    d.ext_chunk_off = ext_chunk_off;
    d.ext_part_sum = ext_part_sum;
    d.ext_part_cnt = ext_part_cnt;
    d.ext_done = ext_done;
    d.n_ext_chunks = n_ext_chunks;
    if (any_sap) {
      d.world_sap = world_sap;
      d.sap_base = sap_base;
      d.sap_cnt = sap_cnt;
      d.sap_off = sap_off;
      d.n_sap_buckets = n_sap_buckets;
      d.sap_ids = sap_ids;
      d.sap_qs = sap_qs;
      d.sap_cursor = sap_cursor;
      d.sap_range = sap_range;
      d.sap_end = sap_end;
    }
    d.lx = lx;
    d.ly = ly;
    d.radius = radius;
    d.emin = emin;
    d.emax = emax;
    d.vx = body[0];
    d.vy = body[1];
    d.w = body[2];
    d.px = body[3];
    d.py = body[4];
    d.th = body[5];
    d.iml = body[6];
    d.imr = body[7];
    d.mu = body[8];
    d.bounce = body[9];
    d.wx = wx;
    d.wy = wy;
    d.nx = nx;
    d.ny = ny;
    d.vf = vf;
    d.ef = ef;
    d.box = box;
    d.boxk = boxk;
    d.flags = flags;
    d.grid_T = grid_T;
    d.grid_base = grid_base;
    d.grid_inv_s = grid_inv_s;
    d.grid_lim = grid_lim;
    d.bucket_cnt = bucket_cnt;
    d.bucket_off = bucket_off;
    d.grid_ent = grid_ent;
    d.cell = cell;
    d.row_mode = row_mode;
    d.large_cnt = large_cnt;
    d.large_ids = large_ids;
    d.n_buckets = n_buckets;
    if (incremental && nbr) {
      d.fatk = fatk;
      d.nbr = nbr;
      d.nbr_cnt = nbr_cnt;
      d.moved = moved;
      d.inc_state = inc_state;
      d.inc_rebuild = inc_rebuild;
      d.inc_moved = inc_moved;
      d.inc_frames = inc_frames;
      d.inc_margin = inc_margin;
      d.nbr_cap = nbr_cap;
    }
    d.row_cnt = row_cnt;
    d.row_hits = row_hits;
    d.row_off = row_off;
    d.pair_a = pair_a;
    d.pair_b = pair_b;
    d.slot_cnt = slot_cnt;
    d.slot_off = slot_off;
    d.slot_feat = slot_feat;
    d.np_perm = np_perm;
    d.np_cls = np_cls;
    d.slot_val = slot_val;
    d.c_key = c_key[write_buf];
    d.c_ga = c_ga;
    d.c_slot = c_slot;
    d.c_gb = c_gb;
    d.c_flip = c_flip;
    d.c_hit = c_hit;
    d.c_val = c_val;
    d.con = con;
    d.lam = lam[write_buf];
    d.old_key = c_key[1 - write_buf];
    d.old_lam = lam[1 - write_buf];
    d.old_cwo = cwo[1 - write_buf];
    d.world_pair_off = world_pair_off;
    d.world_contact_off = cwo[write_buf];
    d.sched_info = sched_info;
    d.sched_list = sched_list;
    d.sched_arr = sched_arr;
    d.sched_body = sched_body;
    d.sched_cur = sched_cur;
    d.gdesc = gdesc;
    d.phase_clock = profiling ? phase_clock : nullptr;
    d.world_levels = world_levels;
    d.group_world_off = group_world_off;
    d.group_worlds = group_worlds;
    d.counters = counters;
    d.world_residual = world_residual;
    d.world_depth = world_depth;
    d.active = active;
    return d;
  }

  void free_row_buffers() {
    dfree(miss_flag); dfree(miss_off); dfree(miss_ids); dfree(miss_n); dfree(mfeat);
    miss_flag = miss_off = miss_ids = miss_n = nullptr;
    mfeat = nullptr;
    miss_cap = 0;
  }

  /* Feature-row buffers for the learned start / sample collection, sized by
   * the contact capacity (allocated on first use). */
  void ensure_row_buffers() {
    if (miss_cap == contact_cap && miss_flag) return;
    if (stream) ck(cudaStreamSynchronize(stream), "sync");
    invalidate_graphs();
    free_row_buffers();
    miss_flag = dalloc<int32_t>(contact_cap, "cudaMalloc rows");
    miss_off = dalloc<int32_t>((size_t)contact_cap + 1, "cudaMalloc rows");
    miss_ids = dalloc<int32_t>(contact_cap, "cudaMalloc rows");
    miss_n = dalloc<int32_t>(1, "cudaMalloc rows");
    mfeat = dalloc<float>((size_t)contact_cap * mlp::kIn, "cudaMalloc rows");
    miss_cap = contact_cap;
  }

  bool learned_on(const shapes_config& cfg) const {
    return (cfg.flags & SHAPES_FLAG_LEARNED) && mlp_model && cfg.warm_start && ds_cap == 0;
  }
  bool collect_on(const shapes_config& cfg) const { return ds_cap > 0 && cfg.warm_start; }

  void free_step_buffers() {
    dfree(pair_a); dfree(pair_b); dfree(slot_cnt); dfree(slot_off); dfree(slot_feat); dfree(slot_val);
    dfree(np_perm);
    np_perm = nullptr;
    for (int k = 0; k < 2; ++k) { dfree(c_key[k]); dfree(lam[k]); }
    dfree(c_ga); dfree(c_gb); dfree(c_slot); dfree(c_flip); dfree(c_hit); dfree(c_val); dfree(con);
    dfree(sched_info); dfree(sched_list); dfree(sched_arr); dfree(gdesc);
    sched_info = nullptr;
    sched_list = sched_arr = nullptr;
    free_scan();
    dfree(snap_key); dfree(snap_lam);
    free_row_buffers();
    dfree(lw_refs); dfree(lw_rank); dfree(lw_hrank); dfree(lw_hitflag);
    dfree(lw_rowflag); dfree(lw_rowoff); dfree(lw_row_start); dfree(lw_side); dfree(lw_lag);
    lw_lag = nullptr;
    lw_rowflag = lw_rowoff = lw_row_start = nullptr;
    lw_side = nullptr;
    dfree(lw_color);
    lw_refs = lw_rank = lw_hrank = lw_hitflag = lw_color = nullptr;
    pair_a = pair_b = slot_cnt = slot_off = slot_feat = nullptr;
    slot_val = nullptr;
    c_key[0] = c_key[1] = nullptr;
    lam[0] = lam[1] = nullptr;
    c_ga = c_gb = c_slot = nullptr;
    c_flip = c_hit = nullptr;
    c_val = nullptr;
    con = nullptr;
    gdesc = nullptr;
    snap_key = nullptr;
    snap_lam = nullptr;
  }

  /* (Re)allocates every buffer sized by pairs/contacts/updates.  Cache
   * contents in c_key/lam[cache_buf] are preserved across a regrowth. */
  void alloc_step_buffers(int32_t new_pair_cap, int32_t new_contact_cap, int iterations) {
    if (stream) ck(cudaStreamSynchronize(stream), "sync");
    invalidate_graphs();
    const int32_t old_cap = contact_cap;
    uint64_t* keep_key = nullptr;
    double* keep_lam = nullptr;
    if (c_key[cache_buf] && old_cap > 0) {
      keep_key = dalloc<uint64_t>(old_cap, "cudaMalloc keep");
      keep_lam = dalloc<double>(2 * (size_t)old_cap, "cudaMalloc keep");
      ck(cudaMemcpyAsync(keep_key, c_key[cache_buf], sizeof(uint64_t) * old_cap, cudaMemcpyDeviceToDevice, stream), "copy");
      ck(cudaMemcpyAsync(keep_lam, lam[cache_buf], sizeof(double) * 2 * old_cap, cudaMemcpyDeviceToDevice, stream), "copy");
      ck(cudaStreamSynchronize(stream), "sync");
    }
    free_step_buffers();
    pair_cap = new_pair_cap;
    contact_cap = new_contact_cap;
    item_cap = (int64_t)(iterations + 1) * contact_cap;
    pair_a = dalloc<int32_t>(pair_cap, "cudaMalloc pairs");
    pair_b = dalloc<int32_t>(pair_cap, "cudaMalloc pairs");
    slot_cnt = dalloc<int32_t>(pair_cap, "cudaMalloc slots");
    slot_off = dalloc<int32_t>((size_t)pair_cap + 1, "cudaMalloc slots");
    slot_feat = dalloc<int32_t>(2 * (size_t)pair_cap, "cudaMalloc slots");
    slot_val = dalloc<double>(10 * (size_t)pair_cap, "cudaMalloc slots");
    np_perm = dalloc<int32_t>(pair_cap, "cudaMalloc slots");
    for (int k = 0; k < 2; ++k) {
      c_key[k] = dalloc<uint64_t>(contact_cap, "cudaMalloc contacts");
      lam[k] = dalloc<double>(2 * (size_t)contact_cap, "cudaMalloc contacts");
    }
    c_ga = dalloc<int32_t>(contact_cap, "cudaMalloc contacts");
    c_slot = dalloc<int32_t>(contact_cap, "cudaMalloc contacts");
    c_gb = dalloc<int32_t>(contact_cap, "cudaMalloc contacts");
    c_flip = dalloc<uint8_t>(contact_cap, "cudaMalloc contacts");
    c_hit = dalloc<uint8_t>(contact_cap, "cudaMalloc contacts");
    c_val = dalloc<double>(5 * (size_t)contact_cap, "cudaMalloc contacts");
    con = dalloc<Con>(contact_cap, "cudaMalloc constraints");
    sched_info = dalloc<int4>(contact_cap, "cudaMalloc constraints");
    sched_list = dalloc<int32_t>(2 * (size_t)contact_cap, "cudaMalloc constraints");
    sched_arr = dalloc<int32_t>(contact_cap, "cudaMalloc constraints");
    gdesc = dalloc<int4>(item_cap + W + 1, "cudaMalloc items");
    alloc_scan();
    if (!large_worlds.empty()) {
      lw_refs = dalloc<int32_t>(2 * (size_t)contact_cap, "cudaMalloc large world");
      lw_rank = dalloc<int32_t>(2 * (size_t)contact_cap, "cudaMalloc large world");
      lw_hrank = dalloc<int32_t>(2 * (size_t)contact_cap, "cudaMalloc large world");
      lw_hitflag = dalloc<int32_t>(contact_cap, "cudaMalloc large world");
      lw_rowflag = dalloc<int32_t>(contact_cap, "cudaMalloc large world");
      lw_rowoff = dalloc<int32_t>((size_t)contact_cap + 1, "cudaMalloc large world");
      lw_row_start = dalloc<int32_t>(contact_cap, "cudaMalloc large world");
      lw_side = dalloc<int4>(2 * (size_t)contact_cap, "cudaMalloc large world");
      lw_lag = dalloc<ulonglong2>(2 * (size_t)contact_cap, "cudaMalloc large world");
      lw_color = dalloc<int32_t>(contact_cap, "cudaMalloc large world");
    }
    snap_cap = contact_cap;
    snap_key = dalloc<uint64_t>(snap_cap, "cudaMalloc snapshot");
    snap_lam = dalloc<double>(2 * (size_t)snap_cap, "cudaMalloc snapshot");
    if (keep_key) {
      ck(cudaMemcpyAsync(c_key[cache_buf], keep_key, sizeof(uint64_t) * old_cap, cudaMemcpyDeviceToDevice, stream), "copy");
      ck(cudaMemcpyAsync(lam[cache_buf], keep_lam, sizeof(double) * 2 * old_cap, cudaMemcpyDeviceToDevice, stream), "copy");
      ck(cudaStreamSynchronize(stream), "sync");
      dfree(keep_key);
      dfree(keep_lam);
    }
  }

  int32_t cached_iterations = -1;

  void ensure_items(int iterations) {
    if ((int64_t)(iterations + 1) * contact_cap <= item_cap) return;
    ck(cudaStreamSynchronize(stream), "sync");
    invalidate_graphs();
    dfree(gdesc);
    item_cap = (int64_t)(iterations + 1) * contact_cap;
    gdesc = dalloc<int4>(item_cap + W + 1, "cudaMalloc items");
  }

  /* Solver groups: worlds sorted by body count (largest first, so the longest
   * dependency chains start first) and packed by the caller's choice of
   * worlds or bodies per group.  Else so that one group falls to each SM, with
   * eight solver warps, while that is at most kLoneGroupBodies bodies (per step,
   * ms, against four groups to an SM: 119 bodies to an SM 0.345 / 0.435, 197
   * 0.326 / 0.364, 215 0.485 / 0.52; 252 0.373 / 0.338, 526 0.686 / 0.662), and
   * above it four groups that close at kAutoGroupBodies bodies. */
  static constexpr int kLoneGroupBodies = 224;
  static constexpr int kAutoGroupBodies = 512;
  int32_t auto_group_target() {
    int64_t total = 0;
    for (int w = 0; w < W; ++w) {
      const int32_t n = h_world_body_off[w + 1] - h_world_body_off[w];
      if (n < large_world_bodies) total += n;
    }
    const int64_t per_sm = total / num_sms();
    return (int32_t)std::max<int64_t>(
        1, per_sm <= kLoneGroupBodies ? per_sm : std::min<int64_t>(kAutoGroupBodies, per_sm / 4));
  }
  void make_groups(int iterations) {
    if (stream) ck(cudaStreamSynchronize(stream), "sync"); /* no kernel may still read the old groups */
    invalidate_graphs();
    std::vector<int32_t> order;
    const bool given = (int)world_order.size() == W;
    for (int k = 0; k < W; ++k) {
      const int w = given ? world_order[k] : k;
      if (h_world_body_off[w + 1] - h_world_body_off[w] < large_world_bodies) order.push_back(w);
    }
    const int n_small = (int)order.size();
    if (!given)
      std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return (h_world_body_off[a + 1] - h_world_body_off[a]) > (h_world_body_off[b + 1] - h_world_body_off[b]);
      });
    const bool by_worlds = worlds_per_group_override > 0;
    const int per_group = by_worlds ? std::min(shapes::kMaxGroupWorlds, worlds_per_group_override) : 0;
    int32_t target = by_worlds ? 0 : target_group_bodies;
    if (!by_worlds && target <= 0) target = auto_group_target();
    h_group_world_off.assign(1, 0);
    int32_t max_bodies = 0, bodies = 0, in_group = 0;
    for (int k = 0; k < n_small; ++k) {
      const int w = order[k];
      bodies += h_world_body_off[w + 1] - h_world_body_off[w];
      ++in_group;
      const bool close = target > 0 ? (bodies >= target || in_group == shapes::kMaxGroupWorlds) : in_group == per_group;
      if (close || k == n_small - 1) {
        h_group_world_off.push_back(k + 1);
        max_bodies = std::max(max_bodies, bodies);
        bodies = 0;
        in_group = 0;
      }
    }
    h_group_worlds = order;
    dfree(group_world_off);
    dfree(group_worlds);
    const size_t G = h_group_world_off.size() - 1;
    group_max_bodies = max_bodies;
    group_world_off = dalloc<int32_t>(G + 1, "cudaMalloc groups");
    group_worlds = dalloc<int32_t>(std::max(n_small, 1), "cudaMalloc groups");
    ck(cudaMemcpy(group_world_off, h_group_world_off.data(), sizeof(int32_t) * (G + 1), cudaMemcpyHostToDevice),
       "upload groups");
    if (n_small > 0)
      ck(cudaMemcpy(group_worlds, h_group_worlds.data(), sizeof(int32_t) * n_small, cudaMemcpyHostToDevice),
         "upload groups");
    grouped_iterations = iterations;
    dfree(phase_clock);
    phase_clock = dalloc<long long>(8 * std::max<size_t>(G, 1), "cudaMalloc groups");
    phase_clock_groups = (int32_t)G;
  }

  int num_groups() const { return (int)h_group_world_off.size() - 1; }

  /* Worlds with at least large_world_bodies bodies are solved by the
   * large-world paths; their per-body scratch is sized for the largest. */
  void setup_large_worlds() {
    dfree(lw_bcnt); dfree(lw_bstart); dfree(lw_bh); dfree(lw_bn); dfree(lw_vel); dfree(lw_color_cnt); dfree(lw_ctl);
    lw_bcnt = lw_bstart = lw_bh = lw_bn = lw_color_cnt = nullptr;
    lw_vel = nullptr;
    lw_ctl = nullptr;
    large_worlds.clear();
    lw_nb_max = 0;
    for (int w = 0; w < W; ++w) {
      const int32_t n = h_world_body_off[w + 1] - h_world_body_off[w];
      if (n >= large_world_bodies) {
        large_worlds.push_back(w);
        lw_nb_max = std::max(lw_nb_max, n);
      }
    }
    if (large_worlds.empty()) return;
    lw_bcnt = dalloc<int32_t>((size_t)lw_nb_max + 1, "cudaMalloc large world");
    lw_bstart = dalloc<int32_t>((size_t)lw_nb_max + 1, "cudaMalloc large world");
    lw_bh = dalloc<int32_t>(lw_nb_max, "cudaMalloc large world");
    lw_bn = dalloc<int32_t>(lw_nb_max, "cudaMalloc large world");
    lw_vel = dalloc<ulonglong2>(3 * (size_t)lw_nb_max, "cudaMalloc large world");
    lw_color_cnt = dalloc<int32_t>(shapes::kMaxColors + 1, "cudaMalloc large world");
    lw_ctl = dalloc<unsigned long long>(8 * large_worlds.size(), "cudaMalloc large world");
    ck(cudaMemset(lw_ctl, 0, sizeof(unsigned long long) * 8 * large_worlds.size()), "memset");
    if (!metric_part) metric_part = dalloc<double>(shapes::kMetricParts, "cudaMalloc large world");
  }

  shapes::LW lw_view(size_t k) const {
    shapes::LW w{};
    w.wld = large_worlds[k];
    w.b0 = h_world_body_off[w.wld];
    w.nb = h_world_body_off[w.wld + 1] - w.b0;
    w.bcnt = lw_bcnt;
    w.bstart = lw_bstart;
    w.refs = lw_refs;
    w.rank = lw_rank;
    w.hrank = lw_hrank;
    w.bh = lw_bh;
    w.bn = lw_bn;
    w.vel = lw_vel;
    w.lag = lw_lag;
    w.hitflag = lw_hitflag;
    w.rowflag = lw_rowflag;
    w.rowoff = lw_rowoff;
    w.row_start = lw_row_start;
    w.side = lw_side;
    w.color = lw_color;
    w.color_cnt = lw_color_cnt;
    w.ctl = lw_ctl + 8 * k;
    return w;
  }

  /* The group solve (frontier.cuh) of every group.  Each CTA's shared memory
   * holds the largest group at two and a half contacts a body (five where it
   * has the SM to itself), up to a third of an SM's where groups share one (a
   * group that does not fit keeps its lists and velocities in global memory).
   * Groups that have an SM to themselves take eight warps, of which four
   * prepare a narrow level while four solve one; groups that share one take
   * four. */
  static constexpr int kFrontierSmem = 220 * 1024;
  SolveShape solve_shape() {
    const int per_sm = std::max(1, (int)(((int64_t)num_groups() * handles_in_flight + num_sms() - 1) / num_sms()));
    SolveShape s{};
    s.chained = chain();
    s.warps = !group_warps_auto ? group_warps : (per_sm <= 1 ? 8 : 4);
    const int64_t contacts = (per_sm <= 1 ? 10LL : 5LL) * group_max_bodies / 2;
    const size_t want = shapes::frontier_bytes(group_max_bodies, contacts, true);
    /* four groups resident in place of three where their lists fit a quarter of the SM, the Lagrangians then in
     * global memory: 500 groups of 560 bodies run in one wave in place of two, 1.90 -> 1.64 ms a step */
    size_t most = kFrontierSmem / std::min(per_sm, 3);
    if (per_sm >= 4 && shapes::frontier_bytes(group_max_bodies, contacts, false) <= kFrontierSmem / 4)
      most = kFrontierSmem / 4;
    s.smem = (int)std::min<size_t>(want, most);
    s.split_limit = per_sm <= 1 ? 16 : 4;
    return s;
  }
  template <int P>
  void launch_frontier(const Dev& d, const shapes_config& cfg, const SolveShape& s) {
    const int G = num_groups();
    ck(cudaFuncSetAttribute(shapes::k_frontier<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFrontierSmem),
       "cudaFuncSetAttribute");
    launch_chained(s.chained, shapes::k_frontier<P>, G, 32 * (P + 1), s.smem, stream, d, cfg.iterations, cfg.warm_start,
                   cfg.external, cfg.accel_x, cfg.accel_y, cfg.dt, G, s.smem, spread_heavy ? num_sms() : 0,
                   s.split_limit, poll_limit_or(shapes::kFrontierPollLimit));
  }
  void launch_groups(const Dev& d, const shapes_config& cfg) {
    const SolveShape s = solve_shape();
    if (s.warps == 1) launch_frontier<1>(d, cfg, s);
    else if (s.warps == 2) launch_frontier<2>(d, cfg, s);
    else if (s.warps == 4) launch_frontier<4>(d, cfg, s);
    else launch_frontier<8>(d, cfg, s);
  }

  /* Solve one large world: ranks of every contact on its bodies, then the
   * ordered dataflow kernel, or the coloured sweep. */
  /* Per-world residual (or largest depth): one warp per world, and for each
   * large world kMetricParts warps plus an ordered combine. */
  void world_metric_kernels(const Dev& d, bool residual) {
    const int split = large_worlds.empty() ? INT32_MAX : large_world_bodies;
    if (residual)
      shapes::k_residual<<<(W * 32 + 127) / 128, 128, 0, stream>>>(d, split);
    else
      shapes::k_world_depth<<<(W * 32 + 127) / 128, 128, 0, stream>>>(d, split);
    for (int wld : large_worlds) {
      if (residual) {
        shapes::k_metric_part<true><<<shapes::kMetricParts / 4, 128, 0, stream>>>(d, wld, metric_part);
        shapes::k_metric_final<true><<<1, 32, 0, stream>>>(d, wld, metric_part);
      } else {
        shapes::k_metric_part<false><<<shapes::kMetricParts / 4, 128, 0, stream>>>(d, wld, metric_part);
        shapes::k_metric_final<false><<<1, 32, 0, stream>>>(d, wld, metric_part);
      }
    }
  }

  void solve_large_world(const Dev& d, size_t k, const shapes_config& cfg) {
    shapes::LW w = lw_view(k);
    const int cap = contact_cap;
    const bool ordered = !(cfg.flags & SHAPES_FLAG_COLOURED);
    stage(3, ordered ? 7 : 5, [&]() {
      shapes::k_lw_setup<<<grid_for(w.nb + 1, 256), 256, 0, stream>>>(d, w);
      shapes::k_lw_count<<<grid_for(cap, 256), 256, 0, stream>>>(d, w, cfg.iterations);
      scan_raw(w.bcnt, w.nb, nullptr, w.bstart);
      shapes::k_lw_scatter<<<grid_for(cap, 256), 256, 0, stream>>>(d, w);
      shapes::k_lw_rank<<<grid_for(w.nb, 128), 128, 0, stream>>>(d, w);
      if (ordered) { /* the sequence's rows, pass skew, side entries */
        scan_raw(w.rowflag, cap, w.ctl + 4, w.rowoff);
        shapes::k_lw_rows<<<grid_for(cap, 256), 256, 0, stream>>>(d, w);
      }
    });
    stage(4, ordered ? 3 : 1, [&]() {
      if (ordered) {
        shapes::k_lw_begin<<<grid_for(2LL * cap, 256), 256, 0, stream>>>(d, w, cfg.external, cfg.accel_x, cfg.accel_y,
                                                                         cfg.dt);
        shapes::k_lw_ordered<<<kSMs * shapes::kOrderedBlocksPerSM, shapes::kOrderedThreads, 0, stream>>>(
            d, w, cfg.iterations, cfg.warm_start, poll_limit > 0 ? poll_limit : shapes::kPollLimit);
        shapes::k_lw_end<<<grid_for(2LL * cap, 256), 256, 0, stream>>>(d, w);
        return;
      }
      cudaLaunchConfig_t lc{};
      lc.gridDim = dim3(num_sms() * shapes::kColourBlocksPerSM);
      lc.blockDim = dim3(shapes::kColourThreads);
      lc.stream = stream;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeCooperative;
      at[0].val.cooperative = 1;
      lc.attrs = at;
      lc.numAttrs = 1;
      ck(cudaLaunchKernelEx(&lc, shapes::k_lw_coloured, d, w, cfg.iterations, cfg.warm_start, cfg.external, cfg.accel_x,
                            cfg.accel_y, cfg.dt, poll_limit_or(shapes::kPollLimit)),
         "k_lw_coloured");
    });
  }

  void free_incremental() {
    dfree(fatk); dfree(nbr); dfree(nbr_cnt); dfree(moved); dfree(inc_state); dfree(inc_rebuild); dfree(inc_moved);
    dfree(inc_frames); dfree(inc_margin);
    fatk = nullptr;
    nbr = nullptr;
    nbr_cnt = nullptr;
    moved = nullptr;
    inc_state = inc_rebuild = inc_moved = inc_frames = nullptr;
    inc_margin = nullptr;
  }

  /* Adjacency lists of nbr_cap entries per body; every world rebuilds next frame. */
  void setup_incremental() {
    free_incremental();
    if (!any_grid) return;
    fatk = dalloc<uint64_t>(4 * (size_t)N, "cudaMalloc grid");
    nbr = dalloc<int32_t>((size_t)N * nbr_cap, "cudaMalloc grid");
    nbr_cnt = dalloc<int32_t>(N, "cudaMalloc grid");
    moved = dalloc<uint8_t>(N, "cudaMalloc grid");
    inc_state = dalloc<int32_t>(W, "cudaMalloc grid");
    inc_rebuild = dalloc<int32_t>(W, "cudaMalloc grid");
    inc_moved = dalloc<int32_t>(W, "cudaMalloc grid");
    inc_frames = dalloc<int32_t>(W, "cudaMalloc grid");
    inc_margin = dalloc<double>(W, "cudaMalloc grid");
    reset_incremental();
  }

  void reset_incremental() {
    if (inc_state) ck(cudaMemsetAsync(inc_state, 0, sizeof(int32_t) * W, stream), "memset");
  }

  /* Worlds with at least grid_min_bodies bodies use the grid broadphase. */
  void setup_grid() {
    dfree(grid_T); dfree(grid_base); dfree(grid_inv_s); dfree(grid_lim); dfree(bucket_cnt); dfree(bucket_off);
    dfree(grid_ent); dfree(cell); dfree(row_mode); dfree(large_cnt); dfree(large_ids);
    std::vector<int32_t> T(W), base(W);
    int64_t nb = 0;
    any_grid = false;
    for (int w = 0; w < W; ++w) {
      const int32_t n = h_world_body_off[w + 1] - h_world_body_off[w];
      int32_t t = 0;
      if (n >= grid_min_bodies) {
        t = 1;
        while (t < 2 * n) t <<= 1;
        any_grid = true;
      }
      T[w] = t;
      base[w] = (int32_t)nb;
      nb += t;
    }
    if (nb > INT32_MAX / 2) throw CudaError{cudaErrorMemoryAllocation};
    n_buckets = (int32_t)nb;
    grid_T = dalloc<int32_t>(W, "cudaMalloc grid");
    grid_base = dalloc<int32_t>(W, "cudaMalloc grid");
    grid_inv_s = dalloc<double>(W, "cudaMalloc grid");
    grid_lim = dalloc<double>(W, "cudaMalloc grid");
    bucket_cnt = dalloc<int32_t>((size_t)n_buckets + 1, "cudaMalloc grid");
    bucket_off = dalloc<int32_t>((size_t)n_buckets + 1, "cudaMalloc grid");
    grid_ent = dalloc<int4>(N, "cudaMalloc grid");
    cell = dalloc<int2>(N, "cudaMalloc grid");
    row_mode = dalloc<uint8_t>(N, "cudaMalloc grid");
    large_cnt = dalloc<int32_t>(W, "cudaMalloc grid");
    large_ids = dalloc<int32_t>(N, "cudaMalloc grid");
    ck(cudaMemcpy(grid_T, T.data(), sizeof(int32_t) * W, cudaMemcpyHostToDevice), "upload grid");
    ck(cudaMemcpy(grid_base, base.data(), sizeof(int32_t) * W, cudaMemcpyHostToDevice), "upload grid");
    ck(cudaMemset(row_mode, 0, N), "memset");
    ck(cudaMemsetAsync(bucket_cnt, 0, sizeof(int32_t) * ((size_t)n_buckets + 1), stream), "memset");
    {
      /* chunks of at most 4096 bodies, never crossing a world (empty worlds have none) */
      dfree(ext_chunk); dfree(ext_chunk_off); dfree(ext_part_sum); dfree(ext_part_cnt); dfree(ext_done);
      std::vector<int32_t> ranges, choff(W + 1, 0);
      for (int w = 0; w < W; ++w) {
        choff[w] = (int32_t)(ranges.size() / 2);
        for (int32_t b = h_world_body_off[w]; b < h_world_body_off[w + 1]; b += 4096) {
          ranges.push_back(b);
          ranges.push_back(std::min<int32_t>(b + 4096, h_world_body_off[w + 1]));
        }
      }
      n_ext_chunks = (int32_t)(ranges.size() / 2);
      choff[W] = n_ext_chunks;
      ext_chunk = dalloc<int32_t>(std::max<size_t>(ranges.size(), 1), "cudaMalloc grid");
      ext_chunk_off = dalloc<int32_t>((size_t)W + 1, "cudaMalloc grid");
      ext_part_sum = dalloc<double>(std::max<int32_t>(n_ext_chunks, 1), "cudaMalloc grid");
      ext_part_cnt = dalloc<int32_t>(std::max<int32_t>(n_ext_chunks, 1), "cudaMalloc grid");
      ext_done = dalloc<int32_t>(W, "cudaMalloc grid");
      ck(cudaMemsetAsync(ext_done, 0, sizeof(int32_t) * W, stream), "memset");
      if (n_ext_chunks)
        ck(cudaMemcpy(ext_chunk, ranges.data(), sizeof(int32_t) * ranges.size(), cudaMemcpyHostToDevice),
           "upload grid");
      ck(cudaMemcpy(ext_chunk_off, choff.data(), sizeof(int32_t) * (W + 1), cudaMemcpyHostToDevice), "upload grid");
    }
    setup_incremental();
    setup_sap();
  }

  /* One exclusive scan; clear, total and overflow as in k_scan. */
  void scan_raw(int32_t* in, int n_cap, const unsigned long long* n_dev, int32_t* out, bool clear = false,
                unsigned long long* total = nullptr, int32_t total_cap = 0, unsigned overflow_bit = 0) {
    const int tiles = n_cap / shapes::kScanTile + 1;
    launch_chained(chain(), shapes::k_scan, std::min(tiles, 2 * kSMs), shapes::kScanThreads, 0, stream, in, n_cap, n_dev,
                   scan_state, out, clear ? 1 : 0, total, total_cap, counters + shapes::kCntOverflow, overflow_bit,
                   counters + shapes::kCntSolveErr);
  }
  template <class... A>
  void scan(A... a) {
    stage(6, 1, [&]() { scan_raw(a...); });
  }

  void pose(int advance, double dt) {
    Dev d = view(0);
    launch_pose(chain(), stream, N, d, dt, advance);
  }

  /* Broadphase + narrowphase into buffer `wb`; with `solve`, also constraint
   * build, warm start, sweeps, integration. */
  void enqueue_step(const shapes_config& cfg, bool solve, int wb) {
    Dev d = view(wb);
    const bool learn = solve && learned_on(cfg), collect = solve && collect_on(cfg);
    if (learn || collect) { /* row buffers were sized by run() before this view */
      d.learned_mask = learned_mask;
      d.miss_flag = miss_flag;
      d.miss_off = miss_off;
      d.miss_ids = miss_ids;
      d.miss_n = miss_n;
      d.mfeat = mfeat;
      d.collect_all = collect ? 1 : 0;
      d.judge_res = judge_res;
      d.judge_depth = judge_depth;
    }
    const bool inc = any_grid && d.nbr != nullptr;
    const bool sap = any_sap && !inc;
    auto by_team = [&](auto launch) {
      if (shapes::row_teams(N)) launch(std::integral_constant<int, shapes::kRowTeam>{});
      else launch(std::integral_constant<int, shapes::kRowPair>{});
    };
    if (!sap) d.world_sap = nullptr;
    /* the bucket counts are zero between steps: their scan leaves them so */
    if (inc) {
      stage(0, 3, [&]() {
        if (n_ext_chunks) launch_chained(chain(), shapes::k_grid_stats, n_ext_chunks, 256, 0, stream, d, 1);
        launch_chained(chain(), shapes::k_inc_mark, grid_for(N, 256), 256, 0, stream, d);
        launch_chained(chain(), shapes::k_inc_update, grid_for(N, 128), 128, 0, stream, d);
      });
      scan(bucket_cnt, n_buckets, nullptr, bucket_off, true);
      stage(0, 2, [&]() {
        launch_chained(chain(), shapes::k_inc_scatter, grid_for(N, 256), 256, 0, stream, d);
        by_team([&](auto team) {
          constexpr int kTeam = decltype(team)::value;
          launch_chained(chain(), shapes::k_inc_query<kTeam>, grid_for((long long)N * kTeam, shapes::kRowThreads),
                         shapes::kRowThreads, 0, stream, d);
        });
      });
    } else if (any_grid) {
      stage(0, 2, [&]() {
        if (n_ext_chunks) launch_chained(chain(), shapes::k_grid_stats, n_ext_chunks, 256, 0, stream, d, 0);
        launch_chained(chain(), shapes::k_grid_bin, grid_for(N, 256), 256, 0, stream, d);
      });
      scan(bucket_cnt, n_buckets, nullptr, bucket_off, true);
      stage(0, 1, [&]() { launch_chained(chain(), shapes::k_grid_scatter, grid_for(N, 256), 256, 0, stream, d); });
      if (sap) {
        stage(0, 1, [&]() { shapes::k_sap_count<<<grid_for(N, 256), 256, 0, stream>>>(d); });
        scan(sap_cnt, n_sap_buckets, nullptr, sap_off, true);
        stage(0, 2, [&]() {
          shapes::k_sap_scatter<<<grid_for(N, 256), 256, 0, stream>>>(d);
          shapes::k_sap_ends<<<grid_for(W, 128), 128, 0, stream>>>(d);
        });
      }
    }
    stage(0, sap ? 2 : 1, [&]() {
      if (any_grid)
        by_team([&](auto team) {
          constexpr int kTeam = decltype(team)::value;
          const int blocks = grid_for((long long)N * kTeam, shapes::kRowThreads);
          if (inc)
            launch_chained(chain(), shapes::k_count_rows<true, kTeam>, blocks, shapes::kRowThreads, 0, stream, d);
          else
            launch_chained(chain(), shapes::k_count_rows<false, kTeam>, blocks, shapes::kRowThreads, 0, stream, d);
        });
      else
        launch_chained(chain(), shapes::k_count_brute, grid_for((long long)N * 32, 256), 256, 0, stream, d);
      if (sap) shapes::k_sap_rows<true><<<grid_for(N, 128), 128, 0, stream>>>(d);
    });
    scan(row_cnt, N, nullptr, row_off, false, counters + shapes::kCntPairs, pair_cap, 1u);
    stage(0, sap ? 3 : 1, [&]() {
      const int blocks = grid_for(N, shapes::kRowThreads);
      if (inc)
        launch_chained(chain(), shapes::k_write_rows<true, true>, blocks, shapes::kRowThreads, 0, stream, d);
      else if (any_grid)
        launch_chained(chain(), shapes::k_write_rows<true, false>, blocks, shapes::kRowThreads, 0, stream, d);
      else
        launch_chained(chain(), shapes::k_write_rows<false, false>, blocks, shapes::kRowThreads, 0, stream, d);
      if (sap) {
        shapes::k_sap_rows<false><<<grid_for(N, 128), 128, 0, stream>>>(d);
        shapes::k_sap_sort_rows<<<grid_for(N, 128), 128, 0, stream>>>(d);
      }
    });
    stage(1, np_lanes > 1 ? 4 : 1, [&]() {
      if (np_lanes <= 1) {
        launch_chained(chain(), shapes::k_narrowphase, grid_for(pair_cap, shapes::kNpThreads), shapes::kNpThreads, 0,
                       stream, d);
        return;
      }
      ck(cudaMemsetAsync(np_cls, 0, sizeof(int32_t) * shapes::kNpClasses, stream), "memset");
      shapes::k_np_count<<<grid_for(pair_cap, 256), 256, 0, stream>>>(d);
      shapes::k_np_offsets<<<1, 32, 0, stream>>>(d);
      shapes::k_np_scatter<<<grid_for(pair_cap, 256), 256, 0, stream>>>(d);
      switch (np_lanes) {
        case 2: shapes::k_narrowphase_lanes<2><<<grid_for(2LL * pair_cap, 128), 128, 0, stream>>>(d); break;
        case 4: shapes::k_narrowphase_lanes<4><<<grid_for(4LL * pair_cap, 128), 128, 0, stream>>>(d); break;
        case 8: shapes::k_narrowphase_lanes<8><<<grid_for(8LL * pair_cap, 128), 128, 0, stream>>>(d); break;
        case 16: shapes::k_narrowphase_lanes<16><<<grid_for(16LL * pair_cap, 128), 128, 0, stream>>>(d); break;
        default: shapes::k_narrowphase_lanes<32><<<grid_for(32LL * pair_cap, 128), 128, 0, stream>>>(d); break;
      }
    });
    scan(slot_cnt, pair_cap, counters + shapes::kCntPairs, slot_off, false, counters + shapes::kCntContacts, contact_cap,
         2u);
    stage(2, 2, [&]() {
      launch_chained(chain(), shapes::k_contact_slots, grid_for(2LL * pair_cap, 256), 256, 0, stream, d);
      const bool staged = shapes::build_staged(contact_cap) && chain();
      launch_chained(chain(), shapes::k_build, grid_for(contact_cap, shapes::kBuildThreads), shapes::kBuildThreads,
                     staged ? shapes::kBuildThreads * sizeof(shapes::Con) : 0, stream, d, cfg.baumgarte / cfg.dt,
                     cfg.slop, cfg.warm_start, solve ? 1 : 0, staged ? 1 : 0);
    });
    if (!solve) return;
    if (learn || collect) {
      stage(7, 2 + (learn ? 2 : 0), [&]() {
        scan_raw(miss_flag, contact_cap, counters + shapes::kCntContacts, miss_off);
        shapes::k_learned_features<<<grid_for(contact_cap, 128), 128, 0, stream>>>(d, cfg.external, cfg.accel_x,
                                                                                  cfg.accel_y, cfg.dt);
        if (learn) {
          ck(mlp::launch_predict_contacts(mlp::device_params(mlp_model), mlp::device_norm(mlp_model), mfeat, miss_n,
                                          miss_ids, d.lam, c_hit, shapes::kInfoHit,
                                          counters + shapes::kCntPredicted,
                                          reinterpret_cast<int*>(counters + shapes::kCntMlpErr), contact_cap, stream),
             "k_mlp_predict");
          if (judge_set) world_metric_kernels(d, false);
        }
      });
    }
    /* groups for cfg.iterations were built by run() before this view */
    if (num_groups() > 0) stage(4, 1, [&]() { launch_groups(d, cfg); });
    for (size_t k = 0; k < large_worlds.size(); ++k) solve_large_world(d, k, cfg);
    if ((cfg.flags & SHAPES_FLAG_RESIDUAL) || (learn && judge_set))
      stage(4, 1 + 2 * (int)large_worlds.size(), [&]() { world_metric_kernels(d, true); });
    if (learn && judge_set)
      stage(7, 1, [&]() { shapes::k_learned_judge<<<grid_for(W, 128), 128, 0, stream>>>(d); });
    if (collect)
      stage(7, 2, [&]() {
        shapes::k_collect<<<grid_for(contact_cap, 256), 256, 0, stream>>>(d, ds_feat, ds_tgt, ds_count, ds_cap);
        shapes::k_collect_advance<<<1, 1, 0, stream>>>(miss_n, ds_count, ds_cap);
      });
    stage(5, 1, [&]() { launch_pose(chain(), stream, N, d, cfg.dt, 1); });
  }

  /* The state a refused or regrown step returns to: the pose-and-velocity
   * fields, the cache (keys, Lagrangians, world offsets), the learned mask and
   * the sample count, copied in one launch. */
  void snapshot_segments(shapes::Segments& sg, int& n, bool to_snap, int cap) {
    n = 0;
    auto add = [&](void* live, void* snap, unsigned long long bytes) {
      sg.src[n] = to_snap ? live : snap;
      sg.dst[n] = to_snap ? snap : live;
      sg.bytes[n] = bytes;
      ++n;
    };
    for (int k = 0; k < 6; ++k) add(body[k], snap_body[k], sizeof(double) * (unsigned long long)N);
    add(c_key[cache_buf], snap_key, sizeof(uint64_t) * (unsigned long long)cap);
    add(lam[cache_buf], snap_lam, sizeof(double) * 2ull * (unsigned long long)cap);
    add(cwo[cache_buf], snap_cwo, sizeof(int32_t) * (unsigned long long)(W + 1));
    if (learned_mask) add(learned_mask, snap_mask, (unsigned long long)W);
    if (ds_count) add(ds_count, snap_ds_count, sizeof(unsigned long long));
  }
  void copy_segments(const shapes::Segments& sg, int n) {
    unsigned long long most = 0;
    for (int k = 0; k < n; ++k) most = std::max(most, sg.bytes[k]);
    const unsigned blocks = (unsigned)std::max<unsigned long long>(1, std::min<unsigned long long>((most / 8 + 255) / 256, 512));
    shapes::k_copy_segments<<<dim3(blocks, (unsigned)n), 256, 0, stream>>>(sg);
    ck(cudaGetLastError(), "launch");
  }
  void snapshot() {
    shapes::Segments sg{};
    int n = 0;
    snapshot_segments(sg, n, true, contact_cap);
    copy_segments(sg, n);
  }

  /* Restore into buffer `buf` (which becomes the cache buffer). */
  void restore(int saved_cap) {
    shapes::Segments sg{};
    int n = 0;
    snapshot_segments(sg, n, false, saved_cap);
    copy_segments(sg, n);
  }

  /* Asynchronous body-state upload for shapes_batches_step_io: caller arrays
   * into the staging arrays with the finiteness check into the bad-input
   * counter, then the staged state into the live arrays unless the check
   * failed, and a re-pose of the bodies whose pose inputs changed. */
  void io_upload(const shapes_bodies* in, double* const* mapped = nullptr);
  void io_commit() {
    shapes::Ptr10 p{};
    for (int k = 0; k < 10; ++k) {
      p.src[k] = body_stage[k];
      p.dst[k] = body[k];
    }
    shapes::k_commit_bodies<<<grid_for(N, 256), 256, 0, stream>>>(p, N, body_changed,
                                                                  counters + shapes::kCntBadInput);
    Dev d = view(0);
    launch_pose(chain(), stream, N, d, 0.0, 0, body_changed);
    ck(cudaGetLastError(), "launch");
  }
  /* The first `fields` body arrays (10: all; kStepFields: velocities and pose,
   * the only ones a step writes) into the caller's arrays. */
  void io_download(shapes_bodies* out, double* const* mapped = nullptr, int fields = 10);
  /* After an io step was enqueued: waits, and on refused input undoes the
   * step (SHAPES_E_NAN); otherwise finishes it, re-running the staged input
   * alone after a buffer regrowth. */
  int io_finish(const shapes_config& cfg, shapes_bodies* out, double* const* mapped_out = nullptr, int fields = 10);

  /* One call of `nsteps` steps (or one collide when !solve) in three parts,
   * so that several handles can have their steps in flight at once
   * (shapes_batches_step): prepare() sizes buffers and groups, enqueue()
   * snapshots the state for a retry and launches the steps and the read-back
   * of the counters without waiting, finish() (after the stream is drained)
   * checks them: kRunRetry means the buffers were too small, the state was
   * restored and grown, and the call must be enqueued again. */
  static constexpr int kRunRetry = 1;
  int run_retries = 0, run_saved_cache_buf = 0, run_saved_cap = 0;
  /* pinned host copy of the step counters (kCntSlots), so that reading them
   * back is an asynchronous copy and the wait happens where the caller waits */
  unsigned long long* run_counters = nullptr;
  /* behind them in the same pinned block, for handles of at most kStageBodies
   * bodies: ten arrays through which get_bodies and set_bodies move pageable
   * caller arrays, with one kernel and ten memcpys in place of ten driver copies.
   * get_bodies took 37 us in place of 112 at 21 bodies and 73 in place of 120
   * at 9,075; at 32,771 the ten memcpys were slower (234 us against 141) */
  static constexpr int kStageBodies = 16384;
  int stage_bodies = 0;
  int stage_stride() const { return (stage_bodies + 1) & ~1; } /* each array on 16 bytes */
  double* stage(int k) const {
    return reinterpret_cast<double*>(run_counters + shapes::kCntSlots) + (size_t)k * stage_stride();
  }
  void pinned_block() {
    const int want = N <= kStageBodies ? N : 0;
    if (run_counters && want <= stage_bodies) return;
    if (run_counters) {
      ck(cudaStreamSynchronize(stream), "sync");
      cudaFreeHost(run_counters);
      run_counters = nullptr;
    }
    stage_bodies = want;
    const size_t bytes = sizeof(unsigned long long) * shapes::kCntSlots;
    ck(cudaMallocHost(&run_counters, bytes + 10 * sizeof(double) * (size_t)stage_stride()), "cudaMallocHost");
    std::memset(run_counters, 0, bytes);
  }

  void prepare(const shapes_config& cfg, bool solve) {
    ensure_items(solve ? cfg.iterations : 0);
    /* (re)build the solver groups before any device view of this call is
     * taken: make_groups reallocates the group arrays */
    if (solve && grouped_iterations != cfg.iterations) make_groups(cfg.iterations);
    if (solve && (learned_on(cfg) || collect_on(cfg))) ensure_row_buffers();
  }

  void enqueue_begin(bool solve) {
    ck(cudaMemsetAsync(counters, 0, sizeof(unsigned long long) * shapes::kCntSlots, stream), "memset");
    if (lw_ctl) /* the large-world timeout flags stay set through the run's steps */
      ck(cudaMemsetAsync(lw_ctl, 0, sizeof(unsigned long long) * 8 * large_worlds.size(), stream), "memset");
    run_saved_cache_buf = cache_buf;
    run_saved_cap = contact_cap;
    if (solve) snapshot();
  }
  void enqueue_one(const shapes_config& cfg, bool solve) {
    const int wb = 1 - cache_buf;
    handles_in_flight = AtWork::on(device);
    if (solve)
      launch_step(cfg, wb);
    else
      enqueue_step(cfg, false, wb);
    if (solve) cache_buf = wb;
    results_buf = wb;
  }
  void enqueue_end() {
    pinned_block();
    ck(cudaMemcpyAsync(run_counters, counters, sizeof(unsigned long long) * shapes::kCntSlots, cudaMemcpyDeviceToHost,
                       stream),
       "read counters");
  }
  void enqueue(const shapes_config& cfg, int32_t nsteps, bool solve) {
    enqueue_begin(solve);
    for (int s = 0; s < (solve ? nsteps : 1); ++s) enqueue_one(cfg, solve);
    enqueue_end();
  }

  int finish(const shapes_config& cfg, bool solve) {
    ck(cudaStreamSynchronize(stream), "step");
    ck(cudaGetLastError(), "launch");
    if (profiling) collect_profile();
    const unsigned long long* agg = run_counters;
    if (agg[shapes::kCntMlpErr]) {
      g_last_error = "learned warm start: a bounded tensor-core wait gave up";
      return SHAPES_E_TIMEOUT;
    }
    if (agg[shapes::kCntSolveErr]) {
      g_last_error = "group solver or scan: a bounded wait gave up";
      return SHAPES_E_TIMEOUT;
    }
    if (!agg[shapes::kCntOverflow] && solve && !large_worlds.empty()) {
      std::vector<unsigned long long> ctl(8 * large_worlds.size());
      ck(cudaMemcpy(ctl.data(), lw_ctl, sizeof(unsigned long long) * ctl.size(), cudaMemcpyDeviceToHost), "ctl");
      for (size_t k = 0; k < large_worlds.size(); ++k)
        if (ctl[8 * k + 1]) {
          g_last_error = "large-world solver: a bounded wait gave up";
          return SHAPES_E_TIMEOUT;
        }
    }
    if (!agg[shapes::kCntOverflow]) {
      stats.pairs = (int64_t)agg[shapes::kCntPairs];
      stats.contacts = (int64_t)agg[shapes::kCntContacts];
      stats.cache_hits = (int64_t)agg[shapes::kCntHits] - (int64_t)agg[shapes::kCntPredicted];
      stats.predicted = (int64_t)agg[shapes::kCntPredicted];
      stats.reverted = (int64_t)agg[shapes::kCntReverted];
      stats.solver_items = (int64_t)agg[shapes::kCntItems];
      stats.solver_levels = (int64_t)agg[shapes::kCntLevels];
      stats.retries = run_retries;
      have_results = true;
      return SHAPES_OK;
    }
    if (++run_retries > 6) return SHAPES_E_CAPACITY;
    /* undo, grow, redo */
    const unsigned long long overflow = agg[shapes::kCntOverflow];
    cache_buf = run_saved_cache_buf;
    if (solve) restore(run_saved_cap);
    ck(cudaStreamSynchronize(stream), "restore");
    if (overflow & 4ull) { /* an adjacency list was full */
      if (nbr_cap > (1 << 14)) return SHAPES_E_CAPACITY;
      nbr_cap *= 2;
      invalidate_graphs();
      setup_incremental();
    }
    reset_incremental(); /* the lists follow the undone steps' poses */
    if (overflow & ~4ull) {
      const int64_t np = (int64_t)pair_cap * ((overflow & 1ull) ? 2 : 1);
      const int64_t nc = (int64_t)contact_cap * 2;
      if (np > INT32_MAX / 2 || nc > INT32_MAX / 2) return SHAPES_E_CAPACITY;
      alloc_step_buffers((int32_t)np, (int32_t)std::max<int64_t>(nc, 2 * np), solve ? cfg.iterations : 0);
    }
    ensure_items(solve ? cfg.iterations : 0);
    if (solve && (learned_on(cfg) || collect_on(cfg))) ensure_row_buffers();
    if (solve) pose(0, 0.0);
    return kRunRetry;
  }

  /* Runs `nsteps` steps (or one collide when !solve) with overflow retries. */
  int run(const shapes_config& cfg, int32_t nsteps, bool solve) {
    const AtWork at_work(device);
    prepare(cfg, solve);
    run_retries = 0;
    for (;;) {
      enqueue(cfg, nsteps, solve);
      const int rc = finish(cfg, solve);
      if (rc != kRunRetry) return rc;
    }
  }

  /* The local points in the caller's convention (a circle as (radius, 0)). */
  std::vector<double> local_xy_host() {
    std::vector<double> xs(V), ys(V), xy(2 * (size_t)V);
    ck(cudaMemcpyAsync(xs.data(), lx, sizeof(double) * V, cudaMemcpyDeviceToHost, stream), "download");
    ck(cudaMemcpyAsync(ys.data(), ly, sizeof(double) * V, cudaMemcpyDeviceToHost, stream), "download");
    ck(cudaStreamSynchronize(stream), "download");
    for (int64_t v = 0; v < V; ++v) {
      xy[2 * v] = xs[v];
      xy[2 * v + 1] = ys[v];
    }
    for (int32_t b = 0; b < N; ++b)
      if (h_radius[b] > 0.0) xy[2 * (size_t)h_vert_off[b]] = h_radius[b];
    return xy;
  }

  /* (Re)builds everything sized by the bodies and vertices from host arrays:
   * world offsets [W+1], the ten body arrays, vertex offsets [N+1] and local
   * vertices [2V].  Used by creation and by appends that change the
   * topology; settings, the stream, the network and the judge stay.  The
   * contact cache comes back empty (the caller restores it). */
  void init_topology(const int32_t* world_body_offsets, double* const bp[10], const int32_t* vert_offsets,
                     const double* local_verts_xy) {
    if (stream) ck(cudaStreamSynchronize(stream), "sync");
    invalidate_graphs();
    free_step_buffers();
    dfree(world_body_off); dfree(body_world); dfree(vert_off); dfree(lx); dfree(ly); dfree(emin); dfree(emax);
    dfree(radius);
    radius = nullptr;
    for (int k = 0; k < 10; ++k) {
      dfree(body[k]);
      dfree(body_stage[k]);
    }
    dfree(wx); dfree(wy); dfree(nx); dfree(ny); dfree(box); dfree(boxk); dfree(flags); dfree(body_changed);
    dfree(vf); dfree(ef);
    dfree(row_cnt); dfree(row_hits); dfree(row_off); dfree(world_pair_off); dfree(sched_body); dfree(sched_cur); dfree(world_levels);
    for (int k = 0; k < 6; ++k) dfree(snap_body[k]);
    dfree(active);
    active = nullptr;
    const int32_t n_worlds = W;
    N = world_body_offsets[n_worlds];
    V = vert_offsets[N];
    h_world_body_off.assign(world_body_offsets, world_body_offsets + n_worlds + 1);
    h_vert_off.assign(vert_offsets, vert_offsets + N + 1);
    h_active.assign(N, 1);
    h_body_world.resize(N);
    for (int w = 0; w < n_worlds; ++w)
      for (int32_t b = world_body_offsets[w]; b < world_body_offsets[w + 1]; ++b) h_body_world[b] = w;
    world_body_off = dalloc<int32_t>(n_worlds + 1, "cudaMalloc");
    body_world = dalloc<int32_t>(N, "cudaMalloc");
    vert_off = dalloc<int32_t>((size_t)N + 1, "cudaMalloc");
    lx = dalloc<double>(V, "cudaMalloc");
    ly = dalloc<double>(V, "cudaMalloc");
    emin = dalloc<int32_t>(V, "cudaMalloc");
    emax = dalloc<int32_t>(V, "cudaMalloc");
    for (int k = 0; k < 10; ++k) body[k] = dalloc<double>(N, "cudaMalloc bodies");
    for (int k = 0; k < 10; ++k) body_stage[k] = dalloc<double>(N, "cudaMalloc bodies");
    wx = dalloc<double>(V, "cudaMalloc");
    wy = dalloc<double>(V, "cudaMalloc");
    nx = dalloc<double>(V, "cudaMalloc");
    ny = dalloc<double>(V, "cudaMalloc");
    vf = dalloc<float4>(V, "cudaMalloc");
    ef = dalloc<float2>(V, "cudaMalloc");
    box = dalloc<double>(4 * (size_t)N, "cudaMalloc");
    boxk = dalloc<uint64_t>(4 * (size_t)N, "cudaMalloc");
    flags = dalloc<uint8_t>(N, "cudaMalloc");
    body_changed = dalloc<uint8_t>(N, "cudaMalloc");
    row_cnt = dalloc<int32_t>(N, "cudaMalloc");
    row_hits = dalloc<int32_t>(shapes::kRowHits * (size_t)N, "cudaMalloc");
    row_off = dalloc<int32_t>((size_t)N + 1, "cudaMalloc");
    world_pair_off = dalloc<int32_t>(n_worlds + 1, "cudaMalloc");
    if (!cwo[0])
      for (int k = 0; k < 2; ++k) cwo[k] = dalloc<int32_t>(n_worlds + 1, "cudaMalloc");
    sched_body = dalloc<int32_t>(4 * (size_t)N, "cudaMalloc");
    sched_cur = dalloc<uint32_t>(N, "cudaMalloc");
    world_levels = dalloc<int32_t>(n_worlds, "cudaMalloc");
    ck(cudaMemset(world_levels, 0, sizeof(int32_t) * n_worlds), "memset");
    if (!counters) counters = dalloc<unsigned long long>(shapes::kCntSlots, "cudaMalloc");
    if (!np_cls) np_cls = dalloc<int32_t>(2 * shapes::kNpClasses + 1, "cudaMalloc");
    if (!world_residual) world_residual = dalloc<double>(n_worlds, "cudaMalloc");
    if (!world_depth) world_depth = dalloc<double>(n_worlds, "cudaMalloc");
    for (int k = 0; k < 6; ++k) snap_body[k] = dalloc<double>(N, "cudaMalloc snapshot");
    if (!snap_cwo) snap_cwo = dalloc<int32_t>(n_worlds + 1, "cudaMalloc snapshot");
    ck(cudaMemcpy(world_body_off, world_body_offsets, sizeof(int32_t) * (n_worlds + 1), cudaMemcpyHostToDevice),
       "upload");
    ck(cudaMemcpy(body_world, h_body_world.data(), sizeof(int32_t) * N, cudaMemcpyHostToDevice), "upload");
    ck(cudaMemcpy(vert_off, vert_offsets, sizeof(int32_t) * (N + 1), cudaMemcpyHostToDevice), "upload");
    /* a circle's one local point (radius, 0) becomes radius[b] and the local
     * centre (0, 0) (circleWithRadius, Contact/Circle.hs:24-25) */
    h_radius.assign(N, 0.0);
    bool any_circle = false;
    for (int32_t b = 0; b < N; ++b)
      if (vert_offsets[b + 1] - vert_offsets[b] == 1) {
        h_radius[b] = local_verts_xy[2 * (size_t)vert_offsets[b]];
        any_circle = true;
      }
    std::vector<double> tmp(V);
    for (int32_t v = 0; v < V; ++v) tmp[v] = local_verts_xy[2 * (size_t)v];
    for (int32_t b = 0; b < N; ++b)
      if (h_radius[b] > 0.0) tmp[vert_offsets[b]] = 0.0;
    ck(cudaMemcpy(lx, tmp.data(), sizeof(double) * V, cudaMemcpyHostToDevice), "upload");
    for (int32_t v = 0; v < V; ++v) tmp[v] = local_verts_xy[2 * (size_t)v + 1];
    for (int32_t b = 0; b < N; ++b)
      if (h_radius[b] > 0.0) tmp[vert_offsets[b]] = 0.0;
    ck(cudaMemcpy(ly, tmp.data(), sizeof(double) * V, cudaMemcpyHostToDevice), "upload");
    if (any_circle) {
      radius = dalloc<double>(N, "cudaMalloc");
      ck(cudaMemcpy(radius, h_radius.data(), sizeof(double) * N, cudaMemcpyHostToDevice), "upload");
    }
    for (int k = 0; k < 10; ++k) ck(cudaMemcpy(body[k], bp[k], sizeof(double) * N, cudaMemcpyHostToDevice), "upload bodies");
    /* empty cache: every world offset 0 */
    for (int k = 0; k < 2; ++k) ck(cudaMemset(cwo[k], 0, sizeof(int32_t) * (n_worlds + 1)), "memset");
    cache_buf = 0;
    results_buf = 0;
    have_results = false;
    residual_valid = false;
    setup_grid();
    setup_large_worlds();
    contact_cap = 0;
    item_cap = 0;
    const int32_t pcap = (int32_t)std::min<int64_t>(std::max<int64_t>(1024, 8LL * N), INT32_MAX / 4);
    alloc_step_buffers(pcap, 2 * pcap, 8);
    make_groups(grouped_iterations > 0 ? grouped_iterations : 2);
    Dev d = view(0);
    launch_chained(chain(), shapes::k_init_extents, grid_for(V, 128), 128, 0, stream, d);
    pose(0, 0.0);
    ck(cudaGetLastError(), "launch");
    ck(cudaStreamSynchronize(stream), "create");
  }

  /* Uploads the filled-slot flags (allocated on first use; the step graphs
   * hold the array, so its first allocation re-captures them) and re-poses,
   * which recomputes every body's broadphase flags. */
  void upload_active() {
    bool all = true;
    for (uint8_t a : h_active) all = all && a;
    if (all && !active) return;
    if (!active) {
      if (stream) ck(cudaStreamSynchronize(stream), "sync");
      active = dalloc<uint8_t>(N, "cudaMalloc");
      invalidate_graphs();
    }
    ck(cudaMemcpyAsync(active, h_active.data(), N, cudaMemcpyHostToDevice, stream), "upload");
    pose(0, 0.0);
    ck(cudaStreamSynchronize(stream), "upload");
    have_results = false;
  }

  ~shapes_batch() {
    if (stream) cudaStreamSynchronize(stream);
    drop_graphs();
    free_step_buffers();
    dfree(world_body_off); dfree(body_world); dfree(vert_off); dfree(lx); dfree(ly);
    dfree(emin); dfree(emax);
    for (int k = 0; k < 10; ++k) {
      dfree(body[k]);
      dfree(body_stage[k]);
    }
    dfree(wx); dfree(wy); dfree(nx); dfree(ny); dfree(box); dfree(boxk); dfree(flags); dfree(body_changed);
    dfree(vf); dfree(ef);
    dfree(row_cnt); dfree(row_hits); dfree(row_off); dfree(world_pair_off);
    dfree(grid_T); dfree(grid_base); dfree(grid_inv_s); dfree(grid_lim); dfree(bucket_cnt); dfree(bucket_off);
    dfree(grid_ent); dfree(cell); dfree(row_mode); dfree(large_cnt); dfree(large_ids);
    dfree(ext_chunk); dfree(ext_chunk_off); dfree(ext_part_sum); dfree(ext_part_cnt); dfree(ext_done);
    free_sap();
    free_incremental();
    dfree(radius);
    dfree(metric_part);
    for (int k = 0; k < 2; ++k) dfree(cwo[k]);
    dfree(sched_body); dfree(sched_cur); dfree(world_levels); dfree(group_world_off); dfree(group_worlds);
    dfree(phase_clock);
    dfree(counters);
    dfree(np_cls);
    dfree(export_keys);
    dfree(export_vals);
    dfree(lw_bcnt); dfree(lw_bstart); dfree(lw_bh); dfree(lw_bn); dfree(lw_vel); dfree(lw_color_cnt); dfree(lw_ctl);
    dfree(world_residual);
    dfree(world_depth);
    dfree(learned_mask); dfree(judge_res); dfree(judge_depth);
    dfree(active);
    dfree(ds_feat); dfree(ds_tgt); dfree(ds_count); dfree(snap_ds_count); dfree(snap_mask);
    for (int k = 0; k < 6; ++k) dfree(snap_body[k]);
    dfree(snap_cwo);
    for (cudaEvent_t e : ev_pool) cudaEventDestroy(e);
    if (run_counters) cudaFreeHost(run_counters);
    if (own_stream) cudaStreamDestroy(own_stream);
  }
};

namespace {

bool body_arrays_ok(const shapes_bodies* b) {
  return b && b->vel_x && b->vel_y && b->rot_vel && b->pos_x && b->pos_y && b->rot &&
         b->inv_mass_lin && b->inv_mass_rot && b->mu && b->bounce;
}

double* const* body_ptrs(const shapes_bodies* b, double* out[10]) {
  out[0] = b->vel_x; out[1] = b->vel_y; out[2] = b->rot_vel; out[3] = b->pos_x; out[4] = b->pos_y;
  out[5] = b->rot; out[6] = b->inv_mass_lin; out[7] = b->inv_mass_rot; out[8] = b->mu; out[9] = b->bounce;
  return out;
}

/* Body arrays a step writes: vel_x, vel_y, rot_vel, pos_x, pos_y, rot (the
 * first six of the shapes_bodies order); inverse masses and material stay. */
constexpr int kStepFields = 6;

/* Strictly convex, counter-clockwise, no zero-length edge. */
int check_hull(int nv, const double* xy) {
  if (nv < 3) return SHAPES_E_INVALID_ARG;
  if (nv > shapes::kMaxVerts) return SHAPES_E_UNSUPPORTED;
  for (int k = 0; k < 2 * nv; ++k)
    if (!std::isfinite(xy[k])) return SHAPES_E_NAN;
  for (int k = 0; k < nv; ++k) {
    const int k1 = (k + 1) % nv, k2 = (k + 2) % nv;
    const double ex = xy[2 * k1] - xy[2 * k], ey = xy[2 * k1 + 1] - xy[2 * k + 1];
    const double fx = xy[2 * k2] - xy[2 * k1], fy = xy[2 * k2 + 1] - xy[2 * k1 + 1];
    if (ex == 0.0 && ey == 0.0) return SHAPES_E_INVALID_ARG;
    if (ex * fy - ey * fx <= 0.0) return SHAPES_E_NONCONVEX;
  }
  return SHAPES_OK;
}

/* A circle is one local point (radius, 0) with 0 < radius < 2^500. */
int check_shape(uint8_t kind, int nv, const double* xy) {
  if (kind == SHAPES_SHAPE_HULL) {
    const int rc = check_hull(nv, xy);
    if (rc != SHAPES_OK) g_last_error = "a hull needs 3..64 finite, strictly convex, counter-clockwise vertices";
    return rc;
  }
  g_last_error = "a circle is one local point (radius, 0) with 0 < radius < 2^500";
  if (kind != SHAPES_SHAPE_CIRCLE || nv != 1) {
    if (kind != SHAPES_SHAPE_CIRCLE) g_last_error = "unknown shape kind";
    return SHAPES_E_INVALID_ARG;
  }
  if (!std::isfinite(xy[0]) || !std::isfinite(xy[1])) return SHAPES_E_NAN;
  if (!(xy[0] > 0.0) || xy[0] >= 0x1p500 || xy[1] != 0.0) return SHAPES_E_INVALID_ARG;
  g_last_error.clear();
  return SHAPES_OK;
}

template <typename F>
int guarded(F&& f) {
  try {
    return f();
  } catch (const CudaError&) {
    return SHAPES_E_CUDA;
  } catch (const std::bad_alloc&) {
    g_last_error = "host allocation failed";
    return SHAPES_E_CAPACITY;
  }
}

}  // namespace

extern "C" {

const char* shapes_strerror(int status) {
  switch (status) {
    case SHAPES_OK: return "ok";
    case SHAPES_E_INVALID_ARG: return "invalid argument";
    case SHAPES_E_UNSUPPORTED: return "unsupported shape or option";
    case SHAPES_E_NONCONVEX: return "hull is not strictly convex and counter-clockwise";
    case SHAPES_E_CAPACITY: return "internal buffer could not grow";
    case SHAPES_E_CUDA: return "CUDA error";
    case SHAPES_E_TIMEOUT: return "bounded device wait gave up";
    case SHAPES_E_NAN: return "non-finite body state";
    case SHAPES_E_BUFFER: return "caller buffer too small";
    default: return "unknown status";
  }
}

const char* shapes_last_error_detail(void) { return g_last_error.c_str(); }

int shapes_batch_create(int32_t n_worlds, const int32_t* world_body_offsets, const shapes_bodies* bodies,
                        const int32_t* vert_offsets, const double* local_verts_xy, const uint8_t* shape_kind,
                        shapes_batch** out) {
  g_last_error.clear();
  if (!out || n_worlds < 1 || !world_body_offsets || !vert_offsets || !local_verts_xy || !body_arrays_ok(bodies))
    return SHAPES_E_INVALID_ARG;
  *out = nullptr;
  if (world_body_offsets[0] != 0) return SHAPES_E_INVALID_ARG;
  for (int w = 0; w < n_worlds; ++w) {
    const int32_t n = world_body_offsets[w + 1] - world_body_offsets[w];
    if (n < 0 || n >= (1 << 20)) return SHAPES_E_INVALID_ARG;
  }
  const int32_t N = world_body_offsets[n_worlds];
  if (N < 1) return SHAPES_E_INVALID_ARG;
  if (vert_offsets[0] != 0) return SHAPES_E_INVALID_ARG;
  for (int32_t b = 0; b < N; ++b) {
    const int32_t nv = vert_offsets[b + 1] - vert_offsets[b];
    const int rc = check_shape(shape_kind ? shape_kind[b] : (uint8_t)SHAPES_SHAPE_HULL, nv,
                               local_verts_xy + 2 * (size_t)vert_offsets[b]);
    if (rc != SHAPES_OK) return rc;
  }
  double* bp[10];
  body_ptrs(bodies, bp);
  for (int k = 0; k < 10; ++k)
    for (int32_t b = 0; b < N; ++b)
      if (!std::isfinite(bp[k][b])) return SHAPES_E_NAN;
  return guarded([&]() -> int {
    shapes_batch* h = new shapes_batch();
    try {
      ck(cudaGetDevice(&h->device), "cudaGetDevice");
      ck(cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking), "cudaStreamCreate");
      h->stream = h->own_stream;
      h->W = n_worlds;
      h->h_empties.assign(n_worlds, {});
      h->init_topology(world_body_offsets, bp, vert_offsets, local_verts_xy);
    } catch (...) {
      delete h;
      throw;
    }
    *out = h;
    return SHAPES_OK;
  });
}

int shapes_world_create(int32_t n_bodies, const shapes_bodies* bodies, const int32_t* vert_offsets,
                        const double* local_verts_xy, const uint8_t* shape_kind, shapes_batch** out) {
  const int32_t off[2] = {0, n_bodies};
  return shapes_batch_create(1, off, bodies, vert_offsets, local_verts_xy, shape_kind, out);
}

void shapes_batch_destroy(shapes_batch* b) { delete b; }

static int check_cfg(const shapes_config* c) {
  if (!c) return SHAPES_E_INVALID_ARG;
  if (!std::isfinite(c->dt) || !std::isfinite(c->baumgarte) || !std::isfinite(c->slop) ||
      !std::isfinite(c->accel_x) || !std::isfinite(c->accel_y))
    return SHAPES_E_INVALID_ARG;
  if (c->iterations < 0 || c->iterations > 64) return SHAPES_E_INVALID_ARG;
  if (c->warm_start != SHAPES_WARM_START_OFF && c->warm_start != SHAPES_WARM_START_CACHE)
    return SHAPES_E_UNSUPPORTED;
  if (c->external != SHAPES_EXTERNAL_NONE && c->external != SHAPES_EXTERNAL_CONSTANT_ACCEL)
    return SHAPES_E_UNSUPPORTED;
  if (c->flags & ~(SHAPES_FLAG_RESIDUAL | SHAPES_FLAG_COLOURED | SHAPES_FLAG_LEARNED)) return SHAPES_E_INVALID_ARG;
  return SHAPES_OK;
}

int shapes_batch_step(shapes_batch* b, const shapes_config* cfg, int32_t nsteps) {
  if (!b || nsteps < 0) return SHAPES_E_INVALID_ARG;
  const int rc = check_cfg(cfg);
  if (rc != SHAPES_OK) return rc;
  if (nsteps == 0) return SHAPES_OK;
  return guarded([&]() -> int {
    ck(cudaSetDevice(b->device), "cudaSetDevice");
    const int rc = b->run(*cfg, nsteps, true);
    b->residual_valid = rc == SHAPES_OK && ((cfg->flags & SHAPES_FLAG_RESIDUAL) || b->learned_on(*cfg));
    return rc;
  });
}

int shapes_batches_step(shapes_batch* const* bs, int32_t n, const shapes_config* cfg, int32_t nsteps) {
  if (!bs || n < 1 || nsteps < 0) return SHAPES_E_INVALID_ARG;
  for (int32_t k = 0; k < n; ++k) {
    if (!bs[k]) return SHAPES_E_INVALID_ARG;
    for (int32_t j = 0; j < k; ++j)
      if (bs[j] == bs[k] || bs[j]->stream == bs[k]->stream) return SHAPES_E_INVALID_ARG;
  }
  const int rc0 = check_cfg(cfg);
  if (rc0 != SHAPES_OK) return rc0;
  if (nsteps == 0) return SHAPES_OK;
  return guarded([&]() -> int {
    const AtWork at_work(bs, n);
    /* every handle's steps in flight on its own stream, launched step by
     * step in turn (a stream's launch queue is finite: launching all of one
     * handle's steps first would block until most of them had run), then
     * each finished */
    for (int32_t k = 0; k < n; ++k) {
      ck(cudaSetDevice(bs[k]->device), "cudaSetDevice");
      bs[k]->prepare(*cfg, true);
      bs[k]->run_retries = 0;
      bs[k]->enqueue_begin(true);
    }
    for (int32_t s = 0; s < nsteps; ++s)
      for (int32_t k = 0; k < n; ++k) bs[k]->enqueue_one(*cfg, true);
    for (int32_t k = 0; k < n; ++k) bs[k]->enqueue_end();
    int rc = SHAPES_OK;
    for (int32_t k = 0; k < n; ++k) {
      shapes_batch* b = bs[k];
      int r = b->finish(*cfg, true);
      while (r == shapes_batch::kRunRetry) { /* this handle alone, as shapes_batch_step would */
        b->enqueue(*cfg, nsteps, true);
        r = b->finish(*cfg, true);
      }
      b->residual_valid = r == SHAPES_OK && ((cfg->flags & SHAPES_FLAG_RESIDUAL) || b->learned_on(*cfg));
      if (r != SHAPES_OK && rc == SHAPES_OK) rc = r;
    }
    return rc;
  });
}

int shapes_batches_step_io(shapes_batch* const* bs, int32_t n, const shapes_config* cfg, const shapes_bodies* in,
                           shapes_bodies* out) {
  if (!bs || n < 1 || !in || !out) return SHAPES_E_INVALID_ARG;
  for (int32_t k = 0; k < n; ++k) {
    if (!bs[k] || !body_arrays_ok(&in[k]) || !body_arrays_ok(&out[k])) return SHAPES_E_INVALID_ARG;
    for (int32_t j = 0; j < k; ++j)
      if (bs[j] == bs[k] || bs[j]->stream == bs[k]->stream) return SHAPES_E_INVALID_ARG;
  }
  const int rc0 = check_cfg(cfg);
  if (rc0 != SHAPES_OK) return rc0;
  return guarded([&]() -> int {
    const AtWork at_work(bs, n);
    for (int32_t k = 0; k < n; ++k) {
      shapes_batch* b = bs[k];
      ck(cudaSetDevice(b->device), "cudaSetDevice");
      b->prepare(*cfg, true);
      b->run_retries = 0;
      b->enqueue_begin(true); /* zeroes the counters and keeps the state a refusal returns to */
      b->io_upload(&in[k]);
      b->io_commit();
    }
    for (int32_t k = 0; k < n; ++k) bs[k]->enqueue_one(*cfg, true);
    for (int32_t k = 0; k < n; ++k) {
      bs[k]->io_download(&out[k]);
      bs[k]->enqueue_end();
    }
    int rc = SHAPES_OK;
    for (int32_t k = 0; k < n; ++k) {
      const int r = bs[k]->io_finish(*cfg, &out[k]);
      if (r != SHAPES_OK && rc == SHAPES_OK) rc = r;
    }
    return rc;
  });
}

static bool mapped_host10(double* const host[10], double* dev[10]);

int shapes_batches_run_io(shapes_batch* const* bs, int32_t n, const shapes_config* cfg, int32_t nsteps,
                          shapes_bodies* state, shapes_step_callback on_step, void* user) {
  if (!bs || n < 1 || nsteps < 0 || !state) return SHAPES_E_INVALID_ARG;
  for (int32_t k = 0; k < n; ++k) {
    if (!bs[k] || !body_arrays_ok(&state[k])) return SHAPES_E_INVALID_ARG;
    for (int32_t j = 0; j < k; ++j)
      if (bs[j] == bs[k] || bs[j]->stream == bs[k]->stream) return SHAPES_E_INVALID_ARG;
  }
  const int rc0 = check_cfg(cfg);
  if (rc0 != SHAPES_OK) return rc0;
  std::vector<int> status(n, SHAPES_OK);
  std::vector<std::string> detail(n);
  const AtWork at_work(bs, n);
  /* handle k's loop: its steps in order, one wait per step */
  auto lane = [&](int32_t k) {
    shapes_batch* b = bs[k];
    status[k] = guarded([&]() -> int {
      ck(cudaSetDevice(b->device), "cudaSetDevice");
      double* bp[10];
      body_ptrs(&state[k], bp);
      double* mapped[10];
      const bool is_mapped = mapped_host10(bp, mapped); /* resolved once for the whole run */
      double* const* mp = is_mapped ? mapped : nullptr;
      for (int32_t s = 0; s < nsteps; ++s) {
        b->prepare(*cfg, true);
        b->run_retries = 0;
        b->enqueue_begin(true);
        b->io_upload(&state[k], mp);
        b->io_commit();
        b->enqueue_one(*cfg, true);
        b->io_download(&state[k], mp, kStepFields); /* the other four arrays are the ones just uploaded */
        b->enqueue_end();
        const int r = b->io_finish(*cfg, &state[k], mp, kStepFields);
        if (r != SHAPES_OK) return r;
        if (on_step && on_step(user, k, s) != 0) break;
      }
      return SHAPES_OK;
    });
    detail[k] = g_last_error;
  };
  std::vector<std::thread> threads;
  try {
    for (int32_t k = 1; k < n; ++k) threads.emplace_back(lane, k);
  } catch (const std::system_error&) {
    for (auto& t : threads) t.join();
    g_last_error = "could not start a host thread";
    return SHAPES_E_CAPACITY;
  }
  lane(0);
  for (auto& t : threads) t.join();
  for (int32_t k = 0; k < n; ++k)
    if (status[k] != SHAPES_OK) {
      g_last_error = detail[k];
      return status[k];
    }
  g_last_error.clear();
  return SHAPES_OK;
}

int shapes_batch_collide(shapes_batch* b) {
  if (!b) return SHAPES_E_INVALID_ARG;
  shapes_config cfg{};
  cfg.dt = 1.0;
  return guarded([&]() -> int {
    ck(cudaSetDevice(b->device), "cudaSetDevice");
    return b->run(cfg, 1, false);
  });
}

/* Device addresses of ten caller arrays when every one is pinned host memory
 * mapped into the device address space (then one copy kernel moves them);
 * false for pageable memory, which goes through cudaMemcpyAsync. */
static bool mapped_host10(double* const host[10], double* dev[10]) {
  for (int k = 0; k < 10; ++k) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, host[k]) != cudaSuccess) {
      cudaGetLastError(); /* clear: an unknown pointer is simply not mapped */
      return false;
    }
    if (a.type != cudaMemoryTypeHost || !a.devicePointer) return false;
    dev[k] = static_cast<double*>(a.devicePointer);
  }
  return true;
}

/* True when every one of ten caller arrays is memory that the host reads and
 * writes directly and the driver does not know (not device or managed memory). */
static bool pageable10(double* const host[10]) {
  for (int k = 0; k < 10; ++k) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, host[k]) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    if (a.type != cudaMemoryTypeUnregistered) return false;
  }
  return true;
}

/* Copies n doubles; false when one is not finite. */
static bool copy_finite(double* dst, const double* src, int n) {
  uint64_t bad = 0;
  for (int i = 0; i < n; ++i) {
    uint64_t u;
    std::memcpy(&u, src + i, sizeof u);
    bad |= (u & 0x7ff0000000000000ull) == 0x7ff0000000000000ull;
    std::memcpy(dst + i, &u, sizeof u);
  }
  return !bad;
}

/* Makes a device current while it lives. */
class OnDevice {
 public:
  explicit OnDevice(int device) {
    ck(cudaGetDevice(&before_), "cudaGetDevice");
    if (before_ != device) ck(cudaSetDevice(device), "cudaSetDevice");
  }
  OnDevice(const OnDevice&) = delete;
  ~OnDevice() {
    int now = before_;
    if (cudaGetDevice(&now) == cudaSuccess && now != before_) cudaSetDevice(before_);
  }

 private:
  int before_ = 0;
};

static dim3 copy10_grid(int n, int fields = 10) {
  const int64_t per_block = 256 * shapes::kCopy10PerThread;
  return dim3((unsigned)std::max<int64_t>(1, std::min<int64_t>((n + per_block - 1) / per_block, 1024)),
              (unsigned)fields);
}

int shapes_batch::io_finish(const shapes_config& cfg, shapes_bodies* out, double* const* mapped_out, int fields) {
  ck(cudaStreamSynchronize(stream), "step");
  if (run_counters[shapes::kCntBadInput]) { /* refused: undo the step taken on the old state */
    cache_buf = run_saved_cache_buf;
    restore(run_saved_cap);
    pose(0, 0.0);
    ck(cudaStreamSynchronize(stream), "restore");
    have_results = false;
    return SHAPES_E_NAN;
  }
  int r = finish(cfg, true);
  while (r == kRunRetry) { /* grown and restored: the staged input again, alone */
    enqueue_begin(true);
    io_commit();
    enqueue_one(cfg, true);
    io_download(out, mapped_out, fields);
    enqueue_end();
    r = finish(cfg, true);
  }
  residual_valid = r == SHAPES_OK && ((cfg.flags & SHAPES_FLAG_RESIDUAL) || learned_on(cfg));
  return r;
}

void shapes_batch::io_upload(const shapes_bodies* in, double* const* mapped) {
  double* bp[10];
  body_ptrs(in, bp);
  double* dp[10];
  if (mapped || mapped_host10(bp, dp)) {
    if (mapped) std::copy(mapped, mapped + 10, dp);
    shapes::Ptr10 p{};
    for (int k = 0; k < 10; ++k) {
      p.src[k] = dp[k];
      p.dst[k] = body_stage[k];
    }
    shapes::k_copy10<<<copy10_grid(N), 256, 0, stream>>>(p, N, counters + shapes::kCntBadInput);
  } else {
    for (int k = 0; k < 10; ++k)
      ck(cudaMemcpyAsync(body_stage[k], bp[k], sizeof(double) * N, cudaMemcpyHostToDevice, stream), "upload");
    shapes::k_check_finite<<<grid_for(10LL * N, 256), 256, 0, stream>>>(
        body_stage[0], body_stage[1], body_stage[2], body_stage[3], body_stage[4], body_stage[5], body_stage[6],
        body_stage[7], body_stage[8], body_stage[9], N, counters + shapes::kCntBadInput);
  }
  ck(cudaGetLastError(), "launch");
}

void shapes_batch::io_download(shapes_bodies* out, double* const* mapped, int fields) {
  double* bp[10];
  body_ptrs(out, bp);
  double* dp[10];
  if (mapped || mapped_host10(bp, dp)) {
    if (mapped) std::copy(mapped, mapped + 10, dp);
    shapes::Ptr10 p{};
    for (int k = 0; k < 10; ++k) {
      p.src[k] = body[k];
      p.dst[k] = dp[k];
    }
    shapes::k_copy10<<<copy10_grid(N, fields), 256, 0, stream>>>(p, N, nullptr);
    ck(cudaGetLastError(), "launch");
  } else {
    for (int k = 0; k < fields; ++k)
      ck(cudaMemcpyAsync(bp[k], body[k], sizeof(double) * N, cudaMemcpyDeviceToHost, stream), "download");
  }
}

int shapes_batch_get_bodies(shapes_batch* b, shapes_bodies* out) {
  if (!b || !body_arrays_ok(out)) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    double* bp[10];
    body_ptrs(out, bp);
    double* dp[10];
    if (b->N > 0 && mapped_host10(bp, dp)) {
      shapes::Ptr10 p{};
      for (int k = 0; k < 10; ++k) {
        p.src[k] = b->body[k];
        p.dst[k] = dp[k];
      }
      shapes::k_copy10<<<copy10_grid(b->N), 256, 0, b->stream>>>(p, b->N, nullptr);
      ck(cudaGetLastError(), "launch");
    } else if (b->N > 0 && b->N <= shapes_batch::kStageBodies && pageable10(bp)) {
      const OnDevice on_device(b->device); /* a kernel, unlike a copy, needs its stream's device to be the current one */
      b->pinned_block();
      shapes::Ptr10 p{};
      for (int k = 0; k < 10; ++k) {
        p.src[k] = b->body[k];
        p.dst[k] = b->stage(k);
      }
      shapes::k_copy10<<<copy10_grid(b->N), 256, 0, b->stream>>>(p, b->N, nullptr);
      ck(cudaGetLastError(), "launch");
      ck(cudaStreamSynchronize(b->stream), "download");
      for (int k = 0; k < 10; ++k) std::memcpy(bp[k], b->stage(k), sizeof(double) * b->N);
      return SHAPES_OK;
    } else {
      for (int k = 0; k < 10; ++k)
        ck(cudaMemcpyAsync(bp[k], b->body[k], sizeof(double) * b->N, cudaMemcpyDeviceToHost, b->stream), "download");
    }
    ck(cudaStreamSynchronize(b->stream), "download");
    return SHAPES_OK;
  });
}

int shapes_batch_set_bodies(shapes_batch* b, const shapes_bodies* in) {
  if (!b || !body_arrays_ok(in)) return SHAPES_E_INVALID_ARG;
  double* bp[10];
  body_ptrs(in, bp);
  return guarded([&]() -> int {
    /* only bodies whose position, rotation or inverse masses changed get a
     * new pose: every other body's pose is already that of the state written
     * back (the live pose always follows the live state).  Copied, not
     * swapped: the live arrays keep their addresses, which the captured step
     * graphs hold. */
    auto commit = [&](shapes::Ptr10& p) -> int {
      for (int k = 0; k < 10; ++k) p.dst[k] = b->body[k];
      shapes::k_commit_bodies<<<grid_for(b->N, 256), 256, 0, b->stream>>>(p, b->N, b->body_changed);
      Dev d = b->view(0);
      launch_pose(true, b->stream, b->N, d, 0.0, 0, b->body_changed);
      ck(cudaGetLastError(), "launch");
      ck(cudaStreamSynchronize(b->stream), "upload");
      b->have_results = false;
      return SHAPES_OK;
    };
    if (b->N > 0 && b->N <= shapes_batch::kStageBodies && pageable10(bp)) {
      b->pinned_block();
      ck(cudaStreamSynchronize(b->stream), "sync");
      shapes::Ptr10 p{};
      for (int k = 0; k < 10; ++k) {
        if (!copy_finite(b->stage(k), bp[k], b->N)) return SHAPES_E_NAN; /* live state untouched */
        p.src[k] = b->stage(k);
      }
      return commit(p);
    }
    ck(cudaMemsetAsync(b->counters + shapes::kCntBadInput, 0, sizeof(unsigned long long), b->stream), "memset");
    double* dp[10];
    if (mapped_host10(bp, dp)) { /* copy and check in one pass over NVLink-C2C / PCIe */
      shapes::Ptr10 p{};
      for (int k = 0; k < 10; ++k) {
        p.src[k] = dp[k];
        p.dst[k] = b->body_stage[k];
      }
      shapes::k_copy10<<<copy10_grid(b->N), 256, 0, b->stream>>>(p, b->N, b->counters + shapes::kCntBadInput);
    } else {
      for (int k = 0; k < 10; ++k)
        ck(cudaMemcpyAsync(b->body_stage[k], bp[k], sizeof(double) * b->N, cudaMemcpyHostToDevice, b->stream),
           "upload");
      shapes::k_check_finite<<<grid_for(10LL * b->N, 256), 256, 0, b->stream>>>(
          b->body_stage[0], b->body_stage[1], b->body_stage[2], b->body_stage[3], b->body_stage[4],
          b->body_stage[5], b->body_stage[6], b->body_stage[7], b->body_stage[8], b->body_stage[9], b->N,
          b->counters + shapes::kCntBadInput);
    }
    ck(cudaGetLastError(), "launch");
    unsigned long long bad = 0;
    ck(cudaMemcpyAsync(&bad, b->counters + shapes::kCntBadInput, sizeof(bad), cudaMemcpyDeviceToHost, b->stream), "download");
    ck(cudaStreamSynchronize(b->stream), "validate");
    if (bad) return SHAPES_E_NAN; /* live state untouched */
    shapes::Ptr10 p{};
    for (int k = 0; k < 10; ++k) p.src[k] = b->body_stage[k];
    return commit(p);
  });
}

int shapes_batch_num_worlds(shapes_batch* b, int32_t* out) {
  if (!b || !out) return SHAPES_E_INVALID_ARG;
  *out = b->W;
  return SHAPES_OK;
}

int shapes_batch_num_bodies(shapes_batch* b, int64_t* out) {
  if (!b || !out) return SHAPES_E_INVALID_ARG;
  *out = b->N;
  return SHAPES_OK;
}

int shapes_batch_num_vertices(shapes_batch* b, int64_t* out) {
  if (!b || !out) return SHAPES_E_INVALID_ARG;
  *out = b->V;
  return SHAPES_OK;
}

int shapes_batch_get_shapes(shapes_batch* b, double* world_xy, double* normal_xy) {
  if (!b || !world_xy || !normal_xy) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    std::vector<double> x(b->V), y(b->V), nx(b->V), ny(b->V);
    ck(cudaMemcpyAsync(x.data(), b->wx, sizeof(double) * b->V, cudaMemcpyDeviceToHost, b->stream), "download");
    ck(cudaMemcpyAsync(y.data(), b->wy, sizeof(double) * b->V, cudaMemcpyDeviceToHost, b->stream), "download");
    ck(cudaMemcpyAsync(nx.data(), b->nx, sizeof(double) * b->V, cudaMemcpyDeviceToHost, b->stream), "download");
    ck(cudaMemcpyAsync(ny.data(), b->ny, sizeof(double) * b->V, cudaMemcpyDeviceToHost, b->stream), "download");
    ck(cudaStreamSynchronize(b->stream), "download");
    for (int32_t v = 0; v < b->V; ++v) {
      world_xy[2 * (size_t)v] = x[v];
      world_xy[2 * (size_t)v + 1] = y[v];
      normal_xy[2 * (size_t)v] = nx[v];
      normal_xy[2 * (size_t)v + 1] = ny[v];
    }
    return SHAPES_OK;
  });
}

int shapes_batch_num_pairs(shapes_batch* b, int64_t* out) {
  if (!b || !out) return SHAPES_E_INVALID_ARG;
  *out = b->have_results ? b->stats.pairs : 0;
  return SHAPES_OK;
}

static void world_counts_from(shapes_batch* b, const int32_t* dev_off, int32_t* counts) {
  std::vector<int32_t> off(b->W + 1);
  ck(cudaMemcpyAsync(off.data(), dev_off, sizeof(int32_t) * (b->W + 1), cudaMemcpyDeviceToHost, b->stream), "download");
  ck(cudaStreamSynchronize(b->stream), "download");
  for (int w = 0; w < b->W; ++w) counts[w] = off[w + 1] - off[w];
}

int shapes_batch_get_pairs(shapes_batch* b, int32_t* ij, int64_t capacity, int32_t* world_counts) {
  if (!b || (!ij && capacity > 0)) return SHAPES_E_INVALID_ARG;
  const int64_t P = b->have_results ? b->stats.pairs : 0;
  if (capacity < P) return SHAPES_E_BUFFER;
  return guarded([&]() -> int {
    std::vector<int32_t> pa(P), pb(P);
    if (P > 0) {
      ck(cudaMemcpyAsync(pa.data(), b->pair_a, sizeof(int32_t) * P, cudaMemcpyDeviceToHost, b->stream), "download");
      ck(cudaMemcpyAsync(pb.data(), b->pair_b, sizeof(int32_t) * P, cudaMemcpyDeviceToHost, b->stream), "download");
      ck(cudaStreamSynchronize(b->stream), "download");
    }
    for (int64_t p = 0; p < P; ++p) {
      const int32_t off = b->h_world_body_off[b->h_body_world[pa[p]]];
      ij[2 * p] = pa[p] - off;
      ij[2 * p + 1] = pb[p] - off;
    }
    if (world_counts) {
      if (b->have_results) world_counts_from(b, b->world_pair_off, world_counts);
      else std::fill(world_counts, world_counts + b->W, 0);
    }
    return SHAPES_OK;
  });
}

int shapes_batch_num_contacts(shapes_batch* b, int64_t* out) {
  if (!b || !out) return SHAPES_E_INVALID_ARG;
  *out = b->have_results ? b->stats.contacts : 0;
  return SHAPES_OK;
}

static void decode_key(uint64_t k, int32_t* out4) {
  out4[0] = (int32_t)(k >> 44);
  out4[1] = (int32_t)((k >> 24) & 0xfffff);
  out4[2] = (int32_t)((k >> 12) & 0xfff);
  out4[3] = (int32_t)(k & 0xfff);
}

int shapes_batch_get_contacts(shapes_batch* b, int32_t* keys5, double* vals5, int64_t capacity,
                              int32_t* world_counts) {
  if (!b || ((!keys5 || !vals5) && capacity > 0)) return SHAPES_E_INVALID_ARG;
  const int64_t C = b->have_results ? b->stats.contacts : 0;
  if (capacity < C) return SHAPES_E_BUFFER;
  return guarded([&]() -> int {
    if (C > 0) {
      /* decoded on the device; straight into the caller's arrays when both
       * are mapped pinned host memory, else through a device staging area */
      cudaPointerAttributes ak{}, av{};
      const bool mk = cudaPointerGetAttributes(&ak, keys5) == cudaSuccess && ak.type == cudaMemoryTypeHost &&
                      ak.devicePointer;
      const bool mv = cudaPointerGetAttributes(&av, vals5) == cudaSuccess && av.type == cudaMemoryTypeHost &&
                      av.devicePointer;
      cudaGetLastError();
      const int grid = (int)std::min<int64_t>((C + 255) / 256, 4096);
      if (mk && mv) {
        shapes::k_export_contacts<<<grid, 256, 0, b->stream>>>(
            b->c_key[b->results_buf], b->c_flip, b->c_val, (int)C, static_cast<int32_t*>(ak.devicePointer),
            static_cast<double*>(av.devicePointer));
        ck(cudaGetLastError(), "launch");
      } else {
        if (b->export_cap < C) {
          dfree(b->export_keys);
          dfree(b->export_vals);
          b->export_keys = nullptr;
          b->export_vals = nullptr;
          b->export_keys = dalloc<int32_t>(5 * (size_t)C, "cudaMalloc export");
          b->export_vals = dalloc<double>(5 * (size_t)C, "cudaMalloc export");
          b->export_cap = C;
        }
        shapes::k_export_contacts<<<grid, 256, 0, b->stream>>>(b->c_key[b->results_buf], b->c_flip, b->c_val,
                                                              (int)C, b->export_keys, b->export_vals);
        ck(cudaGetLastError(), "launch");
        ck(cudaMemcpyAsync(keys5, b->export_keys, sizeof(int32_t) * 5 * C, cudaMemcpyDeviceToHost, b->stream),
           "download");
        ck(cudaMemcpyAsync(vals5, b->export_vals, sizeof(double) * 5 * C, cudaMemcpyDeviceToHost, b->stream),
           "download");
      }
      ck(cudaStreamSynchronize(b->stream), "download");
    }
    if (world_counts) {
      if (b->have_results) world_counts_from(b, b->cwo[b->results_buf], world_counts);
      else std::fill(world_counts, world_counts + b->W, 0);
    }
    return SHAPES_OK;
  });
}

int shapes_batch_num_cache(shapes_batch* b, int64_t* out) {
  if (!b || !out) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    int32_t total = 0;
    ck(cudaMemcpyAsync(&total, b->cwo[b->cache_buf] + b->W, sizeof(int32_t), cudaMemcpyDeviceToHost, b->stream), "download");
    ck(cudaStreamSynchronize(b->stream), "download");
    *out = total;
    return SHAPES_OK;
  });
}

int shapes_batch_get_cache(shapes_batch* b, int32_t* keys4, double* lam2, int64_t capacity, int32_t* world_counts) {
  if (!b) return SHAPES_E_INVALID_ARG;
  int64_t n = 0;
  int rc = shapes_batch_num_cache(b, &n);
  if (rc != SHAPES_OK) return rc;
  if (capacity < n) return SHAPES_E_BUFFER;
  if (n > 0 && (!keys4 || !lam2)) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    std::vector<uint64_t> key(n);
    if (n > 0) {
      ck(cudaMemcpyAsync(key.data(), b->c_key[b->cache_buf], sizeof(uint64_t) * n, cudaMemcpyDeviceToHost, b->stream), "download");
      ck(cudaMemcpyAsync(lam2, b->lam[b->cache_buf], sizeof(double) * 2 * n, cudaMemcpyDeviceToHost, b->stream), "download");
      ck(cudaStreamSynchronize(b->stream), "download");
    }
    for (int64_t c = 0; c < n; ++c) decode_key(key[c], keys4 + 4 * c);
    if (world_counts) world_counts_from(b, b->cwo[b->cache_buf], world_counts);
    return SHAPES_OK;
  });
}

int shapes_batch_set_cache(shapes_batch* b, const int32_t* world_counts, const int32_t* keys4, const double* lam2) {
  if (!b || !world_counts) return SHAPES_E_INVALID_ARG;
  std::vector<int32_t> off(b->W + 1, 0);
  for (int w = 0; w < b->W; ++w) {
    if (world_counts[w] < 0) return SHAPES_E_INVALID_ARG;
    off[w + 1] = off[w] + world_counts[w];
  }
  const int64_t n = off[b->W];
  if (n > 0 && (!keys4 || !lam2)) return SHAPES_E_INVALID_ARG;
  std::vector<uint64_t> key(n);
  for (int w = 0; w < b->W; ++w) {
    const int32_t nw = b->h_world_body_off[w + 1] - b->h_world_body_off[w];
    for (int32_t c = off[w]; c < off[w + 1]; ++c) {
      const int32_t* k = keys4 + 4 * (size_t)c;
      if (k[0] < 0 || k[0] >= nw || k[1] < 0 || k[1] >= nw || k[2] < 0 || k[2] >= 4096 || k[3] < 0 || k[3] >= 4096)
        return SHAPES_E_INVALID_ARG;
      key[c] = ((uint64_t)k[0] << 44) | ((uint64_t)k[1] << 24) | ((uint64_t)k[2] << 12) | (uint64_t)k[3];
      if (c > off[w] && !(key[c] < key[c - 1])) return SHAPES_E_INVALID_ARG;
    }
  }
  return guarded([&]() -> int {
    if (n > b->contact_cap) {
      const int64_t nc = std::max<int64_t>(n, 2LL * b->contact_cap);
      if (nc > INT32_MAX / 2) return SHAPES_E_CAPACITY;
      b->alloc_step_buffers(std::max<int32_t>(b->pair_cap, (int32_t)(nc / 2)), (int32_t)nc, 8);
    }
    if (n > 0) {
      ck(cudaMemcpyAsync(b->c_key[b->cache_buf], key.data(), sizeof(uint64_t) * n, cudaMemcpyHostToDevice, b->stream), "upload");
      ck(cudaMemcpyAsync(b->lam[b->cache_buf], lam2, sizeof(double) * 2 * n, cudaMemcpyHostToDevice, b->stream), "upload");
    }
    ck(cudaMemcpyAsync(b->cwo[b->cache_buf], off.data(), sizeof(int32_t) * (b->W + 1), cudaMemcpyHostToDevice, b->stream), "upload");
    ck(cudaStreamSynchronize(b->stream), "upload");
    return SHAPES_OK;
  });
}

int shapes_batch_get_world_metrics(shapes_batch* b, double* residual, double* max_depth) {
  if (!b) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    if (residual) {
      if (b->residual_valid)
        ck(cudaMemcpy(residual, b->world_residual, sizeof(double) * b->W, cudaMemcpyDeviceToHost), "download");
      else
        std::fill(residual, residual + b->W, std::nan(""));
    }
    if (max_depth) {
      shapes_config cfg{};
      cfg.dt = 1.0;
      const shapes_stats keep = b->stats; /* the counters stay those of the last step call */
      const int rc = b->run(cfg, 1, false);
      b->stats = keep;
      if (rc != SHAPES_OK) return rc;
      Dev d = b->view(b->results_buf);
      b->world_metric_kernels(d, false);
      ck(cudaGetLastError(), "launch");
      ck(cudaMemcpyAsync(max_depth, b->world_depth, sizeof(double) * b->W, cudaMemcpyDeviceToHost, b->stream), "download");
      ck(cudaStreamSynchronize(b->stream), "download");
    }
    return SHAPES_OK;
  });
}

int shapes_batch_get_stats(shapes_batch* b, shapes_stats* out) {
  if (!b || !out) return SHAPES_E_INVALID_ARG;
  *out = b->stats;
  return SHAPES_OK;
}

int shapes_batch_autotune(shapes_batch* b, const shapes_config* cfg, int32_t steps_per_trial,
                          int32_t* chosen_worlds_per_group, int32_t* chosen_threads) {
  if (!b || steps_per_trial < 1) return SHAPES_E_INVALID_ARG;
  const int rc0 = check_cfg(cfg);
  if (rc0 != SHAPES_OK) return rc0;
  return guarded([&]() -> int {
    const int N = b->N, W = b->W;
    /* save the state the trials start from */
    int32_t n_cache = 0;
    ck(cudaMemcpyAsync(&n_cache, b->cwo[b->cache_buf] + W, sizeof(int32_t), cudaMemcpyDeviceToHost, b->stream), "download");
    ck(cudaStreamSynchronize(b->stream), "sync");
    std::vector<void*> saved;
    auto keep = [&](const void* src, size_t bytes) {
      void* p = nullptr;
      ck(cudaMalloc(&p, std::max<size_t>(bytes, 1)), "cudaMalloc autotune");
      saved.push_back(p);
      ck(cudaMemcpyAsync(p, src, bytes, cudaMemcpyDeviceToDevice, b->stream), "copy");
      return p;
    };
    const int cache_buf0 = b->cache_buf;
    void* sb[6];
    for (int k = 0; k < 6; ++k) sb[k] = keep(b->body[k], sizeof(double) * N);
    void* skey = keep(b->c_key[cache_buf0], sizeof(uint64_t) * n_cache);
    void* slam = keep(b->lam[cache_buf0], sizeof(double) * 2 * n_cache);
    void* scwo = keep(b->cwo[cache_buf0], sizeof(int32_t) * (W + 1));
    const int32_t wpg0 = b->worlds_per_group_override, thr0 = b->solve_threads, tgt0 = b->target_group_bodies;
    const int32_t gw0 = b->group_warps;
    const bool auto0 = b->group_warps_auto, spread0 = b->spread_heavy;
    const std::vector<int32_t> order0 = b->world_order;
    const bool prof0 = b->profiling;
    b->profiling = false;
    auto restore_state = [&]() {
      b->cache_buf = cache_buf0;
      for (int k = 0; k < 6; ++k)
        ck(cudaMemcpyAsync(b->body[k], sb[k], sizeof(double) * N, cudaMemcpyDeviceToDevice, b->stream), "copy");
      if (n_cache > b->contact_cap) throw CudaError{cudaErrorMemoryAllocation};
      ck(cudaMemcpyAsync(b->c_key[cache_buf0], skey, sizeof(uint64_t) * n_cache, cudaMemcpyDeviceToDevice, b->stream), "copy");
      ck(cudaMemcpyAsync(b->lam[cache_buf0], slam, sizeof(double) * 2 * n_cache, cudaMemcpyDeviceToDevice, b->stream), "copy");
      ck(cudaMemcpyAsync(b->cwo[cache_buf0], scwo, sizeof(int32_t) * (W + 1), cudaMemcpyDeviceToDevice, b->stream), "copy");
      b->pose(0, 0.0);
    };
    const int base = std::max(1, std::min(shapes::kMaxGroupWorlds, 32 / (cfg->iterations + 1)));
    /* The level-ordered packing: worlds sorted by the dependency levels of
     * one step from the saved state (deepest first, then by size), so that a
     * group's worlds end their levels together. */
    restore_state();
    b->world_order.clear();
    b->make_groups(cfg->iterations);
    const int rc0 = b->run(*cfg, 1, true);
    std::vector<int32_t> lv(W, 0), by_levels(W);
    if (rc0 == SHAPES_OK)
      ck(cudaMemcpy(lv.data(), b->world_levels, sizeof(int32_t) * W, cudaMemcpyDeviceToHost), "download");
    for (int w = 0; w < W; ++w) by_levels[w] = w;
    std::stable_sort(by_levels.begin(), by_levels.end(), [&](int a, int c) {
      if (lv[a] != lv[c]) return lv[a] > lv[c];
      return (b->h_world_body_off[a + 1] - b->h_world_body_off[a]) > (b->h_world_body_off[c + 1] - b->h_world_body_off[c]);
    });
    /* (worlds per group, warps per group, level order, heavy groups spread,
     * target bodies per group: when non-zero, groups close at that many bodies
     * instead of at a world count, so the largest worlds of a ragged batch get
     * groups of their own); ahead of them the packing that was set, kCurrent,
     * and the automatic one, spelled out so that it can be read back and given
     * to another handle */
    constexpr int kCurrent = -1;
    std::vector<std::array<int, 5>> cands;
    const bool was_auto = b->worlds_per_group_override <= 0 && b->target_group_bodies <= 0;
    if (!was_auto || !b->group_warps_auto || b->spread_heavy || !order0.empty()) cands.push_back({kCurrent, 0, 0, 0, 0});
    {
      b->worlds_per_group_override = b->target_group_bodies = 0;
      b->group_warps_auto = true;
      b->make_groups(cfg->iterations);
      cands.push_back({1, b->solve_shape().warps, 0, 0, b->auto_group_target()});
    }
    auto add = [&](int wpg, int gw, int lo, int spread = 0, int target = 0) {
      const std::array<int, 5> c{wpg, gw, lo, spread, target};
      if (wpg >= 1 && wpg <= shapes::kMaxGroupWorlds && std::find(cands.begin(), cands.end(), c) == cands.end())
        cands.push_back(c);
    };
    for (int lo : {0, 1})
      for (int wpg : {1, 2, base, base + 1, 2 * base, 3 * base, 4 * base})
        for (int gw : {1, 2, 4, 8}) {
          add(std::min(wpg, W), gw, lo);
          if (gw > 1) add(std::min(wpg, W), gw, lo, 1);
        }
    int32_t min_n = INT32_MAX, max_n = 0;
    for (int w = 0; w < W; ++w) {
      const int32_t n = b->h_world_body_off[w + 1] - b->h_world_body_off[w];
      if (n >= b->large_world_bodies) continue;
      min_n = std::min(min_n, n);
      max_n = std::max(max_n, n);
    }
    if (max_n > 2 * min_n) /* ragged batches: packings by body count */
      for (int target : {256, 512, 1024, 2048})
        for (int gw : {2, 4, 8}) add(1, gw, 0, 1, target);
    cudaEvent_t e0, e1;
    ck(cudaEventCreate(&e0), "event");
    ck(cudaEventCreate(&e1), "event");
    float best = 1e30f;
    std::array<int, 5> best_c{kCurrent, 0, 0, 0, 0};
    auto apply = [&](const std::array<int, 5>& c) {
      if (c[0] == kCurrent) {
        b->worlds_per_group_override = wpg0;
        b->target_group_bodies = tgt0;
        b->solve_threads = thr0;
        b->group_warps = gw0;
        b->group_warps_auto = auto0;
        b->spread_heavy = spread0;
        b->world_order = order0;
        return;
      }
      b->worlds_per_group_override = c[4] ? 0 : c[0];
      b->target_group_bodies = c[4];
      b->solve_threads = 32 * c[1];
      b->group_warps = c[1];
      b->group_warps_auto = false;
      b->spread_heavy = c[3] != 0;
      if (c[2]) b->world_order = by_levels; else b->world_order.clear();
    };
    int rc = rc0;
    if (rc0 != SHAPES_OK) cands.clear();
    for (const auto& c : cands) {
      restore_state();
      apply(c);
      b->invalidate_graphs();
      b->make_groups(cfg->iterations);
      rc = b->run(*cfg, 1, true); /* untimed: captures this packing's step graphs */
      if (rc != SHAPES_OK) break;
      ck(cudaEventRecord(e0, b->stream), "event");
      rc = b->run(*cfg, steps_per_trial, true);
      if (rc != SHAPES_OK) break;
      ck(cudaEventRecord(e1, b->stream), "event");
      ck(cudaEventSynchronize(e1), "event");
      float ms = 0.f;
      ck(cudaEventElapsedTime(&ms, e0, e1), "event");
      if (ms < best) {
        best = ms;
        best_c = c;
      }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    restore_state();
    apply(rc == SHAPES_OK ? best_c : std::array<int, 5>{kCurrent, 0, 0, 0, 0});
    b->invalidate_graphs();
    b->make_groups(cfg->iterations);
    ck(cudaStreamSynchronize(b->stream), "sync");
    for (void* p : saved) cudaFree(p);
    b->profiling = prof0;
    b->have_results = false;
    if (chosen_worlds_per_group) *chosen_worlds_per_group = b->worlds_per_group_override;
    if (chosen_threads) *chosen_threads = b->solve_threads;
    return rc;
  });
}

/* ---- world mutation (World.append / World.delete) ------------------------ */

int shapes_batch_delete_body(shapes_batch* b, int32_t world, int32_t slot) {
  if (!b || world < 0 || world >= b->W) return SHAPES_E_INVALID_ARG;
  const int32_t n = b->h_world_body_off[world + 1] - b->h_world_body_off[world];
  if (slot < 0 || slot >= n) return SHAPES_E_INVALID_ARG;
  const int32_t g = b->h_world_body_off[world] + slot;
  if (!b->h_active[g]) return SHAPES_E_INVALID_ARG; /* safeDelete: the slot must be filled */
  return guarded([&]() -> int {
    b->h_active[g] = 0;
    b->h_empties[world].push_back(slot);
    b->upload_active();
    return SHAPES_OK;
  });
}

int shapes_batch_append_body(shapes_batch* b, int32_t world, const double* body10, int32_t n_verts,
                             const double* local_verts_xy, int32_t* slot_out) {
  if (!b || !body10 || !local_verts_xy || !slot_out || world < 0 || world >= b->W) return SHAPES_E_INVALID_ARG;
  for (int k = 0; k < 10; ++k)
    if (!std::isfinite(body10[k])) return SHAPES_E_NAN;
  const int hrc = check_shape(n_verts == 1 ? SHAPES_SHAPE_CIRCLE : SHAPES_SHAPE_HULL, n_verts, local_verts_xy);
  if (hrc != SHAPES_OK) return hrc;
  return guarded([&]() -> int {
    const int32_t W = b->W, N = b->N;
    const int32_t w0 = b->h_world_body_off[world];
    auto& empties = b->h_empties[world];
    const bool reuse = !empties.empty();
    const int32_t slot = reuse ? empties.back() : b->h_world_body_off[world + 1] - w0;
    if (slot >= (1 << 20)) return SHAPES_E_CAPACITY;
    if (reuse) {
      const int32_t g = w0 + slot;
      const int32_t v0 = b->h_vert_off[g];
      if (b->h_vert_off[g + 1] - v0 == n_verts) { /* same vertex count: in place */
        ck(cudaStreamSynchronize(b->stream), "sync");
        for (int k = 0; k < 10; ++k)
          ck(cudaMemcpyAsync(b->body[k] + g, body10 + k, sizeof(double), cudaMemcpyHostToDevice, b->stream), "upload");
        std::vector<double> xs(n_verts), ys(n_verts);
        for (int32_t v = 0; v < n_verts; ++v) {
          xs[v] = local_verts_xy[2 * v];
          ys[v] = local_verts_xy[2 * v + 1];
        }
        if (n_verts == 1) { /* a circle into a circle's slot */
          b->h_radius[g] = xs[0];
          xs[0] = ys[0] = 0.0;
          ck(cudaMemcpyAsync(b->radius + g, &b->h_radius[g], sizeof(double), cudaMemcpyHostToDevice, b->stream),
             "upload");
        }
        ck(cudaMemcpyAsync(b->lx + v0, xs.data(), sizeof(double) * n_verts, cudaMemcpyHostToDevice, b->stream), "upload");
        ck(cudaMemcpyAsync(b->ly + v0, ys.data(), sizeof(double) * n_verts, cudaMemcpyHostToDevice, b->stream), "upload");
        Dev d = b->view(0);
        launch_chained(true, shapes::k_init_extents, grid_for(b->V, 128), 128, 0, b->stream, d);
        ck(cudaGetLastError(), "launch");
        empties.pop_back();
        b->h_active[g] = 1;
        b->upload_active();
        if (!b->active) { /* every slot filled again: the in-place shape still needs its pose */
          b->pose(0, 0.0);
          ck(cudaStreamSynchronize(b->stream), "upload");
        }
        *slot_out = slot;
        return SHAPES_OK;
      }
    }
    /* the topology changes: rebuild from the host copies, keeping state and cache */
    std::vector<double> body(10 * (size_t)N);
    shapes_bodies cur{};
    double* bp[10];
    for (int k = 0; k < 10; ++k) bp[k] = body.data() + (size_t)k * N;
    cur.vel_x = bp[0]; cur.vel_y = bp[1]; cur.rot_vel = bp[2]; cur.pos_x = bp[3]; cur.pos_y = bp[4];
    cur.rot = bp[5]; cur.inv_mass_lin = bp[6]; cur.inv_mass_rot = bp[7]; cur.mu = bp[8]; cur.bounce = bp[9];
    int rc = shapes_batch_get_bodies(b, &cur);
    if (rc != SHAPES_OK) return rc;
    int64_t nc = 0;
    rc = shapes_batch_num_cache(b, &nc);
    if (rc != SHAPES_OK) return rc;
    std::vector<int32_t> keys(4 * (size_t)std::max<int64_t>(nc, 1)), wc(W);
    std::vector<double> lam(2 * (size_t)std::max<int64_t>(nc, 1));
    rc = shapes_batch_get_cache(b, keys.data(), lam.data(), nc, wc.data());
    if (rc != SHAPES_OK) return rc;
    const int64_t V = b->V;
    const std::vector<double> xyh = b->local_xy_host();
    const int32_t g = w0 + slot; /* replaced or inserted body */
    const int32_t N2 = reuse ? N : N + 1;
    std::vector<int32_t> off(W + 1);
    for (int w = 0; w <= W; ++w) off[w] = b->h_world_body_off[w] + ((!reuse && w > world) ? 1 : 0);
    std::vector<double> body2(10 * (size_t)N2);
    std::vector<uint8_t> act2(N2);
    std::vector<int32_t> vo2(N2 + 1, 0);
    std::vector<double> xy2;
    xy2.reserve(2 * (size_t)(V + n_verts));
    for (int32_t i = 0; i < N2; ++i) {
      const bool is_new = i == g;
      const int32_t src = (!reuse && i > g) ? i - 1 : i; /* old index */
      for (int k = 0; k < 10; ++k) body2[(size_t)k * N2 + i] = is_new ? body10[k] : body[(size_t)k * N + src];
      act2[i] = is_new ? 1 : b->h_active[src];
      if (is_new) {
        for (int32_t v = 0; v < 2 * n_verts; ++v) xy2.push_back(local_verts_xy[v]);
        vo2[i + 1] = vo2[i] + n_verts;
      } else {
        for (int32_t v = b->h_vert_off[src]; v < b->h_vert_off[src + 1]; ++v) {
          xy2.push_back(xyh[2 * (size_t)v]);
          xy2.push_back(xyh[2 * (size_t)v + 1]);
        }
        vo2[i + 1] = vo2[i] + (b->h_vert_off[src + 1] - b->h_vert_off[src]);
      }
    }
    double* bp2[10];
    for (int k = 0; k < 10; ++k) bp2[k] = body2.data() + (size_t)k * N2;
    b->init_topology(off.data(), bp2, vo2.data(), xy2.data());
    if (reuse) empties.pop_back();
    b->h_active = act2;
    b->upload_active();
    rc = shapes_batch_set_cache(b, wc.data(), keys.data(), lam.data());
    if (rc != SHAPES_OK) return rc;
    *slot_out = slot;
    return SHAPES_OK;
  });
}

int shapes_batch_get_active(shapes_batch* b, uint8_t* out) {
  if (!b || !out) return SHAPES_E_INVALID_ARG;
  std::copy(b->h_active.begin(), b->h_active.end(), out);
  return SHAPES_OK;
}

/* ---- checkpoint file (EngineState: World + EngineCache) ------------------ */

}  // extern "C"

namespace {

constexpr char kCkMagic[8] = {'S', 'H', 'A', 'P', 'E', 'S', 'C', 'K'};
constexpr uint32_t kCkVersion = 1;
constexpr uint32_t kCkEndian = 0x01020304u;

uint64_t fnv1a(const unsigned char* p, size_t n, uint64_t h = 0xcbf29ce484222325ull) {
  for (size_t k = 0; k < n; ++k) {
    h ^= p[k];
    h *= 0x100000001b3ull;
  }
  return h;
}

struct CkWriter {
  std::vector<unsigned char> buf;
  template <class T>
  void put(const T* p, size_t n) {
    const unsigned char* c = reinterpret_cast<const unsigned char*>(p);
    buf.insert(buf.end(), c, c + sizeof(T) * n);
  }
  template <class T>
  void put1(T v) { put(&v, 1); }
};

struct CkReader {
  const std::vector<unsigned char>& buf;
  size_t at = 0;
  bool ok = true;
  template <class T>
  void get(T* p, size_t n) {
    const size_t bytes = sizeof(T) * n;
    if (!ok || buf.size() - at < bytes) {
      ok = false;
      return;
    }
    std::memcpy(p, buf.data() + at, bytes);
    at += bytes;
  }
  template <class T>
  T get1() {
    T v{};
    get(&v, 1);
    return v;
  }
};

}  // namespace

extern "C" {

int shapes_batch_save(shapes_batch* b, const char* path) {
  if (!b || !path) return SHAPES_E_INVALID_ARG;
  const int32_t W = b->W, N = b->N;
  const int64_t V = b->V;
  std::vector<double> body(10 * (size_t)N);
  shapes_bodies out{};
  double* bp[10];
  for (int k = 0; k < 10; ++k) bp[k] = body.data() + (size_t)k * N;
  out.vel_x = bp[0]; out.vel_y = bp[1]; out.rot_vel = bp[2]; out.pos_x = bp[3]; out.pos_y = bp[4];
  out.rot = bp[5]; out.inv_mass_lin = bp[6]; out.inv_mass_rot = bp[7]; out.mu = bp[8]; out.bounce = bp[9];
  int rc = shapes_batch_get_bodies(b, &out);
  if (rc != SHAPES_OK) return rc;
  int64_t nc = 0;
  rc = shapes_batch_num_cache(b, &nc);
  if (rc != SHAPES_OK) return rc;
  std::vector<int32_t> keys(4 * (size_t)std::max<int64_t>(nc, 1)), wc(W);
  std::vector<double> lam(2 * (size_t)std::max<int64_t>(nc, 1));
  rc = shapes_batch_get_cache(b, keys.data(), lam.data(), nc, wc.data());
  if (rc != SHAPES_OK) return rc;
  const std::vector<int32_t>& vo = b->h_vert_off;
  std::vector<double> xy;
  rc = guarded([&]() -> int {
    xy = b->local_xy_host();
    return SHAPES_OK;
  });
  if (rc != SHAPES_OK) return rc;
  CkWriter w;
  w.put(kCkMagic, 8);
  w.put1(kCkVersion);
  w.put1(kCkEndian);
  w.put1(W);
  w.put1(N);
  w.put1(V);
  w.put1(nc);
  w.put(b->h_world_body_off.data(), (size_t)W + 1);
  w.put(vo.data(), (size_t)N + 1);
  w.put(xy.data(), 2 * (size_t)V);
  w.put(body.data(), body.size());
  w.put(wc.data(), (size_t)W);
  w.put(keys.data(), 4 * (size_t)nc);
  w.put(lam.data(), 2 * (size_t)nc);
  w.put(b->h_active.data(), (size_t)N);
  for (int32_t k = 0; k < W; ++k) w.put1((int32_t)b->h_empties[k].size());
  for (int32_t k = 0; k < W; ++k) w.put(b->h_empties[k].data(), b->h_empties[k].size());
  w.put1(fnv1a(w.buf.data(), w.buf.size()));
  const std::string tmp = std::string(path) + ".tmp";
  FILE* f = std::fopen(tmp.c_str(), "wb");
  if (!f) {
    g_last_error = "cannot open " + tmp;
    return SHAPES_E_INVALID_ARG;
  }
  const bool wrote = std::fwrite(w.buf.data(), 1, w.buf.size(), f) == w.buf.size();
  const bool closed = std::fclose(f) == 0;
  if (!wrote || !closed || std::rename(tmp.c_str(), path) != 0) {
    std::remove(tmp.c_str());
    g_last_error = std::string("cannot write ") + path;
    return SHAPES_E_INVALID_ARG;
  }
  return SHAPES_OK;
}

int shapes_batch_load(const char* path, shapes_batch** out) {
  if (!path || !out) return SHAPES_E_INVALID_ARG;
  *out = nullptr;
  std::vector<unsigned char> buf;
  {
    FILE* f = std::fopen(path, "rb");
    if (!f) {
      g_last_error = std::string("cannot open ") + path;
      return SHAPES_E_INVALID_ARG;
    }
    unsigned char chunk[1 << 16];
    size_t got;
    while ((got = std::fread(chunk, 1, sizeof chunk, f)) > 0) buf.insert(buf.end(), chunk, chunk + got);
    std::fclose(f);
  }
  auto bad = [&](const char* why) {
    g_last_error = std::string("checkpoint ") + path + ": " + why;
    return SHAPES_E_INVALID_ARG;
  };
  if (buf.size() < 40 + sizeof(uint64_t)) return bad("too short"); /* 40-byte header + hash */
  uint64_t sum = 0;
  std::memcpy(&sum, buf.data() + buf.size() - sizeof(uint64_t), sizeof sum);
  if (fnv1a(buf.data(), buf.size() - sizeof(uint64_t)) != sum) return bad("checksum mismatch");
  CkReader r{buf};
  char magic[8];
  r.get(magic, 8);
  if (std::memcmp(magic, kCkMagic, 8) != 0) return bad("not a shapes checkpoint");
  if (r.get1<uint32_t>() != kCkVersion) return bad("unsupported version");
  if (r.get1<uint32_t>() != kCkEndian) return bad("byte order differs");
  const int32_t W = r.get1<int32_t>(), N = r.get1<int32_t>();
  const int64_t V = r.get1<int64_t>(), nc = r.get1<int64_t>();
  if (!r.ok || W < 1 || N < 1 || V < 1 || nc < 0 || V > (int64_t)INT32_MAX || nc > (int64_t)INT32_MAX)
    return bad("bad sizes");
  const uint64_t need = 40ull + 4ull * (W + 1) + 4ull * (N + 1) + 16ull * V + 80ull * N + 4ull * W + 16ull * nc +
                        16ull * nc + 1ull * N + 4ull * W + 8ull; /* + the empty-slot stacks */
  if (buf.size() < need) return bad("size does not match the header");
  std::vector<int32_t> off(W + 1), vo(N + 1), wc(W), keys(4 * (size_t)std::max<int64_t>(nc, 1));
  std::vector<double> xy(2 * (size_t)V), body(10 * (size_t)N), lam(2 * (size_t)std::max<int64_t>(nc, 1));
  r.get(off.data(), off.size());
  r.get(vo.data(), vo.size());
  r.get(xy.data(), xy.size());
  r.get(body.data(), body.size());
  r.get(wc.data(), wc.size());
  r.get(keys.data(), 4 * (size_t)nc);
  r.get(lam.data(), 2 * (size_t)nc);
  std::vector<uint8_t> act(N);
  r.get(act.data(), act.size());
  std::vector<int32_t> elen(W);
  r.get(elen.data(), elen.size());
  std::vector<std::vector<int32_t>> empties(W);
  uint64_t total_empty = 0;
  for (int32_t k = 0; k < W && r.ok; ++k) {
    const int32_t nw = off[k + 1] - off[k];
    if (elen[k] < 0 || elen[k] > nw) return bad("bad empty-slot stack");
    total_empty += (uint64_t)elen[k];
    empties[k].resize(elen[k]);
    r.get(empties[k].data(), empties[k].size());
    for (int32_t e : empties[k])
      if (e < 0 || e >= nw || act[off[k] + e]) return bad("bad empty-slot stack");
  }
  if (!r.ok || buf.size() != need + 4ull * total_empty) return bad("size does not match the header");
  shapes_bodies in{};
  double* bp[10];
  for (int k = 0; k < 10; ++k) bp[k] = body.data() + (size_t)k * N;
  in.vel_x = bp[0]; in.vel_y = bp[1]; in.rot_vel = bp[2]; in.pos_x = bp[3]; in.pos_y = bp[4];
  in.rot = bp[5]; in.inv_mass_lin = bp[6]; in.inv_mass_rot = bp[7]; in.mu = bp[8]; in.bounce = bp[9];
  if (vo[0] != 0 || vo[N] != V) return bad("bad vertex offsets");
  std::vector<uint8_t> kind(N);
  for (int32_t i = 0; i < N && r.ok; ++i) {
    if (vo[i + 1] < vo[i] || vo[i + 1] > V) return bad("bad vertex offsets");
    kind[i] = vo[i + 1] - vo[i] == 1 ? SHAPES_SHAPE_CIRCLE : SHAPES_SHAPE_HULL;
  }
  shapes_batch* h = nullptr;
  int rc = shapes_batch_create(W, off.data(), &in, vo.data(), xy.data(), kind.data(), &h);
  if (rc != SHAPES_OK) return rc;
  rc = shapes_batch_set_cache(h, wc.data(), keys.data(), lam.data());
  if (rc == SHAPES_OK)
    rc = guarded([&]() -> int {
      for (int32_t i = 0; i < N; ++i) h->h_active[i] = act[i] ? 1 : 0;
      h->h_empties = empties;
      h->upload_active();
      return SHAPES_OK;
    });
  if (rc != SHAPES_OK) {
    shapes_batch_destroy(h);
    return rc;
  }
  *out = h;
  return SHAPES_OK;
}

int shapes_batch_set_graphs(shapes_batch* b, int32_t enabled) {
  if (!b) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    ck(cudaStreamSynchronize(b->stream), "sync");
    b->graphs_enabled = enabled != 0;
    b->drop_graphs();
    b->invalidate_graphs();
    return SHAPES_OK;
  });
}

int shapes_batch_get_graph_captures(shapes_batch* b, int64_t* captures) {
  if (!b || !captures) return SHAPES_E_INVALID_ARG;
  *captures = b->graph_captures;
  return SHAPES_OK;
}

int shapes_batch_set_mlp(shapes_batch* b, const shapes_mlp* m) {
  if (!b) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    ck(cudaStreamSynchronize(b->stream), "sync");
    if (m && !b->learned_mask) {
      b->learned_mask = dalloc<uint8_t>(b->W, "cudaMalloc");
      b->snap_mask = dalloc<uint8_t>(b->W, "cudaMalloc");
    }
    if (m) ck(cudaMemsetAsync(b->learned_mask, 1, b->W, b->stream), "memset");
    if (m) ck(mlp::prepare_device(), "network set-up");
    b->mlp_model = m;
    b->invalidate_graphs();
    ck(cudaStreamSynchronize(b->stream), "sync");
    return SHAPES_OK;
  });
}

int shapes_batch_get_learned_mask(shapes_batch* b, uint8_t* mask) {
  if (!b || !mask) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    if (!b->learned_mask) {
      std::fill(mask, mask + b->W, (uint8_t)0);
      return SHAPES_OK;
    }
    ck(cudaMemcpyAsync(mask, b->learned_mask, b->W, cudaMemcpyDeviceToHost, b->stream), "download");
    ck(cudaStreamSynchronize(b->stream), "download");
    return SHAPES_OK;
  });
}

int shapes_batch_set_learned_mask(shapes_batch* b, const uint8_t* mask) {
  if (!b || !mask || !b->learned_mask) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    std::vector<uint8_t> m(b->W);
    for (int32_t w = 0; w < b->W; ++w) m[w] = mask[w] ? 1 : 0;
    ck(cudaMemcpyAsync(b->learned_mask, m.data(), b->W, cudaMemcpyHostToDevice, b->stream), "upload");
    ck(cudaStreamSynchronize(b->stream), "upload");
    return SHAPES_OK;
  });
}

int shapes_batch_set_judge(shapes_batch* b, const double* max_residual, const double* max_depth) {
  if (!b) return SHAPES_E_INVALID_ARG;
  for (int32_t w = 0; w < b->W; ++w)
    if ((max_residual && std::isnan(max_residual[w])) || (max_depth && std::isnan(max_depth[w])))
      return SHAPES_E_NAN;
  return guarded([&]() -> int {
    if (!b->judge_res) {
      b->judge_res = dalloc<double>(b->W, "cudaMalloc");
      b->judge_depth = dalloc<double>(b->W, "cudaMalloc");
    }
    const double inf = std::numeric_limits<double>::infinity();
    std::vector<double> r(b->W, inf), dd(b->W, inf);
    if (max_residual) std::copy(max_residual, max_residual + b->W, r.begin());
    if (max_depth) std::copy(max_depth, max_depth + b->W, dd.begin());
    ck(cudaMemcpyAsync(b->judge_res, r.data(), sizeof(double) * b->W, cudaMemcpyHostToDevice, b->stream), "upload");
    ck(cudaMemcpyAsync(b->judge_depth, dd.data(), sizeof(double) * b->W, cudaMemcpyHostToDevice, b->stream),
       "upload");
    ck(cudaStreamSynchronize(b->stream), "upload");
    b->judge_set = max_residual || max_depth;
    b->invalidate_graphs();
    return SHAPES_OK;
  });
}

int shapes_batch_collect(shapes_batch* b, int64_t capacity) {
  if (!b || capacity < 0 || capacity > INT32_MAX) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    ck(cudaStreamSynchronize(b->stream), "sync");
    b->invalidate_graphs();
    dfree(b->ds_feat); dfree(b->ds_tgt); dfree(b->ds_count); dfree(b->snap_ds_count);
    b->ds_feat = b->ds_tgt = nullptr;
    b->ds_count = b->snap_ds_count = nullptr;
    b->ds_cap = 0;
    if (capacity == 0) return SHAPES_OK;
    b->ds_feat = dalloc<float>((size_t)capacity * mlp::kIn, "cudaMalloc samples");
    b->ds_tgt = dalloc<float>((size_t)capacity * mlp::kOut, "cudaMalloc samples");
    b->ds_count = dalloc<unsigned long long>(1, "cudaMalloc samples");
    b->snap_ds_count = dalloc<unsigned long long>(1, "cudaMalloc samples");
    ck(cudaMemsetAsync(b->ds_count, 0, sizeof(unsigned long long), b->stream), "memset");
    ck(cudaStreamSynchronize(b->stream), "sync");
    b->ds_cap = capacity;
    return SHAPES_OK;
  });
}

int shapes_batch_get_samples(shapes_batch* b, float* features, float* targets, int64_t capacity, int64_t* n) {
  if (!b || !n || capacity < 0 || (capacity > 0 && (!features || !targets))) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    unsigned long long cnt = 0;
    if (b->ds_count) {
      ck(cudaMemcpyAsync(&cnt, b->ds_count, sizeof(cnt), cudaMemcpyDeviceToHost, b->stream), "download");
      ck(cudaStreamSynchronize(b->stream), "download");
    }
    *n = (int64_t)cnt;
    const int64_t k = std::min<int64_t>((int64_t)cnt, capacity);
    if (k > 0) {
      ck(cudaMemcpyAsync(features, b->ds_feat, sizeof(float) * mlp::kIn * k, cudaMemcpyDeviceToHost, b->stream),
         "download");
      ck(cudaMemcpyAsync(targets, b->ds_tgt, sizeof(float) * mlp::kOut * k, cudaMemcpyDeviceToHost, b->stream),
         "download");
      ck(cudaStreamSynchronize(b->stream), "download");
    }
    return (int64_t)cnt > capacity ? SHAPES_E_BUFFER : SHAPES_OK;
  });
}

int shapes_batch_set_stream(shapes_batch* b, void* cuda_stream) {
  if (!b) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    ck(cudaStreamSynchronize(b->stream), "sync");
    b->stream = cuda_stream ? static_cast<cudaStream_t>(cuda_stream) : b->own_stream;
    return SHAPES_OK;
  });
}

int shapes_batch_set_incremental(shapes_batch* b, int32_t enabled) {
  if (!b) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    ck(cudaStreamSynchronize(b->stream), "sync");
    b->incremental = enabled != 0;
    b->invalidate_graphs();
    b->reset_incremental();
    return SHAPES_OK;
  });
}

int shapes_batch_set_sweep_prune(shapes_batch* b, int32_t min_bodies) {
  if (!b || min_bodies < 0) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    ck(cudaStreamSynchronize(b->stream), "sync");
    b->sap_min_bodies = min_bodies;
    b->invalidate_graphs();
    b->setup_sap();
    return SHAPES_OK;
  });
}

int shapes_batch_set_wait_limit(shapes_batch* b, int64_t polls) {
  if (!b || polls < 0) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    ck(cudaStreamSynchronize(b->stream), "sync");
    b->poll_limit = (long long)polls;
    b->invalidate_graphs();
    return SHAPES_OK;
  });
}

int shapes_batch_set_narrowphase_lanes(shapes_batch* b, int32_t lanes) {
  if (!b || (lanes != 1 && lanes != 2 && lanes != 4 && lanes != 8 && lanes != 16 && lanes != 32))
    return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    ck(cudaStreamSynchronize(b->stream), "sync");
    b->np_lanes = lanes;
    b->invalidate_graphs();
    return SHAPES_OK;
  });
}

int shapes_batch_set_profiling(shapes_batch* b, int32_t enabled) {
  if (!b) return SHAPES_E_INVALID_ARG;
  b->profiling = enabled != 0;
  for (int k = 0; k < SHAPES_STAGE_COUNT; ++k) {
    b->prof_ms[k] = 0.0;
    b->prof_launches[k] = 0;
  }
  return SHAPES_OK;
}

int shapes_batch_get_profile(shapes_batch* b, double* ms, int64_t* launches) {
  if (!b || !ms || !launches) return SHAPES_E_INVALID_ARG;
  for (int k = 0; k < SHAPES_STAGE_COUNT; ++k) {
    ms[k] = b->prof_ms[k];
    launches[k] = b->prof_launches[k];
    b->prof_ms[k] = 0.0;
    b->prof_launches[k] = 0;
  }
  return SHAPES_OK;
}

int shapes_batch_get_group_clocks(shapes_batch* b, int64_t* out, int32_t* n_groups) {
  if (!b || !n_groups) return SHAPES_E_INVALID_ARG;
  *n_groups = b->phase_clock_groups;
  if (!out) return SHAPES_OK;
  return guarded([&]() -> int {
    ck(cudaMemcpy(out, b->phase_clock, sizeof(long long) * 8 * b->phase_clock_groups, cudaMemcpyDeviceToHost),
       "download");
    return SHAPES_OK;
  });
}

int shapes_batch_set_launch_groups(shapes_batch* b, int32_t worlds_per_group, int32_t threads) {
  if (!b || worlds_per_group < 1 || worlds_per_group > shapes::kMaxGroupWorlds || threads < 0 || threads > 256 ||
      (threads % 32) != 0)
    return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    b->target_group_bodies = 0;
    b->worlds_per_group_override = worlds_per_group;
    b->solve_threads = threads > 0 ? threads : 32;
    b->make_groups(b->grouped_iterations >= 0 ? b->grouped_iterations : 2);
    return SHAPES_OK;
  });
}

int shapes_batch_set_group_warps(shapes_batch* b, int32_t warps) {
  if (!b || (warps != 1 && warps != 2 && warps != 4 && warps != 8)) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    ck(cudaStreamSynchronize(b->stream), "sync");
    b->group_warps = warps;
    b->group_warps_auto = false;
    b->invalidate_graphs();
    return SHAPES_OK;
  });
}

int shapes_batch_set_world_order(shapes_batch* b, const int32_t* order) {
  if (!b) return SHAPES_E_INVALID_ARG;
  if (order) {
    std::vector<char> seen(b->W, 0);
    for (int32_t k = 0; k < b->W; ++k) {
      if (order[k] < 0 || order[k] >= b->W || seen[order[k]]) return SHAPES_E_INVALID_ARG;
      seen[order[k]] = 1;
    }
  }
  return guarded([&]() -> int {
    if (order)
      b->world_order.assign(order, order + b->W);
    else
      b->world_order.clear();
    b->make_groups(b->grouped_iterations >= 0 ? b->grouped_iterations : 2);
    return SHAPES_OK;
  });
}

int shapes_batch_get_world_order(shapes_batch* b, int32_t* order) {
  if (!b || !order) return SHAPES_E_INVALID_ARG;
  if ((int)b->world_order.size() == b->W) {
    std::copy(b->world_order.begin(), b->world_order.end(), order);
  } else {
    for (int32_t k = 0; k < b->W; ++k) order[k] = k;
    std::stable_sort(order, order + b->W, [&](int a, int c) {
      return (b->h_world_body_off[a + 1] - b->h_world_body_off[a]) > (b->h_world_body_off[c + 1] - b->h_world_body_off[c]);
    });
  }
  return SHAPES_OK;
}

int shapes_batch_get_world_levels(shapes_batch* b, int32_t* levels) {
  if (!b || !levels) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    ck(cudaMemcpyAsync(levels, b->world_levels, sizeof(int32_t) * b->W, cudaMemcpyDeviceToHost, b->stream), "download");
    ck(cudaStreamSynchronize(b->stream), "download");
    return SHAPES_OK;
  });
}

int shapes_batch_set_parallel_levels(shapes_batch* b, int32_t enabled) {
  if (!b) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    ck(cudaStreamSynchronize(b->stream), "sync");
    b->parallel_levels = enabled != 0;
    b->invalidate_graphs();
    return SHAPES_OK;
  });
}

int shapes_batch_get_group_target(shapes_batch* b, int32_t* target_bodies) {
  if (!b || !target_bodies) return SHAPES_E_INVALID_ARG;
  *target_bodies = b->target_group_bodies;
  return SHAPES_OK;
}

int shapes_batch_get_launch(shapes_batch* b, int32_t* worlds_per_group, int32_t* threads, int32_t* group_warps) {
  if (!b) return SHAPES_E_INVALID_ARG;
  if (worlds_per_group) *worlds_per_group = b->worlds_per_group_override;
  if (threads) *threads = b->solve_threads;
  if (group_warps) *group_warps = b->group_warps;
  return SHAPES_OK;
}

int shapes_batch_set_spread_heavy(shapes_batch* b, int32_t enabled) {
  if (!b) return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    ck(cudaStreamSynchronize(b->stream), "sync");
    b->spread_heavy = enabled != 0;
    b->invalidate_graphs();
    return SHAPES_OK;
  });
}

int shapes_batch_get_spread_heavy(shapes_batch* b, int32_t* enabled) {
  if (!b || !enabled) return SHAPES_E_INVALID_ARG;
  *enabled = b->spread_heavy ? 1 : 0;
  return SHAPES_OK;
}

int shapes_batch_get_parallel_levels(shapes_batch* b, int32_t* enabled) {
  if (!b || !enabled) return SHAPES_E_INVALID_ARG;
  *enabled = b->parallel_levels ? 1 : 0;
  return SHAPES_OK;
}

int shapes_batch_set_launch(shapes_batch* b, int32_t target_bodies_per_group, int32_t threads) {
  if (!b || target_bodies_per_group < 0 || threads < 0 || threads > 256 || (threads % 32) != 0)
    return SHAPES_E_INVALID_ARG;
  return guarded([&]() -> int {
    b->target_group_bodies = target_bodies_per_group;
    b->worlds_per_group_override = 0;
    b->solve_threads = threads > 0 ? threads : 32;
    b->make_groups(b->grouped_iterations >= 0 ? b->grouped_iterations : 2);
    return SHAPES_OK;
  });
}

}  // extern "C"

/* ------------------------------------------------------------------------ */
/* Broadphase + contact generation without allocating                        */
/* ------------------------------------------------------------------------ */
/*
 * shapes_collide_noalloc serves callers that cannot allocate device memory
 * themselves: plugins whose host application owns every device buffer and
 * hands out pre-planned memory, and loops with a latency budget in which
 * cudaMalloc/cudaFree (which synchronize the whole device) are not allowed.
 * Its scratch lives in the fixed device array below, sized for at most
 * SHAPES_NOALLOC_MAX_BODIES bodies, SHAPES_NOALLOC_MAX_VERTS vertices and
 * SHAPES_NOALLOC_MAX_PAIRS broadphase pairs.  Every GPU that loads this
 * library holds that array until the process exits.
 */
namespace {

constexpr int kNaMaxBodies = SHAPES_NOALLOC_MAX_BODIES;
constexpr int kNaMaxVerts = SHAPES_NOALLOC_MAX_VERTS;
constexpr int kNaMaxPairs = SHAPES_NOALLOC_MAX_PAIRS;
constexpr int kNaMaxContacts = 2 * kNaMaxPairs;
constexpr int kNaTiles = (kNaMaxPairs + 1 + shapes::kScanTile - 1) / shapes::kScanTile + 1;

/* What a call counts on being zero: its counters and what its scans keep.  One
 * block, cleared at the start of every call, so that nothing an earlier call
 * left (calls that overlapped, which is the caller's fault, leave the scans'
 * words of several launches mixed) reaches a later one. */
struct NaWords {
  unsigned long long counters[shapes::kCntSlots];
  unsigned long long tiles[kNaTiles];
  uint32_t scan_ctl[3];
};

/* Byte offsets of the scratch arrays, each 256-byte aligned. */
struct NaPlan {
  size_t world_body_off, body_world, lx, ly, emin, emax, wx, wy, nx, ny, vf, ef, box, boxk, flags, row_mode, row_cnt,
      row_hits, row_off, pair_a, pair_b, slot_cnt, slot_off, slot_feat, slot_val, world_pair_off, cwo, c_key, c_ga, c_gb,
      c_flip, c_hit, c_val, words, total;
};

constexpr size_t na_take(size_t& o, size_t bytes) {
  const size_t at = o;
  o += (bytes + 255) & ~size_t(255);
  return at;
}

constexpr NaPlan na_plan() {
  NaPlan p{};
  size_t o = 0;
  p.world_body_off = na_take(o, 2 * sizeof(int32_t));
  p.body_world = na_take(o, kNaMaxBodies * sizeof(int32_t));
  p.lx = na_take(o, kNaMaxVerts * sizeof(double));
  p.ly = na_take(o, kNaMaxVerts * sizeof(double));
  p.emin = na_take(o, kNaMaxVerts * sizeof(int32_t));
  p.emax = na_take(o, kNaMaxVerts * sizeof(int32_t));
  p.wx = na_take(o, kNaMaxVerts * sizeof(double));
  p.wy = na_take(o, kNaMaxVerts * sizeof(double));
  p.nx = na_take(o, kNaMaxVerts * sizeof(double));
  p.ny = na_take(o, kNaMaxVerts * sizeof(double));
  p.vf = na_take(o, kNaMaxVerts * sizeof(float4));
  p.ef = na_take(o, kNaMaxVerts * sizeof(float2));
  p.box = na_take(o, 4 * kNaMaxBodies * sizeof(double));
  p.boxk = na_take(o, 4 * kNaMaxBodies * sizeof(uint64_t));
  p.flags = na_take(o, kNaMaxBodies);
  p.row_mode = na_take(o, kNaMaxBodies);
  p.row_cnt = na_take(o, kNaMaxBodies * sizeof(int32_t));
  p.row_hits = na_take(o, shapes::kRowHits * kNaMaxBodies * sizeof(int32_t));
  p.row_off = na_take(o, (kNaMaxBodies + 1) * sizeof(int32_t));
  p.pair_a = na_take(o, kNaMaxPairs * sizeof(int32_t));
  p.pair_b = na_take(o, kNaMaxPairs * sizeof(int32_t));
  p.slot_cnt = na_take(o, kNaMaxPairs * sizeof(int32_t));
  p.slot_off = na_take(o, (kNaMaxPairs + 1) * sizeof(int32_t));
  p.slot_feat = na_take(o, 2 * (size_t)kNaMaxPairs * sizeof(int32_t));
  p.slot_val = na_take(o, 10 * (size_t)kNaMaxPairs * sizeof(double));
  p.world_pair_off = na_take(o, 2 * sizeof(int32_t));
  p.cwo = na_take(o, 2 * sizeof(int32_t));
  p.c_key = na_take(o, kNaMaxContacts * sizeof(uint64_t));
  p.c_ga = na_take(o, kNaMaxContacts * sizeof(int32_t));
  p.c_gb = na_take(o, kNaMaxContacts * sizeof(int32_t));
  p.c_flip = na_take(o, kNaMaxContacts);
  p.c_hit = na_take(o, kNaMaxContacts);
  p.c_val = na_take(o, 5 * (size_t)kNaMaxContacts * sizeof(double));
  p.words = na_take(o, sizeof(NaWords));
  p.total = o;
  return p;
}

constexpr NaPlan kNaPlan = na_plan();

}  // namespace

/* The scratch.  Device code may name it directly; in host code the name is a
 * host-side stand-in, not a device address, so the host uses the address that
 * cudaGetSymbolAddress returns (resolved once per device below). */
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaPlan.total];

namespace {

/* Reasons the set-up kernel rejects an input (bits of the bad-input counter). */
constexpr unsigned long long kNaBadOffsets = 1, kNaBadNaN = 2, kNaBadNonconvex = 4, kNaBadEdge = 8;

/* Per-call set-up in scratch: the one-world offsets, de-interleaved local
 * vertices and zeroed row modes.  Validates the caller's input as
 * shapes_batch_create does on the host, so that no later kernel indexes
 * outside the vertex arrays or meets a hull it cannot handle: every body needs
 * 3..64 vertices inside [0, n_verts) (offsets starting at 0 and ending at
 * n_verts), a strictly convex counter-clockwise hull of finite points with no
 * zero-length edge (the same products and comparisons as the host check), and
 * finite position, angle and inverse masses.  The counters were zeroed by the
 * host before this kernel. */
__global__ void k_noalloc_setup(int n, int nv, const int32_t* vert_off, const double* local_xy, const double* px,
                                const double* py, const double* th, const double* iml, const double* imr,
                                unsigned char* base) {
  int32_t* wbo = reinterpret_cast<int32_t*>(base + kNaPlan.world_body_off);
  int32_t* bw = reinterpret_cast<int32_t*>(base + kNaPlan.body_world);
  uint8_t* mode = base + kNaPlan.row_mode;
  double* lx = reinterpret_cast<double*>(base + kNaPlan.lx);
  double* ly = reinterpret_cast<double*>(base + kNaPlan.ly);
  unsigned long long* cnt = reinterpret_cast<NaWords*>(base + kNaPlan.words)->counters;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  if (t0 == 0) {
    wbo[0] = 0;
    wbo[1] = n;
    if (vert_off[0] != 0 || vert_off[n] != nv) atomicOr(&cnt[shapes::kCntBadInput], kNaBadOffsets);
  }
  for (int i = t0; i < n; i += stride) {
    bw[i] = 0;
    mode[i] = 0;
    unsigned long long bad = 0;
    if (!isfinite(px[i]) || !isfinite(py[i]) || !isfinite(th[i]) || !isfinite(iml[i]) || !isfinite(imr[i]))
      bad |= kNaBadNaN;
    const int o0 = vert_off[i], o1 = vert_off[i + 1], c = o1 - o0;
    if (o0 < 0 || o1 > nv || c < 3 || c > shapes::kMaxVerts) {
      bad |= kNaBadOffsets;
    } else { /* the hull lies inside the caller's vertex array: check it */
      const double* xy = local_xy + 2 * (size_t)o0;
      for (int k = 0; k < 2 * c; ++k)
        if (!isfinite(xy[k])) bad |= kNaBadNaN;
      if (!(bad & kNaBadNaN)) {
        for (int k = 0; k < c; ++k) {
          const int k1 = k + 1 < c ? k + 1 : k + 1 - c, k2 = k + 2 < c ? k + 2 : k + 2 - c;
          const double ex = xy[2 * k1] - xy[2 * k], ey = xy[2 * k1 + 1] - xy[2 * k + 1];
          const double fx = xy[2 * k2] - xy[2 * k1], fy = xy[2 * k2 + 1] - xy[2 * k1 + 1];
          if (ex == 0.0 && ey == 0.0) bad |= kNaBadEdge;
          else if (ex * fy - ey * fx <= 0.0) bad |= kNaBadNonconvex;
        }
      }
    }
    if (bad) atomicOr(&cnt[shapes::kCntBadInput], bad);
  }
  for (int v = t0; v < nv; v += stride) {
    lx[v] = local_xy[2 * (size_t)v];
    ly[v] = local_xy[2 * (size_t)v + 1];
  }
}

/* Copies pairs and contacts from scratch into the caller's buffers. */
__global__ void k_noalloc_out(int n_pairs, int n_contacts, const unsigned char* base, int32_t* pairs_ij,
                              int32_t* keys5, double* vals5) {
  const int32_t* pa = reinterpret_cast<const int32_t*>(base + kNaPlan.pair_a);
  const int32_t* pb = reinterpret_cast<const int32_t*>(base + kNaPlan.pair_b);
  const uint64_t* key = reinterpret_cast<const uint64_t*>(base + kNaPlan.c_key);
  const uint8_t* flip = base + kNaPlan.c_flip;
  const double* val = reinterpret_cast<const double*>(base + kNaPlan.c_val);
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  for (int p = t0; p < n_pairs; p += stride) {
    pairs_ij[2 * p] = pa[p];
    pairs_ij[2 * p + 1] = pb[p];
  }
  for (int c = t0; c < n_contacts; c += stride) {
    const uint64_t k = key[c];
    keys5[5 * c] = (int32_t)(k >> 44);
    keys5[5 * c + 1] = (int32_t)((k >> 24) & 0xfffff);
    keys5[5 * c + 2] = (int32_t)((k >> 12) & 0xfff);
    keys5[5 * c + 3] = (int32_t)(k & 0xfff);
    keys5[5 * c + 4] = flip[c];
    for (int q = 0; q < 5; ++q) vals5[5 * c + q] = val[5 * (size_t)c + q];
  }
}

/* Device address of g_noalloc_scratch on the current device, looked up once
 * per device (the first call on a device does this set-up). */
int noalloc_scratch_ptr(unsigned char** out) {
  static std::atomic<unsigned char*> ptrs[kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return SHAPES_E_CUDA;
  unsigned char* p = ptrs[dev].load();
  if (!p) {
    void* addr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&addr, g_noalloc_scratch);
    if (e != cudaSuccess) {
      g_last_error = std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e);
      return SHAPES_E_CUDA;
    }
    p = static_cast<unsigned char*>(addr);
    ptrs[dev].store(p);
  }
  *out = p;
  return SHAPES_OK;
}

}  // namespace

extern "C" int shapes_collide_noalloc(int32_t n_bodies, const double* pos_x, const double* pos_y, const double* rot,
                                      const double* inv_mass_lin, const double* inv_mass_rot,
                                      const int32_t* vert_offsets, const double* local_verts_xy, int32_t n_verts,
                                      int32_t* pairs_ij, int64_t pair_capacity, int32_t* contact_keys5,
                                      double* contact_vals5, int64_t contact_capacity, void* cuda_stream,
                                      int64_t* n_pairs, int64_t* n_contacts) {
  if (!pos_x || !pos_y || !rot || !inv_mass_lin || !inv_mass_rot || !vert_offsets || !local_verts_xy || !n_pairs ||
      !n_contacts || n_bodies < 1 || n_verts < 3 * n_bodies) {
    g_last_error = "shapes_collide_noalloc: a null pointer, no bodies, or fewer than 3 vertices per body";
    return SHAPES_E_INVALID_ARG;
  }
  if (n_bodies > kNaMaxBodies || n_verts > kNaMaxVerts) {
    g_last_error = "shapes_collide_noalloc: more than SHAPES_NOALLOC_MAX_BODIES bodies or SHAPES_NOALLOC_MAX_VERTS vertices";
    return SHAPES_E_CAPACITY;
  }
  unsigned char* base = nullptr;
  const int rc = noalloc_scratch_ptr(&base);
  if (rc != SHAPES_OK) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  Dev d{};
  d.n_worlds = 1;
  d.n_bodies = n_bodies;
  d.n_verts = n_verts;
  d.pair_cap = kNaMaxPairs;
  d.contact_cap = kNaMaxContacts;
  d.world_body_off = reinterpret_cast<int32_t*>(base + kNaPlan.world_body_off);
  d.body_world = reinterpret_cast<int32_t*>(base + kNaPlan.body_world);
  d.vert_off = vert_offsets;
  d.lx = reinterpret_cast<double*>(base + kNaPlan.lx);
  d.ly = reinterpret_cast<double*>(base + kNaPlan.ly);
  d.emin = reinterpret_cast<int32_t*>(base + kNaPlan.emin);
  d.emax = reinterpret_cast<int32_t*>(base + kNaPlan.emax);
  d.px = const_cast<double*>(pos_x);
  d.py = const_cast<double*>(pos_y);
  d.th = const_cast<double*>(rot);
  d.iml = inv_mass_lin;
  d.imr = inv_mass_rot;
  d.wx = reinterpret_cast<double*>(base + kNaPlan.wx);
  d.wy = reinterpret_cast<double*>(base + kNaPlan.wy);
  d.nx = reinterpret_cast<double*>(base + kNaPlan.nx);
  d.ny = reinterpret_cast<double*>(base + kNaPlan.ny);
  d.vf = reinterpret_cast<float4*>(base + kNaPlan.vf);
  d.ef = reinterpret_cast<float2*>(base + kNaPlan.ef);
  d.box = reinterpret_cast<double*>(base + kNaPlan.box);
  d.boxk = reinterpret_cast<uint64_t*>(base + kNaPlan.boxk);
  d.flags = base + kNaPlan.flags;
  d.row_mode = base + kNaPlan.row_mode;
  d.row_cnt = reinterpret_cast<int32_t*>(base + kNaPlan.row_cnt);
  d.row_hits = reinterpret_cast<int32_t*>(base + kNaPlan.row_hits);
  d.row_off = reinterpret_cast<int32_t*>(base + kNaPlan.row_off);
  d.pair_a = reinterpret_cast<int32_t*>(base + kNaPlan.pair_a);
  d.pair_b = reinterpret_cast<int32_t*>(base + kNaPlan.pair_b);
  d.slot_cnt = reinterpret_cast<int32_t*>(base + kNaPlan.slot_cnt);
  d.slot_off = reinterpret_cast<int32_t*>(base + kNaPlan.slot_off);
  d.slot_feat = reinterpret_cast<int32_t*>(base + kNaPlan.slot_feat);
  d.slot_val = reinterpret_cast<double*>(base + kNaPlan.slot_val);
  d.world_pair_off = reinterpret_cast<int32_t*>(base + kNaPlan.world_pair_off);
  d.world_contact_off = reinterpret_cast<int32_t*>(base + kNaPlan.cwo);
  d.c_key = reinterpret_cast<uint64_t*>(base + kNaPlan.c_key);
  d.c_ga = reinterpret_cast<int32_t*>(base + kNaPlan.c_ga);
  d.c_gb = reinterpret_cast<int32_t*>(base + kNaPlan.c_gb);
  d.c_flip = base + kNaPlan.c_flip;
  d.c_hit = base + kNaPlan.c_hit;
  d.c_val = reinterpret_cast<double*>(base + kNaPlan.c_val);
  NaWords* const words = reinterpret_cast<NaWords*>(base + kNaPlan.words);
  d.counters = words->counters;
  const shapes::ScanState scan_state{words->tiles, words->scan_ctl, kNaTiles};
  auto scan = [&](int32_t* in, int n_cap, const unsigned long long* n_dev, int32_t* out, unsigned long long* total,
                  int cap, unsigned bit) {
    launch_chained(true, shapes::k_scan, n_cap / shapes::kScanTile + 1, shapes::kScanThreads, 0, st, in, n_cap, n_dev,
                   scan_state, out, 0, total, cap, d.counters + shapes::kCntOverflow, bit,
                   d.counters + shapes::kCntSolveErr);
  };
  /* counters and scans start at zero; the set-up kernel validates the vertex offsets */
  cudaError_t e = cudaMemsetAsync(words, 0, sizeof(NaWords), st);
  unsigned long long cnt[shapes::kCntSlots] = {0};
  if (e == cudaSuccess) {
    k_noalloc_setup<<<grid_for(std::max(n_bodies, n_verts), 256), 256, 0, st>>>(
        n_bodies, n_verts, vert_offsets, local_verts_xy, pos_x, pos_y, rot, inv_mass_lin, inv_mass_rot, base);
    e = cudaMemcpyAsync(cnt, d.counters, sizeof(cnt), cudaMemcpyDeviceToHost, st);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    g_last_error = std::string("shapes_collide_noalloc: ") + cudaGetErrorString(e);
    return SHAPES_E_CUDA;
  }
  if (const unsigned long long bad = cnt[shapes::kCntBadInput]) {
    if (bad & (kNaBadOffsets | kNaBadEdge)) {
      g_last_error = (bad & kNaBadOffsets)
                         ? "shapes_collide_noalloc: vert_offsets must start at 0, end at n_verts and give every body "
                           "3..64 vertices (circles are not accepted)"
                         : "shapes_collide_noalloc: a hull has a zero-length edge";
      return SHAPES_E_INVALID_ARG;
    }
    if (bad & kNaBadNaN) {
      g_last_error = "shapes_collide_noalloc: a position, angle, inverse mass or hull point is not finite";
      return SHAPES_E_NAN;
    }
    g_last_error = "shapes_collide_noalloc: a hull is not strictly convex and counter-clockwise";
    return SHAPES_E_NONCONVEX;
  }
  launch_chained(true, shapes::k_init_extents, grid_for(n_verts, 128), 128, 0, st, d);
  launch_pose(true, st, n_bodies, d, 0.0, 0);
  launch_chained(true, shapes::k_count_brute, grid_for((long long)n_bodies * 32, 256), 256, 0, st, d);
  scan(d.row_cnt, n_bodies, nullptr, d.row_off, d.counters + shapes::kCntPairs, d.pair_cap, 1u);
  launch_chained(true, shapes::k_write_rows<false, false>, grid_for(n_bodies, shapes::kRowThreads),
                 shapes::kRowThreads, 0, st, d);
  launch_chained(true, shapes::k_narrowphase, grid_for(kNaMaxPairs, shapes::kNpThreads), shapes::kNpThreads, 0, st, d);
  scan(d.slot_cnt, kNaMaxPairs, d.counters + shapes::kCntPairs, d.slot_off, d.counters + shapes::kCntContacts,
       d.contact_cap, 2u);
  launch_chained(true, shapes::k_build, grid_for(2LL * kNaMaxPairs, shapes::kBuildThreads), shapes::kBuildThreads, 0, st,
                 d, 0.0, 0.0, 0, 0, 0);
  e = cudaMemcpyAsync(cnt, d.counters, sizeof(cnt), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    g_last_error = std::string("shapes_collide_noalloc: ") + cudaGetErrorString(e);
    return SHAPES_E_CUDA;
  }
  if (cnt[shapes::kCntSolveErr]) {
    g_last_error = "shapes_collide_noalloc: a scan's bounded wait gave up";
    return SHAPES_E_TIMEOUT;
  }
  *n_pairs = (int64_t)cnt[shapes::kCntPairs];
  *n_contacts = (int64_t)cnt[shapes::kCntContacts];
  if (cnt[shapes::kCntOverflow]) {
    g_last_error = "shapes_collide_noalloc: more than SHAPES_NOALLOC_MAX_PAIRS broadphase pairs";
    return SHAPES_E_CAPACITY;
  }
  if (*n_pairs > pair_capacity || *n_contacts > contact_capacity) {
    g_last_error = "shapes_collide_noalloc: pair_capacity or contact_capacity below *n_pairs / *n_contacts";
    return SHAPES_E_BUFFER;
  }
  if ((*n_pairs > 0 && !pairs_ij) || (*n_contacts > 0 && (!contact_keys5 || !contact_vals5))) {
    g_last_error = "shapes_collide_noalloc: null output buffer";
    return SHAPES_E_INVALID_ARG;
  }
  if (*n_pairs > 0 || *n_contacts > 0) {
    k_noalloc_out<<<grid_for(std::max(*n_pairs, *n_contacts), 256), 256, 0, st>>>(
        (int)*n_pairs, (int)*n_contacts, base, pairs_ij, contact_keys5, contact_vals5);
    e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) {
      g_last_error = std::string("shapes_collide_noalloc: ") + cudaGetErrorString(e);
      return SHAPES_E_CUDA;
    }
  }
  return SHAPES_OK;
}
