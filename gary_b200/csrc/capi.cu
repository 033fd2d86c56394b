// C-ABI glue: error strings, handle lifetime, dispatch of gary_count.
// No C++ exception crosses this boundary: every entry point catches and maps
// to a GARY_ERR_* status (the reference's checkCudaErrors exits the process
// instead, common/HelperCUDA.h:582-595).
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <iterator>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <unordered_map>
#include <vector>

#include "graph.cuh"
#include "internal.cuh"
#include "mlp.cuh"
#include "patterns.cuh"
#include "tc.cuh"

namespace gary {

namespace {
thread_local char g_error[1024] = {0};
}

void set_error(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
}

void clear_error() { g_error[0] = '\0'; }

int device_ordinal() {
  int d = 0;
  cudaGetDevice(&d);
  return d;
}

int sm_count() {
  static int cache[64] = {0};
  int d = device_ordinal();
  if (d >= 0 && d < 64 && cache[d]) return cache[d];
  int v = 0;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d) != cudaSuccess || v <= 0) {
    cudaGetLastError();
    v = 148;
  }
  if (d >= 0 && d < 64) cache[d] = v;
  return v;
}

namespace {
std::mutex g_pool_mu;
cudaMemPool_t g_pools[64] = {};
uint64_t g_pool_keep = ~0ull;  // keep freed scratch mapped, as a caching allocator does
}  // namespace

cudaMemPool_t scratch_pool() {
  const int d = device_ordinal();
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if (d < 0 || d >= 64) {
    cudaMemPool_t p = nullptr;
    cudaDeviceGetDefaultMemPool(&p, d);
    return p;
  }
  if (!g_pools[d]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = d;
    if (cudaMemPoolCreate(&g_pools[d], &props) != cudaSuccess) {
      cudaGetLastError();
      cudaDeviceGetDefaultMemPool(&g_pools[d], d);
    } else {
      uint64_t keep = g_pool_keep;
      cudaMemPoolSetAttribute(g_pools[d], cudaMemPoolAttrReleaseThreshold, &keep);
    }
  }
  return g_pools[d];
}

namespace {
struct BlockInfo {
  size_t bytes;
  int dev;
};
std::mutex g_blk_mu;
std::unordered_map<void *, BlockInfo> g_live;      // blocks handed out
std::multimap<size_t, void *> g_cached[64];         // free blocks by rounded size, per device
uint64_t g_cached_bytes[64] = {};

size_t round_block(size_t b) {
  if (b <= (1u << 20)) {
    size_t r = 256;
    while (r < b) r <<= 1;
    return r;
  }
  const size_t step = 2u << 20;
  return (b + step - 1) / step * step;
}

// Returns cached blocks of device d to the driver, largest first, until at
// most keep bytes stay cached.  Caller holds g_blk_mu.
void trim_blocks_locked(int d, uint64_t keep) {
  auto &c = g_cached[d];
  if (c.empty() || g_cached_bytes[d] <= keep) return;
  int cur = 0;
  cudaGetDevice(&cur);
  if (cur != d) cudaSetDevice(d);
  while (g_cached_bytes[d] > keep && !c.empty()) {
    auto it = std::prev(c.end());
    cudaFree(it->second);
    g_cached_bytes[d] -= it->first;
    c.erase(it);
  }
  if (cur != d) cudaSetDevice(cur);
}

// Tuning key "refuse_block": the k-th block asked for from then on is refused as
// a full device would refuse it (0: none), so that tests reach what a call leaves
// behind when it runs out of memory.
std::atomic<uint64_t> g_refuse_block{0};
bool refuse_block() {
  uint64_t k = g_refuse_block.load(std::memory_order_relaxed);
  while (k && !g_refuse_block.compare_exchange_weak(k, k - 1, std::memory_order_relaxed)) {
  }
  return k == 1;
}
}  // namespace

cudaError_t persistent_alloc(void **p, size_t bytes) {
  if (refuse_block()) return cudaErrorMemoryAllocation;
  const int d = device_ordinal();
  const size_t rb = round_block(bytes);
  if (d >= 0 && d < 64) {
    std::lock_guard<std::mutex> lk(g_blk_mu);
    auto &c = g_cached[d];
    auto it = c.lower_bound(rb);
    if (it != c.end() && it->first <= rb + rb / 8) {
      *p = it->second;
      g_live[*p] = BlockInfo{it->first, d};
      g_cached_bytes[d] -= it->first;
      c.erase(it);
      return cudaSuccess;
    }
  }
  cudaError_t e = cudaMalloc(p, rb);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    release_cached_memory();
    e = cudaMalloc(p, rb);
  }
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(g_blk_mu);
  g_live[*p] = BlockInfo{rb, d};
  return cudaSuccess;
}

void persistent_free(void *p) {
  BlockInfo info{0, -1};
  {
    std::lock_guard<std::mutex> lk(g_blk_mu);
    auto it = g_live.find(p);
    if (it != g_live.end()) {
      info = it->second;
      g_live.erase(it);
    }
  }
  if (info.dev < 0 || info.dev >= 64) {
    cudaFree(p);
    return;
  }
  int cur = 0;
  cudaGetDevice(&cur);
  if (cur != info.dev) cudaSetDevice(info.dev);
  if (cudaDeviceSynchronize() != cudaSuccess) cudaGetLastError();
  {
    std::lock_guard<std::mutex> lk(g_blk_mu);
    g_cached[info.dev].emplace(info.bytes, p);
    g_cached_bytes[info.dev] += info.bytes;
    uint64_t keep;
    {
      std::lock_guard<std::mutex> lk2(g_pool_mu);
      keep = g_pool_keep;
    }
    trim_blocks_locked(info.dev, keep);
  }
  if (cur != info.dev) cudaSetDevice(cur);
}

// ---- pinned result slots ---------------------------------------------------
// Where gary_count reads a launch's scheduler words and count to: page-locked,
// so that the copy is one asynchronous operation on the stream instead of a
// staged copy the host waits in.  One page for the process, handed out slot by
// slot under a lock, returned to the driver by release_cached_memory while no
// slot is out.  With no slot free the caller's own (pageable) struct is used.
struct ResultWords {
  SchedState st;
};

namespace {
constexpr int kResultSlots = 32;
std::mutex g_slot_mu;
ResultWords *g_slots = nullptr;
uint32_t g_slots_used = 0;
}  // namespace

struct ResultSlot {
  ResultWords own{};
  ResultWords *p = &own;
  int index = -1;
  ResultSlot() {
    std::lock_guard<std::mutex> lk(g_slot_mu);
    if (!g_slots && cudaHostAlloc(reinterpret_cast<void **>(&g_slots), sizeof(ResultWords) * kResultSlots,
                                  cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      g_slots = nullptr;
      return;
    }
    for (int k = 0; k < kResultSlots; ++k)
      if (!((g_slots_used >> k) & 1u)) {
        g_slots_used |= 1u << k;
        index = k;
        p = g_slots + k;
        return;
      }
  }
  ResultSlot(const ResultSlot &) = delete;
  ResultSlot &operator=(const ResultSlot &) = delete;
  ResultWords *operator->() { return p; }
  // Gives the slot back, once no copy into it can be in flight.  A call that
  // fails before that keeps it out: at most kResultSlots such calls, and the
  // ones after them use their own struct.
  void done() {
    if (index < 0) return;
    std::lock_guard<std::mutex> lk(g_slot_mu);
    g_slots_used &= ~(1u << index);
    index = -1;
    p = &own;
  }
};

void release_cached_memory() {
  {
    std::lock_guard<std::mutex> lk(g_slot_mu);
    if (g_slots && !g_slots_used) {
      cudaFreeHost(g_slots);
      g_slots = nullptr;
    }
  }
  {
    std::lock_guard<std::mutex> lk(g_blk_mu);
    for (int d = 0; d < 64; ++d) trim_blocks_locked(d, 0);
  }
  std::lock_guard<std::mutex> lk(g_pool_mu);
  for (int d = 0; d < 64; ++d) {
    if (!g_pools[d]) continue;
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != d) cudaSetDevice(d);
    cudaDeviceSynchronize();
    cudaMemPoolTrimTo(g_pools[d], 0);
    if (cur != d) cudaSetDevice(cur);
  }
  cudaGetLastError();
}

void set_pool_keep_bytes(uint64_t bytes) {
  {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    g_pool_keep = bytes;
    for (cudaMemPool_t p : g_pools) {
      if (!p) continue;
      uint64_t keep = bytes;
      cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
      cudaMemPoolTrimTo(p, bytes);
    }
  }
  std::lock_guard<std::mutex> lk(g_blk_mu);
  for (int d = 0; d < 64; ++d) trim_blocks_locked(d, bytes);
}

namespace {
double now_s() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}
bool trace_on() {
  static const bool on = [] {
    const char *e = std::getenv("GARY_TRACE");
    return e && *e && std::strcmp(e, "0") != 0;
  }();
  return on;
}
}  // namespace

PhaseTrace::PhaseTrace(const char *what_, cudaStream_t s_) : what(what_), s(s_), on(trace_on()) {
  if (on) {
    cudaStreamSynchronize(s);
    t0 = t = now_s();
  }
}

void PhaseTrace::mark(const char *phase) {
  if (!on) return;
  cudaStreamSynchronize(s);
  const double x = now_s();
  std::fprintf(stderr, "[gary trace] %s: %-24s %9.3f ms\n", what, phase, (x - t) * 1e3);
  t = x;
}

PhaseTrace::~PhaseTrace() {
  if (on) std::fprintf(stderr, "[gary trace] %s: %-24s %9.3f ms\n", what, "total", (now_s() - t0) * 1e3);
}

int upload(const uint64_t *ptr, const uint32_t *idx, uint32_t n, uint64_t nnz, uint32_t flags,
           cudaStream_t s, gary_graph **out, const uint64_t *group_off, uint32_t ngroups);
int build_coo(PaddedCSR &c, cudaStream_t s);
int download(gary_graph *g, uint64_t *ptr, uint32_t *idx, uint32_t *perm, cudaStream_t s);

void free_plans(gary_graph *g) {
  for (auto &p : g->plans) {
    delete p;
    p = nullptr;
  }
  delete g->k4_plan;
  delete g->c4_plan;
  delete g->c4_shard_plan;
  g->k4_plan = g->c4_plan = g->c4_shard_plan = nullptr;
}

namespace {

template <typename F>
int guarded(const char *what, F &&f) {
  clear_error();
  try {
    return f();
  } catch (const std::bad_alloc &) {
    set_error("%s: out of memory", what);
    return GARY_ERR_OOM;
  } catch (const std::exception &e) {
    set_error("%s: %s", what, e.what());
    return GARY_ERR_CUDA;
  } catch (...) {
    set_error("%s: unknown exception", what);
    return GARY_ERR_CUDA;
  }
}

int plan_slot(int pattern, int sched) { return (pattern - 3) * 2 + sched; }
constexpr int kShardSlot = 2;    // + sched: a shard's plan where the whole count's had no room for rows
constexpr int kProfileSlot = 7;  // the plan of gary_tc_features and gary_tc_profile: no hub rows

// That plan: the counting plan where it has no hub rows, else one of its own.
int profile_plan(gary_graph *g, cudaStream_t s, gary_count_plan **out) {
  gary_count_plan *count = g->plans[plan_slot(GARY_PATTERN_TRIANGLE, GARY_SCHED_PLAIN)];
  if (count && !count->hub.n_list) {
    *out = count;
    return GARY_OK;
  }
  if (!g->plans[kProfileSlot])
    GARY_TRY(build_k3_plan(g, tuned_params(), s, &g->plans[kProfileSlot], nullptr, Rows::kNone));
  *out = g->plans[kProfileSlot];
  return GARY_OK;
}

PlanParams g_tuning;  // process-wide knobs of the counting plans (gary_tune)
std::mutex g_tuning_mu;
std::vector<float> g_model;  // process-wide cost model (gary_set_cost_model)
std::mutex g_model_mu;

// own_word: the caller has no device word; a triangle count goes to the
// plan's SchedState::total (d_out is then the word of the other patterns).
int count_async(gary_graph *g, int pattern, int sched, cudaStream_t s, unsigned long long *d_out,
                uint32_t shard = 0, uint32_t nshards = 1, bool own_word = false) {
  GARY_CHECK_ARG(g != nullptr, "graph is NULL");
  GARY_CHECK_ARG(d_out != nullptr || own_word, "output pointer is NULL");
  GARY_CHECK_ARG(pattern == GARY_PATTERN_TRIANGLE || pattern == GARY_PATTERN_4CYCLE ||
                     pattern == GARY_PATTERN_4CLIQUE,
                 "unknown pattern %d", pattern);
  GARY_CHECK_ARG(sched == GARY_SCHED_PLAIN || sched == GARY_SCHED_LEARNED, "unknown scheduler %d",
                 sched);
  GARY_CHECK_ARG(nshards >= 1 && shard < nshards, "shard %u of %u is out of range", shard, nshards);
  // what a shard covers must not depend on this device's free memory
  const Rows rows = nshards > 1 ? Rows::kRequired : Rows::kOptional;
  if (own_word && pattern != GARY_PATTERN_TRIANGLE) {
    if (!g->result.p) GARY_TRY(g->result.alloc_persistent(1));
    d_out = g->result.p;
  }
  if (pattern == GARY_PATTERN_4CLIQUE) {
    if (g->dag.max_len > kK4MaxOutDegree) {
      set_error("4-clique counting supports out-degree <= %u (graph has %u)", kK4MaxOutDegree,
                g->dag.max_len);
      return GARY_ERR_UNSUPPORTED;
    }
    if (!g->k4_plan) GARY_TRY(build_k4_plan(g, s, &g->k4_plan));
    return launch_k4(g, g->k4_plan, d_out, s, shard, nshards);
  }
  if (pattern == GARY_PATTERN_4CYCLE) {
    PatternPlan *plan = nshards > 1 ? g->c4_shard_plan : g->c4_plan;
    if (nshards > 1 && g->c4_plan && g->c4_plan->rows.shared) plan = g->c4_plan;
    if (!plan) {
      GARY_TRY(build_c4_plan(g, s, &plan, rows));
      (nshards > 1 && (g->c4_plan || !plan->rows.shared) ? g->c4_shard_plan : g->c4_plan) = plan;
    }
    return launch_c4(g, plan, d_out, s, shard, nshards);
  }
  int slot = plan_slot(pattern, sched);
  if (nshards > 1 && g->plans[slot] && !g->plans[slot]->rows_by_graph) slot = kShardSlot + sched;
  if (!g->plans[slot]) {
    if (sched == GARY_SCHED_LEARNED) {
      std::vector<float> model;
      {
        std::lock_guard<std::mutex> lk(g_model_mu);
        model = g_model;
      }
      if (model.empty()) {
        set_error("GARY_SCHED_LEARNED needs a cost model: call gary_set_cost_model first");
        return GARY_ERR_INVALID;
      }
      GARY_TRY(build_k3_plan(g, tuned_params(), s, &g->plans[slot], model.data(), rows));
    } else {
      GARY_TRY(build_k3_plan(g, tuned_params(), s, &g->plans[slot], nullptr, rows));
    }
  }
  return launch_k3(g, g->plans[slot], d_out, s, shard, nshards);
}

}  // namespace

PlanParams tuned_params() {
  std::lock_guard<std::mutex> lk(g_tuning_mu);
  return g_tuning;
}

// GARY_OK, or the status the error word of a counting launch stands for.
int launch_status(uint32_t err) {
  if (!err) return GARY_OK;
  if (err & kLaunchErrTableFull) {
    set_error("a shared-memory table of the counting kernel overflowed (error word 0x%x): the count "
              "is incomplete", err);
    return GARY_ERR_INTERNAL;
  }
  set_error("a bounded device wait expired (error word 0x%x): the count is incomplete", err);
  return GARY_ERR_TIMEOUT;
}

}  // namespace gary

using gary::guarded;

extern "C" int gary_tune(const char *key, uint64_t value) {
  GARY_CHECK_ARG(key != nullptr, "key is NULL");
  std::lock_guard<std::mutex> lk(gary::g_tuning_mu);
  gary::PlanParams &p = gary::g_tuning;
  const std::string k(key);
  const bool pow2 = value && !(value & (value - 1));
  if (k == "warp_tile_cost") p.warp_tile_cost = value;  // 0: from the work
  else if (k == "cta_tile_cost" && value > 0) p.cta_tile_cost = value;
  else if (k == "warp_cap" && value >= 8 && value <= gary::kWarpTableSlots / 2) p.warp_cap = (uint32_t)value;
  else if (k == "cta_set_words" && (value == 0 || (pow2 && value >= 64 && value <= gary::kTcMaxWarps * gary::kWarpTableSlots)))
    p.cta_set_words = (uint32_t)value;
  else if (k == "stage_wait_polls" && value <= gary::kSpinLimit) p.stage_polls = (uint32_t)value;
  else if (k == "vertex_overhead") p.vertex_overhead = value;
  else if (k == "min_blocks" && (value == 0 || value == 2 || value == 3)) p.min_blocks = (uint32_t)value;
  else if (k == "pool_keep_bytes") gary::set_pool_keep_bytes(value);
  else if (k == "refuse_block") gary::g_refuse_block = value;
  else if (k == "reset") p = gary::PlanParams{};
  else {
    gary::set_error("unknown tuning key '%s' or value %llu out of range", key,
                    (unsigned long long)value);
    return GARY_ERR_INVALID;
  }
  return GARY_OK;
}

extern "C" int gary_set_cost_model(const float *params) {
  std::lock_guard<std::mutex> lk(gary::g_model_mu);
  if (!params) {
    gary::g_model.clear();
    return GARY_OK;
  }
  gary::g_model.assign(params, params + gary::kMlpParams);
  return GARY_OK;
}

extern "C" int gary_tc_features(gary_graph *g, float *d_x, uint8_t *d_legal, void *stream) {
  GARY_CHECK_ARG(g && d_x && d_legal, "NULL argument");
  return guarded("gary_tc_features", [&] {
    cudaStream_t s = gary::as_stream(stream);
    gary_count_plan *plan = nullptr;
    GARY_TRY(gary::profile_plan(g, s, &plan));
    return gary::k3_features(g, plan, d_x, d_legal, s);
  });
}

extern "C" int gary_tc_profile(gary_graph *g, int variant, uint64_t *d_cycles, uint64_t *d_count,
                               void *stream) {
  GARY_CHECK_ARG(g && d_cycles && d_count, "NULL argument");
  GARY_CHECK_ARG(variant >= -1 && variant <= 3, "variant must be -1 (plain) or 0..3");
  return guarded("gary_tc_profile", [&] {
    cudaStream_t s = gary::as_stream(stream);
    gary_count_plan *plan = nullptr;
    GARY_TRY(gary::profile_plan(g, s, &plan));
    gary::DevBuf<uint8_t> forced;
    if (variant >= 0) {
      GARY_TRY(forced.alloc(g->n, s));
      GARY_CUDA(cudaMemsetAsync(forced.p, variant, g->n, s));
    }
    GARY_CUDA(cudaMemsetAsync(d_cycles, 0, (uint64_t)g->n * 8, s));
    return gary::launch_k3_ctl(g, plan, reinterpret_cast<unsigned long long *>(d_count), s,
                               0, 1, variant >= 0 ? forced.p : nullptr,
                               reinterpret_cast<unsigned long long *>(d_cycles));
  });
}

// ---- batches ------------------------------------------------------------
struct gary_exec {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

namespace gary {
namespace {
int batch_count(gary_graph *g, unsigned long long *d_counts, unsigned long long *d_total,
                cudaStream_t s, int sched) {
  GARY_CHECK_ARG(g != nullptr && d_counts != nullptr && d_total != nullptr, "NULL argument");
  GARY_CHECK_ARG(g->ngroups > 0, "graph was not uploaded with gary_batch_upload");
  const int slot = plan_slot(GARY_PATTERN_TRIANGLE, sched);
  if (!g->plans[slot]) GARY_TRY(count_async(g, GARY_PATTERN_TRIANGLE, sched, s, d_total));
  GARY_CUDA(cudaMemsetAsync(d_counts, 0, (uint64_t)g->ngroups * 8, s));
  gary_count_plan *plan = g->plans[slot];
  return launch_k3_ctl(g, plan, d_total, s, 0, 1, plan->variant.p, nullptr, d_counts);
}
}  // namespace
}  // namespace gary

extern "C" int gary_batch_count_async(gary_graph *g, int sched, uint64_t *d_counts, uint64_t *d_total,
                                      void *stream) {
  GARY_CHECK_ARG(sched == GARY_SCHED_PLAIN || sched == GARY_SCHED_LEARNED, "unknown scheduler");
  return guarded("gary_batch_count_async", [&] {
    return gary::batch_count(g, reinterpret_cast<unsigned long long *>(d_counts),
                             reinterpret_cast<unsigned long long *>(d_total), gary::as_stream(stream),
                             sched);
  });
}

extern "C" int gary_batch_capture(gary_graph *g, int sched, uint64_t *d_counts, uint64_t *d_total,
                                  void *stream, gary_exec **out) {
  GARY_CHECK_ARG(out != nullptr, "out is NULL");
  GARY_CHECK_ARG(stream != nullptr, "capture needs a non-default stream");
  return guarded("gary_batch_capture", [&] {
    cudaStream_t s = gary::as_stream(stream);
    // plans are built (allocations, host syncs) before the capture begins
    GARY_TRY(gary::batch_count(g, reinterpret_cast<unsigned long long *>(d_counts),
                               reinterpret_cast<unsigned long long *>(d_total), s, sched));
    GARY_CUDA(cudaStreamSynchronize(s));
    auto e = std::make_unique<gary_exec>();
    GARY_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    const int st = gary::batch_count(g, reinterpret_cast<unsigned long long *>(d_counts),
                                     reinterpret_cast<unsigned long long *>(d_total), s, sched);
    cudaGraph_t graph = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(s, &graph);
    if (st != GARY_OK) {
      if (graph) cudaGraphDestroy(graph);
      return st;
    }
    GARY_CUDA(ce);
    e->graph = graph;
    GARY_CUDA(cudaGraphInstantiate(&e->exec, graph, 0));
    *out = e.release();
    return GARY_OK;
  });
}

extern "C" int gary_exec_launch(gary_exec *e, void *stream) {
  GARY_CHECK_ARG(e != nullptr, "exec is NULL");
  GARY_CUDA(cudaGraphLaunch(e->exec, gary::as_stream(stream)));
  return GARY_OK;
}

extern "C" int gary_exec_free(gary_exec *e) {
  if (!e) return GARY_OK;
  if (e->exec) cudaGraphExecDestroy(e->exec);
  if (e->graph) cudaGraphDestroy(e->graph);
  delete e;
  return GARY_OK;
}

extern "C" int gary_graph_drop_plans(gary_graph *g) {
  GARY_CHECK_ARG(g != nullptr, "graph is NULL");
  gary::free_plans(g);
  return GARY_OK;
}

extern "C" const char *gary_last_error(void) { return gary::g_error; }

extern "C" int gary_abi_version(void) { return GARY_ABI_VERSION; }

extern "C" int gary_graph_upload(const uint64_t *ptr, const uint32_t *idx, uint32_t n,
                                 uint64_t nnz, uint32_t flags, void *stream, gary_graph **out) {
  return guarded("gary_graph_upload", [&] {
    return gary::upload(ptr, idx, n, nnz, flags, gary::as_stream(stream), out, nullptr, 0);
  });
}

extern "C" int gary_batch_upload(const uint64_t *group_off, uint32_t ngroups, const uint64_t *ptr,
                                 const uint32_t *idx, uint32_t n, uint64_t nnz, uint32_t flags,
                                 void *stream, gary_graph **out) {
  GARY_CHECK_ARG(group_off != nullptr && ngroups >= 1, "need ngroups >= 1 and host group offsets");
  GARY_CHECK_ARG(!(flags & GARY_KEEP_IDS), "GARY_KEEP_IDS is not supported for batches");
  return guarded("gary_batch_upload", [&] {
    return gary::upload(ptr, idx, n, nnz, flags, gary::as_stream(stream), out, group_off, ngroups);
  });
}

extern "C" int gary_graph_free(gary_graph *g) {
  if (!g) return GARY_OK;
  return guarded("gary_graph_free", [&] {
    gary::free_plans(g);
    if (g->ev0) cudaEventDestroy(g->ev0);
    if (g->ev1) cudaEventDestroy(g->ev1);
    delete g;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      gary::set_error("gary_graph_free: %s", cudaGetErrorString(e));
      return GARY_ERR_CUDA;
    }
    return GARY_OK;
  });
}

extern "C" int gary_graph_get_info(const gary_graph *g, gary_graph_info *out) {
  GARY_CHECK_ARG(g != nullptr && out != nullptr, "NULL argument");
  out->n = g->n;
  out->max_degree = g->max_degree;
  out->max_out_degree = g->dag.max_len;
  out->relabeled = g->keep_ids ? 0u : 1u;
  out->m = g->dag.m;
  out->adj_words = g->dag.words;
  out->wedges = g->wedges;
  out->out_deg_sq = g->out_deg_sq;
  out->alg_bytes = g->alg_bytes;
  out->device_bytes = g->device_bytes();
  return GARY_OK;
}

extern "C" int gary_graph_device_csr(gary_graph *g, gary_device_csr *out) {
  GARY_CHECK_ARG(g != nullptr && out != nullptr, "NULL argument");
  gary::PaddedCSR &c = g->user_view();
  out->m = g->n;
  out->nnz = c.m;
  out->indPtr = c.indptr.p;
  out->colIdx = c.adj.p;
  out->deg = c.outdeg.p;
  return GARY_OK;
}

extern "C" int gary_graph_device_coo(gary_graph *g, gary_device_coo *out) {
  GARY_CHECK_ARG(g != nullptr && out != nullptr, "NULL argument");
  return guarded("gary_graph_device_coo", [&] {
    gary::PaddedCSR &c = g->user_view();
    GARY_TRY(gary::build_coo(c, nullptr));
    out->m = g->n;
    out->nnz = c.m;
    out->rowIdx = c.coo_row.p;
    out->colIdx = c.coo_col.p;
    out->deg = c.outdeg.p;
    return GARY_OK;
  });
}

extern "C" int gary_graph_download(gary_graph *g, uint64_t *ptr, uint32_t *idx, uint32_t *perm) {
  GARY_CHECK_ARG(g != nullptr, "graph is NULL");
  return guarded("gary_graph_download", [&] { return gary::download(g, ptr, idx, perm, nullptr); });
}

extern "C" int gary_count_async(gary_graph *g, int pattern, int sched, void *stream,
                                uint64_t *d_out) {
  return guarded("gary_count_async", [&] {
    return gary::count_async(g, pattern, sched, gary::as_stream(stream),
                             reinterpret_cast<unsigned long long *>(d_out));
  });
}

extern "C" int gary_count(gary_graph *g, int pattern, int sched, void *stream, uint64_t *out) {
  GARY_CHECK_ARG(out != nullptr, "out is NULL");
  GARY_CHECK_ARG(g != nullptr, "graph is NULL");
  return guarded("gary_count", [&] {
    cudaStream_t s = gary::as_stream(stream);
    GARY_TRY(gary::count_async(g, pattern, sched, s, nullptr, 0, 1, true));
    gary::ResultSlot slot;
    GARY_CUDA(cudaMemcpyAsync(&slot->st, g->last_sched, sizeof(gary::SchedState), cudaMemcpyDeviceToHost, s));
    if (pattern != GARY_PATTERN_TRIANGLE)
      GARY_CUDA(cudaMemcpyAsync(&slot->st.total, g->result.p, 8, cudaMemcpyDeviceToHost, s));
    GARY_CUDA(cudaStreamSynchronize(s));
    const gary::SchedState st = slot->st;
    slot.done();
    GARY_TRY(gary::launch_status(st.error));
    const unsigned long long h = st.total;
    *out = h;
    return GARY_OK;
  });
}

extern "C" int gary_count_shard_async(gary_graph *g, int pattern, int sched, uint32_t shard,
                                      uint32_t nshards, void *stream, uint64_t *d_out) {
  return guarded("gary_count_shard_async", [&] {
    return gary::count_async(g, pattern, sched, gary::as_stream(stream),
                             reinterpret_cast<unsigned long long *>(d_out), shard, nshards);
  });
}

extern "C" int gary_count_status(gary_graph *g, void *stream) {
  GARY_CHECK_ARG(g != nullptr, "graph is NULL");
  GARY_CHECK_ARG(g->last_sched != nullptr, "no count has been launched on this graph");
  return guarded("gary_count_status", [&] {
    cudaStream_t s = gary::as_stream(stream);
    gary::SchedState st{};
    GARY_CUDA(cudaMemcpyAsync(&st, g->last_sched, sizeof(st), cudaMemcpyDeviceToHost, s));
    GARY_CUDA(cudaStreamSynchronize(s));
    return gary::launch_status(st.error);
  });
}

extern "C" int gary_count_last_stats(gary_graph *g, gary_count_stats *out) {
  GARY_CHECK_ARG(g != nullptr && out != nullptr, "NULL argument");
  if (g->last_sched) {
    gary::SchedState st{};
    GARY_CUDA(cudaMemcpy(&st, g->last_sched, sizeof(st), cudaMemcpyDeviceToHost));
    for (int k = 0; k < 4; ++k) g->last.cta_path_tiles[k] = st.cta_path[k];
    g->last.error = st.error;
  }
  if (g->last_span && g->last_span_ctas) {
    // makespan of the launch and the mean time at which its CTAs finished,
    // both from the earliest CTA start
    std::vector<unsigned long long> sp(2ull * g->last_span_ctas);
    GARY_CUDA(cudaMemcpy(sp.data(), g->last_span, sp.size() * 8, cudaMemcpyDeviceToHost));
    unsigned long long t0 = ~0ull, t1 = 0;
    for (uint32_t b = 0; b < g->last_span_ctas; ++b) {
      t0 = std::min(t0, sp[2 * b]);
      t1 = std::max(t1, sp[2 * b + 1]);
    }
    double mean = 0;
    for (uint32_t b = 0; b < g->last_span_ctas; ++b) mean += (double)(sp[2 * b + 1] - t0);
    g->last.makespan_ms = (float)((t1 - t0) * 1e-6);
    g->last.mean_cta_finish_ms = (float)(mean / g->last_span_ctas * 1e-6);
  }
  if (g->last_timed) {
    float ms = 0.f;
    cudaError_t e = cudaEventElapsedTime(&ms, g->ev0, g->ev1);
    if (e == cudaErrorNotReady) {
      cudaGetLastError();
      gary::set_error("the last counting kernel has not finished; synchronise its stream first");
      return GARY_ERR_INVALID;
    }
    if (e != cudaSuccess) {
      gary::set_error("cudaEventElapsedTime: %s", cudaGetErrorString(e));
      cudaGetLastError();
      return GARY_ERR_CUDA;
    }
    g->last.kernel_ms = ms;
  }
  *out = g->last;
  return GARY_OK;
}
