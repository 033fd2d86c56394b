// Hub rows of the triangle plan (hub.cuh).
#include <thrust/copy.h>
#include <thrust/execution_policy.h>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>

#include "hub.cuh"

namespace gary {
namespace {

constexpr int kThreads = 256;
static_assert(kHubMin >= 8, "a cut rounded up to an octet stays inside the list");

inline unsigned grid_for(uint64_t items) {
  const uint64_t b = (items + kThreads - 1) / kThreads, cap = (uint64_t)sm_count() * 16;
  return (unsigned)std::max<uint64_t>(std::min(b, cap), 1);
}

// When at least kHubMin ids of N+(u) are hubs, len[u] = the ids below `first`
// rounded up to whole octets (less than d+(u), for kHubMin >= 8); else all of
// N+(u).  sum[0] += suffix ids such vertices save the walk.
__global__ void k_hub_split(const uint2 *__restrict__ row, const uint32_t *__restrict__ adj, uint32_t n,
                            uint32_t first, uint32_t *__restrict__ len, unsigned long long *__restrict__ sum) {
  unsigned long long mine = 0;
  for (uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; u < n; u += (uint64_t)gridDim.x * blockDim.x) {
    const uint2 r = row[u];
    uint32_t l = r.y;
    if (r.y >= kHubMin) {
      const uint32_t *a = adj + (uint64_t)r.x * 4;
      // the kHubMin-th id from the end tells whether there are enough hubs
      if (a[r.y - kHubMin] >= first) {
        uint32_t b = 0, e = r.y - kHubMin;
        while (b < e) {
          const uint32_t m = (b + e) >> 1;
          if (a[m] < first) b = m + 1;
          else e = m;
        }
        l = (b + 7) & ~7u;
        const unsigned long long h = r.y - l;
        mine += h * (h - 1) / 2 + h * l;
      }
    }
    len[u] = l;
  }
  for (int o = 16; o; o >>= 1) mine += __shfl_xor_sync(kFull, mine, o);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(sum, mine);
}

struct IsCounted {
  const uint2 *row;
  const uint32_t *len;
  __host__ __device__ bool operator()(uint32_t u) const { return len[u] < row[u].y; }
};

// One warp per row: bits of the hub neighbours of its vertex.
__global__ void __launch_bounds__(kThreads)
    k_hub_fill(const uint2 *__restrict__ row, const uint32_t *__restrict__ adj, const uint32_t *__restrict__ len,
               const uint32_t *__restrict__ list, uint32_t n_list, uint32_t first, uint32_t *__restrict__ cut,
               uint32_t *__restrict__ rowof, uint4 *__restrict__ rows) {
  __shared__ __align__(16) uint32_t bits[kThreads / 32][kHubIds / 32];
  const int lane = threadIdx.x & 31;
  uint32_t *mine = bits[threadIdx.x >> 5];
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < (uint64_t)kHubIds + n_list; t += warps) {
    const uint32_t v = t < kHubIds ? first + (uint32_t)t : list[t - kHubIds];
    if (t >= kHubIds && lane == 0) cut[t - kHubIds] = len[v];
    if (t >= kHubIds && v >= first) continue;  // a counted hub: its row is among the first
    const uint2 r = row[v];
    const uint32_t l = v >= first || len[v] < 8 ? 0u : len[v] - 8;  // at or before the first hub neighbour
    reinterpret_cast<uint4 *>(mine)[lane] = make_uint4(0, 0, 0, 0);
    __syncwarp();
    const uint32_t *a = adj + (uint64_t)r.x * 4;
    for (uint32_t i = l + lane; i < r.y; i += 32) {
      const uint32_t p = a[i] - first;
      if (p < kHubIds) atomicOr(&mine[p >> 5], 1u << (p & 31u));
    }
    __syncwarp();
    rows[t * kHubRowQuads + lane] = reinterpret_cast<const uint4 *>(mine)[lane];
    if (t >= kHubIds && lane == 0) rowof[v] = (uint32_t)t;
    __syncwarp();
  }
}

// low[u] = ids of N+(u) below `first`; sum[0] += pairs of N+(u) whose second id
// is not, for the u with a row (at least kAdjMin ids from `first` on).
__global__ void k_adj_split(const uint2 *__restrict__ row, const uint32_t *__restrict__ adj, uint32_t n,
                            uint32_t first, uint32_t *__restrict__ low, unsigned long long *__restrict__ sum) {
  unsigned long long mine = 0;
  for (uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; u < n; u += (uint64_t)gridDim.x * blockDim.x) {
    const uint2 r = row[u];
    const uint32_t *a = adj + (uint64_t)r.x * 4;
    uint32_t b = 0, e = u >= first ? 0u : r.y;
    while (b < e) {
      const uint32_t m = (b + e) >> 1;
      if (a[m] < first) b = m + 1;
      else e = m;
    }
    const unsigned long long h = r.y - b;
    if (h >= kAdjMin) mine += h * (h - 1) / 2 + h * b;
    low[u] = b;
  }
  for (int o = 16; o; o >>= 1) mine += __shfl_xor_sync(kFull, mine, o);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(sum, mine);
}

struct NeedsAdjRow {
  const uint2 *row;
  const uint32_t *low;
  uint32_t first;
  __host__ __device__ bool operator()(uint32_t v) const { return v < first && row[v].y - low[v] >= kAdjMin; }
};

// One warp per row of `words` words: row p of the id first + p, row span + i
// (span = n - first) of list[i].
__global__ void __launch_bounds__(kThreads)
    k_adj_fill(const uint2 *__restrict__ row, const uint32_t *__restrict__ adj, const uint32_t *__restrict__ low,
               const uint32_t *__restrict__ list, uint32_t n_list, uint32_t first, uint32_t span, uint32_t words,
               uint32_t *__restrict__ rowof, uint32_t *__restrict__ rows) {
  __shared__ __align__(16) uint32_t bits[kThreads / 32][kAdjRowIds / 32];
  const int lane = threadIdx.x & 31;
  uint32_t *mine = bits[threadIdx.x >> 5];
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < (uint64_t)span + n_list; t += warps) {
    const uint32_t v = t < span ? first + (uint32_t)t : list[t - span];
    const uint2 r = row[v];
    for (uint32_t i = lane; i < words; i += 32) mine[i] = 0;
    __syncwarp();
    const uint32_t *a = adj + (uint64_t)r.x * 4;
    for (uint32_t i = low[v] + lane; i < r.y; i += 32) {
      const uint32_t p = a[i] - first;
      if (p < span) atomicOr(&mine[p >> 5], 1u << (p & 31u));  // always true for a sorted list
    }
    __syncwarp();
    for (uint32_t i = lane; i < words; i += 32) rows[t * words + i] = mine[i];
    if (t >= span && lane == 0) rowof[v] = (uint32_t)t;
    __syncwarp();
  }
}

// A u more than an eighth of whose neighbours have no row keeps no columns in
// them: low[u] = all its neighbours.  One warp per vertex.
__global__ void k_adj_low(const uint2 *__restrict__ row, const uint32_t *__restrict__ adj, uint32_t n, uint32_t first,
                          const uint32_t *__restrict__ rowof, uint32_t *__restrict__ low) {
  const int lane = threadIdx.x & 31;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t u = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n; u += warps) {
    const uint2 r = row[u];
    const uint32_t l = low[u];
    if (l == 0 || l == r.y) continue;  // only the ids below `first` can lack one
    uint32_t none = 0;
    for (uint32_t i = lane; i < l; i += 32) none += rowof[adj[(uint64_t)r.x * 4 + i]] == kNoHubRow;
    none = __reduce_add_sync(kFull, none);
    if (lane == 0 && none * 8 > r.y) low[u] = r.y;
  }
}

}  // namespace

int build_adj_rows(gary_graph *g, cudaStream_t s, AdjRows &adj) {
  const uint32_t n = g->n, span = std::min(n, kAdjRowIds), first = n - span;
  adj.words = 0;
  if (g->dag.max_len <= kAdjMaxShort) return GARY_OK;
  ScratchAlloc pol_alloc{s};
  auto pol = thrust::cuda::par_nosync(pol_alloc).on(s);
  DevBuf<unsigned long long> sum;
  GARY_TRY(sum.alloc(1, s));
  GARY_TRY(adj.low.alloc_persistent(n));
  GARY_CUDA(cudaMemsetAsync(sum.p, 0, 8, s));
  k_adj_split<<<grid_for(n), kThreads, 0, s>>>(g->dag.row.p, g->dag.adj.p, n, first, adj.low.p, sum.p);
  GARY_CUDA(cudaGetLastError());
  DevBuf<uint32_t> list;
  GARY_TRY(list.alloc(n, s));
  const uint32_t nl = (uint32_t)(thrust::copy_if(pol, thrust::counting_iterator<uint32_t>(0),
                                                 thrust::counting_iterator<uint32_t>(n), list.p,
                                                 NeedsAdjRow{g->dag.row.p, adj.low.p, first}) -
                                 list.p);
  unsigned long long pairs = 0;
  GARY_CUDA(cudaMemcpyAsync(&pairs, sum.p, 8, cudaMemcpyDeviceToHost, s));
  GARY_CUDA(cudaStreamSynchronize(s));
  const uint32_t words = ((span + 127) / 128) * 4;  // whole quads
  const uint64_t bytes = ((uint64_t)span + nl) * words * 4;
  if (pairs < (g->out_deg_sq - g->dag.m) / 16 || !room_for_rows(bytes)) {
    adj.low.release();
    return GARY_OK;
  }
  GARY_TRY(adj.rowof.alloc_persistent(n));
  GARY_TRY(adj.rows.alloc_persistent(bytes / 16));
  GARY_CUDA(cudaMemsetAsync(adj.rowof.p, 0xFF, (uint64_t)n * 4, s));
  k_adj_fill<<<grid_for(((uint64_t)span + nl) * 32), kThreads, 0, s>>>(
      g->dag.row.p, g->dag.adj.p, adj.low.p, list.p, nl, first, span, words, adj.rowof.p,
      reinterpret_cast<uint32_t *>(adj.rows.p));
  k_adj_low<<<grid_for((uint64_t)n * 32), kThreads, 0, s>>>(g->dag.row.p, g->dag.adj.p, n, first, adj.rowof.p, adj.low.p);
  GARY_CUDA(cudaGetLastError());
  adj.first = first;
  adj.words = words;
  return GARY_OK;
}

int build_hub_rows(gary_graph *g, cudaStream_t s, Rows use, HubRows &hub, DevBuf<uint32_t> &len) {
  hub.n_list = 0;
  if (use == Rows::kNone) return GARY_OK;
  const uint32_t n = g->n;
  // A union of graphs is ranked graph by graph: its hubs are not the top ids.
  if (n <= 2 * kHubIds || g->ngroups || g->dag.max_len < kHubMin) return GARY_OK;
  const uint32_t first = n - kHubIds;
  ScratchAlloc pol_alloc{s};
  auto pol = thrust::cuda::par_nosync(pol_alloc).on(s);
  DevBuf<unsigned long long> sum;
  GARY_TRY(sum.alloc(1, s));
  GARY_TRY(len.alloc(n, s));
  GARY_CUDA(cudaMemsetAsync(sum.p, 0, 8, s));
  k_hub_split<<<grid_for(n), kThreads, 0, s>>>(g->dag.row.p, g->dag.adj.p, n, first, len.p, sum.p);
  GARY_CUDA(cudaGetLastError());
  unsigned long long saved = 0;
  GARY_CUDA(cudaMemcpyAsync(&saved, sum.p, 8, cudaMemcpyDeviceToHost, s));
  GARY_CUDA(cudaStreamSynchronize(s));
  const uint64_t probes = (g->out_deg_sq - g->dag.m) / 2;
  if (saved < probes / 8) {
    len.release();
    return GARY_OK;
  }
  GARY_TRY(hub.list.alloc_persistent(n));
  const uint32_t nl = (uint32_t)(thrust::copy_if(pol, thrust::counting_iterator<uint32_t>(0),
                                                 thrust::counting_iterator<uint32_t>(n), hub.list.p,
                                                 IsCounted{g->dag.row.p, len.p}) -
                                 hub.list.p);
  const uint64_t quads = ((uint64_t)kHubIds + nl) * kHubRowQuads;
  const bool fits = (uint64_t)nl + kHubIds < (1u << 27);  // rows are numbered in 27 bits
  if (!fits || (use == Rows::kOptional && !room_for_rows(quads * 16))) {
    hub.no_room = fits;
    hub.list.release();
    len.release();
    return GARY_OK;
  }
  GARY_TRY(hub.cut.alloc_persistent(nl));
  GARY_TRY(hub.rowof.alloc_persistent(n));
  GARY_TRY(hub.rows.alloc_persistent(quads));
  GARY_CUDA(cudaMemsetAsync(hub.rowof.p, 0xFF, (uint64_t)n * 4, s));
  k_hub_fill<<<grid_for(((uint64_t)kHubIds + nl) * 32), kThreads, 0, s>>>(
      g->dag.row.p, g->dag.adj.p, len.p, hub.list.p, nl, first, hub.cut.p, hub.rowof.p, hub.rows.p);
  GARY_CUDA(cudaGetLastError());
  hub.n_list = nl;
  hub.first = first;
  return GARY_OK;
}

bool room_for_rows(uint64_t bytes) {
  if (bytes <= (1ull << 30)) return true;
  size_t free_bytes = 0, total_bytes = 0;
  if (cudaMemGetInfo(&free_bytes, &total_bytes) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (bytes > total_bytes / 8) return false;
  if (bytes > free_bytes / 2) {  // cached blocks may hold the room
    release_cached_memory();
    if (cudaMemGetInfo(&free_bytes, &total_bytes) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
  }
  return bytes <= free_bytes / 2;
}

}  // namespace gary
