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

}  // namespace

int build_hub_rows(gary_graph *g, cudaStream_t s, HubRows &hub, DevBuf<uint32_t> &len) {
  hub.n_list = 0;
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
  if ((uint64_t)nl + kHubIds >= (1u << 27)) {  // rows are numbered in 27 bits
    hub.list.release();
    len.release();
    return GARY_OK;
  }
  GARY_TRY(hub.cut.alloc_persistent(nl));
  GARY_TRY(hub.rowof.alloc_persistent(n));
  GARY_TRY(hub.rows.alloc_persistent(((uint64_t)kHubIds + nl) * kHubRowQuads));
  GARY_CUDA(cudaMemsetAsync(hub.rowof.p, 0xFF, (uint64_t)n * 4, s));
  k_hub_fill<<<grid_for(((uint64_t)kHubIds + nl) * 32), kThreads, 0, s>>>(
      g->dag.row.p, g->dag.adj.p, len.p, hub.list.p, nl, first, hub.cut.p, hub.rowof.p, hub.rows.p);
  GARY_CUDA(cudaGetLastError());
  hub.n_list = nl;
  hub.first = first;
  return GARY_OK;
}

}  // namespace gary
