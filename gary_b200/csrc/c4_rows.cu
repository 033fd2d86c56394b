// 4-cycles whose highest vertex is a hub (c4_rows.cuh).
#include <thrust/copy.h>
#include <thrust/execution_policy.h>
#include <thrust/fill.h>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>

#include "c4_rows.cuh"
#include "hub.cuh"
#include "warp_ops.cuh"

namespace gary {
namespace {

constexpr int kThreads = 256;

inline unsigned grid_for(uint64_t items) {
  const uint64_t b = (items + kThreads - 1) / kThreads, cap = (uint64_t)sm_count() * 16;
  return (unsigned)std::max<uint64_t>(std::min(b, cap), 1);
}

// ---- bit-sliced counters ----------------------------------------------------
// p[k] holds bit k of 32 counters.  Adds eight rows' bits: full adders into the
// ones, twos and fours, and the last carry rippled up (14 + 2 (S - 3) logic
// operations; one row at a time takes 2 S).
__device__ __forceinline__ uint32_t carry(uint32_t &s, uint32_t a, uint32_t b) {  // s += a + b
  const uint32_t c = (s & a) | (s & b) | (a & b);
  s = s ^ a ^ b;
  return c;
}
template <int S>
__device__ __forceinline__ void add8(uint32_t (&p)[S], uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e,
                                     uint32_t f, uint32_t g, uint32_t h) {
  const uint32_t t1 = carry(p[0], a, b), t2 = carry(p[0], c, d);
  const uint32_t f1 = carry(p[1], t1, t2);
  const uint32_t t3 = carry(p[0], e, f), t4 = carry(p[0], g, h);
  const uint32_t f2 = carry(p[1], t3, t4);
  uint32_t up = carry(p[2], f1, f2);
#pragma unroll
  for (int k = 3; k < S; ++k) {
    const uint32_t x = p[k] & up;
    p[k] ^= up;
    up = x;
  }
}

// A lane's 128 counters: those of its quad of a row.
template <int S>
struct Planes {
  uint32_t p[4][S];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int k = 0; k < S; ++k) p[j][k] = 0;
  }
  // Adds the rows of lanes 0 .. n - 1 (the other lanes name the zero row).
  __device__ __forceinline__ void add_rows(const uint4 *__restrict__ rows, uint32_t row, uint32_t n, int lane) {
#pragma unroll 1
    for (uint32_t k = 0; k < n; k += 8) {
      uint4 x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) x[q] = rows[(uint64_t)__shfl_sync(kFull, row, k + q) * kC4RowQuads + lane];
      add8(p[0], x[0].x, x[1].x, x[2].x, x[3].x, x[4].x, x[5].x, x[6].x, x[7].x);
      add8(p[1], x[0].y, x[1].y, x[2].y, x[3].y, x[4].y, x[5].y, x[6].y, x[7].y);
      add8(p[2], x[0].z, x[1].z, x[2].z, x[3].z, x[4].z, x[5].z, x[6].z, x[7].z);
      add8(p[3], x[0].w, x[1].w, x[2].w, x[3].w, x[4].w, x[5].w, x[6].w, x[7].w);
    }
  }
};

struct RowsView {
  const uint4 *__restrict__ rows;
  const uint32_t *__restrict__ rowof;
  uint32_t first, end, zero;  // zero: the row without a bit
  // the row of x < end: its neighbours in the slab that lie above it
  __device__ __forceinline__ uint32_t row(uint32_t x) const { return x < first ? rowof[x] : x - first; }
};

// How many ids of a sorted list lie below x (all 32 lanes; few lie above).
__device__ __forceinline__ uint32_t ids_below(const uint32_t *l, uint32_t len, uint32_t x, int lane) {
  uint32_t b = len;
  while (b) {
    const uint32_t at = b >= 32 ? b - 32 : 0u;
    const unsigned m = __ballot_sync(kFull, at + lane < b && l[at + lane] >= x);
    b -= __popc(m);
    if (b != at) break;
  }
  return b;
}

// The 32 counters' lower bits below bit `from` of word `word` cleared.
__device__ __forceinline__ uint32_t word_mask(uint32_t word, uint32_t from) {
  const uint32_t b = word * 32;
  return from <= b ? kFull : from >= b + 32 ? 0u : kFull << (from & 31u);
}

template <int S>
__global__ void __launch_bounds__(kThreads)
    k_c4_rows_warp(GraphView sym, RowsView rv, const uint32_t *__restrict__ list, uint32_t count, uint32_t *next,
                   unsigned long long *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  unsigned long long acc = 0;
  while (true) {
    uint32_t c = 0;
    if (lane == 0) c = atomicAdd(next, 1u);
    c = __shfl_sync(kFull, c, 0);
    if (c >= count) break;
    const uint32_t w = list[c];
    if (w + 1 >= rv.end) continue;  // no hub of the slab lies above w
    const uint2 r = sym.row[w];
    const uint32_t *l = sym.adj + (uint64_t)r.x * 4;
    const uint32_t e = ids_below(l, r.y, rv.end, lane);
    Planes<S> pl;
    pl.clear();
    for (uint32_t b = 0; b < e; b += 32)
      pl.add_rows(rv.rows, b + lane < e ? rv.row(l[b + lane]) : rv.zero, min(32u, e - b), lane);
    if (w >= rv.first) {  // hubs above w only
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t m = word_mask(4 * lane + j, w - rv.first + 1);
#pragma unroll
        for (int k = 0; k < S; ++k) pl.p[j][k] &= m;
      }
    }
    // sum of c (c - 1) / 2 over the counters, slice by slice: the squares are
    // 2^2i per bit of slice i and 2^(i+k+1) per common bit of two slices (a
    // lane's sums stay below 128 * 255^2).  Higher slices are often empty.
    uint32_t cc = 0, c1 = 0;
#pragma unroll
    for (int i = 0; i < S; ++i) {
      if (i && !__any_sync(kFull, pl.p[0][i] | pl.p[1][i] | pl.p[2][i] | pl.p[3][i])) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t u = pl.p[j][i];
        c1 += (uint32_t)__popc(u) << i;
        cc += (uint32_t)__popc(u) << (2 * i);
#pragma unroll
        for (int k = 0; k < i; ++k) cc += (uint32_t)__popc(u & pl.p[j][k]) << (i + k + 1);
      }
    }
    acc += (cc - c1) / 2;
  }
  acc = warp_sum_u64(acc);
  if (lane == 0 && acc) atomicAdd(out, acc);
}

// Vertices of 256 neighbours and more: the CTA's warps take 32 neighbours at a
// time into slices of their own and add these to shared 32-bit counters before
// they can overflow.  Counter of bit b of word 4 lane + j: [(32 j + b) * 32 + lane].
constexpr uint32_t kSliceRows = 255;  // rows 8 slices count

__device__ __forceinline__ void flush(Planes<8> &pl, uint32_t *cnt, int lane) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
#pragma unroll 2
    for (int b = 0; b < 8; ++b) {
      // the counts of bits b, b + 8, b + 16 and b + 24, a byte each
      uint32_t v = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) v |= ((pl.p[j][k] >> b) & 0x01010101u) << k;
      uint32_t *c = cnt + (32 * j + b) * 32 + lane;
      if (v & 0xFFu) atomicAdd(c, v & 0xFFu);
      if (v & 0xFF00u) atomicAdd(c + 8 * 32, (v >> 8) & 0xFFu);
      if (v & 0xFF0000u) atomicAdd(c + 16 * 32, (v >> 16) & 0xFFu);
      if (v >> 24) atomicAdd(c + 24 * 32, v >> 24);
    }
  }
  pl.clear();
}

__global__ void __launch_bounds__(kThreads)
    k_c4_rows_cta(GraphView sym, RowsView rv, const uint32_t *__restrict__ list, uint32_t count, uint32_t *next,
                  unsigned long long *__restrict__ out) {
  __shared__ uint32_t cnt[kC4RowIds];
  __shared__ uint32_t s_i, s_next;
  const int lane = threadIdx.x & 31;
  unsigned long long acc = 0;
  while (true) {
    if (threadIdx.x == 0) {
      s_i = atomicAdd(next, 1u);
      s_next = 0;
    }
    for (uint32_t i = threadIdx.x; i < kC4RowIds; i += kThreads) cnt[i] = 0;
    __syncthreads();
    const uint32_t c = s_i;
    if (c >= count) break;
    const uint32_t w = list[count - 1 - c];  // the largest ranks, with the most neighbours, first
    if (w + 1 < rv.end) {
      const uint2 r = sym.row[w];
      const uint32_t *l = sym.adj + (uint64_t)r.x * 4;
      const uint32_t e = ids_below(l, r.y, rv.end, lane);
      Planes<8> pl;
      pl.clear();
      uint32_t n = 0;  // rows since the last flush
      while (true) {
        uint32_t b = 0;
        if (lane == 0) b = atomicAdd(&s_next, 32u);
        b = __shfl_sync(kFull, b, 0);
        if (b >= e) break;
        if (n + 32 > kSliceRows) {
          flush(pl, cnt, lane);
          n = 0;
        }
        pl.add_rows(rv.rows, b + lane < e ? rv.row(l[b + lane]) : rv.zero, min(32u, e - b), lane);
        n += 32;
      }
      if (n) flush(pl, cnt, lane);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kC4RowIds; i += kThreads) {
      const uint32_t bit = i >> 5, id = (4 * (i & 31u) + (bit >> 5)) * 32 + (bit & 31u);  // hub id - first
      const unsigned long long u = cnt[i];
      if (u > 1 && (w < rv.first || id > w - rv.first)) acc += u * (u - 1) / 2;
    }
    __syncthreads();
  }
  acc = warp_sum_u64(acc);
  if (lane == 0 && acc) atomicAdd(out, acc);
}

// ---- build --------------------------------------------------------------------
// Where the ids of [first, end) lie in a sorted list.
__device__ __forceinline__ uint2 slab_part(const uint32_t *l, uint32_t len, uint32_t first, uint32_t end) {
  auto lower = [&](uint32_t x) {
    uint32_t b = 0, e = len;
    while (b < e) {
      const uint32_t m = (b + e) >> 1;
      if (l[m] < x) b = m + 1;
      else e = m;
    }
    return b;
  };
  return make_uint2(lower(first), lower(end));
}

// One warp per row.
__global__ void __launch_bounds__(kThreads)
    k_c4_fill(const uint2 *__restrict__ srow, const uint32_t *__restrict__ sadj, const uint32_t *__restrict__ list,
              uint32_t n_list, uint32_t first, uint32_t end, uint32_t *__restrict__ rowof, uint4 *__restrict__ rows) {
  __shared__ __align__(16) uint32_t bits[kThreads / 32][kC4RowIds / 32];
  const int lane = threadIdx.x & 31;
  uint32_t *mine = bits[threadIdx.x >> 5];
  const uint32_t span = end - first;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t <= (uint64_t)span + n_list; t += warps) {
    if (t == (uint64_t)span + n_list) {  // the row without a bit
      rows[t * kC4RowQuads + lane] = make_uint4(0, 0, 0, 0);
      break;
    }
    const bool in = t < span;
    const uint32_t v = in ? first + (uint32_t)t : list[t - span];
    const uint2 r = srow[v];
    const uint32_t *l = sadj + (uint64_t)r.x * 4;
    const uint2 part = slab_part(l, r.y, first, end);
    reinterpret_cast<uint4 *>(mine)[lane] = make_uint4(0, 0, 0, 0);
    __syncwarp();
    for (uint32_t i = part.x + lane; i < part.y; i += 32) {
      const uint32_t p = l[i] - first;
      if (p < span && (!in || p > (uint32_t)t)) atomicOr(&mine[p >> 5], 1u << (p & 31u));
    }
    __syncwarp();
    rows[t * kC4RowQuads + lane] = reinterpret_cast<const uint4 *>(mine)[lane];
    if (!in && lane == 0) rowof[v] = (uint32_t)t;
    __syncwarp();
  }
}

// Per slab k (ids from end[k] - kC4RowIds on): stat[k] += wedges under its ids;
// stat[kC4MaxSlabs] += rows a slab's pass reads (nearly every neighbour).
struct SlabEnds {
  uint32_t end[kC4MaxSlabs];
  int slabs;
};
__global__ void k_c4_rows_stat(const uint2 *__restrict__ srow, const uint32_t *__restrict__ sadj,
                               const uint32_t *__restrict__ dplus, uint32_t n, SlabEnds se,
                               unsigned long long *__restrict__ stat) {
  unsigned long long rows = 0, wedges[kC4MaxSlabs] = {0};
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const uint2 r = srow[v];
    if (r.y >= 2) rows += r.y;
    // N(v) holds low ids below v and d+ above: the i-th of the latter, u, has
    // low + i wedges u - v - w
    const uint32_t *l = sadj + (uint64_t)r.x * 4;
    const unsigned long long low = r.y - dplus[v];
    uint32_t b = r.y;
#pragma unroll
    for (int k = 0; k < kC4MaxSlabs; ++k) {
      if (k >= se.slabs || b <= low) break;
      const uint32_t end = se.end[k], first = end > kC4RowIds ? end - kC4RowIds : 0u;
      if (l[b - 1] < first) continue;
      uint32_t x = (uint32_t)low, e = b;
      while (x < e) {
        const uint32_t m = (x + e) >> 1;
        if (l[m] < first) x = m + 1;
        else e = m;
      }
      wedges[k] += (unsigned long long)(b - x) * (x + b - 1) / 2;  // positions x .. b - 1
      b = x;
    }
  }
#pragma unroll
  for (int k = 0; k < kC4MaxSlabs; ++k) {
    const unsigned long long x = warp_sum_u64(wedges[k]);
    if ((threadIdx.x & 31) == 0 && x) atomicAdd(&stat[k], x);
  }
  rows = warp_sum_u64(rows);
  if ((threadIdx.x & 31) == 0 && rows) atomicAdd(&stat[kC4MaxSlabs], rows);
}

// Vertices below `first` with a neighbour in [first, end).
struct TouchesSlab {
  const uint2 *row;
  const uint32_t *adj;
  uint32_t first, end;
  __host__ __device__ bool operator()(uint32_t v) const {
    if (v >= first) return false;
    const uint2 r = row[v];
    const uint32_t *l = adj + (uint64_t)r.x * 4;
    uint32_t b = 0, e = r.y;
    while (b < e) {
      const uint32_t m = (b + e) >> 1;
      if (l[m] < first) b = m + 1;
      else e = m;
    }
    return b < r.y && l[b] < end;
  }
};

struct DegreeIn {
  const uint2 *row;
  uint32_t lo, hi;
  __host__ __device__ bool operator()(uint32_t v) const { return row[v].y >= lo && row[v].y <= hi; }
};

}  // namespace

int build_c4_rows(gary_graph *g, cudaStream_t s, Rows use, C4Rows &r) {
  const uint32_t n = g->n;
  const uint2 *row = g->sym.row.p;
  const uint32_t *adj = g->sym.adj.p, *dplus = g->dag.outdeg.p;
  r.slabs = 0;
  r.lowest = n;
  r.shared = use != Rows::kNone;
  if (use == Rows::kNone) return GARY_OK;
  ScratchAlloc pol_alloc{s};
  auto pol = thrust::cuda::par_nosync(pol_alloc).on(s);
  SlabEnds se{};
  for (uint32_t end = n; end && se.slabs < kC4MaxSlabs; end = end > kC4RowIds ? end - kC4RowIds : 0)
    se.end[se.slabs++] = end;
  DevBuf<unsigned long long> stat;
  GARY_TRY(stat.alloc(kC4MaxSlabs + 1, s));
  GARY_CUDA(cudaMemsetAsync(stat.p, 0, stat.bytes(), s));
  k_c4_rows_stat<<<grid_for(n), kThreads, 0, s>>>(row, adj, dplus, n, se, stat.p);
  GARY_CUDA(cudaGetLastError());
  unsigned long long h[kC4MaxSlabs + 1];
  GARY_CUDA(cudaMemcpyAsync(h, stat.p, sizeof(h), cudaMemcpyDeviceToHost, s));
  GARY_CUDA(cudaStreamSynchronize(s));
  uint64_t used = 0;  // by all slabs' rows
  const uint64_t shard_most = std::max(kC4ShardWordBytes * g->dag.words, kC4ShardLeast);
  DevBuf<uint32_t> list;
  GARY_TRY(list.alloc(n, s));
  for (int k = 0; k < se.slabs && h[k] && h[k] / kC4RowWedges >= h[kC4MaxSlabs]; ++k) {
    C4Slab &sl = r.slab[k];
    sl.end = se.end[k];
    sl.first = sl.end > kC4RowIds ? sl.end - kC4RowIds : 0;
    const uint32_t span = sl.end - sl.first;
    const uint32_t nl = (uint32_t)(thrust::copy_if(pol, thrust::counting_iterator<uint32_t>(0),
                                                   thrust::counting_iterator<uint32_t>(n), list.p,
                                                   TouchesSlab{row, adj, sl.first, sl.end}) - list.p);
    const uint64_t bytes = ((uint64_t)span + nl + 1) * kC4RowQuads * 16;
    const bool in_shards = used + bytes <= shard_most;
    const bool take = use == Rows::kRequired ? in_shards : room_for_rows(used + bytes);
    // both kinds of plan have this slab
    r.shared = r.shared && take && in_shards;
    if (!take) break;
    used += bytes;
    GARY_TRY(sl.rowof.alloc_persistent(n));
    GARY_TRY(sl.rows.alloc_persistent(bytes / 16));
    sl.zero = span + nl;
    thrust::fill(pol, sl.rowof.p, sl.rowof.p + n, sl.zero);
    k_c4_fill<<<grid_for(((uint64_t)span + nl) * 32), kThreads, 0, s>>>(row, adj, list.p, nl, sl.first, sl.end, sl.rowof.p,
                                                                      sl.rows.p);
    GARY_CUDA(cudaGetLastError());
    r.lowest = sl.first;
    r.slabs = k + 1;
  }
  if (!r.slabs) return GARY_OK;
  GARY_TRY(r.queue.alloc_persistent(3 * kC4MaxSlabs));
  GARY_TRY(r.list.alloc_persistent(n));
  auto pick = [&](uint32_t *to, uint32_t lo, uint32_t hi) {
    return (uint32_t)(thrust::copy_if(pol, thrust::counting_iterator<uint32_t>(0), thrust::counting_iterator<uint32_t>(n),
                                      to, DegreeIn{row, lo, hi}) - to);
  };
  r.n5 = pick(r.list.p, 2, 31);
  r.n8 = pick(r.list.p + r.n5, 32, 255);
  r.n32 = pick(r.list.p + r.n5 + r.n8, 256, 0xFFFFFFFFu);
  return GARY_OK;
}

int launch_c4_rows(gary_graph *g, const C4Rows &r, unsigned long long *d_out, cudaStream_t s, uint32_t shard,
                   uint32_t nshards) {
  if (!r.slabs) return GARY_OK;
  const GraphView sym{g->n, g->sym.row.p, g->sym.adj.p, true};
  GARY_CUDA(cudaMemsetAsync(r.queue.p, 0, 3 * kC4MaxSlabs * 4, s));
  for (int k = 0; k < r.slabs; ++k) {
    const C4Slab &sl = r.slab[k];
    const RowsView rv{sl.rows.p, sl.rowof.p, sl.first, sl.end, sl.zero};
    auto run = [&](auto kern, uint32_t begin, uint32_t total, int q) -> int {
      const uint32_t lo = (uint32_t)((uint64_t)total * shard / nshards), hi = (uint32_t)((uint64_t)total * (shard + 1) / nshards);
      if (lo == hi) return GARY_OK;
      int per_sm = 0;
      GARY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, 0));
      kern<<<(unsigned)(sm_count() * std::max(per_sm, 1)), kThreads, 0, s>>>(sym, rv, r.list.p + begin + lo, hi - lo,
                                                                             r.queue.p + 3 * k + q, d_out);
      GARY_CUDA(cudaGetLastError());
      return GARY_OK;
    };
    // the vertices of most neighbours first
    GARY_TRY(run(k_c4_rows_cta, r.n5 + r.n8, r.n32, 0));
    GARY_TRY(run(k_c4_rows_warp<8>, r.n5, r.n8, 1));
    GARY_TRY(run(k_c4_rows_warp<5>, 0, r.n5, 2));
  }
  return GARY_OK;
}

}  // namespace gary
