// Triangle counting on the degree-oriented DAG (pattern K3).
//
// Reference: graph_query::triangleCountHom (include/kernels/GraphQueryHom.cuh:15-43)
// launches one warp per oriented COO edge (u,v) and counts |N+(u) & N+(v)| by
// per-key binary search, one key per lane.  The total is the same number
//     T = sum over (u,v) in E+ of |N+(u) & N+(v)|,
// computed here from the MIDDLE vertex of each triangle u < v < w (ids are
// degree ranks, so every list is sorted in orientation order):
//
//     T = sum over v of  sum over in-edges u->v of |S(u,v) & N+(v)|,
//     S(u,v) = the part of N+(u) after v.
//
// On skewed graphs the suffix ids among the top 4096 are first taken out and
// counted by bit rows (hub.cuh).  For the rest, one warp (or CTA) holds N+(v) as
// a shared-memory bitmap (when its id range is short), hash or pair set
// (pair_set.cuh; the lists of two octets and less need no set), and streams the suffixes S(u,v) of all in-edges of v
// with 16-byte loads over the padded lists, all lanes busy.  The probe count
// is sum over u of C(d+(u), 2), 3.5-4x fewer than streaming N+(v) for every
// edge (sum of d+(v)) on RMAT graphs, and every read is a coalesced sweep.
//
// Work is cut into tiles of bounded probe count over the in-edge index and
// served by a persistent scheduler: CTA tiles (large N+(v)) first, then warp
// tiles.
#include <cub/cub.cuh>
#include <thrust/binary_search.h>
#include <thrust/copy.h>
#include <thrust/execution_policy.h>
#include <thrust/fill.h>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/reverse_iterator.h>
#include <thrust/iterator/transform_iterator.h>
#include <thrust/reduce.h>
#include <thrust/scan.h>
#include <thrust/transform.h>
#include <thrust/transform_reduce.h>

#include <algorithm>
#include <memory>
#include <numeric>

#include "bulk.cuh"
#include "mlp.cuh"
#include "graph.cuh"
#include "pair_set.cuh"
#include "tc.cuh"
#include "warp_ops.cuh"

namespace gary {

// ---------------------------------------------------------------------------
// Plan: in-edge index + tiles
namespace {

constexpr int kThreads = 256;

inline unsigned grid_for(uint64_t items) {
  uint64_t b = (items + kThreads - 1) / kThreads;
  uint64_t cap = (uint64_t)sm_count() * 16;
  return (unsigned)std::max<uint64_t>(std::min(b, cap), 1);
}

inline int bits_for(uint64_t x) {
  int b = 0;
  while (b < 64 && (x - 1) >> b) ++b;
  return std::max(b, 1);
}

__host__ __device__ __forceinline__ uint64_t min_u64(uint64_t a, uint64_t b) { return a < b ? a : b; }

struct MinU64 {
  __host__ __device__ uint64_t operator()(uint64_t a, uint64_t b) const { return a < b ? a : b; }
};

// The records of the padded words w of N+(u): the suffix after v = adj[w], up to
// len[u] (null: the whole list), keyed by v.  They are written in an order that
// follows from the lists' size alone (tile_stride), so that the sort after it
// (stable, by v) moves records only (with hub rows a third of the words hold one at
// RMAT-20 ef16) and leaves every vertex's records in the same order in every plan
// of the graph: split vertices are cut by position, and shards of one count come
// from plans that other processes built.  (Appended in whatever order tiles ran,
// shards of two plans counted some records twice and others never.)
// Two passes, tile by tile of kCandTile words.  This one marks the words with a
// record, a bit each, so that d+(v), a scattered read, is not read twice, and
// counts them: tiles[q] of the q-th tile.  total[0] += the suffix ids past len[u],
// total[1] += the records.  A first count, plan included, takes up to 15 us
// more than with one appending pass (RMAT-16 ef16 0.446 / 0.450 ms, RMAT-20 1.521 /
// 1.537, RMAT-22 6.03 / 6.05).
constexpr int kCandPer = 8;
constexpr uint32_t kCandTile = kThreads * kCandPer;
constexpr int kCandWarps = kThreads / 32;

// Suffix ids after position pos of a list cut to `end` ids.
__device__ __forceinline__ uint32_t kept_suffix(uint32_t end, uint64_t pos) {
  return end > (uint32_t)pos + 1 ? end - (uint32_t)pos - 1 : 0u;
}

__global__ void __launch_bounds__(kThreads)
    k_in_mark(const uint2 *__restrict__ row, const uint32_t *__restrict__ adj, const uint32_t *__restrict__ rowid,
              uint64_t words, uint64_t stride, const uint32_t *__restrict__ len, uint32_t *__restrict__ marks,
              uint64_t *__restrict__ tiles, unsigned long long *__restrict__ total) {
  __shared__ uint32_t s_n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long mine = 0, records = 0;
  const uint64_t nt = (words + kCandTile - 1) / kCandTile;
  for (uint64_t q = blockIdx.x; q < nt; q += gridDim.x) {
    const uint64_t t = q * stride % nt;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < kCandPer; ++i) {
      const uint64_t w = t * kCandTile + (uint64_t)i * kThreads + threadIdx.x;
      bool has = false;
      if (w < words) {
        const uint32_t u = rowid[w];
        const uint2 r = row[u];
        const uint64_t pos = w - (uint64_t)r.x * 4;
        if (pos + 1 < r.y && row[adj[w]].y) {
          const uint32_t keep = kept_suffix(len ? len[u] : r.y, pos);
          mine += r.y - (uint32_t)pos - 1 - keep;
          has = keep != 0;
        }
      }
      const unsigned m = __ballot_sync(kFull, has);
      if (lane == 0) marks[(t * kCandPer + i) * kCandWarps + warp] = m;
      c += __popc(m);
    }
    if (lane == 0) atomicAdd(&s_n, c);
    __syncthreads();
    if (threadIdx.x == 0) {
      tiles[q] = s_n;
      records += s_n;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0 && records) atomicAdd(&total[1], records);
  if (len) {
    mine = warp_sum_u64(mine);
    if (lane == 0 && mine) atomicAdd(&total[0], mine);
  }
}

// Tile q of the record order is tile q * stride mod nt of the words.  From 2^16
// tiles (512 MB of lists, four times the L2) consecutive tiles come from all over
// the graph, smaller lists are taken in word order: ms a count appended as before /
// in word order / strided, RMAT-24 ef32 64.2 / 65.0 / 61.7, RMAT-24 ef16 20.08 /
// 20.22 / 19.98, RMAT-23 ef16 7.85 / 7.87 / 7.78; RMAT-22 ef32 8.65 / 8.62 / 8.67,
// RMAT-22 ef16 3.010 / 3.020 / 3.059, RMAT-20 0.512 / 0.511 / 0.513.
uint64_t tile_stride(uint64_t nt) {
  if (nt < (1u << 16)) return 1;
  uint64_t k = (uint64_t)(0.6180339887 * (double)nt) | 1;  // golden section: even spread
  while (std::gcd(k, nt) != 1) k += 2;
  return k;
}

// Up to so many tiles, every CTA adds up the counts before its own itself; past
// them (RMAT-21 and larger) that reads more than a scan's launches cost (a first
// count with a scan at any size: RMAT-16 0.478 ms, RMAT-20 1.570).
constexpr uint64_t kCandFewTiles = 1u << 14;

// The second pass writes the marked words' records, a CTA those of tiles that
// follow one another in the order.  tiles: each tile's offset (scanned) or its count.
__global__ void __launch_bounds__(kThreads)
    k_in_candidates(const uint2 *__restrict__ row, const uint32_t *__restrict__ adj,
                    const uint32_t *__restrict__ rowid, uint64_t words, uint64_t stride,
                    const uint32_t *__restrict__ len, const uint32_t *__restrict__ marks, const uint64_t *__restrict__ tiles, bool scanned,
                    uint32_t *__restrict__ keys, uint2 *__restrict__ vals) {
  __shared__ uint32_t at[kCandPer * kCandWarps];
  __shared__ unsigned long long s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t nt = (words + kCandTile - 1) / kCandTile, per = (nt + gridDim.x - 1) / gridDim.x;
  const uint64_t t0 = blockIdx.x * per, t1 = min_u64(t0 + per, nt);
  if (t0 >= t1) return;
  if (threadIdx.x == 0) s_base = scanned ? tiles[t0] : 0;
  __syncthreads();
  if (!scanned) {
    unsigned long long before = 0;
    for (uint64_t j = threadIdx.x; j < t0; j += kThreads) before += tiles[j];
    before = warp_sum_u64(before);
    if (lane == 0 && before) atomicAdd(&s_base, before);
    __syncthreads();
  }
  for (uint64_t q = t0; q < t1; ++q) {
    const uint64_t t = q * stride % nt;
    const unsigned long long base = s_base;
    uint32_t all = 0;  // the tile's records
    if (warp == 0) {   // where each warp's part of each row of the tile goes
      const uint32_t *m = marks + t * (kCandPer * kCandWarps);
      const uint32_t a = __popc(m[2 * lane]), b = __popc(m[2 * lane + 1]);
      const uint32_t incl = warp_inclusive_sum(a + b, lane);
      at[2 * lane] = incl - a - b;
      at[2 * lane + 1] = incl - b;
      all = __shfl_sync(kFull, incl, 31);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kCandPer; ++i) {
      const unsigned m = marks[(t * kCandPer + i) * kCandWarps + warp];
      if ((m >> lane) & 1u) {
        const uint64_t w = t * kCandTile + (uint64_t)i * kThreads + threadIdx.x;
        const uint32_t u = rowid[w];
        const uint2 r = row[u];
        const uint64_t o = base + at[i * kCandWarps + warp] + __popc(m & ((1u << lane) - 1u));
        keys[o] = adj[w];
        vals[o] = make_uint2((uint32_t)(w + 1), kept_suffix(len ? len[u] : r.y, w - (uint64_t)r.x * 4));
      }
    }
    if (threadIdx.x == 0) s_base = base + all;
    __syncthreads();
  }
  static_assert(kCandPer * kCandWarps == 64, "two entries a lane");
}

__global__ void k_in_heads(const uint32_t *__restrict__ keys, uint64_t m,
                           uint64_t *__restrict__ inptr) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = keys[i];
    if (i == 0 || keys[i - 1] != v) inptr[v] = i;
  }
}

// work[v] = sum of suffix lengths of v's in-edges (segmented warp scan; keys sorted).
__global__ void k_in_work(const uint32_t *__restrict__ keys, const uint2 *__restrict__ vals,
                          uint64_t m, unsigned long long *__restrict__ work) {
  const int lane = threadIdx.x & 31;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = blockIdx.x * (uint64_t)blockDim.x; base < m; base += stride) {
    const uint64_t i = base + threadIdx.x;
    const bool ok = i < m;
    const uint32_t v = ok ? keys[i] : 0xFFFFFFFFu;
    unsigned long long x = ok ? vals[i].y : 0ull;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(kFull, x, o);
      const uint32_t tv = __shfl_up_sync(kFull, v, o);
      if (lane >= o && tv == v) x += t;
    }
    const uint32_t nv = __shfl_down_sync(kFull, v, 1);
    if (ok && (lane == 31 || nv != v) && x) atomicAdd(&work[v], x);
  }
}

// pcost (optional): predicted cycles of a warp-class vertex, with tile target
// tw_pred in the same unit; without it, costs are probe counts.  tw_pred cycles
// stand for warp_tile_cost probes.
__global__ void k_classify(const uint2 *__restrict__ row, const uint32_t *__restrict__ adj,
                           const uint64_t *__restrict__ work,
                           const uint64_t *__restrict__ inptr, uint32_t n, PlanParams pp,
                           const uint64_t *__restrict__ pcost, uint64_t tw_pred,
                           uint8_t *__restrict__ vclass, uint64_t *__restrict__ costL,
                           uint32_t *__restrict__ kW, uint32_t *__restrict__ kC) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const uint2 rv = row[v];
    const uint32_t dv = rv.y;
    const uint64_t nin = inptr[v + 1] - inptr[v];
    uint8_t cls = kClassNone;
    uint64_t cl = 0;
    uint32_t kw = 0, kc = 0;
    if (dv && nin) {
      // a warp holds N+(v) as a bitmap when its id span is short, else as
      // buckets when d+(v) <= warp_cap; otherwise the CTA shares one set
      const uint32_t span = adj[(uint64_t)rv.x * 4 + dv - 1] - adj[(uint64_t)rv.x * 4];
      const bool bitmap = span <= bitmap_max_span(kWarpTableSlots);
      const bool warp_fits = bitmap || dv <= pp.warp_cap;
      const uint64_t build = bitmap ? (span >> 5) + dv : 4ull * dv;
      const bool pred = pcost && warp_fits;
      // probe cost; a tiny vertex has no set, and each record costs it at
      // least an octet
      const uint64_t cp = dv <= kTinyOut ? work[v] + 8 * nin + 16 : work[v] + build + pp.vertex_overhead;
      // learned: predicted cycles, but never below the probe cost scaled to
      // the same tile target, so that no tile outgrows a plain one (a vertex
      // the model under-rates would otherwise end the launch alone).  The model
      // knows tiny vertices with a set only: theirs is the scaled probe cost.
      auto scaled = [&](uint64_t probes) { return pred ? probes * tw_pred / pp.warp_tile_cost : probes; };
      const uint64_t c = pred && dv > kTinyOut ? max(pcost[v] + 1, scaled(cp)) : max(scaled(cp), (uint64_t)1);
      const uint64_t tw = pred ? tw_pred : pp.warp_tile_cost;
      if (!warp_fits) {
        cls = kClassCta;
        kc = (uint32_t)min_u64((c + pp.cta_tile_cost - 1) / pp.cta_tile_cost, nin);
      } else if (c > tw) {
        cls = kClassSplit;
        const uint64_t piece = max(tw, scaled(pp.split_floor * dv));  // every piece builds the set again
        kw = (uint32_t)min_u64((c + piece - 1) / piece, nin);
      } else {
        cls = kClassLight;
        cl = c;
      }
    }
    vclass[v] = cls;
    costL[v] = cl;
    kW[v] = kw;
    kC[v] = kc;
  }
}

// off[] holds exclusive tile offsets (n+1 entries): vertex v owns tiles
// off[v] .. off[v+1], splitting its in-edge list evenly.
__global__ void k_fill_split_tiles(const uint64_t *__restrict__ inptr, uint32_t n,
                                   const uint32_t *__restrict__ off, Tile *__restrict__ tiles) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t kk = off[v + 1] - off[v];
    if (!kk) continue;
    const uint64_t nin = inptr[v + 1] - inptr[v];
    const uint32_t o = off[v];
    for (uint32_t i = 0; i < kk; ++i) {
      Tile t;
      t.v0 = (uint32_t)v;
      t.v1 = (uint32_t)v + 1;
      t.j0 = (uint32_t)((uint64_t)i * nin / kk);
      t.j1 = (uint32_t)((uint64_t)(i + 1) * nin / kk);
      tiles[o + i] = t;
    }
  }
}

struct GroupTarget {
  uint64_t tw;
  __host__ __device__ uint64_t operator()(uint64_t g) const { return g * tw; }
};

struct IsLight {
  const uint8_t *vclass;
  __host__ __device__ bool operator()(uint32_t v) const { return vclass[v] == kClassLight; }
};

// Predicted cycles of a vertex that is counted with a set.
struct SetCycles {
  const uint2 *row;
  const uint64_t *pcost;
  __host__ __device__ uint64_t operator()(uint32_t v) const { return row[v].y > kTinyOut ? pcost[v] : 0u; }
};

struct LightCost {
  const uint64_t *cost;
  __host__ __device__ uint64_t operator()(uint32_t v) const { return cost[v]; }
};

// Group tiles over the compacted light-vertex list: tile g covers list
// positions [starts[g], starts[g+1]).
__global__ void k_fill_group_tiles(const uint32_t *__restrict__ starts, uint64_t G, uint32_t L,
                                   Tile *__restrict__ tiles) {
  for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < G;
       g += (uint64_t)gridDim.x * blockDim.x) {
    Tile t;
    t.v0 = starts[g];
    t.v1 = g + 1 < G ? starts[g + 1] : L;
    t.j0 = 0;
    t.j1 = kGroupTile;
    tiles[g] = t;
  }
}

}  // namespace

// Cost-model features of middle vertex v (all log2(1 + .)):
//   x0 degree, x1 mean in-edge suffix length (the other endpoints' remaining
//   out-degree), x2 = x0 - x1 (their log ratio), x3 out-degree d+(v),
//   x4 id span of N+(v), x5 number of in-edge records.
// legal[v]: bit k when variant k can run v on a warp (0: not a warp vertex).
__global__ void k_features(const uint2 *__restrict__ row, const uint32_t *__restrict__ adj,
                           const uint32_t *__restrict__ rdeg, const uint64_t *__restrict__ work,
                           const uint64_t *__restrict__ inptr, uint32_t n, uint32_t warp_cap,
                           float *__restrict__ x, uint8_t *__restrict__ legal) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const uint2 rv = row[v];
    const uint32_t d = rv.y;
    const uint64_t nin = inptr[v + 1] - inptr[v];
    const uint32_t span = d ? adj[(uint64_t)rv.x * 4 + d - 1] - adj[(uint64_t)rv.x * 4] : 0u;
    const bool warp_fits = span <= bitmap_max_span(kWarpTableSlots) || d <= warp_cap;
    uint32_t lg = 0;
    if (d && nin && warp_fits)
      for (uint32_t k = 0; k < 4; ++k)
        if (variant_legal(k, d, span)) lg |= 1u << k;
    legal[v] = (uint8_t)lg;
    const float x0 = log2f(1.f + (float)rdeg[v]);
    const float x1 = log2f(1.f + (float)work[v] / (float)(nin ? nin : 1));
    float *xv = x + v * kMlpIn;
    xv[0] = x0;
    xv[1] = x1;
    xv[2] = x0 - x1;
    xv[3] = log2f(1.f + (float)d);
    xv[4] = log2f(1.f + (float)span);
    xv[5] = log2f(1.f + (float)nin);
  }
}

// The cost model over every warp vertex: variant = argmin over legal
// variants of predicted log2 cycles, pcost = predicted cycles of that variant.
__global__ void k_predict(const float *__restrict__ params, const float *__restrict__ x,
                          const uint8_t *__restrict__ legal, uint32_t n, uint8_t *__restrict__ variant,
                          uint64_t *__restrict__ pcost) {
  __shared__ float P[kMlpParams];
  for (int i = threadIdx.x; i < kMlpParams; i += blockDim.x) P[i] = params[i];
  __syncthreads();
  float h1[kMlpH1], h2[kMlpH2];
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t lg = legal[v];
    if (!lg) {
      variant[v] = 0xFF;
      pcost[v] = 0;
      continue;
    }
    float xi[kMlpIn], y[kMlpOut];
#pragma unroll
    for (int f = 0; f < kMlpIn; ++f) xi[f] = (x[v * kMlpIn + f] - P[kMlpMuX + f]) / P[kMlpSdX + f];
    mlp_forward_one(P, xi, h1, h2, y);
    uint32_t best = 0xFF;
    float by = 0.f;
#pragma unroll
    for (int k = 0; k < kMlpOut; ++k) {
      const float yk = y[k] * P[kMlpSdY + k] + P[kMlpMuY + k];
      if (((lg >> k) & 1) && (best == 0xFF || yk < by)) {
        best = k;
        by = yk;
      }
    }
    variant[v] = (uint8_t)best;
    pcost[v] = (uint64_t)exp2f(fminf(fmaxf(by, 0.f), 40.f));
  }
}

namespace {

int build_in_index(gary_graph *g, cudaStream_t s, const DevBuf<uint32_t> &len, InIndex &in) {
  const uint32_t n = g->n;
  const uint64_t W = g->dag.words;
  if (W >= (1ull << 32)) {
    set_error("graph too large for the in-edge index (%llu padded words)", (unsigned long long)W);
    return GARY_ERR_UNSUPPORTED;
  }
  ScratchAlloc pol_alloc{s};
  auto pol = thrust::cuda::par_nosync(pol_alloc).on(s);
  DevBuf<uint32_t> keys, keys2;
  DevBuf<uint2> vals, vals2;
  uint64_t m = 0;
  {
    DevBuf<uint32_t> rowid, marks;
    DevBuf<uint64_t> tiles;
    DevBuf<unsigned long long> total;  // {suffix ids cut off, records}
    const uint64_t nt = (W + kCandTile - 1) / kCandTile;
    const bool scan = nt > kCandFewTiles;
    const uint64_t stride = tile_stride(nt);
    GARY_TRY(total.alloc(2, s));
    GARY_CUDA(cudaMemsetAsync(total.p, 0, 16, s));
    GARY_TRY(tiles.alloc(std::max<uint64_t>(nt, 1), s));
    GARY_TRY(marks.alloc(std::max<uint64_t>(nt * kCandPer * kCandWarps, 1), s));
    GARY_TRY(padded_rowid(g->dag, rowid, s));
    const unsigned grid = grid_for(nt * kThreads);
    if (W)
      k_in_mark<<<grid, kThreads, 0, s>>>(g->dag.row.p, g->dag.adj.p, rowid.p, W, stride, len.p, marks.p, tiles.p, total.p);
    GARY_CUDA(cudaGetLastError());
    if (scan) thrust::exclusive_scan(pol, tiles.p, tiles.p + nt, tiles.p, (uint64_t)0);
    // a word has one record at most: not waiting for their number here keeps the
    // device busy over the allocations and the launch
    GARY_TRY(keys.alloc(std::max<uint64_t>(W, 1), s));
    GARY_TRY(vals.alloc(std::max<uint64_t>(W, 1), s));
    if (W)
      k_in_candidates<<<grid, kThreads, 0, s>>>(g->dag.row.p, g->dag.adj.p, rowid.p, W, stride, len.p, marks.p, tiles.p, scan,
                                                keys.p, vals.p);
    GARY_CUDA(cudaGetLastError());
    unsigned long long h[2] = {0, 0};
    GARY_CUDA(cudaMemcpyAsync(h, total.p, 16, cudaMemcpyDeviceToHost, s));
    GARY_CUDA(cudaStreamSynchronize(s));
    in.hub_work = h[0];
    m = h[1];
  }
  if (m) {
    GARY_TRY(keys2.alloc(m, s));
    GARY_TRY(vals2.alloc(m, s));
    cub::DoubleBuffer<uint32_t> kb(keys.p, keys2.p);
    cub::DoubleBuffer<uint2> vb(vals.p, vals2.p);
    size_t tmp = 0;
    const int eb = bits_for((uint64_t)n);
    GARY_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, kb, vb, m, 0, eb, s));
    DevBuf<uint8_t> t;
    GARY_TRY(t.alloc(tmp, s));
    GARY_CUDA(cub::DeviceRadixSort::SortPairs(t.p, tmp, kb, vb, m, 0, eb, s));
    if (kb.Current() != keys.p) std::swap(keys, keys2);
    if (vb.Current() != vals.p) std::swap(vals, vals2);
  }
  keys2.release();
  vals2.release();
  in.records = m;
  GARY_TRY(in.inptr.alloc_persistent((uint64_t)n + 1));
  thrust::fill(pol, in.inptr.p, in.inptr.p + n + 1, m);
  if (m) k_in_heads<<<grid_for(m), kThreads, 0, s>>>(keys.p, m, in.inptr.p);
  auto rb = thrust::make_reverse_iterator(in.inptr.p + n + 1);
  thrust::inclusive_scan(pol, rb, rb + n + 1, rb, MinU64());
  GARY_TRY(in.inedge.alloc_persistent(std::max<uint64_t>(m, 1)));
  if (m)
    GARY_CUDA(cudaMemcpyAsync(in.inedge.p, vals.p, m * sizeof(uint2), cudaMemcpyDeviceToDevice, s));
  GARY_TRY(in.work.alloc_persistent(n));
  GARY_CUDA(cudaMemsetAsync(in.work.p, 0, (uint64_t)n * 8, s));
  if (m)
    k_in_work<<<grid_for(m), kThreads, 0, s>>>(keys.p, vals.p, m,
                                              reinterpret_cast<unsigned long long *>(in.work.p));
  GARY_CUDA(cudaGetLastError());
  in.total_work = thrust::reduce(pol, in.work.p, in.work.p + n, 0ull);
  return GARY_OK;
}

}  // namespace

PlanParams resolve_params(PlanParams pp, uint64_t total_work, uint64_t records) {
  // Three resident CTAs per SM of 12 warps beat two of 16 from some 2^26 probes
  // on (ms a count, 3 / 2: RMAT-18 0.119 / 0.123, RMAT-20 0.514 / 0.537, RMAT-22
  // 3.02 / 3.22, RMAT-24 ef32 65.5 / 72.4; RMAT-16 0.039 either way).
  if (pp.min_blocks != 2 && pp.min_blocks != 3) pp.min_blocks = total_work >= (1ull << 26) ? 3 : 2;
  const uint64_t slots = (uint64_t)sm_count() * tc_warps(pp.min_blocks) * pp.min_blocks;
  // A vertex is split over tiles no finer than split_floor probes per id of its
  // set, or building the set anew for every piece costs too much (RMAT-22 3.71
  // ms with pieces of any size, 3.23 at 32 probes an id, 3.02 at 128); graphs
  // with little work for each warp need the parallelism more (RMAT-16 0.0384
  // ms at 16 and below, 0.0435 at 64).
  pp.split_floor = total_work / slots >= (1ull << 12) ? 128 : 16;
  if (!pp.warp_tile_cost) {
    // The best warp tile holds about 1/128 of a resident warp's share of the
    // work, between 2^11 and 2^14 probes: larger tiles leave warps idle at the
    // end (RMAT-23 9.16 ms at 1/32 up to 2^15, 8.0 at 1/128), smaller ones pay
    // the per-tile cost.
    const uint64_t want = total_work / (slots * 128);
    uint64_t t = 1ull << 11;
    while (t < want && t < (1ull << 14)) t <<= 1;
    // a graph too small to give every resident warp such a tile is cut into one
    // tile per warp: its time is that of the longest chain of dependent loads
    const uint64_t share = (total_work + 8 * records) / slots;
    if (share < t) t = std::max<uint64_t>(share, 128);
    pp.warp_tile_cost = t;
  }
  return pp;
}

namespace {

int k3_plan(gary_graph *g, const PlanParams &pp_in, cudaStream_t s, gary_count_plan **out, const float *model,
            Rows rows) {
  auto plan = std::make_unique<gary_count_plan>();
  const uint32_t n = g->n;
  ScratchAlloc pol_alloc{s};
  auto pol = thrust::cuda::par_nosync(pol_alloc).on(s);
  PhaseTrace tr("triangle plan", s);
  {
    DevBuf<uint32_t> len;
    GARY_TRY(build_hub_rows(g, s, rows, plan->hub, len));
    plan->rows_by_graph = rows != Rows::kNone && !plan->hub.no_room;
    tr.mark("hub rows");
    GARY_TRY(build_in_index(g, s, len, plan->in));
  }
  tr.mark("in-edge index");
  const PlanParams pp = resolve_params(pp_in, plan->in.total_work, plan->in.records);
  plan->params = pp;
  GARY_TRY(plan->vclass.alloc_persistent(n));
  DevBuf<uint64_t> costV;  // cost of each light vertex, 0 for the others
  DevBuf<uint32_t> kW, kC;
  GARY_TRY(costV.alloc(n, s));
  GARY_TRY(kW.alloc((uint64_t)n + 1, s));
  GARY_TRY(kC.alloc((uint64_t)n + 1, s));
  // learned plans: per-vertex features -> cost model -> variant and predicted cycles
  DevBuf<uint64_t> pcost;
  uint64_t tw = pp.warp_tile_cost;
  if (model) {
    DevBuf<float> x, dmodel;
    DevBuf<uint8_t> legal;
    GARY_TRY(x.alloc((uint64_t)n * kMlpIn, s));
    GARY_TRY(legal.alloc(n, s));
    GARY_TRY(dmodel.alloc(kMlpParams, s));
    GARY_TRY(pcost.alloc(n, s));
    GARY_TRY(plan->variant.alloc_persistent(n));
    GARY_CUDA(cudaMemcpyAsync(dmodel.p, model, kMlpParams * 4, cudaMemcpyHostToDevice, s));
    k_features<<<grid_for(n), kThreads, 0, s>>>(g->dag.row.p, g->dag.adj.p, g->rdeg.p, plan->in.work.p,
                                                plan->in.inptr.p, n, pp.warp_cap, x.p, legal.p);
    k_predict<<<grid_for(n), 128, 0, s>>>(dmodel.p, x.p, legal.p, n, plan->variant.p, pcost.p);
    GARY_CUDA(cudaGetLastError());
    const uint64_t total = thrust::transform_reduce(pol, thrust::counting_iterator<uint32_t>(0),
                                                    thrust::counting_iterator<uint32_t>(n),
                                                    SetCycles{g->dag.row.p, pcost.p}, (uint64_t)0, thrust::plus<uint64_t>());
    // about 32 warp tiles per resident warp, in predicted cycles
    const uint64_t slots = (uint64_t)sm_count() * pp.min_blocks * tc_warps(pp.min_blocks) * 32;
    tw = std::max<uint64_t>(total / std::max<uint64_t>(slots, 1), 4096);
    plan->learned = true;
  }
  k_classify<<<grid_for(n), kThreads, 0, s>>>(g->dag.row.p, g->dag.adj.p, plan->in.work.p, plan->in.inptr.p, n, pp,
                                              model ? pcost.p : nullptr, tw, plan->vclass.p, costV.p, kW.p,
                                              kC.p);
  GARY_CUDA(cudaGetLastError());
  GARY_CUDA(cudaMemsetAsync(kW.p + n, 0, 4, s));
  GARY_CUDA(cudaMemsetAsync(kC.p + n, 0, 4, s));
  const uint64_t totalL = thrust::reduce(pol, costV.p, costV.p + n, 0ull);
  thrust::exclusive_scan(pol, kW.p, kW.p + n + 1, kW.p, 0u);
  thrust::exclusive_scan(pol, kC.p, kC.p + n + 1, kC.p, 0u);
  uint32_t nW = 0, nC = 0;
  GARY_CUDA(cudaMemcpyAsync(&nW, kW.p + n, 4, cudaMemcpyDeviceToHost, s));
  GARY_CUDA(cudaMemcpyAsync(&nC, kC.p + n, 4, cudaMemcpyDeviceToHost, s));
  GARY_CUDA(cudaStreamSynchronize(s));
  tr.mark("classify");
  const uint64_t G = totalL ? (totalL + tw - 1) / tw : 0;
  const uint64_t total = (uint64_t)nC + nW + G;
  if (total >= (1ull << 31)) {
    set_error("tile plan too large (%llu tiles)", (unsigned long long)total);
    return GARY_ERR_UNSUPPORTED;
  }
  plan->n_cta = nC;
  plan->n_warp = (uint32_t)(nW + G);
  GARY_TRY(plan->tiles.alloc_persistent(std::max<uint64_t>(total, 1)));
  k_fill_split_tiles<<<grid_for(n), kThreads, 0, s>>>(plan->in.inptr.p, n, kC.p, plan->tiles.p);
  k_fill_split_tiles<<<grid_for(n), kThreads, 0, s>>>(plan->in.inptr.p, n, kW.p,
                                                     plan->tiles.p + nC);
  GARY_CUDA(cudaGetLastError());
  if (G) {
    // light vertices in id order, and the exclusive prefix of their costs
    GARY_TRY(plan->light.alloc_persistent(n));
    const uint32_t L = (uint32_t)(thrust::copy_if(pol, thrust::counting_iterator<uint32_t>(0),
                                                  thrust::counting_iterator<uint32_t>(n),
                                                  plan->light.p, IsLight{plan->vclass.p}) -
                                  plan->light.p);
    plan->n_light = L;
    DevBuf<uint64_t> lc;
    GARY_TRY(lc.alloc((uint64_t)L + 1, s));
    auto costs = thrust::make_transform_iterator(plan->light.p, LightCost{costV.p});
    thrust::exclusive_scan(pol, costs, costs + L, lc.p, 0ull);
    DevBuf<uint32_t> starts;
    GARY_TRY(starts.alloc(G, s));
    auto targets = thrust::make_transform_iterator(thrust::counting_iterator<uint64_t>(0),
                                                   GroupTarget{tw});
    thrust::lower_bound(pol, lc.p, lc.p + L, targets, targets + G, starts.p);
    k_fill_group_tiles<<<grid_for(G), kThreads, 0, s>>>(starts.p, G, L, plan->tiles.p + nC + nW);
    GARY_CUDA(cudaGetLastError());
  }
  constexpr size_t kSpanBytes = 2ull * kMaxCountCtas * 8;
  GARY_TRY(plan->sched.alloc_persistent(1 + (kSpanBytes + sizeof(SchedState) - 1) / sizeof(SchedState)));
  GARY_CUDA(cudaStreamSynchronize(s));
  tr.mark("tiles");
  *out = plan.release();
  return GARY_OK;
}

}  // namespace

int build_k3_plan(gary_graph *g, const PlanParams &pp, cudaStream_t s, gary_count_plan **out, const float *model,
                  Rows rows) {
  if (rows != Rows::kOptional) return k3_plan(g, pp, s, out, model, rows);
  return with_or_without_rows(s, [&](Rows use) { return k3_plan(g, pp, s, out, model, use); });
}

// ---------------------------------------------------------------------------
// Counting kernel
namespace {

static_assert(kPairWords == kWarpTableSlots, "a pair set fills a warp's region");
constexpr uint32_t kWarpBitmapSpan = bitmap_max_span(kWarpTableSlots);  // ids a warp bitmap covers

// One chunk of at most 32 in-edge records [kb, ke): count the members of each
// suffix that `set` holds.  Suffixes are read as 32-byte-aligned octets of
// ids (two 16-byte loads from one sector); the lanes walk the concatenation of
// the chunk's octets, so short suffixes do not idle lanes.  Lists start on
// 32-byte boundaries and are padded with kSentinel to a multiple of 8 words,
// so an octet only ever holds words of its own list: ids up to and including
// v before the suffix (all below min N+(v)) and padding (a suffix cut short by
// hub rows ends with an octet).  Every set rejects both, so no per-id mask is
// needed: most as out of their [lo, lo + span] range, a pair set as ids that are
// not in it (its entries and slots give an id back exactly, and padding has an
// entry of more than 16 bits).
// All 32 lanes must call.
template <typename Set>
__device__ __forceinline__ uint32_t probe_octet(const uint4 &a, const uint4 &b, const Set &set) {
  return set.contains(a.x) + set.contains(a.y) + set.contains(a.z) + set.contains(a.w) +
         set.contains(b.x) + set.contains(b.y) + set.contains(b.z) + set.contains(b.w);
}

template <typename Set>
__device__ __forceinline__ uint32_t walk_chunk(const uint4 *__restrict__ adj4,
                                               const uint2 *__restrict__ edges, uint64_t kb,
                                               uint64_t ke, int lane, const Set &set) {
  const uint64_t kk = kb + lane;
  uint32_t o0 = 0, no = 0;
  if (kk < ke) {
    const uint2 r = edges[kk];
    o0 = r.x >> 3;
    no = ((r.x + r.y + 7) >> 3) - o0;
  }
  const uint32_t incl = warp_inclusive_sum(no, lane);
  const uint32_t total = __shfl_sync(kFull, incl, 31);
  if (total == 0) return 0;
  // flattened position p of record k's octets maps to octet (o0 - excl) + p
  const uint32_t excl = incl - no;
  const uint32_t bias = o0 - excl;
  // Every record has octets (a suffix is never empty); only the lanes past
  // the last record have none, so the owners follow from the record starts.
  WarpOwners owners(excl, lane);
  auto fetch = [&](uint32_t pb, uint4 &a, uint4 &b) {
    const uint32_t own = owners.owner(pb);
    const uint32_t p = pb + lane;
    const uint32_t oc = __shfl_sync(kFull, bias, own) + p;
    if (p < total) {
      a = adj4[2 * oc];
      b = adj4[2 * oc + 1];
    } else {
      a = b = make_uint4(kSentinel, kSentinel, kSentinel, kSentinel);
    }
  };
  uint32_t cnt = 0;
  // two batches in flight: the next octet loads while this one is probed
  uint4 ca, cb;
  fetch(0, ca, cb);
  for (uint32_t pb = 32; pb < total; pb += 32) {
    uint4 na, nb;
    fetch(pb, na, nb);
    cnt += probe_octet(ca, cb, set);
    ca = na;
    cb = nb;
  }
  cnt += probe_octet(ca, cb, set);
  return cnt;
}

template <typename Set>
__device__ __forceinline__ uint32_t walk_range(const uint4 *__restrict__ adj4,
                                               const uint2 *__restrict__ edges, uint64_t kb,
                                               uint64_t ke, int lane, const Set &set) {
  uint32_t cnt = 0;
  for (uint64_t k = kb; k < ke; k += 32) cnt += walk_chunk(adj4, edges, k, ke, lane, set);
  return cnt;
}

// CTA tile: N+(v) does not fit a warp's set.  All warps share one set in the
// whole shared buffer and claim 32-record chunks of the tile dynamically.
template <int WARPS, typename Set>
__device__ __forceinline__ uint32_t cta_walk(const uint4 *__restrict__ adj4,
                                             const uint2 *__restrict__ edges, uint64_t kb,
                                             uint64_t ke, uint32_t *chunk, int lane,
                                             const Set &set) {
  uint32_t cnt = 0;
  while (true) {
    uint32_t c = 0;
    if (lane == 0) c = atomicAdd(chunk, 1u);
    c = __shfl_sync(kFull, c, 0);
    const uint64_t k = kb + (uint64_t)c * 32;
    if (k >= ke) break;
    cnt += walk_chunk(adj4, edges, k, ke < k + 32 ? ke : k + 32, lane, set);
  }
  return cnt;
}

// How CTA tiles hold N+(v): `words` shared words for the set (a multiple of
// 4, at most the CTA's buffer) and the poll limit of the first wait for a
// staging copy.
struct CtaSetCfg {
  uint32_t words;
  uint32_t polls;
};

// One CTA tile.  N+(v) goes into the cheapest set that fits `cfg.words`
// shared words: a bitmap of its id span, 4-slot hash buckets (d <= words/2),
// the sorted list staged whole by a bulk copy (d <= words; searched in
// shared memory only), or `words` evenly spaced samples of the list for the
// two-phase search (phase 2 in HBM).  Adds the tile's count to cnt_total.
// Returns false when a staging copy did not land within the drain wait: the
// CTA must then stop touching shared memory (the copy may still arrive), so
// the caller abandons its remaining work; the error word records it.
template <int WARPS>
__device__ bool cta_tile(const GraphView &g, const uint2 *__restrict__ inedge,
                         const uint64_t *__restrict__ inptr, const Tile &t, uint32_t *smem,
                         uint32_t *chunk, uint64_t *bar, uint32_t &phase, const CtaSetCfg &cfg,
                         SchedState *sched, const uint32_t *gid, unsigned long long *gcount,
                         unsigned long long &cnt_total) {
  const uint32_t S = cfg.words;
  const int lane = threadIdx.x & 31;
  const uint32_t v = t.v0;
  const uint2 rv = g.row[v];
  const uint32_t d = rv.y;
  const uint32_t *av = g.adj + (uint64_t)rv.x * 4;
  const uint4 *adj4 = reinterpret_cast<const uint4 *>(g.adj);
  const uint64_t base = inptr[v];
  const uint64_t kb = base + t.j0, ke = base + t.j1;
  const uint32_t lo = av[0], span = av[d - 1] - lo;
  auto sync = [] { __syncthreads(); };
  if (threadIdx.x == 0) *chunk = 0;
  uint32_t cnt = 0, path;
  if (span <= bitmap_max_span(S)) {
    path = kPathBitmap;
    const BitmapSet st = build_bitmap(av, d, lo, span, smem, threadIdx.x, blockDim.x, sync);
    cnt = cta_walk<WARPS>(adj4, inedge, kb, ke, chunk, lane, st);
  } else if (2 * d <= S) {
    path = kPathBuckets;
    const BucketSet st =
        build_buckets(av, d, lo, span, smem, S, threadIdx.x, blockDim.x, sync, &sched->error);
    cnt = cta_walk<WARPS>(adj4, inedge, kb, ke, chunk, lane, st);
  } else {
    if (d <= S) {
      // the whole list by one bulk copy (lists start 32-byte aligned and are
      // padded to whole octets, so the 16-byte-rounded size stays in the list)
      path = kPathStaged;
      if (threadIdx.x == 0) bulk_stage(smem, av, ((d + 3) / 4) * 16, bar);
      bool ok = mbar_wait_bounded(bar, phase, cfg.polls);
      if (!ok) {
        atomicOr(&sched->error, kLaunchErrStageWait);
        ok = mbar_wait_bounded(bar, phase);  // drain the copy before going on
      }
      if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) atomicOr(&sched->error, kLaunchErrStageDrain);
        return false;
      }
      phase ^= 1;
    } else {
      path = kPathSampled;
      for (uint32_t i = threadIdx.x; i < S; i += blockDim.x) smem[i] = av[(uint64_t)i * d / S];
      __syncthreads();
    }
    const SearchSet st{av, smem, d, S, lo, span};
    cnt = cta_walk<WARPS>(adj4, inedge, kb, ke, chunk, lane, st);
  }
  if (threadIdx.x == 0) atomicAdd(&sched->cta_path[path], 1u);
  if (gcount) {
    const unsigned long long tw = warp_sum_u64(cnt);
    if (lane == 0 && tw) atomicAdd(&gcount[gid[v]], tw);
  }
  cnt_total += cnt;
  // the next tile rewrites shared memory, possibly through the async proxy
  fence_proxy_async_smem();
  __syncthreads();
  return true;
}

// Sorted copy of N+(v) in shared memory, binary-searched (variant SEARCH).
struct SmemSearchSet {
  const uint32_t *list;
  uint32_t d, lo, span;
  __device__ __forceinline__ uint32_t contains(uint32_t x) const {
    if (x - lo > span) return 0;
    uint32_t b = 0, e = d;
    while (b < e) {
      const uint32_t m = (b + e) >> 1;
      const uint32_t v = list[m];
      if (v == x) return 1;
      if (v < x) b = m + 1;
      else e = m;
    }
    return 0;
  }
};

// Up to 8 ids held in registers in every lane, each probe compared against
// all of them (variant REGS).
struct RegSet8 {
  uint32_t r[8];
  __device__ __forceinline__ uint32_t contains(uint32_t x) const {
    uint32_t f = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) f |= (x == r[k]) ? 1u : 0u;
    return f;
  }
};

// Per-vertex control of the warp path; null pointers give the plain
// dispatch (bitmap when the span fits, else buckets) and no cycle log.
struct VertexCtl {
  const uint8_t *variant;      // intersection variant per middle vertex
  unsigned long long *cycles;  // clock64 cycles spent per middle vertex
  const uint32_t *gid;         // batches: graph of each middle vertex
  unsigned long long *gcount;  // batches: per-graph counts
  unsigned *err;               // the launch's error word
  unsigned long long *span;    // per CTA: start time, finish time of its last warp (ns)
};

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Batches: add a warp's count for middle vertex v to its graph's total.
__device__ __forceinline__ void add_graph_count(const VertexCtl &ctl, uint32_t v, uint32_t c,
                                                int lane) {
  if (!ctl.gcount) return;
  const unsigned long long t = warp_sum_u64(c);
  if (lane == 0 && t) atomicAdd(&ctl.gcount[ctl.gid[v]], t);
}

// What a warp needs of a middle vertex before it builds a set: its list, its
// records [kb, ke) and the list's first id and span.
struct VertexHead {
  uint2 rv;
  uint32_t lo, span;
  uint64_t kb, ke;
};

// One middle vertex v (d+ > 0, some records) on one warp: a set of N+(v) in the
// warp's slots, walk its records.
__device__ __forceinline__ uint32_t warp_vertex(const GraphView &g, const uint2 *__restrict__ inedge, uint32_t v,
                                                const VertexHead &h, uint32_t *tab, int lane, const VertexCtl &ctl) {
  const uint32_t d = h.rv.y, lo = h.lo, span = h.span;
  const uint64_t kb = h.kb, ke = h.ke;
  const long long t0 = ctl.cycles ? clock64() : 0;
  const uint32_t *av = g.adj + (uint64_t)h.rv.x * 4;
  const uint4 *adj4 = reinterpret_cast<const uint4 *>(g.adj);
  auto sync = [] { __syncwarp(); };
  uint32_t var = span <= kWarpBitmapSpan ? kVarBitmap : kVarHash;
  if (ctl.variant) {
    const uint32_t f = ctl.variant[v];
    if (variant_legal(f, d, span)) var = f;
  }
  uint32_t c;
  if (var == kVarBitmap) {
    const BitmapSet st = build_bitmap(av, d, lo, span, tab, lane, 32, sync);
    c = walk_range(adj4, inedge, kb, ke, lane, st);
  } else if (var == kVarHash) {
    // buckets for ids of more than 26 bits, and when a pair set's build gives up
    const int k = pair_log(d, g.n);
    PairSet pair;
    if (k && build_pair_set(av, d, k, tab, lane, pair)) {
      c = walk_range(adj4, inedge, kb, ke, lane, pair);
    } else {
      const BucketSet st = build_buckets(av, d, lo, span, tab, kWarpTableSlots, lane, 32, sync, ctl.err);
      c = walk_range(adj4, inedge, kb, ke, lane, st);
    }
  } else if (var == kVarSearch) {
    for (uint32_t i = lane; i < d; i += 32) tab[i] = av[i];
    __syncwarp();
    const SmemSearchSet st{tab, d, lo, span};
    c = walk_range(adj4, inedge, kb, ke, lane, st);
  } else {
    RegSet8 st;
#pragma unroll
    for (int k = 0; k < 8; ++k) st.r[k] = av[(uint32_t)k < d ? k : d - 1];  // repeats, never padding
    c = walk_range(adj4, inedge, kb, ke, lane, st);
  }
  __syncwarp();
  if (ctl.cycles && lane == 0) atomicAdd(&ctl.cycles[v], (unsigned long long)(clock64() - t0));
  add_graph_count(ctl, v, c, lane);
  return c;
}

// How many of the 8 ids a, b equal one of the 8 ids p, q.
__device__ __forceinline__ uint32_t match_octets(const uint4 &a, const uint4 &b, const uint4 &p, const uint4 &q) {
  auto in = [&](uint32_t x) -> uint32_t {
    return x == p.x || x == p.y || x == p.z || x == p.w || x == q.x || x == q.y || x == q.z || x == q.w;
  };
  return in(a.x) + in(a.y) + in(a.z) + in(a.w) + in(b.x) + in(b.y) + in(b.z) + in(b.w);
}

// All in-edges of the tiny vertices among 32 light ones (lane's list rv and its
// nin_v records from ib on, where `tiny`), without a set: the 32 vertices'
// records are walked flattened, and within a batch of 32 records their octets
// are, so every lane compares one octet of a suffix with the one or two octets
// of N+(v).  Building a set costs
// a vertex some thousands of cycles of dependent loads and shared-memory
// passes whatever its size, which for these vertices is most of their time.
// All 32 lanes must call.
__device__ __forceinline__ uint32_t tiny_vertices(const GraphView &g, const uint2 *__restrict__ inedge, uint32_t ib,
                                                  uint32_t nin_v, uint2 rv, bool tiny, int lane) {
  // N+(v)'s padding equals a suffix's padding: the suffix's is lowered by one
  // (still no vertex id), which is also what lanes without an octet hold.
  constexpr uint32_t kNever = kSentinel - 1u;
  const uint4 *adj4 = reinterpret_cast<const uint4 *>(g.adj);
  const uint32_t nin = tiny ? nin_v : 0u;
  const uint32_t incl = warp_inclusive_sum(nin, lane);
  const uint32_t records = __shfl_sync(kFull, incl, 31);
  // record of flattened position p: rbias + p (mod 2^32, as the octets below) of the owner
  const uint32_t rbias = ib - (incl - nin);
  const uint32_t myset = (rv.x >> 1) | (rv.y > 8 ? 1u << 31 : 0u);  // N+(v)'s first octet; bit 31: it has two
  WarpRuns runs(incl - nin, nin, lane);
  uint32_t cnt = 0;
  auto fetch = [&](uint32_t rb, uint2 &r, uint32_t &set) {
    const int o = (int)runs.owner(rb);
    const uint32_t k = __shfl_sync(kFull, rbias, o) + rb + lane;
    set = __shfl_sync(kFull, myset, o);
    r = rb + lane < records ? inedge[k] : make_uint2(0, 0);
  };
  uint2 r;
  uint32_t set;
  fetch(0, r, set);
  for (uint32_t rb = 0; rb < records; rb += 32) {
    uint2 rn = make_uint2(0, 0);
    uint32_t setn = 0;
    if (rb + 32 < records) fetch(rb + 32, rn, setn);
    const uint32_t o0 = r.x >> 3;
    const uint32_t no = r.y ? ((r.x + r.y + 7) >> 3) - o0 : 0u;
    const uint32_t oincl = warp_inclusive_sum(no, lane);
    const uint32_t total = __shfl_sync(kFull, oincl, 31);
    const uint32_t bias = o0 - (oincl - no);
    WarpOwners owners(oincl - no, lane);
    for (uint32_t pb = 0; pb < total; pb += 32) {
      const int o = (int)owners.owner(pb);
      const uint32_t oc = __shfl_sync(kFull, bias, o) + pb + lane;
      const uint32_t sx = __shfl_sync(kFull, set, o);
      const bool on = pb + lane < total;
      const uint4 never = make_uint4(kNever, kNever, kNever, kNever);
      uint4 a = never, b = never, p = never, q = never;
      const uint32_t so = sx & 0x7FFFFFFFu;
      if (on) {
        a = adj4[2 * (uint64_t)oc];
        b = adj4[2 * (uint64_t)oc + 1];
        p = adj4[2 * (uint64_t)so];
        q = adj4[2 * (uint64_t)so + 1];
        a.x = min(a.x, kNever); a.y = min(a.y, kNever); a.z = min(a.z, kNever); a.w = min(a.w, kNever);
        b.x = min(b.x, kNever); b.y = min(b.y, kNever); b.z = min(b.z, kNever); b.w = min(b.w, kNever);
        cnt += match_octets(a, b, p, q);
        if (sx >> 31) {
          p = adj4[2 * (uint64_t)so + 2];
          q = adj4[2 * (uint64_t)so + 3];
          cnt += match_octets(a, b, p, q);
        }
      }
    }
    r = rn;
    set = setn;
  }
  return cnt;
}

template <int WARPS, int MINB>
__global__ void __launch_bounds__(WARPS * 32, MINB)
    k_tc_mid(GraphView g, const uint2 *__restrict__ inedge, const uint64_t *__restrict__ inptr,
             const uint32_t *__restrict__ light, const Tile *__restrict__ tiles, uint32_t n_cta,
             TileRange rng, HubView hub, SchedState *sched, unsigned long long *__restrict__ out, VertexCtl ctl,
             CtaSetCfg cfg) {
  extern __shared__ __align__(16) uint32_t smem_raw[];
  __shared__ uint64_t bar;
  __shared__ uint32_t s_tile, s_chunk;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long cnt = 0;
  // each warp's region on a multiple of its size (PairSet)
  constexpr uint32_t kRegion = kWarpTableSlots * 4;
  uint32_t *smem = smem_raw + ((0u - (uint32_t)__cvta_generic_to_shared(smem_raw)) & (kRegion - 1)) / 4;

  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
    if (ctl.span) ctl.span[2 * blockIdx.x] = global_ns();
  }
  __syncthreads();
  uint32_t phase = 0;

  // phase 1: CTA tiles (N+(v) does not fit a warp's set)
  bool alive = true;
  while (true) {
    if (threadIdx.x == 0) s_tile = rng.cta_lo + atomicAdd(&sched->next_cta, 1u);
    __syncthreads();
    const uint32_t t = s_tile;
    __syncthreads();
    if (t >= rng.cta_hi) break;
    const Tile tl = tiles[t];
    if (!cta_tile<WARPS>(g, inedge, inptr, tl, smem, &s_chunk, &bar, phase, cfg, sched, ctl.gid,
                         ctl.gcount, cnt)) {
      alive = false;  // a staging copy may still land in shared memory: no more work here
      break;
    }
  }

  // phase 2: warp tiles, each warp on its own slots, and hub rows.  Odd warps
  // begin with the rows, even ones with the tiles, so that the rows' L2 reads
  // and the tiles' shared-memory probes overlap on every SM.
  uint32_t *tab = smem + warp * kWarpTableSlots;
  const Tile *wt = tiles + n_cta;
#pragma unroll 1
  for (int part = 0; part < 2; ++part) {
    if ((part ^ warp) & 1) {
      while (alive && hub.lo < hub.hi) {
        uint32_t i = 0;
        if (lane == 0) i = hub.lo + atomicAdd(&sched->next_aux, 1u);
        i = __shfl_sync(kFull, i, 0);
        if (i >= hub.hi) break;
        cnt += hub_vertex(g, hub, i, lane);
      }
      continue;
    }
    while (alive) {
      uint32_t t = 0;
      if (lane == 0) t = rng.warp_lo + atomicAdd(&sched->next_warp, 1u);
      t = __shfl_sync(kFull, t, 0);
      if (t >= rng.warp_hi) break;
      const Tile tl = wt[t];
      if (tl.j1 != kGroupTile) {  // records [j0, j1) of one vertex
        const uint2 rv = g.row[tl.v0];
        const uint32_t *av = g.adj + (uint64_t)rv.x * 4;
        const uint64_t base = inptr[tl.v0];
        const uint32_t lo = av[0];
        cnt += warp_vertex(g, inedge, tl.v0,
                           VertexHead{rv, lo, av[rv.y - 1] - lo, base + tl.j0, base + tl.j1}, tab, lane, ctl);
        continue;
      }
      // a group of light vertices: list positions [v0, v1), 32 ids per load
      for (uint32_t ib = tl.v0; ib < tl.v1; ib += 32) {
        const uint32_t nb = min(32u, tl.v1 - ib);
        const uint32_t myv = lane < nb ? light[ib + lane] : 0u;
        unsigned left = nb < 32 ? (1u << nb) - 1u : kFull;
        // the tiny ones together, unless per-vertex results are asked for
        bool together = !ctl.cycles;
        uint32_t gid = 0;
        if (together && ctl.gcount) {
          gid = lane < nb ? ctl.gid[myv] : 0u;
          const uint32_t g0 = __shfl_sync(kFull, gid, 0);
          together = __all_sync(kFull, lane >= nb || gid == g0);
          gid = g0;
        }
        // the heads of all 32 in lanes, so that the loads a vertex begins with
        // are waited for once, not by every vertex again (batch of 128 graphs
        // 718 -> 687 us, RMAT-22 ef16 3.04 -> 3.02 ms)
        uint2 rv = make_uint2(0, 0);
        uint64_t kb = 0;
        uint32_t nin = 0;
        if (lane < nb) {
          rv = g.row[myv];
          kb = inptr[myv];
          nin = (uint32_t)(inptr[myv + 1] - kb);
        }
        if (together) {
          const bool tiny = rv.y - 1u < kTinyOut;
          const unsigned tm = __ballot_sync(kFull, tiny);
          if (tm) {
            const uint32_t c = tiny_vertices(g, inedge, (uint32_t)kb, nin, rv, tiny, lane);
            cnt += c;
            if (ctl.gcount) {
              const unsigned long long sum = warp_sum_u64(c);
              if (lane == 0 && sum) atomicAdd(&ctl.gcount[gid], sum);
            }
            left &= ~tm;
          }
        }
        if (left) {
          uint32_t lo = 0, span = 0;
          if ((left >> lane) & 1u) {
            const uint32_t *av = g.adj + (uint64_t)rv.x * 4;
            lo = av[0];
            span = av[rv.y - 1] - lo;
          }
          while (left) {
            const int k = __ffs(left) - 1;
            left &= left - 1;
            VertexHead h;
            h.rv.x = __shfl_sync(kFull, rv.x, k);
            h.rv.y = __shfl_sync(kFull, rv.y, k);
            h.lo = __shfl_sync(kFull, lo, k);
            h.span = __shfl_sync(kFull, span, k);
            h.kb = __shfl_sync(kFull, (uint32_t)kb, k);  // records are numbered in 32 bits (build_in_index)
            h.ke = h.kb + __shfl_sync(kFull, nin, k);
            cnt += warp_vertex(g, inedge, __shfl_sync(kFull, myv, k), h, tab, lane, ctl);
          }
        }
      }
    }
  }

  cnt = warp_sum_u64(cnt);
  if (lane == 0 && cnt) atomicAdd(out, cnt);
  if (lane == 0 && ctl.span) atomicMax(&ctl.span[2 * blockIdx.x + 1], global_ns());
  if (threadIdx.x == 0 && alive) mbar_inval(&bar);
}

}  // namespace

int k3_features(gary_graph *g, gary_count_plan *plan, float *d_x, uint8_t *d_legal, cudaStream_t s) {
  k_features<<<grid_for(g->n), kThreads, 0, s>>>(g->dag.row.p, g->dag.adj.p, g->rdeg.p,
                                                 plan->in.work.p, plan->in.inptr.p, g->n,
                                                 plan->params.warp_cap, d_x, d_legal);
  GARY_CUDA(cudaGetLastError());
  return GARY_OK;
}

template <int MINB>
int launch_k3_impl(gary_graph *g, gary_count_plan *plan, unsigned long long *d_out, cudaStream_t s,
                   uint32_t shard, uint32_t nshards, VertexCtl ctl) {
  constexpr int WARPS = tc_warps(MINB);
  auto kern = k_tc_mid<WARPS, MINB>;
  const size_t smem = (size_t)(WARPS + 1) * kWarpTableSlots * 4;  // + 1: regions start on a multiple of their size
  // the resident CTAs per SM, asked for once per device
  static int resident[64] = {0};
  const int dev = device_ordinal();
  int per_sm = dev < 64 ? resident[dev] : 0;
  if (!per_sm) {
    GARY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    GARY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WARPS * 32, smem));
    if (per_sm < 1) per_sm = 1;
    if (dev < 64) resident[dev] = per_sm;
  }
  const unsigned grid = (unsigned)std::min<int>(sm_count() * per_sm, (int)kMaxCountCtas);
  ctl.span = plan->span();
  const TileRange rng = shard_range(plan->n_cta, plan->n_warp, shard, nshards);
  auto part = [&](uint32_t k) { return (uint32_t)((uint64_t)plan->hub.n_list * k / nshards); };
  const HubView hub{plan->hub.rows.p, plan->hub.rowof.p, plan->hub.list.p, plan->hub.cut.p, plan->hub.first, part(shard), part(shard + 1)};
  const uint32_t words = (uint32_t)(WARPS * kWarpTableSlots);
  const uint32_t cw = plan->params.cta_set_words;
  const CtaSetCfg cfg{cw && cw < words ? cw : words, plan->params.stage_polls};
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  GARY_CUDA(cudaStreamIsCapturing(s, &cap));
  const bool timed = cap == cudaStreamCaptureStatusNone;
  GARY_CUDA(cudaMemsetAsync(plan->sched.p, 0, sizeof(SchedState) + 2ull * grid * 8, s));
  if (d_out) GARY_CUDA(cudaMemsetAsync(d_out, 0, sizeof(unsigned long long), s));
  else d_out = &plan->sched.p->total;
  if (timed) GARY_CUDA(cudaEventRecord(g->ev0, s));
  kern<<<grid, WARPS * 32, smem, s>>>(g->view(), plan->in.inedge.p, plan->in.inptr.p, plan->light.p,
                                      plan->tiles.p, plan->n_cta, rng, hub, plan->sched.p, d_out, ctl, cfg);
  GARY_CUDA(cudaGetLastError());
  if (timed) GARY_CUDA(cudaEventRecord(g->ev1, s));
  g->last = gary_count_stats{};
  g->last.tiles = (rng.cta_hi - rng.cta_lo) + (rng.warp_hi - rng.warp_lo);
  g->last.cta_tiles = rng.cta_hi - rng.cta_lo;
  g->last.work = plan->in.total_work + plan->in.hub_work;
  g->last_timed = timed;
  g->last_sched = plan->sched.p;
  g->last_span = plan->span();
  g->last_span_ctas = grid;
  return GARY_OK;
}

int launch_k3_ctl(gary_graph *g, gary_count_plan *plan, unsigned long long *d_out, cudaStream_t s,
                  uint32_t shard, uint32_t nshards, const uint8_t *variant,
                  unsigned long long *cycles, unsigned long long *gcount) {
  const VertexCtl ctl{variant, cycles, gcount ? g->gid.p : nullptr, gcount, &plan->sched.p->error, nullptr};
  if (plan->params.min_blocks >= 3) return launch_k3_impl<3>(g, plan, d_out, s, shard, nshards, ctl);
  return launch_k3_impl<2>(g, plan, d_out, s, shard, nshards, ctl);
}

int launch_k3(gary_graph *g, gary_count_plan *plan, unsigned long long *d_out, cudaStream_t s,
              uint32_t shard, uint32_t nshards) {
  return launch_k3_ctl(g, plan, d_out, s, shard, nshards, plan->variant.p, nullptr, nullptr);
}

}  // namespace gary
