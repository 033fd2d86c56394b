// Hub rows: the part of the triangle count whose third vertex is a hub.
//
// Ranks are by degree, so the top kHubIds ids are the graph's hubs, and on
// skewed graphs most members of most lists are among them: of the suffix ids
// the middle-vertex walk would probe, 86 % at RMAT-20 ef16, 72 % at RMAT-22
// ef16 and 57 % at RMAT-24 ef32 are hubs.  For the vertices with at least
// kHubMin hub neighbours the plan keeps those neighbours as a row of kHubIds
// bits, and the triangles u < v < w with a hub w are, for every edge u -> v,
//     popcount(row(u) & row(v)),
// 512 bytes read and four words ANDed per lane instead of one probe per hub
// id (about 250 ids per edge on average at RMAT-24).  A vertex u counted this
// way is cut out of the middle-vertex walk from there on, so every triangle is
// still counted once.  The walk reads whole octets of a list and would probe
// every id of its last one, so the cut lies on the next octet boundary, and u's
// own row is masked below the first id past the cut.
//
// A warp takes one u: its row in registers, N+(u) read in order.  v's row is
// usually that of a hub (2 MB in all, L2-resident), and then only the words
// above v's own position are read: N+(v) holds no id below v.
#pragma once
#include <cstdint>
#include <new>

#include "graph.cuh"
#include "internal.cuh"

namespace gary {

// 4096 ids make a row of one 16-byte load per lane.
constexpr uint32_t kHubIds = 4096;
constexpr uint32_t kHubRowQuads = kHubIds / 128;  // uint4 per row: one per lane
static_assert(kHubRowQuads == kWarp, "one quad of a row per lane");
// A row read costs about as much as probing some tens of ids (RMAT-20 ef16 /
// RMAT-22 ef16 / RMAT-24 ef32, ms a count: 1.13 / 6.78 / 118.9 without rows;
// rows from 16 hub neighbours on 0.88 / 5.26 / 76.0, from 32 0.79 / 5.06 /
// 73.1, from 64 0.79 / 4.86 / 73.3, from 96 0.70 / 5.56 / 74.6).
constexpr uint32_t kHubMin = 64;
constexpr uint32_t kHubTop = 1024;   // the last kHubTop ids fill one word per lane
constexpr uint32_t kNoHubRow = 0xFFFFFFFFu;

// Rows of the hubs themselves come first (row p of hub id first + p), then
// those of the other counted vertices: row kHubIds + i of list[i].
struct HubRows {
  DevBuf<uint4> rows;
  DevBuf<uint32_t> rowof;  // per vertex below `first`: its row, or kNoHubRow
  DevBuf<uint32_t> list;   // counted vertices, ascending
  DevBuf<uint32_t> cut;    // per listed vertex: where its counted ids begin in N+(u), a multiple of 8
  uint32_t n_list = 0;     // 0: the plan has no hub rows
  uint32_t first = 0;      // n - kHubIds
  bool no_room = false;    // n_list is 0 for want of memory
};

struct HubView {
  const uint4 *__restrict__ rows;
  const uint32_t *__restrict__ rowof;
  const uint32_t *__restrict__ list;
  const uint32_t *__restrict__ cut;
  uint32_t first, lo, hi;  // this launch counts list[lo .. hi)
};

// Adjacency rows for the 4-clique kernels: bit p of v's row says that v has the
// higher neighbour first + p.  As HubRows, over a wider range of ids (memory
// and the build grow with it, a look-up does not), without a counted list.
struct AdjRows {
  DevBuf<uint4> rows;
  DevBuf<uint32_t> rowof;  // per vertex below `first`: its row, or kNoHubRow
  DevBuf<uint32_t> low;    // per vertex: how many of its higher neighbours the rows do not cover
  uint32_t first = 0;
  uint32_t words = 0;      // per row; 0: no rows
};

// RMAT-22 ef16, ms per count of 4-cliques: 45.1 with rows of 8192 ids, 33.4 with
// 16384, 31.0 with 32768 (twice the memory: 1.2 GB); 119.5 without rows.
constexpr uint32_t kAdjRowIds = 16384;
// Top neighbours a row needs (8 / 16 / 32 / 64: RMAT-22 ef16 33.1 / 33.2 / 33.4 /
// 37.9 ms, RMAT-20 ef5 0.73 / 0.74 / 0.78 / 0.79).
constexpr uint32_t kAdjMin = 16;
// No rows where every list fits one word: they win some 5 us a count and cost 55
// us in the plan (ER n = 20000, 10 edges a vertex: 52 / 57 us a count, first count
// with its plan 214 / 157 us, with / without).
constexpr uint32_t kAdjMaxShort = 32;

// Rows of more than 1 GB take at most an eighth of the device's memory and half of
// what is free.  (Smaller ones do not ask: the driver's answer takes up to 3 ms,
// longer than a count of RMAT-20 with its plan.)
bool room_for_rows(uint64_t bytes);

// Whether a plan has rows.  In the plans of triangles and 4-cycles rows decide
// which part of the count a shard is, and the shards of one count come from plans
// that several processes built, each on a device of its own.  So the plan of a
// shard has the rows that the graph alone decides on (kRequired) or ends with
// GARY_ERR_OOM; the plan of a whole count has them where there is room (kOptional).
enum class Rows { kNone, kOptional, kRequired };

// For a whole count rows are an option: a plan that does not find the memory it
// needs is made again without them.
template <class F>
int with_or_without_rows(cudaStream_t s, F build) {
  int rc;
  try {
    rc = build(Rows::kOptional);
  } catch (const std::bad_alloc &) {  // thrust's temporaries (ScratchAlloc)
    rc = GARY_ERR_OOM;
  }
  if (rc != GARY_ERR_OOM) return rc;
  GARY_CUDA(cudaStreamSynchronize(s));
  release_cached_memory();
  clear_error();
  return build(Rows::kNone);
}

// Builds them when at least an eighth of the pairs of higher neighbours have
// their second id among the top ids and their first vertex a row; words stays 0
// otherwise (sparse graphs without hubs: walking lists is cheaper there).
int build_adj_rows(gary_graph *g, cudaStream_t s, AdjRows &adj);

// Builds the rows of g's DAG when they pay, and len[u], the part of N+(u) the
// middle-vertex walk still covers (all of it for a vertex not counted here).
// Otherwise leaves hub.n_list 0 and len empty; hub.no_room says that they would
// have paid.  (Required rows do not ask for room: a row of 512 bytes takes 57 ids
// or more out of the walk, and each of them saves the plan 12 bytes to sort and 8
// of index.)
int build_hub_rows(gary_graph *g, cudaStream_t s, Rows use, HubRows &hub, DevBuf<uint32_t> &len);

// The bits of word `word` (of a row) from bit position `from` on.
__device__ __forceinline__ uint32_t bits_from(uint32_t x, uint32_t word, uint32_t from) {
  const uint32_t b = word * 32;
  return from <= b ? x : from >= b + 32 ? 0u : x & (kFull << (from & 31u));
}

// Triangles u < v < w with w a hub past u's cut, for one counted u.  All 32
// lanes call; the count is split over them.
__device__ __forceinline__ uint32_t hub_vertex(const GraphView &g, const HubView &hub, uint32_t i, int lane) {
  const uint32_t u = hub.list[i];
  const uint2 ru = g.row[u];
  const uint32_t *au = g.adj + (uint64_t)ru.x * 4;
  const uint32_t d = ru.y, first = hub.first, top = first + (kHubIds - kHubTop);
  const uint4 *mine = hub.rows + (uint64_t)(u >= first ? u - first : kHubIds + i) * kHubRowQuads;
  const uint32_t *mine32 = reinterpret_cast<const uint32_t *>(mine);
  const uint32_t least = au[hub.cut[i]] - first;  // bit of the first counted id
  uint4 r = mine[lane];
  r.x = bits_from(r.x, 4 * lane, least);
  r.y = bits_from(r.y, 4 * lane + 1, least);
  r.z = bits_from(r.z, 4 * lane + 2, least);
  r.w = bits_from(r.w, 4 * lane + 3, least);
  uint32_t cnt = 0;
  uint32_t b = 0;
  // v below the last kHubTop ids: whole rows, from v's own position on
  for (; b < d; b += 32) {
    const uint32_t v = b + lane < d ? au[b + lane] : kSentinel;
    const unsigned in = __ballot_sync(kFull, v < top);
    if (!in) break;
    uint32_t row = kNoHubRow, from = 0;
    if (v < top) {
      if (v >= first) {
        row = v - first;
        from = row >> 7;
      } else {
        row = hub.rowof[v];
      }
    }
    unsigned without = __ballot_sync(kFull, row == kNoHubRow) & in;
    const uint32_t packed = row == kNoHubRow ? 31u << 27 : row | (from << 27);  // rows fit 27 bits (build_hub_rows)
    const uint32_t nv = 32 - __clz(in);
    for (uint32_t k = 0; k < nv; k += 4) {
      uint4 x[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t p = __shfl_sync(kFull, packed, k + j);
        const bool live = lane >= (p >> 27) && k + j < nv && !((without >> (k + j)) & 1u);
        x[j] = make_uint4(0, 0, 0, 0);
        if (live) x[j] = hub.rows[(uint64_t)(p & 0x7FFFFFFu) * kHubRowQuads + lane];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        cnt += __popc(x[j].x & r.x) + __popc(x[j].y & r.y) + __popc(x[j].z & r.z) + __popc(x[j].w & r.w);
    }
    // a v without a row has fewer than kHubMin hub neighbours, the last ids
    // of its list: each is looked up in u's row
    while (without) {
      const int k = __ffs(without) - 1;
      without &= without - 1;
      const uint2 rv = g.row[__shfl_sync(kFull, v, k)];
      const uint32_t *av = g.adj + (uint64_t)rv.x * 4;
      for (uint32_t j = lane; j < rv.y && j < kHubMin; j += 32) {
        const uint32_t w = av[rv.y - 1 - j];
        if (w >= first + least) cnt += (mine32[(w - first) >> 5] >> ((w - first) & 31u)) & 1u;
      }
    }
    if (nv < 32) {
      b += nv;
      break;
    }
  }
  // v among the last kHubTop ids: one word per lane
  const uint32_t r1 = bits_from(mine32[(kHubIds - kHubTop) / 32 + lane], (kHubIds - kHubTop) / 32 + lane, least);
  const uint32_t *rows32 = reinterpret_cast<const uint32_t *>(hub.rows) + (kHubIds - kHubTop) / 32 + lane;
  for (; b < d; b += 32) {
    const uint32_t nv = min(32u, d - b);
    const uint32_t v = lane < nv ? au[b + lane] - first : 0u;
    for (uint32_t k = 0; k < nv; k += 8) {
      uint32_t x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t p = __shfl_sync(kFull, v, k + j);
        x[j] = k + j < nv ? rows32[p * (kHubIds / 32)] : 0u;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) cnt += __popc(x[j] & r1);
    }
  }
  return cnt;
}

}  // namespace gary
