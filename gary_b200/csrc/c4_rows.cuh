// 4-cycles whose highest vertex is a hub.
//
// A 4-cycle with highest vertex u and opposite vertex w is a pair of the
// c(u, w) vertices v < u adjacent to both, so the cycles under u are the sum
// over w < u of C(c(u, w), 2).  The wedge kernels (patterns.cu) build the
// counters c(u, .) by walking every wedge u - v - w, and most wedges lie under
// the graph's few thousand hubs (78 % under the top 4096 ids at RMAT-22 ef16,
// 91 % under the top 8192).  For those u the counters are built from the other
// end: c(., w) for all hubs u at once is a sum of bit rows,
//     c(u, w) = sum over x in N(w) of [u in N(x), u > x],
// and a warp adds 512-byte rows (the hubs above x that x is adjacent to) into
// bit-sliced counters: slice k holds bit k of every hub's count.  A neighbour of
// w costs a row read and some ten logic operations a lane, whatever number of
// wedges (222 on average at RMAT-22) it stands for.
//
// Hubs are taken in slabs of kC4RowIds ids from the top down, as many as pay;
// the wedge kernels keep the vertices u below them.
#pragma once
#include <cstdint>

#include "graph.cuh"
#include "hub.cuh"
#include "internal.cuh"

namespace gary {

constexpr uint32_t kC4RowIds = 4096;
constexpr uint32_t kC4RowQuads = kC4RowIds / 128;
static_assert(kC4RowQuads == kWarp, "one quad of a row per lane");
constexpr int kC4MaxSlabs = 8;
// Wedges a row read must stand for (ms a count with the limit at 5 / 10 / 20 / 40:
// RMAT-20 ef16 8.39 / 8.39 / 9.00 / 8.99, RMAT-22 ef16 75.2 / 76.1 / 76.1 / 85.5;
// without rows 16.4 and 142.7).
constexpr uint64_t kC4RowWedges = 10;

// A shard's slabs take at most so many bytes per padded word of the graph's lists,
// or 128 MB.  The symmetric lists' own build takes more (two arrays of two 8-byte
// keys a word), so a shard is not refused for its rows on a device that could hold
// the lists.
constexpr uint64_t kC4ShardWordBytes = 24, kC4ShardLeast = 128u << 20;

// Rows over the ids [first, end): row p < end - first holds the neighbours of
// first + p above it, the rows after those (rowof) all of an x's below `first`.
struct C4Slab {
  DevBuf<uint4> rows;
  DevBuf<uint32_t> rowof;  // per vertex below `first`: its row, or the zero row
  uint32_t first = 0, end = 0, zero = 0;
};

struct C4Rows {
  C4Slab slab[kC4MaxSlabs];
  int slabs = 0;
  uint32_t lowest = 0;     // the wedge kernels take the u below
  bool shared = false;     // shards and whole counts have these same slabs
  // vertices w of two neighbours and more, by the counters their degree needs:
  // 5 and 8 slices in a warp's registers, and shared 32-bit counters of a CTA
  DevBuf<uint32_t> list;
  uint32_t n5 = 0, n8 = 0, n32 = 0;  // list: n5 vertices, then n8, then n32
  DevBuf<uint32_t> queue;            // three words a slab
};

// Builds the slabs that pay (none: slabs 0, lowest n): for a whole count those
// there is room for, for a shard (Rows::kRequired) those within kC4ShardWordBytes.
int build_c4_rows(gary_graph *g, cudaStream_t s, Rows use, C4Rows &r);

// Adds this shard's cycles to *d_out.
int launch_c4_rows(gary_graph *g, const C4Rows &r, unsigned long long *d_out, cudaStream_t s, uint32_t shard,
                   uint32_t nshards);

}  // namespace gary
