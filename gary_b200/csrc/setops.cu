// Batched set operations: the reference's include/ops layer as kernels.
//
//   gary_search_batch     binary_search (Search.cuh:48-61) and the two-phase
//                         cached search (Search.cuh:93-138) of many keys in one
//                         sorted list -- the kernels of test/SearchTest.cu:14-67
//   gary_intersect_batch  |A & B| (and A & B, sorted) for many pairs of sorted
//                         lists -- intersectBinarySearch (Intersection.cuh:18-135)
//                         and the merge / bitmap paths the reference stubs out
//                         (intersectMerge returns 0, Intersection.cuh:172-180)
//   gary_intersect_num_batch  the same counts restricted to members below a
//                         per-pair bound and outside a per-pair list of
//                         excluded ids -- the intersect_num family the
//                         reference leaves commented out (Intersection.cuh:361-485)
//
// CTAs claim chunks of pairs from a persistent queue and sort each chunk's
// pairs by what they need:
//   few ids (the shorter list at most kTinyKeys)  all such pairs of a warp
//           flattened over its lanes, one key a lane, a binary search each
//   long (more than kLongCost of work)  the whole CTA: every warp takes a part
//           of the shorter list and the stretch of the longer list its values
//           span
//   the rest  one warp a pair
// One warp per pair, whatever its size, left the last pairs of 65536 ids
// running alone for 1.4 ms of a launch, and a warp with nothing but a few
// dependent loads to do for most others (Zipf lengths: half the lists hold at
// most 8 ids).  AUTO, ms before and now: 2^20 pairs counted 3.48 / 2.67 (85 %
// of copy bandwidth in the lists' bytes), 50,001 pairs with lists 1.44 / 0.46.
// Variants, for a pair or a part of one:
//   MERGE   1024-id tiles of the longer list in shared memory, the shorter
//           list's values searched in them 32 at a time
//   SEARCH  lanes take the shorter list's values as keys and search the
//           longer list: phase 1 in shared samples, phase 2 in HBM
//   BITMAP  the longer list as a shared-memory bitmap over 32K-value windows,
//           the shorter list probed window by window
//   AUTO    SEARCH when the longer list is much longer, else MERGE
// Materialised outputs are sorted (every variant emits in key order through
// ballot compaction); the reference's are unsorted (Intersection.cuh:24-47).
#include <algorithm>
#include <cmath>
#include <vector>

#include "internal.cuh"
#include "pairs_gen.cuh"
#include "warp_ops.cuh"

namespace gary {
namespace {

constexpr uint32_t kSoWarpWords = 1024;  // per-warp shared words
constexpr uint32_t kSearchSamples = 256;
constexpr uint32_t kInf = 0xFFFFFFFFu;
constexpr uint32_t kTinyKeys = 16;
constexpr uint32_t kLongCost = 3072;  // ids read, or 8 per searched key
// Pairs a CTA of `warps` warps claims at a time, at most.
constexpr uint32_t chunk_pairs(int warps) { return warps <= 8 ? 128 : 224; }
// Batches of fewer pairs run 16-warp CTAs: the long pairs end sooner, and there
// are not enough pairs to hide them (ms, 16 / 8 warps: 50,001 Zipf pairs with
// lists 0.45 / 0.61, 1,000 pairs 0.046 / 0.059, 200,000 pairs 0.45 / 0.50,
// 300,000 pairs of up to 4096 ids 0.31 / 0.28, 2^20 pairs 2.72 / 2.60).
constexpr uint64_t kManyPairs = 1ull << 18;

struct PairView {
  const uint64_t *a_off, *b_off;
  const uint32_t *a_len, *b_len;
  const uint32_t *a, *b;
};

// Bounded / ancestor-filtered counts (the reference's intersect_num family,
// Intersection.cuh:361-485, left commented out there): per pair an exclusive
// upper bound on the members and a list of excluded ids.
struct PairFilter {
  const uint32_t *bound;   // per pair, or null
  const uint64_t *ex_off;  // per pair offsets into ex (npairs + 1), or null
  const uint32_t *ex;
};

// first index in [0, len) with l[i] >= x (all lanes compute the same answer)
__device__ __forceinline__ uint32_t so_lower_bound(const uint32_t *l, uint32_t len, uint32_t x) {
  uint32_t b = 0, e = len;
  while (b < e) {
    const uint32_t m = (b + e) >> 1;
    if (l[m] < x) b = m + 1;
    else e = m;
  }
  return b;
}

struct PairOut {
  uint64_t *counts;        // per pair, or null
  const uint64_t *out_off; // per pair, or null (count only)
  uint32_t *out;
};

__device__ __forceinline__ unsigned lanemask_lt(int lane) { return (1u << lane) - 1u; }

// first index in [0, len) with l[i] >= x, by all 32 lanes together: each step
// reads 32 evenly spaced ids (len 65536: 4 dependent loads instead of 16)
__device__ __forceinline__ uint32_t warp_lower_bound(const uint32_t *l, uint32_t len, uint32_t x, int lane) {
  uint32_t b = 0, e = len;  // the answer is in [b, e]
  while (e - b > 32) {
    const uint32_t step = (e - b + 31) / 32;
    const uint32_t at = min(b + (lane + 1) * step, e) - 1;  // last id of the lane's stretch
    const unsigned below = __ballot_sync(kFull, l[at] < x);
    const uint32_t k = __popc(below);  // stretches wholly below x
    b = min(b + k * step, e);
    e = min(b + step, e);
  }
  const bool below = b + lane < e && l[b + lane] < x;
  return b + __popc(__ballot_sync(kFull, below));
}

// ---- MERGE ------------------------------------------------------------------
__device__ uint32_t pair_merge(const uint32_t *S, uint32_t ls, const uint32_t *L, uint32_t ll, uint32_t *tile,
                               uint32_t *out, int lane) {
  uint32_t si = 0, found_total = 0;
  auto key = [&](uint32_t i) { return i < ls ? S[i] : 0u; };
  uint32_t x = key(lane), xn = key(32 + lane);  // this window of S and the next, in flight
  for (uint32_t li = 0; li < ll && si < ls; li += kSoWarpWords) {
    const uint32_t n = min(kSoWarpWords, ll - li);
    if (n == kSoWarpWords) {
#pragma unroll 8
      for (uint32_t k = 0; k < kSoWarpWords; k += 32) tile[k + lane] = L[li + k + lane];
    } else {
      for (uint32_t k = lane; k < n; k += 32) tile[k] = L[li + k];
    }
    __syncwarp();
    const uint32_t last = tile[n - 1];
    while (true) {
      // S[si .. si + 32), in x; the values past this tile wait for the next
      const bool in = si + lane < ls && x <= last;
      uint32_t pos = 0;  // ids of the tile below x
#pragma unroll
      for (uint32_t step = kSoWarpWords / 2; step; step >>= 1) {
        const uint32_t at = pos + step - 1;
        if (at < n && tile[at] < x) pos += step;
      }
      const bool hit = in && pos < n && tile[pos] == x;
      const unsigned hm = __ballot_sync(kFull, hit);
      if (out && hit) out[found_total + __popc(hm & lanemask_lt(lane))] = x;
      found_total += __popc(hm);
      const uint32_t done = __popc(__ballot_sync(kFull, in));
      si += done;
      if (done == 32) {
        x = xn;
        xn = key(si + 32 + lane);
      } else if (done) {
        x = key(si + lane);
        xn = key(si + 32 + lane);
      }
      if (done < 32 || si >= ls) break;
    }
    __syncwarp();
  }
  return found_total;
}

// ---- SEARCH (two-phase) ---------------------------------------------------
__device__ uint32_t pair_search(const uint32_t *S, uint32_t ls, const uint32_t *L, uint32_t ll,
                                uint32_t *cache, uint32_t *out, int lane) {
  // a few samples per key; each is a sector of HBM of its own
  const uint32_t want = ls <= 32 ? 64u : ls <= 64 ? 128u : kSearchSamples;
  const uint32_t ns = ll < want ? ll : want;
  for (uint32_t k = lane; k < ns; k += 32) cache[k] = L[(uint64_t)k * ll / ns];
  __syncwarp();
  uint32_t found_total = 0;
  uint32_t xn = lane < ls ? S[lane] : 0u;
  for (uint32_t b = 0; b < ls; b += 32) {
    const bool ok = b + lane < ls;
    const uint32_t x = xn;
    xn = b + 32 + lane < ls ? S[b + 32 + lane] : 0u;
    const bool hit = ok && search_2phase(L, ll, cache, ns, x);
    const unsigned hm = __ballot_sync(kFull, hit);
    if (out && hit) out[found_total + __popc(hm & lanemask_lt(lane))] = x;
    found_total += __popc(hm);
  }
  __syncwarp();
  return found_total;
}

// ---- BITMAP ---------------------------------------------------------------
// Windows of W = 32 * kSoWarpWords values.  In each non-empty window the
// warp sets the bits of L's values, probes S's values, then clears the words
// it set (so the bitmap starts every window zeroed).
__device__ uint32_t pair_bitmap(const uint32_t *S, uint32_t ls, const uint32_t *L, uint32_t ll,
                                uint32_t *bm, uint32_t *out, int lane) {
  constexpr uint32_t W = 32 * kSoWarpWords;
  uint32_t si = 0, li = 0, found_total = 0;
  while (si < ls && li < ll) {
    const uint32_t s0 = S[si], l0 = L[li];
    const uint32_t w0 = (s0 > l0 ? s0 : l0) / W * W;  // window holding the larger head
    const uint64_t w1 = (uint64_t)w0 + W;
    // skip values below the window, and find its end
    auto from = [&](const uint32_t *X, uint32_t n, uint32_t i, uint64_t v) {
      return v > kInf ? n : i + warp_lower_bound(X + i, n - i, (uint32_t)v, lane);
    };
    const uint32_t sb = from(S, ls, si, w0), se = from(S, ls, sb, w1);
    const uint32_t lb = from(L, ll, li, w0), le = from(L, ll, lb, w1);
    for (uint32_t k = lb + lane; k < le; k += 32) {
      const uint32_t o = L[k] - w0;
      atomicOr(&bm[o >> 5], 1u << (o & 31));
    }
    __syncwarp();
    for (uint32_t k = sb; k < se; k += 32) {
      const bool ok = k + lane < se;
      const uint32_t x = ok ? S[k + lane] : w0;
      const uint32_t o = x - w0;
      const bool hit = ok && ((bm[o >> 5] >> (o & 31)) & 1u);
      const unsigned hm = __ballot_sync(kFull, hit);
      if (out && hit) out[found_total + __popc(hm & lanemask_lt(lane))] = x;
      found_total += __popc(hm);
    }
    __syncwarp();
    for (uint32_t k = lb + lane; k < le; k += 32) bm[(L[k] - w0) >> 5] = 0u;
    __syncwarp();
    si = se;
    li = le;
  }
  return found_total;
}

// A pair as the kernel runs it: S the shorter list (ties: A), L the longer.
struct PairJob {
  const uint32_t *S, *L;
  uint32_t ls, ll;
};

__device__ __forceinline__ uint32_t warp_pair(int variant, const PairJob &j, uint32_t *mine, uint32_t *out, int lane) {
  if (variant == GARY_ISECT_MERGE) return pair_merge(j.S, j.ls, j.L, j.ll, mine, out, lane);
  if (variant == GARY_ISECT_SEARCH) return pair_search(j.S, j.ls, j.L, j.ll, mine, out, lane);
  return pair_bitmap(j.S, j.ls, j.L, j.ll, mine, out, lane);
}

// AUTO searches once the longer list exceeds half of |S| log2 |L|.
__device__ __forceinline__ int pair_variant(int variant, uint32_t ls, uint32_t ll) {
  if (variant != GARY_ISECT_AUTO) return variant;
  const uint32_t lg = 32 - __clz(ll);
  return 2ull * ll > (uint64_t)ls * lg ? GARY_ISECT_SEARCH : GARY_ISECT_MERGE;
}

template <int kSoWarps>
__global__ void __launch_bounds__(kSoWarps * 32)
    k_intersect_pairs(PairView pv, uint64_t npairs, uint32_t chunk, int variant, PairOut po, PairFilter pf,
                      unsigned long long *queue, unsigned long long *total) {
  extern __shared__ __align__(16) uint32_t smem[];  // kSoWarps * kSoWarpWords
  constexpr uint32_t kChunkPairs = chunk_pairs(kSoWarps);
  static_assert(kChunkPairs <= 256 && kChunkPairs <= kSoWarps * 32, "a thread per pair, numbered in a byte");
  __shared__ PairJob jobs[kChunkPairs];
  __shared__ uint32_t found[kChunkPairs];  // per pair of the chunk
  __shared__ uint8_t mid[kChunkPairs], big[kChunkPairs];
  __shared__ uint32_t n_mid, n_big, next_mid;
  __shared__ uint32_t piece[kSoWarps];
  __shared__ unsigned long long s_first;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *mine = smem + warp * kSoWarpWords;
  for (uint32_t i = lane; i < kSoWarpWords; i += 32) mine[i] = 0u;
  unsigned long long local = 0;
  while (true) {
    if (threadIdx.x == 0) {
      s_first = atomicAdd(queue, (unsigned long long)chunk);
      n_mid = n_big = next_mid = 0;
    }
    __syncthreads();
    const uint64_t first = s_first;
    if (first >= npairs) break;
    const uint32_t np = (uint32_t)min((unsigned long long)chunk, (unsigned long long)(npairs - first));
    if (threadIdx.x < np) {
      const uint64_t p = first + threadIdx.x;
      uint32_t la = pv.a_len[p], lb = pv.b_len[p];
      const uint32_t *A = pv.a + pv.a_off[p], *B = pv.b + pv.b_off[p];
      if (pf.bound) {  // members < bound only: both lists end at the bound
        const uint32_t bound = pf.bound[p];
        la = so_lower_bound(A, la, bound);
        lb = so_lower_bound(B, lb, bound);
      }
      const bool a_short = la <= lb;
      const PairJob j{a_short ? A : B, a_short ? B : A, a_short ? la : lb, a_short ? lb : la};
      jobs[threadIdx.x] = j;
      found[threadIdx.x] = 0;
      if (j.ls > kTinyKeys) {
        // work in loads: a search's keys cost several each, and a bitmap's may
        // each lie in a window of its own
        const int v = pair_variant(variant, j.ls, j.ll);
        const uint64_t cost = v == GARY_ISECT_SEARCH ? 8ull * j.ls : v == GARY_ISECT_BITMAP ? 64ull * j.ls : (uint64_t)j.ls + j.ll;
        if (cost > kLongCost) big[atomicAdd(&n_big, 1u)] = (uint8_t)threadIdx.x;
        else mid[atomicAdd(&n_mid, 1u)] = (uint8_t)threadIdx.x;
      }
    }
    __syncthreads();
    {  // pairs of few ids: this warp's share of the chunk, one key a lane
      const uint32_t share = (np + kSoWarps - 1) / kSoWarps, q0 = warp * share;
      const uint32_t ls = lane < share && q0 + lane < np ? jobs[q0 + lane].ls : 0u;
      const uint32_t keys = ls <= kTinyKeys ? ls : 0u;
      const uint32_t incl = warp_inclusive_sum(keys, lane);
      const uint32_t all = __shfl_sync(kFull, incl, 31);
      WarpRuns runs(incl - keys, keys, lane);
      for (uint32_t pb = 0; pb < all; pb += 32) {
        const int o = (int)runs.owner(pb);
        const uint32_t start = __shfl_sync(kFull, incl - keys, o);
        const bool on = pb + lane < all;
        bool hit = false;
        uint32_t x = 0;
        if (on) {
          const PairJob j = jobs[q0 + o];
          x = j.S[pb + lane - start];
          uint32_t base = 0;
          for (uint32_t n = j.ll; n > 1;) {  // ids below x: at least base, at most base + n - 1 but for the last
            const uint32_t half = n >> 1;
            if (j.L[base + half - 1] < x) base += half;
            n -= half;
          }
          hit = j.L[base] == x;
        }
        const unsigned hm = __ballot_sync(kFull, hit);
        // the lanes of this pair in the batch: from its first key on
        const uint32_t from = start > pb ? start - pb : 0u;
        const unsigned before = hm & lanemask_lt(lane) & ~lanemask_lt(from);
        const uint32_t had = on ? found[q0 + o] : 0u;
        if (po.out_off && hit) po.out[po.out_off[first + q0 + o] + had + __popc(before)] = x;
        __syncwarp();
        const int next = __shfl_down_sync(kFull, on ? o : -1, 1);
        if (on && (lane == 31 || next != o)) found[q0 + o] = had + __popc(before) + hit;
        __syncwarp();
      }
    }
    while (true) {  // one warp a pair
      uint32_t m = 0;
      if (lane == 0) m = atomicAdd(&next_mid, 1u);
      m = __shfl_sync(kFull, m, 0);
      if (m >= n_mid) break;
      const uint32_t q = mid[m];
      const PairJob j = jobs[q];
      uint32_t *out = po.out_off ? po.out + po.out_off[first + q] : nullptr;
      const uint32_t c = warp_pair(pair_variant(variant, j.ls, j.ll), j, mine, out, lane);
      if (lane == 0) found[q] = c;
    }
    for (uint32_t i = 0; i < n_big; ++i) {  // the CTA together, a part of S a warp
      const uint32_t q = big[i];
      const PairJob j = jobs[q];
      const int v = pair_variant(variant, j.ls, j.ll);
      const uint32_t s0 = (uint32_t)((uint64_t)j.ls * warp / kSoWarps), s1 = (uint32_t)((uint64_t)j.ls * (warp + 1) / kSoWarps);
      PairJob sub{nullptr, nullptr, 0, 0};
      if (s0 < s1) {  // more ids than warps: always
        const uint32_t l0 = warp_lower_bound(j.L, j.ll, j.S[s0], lane);
        const uint32_t l1 = l0 + warp_lower_bound(j.L + l0, j.ll - l0, j.S[s1 - 1], lane);
        sub = PairJob{j.S + s0, j.L + l0, s1 - s0, min(l1 + 1, j.ll) - l0};
      }
      uint32_t c = 0;
      if (sub.ll) c = warp_pair(v, sub, mine, nullptr, lane);
      if (!po.out_off) {
        if (lane == 0 && c) atomicAdd(&found[q], c);
        continue;
      }
      // the places of the parts follow from their counts: a second pass writes
      if (lane == 0) piece[warp] = c;
      __syncthreads();
      uint32_t at = 0, sum = 0;
      for (int w = 0; w < kSoWarps; ++w) {
        at += w < warp ? piece[w] : 0u;
        sum += piece[w];
      }
      if (c) warp_pair(v, sub, mine, po.out + po.out_off[first + q] + at, lane);
      if (threadIdx.x == 0) found[q] = sum;
      __syncthreads();
    }
    __syncthreads();
    if (pf.ex_off) {  // excluded ids that are members (each id once)
      for (uint32_t q = warp; q < np; q += kSoWarps) {
        const PairJob j = jobs[q];
        if (!j.ls) continue;
        const uint64_t e0 = pf.ex_off[first + q], e1 = pf.ex_off[first + q + 1];
        const uint32_t bound = pf.bound ? pf.bound[first + q] : kInf;
        uint32_t drop = 0;
        for (uint64_t k = e0 + lane; k < e1; k += 32) {
          const uint32_t x = pf.ex[k];
          bool is_first = x < bound;
          for (uint64_t i = e0; is_first && i < k; ++i) is_first = pf.ex[i] != x;
          if (is_first) {
            const uint32_t is = so_lower_bound(j.S, j.ls, x), il = so_lower_bound(j.L, j.ll, x);
            drop += is < j.ls && j.S[is] == x && il < j.ll && j.L[il] == x;
          }
        }
        for (int o = 16; o; o >>= 1) drop += __shfl_xor_sync(kFull, drop, o);
        if (lane == 0) found[q] -= drop;
      }
      __syncthreads();
    }
    if (threadIdx.x < np) {
      const uint32_t c = found[threadIdx.x];
      if (po.counts) po.counts[first + threadIdx.x] = c;
      local += c;
    }
    // the next chunk's set-up is ordered after these reads by its claim's barrier
  }
  local = warp_sum_u64(local);
  if (lane == 0 && total && local) atomicAdd(total, local);
}

// One launch over all pairs.
template <int W>
int launch_pairs(const PairView &pv, uint64_t npairs, int variant, const PairOut &po, const PairFilter &pf,
                 uint64_t *d_queue, uint64_t *d_total, cudaStream_t s) {
  constexpr size_t smem = (size_t)W * kSoWarpWords * 4;
  auto kern = k_intersect_pairs<W>;
  static bool done[64] = {false};  // shared memory beyond the default limit, once per device
  const int dev = device_ordinal();
  if (dev >= 64 || !done[dev]) {
    GARY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (dev < 64) done[dev] = true;
  }
  int per_sm = 0;
  GARY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, W * 32, smem));
  if (per_sm < 1) per_sm = 1;
  const unsigned grid = (unsigned)(sm_count() * per_sm);
  // pairs per claim: some claims for every CTA, a pair for every warp
  const uint64_t c = npairs / ((W > 8 ? 2ull : 4ull) * grid);
  const uint32_t chunk = c < W ? (uint32_t)W : c > chunk_pairs(W) ? chunk_pairs(W) : (uint32_t)c;
  kern<<<grid, W * 32, smem, s>>>(pv, npairs, chunk, variant, po, pf, reinterpret_cast<unsigned long long *>(d_queue),
                                  reinterpret_cast<unsigned long long *>(d_total));
  GARY_CUDA(cudaGetLastError());
  return GARY_OK;
}

int launch_pairs_any(const PairView &pv, uint64_t npairs, int variant, const PairOut &po, const PairFilter &pf,
                     uint64_t *d_queue, uint64_t *d_total, cudaStream_t s) {
  return npairs >= kManyPairs ? launch_pairs<8>(pv, npairs, variant, po, pf, d_queue, d_total, s)
                              : launch_pairs<16>(pv, npairs, variant, po, pf, d_queue, d_total, s);
}

// ---- search batch ----------------------------------------------------------
__global__ void __launch_bounds__(256)
    k_search_batch(const uint32_t *__restrict__ list, uint64_t len, const uint32_t *__restrict__ keys,
                   uint64_t nkeys, uint32_t cache_n, uint8_t *__restrict__ found,
                   unsigned long long *count) {
  extern __shared__ uint32_t cache[];
  for (uint32_t k = threadIdx.x; k < cache_n; k += blockDim.x) cache[k] = list[(uint64_t)k * len / cache_n];
  __syncthreads();
  unsigned long long local = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nkeys;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t x = keys[i];
    uint32_t f;
    if (cache_n) {
      f = search_2phase(list, (uint32_t)len, cache, cache_n, x);
    } else {
      uint64_t b = 0, e = len;
      f = 0;
      while (b < e) {
        const uint64_t mid = (b + e) >> 1;
        const uint32_t v = list[mid];
        if (v == x) { f = 1; break; }
        if (v < x) b = mid + 1;
        else e = mid;
      }
    }
    if (found) found[i] = (uint8_t)f;
    local += f;
  }
  if (count) {
    local = warp_sum_u64(local);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(count, local);
  }
}

// Many keys: the list's separators are kept in shared memory as a search tree
// of up to 2^15 - 1 nodes (node k's children are 2k and 2k + 1, so that the nodes
// of a level lie side by side and the lanes of a warp read different banks), and
// each thread takes kSearchIlp keys at a time, whose loads overlap.  A key costs
// `levels` shared loads and then a binary search of the len / 2^levels ids of
// its bucket, begun by interpolation.  What bounds a search is the sectors it
// takes from L2 or HBM, one per step but the last three: 10 with 1024 samples of
// a 4 M list, 2 to 3 here (4 M keys in 4 M ids 217 -> 139 us, 32 M in 32 M 8.3 ->
// 1.4 ms).
constexpr int kSearchThreads = 1024;
constexpr int kSearchIlp = 4;
constexpr int kSearchMaxLevels = 15;

// The node of the r-th separator in order (r from 1).
__device__ __forceinline__ uint32_t separator(uint32_t r, int levels) {
  const int z = __ffs(r) - 1;  // levels above the last
  return (1u << (levels - 1 - z)) + (r >> (z + 1));
}

__global__ void __launch_bounds__(kSearchThreads)
    k_search_tree(const uint32_t *__restrict__ list, uint32_t len, const uint32_t *__restrict__ keys, uint64_t nkeys,
                  int levels, uint8_t *__restrict__ found, unsigned long long *count) {
  extern __shared__ uint32_t tree[];  // 2^levels words, node k at k
  for (uint32_t k = threadIdx.x; k < (1u << levels); k += kSearchThreads) {
    if (!k) continue;
    const int l = 31 - __clz(k);  // node k: number k - 2^l of level l
    const uint32_t rank = (2 * (k - (1u << l)) + 1) << (levels - 1 - l);  // separators up to it, in order
    tree[k] = list[(uint64_t)rank * len >> levels];
  }
  const uint32_t last = list[len - 1];
  __syncthreads();
  uint32_t local = 0;
  const uint64_t step = (uint64_t)gridDim.x * kSearchThreads * kSearchIlp;
  for (uint64_t i0 = (uint64_t)blockIdx.x * kSearchThreads * kSearchIlp + threadIdx.x; i0 < nkeys; i0 += step) {
    uint32_t x[kSearchIlp], k[kSearchIlp], n[kSearchIlp], lo[kSearchIlp], hi[kSearchIlp];
#pragma unroll
    for (int j = 0; j < kSearchIlp; ++j) {
      const uint64_t i = i0 + (uint64_t)j * kSearchThreads;
      x[j] = i < nkeys ? keys[i] : 0u;
      k[j] = 1;
    }
    for (int l = 0; l < levels; ++l)
#pragma unroll
      for (int j = 0; j < kSearchIlp; ++j) k[j] = 2 * k[j] + (tree[k[j]] <= x[j] ? 1u : 0u);
#pragma unroll
    for (int j = 0; j < kSearchIlp; ++j) {  // bucket: [first, first + n)
      const uint64_t b = k[j] - (1u << levels);
      const uint32_t first = (uint32_t)(b * len >> levels);
      n[j] = (uint32_t)((b + 1) * len >> levels) - first;
      k[j] = first;
      // the separators around it (the outermost buckets lack one)
      lo[j] = b ? tree[separator((uint32_t)b, levels)] : 0u;
      hi[j] = b + 1 < (1u << levels) ? tree[separator((uint32_t)b + 1, levels)] : last;
    }
    // x can only be at [k, k + n).  One probe where it would be if the bucket's
    // ids were evenly spaced, one eight ids further towards it, then bisection:
    // two or three sectors where ids are spread evenly, the bisection's five
    // and a little where they are not.
    auto probe = [&](int j, uint32_t at) {  // at < n
      const bool less = list[k[j] + at] < x[j];
      k[j] += less ? at + 1 : 0u;
      n[j] = less ? n[j] - at - 1 : at + 1;
      return less;
    };
    uint32_t g[kSearchIlp];
#pragma unroll
    for (int j = 0; j < kSearchIlp; ++j) {
      const float d = (float)(x[j] - lo[j]) / (float)max(hi[j] - lo[j], 1u);
      g[j] = x[j] < lo[j] ? 0u : min((uint32_t)(d * (float)n[j]), n[j] - 1);
    }
    bool less[kSearchIlp];
#pragma unroll
    for (int j = 0; j < kSearchIlp; ++j) less[j] = probe(j, g[j]);
#pragma unroll
    for (int j = 0; j < kSearchIlp; ++j)
      if (n[j] > 8) probe(j, less[j] ? 7u : n[j] - 9u);
    while (true) {
      uint32_t most = 0;
#pragma unroll
      for (int j = 0; j < kSearchIlp; ++j) most = max(most, n[j]);
      if (most <= 1) break;
#pragma unroll
      for (int j = 0; j < kSearchIlp; ++j)
        if (n[j] > 1) probe(j, (n[j] >> 1) - 1);
    }
#pragma unroll
    for (int j = 0; j < kSearchIlp; ++j) {
      const uint64_t i = i0 + (uint64_t)j * kSearchThreads;
      if (i >= nkeys) continue;
      const uint32_t f = n[j] && list[k[j]] == x[j];
      if (found) found[i] = (uint8_t)f;
      local += f;
    }
  }
  if (count) {
    const uint32_t sum = __reduce_add_sync(kFull, local);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(count, (unsigned long long)sum);
  }
}

// Levels of the tree: no more separators than a CTA's share of the keys (each
// is a scattered read, which the keys must pay back), buckets of 8 ids or more.
// Below 10 levels (lists of up to 8 K ids: 4 M keys in 2000 ids 62 us plain, 69 with
// a tree), or with too few keys for every SM, the plain kernel is used.
int search_levels(uint64_t len, uint64_t nkeys) {
  const uint64_t most = std::min<uint64_t>(len / 8, nkeys / (uint64_t)sm_count());
  int l = 0;
  while (l < kSearchMaxLevels && (2ull << l) <= most) ++l;
  return l;
}

// ---- pair generation -------------------------------------------------------
__global__ void k_pair_lengths(PairGen pg, uint64_t first, uint64_t npairs, uint32_t *__restrict__ la,
                               uint32_t *__restrict__ lb, uint64_t *__restrict__ qa,
                               uint64_t *__restrict__ qb) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < npairs;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t a = pg.length(first + i, 0), b = pg.length(first + i, 1);
    la[i] = a;
    lb[i] = b;
    qa[i] = (a + 3) / 4;  // lists padded to 16 bytes
    qb[i] = (b + 3) / 4;
  }
}

__global__ void k_pair_values(PairGen pg, uint64_t first, uint64_t npairs,
                              const uint32_t *__restrict__ la, const uint32_t *__restrict__ lb,
                              const uint64_t *__restrict__ a_off, const uint64_t *__restrict__ b_off,
                              uint32_t *__restrict__ a, uint32_t *__restrict__ b) {
  const int lane = threadIdx.x & 31;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i = warp; i < npairs; i += nwarps) {
    const uint32_t A = la[i], B = lb[i];
    const uint32_t pa = (A + 3) & ~3u, pb = (B + 3) & ~3u;
    for (uint32_t j = lane; j < pa; j += 32)
      a[a_off[i] + j] = j < A ? pg.value(first + i, 0, j, A, B) : kSentinel;
    for (uint32_t j = lane; j < pb; j += 32)
      b[b_off[i] + j] = j < B ? pg.value(first + i, 1, j, A, B) : kSentinel;
  }
}

PairGen make_gen(uint64_t seed, uint32_t nmax, const uint64_t *cdf, double overlap, uint64_t range) {
  PairGen g;
  g.key = pmix64(seed ^ 0x7F4A7C15F39CC060ull);
  g.range = range;
  const double t = overlap <= 0 ? 0.0 : (overlap >= 1 ? 4294967295.0 : overlap * 4294967296.0);
  g.overlap_thresh = (uint32_t)t;
  g.nmax = nmax;
  g.cdf = cdf;
  return g;
}

}  // namespace
}  // namespace gary

using namespace gary;

extern "C" int gary_zipf_table(uint32_t nmax, double s, uint64_t *cdf) {
  GARY_CHECK_ARG(nmax >= 1 && cdf, "need nmax >= 1 and an output table");
  GARY_CHECK_ARG(s > 0, "exponent must be positive");
  std::vector<long double> w(nmax);
  long double H = 0;
  for (uint32_t x = nmax; x >= 1; --x) {  // small terms first
    w[x - 1] = powl((long double)x, -(long double)s);
    H += w[x - 1];
  }
  long double c = 0;
  for (uint32_t k = 0; k + 1 < nmax; ++k) {
    c += w[k];
    long double f = c / H * 18446744073709551616.0L;
    cdf[k] = f >= 18446744073709551615.0L ? ~0ull : (uint64_t)f;
  }
  cdf[nmax - 1] = ~0ull;
  return GARY_OK;
}

extern "C" int gary_gen_pair_host(uint64_t seed, uint64_t pair, uint32_t nmax, const uint64_t *cdf,
                                  double overlap, uint64_t range, uint32_t *a, uint32_t *la,
                                  uint32_t *b, uint32_t *lb) {
  GARY_CHECK_ARG(cdf && la && lb, "NULL argument");
  GARY_CHECK_ARG(range >= (uint64_t)nmax && range <= (1ull << 32), "range must be in [nmax, 2^32]");
  const PairGen g = make_gen(seed, nmax, cdf, overlap, range);
  const uint32_t A = g.length(pair, 0), B = g.length(pair, 1);
  *la = A;
  *lb = B;
  if (a)
    for (uint32_t j = 0; j < A; ++j) a[j] = g.value(pair, 0, j, A, B);
  if (b)
    for (uint32_t j = 0; j < B; ++j) b[j] = g.value(pair, 1, j, A, B);
  return GARY_OK;
}

extern "C" int gary_gen_pairs_lengths(uint64_t seed, uint64_t first, uint64_t npairs, uint32_t nmax,
                                      const uint64_t *d_cdf, uint32_t *d_la, uint32_t *d_lb,
                                      uint64_t *d_qa, uint64_t *d_qb, void *stream) {
  GARY_CHECK_ARG(npairs == 0 || (d_cdf && d_la && d_lb && d_qa && d_qb), "NULL argument");
  if (!npairs) return GARY_OK;
  const PairGen g = make_gen(seed, nmax, d_cdf, 0.0, 1ull << 26);
  const uint64_t blocks = (npairs + 255) / 256, cap = (uint64_t)sm_count() * 16;
  k_pair_lengths<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, as_stream(stream)>>>(
      g, first, npairs, d_la, d_lb, d_qa, d_qb);
  GARY_CUDA(cudaGetLastError());
  return GARY_OK;
}

extern "C" int gary_gen_pairs_values(uint64_t seed, uint64_t first, uint64_t npairs, uint32_t nmax,
                                     const uint64_t *d_cdf, double overlap, uint64_t range,
                                     const uint32_t *d_la, const uint32_t *d_lb,
                                     const uint64_t *d_a_off, const uint64_t *d_b_off, uint32_t *d_a,
                                     uint32_t *d_b, void *stream) {
  GARY_CHECK_ARG(npairs == 0 || (d_cdf && d_la && d_lb && d_a_off && d_b_off && d_a && d_b),
                 "NULL argument");
  GARY_CHECK_ARG(range >= (uint64_t)nmax && range <= (1ull << 32), "range must be in [nmax, 2^32]");
  if (!npairs) return GARY_OK;
  const PairGen g = make_gen(seed, nmax, d_cdf, overlap, range);
  const uint64_t blocks = (npairs * 32 + 255) / 256, cap = (uint64_t)sm_count() * 16;
  k_pair_values<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, as_stream(stream)>>>(
      g, first, npairs, d_la, d_lb, d_a_off, d_b_off, d_a, d_b);
  GARY_CUDA(cudaGetLastError());
  return GARY_OK;
}

extern "C" int gary_intersect_batch(uint64_t npairs, const uint64_t *d_a_off, const uint32_t *d_a_len,
                                    const uint32_t *d_a, const uint64_t *d_b_off,
                                    const uint32_t *d_b_len, const uint32_t *d_b, int variant,
                                    uint64_t *d_counts, const uint64_t *d_out_off, uint32_t *d_out,
                                    uint64_t *d_total, uint64_t *d_queue, void *stream) {
  GARY_CHECK_ARG(variant >= GARY_ISECT_AUTO && variant <= GARY_ISECT_BITMAP, "unknown variant %d",
                 variant);
  GARY_CHECK_ARG(npairs == 0 || (d_a_off && d_a_len && d_a && d_b_off && d_b_len && d_b),
                 "NULL list argument");
  GARY_CHECK_ARG(!d_out_off || d_out, "d_out is NULL while d_out_off is set");
  GARY_CHECK_ARG(d_queue != nullptr, "d_queue (one device word of scheduler state) is NULL");
  cudaStream_t s = as_stream(stream);
  GARY_CUDA(cudaMemsetAsync(d_queue, 0, 8, s));
  if (d_total) GARY_CUDA(cudaMemsetAsync(d_total, 0, 8, s));
  if (!npairs) return GARY_OK;
  const PairView pv{d_a_off, d_b_off, d_a_len, d_b_len, d_a, d_b};
  const PairOut po{d_counts, d_out_off, d_out};
  return launch_pairs_any(pv, npairs, variant, po, PairFilter{nullptr, nullptr, nullptr}, d_queue, d_total, s);
}

extern "C" int gary_intersect_num_batch(uint64_t npairs, const uint64_t *d_a_off, const uint32_t *d_a_len,
                                        const uint32_t *d_a, const uint64_t *d_b_off,
                                        const uint32_t *d_b_len, const uint32_t *d_b, int variant,
                                        const uint32_t *d_bound, const uint64_t *d_ex_off,
                                        const uint32_t *d_ex, uint64_t *d_counts, uint64_t *d_total,
                                        uint64_t *d_queue, void *stream) {
  GARY_CHECK_ARG(variant >= GARY_ISECT_AUTO && variant <= GARY_ISECT_BITMAP, "unknown variant %d",
                 variant);
  GARY_CHECK_ARG(npairs == 0 || (d_a_off && d_a_len && d_a && d_b_off && d_b_len && d_b),
                 "NULL list argument");
  GARY_CHECK_ARG(!d_ex_off || d_ex, "d_ex is NULL while d_ex_off is set");
  GARY_CHECK_ARG(d_queue != nullptr, "d_queue (one device word of scheduler state) is NULL");
  cudaStream_t s = as_stream(stream);
  GARY_CUDA(cudaMemsetAsync(d_queue, 0, 8, s));
  if (d_total) GARY_CUDA(cudaMemsetAsync(d_total, 0, 8, s));
  if (!npairs) return GARY_OK;
  const PairView pv{d_a_off, d_b_off, d_a_len, d_b_len, d_a, d_b};
  const PairOut po{d_counts, nullptr, nullptr};
  return launch_pairs_any(pv, npairs, variant, po, PairFilter{d_bound, d_ex_off, d_ex}, d_queue, d_total, s);
}

extern "C" int gary_search_batch(const uint32_t *d_list, uint64_t len, const uint32_t *d_keys,
                                 uint64_t nkeys, uint32_t cache_entries, uint8_t *d_found,
                                 uint64_t *d_count, void *stream) {
  GARY_CHECK_ARG(len < (1ull << 32), "list longer than 2^32-1");
  GARY_CHECK_ARG(cache_entries <= 8192, "cache_entries must be <= 8192");
  GARY_CHECK_ARG(nkeys == 0 || (d_keys && (d_list || len == 0)), "NULL argument");
  cudaStream_t s = as_stream(stream);
  if (d_count) GARY_CUDA(cudaMemsetAsync(d_count, 0, 8, s));
  if (!nkeys) return GARY_OK;
  if (len == 0) {
    if (d_found) GARY_CUDA(cudaMemsetAsync(d_found, 0, nkeys, s));
    return GARY_OK;
  }
  const int levels = search_levels(len, nkeys);
  if (levels >= 10 && nkeys >= (uint64_t)sm_count() * kSearchThreads * kSearchIlp) {
    const size_t smem = (size_t)4 << levels;
    static bool done[64] = {false};  // shared memory beyond the default limit, once per device
    const int dev = device_ordinal();
    if (dev >= 64 || !done[dev]) {
      GARY_CUDA(cudaFuncSetAttribute(k_search_tree, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 << kSearchMaxLevels));
      if (dev < 64) done[dev] = true;
    }
    const uint64_t per_sm = levels < kSearchMaxLevels ? 2 : 1;
    const uint64_t blocks = (nkeys + kSearchThreads * kSearchIlp - 1) / (kSearchThreads * kSearchIlp);
    const uint64_t most = (uint64_t)sm_count() * per_sm;
    k_search_tree<<<(unsigned)(blocks < most ? blocks : most), kSearchThreads, smem, s>>>(
        d_list, (uint32_t)len, d_keys, nkeys, levels, d_found, reinterpret_cast<unsigned long long *>(d_count));
    GARY_CUDA(cudaGetLastError());
    return GARY_OK;
  }
  const uint32_t cn = cache_entries && cache_entries > len ? (uint32_t)len : cache_entries;
  const uint64_t blocks = (nkeys + 255) / 256, cap = (uint64_t)sm_count() * 8;
  k_search_batch<<<(unsigned)(blocks < cap ? blocks : cap), 256, cn * 4, s>>>(
      d_list, len, d_keys, nkeys, cn, d_found, reinterpret_cast<unsigned long long *>(d_count));
  GARY_CUDA(cudaGetLastError());
  return GARY_OK;
}
