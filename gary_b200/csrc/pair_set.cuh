// A warp's shared-memory set of sparse ids (N+(v) over an id span too wide for
// a bitmap): two tables of 16-bit entries, one candidate slot of an id in each.
//
// An id x splits into its low k bits and q = x >> k.  It lies in slot
// x mod 2^k of the first table or in slot (x + C q) mod 2^k of the second, and
// the entry there is q: slot and entry together give x back, so 16 bits hold
// an id exactly (for ids below 0xFFFF << k).  A probe is two independent
// 2-byte shared loads and two compares, with no loop and no branch.  The
// 4-slot hash buckets it stands in for read 16 bytes a probe in a loop that
// diverges: at RMAT-22 ef16 the warps spent 25 cycles a probe in buckets
// against 6 in bitmaps.  A count with pair sets instead of buckets: RMAT-20
// ef16 698 -> 590 us, RMAT-22 ef16 4.57 -> 3.76 ms, RMAT-24 ef32 71.3 -> 68.7 ms.
// Lists of 513 to 896 ids fit too, but at RMAT-24 they count faster as CTA
// tiles (71.3 ms with them here).
//
// Building: every id is stored in the first table, the ids found overwritten
// in the second, and those overwritten there (about 1 % at 512 ids) are placed
// one by one with evictions (cuckoo hashing, Pagh and Rodler 2004).  Tables
// are at most a quarter full; a placement that does not end after kPairKicks
// evictions gives up, and the caller uses another set.
#pragma once
#include <cstdint>

#include "internal.cuh"

namespace gary {

constexpr int kPairMaxLog = 10;                       // slots per table, at most
constexpr uint32_t kPairTableBytes = 2u << kPairMaxLog;
constexpr uint32_t kPairWords = 2 * kPairTableBytes / 4;  // the warp's 4 KiB region
constexpr uint32_t kPairMaxIds = 512;
constexpr uint32_t kPairMul = 0x9E3779B1u;
constexpr uint32_t kPairEmpty = 0xFFFFu;
constexpr uint32_t kPairKicks = 64;

// Low bits for a list of d ids: four slots (both tables) or more per id, and
// enough bits that no id below n, member or not, has the entry of an empty
// slot.  (List padding has one too large for any entry.)  0: not representable.
__host__ __device__ __forceinline__ int pair_log(uint32_t d, uint32_t n) {
  int k = 6;
  while (k < kPairMaxLog && ((1u << k) < 2 * d || ((n - 1) >> k) >= kPairEmpty)) ++k;
  return d <= kPairMaxIds && ((n - 1) >> k) < kPairEmpty ? k : 0;
}

struct PairSet {
  uint32_t base;  // shared address of the region, a multiple of its size
  uint32_t mask;  // (2^k - 1) * 2: byte offset of a slot
  int k;
  __device__ __forceinline__ static uint32_t load(uint32_t addr) {
    uint16_t e;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(e) : "r"(addr));
    return e;
  }
  __device__ __forceinline__ static void store(uint32_t addr, uint32_t q) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"((uint16_t)q) : "memory");
  }
  __device__ __forceinline__ uint32_t slot1(uint32_t x) const { return ((2 * x) & mask) | base; }
  __device__ __forceinline__ uint32_t slot2(uint32_t x, uint32_t q) const {
    return ((q * (2 * kPairMul) + 2 * x) & mask) | base;
  }
  __device__ __forceinline__ uint32_t contains(uint32_t x) const {
    const uint32_t q = x >> k;
    const uint32_t e1 = load(slot1(x)), e2 = load(slot2(x, q) + kPairTableBytes);
    return e1 == q || e2 == q;
  }
};

// The warp's set of the d sorted ids at av (k = pair_log(d, n) > 0) in its
// region tab.  False: an id found no place.  All 32 lanes call.
__device__ __forceinline__ bool build_pair_set(const uint32_t *__restrict__ av, uint32_t d, int k, uint32_t *tab,
                                               int lane, PairSet &set) {
  set.base = (uint32_t)__cvta_generic_to_shared(tab);
  set.mask = ((1u << k) - 1) * 2;
  set.k = k;
  const uint32_t quads = (2u << k) / 16;  // per table
  const uint4 empty = make_uint4(kFull, kFull, kFull, kFull);
  for (uint32_t i = lane; i < quads; i += 32) {
    reinterpret_cast<uint4 *>(tab)[i] = empty;
    reinterpret_cast<uint4 *>(tab)[i + kPairTableBytes / 16] = empty;
  }
  __syncwarp();
  for (uint32_t i = lane; i < d; i += 32) PairSet::store(set.slot1(av[i]), av[i] >> k);
  __syncwarp();
  for (uint32_t i = lane; i < d; i += 32) {
    const uint32_t x = av[i], q = x >> k;
    if (PairSet::load(set.slot1(x)) != q) PairSet::store(set.slot2(x, q) + kPairTableBytes, q);
  }
  __syncwarp();
  bool ok = true;
  for (uint32_t b = 0; b < d; b += 32) {
    const uint32_t x = b + lane < d ? av[b + lane] : 0u;
    unsigned homeless = __ballot_sync(kFull, b + lane < d && !set.contains(x));
    while (homeless) {  // one after the other; every lane follows the same chain, one stores
      const int j = __ffs(homeless) - 1;
      homeless &= homeless - 1;
      uint32_t y = __shfl_sync(kFull, x, j);
      bool placed = false;
      for (uint32_t kick = 0; kick < kPairKicks && !placed; ++kick) {
        const uint32_t q = y >> k;
        const bool second = kick & 1u;
        const uint32_t at = second ? set.slot2(y, q) + kPairTableBytes : set.slot1(y);
        const uint32_t out = PairSet::load(at);
        __syncwarp();
        if (lane == 0) PairSet::store(at, q);
        __syncwarp();
        placed = out == kPairEmpty;
        // the evicted id: its entry and its slot's low bits
        const uint32_t low = ((at & set.mask) >> 1) - (second ? out * kPairMul : 0u);
        y = (out << k) | (low & (set.mask >> 1));
      }
      ok = ok && placed;
    }
  }
  __syncwarp();
  return ok;
}

}  // namespace gary
