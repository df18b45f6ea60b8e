// Decoupled look-back of a chained scan: every tile of an ordered sequence
// publishes a word per counter -- its own count first, the inclusive prefix of
// all tiles up to it once known -- and adds up the words of the tiles before it.
// A tile only waits for tiles claimed earlier (from a ticket), by blocks that
// are running and publish before they wait; every wait is bounded, and one that
// gives up raises kErrTimeout.
#pragma once

#include "bh_internal.cuh"

namespace bh {

// tile words: top 2 bits the state, low 62 bits the count
constexpr uint64_t kTileAggregate = 1ull << 62;  // the tile's own count
constexpr uint64_t kTileInclusive = 2ull << 62;  // sum of the counts of tiles 0..t
constexpr uint64_t kTileValue = (1ull << 62) - 1;
constexpr int64_t kLookbackSpins = 1 << 22;      // polls of one look-back; about a second at most

__device__ __forceinline__ uint64_t ld_relaxed(const uint64_t *p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(uint64_t *p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// One counter per thread: publishes `count` for tile t (its word at
// words[t * stride]) and returns the sum of the counts of the tiles before it.
// (Reading 4 or 8 earlier words at once made no sort faster, and a pass of 18 M
// terms 180 instead of 171 us.)
__device__ __forceinline__ int64_t thread_lookback(uint64_t *words, int t, int stride, int64_t count,
                                                   int *err) {
  uint64_t *word = words + (int64_t)t * stride;
  if (t == 0) {
    st_relaxed(word, kTileInclusive | (uint64_t)count);
    return 0;
  }
  st_relaxed(word, kTileAggregate | (uint64_t)count);
  int64_t excl = 0, spins = 0;
  for (int j = t - 1; j >= 0;) {
    const uint64_t w = ld_relaxed(words + (int64_t)j * stride);
    if ((w & ~kTileValue) == 0) {
      if (++spins > kLookbackSpins) { atomicOr(err, kErrTimeout); break; }
      continue;
    }
    excl += (int64_t)(w & kTileValue);
    if ((w & ~kTileValue) == kTileInclusive) break;
    --j;
  }
  st_relaxed(word, kTileInclusive | (uint64_t)(excl + count));
  return excl;
}

// One counter for the whole warp: reads the words of the 32 tiles before the
// window's end at once and adds them up to the nearest inclusive word; a
// window with a word not yet published is read again.
__device__ __forceinline__ int64_t warp_lookback(uint64_t *words, int t, int64_t count, int *err) {
  const int lane = threadIdx.x & (kWarp - 1);
  uint64_t *word = words + t;
  if (t == 0) {
    if (lane == 0) st_relaxed(word, kTileInclusive | (uint64_t)count);
    return 0;
  }
  if (lane == 0) st_relaxed(word, kTileAggregate | (uint64_t)count);
  int64_t excl = 0;
  int j = t - 1;  // the window is tiles j - 31 .. j, lane k reading tile j - k
  int64_t spins = 0;
  for (;;) {
    const int idx = j - lane;
    const uint64_t w = idx >= 0 ? ld_relaxed(words + idx) : kTileInclusive;
    const unsigned incl = __ballot_sync(0xffffffffu, (w & ~kTileValue) == kTileInclusive);
    const unsigned unset = __ballot_sync(0xffffffffu, (w & ~kTileValue) == 0);
    const int stop = incl ? __ffs(incl) - 1 : kWarp - 1;  // the last lane that counts
    const unsigned counted = stop == kWarp - 1 ? 0xffffffffu : ((2u << stop) - 1u);
    if (unset & counted) {
      if (++spins > kLookbackSpins) {
        if (lane == 0) atomicOr(err, kErrTimeout);
        break;
      }
      continue;
    }
    int64_t v = lane <= stop ? (int64_t)(w & kTileValue) : 0;
#pragma unroll
    for (int o = kWarp / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    excl += v;
    if (incl) break;
    j -= kWarp;
  }
  if (lane == 0) st_relaxed(word, kTileInclusive | (uint64_t)(excl + count));
  return excl;
}

}  // namespace bh
