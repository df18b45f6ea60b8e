// Stable LSD radix sort of (64-bit key, 32-bit value) pairs, a device-wide
// exclusive scan, and the gather of particles into key order.
//
// Replaces the stable recursive merge sort of fortran/morton/morton_octree.f90
// :501-560 (argsort).  An LSD radix sort whose every pass is stable produces
// exactly the stable sort's permutation: equal keys keep ascending original
// index, as the merge sort's "ties take the left element" rule (:537-538).
//
// Digit counts of every pass come from one histogram kernel over the keys;
// each pass (8-bit digit) is then ONE kernel with decoupled look-back: a block
// claims the next tile (4096 keys; 1024 for sorts of at most 65,536 keys, whose
// few large tiles would leave most SMs idle) from an atomic counter, ranks its keys inside
// the tile with warp __match_any_sync / popc ranking (element order = warp,
// iteration, lane, so ranks are stable), publishes its per-digit counts, adds
// up the counts of the tiles before it (each tile's word holds either its own
// count or, once known, the inclusive prefix of all tiles up to it), stages
// the tile in shared memory in digit order and writes it out so that runs of
// equal digits land on consecutive addresses.  A block only waits for tiles
// claimed before its own, by blocks that are already running; every wait is
// bounded and a wait that gives up raises an error flag instead of hanging.
#include <math.h>

#include "bh_internal.cuh"
#include "bh_lookback.cuh"

namespace bh {

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / kWarp;
constexpr int kItems = 16;       // keys per thread of a large sort's tile
constexpr int kSmallItems = kSortTileSmall / 256;  // and of a small sort's
constexpr int kTile = kSortThreads * kItems;  // 4096 keys per block (large sorts)
constexpr int kRadix = 256;

// Sum over the systems of n_s^2 up to which bodies are sorted by counting; above
// it the comparisons cost more than the radix passes, which in a batch grow with the
// bodies (more tiles, and passes over the system too).  Whole builds, us, counting /
// radix (Plummer; uniform spheres cross at the same sizes):
//   one system   10,000 (1e8) 151 / 159   12,000 (1.4e8) 156 / 160   14,142 (2e8) 194 / 162
//   2 of 7,071 (1e8) 153 / 168   2 of 8,485 (1.4e8) 180 / 173   2 of 11,180 (2.5e8) 261 / 182
//   4 of 5,000 (1e8) 171 / 175   4 of 6,000 (1.4e8) 197 / 182
//   8 of 4,242 (1.4e8) 208 / 211   8 of 5,000 (2e8) 219 / 216   8 of 6,614 (3.5e8) 235 / 224
//   16 of 4,677 (3.5e8) 227 / 253   16 of 5,590 (5e8) 254 / 256   16 of 6,614 (7e8) 294 / 260
//   32 of 3,952 (5e8) 255 / 268   32 of 4,677 (7e8) 307 / 277
//   128 of 2,338 (7e8) 348 / 388   512 of 1,169 (7e8) 451 / 499
constexpr double kRankPairsOne = 1.44e8;
inline double rank_pairs_batch(int64_t n) { return fmin(3e7 + 4500.0 * (double)n, 7e8); }

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 8;
constexpr int kScanChunk = kScanThreads * kScanItems;

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned r;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(r));
  return r;
}

__device__ __forceinline__ int warp_incl_scan(int v) {
  const int lane = threadIdx.x & (kWarp - 1);
#pragma unroll
  for (int o = 1; o < kWarp; o <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Exclusive scan of one value per thread across the block; `ws` needs
// blockDim/32 ints.  Ends with a barrier so `ws` may be reused.
__device__ int block_excl_scan(int v, int *ws, int *total) {
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  const int nwarps = blockDim.x / kWarp;
  int incl = warp_incl_scan(v);
  if (lane == kWarp - 1) ws[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int s = lane < nwarps ? ws[lane] : 0;
    s = warp_incl_scan(s);
    if (lane < nwarps) ws[lane] = s;
  }
  __syncthreads();
  int off = warp > 0 ? ws[warp - 1] : 0;
  if (total) *total = ws[nwarps - 1];
  __syncthreads();
  return off + incl - v;
}

// Digit counts from the number of keys of every key value v (keys are the
// values 0..n_values-1): pass p's count of digit d sums count[v] over the
// values whose digit p is d -- one read of the counts instead of all keys.
__global__ void __launch_bounds__(kSortThreads)
count_hist_kernel(const int32_t *__restrict__ count, int64_t n_values, int passes,
                  uint32_t *__restrict__ ghist) {
  constexpr int kMaxPasses = 4;  // 32-bit keys
  __shared__ uint32_t h[kMaxPasses][kRadix];
  for (int i = threadIdx.x; i < kMaxPasses * kRadix; i += kSortThreads) (&h[0][0])[i] = 0;
  __syncthreads();
  for (int64_t v = (int64_t)blockIdx.x * kSortThreads + threadIdx.x; v < n_values;
       v += (int64_t)gridDim.x * kSortThreads) {
    const uint32_t c = (uint32_t)count[v];
    if (c == 0) continue;
    for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(v >> (8 * p)) & 0xff], c);
  }
  __syncthreads();
  for (int p = 0; p < passes; ++p) {
    const uint32_t c = h[p][threadIdx.x];  // kSortThreads == kRadix
    if (c) atomicAdd(&ghist[p * kRadix + threadIdx.x], c);
  }
}

// Exclusive scan of each pass's 256 digit counts, in place, one block per pass
// (every block of a pass scanning them itself: 512 systems 22.6 instead of 22.5 ms).
__global__ void __launch_bounds__(kSortThreads) digit_scan_kernel(uint32_t *counts) {
  __shared__ int ws[kSortWarps];
  pdl_enter();
  uint32_t *c = counts + blockIdx.x * kRadix + threadIdx.x;  // kSortThreads == kRadix
  *c = (uint32_t)block_excl_scan((int)*c, ws, nullptr);
}

template <typename K, int ITEMS, bool SYS>
struct PassSmem {
  K sk[ITEMS * kSortThreads];
  int32_t sv[ITEMS * kSortThreads];
  unsigned char sd[SYS ? ITEMS * kSortThreads : 16];  // digits that the key does not hold
  int wh[kSortWarps][kRadix];
  int tile_start[kRadix];
  int gbase[kRadix];
  int ws[kSortWarps];
  int tile;
};

// kout may be null: the pass then writes only the values (a last pass whose
// keys nobody reads).
// 3 blocks per SM (80 registers, no spills; the compiler's own choice was 128
// and 2 blocks): the 181 M-term sort of Dehnen's method 1 ms faster.
// starts: first place of each of the pass's 256 digits.  SYS: the digit is the
// system's (of the body that the value names), not the key's.
template <typename K, int ITEMS, bool SYS>
__global__ void __launch_bounds__(kSortThreads, 3)
onesweep_kernel(const K *__restrict__ kin, const int32_t *__restrict__ vin,
                K *__restrict__ kout, int32_t *__restrict__ vout, int64_t n, int shift,
                const int32_t *__restrict__ sys_of, const uint32_t *__restrict__ starts,
                uint64_t *__restrict__ tiles, int32_t *__restrict__ tile_ctr, int *err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PassSmem<K, ITEMS, SYS> &S = *reinterpret_cast<PassSmem<K, ITEMS, SYS> *>(smem_raw);
  constexpr int kItems = ITEMS;
  constexpr int kTile = ITEMS * kSortThreads;
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  for (int i = threadIdx.x; i < kSortWarps * kRadix; i += kSortThreads) (&S.wh[0][0])[i] = 0;
  pdl_enter();
  if (threadIdx.x == 0) S.tile = atomicAdd(tile_ctr, 1);
  __syncthreads();
  const int t = S.tile;
  const int64_t tile_base = (int64_t)t * kTile;
  if (tile_base >= n) return;  // uniform across the block; later tiles return too
  const int tile_n = (int)bh_min64(kTile, n - tile_base);

  K k[kItems];
  int32_t v[kItems];
  int dig[kItems], rank[kItems];
  const int wbase = warp * kWarp * kItems;
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    int li = wbase + i * kWarp + lane;
    bool valid = li < tile_n;
    k[i] = valid ? kin[tile_base + li] : (K)0;
    v[i] = valid ? vin[tile_base + li] : 0;
    dig[i] = valid ? (int)(((SYS ? (K)sys_of[v[i]] : k[i]) >> shift) & 0xff) : kRadix;
  }
  const unsigned lt = lanemask_lt();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int d = dig[i];
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const int rin = __popc(peers & lt);
    const int pre = d < kRadix ? S.wh[warp][d] : 0;
    __syncwarp();
    if (d < kRadix && rin == 0) S.wh[warp][d] = pre + __popc(peers);
    __syncwarp();
    rank[i] = pre + rin;
  }
  __syncthreads();
  // per digit (thread d): exclusive offsets of the warps and the tile's count
  const int d = threadIdx.x;  // kSortThreads == kRadix
  int cnt = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) {
    const int c = S.wh[w][d];
    S.wh[w][d] = cnt;
    cnt += c;
  }
  // publish, then look back over the earlier tiles for this digit
  const int64_t excl = thread_lookback(tiles + d, t, kRadix, cnt, err);
  S.gbase[d] = (int)(starts[d] + excl);
  int start = block_excl_scan(cnt, S.ws, nullptr);
  S.tile_start[d] = start;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int dd = dig[i];
    if (dd < kRadix) {
      int pos = S.tile_start[dd] + S.wh[warp][dd] + rank[i];
      S.sk[pos] = k[i];
      S.sv[pos] = v[i];
      if (SYS) S.sd[pos] = (unsigned char)dd;
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < tile_n; j += kSortThreads) {
    const K key = S.sk[j];
    const int dd = SYS ? (int)S.sd[j] : (int)((key >> shift) & 0xff);
    const int64_t o = (int64_t)S.gbase[dd] + (j - S.tile_start[dd]);
    if (kout) kout[o] = key;
    vout[o] = S.sv[j];
  }
}

// ---- exclusive scan ----

// Single-pass exclusive scan (chained scan with decoupled look-back): block b
// claims tile t (kScanChunk values) from a ticket, sums it, publishes the sum,
// adds up the earlier tiles' words (an inclusive word ends the walk), then
// writes its outputs.  A block only waits for tiles claimed before its own by
// blocks that are running and publish before they wait; every wait is
// bounded and one that gives up raises kErrTimeout in *err.
// tmp (int32 entries): [0] ticket, [1] unused, then one 64-bit word per tile.
__global__ void __launch_bounds__(kScanThreads)
scan_onepass_kernel(const int32_t *__restrict__ in, int32_t *__restrict__ out, int64_t n, int32_t *tmp,
                    int *err) {
  __shared__ int ws[kScanThreads / kWarp];
  __shared__ int s_tile;
  __shared__ int64_t s_excl;
  if (threadIdx.x == 0) s_tile = atomicAdd(tmp, 1);
  __syncthreads();
  const int t = s_tile;
  uint64_t *words = reinterpret_cast<uint64_t *>(tmp + 2);
  const int64_t base = (int64_t)t * kScanChunk + (int64_t)threadIdx.x * kScanItems;
  int vals[kScanItems];
  int sum = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    vals[i] = (base + i < n) ? in[base + i] : 0;
    sum += vals[i];
  }
  int tile_total;
  int off = block_excl_scan(sum, ws, &tile_total);
  if (threadIdx.x < kWarp) {
    const int64_t excl = warp_lookback(words, t, tile_total, err);
    if (threadIdx.x == 0) s_excl = excl;
  }
  __syncthreads();
  int64_t o = s_excl + off;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (base + i < n) out[base + i] = (int32_t)o;
    o += vals[i];
  }
}

// bodies into key order, from the packed copy the keys kernel wrote
__global__ void __launch_bounds__(256)
gather_kernel(const double4 *__restrict__ packed, const int32_t *__restrict__ perm, int64_t n,
              double4 *__restrict__ spos) {
  pdl_enter();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    spos[i] = packed[perm[i]];
}

// ---- sort by counting (small systems) ----

// Body t's place in its system's key order is the number of that system's keys
// below its own, equal keys of earlier bodies included (the stable order): with
// few bodies counting all of them beats eight dependent passes.  A block takes
// 64 bodies, two per lane, and its 8 warps a slice of the system's keys each (two
// keys per shared-memory read, three instructions a comparison); the bodies then
// go straight to their places, so there is no gather either.
// Bound: the integer pipe, n_s^2 comparisons (1,024 bodies 6 us against 45 for
// eight radix passes and their counts; kRankPairsOne has the crossing).
constexpr int kRankWarps = 8, kRankBodies = 2 * kWarp;

// neg -= (a < b), on the borrow of a - b
__device__ __forceinline__ void count_below(unsigned &neg, uint64_t a, uint64_t b) {
  asm("{\n\t.reg .u32 t, al, ah, bl, bh;\n\t"
      "mov.b64 {al, ah}, %1;\n\tmov.b64 {bl, bh}, %2;\n\t"
      "sub.cc.u32 t, al, bl;\n\tsubc.cc.u32 t, ah, bh;\n\tsubc.u32 %0, %0, 0;\n\t}"
      : "+r"(neg) : "l"(a), "l"(b));
}

__global__ void __launch_bounds__(kRankWarps *kWarp)
rank_sort_kernel(const uint64_t *__restrict__ keys, const double *__restrict__ m,
                 const double *__restrict__ x, const double *__restrict__ y,
                 const double *__restrict__ z, int64_t n, const int32_t *__restrict__ sys_of,
                 const SysScalars *__restrict__ sys, uint64_t *__restrict__ kout,
                 int32_t *__restrict__ vout, double4 *__restrict__ spos) {
  __shared__ __align__(16) uint64_t tile[kRankWarps][2 * kWarp];
  __shared__ unsigned part[kRankWarps][kRankBodies];
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  const int64_t base = (int64_t)blockIdx.x * kRankBodies;
  pdl_enter();
  int64_t t[2];
  uint64_t key[2];
  int mine[2];
  unsigned neg[2] = {0, 0};
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    t[q] = base + q * kWarp + lane;
    key[q] = t[q] < n ? keys[t[q]] : 0;
    mine[q] = t[q] < n ? sys_of[t[q]] : -1;
  }
  const int s_last = sys_of[bh_min64(base + kRankBodies, n) - 1];
  for (int s = sys_of[base]; s <= s_last; ++s) {
    const int64_t off = sys[s].off, ns = sys[s].n;
    const int64_t b = off + ns * (warp + 1) / kRankWarps;
    for (int64_t a = off + ns * warp / kRankWarps; a < b; a += 2 * kWarp) {
      // keys beyond the slice never count
      tile[warp][lane] = a + lane < b ? keys[a + lane] : ~0ull;
      tile[warp][kWarp + lane] = a + kWarp + lane < b ? keys[a + kWarp + lane] : ~0ull;
      __syncwarp();
      const ulonglong2 *k2 = reinterpret_cast<const ulonglong2 *>(tile[warp]);
      if (a + 2 * kWarp <= base || a >= base + kRankBodies) {
        // all earlier bodies (equal keys count: below key + 1) or all later ones
        const uint64_t up = a < base ? 1 : 0;
        const uint64_t b0 = mine[0] == s ? key[0] + up : 0, b1 = mine[1] == s ? key[1] + up : 0;
#pragma unroll 8
        for (int j = 0; j < kWarp; ++j) {
          const ulonglong2 k = k2[j];
          count_below(neg[0], k.x, b0); count_below(neg[0], k.y, b0);
          count_below(neg[1], k.x, b1); count_below(neg[1], k.y, b1);
        }
      } else {
        for (int j = 0; j < kWarp; ++j) {
          const ulonglong2 k = k2[j];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            if (mine[q] != s) continue;
            count_below(neg[q], k.x, key[q] + (a + 2 * j < t[q] ? 1 : 0));
            count_below(neg[q], k.y, key[q] + (a + 2 * j + 1 < t[q] ? 1 : 0));
          }
        }
      }
      __syncwarp();
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) part[warp][q * kWarp + lane] = neg[q];
  __syncthreads();
  if (threadIdx.x < kRankBodies && base + threadIdx.x < n) {
    unsigned c = 0;
#pragma unroll
    for (int w = 0; w < kRankWarps; ++w) c -= part[w][threadIdx.x];
    const int64_t p = base + threadIdx.x, o = sys[sys_of[p]].off + c;
    kout[o] = keys[p];
    vout[o] = (int32_t)p;
    spos[o] = make_double4(x[p], y[p], z[p], m[p]);
  }
}

template <typename K, int ITEMS, bool SYS>
void launch_pass(int64_t ntiles, const K *ki, const int32_t *vi, K *ko, int32_t *vo, int64_t n,
                 int shift, const int32_t *sys_of, const uint32_t *counts, uint64_t *tiles,
                 int32_t *ctr, int *err, cudaStream_t s) {
  constexpr int smem = (int)sizeof(PassSmem<K, ITEMS, SYS>);
  static bool done[64] = {};  // the limit is set once per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!done[dev]) {
    cudaFuncSetAttribute(onesweep_kernel<K, ITEMS, SYS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         smem);
    done[dev] = true;
  }
  launch_pdl(onesweep_kernel<K, ITEMS, SYS>, ntiles, kSortThreads, smem, s, ki, vi, ko, vo, n, shift,
             sys_of, counts, tiles, ctr, err);
}

// scratch layout (int32 entries): digit counts [passes][256], tile counters
// [12], then the tile words (uint64) [passes][ntiles][256]
struct SortScratch {
  uint32_t *counts;
  int32_t *ctr;
  uint64_t *tiles;
  int64_t ntiles, entries;
};
SortScratch sort_scratch(int64_t n, int passes, int32_t *hist) {
  SortScratch c;
  c.counts = reinterpret_cast<uint32_t *>(hist);
  c.ctr = hist + passes * kRadix;
  c.tiles = reinterpret_cast<uint64_t *>(hist + passes * kRadix + 12);
  c.ntiles = (n + sort_tile(n) - 1) / sort_tile(n);
  c.entries = passes * kRadix + 12 + 2 * (int64_t)passes * c.ntiles * kRadix;
  return c;
}

template <typename K, bool SYS>
void one_pass(const SortScratch &c, int pass, int64_t n, int shift, const int32_t *sys_of, const K *ki,
              const int32_t *vi, K *ko, int32_t *vo, int *err, cudaStream_t s) {
  // small sorts take small tiles: more blocks in flight for the same keys
  if (sort_tile(n) == kSortTileSmall)
    launch_pass<K, kSmallItems, SYS>(c.ntiles, ki, vi, ko, vo, n, shift, sys_of,
                                     c.counts + pass * kRadix, c.tiles + pass * c.ntiles * kRadix,
                                     c.ctr + pass, err, s);
  else
    launch_pass<K, kItems, SYS>(c.ntiles, ki, vi, ko, vo, n, shift, sys_of, c.counts + pass * kRadix,
                                c.tiles + pass * c.ntiles * kRadix, c.ctr + pass, err, s);
}

}  // namespace

static_assert(kScanChunk == 8192 && kTile == kSortTileLarge && kRadix == 256 &&
                  kSortThreads * kSmallItems == kSortTileSmall && kMaxSortPasses <= 12,
              "scan_tmp_entries / radix_hist_entries in bh_internal.cuh assume these sizes");

void exclusive_scan(const int32_t *in, int32_t *out, int64_t n, int32_t *tmp, int *err,
                    cudaStream_t s) {
  int nb = (int)((n + kScanChunk - 1) / kScanChunk);
  if (nb < 1) nb = 1;
  cudaMemsetAsync(tmp, 0, (2 + 2 * (int64_t)nb) * sizeof(int32_t), s);
  scan_onepass_kernel<<<nb, kScanThreads, 0, s>>>(in, out, n, tmp, err);
}

int radix_sort_values32(uint32_t *k0, int32_t *v0, uint32_t *k1, int32_t *v1, int64_t n, int bits,
                        int32_t *hist, int *err, cudaStream_t s, const int32_t *key_counts,
                        int64_t n_key_values) {
  int passes = (bits + 7) / 8;
  passes = passes < 1 ? 1 : (passes > 4 ? 4 : passes);
  const SortScratch c = sort_scratch(n, passes, hist);
  cudaMemsetAsync(hist, 0, c.entries * sizeof(int32_t), s);
  count_hist_kernel<<<grid_for(n_key_values, kSortThreads, 148 * 8), kSortThreads, 0, s>>>(
      key_counts, n_key_values, passes, c.counts);
  launch_pdl(digit_scan_kernel, passes, kSortThreads, 0, s, c.counts);
  uint32_t *ki = k0, *ko = k1;
  int32_t *vi = v0, *vo = v1;
  for (int p = 0; p < passes; ++p) {
    one_pass<uint32_t, false>(c, p, n, 8 * p, nullptr, ki, vi, p == passes - 1 ? nullptr : ko, vo, err, s);
    uint32_t *tk = ki; ki = ko; ko = tk;
    int32_t *tv = vi; vi = vo; vo = tv;
  }
  return ki == k0 ? 0 : 1;
}

SortPlan sort_plan(int64_t n, int L, const Buffers &b) {
  SortPlan p;
  p.by_rank = b.sort_pairs <= (b.nsys > 1 ? rank_pairs_batch(n) : kRankPairsOne);
  const int bits = 3 * (L == 0 ? kMaxDepth : L);
  p.kpass = (bits + 7) / 8;
  p.spass = 0;
  while (((int64_t)1 << (8 * p.spass)) < b.nsys) ++p.spass;
  p.scratch = sort_scratch(n, p.kpass + p.spass, nullptr).entries;
  return p;
}

void launch_sort(const double *m, const double *x, const double *y, const double *z, int64_t n,
                 int L, Buffers &b, cudaStream_t s) {
  const SortPlan plan = sort_plan(n, L, b);
  if (plan.by_rank) {
    launch_pdl(rank_sort_kernel, (n + kRankBodies - 1) / kRankBodies, kRankWarps * kWarp, 0, s, b.k1, m,
               x, y, z, n, b.sys_of, b.ss, b.k0, b.v0, b.spos);
    return;
  }
  const int passes = plan.kpass + plan.spass;
  const SortScratch c = sort_scratch(n, passes, b.hist);
  const bool odd = passes & 1;
  launch_pdl(digit_scan_kernel, passes, kSortThreads, 0, s, c.counts);
  uint64_t *ki = odd ? b.k1 : b.k0, *ko = odd ? b.k0 : b.k1;
  int32_t *vi = odd ? b.v1 : b.v0, *vo = odd ? b.v0 : b.v1;
  for (int p = 0; p < passes; ++p) {
    // the key's digits, then the system's: every system's bodies end up
    // together, each range in key order (LSD order)
    if (p < plan.kpass)
      one_pass<uint64_t, false>(c, p, n, 8 * p, nullptr, ki, vi, ko, vo, &b.sc->err, s);
    else
      one_pass<uint64_t, true>(c, p, n, 8 * (p - plan.kpass), b.sys_of, ki, vi, ko, vo, &b.sc->err, s);
    uint64_t *tk = ki; ki = ko; ko = tk;
    int32_t *tv = vi; vi = vo; vo = tv;
  }
  launch_pdl(gather_kernel, grid_for(n, 256, 148 * 16), 256, 0, s,
             reinterpret_cast<const double4 *>(b.cn_oct), b.v0, n, b.spos);
}

}  // namespace bh
