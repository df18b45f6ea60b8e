// Octree from the sorted Morton keys, and the target groups of the walk.
//
// The reference (fortran/morton/morton_octree.f90:420-493) materialises one
// node per distinct key prefix at every level 0..L, so a run of particles that
// does not split between two levels appears once per level (a chain), and
// every lone particle is followed down to level L.  The walk of :627-766
// visits such a chain top-down with the same centre of mass and mass at every
// link and opens the next link while the cell-size test fails; since the cell
// size shrinks with depth, the chain is accepted exactly when its deepest
// link passes.  The compact octree built here keeps one node per distinct
// particle range with >= 2 particles (at the deepest level of its chain), and
// lists lone particles as particle children.  It therefore has the
// reference's topology without the chains, and its node order is the
// reference's node order (level, then first particle) restricted to those
// nodes.
//
// Construction: a binary radix tree over the sorted keys (Karras 2012, with
// the index as tie-break for equal keys), whose nodes get the octal level
// floor(common prefix bits / 3); a binary node whose level is deeper than its
// parent's starts a new octree node.  Nodes of one level hold disjoint ranges
// and a binary node's index lies inside its range, so the order (level, first
// particle) is the order (level, binary index): a count per level and a scan
// place every node, without a sort, and each one enumerates its octree
// children by descending at most three binary levels.
//
// In a batch every system is its own segment of the sorted arrays: the
// binary tree of a segment [s0, s1) uses internal nodes s0 .. s1 - 2 (the slot
// s1 - 1 stays unused) and treats bodies outside the segment as absent, so
// every system gets its own root; all later steps run over all systems at once.
#include "bh_internal.cuh"
#include "bh_lookback.cuh"

namespace bh {

namespace {

__device__ __forceinline__ int delta(const uint64_t *__restrict__ k, int64_t s0, int64_t s1,
                                     int64_t i, uint64_t ki, int64_t j) {
  if (j < s0 || j >= s1) return -1;
  uint64_t kj = k[j];
  if (ki != kj) return __clzll((long long)(ki ^ kj));
  return 64 + __clz((int)(i ^ j));
}

// octal level of a common prefix of d bits (at most L)
__device__ __forceinline__ int octal_level(int d, int lead, int L) {
  const int v = (d - lead) / 3;
  return v > L ? L : v;
}

constexpr int kRankThreads = 256;
constexpr int kNone = kWarp - 1;  // level slot of what is not an octree node (levels reach 21)
static_assert(kMaxDepth < kNone, "a lane per level");
static_assert(kRankThreads == kTreeTile, "build_tmp_entries in bh_internal.cuh assumes this tile");

// The binary radix tree, and every octree node's rank among the nodes of its
// level: a chained scan over tiles of kRankTile binary nodes with a counter per
// level (a lane each).  A node's parent has the longer of the prefixes shared
// across the range's two ends, so whether it starts an octree node is known
// without the parent array.  rank is -1 for binary nodes inside an octree node.
// One launch; with the records below it replaces a marking pass, a scan, a
// 4-pass radix sort with its counts, and three copies (2^20 bodies: about 190 us
// in 16 launches -> 123 in 2; 1,024 bodies: 45 -> 17 us).
template <int kRankItems>
__global__ void __launch_bounds__(kRankThreads)
karras_kernel(const uint64_t *__restrict__ k, int64_t n, const int32_t *__restrict__ sys_of,
              const SysScalars *__restrict__ sys, Scalars *__restrict__ sc,
              int32_t *__restrict__ left, int32_t *__restrict__ right,
              int32_t *__restrict__ first, int32_t *__restrict__ last,
              int32_t *__restrict__ level, int32_t *__restrict__ rank, int32_t *ticket,
              uint64_t *words, int32_t *__restrict__ level_count) {
  constexpr int kRankTile = kRankThreads * kRankItems, kRankRows = kRankTile / kWarp;
  __shared__ int cnt[kRankRows][kWarp];
  __shared__ int before[kWarp];
  __shared__ int s_tile;
  pdl_enter();
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1);
  for (int i = threadIdx.x; i < kRankRows * kWarp; i += kRankThreads) (&cnt[0][0])[i] = 0;
  __syncthreads();
  const int tile = s_tile;
  const int64_t base = (int64_t)tile * kRankTile;
  if (base >= n) return;  // uniform across the block
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  const int L = sc->L;
  const int lead = 64 - 3 * L;  // leading zero bits of every key
  int slot[kRankItems], in_warp[kRankItems];
#pragma unroll
  for (int q = 0; q < kRankItems; ++q) {
    const int64_t i = base + q * kRankThreads + threadIdx.x;
    slot[q] = kNone;
    if (i < n) {
      const SysScalars &ss = sys[sys_of[i]];
      const int64_t s0 = ss.off, s1 = ss.off + ss.n;
      if (i != s1 - 1) {  // not the segment's unused slot
        const uint64_t ki = k[i];
        const int d = (delta(k, s0, s1, i, ki, i + 1) - delta(k, s0, s1, i, ki, i - 1)) > 0 ? 1 : -1;
        const int dmin = delta(k, s0, s1, i, ki, i - d);
        int64_t lmax = 2;
        while (delta(k, s0, s1, i, ki, i + lmax * d) > dmin) lmax <<= 1;
        int64_t l = 0;
        for (int64_t t = lmax >> 1; t >= 1; t >>= 1)
          if (delta(k, s0, s1, i, ki, i + (l + t) * d) > dmin) l += t;
        const int64_t j = i + l * d;
        const int dnode = delta(k, s0, s1, i, ki, j);
        int64_t s = 0, t = l;
        do {
          t = (t + 1) >> 1;
          if (delta(k, s0, s1, i, ki, i + (s + t) * d) > dnode) s += t;
        } while (t > 1);
        const int64_t gamma = i + s * d + (d < 0 ? -1 : 0);
        const int64_t f = min(i, j), la = max(i, j);
        left[i] = (f == gamma) ? ~(int32_t)gamma : (int32_t)gamma;
        right[i] = (la == gamma + 1) ? ~(int32_t)(gamma + 1) : (int32_t)(gamma + 1);
        first[i] = (int32_t)f;
        last[i] = (int32_t)la;
        const int v = octal_level(dnode, lead, L);
        level[i] = v;
        // one end of the range is i itself: its outer prefix is dmin
        const int dother = delta(k, s0, s1, j, k[j], j + d);
        const int dparent = max(dmin, dother);
        if (dparent < 0 || v > octal_level(dparent, lead, L)) slot[q] = v;
      }
    }
    const unsigned peers = __match_any_sync(0xffffffffu, slot[q]);
    in_warp[q] = __popc(peers & ((1u << lane) - 1u));
    if (in_warp[q] == 0) cnt[q * (kRankThreads / kWarp) + warp][slot[q]] = __popc(peers);
  }
  __syncthreads();
  if (warp == 0) {  // lane = level: exclusive counts of the rows, then the earlier tiles
    int total = 0;
#pragma unroll
    for (int r = 0; r < kRankRows; ++r) {
      const int c = cnt[r][lane];
      cnt[r][lane] = total;
      total += c;
    }
    const int64_t excl = thread_lookback(words + lane, tile, kWarp, total, &sc->err);
    before[lane] = (int)excl;
    if (base + kRankTile >= n) level_count[lane] = (int)(excl + total);
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kRankItems; ++q) {
    const int64_t i = base + q * kRankThreads + threadIdx.x;
    if (i < n)
      rank[i] = slot[q] == kNone
                    ? -1
                    : before[slot[q]] + cnt[q * (kRankThreads / kWarp) + warp][slot[q]] + in_warp[q];
  }
}

// Octree records, one thread per binary node: node id = nodes of the shallower
// levels + rank.  Also clears the group flags, and writes the roots, the level
// starts and the node count.
// (Marking the groups' first bodies here as well, from the children's ranges,
// took it from 167 to 450 us at 5,000,011 bodies, to save a launch of 15.)
__global__ void __launch_bounds__(256)
records_kernel(int64_t n, const int32_t *__restrict__ sys_of, SysScalars *__restrict__ sys,
               Scalars *__restrict__ sc, const int32_t *__restrict__ level_count,
               const int32_t *__restrict__ left, const int32_t *__restrict__ right,
               const int32_t *__restrict__ first, const int32_t *__restrict__ last,
               const int32_t *__restrict__ level, const int32_t *__restrict__ rank,
               int32_t *__restrict__ cbin, int4 *__restrict__ meta, int32_t *__restrict__ child,
               int32_t *__restrict__ cparent, int32_t *__restrict__ level_begin,
               int32_t *__restrict__ gflag) {
  __shared__ int begin[kWarp];
  pdl_enter();
  if (threadIdx.x < kWarp) {
    const int l = threadIdx.x;
    const int c = l <= kMaxDepth ? level_count[l] : 0;
    int v = c;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, v, o);
      if (l >= o) v += t;
    }
    begin[l] = v - c;  // entries past kMaxDepth: the node count
    if (blockIdx.x == 0) {
      if (l <= kNumLevels) level_begin[l] = v - c;
      if (l == kNone) sc->n_compact = v;
    }
  }
  __syncthreads();
  const int L = sc->L;
  int err = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    gflag[i] = 0;
    const int32_t r = rank[i];
    SysScalars &ss = sys[sys_of[i]];
    if (i == ss.off && ss.n < 2) ss.root = -1;
    if (r < 0) continue;
    const int f = first[i], la = last[i], v = level[i];
    const int j = begin[v] + r;
    int nc = 0;
    int32_t ch[8];
    if (v < L) {
      int32_t st[8];
      int top = 0;
      st[top++] = right[i];
      st[top++] = left[i];
      int guard = 0;
      while (top > 0) {
        if (++guard > 64) { err |= kErrChildren; break; }
        const int32_t c = st[--top];
        if (c < 0) {
          if (nc < 8) ch[nc] = c;  // particle ~c, stored as ~c (< 0)
          ++nc;
          continue;
        }
        const int32_t cr = rank[c];
        if (cr >= 0) {
          if (nc < 8) ch[nc] = begin[level[c]] + cr;
          ++nc;
        } else {
          if (top + 2 > 8) { err |= kErrChildren; break; }
          st[top++] = right[c];
          st[top++] = left[c];
        }
      }
      if (nc > 8) { err |= kErrChildren; nc = 8; }
    }
    cbin[j] = (int32_t)i;
    meta[j] = make_int4(f, la - f + 1, v, nc);
    for (int c = 0; c < 8; ++c) child[8 * (int64_t)j + c] = c < nc ? ch[c] : 0x7fffffff;
    for (int c = 0; c < nc; ++c)
      if (ch[c] >= 0) cparent[ch[c]] = j;
    if (i == ss.off) {  // the segment's binary root: the system's root node
      ss.root = j;
      cparent[j] = -1;
    }
  }
  if (err) atomicOr(&sc->err, err);
}

// ---- target groups ----
// Units are the subtrees of <= U bodies whose parent holds more than U bodies
// (lone particles included).  Consecutive units under the same parent are
// concatenated in key order and cut into groups of G bodies (the last one of a
// run shorter); a child with more than U bodies ends the run and is cut by its
// own children.  A node of identical keys (no children) with more than U
// bodies, or a root of <= U bodies, is cut into groups of G directly.
// gflag marks the first body of each group.  With U = G this packs small
// siblings; a larger U fills more groups completely at the price of groups
// that span neighbouring subtrees.
__global__ void __launch_bounds__(256)
group_flags_kernel(const int4 *__restrict__ meta, const int32_t *__restrict__ child,
                   const int32_t *__restrict__ cparent, const Scalars *__restrict__ sc, int G,
                   int U, const SysScalars *__restrict__ sys, int nsys,
                   int32_t *__restrict__ gflag) {
  pdl_enter();
  // every system starts a group (this also covers lone bodies, which have no node)
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nsys; q += gridDim.x * blockDim.x)
    if (sys[q].n > 0) gflag[sys[q].off] = 1;
  const int M = sc->n_compact;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < M; j += gridDim.x * blockDim.x) {
    const int4 mt = meta[j];  // first, count, level, nchild
    if (mt.y <= U) {
      if (cparent[j] < 0)  // a system's root
        for (int s = 0; s < mt.y; s += G) gflag[mt.x + s] = 1;
      continue;
    }
    if (mt.w == 0) {
      for (int s = 0; s < mt.y; s += G) gflag[mt.x + s] = 1;
      continue;
    }
    int run_first = -1, run_len = 0;
    for (int c = 0; c <= mt.w; ++c) {
      int cfirst = 0, ccount = U + 1;  // c == nchild: closes the last run
      if (c < mt.w) {
        const int32_t ch = child[8 * j + c];
        if (ch < 0) { cfirst = ~ch; ccount = 1; }
        else { const int4 cm = meta[ch]; cfirst = cm.x; ccount = cm.y; }
      }
      if (ccount > U) {
        for (int s = 0; s < run_len; s += G) gflag[run_first + s] = 1;
        run_first = -1;
        run_len = 0;
        continue;
      }
      if (run_first < 0) run_first = cfirst;
      run_len += ccount;
    }
  }
}

constexpr int kGroupThreads = 256, kGroupItems = 8, kGroupTile = kGroupThreads * kGroupItems;
static_assert(kGroupTile == kGroupScanTile, "build_tmp_entries in bh_internal.cuh assumes this tile");

// The groups' first bodies from the flags, in one launch: a chained scan whose
// blocks write g_first themselves (instead of a scan array and a pass over it).
__global__ void __launch_bounds__(kGroupThreads)
group_first_kernel(int64_t n, const int32_t *__restrict__ gflag, Scalars *__restrict__ sc,
                   int32_t *__restrict__ cursor, int32_t *ticket, uint64_t *words,
                   int32_t *__restrict__ g_first) {
  __shared__ int ws[kGroupThreads / kWarp];
  __shared__ int s_tile, s_before;
  pdl_enter();
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1);
  if (blockIdx.x == 0 && threadIdx.x == 0) *cursor = 0;  // for a walk queued with the build
  __syncthreads();
  const int tile = s_tile;
  const int64_t base = (int64_t)tile * kGroupTile;
  if (base >= n) return;  // uniform across the block
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  // a warp takes 8 rows of 32 consecutive bodies
  const int64_t row0 = base + warp * (kGroupItems * kWarp) + lane;
  unsigned row[kGroupItems];
  int mine = 0;
#pragma unroll
  for (int q = 0; q < kGroupItems; ++q) {
    const int64_t i = row0 + q * kWarp;
    row[q] = __ballot_sync(0xffffffffu, i < n && gflag[i] != 0);
    mine += __popc(row[q]);
  }
  if (lane == 0) ws[warp] = mine;
  __syncthreads();
  int in_block = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kGroupThreads / kWarp; ++w) {
    if (w < warp) in_block += ws[w];
    total += ws[w];
  }
  if (warp == 0) {
    const int64_t excl = warp_lookback(words, tile, total, &sc->err);
    if (lane == 0) {
      s_before = (int)excl;
      if (base + kGroupTile >= n) {
        sc->n_groups = (int)(excl + total);
        g_first[excl + total] = (int32_t)n;
      }
    }
  }
  __syncthreads();
  int o = s_before + in_block;
#pragma unroll
  for (int q = 0; q < kGroupItems; ++q) {
    if ((row[q] >> lane) & 1u) g_first[o + __popc(row[q] & ((1u << lane) - 1u))] = (int32_t)(row0 + q * kWarp);
    o += __popc(row[q]);
  }
}

// Scratch of the tree and group passes in b.scan_tmp (int32 entries): [0], [1]
// the two tickets, then the nodes of every level, the words of the two
// look-backs, and the upward pass's list counters; cleared by the build's first
// kernel.
struct BuildTmp {
  int32_t *tickets, *level_count;
  uint64_t *tree_words, *group_words;
};
BuildTmp build_tmp(int64_t n, Buffers &b) {
  BuildTmp t;
  t.tickets = b.scan_tmp;
  t.level_count = b.scan_tmp + 2;
  t.tree_words = reinterpret_cast<uint64_t *>(b.scan_tmp + 2 + kWarp);
  t.group_words = t.tree_words + kWarp * ((n + kTreeTile - 1) / kTreeTile);
  return t;
}

}  // namespace

int32_t *upward_counters(int64_t n, Buffers &b) {
  return reinterpret_cast<int32_t *>(build_tmp(n, b).group_words + (n + kGroupScanTile - 1) / kGroupScanTile);
}

void launch_build_tree(int64_t n, Buffers &b, cudaStream_t s) {
  const BuildTmp t = build_tmp(n, b);
  // one binary node a thread while the tiles all run at once, four above (fewer
  // tiles to look back over: 2^20 bodies 85 against 107 us; 1,024 bodies 20
  // against 9 us).  The large one is launched ordinarily: started while the
  // gather drains, it and the records after it took 65 us longer at 5,000,011.
  if (n <= (1 << 18))
    launch_pdl(karras_kernel<1>, (n + kRankThreads - 1) / kRankThreads, kRankThreads, 0, s, b.k0, n,
               b.sys_of, b.ss, b.sc, b.bn_left, b.bn_right, b.bn_first, b.bn_last, b.bn_level,
               b.bn_rank, t.tickets, t.tree_words, t.level_count);
  else
    karras_kernel<4><<<(unsigned)((n + 4 * kRankThreads - 1) / (4 * kRankThreads)), kRankThreads, 0, s>>>(
        b.k0, n, b.sys_of, b.ss, b.sc, b.bn_left, b.bn_right, b.bn_first, b.bn_last, b.bn_level,
        b.bn_rank, t.tickets, t.tree_words, t.level_count);
  launch_pdl(records_kernel, grid_for(n, 256, 148 * 16), 256, 0, s, n, b.sys_of, b.ss, b.sc,
             t.level_count, b.bn_left, b.bn_right, b.bn_first, b.bn_last, b.bn_level, b.bn_rank,
             b.cn_bin, b.cn_meta, b.cn_child, b.cn_parent, b.level_begin, b.gflag);
}

void launch_groups(int64_t n, int group_size, int group_span, Buffers &b, cudaStream_t s) {
  const BuildTmp t = build_tmp(n, b);
  launch_pdl(group_flags_kernel, grid_for(n, 256, 148 * 16), 256, 0, s, b.cn_meta, b.cn_child,
             b.cn_parent, b.sc, group_size, group_span, b.ss, b.nsys, b.gflag);
  launch_pdl(group_first_kernel, (n + kGroupTile - 1) / kGroupTile, kGroupThreads, 0, s, n, b.gflag,
             b.sc, b.counters, t.tickets + 1, t.group_words, b.g_first);
}

}  // namespace bh
