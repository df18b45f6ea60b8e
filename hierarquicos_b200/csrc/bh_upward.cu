// Upward pass: mass, centre of mass, quadrupole and octupole of every octree
// node, level by level from the deepest level to the root, in FP64.
//
// Follows the translation method of fortran/octree_default.f90:744-882
// (evaluate_multipole): the node's mass and centre of mass from its children
// (:782-799); for every child, first its own moments (:815-821), then the
// parallel-axis terms m d d (:823-828) and m d d d (:830-844), then the
// octupole cross terms 3 d Q of a child node (:846-872); finally the summary
// sums oct(11) = sum 1..10, oct(12..14) = row sums (:875-880).  Moments are raw
// (not trace-free) moments about the node's centre of mass: quad = xx yy zz xy
// xz yz; oct = xxx xyy xzz yxx yyy yzz zxx zyy zzz xyz (the reference's order).
// Lone particles are point children (mass, position, no moments), so a node's
// children are processed exactly like the reference's twig/leaf children.
//
// Large systems: one launch per level, deepest first; a thread computes one
// node, loading all of its child records before using any so that the loads
// overlap.
//
// Systems of up to kChunkMax bodies, for which the 22 launches cost more than
// their work, run in three stages instead.  A node's range of bodies lies inside an
// aligned chunk of 2^8 or 2^15 bodies or spans those: the stage of the smallest one
// that holds it computes it, so all its children are done by earlier stages or by
// the same block.  Stage 1 takes one block per 256 bodies, a thread per binary
// node, with the chunk's bodies and results in shared memory; nodes that span its
// chunks go on lists (one per chunk of the next stage that holds them), and the
// later stages take one block per list.  Inside a block the levels present run
// deepest first with a block barrier between them.  A level holds at most 127
// nodes that cross one of the 127 inner boundaries of a later stage's chunk,
// which bounds the lists.  The same arithmetic in the same child order: the same
// bits.
// Both are bound by latency (about 300 bytes a node, all in L2).  Stages against
// levels (1,024 and 4,096 bodies: one cooperative launch with a grid barrier per
// level), us: 1,024 bodies 34 / 48, 4,096 39 / 59, 16,384 (monopole) 25 / 59,
// 262,144 114 / 122; but 100,003 (octupole) 153 / 113, 2^20 257 / 183, 5,000,011
// 952 / 460: a block's levels leave most of its threads idle, which costs once
// the blocks run in several waves.
//
// The same pass writes the normalised FP32 copies used by the FP32 walk:
// quadrupole / (M ssa^2) with its trace, octupole / (M ssa^3), where M is the
// total mass and ssa the root cube side, so the walk's values are O(1)
// whatever the physical units.
#include "bh_internal.cuh"

namespace bh {

namespace {

__device__ __forceinline__ double4 ld_com(const double4 *p) {
  const double2 a = __ldcg(reinterpret_cast<const double2 *>(p));
  const double2 b = __ldcg(reinterpret_cast<const double2 *>(p) + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}

// One child's contribution to the moments about (cx, cy, cz): its own
// moments (node children), then the parallel-axis and octupole cross terms.
template <int ORDER>
__device__ __forceinline__ void add_child(double pm, double px, double py, double pz, bool node,
                                          const double *Qd, const double *Od, double cx,
                                          double cy, double cz, double *Q, double *O) {
  const double dx = px - cx, dy = py - cy, dz = pz - cz;
  if (node) {
#pragma unroll
    for (int k = 0; k < 6; ++k) Q[k] = Q[k] + Qd[k];
    if (ORDER >= 8) {
#pragma unroll
      for (int k = 0; k < 14; ++k) O[k] = O[k] + Od[k];
    }
  }
  Q[0] = Q[0] + pm * (dx * dx);
  Q[1] = Q[1] + pm * (dy * dy);
  Q[2] = Q[2] + pm * (dz * dz);
  Q[3] = Q[3] + pm * dx * dy;
  Q[4] = Q[4] + pm * dx * dz;
  Q[5] = Q[5] + pm * dy * dz;
  if (ORDER >= 8) {
    O[0] = O[0] + pm * dx * (dx * dx);
    O[1] = O[1] + pm * dx * (dy * dy);
    O[2] = O[2] + pm * dx * (dz * dz);
    O[3] = O[3] + pm * dy * (dx * dx);
    O[4] = O[4] + pm * dy * (dy * dy);
    O[5] = O[5] + pm * dy * (dz * dz);
    O[6] = O[6] + pm * dz * (dx * dx);
    O[7] = O[7] + pm * dz * (dy * dy);
    O[8] = O[8] + pm * dz * (dz * dz);
    O[9] = O[9] + pm * dx * dy * dz;
    if (node) {
      O[0] = O[0] + 3.0 * dx * Qd[0];
      O[1] = O[1] + 2.0 * dy * Qd[3] + dx * Qd[1];
      O[2] = O[2] + 2.0 * dz * Qd[4] + dx * Qd[2];
      O[3] = O[3] + 2.0 * dx * Qd[3] + dy * Qd[0];
      O[4] = O[4] + 3.0 * dy * Qd[1];
      O[5] = O[5] + 2.0 * dz * Qd[5] + dy * Qd[2];
      O[6] = O[6] + 2.0 * dx * Qd[4] + dz * Qd[0];
      O[7] = O[7] + 2.0 * dy * Qd[5] + dz * Qd[1];
      O[8] = O[8] + 3.0 * dz * Qd[2];
      O[9] = O[9] + dx * Qd[5] + dy * Qd[4] + dz * Qd[3];
    }
  }
}

// ---- level by level ----

// Mass, centre of mass and moments of node j from its children.  For a node
// with child entries, all child records are loaded before any is used, so the
// loads overlap; the sums run in child order either way.  WAIT: the previous
// level's launch may still be running; what it does not write (the records and
// the lone bodies) is loaded before waiting for it.
template <int ORDER, bool WAIT>
__device__ __forceinline__ void compute_node(int j, const int4 *__restrict__ meta, const int32_t *__restrict__ child,
                             const double4 *__restrict__ spos, const int32_t *__restrict__ sys_of,
                             const SysScalars *__restrict__ sys, double4 *com, double *quad,
                             double *oct, float4 *__restrict__ fq, float4 *__restrict__ fo) {
  const int4 mt = meta[j];  // first, count, level, nchild
  const SysScalars &ss = sys[sys_of[mt.x]];
  const double inv_m = 1.0 / ss.mass;
  const double inv_s = 1.0 / ss.ssa;
  const double nq = inv_m * inv_s * inv_s, no = nq * inv_s;
  double M = 0.0, cx = 0.0, cy = 0.0, cz = 0.0;
  double Q[6] = {0, 0, 0, 0, 0, 0};
  double O[14] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  if (mt.w == 0) {  // bucket of identical keys: its bodies are the children
    if (WAIT) cudaGridDependencySynchronize();
    for (int c = 0; c < mt.y; ++c) {
      const double4 p = spos[mt.x + c];
      M = M + p.w;
      cx = cx + p.w * p.x;
      cy = cy + p.w * p.y;
      cz = cz + p.w * p.z;
    }
    if (M == 0.0) {  // massless node: a finite centre (it only enters sums times 0)
      const double4 p = spos[mt.x];
      cx = p.x; cy = p.y; cz = p.z;
    } else {
      cx = cx / M; cy = cy / M; cz = cz / M;
    }
    com[j] = make_double4(cx, cy, cz, M);
    if constexpr (ORDER < 4) {
      return;
    } else {
      for (int c = 0; c < mt.y; ++c) {
        const double4 p = spos[mt.x + c];
        add_child<ORDER>(p.w, p.x, p.y, p.z, false, nullptr, nullptr, cx, cy, cz, Q, O);
      }
    }
  } else {
    const int4 c0 = *reinterpret_cast<const int4 *>(child + 8 * (int64_t)j);
    const int4 c1 = *reinterpret_cast<const int4 *>(child + 8 * (int64_t)j + 4);
    const int32_t ch[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    double4 cd[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      cd[c] = make_double4(0.0, 0.0, 0.0, 0.0);
      if (c < mt.w && ch[c] < 0) cd[c] = spos[~ch[c]];
    }
    if (WAIT) cudaGridDependencySynchronize();
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (c < mt.w && ch[c] >= 0) cd[c] = ld_com(com + ch[c]);
    double Qd[ORDER >= 4 ? 8 : 1][6];
    if (ORDER >= 4) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (c < mt.w && ch[c] >= 0) {
          const double2 *q2 = reinterpret_cast<const double2 *>(quad + 6 * (int64_t)ch[c]);
          const double2 a = __ldcg(q2), b = __ldcg(q2 + 1), e = __ldcg(q2 + 2);
          Qd[c][0] = a.x; Qd[c][1] = a.y; Qd[c][2] = b.x; Qd[c][3] = b.y; Qd[c][4] = e.x; Qd[c][5] = e.y;
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (c < mt.w) {
        M = M + cd[c].w;
        cx = cx + cd[c].w * cd[c].x;
        cy = cy + cd[c].w * cd[c].y;
        cz = cz + cd[c].w * cd[c].z;
      }
    }
    if (M == 0.0) {  // massless node: a finite centre (it only enters sums times 0)
      cx = cd[0].x; cy = cd[0].y; cz = cd[0].z;
    } else {
      cx = cx / M; cy = cy / M; cz = cz / M;
    }
    com[j] = make_double4(cx, cy, cz, M);
    if constexpr (ORDER < 4) {
      return;
    } else {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (c < mt.w) {
          double Od[14];
          if (ORDER >= 8 && ch[c] >= 0) {
#pragma unroll
            for (int k = 0; k < 14; ++k) Od[k] = __ldcg(oct + 14 * (int64_t)ch[c] + k);
          }
          add_child<ORDER>(cd[c].w, cd[c].x, cd[c].y, cd[c].z, ch[c] >= 0, Qd[c], Od, cx, cy, cz,
                           Q, O);
        }
      }
    }
  }
  if constexpr (ORDER >= 4) {
#pragma unroll
    for (int k = 0; k < 6; ++k) quad[6 * (int64_t)j + k] = Q[k];
    const double trq = Q[0] + Q[1] + Q[2];
    fq[2 * (int64_t)j] = make_float4((float)(Q[0] * nq), (float)(Q[1] * nq), (float)(Q[2] * nq),
                                     (float)(Q[3] * nq));
    fq[2 * (int64_t)j + 1] =
        make_float4((float)(Q[4] * nq), (float)(Q[5] * nq), (float)(trq * nq), 0.0f);
    if (ORDER >= 8) {
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < 10; ++k) s = s + O[k];
      O[10] = s;
      O[11] = O[0] + O[1] + O[2];
      O[12] = O[3] + O[4] + O[5];
      O[13] = O[6] + O[7] + O[8];
#pragma unroll
      for (int k = 0; k < 14; ++k) oct[14 * (int64_t)j + k] = O[k];
      float4 *f = fo + 4 * (int64_t)j;
      f[0] = make_float4((float)(O[0] * no), (float)(O[1] * no), (float)(O[2] * no), (float)(O[3] * no));
      f[1] = make_float4((float)(O[4] * no), (float)(O[5] * no), (float)(O[6] * no), (float)(O[7] * no));
      f[2] = make_float4((float)(O[8] * no), (float)(O[9] * no), (float)(O[11] * no), (float)(O[12] * no));
      f[3] = make_float4((float)(O[13] * no), 0.0f, 0.0f, 0.0f);
    }
  }
}

template <int ORDER>
__global__ void __launch_bounds__(128)
upward_level_kernel(int level, const int32_t *__restrict__ level_begin,
                    const int4 *__restrict__ meta, const int32_t *__restrict__ child,
                    const double4 *__restrict__ spos, const int32_t *__restrict__ sys_of,
                    const SysScalars *__restrict__ sys, double4 *com, double *quad, double *oct,
                    float4 *__restrict__ fq, float4 *__restrict__ fo) {
  // The next level's launch may start now.  The records were complete before
  // the deepest level's (ordinary) launch began; every thread waits for the level
  // before this one, which waited for its own predecessor, so the levels complete
  // in order.
  cudaTriggerProgrammaticLaunchCompletion();
  const int lb = level_begin[level], le = level_begin[level + 1];
  int j = lb + blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= le) {
    cudaGridDependencySynchronize();
    return;
  }
  compute_node<ORDER, true>(j, meta, child, spos, sys_of, sys, com, quad, oct, fq, fo);
  for (j += gridDim.x * blockDim.x; j < le; j += gridDim.x * blockDim.x)
    compute_node<ORDER, false>(j, meta, child, spos, sys_of, sys, com, quad, oct, fq, fo);
}

// ---- by chunks of bodies ----

// Moments of one node as its parent reads them.
template <int ORDER> struct __align__(16) Moments {
  double x, y, z, m;
  double q[ORDER >= 4 ? 6 : 1];
  double o[ORDER >= 8 ? 14 : 1];
};

// Mass, centre of mass and moments of a node from its nch children, which
// child(c, body) names: the moments record of a child node, or the body (and
// null) of a lone particle or bucket body.  The sums run in child order.
// MAX > 0: at most MAX children, unrolled (for children held in registers).
template <int ORDER, int MAX, typename ChildFn>
__device__ __forceinline__ void combine(int nch, ChildFn &&child, Moments<ORDER> &r) {
  constexpr int kUnroll = MAX > 0 ? MAX : 1;
  double M = 0.0, cx = 0.0, cy = 0.0, cz = 0.0;
#pragma unroll kUnroll
  for (int c = 0; c < (MAX > 0 ? MAX : nch); ++c) {
    if (MAX > 0 && c >= nch) continue;
    double4 p;
    child(c, p);
    M = M + p.w;
    cx = cx + p.w * p.x;
    cy = cy + p.w * p.y;
    cz = cz + p.w * p.z;
  }
  if (M == 0.0) {  // massless node: a finite centre (it only enters sums times 0)
    double4 p;
    child(0, p);
    cx = p.x; cy = p.y; cz = p.z;
  } else {
    cx = cx / M; cy = cy / M; cz = cz / M;
  }
  r.x = cx; r.y = cy; r.z = cz; r.m = M;
  if constexpr (ORDER >= 4) {
    double Q[6] = {0, 0, 0, 0, 0, 0};
    double O[14] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll kUnroll
    for (int c = 0; c < (MAX > 0 ? MAX : nch); ++c) {
      if (MAX > 0 && c >= nch) continue;
      double4 p;
      const Moments<ORDER> *d = child(c, p);
      add_child<ORDER>(p.w, p.x, p.y, p.z, d != nullptr, d ? d->q : nullptr, d ? d->o : nullptr, cx,
                       cy, cz, Q, O);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) r.q[k] = Q[k];
    if constexpr (ORDER >= 8) {
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < 10; ++k) s = s + O[k];
      O[10] = s;
      O[11] = O[0] + O[1] + O[2];
      O[12] = O[3] + O[4] + O[5];
      O[13] = O[6] + O[7] + O[8];
#pragma unroll
      for (int k = 0; k < 14; ++k) r.o[k] = O[k];
    }
  }
}

struct UpArgs {
  const int32_t *first, *last, *level, *rank, *level_begin, *cbin, *child, *sys_of;
  const int4 *meta;
  const double4 *spos;
  const SysScalars *sys;
  double4 *com;
  double *quad, *oct;
  float4 *fq, *fo;
  int32_t *list1, *list2, *count;  // lists of stages 2 and 3
  int *err;
  int64_t n;
};

// Node j's results to global memory, with the normalised FP32 copies.
template <int ORDER>
__device__ __forceinline__ void store_node(const UpArgs &a, int64_t j, const Moments<ORDER> &r,
                                           double nq, double no) {
  a.com[j] = make_double4(r.x, r.y, r.z, r.m);
  if constexpr (ORDER >= 4) {
    double2 *q2 = reinterpret_cast<double2 *>(a.quad + 6 * j);
    q2[0] = make_double2(r.q[0], r.q[1]); q2[1] = make_double2(r.q[2], r.q[3]);
    q2[2] = make_double2(r.q[4], r.q[5]);
    const double trq = r.q[0] + r.q[1] + r.q[2];
    a.fq[2 * j] = make_float4((float)(r.q[0] * nq), (float)(r.q[1] * nq), (float)(r.q[2] * nq),
                              (float)(r.q[3] * nq));
    a.fq[2 * j + 1] =
        make_float4((float)(r.q[4] * nq), (float)(r.q[5] * nq), (float)(trq * nq), 0.0f);
  }
  if constexpr (ORDER >= 8) {
    const double *O = r.o;
#pragma unroll
    for (int k = 0; k < 14; ++k) a.oct[14 * j + k] = O[k];
    float4 *f = a.fo + 4 * j;
    f[0] = make_float4((float)(O[0] * no), (float)(O[1] * no), (float)(O[2] * no), (float)(O[3] * no));
    f[1] = make_float4((float)(O[4] * no), (float)(O[5] * no), (float)(O[6] * no), (float)(O[7] * no));
    f[2] = make_float4((float)(O[8] * no), (float)(O[9] * no), (float)(O[11] * no), (float)(O[12] * no));
    f[3] = make_float4((float)(O[13] * no), 0.0f, 0.0f, 0.0f);
  }
}

constexpr int kChunkBits = 8, kChunk = 1 << kChunkBits, kStageBits = 7;
constexpr int kListCap = ((1 << kStageBits) - 1) * (kMaxDepth + 1);  // nodes of one list
constexpr int kUpThreads = 256;
constexpr int64_t kChunkMax = 65536;  // the most bodies that go in stages
static_assert(kChunkMax <= (int64_t)1 << (kChunkBits + 2 * kStageBits), "three stages hold every node");
static_assert((kChunkMax >> (kChunkBits + kStageBits)) + 2 <= kUpwardCounters, "a counter per list");

// list of a chunk of stage 2 (2^15 bodies) or 3 (all of them).  Stage 2's lists are
// kListCap entries apart; a last, partial chunk holds fewer nodes than bodies, so the
// arrays of n entries hold them all.
__device__ __forceinline__ int32_t *up_list(const UpArgs &a, int stage, int64_t chunk,
                                            int32_t *&count) {
  if (stage == 2) {
    count = a.count + chunk;
    return a.list1 + chunk * kListCap;
  }
  count = a.count + (a.n >> (kChunkBits + kStageBits)) + 1;
  return a.list2;
}

// Stage 1: one block per 256 bodies, thread t the binary node at base + t.
template <int ORDER>
__global__ void __launch_bounds__(kUpThreads)
upward_chunk_kernel(UpArgs a) {
  extern __shared__ __align__(16) unsigned char up_smem[];
  double4 *body = reinterpret_cast<double4 *>(up_smem);
  Moments<ORDER> *node = reinterpret_cast<Moments<ORDER> *>(body + kChunk);
  __shared__ unsigned levels;
  const int64_t base = (int64_t)blockIdx.x * kChunk;
  const int64_t i = base + threadIdx.x;
  pdl_enter();
  if (threadIdx.x == 0) levels = 0;
  int64_t j = -1;
  int lev = -1, nch = 0, bucket = 0;
  int32_t ch[8];
  double nq = 0.0, no = 0.0;
  if (i < a.n) body[threadIdx.x] = a.spos[i];
  __syncthreads();
  const int r = i < a.n ? a.rank[i] : -1;
  if (r >= 0) {
    const int f = a.first[i], la = a.last[i], v = a.level[i];
    const int64_t id = a.level_begin[v] + r;
    const int span = 31 - __clz(f ^ la);  // highest bit in which the range's ends differ
    if (span < kChunkBits) {
      j = id;
      lev = v;
      const int4 mt = a.meta[j];
      nch = mt.w;
      if (nch == 0) {  // bucket of identical keys: its bodies are the children
        bucket = 1;
        nch = mt.y;
        ch[0] = (int32_t)(mt.x - base);
      } else {
        const int4 c0 = *reinterpret_cast<const int4 *>(a.child + 8 * j);
        const int4 c1 = *reinterpret_cast<const int4 *>(a.child + 8 * j + 4);
        const int32_t raw[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
        for (int c = 0; c < 8; ++c)  // local: bodies ~p, nodes by their binary index
          ch[c] = c < nch ? (raw[c] < 0 ? ~(int32_t)(~raw[c] - base) : (int32_t)(a.cbin[raw[c]] - base)) : 0;
      }
      const SysScalars &ss = a.sys[a.sys_of[f]];
      const double inv_m = 1.0 / ss.mass, inv_s = 1.0 / ss.ssa;
      nq = inv_m * inv_s * inv_s; no = nq * inv_s;
      atomicOr(&levels, 1u << v);
    } else {
      const int stage = 2 + (span - kChunkBits) / kStageBits;
      int32_t *count;
      int32_t *list = up_list(a, stage, (int64_t)f >> (kChunkBits + kStageBits * (stage - 1)), count);
      const int k = atomicAdd(count, 1);
      if (k < kListCap) list[k] = (int32_t)id;
      else atomicOr(a.err, kErrIndex);  // cannot happen: see kListCap
    }
  }
  __syncthreads();
  for (unsigned todo = levels; todo;) {
    const int l = 31 - __clz(todo);
    todo ^= 1u << l;
    if (lev == l) {
      Moments<ORDER> res;
      if (bucket) {
        combine<ORDER, 0>(nch, [&](int c, double4 &p) -> const Moments<ORDER> * {
          p = body[ch[0] + c];
          return nullptr;
        }, res);
      } else {
        combine<ORDER, 8>(nch, [&](int c, double4 &p) -> const Moments<ORDER> * {
          // a body is (x, y, z, m) and a node's record starts with the same
          const Moments<ORDER> *d = node + ch[c];
          p = *(ch[c] < 0 ? body + ~ch[c] : reinterpret_cast<const double4 *>(d));
          return ch[c] < 0 ? nullptr : d;
        }, res);
      }
      node[threadIdx.x] = res;
      store_node<ORDER>(a, j, res, nq, no);
    }
    __syncthreads();
  }
}

// One node of a list, in shared memory: what does not depend on other nodes is
// loaded before the levels run, so a level waits for one trip to L2.
struct __align__(16) ListEntry {
  int32_t ch[8];
  double nq, no;
  int32_t id, nch, first, pad;  // nch < 0: a bucket of -nch bodies from `first`
};

// Later stages: one block per list.  Children are read from global memory
// (through L2: a node of this list may have been written by another thread of
// the block).
template <int ORDER>
__global__ void __launch_bounds__(kUpThreads)
upward_list_kernel(UpArgs a, int stage) {
  extern __shared__ __align__(16) unsigned char up_smem[];
  ListEntry *entry = reinterpret_cast<ListEntry *>(up_smem);  // by level
  __shared__ int begin[kWarp + 1], fill[kWarp];
  pdl_enter();
  int32_t *cnt;
  const int32_t *list = up_list(a, stage, blockIdx.x, cnt);
  const int n = min(*cnt, kListCap);
  if (n == 0) return;  // uniform across the block
  if (threadIdx.x < kWarp) fill[threadIdx.x] = 0;
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += kUpThreads) atomicAdd(&fill[a.meta[list[k]].z], 1);
  __syncthreads();
  if (threadIdx.x < kWarp) {
    const int c = fill[threadIdx.x];
    int v = c;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, v, o);
      if ((int)threadIdx.x >= o) v += t;
    }
    begin[threadIdx.x + 1] = v;
    if (threadIdx.x == 0) begin[0] = 0;
    fill[threadIdx.x] = v - c;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += kUpThreads) {
    const int32_t j = list[k];
    const int4 mt = a.meta[j];
    const int4 *cp = reinterpret_cast<const int4 *>(a.child + 8 * (int64_t)j);
    const int4 c0 = cp[0], c1 = cp[1];
    const SysScalars &ss = a.sys[a.sys_of[mt.x]];
    const double inv_m = 1.0 / ss.mass, inv_s = 1.0 / ss.ssa;
    ListEntry &e = entry[atomicAdd(&fill[mt.z], 1)];  // any order within a level
    *reinterpret_cast<int4 *>(e.ch) = c0;
    *reinterpret_cast<int4 *>(e.ch + 4) = c1;
    e.nq = inv_m * inv_s * inv_s;
    e.no = e.nq * inv_s;
    e.id = j;
    e.nch = mt.w == 0 ? -mt.y : mt.w;
    e.first = mt.x;
  }
  __syncthreads();
  for (int l = kMaxDepth; l >= 0; --l) {
    if (begin[l] == begin[l + 1]) continue;  // uniform across the block
    for (int k = begin[l] + threadIdx.x; k < begin[l + 1]; k += kUpThreads) {
      const ListEntry &e = entry[k];
      Moments<ORDER> res;
      if (e.nch < 0) {  // a bucket that spans chunks
        combine<ORDER, 0>(-e.nch, [&](int c, double4 &p) -> const Moments<ORDER> * {
          p = a.spos[e.first + c];
          return nullptr;
        }, res);
      } else {
        // the child records are loaded before any is used, so the loads overlap
        // (the octupole's third moments, which would not fit the registers, later)
        const int nch = e.nch;
        Moments<(ORDER >= 4 ? 4 : 1)> d[8];
        int32_t ch[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          ch[c] = e.ch[c];
          if (c >= nch) continue;
          const double2 *p = reinterpret_cast<const double2 *>(ch[c] < 0 ? a.spos + ~ch[c] : a.com + ch[c]);
          const double2 u = __ldcg(p), v = __ldcg(p + 1);
          d[c].x = u.x; d[c].y = u.y; d[c].z = v.x; d[c].m = v.y;
          if constexpr (ORDER >= 4) {
            if (ch[c] >= 0) {
              const double2 *q2 = reinterpret_cast<const double2 *>(a.quad + 6 * (int64_t)ch[c]);
#pragma unroll
              for (int k = 0; k < 3; ++k) {
                const double2 w = __ldcg(q2 + k);
                d[c].q[2 * k] = w.x; d[c].q[2 * k + 1] = w.y;
              }
            }
          }
        }
        Moments<ORDER> full;
        combine<ORDER, 8>(nch, [&](int c, double4 &p) -> const Moments<ORDER> * {
          p = make_double4(d[c].x, d[c].y, d[c].z, d[c].m);
          if (ch[c] < 0) return nullptr;
          if constexpr (ORDER >= 4) {
#pragma unroll
            for (int k = 0; k < 6; ++k) full.q[k] = d[c].q[k];
          }
          if constexpr (ORDER >= 8) {
            const double2 *o2 = reinterpret_cast<const double2 *>(a.oct + 14 * (int64_t)ch[c]);
#pragma unroll
            for (int k = 0; k < 7; ++k) {
              const double2 w = __ldcg(o2 + k);
              full.o[2 * k] = w.x; full.o[2 * k + 1] = w.y;
            }
          }
          return &full;
        }, res);
      }
      store_node<ORDER>(a, e.id, res, e.nq, e.no);
    }
    __syncthreads();
  }
}

template <int ORDER>
void launch_upward_t(const UpArgs &a, cudaStream_t s) {
  constexpr int chunk_smem = kChunk * (int)(sizeof(double4) + sizeof(Moments<ORDER>));
  static bool done[64] = {};  // the shared-memory limit is set once per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!done[dev]) {
    cudaFuncSetAttribute(upward_chunk_kernel<ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         chunk_smem);
    cudaFuncSetAttribute(upward_list_kernel<ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         kListCap * (int)sizeof(ListEntry));
    done[dev] = true;
  }
  launch_pdl(upward_chunk_kernel<ORDER>, (a.n + kChunk - 1) / kChunk, kUpThreads, chunk_smem, s, a);
  for (int stage = 2; a.n > ((int64_t)1 << (kChunkBits + kStageBits * (stage - 2))); ++stage) {
    const int bits = kChunkBits + kStageBits * (stage - 1);
    launch_pdl(upward_list_kernel<ORDER>, (a.n + ((int64_t)1 << bits) - 1) >> bits, kUpThreads,
               (size_t)bh_min64(kListCap, a.n) * sizeof(ListEntry), s, a, stage);
  }
}

template <int ORDER>
void launch_levels(int64_t n, Buffers &b, cudaStream_t s) {
  const int grid = grid_for(n / 2 + 1, 128, 148 * 8);
  for (int level = kMaxDepth; level >= 0; --level) {
    if (level == kMaxDepth)
      upward_level_kernel<ORDER><<<grid, 128, 0, s>>>(level, b.level_begin, b.cn_meta, b.cn_child,
                                                      b.spos, b.sys_of, b.ss, b.cn_com, b.cn_quad,
                                                      b.cn_oct, b.cn_fq, b.cn_fo);
    else
      launch_pdl(upward_level_kernel<ORDER>, grid, 128, 0, s, level, b.level_begin, b.cn_meta,
                 b.cn_child, b.spos, b.sys_of, b.ss, b.cn_com, b.cn_quad, b.cn_oct, b.cn_fq, b.cn_fo);
  }
}

}  // namespace

void launch_upward(int64_t n, int order, Buffers &b, cudaStream_t s) {
  if (n > kChunkMax) {
    if (order >= 8) launch_levels<8>(n, b, s);
    else if (order >= 4) launch_levels<4>(n, b, s);
    else launch_levels<1>(n, b, s);
    return;
  }
  UpArgs a;
  a.first = b.bn_first; a.last = b.bn_last; a.level = b.bn_level; a.rank = b.bn_rank;
  a.level_begin = b.level_begin; a.cbin = b.cn_bin; a.child = b.cn_child; a.sys_of = b.sys_of;
  a.meta = b.cn_meta; a.spos = b.spos; a.sys = b.ss;
  a.com = b.cn_com; a.quad = b.cn_quad; a.oct = b.cn_oct; a.fq = b.cn_fq; a.fo = b.cn_fo;
  a.list1 = b.up_list; a.list2 = b.gscan; a.count = upward_counters(n, b);
  a.err = &b.sc->err;
  a.n = n;
  if (order >= 8) launch_upward_t<8>(a, s);
  else if (order >= 4) launch_upward_t<4>(a, s);
  else launch_upward_t<1>(a, s);
}

}  // namespace bh
