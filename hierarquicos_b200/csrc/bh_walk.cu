// Tree walks.
//
// 1. Group walk (the production path), after Barnes (1990) as restated by
//    fortran/octree_default.f90:1811-2095 (forces_groups / group_worker): one
//    warp per group of <= 64 Morton-contiguous targets.  The warp walks the
//    tree 32 nodes at a time from a per-warp stack, tests each node with the
//    box-distance MAC of :1927-1936 (size^2 <= theta^2 * dist^2 from the
//    node's centre of mass to the group's bounding box), queues accepted
//    nodes as cells and the bodies of opened leaves / lone particles as
//    bodies, and evaluates the queues in batches of 32: lane j stages entry j
//    (a coalesced load) into shared memory and every lane then sweeps the 32
//    staged entries (broadcast reads) for its own 1 or 2 targets.  Each batch
//    is summed in registers and Kahan-added (Kahan 1965) into the per-target
//    accumulator.  Positions are taken relative to the group's centre in FP64
//    and only then rounded, and everything is scaled to the root cube side and
//    total mass, so the FP32 arithmetic sees O(1) numbers.  The cell formulas
//    are the reference's (:1993-2083) with r^-3 factored out so that no
//    intermediate power of r overflows FP32.
//    Because the box distance never exceeds a member's own distance, every
//    accepted cell also passes the per-target MAC of the classic walk.
//
// 2. Reference walk: one thread per target with the semantics of
//    fortran/morton/morton_octree.f90:627-766 (barnes_hut) in FP64 over the
//    compact tree: the node containing the target is always opened, cells are
//    tested with the target-to-centre distance, lone particles are monopoles
//    at m*q/m, level-L leaves are summed particle by particle.  Used to check
//    the tree against the reference and to count the reference's interactions.
#include <math.h>
#include <stdint.h>

#include "bh_fp64.cuh"
#include "bh_internal.cuh"

namespace bh {

namespace {

// The walk runs one warp per block.  The FP32 walk is compiled for 16 resident
// blocks per SM (128 registers a thread).
constexpr int kWalkBlocksPerSm = 16;
// One-warp blocks per SM the walk is compiled for, FP64 as FP32: 16 (128
// registers) against the compiler's own choice for FP64 (182 / 222 registers,
// 11 / 9 warps per SM) took the FP64 walk at 2^20 from 15.5 to 12.3 ms
// (quadrupole) and from 29.4 to 26.3 ms (octupole, despite 592 bytes of
// spills; 12 blocks: 27.1 ms), the same bits.  Of the FP64 octupole walk, whose
// block has 13,696 bytes of shared memory, 15 fit on an SM.
template <typename T, int ORDER> constexpr int walk_min_blocks() { return kWalkBlocksPerSm; }
constexpr int kCellQ = 64;
constexpr int kBodyPerLane = 16;
constexpr int kBodyQ = 32 + kWarp * kBodyPerLane;  // 544
constexpr unsigned kFull = 0xffffffffu;
constexpr int32_t kNoChild = 0x7fffffff;  // unused entry of a node's child list (records_kernel)

template <typename T> struct Ops;
template <> struct Ops<float> {
  static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ float rsq(float r2) { return r2 > 0.0f ? rsqrtf(r2) : 0.0f; }
};
template <> struct Ops<double> {
  static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
  static __device__ __forceinline__ double rsq(double r2) { return r2 > 0.0 ? rsqrt(r2) : 0.0; }
};

template <typename T>
__device__ __forceinline__ void kahan_add(T &s, T &c, T x) {
  T y = Ops<T>::sub(x, c);
  T t = Ops<T>::add(s, y);
  c = Ops<T>::sub(Ops<T>::sub(t, s), y);
  s = t;
}

template <int ORDER> struct StageWords { static constexpr int value = ORDER >= 8 ? 24 : (ORDER >= 4 ? 12 : 4); };

template <typename T> struct __align__(16) Vec4 { T x, y, z, w; };

// Shared memory of one tree walk: the queues, the members and the members'-MAC
// candidates of the current group, and the top of the walk's stack.
constexpr int kSamples = 8;         // members of the first look of the members' MAC
constexpr int kStackWindow = 512;  // stack entries kept in shared memory (a power of two)
template <typename T>
struct __align__(16) WalkSmem {
  Vec4<T> member[2 * kWarp];  // group-frame position of every target slot
  Vec4<T> cand[kWarp];        // centre of mass and size^2 of the nodes to test
  int window[kStackWindow];
  int cellq[kCellQ];
  int bodyq[kBodyQ];
};

template <typename T, int ORDER>
struct __align__(16) WarpSmem {
  T stage[kWarp * StageWords<ORDER>::value];
  WalkSmem<T> w;
};

struct WalkArgs {
  const int4 *meta;
  const int32_t *child;
  const double4 *com;
  const double *quad;
  const double *oct;
  const float4 *fq;
  const float4 *fo;
  const double4 *spos;
  const int32_t *perm;
  const int32_t *g_first;
  const int32_t *sys_of;
  const SysScalars *ss;
  Scalars *sc;
  int32_t *cursor;
  int32_t *stack;
  int64_t stack_cap;
  int64_t slots;
  unsigned long long *stats;
  double *out;
  int64_t n;
  double theta2, G, eps2;
  int out_kind, leaf_cap, count_stats, mac;
  int g_begin, g_end;  // groups walked: [g_begin, g_end), g_end < 0 = all
  int pipeline;        // producer / consumer warps
  int64_t largest;     // choose_walk: bodies of the largest system,
  double walk_groups;  // and groups weighed by the length of their walks
};

// a predicated shared-memory store: no branch, whatever the lanes decide
__device__ __forceinline__ void store_if(int *p, int v, bool yes) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\t@q st.shared.s32 [%0], %1;\n\t}"
               ::"r"((unsigned)__cvta_generic_to_shared(p)), "r"(v), "r"((int)yes)
               : "memory");
}

template <typename T>
__device__ __forceinline__ T warp_min(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(kFull, v, o));
  return v;
}
template <typename T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(kFull, v, o));
  return v;
}

__device__ __forceinline__ int warp_excl_scan(int v, int lane, int &total) {
  int x = v;
#pragma unroll
  for (int o = 1; o < kWarp; o <<= 1) {
    int t = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += t;
  }
  total = __shfl_sync(kFull, x, kWarp - 1);
  return x - v;
}

// Stage one cell (node j) as T words, all in the group's frame (positions
// relative to the group centre over the root cube side, masses over the total
// mass):
//   [0..3]   x, y, z, m
//   [4..7]   7.5 Qxx, 7.5 Qyy, 7.5 Qzz, 7.5 Qxy
//   [8..11]  7.5 Qxz, 7.5 Qyz, -1.5 trQ, O14
//   [12..23] O1..O10, O12, O13     (octupole only)
// The factors 7.5 and -1.5 of the reference's cell formula
// (octree_default.f90:2024-2027) are folded in here once per staged cell.
// Word k goes to w[k * STR]: STR = 1 for the FP64 walk, 2 for the paired FP32
// walk, whose stage holds cells 2i and 2i+1 interleaved word by word.
template <typename T, int ORDER, int STR = 1>
__device__ __forceinline__ void stage_cell(T *w, int j, const WalkArgs &a, const double gc[3],
                                           double inv_s, double inv_m, double nq, double no) {
  const double4 c = a.com[j];
  w[0 * STR] = (T)((c.x - gc[0]) * inv_s);
  w[1 * STR] = (T)((c.y - gc[1]) * inv_s);
  w[2 * STR] = (T)((c.z - gc[2]) * inv_s);
  w[3 * STR] = (T)(c.w * inv_m);
  if (ORDER >= 4) {
    if (sizeof(T) == 4) {
      const float4 q0 = a.fq[2 * (int64_t)j], q1 = a.fq[2 * (int64_t)j + 1];
      w[4 * STR] = (T)(7.5f * q0.x); w[5 * STR] = (T)(7.5f * q0.y); w[6 * STR] = (T)(7.5f * q0.z);
      w[7 * STR] = (T)(7.5f * q0.w); w[8 * STR] = (T)(7.5f * q1.x); w[9 * STR] = (T)(7.5f * q1.y);
      w[10 * STR] = (T)(-1.5f * q1.z);
    } else {
      const double *q = a.quad + 6 * (int64_t)j;
      const double q0 = q[0] * nq, q1 = q[1] * nq, q2 = q[2] * nq;
      w[4 * STR] = (T)(7.5 * q0); w[5 * STR] = (T)(7.5 * q1); w[6 * STR] = (T)(7.5 * q2);
      w[7 * STR] = (T)(7.5 * q[3] * nq); w[8 * STR] = (T)(7.5 * q[4] * nq);
      w[9 * STR] = (T)(7.5 * q[5] * nq);
      w[10 * STR] = (T)(-1.5 * (q0 + q1 + q2));
    }
    w[11 * STR] = (T)0;
  }
  if (ORDER >= 8) {
    if (sizeof(T) == 4) {
      const float4 *f = a.fo + 4 * (int64_t)j;
      const float4 o0 = f[0], o1 = f[1], o2 = f[2], o3 = f[3];
      w[12 * STR] = (T)o0.x; w[13 * STR] = (T)o0.y; w[14 * STR] = (T)o0.z; w[15 * STR] = (T)o0.w;
      w[16 * STR] = (T)o1.x; w[17 * STR] = (T)o1.y; w[18 * STR] = (T)o1.z; w[19 * STR] = (T)o1.w;
      w[20 * STR] = (T)o2.x; w[21 * STR] = (T)o2.y; w[22 * STR] = (T)o2.z; w[23 * STR] = (T)o2.w;
      w[11 * STR] = (T)o3.x;
    } else {
      const double *o = a.oct + 14 * (int64_t)j;
      for (int k = 0; k < 10; ++k) w[(12 + k) * STR] = (T)(o[k] * no);
      w[22 * STR] = (T)(o[11] * no);
      w[23 * STR] = (T)(o[12] * no);
      w[11 * STR] = (T)(o[13] * no);
    }
  }
}

// Vector loads of W staged words (float4 / double2).
template <int W>
__device__ __forceinline__ void load_words(const float *p, float (&w)[W]) {
#pragma unroll
  for (int k = 0; k < W; k += 4) {
    const float4 v = *reinterpret_cast<const float4 *>(p + k);
    w[k] = v.x; w[k + 1] = v.y; w[k + 2] = v.z; w[k + 3] = v.w;
  }
}
template <int W>
__device__ __forceinline__ void load_words(const double *p, double (&w)[W]) {
#pragma unroll
  for (int k = 0; k < W; k += 2) {
    const double2 v = *reinterpret_cast<const double2 *>(p + k);
    w[k] = v.x; w[k + 1] = v.y;
  }
}

// Reciprocal square root.  FP32: one approximate hardware instruction
// (rel. error ~2^-22.9) with subnormals flushed: every input is a squared
// distance in units of the root cube side, never subnormal.  FP64: the
// binomial series of bh_fp64.cuh (the same range holds; kEps2Max bounds it
// above).
__device__ __forceinline__ float fast_rsqrt(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ double fast_rsqrt(double x) { return inv_sqrt64(x); }

// m r^-3 from r^2
__device__ __forceinline__ float mass_r3(float r2, float m) {
  const float ri = fast_rsqrt(r2);
  return (m * ri) * (ri * ri);
}
__device__ __forceinline__ double mass_r3(double r2, double m) { return mass_over_r3(r2, m); }

// A softening beyond this (squared, in root sides) gives zero forces either
// way; larger squares would leave the series' range.
constexpr double kEps2Max = 1e250;

// (2^-level)^2 = 2^(-2 level), exact, from the exponent bits (level <= 21)
template <typename T> __device__ __forceinline__ T pow2_neg2(int level);
template <> __device__ __forceinline__ float pow2_neg2<float>(int level) {
  return __int_as_float((127 - 2 * level) << 23);
}
template <> __device__ __forceinline__ double pow2_neg2<double>(int level) {
  return __longlong_as_double((long long)(1023 - 2 * level) << 52);
}

// Smallest r^2 of a body pair when there is no softening: a body meets itself
// (d = 0, contribution exactly 0) and exactly coincident bodies contribute 0;
// r^-3 stays finite in T.
template <typename T> __device__ __forceinline__ T r2_floor();
template <> __device__ __forceinline__ float r2_floor<float>() { return 1e-24f; }
template <> __device__ __forceinline__ double r2_floor<double>() { return 1e-200; }

// One body-body term added to (bx, by, bz) (morton_octree.f90:676-686).
template <typename T, bool SOFT>
__device__ __forceinline__ void body_force(T sx, T sy, T sz, T sm, T rx, T ry, T rz, T eps2,
                                           T &bx, T &by, T &bz) {
  const T dx = sx - rx, dy = sy - ry, dz = sz - rz;
  T r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
  if (!SOFT) r2 = max(r2, r2_floor<T>());
  const T f = mass_r3(r2, sm);
  bx = fma(f, dx, bx); by = fma(f, dy, by); bz = fma(f, dz, bz);
}

// One cell term added to (bx, by, bz): the reference's grouped-walk formula
// (octree_default.f90:1993-2083) with r^-3 factored out of every term:
//   a += r^-3 [ (M - 1.5 trQ r^-2 + 7.5 dQd r^-4) d - 3 r^-2 Q d + r^3 O(d) ].
// Accepted cells never coincide with a target (the group box lies outside the
// MAC radius), so r^2 > 0.
template <typename T, int ORDER>
__device__ __forceinline__ void cell_force(const T *w, T rx, T ry, T rz, T eps2, T &bx, T &by,
                                           T &bz) {
  const T dx = w[0] - rx, dy = w[1] - ry, dz = w[2] - rz;
  const T r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
  const T rinv = fast_rsqrt(r2);
  const T r2i = rinv * rinv;
  const T r3i = rinv * r2i;
  if (ORDER < 4) {
    const T f = w[3] * r3i;
    bx = fma(f, dx, bx); by = fma(f, dy, by); bz = fma(f, dz, bz);
    return;
  }
  // w[4..9] = 7.5 Q, w[10] = -1.5 trQ
  const T qx = fma(w[4], dx, fma(w[7], dy, w[8] * dz));
  const T qy = fma(w[7], dx, fma(w[5], dy, w[9] * dz));
  const T qz = fma(w[8], dx, fma(w[9], dy, w[6] * dz));
  const T dqd = fma(dx, qx, fma(dy, qy, dz * qz));          // 7.5 dQd
  const T A = fma(dqd, r2i * r2i, fma(w[10], r2i, w[3]));  // M - 1.5 tr r^-2 + 7.5 dQd r^-4
  const T sA = r3i * A;
  const T t = (T)-0.4 * (r3i * r2i);                        // -3 r^-5 / 7.5
  if (ORDER < 8) {
    bx = fma(sA, dx, fma(t, qx, bx));
    by = fma(sA, dy, fma(t, qy, by));
    bz = fma(sA, dz, fma(t, qz, bz));
    return;
  }
  const T O1 = w[12], O2 = w[13], O3 = w[14], O4 = w[15], O5 = w[16], O6 = w[17], O7 = w[18],
          O8 = w[19], O9 = w[20], O10 = w[21], O12 = w[22], O13 = w[23], O14 = w[11];
  const T s7 = (T)7.5 * r2i * r2i;          // 7.5 r^-4
  const T s5 = (T)-1.5 * r2i;               // -1.5 r^-2
  const T s9 = (T)-17.5 * r2i * r2i * r2i;  // -17.5 r^-6
  const T xx = dx * dx, yy = dy * dy, zz = dz * dz, xy = dx * dy, xz = dx * dz, yz = dy * dz;
  const T oc = s7 * fma(dx, O12, fma(dy, O13, dz * O14));
  T ox = fma(s5, O12, dx * oc), oy = fma(s5, O13, dy * oc), oz = fma(s5, O14, dz * oc);
  ox = fma(s7, fma(xx, O1, fma(yy, O2, zz * O3)) + (T)2 * fma(xy, O4, fma(xz, O7, yz * O10)), ox);
  oy = fma(s7, fma(xx, O4, fma(yy, O5, zz * O6)) + (T)2 * fma(xy, O2, fma(xz, O10, yz * O8)), oy);
  oz = fma(s7, fma(xx, O7, fma(yy, O8, zz * O9)) + (T)2 * fma(xy, O10, fma(xz, O3, yz * O6)), oz);
  T c3 = fma(xx * dx, O1, fma(yy * dy, O5, zz * dz * O9));
  c3 = fma((T)3, fma(xx * dy, O4, fma(xx * dz, O7, xy * dy * O2)), c3);
  c3 = fma((T)3, fma(yy * dz, O8, fma(xz * dz, O3, yz * dz * O6)), c3);
  c3 = fma((T)6 * xy, dz * O10, c3);
  c3 = s9 * c3;
  ox = fma(dx, c3, ox); oy = fma(dy, c3, oy); oz = fma(dz, c3, oz);
  bx = fma(sA, dx, fma(t, qx, fma(r3i, ox, bx)));
  by = fma(sA, dy, fma(t, qy, fma(r3i, oy, by)));
  bz = fma(sA, dz, fma(t, qz, fma(r3i, oz, bz)));
}

// ---- paired FP32 (sm_100 f32x2 instructions) ----
//
// The FP32 walk evaluates two staged entries (cells j and j+1, or bodies) per
// instruction: every operand is a float2 whose halves belong to the two
// entries, and the target's coordinates are the same in both halves.  Each half
// is rounded exactly like the scalar operation it replaces.
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 splat(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 rsqrt2(float2 x) { return make_float2(fast_rsqrt(x.x), fast_rsqrt(x.y)); }

// Two body-body terms; (nrx, nry, nrz) is minus the target's position.
template <bool SOFT>
__device__ __forceinline__ void body_force2(float2 sx, float2 sy, float2 sz, float2 sm, float2 nrx,
                                            float2 nry, float2 nrz, float2 eps2, float2 &bx,
                                            float2 &by, float2 &bz) {
  const float2 dx = add2(sx, nrx), dy = add2(sy, nry), dz = add2(sz, nrz);
  float2 r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, eps2)));
  if (!SOFT) { r2.x = fmaxf(r2.x, r2_floor<float>()); r2.y = fmaxf(r2.y, r2_floor<float>()); }
  const float2 ri = rsqrt2(r2);
  const float2 f = mul2(mul2(sm, ri), mul2(ri, ri));
  bx = fma2(f, dx, bx); by = fma2(f, dy, by); bz = fma2(f, dz, bz);
}

// Two cell terms, the formula of cell_force; w[k] holds word k of both cells.
template <int ORDER>
__device__ __forceinline__ void cell_force2(const float2 *w, float2 nrx, float2 nry, float2 nrz,
                                            float2 eps2, float2 &bx, float2 &by, float2 &bz) {
  const float2 dx = add2(w[0], nrx), dy = add2(w[1], nry), dz = add2(w[2], nrz);
  const float2 r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, eps2)));
  const float2 rinv = rsqrt2(r2);
  const float2 r2i = mul2(rinv, rinv);
  const float2 r3i = mul2(rinv, r2i);
  if (ORDER < 4) {
    const float2 f = mul2(w[3], r3i);
    bx = fma2(f, dx, bx); by = fma2(f, dy, by); bz = fma2(f, dz, bz);
    return;
  }
  const float2 qx = fma2(w[4], dx, fma2(w[7], dy, mul2(w[8], dz)));
  const float2 qy = fma2(w[7], dx, fma2(w[5], dy, mul2(w[9], dz)));
  const float2 qz = fma2(w[8], dx, fma2(w[9], dy, mul2(w[6], dz)));
  const float2 dqd = fma2(dx, qx, fma2(dy, qy, mul2(dz, qz)));
  const float2 A = fma2(dqd, mul2(r2i, r2i), fma2(w[10], r2i, w[3]));
  const float2 sA = mul2(r3i, A);
  const float2 t = mul2(splat(-0.4f), mul2(r3i, r2i));
  if (ORDER < 8) {
    bx = fma2(sA, dx, fma2(t, qx, bx));
    by = fma2(sA, dy, fma2(t, qy, by));
    bz = fma2(sA, dz, fma2(t, qz, bz));
    return;
  }
  const float2 O1 = w[12], O2 = w[13], O3 = w[14], O4 = w[15], O5 = w[16], O6 = w[17], O7 = w[18],
               O8 = w[19], O9 = w[20], O10 = w[21], O12 = w[22], O13 = w[23], O14 = w[11];
  const float2 r4i = mul2(r2i, r2i);
  const float2 s7 = mul2(splat(7.5f), r4i);
  const float2 s5 = mul2(splat(-1.5f), r2i);
  const float2 s9 = mul2(mul2(splat(-17.5f), r4i), r2i);
  const float2 xx = mul2(dx, dx), yy = mul2(dy, dy), zz = mul2(dz, dz), xy = mul2(dx, dy),
               xz = mul2(dx, dz), yz = mul2(dy, dz);
  const float2 two = splat(2.0f), three = splat(3.0f);
  const float2 oc = mul2(s7, fma2(dx, O12, fma2(dy, O13, mul2(dz, O14))));
  float2 ox = fma2(s5, O12, mul2(dx, oc)), oy = fma2(s5, O13, mul2(dy, oc)),
         oz = fma2(s5, O14, mul2(dz, oc));
  ox = fma2(s7, fma2(two, fma2(xy, O4, fma2(xz, O7, mul2(yz, O10))),
                     fma2(xx, O1, fma2(yy, O2, mul2(zz, O3)))), ox);
  oy = fma2(s7, fma2(two, fma2(xy, O2, fma2(xz, O10, mul2(yz, O8))),
                     fma2(xx, O4, fma2(yy, O5, mul2(zz, O6)))), oy);
  oz = fma2(s7, fma2(two, fma2(xy, O10, fma2(xz, O3, mul2(yz, O6))),
                     fma2(xx, O7, fma2(yy, O8, mul2(zz, O9)))), oz);
  float2 c3 = fma2(mul2(xx, dx), O1, fma2(mul2(yy, dy), O5, mul2(mul2(zz, dz), O9)));
  c3 = fma2(three, fma2(mul2(xx, dy), O4, fma2(mul2(xx, dz), O7, mul2(mul2(xy, dy), O2))), c3);
  c3 = fma2(three, fma2(mul2(yy, dz), O8, fma2(mul2(xz, dz), O3, mul2(mul2(yz, dz), O6))), c3);
  c3 = fma2(mul2(splat(6.0f), xy), mul2(dz, O10), c3);
  c3 = mul2(s9, c3);
  ox = fma2(dx, c3, ox); oy = fma2(dy, c3, oy); oz = fma2(dz, c3, oz);
  bx = fma2(sA, dx, fma2(t, qx, fma2(r3i, ox, bx)));
  by = fma2(sA, dy, fma2(t, qy, fma2(r3i, oy, by)));
  bz = fma2(sA, dz, fma2(t, qz, fma2(r3i, oz, bz)));
}

// Accepted nodes of at most this many bodies are evaluated body by body
// (6 for the octupole: 12.4 instead of 13.2 ms at N = 2^20; for the
// quadrupole and the monopole no count pays).
template <int ORDER> __host__ __device__ constexpr int bodies_as_cell() { return ORDER >= 8 ? 6 : 1; }

// A staged entry that contributes exactly zero: no mass, no moments, far from
// every target (positions are in root-cube units, |x| <= ~1).
constexpr float kPadPos = 1.0e4f;

struct WalkCounters {
  unsigned long long pp = 0, pc = 0, tests = 0;
  int err = 0;
};

// The tree walk of one group (the box-distance MAC of octree_default.f90
// :1927-1936, optionally with every member's own MAC): accepted nodes are
// queued as cells and the bodies of opened leaves and lone particles as
// bodies; eval_cells(end, k) / eval_bodies(end, k) consume the k queue entries
// that end at position `end`, 32 at a time and the remainders at the end.
// Positions are relative to the group centre gc in units of the root side;
// S.member holds the group's targets (32 TPL slots, unused ones repeating the
// first target).  An accepted node of at most ASB bodies is queued as its
// bodies: for the octupole, whose cell term costs as much as about 8 body
// terms, that is cheaper and exact.
//
// Bound: latency; one pass over 32 nodes is a chain of dependent steps.  The
// members' MAC candidates share the warp (one at a time they took 4,000 of the
// 10,200 cycles of a pass at N = 1,024, where 14 of the 32 nodes are
// candidates; now 860), the stack's top kStackWindow entries stay in shared
// memory (older ones move to the global stack), one scan places both the
// children and the bodies of a pass, and the appends are predicated stores.
// EAGER walks (few groups, nothing else to hide the latency behind) load the
// next pass's records, every node's children among them, before handing this
// pass's batches on, and refuse most candidates by a look at kSamples members:
// about 3,500 cycles a pass.  With many groups the extra loads and tests only
// take issue slots from the consumers (2^20 bodies: 5.17 ms without, 5.29 with).
template <typename T, int TPL, int ASB, bool EAGER, typename CellsFn, typename BodiesFn>
__device__ __forceinline__ void tree_walk(const WalkArgs &a, WalkSmem<T> &S, int32_t *stack,
                                          int stack_cap, int gf, int gn, int root,
                                          const double gc[3], double inv_s, const T blo[3],
                                          const T bhi[3], T theta2, T inv_theta2, T diag, T rad,
                                          WalkCounters &wc, CellsFn &&eval_cells,
                                          BodiesFn &&eval_bodies) {
  const int lane = threadIdx.x & (kWarp - 1);
  const unsigned lt = (1u << lane) - 1u;
  // distance at which a node of level `lane` passes the MAC
  const T reach_of_level = sqrt(pow2_neg2<T>(min(lane, kMaxDepth)) * inv_theta2);
  // stack entries [low, top) are in the window, [0, low) in global memory
  int top = 1, low = 0, ncell = 0, nbody = 0;
  // a tree visits every node at most once per group: more tests than nodes
  // means a malformed tree, and the walk stops with an error instead of
  // looping
  const int max_tests = a.sc->n_compact + kWarp;
  int group_tests = 0;
  if (root < 0) top = 0;  // a lone body: no tree, no force
  if (lane == 0) S.window[0] = root;
  __syncwarp();
  // the nodes of the next pass (the top of the stack) and their records
  int take = 0, node = -1;
  int4 mt = make_int4(0, 0, 0, 0), c0 = mt, c1 = mt;
  double4 c = make_double4(0.0, 0.0, 0.0, 0.0);
  auto fetch = [&]() {
    take = min(top, kWarp);
    const int base = top - take;
    if (base < low) {  // older entries come back from the global stack
      const int from = max(0, low - kStackWindow / 2);
      for (int i = from + lane; i < low; i += kWarp) S.window[i & (kStackWindow - 1)] = stack[i];
      low = from;
      __syncwarp();
    }
    node = lane < take ? S.window[(base + lane) & (kStackWindow - 1)] : -1;
    top = base;
    if (node >= 0) {
      mt = a.meta[node];
      c = a.com[node];
      if (EAGER) {
        const int4 *cp = reinterpret_cast<const int4 *>(a.child + 8 * (int64_t)node);
        c0 = cp[0]; c1 = cp[1];
      }
    }
    __syncwarp();
  };
  fetch();
  while (take > 0) {
    if (group_tests > max_tests) { wc.err |= kErrIndex; break; }
    int cls = 0;  // 1 cell, 2 open leaf, 3 open internal
    T dx = (T)0, dy = (T)0, dz = (T)0, size2 = (T)0;
    bool cand = false;
    const T reach = __shfl_sync(kFull, reach_of_level, mt.z);
    if (node >= 0) {
      dx = (T)((c.x - gc[0]) * inv_s); dy = (T)((c.y - gc[1]) * inv_s); dz = (T)((c.z - gc[2]) * inv_s);
      const T ex = max(max(blo[0] - dx, (T)0), dx - bhi[0]);
      const T ey = max(max(blo[1] - dy, (T)0), dy - bhi[1]);
      const T ez = max(max(blo[2] - dz, (T)0), dz - bhi[2]);
      const T d2 = fma(ex, ex, fma(ey, ey, ez * ez));
      size2 = pow2_neg2<T>(mt.z);
      if (size2 <= theta2 * d2) {
        cls = 1;
      } else {
        cls = (mt.y <= a.leaf_cap || mt.w == 0) ? 2 : 3;
        if (a.mac == 1 && (mt.x + mt.y <= gf || mt.x >= gf + gn)) {
          // holds no member: accept when every member passes its own MAC.
          // Every member is at least |c| - rad from the centre of mass (the
          // sphere bound); otherwise the members are tested one by one below
          // if the nearest of them (at most `diag` beyond the box) may pass.
          const T dc = sqrt(fma(dx, dx, fma(dy, dy, dz * dz)));
          if (dc - rad >= reach) {
            cls = 1;
          } else {
            const T r2 = reach - diag;
            cand = r2 <= (T)0 || r2 * r2 <= d2;
          }
        }
      }
    }
    // members' own MAC (morton_octree.f90:701-706: size^2 <= theta^2 d^2 with
    // d from the member to the centre of mass).  Every lane first tests its own
    // node against a few members spread over the group, which refuses most;
    // the remaining candidates are gathered and share the warp: 2^sh lanes per
    // candidate, each over its part of the members (interleaved, so that the
    // reads of one step are adjacent), four at a time.
    if (EAGER && __any_sync(kFull, cand)) {
      T dmin = (T)INFINITY;
#pragma unroll
      for (int k = 0; k < kSamples; ++k) {
        const Vec4<T> q = S.member[k * (kWarp * TPL / kSamples)];
        const T ux = dx - q.x, uy = dy - q.y, uz = dz - q.z;
        dmin = min(dmin, fma(ux, ux, fma(uy, uy, uz * uz)));
      }
      cand = cand && size2 <= theta2 * dmin;
    }
    const unsigned pend = __ballot_sync(kFull, cand);
    if (pend) {
      const int nc = __popc(pend), rank = __popc(pend & lt);
      if (cand) S.cand[rank] = Vec4<T>{dx, dy, dz, size2};
      __syncwarp();
      const int sh = min(__clz(nc - 1) - 27, TPL == 2 ? 4 : 3);  // 5 - ceil(log2 nc)
      const int step = 1 << sh;
      const Vec4<T> t = S.cand[min(lane >> sh, nc - 1)];
      T dm[4] = {(T)INFINITY, (T)INFINITY, (T)INFINITY, (T)INFINITY};
      for (int i = lane & (step - 1); i < kWarp * TPL; i += 4 * step) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const Vec4<T> q = S.member[i + k * step];
          const T ux = t.x - q.x, uy = t.y - q.y, uz = t.z - q.z;
          dm[k] = min(dm[k], fma(ux, ux, fma(uy, uy, uz * uz)));
        }
      }
      T dmin = min(min(dm[0], dm[1]), min(dm[2], dm[3]));
      for (int o = step >> 1; o > 0; o >>= 1) dmin = min(dmin, __shfl_xor_sync(kFull, dmin, o));
      const unsigned pass = __ballot_sync(kFull, t.w <= theta2 * dmin);
      if (cand && ((pass >> (rank << sh)) & 1u)) cls = 1;
    }
    if (cls == 1 && mt.y <= ASB) cls = 2;
    group_tests += take;
    // cells
    const unsigned cm = __ballot_sync(kFull, cls == 1);
    store_if(&S.cellq[ncell + __popc(cm & lt)], node, cls == 1);
    ncell += __popc(cm);
    // children of opened internal nodes; bodies: lone-particle children (<= 8)
    // and leaf ranges, kBodyPerLane at a time.  A child entry is a node (>= 0),
    // a particle (< 0) or unused (kNoChild).
    if (!EAGER && cls == 3) {
      const int4 *cp = reinterpret_cast<const int4 *>(a.child + 8 * (int64_t)node);
      c0 = cp[0]; c1 = cp[1];
    }
    const int32_t ch[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const bool open = cls == 3;
    int nnc = 0, npc = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      nnc += (unsigned)ch[k] < (unsigned)kNoChild ? 1 : 0;
      npc += ch[k] < 0 ? 1 : 0;
    }
    int rf = mt.x, rn = cls == 2 ? mt.y : 0;
    int give = open ? npc : min(rn, kBodyPerLane);
    int both;
    const int off = warp_excl_scan((open ? nnc : 0) | (give << 16), lane, both);
    const int tot = both & 0xffff;
    int btot = both >> 16;
    int boff = nbody + (off >> 16);
    if (top + tot > stack_cap) {
      // capacity exceeded: the group's result is incomplete and flagged;
      // the host repeats the walk with a larger stack
      wc.err |= kErrStackOverflow;
    } else {
      if (top + tot - low > kStackWindow) {  // the oldest entries move out
        const int to = max(low, top - kStackWindow / 4);
        for (int i = low + lane; i < to; i += kWarp) stack[i] = S.window[i & (kStackWindow - 1)];
        low = to;
        __syncwarp();
      }
      if (tot > 0) {
        int k = top + (off & 0xffff);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const bool is = open && (unsigned)ch[q] < (unsigned)kNoChild;
          store_if(&S.window[k & (kStackWindow - 1)], ch[q], is);
          k += is ? 1 : 0;
        }
      }
      top += tot;
    }
    if (btot > 0) {
      int k = boff;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const bool is = open && ch[q] < 0;
        store_if(&S.bodyq[k], ~ch[q], is);
        k += is ? 1 : 0;
      }
    }
    __syncwarp();
    // the next pass's records load while this one's batches are handed on
    if (EAGER) fetch();
    if (btot > 0) {
      if (open) give = 0;
      for (;;) {
#pragma unroll
        for (int k = 0; k < kBodyPerLane / 2; ++k) store_if(&S.bodyq[boff + k], rf + k, k < give);
        if (__any_sync(kFull, give > kBodyPerLane / 2)) {
#pragma unroll
          for (int k = kBodyPerLane / 2; k < kBodyPerLane; ++k)
            store_if(&S.bodyq[boff + k], rf + k, k < give);
        }
        rf += give; rn -= give;
        nbody += btot;
        __syncwarp();
        while (nbody >= kWarp) { eval_bodies(nbody, kWarp); nbody -= kWarp; }
        if (__ballot_sync(kFull, rn > 0) == 0u) break;
        give = min(rn, kBodyPerLane);
        boff = nbody + warp_excl_scan(give, lane, btot);
      }
    }
    while (ncell >= kWarp) { eval_cells(ncell, kWarp); ncell -= kWarp; }
    __syncwarp();
    if (!EAGER) fetch();
  }
  wc.tests += group_tests;
  if (ncell > 0) eval_cells(ncell, ncell);
  if (nbody > 0) eval_bodies(nbody, nbody);
}

// A lane's TPL targets in the group frame, as the evaluation reads them: the
// FP32 walk wants them negated in both halves of a pair.
template <typename T, int TPL> struct Targets {
  T x[TPL], y[TPL], z[TPL];
  __device__ __forceinline__ void set(int t, T a, T b, T c) { x[t] = a; y[t] = b; z[t] = c; }
};
template <int TPL> struct Targets<float, TPL> {
  float2 x[TPL], y[TPL], z[TPL];
  __device__ __forceinline__ void set(int t, float a, float b, float c) {
    x[t] = splat(-a); y[t] = splat(-b); z[t] = splat(-c);
  }
};

// Staging of one batch, lane j entry j (j < n).  FP64: entry j at [W j, W (j + 1)).
// FP32: entries 2i and 2i + 1 interleaved word by word at [2W i, 2W (i + 1)), an odd
// count padded with an empty far entry.
template <typename T, int ORDER>
__device__ __forceinline__ void stage_cells(T *stage, int lane, int nc, int node, const WalkArgs &a,
                                            const double gc[3], double inv_s, double inv_m,
                                            double nq, double no) {
  constexpr int W = StageWords<ORDER>::value;
  if constexpr (sizeof(T) == 4) {
    float *w = stage + (lane >> 1) * 2 * W + (lane & 1);
    if (lane < nc) {
      stage_cell<float, ORDER, 2>(w, node, a, gc, inv_s, inv_m, nq, no);
    } else if (lane == nc && (nc & 1)) {
#pragma unroll
      for (int k = 3; k < W; ++k) w[2 * k] = 0.0f;
      w[0] = w[2] = w[4] = kPadPos;
    }
  } else {
    if (lane < nc) stage_cell<T, ORDER>(stage + lane * W, node, a, gc, inv_s, inv_m, nq, no);
  }
}
template <typename T>
__device__ __forceinline__ void stage_bodies(T *stage, int lane, int nb, int body, const WalkArgs &a,
                                             const double gc[3], double inv_s, double inv_m) {
  constexpr int STR = sizeof(T) == 4 ? 2 : 1;
  T *w = sizeof(T) == 4 ? stage + (lane >> 1) * 8 + (lane & 1) : stage + lane * 4;
  if (lane < nb) {
    const double4 s = a.spos[body];
    w[0] = (T)((s.x - gc[0]) * inv_s);
    w[STR] = (T)((s.y - gc[1]) * inv_s);
    w[2 * STR] = (T)((s.z - gc[2]) * inv_s);
    w[3 * STR] = (T)(s.w * inv_m);
  } else if (sizeof(T) == 4 && lane == nb && (nb & 1)) {
    w[0] = w[STR] = w[2 * STR] = (T)kPadPos;
    w[3 * STR] = (T)0;
  }
}

// The sum of one staged batch for every target of the lane.
template <typename T, int ORDER, int TPL>
__device__ __forceinline__ void sum_cells(const T *stage, int nc, const Targets<T, TPL> &g, T eps2,
                                          T (&sx)[TPL], T (&sy)[TPL], T (&sz)[TPL]) {
  constexpr int W = StageWords<ORDER>::value;
  if constexpr (sizeof(T) == 4) {
    const float2 eps2p = splat(eps2);
    float2 bx[TPL], by[TPL], bz[TPL];
#pragma unroll
    for (int t = 0; t < TPL; ++t) bx[t] = by[t] = bz[t] = make_float2(0.0f, 0.0f);
    const int np = (nc + 1) >> 1;
#pragma unroll 2
    for (int j = 0; j < np; ++j) {
      const float4 *st = reinterpret_cast<const float4 *>(stage) + j * (W / 2);
      float2 cw[W];
#pragma unroll
      for (int k = 0; k < W / 2; ++k) {
        const float4 v = st[k];
        cw[2 * k] = make_float2(v.x, v.y);
        cw[2 * k + 1] = make_float2(v.z, v.w);
      }
#pragma unroll
      for (int t = 0; t < TPL; ++t)
        cell_force2<ORDER>(cw, g.x[t], g.y[t], g.z[t], eps2p, bx[t], by[t], bz[t]);
    }
#pragma unroll
    for (int t = 0; t < TPL; ++t) {
      sx[t] = bx[t].x + bx[t].y; sy[t] = by[t].x + by[t].y; sz[t] = bz[t].x + bz[t].y;
    }
  } else {
#pragma unroll
    for (int t = 0; t < TPL; ++t) sx[t] = sy[t] = sz[t] = (T)0;
#pragma unroll 2
    for (int j = 0; j < nc; ++j) {
      T w[W];
      load_words<W>(stage + j * W, w);
#pragma unroll
      for (int t = 0; t < TPL; ++t)
        cell_force<T, ORDER>(w, g.x[t], g.y[t], g.z[t], eps2, sx[t], sy[t], sz[t]);
    }
  }
}
template <typename T, int TPL, bool SOFT>
__device__ __forceinline__ void sum_bodies(const T *stage, int nb, const Targets<T, TPL> &g, T eps2,
                                           T (&sx)[TPL], T (&sy)[TPL], T (&sz)[TPL]) {
  if constexpr (sizeof(T) == 4) {
    const float2 eps2p = splat(eps2);
    float2 bx[TPL], by[TPL], bz[TPL];
#pragma unroll
    for (int t = 0; t < TPL; ++t) bx[t] = by[t] = bz[t] = make_float2(0.0f, 0.0f);
    const int np = (nb + 1) >> 1;
    const float4 *st = reinterpret_cast<const float4 *>(stage);
    for (int j = 0; j < np; ++j) {
      const float4 u = st[2 * j], v = st[2 * j + 1];
      const float2 px = make_float2(u.x, u.y), py = make_float2(u.z, u.w);
      const float2 pz = make_float2(v.x, v.y), pm = make_float2(v.z, v.w);
#pragma unroll
      for (int t = 0; t < TPL; ++t)
        body_force2<SOFT>(px, py, pz, pm, g.x[t], g.y[t], g.z[t], eps2p, bx[t], by[t], bz[t]);
    }
#pragma unroll
    for (int t = 0; t < TPL; ++t) {
      sx[t] = bx[t].x + bx[t].y; sy[t] = by[t].x + by[t].y; sz[t] = bz[t].x + bz[t].y;
    }
  } else {
#pragma unroll
    for (int t = 0; t < TPL; ++t) sx[t] = sy[t] = sz[t] = (T)0;
#pragma unroll 2
    for (int j = 0; j < nb; ++j) {
      T w[4];
      load_words<4>(stage + j * 4, w);
#pragma unroll
      for (int t = 0; t < TPL; ++t)
        body_force<T, SOFT>(w[0], w[1], w[2], w[3], g.x[t], g.y[t], g.z[t], eps2, sx[t], sy[t], sz[t]);
    }
  }
}

// Running sums of a lane's targets: Kahan-compensated in FP32.
template <typename T, int TPL> struct Sums {
  static constexpr bool kKahan = sizeof(T) == 4;
  T ax[TPL], ay[TPL], az[TPL], cx[TPL], cy[TPL], cz[TPL];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int t = 0; t < TPL; ++t) ax[t] = ay[t] = az[t] = cx[t] = cy[t] = cz[t] = (T)0;
  }
  __device__ __forceinline__ void add(const T (&sx)[TPL], const T (&sy)[TPL], const T (&sz)[TPL]) {
#pragma unroll
    for (int t = 0; t < TPL; ++t) {
      if (kKahan) {
        kahan_add(ax[t], cx[t], sx[t]); kahan_add(ay[t], cy[t], sy[t]); kahan_add(az[t], cz[t], sz[t]);
      } else {
        ax[t] += sx[t]; ay[t] += sy[t]; az[t] += sz[t];
      }
    }
  }
  // forces in the original order; every system's result is an (n_s, 3)
  // Fortran-ordered block at 3 * off_s
  __device__ __forceinline__ void write(const WalkArgs &a, const SysScalars &ss, int gf, int gn,
                                        int lane) const {
    const double inv_s = 1.0 / ss.ssa;
    const double scale = a.G * ss.mass * inv_s * inv_s;
    double *out = a.out + 3 * ss.off;
    const int64_t ns = ss.n;
#pragma unroll
    for (int t = 0; t < TPL; ++t) {
      if (lane + kWarp * t >= gn) continue;
      const int i = gf + lane + kWarp * t;
      const int64_t p = a.perm[i] - ss.off;
      double fxs = (double)ax[t], fys = (double)ay[t], fzs = (double)az[t];
      if (kKahan) { fxs -= (double)cx[t]; fys -= (double)cy[t]; fzs -= (double)cz[t]; }
      double sc = scale;
      if (a.out_kind == 0) sc *= a.spos[i].w;
      out[p] = fxs * sc;
      out[ns + p] = fys * sc;
      out[2 * ns + p] = fzs * sc;
    }
  }
};

template <typename T>
__device__ __forceinline__ T group_eps2(const WalkArgs &a, double inv_s) {
  const double e2 = a.eps2 * inv_s * inv_s;
  return (T)(sizeof(T) == 8 ? fmin(e2, kEps2Max) : e2);
}

// The frame of one group (its <= 32 TPL bodies start at gf): centre gc and box
// of the members, which go to S.member, and the tree walk with the given
// consumers of the queues.
template <typename T, int ORDER, int TPL, bool EAGER, typename CellsFn, typename BodiesFn,
          typename BeginFn>
__device__ __forceinline__ void walk_members(const WalkArgs &a, WalkSmem<T> &S, int32_t *stack,
                                             int stack_cap, int gf, int gn, const SysScalars &ss,
                                             T theta2, double gc[3], WalkCounters &wc,
                                             BeginFn &&begin, CellsFn &&eval_cells,
                                             BodiesFn &&eval_bodies) {
  const int lane = threadIdx.x & (kWarp - 1);
  const double inv_s = 1.0 / ss.ssa;
  double px[TPL], py[TPL], pz[TPL];
#pragma unroll
  for (int t = 0; t < TPL; ++t) {
    const int k = lane + kWarp * t;
    const double4 p = a.spos[gf + (k < gn ? k : 0)];
    px[t] = p.x; py[t] = p.y; pz[t] = p.z;
  }
  double lo[3] = {px[0], py[0], pz[0]}, hi[3] = {px[0], py[0], pz[0]};
#pragma unroll
  for (int t = 1; t < TPL; ++t) {
    lo[0] = fmin(lo[0], px[t]); hi[0] = fmax(hi[0], px[t]);
    lo[1] = fmin(lo[1], py[t]); hi[1] = fmax(hi[1], py[t]);
    lo[2] = fmin(lo[2], pz[t]); hi[2] = fmax(hi[2], pz[t]);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) gc[k] = 0.5 * (warp_min(lo[k]) + warp_max(hi[k]));
  T rx[TPL], ry[TPL], rz[TPL], blo[3], bhi[3];
#pragma unroll
  for (int t = 0; t < TPL; ++t) {
    rx[t] = (T)((px[t] - gc[0]) * inv_s);
    ry[t] = (T)((py[t] - gc[1]) * inv_s);
    rz[t] = (T)((pz[t] - gc[2]) * inv_s);
    S.member[lane + kWarp * t] = Vec4<T>{rx[t], ry[t], rz[t], (T)0};
    if (t == 0) { blo[0] = bhi[0] = rx[0]; blo[1] = bhi[1] = ry[0]; blo[2] = bhi[2] = rz[0]; }
    else {
      blo[0] = min(blo[0], rx[t]); bhi[0] = max(bhi[0], rx[t]);
      blo[1] = min(blo[1], ry[t]); bhi[1] = max(bhi[1], ry[t]);
      blo[2] = min(blo[2], rz[t]); bhi[2] = max(bhi[2], rz[t]);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) { blo[k] = warp_min(blo[k]); bhi[k] = warp_max(bhi[k]); }
  // every member lies within `diag` of every point of the box
  const T diag = sqrt((bhi[0] - blo[0]) * (bhi[0] - blo[0]) + (bhi[1] - blo[1]) * (bhi[1] - blo[1]) +
                      (bhi[2] - blo[2]) * (bhi[2] - blo[2]));
  const T inv_theta2 = theta2 > (T)0 ? (T)1 / theta2 : (T)INFINITY;
  // radius of the members' sphere about the group centre
  T rad2 = (T)0;
#pragma unroll
  for (int t = 0; t < TPL; ++t) rad2 = max(rad2, fma(rx[t], rx[t], fma(ry[t], ry[t], rz[t] * rz[t])));
  const T rad = sqrt(warp_max(rad2));
  begin(rx, ry, rz);
  tree_walk<T, TPL, bodies_as_cell<ORDER>(), EAGER>(a, S, stack, stack_cap, gf, gn, ss.root, gc, inv_s,
                                             blo, bhi, theta2, inv_theta2, diag, rad, wc,
                                             eval_cells, eval_bodies);
}

// One group on one warp: TPL targets per lane.
template <typename T, int ORDER, int TPL, bool SOFT>
__device__ __forceinline__ void walk_group(const WalkArgs &a, WarpSmem<T, ORDER> &S,
                                           int32_t *stack, int stack_cap, int gf, int gn,
                                           const SysScalars &ss, T theta2, WalkCounters &wc) {
  const int lane = threadIdx.x & (kWarp - 1);
  const double inv_s = 1.0 / ss.ssa, inv_m = 1.0 / ss.mass;
  const double nq = inv_m * inv_s * inv_s, no = nq * inv_s;
  const T eps2 = group_eps2<T>(a, inv_s);
  double gc[3];
  Targets<T, TPL> tg;
  Sums<T, TPL> acc;
  acc.clear();
  walk_members<T, ORDER, TPL, false>(
      a, S.w, stack, stack_cap, gf, gn, ss, theta2, gc, wc,
      [&](const T (&rx)[TPL], const T (&ry)[TPL], const T (&rz)[TPL]) {
#pragma unroll
        for (int t = 0; t < TPL; ++t) tg.set(t, rx[t], ry[t], rz[t]);
      },
      [&](int end, int nc) {
        stage_cells<T, ORDER>(S.stage, lane, nc, lane < nc ? S.w.cellq[end - nc + lane] : 0, a, gc,
                              inv_s, inv_m, nq, no);
        __syncwarp();
        T sx[TPL], sy[TPL], sz[TPL];
        sum_cells<T, ORDER, TPL>(S.stage, nc, tg, eps2, sx, sy, sz);
        acc.add(sx, sy, sz);
        wc.pc += (unsigned long long)nc * gn;
        __syncwarp();
      },
      [&](int end, int nb) {
        stage_bodies<T>(S.stage, lane, nb, lane < nb ? S.w.bodyq[end - nb + lane] : 0, a, gc, inv_s,
                        inv_m);
        __syncwarp();
        T sx[TPL], sy[TPL], sz[TPL];
        sum_bodies<T, TPL, SOFT>(S.stage, nb, tg, eps2, sx, sy, sz);
        acc.add(sx, sy, sz);
        wc.pp += (unsigned long long)nb * gn;
        __syncwarp();
      });
  acc.write(a, ss, gf, gn, lane);
}

// Persistent warps, one per block, take groups from a global cursor until
// none is left; block b uses stack slot b.  With 64-body groups a group of
// <= 32 bodies runs the one-target-per-lane path.
template <typename T, int ORDER, int MAXTPL, bool SOFT>
__global__ void __launch_bounds__(kWarp, walk_min_blocks<T, ORDER>())
group_walk_kernel(WalkArgs a) {
  __shared__ WarpSmem<T, ORDER> S;
  pdl_enter();
  const int lane = threadIdx.x;
  int32_t *stack = a.stack + (int64_t)blockIdx.x * a.stack_cap;
  const int stack_cap = (int)a.stack_cap;
  const int ngroups = a.g_end >= 0 ? min(a.g_end, a.sc->n_groups) : a.sc->n_groups;
  const T theta2 = (T)a.theta2;
  WalkCounters wc;
  for (;;) {
    int g = 0;
    if (lane == 0) g = a.g_begin + atomicAdd(a.cursor, 1);
    g = __shfl_sync(kFull, g, 0);
    if (g >= ngroups) break;
    const int gf = a.g_first[g];
    const int gn = a.g_first[g + 1] - gf;
    const SysScalars &ss = a.ss[a.sys_of[gf]];
    if (MAXTPL == 2 && gn > kWarp)
      walk_group<T, ORDER, 2, SOFT>(a, S, stack, stack_cap, gf, gn, ss, theta2, wc);
    else
      walk_group<T, ORDER, 1, SOFT>(a, S, stack, stack_cap, gf, gn, ss, theta2, wc);
  }
  if (wc.err && lane == 0) atomicOr(&a.sc->err, wc.err);
  if (a.count_stats && lane == 0) {
    atomicAdd(&a.stats[0], wc.pp);
    atomicAdd(&a.stats[1], wc.pc);
    atomicAdd(&a.stats[3], wc.tests);
  }
}

// ---- warp-specialised group walk (pipeline = 1) ----
//
// A block is one producer warp and CONS consumer warps.  The producer
// takes groups from the global cursor, walks the tree exactly as the one-warp
// walk does and hands every batch of 32 cells or bodies on as a list of ids in
// a ring of shared-memory slots.  Batch i belongs to consumer
// i mod CONS, which loads and stages the entries itself (so no load of
// theirs delays the walk), sums the batch for the group's targets and then, in
// batch order, adds its sums to the running (Kahan) sums that the consumers
// hand on to each other through shared memory.  Every target sees the batches
// of the one-warp walk in the same order with the same arithmetic, so the
// results are the same bit for bit; the tree walk of one group overlaps the
// evaluation of the previous one, and a group's batches overlap one another.
// Each slot has a "full" mbarrier (the producer's arrival), an "empty" one (its
// consumer's, once the ids are read) and a "turn" one (the arrival of the
// consumer of the batch before it, once its sums are added).  Every wait is
// bounded: a wait that lasts more than about 2 s, or sees the block's abort
// flag, gives up, sets the flag and reports an error; every warp of the block
// then leaves its loop.
// 7 consumers a block: N = 1,024 81 -> 30 us, 4,096 196 -> 79 us, 16,384 371 ->
// 157 us against one team (below) per group; the FP64 walk at 65,536 bodies
// (3 consumers, 4 blocks per SM) 2.37 -> 1.16 ms against one warp per group
// evaluating its own batches.  choose_walk has the sizes where each wins.

constexpr long long kWaitCycles = 4000000000LL;
constexpr int kRingStart = 1, kRingCells = 2, kRingBodies = 3, kRingEnd = 4, kRingQuit = 5;

struct __align__(16) WideSlot {
  int kind, count, g, first;  // first: nothing of the group was added before
  double gc[3];
  double unused;
  int id[kWarp];
};

template <typename T, int ORDER, int CONS>
struct __align__(16) WideSmem {
  static constexpr int kSlots = 2 * CONS;  // of the ring
  unsigned long long full[kSlots], empty[kSlots], turn[kSlots];
  int abort_flag;
  WalkSmem<T> walk;
  WideSlot ring[kSlots];
  T sums[6][2 * kWarp];  // running sums of the group whose turn it is
  T stage[CONS][kWarp * StageWords<ORDER>::value];
};

__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long *b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned long long *b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// The whole warp waits for the phase of parity `parity` of barrier b to
// complete; false when the block was aborted or the wait lasted more than
// `limit` cycles (which aborts the block).
__device__ __forceinline__ bool mbar_wait_warp(unsigned long long *b, unsigned parity,
                                               volatile int *abort_flag,
                                               long long limit = kWaitCycles) {
  if (__all_sync(kFull, mbar_test(b, parity))) return true;
  const long long t0 = clock64();
  for (;;) {
    if (__all_sync(kFull, mbar_test(b, parity))) return true;
    int stop = 0;
    if ((threadIdx.x & (kWarp - 1)) == 0) {
      if (*abort_flag) stop = 1;
      else if (clock64() - t0 > limit) { *abort_flag = 1; stop = 1; }
    }
    if (__shfl_sync(kFull, stop, 0)) return false;
  }
}

// Producer side of one group: the walk of walk_group, with every batch's ids
// put into the ring.  `alive` turns false (for the rest of the kernel) when a
// wait gave up.
template <typename T, int ORDER, int TPL, int CONS>
__device__ __forceinline__ void wide_produce(const WalkArgs &a, WideSmem<T, ORDER, CONS> &P, unsigned &it,
                                              bool &alive, volatile int *abort_flag,
                                              int32_t *stack, int stack_cap, int g, int gf,
                                              int gn, const SysScalars &ss, T theta2,
                                              WalkCounters &wc) {
  constexpr unsigned kSlots = WideSmem<T, ORDER, CONS>::kSlots;
  const int lane = threadIdx.x & (kWarp - 1);
  double gc[3];
  int first = 1;
  auto emit = [&](int kind, int count, const int *ids) {
    const unsigned slot = it % kSlots, round = it / kSlots;
    if (alive && round > 0 && !mbar_wait_warp(&P.empty[slot], (round - 1) & 1u, abort_flag))
      alive = false;
    if (!alive) return;
    WideSlot &R = P.ring[slot];
    if (lane < count) R.id[lane] = ids[lane];
    if (lane == 0) {
      R.kind = kind; R.count = count; R.g = g; R.first = first;
      R.gc[0] = gc[0]; R.gc[1] = gc[1]; R.gc[2] = gc[2];
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&P.full[slot]);
    ++it;
    first = 0;
  };
  walk_members<T, ORDER, TPL, true>(
      a, P.walk, stack, stack_cap, gf, gn, ss, theta2, gc, wc,
      [](const T (&)[TPL], const T (&)[TPL], const T (&)[TPL]) {},
      [&](int end, int nc) {
        emit(kRingCells, nc, P.walk.cellq + end - nc);
        wc.pc += (unsigned long long)nc * gn;
      },
      [&](int end, int nb) {
        emit(kRingBodies, nb, P.walk.bodyq + end - nb);
        wc.pp += (unsigned long long)nb * gn;
      });
  emit(kRingEnd, 0, P.walk.cellq);
}

// One slot of a group on its consumer: the batch's sums, then the turn.
// False when a wait gave up.
template <typename T, int ORDER, int TPL, bool SOFT, int CONS>
__device__ __forceinline__ bool consume_slot(const WalkArgs &a, WideSmem<T, ORDER, CONS> &P, T *stage,
                                             unsigned it, volatile int *abort_flag, int kind,
                                             int count, int first, int id, int gf, int gn,
                                             const double gc[3], const SysScalars &ss,
                                             const Targets<T, TPL> &tg, double inv_s, T eps2) {
  constexpr unsigned kSlots = WideSmem<T, ORDER, CONS>::kSlots;
  const int lane = threadIdx.x & (kWarp - 1);
  T sx[TPL], sy[TPL], sz[TPL];
  if (kind == kRingCells) {
    const double inv_m = 1.0 / ss.mass, nq = inv_m * inv_s * inv_s, no = nq * inv_s;
    stage_cells<T, ORDER>(stage, lane, count, id, a, gc, inv_s, inv_m, nq, no);
    __syncwarp();
    sum_cells<T, ORDER, TPL>(stage, count, tg, eps2, sx, sy, sz);
  } else if (kind == kRingBodies) {
    const double inv_m = 1.0 / ss.mass;
    stage_bodies<T>(stage, lane, count, id, a, gc, inv_s, inv_m);
    __syncwarp();
    sum_bodies<T, TPL, SOFT>(stage, count, tg, eps2, sx, sy, sz);
  }
  const unsigned slot = it % kSlots, round = it / kSlots;
  if (!mbar_wait_warp(&P.turn[slot], round & 1u, abort_flag)) return false;
  Sums<T, TPL> acc;
  if (first) acc.clear();
  else {
#pragma unroll
    for (int t = 0; t < TPL; ++t) {
      const int k = lane + kWarp * t;
      acc.ax[t] = P.sums[0][k]; acc.ay[t] = P.sums[1][k]; acc.az[t] = P.sums[2][k];
      if (acc.kKahan) { acc.cx[t] = P.sums[3][k]; acc.cy[t] = P.sums[4][k]; acc.cz[t] = P.sums[5][k]; }
    }
  }
  if (kind != kRingEnd) {
    acc.add(sx, sy, sz);
#pragma unroll
    for (int t = 0; t < TPL; ++t) {
      const int k = lane + kWarp * t;
      P.sums[0][k] = acc.ax[t]; P.sums[1][k] = acc.ay[t]; P.sums[2][k] = acc.az[t];
      if (acc.kKahan) { P.sums[3][k] = acc.cx[t]; P.sums[4][k] = acc.cy[t]; P.sums[5][k] = acc.cz[t]; }
    }
  }
  __syncwarp();
  if (lane == 0) mbar_arrive(&P.turn[(it + 1) % kSlots]);
  if (kind == kRingEnd) acc.write(a, ss, gf, gn, lane);
  return true;
}

template <int CONS> constexpr int wide_threads() { return (1 + CONS) * kWarp; }
// resident blocks per SM the kernel is compiled for: 16 warps of 128 registers
template <int CONS> constexpr int wide_blocks() { return 16 / (1 + CONS); }

template <typename T, int ORDER, int MAXTPL, bool SOFT, int CONS>
__global__ void __launch_bounds__(wide_threads<CONS>(), wide_blocks<CONS>())
wide_walk_kernel(WalkArgs a) {
  extern __shared__ __align__(16) unsigned char wide_smem_raw[];
  constexpr unsigned kSlots = WideSmem<T, ORDER, CONS>::kSlots;
  pdl_enter();
  WideSmem<T, ORDER, CONS> &P = *reinterpret_cast<WideSmem<T, ORDER, CONS> *>(wide_smem_raw);
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x & (kWarp - 1);
  if (threadIdx.x == 0) {
    for (unsigned r = 0; r < kSlots; ++r) {
      mbar_init(&P.full[r], 1);
      mbar_init(&P.empty[r], 1);
      mbar_init(&P.turn[r], 1);
    }
    P.abort_flag = 0;
    mbar_arrive(&P.turn[0]);  // the first batch has nobody before it
  }
  __syncthreads();
  volatile int *abort_flag = &P.abort_flag;
  if (warp == 0) {
    const int ngroups = a.g_end >= 0 ? min(a.g_end, a.sc->n_groups) : a.sc->n_groups;
    int32_t *stack = a.stack + (int64_t)blockIdx.x * a.stack_cap;
    const int stack_cap = (int)a.stack_cap;
    const T theta2 = (T)a.theta2;
    WalkCounters wc;
    bool alive = true;
    unsigned it = 0;
    for (;;) {
      int g = 0;
      if (lane == 0) g = a.g_begin + atomicAdd(a.cursor, 1);
      g = __shfl_sync(kFull, g, 0);
      if (g >= ngroups) break;
      const int gf = a.g_first[g];
      const int gn = a.g_first[g + 1] - gf;
      const SysScalars &ss = a.ss[a.sys_of[gf]];
      if (MAXTPL == 2 && gn > kWarp)
        wide_produce<T, ORDER, 2, CONS>(a, P, it, alive, abort_flag, stack, stack_cap, g, gf, gn, ss,
                                   theta2, wc);
      else
        wide_produce<T, ORDER, 1, CONS>(a, P, it, alive, abort_flag, stack, stack_cap, g, gf, gn, ss,
                                   theta2, wc);
      if (!alive) break;
    }
    // tell every consumer there is nothing more
    for (int c = 0; alive && c < CONS; ++c, ++it) {
      const unsigned slot = it % kSlots, round = it / kSlots;
      if (round > 0 && !mbar_wait_warp(&P.empty[slot], (round - 1) & 1u, abort_flag)) {
        alive = false;
        break;
      }
      if (lane == 0) { P.ring[slot].kind = kRingQuit; mbar_arrive(&P.full[slot]); }
    }
    if (lane == 0) {
      if (wc.err) atomicOr(&a.sc->err, wc.err);
      if (!alive) atomicOr(&a.sc->err, kErrTimeout);
      if (a.count_stats) {
        atomicAdd(&a.stats[0], wc.pp);
        atomicAdd(&a.stats[1], wc.pc);
        atomicAdd(&a.stats[3], wc.tests);
      }
    }
  } else {
    T *stage = P.stage[warp - 1];
    int cur = -1, gf = 0, gn = 0;
    double gc[3] = {0.0, 0.0, 0.0}, inv_s = 0.0;
    T eps2 = (T)0;
    const SysScalars *ss = a.ss;
    Targets<T, MAXTPL> tg;
    bool ok = true;
    for (unsigned it = warp - 1;; it += CONS) {
      const unsigned slot = it % kSlots, round = it / kSlots;
      ok = mbar_wait_warp(&P.full[slot], round & 1u, abort_flag);
      if (!ok) break;
      const WideSlot &R = P.ring[slot];
      const int kind = R.kind, count = R.count, g = R.g, first = R.first, id = R.id[lane];
      if (kind == kRingQuit) break;
      if (g != cur) {  // the group's targets
        cur = g;
        gc[0] = R.gc[0]; gc[1] = R.gc[1]; gc[2] = R.gc[2];
        gf = a.g_first[g];
        gn = a.g_first[g + 1] - gf;
        ss = a.ss + a.sys_of[gf];
        inv_s = 1.0 / ss->ssa;
        eps2 = group_eps2<T>(a, inv_s);
#pragma unroll
        for (int t = 0; t < MAXTPL; ++t) {
          const int k = lane + kWarp * t;
          const double4 p = a.spos[gf + (k < gn ? k : 0)];
          tg.set(t, (T)((p.x - gc[0]) * inv_s), (T)((p.y - gc[1]) * inv_s),
                 (T)((p.z - gc[2]) * inv_s));
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&P.empty[slot]);
      if (MAXTPL == 2 && gn > kWarp) {
        ok = consume_slot<T, ORDER, MAXTPL, SOFT, CONS>(a, P, stage, it, abort_flag, kind, count, first,
                                                  id, gf, gn, gc, *ss, tg, inv_s, eps2);
      } else {
        Targets<T, 1> t1;
        t1.x[0] = tg.x[0]; t1.y[0] = tg.y[0]; t1.z[0] = tg.z[0];
        ok = consume_slot<T, ORDER, 1, SOFT, CONS>(a, P, stage, it, abort_flag, kind, count, first, id,
                                             gf, gn, gc, *ss, t1, inv_s, eps2);
      }
      if (!ok) break;
    }
    if (!ok && lane == 0) atomicOr(&a.sc->err, kErrTimeout);
  }
}

// ---- warp-specialised FP32 walk for many groups ----
//
// A block holds kTeams teams of one producer warp and one consumer warp.  The
// producer walks groups from the global cursor and stages every batch of 32
// cells or bodies into a ring of kRing shared-memory slots; its consumer sums
// the batches and writes the forces: the batches, order and arithmetic of the
// one-warp walk, so the same bits.  The consumers (warpgroup 0) take registers
// over from the producers (warpgroup 1) with setmaxnreg.
// Bound: the FP32 FMA pipe (66 % busy at 524,288 bodies; the evaluation loop alone
// reaches 84 % with 2-5 warps per scheduler, and the producers' instructions
// take the difference).  2^20 Hernquist bodies 5.20 -> 5.17 ms, 5,000,011 in a
// uniform sphere 7.00 -> 6.76 ms with the walk's gathered candidates and
// shared-memory stack; consumers as the lower warpgroup took 1.3 % off.  Tried
// and slower at 2^20: two batches at once, one per half-warp with four targets a
// lane (2 blocks per SM: 7.1 ms), the consumers staging (7.0-9.0 ms), eight lanes
// per opened node instead of the scan (5.47 ms), branches instead of the
// predicated appends (5.45 ms).

constexpr int kTeams = 4;
constexpr int kRing = 4;

template <int ORDER>
struct __align__(16) TeamSlot {
  int kind, count, g, unused;
  double gc[3];
  double unused2;
  float stage[kWarp * StageWords<ORDER>::value];
};

template <int ORDER>
struct __align__(16) TeamSmem {
  unsigned long long full[kTeams][kRing];
  unsigned long long empty[kTeams][kRing];
  int abort_flag;
  WalkSmem<float> walk[kTeams];
  TeamSlot<ORDER> ring[kTeams][kRing];
};

// Producer side of one group: the walk of walk_group, with every batch staged
// into the ring.  `alive` turns false (for the rest of the kernel) when a wait
// gave up.
template <int ORDER, int TPL>
__device__ __forceinline__ void team_produce(const WalkArgs &a, TeamSmem<ORDER> &P, int team,
                                             unsigned &it, bool &alive, volatile int *abort_flag,
                                             int32_t *stack, int stack_cap, int g, int gf, int gn,
                                             const SysScalars &ss, float theta2, WalkCounters &wc) {
  const double inv_s = 1.0 / ss.ssa, inv_m = 1.0 / ss.mass;
  const double nq = inv_m * inv_s * inv_s, no = nq * inv_s;
  const int lane = threadIdx.x & (kWarp - 1);
  double gc[3];
  // the next slot, once its consumer has released it
  auto acquire = [&]() -> TeamSlot<ORDER> & {
    const unsigned slot = it % kRing, round = it / kRing;
    if (alive && round > 0 && !mbar_wait_warp(&P.empty[team][slot], (round - 1) & 1u, abort_flag))
      alive = false;
    return P.ring[team][slot];
  };
  auto publish = [&]() {
    __syncwarp();
    if (lane == 0) mbar_arrive(&P.full[team][it % kRing]);
    ++it;
  };
  walk_members<float, ORDER, TPL, false>(
      a, P.walk[team], stack, stack_cap, gf, gn, ss, theta2, gc, wc,
      [&](const float (&)[TPL], const float (&)[TPL], const float (&)[TPL]) {
        TeamSlot<ORDER> &R = acquire();
        if (!alive) return;
        if (lane == 0) {
          R.kind = kRingStart; R.g = g; R.count = gn;
          R.gc[0] = gc[0]; R.gc[1] = gc[1]; R.gc[2] = gc[2];
        }
        publish();
      },
      [&](int end, int nc) {
        TeamSlot<ORDER> &R = acquire();
        if (!alive) return;
        stage_cells<float, ORDER>(R.stage, lane, nc,
                                  lane < nc ? P.walk[team].cellq[end - nc + lane] : 0, a, gc, inv_s,
                                  inv_m, nq, no);
        if (lane == 0) { R.kind = kRingCells; R.count = nc; }
        wc.pc += (unsigned long long)nc * gn;
        publish();
      },
      [&](int end, int nb) {
        TeamSlot<ORDER> &R = acquire();
        if (!alive) return;
        stage_bodies<float>(R.stage, lane, nb, lane < nb ? P.walk[team].bodyq[end - nb + lane] : 0,
                            a, gc, inv_s, inv_m);
        if (lane == 0) { R.kind = kRingBodies; R.count = nb; }
        wc.pp += (unsigned long long)nb * gn;
        publish();
      });
  TeamSlot<ORDER> &R = acquire();
  if (!alive) return;
  if (lane == 0) R.kind = kRingEnd;
  publish();
}

// Consumer side of one group (its start slot already read and released):
// sums the batches until the group's end slot, then writes the forces; false
// when a wait gave up.
template <int ORDER, int TPL, bool SOFT>
__device__ __forceinline__ bool team_consume(const WalkArgs &a, TeamSmem<ORDER> &P, int team,
                                             unsigned &it, volatile int *abort_flag, int gf, int gn,
                                             const double gc[3], const SysScalars &ss) {
  const int lane = threadIdx.x & (kWarp - 1);
  const double inv_s = 1.0 / ss.ssa;
  const float eps2 = group_eps2<float>(a, inv_s);
  Targets<float, TPL> tg;
#pragma unroll
  for (int t = 0; t < TPL; ++t) {
    const int k = lane + kWarp * t;
    const double4 p = a.spos[gf + (k < gn ? k : 0)];
    tg.set(t, (float)((p.x - gc[0]) * inv_s), (float)((p.y - gc[1]) * inv_s),
           (float)((p.z - gc[2]) * inv_s));
  }
  Sums<float, TPL> acc;
  acc.clear();
  for (;;) {
    const unsigned slot = it % kRing, round = it / kRing;
    if (!mbar_wait_warp(&P.full[team][slot], round & 1u, abort_flag)) return false;
    const TeamSlot<ORDER> &R = P.ring[team][slot];
    const int kind = R.kind, count = R.count;
    float sx[TPL], sy[TPL], sz[TPL];
    if (kind == kRingCells) {
      sum_cells<float, ORDER, TPL>(R.stage, count, tg, eps2, sx, sy, sz);
      acc.add(sx, sy, sz);
    } else if (kind == kRingBodies) {
      sum_bodies<float, TPL, SOFT>(R.stage, count, tg, eps2, sx, sy, sz);
      acc.add(sx, sy, sz);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&P.empty[team][slot]);
    ++it;
    if (kind == kRingEnd) break;
  }
  acc.write(a, ss, gf, gn, lane);
  return true;
}

// TeamRegs<ORDER>::blocks blocks of 2 kTeams warps per SM.  At launch every
// thread holds `regs` registers (the most that `blocks` blocks allow); the
// producer warpgroup then gives registers up to the consumer warpgroup:
// producer + consumer = 2 regs, so the consumers' request is always covered by
// the block's own registers (the host checks the launch count first).
constexpr int kTeamThreads = 2 * kTeams * kWarp;
static_assert(kTeams == 4, "one warpgroup of producers, one of consumers");
template <int ORDER> struct TeamRegs {
  static constexpr int blocks = ORDER >= 8 ? 2 : 3;
  static constexpr int regs = ORDER >= 8 ? 128 : 80;
  static constexpr int producer = ORDER >= 8 ? 96 : 64;
  static constexpr int consumer = 2 * regs - producer;
  static_assert(regs * kTeamThreads * blocks <= 65536, "register file");
  static_assert(regs % 8 == 0 && producer % 8 == 0 && consumer <= 256, "setmaxnreg counts");
};

template <int ORDER, int MAXTPL, bool SOFT>
__global__ void __launch_bounds__(kTeamThreads, TeamRegs<ORDER>::blocks)
team_walk_kernel(WalkArgs a) {
  extern __shared__ __align__(16) unsigned char team_smem_raw[];
  TeamSmem<ORDER> &P = *reinterpret_cast<TeamSmem<ORDER> *>(team_smem_raw);
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x & (kWarp - 1);
  if (threadIdx.x == 0) {
    for (int q = 0; q < kTeams; ++q)
      for (int r = 0; r < kRing; ++r) {
        mbar_init(&P.full[q][r], 1);
        mbar_init(&P.empty[q][r], 1);
      }
    P.abort_flag = 0;
  }
  __syncthreads();
  volatile int *abort_flag = &P.abort_flag;
  unsigned it = 0;
  if (warp >= kTeams) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(TeamRegs<ORDER>::producer));
    const int ngroups = a.g_end >= 0 ? min(a.g_end, a.sc->n_groups) : a.sc->n_groups;
    const int team = warp - kTeams;
    int32_t *stack = a.stack + ((int64_t)blockIdx.x * kTeams + team) * a.stack_cap;
    const int stack_cap = (int)a.stack_cap;
    const float theta2 = (float)a.theta2;
    WalkCounters wc;
    bool alive = true;
    for (;;) {
      int g = 0;
      if (lane == 0) g = a.g_begin + atomicAdd(a.cursor, 1);
      g = __shfl_sync(kFull, g, 0);
      if (g >= ngroups) break;
      const int gf = a.g_first[g];
      const int gn = a.g_first[g + 1] - gf;
      const SysScalars &ss = a.ss[a.sys_of[gf]];
      if (MAXTPL == 2 && gn > kWarp)
        team_produce<ORDER, 2>(a, P, team, it, alive, abort_flag, stack, stack_cap, g, gf, gn, ss,
                               theta2, wc);
      else
        team_produce<ORDER, 1>(a, P, team, it, alive, abort_flag, stack, stack_cap, g, gf, gn, ss,
                               theta2, wc);
      if (!alive) break;
    }
    if (alive) {  // tell the consumer there is nothing more
      const unsigned slot = it % kRing, round = it / kRing;
      if (round == 0 || mbar_wait_warp(&P.empty[team][slot], (round - 1) & 1u, abort_flag)) {
        if (lane == 0) { P.ring[team][slot].kind = kRingQuit; mbar_arrive(&P.full[team][slot]); }
      } else {
        alive = false;
      }
    }
    if (lane == 0) {
      if (wc.err) atomicOr(&a.sc->err, wc.err);
      if (!alive) atomicOr(&a.sc->err, kErrTimeout);
      if (a.count_stats) {
        atomicAdd(&a.stats[0], wc.pp);
        atomicAdd(&a.stats[1], wc.pc);
        atomicAdd(&a.stats[3], wc.tests);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(TeamRegs<ORDER>::consumer));
    const int team = warp;
    bool ok;
    for (;;) {
      ok = mbar_wait_warp(&P.full[team][it % kRing], (it / kRing) & 1u, abort_flag);
      if (!ok) break;
      const TeamSlot<ORDER> &R = P.ring[team][it % kRing];
      const int kind = R.kind, g = R.g, gn = R.count;
      const double gc[3] = {R.gc[0], R.gc[1], R.gc[2]};
      if (kind != kRingStart) break;  // the producer has no more groups
      __syncwarp();
      if (lane == 0) mbar_arrive(&P.empty[team][it % kRing]);
      ++it;
      const int gf = a.g_first[g];
      const SysScalars &ss = a.ss[a.sys_of[gf]];
      if (MAXTPL == 2 && gn > kWarp)
        ok = team_consume<ORDER, 2, SOFT>(a, P, team, it, abort_flag, gf, gn, gc, ss);
      else
        ok = team_consume<ORDER, 1, SOFT>(a, P, team, it, abort_flag, gf, gn, gc, ss);
      if (!ok) break;
    }
    if (!ok && lane == 0) atomicOr(&a.sc->err, kErrTimeout);
  }
}

// Check of the bounded waits above on one block of two warps.  Warp 0 arrives
// at barrier 2 (a phase that completes), waits until warp 1 has seen it
// complete, then waits on barrier 0, at which nothing ever arrives, for
// `limit` cycles.  Warp 1 waits on barrier 2, acknowledges on barrier 1, then
// waits on barrier 0 with the walk's full limit: it must be released by the
// abort flag that warp 0 sets when it gives up.  out: [0] warp 0's result on
// barrier 0, [1] warp 1's result on barrier 2, [2] warp 1's result on barrier
// 0, [3] the cycles warp 1 waited there, [4] the abort flag at the end.
__global__ void __launch_bounds__(2 * kWarp) wait_probe_kernel(long long limit, long long *out) {
  __shared__ __align__(8) unsigned long long bar[3];
  __shared__ int abort_flag;
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x & (kWarp - 1);
  if (threadIdx.x == 0) {
    for (int k = 0; k < 3; ++k) mbar_init(&bar[k], kWarp);
    abort_flag = 0;
  }
  __syncthreads();
  volatile int *af = &abort_flag;
  if (warp == 0) {
    mbar_arrive(&bar[2]);
    const bool acked = mbar_wait_warp(&bar[1], 0, af, limit);
    const bool ok = acked && mbar_wait_warp(&bar[0], 0, af, limit);
    if (lane == 0) out[0] = ok ? 1 : 0;
  } else {
    const bool seen = mbar_wait_warp(&bar[2], 0, af, limit);
    if (lane == 0) out[1] = seen ? 1 : 0;
    mbar_arrive(&bar[1]);
    const long long t0 = clock64();
    const bool ok = mbar_wait_warp(&bar[0], 0, af);
    const long long dt = clock64() - t0;
    if (lane == 0) { out[2] = ok ? 1 : 0; out[3] = dt; }
  }
  __syncthreads();
  if (threadIdx.x == 0) out[4] = abort_flag;
}

// ---- reference-semantics walk (FP64, one thread per target) ----

__device__ __forceinline__ void ref_pp(double bx, double by, double bz, double bm, double qp0,
                                       double qp1, double qp2, double mp, double G, double eps2,
                                       double &fx, double &fy, double &fz) {
  // morton_octree.f90:676-686
  const double dx = bx - qp0, dy = by - qp1, dz = bz - qp2;
  const double dist2 = dx * dx + dy * dy + dz * dz + eps2;
  double inv = 1.0 / sqrt(dist2);
  inv = inv * inv * inv;
  const double f = G * mp * bm * inv;
  fx = fx + f * dx; fy = fy + f * dy; fz = fz + f * dz;
}

template <int ORDER>
__global__ void __launch_bounds__(128)
reference_walk_kernel(WalkArgs a, const int64_t *__restrict__ targets, int64_t nt,
                      const int32_t *__restrict__ inv_perm, int64_t *__restrict__ counts) {
  const int L = a.sc->L;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nt;
       k += (int64_t)gridDim.x * blockDim.x) {
    if (targets && (targets[k] < 0 || targets[k] >= a.n)) {
      a.out[k] = a.out[nt + k] = a.out[2 * nt + k] = nan("");
      if (counts) counts[2 * k] = counts[2 * k + 1] = -1;
      continue;
    }
    const int p = targets ? inv_perm[targets[k]] : (int)k;
    const SysScalars &ss = a.ss[a.sys_of[p]];
    const double ssa = ss.ssa;
    const double4 q = a.spos[p];
    const double qp0 = q.x, qp1 = q.y, qp2 = q.z, mp = q.w;
    double fx = 0.0, fy = 0.0, fz = 0.0;
    int64_t npp = 0, npc = 0;
    // stack entries: node j >= 0; lone particle b as ~b (monopole at m q / m);
    // level-L lone particle b as ~b - 2^30 (summed at its exact position)
    int32_t st[8 * (kMaxDepth + 2) + 8];
    int top = 0;
    if (ss.root >= 0) st[top++] = ss.root;
    const int64_t max_pops = (int64_t)a.sc->n_compact + a.n + 8;
    int64_t pops = 0;
    while (top > 0) {
      if (++pops > max_pops) { atomicOr(&a.sc->err, kErrIndex); break; }
      const int32_t e = st[--top];
      if (e < 0) {
        const bool exact = e < -(1 << 30);
        const int b = exact ? ~(e + (1 << 30)) : ~e;
        if (b == p) continue;
        const double4 s = a.spos[b];
        if (exact) {
          ref_pp(s.x, s.y, s.z, s.w, qp0, qp1, qp2, mp, a.G, a.eps2, fx, fy, fz);
        } else {
          // single-particle node: qcm = (m q) / m (morton_octree.f90:446-458)
          const double cx = (s.w * s.x) / s.w, cy = (s.w * s.y) / s.w, cz = (s.w * s.z) / s.w;
          if (s.w > 0) ref_pp(cx, cy, cz, s.w, qp0, qp1, qp2, mp, a.G, a.eps2, fx, fy, fz);
        }
        ++npp;
        continue;
      }
      const int4 mt = a.meta[e];
      if (mt.w == 0) {  // level-L leaf: particle by particle (:672-691)
        for (int b = mt.x; b < mt.x + mt.y; ++b) {
          if (b == p) continue;
          const double4 s = a.spos[b];
          ref_pp(s.x, s.y, s.z, s.w, qp0, qp1, qp2, mp, a.G, a.eps2, fx, fy, fz);
          ++npp;
        }
        continue;
      }
      bool open = (mt.x <= p && p < mt.x + mt.y);  // :694-697
      if (!open) {
        const double4 c = a.com[e];
        const double dx = c.x - qp0, dy = c.y - qp1, dz = c.z - qp2;
        double dist2 = dx * dx + dy * dy + dz * dz;
        const double size = ssa * ldexp(1.0, -mt.z);
        if (size * size <= a.theta2 * dist2) {  // :706
          if (c.w > 0) {
            dist2 = dist2 + a.eps2;
            if (ORDER < 4) {
              double inv = 1.0 / sqrt(dist2);
              inv = inv * inv * inv;
              const double f = a.G * mp * c.w * inv;
              fx = fx + f * dx; fy = fy + f * dy; fz = fz + f * dz;
            } else {  // :721-753
              const double *Q = a.quad + 6 * (int64_t)e;
              const double invR = 1.0 / sqrt(dist2);
              const double invR2 = 1.0 / dist2;
              const double invR3 = invR * invR2;
              const double invR5 = invR3 * invR * invR;
              const double mx = dx * invR3 * c.w, my = dy * invR3 * c.w, mz = dz * invR3 * c.w;
              const double dx2 = 15.0 * dx * dx * invR2 - 3.0;
              const double dy2 = 15.0 * dy * dy * invR2 - 3.0;
              const double dz2 = 15.0 * dz * dz * invR2 - 3.0;
              const double dxyz = 15.0 * dx * dy * dz * invR2;
              double Qx = (Q[0] * (dx2 - 6.0) + Q[1] * dy2 + Q[2] * dz2) * 0.5 * dx;
              double Qy = (Q[1] * (dy2 - 6.0) + Q[2] * dz2 + Q[0] * dx2) * 0.5 * dy;
              double Qz = (Q[2] * (dz2 - 6.0) + Q[0] * dx2 + Q[1] * dy2) * 0.5 * dz;
              Qx = Qx + Q[3] * dy * dx2 + Q[4] * dz * dx2 + Q[5] * dxyz;
              Qy = Qy + Q[5] * dz * dy2 + Q[3] * dx * dy2 + Q[4] * dxyz;
              Qz = Qz + Q[4] * dx * dz2 + Q[5] * dy * dz2 + Q[3] * dxyz;
              if (ORDER < 8) {
                fx = fx + a.G * mp * (mx + invR5 * Qx);
                fy = fy + a.G * mp * (my + invR5 * Qy);
                fz = fz + a.G * mp * (mz + invR5 * Qz);
              } else {  // octupole terms of octree_default.f90:1012-1063
                const double *o = a.oct + 14 * (int64_t)e;
                const double invR7 = invR5 * invR * invR;
                const double invR9 = invR7 * invR * invR;
                double Ox = -1.5 * invR5 * o[11], Oy = -1.5 * invR5 * o[12], Oz = -1.5 * invR5 * o[13];
                double Oc = 7.5 * invR7 * (dx * o[11] + dy * o[12] + dz * o[13]);
                Ox = Ox + dx * Oc; Oy = Oy + dy * Oc; Oz = Oz + dz * Oc;
                const double ddx = dx * dx, ddy = dy * dy, ddz = dz * dz;
                Ox = Ox + 7.5 * invR7 * (ddx * o[0] + ddy * o[1] + ddz * o[2] + 2.0 * dx * dy * o[3] +
                                         2.0 * dx * dz * o[6] + 2.0 * dy * dz * o[9]);
                Oy = Oy + 7.5 * invR7 * (ddx * o[3] + ddy * o[4] + ddz * o[5] + 2.0 * dx * dy * o[1] +
                                         2.0 * dx * dz * o[9] + 2.0 * dy * dz * o[7]);
                Oz = Oz + 7.5 * invR7 * (ddx * o[6] + ddy * o[7] + ddz * o[8] + 2.0 * dx * dy * o[9] +
                                         2.0 * dx * dz * o[2] + 2.0 * dy * dz * o[5]);
                Oc = -17.5 * invR9 *
                     (ddx * dx * o[0] + ddy * dy * o[4] + ddz * dz * o[8] + 3.0 * ddx * dy * o[3] +
                      3.0 * ddx * dz * o[6] + 3.0 * ddy * dx * o[1] + 3.0 * ddy * dz * o[7] +
                      3.0 * ddz * dx * o[2] + 3.0 * ddz * dy * o[5] + 6.0 * dx * dy * dz * o[9]);
                Ox = Ox + dx * Oc; Oy = Oy + dy * Oc; Oz = Oz + dz * Oc;
                fx = fx + a.G * mp * (mx + invR5 * Qx + Ox);
                fy = fy + a.G * mp * (my + invR5 * Qy + Oy);
                fz = fz + a.G * mp * (mz + invR5 * Qz + Oz);
              }
            }
          }
          ++npc;
          continue;
        }
      }
      // open: push children in reverse so they pop in key order
      const bool deepest = (mt.z + 1 == L);
      for (int c = mt.w - 1; c >= 0; --c) {
        const int32_t ch = a.child[8 * (int64_t)e + c];
        if (top >= (int)(sizeof(st) / sizeof(st[0]))) break;
        st[top++] = (ch < 0 && deepest) ? ch - (1 << 30) : ch;
      }
    }
    double sc = 1.0;
    if (a.out_kind == 1) sc = 1.0 / mp;
    if (targets) {
      a.out[k] = fx * sc; a.out[nt + k] = fy * sc; a.out[2 * nt + k] = fz * sc;
    } else {
      double *out = a.out + 3 * ss.off;
      const int64_t orig = a.perm[p] - ss.off, ns = ss.n;
      out[orig] = fx * sc; out[ns + orig] = fy * sc; out[2 * ns + orig] = fz * sc;
    }
    if (counts) { counts[2 * k] = npp; counts[2 * k + 1] = npc; }
  }
}

int g_sm_count[64] = {0};

int sm_count() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (g_sm_count[dev] == 0) {
    int c = 0;
    cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
    g_sm_count[dev] = c > 0 ? c : 148;
  }
  return g_sm_count[dev];
}

}  // namespace

// stack slots: one per resident walk block of the FP32 walk (the most of any
// instantiation)
int64_t walk_slots() { return (int64_t)sm_count() * kWalkBlocksPerSm; }

int probe_bounded_wait(long long cycles, long long *out5) {
  long long *d = nullptr;
  if (cudaMalloc(&d, 5 * sizeof(long long)) != cudaSuccess) return 1;
  int rc = 0;
  if (cudaMemset(d, 0xff, 5 * sizeof(long long)) != cudaSuccess) rc = 1;
  if (!rc) {
    wait_probe_kernel<<<1, 2 * kWarp>>>(cycles, d);
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) rc = 1;
  }
  if (!rc && cudaMemcpy(out5, d, 5 * sizeof(long long), cudaMemcpyDeviceToHost) != cudaSuccess)
    rc = 1;
  cudaFree(d);
  return rc;
}

// exactly the blocks that are resident at once: no block waits for a second
// wave behind the walk (which would also hold back other streams); occupancy
// and the shared-memory limit are properties of the device, so they are kept
// per device.  regs > 0: the kernel's setmaxnreg split assumes that launch
// count; a block launched with fewer would wait for ever, so a kernel compiled
// otherwise is never launched (-1).
template <typename K>
static int resident_blocks(int (&per_sm)[64], K *kernel, int threads, size_t smem, int regs = 0) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (per_sm[dev] == 0) {
    int v = 0;
    if (smem)
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kernel, threads, smem);
    cudaFuncAttributes fa{};
    cudaFuncGetAttributes(&fa, kernel);
    per_sm[dev] = regs > 0 && (fa.numRegs != regs || v < 1) ? -1 : (v > 0 ? v : 1);
  }
  return per_sm[dev];
}

template <int ORDER, int MAXTPL, bool SOFT>
static bool launch_team_walk(const WalkArgs &a, cudaStream_t s) {
  static int per_sm[64] = {};
  const size_t smem = sizeof(TeamSmem<ORDER>);
  const int per = resident_blocks(per_sm, team_walk_kernel<ORDER, MAXTPL, SOFT>, kTeamThreads, smem,
                                  TeamRegs<ORDER>::regs);
  if (per < 0 || a.slots < kTeams) return false;
  const int64_t blocks = bh_min64(a.slots / kTeams, (int64_t)sm_count() * per);  // a stack per producer
  team_walk_kernel<ORDER, MAXTPL, SOFT><<<(unsigned)blocks, kTeamThreads, smem, s>>>(a);
  return true;
}

template <typename T, int ORDER, int MAXTPL, bool SOFT, int CONS>
static void launch_wide_walk(const WalkArgs &a, cudaStream_t s) {
  static int per_sm[64] = {};
  const size_t smem = sizeof(WideSmem<T, ORDER, CONS>);
  const int per = resident_blocks(per_sm, wide_walk_kernel<T, ORDER, MAXTPL, SOFT, CONS>,
                                  wide_threads<CONS>(), smem);
  const int64_t blocks = bh_min64(a.slots, (int64_t)sm_count() * per);  // one stack per block
  launch_pdl(wide_walk_kernel<T, ORDER, MAXTPL, SOFT, CONS>, blocks, wide_threads<CONS>(), smem, s, a);
}

// Which walk a launch takes (pipeline 1).  Few groups leave most of the chip idle,
// so the more warps share a group the better; with more groups than a kernel has
// producers (296 with 7 consumers a block, 592 with 3, 1,776 in teams, 2,368 one-warp
// walks) the shared ones fall behind.  Where the lines lie depends on how long a
// group's walk is: the walk of a small system is a pass or two, over before its
// consumers gain anything.  So the choice goes by the number of groups, each
// weighed by the length of its walk against the longest (about the square root of
// the system's bodies, launch time taken off), and by the size of the largest system.
// Walk times in us, 7 consumers / 3 consumers / teams / one warp a group (theta 0.5,
// Plummer; g: ceil(n_s / group size) summed over the systems):
//  FP32 quadrupole, one system    16,384 (g 256): 157 / 182 / 359 / -
//                  20,480 (320): 196 / 204 / 404 / -   65,536 (1,024): 582 / 459 / 510 / -
//                  100,003 (1,563): 876 / 654 / 549 / -
//     monopole 20,480: 182 / 162 / 268   65,536: 526 / 354 / 326   octupole 32,768:
//     450 / 497 / 635   65,536: 942 / 975 / 810
//  FP32, groups of 32   6,000 (g 188): 88 / 100 / 153   20,000 (625): 247 / 173 / 240
//                       40,000 (1,250): 481 / 317 / 285   65,000 (2,032): 810 / 506 / 385
//     octupole 6,000: 104 / 126 / 200   20,000: 296 / 220 / 333   40,000: 599 / 465 / 500
//              65,000: 1,023 / 753 / 754
//  FP32, batches   4,000 systems of 10: 68 / 43 / 28 / 25   600 of 64: 35 / 28 / 27 / 29
//     75 of 100 (g 150): 25 / 26 / 31 / 32   300 of 100 (600): 39 / 32 / 32 / 35
//     37 of 500 (296): 55 / 43 / 63 / 73   75 of 500 (600): 90 / 71 / 64 / 75
//     37 of 1,000 (592): 114 / 90 / 100 / -   62 of 1,000 (992): 178 / 140 / 103 / -
//     15 of 4,000 (945): 276 / 217 / 244 / -   31 of 4,000 (1,953): 512 / 404 / 333 / -
//     octupole, 75 of 100: 25 / 27 / 28   300 of 100: 41 / 33 / 28
//  FP64 quadrupole, batches   300 of 10: 23 / 21 / - / 21   2,000 of 30: 62 / 43 / - / 28
//     75 of 100: 27 / 29 / - / 41   500 of 100 (g 1,000): 58 / 43 / - / 48
//     1,000 of 100 (2,000): 92 / 66 / - / 50   250 of 200 (1,000): 111 / 87 / - / 71
//     1,000 of 200 (4,000): 400 / 330 / - / 158   62 of 1,000 (992): 235 / 196 / - / 238
//     125 of 1,000 (2,000): 426 / 365 / - / 268   31 of 4,000 (1,953): 675 / 620 / - / 644
//     63 of 4,000 (3,969): 1,301 / 1,169 / - / 1,035
//  FP64, one system (theta 0.4 and 0.6, Hernquist and uniform sphere, 3 consumers over
//     one warp a group, means of the four): quadrupole 131,072 0.85, 230,000 0.95,
//     300,000 0.97, 350,000 1.03, 524,288 1.06; monopole 131,072 0.94, 196,608 1.16;
//     octupole (7 consumers) 131,072 0.88, 196,608 1.04.
//  Ranges of a 2^20-body system's groups, FP32 quadrupole   200: 251 / 311 / 653
//     800: 489 / 387 / 666; FP64 quadrupole of 2^19   2,000: 1,473 / 1,408 / - / 1,766
//     4,000: 2,761 / 2,572 / - / 2,744
enum class Walk { kOneWarp, kTeams, kWide3, kWide7 };
constexpr int64_t kLongWalks = 2048;  // bodies from which a system's walks are long

template <typename T, int ORDER, int MAXTPL>
static Walk choose_walk(const WalkArgs &a) {
  if (!a.pipeline) return Walk::kOneWarp;
  double g = a.walk_groups;
  if (a.g_end >= 0) g = fmin(g, (double)(a.g_end - a.g_begin));
  const double root = sqrt((double)a.largest);
  const bool lone = a.largest >= kLongWalks;
  double seven = 200.0, three;  // the most weighed groups of each
  if constexpr (sizeof(T) == 8) {
    const double most = ORDER >= 8 ? 2900.0 : (ORDER >= 4 ? 5000.0 : 2400.0);
    three = a.largest <= kWarp ? 400.0 : fmin(fmax(40.0 * root, 800.0), most);
    if (lone) seven = ORDER >= 8 ? three : 384.0;
  } else if constexpr (ORDER >= 8) {
    three = lone ? (MAXTPL == 2 ? 768.0 : 1400.0) : 400.0;
    if (lone) seven = MAXTPL == 2 ? 768.0 : 400.0;
  } else {
    three = fmin(fmax(20.0 * root, 512.0), 1024.0);
    if (lone) seven = 320.0;
  }
  if (g <= seven) return Walk::kWide7;
  if (g <= three) return Walk::kWide3;
  return sizeof(T) == 4 ? Walk::kTeams : Walk::kOneWarp;
}

template <typename T, int ORDER, int MAXTPL, bool SOFT>
static void launch_group_walk(const WalkArgs &a, cudaStream_t s) {
  Walk kind = choose_walk<T, ORDER, MAXTPL>(a);
  if constexpr (sizeof(T) == 4) {
    if (kind == Walk::kTeams) {
      if (launch_team_walk<ORDER, MAXTPL, SOFT>(a, s)) return;
      kind = Walk::kWide3;
    }
  }
  if (kind == Walk::kWide7) return launch_wide_walk<T, ORDER, MAXTPL, SOFT, 7>(a, s);
  if (kind == Walk::kWide3) return launch_wide_walk<T, ORDER, MAXTPL, SOFT, 3>(a, s);
  static int per_sm[64] = {};
  const int per = resident_blocks(per_sm, group_walk_kernel<T, ORDER, MAXTPL, SOFT>, kWarp, 0);
  const int64_t blocks = bh_min64(a.slots, (int64_t)sm_count() * per);  // one stack per block
  launch_pdl(group_walk_kernel<T, ORDER, MAXTPL, SOFT>, blocks, kWarp, 0, s, a);
}

static WalkArgs make_args(int64_t n, const WalkParams &p, Buffers &b, double *out) {
  WalkArgs a;
  a.meta = b.cn_meta; a.child = b.cn_child; a.com = b.cn_com; a.quad = b.cn_quad; a.oct = b.cn_oct;
  a.fq = b.cn_fq; a.fo = b.cn_fo; a.spos = b.spos; a.perm = b.v0; a.g_first = b.g_first;
  a.sys_of = b.sys_of; a.ss = b.ss;
  a.sc = b.sc; a.cursor = b.counters; a.stack = b.wstack; a.stack_cap = b.wstack_cap;
  a.slots = b.wstack_slots;
  a.stats = b.stats; a.out = out; a.n = n;
  a.theta2 = p.theta2; a.G = p.G; a.eps2 = p.eps2;
  a.out_kind = p.out_kind; a.leaf_cap = p.leaf_cap; a.count_stats = p.count_stats;
  a.mac = p.mac;
  a.g_begin = p.g_begin; a.g_end = p.g_end;
  a.pipeline = p.pipeline;
  a.largest = b.largest;
  a.walk_groups = b.walk_groups[p.group_size > 32 ? 1 : 0];
  return a;
}

template <typename T, int ORDER>
static void launch_walk_t(const WalkArgs &a, bool two, bool soft, cudaStream_t s) {
  if (two) {
    if (soft) launch_group_walk<T, ORDER, 2, true>(a, s);
    else launch_group_walk<T, ORDER, 2, false>(a, s);
  } else {
    if (soft) launch_group_walk<T, ORDER, 1, true>(a, s);
    else launch_group_walk<T, ORDER, 1, false>(a, s);
  }
}

void launch_walk(int64_t n, const WalkParams &p, Buffers &b, double *out, cudaStream_t s) {
  WalkArgs a = make_args(n, p, b, out);
  if (!p.after_build) cudaMemsetAsync(b.counters, 0, sizeof(int32_t), s);
  const bool two = p.group_size > 32;
  const bool soft = p.eps2 > 0.0;
  if (p.precision == BH_PREC_FP64) {
    if (p.order >= 8) launch_walk_t<double, 8>(a, two, soft, s);
    else if (p.order >= 4) launch_walk_t<double, 4>(a, two, soft, s);
    else launch_walk_t<double, 1>(a, two, soft, s);
  } else {
    if (p.order >= 8) launch_walk_t<float, 8>(a, two, soft, s);
    else if (p.order >= 4) launch_walk_t<float, 4>(a, two, soft, s);
    else launch_walk_t<float, 1>(a, two, soft, s);
  }
}

__global__ void inv_perm_kernel(const int32_t *__restrict__ perm, int64_t n, int32_t *__restrict__ inv) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    inv[perm[i]] = (int32_t)i;
}

void launch_reference_walk(int64_t n, const WalkParams &p, Buffers &b, double *out,
                           const int64_t *targets, int64_t ntargets, int64_t *counts,
                           cudaStream_t s) {
  WalkArgs a = make_args(n, p, b, out);
  int32_t *inv = nullptr;
  if (targets) {
    inv = b.gscan;  // free after the group pass
    inv_perm_kernel<<<grid_for(n, 256, 148 * 8), 256, 0, s>>>(b.v0, n, inv);
  }
  const int64_t nt = targets ? ntargets : n;
  const int grid = grid_for(nt, 128, 148 * 32);
  if (p.order >= 8)
    reference_walk_kernel<8><<<grid, 128, 0, s>>>(a, targets, nt, inv, counts);
  else if (p.order >= 4)
    reference_walk_kernel<4><<<grid, 128, 0, s>>>(a, targets, nt, inv, counts);
  else
    reference_walk_kernel<1><<<grid, 128, 0, s>>>(a, targets, nt, inv, counts);
}

}  // namespace bh
