// FP64 direct summation (the error oracle of every result) and the FMA
// throughput probe used as the roofline denominator of the walk.
//
// The pair force is that of fortran/direct_forces.f90:24-26 and
// fortran/api3d.f90:54-59: f = G m_a m_b / (dist * dist2), dist2 = |d|^2 + eps^2.
//
// Bound: the FP64 pipe, 16 operations a pair (3 differences, 3 for dist2, 7
// for m / dist^3 -- mass_over_r3 -- and 3 sums).  A CTA takes 64 targets; the
// sources are cut into kDirSplits slices, one per CTA of a cluster, and inside
// a CTA into kDirSubs groups of 64 threads, so that 2,048 targets already put
// warps on every SM.  The partial sums meet in a fixed order (groups, then
// slices through distributed shared memory) that depends on n alone.
// 16,384 bodies: 0.32 ms (13.5 T FP64 operations/s of the 18.3 T that the FMA
// probe reaches) against 3.00 ms with a square root and a division a pair and
// one block per 256 targets walking all sources (64 blocks for 148 SMs); 1,024
// bodies 11 us.  Also measured at 16,384: 2 groups 0.326 ms, 1 group 0.351,
// 8 groups 0.348; two targets a thread with 1, 2, 4 groups 0.356, 0.336,
// 0.329; four targets a thread 0.35: one target and 4 groups is the best or
// within 1.5 % of it from 2,048 to 40,000 bodies.
#include <cooperative_groups.h>
#include <math.h>

#include "bh_fp64.cuh"
#include "bh_internal.cuh"

namespace cg = cooperative_groups;

namespace bh {

namespace {

constexpr int kDirSplits = 8;  // CTAs of a cluster (the portable limit), one source slice each
constexpr int kDirLanes = 64;  // threads of a group, one target each
constexpr int kDirSubs = 4;    // groups of a CTA
constexpr int kDirThreads = kDirLanes * kDirSubs;
static_assert(kDirLanes == 2 * kWarp, "two warps of targets");

// SELF: the target may be among the sources of this tile
template <bool SELF>
__device__ __forceinline__ void direct_tile(const double4 *tile, int cnt, int64_t src, int64_t a,
                                            double xa, double ya, double za, double eps2,
                                            double &fx, double &fy, double &fz) {
#pragma unroll 4
  for (int j = 0; j < cnt; ++j) {
    const double4 s = tile[j];
    const double dx = s.x - xa, dy = s.y - ya, dz = s.z - za;
    double r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
    if (SELF && src + j == a) r2 = 1.0;  // d = 0: the term is exactly 0
    const double w = mass_over_r3(r2, s.w);
    fx = fma(w, dx, fx); fy = fma(w, dy, fy); fz = fma(w, dz, fz);
  }
}

// Component q of target `lane`: the partial sums of the groups, slice by slice.
__device__ __forceinline__ double cluster_sum(const cg::cluster_group &cluster, double *part, int q,
                                              int lane) {
  double f = 0.0;
  for (int r = 0; r < kDirSplits; ++r) {
    const double *p = cluster.map_shared_rank(part, r);
    for (int g = 0; g < kDirSubs; ++g) f += p[(g * 3 + q) * kDirLanes + lane];
  }
  return f;
}

// What a thread of the cluster works on: target a (entry k of the output) and the
// sources [s0, s1).
struct DirSlot {
  int64_t k, a, s0, s1;
  bool bad;  // invalid target index: NaN result
};
__device__ __forceinline__ DirSlot direct_slot(int rank, int64_t n, const int64_t *targets, int64_t nt) {
  DirSlot d;
  d.k = (int64_t)(blockIdx.x / kDirSplits) * kDirLanes + threadIdx.x % kDirLanes;
  d.a = d.k < nt ? (targets ? targets[d.k] : d.k) : 0;
  d.bad = d.a < 0 || d.a >= n;
  if (d.bad) d.a = 0;
  d.s0 = n * rank / kDirSplits;
  d.s1 = n * (rank + 1) / kDirSplits;
  return d;
}

// Sums that did not come out finite, made again with the reference's own
// operations by the whole cluster: coincident unsoftened bodies, non-finite inputs
// and squared distances beyond the range of mass_over_r3 give what these operations
// give.  `redo` has the targets of the thread's warp.  Not inlined and not unrolled:
// with this sum in its body the kernel took 66 registers, which leaves 3 blocks per
// SM (16,384 bodies 0.354 ms), or spills at 64 (0.322).  One NaN among 16,384 bodies, so that every sum
// is made again: 1.0 ms, against 17.8 by the first warps of one CTA; a coincident pair
// 0.34 against 4.4.
__device__ __noinline__ void direct_again(const double *__restrict__ m, const double *__restrict__ x,
                                          const double *__restrict__ y,
                                          const double *__restrict__ z, int64_t n,
                                          const int64_t *__restrict__ targets, int64_t nt, double G,
                                          double eps2, int out_kind, double *__restrict__ out,
                                          double4 *tile, double *part, unsigned redo) {
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int sub = threadIdx.x / kDirLanes, lane = threadIdx.x % kDirLanes;
  const DirSlot d = direct_slot(rank, n, targets, nt);
  const double gm = G * (out_kind == 1 ? 1.0 : m[d.a]);
  const double xa = x[d.a], ya = y[d.a], za = z[d.a];
  double fx = 0.0, fy = 0.0, fz = 0.0;
  for (int64_t src = d.s0; src < d.s1; src += kDirThreads) {
    const int64_t j = src + threadIdx.x;
    __syncthreads();
    if (j < d.s1) tile[threadIdx.x] = make_double4(x[j], y[j], z[j], m[j]);
    __syncthreads();
    const int64_t first = src + sub * kDirLanes;  // this group's part of the tile
    const int cnt = (int)(redo && first < d.s1 ? bh_min64(kDirLanes, d.s1 - first) : 0);
#pragma unroll 1
    for (int i = 0; i < cnt; ++i) {
      if (first + i == d.a) continue;
      const double4 s = tile[sub * kDirLanes + i];
      const double dx = s.x - xa, dy = s.y - ya, dz = s.z - za;
      const double dist2 = dx * dx + dy * dy + dz * dz + eps2;
      const double dist = sqrt(dist2);
      const double w = gm * s.w / (dist * dist2);
      fx = fx + w * dx; fy = fy + w * dy; fz = fz + w * dz;
    }
  }
  part[(sub * 3 + 0) * kDirLanes + lane] = fx;
  part[(sub * 3 + 1) * kDirLanes + lane] = fy;
  part[(sub * 3 + 2) * kDirLanes + lane] = fz;
  cluster.sync();
  if (rank == 0 && sub == 0 && (redo >> (lane % kWarp) & 1u))
    for (int q = 0; q < 3; ++q) out[q * nt + d.k] = cluster_sum(cluster, part, q, lane);
  cluster.sync();
}

__global__ void __launch_bounds__(kDirThreads)
direct_kernel(const double *__restrict__ m, const double *__restrict__ x,
              const double *__restrict__ y, const double *__restrict__ z, int64_t n,
              const int64_t *__restrict__ targets, int64_t nt, double G, double eps2,
              int out_kind, double *__restrict__ out) {
  __shared__ double4 tile[kDirThreads];
  __shared__ double part[kDirSubs][3][kDirLanes];
  __shared__ unsigned again[kDirLanes / kWarp];  // targets whose sum is not finite
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int sub = threadIdx.x / kDirLanes, lane = threadIdx.x % kDirLanes;
  const DirSlot d = direct_slot(rank, n, targets, nt);
  if (threadIdx.x < kDirLanes / kWarp) again[threadIdx.x] = 0;
  const int64_t a = d.a, s0 = d.s0, s1 = d.s1;
  const double xa = x[a], ya = y[a], za = z[a];
  double fx = 0.0, fy = 0.0, fz = 0.0;
  for (int64_t src = s0; src < s1; src += kDirThreads) {
    const int64_t j = src + threadIdx.x;
    __syncthreads();
    if (j < s1) tile[threadIdx.x] = make_double4(x[j], y[j], z[j], m[j]);
    __syncthreads();
    const int64_t first = src + sub * kDirLanes;  // this group's part of the tile
    const int cnt = (int)(first < s1 ? bh_min64(kDirLanes, s1 - first) : 0);
    const double4 *mine = tile + sub * kDirLanes;
    if (__any_sync(0xffffffffu, a >= first && a < first + cnt))
      direct_tile<true>(mine, cnt, first, a, xa, ya, za, eps2, fx, fy, fz);
    else
      direct_tile<false>(mine, cnt, first, a, xa, ya, za, eps2, fx, fy, fz);
  }
  part[sub][0][lane] = fx; part[sub][1][lane] = fy; part[sub][2][lane] = fz;
  cluster.sync();
  if (rank == 0 && sub == 0) {
    const double gm = G * (out_kind == 1 ? 1.0 : m[d.a]);
    double f[3];
    for (int q = 0; q < 3; ++q) f[q] = gm * cluster_sum(cluster, &part[0][0][0], q, lane);
    const bool finite = isfinite(f[0]) && isfinite(f[1]) && isfinite(f[2]);
    const unsigned redo = __ballot_sync(0xffffffffu, d.k < nt && !d.bad && !finite);
    if (redo && lane % kWarp < kDirSplits)  // every CTA of the cluster gets the word
      cluster.map_shared_rank(again, lane % kWarp)[lane / kWarp] = redo;
    if (d.bad) f[0] = f[1] = f[2] = nan("");
    if (d.k < nt)
      for (int q = 0; q < 3; ++q) out[q * nt + d.k] = f[q];
  }
  cluster.sync();  // the words are set, and rank 0 has read the other CTAs' shared memory
  if ((again[0] | again[1]) != 0)  // the same words in every CTA
    direct_again(m, x, y, z, n, targets, nt, G, eps2, out_kind, out, tile, &part[0][0][0],
                 again[lane / kWarp]);
}

constexpr int kProbeIters = 4096;

template <typename T>
__global__ void __launch_bounds__(256) fma_probe_kernel(T *sink, T a, T b) {
  T v0 = (T)threadIdx.x, v1 = v0 + 1, v2 = v0 + 2, v3 = v0 + 3, v4 = v0 + 4, v5 = v0 + 5,
    v6 = v0 + 6, v7 = v0 + 7;
#pragma unroll 16
  for (int i = 0; i < kProbeIters; ++i) {
    v0 = fma(v0, a, b); v1 = fma(v1, a, b); v2 = fma(v2, a, b); v3 = fma(v3, a, b);
    v4 = fma(v4, a, b); v5 = fma(v5, a, b); v6 = fma(v6, a, b); v7 = fma(v7, a, b);
  }
  T s = v0 + v1 + v2 + v3 + v4 + v5 + v6 + v7;
  if (s == (T)12345.678) sink[threadIdx.x] = s;  // keeps the chains alive
}

// The same chains with paired FP32 instructions (two FMAs per instruction).
__global__ void __launch_bounds__(256) fma2_probe_kernel(float *sink, float a, float b) {
  const float2 av = make_float2(a, a), bv = make_float2(b, b);
  const float f = (float)threadIdx.x;
  float2 v0 = make_float2(f, f + 1), v1 = make_float2(f + 2, f + 3), v2 = make_float2(f + 4, f + 5),
         v3 = make_float2(f + 6, f + 7);
#pragma unroll 16
  for (int i = 0; i < kProbeIters; ++i) {
    v0 = __ffma2_rn(v0, av, bv); v1 = __ffma2_rn(v1, av, bv);
    v2 = __ffma2_rn(v2, av, bv); v3 = __ffma2_rn(v3, av, bv);
  }
  const float s = v0.x + v0.y + v1.x + v1.y + v2.x + v2.y + v3.x + v3.y;
  if (s == 12345.678f) sink[threadIdx.x] = s;
}

}  // namespace

void launch_direct(const double *m, const double *x, const double *y, const double *z, int64_t n,
                   const int64_t *targets, int64_t ntargets, double G, double eps2, int out_kind,
                   double *out, cudaStream_t s) {
  const int64_t nt = targets ? ntargets : n;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((nt + kDirLanes - 1) / kDirLanes * kDirSplits));
  cfg.blockDim = dim3(kDirThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kDirSplits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, direct_kernel, m, x, y, z, n, targets, nt, G, eps2, out_kind, out);
}

// GFLOP/s of FMA (2 flops each) on independent chains: [0] FP32, [1] FP64,
// [2] FP32 issued as paired (f32x2) instructions.
int probe_fma(double *gflops2) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int blocks = sms * 8, threads = 256;
  float *fs = nullptr;
  double *ds = nullptr;
  if (cudaMalloc(&fs, threads * sizeof(float)) != cudaSuccess) return 1;
  if (cudaMalloc(&ds, threads * sizeof(double)) != cudaSuccess) { cudaFree(fs); return 1; }
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const double flops = 2.0 * 8.0 * kProbeIters * (double)blocks * threads;
  for (int which = 0; which < 3; ++which) {
    float best = 1e30f;
    for (int rep = 0; rep < 5; ++rep) {
      cudaEventRecord(e0);
      if (which == 0) fma_probe_kernel<float><<<blocks, threads>>>(fs, 0.999f, 1e-3f);
      else if (which == 1) fma_probe_kernel<double><<<blocks, threads>>>(ds, 0.999, 1e-3);
      else fma2_probe_kernel<<<blocks, threads>>>(fs, 0.999f, 1e-3f);
      cudaEventRecord(e1);
      cudaEventSynchronize(e1);
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (rep > 0 && ms < best) best = ms;
    }
    gflops2[which] = flops / (best * 1e-3) / 1e9;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(fs);
  cudaFree(ds);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

}  // namespace bh
