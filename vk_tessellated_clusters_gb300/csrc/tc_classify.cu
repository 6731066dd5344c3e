// tc_classify.cu — cluster_classify: per-triangle edge segment counts and the
// full / part / split classification of every visible cluster.
//
// shaders/cluster_classify.comp.glsl:150-666 (RT target, plain path), and with
// TC_FLAG_TRANSIENT_1X / _2X :254-905 (transient CLAS builds of untessellated
// triangles and of 2X batches) through a count variant and a write kernel of
// their own.
//
// GB300 mapping, three launches per stage, none with a cross-block wait. Block
// b of the write grid owns the contiguous range of visible clusters
// [b * per, (b + 1) * per):
//   count : warps stride over the whole list, one cluster at a time per warp
//           (<= 64 triangles, two per lane), vertices staged in shared
//           memory; segment counts, configs and the cluster's counts (part /
//           split triangles, full-cluster vertices, CLAS bytes) go to
//           scratch, and 64-bit atomics add them to the sums of the cluster's
//           range
//   write : every block adds up the sums of the ranges before its own (the
//           counters' values before the launch included), then scans its own
//           clusters' counts in shared memory, so every offset equals what a
//           serial loop over the clusters gives; part / split triangles and
//           instantiation arguments go to those offsets, and the grid's last
//           block writes the counters' new totals
//   full vertices : the displaced vertices of the accepted full clusters, from
//           the records write leaves (a launch of its own, beside later work)
#include <algorithm>

#include "tc_deform.cuh"
#include "tc_kernels.h"
#include "tc_stage.cuh"
#include "tc_vertex.cuh"
#include "tc_walk.cuh"

namespace tc {

namespace {

constexpr u32 kBlock = 256;  // threads of the count and write blocks
constexpr u32 kWarps = kBlock / 32;

enum : int
{
  kCntParts = 0,
  kCntSplits,
  kCntGen,
  kCntVerts,
  kCntData,
  kNumCounters
};

// per-cluster counts: x = parts | splits << 7 | full << 14 | fullVertices << 15 | fullTriangles << 22,
// y = CLAS bytes
__device__ __forceinline__ uint2 pack_counts(u32 parts, u32 splits, bool full, u32 nv, u32 nt, u32 data)
{
  return make_uint2(parts | (splits << 7) | ((full ? 1u : 0u) << 14) | ((full ? nv : 0u) << 15) | ((full ? nt : 0u) << 22),
                    full ? data : 0u);
}
__device__ __forceinline__ u32 cnt_parts(uint2 r) { return r.x & 0x7F; }
__device__ __forceinline__ u32 cnt_splits(uint2 r) { return (r.x >> 7) & 0x7F; }
__device__ __forceinline__ u32 cnt_full(uint2 r) { return (r.x >> 14) & 1; }
__device__ __forceinline__ u32 cnt_verts(uint2 r) { return (r.x >> 15) & 0x7F; }
__device__ __forceinline__ u32 cnt_tris(uint2 r) { return (r.x >> 22) & 0x7F; }

// tessellation.glsl:119-144 tess_getConfig, also reporting how the three
// sub-triangle corners were rotated (0: none, 1: .yzx, 2: .zxy)
__device__ __forceinline__ u32 get_config_rot(uint3 f, u32& rot)
{
  u32 m = max(max(f.x, f.y), f.z);
  rot   = 0;
  if(m == f.y)
  {
    f   = make_uint3(f.y, f.z, f.x);
    rot = 1;
  }
  else if(m == f.z)
  {
    f   = make_uint3(f.z, f.x, f.y);
    rot = 2;
  }
  const u32 L   = TC_TESSTABLE_LOOKUP_SIZE;
  u32       idx = f.x + f.y * L + f.z * L * L - (1 + L + L * L);
  if(f.z > f.y)
    idx |= 1u << 15;
  return idx;
}

// per-triangle word: config | rotation << 16 | split << 18
__device__ __forceinline__ u32 classify_triangle(uint3 f, u32 sf)
{
  const u32  m     = max(max(f.x, f.y), f.z);
  const bool split = m > TC_TESSTABLE_SIZE;
  if(split)
    f = make_uint3(split_factor1(f.x, sf), split_factor1(f.y, sf), split_factor1(f.z, sf));
  u32       rot;
  const u32 cfg = get_config_rot(f, rot);
  return cfg | (rot << 16) | ((split ? 1u : 0u) << 18);
}

struct ClassifyScratch
{
  uint2*          counts;     // per visible cluster of the window
  u32*            triWords;   // 64 per visible cluster
  RangeSums*      rangeSums;  // per write block's range: the counts' sums, zero before count
  ClusterOffsets* bases;      // the counters before the launch
  u32             writeBlocks;  // the write launch's grid (its blocks' ranges)
  u32             listed;       // k_classify_write leaves the clusters with parts to k_classify_emit
  uint2*          fullRecs;   // per full cluster (generated-cluster slot - first slot): visible index, first vertex
  u32*            fullRange;  // [2]: the launch's generated-cluster slots [begin, end); [2]: transRecs' count
  const uint4*    groups;     // instance groups, or null; with them fullRecs are per visible cluster
  const u32*      members;
  u32*            groupHead;
  const u32*      instBounds;  // per instance: its first entry of bounds
  const float4*   bounds;      // two words per cluster of each group (k_cluster_bounds)
  uint4*          transRecs;  // per cluster left to k_classify_emit (two words) or k_classify_emit_transient (three)
};

constexpr u32 kRejected = 0xFFFFFFFFu;  // fullRecs: a full cluster that did not fit the capacities

// the contiguous range of visible clusters block `blk` of `nb` owns
__device__ __forceinline__ void block_range(u32 n, u32 blk, u32 nb, u32& v0, u32& v1)
{
  const u32 per = (n + nb - 1) / nb;
  v0            = min(n, blk * per);
  v1            = min(n, v0 + per);
}

// Visible cluster v when the list is every cluster in instance order (RT
// semantics: clusters_cull keeps them all): the instance whose first flat
// index is the last one <= v.
// `starts`: the instances' first flat indices (instClusterStart, or the
// block's shared copy of it)
__device__ __forceinline__ tc_ClusterInfo flat_cluster(const u32* starts, u32 numInstances, u32 v)
{
  u32 lo = 0, hi = numInstances;
  while(hi - lo > 1)
  {
    const u32 mid = (lo + hi) >> 1;
    if(starts[mid] <= v)
      lo = mid;
    else
      hi = mid;
  }
  return {lo, v - starts[lo]};
}

// Instance counts up to kFlatShared keep the prefix in shared memory, where
// the binary search of every cluster lookup runs.
constexpr u32 kFlatShared = 1024;

struct FlatStarts
{
  u32 v[kFlatShared];
};

// Called by every thread of the block (contains a barrier); returns the
// prefix the block's lookups use.
__device__ __forceinline__ const u32* stage_flat_starts(const StageCtx& c, FlatStarts& sh)
{
  if(!c.flatVisible || c.numInstances > kFlatShared)
    return c.instClusterStart;
  for(u32 i = threadIdx.x; i < c.numInstances; i += blockDim.x)
    sh.v[i] = c.instClusterStart[i];
  __syncthreads();
  return sh.v;
}

__device__ __forceinline__ tc_ClusterInfo visible_cluster(const StageCtx& c, const u32* starts,
                                                          const tc_ClusterInfo* vis, u32 v)
{
  return c.flatVisible ? flat_cluster(starts, c.numInstances, v) : vis[v];
}

// visible clusters of the instance window (visibleClusters is sorted by instance)
__device__ inline void window_range(const StageCtx& c, u32& lo, u32& hi)
{
  if(c.flatVisible)  // whole window, every cluster listed (clusters_cull runs beside classify)
  {
    lo = 0;
    hi = min(c.instClusterStart[c.numInstances], c.caps.maxVisibleClusters);
    return;
  }
  const tc_ClusterInfo* vis = reinterpret_cast<const tc_ClusterInfo*>(c.build->visibleClusters);
  lo                        = 0;
  hi                        = min(c.build->visibleClusterCounter, c.caps.maxVisibleClusters);
  if(!whole_window(c))
  {
    auto get = [&](u32 i) { return vis[i].instanceID; };
    u32  e   = lower_bound_instance(lo, hi, c.instEnd, get);
    lo       = lower_bound_instance(lo, e, c.instBegin, get);
    hi       = e;
  }
}

__device__ __forceinline__ FactorParams factor_params(const StageCtx& c)
{
  FactorParams fp;
  fp.viewPos   = {c.build->viewPos.x, c.build->viewPos.y, c.build->viewPos.z};
  fp.nearPlane = c.view->nearPlane;
  fp.viewportH = c.view->viewportf.y;
  fp.tessRate  = c.view->tessRate;
  return fp;
}

// ---------------------------------------------------------------------------
// scans
// ---------------------------------------------------------------------------

// block-wide exclusive scan of N values per thread (totals in tot)
template <int N>
__device__ inline void block_scan_n(u64 (&v)[N], u64 (&tot)[N], u64 (*s_warp)[N])
{
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  u64       inc[N];
#pragma unroll
  for(int q = 0; q < N; q++)
  {
    inc[q] = warp_inclusive<u64>(v[q], lane);
    if(lane == 31)
      s_warp[warp][q] = inc[q];
  }
  __syncthreads();
  if(warp == 0)
  {
#pragma unroll
    for(int q = 0; q < N; q++)
    {
      u64 w = lane < nw ? s_warp[lane][q] : 0;
      u64 s = warp_inclusive<u64>(w, lane);
      __syncwarp();
      if(lane < nw)
        s_warp[lane][q] = s - w;
      if(lane == 31)
        s_warp[32][q] = s;
    }
  }
  __syncthreads();
#pragma unroll
  for(int q = 0; q < N; q++)
  {
    tot[q] = s_warp[32][q];
    v[q]   = s_warp[warp][q] + inc[q] - v[q];
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// count
// ---------------------------------------------------------------------------

// The offsets at which block `blockIdx.x` of the write launch starts: the
// counters' values before the launch plus the sums of all blocks before it.
__device__ inline void block_prefix(const ClassifyScratch& cs, u64 (&pre)[kNumCounters],
                                    u64 (*s_warp)[kNumCounters])
{
  u64 x[kNumCounters] = {0, 0, 0, 0, 0};
  for(u32 i = threadIdx.x; i < blockIdx.x; i += blockDim.x)
  {
    const RangeSums o = cs.rangeSums[i];
    x[kCntParts] += (u32)o.partsSplits;
    x[kCntSplits] += (u32)(o.partsSplits >> 32);
    x[kCntGen] += (u32)o.fullVerts;
    x[kCntVerts] += (u32)(o.fullVerts >> 32);
    x[kCntData] += o.data;
  }
  u64 tot[kNumCounters];
  block_scan_n<kNumCounters>(x, tot, s_warp);
  const ClusterOffsets b0 = *cs.bases;
  pre[kCntParts]          = b0.part + tot[kCntParts];
  pre[kCntSplits]         = b0.split + tot[kCntSplits];
  pre[kCntGen]            = b0.gen + tot[kCntGen];
  pre[kCntVerts]          = b0.vert + tot[kCntVerts];
  pre[kCntData]           = b0.data + tot[kCntData];
}

// ---------------------------------------------------------------------------
// transient builds (TC_FLAG_TRANSIENT_1X / _2X)
// ---------------------------------------------------------------------------

// per-triangle word bits beyond config | rotation << 16 | split << 18
constexpr u32 kWordMini        = 1u << 19;  // packed into a 2X batch
constexpr u32 kWordSubset      = 1u << 20;  // in the cluster's 1X subset
constexpr u32 kWordFactorShift = 21;        // edge factors - 1 (3 bits) of a triangle with factors <= 2

constexpr u32 kClusterInfoBytes = 8, kTessInfoBytes = 24;
constexpr u32 kMiniBatch        = TC_2X_MINI_BATCHSIZE;
constexpr u32 kMiniBatchTris    = TC_2X_MINI_BATCHSIZE * TC_2X_MINI_TRIANGLES;
constexpr u32 kMiniBatchVerts   = TC_2X_MINI_BATCHSIZE * TC_2X_MINI_VERTICES;
constexpr u32 kMiniVertexSize   = kMiniBatchVerts + (kMiniBatchTris * 3 + 11) / 12;  // vertices, then index bytes
constexpr u32 kMiniPartSlots    = (kClusterInfoBytes + kMiniBatchTris * 2 + kTessInfoBytes - 1) / kTessInfoBytes;
__device__ __forceinline__ u32 subset_vertex_size(u32 nv, u32 simple) { return nv + (simple * 3 + 11) / 12; }
__device__ __forceinline__ u32 subset_part_slots(u32 simple)
{
  return (kClusterInfoBytes + simple + kTessInfoBytes - 1) / kTessInfoBytes;
}

// per-cluster counts with transient builds (16 bytes):
// x = parts | splits << 7 | generated clusters << 14 | transient builds << 19 | back slots << 23 | full << 28 | 1X << 29
// y = vertices | simple triangles << 10 | numVertices << 17 | numTriangles << 24, z = CLAS bytes
__device__ __forceinline__ u32 t_parts(uint4 r) { return r.x & 0x7F; }
__device__ __forceinline__ u32 t_splits(uint4 r) { return (r.x >> 7) & 0x7F; }
__device__ __forceinline__ u32 t_gen(uint4 r) { return (r.x >> 14) & 0x1F; }
__device__ __forceinline__ u32 t_trans(uint4 r) { return (r.x >> 19) & 0xF; }
__device__ __forceinline__ u32 t_back(uint4 r) { return (r.x >> 23) & 0x1F; }
__device__ __forceinline__ bool t_full(uint4 r) { return (r.x >> 28) & 1; }
__device__ __forceinline__ bool t_subset(uint4 r) { return (r.x >> 29) & 1; }
__device__ __forceinline__ u32 t_verts(uint4 r) { return r.y & 0x3FF; }
__device__ __forceinline__ u32 t_simple(uint4 r) { return (r.y >> 10) & 0x7F; }
__device__ __forceinline__ u32 t_nv(uint4 r) { return (r.y >> 17) & 0x7F; }
__device__ __forceinline__ u32 t_nt(uint4 r) { return (r.y >> 24) & 0x7F; }

// cluster_classify.comp.glsl:254-343 and 543-790, counting only: which
// triangles go to the 1X subset, to parts, to splits and to 2X batches, and
// what the cluster takes from every counter (each allocation counts whether or
// not it will fit, like the reference's atomics). m0/m1, w0/w1: the max factor
// and word of triangles lane and lane + 32.
__device__ __forceinline__ void count_transient(const StageCtx& c, const ClassifyScratch& cs, u32 v, u32 perRange, u32 nv,
                                             u32 nt, u32 simple, u32 m0, u32 m1, u32 w0, u32 w1, u32 templateSize)
{
  const u32  lane   = threadIdx.x & 31;
  const bool full   = simple == nt;
  const bool subset = (c.flags & TC_FLAG_TRANSIENT_1X) && !full && simple > 1;
  const bool mini2x = (c.flags & TC_FLAG_TRANSIENT_2X) != 0;
  const u32* basic  = reinterpret_cast<const u32*>(c.build->basicClusterSizes);
  u32        parts = 0, splits = 0, batches = 0;
  if(!full)
  {
    auto mark = [&](u32 m, u32& w) {  // :573-590
      if(subset && m == 1)
        w |= kWordSubset;
      else if(m <= TC_TESSTABLE_SIZE && mini2x && m <= 2)
        w |= kWordMini;
    };
    if(lane < nt)
      mark(m0, w0);
    if(lane + 32 < nt)
      mark(m1, w1);
    const bool v0 = lane < nt, v1 = lane + 32 < nt;
    parts  = __popc(__ballot_sync(0xFFFFFFFFu, v0 && (w0 & (kWordMini | kWordSubset | (1u << 18))) == 0))
             + __popc(__ballot_sync(0xFFFFFFFFu, v1 && (w1 & (kWordMini | kWordSubset | (1u << 18))) == 0));
    splits = __popc(__ballot_sync(0xFFFFFFFFu, v0 && (w0 & (1u << 18)))) + __popc(__ballot_sync(0xFFFFFFFFu, v1 && (w1 & (1u << 18))));
    const u32 mini0 = __popc(__ballot_sync(0xFFFFFFFFu, v0 && (w0 & kWordMini)));
    const u32 mini1 = __popc(__ballot_sync(0xFFFFFFFFu, v1 && (w1 & kWordMini)));
    batches         = (mini0 + kMiniBatch - 1) / kMiniBatch + (mini1 + kMiniBatch - 1) / kMiniBatch;
    u32* tw         = cs.triWords + (u64)v * TC_MAX_CLUSTER_TRIANGLES;
    if(v0)
      tw[lane] = w0;
    if(v1)
      tw[lane + 32] = w1;
  }
  if(lane != 0)
    return;
  const u32 one   = (full || subset) ? 1u : 0u;
  const u32 gen   = one + batches, trans = (subset ? 1u : 0u) + batches;
  const u32 verts = (full ? nv : (subset ? subset_vertex_size(nv, simple) : 0u)) + kMiniVertexSize * batches;
  const u32 back  = (subset ? subset_part_slots(simple) : 0u) + kMiniPartSlots * batches;
  u64       data  = full ? (u64)templateSize : (subset ? (u64)basic[simple] : 0ull);
  if(batches)
    data += (u64)basic[kMiniBatchTris] * batches;
  reinterpret_cast<uint4*>(cs.counts)[v] =
      make_uint4(parts | (splits << 7) | (gen << 14) | (trans << 19) | (back << 23) | ((full ? 1u : 0u) << 28)
                     | ((subset ? 1u : 0u) << 29),
                 verts | (simple << 10) | (nv << 17) | (nt << 24), (u32)data, 0u);
  RangeSums& rs = cs.rangeSums[v / perRange];
  if(parts | splits)
    atomicAdd(&rs.partsSplits, (unsigned long long)parts | ((unsigned long long)splits << 32));
  if(gen)
  {
    atomicAdd(&rs.fullVerts, (unsigned long long)gen | ((unsigned long long)verts << 32));
    if(data)
      atomicAdd(&rs.data, (unsigned long long)data);
  }
  if(trans)
    atomicAdd(&rs.backTrans, (unsigned long long)back | ((unsigned long long)trans << 32));
}

// ---------------------------------------------------------------------------
// bounds of the clusters of instance groups (tc_groups.cuh)
// ---------------------------------------------------------------------------

// The smallest normal float, added to the squares whose roots bound a length
// from above: squares of less underflow, by at most 2^-149 for each product. (A
// mesh of 1e-23 units under a scale of 1e18 had bounds of zero, and its clusters
// were accepted wherever they lay. A scale whose square overflows fails the test.)
constexpr float kBoundsTiny = 1.17549435e-38f;

// Object-space bounds of the groups' clusters, one warp each: a sphere around
// the vertices and the longest triangle edge, both rounded up. They let the
// count kernel accept a whole cluster of an instance without its vertices
// (bounds_factor_one), so they pay when instances share clusters: head is 0
// when the frame's clusters are fewer than four per bounded one.
__global__ void __launch_bounds__(kBlock, 4) k_cluster_bounds(StageCtx c, GroupTables g)
{
  stage_prologue();
  __shared__ f3 s_vert[kWarps][TC_MAX_CLUSTER_VERTICES];
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const u32 total = g.head[kHeadBounds], reps = g.head[kHeadReps];
  for(u32 u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < total; u += (gridDim.x * blockDim.x) >> 5)
  {
    u32 lo = 0, hi = reps;  // the last representative whose first cluster is at most u
    while(hi - lo > 1)
    {
      const u32 mid = (lo + hi) >> 1;
      if(g.reps[mid].x <= u)
        lo = mid;
      else
        hi = mid;
    }
    const uint2              r  = g.reps[lo];
    const tc_RenderInstance& in = c.instances[r.y];
    const tc_Cluster         cl = reinterpret_cast<const tc_Cluster*>(in.clusters)[u - r.x];
    const u32                nt = min((u32)cl.numTriangles, TC_MAX_CLUSTER_TRIANGLES);
    const u32                nv = min((u32)cl.numVertices, TC_MAX_CLUSTER_VERTICES);
    const uint8_t*           lt = reinterpret_cast<const uint8_t*>(in.clusterLocalTriangles) + cl.firstLocalTriangle;
    const float              inf = __int_as_float(0x7F800000);
    f3                       p[2], mn = {inf, inf, inf}, mx = {-inf, -inf, -inf};
#pragma unroll
    for(u32 h = 0; h < 2; h++)
    {
      const u32 i = lane + 32 * h;
      if(i >= nv)
        continue;
      p[h]            = ldg3(reinterpret_cast<const float*>(in.positions), cl.firstLocalVertex + i);
      s_vert[warp][i] = p[h];
      mn = {fminf(mn.x, p[h].x), fminf(mn.y, p[h].y), fminf(mn.z, p[h].z)};
      mx = {fmaxf(mx.x, p[h].x), fmaxf(mx.y, p[h].y), fmaxf(mx.z, p[h].z)};
    }
#pragma unroll
    for(int o = 16; o > 0; o >>= 1)
    {
      mn = {fminf(mn.x, __shfl_xor_sync(0xFFFFFFFFu, mn.x, o)), fminf(mn.y, __shfl_xor_sync(0xFFFFFFFFu, mn.y, o)),
            fminf(mn.z, __shfl_xor_sync(0xFFFFFFFFu, mn.z, o))};
      mx = {fmaxf(mx.x, __shfl_xor_sync(0xFFFFFFFFu, mx.x, o)), fmaxf(mx.y, __shfl_xor_sync(0xFFFFFFFFu, mx.y, o)),
            fmaxf(mx.z, __shfl_xor_sync(0xFFFFFFFFu, mx.z, o))};
    }
    const f3 mid = {0.5f * (mn.x + mx.x), 0.5f * (mn.y + mx.y), 0.5f * (mn.z + mx.z)};
    float    r2  = 0.0f, e2 = 0.0f;
    bool     bad = false;  // NaN vertices, indices outside the cluster: no bound
#pragma unroll
    for(u32 h = 0; h < 2; h++)
      if(lane + 32 * h < nv)
      {
        const f3    d = sub3(p[h], mid);
        const float q = dot3(d, d);
        bad |= !(q < inf);
        r2 = fmaxf(r2, q);
      }
    __syncwarp();
    for(u32 t = lane; t < nt; t += 32)
    {
      const u32 i0 = lt[3 * t], i1 = lt[3 * t + 1], i2 = lt[3 * t + 2];
      if(max(i0, max(i1, i2)) >= nv)
      {
        bad = true;
        continue;
      }
      const f3 a = s_vert[warp][i0], b = s_vert[warp][i1], d = s_vert[warp][i2];
      const f3 ab = sub3(a, b), bd = sub3(b, d), da = sub3(d, a);
      e2 = fmaxf(e2, fmaxf(dot3(ab, ab), fmaxf(dot3(bd, bd), dot3(da, da))));
    }
#pragma unroll
    for(int o = 16; o > 0; o >>= 1)
    {
      r2 = fmaxf(r2, __shfl_xor_sync(0xFFFFFFFFu, r2, o));
      e2 = fmaxf(e2, __shfl_xor_sync(0xFFFFFFFFu, e2, o));
    }
    bad = __any_sync(0xFFFFFFFFu, bad);
    if(lane == 0)
    {
      // (1e-5 covers the roundings of the differences, dot products and roots,
      // kBoundsTiny squares that underflow)
      const float r = __fsqrt_rn(r2 + kBoundsTiny) * (1.0f + 1e-5f), e = __fsqrt_rn(e2 + kBoundsTiny) * (1.0f + 1e-5f);
      g.bounds[2 * (u64)u]     = make_float4(mid.x, mid.y, mid.z, r);
      g.bounds[2 * (u64)u + 1] = make_float4(bad ? inf : e, (len3(mid) + r) * (1.0f + 1e-5f), 0.0f, 0.0f);
    }
    __syncwarp();  // the vertices are rewritten by the warp's next cluster
  }
}

// Whether every edge of a cluster with object-space bounds b0, b1 certainly has
// factor 1 (see edge_factor) under world matrix m. With u = 2^-24, s >= the
// matrix' largest singular value (the root of the largest row sum of |A^T A|,
// which bounds its largest eigenvalue) and W >= s |p| + |t| for every vertex p:
// a vertex' world position carries an error below 7 u W in length
// (xform_point: four roundings per component, each of at most s |p| + |t|), so
// an edge of the computed positions is at most s E + 14 u W long and a vertex
// at least |A c + t - view| - s r - 14 u W away; 2e-6 W is 33 u W. The factor's
// product is then below 1.4999 / (1 - 1e-5) * (1 + 10 u) < 1.5: the factor is 1.
// NaN and infinite values fail the test.
__device__ __forceinline__ bool bounds_factor_one(const float* m, float4 b0, float4 b1, const FactorParams& fp, float kRate)
{
  const f3    a0 = {m[0], m[1], m[2]}, a1 = {m[4], m[5], m[6]}, a2 = {m[8], m[9], m[10]}, t = {m[12], m[13], m[14]};
  const float g01 = fabsf(dot3(a0, a1)), g02 = fabsf(dot3(a0, a2)), g12 = fabsf(dot3(a1, a2));
  const float s2  = fmaxf(dot3(a0, a0) + g01 + g02, fmaxf(dot3(a1, a1) + g01 + g12, dot3(a2, a2) + g02 + g12));
  const float s   = __fsqrt_rn(s2 + kBoundsTiny) * (1.0f + 1e-5f);
  const float err = 2e-6f * (s * b1.y + len3(t));
  const float d   = dist3(xform_point(m, {b0.x, b0.y, b0.z}), fp.viewPos) - s * b0.w - err;
  return (s * b1.x + err) * kRate < 1.4999f * fmaxf(fp.nearPlane, d * (1.0f - 1e-5f));
}

// the counts of visible cluster v as a full cluster
template <bool Trans>
__device__ __forceinline__ void store_full_counts(const ClassifyScratch& cs, u32 v, u32 nv, u32 nt, u32 data)
{
  if constexpr(Trans)
    reinterpret_cast<uint4*>(cs.counts)[v] = make_uint4((1u << 14) | (1u << 28), nv | (nt << 10) | (nv << 17) | (nt << 24), data, 0u);
  else
    cs.counts[v] = pack_counts(0u, 0u, true, nv, nt, data);
}

__device__ __forceinline__ void add_full_sums(RangeSums& rs, u32 clusters, u32 vertices, u64 data)
{
  atomicAdd(&rs.fullVerts, (unsigned long long)clusters | ((unsigned long long)vertices << 32));
  if(data)
    atomicAdd(&rs.data, (unsigned long long)data);
}

// the visible clusters' counter and set-up when every cluster is visible
__device__ __forceinline__ void visible_set_up(const StageCtx& c)
{
  c.build->visibleClusterCounter = c.instClusterStart[c.numInstances];
  build_setup_apply(c, TC_BUILD_SETUP_CLASSIFY);
}

// With bounds: one thread per visible cluster writes the visible list (RT
// semantics: every cluster in instance order, clusters_cull.comp.glsl:112-161,
// and its set-up) and counts the clusters that are full
// clusters for certain, without their vertices (of an invisible instance, or
// too small for their distance by their bounds), and lists the others for
// k_classify_count. Neighbouring threads take neighbouring clusters, so the
// instance's matrix is one broadcast load and a warp adds to its range's sums
// once. Measured on a GB300, 207,360 clusters of 1,024 instances, 10,700 of
// them listed: the count 88 -> 24 us (bounds 4, this 8, the listed clusters 12),
// the frame 233 -> 162 us. A frame that turns out to have no bounds leaves
// everything to k_classify_count, whose lanes then write the list: written here,
// in front of the count, it costs 2.5 us of 262 with 1,000 instances that share
// nothing and 1.6 of 93 with 256 (by clusters_cull on a side stream 17 and 4: its
// blocks are placed before this kernel's).
template <bool Trans>
__global__ void __launch_bounds__(kBlock) k_classify_whole(StageCtx c, ClassifyScratch cs)
{
  stage_prologue();
  __shared__ FlatStarts s_starts;
  if(cs.groupHead[kHeadBounds] == 0)
    return;
  const u32* starts = stage_flat_starts(c, s_starts);
  if(blockIdx.x == 0 && threadIdx.x == 0)
    visible_set_up(c);
  tc_ClusterInfo*    vis     = reinterpret_cast<tc_ClusterInfo*>(c.build->visibleClusters);
  const u32          n       = min(min(c.instClusterStart[c.numInstances], c.caps.maxVisibleClusters), c.scratch.itemCapacity);
  const u32          lane    = threadIdx.x & 31;
  const FactorParams fp      = factor_params(c);
  const float        kRate   = fp.viewportH * fp.tessRate;
  const bool         culling = (c.flags & TC_FLAG_CULLING) != 0;
  const u32*         states  = reinterpret_cast<const u32*>(c.build->instanceStates);
  const u32          perRange = (n + cs.writeBlocks - 1) / cs.writeBlocks;
  u32*               list    = reinterpret_cast<u32*>(cs.transRecs);
  for(u32 v0 = (blockIdx.x * kBlock + threadIdx.x) & ~31u; v0 < n; v0 += gridDim.x * kBlock)
  {
    const u32 v     = v0 + lane;
    bool      whole = false;
    u32       nv = 0, nt = 0, data = 0;
    if(v < n)
    {
      const tc_ClusterInfo     ci = flat_cluster(starts, c.numInstances, v);
      const tc_RenderInstance* in = c.instances + ci.instanceID;
      reinterpret_cast<uint2*>(vis)[v] = make_uint2(ci.instanceID, ci.clusterID);
      const tc_Cluster cl = reinterpret_cast<const tc_Cluster*>(in->clusters)[ci.clusterID];
      nt = cl.numTriangles, nv = cl.numVertices;
      data = __ldg(reinterpret_cast<const u32*>(in->clusterTemplateInstantiatonSizes) + ci.clusterID);
      const float4* bd = cs.bounds + 2 * (u64)(cs.instBounds[ci.instanceID] + ci.clusterID);
      // (a malformed cluster is k_classify_count's to report)
      whole = nt <= TC_MAX_CLUSTER_TRIANGLES && nv <= TC_MAX_CLUSTER_VERTICES
              && ((culling && (states[ci.instanceID] & TC_INSTANCE_VISIBLE_BIT) == 0)
                  || bounds_factor_one(in->worldMatrix.m, bd[0], bd[1], fp, kRate));
      if(whole)
        store_full_counts<Trans>(cs, v, nv, nt, data);
    }
    const u32 wm = __ballot_sync(0xFFFFFFFFu, whole), om = __ballot_sync(0xFFFFFFFFu, v < n && !whole);
    // the warp's range (two where one ends inside it)
    for(u32 left = wm; left;)
    {
      const u32  r    = (v0 + __ffs(left) - 1) / perRange;
      const bool mine = whole && v / perRange == r;
      const u32  sel  = __ballot_sync(0xFFFFFFFFu, mine);
      const u32  verts = __reduce_add_sync(0xFFFFFFFFu, mine ? nv : 0u);
      const u64  bytes = warp_sum_u64(mine ? data : 0u);
      left &= ~sel;
      if(lane == 0)
        add_full_sums(cs.rangeSums[r], __popc(sel), verts, bytes);
    }
    if(om)
    {
      u32 at = 0;
      if(lane == 0)
        at = atomicAdd(cs.groupHead + kHeadList, __popc(om));
      at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(om & ((1u << lane) - 1u));
      if(v < n && !whole)
        list[at] = v;
    }
  }
}

// MinBlocks: resident 256-thread blocks per SM the registers are sized for
// (4: 64 registers, 6: 40, 8: 32); more resident warps hide more of the
// dependent-load latency per cluster at the cost of some spills.
template <int MinBlocks, bool Trans = false>
__global__ void __launch_bounds__(kBlock, MinBlocks) k_classify_count(StageCtx c, ClassifyScratch cs)
{
  stage_prologue();
  __shared__ f3  s_vert[kWarps][TC_MAX_CLUSTER_VERTICES];
  __shared__ f2  s_dist[kWarps][TC_MAX_CLUSTER_VERTICES];  // per vertex: distance to the view position, its reciprocal
  __shared__ u32 s_range[2];
  __shared__ FlatStarts s_starts;
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if(threadIdx.x == 0)
    window_range(c, s_range[0], s_range[1]);
  __syncthreads();
  const u32* starts = stage_flat_starts(c, s_starts);
  const u32 begin = s_range[0];
  const u32 n     = min(s_range[1] - s_range[0], c.scratch.itemCapacity);

  const tc_SceneBuilding* b       = c.build;
  const tc_ClusterInfo*   vis     = reinterpret_cast<const tc_ClusterInfo*>(b->visibleClusters);
  const FactorParams      fp      = factor_params(c);
  const float             rNear   = __fdiv_rn(1.0f, fp.nearPlane);
  const float             kRate   = fp.viewportH * fp.tessRate;
  const float             k2      = kRate * kRate;
  const float             near2   = fp.nearPlane * fp.nearPlane;
  const bool              culling = (c.flags & TC_FLAG_CULLING) != 0;
  const u32               sf      = clamp_split_factor(c.caps.splitFactor);
  const u32               wordOnes = classify_triangle(make_uint3(1u, 1u, 1u), sf);  // a triangle of factors 1
  if(blockIdx.x == 0 && threadIdx.x == 0)  // the offsets continue from the counters' current values
  {
    cs.fullRange[2] = 0;
    if constexpr(Trans)
    {
      // parts from the front of the two-sided counter (build.glsl:52-82)
      *cs.bases = {(u32)b->dualPartTriangleCounter, (u32)b->splitTriangleCounter, b->genClusterCounter,
                   b->genVertexCounter, b->genClusterDataCounter};
      *reinterpret_cast<TransBases*>(cs.bases + 1) = {(u32)(b->dualPartTriangleCounter >> 32), b->transBuildCounter,
                                                      b->tempInstantiateCounter, 0u};
    }
    else
      *cs.bases = {b->partTriangleCounter, (u32)b->splitTriangleCounter, b->genClusterCounter, b->genVertexCounter,
                   b->genClusterDataCounter};
  }
  // the write launch's block ranges, which collect the counts' sums
  const u32 perRange = (n + cs.writeBlocks - 1) / cs.writeBlocks;

  // the warp's clusters are v = gw + nwarps * j, j < cntW (spread over the
  // whole list, which evens out instances of uneven cost); their cluster
  // records load one lane per cluster, 32 at a time, so that only the vertex
  // and index loads remain on each cluster's dependent path
  const u32  gw     = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const u32  nwarps = (gridDim.x * blockDim.x) >> 5;
  // with bounds k_classify_whole has counted the others: the list it left
  const bool bounded = cs.groups != nullptr && cs.groupHead[kHeadBounds] != 0;
  const u32* list    = reinterpret_cast<const u32*>(cs.transRecs);
  const u32  items   = bounded ? cs.groupHead[kHeadList] : n;
  const bool write   = cs.groups != nullptr && !bounded;  // the visible list
  if(write && blockIdx.x == 0 && threadIdx.x == 0)
    visible_set_up(c);
  const u32  cntW   = gw < items ? (items - gw + nwarps - 1) / nwarps : 0u;
  const u32* states = reinterpret_cast<const u32*>(b->instanceStates);
  for(u32 j0 = 0; j0 < cntW; j0 += 32)
  {
    const u32 jn = min(32u, cntW - j0);
    u32       hV = 0, hInst = 0, hMeta = 0, hFirstV = 0, hFirstT = 0, hData = 0;
    bool      whole = false;
    if(lane < jn)
    {
      const u32                at = gw + nwarps * (j0 + lane);
      const u32                v  = bounded ? list[at] : at;
      const tc_ClusterInfo     ci = visible_cluster(c, starts, vis, begin + v);
      const tc_RenderInstance* in = c.instances + ci.instanceID;
      const tc_Cluster         cl = reinterpret_cast<const tc_Cluster*>(in->clusters)[ci.clusterID];
      u32                      nt = cl.numTriangles, nv = cl.numVertices;
      if(write)
        reinterpret_cast<uint2*>(c.build->visibleClusters)[v] = make_uint2(ci.instanceID, ci.clusterID);
      if(nt > TC_MAX_CLUSTER_TRIANGLES || nv > TC_MAX_CLUSTER_VERTICES)
      {
        atomicOr(c.errorWord, TC_DEVERR_BAD_CLUSTER);
        nt = min(nt, TC_MAX_CLUSTER_TRIANGLES);
        nv = min(nv, TC_MAX_CLUSTER_VERTICES);
      }
      hInst   = ci.instanceID;
      hMeta   = nv | (nt << 8);
      hFirstV = cl.firstLocalVertex;
      hFirstT = cl.firstLocalTriangle;
      hData   = __ldg(reinterpret_cast<const u32*>(in->clusterTemplateInstantiatonSizes) + ci.clusterID);
      hV      = v;
      // cluster_classify.comp.glsl:203-211: invisible instance, no tessellation
      // (one lane for such a cluster, not a warp)
      whole = culling && (states[ci.instanceID] & TC_INSTANCE_VISIBLE_BIT) == 0;
    }
    for(u32 left = __ballot_sync(0xFFFFFFFFu, lane < jn && !whole); left; left &= left - 1)
    {
      const u32                jj     = __ffs(left) - 1;
      const u32                v      = __shfl_sync(0xFFFFFFFFu, hV, jj);
      const u32                meta   = __shfl_sync(0xFFFFFFFFu, hMeta, jj);
      const u32                nv     = meta & 0xFF, nt = (meta >> 8) & 0xFF;
      const tc_RenderInstance* in     = c.instances + __shfl_sync(0xFFFFFFFFu, hInst, jj);
      const u32                firstV = __shfl_sync(0xFFFFFFFFu, hFirstV, jj);
      const u32                firstT = __shfl_sync(0xFFFFFFFFu, hFirstT, jj);
      u32                      m0 = 0, m1 = 0, w0 = 0, w1 = 0;
      u32                      simple = nt;
      {
        // indices first (their loads overlap the vertex loads); masked to the
        // staged range: a malformed index reads a wrong vertex of the same
        // cluster, never outside shared memory
        const uint8_t* lt = reinterpret_cast<const uint8_t*>(in->clusterLocalTriangles) + firstT;
        u32            ia = 0, ib = 0;
        if(lane < nt)
          ia = (lt[lane * 3 + 0] & 63u) | ((lt[lane * 3 + 1] & 63u) << 8) | ((lt[lane * 3 + 2] & 63u) << 16);
        if(lane + 32 < nt)
          ib = (lt[lane * 3 + 96] & 63u) | ((lt[lane * 3 + 97] & 63u) << 8) | ((lt[lane * 3 + 98] & 63u) << 16);
        // cluster_classify.comp.glsl:180-198 vertices, then 217-246 factors; each
        // vertex is taken to world space once here (the same operations the
        // shader applies per triangle corner, so the same bits)
        const float* pos = reinterpret_cast<const float*>(in->positions);
        float        m[16];
#pragma unroll
        for(int q = 0; q < 16; q++)
          m[q] = __ldg(in->worldMatrix.m + q);
        for(u32 i = lane; i < nv; i += 32)
        {
          const f3 w  = xform_point(m, ldg3(pos, firstV + i));
          const f3 dv = sub3(w, fp.viewPos);
          s_vert[warp][i]   = w;
          s_dist[warp][i].x = dot3(dv, dv);  // squared: the distance and its reciprocal only when needed
        }
        __syncwarp();
        // A cluster whose every edge provably has factor 1 (edge_factor_one_sq:
        // squared lengths and distances, no roots or divisions) is classified
        // without the distances; the word is that of factors (1, 1, 1).
        auto allOne = [&](u32 idx) {
          const u32   i0 = idx & 0xFF, i1 = (idx >> 8) & 0xFF, i2 = idx >> 16;
          const f3    v0 = s_vert[warp][i0], v1 = s_vert[warp][i1], v2 = s_vert[warp][i2];
          const float q0 = s_dist[warp][i0].x, q1 = s_dist[warp][i1].x, q2 = s_dist[warp][i2].x;
          return edge_factor_one_sq(v0, v1, q0, q1, k2, near2) && edge_factor_one_sq(v1, v2, q1, q2, k2, near2)
                 && edge_factor_one_sq(v2, v0, q2, q0, k2, near2);
        };
        if(__all_sync(0xFFFFFFFFu, (lane >= nt || allOne(ia)) && (lane + 32 >= nt || allOne(ib))))
        {
          if(lane < nt)
            m0 = 1, w0 = wordOnes;
          if(lane + 32 < nt)
            m1 = 1, w1 = wordOnes;
          simple = nt;
        }
        else
        {
          for(u32 i = lane; i < nv; i += 32)
          {
            const float d     = __fsqrt_rn(s_dist[warp][i].x);  // dist3(w, viewPos)
            s_dist[warp][i].y = __fdiv_rn(1.0f, d);
            s_dist[warp][i].x = d;
          }
          __syncwarp();
          auto classify = [&](u32 idx, u32& mOut, u32& wOut) {
            const u32   i0 = idx & 0xFF, i1 = (idx >> 8) & 0xFF, i2 = idx >> 16;
            const f2    d0 = s_dist[warp][i0], d1 = s_dist[warp][i1], d2 = s_dist[warp][i2];
            const uint3 f  = tess_factors_hoisted(s_vert[warp][i0], s_vert[warp][i1], s_vert[warp][i2], d0.x, d1.x,
                                                  d2.x, d0.y, d1.y, d2.y, rNear, fp);
            mOut           = max(max(f.x, f.y), f.z);
            wOut           = classify_triangle(f, sf);
            if constexpr(Trans)  // factors of a 2X candidate, for its triangle map (cluster_classify.comp.glsl:817)
              if(mOut <= 2)
                wOut |= ((f.x - 1) | ((f.y - 1) << 1) | ((f.z - 1) << 2)) << kWordFactorShift;
          };
          if(lane < nt)
            classify(ia, m0, w0);
          if(lane + 32 < nt)
            classify(ib, m1, w1);
          simple = __popc(__ballot_sync(0xFFFFFFFFu, lane < nt && m0 == 1))
                   + __popc(__ballot_sync(0xFFFFFFFFu, lane + 32 < nt && m1 == 1));
        }
        __syncwarp();  // s_vert is reused by the next cluster
      }
      const bool full  = simple == nt;
      if constexpr(Trans)
      {
        count_transient(c, cs, v, perRange, nv, nt, simple, m0, m1, w0, w1, __shfl_sync(0xFFFFFFFFu, hData, jj));
        continue;
      }
      u32        parts = 0, splits = 0;
      if(!full)
      {
        parts  = __popc(__ballot_sync(0xFFFFFFFFu, lane < nt && m0 <= TC_TESSTABLE_SIZE))
                 + __popc(__ballot_sync(0xFFFFFFFFu, lane + 32 < nt && m1 <= TC_TESSTABLE_SIZE));
        splits = nt - parts;
        u32* tw = cs.triWords + (u64)v * TC_MAX_CLUSTER_TRIANGLES;
        if(lane < nt)
          tw[lane] = w0;
        if(lane + 32 < nt)
          tw[lane + 32] = w1;
      }
      const u32 data = __shfl_sync(0xFFFFFFFFu, hData, jj);
      if(lane == 0)
      {
        cs.counts[v] = pack_counts(parts, splits, full, nv, nt, data);
        RangeSums& rs = cs.rangeSums[v / perRange];
        if(full)
        {
          atomicAdd(&rs.fullVerts, 1ull | ((unsigned long long)nv << 32));
          if(data)
            atomicAdd(&rs.data, (unsigned long long)data);
        }
        else
          atomicAdd(&rs.partsSplits, (unsigned long long)parts | ((unsigned long long)splits << 32));
      }
    }
    // (after the others: in front of them it delayed their chains of loads, 0.2 us
    // of a frame, 0.3 of the stage call)
    if(whole)
    {
      store_full_counts<Trans>(cs, hV, hMeta & 0xFF, (hMeta >> 8) & 0xFF, hData);
      add_full_sums(cs.rangeSums[hV / perRange], 1u, hMeta & 0xFF, hData);
    }
  }
}

// ---------------------------------------------------------------------------
// write
// ---------------------------------------------------------------------------

__device__ __forceinline__ void store_tess_info(tc_TessTriangleInfo* dst, const tc_ClusterInfo& ci, u32 v0, u32 v1,
                                                u32 v2, u32 tc)
{
  uint2* p = reinterpret_cast<uint2*>(dst);
  p[0]     = make_uint2(ci.instanceID, ci.clusterID);
  p[1]     = make_uint2(v0, v1);
  p[2]     = make_uint2(v2, tc);
}

// part / split triangle from its per-triangle word (cluster_classify.comp.glsl:608-666)
__device__ __forceinline__ void emit_triangle(tc_TessTriangleInfo* dst, const tc_ClusterInfo& ci, u32 tri, u32 word)
{
  u32       v0 = 0, v1 = TC_TESSTABLE_COORD_MAX, v2 = TC_TESSTABLE_COORD_MAX << 16;
  const u32 rot = (word >> 16) & 3;
  if(rot == 1)
  {
    u32 t = v0;
    v0 = v1, v1 = v2, v2 = t;
  }
  else if(rot == 2)
  {
    u32 t = v2;
    v2 = v1, v1 = v0, v0 = t;
  }
  store_tess_info(dst, ci, v0, v1, v2, tri | ((word & 0xFFFFu) << 16));
}

// cluster_classify.comp.glsl:543-666: the part and split triangles of one
// cluster by one warp, from the words of triangles lane and lane + 32. The
// cluster's parts are consecutive records of 24 bytes: they are put together
// in the warp's `stage` and stored as consecutive 8-byte words (a lane that
// stores its own record touches 24 sectors per store instruction, eight when
// the lanes' words are consecutive).
__device__ __forceinline__ void emit_cluster(const StageCtx& c, const tc_ClusterInfo& ci, u32 nt, u32 offPart,
                                             u32 offSplit, u32 w0, u32 w1, uint2* stage)
{
  const tc_SceneBuilding* b      = c.build;
  const tc_caps&          k      = c.caps;
  tc_TessTriangleInfo*    splits = reinterpret_cast<tc_TessTriangleInfo*>(b->splitTriangles);
  tc_TessTriangleInfo*    parts  = reinterpret_cast<tc_TessTriangleInfo*>(b->partTriangles);
  const u32  lane = threadIdx.x & 31, ltm = (1u << lane) - 1u;
  const bool s0  = lane < nt && (w0 >> 18) != 0, p0 = lane < nt && (w0 >> 18) == 0;
  const bool s1  = lane + 32 < nt && (w1 >> 18) != 0, p1 = lane + 32 < nt && (w1 >> 18) == 0;
  const u32  bs0 = __ballot_sync(0xFFFFFFFFu, s0), bp0 = __ballot_sync(0xFFFFFFFFu, p0);
  const u32  bs1 = __ballot_sync(0xFFFFFFFFu, s1), bp1 = __ballot_sync(0xFFFFFFFFu, p1);
  tc_TessTriangleInfo* local = reinterpret_cast<tc_TessTriangleInfo*>(stage);
  if(p0)
    emit_triangle(local + __popc(bp0 & ltm), ci, lane, w0);
  if(p1)
    emit_triangle(local + __popc(bp0) + __popc(bp1 & ltm), ci, lane + 32, w1);
  __syncwarp();
  const u32 np   = min((u32)__popc(bp0) + (u32)__popc(bp1), k.maxPartTriangles - min(offPart, k.maxPartTriangles));
  uint2*    dst  = reinterpret_cast<uint2*>(parts + offPart);
  for(u32 q = lane; q < 3 * np; q += 32)
    dst[q] = stage[q];
  __syncwarp();  // the stage is rewritten by the warp's next cluster
  if((bs0 | bs1) == 0)
    return;
  // split items also carry their base triangle's world positions (read by
  // every split pass instead of the instance / cluster / vertex chain)
  const tc_RenderInstance* in = c.instances + ci.instanceID;
  const tc_Cluster         cl = reinterpret_cast<const tc_Cluster*>(in->clusters)[ci.clusterID];
  float                    m[16];
#pragma unroll
  for(int j = 0; j < 16; j++)
    m[j] = __ldg(in->worldMatrix.m + j);
  auto split = [&](u64 o, u32 tri, u32 w) {
    if(o >= k.maxSplitTriangles)
      return;
    emit_triangle(splits + o, ci, tri, w);
    const uint8_t* lt  = reinterpret_cast<const uint8_t*>(in->clusterLocalTriangles) + cl.firstLocalTriangle;
    const float*   pos = reinterpret_cast<const float*>(in->positions);
    float*         d   = c.splitBase + 9 * o;
#pragma unroll
    for(int vv = 0; vv < 3; vv++)
    {
      const f3 wp = xform_point(m, ldg3(pos, cl.firstLocalVertex + lt[tri * 3 + vv]));
      d[3 * vv + 0] = wp.x, d[3 * vv + 1] = wp.y, d[3 * vv + 2] = wp.z;
    }
  };
  if(s0)
    split((u64)offSplit + __popc(bs0 & ltm), lane, w0);
  if(s1)
    split((u64)offSplit + __popc(bs0) + __popc(bs1 & ltm), lane + 32, w1);
}

// the words of cluster v's triangles lane and lane + 32
__device__ __forceinline__ uint2 cluster_words(const ClassifyScratch& cs, u32 v, u32 nt)
{
  const u32  lane = threadIdx.x & 31;
  const u32* tw   = cs.triWords + (u64)v * TC_MAX_CLUSTER_TRIANGLES;
  return make_uint2(lane < nt ? tw[lane] : 0u, lane + 32 < nt ? tw[lane + 32] : 0u);
}

// Listed: the clusters with part or split triangles go to a list that
// k_classify_emit's warps stride over, instead of being written by their
// range's block. The visible clusters of an instance lie next to each other,
// so of the 608 ranges of 341 clusters of a frame with 207,360 clusters, 4,694
// of them tessellated, a few hold them all: from the count's end to the last
// write 39 us in one kernel, 22 us in two (terrain of 32,768 clusters, nearly
// all tessellated: 36 -> 23 us). Ranges of up to 32 clusters, four per warp,
// are written at once: the second launch costs what it gains.
template <int MinBlocks>
__global__ void __launch_bounds__(kBlock, MinBlocks) k_classify_write(StageCtx c, ClassifyScratch cs)
{
  stage_prologue();
  __shared__ u32            s_range[2];
  __shared__ u64            s_warp[33][kNumCounters];
  __shared__ ClusterOffsets s_off[kBlock];  // offsets of the chunk's clusters
  __shared__ uint2          s_cnt[kBlock];  // counts of the chunk's clusters
  __shared__ tc_ClusterInfo s_ci[kBlock];   // the chunk's clusters
  __shared__ uint2          s_stage[kWarps][3 * TC_MAX_CLUSTER_TRIANGLES];
  __shared__ FlatStarts     s_starts;
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if(threadIdx.x == 0)
    window_range(c, s_range[0], s_range[1]);
  __syncthreads();
  const u32* starts = stage_flat_starts(c, s_starts);
  const u32 begin = s_range[0];
  const u32 n     = min(s_range[1] - s_range[0], c.scratch.itemCapacity);

  tc_SceneBuilding*     b            = c.build;
  const tc_caps&        k            = c.caps;
  const tc_ClusterInfo* vis          = reinterpret_cast<const tc_ClusterInfo*>(b->visibleClusters);
  const u64             maxData      = (u64)k.maxGeneratedClusterMegs * 1024ull * 1024ull;
  tc_BlasBuildInfo*     blas         = reinterpret_cast<tc_BlasBuildInfo*>(b->blasBuildInfos);
  const u32             ltm          = (1u << lane) - 1u;
  u32                   statTris = 0, statTemp = 0;

  u64 pre[kNumCounters];  // offsets of the next chunk's first cluster
  block_prefix(cs, pre, s_warp);
  const u32 genBase = cs.bases->gen;
  u32       vBegin, vEnd;
  block_range(n, blockIdx.x, gridDim.x, vBegin, vEnd);
  for(u32 c0 = vBegin; c0 < vEnd; c0 += kBlock)
  {
    // exclusive scan of the chunk's counts, in cluster order
    const u32 len = min(kBlock, vEnd - c0);
    {
      const uint2 r = threadIdx.x < len ? cs.counts[c0 + threadIdx.x] : make_uint2(0, 0);
      if(threadIdx.x < len)  // looked up once per cluster, in parallel
        s_ci[threadIdx.x] = visible_cluster(c, starts, vis, begin + c0 + threadIdx.x);
      u64 x[kNumCounters] = {cnt_parts(r), cnt_splits(r), cnt_full(r), cnt_verts(r), r.y};
      u64 tot[kNumCounters];
      block_scan_n<kNumCounters>(x, tot, s_warp);
      s_cnt[threadIdx.x] = r;
      s_off[threadIdx.x] = {(u32)(pre[kCntParts] + x[kCntParts]), (u32)(pre[kCntSplits] + x[kCntSplits]),
                            (u32)(pre[kCntGen] + x[kCntGen]), (u32)(pre[kCntVerts] + x[kCntVerts]),
                            pre[kCntData] + x[kCntData]};
#pragma unroll
      for(int q = 0; q < kNumCounters; q++)
        pre[q] += tot[q];
    }
    __syncthreads();
    // each warp takes a contiguous part of the chunk (instance-sorted), so its
    // full-cluster BLAS reference counts collapse into one atomic per instance
    // it touches and its full clusters' vertices are contiguous
    const u32 perW = (len + kWarps - 1) / kWarps;
    const u32 lo = min(len, warp * perW), hi = min(len, lo + perW);

    // ---- phase 1: part and split triangles ------------------------------------
    const u32  mine  = lo + lane;
    const bool cut   = mine < hi && !cnt_full(s_cnt[min(mine, kBlock - 1)]);
    u32        left  = __ballot_sync(0xFFFFFFFFu, cut);
    if(cs.listed && left)
    {
      u32 at = 0;
      if(lane == 0)
        at = atomicAdd(cs.fullRange + 2, __popc(left));
      at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(left & ltm);
      if(cut)
      {
        uint4* rec = cs.transRecs + 2 * (u64)at;
        rec[0] = make_uint4(s_ci[mine].instanceID, s_ci[mine].clusterID, s_off[mine].part, s_off[mine].split);
        rec[1] = make_uint4(c0 + mine, cnt_parts(s_cnt[mine]) + cnt_splits(s_cnt[mine]), 0u, 0u);
      }
      left = 0;
    }
    for(; left; left &= left - 1)
    {
      const u32   i  = lo + (u32)__ffs(left) - 1;
      const u32   nt = cnt_parts(s_cnt[i]) + cnt_splits(s_cnt[i]);
      const uint2 w  = cluster_words(cs, c0 + i, nt);
      emit_cluster(c, s_ci[i], nt, s_off[i].part, s_off[i].split, w.x, w.y, s_stage[warp]);
    }

    // ---- phase 2: full clusters of the warp's part, 32 at a time ---------------
    // cluster_classify.comp.glsl:271-488: instantiation arguments, one lane per
    // cluster (the instance loads of 32 clusters overlap). The displaced
    // vertices (:457-482) are written by k_classify_full_vertices from the
    // records left here.
    for(u32 i0 = lo; i0 < hi; i0 += 32)
    {
      const u32 i    = i0 + lane;
      bool      full = false;
      u32       inst = 0xFFFFFFFFu;
      if(i < hi)
      {
        const uint2 r = s_cnt[i];
        if(cnt_full(r))
        {
          const ClusterOffsets off = s_off[i];
          const u32            v   = c0 + i;
          full = !((u64)off.vert + cnt_verts(r) > k.maxGeneratedVertices || (u64)off.gen + 1 > k.maxGeneratedClusters
                   || off.data + r.y > maxData);
          cs.fullRecs[cs.groups ? v : off.gen - genBase] = full ? make_uint2(begin + v, off.vert) : make_uint2(kRejected, 0u);
          if(full)
          {
            const tc_ClusterInfo     ci = s_ci[i];
            const tc_RenderInstance* in = c.instances + ci.instanceID;
            // accepted instantiations form a prefix of the serial order, so the
            // instantiation slot equals the generated-cluster slot
            const u32                  tempOffset = off.gen;
            tc_TemplateInstantiateInfo ti;
            ti.clusterIdOffset        = 0;
            ti.geometryIndexOffset    = 0;
            ti.clusterTemplateAddress = __ldg(reinterpret_cast<const u64*>(in->clusterTemplateAdresses) + ci.clusterID);
            ti.vertexBufferAddress    = b->genVertices + (u64)off.vert * 12ull;
            ti.vertexBufferStride     = 12;
            reinterpret_cast<tc_TemplateInstantiateInfo*>(b->tempInstantiations)[tempOffset] = ti;
            reinterpret_cast<u32*>(b->tempInstanceIDs)[tempOffset]                          = ci.instanceID;
            reinterpret_cast<u64*>(b->tempClusterAddresses)[tempOffset]                     = b->genClusterData + off.data;
            if((c.flags & TC_FLAG_WRITE_FULLCLUSTERS) && b->fullClusters)
              reinterpret_cast<tc_ClusterInfo*>(b->fullClusters)[tempOffset] = ci;
            statTemp += 1;
            statTris += cnt_tris(r);
            inst = ci.instanceID;
          }
        }
        else if(cs.groups)
          cs.fullRecs[c0 + i] = make_uint2(kRejected, 0u);
      }
      const u32 fm = __ballot_sync(0xFFFFFFFFu, full);
      // CLAS reference counts: one atomic per distinct instance of the batch
      for(u32 remaining = fm; remaining;)
      {
        const int src = __ffs(remaining) - 1;
        const u32 gk  = __shfl_sync(0xFFFFFFFFu, inst, src);
        const u32 sel = __ballot_sync(0xFFFFFFFFu, full && inst == gk);
        remaining &= ~sel;
        if((int)lane == src)
          atomicAdd(&blas[gk].clusterReferencesCount, __popc(sel));
      }
    }
    __syncthreads();  // s_off / s_cnt are rewritten by the next chunk
  }

  // statistics: one atomic each per warp
#pragma unroll
  for(int o = 16; o > 0; o >>= 1)
  {
    statTemp += __shfl_xor_sync(0xFFFFFFFFu, statTemp, o);
    statTris += __shfl_xor_sync(0xFFFFFFFFu, statTris, o);
  }
  if(lane == 0)
  {
    if(statTemp)
      atomicAdd(&b->tempInstantiateCounter, statTemp);
    if(statTris)
      atomicAdd(&c.readback->numTotalTriangles, statTris);
  }

  // the last block's running offsets are the totals; no block reads the
  // counters after count took their values
  if(blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
  {
    cs.fullRange[0] = cs.groups ? 0u : genBase;
    cs.fullRange[1] = cs.groups ? n : (u32)pre[kCntGen];
    if(n)
    {
      const ClusterOffsets b0  = *cs.bases;
      b->partTriangleCounter   = (u32)pre[kCntParts];
      b->splitTriangleCounter  = (int32_t)(u32)pre[kCntSplits];
      b->genClusterCounter     = (u32)pre[kCntGen];
      b->genVertexCounter      = (u32)pre[kCntVerts];
      b->genClusterDataCounter = pre[kCntData];
      // cluster_classify.comp.glsl:299 counts every full cluster, accepted or not
      c.readback->numFullClusters += (u32)pre[kCntGen] - b0.gen;
    }
    if(c.fuseSetup != kNoSetup)
      build_setup_apply(c, c.fuseSetup);
  }
}

// The clusters k_classify_write listed: a warp's next cluster is loaded while
// the current one is written.
__global__ void __launch_bounds__(kBlock, 4) k_classify_emit(StageCtx c, ClassifyScratch cs)
{
  stage_prologue();
  __shared__ uint2 s_stage[kWarps][3 * TC_MAX_CLUSTER_TRIANGLES];
  const u32 count = cs.fullRange[2], warp = threadIdx.x >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
  u32       i     = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if(i >= count)
    return;
  uint4 a = cs.transRecs[2 * (u64)i], v = cs.transRecs[2 * (u64)i + 1];
  uint2 w = cluster_words(cs, v.x, v.y);
  for(;;)
  {
    const uint4 ca = a, cv = v;
    const uint2 cw = w;
    i += nwarps;
    if(i < count)
    {
      a = cs.transRecs[2 * (u64)i], v = cs.transRecs[2 * (u64)i + 1];
      w = cluster_words(cs, v.x, v.y);
    }
    emit_cluster(c, {ca.x, ca.y}, cv.y, ca.z, ca.w, cw.x, cw.y, s_stage[warp]);
    if(i >= count)
      break;
  }
}

// ---------------------------------------------------------------------------
// write, with transient builds
// ---------------------------------------------------------------------------

enum : int
{
  kTFront = 0,
  kTSplit,
  kTGen,
  kTVert,
  kTData,
  kTBack,
  kTTrans,
  kTNum
};

// a cluster's offsets into every counter (exclusive, in the canonical order)
struct TransOffsets
{
  u32 front, split, gen, vert, back, trans;
  u64 data;
};

// build.glsl:52-66: slots from the back of partTriangles; maxPartTriangles
// when the two ends would meet (the counter advances either way)
__device__ __forceinline__ u32 back_alloc(u32 x, u32& y, u32 m, u32 maxParts)
{
  const u32 off = ((u64)x + y + m + 1 > maxParts) ? maxParts : maxParts - y - m;
  y += m;
  return off;
}

// cluster_classify.comp.glsl:401-431 / 751-786
__device__ __forceinline__ void store_clas_build(tc_ClasBuildInfo* dst, u32 mode, u32 partOffset, u32 numTriangles,
                                                 u32 numVertices, u32 truncateBits, u64 vertexBuffer)
{
  uint4* d = reinterpret_cast<uint4*>(dst);
  d[0]     = make_uint4((mode << 30) | partOffset, 0u, numTriangles | (numVertices << 9) | (truncateBits << 18) | (1u << 24),
                        4u << 29);
  d[1]     = make_uint4(1u | (12u << 16), 0u, (u32)(vertexBuffer + (u64)numVertices * 12), (u32)((vertexBuffer + (u64)numVertices * 12) >> 32));
  d[2]     = make_uint4((u32)vertexBuffer, (u32)(vertexBuffer >> 32), 0u, 0u);
  d[3]     = make_uint4(0u, 0u, 0u, 0u);
}

// a 2X batch's base triangle: its u16 map entries and u8 indices (:880-903)
__device__ inline void mini_indices(const StageCtx& c, u32 tri, u32 word, u32 rel, u32 baseTris, u32 vertexOffset,
                                    u32 partOffset)
{
  tc_SceneBuilding*       b   = c.build;
  const u32               cfg = word & 0xFFFFu;
  const tc_TessTableEntry e   = table_entry(c.table, cfg);
  const u32 pf  = (word >> kWordFactorShift) & 7;
  uint8_t*  idx = reinterpret_cast<uint8_t*>(b->genVertices) + ((u64)vertexOffset + kMiniBatchVerts) * 12;
  uint16_t* map = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(b->partTriangles) + (u64)partOffset * kTessInfoBytes
                                              + kClusterInfoBytes);
  for(u32 i = 0; i < e.numTriangles; i++)
  {
    const uint3 ct        = cfg_triangle(c.table, e, cfg, i);
    const u32   triOffset = baseTris + i;
    map[triOffset]        = (uint16_t)(tri | (i << 8) | (pf << 12));
    idx[triOffset * 3 + 0] = (uint8_t)(ct.x + rel * TC_2X_MINI_VERTICES);
    idx[triOffset * 3 + 1] = (uint8_t)(ct.y + rel * TC_2X_MINI_VERTICES);
    idx[triOffset * 3 + 2] = (uint8_t)(ct.z + rel * TC_2X_MINI_VERTICES);
  }
}

// the warp zeroes `words` 32-bit words at p (4-byte aligned)
__device__ __forceinline__ void warp_zero(void* p, u32 words)
{
  u32* w = reinterpret_cast<u32*>(p);
  for(u32 i = threadIdx.x & 31; i < words; i += 32)
    w[i] = 0u;
}

// cluster_classify.comp.glsl:254-905 with transient builds, for one cluster
// that is not a full one, by one warp, in the canonical order: the 1X
// allocation, then per 32-triangle chunk its parts and splits followed by its
// 2X batches. Offsets come from the block scan; every allocation is tested like
// the reference's (the counters advance whether or not it fits). Bytes the
// reference leaves unwritten inside an allocation are written as zeros.
__device__ inline void write_cluster_transient(const StageCtx& c, const ClassifyScratch& cs, u32 visIndex, u32 v,
                                               const tc_ClusterInfo& ci, uint4 r, TransOffsets o, u32& statTrans,
                                               u32& statTris)
{
  const u32         lane = threadIdx.x & 31, ltm = (1u << lane) - 1u;
  tc_SceneBuilding* b    = c.build;
  const tc_caps&    k    = c.caps;
  const u64         maxData = (u64)k.maxGeneratedClusterMegs * 1024ull * 1024ull;
  const u32*        basic   = reinterpret_cast<const u32*>(b->basicClusterSizes);
  tc_BlasBuildInfo* blas    = reinterpret_cast<tc_BlasBuildInfo*>(b->blasBuildInfos);
  const u32         nt = t_nt(r), nv = t_nv(r), simple = t_simple(r);
  const bool        subset = t_subset(r);
  const tc_RenderInstance* in = c.instances + ci.instanceID;
  const tc_Cluster         cl = reinterpret_cast<const tc_Cluster*>(in->clusters)[ci.clusterID];
  u32 x = o.front, y = o.back, s = o.split, g = o.gen, vo = o.vert, tr = o.trans;
  u64 d = o.data;
  auto fits = [&](u32 vertexSize, u64 dataSize, u32 partOffset, u32 partSize) {
    return !((u64)vo + vertexSize > k.maxGeneratedVertices || (u64)g + 1 > k.maxGeneratedClusters
             || d + dataSize > maxData || (u64)partOffset + partSize > k.maxPartTriangles);
  };
  uint8_t* gvb = reinterpret_cast<uint8_t*>(b->genVertices);
  uint8_t* ptb = reinterpret_cast<uint8_t*>(b->partTriangles);

  // ---- :254-437 1X subset ----------------------------------------------------------
  if(subset)
  {
    const u32  vertexSize = subset_vertex_size(nv, simple);
    const u64  dataSize   = (u64)basic[simple];
    const u32  partSize   = subset_part_slots(simple);
    const u32  partOffset = back_alloc(x, y, partSize, k.maxPartTriangles);
    const bool ok         = fits(vertexSize, dataSize, partOffset, partSize);
    if(lane == 0)  // the vertex walk's record, per visible cluster with transient builds
      cs.fullRecs[v] = ok ? make_uint2(visIndex, vo) : make_uint2(kRejected, 0u);
    if(ok)
    {
      if(lane == 0)
      {
        store_clas_build(reinterpret_cast<tc_ClasBuildInfo*>(b->transBuilds) + tr, TC_RT_CLUSTER_MODE_1X_SUBSET_CLUSTER,
                         partOffset, simple, nv, b->positionTruncateBitCount, b->genVertices + (u64)vo * 12ull);
        reinterpret_cast<u32*>(b->transInstanceIDs)[tr]      = ci.instanceID;
        reinterpret_cast<u64*>(b->transClusterAddresses)[tr] = b->genClusterData + d;
        statTrans += 1;
        statTris += simple;
        atomicAdd(&blas[ci.instanceID].clusterReferencesCount, 1u);
      }
      // :489-535 indices after the vertices, triangle map after the header
      uint8_t* idx = gvb + ((u64)vo + nv) * 12;
      uint8_t* map = ptb + (u64)partOffset * kTessInfoBytes;
      warp_zero(idx, (simple * 3 + 11) / 12 * 3);
      warp_zero(map, partSize * kTessInfoBytes / 4);
      __syncwarp();
      if(lane == 0)
        *reinterpret_cast<uint2*>(map) = make_uint2(ci.instanceID, ci.clusterID);
      const u32* tw = cs.triWords + (u64)v * TC_MAX_CLUSTER_TRIANGLES;
      const uint8_t* lt = reinterpret_cast<const uint8_t*>(in->clusterLocalTriangles) + cl.firstLocalTriangle;
      u32 out = 0;
      for(u32 t0 = 0; t0 < nt; t0 += 32)
      {
        const u32  tri = t0 + lane;
        const bool sub = tri < nt && (tw[tri] & kWordSubset);
        const u32  bm  = __ballot_sync(0xFFFFFFFFu, sub);
        if(sub)
        {
          const u32 q = out + __popc(bm & ltm);
          map[kClusterInfoBytes + q] = (uint8_t)tri;
          idx[q * 3 + 0]            = lt[tri * 3 + 0];
          idx[q * 3 + 1]            = lt[tri * 3 + 1];
          idx[q * 3 + 2]            = lt[tri * 3 + 2];
        }
        out += __popc(bm);
      }
    }
    g += 1, vo += vertexSize, d += dataSize, tr += 1;
  }
  else if(lane == 0)
    cs.fullRecs[v] = make_uint2(kRejected, 0u);

  // ---- :543-905 the other triangles, one 32-triangle chunk at a time -------------
  const u32*   tw  = cs.triWords + (u64)v * TC_MAX_CLUSTER_TRIANGLES;
  tc_TessTriangleInfo* splits = reinterpret_cast<tc_TessTriangleInfo*>(b->splitTriangles);
  tc_TessTriangleInfo* parts  = reinterpret_cast<tc_TessTriangleInfo*>(b->partTriangles);
  for(u32 t0 = 0; t0 < nt; t0 += 32)
  {
    const u32  tri   = t0 + lane;
    const bool valid = tri < nt;
    const u32  word  = valid ? tw[tri] : 0u;
    const bool split = valid && (word & (1u << 18));
    const bool mini  = valid && (word & kWordMini);
    const bool part  = valid && !split && !mini && !(word & kWordSubset);
    const u32  bp = __ballot_sync(0xFFFFFFFFu, part), bs = __ballot_sync(0xFFFFFFFFu, split);
    const u32  bm = __ballot_sync(0xFFFFFFFFu, mini);
    // parts from the front of the two-sided counter: the chunk fits as a whole or not at all
    const u32  nPart   = __popc(bp);
    const bool frontOk = nPart != 0 && (u64)x + y + nPart + 1 <= k.maxPartTriangles;
    if(part && frontOk)
      emit_triangle(parts + x + __popc(bp & ltm), ci, tri, word);
    if(frontOk && lane == 0)  // the written front's end
      atomicMax(&b->partTriangleCounter, x + nPart);
    x += nPart;
    if(split)
    {
      const u64 so = (u64)s + __popc(bs & ltm);
      if(so < k.maxSplitTriangles)
      {
        emit_triangle(splits + so, ci, tri, word);
        const uint8_t* lt  = reinterpret_cast<const uint8_t*>(in->clusterLocalTriangles) + cl.firstLocalTriangle;
        const float*   pos = reinterpret_cast<const float*>(in->positions);
        float          m[16];
#pragma unroll
        for(int j = 0; j < 16; j++)
          m[j] = __ldg(in->worldMatrix.m + j);
        float* dd = c.splitBase + 9 * so;
#pragma unroll
        for(int vv = 0; vv < 3; vv++)
        {
          const f3 wp = xform_point(m, ldg3(pos, cl.firstLocalVertex + lt[tri * 3 + vv]));
          dd[3 * vv + 0] = wp.x, dd[3 * vv + 1] = wp.y, dd[3 * vv + 2] = wp.z;
        }
      }
    }
    s += __popc(bs);
    // :675-790 the chunk's 2X batches, kMiniBatch triangles each, in triangle
    // order. Batch q's offsets follow from the chunk's (every batch takes the
    // same amounts), so all of them are set up and written at once: lane by
    // lane for the base triangles, the batch's first triangle for the build.
    const u32 nMini = __popc(bm);
    if(nMini)
    {
      const u32  nb       = (nMini + kMiniBatch - 1) / kMiniBatch;
      const u64  dataSize = (u64)basic[kMiniBatchTris];
      const u32  rank = __popc(bm & ltm), q = rank / kMiniBatch, rel = rank % kMiniBatch;
      // the lanes of this lane's batch, the sum of their table triangles and this one's start
      const u32  group   = __match_any_sync(0xFFFFFFFFu, mini ? q : 0xFFFFFFFFu);
      const u32  ntris   = mini ? (u32)table_entry(c.table, word & 0xFFFFu).numTriangles : 0u;
      const u32  incl    = warp_inclusive<u32>(ntris, lane);
      const u32  first   = __shfl_sync(0xFFFFFFFFu, incl - ntris, __ffs(group) - 1);
      const u32  last    = __shfl_sync(0xFFFFFFFFu, incl, 31 - __clz(group));
      auto       back_of = [&](u32 qq) {  // build.glsl:52-66 for batch qq of the chunk
        const u32 yq = y + kMiniPartSlots * qq;
        return ((u64)x + yq + kMiniPartSlots + 1 > k.maxPartTriangles) ? k.maxPartTriangles
                                                                        : k.maxPartTriangles - yq - kMiniPartSlots;
      };
      auto fits_q = [&](u32 qq) {
        const u32 po = back_of(qq);
        return !((u64)vo + kMiniVertexSize * (qq + 1) > k.maxGeneratedVertices
                 || (u64)g + qq + 1 > k.maxGeneratedClusters || d + dataSize * (qq + 1) > maxData
                 || (u64)po + kMiniPartSlots > k.maxPartTriangles);
      };
      for(u32 qq = 0; qq < nb; qq++)  // zero the accepted batches' regions
        if(fits_q(qq))
        {
          warp_zero(gvb + ((u64)vo + kMiniVertexSize * qq) * 12, kMiniVertexSize * 3);
          warp_zero(ptb + (u64)back_of(qq) * kTessInfoBytes, kMiniPartSlots * kTessInfoBytes / 4);
        }
      __syncwarp();
      if(mini && fits_q(q))
      {
        const u32 vq = vo + kMiniVertexSize * q, po = back_of(q);
        if(rel == 0)
        {
          const u32 trq = tr + q;
          store_clas_build(reinterpret_cast<tc_ClasBuildInfo*>(b->transBuilds) + trq,
                           TC_RT_CLUSTER_MODE_2X_BATCHED_TESSELLATED, po, last - first, kMiniBatchVerts,
                           b->positionTruncateBitCount, b->genVertices + (u64)vq * 12ull);
          reinterpret_cast<u32*>(b->transInstanceIDs)[trq]      = ci.instanceID;
          reinterpret_cast<u64*>(b->transClusterAddresses)[trq] = b->genClusterData + d + dataSize * q;
          *reinterpret_cast<uint2*>(ptb + (u64)po * kTessInfoBytes) = make_uint2(ci.instanceID, ci.clusterID);
          atomicAdd(&blas[ci.instanceID].clusterReferencesCount, 1u);
          statTrans += 1;
          statTris += last - first;
        }
        mini_indices(c, tri, word, rel, incl - ntris - first, vq, po);
      }
      g += nb, vo += kMiniVertexSize * nb, d += dataSize * nb, tr += nb, y += kMiniPartSlots * nb;
    }
  }
}

// The offsets at which block `blockIdx.x` of the write launch starts, with
// transient builds (the seven counters of TransOffsets).
__device__ inline void block_prefix_transient(const ClassifyScratch& cs, u64 (&pre)[kTNum], u64 (*s_warp)[kTNum])
{
  u64 x[kTNum] = {0, 0, 0, 0, 0, 0, 0};
  for(u32 i = threadIdx.x; i < blockIdx.x; i += blockDim.x)
  {
    const RangeSums o = cs.rangeSums[i];
    x[kTFront] += (u32)o.partsSplits;
    x[kTSplit] += (u32)(o.partsSplits >> 32);
    x[kTGen] += (u32)o.fullVerts;
    x[kTVert] += (u32)(o.fullVerts >> 32);
    x[kTData] += o.data;
    x[kTBack] += (u32)o.backTrans;
    x[kTTrans] += (u32)(o.backTrans >> 32);
  }
  u64 tot[kTNum];
  block_scan_n<kTNum>(x, tot, s_warp);
  const ClusterOffsets b0 = *cs.bases;
  const TransBases     t0 = *reinterpret_cast<const TransBases*>(cs.bases + 1);
  pre[kTFront] = b0.part + tot[kTFront];
  pre[kTSplit] = b0.split + tot[kTSplit];
  pre[kTGen]   = b0.gen + tot[kTGen];
  pre[kTVert]  = b0.vert + tot[kTVert];
  pre[kTData]  = b0.data + tot[kTData];
  pre[kTBack]  = t0.back + tot[kTBack];
  pre[kTTrans] = t0.trans + tot[kTTrans];
}

// The offsets of every cluster, the full clusters' arguments (32 clusters at a
// time, one per lane, like k_classify_write), and a list of the others, which
// k_classify_emit_transient takes one per warp: a cluster with 1X and 2X builds
// takes a warp about 10 us of dependent steps, and the visible, tessellated
// clusters lie next to each other in the list, so a block that wrote its own
// range's clusters had up to 57 of them while most blocks had none.
// Measured on a GB300, 51,840 clusters of 256 instances, 1,217 of them partly
// tessellated: 79 us from the count's end to the last write in one kernel,
// 31 us in two. Not Listed (a range has no more clusters than warps): the range's
// warps write them, without the second launch (24 instances with every option
// 66.5 -> 60.9 us a frame, 34 with transient builds 68.5 -> 62.2; at two clusters
// to a warp, 60 instances, 80.6 with the list and 82.7 without).
template <bool Listed>
__global__ void __launch_bounds__(kBlock, Listed ? 6 : 4) k_classify_write_transient(StageCtx c, ClassifyScratch cs)
{
  stage_prologue();
  __shared__ u32            s_range[2];
  __shared__ u64            s_warp[33][kTNum];
  __shared__ TransOffsets   s_off[kBlock];
  __shared__ uint4          s_cnt[kBlock];
  __shared__ tc_ClusterInfo s_ci[kBlock];
  __shared__ FlatStarts     s_starts;
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if(threadIdx.x == 0)
    window_range(c, s_range[0], s_range[1]);
  __syncthreads();
  const u32* starts = stage_flat_starts(c, s_starts);
  const u32  begin  = s_range[0];
  const u32  n      = min(s_range[1] - s_range[0], c.scratch.itemCapacity);
  tc_SceneBuilding*     b   = c.build;
  const tc_ClusterInfo* vis = reinterpret_cast<const tc_ClusterInfo*>(b->visibleClusters);
  const uint4*          counts = reinterpret_cast<const uint4*>(cs.counts);
  const tc_caps&        k       = c.caps;
  const u64             maxData = (u64)k.maxGeneratedClusterMegs * 1024ull * 1024ull;
  tc_BlasBuildInfo*     blas    = reinterpret_cast<tc_BlasBuildInfo*>(b->blasBuildInfos);
  u32                   statTemp = 0, statTris = 0, statTrans = 0;

  u64 pre[kTNum];
  block_prefix_transient(cs, pre, s_warp);
  const u32        genBase = cs.bases->gen;
  const TransBases tb      = *reinterpret_cast<const TransBases*>(cs.bases + 1);
  u32              vBegin, vEnd;
  block_range(n, blockIdx.x, gridDim.x, vBegin, vEnd);
  for(u32 c0 = vBegin; c0 < vEnd; c0 += kBlock)
  {
    const u32 len = min(kBlock, vEnd - c0);
    {
      const uint4 r = threadIdx.x < len ? counts[c0 + threadIdx.x] : make_uint4(0, 0, 0, 0);
      if(threadIdx.x < len)
        s_ci[threadIdx.x] = visible_cluster(c, starts, vis, begin + c0 + threadIdx.x);
      u64 x[kTNum] = {t_parts(r), t_splits(r), t_gen(r), t_verts(r), r.z, t_back(r), t_trans(r)};
      u64 tot[kTNum];
      block_scan_n<kTNum>(x, tot, s_warp);
      s_cnt[threadIdx.x] = r;
      s_off[threadIdx.x] = {(u32)(pre[kTFront] + x[kTFront]), (u32)(pre[kTSplit] + x[kTSplit]),
                            (u32)(pre[kTGen] + x[kTGen]),     (u32)(pre[kTVert] + x[kTVert]),
                            (u32)(pre[kTBack] + x[kTBack]),   (u32)(pre[kTTrans] + x[kTTrans]),
                            pre[kTData] + x[kTData]};
#pragma unroll
      for(int q = 0; q < kTNum; q++)
        pre[q] += tot[q];
    }
    __syncthreads();
    const u32 perW = (len + kWarps - 1) / kWarps;
    const u32 lo = min(len, warp * perW), hi = min(len, lo + perW);
    for(u32 i0 = lo; i0 < hi; i0 += 32)
    {
      const u32  i       = i0 + lane;
      const bool valid   = i < hi;
      const uint4 r      = valid ? s_cnt[i] : make_uint4(0u, 0u, 0u, 0u);
      const bool isFull  = valid && t_full(r);
      u32        inst    = 0xFFFFFFFFu;
      bool       full    = false;
      // cluster_classify.comp.glsl:254-437, full clusters
      if(isFull)
      {
        const TransOffsets o = s_off[i];
        full = !((u64)o.vert + t_nv(r) > k.maxGeneratedVertices || (u64)o.gen + 1 > k.maxGeneratedClusters
                 || o.data + r.z > maxData);
        cs.fullRecs[c0 + i] = full ? make_uint2(begin + c0 + i, o.vert) : make_uint2(kRejected, 0u);
        if(full)
        {
          const tc_ClusterInfo       ci = s_ci[i];
          const tc_RenderInstance*   in = c.instances + ci.instanceID;
          const u32                  tempOffset = tb.temp + (o.gen - genBase) - (o.trans - tb.trans);
          tc_TemplateInstantiateInfo ti;
          ti.clusterIdOffset        = 0;
          ti.geometryIndexOffset    = 0;
          ti.clusterTemplateAddress = __ldg(reinterpret_cast<const u64*>(in->clusterTemplateAdresses) + ci.clusterID);
          ti.vertexBufferAddress    = b->genVertices + (u64)o.vert * 12ull;
          ti.vertexBufferStride     = 12;
          reinterpret_cast<tc_TemplateInstantiateInfo*>(b->tempInstantiations)[tempOffset] = ti;
          reinterpret_cast<u32*>(b->tempInstanceIDs)[tempOffset]                          = ci.instanceID;
          reinterpret_cast<u64*>(b->tempClusterAddresses)[tempOffset]                     = b->genClusterData + o.data;
          if((c.flags & TC_FLAG_WRITE_FULLCLUSTERS) && b->fullClusters)
            reinterpret_cast<tc_ClusterInfo*>(b->fullClusters)[tempOffset] = ci;
          statTemp += 1;
          statTris += t_simple(r);
          inst = ci.instanceID;
        }
      }
      // CLAS reference counts: one atomic per distinct instance of the batch
      for(u32 remaining = __ballot_sync(0xFFFFFFFFu, full); remaining;)
      {
        const int src = __ffs(remaining) - 1;
        const u32 gk  = __shfl_sync(0xFFFFFFFFu, inst, src);
        const u32 sel = __ballot_sync(0xFFFFFFFFu, full && inst == gk);
        remaining &= ~sel;
        if((int)lane == src)
          atomicAdd(&blas[gk].clusterReferencesCount, __popc(sel));
      }
      const u32 others = __ballot_sync(0xFFFFFFFFu, valid && !isFull);
      if constexpr(!Listed)
      {
        for(u32 left = others; left; left &= left - 1)
        {
          const u32 k = i0 + (u32)__ffs(left) - 1;
          write_cluster_transient(c, cs, begin + c0 + k, c0 + k, s_ci[k], s_cnt[k], s_off[k], statTrans, statTris);
        }
      }
      else if(others)
      {
        u32 at = 0;
        if(lane == 0)
          at = atomicAdd(cs.fullRange + 2, __popc(others));
        at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(others & ((1u << lane) - 1u));
        if(valid && !isFull)
        {
          const TransOffsets o   = s_off[i];
          uint4*             rec = cs.transRecs + 3 * (u64)at;
          rec[0]                 = make_uint4(c0 + i, s_ci[i].instanceID, s_ci[i].clusterID, o.front);
          rec[1]                 = make_uint4(o.split, o.gen, o.vert, o.back);
          rec[2]                 = make_uint4(o.trans, (u32)o.data, (u32)(o.data >> 32), 0u);
        }
      }
    }
    __syncthreads();
  }
  statTemp  = __reduce_add_sync(0xFFFFFFFFu, statTemp);
  statTris  = __reduce_add_sync(0xFFFFFFFFu, statTris);
  statTrans = __reduce_add_sync(0xFFFFFFFFu, statTrans);
  if(lane == 0)
  {
    if(statTemp)
      atomicAdd(&b->tempInstantiateCounter, statTemp);
    if(statTrans)
      atomicAdd(&b->transBuildCounter, statTrans);
    if(statTris)
      atomicAdd(&c.readback->numTotalTriangles, statTris);
  }
  if(blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
  {
    cs.fullRange[0] = 0;  // the walk's records are per visible cluster here
    cs.fullRange[1] = n;
    if(n)
    {
      const ClusterOffsets b0 = *cs.bases;
      b->dualPartTriangleCounter = (u64)(u32)pre[kTFront] | ((u64)(u32)pre[kTBack] << 32);
      b->splitTriangleCounter    = (int32_t)(u32)pre[kTSplit];
      b->genClusterCounter       = (u32)pre[kTGen];
      b->genVertexCounter        = (u32)pre[kTVert];
      b->genClusterDataCounter   = pre[kTData];
      // :299 counts every full-cluster attempt; the full attempts also bound
      // the full clusters' run of the instantiation list
      const u32 fullAttempts = ((u32)pre[kTGen] - b0.gen) - ((u32)pre[kTTrans] - tb.trans);
      c.readback->numFullClusters += fullAttempts;
      c.runStarts[kFullAttemptsSlot] += fullAttempts;
    }
    if(c.fuseSetup != kNoSetup)
      build_setup_apply(c, c.fuseSetup);
  }
}

// The clusters k_classify_write_transient listed: warps stride over them.
__global__ void __launch_bounds__(kBlock, 4) k_classify_emit_transient(StageCtx c, ClassifyScratch cs)
{
  stage_prologue();
  __shared__ u32 s_range[2];
  if(threadIdx.x == 0)
    window_range(c, s_range[0], s_range[1]);
  __syncthreads();
  const u32 begin = s_range[0], count = cs.fullRange[2];
  const u32 lane = threadIdx.x & 31, nwarps = (gridDim.x * blockDim.x) >> 5;
  u32       statTrans = 0, statTris = 0;
  for(u32 i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < count; i += nwarps)
  {
    const uint4*         rec = cs.transRecs + 3 * (u64)i;
    const uint4          a = rec[0], b = rec[1], d = rec[2];
    const tc_ClusterInfo ci = {a.y, a.z};
    const TransOffsets   o  = {a.w, b.x, b.y, b.z, b.w, d.x, (u64)d.y | ((u64)d.z << 32)};
    write_cluster_transient(c, cs, begin + a.x, a.x, ci, reinterpret_cast<const uint4*>(cs.counts)[a.x], o, statTrans,
                            statTris);
  }
  statTrans = __reduce_add_sync(0xFFFFFFFFu, statTrans);
  statTris  = __reduce_add_sync(0xFFFFFFFFu, statTris);
  if(lane == 0)
  {
    if(statTrans)
      atomicAdd(&c.build->transBuildCounter, statTrans);
    if(statTris)
      atomicAdd(&c.readback->numTotalTriangles, statTris);
  }
}

// cluster_classify.comp.glsl:810-878: the vertices of the launch's accepted 2X
// batches, from their build records: the batch's base triangles are the first
// entries of its triangle map (table triangle 0), whose edge factors give the
// configuration. A warp takes two builds at a time (one lane per base
// triangle), one when there are not enough for every warp, then one lane per
// vertex (3 to 6 per base triangle; tc_deform.cuh).
__global__ void __launch_bounds__(kDeformBlock, kDeformBlocksPerSM) k_classify_mini_vertices(StageCtx c, ClassifyScratch cs)
{
  stage_prologue();
  __shared__ DeformRecords s_rec[kDeformWarps];
  __shared__ uint4         s_lane[kDeformWarps][32];
  const u32                lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ltm = (1u << lane) - 1u;
  const tc_SceneBuilding*  b      = c.build;
  const tc_ClasBuildInfo*  builds = reinterpret_cast<const tc_ClasBuildInfo*>(b->transBuilds);
  const uint8_t*           ptb    = reinterpret_cast<const uint8_t*>(b->partTriangles);
  float*                   gv     = reinterpret_cast<float*>(b->genVertices);
  const bool               pn     = (c.flags & TC_FLAG_PN) != 0;
  const RippleParams       rp     = ripple_params(*c.view, (c.flags & TC_FLAG_RIPPLE) != 0);
  // accepted builds take consecutive slots after those before the launch
  const u32 first = reinterpret_cast<const TransBases*>(cs.bases + 1)->trans;
  const u32 count = max(b->transBuildCounter, first) - first;
  const u32 nwarps = (gridDim.x * blockDim.x) >> 5;
  u32       per    = kDeformParts / kMiniBatch;
  while(per > 1 && (count + per / 2 - 1) / (per / 2) <= nwarps)
    per >>= 1;
  DeformRecords& rec = s_rec[warp];
  for(u32 k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k * per < count; k += nwarps)
  {
    // lane's base triangle: number lane % 8 of build lane / 8
    const u32 j    = k * per + lane / kMiniBatch, rel = lane % kMiniBatch;
    u32       part = 0, vo = 0, ntri = 0;
    bool      take = false;
    if(lane / kMiniBatch < per && j < count)
    {
      const tc_ClasBuildInfo& bi = builds[first + j];
      part = bi.clusterID & 0x3FFFFFFFu;
      ntri = bi.packed & 0x1FFu;
      vo   = (u32)((bi.vertexBuffer - b->genVertices) / 12);
      take = bi.clusterID >> 30 == TC_RT_CLUSTER_MODE_2X_BATCHED_TESSELLATED;
    }
    // the rel-th of the map's entries that start a base triangle: each of the
    // build's lanes tests four of the 32 entries
    const uint16_t* map    = reinterpret_cast<const uint16_t*>(ptb + (u64)part * kTessInfoBytes + kClusterInfoBytes);
    u32             starts = 0;
    if(take)
    {
      const uint2 e = reinterpret_cast<const uint2*>(map)[rel];
#pragma unroll
      for(u32 i = 0; i < 4; i++)
        if(4 * rel + i < ntri && (((i & 2 ? e.y : e.x) >> (16 * (i & 1) + 8)) & 3u) == 0)
          starts |= 1u << (4 * rel + i);
    }
    starts = __reduce_or_sync(0xFFu << (lane & 24u), starts);
    for(u32 i = 0; i < rel; i++)
      starts &= starts - 1;
    const bool found = starts != 0;
    const u32  word  = found ? map[__ffs(starts) - 1] : 0u;
    const u32 tm = __ballot_sync(0xFFFFFFFFu, found);
    if(found)
    {
      const uint2              hdr = *reinterpret_cast<const uint2*>(ptb + (u64)part * kTessInfoBytes);
      const tc_RenderInstance& in  = c.instances[hdr.x];
      const tc_Cluster         cl  = reinterpret_cast<const tc_Cluster*>(in.clusters)[hdr.y];
      u32                      corner[3] = {0u, TC_TESSTABLE_COORD_MAX, TC_TESSTABLE_COORD_MAX << 16};
      const u32                cfg = get_config(make_uint3(1u + ((word >> 12) & 1u), 1u + ((word >> 13) & 1u), 1u + ((word >> 14) & 1u)),
                                                corner[0], corner[1], corner[2]);
      const tc_TessTableEntry  e    = table_entry(c.table, cfg);
      const u32                slot = __popc(tm & ltm);
      setup_deform(c, in, cl, word & 0xFFu, cfg, corner, e.firstVertex, pn, rec.affine[slot], rec.pn[slot]);
      s_lane[warp][slot] = make_uint4(e.firstVertex | (u32)e.numVertices << 16, vo + rel * TC_2X_MINI_VERTICES, hdr.x,
                                      __float_as_uint(in.geoHi.w));
    }
    __syncwarp();
    const u32        owners = __popc(tm);
    const uint4      l      = lane < owners ? s_lane[warp][lane] : make_uint4(0u, 0u, 0u, 0u);
    const DeformLane d      = {l.x >> 16, l.x & 0xFFFFu, l.y, l.z, __uint_as_float(l.w)};
    deform_walk(c, rec, owners, d, pn, rp, gv);
    __syncwarp();  // the records are rewritten by the warp's next builds
  }
}

// ---------------------------------------------------------------------------
// full clusters' vertices
// ---------------------------------------------------------------------------

// cluster_classify.comp.glsl:457-482: the displaced vertices of the full
// clusters the write launch accepted. A warp takes `per` <= 32 consecutive
// records (per: the records spread over all of the grid's warps): one lane per
// cluster, then the clusters' vertex ranges, contiguous in genVertices, are
// walked on consecutive lanes.
__device__ __forceinline__ void full_slots(const StageCtx& c, const ClassifyScratch& cs, const u32* starts,
                                           FullRecord* rec, float* gv, const RippleParams& rp)
{
  const u32             lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const u32             count        = cs.fullRange[1] - cs.fullRange[0];
  const u32             totalWarps   = gridDim.x * kWarps;
  const u32             per          = min(32u, max(1u, (count + totalWarps - 1) / totalWarps));
  const u32             numChunks    = (count + per - 1) / per;
  const tc_ClusterInfo* vis          = reinterpret_cast<const tc_ClusterInfo*>(c.build->visibleClusters);
  for(u32 chunk = blockIdx.x * kWarps + warp; chunk < numChunks; chunk += totalWarps)
  {
    const u32  slot  = chunk * per + lane;
    bool       owner = false;
    FullRecord fr;
    if(lane < per && slot < count)
    {
      const uint2 fs = cs.fullRecs[slot];
      if(fs.x != kRejected)
      {
        owner = true;
        fr    = full_record(c, visible_cluster(c, starts, vis, fs.x), fs.y);
      }
    }
    full_batch(rec, owner, fr, gv, rp);
    __syncwarp();  // records are rewritten by the next batch
  }
}

// Its own launch so that it can overlap other work.
template <int MinBlocks>
__global__ void __launch_bounds__(kBlock, MinBlocks) k_classify_full_vertices(StageCtx c, ClassifyScratch cs)
{
  stage_prologue();
  __shared__ FullRecord s_full[kWarps][32];
  __shared__ FlatStarts s_starts;
  const u32*            starts = stage_flat_starts(c, s_starts);
  full_slots(c, cs, starts, s_full[threadIdx.x >> 5], reinterpret_cast<float*>(c.build->genVertices),
             ripple_params(*c.view, (c.flags & TC_FLAG_RIPPLE) != 0));
}

// The same vertices by instance groups (find_groups). They are in object
// space, so instances of one mesh, map, scale and offset have the same ones:
// a warp evaluates a cluster's vertices once for a subgroup and stores them for
// each member whose cluster is a full one, as consecutive words. One at a
// time, the walk above reads 32 bytes of attributes and its texel sectors for
// each vertex through L2, which bounds it (about 9 TB/s). Measured on a GB300:
// 2.4 M vertices of 256 instances 34 -> 14 us, 9.9 M of 1,024 instances
// 115 -> 35 us (the frames 109 -> 101 and 287 -> 233 us). Under the ripple,
// which differs by instance, the lanes take (member, vertex) pairs.
__global__ void __launch_bounds__(kBlock, 4) k_classify_full_groups(StageCtx c, ClassifyScratch cs)
{
  stage_prologue();
  __shared__ union
  {
    FullRecord full[kWarps][32];
    float      words[kWarps][3 * TC_MAX_CLUSTER_VERTICES];
  } s;
  __shared__ uint2      s_member[kWarps][kGroupMembers];
  __shared__ FlatStarts s_starts;
  const u32*            starts = stage_flat_starts(c, s_starts);
  const u32             lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float*                gv   = reinterpret_cast<float*>(c.build->genVertices);
  const RippleParams    rp   = ripple_params(*c.view, (c.flags & TC_FLAG_RIPPLE) != 0);
  if(cs.groupHead[kHeadGrouped] == 0)
  {
    full_slots(c, cs, starts, s.full[warp], gv, rp);
    return;
  }
  const u32 subs = cs.groupHead[kHeadSubgroups], tasks = cs.groupHead[kHeadTasks], n = cs.fullRange[1];
  const u32 gwarp = blockIdx.x * kWarps + warp, nwarps = gridDim.x * kWarps;
  float*    words = s.words[warp];
  for(u32 t0 = gwarp; t0 < tasks; t0 += 32 * nwarps)
  {
    // lane's task t0 + lane * nwarps: its representative instance, cluster and
    // the members' first vertices (~0: the cluster is not a full one there)
    u32        rep = 0, firstV = 0, nv = 0, member = 0;
    u32        vo[kGroupMembers];
    const u64  t     = (u64)t0 + (u64)lane * nwarps;
    const bool valid = t < tasks;
#pragma unroll
    for(u32 m = 0; m < kGroupMembers; m++)
      vo[m] = ~0u;
    if(valid)
    {
      u32 lo = 0, hi = subs;  // the last subgroup whose first task is at most t
      while(hi - lo > 1)
      {
        const u32 mid = (lo + hi) >> 1;
        if(cs.groups[mid].x <= (u32)t)
          lo = mid;
        else
          hi = mid;
      }
      const uint4      g  = cs.groups[lo];
      const u32        k  = (u32)t - g.x;
      const tc_Cluster cl = reinterpret_cast<const tc_Cluster*>(c.instances[g.w].clusters)[k];
      rep = g.w, member = g.y, firstV = cl.firstLocalVertex;
      nv  = min((u32)cl.numVertices, TC_MAX_CLUSTER_VERTICES);
      u32 v[kGroupMembers];
#pragma unroll
      for(u32 m = 0; m < kGroupMembers; m++)
        v[m] = m < g.z ? starts[cs.members[g.y + m]] + k : ~0u;
#pragma unroll
      for(u32 m = 0; m < kGroupMembers; m++)
        if(v[m] < n)
        {
          const uint2 r = cs.fullRecs[v[m]];
          vo[m]         = r.x != kRejected ? r.y : ~0u;
        }
    }
    bool any = false;
#pragma unroll
    for(u32 m = 0; m < kGroupMembers; m++)
      any |= vo[m] != ~0u;
    for(u32 left = __ballot_sync(0xFFFFFFFFu, any); left; left &= left - 1)
    {
      const int  src = __ffs(left) - 1;
      const u32  cv  = __shfl_sync(0xFFFFFFFFu, nv, src);
      FullRecord fr  = full_attributes(c, __shfl_sync(0xFFFFFFFFu, rep, src));
      fr.first       = __shfl_sync(0xFFFFFFFFu, firstV, src);
      for(u32 i = lane; i < cv; i += 32)
      {
        const f3 p = full_vertex(fr, i);
        words[3 * i] = p.x, words[3 * i + 1] = p.y, words[3 * i + 2] = p.z;
      }
      if(rp.enabled)  // cluster_classify.comp.glsl:483-485: by instance; the lanes take (member, vertex) pairs
      {
        u32 count = 0;
#pragma unroll
        for(u32 m = 0; m < kGroupMembers; m++)
          if((int)lane == src && vo[m] != ~0u)
            s_member[warp][count++] = make_uint2(vo[m], member + m);
        count = __shfl_sync(0xFFFFFFFFu, count, src);
        __syncwarp();
        u32   first = 0, inst = 0;
        float size = 0.0f;
        if(lane < count)
        {
          first = s_member[warp][lane].x;
          inst  = cs.members[s_member[warp][lane].y];
          size  = c.instances[inst].geoHi.w;
        }
        u32 m = 0, i = lane;
        for(u32 base = 0; base < count * cv; base += 32, i += 32)
        {
          for(; i >= cv; i -= cv)
            m++;
          const u32   mFirst = __shfl_sync(0xFFFFFFFFu, first, m & 31), mInst = __shfl_sync(0xFFFFFFFFu, inst, m & 31);
          const float mSize  = __shfl_sync(0xFFFFFFFFu, size, m & 31);
          if(m < count)
          {
            const f3 q = ripple({words[3 * i], words[3 * i + 1], words[3 * i + 2]}, mInst, mSize, rp);
            float*   d = gv + 3 * ((u64)mFirst + i);
            d[0] = q.x, d[1] = q.y, d[2] = q.z;
          }
        }
      }
      else
      {
        __syncwarp();
        float w[6];
#pragma unroll
        for(u32 q = 0; q < 6; q++)
          w[q] = lane + 32 * q < 3 * cv ? words[lane + 32 * q] : 0.0f;
#pragma unroll
        for(u32 m = 0; m < kGroupMembers; m++)
        {
          const u32 first = __shfl_sync(0xFFFFFFFFu, vo[m], src);
          if(first == ~0u)
            continue;
          float* dst = gv + 3 * (u64)first;
#pragma unroll
          for(u32 q = 0; q < 6; q++)
            if(lane + 32 * q < 3 * cv)
              dst[lane + 32 * q] = w[q];
        }
      }
      __syncwarp();  // the words are rewritten by the warp's next cluster
    }
  }
}

}  // namespace

cudaError_t launch_cluster_classify(const StageCtx& c, const ClassifyBuffers& buf, u32 maxClusters, u32 numSMs,
                                    u32 warpBlocksPerSM, cudaStream_t s)
{
  // the write launch's blocks own contiguous ranges of clusters, whose count
  // sums the count launch accumulates (its warps stride over the whole list)
  const u32 grid = std::max(1u, std::min(classify_max_blocks(maxClusters), numSMs * std::max(1u, warpBlocksPerSM)));
  ClassifyScratch cs{buf.counts, buf.triWords, buf.rangeSums, buf.bases, grid, 0, buf.fullRecs, buf.fullRange, buf.groups.groups,
                     buf.groups.members, buf.groups.head, buf.groups.instBounds, buf.groups.bounds, buf.transRecs};
  const u32 wholeGrid = std::max(1u, std::min((maxClusters + kBlock - 1) / kBlock, numSMs * 8));
  // register budget from the requested residency: 4 or less -> 64, 5-7 -> 40, 8 and more -> 32
  if(c.flags & (TC_FLAG_TRANSIENT_1X | TC_FLAG_TRANSIENT_2X))
  {
    // the transient write is latency-bound per cluster: a full wave of its
    // six resident blocks per SM (the count uses the same ranges)
    const u32  tgrid  = std::max(1u, std::min(classify_max_blocks(maxClusters), numSMs * std::max(6u, warpBlocksPerSM)));
    const bool listed = classify_lists_clusters(maxClusters, numSMs, warpBlocksPerSM, true);
    ClassifyScratch ts = cs;
    ts.writeBlocks     = tgrid;
    cudaError_t e      = cs.groups ? launch_pdl_critical(k_classify_whole<true>, wholeGrid, kBlock, s, c, ts) : cudaSuccess;
    if(e != cudaSuccess)
      return e;
    e = launch_pdl_critical(k_classify_count<4, true>, tgrid, kBlock, s, c, ts);
    if(e != cudaSuccess)
      return e;
    e = listed ? launch_pdl_critical(k_classify_write_transient<true>, tgrid, kBlock, s, c, ts)
               : launch_pdl_critical(k_classify_write_transient<false>, tgrid, kBlock, s, c, ts);
    if(e != cudaSuccess || !listed)
      return e;
    const u32 egrid = std::max(1u, std::min((maxClusters + kWarps - 1) / kWarps, numSMs * 4));
    return launch_pdl_critical(k_classify_emit_transient, egrid, kBlock, s, c, ts);
  }
  cs.listed       = classify_lists_clusters(maxClusters, numSMs, warpBlocksPerSM, false) ? 1u : 0u;
  const int   occ = warpBlocksPerSM >= 8 ? 8 : (warpBlocksPerSM >= 5 ? 6 : 4);
  cudaError_t e   = cs.groups ? launch_pdl_critical(k_classify_whole<false>, wholeGrid, kBlock, s, c, cs) : cudaSuccess;
  if(e != cudaSuccess)
    return e;
  e = occ == 8   ? launch_pdl_critical(k_classify_count<8>, grid, kBlock, s, c, cs)
      : occ == 6 ? launch_pdl_critical(k_classify_count<6>, grid, kBlock, s, c, cs)
                 : launch_pdl_critical(k_classify_count<4>, grid, kBlock, s, c, cs);
  if(e != cudaSuccess)
    return e;
  e = occ == 8   ? launch_pdl_critical(k_classify_write<8>, grid, kBlock, s, c, cs)
      : occ == 6 ? launch_pdl_critical(k_classify_write<6>, grid, kBlock, s, c, cs)
                 : launch_pdl_critical(k_classify_write<4>, grid, kBlock, s, c, cs);
  if(e != cudaSuccess || !cs.listed)
    return e;
  const u32 egrid = std::max(1u, std::min((maxClusters + kWarps - 1) / kWarps, numSMs * 4));
  return launch_pdl_critical(k_classify_emit, egrid, kBlock, s, c, cs);
}

cudaError_t launch_cluster_bounds(const StageCtx& c, const GroupTables& g, u32 numSMs, cudaStream_t s)
{
  const u32 grid = std::max(1u, std::min((g.boundsCap + kWarps - 1) / kWarps, numSMs * 4));
  return launch_pdl_critical(k_cluster_bounds, grid, kBlock, s, c, g);
}

cudaError_t launch_classify_full_vertices(const StageCtx& c, const ClassifyBuffers& buf, u32 maxClusters, u32 numSMs,
                                          u32 blocksPerSM, cudaStream_t s)
{
  ClassifyScratch cs{buf.counts, buf.triWords, buf.rangeSums, buf.bases, 0, 0, buf.fullRecs, buf.fullRange, buf.groups.groups,
                     buf.groups.members, buf.groups.head, buf.groups.instBounds, buf.groups.bounds, buf.transRecs};
  // every warp of the grid takes a share of the slots
  const u32 grid = std::max(1u, std::min((maxClusters + kWarps - 1) / kWarps, numSMs * std::max(1u, blocksPerSM)));
  // register budget from the requested residency: 4 or less -> 64, 5-6 -> 40, 7 and more -> 32
  cudaError_t e = cs.groups          ? launch_pdl(k_classify_full_groups, grid, kBlock, s, c, cs)
                  : blocksPerSM >= 7 ? launch_pdl(k_classify_full_vertices<8>, grid, kBlock, s, c, cs)
                  : blocksPerSM >= 5 ? launch_pdl(k_classify_full_vertices<6>, grid, kBlock, s, c, cs)
                                     : launch_pdl(k_classify_full_vertices<4>, grid, kBlock, s, c, cs);
  if(e != cudaSuccess || !(c.flags & TC_FLAG_TRANSIENT_2X))
    return e;
  // the 2X batches' vertices (at most eight builds per cluster): warps stride
  // over the builds, one resident wave of the kernel's blocks (less kDeformRoom)
  const u32 miniGrid = std::max(1u, std::min((maxClusters * 8 + kDeformWarps - 1) / kDeformWarps, numSMs * (u32)(kDeformBlocksPerSM - kDeformRoom)));
  return launch_pdl(k_classify_mini_vertices, miniGrid, kDeformBlock, s, c, cs);
}

bool classify_lists_clusters(u32 maxClusters, u32 numSMs, u32 warpBlocksPerSM, bool transient)
{
  return transient ? maxClusters > (u64)kWarps * numSMs * std::max(6u, warpBlocksPerSM)
                   : maxClusters > 32ull * numSMs * std::max(1u, warpBlocksPerSM);
}

u32 classify_max_blocks(u32 maxClusters) { return std::max(1u, (maxClusters + kWarps - 1) / kWarps); }

}  // namespace tc
