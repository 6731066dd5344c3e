// tc_raster.cu — raster-style batching of the frame's part triangles:
// render_raster_clusters_batched.task.glsl:115-215 (the linear fill of 32
// parts into batches of <= 96 vertices and <= 121 triangles) and
// render_raster_clusters_batched.mesh.glsl:141-435 (the batch's displaced
// vertices in world and clip space, its triangles' local indices and
// primitive IDs) as compute kernels writing plain vertex and index arrays.
//
// Three launches: per group of 32 parts (one warp) its batch, vertex and
// triangle counts; one block scans the groups' counts into offsets; per group
// again the batch records, then the group's vertices and triangles, each as
// one contiguous range over which the lanes take consecutive elements.
#include "tc_deform.cuh"
#include <type_traits>

#include "tc_kernels.h"
#include "tc_stage.cuh"
#include "tc_vertex.cuh"

namespace tc {

namespace {

constexpr u32 kRasterBlock = 256;  // counts
constexpr u32 kWriteBlock  = 128;  // k_raster_write: its part records fill the shared memory of a block
constexpr u32 kWriteWarps  = kWriteBlock / 32;

// the group's parts: per lane (part g0 + lane) its inclusive vertex and
// triangle sums; lanes past the parts count as a full batch (they never fit)
struct GroupSums
{
  u32 v, t;        // this lane's part
  u32 sumV, sumT;  // inclusive
};

__device__ __forceinline__ GroupSums group_sums(const StageCtx& c, u32 g0, u32 local)
{
  const u32                  lane  = threadIdx.x & 31;
  const tc_TessTriangleInfo* parts = reinterpret_cast<const tc_TessTriangleInfo*>(c.build->partTriangles);
  GroupSums                  s;
  s.v = TC_RASTER_BATCH_VERTICES, s.t = TC_RASTER_BATCH_TRIANGLES;
  if(lane < local)
  {
    const tc_TessTableEntry e = table_entry(c.table, parts[g0 + lane].subTriangle.triangleID_config >> 16);
    s.v = e.numVertices, s.t = e.numTriangles;
  }
  s.sumV = s.v, s.sumT = s.t;
#pragma unroll
  for(int d = 1; d < 32; d <<= 1)
  {
    const u32 a = __shfl_up_sync(0xFFFFFFFFu, s.sumV, d), b = __shfl_up_sync(0xFFFFFFFFu, s.sumT, d);
    if(lane >= (u32)d)
      s.sumV += a, s.sumT += b;
  }
  return s;
}

// task.glsl:150-205: batch q's last part (its end) for every batch, calling
// fn(q, start, end, vertices before start, triangles before start)
template <class F>
__device__ __forceinline__ u32 group_batches(const GroupSums& s, u32 local, F&& fn)
{
  u32 start = 0, lastV = 0, lastT = 0, left = local, q = 0;
  while(left != 0 && q < 32)
  {
    // unsigned differences: parts before the batch do not fit
    const u32 fit = __ballot_sync(0xFFFFFFFFu, s.sumV - lastV <= TC_RASTER_BATCH_VERTICES
                                                   && s.sumT - lastT <= TC_RASTER_BATCH_TRIANGLES);
    const u32 end = 31 - __clz(fit);
    fn(q, start, end, lastV, lastT);
    const u32 count = 1 + end - start;
    lastV           = __shfl_sync(0xFFFFFFFFu, s.sumV, end);
    lastT           = __shfl_sync(0xFFFFFFFFu, s.sumT, end);
    start           = end + 1;
    left -= min(count, left);
    q++;
  }
  return q;
}

__device__ __forceinline__ u32 num_parts(const StageCtx& c)
{
  return min(c.build->partTriangleCounter, c.caps.maxPartTriangles);
}

__global__ void __launch_bounds__(kRasterBlock) k_raster_counts(StageCtx c, uint4* groups)
{
  stage_prologue();
  const u32 lane = threadIdx.x & 31, n = num_parts(c), ngroups = (n + 31) / 32;
  for(u32 g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ngroups; g += (gridDim.x * blockDim.x) >> 5)
  {
    const u32       g0 = g * 32, local = min(32u, n - g0);
    const GroupSums s  = group_sums(c, g0, local);
    const u32       nb = group_batches(s, local, [](u32, u32, u32, u32, u32) {});
    const u32       vTot = __shfl_sync(0xFFFFFFFFu, s.sumV, local - 1), tTot = __shfl_sync(0xFFFFFFFFu, s.sumT, local - 1);
    if(lane == 0)
      groups[g] = make_uint4(nb, vTot, tTot, 0u);
  }
}

// one block: exclusive scan of the groups' counts, in place; totals to
// counts[3]. Four consecutive groups per thread and round: a round costs two
// barriers and a memory round trip, so a frame of 160,000 parts (5,100 groups)
// takes two rounds.
constexpr u32 kScanGroups = 4;

__global__ void __launch_bounds__(1024) k_raster_scan(StageCtx c, uint4* groups, u32* counts)
{
  stage_prologue();
  __shared__ uint3 s_warp[2][33];
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const u32 ngroups = (num_parts(c) + 31) / 32;
  uint3     carry   = make_uint3(0, 0, 0);
  u32       round   = 0;
  for(u32 base = 0; base < ngroups; base += blockDim.x * kScanGroups, round ^= 1)
  {
    const u32 i = base + threadIdx.x * kScanGroups;
    uint4     v[kScanGroups];
    uint3     sum = make_uint3(0, 0, 0);
#pragma unroll
    for(u32 k = 0; k < kScanGroups; k++)
      v[k] = i + k < ngroups ? groups[i + k] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for(u32 k = 0; k < kScanGroups; k++)
      sum.x += v[k].x, sum.y += v[k].y, sum.z += v[k].z;
    uint3 inc = sum;
#pragma unroll
    for(int d = 1; d < 32; d <<= 1)
    {
      const u32 a = __shfl_up_sync(0xFFFFFFFFu, inc.x, d), b = __shfl_up_sync(0xFFFFFFFFu, inc.y, d),
                e = __shfl_up_sync(0xFFFFFFFFu, inc.z, d);
      if(lane >= (u32)d)
        inc.x += a, inc.y += b, inc.z += e;
    }
    if(lane == 31)
      s_warp[round][warp] = inc;
    __syncthreads();
    if(warp == 0)
    {
      const uint3 w  = s_warp[round][lane];
      uint3       wi = w;
#pragma unroll
      for(int d = 1; d < 32; d <<= 1)
      {
        const u32 a = __shfl_up_sync(0xFFFFFFFFu, wi.x, d), b = __shfl_up_sync(0xFFFFFFFFu, wi.y, d),
                  e = __shfl_up_sync(0xFFFFFFFFu, wi.z, d);
        if(lane >= (u32)d)
          wi.x += a, wi.y += b, wi.z += e;
      }
      s_warp[round][lane] = make_uint3(wi.x - w.x, wi.y - w.y, wi.z - w.z);
      if(lane == 31)
        s_warp[round][32] = wi;
    }
    __syncthreads();
    // (the next round writes the other copy; its first barrier orders the one after)
    const uint3 ww = s_warp[round][warp], tot = s_warp[round][32];
    uint3       ex = make_uint3(carry.x + ww.x + inc.x - sum.x, carry.y + ww.y + inc.y - sum.y, carry.z + ww.z + inc.z - sum.z);
#pragma unroll
    for(u32 k = 0; k < kScanGroups; k++)
    {
      if(i + k < ngroups)
        groups[i + k] = make_uint4(ex.x, ex.y, ex.z, 0u);
      ex.x += v[k].x, ex.y += v[k].y, ex.z += v[k].z;
    }
    carry.x += tot.x, carry.y += tot.y, carry.z += tot.z;
  }
  if(threadIdx.x == 0)
  {
    counts[0] = carry.x, counts[1] = carry.y, counts[2] = carry.z;
  }
}

// Bound by instruction issue and the latency of a group's dependent loads.
// A part has about five vertices and four triangles, so a warp that takes its
// parts one by one uses a sixth of its lanes; here every part of the group is
// set up once in shared memory, one part per lane (its affine form as in the
// vertex kernels, tc_vertex.cuh, and its world matrix), and the lanes walk the
// group's vertices, then its triangles, in order. When the frame has fewer
// groups than the grid has warps, several warps share a group, each walking a
// part of its parts. Measured on a GB300, 163,000 parts (992,000 vertices) of
// 256 instances: the kernel 104 -> 36 us, the call 112 -> 46 us.
// Deform: with PN triangles or the ripple.
template <bool Deform>
__global__ void __launch_bounds__(kWriteBlock, 4) k_raster_write(StageCtx c, const uint4* groups, tc_raster_outputs o)
{
  stage_prologue();
  __shared__ PartAffine s_part[kWriteWarps][32];
  __shared__ float4     s_world[kWriteWarps][32][3];  // rows of the world matrix
  __shared__ PartPn     s_pn[Deform ? kWriteWarps : 1][Deform ? 32 : 1];
  const u32                  lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const u32                  n = num_parts(c), ngroups = (n + 31) / 32;
  const tc_TessTriangleInfo* parts = reinterpret_cast<const tc_TessTriangleInfo*>(c.build->partTriangles);
  tc_raster_batch*           batches = reinterpret_cast<tc_raster_batch*>(o.batches);
  float*                     clip    = reinterpret_cast<float*>(o.clipPositions);
  float*                     world   = reinterpret_cast<float*>(o.worldPositions);
  uint8_t*                   idx     = reinterpret_cast<uint8_t*>(o.indices);
  u32*                       prim    = reinterpret_cast<u32*>(o.primitiveIDs);
  const bool                 clip16 = (o.clipPositions & 15) == 0;
  const bool                 visTriangles = c.view->visualize == TC_VISUALIZE_TRIANGLES;
  const bool                 pn = Deform && (c.flags & TC_FLAG_PN) != 0;
  const RippleParams         rp = ripple_params(*c.view, Deform && (c.flags & TC_FLAG_RIPPLE) != 0);
  float                      vp[16];
#pragma unroll
  for(int q = 0; q < 16; q++)
    vp[q] = c.view->viewProjMatrix.m[q];
  PartAffine* sp       = s_part[warp];
  const u32   below    = (2u << lane) - 2u;
  bool        overflow = false;
  // warps per group: as many of 1, 2 and 4 as the grid has warps for
  const u32 nwarps   = (gridDim.x * blockDim.x) >> 5;
  const u32 share    = ngroups * 4 <= nwarps ? 4u : (ngroups * 2 <= nwarps ? 2u : 1u);
  const u32 perShare = 32 / share;
  for(u32 gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; gw < ngroups * share; gw += nwarps)
  {
    const u32       g = gw / share, sub = gw % share;
    const u32       g0 = g * 32, local = min(32u, n - g0);
    const uint4     off = groups[g];  // batches, vertices, triangles before this group
    const GroupSums s   = group_sums(c, g0, local);
    // the vertex count before this lane's part's batch: its batch-local vertex start
    u32 batchStartV = 0;
    group_batches(s, local, [&](u32 q, u32 start, u32 end, u32 lastV, u32 lastT) {
      const u32 ev = __shfl_sync(0xFFFFFFFFu, s.sumV, end), et = __shfl_sync(0xFFFFFFFFu, s.sumT, end);
      if(lane >= start && lane <= end)
        batchStartV = lastV;
      if(lane == 0 && sub == 0)
      {
        const u32 slot = off.x + q;
        if(slot < o.maxBatches)
        {
          tc_raster_batch r;
          r.firstPart     = g0 + start;
          r.partCount     = 1 + end - start;
          r.firstVertex   = off.y + lastV;
          r.numVertices   = ev - lastV;
          r.firstTriangle = off.z + lastT;
          r.numTriangles  = et - lastT;
          batches[slot]   = r;
        }
        else
          overflow = true;
      }
    });
    // mesh.glsl:190-435: this warp's parts [pBegin, pEnd) of the group, one per lane
    const u32  pBegin = min(local, sub * perShare), pEnd = min(local, pBegin + perShare);
    const bool owner = lane >= pBegin && lane < pEnd;
    const u32  exV = s.sumV - s.v, exT = s.sumT - s.t;  // vertices and triangles before this lane's part
    u32        tvBase = 0, triBase = 0, meta = 0, inst = 0;
    float      size = 0.0f;
    if(owner)
    {
      const uint2*            raw = reinterpret_cast<const uint2*>(parts + g0 + lane);
      const uint2             r0 = __ldg(raw), r1 = __ldg(raw + 1), r2 = __ldg(raw + 2);
      const u32               cfg = r2.y >> 16, tri = r2.y & 0xFFFFu;
      const tc_TessTableEntry e   = table_entry(c.table, cfg);
      const tc_RenderInstance& in = c.instances[r0.x];
      const tc_Cluster         cl = reinterpret_cast<const tc_Cluster*>(in.clusters)[r0.y];
      const u32               corner[3] = {r1.x, r1.y, r2.x};
      setup_deform(c, in, cl, tri, cfg, corner, e.firstVertex, pn, sp[lane], s_pn[Deform ? warp : 0][Deform ? lane : 0]);
      const float* m = in.worldMatrix.m;
#pragma unroll
      for(int r = 0; r < 3; r++)
        s_world[warp][lane][r] = make_float4(__ldg(m + r), __ldg(m + 4 + r), __ldg(m + 8 + r), __ldg(m + 12 + r));
      u32 partID = 0;
#pragma unroll
      for(int v = 0; v < 3; v++)
        partID ^= (corner[v] >> 20) | ((corner[v] >> 4) & 0xFFFu);
      tvBase  = e.firstVertex - exV;    // table vertex of group vertex j: tvBase + j
      triBase = e.firstTriangle - exT;  // table triangle of group triangle j: triBase + j
      meta    = (exV - batchStartV) | ((tri & 0xFFu) << 8) | (partID << 16) | (cfg_flipped(cfg) ? 1u << 28 : 0u);
      inst    = r0.x;
      size    = in.geoHi.w;
    }
    __syncwarp();
    if(pBegin < pEnd)
    {
      const u32 vBegin = __shfl_sync(0xFFFFFFFFu, exV, pBegin), vEnd = __shfl_sync(0xFFFFFFFFu, s.sumV, pEnd - 1);
      const u32 vFit = o.maxVertices > off.y ? min(vEnd, o.maxVertices - off.y) : 0u;
      overflow |= vFit < vEnd;
      // one specialisation when the group's parts share a map kind (format and
      // wrapping resolved per vertex: 46.6 us a call, so 41.7)
      auto walk = [&](auto tag) {
        constexpr u32 kKind = decltype(tag)::value;
#pragma unroll 2  // two steps in flight: their loads overlap
        for(u32 base = vBegin; base < vFit; base += 32)
        {
          // lane's part: those starting at or before the step's first vertex,
          // plus those starting inside the step up to the lane (one bit each)
          const u32 before = __popc(__ballot_sync(0xFFFFFFFFu, owner && exV <= base));
          const u32 inside =
              __reduce_or_sync(0xFFFFFFFFu, (owner && exV > base && exV < base + 32) ? 1u << (exV - base) : 0u);
          const u32 pi = (pBegin + before - 1 + __popc(inside & below)) & 31;
          const u32 jj = base + lane;
          const u32 tvIdx = __shfl_sync(0xFFFFFFFFu, tvBase, pi);
          u32       vInst = 0;
          float     vSize = 0.0f;
          if constexpr(Deform)
          {
            vInst = __shfl_sync(0xFFFFFFFFu, inst, pi);
            vSize = __shfl_sync(0xFFFFFFFFu, size, pi);
          }
          if(jj < vFit)
          {
            const u32 tv = __ldg(c.table.vertices + (tvIdx + jj));
            const f3  p  = Deform ? deform_vertex<~0u>(sp[pi], s_pn[Deform ? warp : 0][Deform ? pi : 0], tv, pn, vInst, vSize, rp)
                                : affine_vertex_k<kKind>(sp[pi], tv);
            const float4 mx = s_world[warp][pi][0], my = s_world[warp][pi][1], mz = s_world[warp][pi][2];
            const f3     wp = {((mx.x * p.x + mx.y * p.y) + mx.z * p.z) + mx.w, ((my.x * p.x + my.y * p.y) + my.z * p.z) + my.w,
                               ((mz.x * p.x + mz.y * p.y) + mz.z * p.z) + mz.w};
            const f3     cp = xform_point(vp, wp);
            const float  cw = ((vp[3] * wp.x + vp[7] * wp.y) + vp[11] * wp.z) + vp[15];
            float*       wo = world + 3 * (u64)(off.y + jj);
            float*       co = clip + 4 * (u64)(off.y + jj);
            wo[0] = wp.x, wo[1] = wp.y, wo[2] = wp.z;
            if(clip16)
              *reinterpret_cast<float4*>(co) = make_float4(cp.x, cp.y, cp.z, cw);
            else
              co[0] = cp.x, co[1] = cp.y, co[2] = cp.z, co[3] = cw;
          }
        }
      };
      const u32 kind  = owner ? affine_kind_of(sp[lane]) : ~0u;
      const u32 kind0 = __shfl_sync(0xFFFFFFFFu, kind, __ffs(__ballot_sync(0xFFFFFFFFu, owner)) - 1);
      const u32 kw    = Deform || !__all_sync(0xFFFFFFFFu, !owner || kind == kind0) ? ~0u : kind0;
#define TC_RASTER_KIND(K)                                                                                              \
  case K:                                                                                                              \
    if constexpr(!Deform)                                                                                              \
      walk(std::integral_constant<u32, K>());                                                                          \
    break
      switch(kw)
      {
        TC_RASTER_KIND(affine_kind(TC_TEXEL_F16, true));
        TC_RASTER_KIND(affine_kind(TC_TEXEL_F32, true));
        TC_RASTER_KIND(affine_kind(TC_TEXEL_UNORM16, true));
        TC_RASTER_KIND(affine_kind(TC_TEXEL_F16, false));
        TC_RASTER_KIND(affine_kind(TC_TEXEL_F32, false));
        TC_RASTER_KIND(affine_kind(TC_TEXEL_UNORM16, false));
        TC_RASTER_KIND(kAffineFlat);
        default: walk(std::integral_constant<u32, ~0u>()); break;
      }
#undef TC_RASTER_KIND
      const u32 tBegin = __shfl_sync(0xFFFFFFFFu, exT, pBegin), tEnd = __shfl_sync(0xFFFFFFFFu, s.sumT, pEnd - 1);
      const u32 tFit = o.maxTriangles > off.z ? min(tEnd, o.maxTriangles - off.z) : 0u;
      overflow |= tFit < tEnd;
#pragma unroll 2
      for(u32 base = tBegin; base < tFit; base += 32)
      {
        const u32 before = __popc(__ballot_sync(0xFFFFFFFFu, owner && exT <= base));
        const u32 inside =
            __reduce_or_sync(0xFFFFFFFFu, (owner && exT > base && exT < base + 32) ? 1u << (exT - base) : 0u);
        const u32 pi = (pBegin + before - 1 + __popc(inside & below)) & 31;
        const u32 jj = base + lane;
        const u32 tb = __shfl_sync(0xFFFFFFFFu, triBase, pi), mt = __shfl_sync(0xFFFFFFFFu, meta, pi);
        const u32 first = __shfl_sync(0xFFFFFFFFu, exT, pi);
        if(jj < tFit)
        {
          const u32 packed = __ldg(c.table.triangles + (tb + jj));
          const u32 a = packed & 0xFF, b1 = (packed >> 8) & 0xFF, b2 = (packed >> 16) & 0xFF;
          const bool flip = (mt >> 28) != 0;  // tessellation.glsl:165-176 (flip -> .xzy)
          const u32  vs = mt & 0xFF, ID = visTriangles ? (jj - first) * 3 : (mt >> 16) & 0xFFFu;
          uint8_t*   d = idx + 3 * (u64)(off.z + jj);
          d[0] = (uint8_t)(a + vs), d[1] = (uint8_t)((flip ? b2 : b1) + vs), d[2] = (uint8_t)((flip ? b1 : b2) + vs);
          prim[off.z + jj] = ((mt >> 8) & 0xFFu) | ((ID | 1u) << 8);
        }
      }
    }
    __syncwarp();  // the records are rewritten by the warp's next group
  }
  if(overflow)
    atomicOr(c.errorWord, TC_DEVERR_CAPACITY);
}

}  // namespace

cudaError_t launch_raster_batches(const StageCtx& c, uint4* groups, const tc_raster_outputs& o, u32 maxParts,
                                  u32 numSMs, cudaStream_t s)
{
  const u32   ngroups = std::max(1u, (maxParts + 31) / 32);
  const u32   grid    = std::max(1u, std::min((ngroups + 7) / 8, numSMs * 8));
  // Two waves of the write blocks: four are resident per SM (106 registers), and
  // eight per SM even out the groups (992,000 vertices 35.5 us a call, 42.2 with
  // one wave; 286,000 24.9 and 30.2). One with PN or the ripple, where the records
  // take the shared memory of four. Small capacities get four warps per group.
  const bool  deform = (c.flags & (TC_FLAG_PN | TC_FLAG_RIPPLE)) != 0;
  const u32   wgrid  = std::max(1u, std::min(ngroups, numSMs * (deform ? 4u : 8u)));
  cudaError_t e       = launch_pdl(k_raster_counts, grid, kRasterBlock, s, c, groups);
  if(e != cudaSuccess)
    return e;
  e = launch_pdl(k_raster_scan, 1u, 1024u, s, c, groups, reinterpret_cast<u32*>(o.counts));
  if(e != cudaSuccess)
    return e;
  if(deform)
    return launch_pdl(k_raster_write<true>, wgrid, kWriteBlock, s, c, const_cast<const uint4*>(groups), o);
  return launch_pdl(k_raster_write<false>, wgrid, kWriteBlock, s, c, const_cast<const uint4*>(groups), o);
}

}  // namespace tc
