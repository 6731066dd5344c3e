// tc_walk.cuh — the vertices of a batch of parts or full clusters by one warp:
// one lane sets up one part or cluster, then the lanes walk the batch's
// contiguous vertex range on consecutive vertices. Used by the frame's vertex
// kernels and by the frozen frame's forward, whose outputs are the same bits.
#pragma once

#include "tc_stage.cuh"
#include "tc_vertex.cuh"

namespace tc {

constexpr u32 kPartsPerWarp = 32;  // parts per warp and chunk: one per lane

template <class T>
__device__ __forceinline__ T warp_inclusive(T x, u32 lane)
{
#pragma unroll
  for(int d = 1; d < 32; d <<= 1)
  {
    T y = __shfl_up_sync(0xFFFFFFFFu, x, d);
    if(lane >= (u32)d)
      x += y;
  }
  return x;
}

// ---------------------------------------------------------------------------
// part triangles
// ---------------------------------------------------------------------------

// Uniform: every part of the chunk has the map, scale and offset in `m`,
// `scale`, `offset` (held in registers; the records' q6-q8 are not read).
// `tvBase`: per owner lane, its part's first table vertex minus its first
// vertex within the chunk (table index of chunk vertex jj = tvBase + jj).
// Bound by instruction issue (185 for each 32 vertices, a seventh of them the
// parts' set-up) and the latency of the texel and table loads. Steps: steps of
// 32 vertices unrolled. No lane branches: those past the end repeat the last
// vertex, so that the steps' loads overlap. With a branch around each vertex
// the frame of a 2 M triangle terrain takes 338 us, without 332 with two steps
// and 328 with four; the stage kernel, short of registers, is better with one
// (314 us with the branch, 312 with two, 309 with one).
template <u32 Kind, bool Uniform, int Steps>
__device__ __forceinline__ void chunk_vertices(const StageCtx& c, const PartAffine* sp, u32 owner, u32 start, u32 tvBase,
                                               u32 total, float* dst, const MapDesc& m, float scale, float offset)
{
  const u32 lane  = threadIdx.x & 31;
  const u32 below = (2u << lane) - 2u;  // bits 1..lane
#pragma unroll Steps
  for(u32 base = 0; base < total; base += 32)
  {
    // lane's part: those starting at or before the step's first vertex, plus
    // those starting inside the step up to the lane (one bit each)
    const u32         before = __popc(__ballot_sync(0xFFFFFFFFu, owner && start <= base));
    const u32         inside = __reduce_or_sync(0xFFFFFFFFu,
                                                (owner && start > base && start < base + 32) ? 1u << (start - base) : 0u);
    const u32         pi     = before - 1 + __popc(inside & below);
    const u32         tvIdx  = __shfl_sync(0xFFFFFFFFu, tvBase, pi & 31);
    const u32         jj     = min(base + lane, total - 1);
    const PartAffine& r      = sp[pi];
    const u32         tv     = __ldg(c.table.vertices + (tvIdx + jj));
    const f3          q      = Uniform ? affine_vertex_u<Kind>(r, tv, m, scale, offset) : affine_vertex_k<Kind>(r, tv);
    float*            d      = dst + 3 * (u64)jj;
    d[0] = q.x, d[1] = q.y, d[2] = q.z;
  }
}

// One lane's part (records r0..r2 of its TessTriangleInfo): its affine
// record in `rec` (tc_vertex.cuh), vertex count, map kind and description,
// first table vertex, displacement scale and offset.
__device__ __forceinline__ void lane_part(const StageCtx& c, uint2 r0, uint2 r1, uint2 r2, PartAffine& rec, u32& nv,
                                          u32& kind, u32& tvBase, float& scale, float& offset, MapDesc& map)
{
  const u32                cfg = r2.y >> 16;
  const u32                tri = r2.y & 0xFFFFu;
  const tc_TessTableEntry  e   = table_entry(c.table, cfg);
  const tc_RenderInstance& in  = c.instances[r0.x];
  const tc_Cluster         cl  = reinterpret_cast<const tc_Cluster*>(in.clusters)[r0.y];
  const uint8_t*           lt  = reinterpret_cast<const uint8_t*>(in.clusterLocalTriangles) + cl.firstLocalTriangle;
  const u32                corner[3] = {r1.x, r1.y, r2.x};
  tc_DisplacementTexture   tx = {};
  if(c.numTextures > 0 && c.textures != nullptr && in.displacementIndex >= 0)
  {
    if((u32)in.displacementIndex < c.numTextures)
      tx = c.textures[in.displacementIndex];
    else
      atomicOr(c.errorWord, TC_DEVERR_BAD_CLUSTER);
  }
  scale  = in.displacementScale * c.view->displacementScale;
  offset = in.displacementOffset + c.view->displacementOffset;
  part_affine(rec, corner, cfg_flipped(cfg), reinterpret_cast<const float*>(in.positions),
              reinterpret_cast<const float*>(in.normals), reinterpret_cast<const float*>(in.texcoords),
              cl.firstLocalVertex, lt + tri * 3, e.firstVertex, tx, scale, offset);
  map    = make_map_desc(tx);
  nv     = e.numVertices;
  kind   = map.kind;
  tvBase = e.firstVertex;
}

// The vertices of one chunk, after every lane set up its part's record in
// `sp[lane]` (nv = 0: no part): lanes walk the chunk's contiguous vertex
// range (first generated vertex: lane 0's `vo`) on consecutive vertices, with
// one specialisation for the whole chunk when its parts share a map kind, and
// the map, scale and offset in registers when they share those too.
template <int Steps>
__device__ __forceinline__ void chunk_generate(const StageCtx& c, const PartAffine* sp, float* gv, u32 vo, u32 nv,
                                             u32 kind, u32 tvBase, const MapDesc& map, float scale, float offset)
{
  const u32 lane = threadIdx.x & 31;
  const u32  inc   = warp_inclusive<u32>(nv, lane);
  const u32  start = inc - nv;  // first vertex of this lane's part within the chunk
  const u32  total = __shfl_sync(0xFFFFFFFFu, inc, kPartsPerWarp - 1);
  const u32  v0    = __shfl_sync(0xFFFFFFFFu, vo, 0);
  const bool owner = lane < kPartsPerWarp && nv > 0;
  tvBase -= start;  // table index of chunk vertex jj: tvBase + jj
  // one specialisation for the whole chunk when its parts share a map kind
  const u32 kind0 = __shfl_sync(0xFFFFFFFFu, kind, 0);
  const u32 kw    = __all_sync(0xFFFFFFFFu, !owner || kind == kind0) ? kind0 : ~0u;
  // the usual chunk: every part displaced from one map with one scale and
  // offset (lane 0 always owns a part: accepted parts form a prefix)
  MapDesc um;
  um.q7 = make_float4(__shfl_sync(0xFFFFFFFFu, map.q7.x, 0), __shfl_sync(0xFFFFFFFFu, map.q7.y, 0),
                      __shfl_sync(0xFFFFFFFFu, map.q7.z, 0), __shfl_sync(0xFFFFFFFFu, map.q7.w, 0));
  um.q8 = make_float4(__shfl_sync(0xFFFFFFFFu, map.q8.x, 0), __shfl_sync(0xFFFFFFFFu, map.q8.y, 0),
                      __shfl_sync(0xFFFFFFFFu, map.q8.z, 0), __shfl_sync(0xFFFFFFFFu, map.q8.w, 0));
  um.kind            = kind0;
  const float uScale = __shfl_sync(0xFFFFFFFFu, scale, 0), uOffset = __shfl_sync(0xFFFFFFFFu, offset, 0);
  const bool  same   = !owner
                    || (__float_as_uint(map.q7.x) == __float_as_uint(um.q7.x)
                        && __float_as_uint(map.q7.y) == __float_as_uint(um.q7.y)
                        && __float_as_uint(map.q7.z) == __float_as_uint(um.q7.z)
                        && __float_as_uint(map.q7.w) == __float_as_uint(um.q7.w)
                        && __float_as_uint(scale) == __float_as_uint(uScale)
                        && __float_as_uint(offset) == __float_as_uint(uOffset) && kind == kind0);
  const bool  uni    = __all_sync(0xFFFFFFFFu, same);
  __syncwarp();
  float* dst = gv + 3 * (u64)v0;
#define TC_CHUNK(K)                                                                                                    \
  (uni ? chunk_vertices<K, true, Steps>(c, sp, owner, start, tvBase, total, dst, um, uScale, uOffset)                       \
       : chunk_vertices<K, false, Steps>(c, sp, owner, start, tvBase, total, dst, um, uScale, uOffset))
  // (maps of sizes that are no powers of two, at run time before: a terrain of
  // 700,000 triangles with a map of 759 x 759 166 -> 146 us a frame, 221 -> 209 in
  // stages; 256 instances with maps of 300 x 300 85 -> 80 us)
  switch(kw)
  {
    case affine_kind(TC_TEXEL_F16, true): TC_CHUNK(affine_kind(TC_TEXEL_F16, true)); break;
    case affine_kind(TC_TEXEL_F32, true): TC_CHUNK(affine_kind(TC_TEXEL_F32, true)); break;
    case affine_kind(TC_TEXEL_UNORM16, true): TC_CHUNK(affine_kind(TC_TEXEL_UNORM16, true)); break;
    case affine_kind(TC_TEXEL_F16, false): TC_CHUNK(affine_kind(TC_TEXEL_F16, false)); break;
    case affine_kind(TC_TEXEL_F32, false): TC_CHUNK(affine_kind(TC_TEXEL_F32, false)); break;
    case affine_kind(TC_TEXEL_UNORM16, false): TC_CHUNK(affine_kind(TC_TEXEL_UNORM16, false)); break;
    case kAffineFlat:
      chunk_vertices<kAffineFlat, false, Steps>(c, sp, owner, start, tvBase, total, dst, um, uScale, uOffset);
      break;
    default: chunk_vertices<~0u, false, Steps>(c, sp, owner, start, tvBase, total, dst, um, uScale, uOffset); break;
  }
#undef TC_CHUNK
}

// Parts per chunk of a launch with `n` parts, `vertices` vertices in all (about)
// and `nwarps` warps: `most` (a lane sets up one part), halved
//  - while the chunks still take no more than half of the warps. The parts of
//    a small frame have up to 78 vertices each, so 32 of them in a row keep
//    one warp busy for 50 us while most of the chip idles: 1,280 parts of 36
//    vertices took 54.7 us in 40 chunks of 32 and take 11.7 us in 1,280 chunks
//    of one (the frame 69.8 -> 48.3 us);
//  - while there are no more chunks than warps and a chunk keeps 64 vertices
//    (two steps of the walk);
//  - while there are fewer than two chunks per warp for the ticket to even
//    out, as long as a chunk keeps 256 vertices for its set-up: 25,600 parts of
//    70 vertices, with PN, took 70.7 us in 800 chunks of 32.
// Parts of five vertices stay at 32 (60,000 of them in 16s: the frame 0.5 %
// slower; the full clusters' vertices and the allocations run beside).
__device__ __forceinline__ u32 chunk_parts(u32 n, u32 vertices, u32 nwarps, u32 most)
{
  u32 w = most;
  while(w > 1)
  {
    const u32 chunks = (n + w / 2 - 1) / (w / 2);
    if(chunks > nwarps / 2 && (chunks > 2 * nwarps || vertices / chunks < (chunks > nwarps ? 256u : 64u)))
      break;
    w >>= 1;
  }
  return w;
}

// ---------------------------------------------------------------------------
// full clusters
// ---------------------------------------------------------------------------

// what the vertex walk of a full cluster needs (phase 2 of k_classify_write)
struct FullRecord
{
  MapDesc      map;
  const float* pos;
  const float* nrm;
  const float* uvs;
  u32          first;  // firstLocalVertex
  float        scale;  // instance x view displacement scale
  float        offset; // instance + view displacement offset
  u32          vo;     // first generated vertex
  u32          nv;     // vertex count
  u32          inst;   // instance (the ripple's seed)
  float        size;   // its geometry size (RenderInstance.geoHi.w)
};

// the vertex walk over a batch of full clusters (records in `rec`), for
// records of map kind Kind (~0u: any)
template <u32 Kind>
__device__ __forceinline__ void full_steps(const FullRecord* rec, bool owner, u32 rStart, u32 rEnd, float* dst,
                                           const RippleParams& rp)
{
  const u32 lane = threadIdx.x & 31;
#pragma unroll 2  // two steps in flight: their loads overlap
  for(u32 base = 0; base < rEnd; base += 32)
  {
    const u32 before = __popc(__ballot_sync(0xFFFFFFFFu, owner && rStart <= base));
    const u32 inside = __reduce_or_sync(0xFFFFFFFFu,
                                        (owner && rStart > base && rStart < base + 32) ? 1u << (rStart - base) : 0u);
    const u32 ri     = before - 1 + __popc(inside & ((2u << lane) - 2u));
    const u32 rs     = __shfl_sync(0xFFFFFFFFu, rStart, ri & 31);
    const u32 jj     = base + lane;
    const FullRecord& fr = rec[ri];
    // (transient builds leave index bytes and 2X batches between the ranges)
    if(jj < rEnd && jj - rs < fr.nv)
    {
      const u32 vi = fr.first + (jj - rs);
      f3                p  = ldg3(fr.pos, vi);
      if(Kind != kAffineFlat)
        p = full_vertex_k<Kind>(p, ldg3(fr.nrm, vi), ldg2(fr.uvs, vi), fr.map, fr.scale, fr.offset);
      if(rp.enabled)  // cluster_classify.comp.glsl:483-485
        p = ripple(p, fr.inst, fr.size, rp);
      float* d = dst + (u64)jj * 3;
      d[0]     = p.x;
      d[1]     = p.y;
      d[2]     = p.z;
    }
  }
}

// full_steps for a batch whose records share the attribute arrays, map,
// displacement scale and offset (and, with the ripple, the instance): those
// stay in registers (`u`, read once per batch), and each step takes only its
// record's vertex-index offset and range end from the record's lane (two
// shuffles) instead of the record from shared memory. Same operations, so the
// same bits.
template <u32 Kind>
__device__ __forceinline__ void full_steps_uniform(const FullRecord& u, bool owner, u32 rStart, u32 rOff, u32 rStop,
                                                   u32 rEnd, float* dst, const RippleParams& rp)
{
  const u32 lane  = threadIdx.x & 31;
  const u32 below = (2u << lane) - 2u;
#pragma unroll 2  // two steps in flight: their loads overlap
  for(u32 base = 0; base < rEnd; base += 32)
  {
    const u32 before = __popc(__ballot_sync(0xFFFFFFFFu, owner && rStart <= base));
    const u32 inside = __reduce_or_sync(0xFFFFFFFFu,
                                        (owner && rStart > base && rStart < base + 32) ? 1u << (rStart - base) : 0u);
    const u32 ri     = (before - 1 + __popc(inside & below)) & 31;
    const u32 off    = __shfl_sync(0xFFFFFFFFu, rOff, ri);
    const u32 stop   = __shfl_sync(0xFFFFFFFFu, rStop, ri);
    const u32 jj     = base + lane;
    // (transient builds leave index bytes and 2X batches between the ranges)
    if(jj < stop)
    {
      const u32 vi = off + jj;
      f3        p  = ldg3(u.pos, vi);
      if(Kind != kAffineFlat)
        p = full_vertex_k<Kind>(p, ldg3(u.nrm, vi), ldg2(u.uvs, vi), u.map, u.scale, u.offset);
      if(rp.enabled)  // cluster_classify.comp.glsl:483-485
        p = ripple(p, u.inst, u.size, rp);
      float* d = dst + (u64)jj * 3;
      d[0]     = p.x;
      d[1]     = p.y;
      d[2]     = p.z;
    }
  }
}

// what the vertices of instance `inst`'s full clusters share
__device__ __forceinline__ FullRecord full_attributes(const StageCtx& c, u32 inst)
{
  const tc_RenderInstance* in = c.instances + inst;
  FullRecord               fr = {};
  fr.pos                    = reinterpret_cast<const float*>(in->positions);
  fr.nrm                    = reinterpret_cast<const float*>(in->normals);
  fr.uvs                    = reinterpret_cast<const float*>(in->texcoords);
  tc_DisplacementTexture tx = {};
  if(c.numTextures > 0 && c.textures != nullptr && in->displacementIndex >= 0)
  {
    if((u32)in->displacementIndex < c.numTextures)
      tx = c.textures[in->displacementIndex];
    else
      atomicOr(c.errorWord, TC_DEVERR_BAD_CLUSTER);
  }
  fr.map    = make_map_desc(tx);
  fr.scale  = in->displacementScale * c.view->displacementScale;
  fr.offset = in->displacementOffset + c.view->displacementOffset;
  fr.inst   = inst;
  fr.size   = in->geoHi.w;
  return fr;
}

// the record of full cluster `ci` whose first generated vertex is `vo`
__device__ __forceinline__ FullRecord full_record(const StageCtx& c, const tc_ClusterInfo& ci, u32 vo)
{
  const tc_Cluster cl = reinterpret_cast<const tc_Cluster*>(c.instances[ci.instanceID].clusters)[ci.clusterID];
  FullRecord       fr = full_attributes(c, ci.instanceID);
  fr.vo               = vo;
  fr.nv               = min((u32)cl.numVertices, TC_MAX_CLUSTER_VERTICES);
  fr.first            = cl.firstLocalVertex;
  return fr;
}

// vertex i of the cluster in `fr`, before the ripple
__device__ __forceinline__ f3 full_vertex(const FullRecord& fr, u32 i)
{
  const u32 vi = fr.first + i;
  const f3  p  = ldg3(fr.pos, vi);
  return fr.map.kind == kAffineFlat ? p
                                    : full_vertex_k<~0u>(p, ldg3(fr.nrm, vi), ldg2(fr.uvs, vi), fr.map, fr.scale, fr.offset);
}

// The vertices of up to 32 full clusters: owner lanes hold their record `fr`,
// in the order of their generated vertices (the ranges follow each other, with
// gaps only where transient builds placed other data); `rec`: the warp's 32
// records.
__device__ __forceinline__ void full_batch(FullRecord* rec, bool owner, const FullRecord& fr, float* gv,
                                           const RippleParams& rp)
{
  const u32 lane = threadIdx.x & 31, ltm = (1u << lane) - 1u;
  const u32 fm = __ballot_sync(0xFFFFFFFFu, owner);
  if(fm == 0)
    return;
  if(owner)
    rec[__popc(fm & ltm)] = fr;
  __syncwarp();
  // per record (lane r < nrec): first vertex within the batch and vertex count
  const u32  nrec   = __popc(fm);
  const u32  vBase  = rec[0].vo;
  const u32  rStart = lane < nrec ? rec[lane].vo - vBase : 0u;
  const u32  rCount = lane < nrec ? rec[lane].nv : 0u;
  const u32  rEnd   = __shfl_sync(0xFFFFFFFFu, rStart + rCount, nrec - 1);
  const bool own    = lane < nrec;
  // one specialisation when the batch's clusters share a map kind
  const u32 kind  = own ? rec[lane].map.kind : 0u;
  const u32 kind0 = rec[0].map.kind;
  const u32 kw    = __all_sync(0xFFFFFFFFu, !own || kind == kind0) ? kind0 : ~0u;
  float*    dst   = gv + (u64)vBase * 3;
  // the usual batch: consecutive clusters of instances of one mesh and map
  const FullRecord u    = rec[0];
  const bool       same = !own
                    || (rec[lane].pos == u.pos && rec[lane].nrm == u.nrm && rec[lane].uvs == u.uvs
                        && rec[lane].map.kind == u.map.kind
                        && __float_as_uint(rec[lane].map.q7.x) == __float_as_uint(u.map.q7.x)
                        && __float_as_uint(rec[lane].map.q7.y) == __float_as_uint(u.map.q7.y)
                        && __float_as_uint(rec[lane].map.q7.z) == __float_as_uint(u.map.q7.z)
                        && __float_as_uint(rec[lane].map.q7.w) == __float_as_uint(u.map.q7.w)
                        && __float_as_uint(rec[lane].scale) == __float_as_uint(u.scale)
                        && __float_as_uint(rec[lane].offset) == __float_as_uint(u.offset)
                        && (!rp.enabled || (rec[lane].inst == u.inst && __float_as_uint(rec[lane].size) == __float_as_uint(u.size))));
  if(__all_sync(0xFFFFFFFFu, same))
  {
    // per record (lane r): vertex index of batch vertex jj is rOff + jj, for jj < rStop
    const u32 rOff  = own ? rec[lane].first - rStart : 0u;
    const u32 rStop = own ? rStart + rCount : 0u;
    switch(u.map.kind)
    {
      case affine_kind(TC_TEXEL_F32, true):
        full_steps_uniform<affine_kind(TC_TEXEL_F32, true)>(u, own, rStart, rOff, rStop, rEnd, dst, rp);
        break;
      case affine_kind(TC_TEXEL_F16, true):
        full_steps_uniform<affine_kind(TC_TEXEL_F16, true)>(u, own, rStart, rOff, rStop, rEnd, dst, rp);
        break;
      case kAffineFlat: full_steps_uniform<kAffineFlat>(u, own, rStart, rOff, rStop, rEnd, dst, rp); break;
      default: full_steps_uniform<~0u>(u, own, rStart, rOff, rStop, rEnd, dst, rp); break;
    }
  }
  else
    switch(kw)
    {
      case affine_kind(TC_TEXEL_F32, true):
        full_steps<affine_kind(TC_TEXEL_F32, true)>(rec, own, rStart, rEnd, dst, rp);
        break;
      case affine_kind(TC_TEXEL_F16, true):
        full_steps<affine_kind(TC_TEXEL_F16, true)>(rec, own, rStart, rEnd, dst, rp);
        break;
      case kAffineFlat: full_steps<kAffineFlat>(rec, own, rStart, rEnd, dst, rp); break;
      default: full_steps<~0u>(rec, own, rStart, rEnd, dst, rp); break;
    }
}

}  // namespace tc
