// tc_deform.cuh — vertices of part triangles with PN displacement and / or the
// ripple (TESS_USE_PN, DO_ANIMATION), one lane per vertex.
//
// A lane sets up one part in shared memory (its affine form, tc_vertex.cuh,
// and with PN the base triangle's control points); the warp's lanes then walk
// the parts' vertices as one range. Parts average three to six vertices, so
// lanes that loop over the vertices of a part of their own, with the 30 floats
// of the PN basis in registers, leave most of the warp idle at the end of each
// part and run at two blocks per SM. Bound by instruction issue and latency
// (280 instructions for each step of 32 vertices with PN). Measured on a GB300:
// 63,300 parts of 48 vertices with PN, the split passes' 25,600 of them
// 75 -> 46 us; the vertices of 7,900 2X batches 84 -> 36 us; close-up frame
// 175 -> 146 us, 256 instances with PN, ripple and transient builds
// 238 -> 198 us.
#pragma once

#include "tc_stage.cuh"
#include "tc_vertex.cuh"

namespace tc {

constexpr u32 kDeformBlock = 128;
constexpr u32 kDeformWarps = kDeformBlock / 32;
// Parts per warp: their records (320 B each) take 20 KB of a block's shared
// memory, which leaves the registers to bound the resident blocks
constexpr u32 kDeformParts = 16;
constexpr int kDeformBlocksPerSM = 7;  // 72 registers per thread
// blocks per SM left out where kernels of the frame's critical path run beside:
// room for one of their blocks
constexpr int kDeformRoom = 2;

// A warp's part records, and what its walk reads of part `lane` by shuffles.
struct DeformRecords
{
  PartAffine affine[kDeformParts];
  PartPn     pn[kDeformParts];
};

struct DeformLane
{
  u32   nv;       // vertices (0: no part)
  u32   tvFirst;  // first table vertex
  u32   dst;      // first generated vertex
  u32   inst;     // the ripple's seed
  float size;     // the geometry's size
};

// The displacement map of an instance as the reference samples it: an empty
// map reads as 0 (the offsets still displace), no map displaces nothing.
__device__ __forceinline__ tc_DisplacementTexture sampled_map(const StageCtx& c, const tc_RenderInstance& in)
{
  tc_DisplacementTexture tx = {};
  if(c.numTextures > 0 && c.textures != nullptr && in.displacementIndex >= 0)
  {
    if((u32)in.displacementIndex < c.numTextures)
    {
      tx = c.textures[in.displacementIndex];
      if(tx.width == 0)
        tx.width = 1, tx.height = 0;
    }
    else
      atomicOr(c.errorWord, TC_DEVERR_BAD_CLUSTER);
  }
  return tx;
}

// Records of base triangle `tri` of cluster `cl` with the sub-triangle corners
// and configuration of a part.
__device__ __forceinline__ void setup_deform(const StageCtx& c, const tc_RenderInstance& in, const tc_Cluster& cl, u32 tri,
                                             u32 cfg, const u32 corner[3], u32 firstVertex, bool pn, PartAffine& a,
                                             PartPn& p)
{
  const uint8_t* lt  = reinterpret_cast<const uint8_t*>(in.clusterLocalTriangles) + cl.firstLocalTriangle + tri * 3;
  const float*   pos = reinterpret_cast<const float*>(in.positions);
  const float*   nrm = reinterpret_cast<const float*>(in.normals);
  part_affine(a, corner, cfg_flipped(cfg), pos, nrm, reinterpret_cast<const float*>(in.texcoords), cl.firstLocalVertex, lt,
              firstVertex, sampled_map(c, in), in.displacementScale * c.view->displacementScale,
              in.displacementOffset + c.view->displacementOffset);
  if(pn)
  {
    f3 v[3], n[3];
#pragma unroll
    for(int k = 0; k < 3; k++)
    {
      const u32 i = cl.firstLocalVertex + lt[k];
      v[k]        = ldg3(pos, i);
      n[k]        = normalize3(ldg3(nrm, i));
    }
    write_part_pn(p, corner, cfg_flipped(cfg), v, n);
  }
}

template <u32 Kind>
__device__ __forceinline__ f3 deform_vertex(const PartAffine& a, const PartPn& p, u32 tv, bool pn, u32 inst, float size,
                                            const RippleParams& rp)
{
  f3 q = pn ? affine_displace<Kind>(a, tv, part_pn_position(p, tv)) : affine_vertex_k<Kind>(a, tv);
  if(rp.enabled)
    q = ripple(q, inst, size, rp);
  return q;
}

// The vertex walk of deform_walk for parts of map kind Kind (~0u: any), the
// lanes past the end repeating the last vertex. (One step at a time: with PN two
// in flight take 129 us instead of 128 a close-up frame, four 150; any kind at
// run time 130.7.)
template <u32 Kind>
__device__ __forceinline__ void deform_steps(const StageCtx& c, const DeformRecords& rec, bool owner, u32 start, u32 total,
                                             u32 tvBase, u32 dstBase, const DeformLane& d, bool pn,
                                             const RippleParams& rp, float* gv)
{
  const u32 lane  = threadIdx.x & 31;
  const u32 below = (2u << lane) - 2u;  // bits 1..lane
  for(u32 base = 0; base < total; base += 32)
  {
    // lane's part: those starting at or before the step's first vertex, plus
    // those starting inside the step up to the lane (one bit each)
    const u32 before = __popc(__ballot_sync(0xFFFFFFFFu, owner && start <= base));
    const u32 inside = __reduce_or_sync(0xFFFFFFFFu,
                                        (owner && start > base && start < base + 32) ? 1u << (start - base) : 0u);
    const u32   pi   = (before - 1 + __popc(inside & below)) & 31;
    const u32   jj   = min(base + lane, total - 1);
    const u32   tvi  = __shfl_sync(0xFFFFFFFFu, tvBase, pi) + jj;
    const u32   vo   = __shfl_sync(0xFFFFFFFFu, dstBase, pi) + jj;
    const u32   inst = rp.enabled ? __shfl_sync(0xFFFFFFFFu, d.inst, pi) : 0u;
    const float size = rp.enabled ? __shfl_sync(0xFFFFFFFFu, d.size, pi) : 0.0f;
    const f3 q = deform_vertex<Kind>(rec.affine[pi], rec.pn[pi], __ldg(c.table.vertices + tvi), pn, inst, size, rp);
    float*   o = gv + 3 * (u64)vo;
    o[0] = q.x, o[1] = q.y, o[2] = q.z;
  }
}

// The vertices of the warp's parts: lane l < count owns record l (d.nv > 0).
__device__ __forceinline__ void deform_walk(const StageCtx& c, const DeformRecords& rec, u32 count, const DeformLane& d,
                                            bool pn, const RippleParams& rp, float* gv)
{
  const u32  lane  = threadIdx.x & 31;
  const bool owner = lane < count;
  u32        incl  = owner ? d.nv : 0u;
#pragma unroll
  for(int s = 1; s < 32; s <<= 1)
  {
    const u32 y = __shfl_up_sync(0xFFFFFFFFu, incl, s);
    if(lane >= (u32)s)
      incl += y;
  }
  const u32 start  = incl - (owner ? d.nv : 0u);
  const u32 total  = __shfl_sync(0xFFFFFFFFu, incl, 31);
  const u32 tvBase = d.tvFirst - start, dstBase = d.dst - start;
  // one specialisation for the parts when they share a map kind
  const u32 kind  = owner ? affine_kind_of(rec.affine[lane]) : ~0u;
  const u32 kind0 = __shfl_sync(0xFFFFFFFFu, kind, 0);
  const u32 kw    = __all_sync(0xFFFFFFFFu, !owner || kind == kind0) ? kind0 : ~0u;
#define TC_DEFORM(K) deform_steps<K>(c, rec, owner, start, total, tvBase, dstBase, d, pn, rp, gv)
  switch(kw)
  {
    case affine_kind(TC_TEXEL_F16, true): TC_DEFORM(affine_kind(TC_TEXEL_F16, true)); break;
    case affine_kind(TC_TEXEL_F32, true): TC_DEFORM(affine_kind(TC_TEXEL_F32, true)); break;
    case affine_kind(TC_TEXEL_UNORM16, true): TC_DEFORM(affine_kind(TC_TEXEL_UNORM16, true)); break;
    case affine_kind(TC_TEXEL_F16, false): TC_DEFORM(affine_kind(TC_TEXEL_F16, false)); break;
    case affine_kind(TC_TEXEL_F32, false): TC_DEFORM(affine_kind(TC_TEXEL_F32, false)); break;
    case affine_kind(TC_TEXEL_UNORM16, false): TC_DEFORM(affine_kind(TC_TEXEL_UNORM16, false)); break;
    default: TC_DEFORM(~0u); break;
  }
#undef TC_DEFORM
}

}  // namespace tc
