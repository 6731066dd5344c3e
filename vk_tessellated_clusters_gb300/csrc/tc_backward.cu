// tc_backward.cu — adjoint of the vertex generation with the tessellation
// decisions (factors, configs, split tree, allocation) of the forward frame
// held fixed: they are piecewise constant in the inputs.
//
// Forward being differentiated (per generated vertex):
//   part triangle   (triangle_tess_template_instantiate.comp.glsl:343-371)
//     w = interp(bb, tableVertex);  P = sum_k w_k p_k
//     N = sum_k w_k normalize(n_k);  uv = sum_k w_k uv_k
//     h = bilinear(tex, uv) * s + o;  v = P + normalize(N) * h
//   full cluster    (cluster_classify.comp.glsl:457-482)
//     v = p + normalize(n) * (bilinear(tex, uv) * s + o)
// with s = instance.displacementScale * view.displacementScale.
//
// Gradients scattered: dL/dp, dL/dn (per base vertex) and dL/dtexel (the four
// bilinear taps). Full clusters: up to 32 instantiations per warp, one lane sets
// up one of them, then the lanes walk their vertices, direct atomics. Part
// triangles likewise; the per-base-vertex terms of a part's vertices are summed
// first and added once.
#include "tc_groups.cuh"
#include "tc_kernels.h"
#include "tc_stage.cuh"
#include "tc_vertex.cuh"
#include "tc_walk.cuh"

namespace tc {

namespace {

// Additions to global memory without a result. (atomicAdd on a pointer that
// was itself loaded compiles to the form that returns the old value.)
__device__ __forceinline__ void red_add(float* p, float v)
{
  asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "f"(v) : "memory");
}
__device__ __forceinline__ void red_add2(float* p, float v0, float v1)  // p: 8-byte aligned
{
  asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(__cvta_generic_to_global(p)), "f"(v0), "f"(v1)
               : "memory");
}

// two neighbouring texels: one access where they lie on 8 bytes
__device__ __forceinline__ void red_add_texels(float* row, int x0, int x1, float v0, float v1)
{
  if(x1 == x0 + 1 && (reinterpret_cast<uintptr_t>(row + x0) & 7) == 0)
    red_add2(row + x0, v0, v1);
  else
  {
    red_add(row + x0, v0);
    red_add(row + x1, v1);
  }
}

__device__ __forceinline__ void scatter_texels(float* grad, const tc_DisplacementTexture& tx, const Taps& t, float dB)
{
  const float gx = 1.0f - t.fx, gy = 1.0f - t.fy;
  red_add_texels(grad + (u64)t.y0 * tx.width, t.x0, t.x1, (gy * gx) * dB, (gy * t.fx) * dB);
  red_add_texels(grad + (u64)t.y1 * tx.width, t.x0, t.x1, (t.fy * gx) * dB, (t.fy * t.fx) * dB);
}

// two accesses: of the first two components where those lie on 8 bytes, else
// of the last two
__device__ __forceinline__ void red_add3(float* base, u64 index, f3 v)
{
  float*     a    = base + 3 * index;
  const bool even = (reinterpret_cast<uintptr_t>(a) & 7) == 0;
  red_add2(even ? a : a + 1, even ? v.x : v.y, even ? v.y : v.z);
  red_add(even ? a + 2 : a, even ? v.z : v.x);
}

constexpr u32 kWarps = 8;      // of the forward's blocks
constexpr u32 kBackWarps = 4;  // of the adjoint's
constexpr int kBackBlocksPerSM = 7;  // 72 registers per thread
// Vertices of parts a warp takes at a time (the parts that start in them), by
// those of all parts and the number of warps: whole rounds of all warps, of
// about kBackChunk each, but no less than 64, since the last step of a walk is
// half empty, or 32 where a round takes no more (a warp's chain of loads is then
// the time). Measured with 32, 64, 96 and 128: 95,000 vertices 10.8, 11.6, 12.6 and
// 16.1 us; 1.7 M 111, 87, 81 and 79 (72 in whole rounds); 4.6 M 329, 253, 225 and
// 225 (216). 312,000 in one round of 74 36.3, in chunks of 64 48.2.
constexpr u32 kBackChunk = 128;
__device__ __forceinline__ u32 back_chunk(u64 vertices, u32 nwarps)
{
  const u32 per = (u32)((vertices + nwarps - 1) / nwarps), rounds = max(1u, (per + kBackChunk / 2) / kBackChunk);
  return per <= 32 ? 32u : max(64u, (per + rounds - 1) / rounds);
}
constexpr int kBackSteps = 2;  // steps of 32 vertices whose loads are in flight together

// number of leading full-cluster instantiations (they precede all parts)
__device__ __forceinline__ u32 full_count(const StageCtx& c, u32 temps)
{
  return min(c.runStarts[kMaxRuns + 1], temps);
}

// ---------------------------------------------------------------------------
// Full clusters by instance groups
//
// The adjoint of a full cluster is linear in dL/dv, with factors that depend on
// the mesh, map, scale and offset alone: a warp adds up dL/dv over the members
// of a subgroup and scatters once. Without that the additions in L2 (12 M
// sectors for 2.4 M vertices) and the reads of the mesh and map are repeated for
// each instance. Measured on a GB300, 50,200 full clusters of 256 instances and
// 105,000 parts, both kernels: 98 -> 49.5 us; of 96 instances 43 -> 27.5 us.
// ---------------------------------------------------------------------------

enum : u32
{
  kBackSubgroups = 0,
  kBackTasks,
  kBackGrouped,  // whether instances share enough (two to a group on average)
};

constexpr u32 kBackTable = 2 * kBackInstances;

// A full cluster's place in `slots`: its number among the instances' clusters
// (the frame's prefix; ~0 or one taken by another: the cluster is left out of
// the groups).
__device__ __forceinline__ u32 back_slot(const StageCtx& c, const BackGroups& g, const tc_ClusterInfo& ci)
{
  if(ci.instanceID >= c.numInstances || ci.clusterID >= c.instances[ci.instanceID].numClusters)
    return ~0u;
  const u32 slot = c.instClusterStart[ci.instanceID] + ci.clusterID;
  return slot < g.slotCap ? slot : ~0u;
}

__device__ __forceinline__ bool same_targets(const tc_GradTargets& a, const tc_GradTargets& b)
{
  return a.dPositions == b.dPositions && a.dNormals == b.dNormals;
}

// Whether full cluster `j` is one of its group's (else it is taken alone).
__device__ __forceinline__ bool back_grouped(const StageCtx& c, const BackGroups& g, const tc_GradTargets* targets,
                                             const tc_ClusterInfo& ci, u32 j)
{
  const u32 slot = back_slot(c, g, ci);
  return slot != ~0u && g.slots[slot] == j
         && same_targets(targets[ci.instanceID], targets[g.members[g.cap + ci.instanceID]]);
}

// Block 0: the groups of instances (representative: the first), cut into
// subgroups of at most kGroupMembers, a task for every cluster of a subgroup.
// Other blocks: the full clusters' slots. Everything written is a function of
// the frame alone, so calls on several streams write the same words.
__global__ void __launch_bounds__(kBackInstances) k_backward_index(StageCtx c, BackGroups g)
{
  stage_prologue();
  if(blockIdx.x != 0)
  {
    const tc_ClusterInfo* fulls = reinterpret_cast<const tc_ClusterInfo*>(c.build->fullClusters);
    const u32 nfull = fulls ? full_count(c, min(c.build->tempInstantiateCounter, c.caps.maxGeneratedClusters)) : 0u;
    for(u32 j = (blockIdx.x - 1) * blockDim.x + threadIdx.x; j < nfull; j += (gridDim.x - 1) * blockDim.x)
    {
      const u32 slot = back_slot(c, g, fulls[j]);
      if(slot != ~0u)
        g.slots[slot] = j;
    }
    return;
  }
  __shared__ unsigned short s_table[kBackTable], s_print[kBackInstances];
  __shared__ u32 s_first[kBackTable], s_rep[kBackInstances], s_count[kBackInstances], s_rank[kBackInstances], s_scan[33];
  constexpr unsigned short kEmpty = 0xFFFF;
  const u32                i = threadIdx.x, n = min(c.numInstances, min(g.cap, kBackInstances));
  for(u32 k = i; k < kBackTable; k += kBackInstances)
    s_table[k] = kEmpty, s_first[k] = ~0u;
  s_count[i] = 0;
  GroupKey key = {};
  if(i < n)
    key = group_key(c.instances[i]);
  const u64            hash  = group_hash(key);
  const unsigned short print = group_print(hash);
  s_print[i]                 = print;
  __syncthreads();
  // the key's slot (as in find_groups), then the first instance with that key
  u32 slot = group_slot(hash) % kBackTable;
  for(bool found = i >= n; !found;)
  {
    const unsigned short other = atomicCAS(&s_table[slot], kEmpty, (unsigned short)i);
    found = other == kEmpty || (s_print[other] == print && same_key(key, group_key(c.instances[other])));
    if(!found)
      slot = (slot + 1) % kBackTable;
  }
  if(i < n)
    atomicMin(&s_first[slot], i);
  __syncthreads();
  const u32 rep = i < n ? s_first[slot] : i;
  s_rep[i]      = rep;
  __syncthreads();
  if(i < 32)  // ranks in instance order
    for(u32 base = 0; base < n; base += 32)
    {
      const bool valid = base + i < n;
      const u32  q     = valid ? s_rep[base + i] : ~0u;
      const u32  peers = __match_any_sync(0xFFFFFFFFu, q);
      const u32  rank  = (valid ? s_count[q] : 0u) + __popc(peers & ((1u << i) - 1u));
      __syncwarp();
      if(valid && (peers >> i) == 1u)  // the last of them
        s_count[q] = rank + 1;
      s_rank[base + i] = rank;
      __syncwarp();
    }
  __syncthreads();
  const bool first = i < n && rep == i;
  const u32  m     = first ? s_count[i] : 0u, subs = (m + kGroupMembers - 1) / kGroupMembers;
  u32        totalM, totalS, totalT, totalR;
  const u32  atM = block_exclusive_scan(m, s_scan, &totalM);
  const u32  atS = block_exclusive_scan(subs, s_scan, &totalS);
  const u32  atT = block_exclusive_scan(subs * key.numClusters, s_scan, &totalT);
  block_exclusive_scan(first ? 1u : 0u, s_scan, &totalR);
  for(u32 k = 0; k < subs; k++)
    g.groups[atS + k] = make_uint4(atT + k * key.numClusters, atM + k * kGroupMembers, min(kGroupMembers, m - k * kGroupMembers), i);
  __syncthreads();
  if(first)
    s_count[i] = atM;
  __syncthreads();
  if(i < n)
  {
    g.members[s_count[rep] + s_rank[i]] = i;
    g.members[g.cap + i]                = rep;
  }
  if(i == 0)
    g.head[kBackSubgroups] = totalS, g.head[kBackTasks] = totalT, g.head[kBackGrouped] = n >= 2 * totalR ? 1u : 0u;
}

// A full cluster as its adjoint reads it.
struct BackRecord
{
  tc_DisplacementTexture tx;
  const float*           nrm;
  const float*           uvs;
  float*                 dPositions;
  float*                 dNormals;
  float*                 dTexels;
  u64                    vo;     // generated vertex of batch vertex jj: vo + jj
  u32                    first;  // base vertex of batch vertex jj: first + jj
  float                  scale, offset;  // the instance's displacement
};

// The adjoint of vertex `vi` of the full cluster in `q`, dL/dv = g, its normal
// and uv read when the cluster is displaced.
__device__ __forceinline__ void full_backward(const BackRecord& q, u32 vi, f3 g, f3 n, f2 uv, float viewScale, float viewOffset)
{
  if(q.dPositions)
    red_add3(q.dPositions, vi, g);
  if(!q.tx.width)
    return;
  const float nl   = len3(n);
  const f3    nh   = normalize3(n);
  const Taps  taps = bilinear_taps(q.tx, uv);
  const float hraw = q.tx.height ? sample_taps(q.tx, taps) : 0.0f;
  const float h    = ((hraw * q.scale) * viewScale + q.offset) + viewOffset;
  const float dh   = dot3(nh, g);
  if(q.dNormals)
  {
    // d normalize(n) / dn = (I - nh nh^T) / |n|
    const float kn = h / nl;
    const f3    dn = {kn * (g.x - nh.x * dh), kn * (g.y - nh.y * dh), kn * (g.z - nh.z * dh)};
    red_add3(q.dNormals, vi, dn);
  }
  if(q.dTexels)
    scatter_texels(q.dTexels, q.tx, taps, dh * (q.scale * viewScale));
}

// what the full clusters of instance `inst` share
__device__ __forceinline__ BackRecord back_record(const StageCtx& c, const tc_GradTargets* targets,
                                                  float* const* gradTexels, u32 inst)
{
  const tc_RenderInstance& in = c.instances[inst];
  const tc_GradTargets     gt = targets[inst];
  BackRecord               q  = {};
  if(c.numTextures > 0 && c.textures != nullptr && in.displacementIndex >= 0 && (u32)in.displacementIndex < c.numTextures)
    q.tx = c.textures[in.displacementIndex];
  q.nrm        = reinterpret_cast<const float*>(in.normals);
  q.uvs        = reinterpret_cast<const float*>(in.texcoords);
  q.dPositions = reinterpret_cast<float*>(gt.dPositions);
  q.dNormals   = reinterpret_cast<float*>(gt.dNormals);
  q.dTexels    = q.tx.width && q.tx.height ? gradTexels[in.displacementIndex] : nullptr;
  q.scale      = in.displacementScale;
  q.offset     = in.displacementOffset;
  return q;
}

// The full clusters that are in groups: a task (subgroup and cluster) per warp,
// each lane having looked up one.
__device__ void back_groups(const StageCtx& c, const BackGroups& g, BackRecord* rec, const tc_ClusterInfo* fulls,
                            u32 nfull, u32 gwarp, u32 nwarp, const float* gradVertices, const tc_GradTargets* targets,
                            float* const* gradTexels)
{
  const u32                         lane = threadIdx.x & 31;
  const u32                         subs = g.head[kBackSubgroups], tasks = g.head[kBackTasks];
  const tc_TemplateInstantiateInfo* ti   = reinterpret_cast<const tc_TemplateInstantiateInfo*>(c.build->tempInstantiations);
  const float viewScale = c.view->displacementScale, viewOffset = c.view->displacementOffset;
  for(u32 t0 = gwarp; t0 < tasks; t0 += 32 * nwarp)
  {
    // lane's task t0 + lane * nwarp: its representative, cluster and the
    // members' first vertices (~0: not a full cluster there)
    u32       nv = 0;
    u32       vo[kGroupMembers];
    const u64 t   = (u64)t0 + (u64)lane * nwarp;
    bool      any = false;
#pragma unroll
    for(u32 m = 0; m < kGroupMembers; m++)
      vo[m] = ~0u;
    if(t < tasks)
    {
      u32 lo = 0, hi = subs;  // the last subgroup whose first task is at most t
      while(hi - lo > 1)
      {
        const u32 mid = (lo + hi) >> 1;
        if(g.groups[mid].x <= (u32)t)
          lo = mid;
        else
          hi = mid;
      }
      const uint4          q  = g.groups[lo];
      const u32            k  = (u32)t - q.x;
      const tc_Cluster     cl = reinterpret_cast<const tc_Cluster*>(c.instances[q.w].clusters)[k];
      const tc_GradTargets gt = targets[q.w];
      nv              = min((u32)cl.numVertices, TC_MAX_CLUSTER_VERTICES);
      rec[lane]       = back_record(c, targets, gradTexels, q.w);
      rec[lane].first = cl.firstLocalVertex;
      // level by level, so that the members' loads overlap (a task's member has
      // cluster k: equal keys have equal cluster counts)
      u32            inst[kGroupMembers], slot[kGroupMembers], j[kGroupMembers];
      tc_ClusterInfo ci[kGroupMembers];
      tc_GradTargets mt[kGroupMembers];
#pragma unroll
      for(u32 m = 0; m < kGroupMembers; m++)
        inst[m] = m < q.z ? g.members[q.y + m] : q.w;
#pragma unroll
      for(u32 m = 0; m < kGroupMembers; m++)
        slot[m] = c.instClusterStart[inst[m]] + k, mt[m] = targets[inst[m]];
#pragma unroll
      for(u32 m = 0; m < kGroupMembers; m++)
        j[m] = slot[m] < g.slotCap ? g.slots[slot[m]] : ~0u;
#pragma unroll
      for(u32 m = 0; m < kGroupMembers; m++)
      {
        const u32 at = min(j[m], nfull - 1);
        ci[m]        = fulls[at];
        vo[m]        = (u32)((ti[at].vertexBufferAddress - c.build->genVertices) / 12);
      }
#pragma unroll
      for(u32 m = 0; m < kGroupMembers; m++)
      {
        const bool in = m < q.z && j[m] < nfull && ci[m].instanceID == inst[m] && ci[m].clusterID == k && same_targets(gt, mt[m]);
        vo[m]         = in ? vo[m] : ~0u;
        any |= in;
      }
    }
    __syncwarp();
    for(u32 left = __ballot_sync(0xFFFFFFFFu, any); left; left &= left - 1)
    {
      const int         src = __ffs(left) - 1;
      const u32         cv  = __shfl_sync(0xFFFFFFFFu, nv, src);
      const BackRecord& q   = rec[src];
      u32               v[kGroupMembers];
#pragma unroll
      for(u32 m = 0; m < kGroupMembers; m++)
        v[m] = __shfl_sync(0xFFFFFFFFu, vo[m], src);
      // a member without the cluster reads another's words and adds nothing, and
      // lanes past the end read the last vertex: no branch keeps the loads apart
      u32 other = 0;
#pragma unroll
      for(u32 m = 0; m < kGroupMembers; m++)
        other = v[m] != ~0u ? v[m] : other;
      for(u32 base = lane; base < cv + lane; base += 64)  // two vertices per lane
      {
        f3 sum[2] = {{0, 0, 0}, {0, 0, 0}}, n[2] = {{0, 0, 1}, {0, 0, 1}};
        f2 uv[2]  = {{0, 0}, {0, 0}};
#pragma unroll
        for(u32 k = 0; k < 2; k++)
        {
          const u32 i = min(base + 32 * k, cv - 1);
          if(q.tx.width)
            n[k] = ldg3(q.nrm, q.first + i), uv[k] = ldg2(q.uvs, q.first + i);
#pragma unroll
          for(u32 m = 0; m < kGroupMembers; m++)
          {
            const f3 d = ldg3(gradVertices, (u64)(v[m] != ~0u ? v[m] : other) + i);
            sum[k]     = v[m] != ~0u ? f3{sum[k].x + d.x, sum[k].y + d.y, sum[k].z + d.z} : sum[k];
          }
        }
#pragma unroll
        for(u32 k = 0; k < 2; k++)
          if(base + 32 * k < cv)
            full_backward(q, q.first + base + 32 * k, sum[k], n[k], uv[k], viewScale, viewOffset);
      }
    }
    __syncwarp();  // the records are rewritten
  }
}

// A part triangle as its adjoint reads it: base triangle's terms, map, targets.
struct __align__(16) BackPart
{
  float4                 q[7];
  // q[0..2]: sub-triangle corners bb0, bb1, bb2 (xyz each), then nh0; q[3..4]: nh1, nh2; q[4].zw: uv0;
  // q[5]: uv1, uv2; q[6]: 1 / |n0|, 1 / |n1|, 1 / |n2|, flipped (bits)
  u32                    vi[3];
  u32                    tv;  // table vertex of the chunk's vertex jj: tv + jj
  tc_DisplacementTexture tx;
  float*                 dPositions;
  float*                 dNormals;
  float*                 dTexels;
  float                  scale, offset;
  u32                    pad[4];
};
static_assert(sizeof(BackPart) % 32 == 16, "consecutive records start in different bank groups");

// The vertices of up to 32 parts: lane l owns part l (record `lane`, `nv`
// vertices, of which the first is vertex `start` of a walk of `total`; no part:
// nv = 0). `carry`: 18 words of the warp. A part's terms are added to
// memory once, by the lane that has its first vertex in its last step: one
// addition for each step or chunk a part lies in rounds the sums more often (a
// frame of 158,000 parts of 46 vertices: an error of 5.1e-7 of the positions'
// gradients instead of 3.7e-7; 224,000 of 54: 2.4e-6 instead of below 2.0e-6).
__device__ __forceinline__ void back_parts(const StageCtx& c, const BackPart* rec, float* carry, u32 nv, u32 start, u32 total,
                                           u64 from, const float* gradVertices, float viewScale, float viewOffset)
{
  const u32 lane = threadIdx.x & 31;
  const u32 upto = (2u << lane) - 1u;  // bits 0..lane
  bool      open = false;              // the step's first part began in the step before
  __syncwarp();
  for(u32 base = 0; base < total; base += 32)
  {
    // lane's part, and the lanes that start one (a part that began before the step starts at lane 0)
    const u32 before = __popc(__ballot_sync(0xFFFFFFFFu, nv && start <= base));
    const u32 heads  = 1u | __reduce_or_sync(0xFFFFFFFFu, (nv && start > base && start < base + 32) ? 1u << (start - base) : 0u);
    const u32 pi     = (before - 2 + __popc(heads & upto)) & 31;
    const u32 jj     = base + lane;
    const u32 within = jj - __shfl_sync(0xFFFFFFFFu, start, pi), count = __shfl_sync(0xFFFFFFFFu, nv, pi);
    const bool on    = within < count;
    const bool adds  = on || (open && lane == 0);
    const BackPart& r = rec[pi];
    f3 dP[3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, dNh[3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    const bool tex = r.tx.width != 0;
    const float4 q2 = r.q[2], q3 = r.q[3], q4 = r.q[4], q6 = r.q[6];
    const f3     nh[3] = {{q2.y, q2.z, q2.w}, {q3.x, q3.y, q3.z}, {q3.w, q4.x, q4.y}};
    if(on)
    {
      const f3 g = ldg3(gradVertices, from + jj);
      f3       w = decode_bary(__ldg(c.table.vertices + (r.tv + jj)));
      if(__float_as_uint(q6.w))
      {
        const float x = w.x;
        w.x           = w.y;
        w.y           = x;
      }
      const float4 q0 = r.q[0], q1 = r.q[1];
      w                 = interp3({q0.x, q0.y, q0.z}, {q0.w, q1.x, q1.y}, {q1.z, q1.w, q2.x}, w);
      const float wk[3] = {w.x, w.y, w.z};
#pragma unroll
      for(int k = 0; k < 3; k++)
        dP[k] = {wk[k] * g.x, wk[k] * g.y, wk[k] * g.z};
      if(tex)
      {
        const float4 q5   = r.q[5];
        const f3     N    = interp3(nh[0], nh[1], nh[2], w);
        const f2     uv   = interp2({q4.z, q4.w}, {q5.x, q5.y}, {q5.z, q5.w}, w);
        const float  Nl   = len3(N);
        const f3     m    = normalize3(N);
        const Taps   taps = bilinear_taps(r.tx, uv);
        const float  hraw = r.tx.height ? sample_taps(r.tx, taps) : 0.0f;
        const float  h    = ((hraw * r.scale) * viewScale + r.offset) + viewOffset;
        const float  dh   = dot3(m, g);
        // d normalize(N) / dN = (I - m m^T) / |N|
        const float kN = h / Nl;
        const f3    gN = {kN * (g.x - m.x * dh), kN * (g.y - m.y * dh), kN * (g.z - m.z * dh)};
#pragma unroll
        for(int k = 0; k < 3; k++)
          dNh[k] = {wk[k] * gN.x, wk[k] * gN.y, wk[k] * gN.z};
        if(r.dTexels)
          scatter_texels(r.dTexels, r.tx, taps, dh * (r.scale * viewScale));
      }
    }
    if(open && lane == 0)
#pragma unroll
      for(int k = 0; k < 3; k++)
      {
        dP[k]  = {dP[k].x + carry[6 * k], dP[k].y + carry[6 * k + 1], dP[k].z + carry[6 * k + 2]};
        dNh[k] = {dNh[k].x + carry[6 * k + 3], dNh[k].y + carry[6 * k + 4], dNh[k].z + carry[6 * k + 5]};
      }
    // a part's sums within the step to its first lane
    const u32  above = heads & ~upto;
    const u32  last  = above ? (u32)__ffs(above) - 2u : 31u;
    const bool any   = __any_sync(0xFFFFFFFFu, tex);
    for(u32 d = 1; d < 32 && __any_sync(0xFFFFFFFFu, lane + d <= last); d <<= 1)
    {
      const float keep = lane + d <= last ? 1.0f : 0.0f;
#pragma unroll
      for(int k = 0; k < 3; k++)
      {
        const f3 o = {__shfl_down_sync(0xFFFFFFFFu, dP[k].x, d), __shfl_down_sync(0xFFFFFFFFu, dP[k].y, d),
                      __shfl_down_sync(0xFFFFFFFFu, dP[k].z, d)};
        if(keep != 0.0f)
          dP[k] = {dP[k].x + o.x, dP[k].y + o.y, dP[k].z + o.z};
      }
      if(any)
#pragma unroll
        for(int k = 0; k < 3; k++)
        {
          const f3 o = {__shfl_down_sync(0xFFFFFFFFu, dNh[k].x, d), __shfl_down_sync(0xFFFFFFFFu, dNh[k].y, d),
                        __shfl_down_sync(0xFFFFFFFFu, dNh[k].z, d)};
          if(keep != 0.0f)
            dNh[k] = {dNh[k].x + o.x, dNh[k].y + o.y, dNh[k].z + o.z};
        }
    }
    // whether the step's last part goes on in the next one: no part starts there
    open = base + 32 < total && !__any_sync(0xFFFFFFFFu, nv && start == base + 32);
    __syncwarp();  // the carry is rewritten
    if(adds && ((heads >> lane) & 1u))
    {
      if(open && last == 31)
      {
#pragma unroll
        for(int k = 0; k < 3; k++)
        {
          carry[6 * k] = dP[k].x, carry[6 * k + 1] = dP[k].y, carry[6 * k + 2] = dP[k].z;
          carry[6 * k + 3] = dNh[k].x, carry[6 * k + 4] = dNh[k].y, carry[6 * k + 5] = dNh[k].z;
        }
      }
      else
      {
        const float rr[3] = {q6.x, q6.y, q6.z};
#pragma unroll
        for(int k = 0; k < 3; k++)
        {
          if(r.dPositions)
            red_add3(r.dPositions, r.vi[k], dP[k]);
          if(tex && r.dNormals)
          {
            // d normalize(n_k) / dn_k = (I - nh nh^T) / |n_k|
            const float d = dot3(nh[k], dNh[k]);
            red_add3(r.dNormals, r.vi[k],
                     {rr[k] * (dNh[k].x - nh[k].x * d), rr[k] * (dNh[k].y - nh[k].y * d), rr[k] * (dNh[k].z - nh[k].z * d)});
          }
        }
      }
    }
    __syncwarp();
  }
}

// What bounds it: the chains of dependent loads (arguments, cluster reference,
// instance, cluster, map, texels) at a low issue rate, so every chain is walked
// by 32 lanes for as many instantiations, and no access returns a value. A warp
// for each full cluster and a lane for each part, at 117 registers, took 147 us
// for 50,600 full clusters and 77,400 parts (2.8 M vertices) and 19.5 us for
// 20,480 parts; now 45 us after the index's 5 and 11 us.
__global__ void __launch_bounds__(kBackWarps * 32, kBackBlocksPerSM) k_instantiate_backward(StageCtx c, const float* gradVertices,
                                                                      const tc_GradTargets* targets,
                                                                      float* const* gradTexels, BackGroups groups)
{
  stage_prologue();
  union Records
  {
    BackRecord full[32];
    BackPart   part[kPartsPerWarp];
  };
  __shared__ __align__(16) unsigned char s_records[kBackWarps][sizeof(Records)];
  __shared__ float  s_carry[kBackWarps][18];
  Records&          records = *reinterpret_cast<Records*>(s_records[threadIdx.x >> 5]);
  const u32         lane  = threadIdx.x & 31;
  const u32         gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const u32         nwarp = (gridDim.x * blockDim.x) >> 5;
  tc_SceneBuilding* b     = c.build;
  const u32         temps = min(b->tempInstantiateCounter, c.caps.maxGeneratedClusters);
  const u32         nfull = full_count(c, temps);
  const tc_TemplateInstantiateInfo* ti    = reinterpret_cast<const tc_TemplateInstantiateInfo*>(b->tempInstantiations);
  const tc_ClusterInfo*             fulls = reinterpret_cast<const tc_ClusterInfo*>(b->fullClusters);
  const float viewScale = c.view->displacementScale, viewOffset = c.view->displacementOffset;

  // full clusters: every generated vertex is one base vertex
  // (cluster_classify.comp.glsl:457-482); spread evenly over the warps, at most
  // 32 at a time
  const bool grouped = groups.head != nullptr && fulls && groups.head[kBackGrouped] != 0;
  if(grouped && nfull)
    back_groups(c, groups, records.full, fulls, nfull, gwarp, nwarp, gradVertices, targets, gradTexels);
  BackRecord* rec = records.full;
  const u32   per = min(32u, max(1u, (nfull + nwarp - 1) / nwarp));
  for(u32 j0 = gwarp * per; fulls && j0 < nfull; j0 += nwarp * per)
  {
    const u32  j     = j0 + lane;
    const bool owner = lane < per && j < nfull;
    u32        nv    = 0;
    BackRecord q     = {};
    if(owner)
    {
      const tc_ClusterInfo ci = fulls[j];
      if(!grouped || !back_grouped(c, groups, targets, ci, j))
      {
        const tc_Cluster cl = reinterpret_cast<const tc_Cluster*>(c.instances[ci.instanceID].clusters)[ci.clusterID];
        q                   = back_record(c, targets, gradTexels, ci.instanceID);
        q.vo                = (ti[j].vertexBufferAddress - b->genVertices) / 12;
        q.first             = cl.firstLocalVertex;
        nv                  = min((u32)cl.numVertices, TC_MAX_CLUSTER_VERTICES);
      }
    }
    const u32 incl  = warp_inclusive<u32>(nv, lane);
    const u32 start = incl - nv, total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    const u32 used  = __ballot_sync(0xFFFFFFFFu, nv != 0);
    q.vo -= start;
    q.first -= start;
    if(nv)  // records of clusters with vertices, in order
      rec[__popc(used & ((1u << lane) - 1u))] = q;
    __syncwarp();
    for(u32 base = 0; base < total; base += 32 * kBackSteps)
    {
      u32  ri[kBackSteps], vi[kBackSteps];
      bool on[kBackSteps];
      f3   g[kBackSteps], n[kBackSteps];
      f2   uv[kBackSteps];
#pragma unroll
      for(int k = 0; k < kBackSteps; k++)
      {
        const u32 at     = base + 32 * k;
        const u32 before = __popc(__ballot_sync(0xFFFFFFFFu, nv && start <= at));
        const u32 inside = __reduce_or_sync(0xFFFFFFFFu, (nv && start > at && start < at + 32) ? 1u << (start - at) : 0u);
        ri[k]                = (before - 1 + __popc(inside & ((2u << lane) - 2u))) & 31;
        const BackRecord& w  = rec[ri[k]];
        on[k]                = at + lane < total;
        vi[k]                = w.first + at + lane;
        g[k]                 = on[k] ? ldg3(gradVertices, w.vo + at + lane) : f3{0, 0, 0};
        n[k]                 = on[k] && w.tx.width ? ldg3(w.nrm, vi[k]) : f3{0, 0, 1};
        uv[k]                = on[k] && w.tx.width ? ldg2(w.uvs, vi[k]) : f2{0, 0};
      }
#pragma unroll
      for(int k = 0; k < kBackSteps; k++)
      {
        if(on[k])
          full_backward(rec[ri[k]], vi[k], g[k], n[k], uv[k], viewScale, viewOffset);
      }
    }
    __syncwarp();  // the records are rewritten by the warp's next batch
  }

  // part triangles (triangle_tess_template_instantiate.comp.glsl:343-371), the
  // last warps first: they have the fewest full clusters
  const u32 nparts = temps - nfull;
  if(nparts == 0)
    return;
  const tc_TessTriangleInfo* parts = reinterpret_cast<const tc_TessTriangleInfo*>(b->partTriangles);
  auto first_vertex = [&](u32 j) { return (ti[j].vertexBufferAddress - b->genVertices) / 12; };
  // cut by vertices: parts have 3 to 78 of them, and those of an instance near
  // the camera have the most. A chunk's parts are those that start in it.
  const u64 vFirst = first_vertex(nfull), vLast = first_vertex(temps - 1);
  const u64 span   = (vLast > vFirst ? min(vLast - vFirst, (u64)c.caps.maxGeneratedVertices) : 0ull) + 1;
  const u32 width  = back_chunk(span, nwarp);
  const u32 chunks = (u32)((span + width - 1) / width);
  for(u32 t = nwarp - 1 - gwarp; t < chunks; t += nwarp)
  {
    const u64 from = vFirst + (u64)t * width;
    // the first part that starts at or after `from`, among 32 at a time
    u32 p0 = 0;
    for(u32 hi = nparts; p0 < hi;)
    {
      const u32 step = (hi - p0 + 31) / 32, q = p0 + lane * step;
      const u32 k    = __popc(__ballot_sync(0xFFFFFFFFu, q < hi && first_vertex(nfull + q) < from));
      if(k == 0)
        break;
      hi = min(hi, p0 + k * step);
      p0 += (k - 1) * step + 1;
    }
    for(; p0 < nparts; p0 += 32)
    {
      const u32  j   = nfull + p0 + lane;
      const u64  vo  = j < temps ? first_vertex(j) : ~0ull;
      const bool own = j < temps && vo < from + width;
      u32        nv  = 0;
      // (lane 0 owns a part if any does: parts are in the order of their vertices)
      const u64 walk  = __shfl_sync(0xFFFFFFFFu, vo, 0);
      const u32 start = (u32)(vo - walk);
      if(own)
      {
        const tc_TessTriangleInfo pt  = parts[ti[j].clusterIdOffset & 0x3FFFFFFFu];
        const u32                 cfg = pt.subTriangle.triangleID_config >> 16;
        const u32                 tri = pt.subTriangle.triangleID_config & 0xFFFFu;
        const tc_RenderInstance&  in  = c.instances[pt.cluster.instanceID];
        const tc_Cluster          cl  = reinterpret_cast<const tc_Cluster*>(in.clusters)[pt.cluster.clusterID];
        const uint8_t*            lt  = reinterpret_cast<const uint8_t*>(in.clusterLocalTriangles) + cl.firstLocalTriangle;
        const tc_TessTableEntry   e   = table_entry(c.table, cfg);
        const BackRecord          q   = back_record(c, targets, gradTexels, pt.cluster.instanceID);
        BackPart&                 r   = records.part[lane];
        nv                            = e.numVertices;
        f3    bb[3], nh[3];
        f2    uvb[3];
        float nl[3];
#pragma unroll
        for(int k = 0; k < 3; k++)
        {
          r.vi[k]    = cl.firstLocalVertex + lt[tri * 3 + k];
          bb[k]      = decode_bary(pt.subTriangle.vtxEncoded[k]);
          const f3 n = ldg3(q.nrm, r.vi[k]);
          nl[k]      = len3(n);
          nh[k]      = normalize3(n);
          uvb[k]     = ldg2(q.uvs, r.vi[k]);
        }
        r.q[0]       = make_float4(bb[0].x, bb[0].y, bb[0].z, bb[1].x);
        r.q[1]       = make_float4(bb[1].y, bb[1].z, bb[2].x, bb[2].y);
        r.q[2]       = make_float4(bb[2].z, nh[0].x, nh[0].y, nh[0].z);
        r.q[3]       = make_float4(nh[1].x, nh[1].y, nh[1].z, nh[2].x);
        r.q[4]       = make_float4(nh[2].y, nh[2].z, uvb[0].x, uvb[0].y);
        r.q[5]       = make_float4(uvb[1].x, uvb[1].y, uvb[2].x, uvb[2].y);
        r.q[6]       = make_float4(1.0f / nl[0], 1.0f / nl[1], 1.0f / nl[2], __uint_as_float(cfg_flipped(cfg) ? 1u : 0u));
        r.tv         = e.firstVertex - start;
        r.tx         = q.tx;
        r.dPositions = q.dPositions, r.dNormals = q.dNormals, r.dTexels = q.dTexels;
        r.scale = q.scale, r.offset = q.offset;
      }
      if(!__any_sync(0xFFFFFFFFu, own))
        break;
      back_parts(c, records.part, s_carry[threadIdx.x >> 5], nv, start, __reduce_max_sync(0xFFFFFFFFu, nv ? start + nv : 0u), walk,
                 gradVertices, viewScale, viewOffset);
      if(!__all_sync(0xFFFFFFFFu, own))
        break;
    }
  }
}

// Forward of the same frozen frame: regenerates every accepted instantiation's
// vertices with the batch walks of the build kernels (tc_walk.cuh; identical
// bits): up to 32 full clusters or parts per warp, one lane per record, so the
// records' dependent loads overlap. Measured on a GB300, 50,600 full clusters
// and 77,400 parts (2.8 M vertices): 84 -> 36 us.
__global__ void __launch_bounds__(kWarps * 32, 4) k_generate_vertices(StageCtx c)
{
  stage_prologue();
  union Records
  {
    PartAffine part[kPartsPerWarp];
    FullRecord full[32];
  };
  __shared__ __align__(16) unsigned char s_records[kWarps][sizeof(Records)];
  Records&          rec   = *reinterpret_cast<Records*>(s_records[threadIdx.x >> 5]);
  const u32         lane  = threadIdx.x & 31;
  const u32         gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const u32         nwarp = (gridDim.x * blockDim.x) >> 5;
  tc_SceneBuilding* b     = c.build;
  const u32         temps = min(b->tempInstantiateCounter, c.caps.maxGeneratedClusters);
  const u32         nfull = full_count(c, temps), nparts = temps - nfull;
  const tc_TemplateInstantiateInfo* ti    = reinterpret_cast<const tc_TemplateInstantiateInfo*>(b->tempInstantiations);
  const tc_TessTriangleInfo*        parts = reinterpret_cast<const tc_TessTriangleInfo*>(b->partTriangles);
  const tc_ClusterInfo*             fulls = reinterpret_cast<const tc_ClusterInfo*>(b->fullClusters);
  float*                            gv    = reinterpret_cast<float*>(b->genVertices);
  const RippleParams                rp    = {};
  auto first_vertex = [&](u32 j) { return (u32)((ti[j].vertexBufferAddress - b->genVertices) / 12); };

  // full clusters spread evenly over the warps, at most 32 at a time
  const u32 per        = min(32u, max(1u, (nfull + nwarp - 1) / nwarp));
  const u32 fullChunks = fulls ? (nfull + per - 1) / per : 0u;
  const u32 width      = nparts ? chunk_parts(nparts, first_vertex(temps - 1) - first_vertex(nfull), nwarp, kPartsPerWarp) : 1u;
  const u32 tasks      = fullChunks + (nparts + width - 1) / width;
  for(u32 t = gwarp; t < tasks; t += nwarp)
  {
    if(t < fullChunks)
    {
      const u32  j     = t * per + lane;
      const bool owner = lane < per && j < nfull;
      FullRecord fr;
      if(owner)
        fr = full_record(c, fulls[j], first_vertex(j));
      full_batch(rec.full, owner, fr, gv, rp);
    }
    else
    {
      const u32  q     = (t - fullChunks) * width + lane;
      const bool owner = lane < width && q < nparts;
      u32        vo = 0, nv = 0, kind = 0, tvBase = 0;
      float      scale = 0.0f, offset = 0.0f;
      MapDesc    map   = {};
      if(owner)
      {
        const u32    j   = nfull + q;
        const uint2* raw = reinterpret_cast<const uint2*>(parts + (ti[j].clusterIdOffset & 0x3FFFFFFFu));
        vo               = first_vertex(j);
        lane_part(c, raw[0], raw[1], raw[2], rec.part[lane], nv, kind, tvBase, scale, offset, map);
      }
      chunk_generate<2>(c, rec.part, gv, vo, nv, kind, tvBase, map, scale, offset);
    }
    __syncwarp();  // the records are rewritten by the warp's next batch
  }
}

}  // namespace

cudaError_t launch_generate_vertices(const StageCtx& c, u32 grid, cudaStream_t s)
{
  return launch_pdl(k_generate_vertices, grid, kWarps * 32, s, c);
}

cudaError_t launch_backward_index(const StageCtx& c, const BackGroups& g, u32 grid, cudaStream_t s)
{
  return launch_pdl(k_backward_index, 1 + grid, kBackInstances, s, c, g);
}

cudaError_t launch_instantiate_backward(const StageCtx& c, const float* gradVertices, const tc_GradTargets* targets,
                                        float* const* gradTexels, const BackGroups& g, u32 numSMs, cudaStream_t s)
{
  return launch_pdl(k_instantiate_backward, numSMs * kBackBlocksPerSM, kBackWarps * 32, s, c, gradVertices, targets, gradTexels, g);
}

}  // namespace tc
