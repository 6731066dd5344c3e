// tc_groups.cuh — instances that share their mesh, displacement map, scale and
// offset, grouped by one block of the batched frame's first kernel.
#pragma once

#include "tc_group_key.h"
#include "tc_kernels.h"
#include "tc_stage.cuh"

namespace tc {

__device__ __forceinline__ GroupKey group_key(const tc_RenderInstance& in)
{
  return {in.positions, in.normals, in.texcoords, in.clusters, in.clusterLocalTriangles, (u32)in.displacementIndex, in.numClusters,
          __float_as_uint(in.displacementScale), __float_as_uint(in.displacementOffset)};
}

// One block groups the frame's instances by key (a hash table of their indices
// in shared memory), cuts the groups into subgroups of at most kGroupMembers
// and makes a task of every cluster of a subgroup. It reads the instance
// records alone, so it runs beside the reset and the classification of the
// instances (a block of their launch; as a kernel of its own it would be a
// second root of the frame's graph, which starts 10 us late). With the records
// in host memory every access is a round trip over the host link: a thread
// loads the keys of four instances at once, and a probe compares 16 bits of the
// hash in shared memory before it reads a record. Grouping is left out (kHeadGrouped 0)
// when instances have fewer than two in a group on average.
constexpr u32 kGroupTable = 1u << kGroupTableBits;
static_assert(kGroupTable == 2 * kGroupInstances, "the table is at most half full");

__device__ inline void find_groups(const StageCtx& c, const GroupTables& g)
{
  __shared__ unsigned short s_table[kGroupTable];
  __shared__ unsigned short s_print[kGroupInstances];
  __shared__ u32            s_count[kGroupInstances], s_scan[33];
  constexpr unsigned short  kEmpty = 0xFFFF;
  const u32                 n      = min(c.numInstances, min(g.cap, kGroupInstances));
  u32*                      place  = g.members + g.cap;  // per instance: representative | rank << 16
  for(u32 i = threadIdx.x; i < kGroupTable; i += blockDim.x)
    s_table[i] = kEmpty;
  for(u32 i = threadIdx.x; i < kGroupInstances; i += blockDim.x)
    s_count[i] = 0;
  __syncthreads();
  constexpr u32 kBatch = 4;
  for(u32 base = threadIdx.x; base < n; base += kBatch * blockDim.x)
  {
    GroupKey key[kBatch];
#pragma unroll
    for(u32 q = 0; q < kBatch; q++)
      if(base + q * blockDim.x < n)
        key[q] = group_key(c.instances[base + q * blockDim.x]);
#pragma unroll
    for(u32 q = 0; q < kBatch; q++)
    {
      const u32 i = base + q * blockDim.x;
      if(i >= n)
        continue;
      const u64            hash  = group_hash(key[q]);
      const unsigned short print = group_print(hash);
      s_print[i]                 = print;
      __threadfence_block();  // (before the instance is seen in the table)
      u32 rep = ~0u;
      for(u32 slot = group_slot(hash); rep == ~0u; slot = (slot + 1) % kGroupTable)
      {
        // (the table has twice as many slots as instances)
        const unsigned short found = atomicCAS(&s_table[slot], kEmpty, (unsigned short)i);
        if(found == kEmpty)
          rep = i;
        else if(*(volatile unsigned short*)&s_print[found] == print && same_key(key[q], group_key(c.instances[found])))
          rep = found;
      }
      place[i]        = rep | atomicAdd(&s_count[rep], 1u) << 16;
      g.instBounds[i] = key[q].numClusters;  // for the scans below
    }
  }
  __syncthreads();
  // the representatives' members, subgroups and tasks, scanned in instance order
  const u32 per = (n + blockDim.x - 1) / blockDim.x;
  const u32 i0 = min(n, threadIdx.x * per), i1 = min(n, i0 + per);
  u32       sumM = 0, sumS = 0, sumT = 0, sumC = 0, reps = 0, all = 0;
  for(u32 i = i0; i < i1; i++)
  {
    const u32 nc = g.instBounds[i];
    all += nc;
    if((place[i] & 0xFFFFu) == i)
    {
      const u32 m = s_count[i], subs = (m + kGroupMembers - 1) / kGroupMembers;
      sumM += m, sumS += subs, sumT += subs * nc, sumC += nc, reps++;
    }
  }
  u32 totalM, totalS, totalT, totalC, totalR, totalAll;
  u32 atM = block_exclusive_scan(sumM, s_scan, &totalM);
  u32 atS = block_exclusive_scan(sumS, s_scan, &totalS);
  u32 atT = block_exclusive_scan(sumT, s_scan, &totalT);
  u32 atC = block_exclusive_scan(sumC, s_scan, &totalC);
  u32 atR = block_exclusive_scan(reps, s_scan, &totalR);
  block_exclusive_scan(all, s_scan, &totalAll);
  for(u32 i = i0; i < i1; i++)
    if((place[i] & 0xFFFFu) == i)
    {
      const u32 m = s_count[i], nc = g.instBounds[i];
      s_count[i]  = atM;  // now the group's first member
      for(u32 k = 0; k < m; k += kGroupMembers)
      {
        g.groups[atS++] = make_uint4(atT, atM + k, min(kGroupMembers, m - k), i);
        atT += nc;
      }
      atM += m;
      g.reps[atR++]   = make_uint2(atC, i);
      g.instBounds[i] = atC;
      atC += nc;
    }
  __syncthreads();
  for(u32 i = threadIdx.x; i < n; i += blockDim.x)
  {
    const u32 rep = place[i] & 0xFFFFu;
    g.members[s_count[rep] + (place[i] >> 16)] = i;
    if(rep != i)
      g.instBounds[i] = g.instBounds[rep];
  }
  if(threadIdx.x == 0)
  {
    g.head[kHeadSubgroups] = totalS, g.head[kHeadTasks] = totalT, g.head[kHeadReps] = totalR;
    g.head[kHeadGrouped]   = n >= 2 * totalR ? 1u : 0u;
    g.head[kHeadBounds]    = totalC <= g.boundsCap && (u64)totalC * 4 <= totalAll ? totalC : 0u;
    g.head[kHeadList]      = 0;
  }
}

}  // namespace tc
