// tc_group_key.h — what instances are grouped by (tc_groups.cuh), and its
// hash. Plain C++ as well as CUDA, so that the hash can be tested on the host.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define TC_KEY_FN __host__ __device__ __forceinline__
#else
#define TC_KEY_FN inline
#endif

namespace tc {

// what the vertices of an instance's full clusters depend on
struct GroupKey
{
  uint64_t positions, normals, texcoords, clusters, localTriangles;
  uint32_t map, numClusters;
  uint32_t scale, offset;  // the bits of the displacement's floats
};

TC_KEY_FN bool same_key(const GroupKey& a, const GroupKey& b)
{
  return a.positions == b.positions && a.normals == b.normals && a.texcoords == b.texcoords && a.clusters == b.clusters
         && a.localTriangles == b.localTriangles && a.map == b.map && a.numClusters == b.numClusters && a.scale == b.scale
         && a.offset == b.offset;
}

// Fibonacci hashing of every compared word in turn: the high bits of a multiple
// of 2^64 / golden ratio, folded down before the next word. Each step is one to
// one in its word, so keys that differ in a single word never share a hash.
// (Without the offset, which scenes give each instance, 1,000 instances of 1,000
// offsets took 780 us a frame in one chain of probes, 270 with it; 3,000 of them
// 15 ms and 0.5.)
TC_KEY_FN uint64_t group_hash(const GroupKey& k)
{
  const uint64_t words[7] = {k.positions, k.normals, k.texcoords, k.clusters, k.localTriangles,
                             k.map | (uint64_t)k.numClusters << 32, k.scale | (uint64_t)k.offset << 32};
  uint64_t       h        = 0;
#ifdef __CUDACC__
#pragma unroll
#endif
  for(int i = 0; i < 7; i++)
    h = ((h ^ h >> 32) ^ words[i]) * 0x9E3779B97F4A7C15ull;
  return h;
}

// The grouping's table: a slot from the hash's top bits, and from those below
// a fingerprint that is compared before the instance's record is read.
constexpr uint32_t kGroupTableBits = 13;
TC_KEY_FN uint32_t group_slot(uint64_t hash) { return (uint32_t)(hash >> (64 - kGroupTableBits)); }
TC_KEY_FN uint16_t group_print(uint64_t hash) { return (uint16_t)(hash >> (48 - kGroupTableBits)); }

}  // namespace tc
