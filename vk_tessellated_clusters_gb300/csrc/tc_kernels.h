// tc_kernels.h — host-side launchers of the stage kernels (implemented in the
// tc_*.cu files). Internal to the library.
#pragma once

#include <cuda_runtime.h>

#include "tc_tessellation.h"

namespace tc {

struct StageCtx;
typedef uint32_t u32;

// exclusive offsets of one visible cluster's appends
struct ClusterOffsets
{
  u32                part, split, gen, vert;
  unsigned long long data;
};
static_assert(sizeof(ClusterOffsets) == 24, "ClusterOffsets: three 8-byte words");

// with transient builds, the bases of the counters only they use (stored
// right after the ClusterOffsets bases): the back of the two-sided part
// counter, the transient builds and the template instantiations so far
struct TransBases
{
  u32 back, trans, temp, _pad;
};

// per range of visible clusters: the sums of the clusters' counts, packed
// (parts | splits << 32, full clusters | their vertices << 32, CLAS bytes;
// with transient builds: generated clusters | vertices << 32, and back slots |
// transient builds << 32 in backTrans)
struct RangeSums
{
  unsigned long long partsSplits, fullVerts, data, backTrans;
};

// Instances that share their mesh, displacement map, scale and offset, and so
// the vertices of their full clusters: found by the batched frame's first
// kernel (tc_groups.cuh) for up to kGroupInstances instances, in subgroups of
// at most kGroupMembers, with object-space bounds of their clusters when many
// instances share them.
constexpr u32 kGroupInstances = 4096;
constexpr u32 kGroupMembers   = 8;
enum : int
{
  kHeadSubgroups = 0,
  kHeadTasks,
  kHeadGrouped,  // whether the full clusters' vertices are written by groups
  kHeadBounds,   // clusters with bounds; 0: none are used
  kHeadReps,     // groups
  kHeadList,     // visible clusters left to k_classify_count (bounds in use)
};
struct GroupTables
{
  uint4*  groups;      // per subgroup: first task, first member, members, representative instance; null: no groups
  u32*    members;     // [2 * cap]: the groups' instances, and scratch
  u32*    head;        // kHead* words
  uint2*  reps;        // per group: its first entry of bounds, representative
  u32*    instBounds;  // per instance: its first entry of bounds
  float4* bounds;      // [2] per cluster of a group
  u32     cap, boundsCap;
};

// cluster_classify scratch: per visible cluster of a launch's window, and per
// block of the classify grid (each write block owns a contiguous range of clusters)
struct ClassifyBuffers
{
  uint2*          counts;     // 8 bytes per cluster (16 with transient builds)
  u32*            triWords;   // 64 per cluster
  RangeSums*      rangeSums;  // per block: the sums of its range's counts (zero before the launch)
  ClusterOffsets* bases;      // one: the counters before the launch (then one TransBases)
  uint2*          fullRecs;   // per full cluster of the window: visible index, first generated vertex
  u32*            fullRange;  // [2]: the window's generated-cluster slots; [2]: transRecs' count
  uint4*          transRecs;  // 48 bytes per cluster that is not a full one
  GroupTables     groups;     // instance groups, or all null: none this frame
};

cudaError_t launch_frame_begin(const StageCtx& c, u32 grid, cudaStream_t s);
cudaError_t launch_decode_hits(const StageCtx& c, const tc_hit* hits, u32 count, tc_base_hit* out, cudaStream_t s);
cudaError_t launch_instances_classify(const StageCtx& c, u32 grid, u32 block, cudaStream_t s);
// frame_begin and instances_classify in one launch (block = kInstanceTile)
// (with groups: one more block, which finds the instance groups)
cudaError_t launch_frame_begin_instances(const StageCtx& c, const GroupTables& g, u32 grid, cudaStream_t s);
// the bounds of the groups' clusters, before launch_cluster_classify
cudaError_t launch_cluster_bounds(const StageCtx& c, const GroupTables& g, u32 numSMs, cudaStream_t s);
// side: launched on a side stream beside classify (an ordinary launch, see
// launch_side); otherwise programmatically after the kernel before it
cudaError_t launch_clusters_cull(const StageCtx& c, u32 grid, u32 block, cudaStream_t s, bool side = false);
cudaError_t launch_build_setup(const StageCtx& c, u32 mode, cudaStream_t s);
// a frame's host traffic: `bytes` from mapped pinned host memory (src, its
// device alias) to device memory, both 16-byte aligned; the Readback to
// mapped pinned host memory (dst, its device alias, 4-byte aligned)
struct HostUpload
{
  const void*        src;
  void*              dst;
  unsigned long long bytes;
};
// on its own (at most maxGrid blocks), or inside the batched frame's first
// kernel (launch_frame_begin_instances with the upload; c's frame constants
// and instance records point into the host block)
cudaError_t launch_host_upload(const HostUpload& u, u32 maxGrid, cudaStream_t s);
cudaError_t launch_frame_begin_instances_upload(const StageCtx& c, const GroupTables& g, const HostUpload& u, u32 grid,
                                                cudaStream_t s);
cudaError_t launch_host_readback(const tc_Readback* src, void* dst, cudaStream_t s);
// the bounded look-back wait on its own (state: 3 words, zeroed here)
cudaError_t launch_lookback_probe(unsigned long long* state, u32 published, u32* errorWord, u32 spinLimit,
                                  cudaStream_t s);
cudaError_t launch_cluster_classify(const StageCtx& c, const ClassifyBuffers& buf, u32 maxClusters, u32 numSMs,
                                    u32 warpBlocksPerSM, cudaStream_t s);
// the full clusters' displaced vertices of the last launch_cluster_classify
cudaError_t launch_classify_full_vertices(const StageCtx& c, const ClassifyBuffers& buf, u32 maxClusters, u32 numSMs,
                                          u32 blocksPerSM, cudaStream_t s);
u32         classify_max_blocks(u32 maxClusters);
// whether launch_cluster_classify launches a kernel of its own for the
// clusters with part or split triangles (or transient builds)
bool        classify_lists_clusters(u32 maxClusters, u32 numSMs, u32 warpBlocksPerSM, bool transient);
cudaError_t launch_triangle_split(const StageCtx& c, u32 blockSize, u32 grid, cudaStream_t s);
// every split pass in one launch: per level its look-back rows and control
// words (a scratch slot each; the ticket of level 0's slot is the launch's)
constexpr u32 kMaxSplitLevels = 16;
constexpr u32 kSplitCtrlWords = 16;  // of a level's slot
struct SplitLevels
{
  unsigned long long* lbState[kMaxSplitLevels];  // [4][stride] per level (split, part, next level's children, index)
  u32*                ctrl[kMaxSplitLevels];     // kSplitCtrlWords per level (see tc_split.cu)
  u32                 stride;                    // tiles per level the rows hold
  u32                 levels;                    // split passes
};
cudaError_t launch_triangle_split_levels(const StageCtx& c, const SplitLevels& lv, u32 blockSize, u32 grid,
                                         cudaStream_t s);
// triangle_tess_template_instantiate scratch, per part triangle
struct InstantiateBuffers
{
  u32*                vertexOffset;  // first generated vertex of each accepted part, ~0 otherwise
  unsigned long long* chunkSums;     // per 32 parts: packed (CLAS bytes << 20 | vertices)
};

// four launches (tile sums, tile scan, args, vertices); the slot needs 3 state rows of
// instantiate_alloc_tiles(maxParts)
cudaError_t launch_triangle_instantiate(const StageCtx& c, const InstantiateBuffers& buf, u32 maxParts, u32 numSMs,
                                        u32 scanBlocksPerSM, u32 vertexBlocksPerSM, u32 vertexGridPerSM,
                                        cudaStream_t s);
// the two halves of launch_triangle_instantiate: allocation and arguments
// (tile sums, tile scan, args), then the displaced vertices, which depend on
// the allocation alone
cudaError_t launch_instantiate_alloc(const StageCtx& c, const InstantiateBuffers& buf, u32 maxParts, u32 numSMs,
                                     u32 scanBlocksPerSM, cudaStream_t s);
// its two parts: the offsets (tile sums and scan; they advance the counters,
// the instantiation counter by the run's accepted parts), then the arguments
cudaError_t launch_instantiate_prefix(const StageCtx& c, const InstantiateBuffers& buf, u32 maxParts, u32 numSMs,
                                      u32 scanBlocksPerSM, cudaStream_t s);
cudaError_t launch_instantiate_args(const StageCtx& c, const InstantiateBuffers& buf, u32 maxParts, u32 numSMs,
                                    u32 scanBlocksPerSM, cudaStream_t s);
cudaError_t launch_instantiate_vertices(const StageCtx& c, const InstantiateBuffers& buf, u32 maxParts, u32 numSMs,
                                        u32 vertexBlocksPerSM, u32 vertexGridPerSM, bool leaveRoom, cudaStream_t s);
u32         instantiate_alloc_tiles(u32 maxParts);
// the stage entry point's form: tile sums, tile scan, then arguments and
// vertices in one kernel (PN / ripple: launch_triangle_instantiate)
cudaError_t launch_instantiate_fused(const StageCtx& c, const InstantiateBuffers& buf, u32 maxParts, u32 numSMs,
                                     u32 scanBlocksPerSM, u32 vertexBlocksPerSM, u32 vertexGridPerSM, cudaStream_t s);
cudaError_t launch_blas_setup_insertion(const StageCtx& c, u32 grid, u32 block, cudaStream_t s);
cudaError_t launch_blas_clusters_insert(const StageCtx& c, u32* segStart, u32* segEnd, u32 stride, u32 grid,
                                        cudaStream_t s);
// raster batching of the frame's parts; `groups`: one uint4 per 32 parts
cudaError_t launch_raster_batches(const StageCtx& c, uint4* groups, const tc_raster_outputs& o, u32 maxParts,
                                  u32 numSMs, cudaStream_t s);
cudaError_t launch_generate_vertices(const StageCtx& c, u32 grid, cudaStream_t s);
// instance groups of the adjoint's full clusters, in scratch (head null: none)
constexpr u32 kBackInstances = 1024;  // instances grouped (one block, a thread each)
struct BackGroups
{
  uint4* groups;   // per subgroup: first task, first member, members, representative instance
  u32*   members;  // [2 * cap]: the groups' instances, then per instance its representative
  u32*   head;     // subgroups, tasks, whether the groups are used
  u32*   slots;    // per cluster of the instances: its full cluster (anything where it has none)
  u32    cap, slotCap;
};
cudaError_t launch_backward_index(const StageCtx& c, const BackGroups& g, u32 grid, cudaStream_t s);
cudaError_t launch_instantiate_backward(const StageCtx& c, const float* gradVertices, const tc_GradTargets* targets,
                                        float* const* gradTexels, const BackGroups& g, u32 numSMs, cudaStream_t s);

// tiles per launch for each stage (used to size the look-back scratch)
constexpr u32 kInstanceTile     = 256;  // instances per tile (instances_classify, blas_setup)
constexpr u32 kCullTile         = 256;  // clusters per tile
constexpr u32 kSplitRowItems    = 16;   // split items of the capacity per look-back tile of a split level
constexpr u32 kInstantiateTile  = 1024; // part triangles per instantiate tile

}  // namespace tc
