// tc_split.cu — one pass of the recursive triangle split.
//
// shaders/triangle_split.comp.glsl:146-331 (processSubTask) and 598-632
// (main_multipass): every split item of the current level spawns the
// triangles of its tessellation config as children; each child's barycentrics
// are composed with the parent's, re-encoded, its segment counts re-evaluated
// on the interpolated world positions, and it is appended either to the split
// queue (next level) or to the part triangles.
//
// GB300 mapping: items have from 2 to 64 children and more (a terrain's: half
// have 2, one in a hundred over 31, and those lie together), so the work is cut
// by children: a tile is B consecutive children of the level, one per thread,
// whatever items they belong to. A level's items carry their running child
// count (StageCtx::splitEnds) and every B-th child its item (splitFirst): the
// first level's from a scan of its items at the launch's start, a later level's
// written with the items themselves (a third look-back counter). Tiles of 32
// items (73 children in the median, 2,048 at most) left most threads of a block
// idle and a few blocks with eight rounds. With 73,000 items in one launch
// beside the first part run it took 146 us and takes 96 (the frame 360 -> 338
// us); in four launches the frame went from 348 to 315 us; a PN close-up's, of
// 13,000 items, from 143 to 132 us. What bounds a tile is its chain of loads
// and the look-back, about 10 us, so tiles are large: 512 children rather than
// 256 took the terrain's frame from 354 to 338 us. (The next ticket fetched
// ahead costs 90 us: the blocks that start late hold up everyone's look-back.)
// A thread classifies its child and keeps it in registers; each warp counts its
// own; one warp per counter turns the counts into offsets and a decoupled
// look-back orders the tile's appends after all earlier tiles; then the
// children are written in (parent, child) order. Split items carry their base
// triangle's world positions in a side array, so a tile's set-up is one load
// level instead of the instance / cluster / index / vertex chain. Persistent
// grid, tiles from a ticket.
//
// Two kernels share the tile body (split_tile):
//   k_triangle_split        one pass per launch (the reference's
//                           main_multipass dispatch; per-stage and
//                           per-instance entry points);
//   k_triangle_split_levels every pass in one launch (the batched frame and
//                           its graph): the persistent blocks take tiles of
//                           all levels from one ticket, level by level; the
//                           block that completes a level's last tile publishes
//                           the next level's item range, for which the blocks
//                           holding later tickets wait (bounded); the one that
//                           completes the last level applies every pass's
//                           build_setup (what the multipass kernel's last
//                           block does). An empty first level leaves every
//                           level empty: one block then runs the passes'
//                           set-ups and the others return.
#include "tc_kernels.h"
#include "tc_stage.cuh"

namespace tc {

namespace {

enum : int
{
  kCntSplit = 0,
  kCntPart,
  kNumCounters,
  kCntKids = kNumCounters,  // children of the next level's items
  kRowScan                  // the scan of the first level's items
};

// k_triangle_split's index words, counted from the slot's first (ticket, done,
// totals); words 2 to 5 are the totals
constexpr u32 kIndexWords = 8;
static_assert(2 + 2 * kNumCounters <= kIndexWords && kIndexWords + 2 <= kSplitCtrlWords, "the index words follow the totals");

constexpr u32 kMaxChildrenPerItem = TC_TESSTABLE_SIZE * TC_TESSTABLE_SIZE;  // 121

struct SplitItem
{
  tc_ClusterInfo ci;
  u32            vtx[3];
  u32            tc;
  f3             bp[3];  // world positions of the base triangle
  u32            firstTriangle;
  u32            firstVertex;
  u32            count;  // children
};

struct Child
{
  u32  vtx[3];
  u32  tc;
  bool split;
};

__device__ __forceinline__ Child make_child(const Table& table, const SplitItem& it, u32 sub, const FactorParams& fp, u32 sf)
{
  const u32 cfg = it.tc >> 16;
  // tessellation.glsl:165-176 triangle of the pattern, flip-aware
  u32   p  = __ldg(table.triangles + it.firstTriangle + sub);
  uint3 tv = make_uint3(p & 0xFF, (p >> 8) & 0xFF, (p >> 16) & 0xFF);
  if(cfg_flipped(cfg))
  {
    u32 s = tv.y;
    tv.y  = tv.z;
    tv.z  = s;
  }
  const f3 bb0 = decode_bary(it.vtx[0]);
  const f3 bb1 = decode_bary(it.vtx[1]);
  const f3 bb2 = decode_bary(it.vtx[2]);
  Child    ch;
  const u32 tvs[3] = {tv.x, tv.y, tv.z};
#pragma unroll
  for(int v = 0; v < 3; v++)
  {
    f3 w = decode_bary(__ldg(table.vertices + it.firstVertex + tvs[v]));
    if(cfg_flipped(cfg))
    {
      float s = w.x;
      w.x     = w.y;
      w.y     = s;
    }
    ch.vtx[v] = encode_bary(interp3(bb0, bb1, bb2, w));  // triangle_split.comp.glsl:236-243
  }
  const f3 w0 = interp3(it.bp[0], it.bp[1], it.bp[2], decode_bary(ch.vtx[0]));
  const f3 w1 = interp3(it.bp[0], it.bp[1], it.bp[2], decode_bary(ch.vtx[1]));
  const f3 w2 = interp3(it.bp[0], it.bp[1], it.bp[2], decode_bary(ch.vtx[2]));
  uint3    f  = tess_factors(w0, w1, w2, fp);
  u32      m  = max(max(f.x, f.y), f.z);
  ch.split    = m > TC_TESSTABLE_SIZE;
  if(ch.split)
    f = make_uint3(split_factor1(f.x, sf), split_factor1(f.y, sf), split_factor1(f.z, sf));
  const u32 ncfg = get_config(f, ch.vtx[0], ch.vtx[1], ch.vtx[2]);
  ch.tc          = (it.tc & 0xFFFFu) | (ncfg << 16);
  return ch;
}

// the part counter a split pass continues from: the front of the two-sided
// counter with transient builds
__device__ __forceinline__ u32 part_base(const StageCtx& c)
{
  return (c.flags & (TC_FLAG_TRANSIENT_1X | TC_FLAG_TRANSIENT_2X)) ? (u32)__ldcg(&c.build->dualPartTriangleCounter)
                                                                    : __ldcg(&c.build->partTriangleCounter);
}
__device__ __forceinline__ u32 part_cap(const StageCtx& c)
{
  const u32 m = c.caps.maxPartTriangles;
  if(!(c.flags & (TC_FLAG_TRANSIENT_1X | TC_FLAG_TRANSIENT_2X)))
    return m;
  const u32 y = (u32)(c.build->dualPartTriangleCounter >> 32);
  return (u64)y + 1 < m ? m - y - 1 : 0u;
}

// Children an item takes in its level's order. At least one: an item whose
// config has no triangle takes a place without a child, so that B consecutive
// children never touch more than B items.
__device__ __forceinline__ u32 child_places(const StageCtx& c, u32 cfg)
{
  return min(max((u32)table_entry(c.table, cfg).numTriangles, 1u), kMaxChildrenPerItem);
}

// One level's items [begin, end) by their children.
struct Level
{
  u32        begin, end;
  u64        total;  // child places of all items (past 2^32 from 35.5 M items of 121 on)
  u32        tiles;  // of `chunks` x B child places each
  u32        chunks;
  const u32* first;  // per B child places: the item the first belongs to (null: level not known yet)
};

// Tiles of B child places; several (up to 16) only where the look-back rows
// hold fewer tiles than that (stride: one per kSplitRowItems items of the capacity).
template <int B>
__device__ __forceinline__ Level make_level(u32 begin, u32 end, u64 total, const u32* first, u32 stride)
{
  Level     lv = {begin, end, min(total, (u64)(end - begin) * kMaxChildrenPerItem), 0u, 1u, first};
  const u64 n  = (lv.total + B - 1) / B;
  lv.chunks    = max(1u, (u32)((n + stride - 1) / stride));
  lv.tiles     = (u32)((n + lv.chunks - 1) / lv.chunks);
  return lv;
}

// Shared memory of one split tile (kernel-scope; one per block).
template <int B>
struct SplitShared
{
  static constexpr u32 kW         = B / 32;
  static constexpr u32 kMaxChunks = (kMaxChildrenPerItem * kSplitRowItems + B - 1) / B;
  static constexpr u32 kSlots     = kMaxChunks * kW;  // (chunk, warp) count slots, in serial order
  static_assert(kSlots <= 64, "one warp scans the count slots, two per lane");
  static_assert(B >= (int)kMaxChildrenPerItem, "an item holds at most one chunk's first child");

  SplitItem item[B];
  int       end[B];                  // per item: its last child place + 1, relative to the chunk's first
  u32       cnt[kCntKids + 1][kSlots];  // per (chunk, warp): count, then exclusive offset within the tile
  u64       excl[kCntKids + 1];
  u64       total;
  u32       scan[33];
  u32       tile, flag, range[2];
};

// An item's entry in its level's index: its running child count and, where
// every B-th child is its own, the item's place in `first`.
template <int B>
__device__ __forceinline__ void index_item(const StageCtx& c, u32* first, u32 item, u64 start, u32 places)
{
  c.splitEnds[item] = start + places;
  const u64 g       = (start + B - 1) / B;
  if(g * B < start + places && g < c.splitFirstStride)
    first[g] = item;
}

// Items [begin, end)'s index from their configs, by this block alone: B items
// at a time. Returns the level's child places.
template <int B>
__device__ u64 index_local(const StageCtx& c, SplitShared<B>& sm, u32 begin, u32 end)
{
  const tc_TessTriangleInfo* queue = reinterpret_cast<const tc_TessTriangleInfo*>(c.build->splitTriangles);
  u64                        base  = 0;
  for(u32 i0 = begin; i0 < end; i0 += B)
  {
    const u32 item = i0 + threadIdx.x;
    const u32 n    = item < end ? child_places(c, __ldcg(&reinterpret_cast<const uint2*>(queue + item)[2].y) >> 16) : 0u;
    u32       total;
    const u32 excl = block_exclusive_scan(n, sm.scan, &total);
    if(n)
      index_item<B>(c, c.splitFirst, item, base + excl, n);
    base += total;
  }
  __syncthreads();  // (the block's own writes, read by its other threads)
  return base;
}

// One tile (B items) of the same by all blocks, ordered by a look-back on `row`.
template <int B>
__device__ void index_tile(const StageCtx& c, SplitShared<B>& sm, u64* row, u32 tile, u32 begin, u32 end)
{
  const tc_TessTriangleInfo* queue = reinterpret_cast<const tc_TessTriangleInfo*>(c.build->splitTriangles);
  const u32                  item  = begin + tile * B + threadIdx.x;
  const u32 n = item < end ? child_places(c, __ldcg(&reinterpret_cast<const uint2*>(queue + item)[2].y) >> 16) : 0u;
  u32       total;
  const u32 excl = block_exclusive_scan(n, sm.scan, &total);
  if(threadIdx.x < 32)
  {
    const u64 ex = warp_lookback_exclusive(row, tile, total, 0, c.errorWord, c.spinLimit);
    if(threadIdx.x == 0)
      sm.excl[0] = ex;
  }
  __syncthreads();
  if(n)
    index_item<B>(c, c.splitFirst, item, sm.excl[0] + excl, n);
  __syncthreads();
}

// up to this many tiles' items every block indexes for itself, without waiting
// for the others
constexpr u32 kIndexLocalTiles = 4;

// Waits (thread 0) until `flag` is set; false after the limit.
__device__ __forceinline__ bool wait_flag(const StageCtx& c, const u32* flag)
{
  u32 spins = 0;
  while(ld_acquire_u32(flag) == 0u)
  {
    if(++spins > c.spinLimit)
    {
      atomicOr(c.errorWord, TC_DEVERR_LOOKBACK_TIMEOUT);
      return false;
    }
    __nanosleep(spins > 64 ? 256 : 32);
  }
  return true;
}

__device__ __forceinline__ void st_release_u32(u32* p, u32 v)
{
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// One child place and its child.
struct Lane
{
  Child child;
  u32   item;  // within the chunk's items
  bool  valid;
};

// Chunk g's items into shared memory, then the thread's child.
template <int B>
__device__ __forceinline__ Lane chunk_child(const StageCtx& c, SplitShared<B>& sm, const Level& lv, u32 g,
                                            const FactorParams& fp, u32 sf)
{
  const tc_TessTriangleInfo* queue = reinterpret_cast<const tc_TessTriangleInfo*>(c.build->splitTriangles);
  const u64                  from = (u64)g * B;
  // the chunk's items: from its first child's to the next chunk's first
  // child's. (Clamped: after a look-back that ran out they may be anything.)
  const u32 a = min(max(__ldcg(lv.first + g), lv.begin), lv.end - 1);
  const u32 z = from + B < lv.total ? min(max(__ldcg(lv.first + g + 1), a), lv.end - 1) : lv.end - 1;
  const u32 n = min(z - a + 1, (u32)B);
  __syncthreads();  // the previous chunk's items are no longer read
  if(threadIdx.x < n)
  {
    const u32 item = a + threadIdx.x;
    // triangle_split.comp.glsl:146-180 fillBaseVertices; the base
    // triangle's world positions travel with the item (splitBase)
    // through L2: with every pass in one launch, other blocks wrote these items
    const uint2* raw = reinterpret_cast<const uint2*>(queue + item);
    const uint2  r0 = __ldcg(raw), r1 = __ldcg(raw + 1), r2 = __ldcg(raw + 2);
    SplitItem    it;
    it.ci     = {r0.x, r0.y};
    it.vtx[0] = r1.x;
    it.vtx[1] = r1.y;
    it.vtx[2] = r2.x;
    it.tc     = r2.y;
    sm.end[threadIdx.x] = (int)((long long)__ldcg(c.splitEnds + item) - (long long)from);
    const float* sb     = c.splitBase + 9 * (u64)item;
#pragma unroll
    for(int v = 0; v < 3; v++)
      it.bp[v] = {__ldcg(sb + 3 * v), __ldcg(sb + 3 * v + 1), __ldcg(sb + 3 * v + 2)};
    const tc_TessTableEntry e = table_entry(c.table, it.tc >> 16);
    it.firstTriangle     = e.firstTriangle;
    it.firstVertex       = e.firstVertex;
    it.count             = min((u32)e.numTriangles, kMaxChildrenPerItem);
    sm.item[threadIdx.x] = it;
  }
  __syncthreads();
  // the place's item: the first that ends after it
  u32 lo = 0, hi = n - 1;
  while(lo < hi)
  {
    const u32 mid = (lo + hi) >> 1;
    if(sm.end[mid] > (int)threadIdx.x)
      hi = mid;
    else
      lo = mid + 1;
  }
  const SplitItem& it  = sm.item[lo];
  const u32        sub = threadIdx.x - (u32)(sm.end[lo] - (int)max(it.count, 1u));
  Lane             l;
  l.item        = lo;
  l.valid       = from + threadIdx.x < lv.total && sub < it.count;
  l.child.split = false;
  if(l.valid)
    l.child = make_child(c.table, it, sub, fp, sf);
  return l;
}

// One tile: its children classified, ordered after every earlier tile of the
// level (look-back on `lbState` rows of `lbStride`, tile 0 from the counters'
// values before the pass: `bases`) and written. The last tile publishes the
// level's totals. `next`: where the next level's `first` is written, null in a
// launch of one pass.
template <int B>
__device__ void split_tile(const StageCtx& c, SplitShared<B>& sm, u32 tile, const Level& lv, u64* lbState, u32 lbStride,
                           u64* totals, const u32* bases, u32* next, const FactorParams& fp, u32 sf, u32 partCap)
{
  using S                  = SplitShared<B>;
  constexpr u32 kW         = S::kW;
  const u32     lane       = threadIdx.x & 31;
  const u32     warp       = threadIdx.x >> 5;
  const u32     ltm        = (1u << lane) - 1u;
  tc_SceneBuilding*    b     = c.build;
  const tc_caps&       k     = c.caps;
  tc_TessTriangleInfo* queue = reinterpret_cast<tc_TessTriangleInfo*>(b->splitTriangles);
  const u32            g0 = tile * lv.chunks, chunks = min(lv.chunks, (u32)((lv.total + B - 1) / B) - g0);

  // ---- classify; every warp counts its own slots ----------------------------
  Lane l;
  for(u32 ch = 0; ch < chunks; ch++)
  {
    l                = chunk_child<B>(c, sm, lv, g0 + ch, fp, sf);
    const bool split = l.valid && l.child.split;
    const u32  bs = __ballot_sync(0xFFFFFFFFu, split), bp = __ballot_sync(0xFFFFFFFFu, l.valid && !split);
    u32        kids = 0;
    if(next && bs)
      kids = __reduce_add_sync(0xFFFFFFFFu, split ? child_places(c, l.child.tc >> 16) : 0u);
    if(lane == 0)
    {
      sm.cnt[kCntSplit][ch * kW + warp] = __popc(bs);
      sm.cnt[kCntPart][ch * kW + warp]  = __popc(bp);
      sm.cnt[kCntKids][ch * kW + warp]  = kids;
    }
  }
  __syncthreads();

  // ---- slot offsets within the tile, tile totals, look-back -----------------
  if(warp < (next ? kCntKids + 1 : kNumCounters))
  {
    const u32 q     = warp;
    const u32 slots = chunks * kW;
    const u32 i0 = 2 * lane, i1 = i0 + 1;
    const u32 v0 = i0 < slots ? sm.cnt[q][i0] : 0u, v1 = i1 < slots ? sm.cnt[q][i1] : 0u;
    u32       incl = v0 + v1;
#pragma unroll
    for(int d = 1; d < 32; d <<= 1)
    {
      const u32 y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if(lane >= (u32)d)
        incl += y;
    }
    const u32 run = incl - v0 - v1;
    if(i0 < slots)
      sm.cnt[q][i0] = run;
    if(i1 < slots)
      sm.cnt[q][i1] = run + v0;
    const u32 agg  = __shfl_sync(0xFFFFFFFFu, incl, 31);
    u64       base = 0;
    if(tile == 0 && q < kNumCounters)  // the counters as the previous pass left them (through L2: see above)
      base = bases ? __ldcg(bases + q) : (q == kCntSplit ? __ldcg(&b->splitWriteCounter) : part_base(c));
    const u64 ex = warp_lookback_exclusive(lbState + (u64)q * lbStride, tile, agg, base, c.errorWord, c.spinLimit);
    if(lane == 0)
    {
      sm.excl[q] = ex;
      if(tile == lv.tiles - 1 && q < kNumCounters)
        totals[q] = ex + agg;
    }
  }
  __syncthreads();

  // ---- write (the children of a tile of several chunks once more) -----------
  for(u32 ch = 0; ch < chunks; ch++)
  {
    if(chunks > 1)
      l = chunk_child<B>(c, sm, lv, g0 + ch, fp, sf);
    const Child&     child = l.child;
    const SplitItem& item  = sm.item[l.item];
    const bool       split = l.valid && child.split, part = l.valid && !child.split;
    const u32        bs = __ballot_sync(0xFFFFFFFFu, split), bp = __ballot_sync(0xFFFFFFFFu, part);
    u32              places = 0, before = 0;
    if(next && bs)
    {
      places = split ? child_places(c, child.tc >> 16) : 0u;
      before = places;
#pragma unroll
      for(int d = 1; d < 32; d <<= 1)
      {
        const u32 y = __shfl_up_sync(0xFFFFFFFFu, before, d);
        if(lane >= (u32)d)
          before += y;
      }
      before -= places;
    }
    if(split)
    {
      const u64 o = sm.excl[kCntSplit] + sm.cnt[kCntSplit][ch * kW + warp] + __popc(bs & ltm);
      if(o < k.maxSplitTriangles)
      {
        uint2* dst = reinterpret_cast<uint2*>(queue + o);
        dst[0]     = make_uint2(item.ci.instanceID, item.ci.clusterID);
        dst[1]     = make_uint2(child.vtx[0], child.vtx[1]);
        dst[2]     = make_uint2(child.vtx[2], child.tc);
        float* d   = c.splitBase + 9 * o;
#pragma unroll
        for(int v = 0; v < 3; v++)
          d[3 * v] = item.bp[v].x, d[3 * v + 1] = item.bp[v].y, d[3 * v + 2] = item.bp[v].z;
        if(next)
          index_item<B>(c, next, (u32)o, sm.excl[kCntKids] + sm.cnt[kCntKids][ch * kW + warp] + before,
                        places);
      }
    }
    else if(part)
    {
      const u64 o = sm.excl[kCntPart] + sm.cnt[kCntPart][ch * kW + warp] + __popc(bp & ltm);
      if(o < partCap)
      {
        uint2* dst = reinterpret_cast<uint2*>(reinterpret_cast<tc_TessTriangleInfo*>(b->partTriangles) + o);
        dst[0]     = make_uint2(item.ci.instanceID, item.ci.clusterID);
        dst[1]     = make_uint2(child.vtx[0], child.vtx[1]);
        dst[2]     = make_uint2(child.vtx[2], child.tc);
      }
    }
  }
  __syncthreads();  // the item and count arrays are rewritten by the next tile
}

// The counters after a pass (triangle_split.comp.glsl:321-328 and the
// multipass dispatch's bookkeeping): run by one thread once every tile of the
// pass is done; `totals` are the last tile's inclusive totals.
__device__ inline void split_pass_counters(const StageCtx& c, u32 numTiles, const u64* totals, u32 partCap)
{
  tc_SceneBuilding* b = c.build;
  if(!numTiles)
    return;
  // another block's last tile wrote the totals: read them through L2
  b->splitWriteCounter = (u32)__ldcg(totals + kCntSplit);
  const u32 total      = (u32)__ldcg(totals + kCntPart);
  if(c.flags & (TC_FLAG_TRANSIENT_1X | TC_FLAG_TRANSIENT_2X))
  {
    // requests to the counter's front half; partTriangleCounter is the
    // end of the written front (triangle_split.comp.glsl:321-328)
    const u32 start = (u32)b->dualPartTriangleCounter, written = min(total, partCap);
    b->dualPartTriangleCounter = (b->dualPartTriangleCounter & 0xFFFFFFFF00000000ull) | total;
    if(written > start)
      b->partTriangleCounter = max(b->partTriangleCounter, written);
  }
  else
    b->partTriangleCounter = total;
}

__device__ inline FactorParams split_factor_params(const StageCtx& c)
{
  FactorParams fp;
  fp.viewPos   = {c.build->viewPos.x, c.build->viewPos.y, c.build->viewPos.z};
  fp.nearPlane = c.view->nearPlane;
  fp.viewportH = c.view->viewportf.y;
  fp.tessRate  = c.view->tessRate;
  return fp;
}

template <int B>
__global__ void __launch_bounds__(B) k_triangle_split(StageCtx c)
{
  stage_prologue();
  __shared__ SplitShared<B> sm;
  tc_SceneBuilding* b = c.build;
  // with transient builds a child part fits when it leaves the back's slots
  // and one more free (build.glsl:68-82, one child at a time)
  const u32            partCap = part_cap(c);
  tc_TessTriangleInfo* queue   = reinterpret_cast<tc_TessTriangleInfo*>(b->splitTriangles);

  if(threadIdx.x == 0)
  {
    u32 hi = min(b->splitPassEnd, c.caps.maxSplitTriangles);
    u32 lo = min(b->splitPassStart, hi);
    if(!whole_window(c))
    {
      auto get = [&](u32 i) { return queue[i].cluster.instanceID; };
      u32  e   = lower_bound_instance(lo, hi, c.instEnd, get);
      lo       = lower_bound_instance(lo, e, c.instBegin, get);
      hi       = e;
    }
    sm.range[0] = lo;
    sm.range[1] = hi;
  }
  __syncthreads();
  const u32 begin = sm.range[0], end = sm.range[1];
  // no item: nothing is counted or written, the first block runs the set-up (an
  // empty pass leaves the next one's range empty as well, so a block that reads
  // it late finds the same)
  if(begin == end)
  {
    if(blockIdx.x == 0 && threadIdx.x == 0 && c.fuseSetup != kNoSetup)
      build_setup_apply(c, c.fuseSetup);
    return;
  }
  const FactorParams fp = split_factor_params(c);
  const u32          sf = clamp_split_factor(c.caps.splitFactor);
  u32*               indexed  = c.scratch.ticket + kIndexWords;  // index tiles done; index complete
  const u32          own      = (end - begin) <= kIndexLocalTiles * B;
  const u32          idxTiles = own ? 0u : (end - begin + B - 1) / B;
  Level              lv       = {};
  if(own)
    lv = make_level<B>(begin, end, index_local<B>(c, sm, begin, end), c.splitFirst, c.scratch.lbStride);

  for(;;)
  {
    u32 tile = next_tile(c, &sm.tile);
    if(tile < idxTiles)
    {
      index_tile<B>(c, sm, c.scratch.lbState + (u64)kRowScan * c.scratch.lbStride, tile, begin, end);
      if(threadIdx.x == 0)
      {
        __threadfence();
        if(atomicAdd(indexed, 1u) == idxTiles - 1)
          st_release_u32(indexed + 1, 1u);
      }
      continue;
    }
    tile -= idxTiles;
    if(idxTiles && lv.first == nullptr)
    {
      if(threadIdx.x == 0)
        sm.total = wait_flag(c, indexed + 1) ? __ldcg(c.splitEnds + end - 1) : 0ull;
      __syncthreads();
      lv = make_level<B>(begin, end, sm.total, c.splitFirst, c.scratch.lbStride);
    }
    if(tile >= lv.tiles)
      break;
    split_tile<B>(c, sm, tile, lv, c.scratch.lbState, c.scratch.lbStride, c.scratch.totals, nullptr, nullptr, fp, sf,
                  partCap);
  }

  if(last_block_done(c, &sm.flag))
  {
    if(threadIdx.x == 0)
    {
      split_pass_counters(c, lv.tiles, c.scratch.totals, partCap);
      if(c.fuseSetup != kNoSetup)
        build_setup_apply(c, c.fuseSetup);
    }
    // (without the index, its wait having run out, what the others used is not known)
    scratch_release(c, lv.tiles == 0 ? c.scratch.lbStride : lv.tiles, kNumCounters);
    if(c.scratch.selfClean)
    {
      for(u32 t = threadIdx.x; t < idxTiles; t += B)
        c.scratch.lbState[(u64)kRowScan * c.scratch.lbStride + t] = 0;
      if(threadIdx.x == 0)
        indexed[0] = indexed[1] = 0;
    }
  }
}

// ---------------------------------------------------------------------------
// every pass in one launch
// ---------------------------------------------------------------------------

// Per-level control words, in the level's scratch slot (zeroed with the
// frame): [1] tiles done, [2..] u64 totals (split, part), [6] / [7] the split
// and part counters before the level, [8] u64 the level's child places (not of
// level 0), [11] next level's range published, [12] finalised, [13] start, [14]
// end. Level 0's [0] is the ticket all levels share, its [8] counts index tiles,
// its [9] is set with the index complete, and its [15] before the set-ups are
// written.
__device__ __forceinline__ u32* lv_done(const SplitLevels& lv, u32 L) { return lv.ctrl[L] + 1; }
__device__ __forceinline__ u64* lv_totals(const SplitLevels& lv, u32 L) { return reinterpret_cast<u64*>(lv.ctrl[L] + 2); }
__device__ __forceinline__ u32* lv_bases(const SplitLevels& lv, u32 L) { return lv.ctrl[L] + 6; }
__device__ __forceinline__ u64* lv_places(const SplitLevels& lv, u32 L) { return reinterpret_cast<u64*>(lv.ctrl[L] + 8); }
__device__ __forceinline__ u32* lv_ready(const SplitLevels& lv, u32 L) { return lv.ctrl[L] + 11; }
__device__ __forceinline__ u32* lv_final(const SplitLevels& lv, u32 L) { return lv.ctrl[L] + 12; }

// Every level is complete: the counters and set-ups of all passes
// (split_pass_counters and TC_BUILD_SETUP_SPLIT_PASS for each, then the fused
// set-up), from the levels' totals, by one thread. Done here once, in
// registers: at each level's end it kept the next level's tiles waiting for
// five dependent accesses. With no split item at all (levels empty) nothing
// but the set-ups is left, 7 us of every frame without splits, now 3.
__device__ void finalize_levels(const StageCtx& c, const SplitLevels& lv, u32 partCap)
{
  // a block that starts only now must not take the range written below for level 0's
  st_release_u32(lv.ctrl[0] + 15, 1u);
  __threadfence();
  tc_SceneBuilding* b     = c.build;
  const u32         most  = c.caps.maxSplitTriangles;
  const bool        trans = (c.flags & (TC_FLAG_TRANSIENT_1X | TC_FLAG_TRANSIENT_2X)) != 0;
  u32 write = b->splitWriteCounter, start = b->splitPassStart, end = b->splitPassEnd, pass = b->splitPass;
  u32 part  = b->partTriangleCounter;
  u64 dual  = b->dualPartTriangleCounter;
  for(u32 L = 0; L < lv.levels; L++)
  {
    const u32 last = min(end, most), first = min(start, last);
    if(last > first)
    {
      // split_pass_counters
      write           = (u32)__ldcg(lv_totals(lv, L) + kCntSplit);
      const u32 total = (u32)__ldcg(lv_totals(lv, L) + kCntPart);
      if(trans)
      {
        const u32 from = (u32)dual, written = min(total, partCap);
        dual           = (dual & 0xFFFFFFFF00000000ull) | total;
        if(written > from)
          part = max(part, written);
      }
      else
        part = total;
    }
    if(L + 1 == lv.levels)
      break;
    // TC_BUILD_SETUP_SPLIT_PASS (build_setup_apply)
    pass++;
    start = min(end, most);
    end   = min(write, most);
    if(pass + 1 <= kMaxRuns)
      c.runStarts[pass + 1] = part;
  }
  b->splitWriteCounter   = write;
  b->partTriangleCounter = part;
  if(trans)
    b->dualPartTriangleCounter = dual;
  if(lv.levels > 1)
  {
    b->splitPass             = pass;
    b->splitPassStart        = start;
    b->splitPassEnd          = end;
    b->dispatchTriangleSplit = {(end - start + 63) / 64, 1, 1};
  }
  if(c.fuseSetup != kNoSetup)
    build_setup_apply(c, c.fuseSetup);
}

// Level L, of items up to `end`, is complete (every tile done, or none): the
// next level's item range and counters, published with release semantics.
// Run by one thread.
__device__ void publish_level(const StageCtx& c, const SplitLevels& lv, u32 L, u32 end, u32 numTiles)
{
  if(L + 1 >= lv.levels)
    return;
  const u32 most = c.caps.maxSplitTriangles;
  // another block's last tile wrote the totals: read them through L2
  u32 write, part;
  if(numTiles)
    write = (u32)__ldcg(lv_totals(lv, L) + kCntSplit), part = (u32)__ldcg(lv_totals(lv, L) + kCntPart);
  else  // (not level 0: without split items no level is published)
    write = __ldcg(lv_bases(lv, L) + kCntSplit), part = __ldcg(lv_bases(lv, L) + kCntPart);
  u32* next = lv.ctrl[L + 1];
  next[6 + kCntSplit] = write, next[6 + kCntPart] = part;
  const u32 first = min(end, most), last = min(write, most);
  *lv_places(lv, L + 1) = last > first ? __ldcg(c.splitEnds + last - 1) : 0ull;
  next[13] = first, next[14] = last;
  __threadfence();
  st_release_u32(lv_ready(lv, L), 1u);
}

template <int B>
__global__ void __launch_bounds__(B) k_triangle_split_levels(StageCtx c, SplitLevels lv)
{
  stage_prologue();
  __shared__ SplitShared<B> sm;
  __shared__ Level          s_lv;
  __shared__ u32            s_level[3];  // level, its first ticket, status (1: stop)
  const u32          partCap  = part_cap(c);
  const FactorParams fp       = split_factor_params(c);
  const u32          sf       = clamp_split_factor(c.caps.splitFactor);
  const u32          levels   = lv.levels;
  u32*               indexed  = lv.ctrl[0] + kIndexWords;

  // level 0: the range the classify set-up (BUILD_SETUP_SPLIT) left, unless
  // the launch is complete and the range already the last level's (the flag is
  // read after the range, and set before it changes)
  if(threadIdx.x == 0)
  {
    const volatile tc_SceneBuilding* b = c.build;
    const u32 hi = min(b->splitPassEnd, c.caps.maxSplitTriangles), lo = min(b->splitPassStart, hi);
    __threadfence();
    sm.range[0] = lo, sm.range[1] = hi;
    sm.flag = ld_acquire_u32(lv.ctrl[0] + 15);
  }
  __syncthreads();
  const u32 begin0 = sm.range[0], end0 = sm.range[1];
  if(sm.flag)
    return;
  if(begin0 == end0)
  {
    // no split item: every level is empty; one block runs the passes' set-ups
    if(blockIdx.x == 0 && threadIdx.x == 0)
      finalize_levels(c, lv, partCap);
    return;
  }
  const bool own      = end0 - begin0 <= kIndexLocalTiles * B;
  const u32  idxTiles = own ? 0u : (end0 - begin0 + B - 1) / B;
  Level      cur      = {};
  u32        level    = 0, first = idxTiles;
  if(own)
    cur = make_level<B>(begin0, end0, index_local<B>(c, sm, begin0, end0), c.splitFirst, lv.stride);

  for(;;)
  {
    const u32 g = next_tile(c, &sm.tile);  // one ticket over the index and all levels
    if(g < idxTiles)
    {
      index_tile<B>(c, sm, lv.lbState[0] + (u64)kRowScan * lv.stride, g, begin0, end0);
      if(threadIdx.x == 0)
      {
        __threadfence();
        if(atomicAdd(indexed, 1u) == idxTiles - 1)
          st_release_u32(indexed + 1, 1u);
      }
      continue;
    }
    // the level of ticket g (later levels wait for the earlier ones' completion)
    if(threadIdx.x == 0)
    {
      u32 stop = 0;
      if(cur.first == nullptr)  // level 0's index
      {
        stop = wait_flag(c, indexed + 1) ? 0u : 1u;
        if(!stop)
          cur = make_level<B>(begin0, end0, __ldcg(c.splitEnds + end0 - 1), c.splitFirst, lv.stride);
      }
      while(!stop && g >= first + cur.tiles)
      {
        // level `level` has no tile for this ticket: move on to the next one
        if(cur.tiles == 0 && atomicCAS(lv_final(lv, level), 0u, 1u) == 0u)
        {
          __threadfence();
          publish_level(c, lv, level, cur.end, 0);
          if(level + 1 == levels)
            finalize_levels(c, lv, partCap);
        }
        first += cur.tiles;
        if(++level >= levels || !wait_flag(c, lv_ready(lv, level - 1)))
        {
          stop = 1;
          break;
        }
        const u32* w = lv.ctrl[level];
        const u32  lo = __ldcg(w + 13), hi = __ldcg(w + 14);
        cur = make_level<B>(lo, hi, __ldcg(lv_places(lv, level)), c.splitFirst + c.splitFirstStride * (1 + (level & 1)), lv.stride);
      }
      s_lv       = cur;
      s_level[0] = level, s_level[1] = first, s_level[2] = stop;
    }
    __syncthreads();
    if(s_level[2])
      break;
    cur   = s_lv;
    level = s_level[0];
    first = s_level[1];
    split_tile<B>(c, sm, g - first, cur, lv.lbState[level], lv.stride, lv_totals(lv, level),
                  level ? lv_bases(lv, level) : nullptr,
                  level + 1 < levels ? c.splitFirst + c.splitFirstStride * (1 + ((level + 1) & 1)) : nullptr, fp, sf,
                  partCap);
    // the block completing the level's last tile publishes the next level
    if(threadIdx.x == 0)
    {
      __threadfence();
      if(atomicAdd(lv_done(lv, level), 1u) == cur.tiles - 1)
      {
        __threadfence();
        publish_level(c, lv, level, cur.end, cur.tiles);
        if(level + 1 == levels)
          finalize_levels(c, lv, partCap);
      }
    }
    __syncthreads();
  }
}

}  // namespace

cudaError_t launch_triangle_split_levels(const StageCtx& c, const SplitLevels& lv, u32 blockSize, u32 grid, cudaStream_t s)
{
  const int prio = high_launch_priority();
  switch(blockSize)
  {
    case 128:
      return launch_pdl_prio(k_triangle_split_levels<128>, grid, 128, prio, s, c, lv);
    case 512:
      return launch_pdl_prio(k_triangle_split_levels<512>, grid, 512, prio, s, c, lv);
    default:
      return launch_pdl_prio(k_triangle_split_levels<256>, grid, 256, prio, s, c, lv);
  }
}

cudaError_t launch_triangle_split(const StageCtx& c, u32 blockSize, u32 grid, cudaStream_t s)
{
  // the split passes are the latency-critical branch of the frame: their
  // blocks take precedence over the concurrent instantiation's
  const int prio = high_launch_priority();
  switch(blockSize)
  {
    case 128:
      return launch_pdl_prio(k_triangle_split<128>, grid, 128, prio, s, c);
    case 512:
      return launch_pdl_prio(k_triangle_split<512>, grid, 512, prio, s, c);
    default:
      return launch_pdl_prio(k_triangle_split<256>, grid, 256, prio, s, c);
  }
}

}  // namespace tc
