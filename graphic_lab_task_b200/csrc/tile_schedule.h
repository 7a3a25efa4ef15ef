// tile_schedule.h — the order in which the warps of an image-order launch take
// its tiles.  Device code that names nothing but the schedule's buffers and a
// few intrinsics, so that it can be run on the host as well, with a clock and
// warps of the caller's making.
#pragma once
#include <stdint.h>

#include "device_layout.h"

namespace lrt {

// Longest-first order of the tiles of an image-order launch.  Each launch
// times its tiles on lane 0 and sorts the slow ones into three classes by
// their cost against the previous launch's longest tile (at least 5/8, 3/8,
// 1/8 of it); the next launch of the same image size on the same stream
// (rd) hands out class 0, then 1, then 2, each in the order the tiles
// finished, then every other tile in natural order (a bitmap skips the
// listed ones).  If the previous launch was tail-bound (its longest tile
// took longer than its warps' mean busy time), a class-0 tile goes out as
// 2, 4 or 8 work items, each traced by one warp on its own rows (or half
// rows) of the tile; the parts' costs add up in the tile's accumulator and the
// last part to finish records the tile.  Only which warp traces which ray, and when,
// depends on it.
// rd == nullptr: natural order; wr == nullptr: nothing recorded.  Buffer
// layout: sched_words and the offsets beside it (device_layout.h).  The
// per-warp state lives in shared memory so that the traversal keeps its
// registers.
//
// A work item is a tile index (below 2^31: more tiles than fit any memory) or
// the part of a split tile: bit 31, log2 of the parts in bits 28..29, the part
// in bits 24..27 and the tile below them, so that launches of more than 2^24
// tiles split none.
struct WarpClock {
  long long start;  // clock64 when the warp took its current item
  uint32_t item;    // that item, ~0u before the first
  uint32_t longest; // longest tile this warp has reported
  uint32_t level;   // log2 of the parts that this launch splits tiles into
  uint32_t pos;     // a split item's position in the concatenated class lists
  unsigned long long busy; // sum of the costs of the items this warp traced
};
constexpr uint32_t kItemSplit = 0x80000000u;
constexpr uint32_t kItemTileMask = 0x00FFFFFFu;

__device__ __forceinline__ uint32_t item_tile(uint32_t item)
{
  return item & kItemSplit ? item & kItemTileMask : item;
}

// Whether `lane` traces its pixel of the item's tile: every lane for a whole
// tile, its part's share of them for a part.
__device__ __forceinline__ bool item_has_lane(uint32_t item, uint32_t lane)
{
  return !(item & kItemSplit) || lane >> (5u - ((item >> 28) & 3u)) == ((item >> 24) & 0xFu);
}

// lane 0: records that a tile took `cost` (longest, class list, bitmap).
// `listed`, no less than that for a split tile, is what its class goes by.
__device__ __forceinline__ void sched_record(const uint32_t* __restrict__ rd, uint32_t* wr, uint32_t tiles,
                                             uint32_t tile, uint32_t cost, uint32_t listed, WarpClock& wc)
{
  const uint64_t lists = sched_lists_offset(tiles);
  if (cost > wc.longest) {
    wc.longest = cost;
    atomicMax(wr, cost);
  }
  const uint32_t mx = rd ? __ldg(rd) : 0u;
  if (mx) {
    const int cls = listed >= mx / 8 * 5 ? 0 : listed >= mx / 8 * 3 ? 1 : listed >= mx / 8 ? 2 : 3;
    if (cls < 3) {
      const uint32_t slot = atomicAdd(wr + 1 + cls, 1u);
      if (slot < tiles) wr[lists + cls * tiles + slot] = tile;
      atomicOr(wr + kSchedHeader + (tile >> 5), 1u << (tile & 31));
    }
  }
}

// What a tile traced in 2^lg parts would have cost whole, from the sum of its
// parts: they repeat the node loads that a whole tile shares, so that the sum
// grows with the level, by about 1.5 for each (the longest tile's in 2 / 4 / 8
// parts against whole: a 200k-triangle mesh at 256^2 1.4 / 1.7 / 2.1, at
// 1920x1080 1.4 / 2.3 / 3.2, voxel sets 1.6 / 2.5 / 4.1 and 1.7 / 3.2 / 5.2,
// 256 instances 1.4 / 2.1 / 2.8, 512^3 bricks 1.6 / 2.7 / 3.6).  Split levels
// and the bounds of the classes are of whole tiles' costs: from the plain sums
// a split tile looked longer than it was and was split further, while the
// tiles that became slow beside it as the camera moved stayed below its class.
__device__ __forceinline__ uint32_t whole_cost(uint64_t sum, uint32_t lg)
{
  const float whole = float(sum) * (lg == 1 ? 0.6667f : lg == 2 ? 0.4444f : 0.2963f);
  return whole < 4e9f ? uint32_t(whole) : 4000000000u;
}

// What a split tile's class goes by: enough of the sum to keep it in class 0
// (5/8 of the longest) if its parts share nothing, so that a tile whose parts
// are cheap is not whole again in every other launch.  (The whole sum in 2
// parts: multi-layer renders of 256^3 bricks at 1920x1080 5,070 -> 5,700 us; 1.25
// of the whole cost for all: repeated rows of 256 instances 185 -> 206.)
__device__ __forceinline__ uint32_t listed_cost(uint64_t sum, uint32_t lg)
{
  const float cost = float(sum) * (lg == 1 ? 0.8f : lg == 2 ? 0.72f : 0.64f);
  return cost < 4e9f ? uint32_t(cost) : 4000000000u;
}

// In how many parts (log2) the class-0 tiles of a launch go out, from the
// longest tile of the launch before, its warps, their busy time and its level:
// whole if that tile took no longer than the warps' mean busy time, else 2, and
// from 2 times on 4 and from 3 times on 8 parts (half rows), as far as `most`.
// A level is left at half the cost from which it is taken, so that repeated
// launches settle: the sum's factor differs by half between scenes.
// Measured in 2 / 4 / 8 parts (us; longest tile in mean busy times): 1.5, 256
// moving instances 484 / 534 / 558 (whole 575); 1.5, voxel set at 1920x1080
// 272 / 275 / 302 (278); 2.7, voxel set at 1001x777 284 / 263 / 249 (312);
// 3.0, mesh at 1920x1080 in rows 307 / 288 / 319 (349); 3.6, 256 instances
// 251 / 218 / 230 (316); 3.8, mesh at 1920x1080 321 / 270 / 231 (364); 17, mesh
// at 256^2 198 / 183 / 166 (204).
inline __host__ __device__ uint32_t split_level(uint32_t was, uint64_t longest, uint64_t warps, uint64_t busy,
                                                uint32_t most)
{
  const uint64_t span = longest * warps;
  uint32_t lg = 0;
  while (lg < most && 2 * span > (lg < was ? 1 : 2) * (lg + 1) * busy) lg++;
  return lg;
}

// The most parts (log2), by the scene's geometry kind: bricks share most of
// their loads (512^3 at 1920x1080, camera moving, 451 / 458 / 469 us in 2 / 4 /
// 8 parts), and mixed scenes lose when the schedule comes from another view
// (1280x720, two views in turn, 563 / 642 / 643 us).
template <uint32_t KIND>
__device__ __forceinline__ uint32_t split_log2(const uint32_t* __restrict__ rd, uint32_t tiles)
{
  if (!rd || tiles > kItemTileMask + 1) return 0u;
  return split_level(__ldg(rd + kSchedLevel), __ldg(rd), __ldg(rd + kSchedWarps),
                     __ldg(reinterpret_cast<const unsigned long long*>(rd + kSchedBusy)),
                     KIND == kKindNoBricks ? 3u : 1u);
}

// lane 0, after the warp has finished its current item (if any): records
// that item's duration and returns the next item of `tiles`, ~0u when none
// is left.
template <uint32_t KIND>
__device__ __forceinline__ uint32_t sched_next(const uint32_t* __restrict__ rd, uint32_t* wr, uint32_t tiles,
                                               unsigned long long* counter, WarpClock& wc)
{
  const uint64_t lists = sched_lists_offset(tiles);
  if (wc.item == ~0u) wc.level = split_log2<KIND>(rd, tiles); // the warp's first item
  const uint32_t lg = wc.level, parts = 1u << lg;
  if (wr && wc.item != ~0u) {
    const long long dt = (clock64() - wc.start) >> 4;
    uint32_t cost = uint32_t(dt < 0xFFFFFFFFll ? dt : 0xFFFFFFFFll);
    uint32_t listed = cost;
    bool record = true;
    wc.busy += cost;
    if (wc.item & kItemSplit) { // parts add up; the last one records the tile
      unsigned long long* acc = reinterpret_cast<unsigned long long*>(wr + sched_acc_offset(tiles));
      const unsigned long long prev = atomicAdd(acc + wc.pos, (1ull << 40) | cost);
      record = (prev >> 40) + 1 == parts;
      const uint64_t sum = (prev & ((1ull << 40) - 1)) + cost;
      cost = whole_cost(sum, lg);
      listed = listed_cost(sum, lg);
    }
    if (record) sched_record(rd, wr, tiles, item_tile(wc.item), cost, listed, wc);
  }
  static_assert(kSchedClasses == 3, "three cost classes");
  uint32_t n[3] = {0, 0, 0};
  if (rd)
    for (int c = 0; c < 3; c++) n[c] = min(__ldg(rd + 1 + c), tiles);
  const uint64_t nAll = uint64_t(n[0]) + n[1] + n[2];
  const uint64_t nSplit = lg ? n[0] : 0;
  const uint64_t nItems = nSplit * parts + (nAll - nSplit);
  for (;;) {
    const unsigned long long k = atomicAdd(counter, 1ull);
    uint32_t item;
    if (k < nItems) {
      const bool split = k < nSplit * parts;
      const uint64_t j = split ? k / parts : k - nSplit * (parts - 1);
      const int cls = j < n[0] ? 0 : j < uint64_t(n[0]) + n[1] ? 1 : 2;
      const uint64_t jj = cls == 0 ? j : cls == 1 ? j - n[0] : j - n[0] - n[1];
      const uint32_t tile = __ldg(rd + lists + cls * tiles + jj);
      if (tile >= tiles) continue;
      item = split ? tile | kItemSplit | (lg << 28) | (uint32_t(k & (parts - 1)) << 24) : tile;
      wc.pos = uint32_t(j);
    } else {
      if (k - nItems >= tiles) { // none left: report this warp's busy time
        if (wr) {
          atomicAdd(reinterpret_cast<unsigned long long*>(wr + kSchedBusy), wc.busy);
          atomicAdd(wr + kSchedWarps, 1u);
          wr[kSchedLevel] = lg; // (every warp's)
        }
        return wc.item = ~0u;
      }
      item = uint32_t(k - nItems);
      if (nAll && ((__ldg(rd + kSchedHeader + (item >> 5)) >> (item & 31)) & 1u)) continue;
    }
    wc.start = clock64();
    return wc.item = item;
  }
}

} // namespace lrt
