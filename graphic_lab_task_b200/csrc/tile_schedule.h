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
// their cost against the previous launch's longest tile (at least 1/2, 1/4,
// 1/8 of it); the next launch of the same image size on the same stream
// (rd) hands out class 0, then 1, then 2, each in the order the tiles
// finished, then every other tile in natural order (a bitmap skips the
// listed ones).  If the previous launch was tail-bound (its longest tile
// took longer than its warps' mean busy time), a class-0 tile goes out as
// 2, 4 or 8 work items, each traced by one warp on its own rows (or half
// rows) of the tile; the parts' costs add up in the tile's accumulator and the last part
// to finish records the tile.  Only which warp traces which ray, and when,
// depends on it.
// rd == nullptr: natural order; wr == nullptr: nothing recorded.  Buffer
// layout: sched_words and the offsets beside it (device_layout.h).  The
// per-warp state lives in shared memory so that the traversal keeps its
// registers.
//
// A work item is a tile index with, for the part of a split tile, bit 31 set
// log2 of its parts in bits 28..29 and the part in bits 24..27 (tile counts
// stay below 2^24).
struct WarpClock {
  long long start;  // clock64 when the warp took its current item
  uint32_t item;    // that item, ~0u before the first
  uint32_t longest; // longest tile this warp has reported
  uint32_t pos;     // a split item's position in the concatenated class lists
  unsigned long long busy; // sum of the costs of the items this warp traced
};
constexpr uint32_t kItemSplit = 0x80000000u;
constexpr uint32_t kItemTileMask = 0x00FFFFFFu;

__device__ __forceinline__ uint32_t item_tile(uint32_t item) { return item & kItemTileMask; }

// Whether `lane` traces its pixel of the item's tile: every lane for a whole
// tile, its part's share of them for a part.
__device__ __forceinline__ bool item_has_lane(uint32_t item, uint32_t lane)
{
  return !(item & kItemSplit) || lane >> (5u - ((item >> 28) & 3u)) == ((item >> 24) & 0xFu);
}

// lane 0: records that a tile took `cost` (longest, class list, bitmap).
__device__ __forceinline__ void sched_record(const uint32_t* __restrict__ rd, uint32_t* wr, uint32_t tiles,
                                             uint32_t tile, uint32_t cost, WarpClock& wc)
{
  const uint64_t lists = sched_lists_offset(tiles);
  if (cost > wc.longest) {
    wc.longest = cost;
    atomicMax(wr, cost);
  }
  const uint32_t mx = rd ? __ldg(rd) : 0u;
  if (mx) {
    const int cls = cost >= mx / 2 ? 0 : cost >= mx / 4 ? 1 : cost >= mx / 8 ? 2 : 3;
    if (cls < 3) {
      const uint32_t slot = atomicAdd(wr + 1 + cls, 1u);
      if (slot < tiles) wr[lists + cls * tiles + slot] = tile;
      atomicOr(wr + kSchedHeader + (tile >> 5), 1u << (tile & 31));
    }
  }
}

// In how many parts (log2) the previous launch's class-0 tiles go out, by how
// far its longest tile outlasted its warps' mean busy time: whole tiles if it
// did not, else 2, and in scenes without bricks from 2 times on 4 and from 4
// times on 8 (one row is the least that keeps a part's pixels together).
// Parts repeat the node loads that a whole tile shares, which a launch that is
// hardly tail-bound pays for: in 2 / 4 / 8 parts an animated 256-instance frame
// took 457 / 500 / 588 us, a 200k-triangle mesh at 256^2 in image order 194 /
// 175 / 128, a voxel set at 1001x777 231 / 193 / 196.  Bricks share most (512^3
// at 1920x1080 393 / 418 us in 2 / 4 parts), and mixed scenes lose when the
// schedule comes from another view (1,742 -> 1,913 us in up to 8).
template <uint32_t KIND>
__device__ __forceinline__ uint32_t split_log2(const uint32_t* __restrict__ rd)
{
  if (!rd) return 0u;
  const uint64_t span = uint64_t(__ldg(rd)) * __ldg(rd + kSchedWarps);
  const uint64_t busy = __ldg(reinterpret_cast<const unsigned long long*>(rd + kSchedBusy));
  if (span <= busy) return 0u;
  if (KIND != kKindNoBricks) return 1u;
  return span > 4 * busy ? 3u : span > 2 * busy ? 2u : 1u;
}

// lane 0, after the warp has finished its current item (if any): records
// that item's duration and returns the next item of `tiles`, ~0u when none
// is left.
template <uint32_t KIND>
__device__ __forceinline__ uint32_t sched_next(const uint32_t* __restrict__ rd, uint32_t* wr, uint32_t tiles,
                                               unsigned long long* counter, WarpClock& wc)
{
  const uint64_t lists = sched_lists_offset(tiles);
  const uint32_t lg = split_log2<KIND>(rd), parts = 1u << lg;
  if (wr && wc.item != ~0u) {
    const long long dt = (clock64() - wc.start) >> 4;
    uint32_t cost = uint32_t(dt < 0xFFFFFFFFll ? dt : 0xFFFFFFFFll);
    bool record = true;
    wc.busy += cost;
    if (wc.item & kItemSplit) { // parts add up; the last one records the tile
      unsigned long long* acc = reinterpret_cast<unsigned long long*>(wr + sched_acc_offset(tiles));
      const unsigned long long prev = atomicAdd(acc + wc.pos, (1ull << 40) | cost);
      record = (prev >> 40) + 1 == parts;
      const unsigned long long sum = (prev & ((1ull << 40) - 1)) + cost;
      cost = uint32_t(sum < 0xFFFFFFFFull ? sum : 0xFFFFFFFFull);
    }
    if (record) sched_record(rd, wr, tiles, item_tile(wc.item), cost, wc);
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
