// Runs the tile schedule's device code on the host: warps in simulated time
// take the items of an image-order launch until none is left.  Built and run
// by test_host_schedule.py; prints one line per check that fails.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <functional>
#include <queue>
#include <vector>

#include <cuda_runtime.h>

using std::min;
static long long g_clock;
static long long clock64() { return g_clock; }
template <class T>
static T __ldg(const T* p)
{
  return *p;
}
template <class T>
static T atomicAdd(T* p, T v)
{
  const T old = *p;
  *p += v;
  return old;
}
static void atomicMax(uint32_t* p, uint32_t v) { *p = std::max(*p, v); }
static void atomicOr(uint32_t* p, uint32_t v) { *p |= v; }

#include "tile_schedule.h"

using namespace lrt;

static int failed = 0;
static void expect(bool ok, const char* what, long long a = 0, long long b = 0)
{
  if (ok) return;
  std::printf("%s (%lld, %lld)\n", what, a, b);
  failed++;
}

struct Launch {
  std::vector<uint32_t> wr;
  std::vector<uint32_t> lanes;   // per tile: the lanes that were traced
  std::vector<uint32_t> items;   // per tile: in how many items
  uint64_t busy = 0;             // of all warps, in the schedule's unit
  long long span = 0;            // when the last warp ended
};

// One launch of `tiles` tiles on `warps` warps; cost(tile, lanes) in clocks / 16.
template <uint32_t KIND>
Launch run(uint32_t tiles, uint32_t warps, const uint32_t* rd, const std::function<uint32_t(uint32_t, uint32_t)>& cost)
{
  Launch L;
  L.wr.assign(sched_words(tiles), 0u);
  L.lanes.assign(tiles, 0u);
  L.items.assign(tiles, 0u);
  std::vector<WarpClock> wc(warps);
  for (WarpClock& w : wc) {
    std::memset(&w, 0, sizeof(w));
    w.item = ~0u;
  }
  typedef std::pair<long long, uint32_t> At; // time, warp
  std::priority_queue<At, std::vector<At>, std::greater<At>> next;
  for (uint32_t w = 0; w < warps; w++) next.push({0, w});
  unsigned long long counter = 0;
  while (!next.empty()) {
    const auto [now, w] = next.top();
    next.pop();
    g_clock = now;
    const uint32_t item = sched_next<KIND>(rd, L.wr.data(), tiles, &counter, wc[w]);
    if (item == ~0u) {
      L.span = std::max(L.span, now / 16);
      continue;
    }
    const uint32_t tile = item_tile(item);
    if (tile >= tiles) {
      expect(false, "item past the last tile", tile, tiles);
      break;
    }
    uint32_t mask = 0;
    for (uint32_t lane = 0; lane < 32; lane++)
      if (item_has_lane(item, lane)) mask |= 1u << lane;
    expect(!(L.lanes[tile] & mask), "a lane is traced twice", tile, mask);
    L.lanes[tile] |= mask;
    L.items[tile]++;
    const uint32_t c = cost(tile, mask);
    L.busy += c;
    next.push({now + 16ll * c, w});
  }
  uint64_t told = 0;
  std::memcpy(&told, &L.wr[kSchedBusy], 8);
  for (uint32_t t = 0; t < tiles; t++) expect(L.lanes[t] == ~0u, "a tile is not traced whole", t, L.lanes[t]);
  expect(told == L.busy, "the warps' busy time is not what their items took", told, L.busy);
  expect(L.wr[kSchedWarps] == warps, "warps that reported", L.wr[kSchedWarps], warps);
  return L;
}

// A few slow tiles, whose parts take their share of the time.
static uint32_t slow_tiles(uint32_t tile, uint32_t lanes)
{
  const uint32_t whole = tile % 97 == 5 ? 6400 : 64 + tile % 7;
  return std::max(1u, whole * uint32_t(__builtin_popcount(lanes)) / 32);
}

template <uint32_t KIND>
static void launches(uint32_t tiles, uint32_t warps)
{
  std::vector<uint32_t> prev;
  for (int k = 0; k < 6; k++) {
    Launch L = run<KIND>(tiles, warps, prev.empty() ? nullptr : prev.data(), slow_tiles);
    prev = L.wr;
  }
}

int main()
{
  for (uint32_t tiles : {1u, 31u, 32u, 300u, 2048u})
    for (uint32_t warps : {1u, 7u, 64u, 600u}) {
      launches<kKindNoBricks>(tiles, warps);
      launches<kKindBricks>(tiles, warps);
      launches<kKindAll>(tiles, warps);
    }
  return failed != 0;
}
