// Runs the tile schedule's device code on the host: warps in simulated time
// take the items of an image-order launch until none is left.  Built and run
// by test_host_schedule.py; prints one line per check that fails.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <queue>
#include <vector>

#include <cuda_runtime.h>

using std::max;
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
  if (failed > 40) std::exit(1);
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

// Repeats of one launch: every tile is traced once whatever the level, and the
// level settles.  Returns it.
template <uint32_t KIND>
static uint32_t launches(uint32_t tiles, uint32_t warps, const std::function<uint32_t(uint32_t, uint32_t)>& cost,
                         long long* spans = nullptr)
{
  std::vector<uint32_t> prev;
  uint32_t level = 0;
  for (int k = 0; k < 20; k++) {
    Launch L = run<KIND>(tiles, warps, prev.empty() ? nullptr : prev.data(), cost);
    if (k > 8) expect(L.wr[kSchedLevel] == level, "the split level does not settle", L.wr[kSchedLevel], level);
    level = L.wr[kSchedLevel];
    const uint32_t most = *std::max_element(L.items.begin(), L.items.end());
    expect(most <= 1u << level, "more parts than the level's", most, 1u << level);
    if (spans && (k == 0 || k == 19)) spans[k != 0] = L.span;
    prev = L.wr;
  }
  return level;
}

// A launch that starts from a planted level, all tiles listed in class 0.
template <uint32_t KIND>
static void planted(uint32_t tiles, uint32_t warps, uint32_t was, uint32_t longest, uint64_t busy, uint32_t want)
{
  std::vector<uint32_t> rd(sched_words(tiles), 0u);
  rd[0] = longest;
  rd[1] = tiles;
  rd[kSchedWarps] = warps;
  rd[kSchedLevel] = was;
  std::memcpy(&rd[kSchedBusy], &busy, 8);
  for (uint32_t t = 0; t < tiles; t++) {
    rd[sched_lists_offset(tiles) + t] = tiles - 1 - t;
    rd[kSchedHeader + t / 32] |= 1u << (t % 32);
  }
  Launch L = run<KIND>(tiles, warps, rd.data(), slow_tiles);
  expect(L.wr[kSchedLevel] == want, "level after a planted schedule", L.wr[kSchedLevel], want);
  for (uint32_t t = 0; t < tiles; t++) expect(L.items[t] == 1u << want, "parts of a planted tile", L.items[t], want);
}

int main()
{
  for (uint32_t tiles : {1u, 31u, 32u, 300u, 2048u})
    for (uint32_t warps : {1u, 7u, 64u, 600u}) {
      launches<kKindNoBricks>(tiles, warps, slow_tiles);
      launches<kKindBricks>(tiles, warps, slow_tiles);
      launches<kKindAll>(tiles, warps, slow_tiles);
    }
  // the slowest tiles take little more than the mean busy time, and their
  // parts repeat much of what a whole tile shares: from the sums the level
  // would grow to the most
  auto shared = [](uint32_t tile, uint32_t lanes) {
    const uint32_t n = uint32_t(__builtin_popcount(lanes));
    return tile % 50 == 0 ? 270 + 17 * n : 100u;
  };
  long long span[2];
  uint32_t lg = launches<kKindNoBricks>(2000, 400, shared, span);
  expect(lg == 1 && span[1] < span[0], "launch whose parts share most of their time", lg, span[1]);
  lg = launches<kKindNoBricks>(2000, 20, shared, span);
  expect(lg == 0, "balanced launch", lg);
  lg = launches<kKindNoBricks>(2048, 2048, slow_tiles, span);
  expect(lg == 3 && 4 * span[1] < span[0], "launch as long as its slowest tiles", lg, span[1]);
  // tiles that become slow are split like those that were: the same number
  // of other tiles is slow in every launch
  std::vector<uint32_t> prev;
  for (int k = 0; k < 8; k++) {
    auto moving = [k](uint32_t tile, uint32_t lanes) {
      const bool slow = tile % 97 == 5 || tile % 97 == 40 + uint32_t(k) || tile % 97 == 41 + uint32_t(k);
      return (slow ? 3200u : 64u) * uint32_t(__builtin_popcount(lanes)) / 32 + (slow ? 500u : 0u);
    };
    Launch L = run<kKindNoBricks>(970, 500, prev.empty() ? nullptr : prev.data(), moving);
    if (k > 2) expect(L.items[41 + k] == 1 && L.items[40 + k] == 8, "tile that was slow is not split", k, L.items[40 + k]);
    prev = L.wr;
  }
  // a mean busy time of 100: a level is taken above once, twice and three
  // times it and left at half of that
  for (uint32_t was = 0; was < 4; was++) {
    planted<kKindNoBricks>(100, 10, was, 301, 1000, 3);
    planted<kKindNoBricks>(100, 10, was, 300, 1000, was == 3 ? 3 : 2);
    planted<kKindNoBricks>(100, 10, was, 201, 1000, was == 3 ? 3 : 2);
    planted<kKindNoBricks>(100, 10, was, 150, 1000, was > 1 ? 2 : 1);
    planted<kKindNoBricks>(100, 10, was, 101, 1000, was > 1 ? 2 : 1);
    planted<kKindNoBricks>(100, 10, was, 100, 1000, was > 0 ? 1 : 0);
    planted<kKindNoBricks>(100, 10, was, 51, 1000, was > 0 ? 1 : 0);
    planted<kKindNoBricks>(100, 10, was, 50, 1000, 0);
  }
  for (uint32_t was = 0; was < 2; was++) {
    planted<kKindAll>(33, 10, was, 900, 1000, 1);
    planted<kKindBricks>(33, 10, was, 900, 1000, 1);
    planted<kKindBricks>(33, 10, was, 50, 1000, 0);
  }
  // more tiles than a part's item can number
  std::vector<uint32_t> head(kSchedHeader, 0u);
  head[0] = 1000;
  head[kSchedWarps] = head[kSchedBusy] = 1;
  const uint32_t many = (1u << 24) + 40;
  std::vector<uint32_t> rd(sched_words(many), 0u);
  std::copy(head.begin(), head.end(), rd.begin());
  rd[1] = 2; // two of them listed
  rd[sched_lists_offset(many)] = 7;
  rd[sched_lists_offset(many) + 1] = many - 1;
  rd[kSchedHeader] = 1u << 7;
  rd[kSchedHeader + (many - 1) / 32] = 1u << (many - 1) % 32;
  for (uint32_t first : {0u, (1u << 24) - 2}) {
    WarpClock wc;
    std::memset(&wc, 0, sizeof(wc));
    wc.item = ~0u;
    unsigned long long counter = first;
    std::vector<uint32_t> got;
    for (int k = 0; k < 60 && (k == 0 || wc.item != ~0u); k++) {
      const uint32_t item = sched_next<kKindNoBricks>(rd.data(), nullptr, many, &counter, wc);
      if (item == ~0u) break;
      expect(item_has_lane(item, 0) && item_has_lane(item, 31), "a tile of a launch of many tiles is split", item);
      got.push_back(item_tile(item));
    }
    std::vector<uint32_t> want;
    if (first == 0)
      want = {7, many - 1, 0, 1, 2, 3, 4, 5, 6, 8, 9}; // the listed ones first
    else
      for (uint32_t t = first - 2; t < many - 1; t++) want.push_back(t);
    got.resize(std::min(got.size(), want.size()));
    expect(got == want, "tiles of a launch of many tiles", got.empty() ? 0 : got.back(), want.back());
  }
  return failed != 0;
}
