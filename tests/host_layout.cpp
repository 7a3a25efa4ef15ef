// Checks of the host builders of the derived layouts that need no GPU; built
// and run by test_host_layout.py.  Prints one line per check that fails.
#include <cstdio>
#include <cstring>

#include "layout.h"

using namespace lrt;

static int failed = 0;
static void expect(bool ok, const char* what)
{
  if (ok) return;
  std::printf("%s\n", what);
  failed++;
}

// A leaf table with a gap and with entries of no triangles that start anywhere.
static void slots()
{
  HostArrays h;
  h.geomData.resize(1);
  std::memset(&h.geomData[0], 0, sizeof(lrt_geom_data));
  h.geomTags = {LRT_TAG_TRIANGLE};
  h.startEnd = {0, 4};
  h.primIdCount = {0x20000000u | 1u, 0x0FFFFFF0u, 0x80000000u | 0x0FFFFFFFu, 0x90000000u | 9u};
  expect(triangle_slots(h, 0) == 10, "entries of no triangles count as triangle slots");
  h.primIdCount = {0x0FFFFFF0u, 5u, 0u, 0x80000000u};
  expect(triangle_slots(h, 0) == 0, "a table of no triangles has slots");
}

// Rays to a warp around the sizes from which a launch takes larger groups,
// whatever the scene's kernels (28 warps on each of 148 SMs).
static void rows()
{
  const struct {
    uint64_t n;
    uint32_t group;
  } want[] = {{1, 8},      {33152, 8},  {33153, 16}, {47000, 16},  {56832, 16},
              {65536, 16}, {66304, 16}, {66305, 32}, {262144, 32}, {1ull << 33, 32}};
  for (const auto& w : want) expect(rays_per_warp(w.n, 148) == w.group, "rays to a warp");
  expect(rays_per_warp(66304, 74) == 32, "rays to a warp of half the SMs");
}

int main()
{
  slots();
  rows();
  return failed;
}
