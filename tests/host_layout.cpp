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

int main()
{
  slots();
  return failed;
}
