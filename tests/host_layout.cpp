// Checks of the host builders of the derived layouts that need no GPU; built
// and run by test_host_layout.py.  Prints one line per check that fails.
#include <cmath>
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

// A scene of meshes whose tables have gaps, empty entries and more leaves than
// a block of the soup's kernel, in slots of their own or shared.
static HostArrays meshes(bool shared)
{
  HostArrays h;
  const uint32_t leaves[3] = {1, 257, 600};
  for (uint32_t g = 0; g < 3; g++) {
    lrt_geom_data gd;
    std::memset(&gd, 0, sizeof(gd));
    gd.offset[0] = shared && g == 2 ? h.geomData[1].offset[0] : uint32_t(h.indices.size());
    gd.offset[1] = uint32_t(h.vertPos.size() / 4);
    h.geomData.push_back(gd);
    h.geomTags.push_back(LRT_TAG_TRIANGLE);
    h.startEnd.push_back(uint32_t(h.primIdCount.size()));
    uint32_t slot = 0;
    for (uint32_t l = 0; l < leaves[g]; l++) {
      const uint32_t cnt = l % 8;
      h.primIdCount.push_back(0x80000000u | (cnt << 28) | (cnt ? slot : 0x0FFFFFFFu));
      slot += cnt + l % 3; // a gap after two of three
    }
    h.startEnd.push_back(uint32_t(h.primIdCount.size()));
    for (uint32_t v = 0; v < 50 * 4; v++) h.vertPos.push_back(float(v * (g + 1)) * 0.37f);
    if (shared && g == 2) h.indices.resize(gd.offset[0]);
    for (uint32_t i = 0; i < 3 * slot; i++) h.indices.push_back(0xFFFFFF00u);
    for (uint32_t l = 0; l < leaves[g]; l++) {
      const uint32_t pk = h.primIdCount[h.startEnd[2 * g] + l], cnt = (pk >> 28) & 7u;
      for (uint32_t t = pk & kStartMask; cnt && t < (pk & kStartMask) + cnt; t++)
        for (uint32_t c = 0; c < 3; c++) h.indices[gd.offset[0] + 3 * t + c] = (7 * t + 13 * c + l) % 50;
    }
  }
  return h;
}

// The blocks of the device's soup cover every leaf entry once, in the
// geometries' order; the host's soup is what their threads would write.
static void soup()
{
  for (bool shared : {false, true}) {
    const HostArrays h = meshes(shared);
    std::vector<SoupBlock> blocks;
    expect(build_soup_blocks(h, blocks) == !shared, "meshes that share slots");
    std::vector<int> seen(h.primIdCount.size(), 0);
    std::vector<float> want(h.indices.size() / 3 * 12, 0.0f), got;
    uint32_t last = 0;
    for (const SoupBlock& b : blocks) {
      expect(b.geom >= last, "blocks out of the geometries' order");
      last = b.geom;
      for (uint32_t a = b.firstLeaf; a < b.firstLeaf + kSoupThreads && a < h.startEnd[2 * b.geom + 1]; a++) {
        seen[a]++;
        const uint32_t cnt = (h.primIdCount[a] >> 28) & 7u;
        for (uint32_t k = 0; k < cnt; k++) {
          const uint64_t t = h.geomData[b.geom].offset[0] / 3 + (h.primIdCount[a] & kStartMask) + k;
          float* o = want.data() + 12 * t;
          for (int c = 0; c < 3; c++)
            for (int x = 0; x < 3; x++) {
              const float* P = h.vertPos.data() + 4 * h.geomData[b.geom].offset[1];
              o[4 * c + x] = P[4 * h.indices[3 * t + c] + x] - (c ? P[4 * h.indices[3 * t] + x] : 0.0f);
            }
        }
      }
    }
    for (int n : seen) expect(n == 1, "a leaf entry in no or two blocks");
    if (shared) continue; // (a slot's indices are the last mesh's, out of the first one's vertices)
    build_tri_soup(h, got);
    expect(got == want, "the host's triangle soup");
  }
}

// Node records made on the host: boxes side by side, leaf entries in the leaf
// words of owned pairs, NaN boxes told apart.
static void records()
{
  HostArrays h;
  h.primIdCount = {0x12345u, 0xA0000007u};
  h.allNodePairs.resize(3);
  HostVec<uint32_t> owner(3);
  owner[0] = owner[1] = 0, owner[2] = ~0u;
  std::vector<DevGeom> geoms(1);
  std::memset(geoms.data(), 0, sizeof(DevGeom));
  const uint32_t words[3][2] = {{1u, 0x90000001u}, {kLeafNormal, 0x80000000u}, {0x80000002u, 0x80000000u}};
  for (uint32_t i = 0; i < 3; i++)
    for (uint32_t j = 0; j < 2; j++) {
      lrt_bvh_node& n = j ? h.allNodePairs[i].right : h.allNodePairs[i].left;
      for (uint32_t k = 0; k < 3; k++) n.boxMin[k] = float(i + 10 * j + k), n.boxMax[k] = n.boxMin[k] + 0.5f;
      n.leftOffset = words[i][j];
      n.escapeIndex = 77 + i;
    }
  HostVec<lrt_bvh_node_pair> out;
  expect(build_node_records(h, geoms, owner, out), "records of sound pairs");
  const uint32_t want[3][2] = {{1u, 0xA0000007u}, {kLeafNormal, 0x80012345u}, {0x80000002u, 0x80000000u}};
  for (uint32_t i = 0; i < 3; i++)
    for (uint32_t j = 0; j < 2; j++) {
      float r[8];
      uint32_t w[8];
      std::memcpy(r, j ? &out[i].right : &out[i].left, 32);
      std::memcpy(w, r, 32);
      const float lo = float(i + 10 * j);
      expect(r[0] == lo && r[1] == lo + 0.5f && r[2] == lo + 1 && r[3] == lo + 1.5f && r[4] == lo + 2 && r[5] == lo + 2.5f,
             "slabs side by side");
      expect(w[6] == want[i][j] && w[7] == 77 + i, "words of a record");
    }
  h.allNodePairs[1].left.boxMin[1] = NAN;
  expect(!build_node_records(h, geoms, owner, out), "a box with one NaN is not clean");
  for (int k = 0; k < 3; k++) h.allNodePairs[1].left.boxMin[k] = h.allNodePairs[1].left.boxMax[k] = NAN;
  expect(build_node_records(h, geoms, owner, out), "a box of NaNs is clean");
}

// Kernels by geometry kind; those for all kinds where a leaf entry would read
// as the empty leaf's word.
static void kinds()
{
  HostArrays h;
  h.primIdCount = {1u, 0x7FFFFFFEu};
  const struct {
    std::vector<uint32_t> tags;
    uint32_t kind;
  } want[] = {{{LRT_TAG_TRIANGLE}, kKindNoBricks},
              {{LRT_TAG_SDF_NODE, LRT_TAG_TRIANGLE}, kKindNoBricks},
              {{LRT_TAG_NONE}, kKindNoBricks},
              {{LRT_TAG_SDF_BRICK}, kKindBricks},
              {{LRT_TAG_SDF_BRICK, LRT_TAG_SDF_NODE}, kKindAll}};
  for (uint32_t odd : {0u, 0x7FFFFFFFu, 0xFFFFFFFFu}) {
    h.primIdCount.back() = odd;
    for (const auto& w : want) {
      h.geomTags = w.tags;
      expect(kernel_kind(h) == (odd && w.kind == kKindNoBricks ? kKindAll : w.kind), "kernels of a scene");
    }
  }
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
  soup();
  records();
  kinds();
  rows();
  return failed;
}
