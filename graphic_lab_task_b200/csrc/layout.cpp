// layout.cpp — builds the derived device layouts of device_layout.h on the
// host (compiled with -ffp-contract=off so every float is computed exactly
// as the reference computes it on the fly).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <limits>
#include <utility>

#include "layout.h"

namespace lrt {

void build_geoms(const HostArrays& h, std::vector<DevGeom>& out)
{
  out.resize(h.geomData.size());
  for (size_t g = 0; g < h.geomData.size(); g++) {
    const lrt_geom_data& gd = h.geomData[g];
    DevGeom d;
    std::memset(&d, 0, sizeof(d));
    d.tag = h.geomTags[g];
    d.type = gd.type;
    d.bvhOffset = gd.bvhOffset;
    d.aabbBase = h.startEnd[2 * g];
    if (d.tag == LRT_TAG_TRIANGLE) {
      d.triBase = gd.offset[0] / 3;
      d.firstVert = gd.offset[1];
    } else {
      d.sdfId = gd.offset[0];
      if (d.tag == LRT_TAG_SDF_BRICK) d.sdfRoot = h.sdfSBSRoots[d.sdfId];
      else if (gd.type == LRT_TYPE_SDF_FRAME_OCTREE) d.sdfRoot = h.sdfFrameOctreeRoots[d.sdfId];
      else if (gd.type == LRT_TYPE_SDF_SVS) d.sdfRoot = h.sdfSVSRoots[d.sdfId];
    }
    out[g] = d;
  }
}

uint64_t triangle_slots(const HostArrays& h, size_t g)
{
  uint64_t ntri = 0;
  for (uint32_t a = h.startEnd[2 * g]; a < h.startEnd[2 * g + 1]; a++) {
    const uint32_t pk = h.primIdCount[a], cnt = (pk & kSizeMask) >> 28;
    if (cnt) ntri = std::max<uint64_t>(ntri, uint64_t(pk & kStartMask) + cnt);
  }
  return ntri;
}

// {A, B-A, C-A} per reordered triangle slot; IntersectAllTrianglesInLeaf
// computes exactly these differences (BVH2Common.cpp:1585-1589).
void build_tri_soup(const HostArrays& h, std::vector<float>& soup)
{
  soup.assign(h.indices.size() / 3 * 12, 0.0f);
  for (size_t g = 0; g < h.geomData.size(); g++) {
    if (h.geomTags[g] != LRT_TAG_TRIANGLE) continue;
    const uint64_t base = h.geomData[g].offset[0] / 3, firstVert = h.geomData[g].offset[1];
    for (uint32_t a = h.startEnd[2 * g]; a < h.startEnd[2 * g + 1]; a++) {
      const uint32_t pk = h.primIdCount[a];
      const uint64_t first = base + (pk & kStartMask), end = first + ((pk & kSizeMask) >> 28);
      for (uint64_t t = first; t < end; t++) {
        const float* P[3];
        for (int c = 0; c < 3; c++) P[c] = h.vertPos.data() + 4 * (firstVert + h.indices[3 * t + c]);
        float* o = soup.data() + 12 * t;
        for (int k = 0; k < 3; k++) {
          o[k] = P[0][k];
          o[4 + k] = P[1][k] - P[0][k];
          o[8 + k] = P[2][k] - P[0][k];
        }
      }
    }
  }
}

bool build_soup_blocks(const HostArrays& h, std::vector<SoupBlock>& blocks)
{
  blocks.clear();
  std::vector<std::pair<uint64_t, uint64_t>> ranges; // slots
  size_t meshes = 0;
  for (uint32_t tag : h.geomTags) meshes += tag == LRT_TAG_TRIANGLE;
  for (size_t g = 0; g < h.geomData.size(); g++) {
    if (h.geomTags[g] != LRT_TAG_TRIANGLE) continue;
    for (uint64_t a = h.startEnd[2 * g]; a < h.startEnd[2 * g + 1]; a += kSoupThreads)
      blocks.push_back({uint32_t(g), uint32_t(a)});
    const uint64_t base = h.geomData[g].offset[0] / 3, slots = meshes > 1 ? triangle_slots(h, g) : 0;
    if (slots) ranges.push_back({base, base + slots});
  }
  std::sort(ranges.begin(), ranges.end());
  for (size_t i = 1; i < ranges.size(); i++)
    if (ranges[i].first < ranges[i - 1].second) return false;
  return true;
}

uint32_t kernel_kind(const HostArrays& h)
{
  uint32_t kinds = 0;
  for (uint32_t t : h.geomTags)
    kinds |= t == LRT_TAG_TRIANGLE ? kKindTriangles : t == LRT_TAG_SDF_NODE ? kKindNodes
           : t == LRT_TAG_SDF_BRICK ? kKindBricks : 0u;
  if (kinds == kKindBricks) return kKindBricks;
  if (kinds & kKindBricks) return kKindAll;
  // (of 7 primitives from 2^28 - 1 on, or of a geometry without leaf code)
  bool asEmpty = false;
  for (uint32_t entry : h.primIdCount) asEmpty |= (entry | kLeafBit) == kLeafNormal;
  return asEmpty ? kKindAll : kKindNoBricks;
}

bool build_node_records(const HostArrays& h, const std::vector<DevGeom>& geoms, const HostVec<uint32_t>& owner,
                        HostVec<lrt_bvh_node_pair>& records)
{
  records.resize(h.allNodePairs.size());
  bool clean = true;
  for (size_t i = 0; i < records.size(); i++) {
    const lrt_bvh_node* in[2] = {&h.allNodePairs[i].left, &h.allNodePairs[i].right};
    lrt_bvh_node* out[2] = {&records[i].left, &records[i].right};
    for (int j = 0; j < 2; j++) {
      const lrt_bvh_node n = *in[j];
      uint32_t word = n.leftOffset;
      if ((word & kLeafBit) && word != kLeafNormal && owner[i] != ~0u)
        word = kLeafBit | (h.primIdCount[geoms[owner[i]].aabbBase + (word & kStartMask)] & ~kLeafBit);
      int nans = 0;
      for (int k = 0; k < 3; k++) nans += std::isnan(n.boxMin[k]) + std::isnan(n.boxMax[k]);
      clean = clean && (nans == 0 || nans == 6);
      const float box[6] = {n.boxMin[0], n.boxMax[0], n.boxMin[1], n.boxMax[1], n.boxMin[2], n.boxMax[2]};
      char* o = reinterpret_cast<char*>(out[j]);
      std::memcpy(o, box, sizeof(box));
      std::memcpy(o + 24, &word, 4);
      std::memcpy(o + 28, &n.escapeIndex, 4);
    }
  }
  return clean;
}

// Surface-voxel masks of every brick from its dense corner grid (see
// device_layout.h): vmin is reduced exactly as load_distance_values does
// (BVH2Common.cpp:861-866), so the bit equals the reference's `vmin <= 0`.
void build_sbs_masks(const HostArrays& h, std::vector<DevSbs>& sbs, const std::vector<float>& dense,
                     std::vector<uint32_t>& mask)
{
  uint64_t total = 0;
  for (size_t i = 0; i < sbs.size(); i++) {
    const uint32_t bs = sbs[i].brick_size;
    sbs[i].maskStride = 1 + (bs * bs * bs + 31) / 32;
    sbs[i].maskBase = total;
    total += uint64_t(sbs[i].nodeCount) * sbs[i].maskStride;
  }
  mask.assign(total, 0u);
  for (size_t i = 0; i < sbs.size(); i++) {
    const DevSbs& d = sbs[i];
    const uint32_t bs = d.brick_size, V1 = bs + 1;
#pragma omp parallel for schedule(static)
    for (int64_t k = 0; k < int64_t(d.nodeCount); k++) {
      const float* g = dense.data() + d.denseBase + uint64_t(k) * d.denseStride;
      uint32_t* m = mask.data() + d.maskBase + uint64_t(k) * d.maskStride;
      for (uint32_t x = 0; x < bs; x++)
        for (uint32_t y = 0; y < bs; y++)
          for (uint32_t z = 0; z < bs; z++) {
            float vmin = 1e6f;
            for (int c = 0; c < 8; c++) {
              const float v = g[((x + ((c & 4) >> 2)) * V1 + (y + ((c & 2) >> 1))) * V1 + (z + (c & 1))];
              vmin = (v < vmin) ? v : vmin;
            }
            if (vmin <= 0.0f) {
              const uint32_t vid = (x * bs + y) * bs + z;
              m[1 + vid / 32] |= 1u << (vid % 32);
              m[0] = 1;
            }
          }
    }
  }
  (void)h;
}

// Device copy of the BLAS node pairs in which every child subtree of an SBS
// BLAS that holds no brick able to start a sphere trace gets a NaN box.  A
// NaN box fails the child test of BVH2TraverseF32 (tmin <= tmax is false) for
// every ray, so such a subtree is never entered.  This cannot change a
// result: the pruned leaves never touch the hit, and the depth-first
// near-first order of the remaining leaves is unchanged — at a node whose
// other child is pruned the reference would visit that child (before or
// after) without effect.  Returns the number of pruned children.
uint64_t prune_sbs_pairs(const HostArrays& h, const std::vector<DevGeom>& geoms, const std::vector<DevSbs>& sbs,
                         const std::vector<uint32_t>& mask, HostVec<lrt_bvh_node_pair>& pairs)
{
  pairs = h.allNodePairs;
  const float qnan = std::numeric_limits<float>::quiet_NaN();
  uint64_t pruned = 0;
  for (size_t g = 0; g < geoms.size(); g++) {
    if (geoms[g].tag != LRT_TAG_SDF_BRICK) continue;
    const DevSbs& sb = sbs[geoms[g].sdfId];
    const uint32_t base = geoms[g].bvhOffset, a0 = geoms[g].aabbBase;
    // returns true if the subtree under `lo` (a child word) can produce a hit
    std::function<bool(uint32_t)> live = [&](uint32_t lo) -> bool {
      if (lo & kLeafBit) {
        if (lo == kLeafNormal) return false;
        const uint32_t primId = h.primIdCount[a0 + (lo & kStartMask)] & kStartMask;
        if (primId >= sb.nodeCount) return false;
        return mask[sb.maskBase + uint64_t(primId) * sb.maskStride] != 0;
      }
      lrt_bvh_node_pair& p = pairs[base + lo];
      const bool l = live(p.left.leftOffset), r = live(p.right.leftOffset);
      for (int j = 0; j < 2; j++) {
        lrt_bvh_node& n = j ? p.right : p.left;
        if (!(j ? r : l)) {
          for (int k = 0; k < 3; k++) n.boxMin[k] = n.boxMax[k] = qnan;
          pruned++;
        }
      }
      return l || r;
    };
    live(0); // the root pair
  }
  return pruned;
}

void build_prune_tree(const HostArrays& h, const std::vector<DevGeom>& geoms, const std::vector<DevSbs>& sbs,
                      std::vector<PruneLeaf>& leaves, std::vector<uint32_t>& parent)
{
  leaves.clear();
  parent.clear();
  if (h.sdfSBSNodes.empty() || h.allNodePairs.size() >= (1u << 30)) return;
  for (const DevSbs& sb : sbs)
    if (sb.maskBase + uint64_t(sb.nodeCount) * sb.maskStride >= 0xFFFFFFFFull) return;
  parent.assign(h.allNodePairs.size(), kPruneOther);
  std::vector<uint32_t> todo;
  for (size_t g = 0; g < geoms.size(); g++) {
    if (geoms[g].tag != LRT_TAG_SDF_BRICK) continue;
    const DevSbs& sb = sbs[geoms[g].sdfId];
    const uint32_t base = geoms[g].bvhOffset, a0 = geoms[g].aabbBase;
    parent[base] = kPruneRoot;
    todo.assign(1, base);
    while (!todo.empty()) {
      const uint32_t p = todo.back();
      todo.pop_back();
      for (uint32_t j = 0; j < 2; j++) {
        const uint32_t lo = (j ? h.allNodePairs[p].right : h.allNodePairs[p].left).leftOffset;
        const uint32_t slot = (p << 1) | j;
        if (!(lo & kLeafBit)) {
          parent[base + lo] = slot;
          todo.push_back(base + lo);
        } else if (lo != kLeafNormal) {
          const uint32_t primId = h.primIdCount[a0 + (lo & kStartMask)] & kStartMask;
          if (primId < sb.nodeCount)
            leaves.push_back({slot, uint32_t(sb.maskBase + uint64_t(primId) * sb.maskStride)});
        }
      }
    }
  }
}

// Dense (brick_size+1)^3 corner grids per SBS node; values as
// load_distance_values returns them (BVH2Common.cpp:846-882).
void build_sbs_dense(const HostArrays& h, std::vector<DevSbs>& sbs, std::vector<float>& dense)
{
  const size_t nsdf = h.sdfSBSRoots.size();
  sbs.assign(nsdf, DevSbs{});
  uint64_t total = 0;
  std::vector<uint64_t> counts(nsdf);
  for (size_t i = 0; i < nsdf; i++) {
    const uint32_t root = h.sdfSBSRoots[i];
    uint64_t next = h.sdfSBSNodes.size();
    for (size_t j = 0; j < nsdf; j++)
      if (h.sdfSBSRoots[j] > root) next = std::min<uint64_t>(next, h.sdfSBSRoots[j]);
    counts[i] = next > root ? next - root : 0;
    const lrt_sdf_sbs_header& hd = h.sdfSBSHeaders[i];
    const uint32_t V1 = hd.brick_size + 1;
    const uint32_t v = hd.brick_size + 2 * hd.brick_pad + 1;
    DevSbs& d = sbs[i];
    d.nodeCount = uint32_t(counts[i]);
    d.denseBase = total;
    d.denseStride = V1 * V1 * V1;
    d.brick_size = hd.brick_size;
    d.v3 = v * v * v;
    d.pad = hd.brick_pad;
    d.vsize = v;
    const uint32_t layout = hd.aux_data & LRT_SBS_LAYOUT_MASK;
    d.colorLayout = (layout == LRT_SBS_LAYOUT_ID32F_IRGB32F || layout == LRT_SBS_LAYOUT_ID32F_IRGB32F_IN) ? 1u : 0u;
    total += counts[i] * d.denseStride;
  }
  dense.assign(total, 0.0f);
  for (size_t i = 0; i < nsdf; i++) {
    const lrt_sdf_sbs_header& hd = h.sdfSBSHeaders[i];
    const DevSbs& d = sbs[i];
    const uint32_t bs = hd.brick_size, pad = hd.brick_pad, V1 = bs + 1;
    const uint32_t v = bs + 2 * pad + 1;
    const bool indexed = d.colorLayout != 0;
    const uint32_t vals_per_int = indexed ? 1 : 4 / hd.bytes_per_value;
    const uint32_t bits = indexed ? 32 : 8 * hd.bytes_per_value;
    const uint32_t max_val = (!indexed && hd.bytes_per_value != 4) ? ((1u << bits) - 1) : 0xFFFFFFFFu;
    const uint32_t root = h.sdfSBSRoots[i];
#pragma omp parallel for schedule(static)
    for (int64_t k = 0; k < int64_t(counts[i]); k++) {
      const lrt_sdf_sbs_node& nd = h.sdfSBSNodes[root + k];
      const uint32_t off = nd.data_offset;
      float* o = dense.data() + d.denseBase + uint64_t(k) * d.denseStride;
      const float sz = float(nd.pos_z_lod_size & 0x0000FFFF);
      const float sz_inv = 2.0f / sz;
      const float d_max = 1.73205081f * sz_inv;
      const float mult = 2 * d_max / max_val;
      for (uint32_t x = 0; x < V1; x++)
        for (uint32_t y = 0; y < V1; y++)
          for (uint32_t z = 0; z < V1; z++) {
            const uint32_t vId = (x + pad) * v * v + (y + pad) * v + (z + pad);
            float val;
            if (indexed) {
              val = h.sdfSBSDataF[h.sdfSBSData[off + vId]];
            } else {
              const uint32_t word = h.sdfSBSData[off + vId / vals_per_int];
              const uint32_t sh = bits * (vId % vals_per_int);
              const uint32_t field = (sh >= 32 ? 0u : (word >> sh)) & max_val;
              val = -d_max + mult * field;
            }
            o[(x * V1 + y) * V1 + z] = val;
          }
    }
  }
}

} // namespace lrt
