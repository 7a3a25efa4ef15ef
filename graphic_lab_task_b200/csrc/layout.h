// layout.h — host builders of the derived device layouts (layout.cpp).
#pragma once
#include <vector>

#include "device_layout.h"
#include "scene.h"

namespace lrt {

void build_geoms(const HostArrays& h, std::vector<DevGeom>& out);
// Records of triangle geometry g in the triangle soup (one past the largest
// leaf range of its leaf table).
uint64_t triangle_slots(const HostArrays& h, size_t g);
// The triangle soup, made on the host: the slots that a leaf covers (geometry
// by geometry), zeros elsewhere.
void build_tri_soup(const HostArrays& h, std::vector<float>& soup);
// The blocks that make it on the device, geometry by geometry.  False if two
// geometries share slots: their blocks must then run in that order.
bool build_soup_blocks(const HostArrays& h, std::vector<SoupBlock>& blocks);
// The kind of kernels that trace the scene: kKindBricks, kKindNoBricks or
// kKindAll.  The last serves all scenes, and also one without bricks whose leaf
// table holds an entry that would read as the empty leaf's word in a record.
uint32_t kernel_kind(const HostArrays& h);
// The node records of a scene of kKindNoBricks (owner: the geometry of each
// pair), made on the host.  False if a box has some but not six NaN coordinates.
bool build_node_records(const HostArrays& h, const std::vector<DevGeom>& geoms, const HostVec<uint32_t>& owner,
                        HostVec<lrt_bvh_node_pair>& records);
void build_sbs_dense(const HostArrays& h, std::vector<DevSbs>& sbs, std::vector<float>& dense);
void build_sbs_masks(const HostArrays& h, std::vector<DevSbs>& sbs, const std::vector<float>& dense,
                     std::vector<uint32_t>& mask);
uint64_t prune_sbs_pairs(const HostArrays& h, const std::vector<DevGeom>& geoms, const std::vector<DevSbs>& sbs,
                         const std::vector<uint32_t>& mask, HostVec<lrt_bvh_node_pair>& pairs);
// The tree of the SBS node pairs as k_prune_mark climbs it; empty without SBS
// geometry, or if its indices do not fit 32 bits.
void build_prune_tree(const HostArrays& h, const std::vector<DevGeom>& geoms, const std::vector<DevSbs>& sbs,
                      std::vector<PruneLeaf>& leaves, std::vector<uint32_t>& parent);

} // namespace lrt
