/*
 * bvh.h - binned-SAH binary BVH over world-space primitive boxes, emitted in
 * the "children boxes in the parent" layout of DNode (device_scene.h).
 * Replaces the Star-3D acceleration structure (src/ssol_scene.c:410-413).
 */
#ifndef SSOL_B200_BVH_H
#define SSOL_B200_BVH_H

#include "device_scene.h"

#include <cstdint>
#include <vector>

namespace ssolb {

struct PrimBox {
  double lo[3], hi[3];
  uint32_t ref; /* primref_make(kind, index) */
};

struct BvhBuildParams {
  int max_leaf = 4; /* primitives per leaf; a snapshot takes 0 as 1, and may join pairs */
  int bins = 16; /* SAH bins per axis */
  int max_depth = 30; /* the device traversal stack holds 32 entries */
  int threads = 1; /* host threads for the subtrees of large scenes */
  /* Leave the tree to the device builder (lbvh.cu): the snapshot keeps the
   * primitive boxes instead (scenes of at least device_min primitives, 2 or
   * more) */
  bool device = false;
  size_t device_min = 2;
};

/* device_min of the renderers and the adjoint, where the caller leaves the
 * builder open: below, the host builds the tree in less time than the device's
 * one block, its launch and the read-back of the depth take. us a call, host /
 * device: draft of 64 x 64 pixels, 34 primitives 74 / 182, 130 110 / 265, 228
 * 173 / 302, 328 218 / 297, 428 317 / 332, 528 410 / 360, 928 744 / 438;
 * adjoint, 1e3 paths, 130 282 / 443, 328 483 / 549, 428 571 / 578, 528 668 /
 * 615, 928 1084 / 743. */
constexpr size_t DEVICE_BUILD_MIN = 449;

struct BvhResult {
  std::vector<double> lo, hi; /* per node child boxes: node*2+k, 3 each */
  std::vector<int32_t> child, count; /* per node*2+k */
  std::vector<uint32_t> primrefs;
  int depth = 0;
};

void build_bvh(std::vector<PrimBox> prims, const BvhBuildParams& params,
               BvhResult& out);

/* A primitive's box in precision R, rounded outward: lo xyz, hi xyz */
template<class R> void round_box_outward(const PrimBox& b, R out[6]);

/* Convert to device nodes of precision R, rounding boxes outward */
template<class R> std::vector<DNode<R>> bvh_nodes(const BvhResult& b);

/* Turn each node of two single primitives, but the root, into a pair in its
 * parent (PAIR_LEAF), its slot 0 first; the pairs' references are appended */
template<class R> void join_pairs(std::vector<DNode<R>>& nodes, std::vector<uint32_t>& primrefs);

} /* namespace ssolb */

#endif /* SSOL_B200_BVH_H */
