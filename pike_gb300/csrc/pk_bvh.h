// pk_bvh.h -- GPU builder of the reference BVH (bvh.js sweep SAH + trace_pass.js packing).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <string>

#include "pk_util.h"

namespace pk {

struct BvhOut {
  DevBuf<int32_t> nodes5;   // BFS nodes, 5 words each (BVHNodeStruct)
  DevBuf<int4> tri4_leaf;   // leaf-ordered {i0, i1, i2, matId}
  DevBuf<float4> verts4;    // normalised positions (xyz, 0)
  DevBuf<double> node_box;  // exact double bounds per BFS node {min xyz, max xyz} (raycaster.js uses them)
  uint32_t n_nodes = 0, n_leaf_tris = 0, depth = 0, largest_leaf = 0;
  double norm[4] = {0, 0, 0, 0};  // centre xyz, scale = 2 / longest
};

// Rebuild of bvh.js:12-223 with identical topology and primitive order: every
// sweep cost of #computeSplit in binary32 with a bound on its error, the costs
// within the bound of the smallest again in double, the first minimum in (axis,
// index) order, `cost > n` a leaf, a stable partition of the other two axis
// orders.  Nodes of more than 512 triangles level by level, the rest a subtree per
// block; nodes come out in BFS order, which is serializeTree's.  Returns non-zero
// with a reason on failure; throws CudaError when a look-back timed out.
int build_bvh_sweep(const Scratch& scratch, const double* pos3, uint32_t n_verts, const int4* tri4, uint32_t n_tris,
                    BvhOut& out, std::string& why);

// Binned SAH (16 bins per axis, leaves of at most 8 triangles): a different,
// faster-to-build topology than bvh.js; same output layout.
int build_bvh_binned(const Scratch& scratch, const double* pos3, uint32_t n_verts, const int4* tri4, uint32_t n_tris,
                     BvhOut& out, std::string& why);

}  // namespace pk
