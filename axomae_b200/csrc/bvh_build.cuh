/* On-device binned-SAH BVH build (declarations).  See bvh_build.cu. */
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace nb {

struct BvhBuildParams {
  int max_leaf;     /* preferred maximum leaf size (SAH may stop earlier); hard cap 16 */
  int hard_leaf;    /* nodes with more primitives are always split (median when SAH finds no plane) */
  int bins;         /* SAH bins per axis (<= 32) */
  float cost_trav;  /* SAH cost of one inner-node visit relative to one triangle test */
  uint32_t small_task; /* nodes of at most this many primitives (<= 256) are built whole by one CTA (0: default) */
};

struct BvhBuildResult {
  uint32_t n_nodes;
  uint32_t n_leaves;
  int max_depth;
  double ms;
};

/* Builds a binary BVH over n primitive boxes (lo/hi: world-space, float4 with w unused; no coordinate -0, which
 * the build's float minima by integer atomics would take for the least value of all, cutting boxes off at zero:
 * making it +0 in every atomic took 5 % of a 3 M triangle build, in the boxes nothing).
 * nodes: room for n + 1 nodes (4 float4 each, layout in device_scene.cuh).
 * order: receives, for every leaf slot, the index (into lo/hi) of the primitive stored there.
 * Returns a CUDA error code (cudaSuccess on success). */
cudaError_t build_bvh(const float4 *lo, const float4 *hi, uint32_t n, const BvhBuildParams &p, float4 *nodes,
                      uint32_t *order, cudaStream_t stream, BvhBuildResult *res);

}  // namespace nb
