// bvh_wide.h — the traversal's 8-wide BVH, made on the GPU from the builders'
// binary trees (bvh_wide.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "dev_types.h"

namespace asuna {

struct WideBvh {
  WideNode* nodes = nullptr;  // device; the caller owns it, also on failure
  TriDev* tris = nullptr;     // device; leaf triangles in wide-leaf order (caller owned, also on failure)
  uint32_t* instIds = nullptr;  // device; instances in wide-leaf order of the top level (in the block of `tris`)
  size_t bytes = 0;             // of both blocks
  uint32_t nodeCount = 0;
  uint32_t levels = 0;        // of the deepest tree
  std::vector<uint32_t> rootLeaves;  // InstDev::rootLeaves of every root
};

// Collapses binary trees into 8-wide nodes on `stream` and waits for it.
// `nodes`: every binary node of the scene on the device; `roots`: the root
// node of each bottom-level tree, then the top level's, whose leaves name
// instances.  Root k of the list becomes wide node k.  `maxDepth`: no leaf
// lies deeper below a root.
int buildWide(const BvhNode* nodes, uint32_t nodeCount, const TriDev* tris, uint32_t triCount, uint32_t instCount,
              const std::vector<int32_t>& roots, uint32_t maxDepth, cudaStream_t stream, WideBvh& out);

}  // namespace asuna
