// mesh_upload.h — the meshes of a scene description, packed on the device
// into the layout that the builders and the shading kernels read.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "dev_types.h"

namespace asuna {

// Copies every mesh's vertices and indices to the device and packs them into
// vtx (vtxBase.back() records) and idx (triBase.back()), both allocated by
// the caller.  `bad` counts triangles with an index past their mesh's
// vertices (their packed indices are 0).  Waits for the stream.
int uploadMeshes(const asuna_scene_desc* d, const std::vector<uint32_t>& triBase, const std::vector<uint32_t>& vtxBase,
                 VtxDev* vtx, uint4* idx, cudaStream_t st, uint32_t& bad);

}  // namespace asuna
