// mesh_upload.cu — the caller's vertex and index arrays copied to the device
// as they lie and packed there.
//
// The 44-byte vertices (without the tangent) become the two 16-byte halves of
// VtxDev and the index triples one uint4 each: two passes over memory, bound
// by HBM and far below the host-to-device copies in front of them.  Packing
// on one host thread took 112 ms for 21M triangles, most of it page faults of
// the packed copies; the whole of scene creation went from 205 to 103 ms.
// The index check of the scene validation runs in the same pass.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "common.h"
#include "mesh_upload.h"

namespace asuna {
namespace {

constexpr int kThreads = 256;
constexpr int kVtxWords = sizeof(asuna_vertex) / 4;
static_assert(kVtxWords == 11 && offsetof(asuna_vertex, uv) == 12 && offsetof(asuna_vertex, normal) == 20,
              "asuna_vertex: position, uv, normal, tangent");
// Consecutive meshes up to this size are gathered into one copy: a copy costs
// about 10 us however short it is, as long as gathering 64 KB takes.
constexpr size_t kGatherBytes = 64 << 10, kGatherBlock = 1 << 20;

// A block loads its vertices as one contiguous run of words and picks its
// fields from shared memory (stride 11: no bank conflicts).
__global__ void __launch_bounds__(kThreads) k_packVertices(const uint32_t* __restrict__ raw, uint32_t n, VtxDev* vtx) {
  __shared__ float w[kThreads * kVtxWords];
  const uint32_t first = blockIdx.x * kThreads;
  const uint32_t cnt = min(uint32_t(kThreads), n - first);
  const uint32_t* src = raw + size_t(first) * kVtxWords;
  for (uint32_t i = threadIdx.x; i < cnt * kVtxWords; i += kThreads) w[i] = __uint_as_float(__ldg(&src[i]));
  __syncthreads();
  if (threadIdx.x >= cnt) return;
  const float* v = w + threadIdx.x * kVtxWords;
  VtxDev o;
  o.pu = make_float4(v[0], v[1], v[2], v[3]);
  o.nv = make_float4(v[5], v[6], v[7], v[4]);
  vtx[first + threadIdx.x] = o;
}

__global__ void __launch_bounds__(kThreads) k_packIndices(const uint32_t* __restrict__ raw, uint32_t n,
                                                          const uint32_t* __restrict__ triBase,
                                                          const uint32_t* __restrict__ vtxBase, int nm, uint4* idx,
                                                          uint32_t* bad) {
  const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  int a = 0, b = nm;
  while (b - a > 1) {
    const int mid = (a + b) / 2;
    if (__ldg(&triBase[mid]) <= i) a = mid; else b = mid;
  }
  const uint32_t nv = __ldg(&vtxBase[a + 1]) - __ldg(&vtxBase[a]);
  const uint32_t* t = raw + 3 * size_t(i);
  uint4 o = make_uint4(__ldg(t), __ldg(t + 1), __ldg(t + 2), 0u);
  if (o.x >= nv || o.y >= nv || o.z >= nv) {
    atomicAdd(bad, 1u);
    o = make_uint4(0u, 0u, 0u, 0u);
  }
  idx[i] = o;
}

// Copies the meshes' arrays one behind the other to `dst`.
template <class Get>
int copyRuns(uint32_t nm, char* dst, cudaStream_t st, Get&& get) {
  std::vector<char> run;
  size_t at = 0;
  auto flush = [&]() -> int {
    if (!run.empty()) {
      // (a pageable source is consumed before the call returns)
      ASUNA_CUDA_TRY(cudaMemcpyAsync(dst + at, run.data(), run.size(), cudaMemcpyHostToDevice, st));
      ASUNA_CUDA_TRY(cudaStreamSynchronize(st));
      at += run.size();
      run.clear();
    }
    return ASUNA_OK;
  };
  for (uint32_t m = 0; m < nm; ++m) {
    const void* src = nullptr;
    size_t bytes = 0;
    get(m, src, bytes);
    if (!bytes) continue;
    int rc = ASUNA_OK;
    if (bytes > kGatherBytes || run.size() + bytes > kGatherBlock)
      if ((rc = flush())) return rc;
    if (bytes > kGatherBytes) {
      ASUNA_CUDA_TRY(cudaMemcpyAsync(dst + at, src, bytes, cudaMemcpyHostToDevice, st));
      at += bytes;
    } else {
      run.insert(run.end(), static_cast<const char*>(src), static_cast<const char*>(src) + bytes);
    }
  }
  return flush();
}

}  // namespace

int uploadMeshes(const asuna_scene_desc* d, const std::vector<uint32_t>& triBase, const std::vector<uint32_t>& vtxBase,
                 VtxDev* vtx, uint4* idx, cudaStream_t st, uint32_t& bad) {
  const uint32_t nm = d->num_meshes, nt = triBase[nm], nv = vtxBase[nm];
  bad = 0;
  if (nt == 0 && nv == 0) return ASUNA_OK;
  auto pad = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t oIdx = pad(size_t(nv) * sizeof(asuna_vertex)), oTri = oIdx + pad(size_t(nt) * 12),
               oVtx = oTri + pad((size_t(nm) + 1) * 4), oBad = oVtx + pad((size_t(nm) + 1) * 4);
  struct Tmp {
    char* p = nullptr;
    ~Tmp() { cudaFree(p); }
  } tmp;
  ASUNA_CUDA_TRY(cudaMalloc(reinterpret_cast<void**>(&tmp.p), oBad + 4));
  ASUNA_CUDA_TRY(cudaMemcpyAsync(tmp.p + oTri, triBase.data(), (size_t(nm) + 1) * 4, cudaMemcpyHostToDevice, st));
  ASUNA_CUDA_TRY(cudaMemcpyAsync(tmp.p + oVtx, vtxBase.data(), (size_t(nm) + 1) * 4, cudaMemcpyHostToDevice, st));
  ASUNA_CUDA_TRY(cudaMemsetAsync(tmp.p + oBad, 0, 4, st));
  int rc;
  if ((rc = copyRuns(nm, tmp.p, st, [&](uint32_t m, const void*& p, size_t& b) {
         p = d->meshes[m].vertices;
         b = size_t(d->meshes[m].num_vertices) * sizeof(asuna_vertex);
       })))
    return rc;
  if (nv)
    k_packVertices<<<(nv + kThreads - 1) / kThreads, kThreads, 0, st>>>(reinterpret_cast<const uint32_t*>(tmp.p), nv,
                                                                      vtx);
  if ((rc = copyRuns(nm, tmp.p + oIdx, st, [&](uint32_t m, const void*& p, size_t& b) {
         p = d->meshes[m].indices;
         b = size_t(d->meshes[m].num_triangles) * 12;
       })))
    return rc;
  if (nt)
    k_packIndices<<<(nt + kThreads - 1) / kThreads, kThreads, 0, st>>>(
        reinterpret_cast<const uint32_t*>(tmp.p + oIdx), nt, reinterpret_cast<const uint32_t*>(tmp.p + oTri),
        reinterpret_cast<const uint32_t*>(tmp.p + oVtx), int(nm), idx, reinterpret_cast<uint32_t*>(tmp.p + oBad));
  ASUNA_CUDA_TRY(cudaGetLastError());
  ASUNA_CUDA_TRY(cudaMemcpyAsync(&bad, tmp.p + oBad, 4, cudaMemcpyDeviceToHost, st));
  ASUNA_CUDA_TRY(cudaStreamSynchronize(st));
  return ASUNA_OK;
}

}  // namespace asuna
