// trace.cu — the traversal kernels of a wavefront pass (extend: closest hit;
// connect: occlusion) and of ray queries, over trace.cuh.
#include "trace.cuh"

namespace asuna {
namespace {

// TB: threads per block; MINB: resident blocks per SM the variant is
// compiled for (its register cap); SHS: 8-byte stack entries in shared memory
template <bool ANY, bool COUNT, int TB, int MINB, int SHS>
__global__ void __launch_bounds__(TB, MINB) k_trace(KParams P) {
  __shared__ uint2 sstack[SHS * TB];
  uint2 lstack[kStackDepth - SHS];
  uint2* sh = sstack + threadIdx.x;
  const WaveDev& W = P.W;
  const Pass pass = passOf(P);
  const int cur = pass.cur;
  uint32_t* countPtr = ANY ? &W.cnt->c[kCntShadow] : &W.cnt->c[kCntExtend0 + cur];
  QueueSrc<ANY> src;
  src.W = &P.W;
  src.P = &P;
  src.fetchCtr = ANY ? &W.cnt->c[kCntFetchShadow] : &W.cnt->c[kCntFetchExtend];
  src.count = *countPtr;
  src.warps = gridDim.x * (TB / 32);
  src.wave = pass.wave;
  src.rO = ANY ? W.shO : W.rayO[cur];
  src.rD = ANY ? W.shD : W.rayD[cur];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (ANY) {
      W.cnt->shadowRays += src.count;
      W.cnt->c[kCntFetchExtend] = 0;  // the next extend pass fetches from 0
    } else {
      W.cnt->extendRays += src.count;
      W.cnt->c[kCntExtend0 + (cur ^ 1)] = 0;  // shade appends into the other queue
      W.cnt->c[kCntShadow] = 0;
      for (int k = 0; k < kNumShadeClasses; ++k) W.cnt->c[kCntCls0 + k] = 0;  // classify appends
    }
  }
  uint32_t nNodes = 0, nTris = 0;
  bool ovf = false;
  // (the instrumented variant walks without speculation, so its node counts
  // are those of the ordered traversal)
  // (P.stackLimit is in [1, kStackDepth]: the host clamps it)
  traceWarp<ANY, COUNT, TB, SHS>(P.S, src, sh, lstack, P.refillLanes, !COUNT && P.speculate != 0, P.stackLimit, nNodes,
                                 nTris, ovf);
  if (ovf) atomicAdd(&W.cnt->stackOverflow, 1ull);
  if (COUNT) {
    const unsigned lane = threadIdx.x & 31u;
    unsigned long long a = nNodes, b = nTris;
    for (int off = 16; off; off >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, off);
      b += __shfl_down_sync(0xffffffffu, b, off);
    }
    if (lane == 0) {
      atomicAdd(ANY ? &W.cnt->shNodes : &W.cnt->nodes, a);
      atomicAdd(ANY ? &W.cnt->shTris : &W.cnt->tris, b);
    }
  }
}

// Rays given as arrays (asuna_scene_trace): each warp walks its own
// contiguous slice of the rays with the same warp loop.
struct ArraySrc {
  const float4 *o, *d;
  float4* hit;
  uint32_t* inst;
  uint32_t cursor, count;
  int anyHit;
  static constexpr uint32_t warps = 1u;  // each warp has its own slice
  __device__ __forceinline__ uint32_t fetch(uint32_t) { return cursor; }
  __device__ __forceinline__ bool stopAtHit() const { return false; }
  // every lane of the warp advances its copy of the cursor alike
  __device__ __forceinline__ void commit(uint32_t base, uint32_t n) { cursor = base + n; }
  template <class T>
  __device__ __forceinline__ void load(const SceneDev& S, uint32_t r, T& tr) {
    const float4 o4 = o[r], d4 = d[r];
    tr.init(S, make_float3(o4.x, o4.y, o4.z), make_float3(d4.x, d4.y, d4.z), d4.w);
  }
  __device__ __forceinline__ float tmin(uint32_t r) const { return o[r].w; }
  __device__ __forceinline__ void world(uint32_t r, float3& wo, float3& wd) const {
    const float4 o4 = o[r], d4 = d[r];
    wo = make_float3(o4.x, o4.y, o4.z);
    wd = make_float3(d4.x, d4.y, d4.z);
  }
  __device__ __forceinline__ void store(uint32_t i, float t, float u, float v, uint32_t prim, uint32_t in) {
    hit[i] = make_float4(t, u, v, __uint_as_float(prim));
    inst[i] = in;
  }
  __device__ __forceinline__ bool later(uint32_t i, uint32_t in, uint32_t prim) const {
    return in < inst[i] || (in == inst[i] && prim < __float_as_uint(hit[i].w));
  }
  __device__ __forceinline__ void finish(uint32_t i, bool found) {
    if (found) {
      if (anyHit) {
        hit[i] = make_float4(1.0f, 0.0f, 0.0f, 0.0f);
        inst[i] = 0u;
      }
    } else {
      hit[i] = make_float4(-1.0f, 0.0f, 0.0f, 0.0f);
      inst[i] = 0xffffffffu;
    }
  }
};

__global__ void __launch_bounds__(kTraceThreads) k_query(SceneDev S, const float4* o, const float4* d, uint32_t n,
                                                         int anyHit, float4* hit, uint32_t* inst, uint32_t* cut) {
  constexpr int SHS = kSharedStack / 2;
  __shared__ uint2 sstack[SHS * kTraceThreads];
  uint2 lstack[kStackDepth - SHS];
  uint2* sh = sstack + threadIdx.x;
  const uint32_t warps = gridDim.x * (blockDim.x / 32u);
  const uint32_t w = blockIdx.x * (blockDim.x / 32u) + threadIdx.x / 32u;
  const uint32_t per = (n + warps - 1) / warps;
  const uint32_t lo = min(n, w * per), hi = min(n, lo + per);
  // indices are relative to the slice
  ArraySrc src{o + lo, d + lo, hit + lo, inst + lo, 0u, hi - lo, anyHit};
  uint32_t a = 0, b = 0;
  bool ovf = false;
  if (anyHit)
    traceWarp<true, false, kTraceThreads, SHS>(S, src, sh, lstack, kRefillLanes, true, kStackDepth, a, b, ovf);
  else
    traceWarp<false, false, kTraceThreads, SHS>(S, src, sh, lstack, kRefillLanes, true, kStackDepth, a, b, ovf);
  if (ovf) atomicAdd(cut, 1u);
}

}  // namespace

namespace {
// Kernel variants: threads per block (64, 128, 256) x resident warps per SM
// (32, 40, 48: the occupancy class 8, 10, 12 of 128-thread blocks) x stack
// bytes in shared memory (16, 24, 32 words, two per entry).
template <bool ANY, int TB, int OCC>
void launchOcc(const KParams& P, int grid, cudaStream_t s) {
  constexpr int MINB = OCC * 128 / TB;
  if (P.sharedStack >= 32)
    k_trace<ANY, false, TB, MINB, 16><<<grid, TB, 0, s>>>(P);
  else if (P.sharedStack > 0 && P.sharedStack <= 16)
    k_trace<ANY, false, TB, MINB, 8><<<grid, TB, 0, s>>>(P);
  else
    k_trace<ANY, false, TB, MINB, 12><<<grid, TB, 0, s>>>(P);
}
template <bool ANY, int TB>
void launchTb(const KParams& P, int grid, cudaStream_t s) {
  if (P.occupancy >= 12)
    launchOcc<ANY, TB, 12>(P, grid, s);
  else if (P.occupancy >= 10)
    launchOcc<ANY, TB, 10>(P, grid, s);
  else
    launchOcc<ANY, TB, kTraceMinBlocks>(P, grid, s);
}
template <bool ANY>
void launchTrace(const KParams& P, int grid, cudaStream_t s) {
  if (P.counters)
    k_trace<ANY, true, kTraceThreads, kTraceMinBlocks, kSharedStack / 2><<<grid, kTraceThreads, 0, s>>>(P);
  else if (P.blockThreads == 64)
    launchTb<ANY, 64>(P, grid, s);
  else if (P.blockThreads == 256)
    launchTb<ANY, 256>(P, grid, s);
  else
    launchTb<ANY, 128>(P, grid, s);
}
template <int TB, int OCC, int SHS>
int blocksOf() {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_trace<false, false, TB, OCC * 128 / TB, SHS>, TB, 0);
  return n;
}
template <int TB, int OCC>
int blocksOcc(int sharedStack) {
  return sharedStack >= 32 ? blocksOf<TB, OCC, 16>()
         : (sharedStack > 0 && sharedStack <= 16) ? blocksOf<TB, OCC, 8>() : blocksOf<TB, OCC, 12>();
}
template <int TB>
int blocksTb(int occupancy, int sharedStack) {
  return occupancy >= 12 ? blocksOcc<TB, 12>(sharedStack)
         : occupancy >= 10 ? blocksOcc<TB, 10>(sharedStack) : blocksOcc<TB, kTraceMinBlocks>(sharedStack);
}
}  // namespace

void launchExtend(const KParams& P, int grid, cudaStream_t s) { launchTrace<false>(P, grid, s); }
void launchConnect(const KParams& P, int grid, cudaStream_t s) { launchTrace<true>(P, grid, s); }
int traceBlocksPerSm(int occupancy, int blockThreads, int sharedStack) {
  const int n = blockThreads == 64    ? blocksTb<64>(occupancy, sharedStack)
                : blockThreads == 256 ? blocksTb<256>(occupancy, sharedStack)
                                      : blocksTb<128>(occupancy, sharedStack);
  return n > 0 ? n : 1;
}
void launchTraceQuery(const SceneDev& S, const float4* o, const float4* d, uint32_t n, int anyHit, float4* hit,
                      uint32_t* inst, uint32_t* cut, cudaStream_t s) {
  int grid = int((n + kTraceThreads - 1) / kTraceThreads);
  if (grid > 4096) grid = 4096;
  if (grid < 1) grid = 1;
  k_query<<<grid, kTraceThreads, 0, s>>>(S, o, d, n, anyHit, hit, inst, cut);
}

}  // namespace asuna
