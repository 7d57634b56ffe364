// path.cu — the path kernel: takes the rays of an extend queue and follows each
// one's path to its end, closest hit, shading and occlusion in turn, without
// leaving the kernel.
//
// A wavefront pass costs a handful of launches and the latency of its slowest
// ray however few rays there are; a small wave, or the last rays of a large
// one, spends most of its time on that.  Here a path waits for nothing but
// itself, and a short queue is spread over all warps (down to one path a
// warp), so that nothing is serialised.  The state lives where the wavefront
// keeps it (the path's records, and the queue slot that the lane took), every
// operation is the wavefront's own, and a path's operations come in the same
// order: the results are bit-identical.  Bound by the latency of one path's
// chain of node fetches; the instruction cache and the divergence between
// materials make it slower than the wavefront when the warps are full.
//
// Compiled with -fmad=false like the shading kernels (the traversal spells its
// fused operations).
#include "shade.cuh"
#include "trace.cuh"

namespace asuna {
namespace {

constexpr int kPathThreads = 128;
constexpr int kPathMinBlocks = 4;
constexpr int kPathStack = kSharedStack / 2;
constexpr uint32_t kCoreClasses = 1u << kClsTerminal | 1u << kClsLambertian | 1u << kClsRoughPlastic |
                                  1u << kClsDielectric;
constexpr uint32_t kAllClasses = (1u << kNumShadeClasses) - 1u;

// Traces the queue's ray `idx` of every lane with `active`.
template <bool ANY>
__device__ __forceinline__ void traceLanes(const KParams& P, const Pass& pass, bool active, uint32_t idx, int nodeLanes,
                                           uint2* sh, uint2* loc, bool& ovf) {
  QueueSrc<ANY, true> src;
  src.W = &P.W;
  src.P = &P;
  src.fetchCtr = nullptr;
  src.count = src.warps = 0u;
  src.wave = pass.wave;
  src.rO = ANY ? P.W.shO : P.W.rayO[pass.cur];
  src.rD = ANY ? P.W.shD : P.W.rayD[pass.cur];
  Trav<kPathThreads, kPathStack> tr;
  tr.gMask = tr.tMask = 0u;
  tr.bottom = 0;
  if (active) src.load(P.S, idx, tr);
  uint32_t events = 0, a = 0, b = 0;
  for (;;) {
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (!act) break;
    bool stop = false;
    const bool done = traceRound<ANY, false>(P.S, src, tr, idx, active, act, nodeLanes, false, P.stackLimit, events, sh,
                                             loc, a, b, ovf, stop);
    if (stop) break;
    if (done) {
      active = false;
      events = 0;
      src.finish(idx, tr.found);
    }
  }
}

template <uint32_t MASK>
__device__ __forceinline__ void shadeAny(const KParams& P, const Pass& pass, uint32_t i, ShadeOut& out) {
  switch (classOf(P.S, P.W.hitInst[i])) {
#define ASUNA_SHADE(C)                                \
  case C:                                             \
    if (MASK >> C & 1u) shadeHit<C>(P, pass, i, out); \
    break;
    ASUNA_SHADE(kClsTerminal)
    ASUNA_SHADE(kClsLambertian)
    ASUNA_SHADE(kClsRoughPlastic)
    ASUNA_SHADE(kClsDielectric)
    ASUNA_SHADE(kClsPlastic)
    ASUNA_SHADE(kClsMirror)
    ASUNA_SHADE(kClsConductor)
    ASUNA_SHADE(kClsRoughConductor)
    ASUNA_SHADE(kClsPhong)
    ASUNA_SHADE(kClsPbr)
    ASUNA_SHADE(kClsDisney)
    ASUNA_SHADE(kClsKang18)
#undef ASUNA_SHADE
  }
}

// MASK: the shading classes compiled in (bit k = class k).  See launchPath.
template <uint32_t MASK>
__global__ void __launch_bounds__(kPathThreads, kPathMinBlocks)
    k_path(KParams P, uint32_t lastPass, uint32_t most, cudaGraphConditionalHandle handle) {
  __shared__ uint2 sstack[kPathStack * kPathThreads];
  uint2 lstack[kStackDepth - kPathStack];
  uint2* sh = sstack + threadIdx.x;
  const WaveDev& W = P.W;
  Pass pass = passOf(P);
  if (handle) pass = Pass{pass.wave + 1u, pass.cur ^ 1};
  const uint32_t n = W.cnt->c[kCntExtend0 + pass.cur], from = pass.wave;
  const unsigned lane = threadIdx.x & 31u;
  const bool take = n <= most;  // (the same in every block: the queue is emptied after all have read it)
  if (take && n) {
    const uint32_t warps = gridDim.x * (kPathThreads / 32), warp = blockIdx.x * (kPathThreads / 32) + threadIdx.x / 32u;
    const uint32_t use = min(32u, (n + warps - 1u) / warps);
    const int nodeLanes = int(use) * kNodeLanes / 32;
    uint32_t extends = 0, shadows = 0;
    bool ovf = false;
    for (uint32_t base = warp * use; base < n; base += warps * use) {
      const uint32_t i = base + lane;
      bool alive = lane < use && i < n;
      for (pass.wave = from; pass.wave <= lastPass && __any_sync(0xffffffffu, alive); ++pass.wave) {
        traceLanes<false>(P, pass, alive, i, nodeLanes, sh, lstack, ovf);
        ShadeOut out;
        if (alive) {
          ++extends;
          shadeAny<MASK>(P, pass, i, out);
        }
        __syncwarp();
        if (out.shadow) {
          ++shadows;
          storeShadow(W, i, out);
        }
        if (out.next) storeNext(W, pass.cur, i, out);
        traceLanes<true>(P, pass, out.shadow, i, nodeLanes, sh, lstack, ovf);
        alive = out.next;
      }
    }
    if (ovf) atomicAdd(&W.cnt->stackOverflow, 1ull);
    extends = __reduce_add_sync(0xffffffffu, extends);
    shadows = __reduce_add_sync(0xffffffffu, shadows);
    if (lane == 0 && extends) atomicAdd(&W.cnt->extendRays, static_cast<unsigned long long>(extends));
    if (lane == 0 && shadows) atomicAdd(&W.cnt->shadowRays, static_cast<unsigned long long>(shadows));
  }
  // the last block to leave empties the queue and decides how it goes on
  if (threadIdx.x == 0 && atomicAdd(&W.cnt->c[kCntTicket], 1u) + 1u == gridDim.x) {
    W.cnt->c[kCntTicket] = 0u;
    if (take) W.cnt->c[kCntExtend0 + pass.cur] = 0u;
    if (handle) {
      W.cnt->c[kCntPass] = from;
      cudaGraphSetConditional(handle, n != 0u && !take && from <= lastPass ? 1u : 0u);
    }
  }
}

}  // namespace

void launchPath(const KParams& P, int lastPass, uint32_t most, int grid, cudaGraphConditionalHandle handle,
                cudaStream_t s) {
  if (P.S.classMask & ~kCoreClasses)
    k_path<kAllClasses><<<grid, kPathThreads, 0, s>>>(P, uint32_t(lastPass), most, handle);
  else
    k_path<kCoreClasses><<<grid, kPathThreads, 0, s>>>(P, uint32_t(lastPass), most, handle);
}
// Measured on whole renders (ms, wavefront passes / path kernel).  Scenes of
// Lambertian, rough plastic and dielectric surfaces: 4,096 paths 0.47 / 0.20
// (box), 0.73 / 0.19 (2M triangles); 65,536 paths 0.61 / 0.43, 1.27 / 0.68;
// 131,072 paths 0.67 / 0.77, 1.35 / 1.03.  With the other materials, whose code
// serialises a warp and fills the registers: 4,096 paths 2.0 / 0.58, 16,384
// 2.2 / 1.5, 32,768 2.3 / 2.3.
uint32_t pathMost(uint32_t classMask) { return classMask & ~kCoreClasses ? 24576u : 98304u; }
int pathBlocksPerSm() {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_path<kAllClasses>, kPathThreads, 0);
  return n > 0 ? n : 1;
}

}  // namespace asuna
