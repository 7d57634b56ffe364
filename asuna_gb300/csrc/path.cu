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

// The ray that a lane is tracing: its path's closest hit or occlusion ray, in
// the queue slot that the lane took.  The running kernel writes both.
struct PathSrc {
  QueueSrc<false, true> hit;
  QueueSrc<true, true> shadow;
  bool any;
  __device__ __forceinline__ bool stopAtHit() const { return any; }
  __device__ __forceinline__ float tmin(uint32_t i) const { return any ? shadow.tmin(i) : hit.tmin(i); }
  template <class T>
  __device__ __forceinline__ void load(const SceneDev& S, uint32_t i, T& tr) {
    if (any)
      shadow.load(S, i, tr);
    else
      hit.load(S, i, tr);
  }
  __device__ __forceinline__ void world(uint32_t i, float3& o, float3& d) const {
    if (any)
      shadow.world(i, o, d);
    else
      hit.world(i, o, d);
  }
  __device__ __forceinline__ void store(uint32_t i, float t, float u, float v, uint32_t prim, uint32_t inst) {
    hit.store(i, t, u, v, prim, inst);
  }
  __device__ __forceinline__ bool later(uint32_t i, uint32_t inst, uint32_t prim) const {
    return hit.later(i, inst, prim);
  }
  __device__ __forceinline__ void finish(uint32_t i, bool found) {
    if (any)
      shadow.finish(i, found);
    else
      hit.finish(i, found);
  }
};

// What a lane's path is doing.  After shading, each lane traces its occlusion
// ray and then its next closest hit without waiting for the others in between
// (separate rounds for the two kinds: 32x32 box of 2 frames 172 -> 143 us, sky
// 641x427 0.91 -> 0.83 ms, 1280x720 frame of 2.6M triangles 2.14 -> 1.94 ms).
// Lanes that have their hit do wait for the last one: shading part of a warp
// at a time costs more than it hides (once seven of eight wait: 0.90 and 2.06
// ms, half of them: 1.04 and 2.33 ms).
enum PathState : int { kPathNone, kPathHit, kPathShadow, kPathShade };

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
  // The last block to leave rewrites the pass and the count.  Every thread has
  // read both before this barrier, and its block's ticket is taken behind it, so
  // the tickets (with the fences around them) order all reads before the writes.
  __syncthreads();
  const unsigned lane = threadIdx.x & 31u;
  const bool take = n <= most;  // (the same in every block)
  if (take && n) {
    const uint32_t warps = gridDim.x * (kPathThreads / 32), warp = blockIdx.x * (kPathThreads / 32) + threadIdx.x / 32u;
    const uint32_t use = min(32u, (n + warps - 1u) / warps);
    const int nodeLanes = int(use) * kNodeLanes / 32;
    uint32_t extends = 0, shadows = 0, events = 0, nn = 0, nt = 0;
    bool ovf = false, more = false, stop = false;
    PathSrc src;
    src.hit.W = src.shadow.W = &P.W;
    src.hit.P = src.shadow.P = &P;
    src.hit.rO = P.W.rayO[pass.cur];
    src.hit.rD = P.W.rayD[pass.cur];
    src.shadow.rO = P.W.shO;
    src.shadow.rD = P.W.shD;
    src.any = false;
    Trav<kPathThreads, kPathStack> tr;
    tr.gMask = tr.tMask = 0u;
    tr.bottom = 0;
    uint32_t i = warp * use + lane;
    int state = lane < use && i < n && from <= lastPass ? kPathHit : kPathNone;
    if (state == kPathHit) src.load(P.S, i, tr);
    while (!stop) {
      const unsigned tracing = __ballot_sync(0xffffffffu, state == kPathHit || state == kPathShadow);
      const unsigned waiting = __ballot_sync(0xffffffffu, state == kPathShade);
      if (!(tracing | waiting)) break;
      bool next = false;  // the path's next closest hit, or the next path
      if (!tracing) {
        if (state == kPathShade) {
          ShadeOut out;
          shadeAny<MASK>(P, pass, i, out);
          ++extends;
          if (out.next) storeNext(W, pass.cur, i, out);
          more = out.next && pass.wave < lastPass;
          next = !out.shadow;
          if (out.shadow) {
            ++shadows;
            storeShadow(W, i, out);
            state = kPathShadow;
            src.any = true;
            src.shadow.wave = pass.wave;
            events = 0;
            src.load(P.S, i, tr);
          }
        }
        __syncwarp();
      } else {
        const bool on = tracing >> lane & 1u;
        if (traceRound<false, false>(P.S, src, tr, i, on, tracing, nodeLanes, false, P.stackLimit, events, sh, lstack,
                                     nn, nt, ovf, stop)) {
          src.finish(i, tr.found);
          next = state == kPathShadow;
          state = kPathShade;
        }
      }
      if (next) {
        if (more) {
          ++pass.wave;
        } else {
          i += warps * use;
          pass.wave = from;
        }
        more = more || i < n;
        state = more ? kPathHit : kPathNone;
        if (more) {
          src.any = false;
          events = 0;
          src.load(P.S, i, tr);
        }
        more = false;
      }
    }
    if (ovf) atomicAdd(&W.cnt->stackOverflow, 1ull);
    extends = __reduce_add_sync(0xffffffffu, extends);
    shadows = __reduce_add_sync(0xffffffffu, shadows);
    if (lane == 0 && extends) atomicAdd(&W.cnt->extendRays, static_cast<unsigned long long>(extends));
    if (lane == 0 && shadows) atomicAdd(&W.cnt->shadowRays, static_cast<unsigned long long>(shadows));
  }
  // the last block to leave empties the queue and decides how it goes on
  if (threadIdx.x != 0) return;
  __threadfence();
  if (atomicAdd(&W.cnt->c[kCntTicket], 1u) + 1u == gridDim.x) {
    __threadfence();
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
// 2.2 / 1.5, 32,768 2.3 / 2.3.  (Before a lane's occlusion ray and next closest
// hit were traced without a wait in between, 5 to 17% less for the path kernel;
// 65,536, 131,072 and 196,608 measured again since: within 1% at 720p, 19.5,
// 20.0 and 21.3 ms against 19.7 for 1920x1080 of 8 frames.)
uint32_t pathMost(uint32_t classMask) { return classMask & ~kCoreClasses ? 24576u : 98304u; }
int pathBlocksPerSm() {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_path<kAllClasses>, kPathThreads, 0);
  return n > 0 ? n : 1;
}

}  // namespace asuna
