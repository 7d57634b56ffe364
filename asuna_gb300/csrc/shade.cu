// shade.cu — ray generation, shading and film accumulation kernels.
//
// One wavefront iteration per path depth: raygen fills extend queue 0 with
// camera rays; after each closest-hit pass, `shade` runs the miss shader or
// the closest-hit shader of the hit material (emitters use the Lambertian
// light branch), writes next-event shadow rays into the shadow queue and the
// continuation rays into the other extend queue (warp-aggregated ballot/popc
// compaction, one atomic per warp); `accumulate` folds the finished samples
// into the film in frame order.
//
// Restates (file:line of the reference):
//   raygen      raytrace.projective.rgen:26-100 (seed, jitter, cameras)
//   shade/miss  raytrace.default.rmiss:24-56
//   shade/hit   rchit_layouts.glsl:61-167, brdf_lambertian.rchit:12-151,
//               brdf_rough_plastic.rchit:191-269, bsdf_dielectric.rchit:74-139,
//               brdf_emissive.rchit:12-27, brdf_plastic.rchit:43-205,
//               brdf_mirror.rchit:12-106, brdf_conductor.rchit:14-164,
//               brdf_rough_conductor.rchit, brdf_phong.rchit:12-194,
//               brdf_pbr_metalness_roughness.rchit:12-219,
//               brdf_disney.rchit:31-477, brdf_kang18.rchit:11-249
//   accumulate  raytrace.projective.rgen:134-179
//
// Compiled with -fmad=false: the float arithmetic rounds operation by
// operation in the order of the reference's GLSL source.
#include <cuda_runtime.h>

#include "common.h"
#include "kernels.h"
#include "shade.cuh"

namespace asuna {
using namespace dm;

namespace {

__device__ __forceinline__ uint32_t laneId() { return threadIdx.x & 31u; }

// Block-aggregated appends to the shadow queue and the next extend queue:
// every thread of the block calls it once per round (the barriers are
// uniform); one shared-memory add per warp and queue, then one global add per
// queue and block, so the two hot queue counters see an eighth of the
// atomics of per-warp appends.  Returns the slots of the thread's entries.
__device__ __forceinline__ void blockAppend2(bool wantA, bool wantB, uint32_t* counterA, uint32_t* counterB,
                                             uint32_t* shCount, uint32_t* shBase, uint32_t& slotA,
                                             uint32_t& slotB) {
  if (threadIdx.x < 2) shCount[threadIdx.x] = 0u;
  __syncthreads();
  const unsigned ma = __ballot_sync(0xffffffffu, wantA), mb = __ballot_sync(0xffffffffu, wantB);
  uint32_t offA = 0, offB = 0;
  if (laneId() == 0) {
    if (ma) offA = atomicAdd(&shCount[0], uint32_t(__popc(ma)));
    if (mb) offB = atomicAdd(&shCount[1], uint32_t(__popc(mb)));
  }
  offA = __shfl_sync(0xffffffffu, offA, 0);
  offB = __shfl_sync(0xffffffffu, offB, 0);
  __syncthreads();
  if (threadIdx.x == 0 && shCount[0]) shBase[0] = atomicAdd(counterA, shCount[0]);
  if (threadIdx.x == 1 && shCount[1]) shBase[1] = atomicAdd(counterB, shCount[1]);
  __syncthreads();
  const unsigned below = (1u << laneId()) - 1u;
  slotA = wantA ? shBase[0] + offA + uint32_t(__popc(ma & below)) : 0u;
  slotB = wantB ? shBase[1] + offB + uint32_t(__popc(mb & below)) : 0u;
}

__device__ __forceinline__ uint32_t findRange(const RangeDev* r, uint32_t n, uint32_t p) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (__ldg(&r[mid].pathBegin) <= p)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

}  // namespace

// ---------------------------------------------------------------------------
// raygen: raytrace.projective.rgen:26-100
__global__ void __launch_bounds__(256) k_raygen(KParams P) {
  const WaveDev& W = P.W;
  const uint32_t stride = gridDim.x * blockDim.x;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    W.cnt->c[kCntExtend0] = W.numPaths;
    W.cnt->c[kCntExtend1] = 0;
    W.cnt->c[kCntShadow] = 0;
    W.cnt->c[kCntFetchExtend] = 0;
    W.cnt->c[kCntFetchShadow] = 0;
    W.cnt->c[kCntPass] = 1;
    W.cnt->c[kCntTicket] = 0;
    W.cnt->paths += W.numPaths;
  }
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < W.numPaths; p += stride) {
    const uint32_t ri = findRange(W.ranges, W.numRanges, p);
    const RangeDev R = W.ranges[ri];
    const ShotDev& sh = W.shots[R.shot];
    const uint32_t local = p - R.pathBegin;
    const uint32_t frame = R.frameBegin + local / R.npix;
    const uint32_t pix = local % R.npix;
    const uint32_t x = pix % sh.width, y = pix / sh.width;
    uint32_t seed = xxhash32(x, y, hashFrame(frame, sh.seed));
    const asuna_camera& cam = sh.cam;
    f3 origin = transformPoint(cam.camera_to_world, splat(0.0f));
    f2 jitter = (frame == 0) ? f2{0.5f, 0.5f} : rnd2(seed);
    f2 pixel{float(x) + jitter.x, float(y) + jitter.y};
    f3 ro = origin, rd = splat(0.0f);
    if (cam.type == ASUNA_CAMERA_PERSPECTIVE) {
      f3 pCamera = transformPoint(cam.raster_to_camera, f3{pixel.x, pixel.y, 0.0f});
      f3 r = makeNormal(pCamera);
      if (cam.aperture > 0.0f) {
        f2 uLens = rnd2(seed);
        f2 d = concentricSampleDisk(uLens);
        f2 pLens{cam.aperture * d.x, cam.aperture * d.y};
        float ft = cam.focal_distance / r.z;
        f3 pFocus = ft * r;
        f3 o{pLens.x, pLens.y, 0.0f};
        ro = transformPoint(cam.camera_to_world, o);
        r = pFocus - o;
      }
      rd = transformDirection(cam.camera_to_world, r);
    } else if (cam.type == ASUNA_CAMERA_OPENCV) {
      float px = (pixel.x - cam.fxfycxcy[2]) / cam.fxfycxcy[0];
      float py = (pixel.y - cam.fxfycxcy[3]) / cam.fxfycxcy[1];
      rd = transformDirection(cam.camera_to_world, f3{px, py, 1.0f});
    }
    // Gaussian filter weight of this sample, rgen:134-145
    const float alpha = -2.0f;
    const float expXY = mexp(alpha * 2.0f * 2.0f);
    float ox = jitter.x - 0.5f, oy = jitter.y - 0.5f;
    float fw = gmax(0.0f, mexp(alpha * ox * ox) - expXY) * gmax(0.0f, mexp(alpha * oy * oy) - expXY);
    W.rayO[0][p] = make_float4(ro.x, ro.y, ro.z, INF);
    W.rayD[0][p] = make_float4(rd.x, rd.y, rd.z, __uint_as_float(p));
    W.path[p].thp = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    W.rad[p] = make_float4(0.0f, 0.0f, 0.0f, fw);
    W.path[p].info = make_uint4(seed, EBsdfNull, ri, local);
    if (P.records) W.rec[p] = make_uint4(0u, 0u, 0u, 1u);
    if (frame == 0) {
      // AOV images are rewritten at frame 0 (rgen:155-162): clear to (0,0,0,1)
      const uint32_t npx = sh.width * sh.height;
      for (uint32_t c = 0; c < sh.state.n_multi_channel && c < ASUNA_MAX_CHANNELS; ++c)
        sh.filmCh[size_t(c) * npx + pix] = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
    }
  }
}

// ---------------------------------------------------------------------------
// Splits the hits of the extend queue into the shading classes (material
// sort).  A block takes 256 hits at a time: lanes are grouped by class in
// each warp (one shared-memory add per class present), then one global
// append per class present in the block, so the few class counters see
// eight times fewer atomics than with per-warp appends.  Classes that no hit
// of a pass uses cost one empty launch.
__global__ void __launch_bounds__(256) k_classify(KParams P) {
  __shared__ uint32_t count[kNumShadeClasses], base[kNumShadeClasses];
  const WaveDev& W = P.W;
  const SceneDev& S = P.S;
  const uint32_t n = W.cnt->c[kCntExtend0 + passOf(P).cur];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    // the connect kernel that follows fetches shadow rays from 0
    W.cnt->c[kCntFetchShadow] = 0;
  }
  const uint32_t stride = gridDim.x * blockDim.x;
  // (i0 is the same for every thread of the block: the barriers are uniform)
  for (uint32_t i0 = blockIdx.x * blockDim.x; i0 < n; i0 += stride) {
    if (threadIdx.x < kNumShadeClasses) count[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t i = i0 + threadIdx.x;
    const int cls = i < n ? classOf(S, W.hitInst[i]) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, cls);
    const int leader = __ffs(peers) - 1;
    uint32_t off = 0;
    if (int(laneId()) == leader && cls >= 0) off = atomicAdd(&count[cls], uint32_t(__popc(peers)));
    off = __shfl_sync(0xffffffffu, off, leader);
    __syncthreads();
    if (threadIdx.x < kNumShadeClasses && count[threadIdx.x])
      base[threadIdx.x] = atomicAdd(&W.cnt->c[kCntCls0 + threadIdx.x], count[threadIdx.x]);
    __syncthreads();
    // (count was last read before the barrier above and base is written
    // again only after two more: the next round may start at once)
    if (cls >= 0) W.cls[cls][base[cls] + off + uint32_t(__popc(peers & ((1u << laneId()) - 1u)))] = i;
  }
}

// Shades the rays of one class.
template <int CLS>
__global__ void __launch_bounds__(256, kShadeMinBlocks) k_shadeClass(KParams P) {
  __shared__ uint32_t appendCount[2], appendBase[2];
  const WaveDev& W = P.W;
  const Pass pass = passOf(P);
  const int nxt = pass.cur ^ 1;
  const uint32_t n = W.cnt->c[kCntCls0 + CLS];
  const uint32_t* list = W.cls[CLS];
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i0 = blockIdx.x * blockDim.x; i0 < n; i0 += stride) {
    ShadeOut out;
    if (i0 + threadIdx.x < n) shadeHit<CLS>(P, pass, list[i0 + threadIdx.x], out);
    __syncwarp();
    if (CLS != kClsTerminal) {  // terminal paths append nothing
      // (i0 is the same for every thread of the block: the barriers inside
      // are reached by all of them, round by round)
      uint32_t sslot, nslot;
      blockAppend2(out.shadow, out.next, &W.cnt->c[kCntShadow], &W.cnt->c[kCntExtend0 + nxt], appendCount,
                   appendBase, sslot, nslot);
      if (out.shadow) storeShadow(W, sslot, out);
      if (out.next) storeNext(W, nxt, nslot, out);
    }
  }
}

// ---------------------------------------------------------------------------
// accumulate: rgen:147-179, frames in order, one thread per pixel of a range
__global__ void __launch_bounds__(256) k_accumulate(KParams P) {
  const WaveDev& W = P.W;
  const RangeDev R = W.ranges[blockIdx.y];
  const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= R.npix) return;
  const ShotDev& sh = W.shots[R.shot];
  float4 old = sh.filmRad[pix];
  float ow = sh.filmW[pix].x;
  for (uint32_t f = 0; f < R.nframes; ++f) {
    const uint32_t p = R.pathBegin + f * R.npix + pix;
    const uint32_t frame = R.frameBegin + f;
    const float4 r4 = W.rad[p];
    const float fw = r4.w;
    float rcl[3] = {gclamp(r4.x, 0.0f, 10.0f), gclamp(r4.y, 0.0f, 10.0f), gclamp(r4.z, 0.0f, 10.0f)};
    float rws[3] = {fw * rcl[0], fw * rcl[1], fw * rcl[2]};
    if (frame == 0) {
      old = make_float4(rws[0] / fw, rws[1] / fw, rws[2] / fw, 1.0f);
      ow = fw;
    } else {
      float nw = ow + fw;
      old = make_float4((old.x * ow + rws[0]) / nw, (old.y * ow + rws[1]) / nw, (old.z * ow + rws[2]) / nw, 1.0f);
      ow = nw;
    }
  }
  sh.filmRad[pix] = old;
  sh.filmW[pix] = make_float4(ow, ow, ow, ow);
}

// ---------------------------------------------------------------------------
// parity records: copy per-path radiance / filter weight with the record
__global__ void __launch_bounds__(256) k_records(KParams P, asuna_path_record* out) {
  const WaveDev& W = P.W;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < W.numPaths; p += gridDim.x * blockDim.x) {
    const float4 r4 = W.rad[p];
    const uint4 rc = W.rec[p];
    asuna_path_record o;
    o.radiance[0] = r4.x;
    o.radiance[1] = r4.y;
    o.radiance[2] = r4.z;
    o.filter_weight = r4.w;
    o.depth = rc.w;
    o.signature = rc.x;
    o.events = rc.y;
    o.shadows = rc.z;
    out[p] = o;
  }
}

// ---------------------------------------------------------------------------
// The sky's direction-independent part, once per scene.  Evaluated for every
// direction it was most of a sky scene's shading: 25 sky evaluations for each
// direction below the horizon (641x427x8 frames: shading 2.55 -> 0.41 ms).
__global__ void k_skyState(asuna_sun_and_sky sky, asuna_sky::SkyState<float>* out) {
  *out = asuna_sky::skyState<float>(asuna_sky::paramsOf<float>(sky));
}
int prepareSky(SceneDev& S, cudaStream_t s) {
  asuna_sky::SkyState<float>* d = nullptr;
  ASUNA_CUDA_TRY(cudaMalloc(reinterpret_cast<void**>(&d), sizeof(*d)));
  k_skyState<<<1, 1, 0, s>>>(S.sky, d);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(&S.skyState, d, sizeof(*d), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFree(d);
  ASUNA_CUDA_TRY(e);
  return ASUNA_OK;
}

void launchRaygen(const KParams& P, int grid, cudaStream_t s) { k_raygen<<<grid, 256, 0, s>>>(P); }
// classify, then one kernel per shading class the scene's materials can
// reach (each a persistent grid over its own list).  The classes are
// independent of each other: with `fork` they run side by side from three
// classes on (two gain nothing), so that a pass with few rays waits for the
// slowest class instead of for their sum.
void launchShade(const KParams& P, int grid, cudaStream_t s, const ShadeFork* fork) {
  k_classify<<<grid, 256, 0, s>>>(P);
  const uint32_t m = P.S.classMask | (1u << kClsTerminal);
  const int nc = __builtin_popcount(m), lanes = fork && nc > 2 ? (nc < kShadeForks + 1 ? nc : kShadeForks + 1) : 1;
  if (lanes > 1) {
    cudaEventRecord(fork->begin, s);
    for (int k = 0; k + 1 < lanes; ++k) cudaStreamWaitEvent(fork->stream[k], fork->begin, 0);
  }
  int at = 0;
  auto next = [&] {
    const int k = at++ % lanes;
    return k == 0 ? s : fork->stream[k - 1];
  };
  if (m & (1u << kClsTerminal)) k_shadeClass<kClsTerminal><<<grid, 256, 0, next()>>>(P);
  if (m & (1u << kClsLambertian)) k_shadeClass<kClsLambertian><<<grid, 256, 0, next()>>>(P);
  if (m & (1u << kClsRoughPlastic)) k_shadeClass<kClsRoughPlastic><<<grid, 256, 0, next()>>>(P);
  if (m & (1u << kClsDielectric)) k_shadeClass<kClsDielectric><<<grid, 256, 0, next()>>>(P);
  if (m & (1u << kClsPlastic)) k_shadeClass<kClsPlastic><<<grid, 256, 0, next()>>>(P);
  if (m & (1u << kClsMirror)) k_shadeClass<kClsMirror><<<grid, 256, 0, next()>>>(P);
  if (m & (1u << kClsConductor)) k_shadeClass<kClsConductor><<<grid, 256, 0, next()>>>(P);
  if (m & (1u << kClsRoughConductor)) k_shadeClass<kClsRoughConductor><<<grid, 256, 0, next()>>>(P);
  if (m & (1u << kClsPhong)) k_shadeClass<kClsPhong><<<grid, 256, 0, next()>>>(P);
  if (m & (1u << kClsPbr)) k_shadeClass<kClsPbr><<<grid, 256, 0, next()>>>(P);
  if (m & (1u << kClsDisney)) k_shadeClass<kClsDisney><<<grid, 256, 0, next()>>>(P);
  if (m & (1u << kClsKang18)) k_shadeClass<kClsKang18><<<grid, 256, 0, next()>>>(P);
  for (int k = 0; k + 1 < lanes; ++k) {
    cudaEventRecord(fork->end[k], fork->stream[k]);
    cudaStreamWaitEvent(s, fork->end[k], 0);
  }
}
int shadeLaunches(uint32_t classMask) { return 1 + __builtin_popcount(classMask | (1u << kClsTerminal)); }
int shadeBlocksPerSm() {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_shadeClass<kClsRoughPlastic>, 256, 0);
  return n > 0 ? n : 1;
}
void launchAccumulate(const KParams& P, uint32_t maxPix, uint32_t nranges, cudaStream_t s) {
  dim3 g((maxPix + 255) / 256, nranges);
  k_accumulate<<<g, 256, 0, s>>>(P);
}
void launchRecords(const KParams& P, asuna_path_record* out, int grid, cudaStream_t s) {
  k_records<<<grid, 256, 0, s>>>(P, out);
}

}  // namespace asuna
