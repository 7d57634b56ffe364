// kernels.h — launch interface of the wavefront kernels.
#pragma once
#include <cuda_runtime.h>

#include "dev_types.h"

namespace asuna {

struct KParams {
  SceneDev S;
  WaveDev W;
  uint32_t depth;  // bounce being processed (1-based)
  int32_t cur;     // extend queue holding this bounce's rays (0/1); -1: both from the counters (passOf)
  int32_t records; // write per-path parity records
  int32_t counters;
  uint32_t refillLanes;  // traversal: idle lanes of a warp that trigger a queue fetch
  int32_t speculate;     // traversal: postponed leaves walk on speculatively
  int32_t occupancy;     // traversal: resident blocks per SM of the kernel variant (8, 10 or 12)
  int32_t stackLimit;    // traversal: stack entries a ray may use, in [1, kStackDepth] (the host clamps it)
  int32_t blockThreads;  // traversal: threads per block (64, 128, 256; 0 = 128)
  int32_t sharedStack;   // traversal: stack words in shared memory (16, 24, 32; 0 = 24), two an entry
};

// The wavefront pass that a kernel works on.  A pass that a graph repeats
// while rays are left finds its number in the counters; without the queue
// sort the queues alternate with it.
struct Pass {
  uint32_t wave;
  int cur;
};
__device__ __forceinline__ Pass passOf(const KParams& P) {
  if (P.cur >= 0) return Pass{P.depth, P.cur};
  const uint32_t w = P.W.cnt->c[kCntPass];
  return Pass{w, int((w - 1u) & 1u)};
}

constexpr int kTraceThreads = 128;
constexpr int kTraceMinBlocks = 8;   // resident blocks per SM the traversal kernels are compiled for
constexpr int kStackDepth = 64;      // traversal stack entries per ray
constexpr int kSharedStack = 24;     // words in shared memory, two an entry (the rest in local memory)
constexpr int kRefillLanes = 8;      // default idle lanes of a warp that trigger a queue fetch
constexpr int kShadeMinBlocks = 3;   // resident 256-thread blocks per SM the shading kernel is compiled for

// S.skyState of S.sky (evaluated on the device, with the shading kernels'
// rounding; waits for the stream)
int prepareSky(SceneDev& S, cudaStream_t s);
// the importance tables of an uploaded W x H environment map (waits for the stream)
int prepareEnvTables(const float4* env, int W, int H, float2* marg, float2* cond, cudaStream_t s);
void launchRaygen(const KParams& P, int grid, cudaStream_t s);
// Streams and events for the shading classes of a pass to run side by side:
// one for every class but the pass's own stream's (a scene of twelve classes,
// 480x270, 4 frames: 4.22 ms in a row, 3.30 on 3 side streams, 3.03 on 11).
constexpr int kShadeForks = kNumShadeClasses - 1;
struct ShadeFork {
  cudaStream_t stream[kShadeForks] = {};
  cudaEvent_t begin = nullptr, end[kShadeForks] = {};
};
void launchShade(const KParams& P, int grid, cudaStream_t s, const ShadeFork* fork = nullptr);
// kernels launchShade issues for a scene's class mask (classify included)
int shadeLaunches(uint32_t classMask);
void launchAccumulate(const KParams& P, uint32_t maxPix, uint32_t nranges, cudaStream_t s);
// counting-sorts extend queue P.cur into queue P.cur ^ 1 (count, scan,
// scatter); mode 1: octant + 4^3 origin cells, 2: octant + 8^3 (Morton)
void launchSortQueue(const KParams& P, int mode, int grid, cudaStream_t s);
void launchRecords(const KParams& P, asuna_path_record* out, int grid, cudaStream_t s);
void launchExtend(const KParams& P, int grid, cudaStream_t s);
// The path kernel: follows the rays of pass P.depth (queue P.cur) to pass
// `lastPass` if there are at most `most`, and empties the queue.  With a
// conditional `handle` it works on the pass after the counters' one, makes
// that the current pass and sets the condition to whether it has rays left.
void launchPath(const KParams& P, int lastPass, uint32_t most, int grid, cudaGraphConditionalHandle handle,
                cudaStream_t s);
// rays up to which the path kernel is faster than wavefront passes
uint32_t pathMost(uint32_t classMask);
int pathBlocksPerSm();
void launchConnect(const KParams& P, int grid, cudaStream_t s);
// resident blocks per SM of the traversal variant (occupancy class 8/10/12 =
// 32/40/48 resident warps, block size, shared-memory stack words)
int traceBlocksPerSm(int occupancy = kTraceMinBlocks, int blockThreads = kTraceThreads,
                     int sharedStack = kSharedStack);
int shadeBlocksPerSm();

// Standalone ray queries (tests): rays are (o.xyz, tmin), (d.xyz, tmax).  Adds
// the lanes with a traversal cut short to `cut`.
void launchTraceQuery(const SceneDev& S, const float4* o, const float4* d, uint32_t n, int anyHit, float4* hit,
                      uint32_t* inst, uint32_t* cut, cudaStream_t s);

}  // namespace asuna
