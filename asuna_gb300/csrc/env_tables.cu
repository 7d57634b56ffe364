// env_tables.cu — the environment map's importance tables, made on the device.
//
// The operations and their order are those of asuna_envmap_tables
// (host_scene.cpp; src/core/texture.cpp:144-226 of the reference): float sums
// in texel order, double literals and divisions stored to float, lower bounds.
// A texel's weight takes the two fused multiply-adds that the compiler of the
// GB300's Arm host makes of the expression there, so that a map's tables do not
// depend on which side made them.
// A warp sums a row (32 texels loaded at once, added one after the other in
// registers), one block sums the rows, and the inverse lookups run a texel per
// thread.  Creating a scene under a 512x256 map: 5.2 -> 1.2 ms; the cost here
// is the latency of the in-order sums.
// Compiled with -fmad=false.
#include <cuda_runtime.h>

#include "common.h"
#include "kernels.h"

namespace asuna {
namespace {

constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ float weightOf(float4 c) {
  return float(__fma_rn(0.1, double(c.z), __fma_rn(0.3, double(c.x), __dmul_rn(0.6, double(c.y)))));
}
__device__ __forceinline__ float over(float v, float sum) { return float(__ddiv_rn(double(v), __dadd_rn(double(sum), 1e-7))); }

// the first i in [lo, hi) with a[i] >= v, else hi
__device__ __forceinline__ int lowerBound(const float* a, int lo, int hi, float v) {
  while (lo < hi) {
    const int mid = (lo + hi) / 2;
    if (a[mid] < v)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// one warp per row: normalised pdf and cdf of the row, its sum
__global__ void __launch_bounds__(128) k_envRows(const float4* __restrict__ env, int W, int H, float* pdf, float* cdf,
                                                 float* rowSum) {
  const int lane = threadIdx.x & 31, row = int(blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32);
  if (row >= H) return;
  const size_t at = size_t(row) * W;
  float sum = 0.0f;
  for (int x0 = 0; x0 < W; x0 += 32) {
    const int x = x0 + lane;
    const float w = x < W ? weightOf(__ldg(&env[at + x])) : 0.0f;
    float mine = 0.0f;
    const int n = min(32, W - x0);
    for (int k = 0; k < n; ++k) {
      sum = __fadd_rn(sum, __shfl_sync(kAll, w, k));
      if (lane == k) mine = sum;
    }
    if (x < W) {
      pdf[at + x] = w;
      cdf[at + x] = mine;
    }
  }
  for (int x = lane; x < W; x += 32) {
    pdf[at + x] = over(pdf[at + x], sum);
    cdf[at + x] = over(cdf[at + x], sum);
  }
  if (lane == 0) rowSum[row] = sum;
}

// one block: the rows' cdf and the marginal table (first column; the rest 0)
__global__ void __launch_bounds__(1024) k_envMarginal(const float* __restrict__ rowSum, int W, int H, float* cdf,
                                                      float2* marg) {
  __shared__ float total;
  if (threadIdx.x < 32) {
    float sum = 0.0f;
    for (int j0 = 0; j0 < H; j0 += 32) {
      const int j = j0 + int(threadIdx.x);
      const float w = j < H ? rowSum[j] : 0.0f;
      float mine = 0.0f;
      const int n = min(32, H - j0);
      for (int k = 0; k < n; ++k) {
        sum = __fadd_rn(sum, __shfl_sync(kAll, w, k));
        if (int(threadIdx.x) == k) mine = sum;
      }
      if (j < H) cdf[j] = mine;
    }
    if (threadIdx.x == 0) total = sum;
  }
  __syncthreads();
  for (int j = threadIdx.x; j < H; j += blockDim.x) cdf[j] = over(cdf[j], total);
  __syncthreads();
  for (int j = threadIdx.x; j < H; j += blockDim.x) {
    const float row = float(lowerBound(cdf, 0, H, __fdiv_rn(float(j + 1), float(H))));
    marg[size_t(j) * W] = make_float2(__fdiv_rn(row, float(H)), over(rowSum[j], total));
  }
}

__global__ void __launch_bounds__(256) k_envConditional(const float* __restrict__ pdf, const float* __restrict__ cdf,
                                                        int W, int H, float2* cond) {
  const size_t n = size_t(W) * H;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
    const int x = int(i % W);
    const float* row = cdf + (i - x);
    const float col = float(lowerBound(row, 0, W, __fdiv_rn(float(x + 1), float(W))));
    cond[i] = make_float2(__fdiv_rn(col, float(W)), pdf[i]);
  }
}

}  // namespace

int prepareEnvTables(const float4* env, int W, int H, float2* marg, float2* cond, cudaStream_t s) {
  const size_t n = size_t(W) * H;
  struct Tmp {
    float* p = nullptr;
    ~Tmp() { cudaFree(p); }
  } tmp;
  ASUNA_CUDA_TRY(cudaMalloc(reinterpret_cast<void**>(&tmp.p), (2 * n + 2 * size_t(H)) * sizeof(float)));
  float *pdf = tmp.p, *cdf = pdf + n, *rowSum = cdf + n, *cdf1 = rowSum + H;
  ASUNA_CUDA_TRY(cudaMemsetAsync(marg, 0, n * sizeof(float2), s));
  k_envRows<<<unsigned((H + 3) / 4), 128, 0, s>>>(env, W, H, pdf, cdf, rowSum);
  k_envMarginal<<<1, 1024, 0, s>>>(rowSum, W, H, cdf1, marg);
  k_envConditional<<<unsigned(n / 256 + 1 < 4096 ? n / 256 + 1 : 4096), 256, 0, s>>>(pdf, cdf, W, H, cond);
  ASUNA_CUDA_TRY(cudaGetLastError());
  ASUNA_CUDA_TRY(cudaStreamSynchronize(s));
  return ASUNA_OK;
}

}  // namespace asuna
