// conv_tc.h — the tcgen05 3x3 convolution as the denoiser calls it: operands
// in rows (NHWC) or planes, and the layer's neighbours (pooling, upsampling,
// the network's output) in its epilogue.
#pragma once
#include <cuda_runtime.h>

namespace asuna {
namespace tc {

// An activation of c channels over n images of h x w pixels (P = n h w) is
// either [P][c] ("rows") or [c / 8][P][8] ("planes", bf16 only).
struct Conv {
  const void* in = nullptr;
  int n = 0, h = 0, w = 0, cin = 0;
  const void* weights = nullptr;  // asuna_nn_weights_tc's layout
  const float* bias = nullptr;
  int cout = 0;
  bool relu = false;
  bool planes = false;         // layout of in, mask and out
  const void* mask = nullptr;  // out *= (mask > 0)
  void* out = nullptr;
  bool f32 = false;  // out is fp32 (rows)
  // The grid may be launched while the stream's previous kernel still runs: it
  // waits for that kernel's end before it touches an activation, but reads the
  // weights and may read the bias at once (that kernel does not write them).
  bool chained = false;
  // planes only, all of them further results; out may then be null
  void* pool = nullptr;   // the 2x2 mean of the bf16 output (h and w even)
  void* up = nullptr;     // each output pixel four times, 2h x 2w
  float4* head = nullptr;  // channels 0..2 in fp32, one float4 per pixel
  // max(expm1(channel + log1p(radiance)), 0) of the imgH x imgW pixels that
  // the network's input was padded from
  float4* image = nullptr;
  const float4* radiance = nullptr;
  int imgH = 0, imgW = 0;
};

int conv3x3(cudaStream_t s, const Conv& c);

// Output channels of a weight slice: nt in asuna_nn_weights_tc's layout.
int sliceWidth(int cout);

}  // namespace tc
}  // namespace asuna
