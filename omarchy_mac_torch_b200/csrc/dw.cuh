// Depthwise convolution: what the kernels of dw.cu and dw_tile.cu share.
#pragma once

#include "common.cuh"

namespace omt {

struct DwArgs {
  ActView x, y;  // fwd: x in, y out. dgrad: x = gy (in), y = dx (out). wgrad: x = x, y = gy.
  const float* w;
  const float* bias;
  int n, c, ih, iw, oh, ow, ks, stride, pad;
  uint32_t flags;
};

// dw_tile.cu: dense channels-last tensors, ks 3, 5 or 7, stride 1 or 2, any channel count; `vec`: c % 4 == 0 and 16-byte aligned
// tensors. `a` describes the convolution that the kernel performs (for the flipped input gradient: gy -> dx with stride 1).
bool dw_tile_ok(const DwArgs& a);
int dw_tile_conv(const DwArgs& a, bool flip, cudaStream_t s);
int dw_tile_wgrad(const DwArgs& a, bool vec, float scale, float* dw, omt_stream_t stream);
int dw_wgrad_finish(const float* part, int64_t total, int kk, int slices, float scale, float* dw, cudaStream_t s);  // dw.cu

}  // namespace omt
