// unet_conv.cu -- 3x3 convolutions of the learned preconditioner on the
// 5th-generation tensor cores (unet_conv_tile.h): the entry point, its choice
// of a tile, and the 64 x 64 instantiations.  The weight gradient and the
// 8-channel first layer are in unet_ops.cu.
#include "unet_conv_tile.h"

using Fprop64x64 = Fprop<64, 64>;
using Dgrad64x64 = Dgrad<64, 64>;
UNET_CONV_DEFINE(conv_fprop_64_64, Fprop64x64)
UNET_CONV_DEFINE(conv_dgrad_64_64, Dgrad64x64)
int conv_fprop_32_32(UNET_CONV_ARGS);  // unet_conv_k32.cu
int conv_fprop_64_32(UNET_CONV_ARGS);
int conv_dgrad_32_32(UNET_CONV_ARGS);
int conv_dgrad_64_32(UNET_CONV_ARGS);
int conv_fprop_32_64(UNET_CONV_ARGS);  // unet_conv_n32.cu
int unet_conv8(int n, int h, int w, int k, const void *x, const void *wt, const void *bias, void *y, void *stream);

// Tiles by channel counts: a tile wider than the layer computes and stages
// zeros (half of a 64 x 64 tile, and of its im2col loads, for 32 channels),
// and a contraction step below the channel count would change the order of
// the sums, so 32 only where all channels fit in it: the same bits throughout.
// Measured (us, 64 x 64 tile -> the one chosen): fprop 32 -> 32 at 1025^2
// 202 -> 68, 96 -> 32 at 1025^2 347 -> 174, 32 -> 64 at 513^2 39 -> 25; dgrad at
// 4 x 128^2 of 32 -> 32 17.3 -> 10.3, of 96 -> 32 27 -> 14.5.  8 channels: 343 -> 52.
extern "C" int unet_conv(int32_t op, int32_t n, int32_t h, int32_t w, int32_t c, int32_t k, const void *a,
                         const void *b, void *d, const void *bias, void *workspace, size_t ws_bytes,
                         size_t *ws_need, void *stream) {
  if (n < 1 || h < 1 || w < 1 || c < 8 || k < 8 || (c % 8) || (k % 8)) return UNET_ERR_SHAPE;
  const bool query = (ws_need && !workspace && !stream);
  if (!query && (!a || !b || !d)) return UNET_ERR_SHAPE;
  auto call = [&](auto *f) { return f(n, h, w, c, k, a, b, bias, d, workspace, ws_bytes, ws_need, stream); };
  if (op == UNET_FPROP_RELU) {
    if (!query && !bias) return UNET_ERR_SHAPE;
    // 4-byte operands of whole rows, pixels counted in 32 bits
    if (c == 8 && !query && (((uintptr_t)a | (uintptr_t)b | (uintptr_t)d) & 3) == 0 && (int64_t)n * h * w < ((int64_t)1 << 31) - 64) {
      if (ws_need) *ws_need = 0;
      return unet_conv8(n, h, w, k, a, b, bias, d, stream);
    }
    if (c <= 32) return k <= 32 ? call(&conv_fprop_32_32) : call(&conv_fprop_64_32);
    return k <= 32 ? call(&conv_fprop_32_64) : call(&conv_fprop_64_64);
  }
  if (op == UNET_DGRAD) {  // contracts k, writes c
    if (k <= 32) return c <= 32 ? call(&conv_dgrad_32_32) : call(&conv_dgrad_64_32);
    return call(&conv_dgrad_64_64);
  }
  return UNET_ERR_SHAPE;
}
