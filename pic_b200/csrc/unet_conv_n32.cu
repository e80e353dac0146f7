// unet_conv_n32.cu -- the forward convolution to at most 32 channels from more
// (unet_conv_tile.h): instantiation only.
#include "unet_conv_tile.h"

using Fprop32x64 = Fprop<32, 64>;
UNET_CONV_DEFINE(conv_fprop_32_64, Fprop32x64)
