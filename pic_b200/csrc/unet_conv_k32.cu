// unet_conv_k32.cu -- convolutions that contract at most 32 channels
// (unet_conv_tile.h): instantiations only.
#include "unet_conv_tile.h"

using Fprop32x32 = Fprop<32, 32>;
using Fprop64x32 = Fprop<64, 32>;
using Dgrad32x32 = Dgrad<32, 32>;
using Dgrad64x32 = Dgrad<64, 32>;
UNET_CONV_DEFINE(conv_fprop_32_32, Fprop32x32)
UNET_CONV_DEFINE(conv_fprop_64_32, Fprop64x32)
UNET_CONV_DEFINE(conv_dgrad_32_32, Dgrad32x32)
UNET_CONV_DEFINE(conv_dgrad_64_32, Dgrad64x32)
