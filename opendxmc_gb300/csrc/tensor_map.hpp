// tensor_map.hpp -- TMA descriptors of the denoiser's tensors.
// This part has no counterpart in the reference.
#pragma once

#include <cuda.h>

namespace dxmcg {
namespace nn {
// 5-D map (C, W, H, D, B) of a channels-last bf16 tensor with boxes of 16 channels by bx, by
// and bz voxels in the 32-byte swizzle, zero outside the tensor; false if it cannot be made
bool brickTensorMap(CUtensorMap* m, const void* base, int B, int D, int H, int W, int C, int bx, int by, int bz);
} // namespace nn
} // namespace dxmcg
