// Means of whole planes from the sums that a block's threads left in shared memory: what the squeeze-and-excite block
// behind a depthwise convolution starts from.
#pragma once
#include <cuda_runtime.h>

namespace ac {

// Plane i of the block has the sums [i * len, (i + 1) * len): a warp each, added in a fixed order.
__device__ __forceinline__ void plane_means(const float* sums, unsigned here, unsigned len, float* means, unsigned plane0, unsigned planes,
                                            int pixels) {
  const unsigned lane = threadIdx.x & 31, warps = (blockDim.x + 31) >> 5;
  for (unsigned i = threadIdx.x >> 5; i < here && plane0 + i < planes; i += warps) {
    float v = 0.f;
    for (unsigned j = lane; j < len; j += 32) v = __fadd_rn(v, sums[i * len + j]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) means[plane0 + i] = __fdiv_rn(v, (float)pixels);
  }
}

}  // namespace ac
