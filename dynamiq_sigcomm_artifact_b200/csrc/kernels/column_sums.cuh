// The second half of every column sum: partial rows, one per CTA of the first half, added in a fixed order.
//
// A dependent launch (dependent_launch.cuh) behind the first half.  Forked to another stream instead, the sums delayed the
// GEMMs beside them (26 -> 43 us for a weight gradient of GPT-2 small).
#pragma once
#include <cuda_runtime.h>

#include "dependent_launch.cuh"

namespace dq {

inline int device_sms() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// out[a][c] = sum over the parts of array a: 32 columns x 32 part groups per CTA, blockIdx.y = array
static __global__ void __launch_bounds__(1024) reduce_arrays_kernel(const float* __restrict__ part, float* out0, float* out1,
                                                                    float* out2, int nparts, int cols) {
  __shared__ float sm[32][33];
  wait_for_previous();
  float* out = blockIdx.y == 0 ? out0 : (blockIdx.y == 1 ? out1 : out2);
  const float* p = part + static_cast<size_t>(blockIdx.y) * nparts * cols;
  const int c = blockIdx.x * 32 + threadIdx.x, g = threadIdx.y;
  float s = 0.f;
  if (c < cols)
    for (int i = g; i < nparts; i += 32) s += p[static_cast<size_t>(i) * cols + c];
  sm[g][threadIdx.x] = s;
  __syncthreads();
  float t = sm[threadIdx.x][g];  // transposed: warp g sums column g of the tile
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
  const int col = blockIdx.x * 32 + g;
  if (threadIdx.x == 0 && col < cols) out[col] = t;
}

inline void reduce_arrays(const float* part, float* out0, float* out1, float* out2, int arrays, int nparts, int cols,
                          cudaStream_t stream) {
  launch_dependent(reduce_arrays_kernel, dim3((cols + 31) / 32, arrays), dim3(32, 32), 0, stream, part, out0, out1, out2, nparts,
                   cols);
}

}  // namespace dq
