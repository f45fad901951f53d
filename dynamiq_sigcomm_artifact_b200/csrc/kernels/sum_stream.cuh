// Where the second half of a column sum runs.
//
// A parameter gradient that is a column sum has no reader before its bucket's optimizer step, so the small launch that
// adds the partial rows need not stand between the kernels of backward: with a stream given (the one that the optimizer
// steps run on) it is forked off there.  48 such launches of 3 us each stood in a GPT-2 small step.
#pragma once
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDACachingAllocator.h>

#include "column_sums.cuh"

namespace dq {

// sums of `arrays` arrays of partial rows in `part`, on the stream with handle `sum_stream` (0: the current one) behind
// what the current stream holds now
inline void finish_sums(const at::Tensor& part, float* out0, float* out1, float* out2, int arrays, int nparts, int cols,
                        int64_t sum_stream) {
  const auto current = at::cuda::getCurrentCUDAStream();
  auto stream = current;
  if (sum_stream != 0 && sum_stream != reinterpret_cast<int64_t>(current.stream())) {
    stream = at::cuda::getStreamFromExternal(reinterpret_cast<cudaStream_t>(sum_stream), part.device().index());
    at::cuda::CUDAEvent ready;
    ready.record(current);
    ready.block(stream);
    c10::cuda::CUDACachingAllocator::recordStream(part.storage().data_ptr(), stream);
  }
  reduce_arrays(part.data_ptr<float>(), out0, out1, out2, arrays, nparts, cols, stream);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
}

}  // namespace dq
