// Elementwise halves of the THC baseline as single kernels: clip + scale + stochastic rounding to integer bins
// (rounding offsets from the counter-based generator, so a run is reproducible from its seed), and the inverse.
// The Hadamard rotation around them is fwht_pow2.cu; the bins travel over the fused
// kernel's identity wire.
//
// Reference counterparts (chains of torch operators): testbed_evaluation/new_comm_hooks/thc_hooks.py:152-223
// (quantise), :226-270 (dequantise); simulation stack simulations_llm/new_comm_hooks/thc_hooks.py:123-339.
//
// `stats` is what one small sum all-reduce leaves on every rank: stats[r] = ||g_r|| for r < world (each rank
// contributes its own entry), stats[world] = sum over ranks of the first rotated coordinate, which THC sends
// exactly.  range = T * max_r stats[r] / sqrt(d), at least 1e-30.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "../common/exact_div.cuh"
#include "../common/philox.cuh"
#include "dependent_launch.cuh"

namespace dq {
namespace {

__device__ __forceinline__ float thc_range(const float* stats, int world, float t_over_sqrt_d) {
  float m = 0.0f;
  for (int r = 0; r < world; ++r) m = fmaxf(m, stats[r]);
  return fmaxf(__fmul_rn(t_over_sqrt_d, m), 1e-30f);
}

__device__ __forceinline__ float thc_bin(float y, uint32_t byte, float range, const SharedDivisor& by_two_range, float top) {
  const float u = __fmul_rn(__fadd_rn(static_cast<float>(byte), 0.5f), 1.0f / 256.0f);
  const float c = fminf(fmaxf(y, -range), range);
  const float t = __fmul_rn(by_two_range(__fadd_rn(c, range)), top);
  return fminf(fmaxf(floorf(__fadd_rn(t, u)), 0.0f), top);
}

// bins = clamp(floor((clamp(y, -range, range) + range) / (2 range) * (levels - 1) + u), 0, levels - 1),
// u = (byte + 0.5) / 256 with byte i from Philox-4x32-7 counter (i / 16, 0, stream, step).
// A warp takes 512 values: lane l draws the 16 bytes of values 16 l .. 16 l + 15, and every memory access is 512
// contiguous bytes, so the bytes change lanes (a lane's four values need one word of another lane's draw).  With a
// thread per draw the scalar accesses were 64 bytes apart: 2^22 values took 24 us.
__global__ void __launch_bounds__(256) thc_quantize_kernel(float* __restrict__ y, const float* __restrict__ stats, int world,
                                                           float t_over_sqrt_d, int levels, long long d, uint32_t stream,
                                                           uint32_t step, uint32_t seed_lo, uint32_t seed_hi) {
  wait_for_previous();
  let_next_start();
  const float range = thc_range(stats, world, t_over_sqrt_d);
  const float top = static_cast<float>(levels - 1);
  const SharedDivisor two_range(__fmul_rn(2.0f, range));
  const int lane = threadIdx.x & 31;
  const long long warp = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const long long nwarps = (gridDim.x * static_cast<long long>(blockDim.x)) >> 5;
  const bool aligned = (reinterpret_cast<uintptr_t>(y) & 15u) == 0;
  for (long long base = warp * 512; base < d; base += nwarps * 512) {
    const U4 r = philox4x32<7>(static_cast<uint32_t>(base / 16 + lane), 0u, stream, step, seed_lo, seed_hi);
    float4 q[4];
    const bool whole = aligned && base + 512 <= d;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long i = base + j * 128 + lane * 4;
      if (whole) {
        q[j] = *reinterpret_cast<const float4*>(y + i);
      } else {
        q[j].x = i < d ? y[i] : 0.f, q[j].y = i + 1 < d ? y[i + 1] : 0.f;
        q[j].z = i + 2 < d ? y[i + 2] : 0.f, q[j].w = i + 3 < d ? y[i + 3] : 0.f;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int from = j * 8 + (lane >> 2);
      const uint32_t w0 = __shfl_sync(0xFFFFFFFFu, r.x, from), w1 = __shfl_sync(0xFFFFFFFFu, r.y, from);
      const uint32_t w2 = __shfl_sync(0xFFFFFFFFu, r.z, from), w3 = __shfl_sync(0xFFFFFFFFu, r.w, from);
      const uint32_t w = (lane & 2) ? ((lane & 1) ? w3 : w2) : ((lane & 1) ? w1 : w0);
      q[j].x = thc_bin(q[j].x, w & 0xFFu, range, two_range, top);
      q[j].y = thc_bin(q[j].y, (w >> 8) & 0xFFu, range, two_range, top);
      q[j].z = thc_bin(q[j].z, (w >> 16) & 0xFFu, range, two_range, top);
      q[j].w = thc_bin(q[j].w, w >> 24, range, two_range, top);
      const long long i = base + j * 128 + lane * 4;
      if (whole) {
        *reinterpret_cast<float4*>(y + i) = q[j];
      } else {
        if (i < d) y[i] = q[j].x;
        if (i + 1 < d) y[i + 1] = q[j].y;
        if (i + 2 < d) y[i + 2] = q[j].z;
        if (i + 3 < d) y[i + 3] = q[j].w;
      }
    }
  }
}

// mean = (total / (levels - 1) * (2 range) - world * range) / world; mean[0] = stats[world] / world
// Four values per access and two accesses in flight (one scalar at a time left 2^22 values at 15 us).  The middle
// bin of an odd number of levels gives a zero, which the ordinary division sends down its slow path: see exact_div.cuh.
__global__ void __launch_bounds__(256) thc_dequantize_kernel(float* __restrict__ total, const float* __restrict__ stats,
                                                             int world, float t_over_sqrt_d, int levels, long long d) {
  wait_for_previous();
  let_next_start();
  const float range = thc_range(stats, world, t_over_sqrt_d);
  const float two_range = __fmul_rn(2.0f, range), top = static_cast<float>(levels - 1);
  const float w = static_cast<float>(world), shift = __fmul_rn(w, range);
  const SharedDivisor by_top(top), by_world(w);
  auto mean = [&](float t) { return by_world(__fsub_rn(__fmul_rn(by_top(t), two_range), shift)); };
  const long long d4 = (reinterpret_cast<uintptr_t>(total) & 15u) == 0 ? d >> 2 : 0;
  const long long first = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  const long long step = gridDim.x * static_cast<long long>(blockDim.x);
  const float exact = __fdiv_rn(stats[world], w);
#pragma unroll 2
  for (long long i = first; i < d4; i += step) {
    float4 q = reinterpret_cast<const float4*>(total)[i];
    q = make_float4(mean(q.x), mean(q.y), mean(q.z), mean(q.w));
    if (i == 0) q.x = exact;
    reinterpret_cast<float4*>(total)[i] = q;
  }
  for (long long i = 4 * d4 + first; i < d; i += step) total[i] = i == 0 ? exact : mean(total[i]);
}

void check_thc(const at::Tensor& y, const at::Tensor& stats, int64_t world, int64_t levels) {
  TORCH_CHECK(y.is_cuda() && y.scalar_type() == at::kFloat && y.is_contiguous() && y.dim() == 1, "thc: flat fp32 CUDA tensor");
  TORCH_CHECK(stats.is_cuda() && stats.scalar_type() == at::kFloat && stats.is_contiguous() && stats.numel() >= world + 1,
              "thc: stats needs world + 1 fp32 entries on the device");
  TORCH_CHECK(world >= 1 && world <= 4096 && levels >= 2, "thc: bad world / levels");
}

}  // namespace

void thc_quantize_(at::Tensor y, at::Tensor stats, int64_t world, double t_over_sqrt_d, int64_t levels, int64_t stream,
                   int64_t step, int64_t seed) {
  check_thc(y, stats, world, levels);
  c10::cuda::CUDAGuard guard(y.device());
  const long long d = y.numel();
  if (d == 0) return;
  const int grid = static_cast<int>(std::min<long long>((d + 4095) / 4096, 148 * 8));
  const uint64_t s = static_cast<uint64_t>(seed);
  C10_CUDA_CHECK(launch_dependent(
      thc_quantize_kernel, grid, 256, 0, at::cuda::getCurrentCUDAStream(), y.data_ptr<float>(), stats.data_ptr<float>(), static_cast<int>(world), static_cast<float>(t_over_sqrt_d),
      static_cast<int>(levels), d, static_cast<uint32_t>(stream), static_cast<uint32_t>(step),
      static_cast<uint32_t>(s & 0xFFFFFFFFull), static_cast<uint32_t>(s >> 32)));
}

void thc_dequantize_(at::Tensor total, at::Tensor stats, int64_t world, double t_over_sqrt_d, int64_t levels) {
  check_thc(total, stats, world, levels);
  c10::cuda::CUDAGuard guard(total.device());
  const long long d = total.numel();
  if (d == 0) return;
  const int grid = static_cast<int>(std::min<long long>((d + 1023) / 1024, 148 * 8));
  C10_CUDA_CHECK(launch_dependent(
      thc_dequantize_kernel, grid, 256, 0, at::cuda::getCurrentCUDAStream(), total.data_ptr<float>(), stats.data_ptr<float>(), static_cast<int>(world), static_cast<float>(t_over_sqrt_d),
      static_cast<int>(levels), d));
}

}  // namespace dq
