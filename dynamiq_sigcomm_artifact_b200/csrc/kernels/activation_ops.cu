// GELU of (pre + bias), and its backward together with the bias gradient.
//
// The bias of the linear layer in front is added here in fp32 instead of in the GEMM's epilogue, so that its gradient
// - the column sums of the gradient this kernel writes - falls out of the pass that has those values in registers:
// activation gradient and bias gradient of an [8192, 3072] layer were 33.6 + 7.4 + 3.9 us in three launches over
// 200 MB, and are one pass over 150 MB plus a sum of partial rows.  Bound by memory (tanh form: two special-function
// instructions a value either way).
//
// Reference counterpart: the Hugging Face MLPs of testbed_evaluation/train_llm_causal.py:490-497.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "column_sums.cuh"
#include "norm_kernels.cuh"

namespace dq {
namespace {

using normk::Raw8;
using normk::Vec8;

constexpr float kSqrt2OverPi = 0.79788456f, kCubic = 0.044715f, kInvSqrt2 = 0.70710678f, kInvSqrt2Pi = 0.39894228f;

// tanh form as x * sigmoid(2 u): no cancellation for negative x
__device__ __forceinline__ float sigmoid_2u(float x) {
  const float u = kSqrt2OverPi * x * fmaf(kCubic * x, x, 1.0f);
  return __fdividef(1.0f, 1.0f + __expf(-2.0f * u));
}

// Normal distribution function from a rational approximation of erfc (C. Hastings, Approximations for Digital Computers,
// 1955; Abramowitz and Stegun 7.1.26): |error| < 1e-7, below the rounding of bf16 results by four decimal digits; a
// reciprocal, an exponential and six multiply-adds where the library's erff takes some thirty instructions.  `e` is
// exp(-x^2 / 2), which the density needs as well.
__device__ __forceinline__ float normal_cdf(float x, float e) {
  const float t = __fdividef(1.0f, fmaf(0.3275911f * kInvSqrt2, fabsf(x), 1.0f));
  float p = fmaf(1.061405429f, t, -1.453152027f);
  p = fmaf(p, t, 1.421413741f);
  p = fmaf(p, t, -0.284496736f);
  p = fmaf(p, t, 0.254829592f);
  const float tail = 0.5f * p * t * e;
  return x < 0.0f ? tail : 1.0f - tail;
}

// fp32 activations keep the library's error function
template <typename T, bool TANH>
__device__ __forceinline__ float gelu(float x) {
  if (TANH) return x * sigmoid_2u(x);
  if (sizeof(T) == 2) return x * normal_cdf(x, __expf(-0.5f * x * x));
  return 0.5f * x * (1.0f + erff(x * kInvSqrt2));
}

template <typename T, bool TANH>
__device__ __forceinline__ float gelu_slope(float x) {
  if (TANH) {
    const float s = sigmoid_2u(x);
    const float du = kSqrt2OverPi * fmaf(3.0f * kCubic * x, x, 1.0f);
    return fmaf(2.0f * x * du, s * (1.0f - s), s);
  }
  const float e = __expf(-0.5f * x * x);
  if (sizeof(T) == 2) return fmaf(x * kInvSqrt2Pi, e, normal_cdf(x, e));
  return fmaf(x * kInvSqrt2Pi, e, 0.5f * (1.0f + erff(x * kInvSqrt2)));
}

// A thread keeps its eight columns (and their bias) and walks down the rows, a few of them at a time with all their loads
// in flight before the arithmetic (with one row at a time the kernels waited for memory: 0.57 - 0.71 of the copy rate).
constexpr int kActWarps = 8, kTileCols = 256;
template <typename T>
constexpr int rows_ahead() { return sizeof(T) == 2 ? 4 : 2; }

template <typename T, bool TANH>
__global__ void __launch_bounds__(kActWarps * 32, 5) gelu_fwd_kernel(const T* __restrict__ pre, const float* __restrict__ bias,
                                                                     T* __restrict__ act, int rows, int cols,
                                                                     int rows_per_split) {
  constexpr int N = rows_ahead<T>();
  const int c = blockIdx.x * kTileCols + (threadIdx.x & 31) * 8;
  if (c >= cols) return;
  float bb[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (bias != nullptr) Vec8<float>::load(bias + c, bb);
  const int r0 = blockIdx.y * rows_per_split, r1 = min(rows, r0 + rows_per_split);
  for (int r = r0 + (threadIdx.x >> 5); r < r1; r += N * kActWarps) {
    Raw8<T> raw[N];
#pragma unroll
    for (int u = 0; u < N; ++u)
      if (r + u * kActWarps < r1) raw[u].load(pre + static_cast<size_t>(r + u * kActWarps) * cols + c);
#pragma unroll
    for (int u = 0; u < N; ++u) {
      if (r + u * kActWarps < r1) {
        float v[8];
        raw[u].get(v);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = gelu<T, TANH>(v[k] + bb[k]);
        Vec8<T>::store(act + static_cast<size_t>(r + u * kActWarps) * cols + c, v);
      }
    }
  }
}

// dpre = dact * gelu'(pre + bias); part[split][cols] = column sums of dpre over the split's rows
template <typename T, bool TANH>
__global__ void __launch_bounds__(kActWarps * 32, 3) gelu_bwd_kernel(const T* __restrict__ dact, const T* __restrict__ pre,
                                                                     const float* __restrict__ bias, T* __restrict__ dpre,
                                                                     float* __restrict__ part, int rows, int cols,
                                                                     int rows_per_split) {
  constexpr int N = rows_ahead<T>();
  __shared__ float sm[kActWarps][kTileCols];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * kTileCols + lane * 8;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (c < cols) {
    float bb[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (bias != nullptr) Vec8<float>::load(bias + c, bb);
    const int r0 = blockIdx.y * rows_per_split, r1 = min(rows, r0 + rows_per_split);
    for (int r = r0 + warp; r < r1; r += N * kActWarps) {
      Raw8<T> rv[N], rd[N];
#pragma unroll
      for (int u = 0; u < N; ++u) {
        if (r + u * kActWarps < r1) {
          const size_t at = static_cast<size_t>(r + u * kActWarps) * cols + c;
          rv[u].load(pre + at);
          rd[u].load(dact + at);
        }
      }
#pragma unroll
      for (int u = 0; u < N; ++u) {
        if (r + u * kActWarps < r1) {
          float v[8], d[8];
          rv[u].get(v);
          rd[u].get(d);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            d[k] *= gelu_slope<T, TANH>(v[k] + bb[k]);
            acc[k] += d[k];
          }
          Vec8<T>::store(dpre + static_cast<size_t>(r + u * kActWarps) * cols + c, d);
        }
      }
    }
  }
  if (part == nullptr) return;
  Vec8<float>::store(&sm[warp][lane * 8], acc);
  __syncthreads();
  const int col = blockIdx.x * kTileCols + threadIdx.x;
  if (col < cols) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kActWarps; ++w) s += sm[w][threadIdx.x];
    part[static_cast<size_t>(blockIdx.y) * cols + col] = s;
  }
}

// rows are split so that about `per_sm` CTAs per SM exist, each with at least 16 rows
void split_rows(int rows, int tiles, int per_sm, int& splits, int& rows_per_split) {
  const int want = std::max(1, device_sms() * per_sm / tiles);
  splits = std::max(1, std::min(want, (rows + 15) / 16));
  rows_per_split = (rows + splits - 1) / splits;
  splits = (rows + rows_per_split - 1) / rows_per_split;
}

void check_act(const at::Tensor& t, const c10::optional<at::Tensor>& bias) {
  TORCH_CHECK(t.is_cuda() && t.is_contiguous() && t.dim() >= 1 && t.size(-1) % 8 == 0 &&
                  (t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kFloat) &&
                  reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0,
              "gelu: contiguous 16-byte aligned bf16 or fp32 CUDA tensor whose last dimension is a multiple of 8");
  TORCH_CHECK(!bias.has_value() || (bias->is_cuda() && bias->scalar_type() == at::kFloat && bias->is_contiguous() &&
                                    bias->numel() == t.size(-1)), "gelu: fp32 bias of the last dimension's size");
}

}  // namespace

at::Tensor gelu_fwd(at::Tensor pre, c10::optional<at::Tensor> bias, bool tanh_form) {
  check_act(pre, bias);
  c10::cuda::CUDAGuard guard(pre.device());
  at::Tensor act = at::empty_like(pre);
  if (pre.numel() == 0) return act;
  const int cols = static_cast<int>(pre.size(-1)), rows = static_cast<int>(pre.numel() / cols);
  const int tiles = (cols + kTileCols - 1) / kTileCols;
  int splits, per;
  split_rows(rows, tiles, 5, splits, per);
  const float* bp = bias.has_value() ? bias->data_ptr<float>() : nullptr;
  auto stream = at::cuda::getCurrentCUDAStream();
#define DQ_CALL(T, TANH)                                                                                       \
  gelu_fwd_kernel<T, TANH><<<dim3(tiles, splits), kActWarps * 32, 0, stream>>>(                                \
      reinterpret_cast<const T*>(pre.data_ptr()), bp, reinterpret_cast<T*>(act.data_ptr()), rows, cols, per)
  if (pre.scalar_type() == at::kBFloat16) {
    if (tanh_form) DQ_CALL(__nv_bfloat16, true); else DQ_CALL(__nv_bfloat16, false);
  } else {
    if (tanh_form) DQ_CALL(float, true); else DQ_CALL(float, false);
  }
#undef DQ_CALL
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return act;
}

// (dpre, dbias); dbias is empty without a bias, and written to dbias_out when that is given
std::tuple<at::Tensor, at::Tensor> gelu_bwd(at::Tensor dact, at::Tensor pre, c10::optional<at::Tensor> bias, bool tanh_form,
                                            c10::optional<at::Tensor> dbias_out) {
  check_act(pre, bias);
  check_act(dact, bias);
  TORCH_CHECK(dact.scalar_type() == pre.scalar_type() && dact.numel() == pre.numel(), "gelu_bwd: gradient and input must agree");
  c10::cuda::CUDAGuard guard(pre.device());
  at::Tensor dpre = at::empty_like(pre);
  const int cols = static_cast<int>(pre.size(-1)), rows = static_cast<int>(pre.numel() / std::max(cols, 1));
  auto fopt = pre.options().dtype(at::kFloat);
  at::Tensor dbias = !bias.has_value() ? at::empty({0}, fopt) : (dbias_out.has_value() ? *dbias_out : at::empty({cols}, fopt));
  TORCH_CHECK(!bias.has_value() || (dbias.is_cuda() && dbias.scalar_type() == at::kFloat && dbias.is_contiguous() &&
                                    dbias.numel() == cols), "gelu_bwd: dbias must be a contiguous fp32 CUDA vector");
  if (pre.numel() == 0) return {dpre, dbias.zero_()};
  const int tiles = (cols + kTileCols - 1) / kTileCols;
  int splits, per;
  split_rows(rows, tiles, 3, splits, per);
  at::Tensor part = at::empty({bias.has_value() ? splits : 0, cols}, fopt);
  const float* bp = bias.has_value() ? bias->data_ptr<float>() : nullptr;
  float* pp = bias.has_value() ? part.data_ptr<float>() : nullptr;
  auto stream = at::cuda::getCurrentCUDAStream();
#define DQ_CALL(T, TANH)                                                                                         \
  gelu_bwd_kernel<T, TANH><<<dim3(tiles, splits), kActWarps * 32, 0, stream>>>(                                  \
      reinterpret_cast<const T*>(dact.data_ptr()), reinterpret_cast<const T*>(pre.data_ptr()), bp,               \
      reinterpret_cast<T*>(dpre.data_ptr()), pp, rows, cols, per)
  if (pre.scalar_type() == at::kBFloat16) {
    if (tanh_form) DQ_CALL(__nv_bfloat16, true); else DQ_CALL(__nv_bfloat16, false);
  } else {
    if (tanh_form) DQ_CALL(float, true); else DQ_CALL(float, false);
  }
#undef DQ_CALL
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  if (bias.has_value()) {
    reduce_arrays(pp, dbias.data_ptr<float>(), nullptr, nullptr, 1, splits, cols, stream);
    C10_CUDA_KERNEL_LAUNCH_CHECK();
  }
  return {dpre, dbias};
}

}  // namespace dq
