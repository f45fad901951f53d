// LayerNorm / RMSNorm with the residual addition in front of it, forward and backward.
//
//   forward   s = x + (delta + bias),  y = norm(s) * w (+ b)
//   backward  dx = norm'(dy + dy2), or norm'(dy) + ds;  dw, db and - the bias of the linear layer that made `delta` -
//             dbias = sum over rows of dx
//
// A transformer block adds a sub-layer's output to the residual stream and normalises the sum; backward adds the
// stream's own gradient to the norm's and needs the column sums of the result for the sub-layer's bias.  As separate
// kernels these were an addition each way and a two-launch column sum per norm: 8192 x 768 bf16 took 8.9 + 6.4 us
// forward and 15.9 + 6.0 + 6.4 + 11.3 us backward; every value here is read and written once.
//
// A row stays in registers between the statistics and the result (H <= 2048), eight columns per thread: a warp per row
// up to 256 columns, a CTA of H / 8 threads per row above, so that enough rows are in flight per SM to cover the
// latency of memory (a warp holding a whole longer row ran at 0.56 - 0.61 of the copy rate).  Backward: norm_kernels.cuh;
// its partial column sums are added by a second launch in a fixed order, no atomics.  Bound by memory.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "column_sums.cuh"
#include "norm_kernels.cuh"

namespace dq {
namespace {

using namespace normk;

template <typename T>
__device__ __forceinline__ float as_stored(float v) { return to_f(from_f<T>(v)); }

// WARP: a warp per row, else a CTA per row; either way thread t of the row owns columns 8 t .. 8 t + 7
template <typename T, bool RMS, bool WARP>
__global__ void __launch_bounds__(256) add_norm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ delta,
                                                           const float* __restrict__ bias, const float* __restrict__ w,
                                                           const float* __restrict__ b, T* __restrict__ s_out, T* __restrict__ y,
                                                           float* __restrict__ mean, float* __restrict__ rstd, int rows, int H,
                                                           float eps) {
  __shared__ float red[2][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int row = WARP ? blockIdx.x * nwarps + warp : blockIdx.x, c = (WARP ? lane : threadIdx.x) * 8;
  if (row >= rows) return;  // whole warps (WARP) or never
  const bool on = c < H;
  const size_t at = static_cast<size_t>(row) * H + c;
  const float inv_h = 1.0f / static_cast<float>(H);
  auto row_sum = [&](float v, int slot) {
    v = warp_sum(v);
    if (!WARP) {
      if (lane == 0) red[slot][warp] = v;
      __syncthreads();
      v = 0.f;
      for (int i = 0; i < nwarps; ++i) v += red[slot][i];
    }
    return v;
  };
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, g[8], bb[8], sum = 0.f;
  if (on) {
    Raw8<T> rx, rd;
    rx.load(x + at);
    if (delta != nullptr) rd.load(delta + at);
    Vec8<float>::load(w + c, g);
    if (!RMS) Vec8<float>::load(b + c, bb);
    rx.get(v);
    if (delta != nullptr) {
      float d[8];
      rd.get(d);
      if (bias != nullptr) {
        float p[8];
        Vec8<float>::load(bias + c, p);
#pragma unroll
        for (int k = 0; k < 8; ++k) d[k] += p[k];
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = as_stored<T>(v[k] + d[k]);
      Vec8<T>::store(s_out + at, v);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) sum += RMS ? v[k] * v[k] : v[k];
  }
  sum = row_sum(sum, 0) * inv_h;
  const float mu = RMS ? 0.f : sum;
  float var = sum;
  if (!RMS) {
    var = 0.f;
    if (on) {
#pragma unroll
      for (int k = 0; k < 8; ++k) var += (v[k] - mu) * (v[k] - mu);
    }
    var = row_sum(var, 1) * inv_h;
  }
  const float rs = rsqrtf(var + eps);
  if (c == 0) {
    if (!RMS) mean[row] = mu;
    rstd[row] = rs;
  }
  if (on) {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = RMS ? v[k] * rs * g[k] : (v[k] - mu) * rs * g[k] + bb[k];
    Vec8<T>::store(y + at, v);
  }
}

// s = x + (delta + bias), rounded as the normalising kernel rounds it
template <typename T>
__global__ void __launch_bounds__(256) residual_add_kernel(const T* __restrict__ x, const T* __restrict__ delta,
                                                           const float* __restrict__ bias, T* __restrict__ s, unsigned groups,
                                                           unsigned row_groups) {
  for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < groups; i += gridDim.x * 256) {
    float v[8], d[8];
    Vec8<T>::load(x + 8ull * i, v);
    Vec8<T>::load(delta + 8ull * i, d);
    if (bias != nullptr) {
      float bb[8];
      Vec8<float>::load(bias + (i % row_groups) * 8, bb);
#pragma unroll
      for (int k = 0; k < 8; ++k) d[k] += bb[k];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] += d[k];
    Vec8<T>::store(s + 8ull * i, v);
  }
}

void check_rows(const at::Tensor& t, const at::Tensor& like, const char* what) {
  TORCH_CHECK(t.is_cuda() && t.is_contiguous() && t.scalar_type() == like.scalar_type() && t.numel() == like.numel(), "norm: ",
              what, " must match x");
  TORCH_CHECK(reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0, "norm: ", what, " must be 16-byte aligned");
}

template <typename T>
T* rows_of(const c10::optional<at::Tensor>& t) {
  return t.has_value() ? reinterpret_cast<T*>(t->data_ptr()) : nullptr;
}

// an fp32 vector of H elements: the given one or a new one
at::Tensor vector_out(const c10::optional<at::Tensor>& out, int H, const at::Tensor& like) {
  if (!out.has_value()) return at::empty({H}, like.options().dtype(at::kFloat));
  TORCH_CHECK(out->is_cuda() && out->scalar_type() == at::kFloat && out->is_contiguous() && out->numel() == H,
              "norm_bwd: an output gradient must be a contiguous CUDA fp32 tensor of H elements");
  return *out;
}

}  // namespace

bool norm_rows_fit(int64_t H) { return H % 8 == 0 && H <= 2048; }

// x, delta: [.., H] bf16 / fp32; bias: fp32 [H] added to delta.  Returns (s, y, mean, rstd); s is x without a delta,
// mean is empty for RMSNorm.
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> add_norm_fwd(at::Tensor x, c10::optional<at::Tensor> delta,
                                                                        c10::optional<at::Tensor> bias, at::Tensor w,
                                                                        c10::optional<at::Tensor> b, double eps, bool rms) {
  TORCH_CHECK(x.is_cuda() && x.is_contiguous(), "norm: x must be a contiguous CUDA tensor");
  TORCH_CHECK(x.scalar_type() == at::kBFloat16 || x.scalar_type() == at::kFloat, "norm: bf16 or fp32 activations");
  const int H = static_cast<int>(x.size(-1));
  TORCH_CHECK(norm_rows_fit(H), "add_norm: hidden size must be a multiple of 8, at most 2048");
  check_rows(x, x, "x");
  if (delta.has_value()) check_rows(*delta, x, "delta");
  auto vec = [&](const at::Tensor& t, const char* what) {
    TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous() && t.numel() == H, "norm: ", what,
                " must be a contiguous fp32 CUDA vector of the hidden size");
    return t.data_ptr<float>();
  };
  const float* wp = vec(w, "weight");
  TORCH_CHECK(rms || b.has_value(), "layernorm needs an fp32 bias");
  const float* bp = rms ? nullptr : vec(*b, "bias");
  const float* addp = bias.has_value() && delta.has_value() ? vec(*bias, "the added bias") : nullptr;
  c10::cuda::CUDAGuard guard(x.device());
  const int rows = static_cast<int>(x.numel() / H);
  auto fopt = x.options().dtype(at::kFloat);
  at::Tensor s = delta.has_value() ? at::empty_like(x) : x, y = at::empty_like(x);
  at::Tensor mean = at::empty({rms ? 0 : rows}, fopt), rstd = at::empty({rows}, fopt);
  if (rows == 0) return {s, y, mean, rstd};
  const bool warp = H <= 256;
  const int threads = warp ? kNormWarps * 32 : norm_group_threads(H), grid = warp ? (rows + kNormWarps - 1) / kNormWarps : rows;
  auto stream = at::cuda::getCurrentCUDAStream();
#define DQ_FWD(T, RMS, WARP)                                                                                            \
  add_norm_fwd_kernel<T, RMS, WARP><<<grid, threads, 0, stream>>>(                                                      \
      reinterpret_cast<const T*>(x.data_ptr()), rows_of<const T>(delta), addp, wp, bp, reinterpret_cast<T*>(s.data_ptr()), \
      reinterpret_cast<T*>(y.data_ptr()), rms ? nullptr : mean.data_ptr<float>(), rstd.data_ptr<float>(), rows, H,      \
      static_cast<float>(eps))
#define DQ_FWD_T(T)                                                                      \
  if (rms) { if (warp) DQ_FWD(T, true, true); else DQ_FWD(T, true, false); }             \
  else { if (warp) DQ_FWD(T, false, true); else DQ_FWD(T, false, false); }
  if (x.scalar_type() == at::kBFloat16) { DQ_FWD_T(__nv_bfloat16) } else { DQ_FWD_T(float) }
#undef DQ_FWD_T
#undef DQ_FWD
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return {s, y, mean, rstd};
}

// Returns (dx, dw, db, dbias); db is empty for RMSNorm, dbias unless `want_bias`.  dw_out / db_out / dbias_out: where
// the column sums go instead of new tensors.
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> add_norm_bwd(
    at::Tensor dy, c10::optional<at::Tensor> dy2, c10::optional<at::Tensor> ds, at::Tensor s, at::Tensor w, at::Tensor mean,
    at::Tensor rstd, bool rms, bool want_bias, c10::optional<at::Tensor> dw_out, c10::optional<at::Tensor> db_out,
    c10::optional<at::Tensor> dbias_out) {
  TORCH_CHECK(s.is_cuda() && s.is_contiguous() && (s.scalar_type() == at::kBFloat16 || s.scalar_type() == at::kFloat),
              "norm_bwd: contiguous bf16 or fp32 CUDA activations");
  const int H = static_cast<int>(s.size(-1));
  TORCH_CHECK(norm_rows_fit(H), "add_norm: hidden size must be a multiple of 8, at most 2048");
  check_rows(s, s, "s");
  check_rows(dy, s, "dy");
  if (dy2.has_value()) check_rows(*dy2, s, "dy2");
  if (ds.has_value()) check_rows(*ds, s, "ds");
  TORCH_CHECK(!(dy2.has_value() && ds.has_value()), "norm_bwd: a second gradient of y or one of s, not both");
  TORCH_CHECK(w.is_cuda() && w.scalar_type() == at::kFloat && w.is_contiguous() && w.numel() == H, "norm: fp32 weight");
  c10::cuda::CUDAGuard guard(s.device());
  const int rows = static_cast<int>(s.numel() / H);
  at::Tensor dx = at::empty_like(s);
  auto fopt = s.options().dtype(at::kFloat);
  at::Tensor dw = vector_out(dw_out, H, s);
  at::Tensor db = rms ? at::empty({0}, fopt) : vector_out(db_out, H, s);
  at::Tensor dbias = want_bias ? vector_out(dbias_out, H, s) : at::empty({0}, fopt);
  if (rows == 0) {
    dw.zero_(), db.zero_(), dbias.zero_();
    return {dx, dw, db, dbias};
  }
  const int arrays = 1 + (rms ? 0 : 1) + (want_bias ? 1 : 0);
  const int grid = norm_bwd_grid(rows, H, device_sms()), nt = norm_group_threads(H), threads = nt * norm_groups(H);
  at::Tensor part = at::empty({arrays, grid, H}, fopt);
  auto stream = at::cuda::getCurrentCUDAStream();
#define DQ_BWD(T, RMS, BIAS)                                                                                              \
  C10_CUDA_CHECK(cudaFuncSetAttribute(add_norm_bwd_kernel<T, RMS, BIAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kNormBwdMaxSmem)); \
  add_norm_bwd_kernel<T, RMS, BIAS><<<grid, threads, norm_bwd_smem(H), stream>>>(                                         \
      reinterpret_cast<const T*>(dy.data_ptr()), rows_of<const T>(dy2.has_value() ? dy2 : ds), dy2.has_value(),           \
      reinterpret_cast<const T*>(s.data_ptr()), w.data_ptr<float>(), rms ? nullptr : mean.data_ptr<float>(),              \
      rstd.data_ptr<float>(), reinterpret_cast<T*>(dx.data_ptr()), part.data_ptr<float>(), rows, H, nt)
#define DQ_BWD_T(T)                                                              \
  if (rms) { if (want_bias) { DQ_BWD(T, true, true); } else { DQ_BWD(T, true, false); } }  \
  else { if (want_bias) { DQ_BWD(T, false, true); } else { DQ_BWD(T, false, false); } }
  if (s.scalar_type() == at::kBFloat16) { DQ_BWD_T(__nv_bfloat16) } else { DQ_BWD_T(float) }
#undef DQ_BWD_T
#undef DQ_BWD
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  float* second = rms ? (want_bias ? dbias.data_ptr<float>() : nullptr) : db.data_ptr<float>();
  reduce_arrays(part.data_ptr<float>(), dw.data_ptr<float>(), second, want_bias ? dbias.data_ptr<float>() : nullptr, arrays,
                grid, H, stream);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return {dx, dw, db, dbias};
}

// x + (delta + bias) for a sub-layer whose sum is not normalised next
at::Tensor residual_add(at::Tensor x, at::Tensor delta, c10::optional<at::Tensor> bias) {
  TORCH_CHECK(x.is_cuda() && x.is_contiguous() && (x.scalar_type() == at::kBFloat16 || x.scalar_type() == at::kFloat) &&
                  x.size(-1) % 8 == 0, "residual_add: contiguous bf16 or fp32 CUDA tensor, last dimension a multiple of 8");
  check_rows(x, x, "x");
  check_rows(delta, x, "delta");
  TORCH_CHECK(!bias.has_value() || (bias->is_cuda() && bias->scalar_type() == at::kFloat && bias->is_contiguous() &&
                                    bias->numel() == x.size(-1)), "residual_add: fp32 bias of the last dimension's size");
  TORCH_CHECK(x.numel() / 8 < (1ll << 31), "residual_add: too large");
  c10::cuda::CUDAGuard guard(x.device());
  at::Tensor s = at::empty_like(x);
  const unsigned groups = static_cast<unsigned>(x.numel() / 8), row_groups = static_cast<unsigned>(x.size(-1) / 8);
  if (groups == 0) return s;
  const int grid = static_cast<int>(std::min<long long>((groups + 255) / 256, device_sms() * 16LL));
  const float* bp = bias.has_value() ? bias->data_ptr<float>() : nullptr;
  auto stream = at::cuda::getCurrentCUDAStream();
  if (x.scalar_type() == at::kBFloat16)
    residual_add_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(
        reinterpret_cast<const __nv_bfloat16*>(x.data_ptr()), reinterpret_cast<const __nv_bfloat16*>(delta.data_ptr()), bp,
        reinterpret_cast<__nv_bfloat16*>(s.data_ptr()), groups, row_groups);
  else
    residual_add_kernel<float><<<grid, 256, 0, stream>>>(x.data_ptr<float>(), delta.data_ptr<float>(), bp, s.data_ptr<float>(),
                                                         groups, row_groups);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return s;
}

}  // namespace dq
