// Input embedding: x = bf16(token row + position row [+ type row 0]), and its backward.
//
// Forward was two gathers, one or two broadcast additions in fp32 and a cast; backward two casts of the gradient to
// fp32, a sort-free scatter for the positions, an indexed addition for the tokens and the sums for the type row (GPT-2
// small, 8 x 1024 tokens: 47 us forward, 120 us backward).  Here each way is one pass over the [B, S, H] tensor.
// Backward: a thread owns eight columns of one position and walks over the batch, so the position's gradient needs no
// atomics; the token rows go out as 16-byte vector reductions to L2 (order not fixed, as with any scatter-add).
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "column_sums.cuh"
#include "norm_kernels.cuh"

namespace dq {
namespace {

using normk::Vec8;

__global__ void __launch_bounds__(256) embed_fwd_kernel(const long long* __restrict__ ids, const __nv_bfloat16* __restrict__ tok,
                                                        const float* __restrict__ pos, const float* __restrict__ typ,
                                                        __nv_bfloat16* __restrict__ x, unsigned total, int S, int H,
                                                        long long vocab_rows) {
  const unsigned groups = H / 8;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned row = i / groups, c = (i - row * groups) * 8;
    const long long id = ids[row];
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, p[8];
    if (id >= 0 && id < vocab_rows) Vec8<__nv_bfloat16>::load(tok + id * H + c, v);
    if (pos != nullptr) {
      Vec8<float>::load(pos + static_cast<size_t>(row % S) * H + c, p);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += p[k];
    }
    if (typ != nullptr) {
      Vec8<float>::load(typ + c, p);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += p[k];
    }
    Vec8<__nv_bfloat16>::store(x + static_cast<size_t>(row) * H + c, v);
  }
}

__device__ __forceinline__ void red_add4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// positions S .. pos_rows - 1 get zeros; chunk: batch entries per thread (gridDim.y chunks; > 1 only without positions)
__global__ void __launch_bounds__(256) embed_bwd_kernel(const __nv_bfloat16* __restrict__ dx, const long long* __restrict__ ids,
                                                        float* __restrict__ tok_grad, float* __restrict__ pos_grad, int B, int S,
                                                        int H, long long vocab_rows, int pos_rows, int chunk) {
  const unsigned groups = H / 8, i = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned s = i / groups, c = (i - s * groups) * 8;
  if (s >= static_cast<unsigned>(max(S, pos_rows))) return;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (s < static_cast<unsigned>(S)) {
    const int b0 = blockIdx.y * chunk, b1 = min(B, b0 + chunk);
    for (int b = b0; b < b1; ++b) {
      const size_t row = static_cast<size_t>(b) * S + s;
      float d[8];
      Vec8<__nv_bfloat16>::load(dx + row * H + c, d);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += d[k];
      const long long id = ids[row];
      if (tok_grad != nullptr && id >= 0 && id < vocab_rows) {
        float* g = tok_grad + id * H + c;
        red_add4(g, d[0], d[1], d[2], d[3]);
        red_add4(g + 4, d[4], d[5], d[6], d[7]);
      }
    }
  }
  if (pos_grad != nullptr) Vec8<float>::store(pos_grad + static_cast<size_t>(s) * H + c, acc);
}

void check_vector(const at::Tensor& t, int64_t H, const char* what) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous() && t.size(-1) == H &&
                  reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0, "embedding: ", what, " must be fp32 rows of the hidden size");
}

}  // namespace

// ids [B, S] int64; tok [V, H] bf16; pos [>= S, H] fp32; typ [types, H] fp32 (row 0).  Rows of ids outside the table
// come out as position and type alone.
at::Tensor embed_fwd(at::Tensor ids, at::Tensor tok, c10::optional<at::Tensor> pos, c10::optional<at::Tensor> typ) {
  TORCH_CHECK(ids.is_cuda() && ids.scalar_type() == at::kLong && ids.dim() == 2 && ids.is_contiguous(), "embedding: ids must be int64 [B, S]");
  TORCH_CHECK(tok.is_cuda() && tok.scalar_type() == at::kBFloat16 && tok.dim() == 2 && tok.is_contiguous() && tok.size(1) % 8 == 0 &&
                  reinterpret_cast<uintptr_t>(tok.data_ptr()) % 16 == 0, "embedding: bf16 table, row length a multiple of 8");
  const int64_t B = ids.size(0), S = ids.size(1), H = tok.size(1);
  if (pos.has_value()) {
    check_vector(*pos, H, "positions");
    TORCH_CHECK(pos->size(0) >= S, "embedding: sequence longer than the position table");
  }
  if (typ.has_value()) check_vector(*typ, H, "types");
  c10::cuda::CUDAGuard guard(ids.device());
  at::Tensor x = at::empty({B, S, H}, tok.options());
  const long long total = B * S * (H / 8);
  TORCH_CHECK(total < (1ll << 31), "embedding: too large");
  if (total == 0) return x;
  embed_fwd_kernel<<<static_cast<int>(std::min<long long>((total + 255) / 256, device_sms() * 16LL)), 256, 0,
                     at::cuda::getCurrentCUDAStream()>>>(
      reinterpret_cast<const long long*>(ids.data_ptr<int64_t>()), reinterpret_cast<const __nv_bfloat16*>(tok.data_ptr()),
      pos.has_value() ? pos->data_ptr<float>() : nullptr, typ.has_value() ? typ->data_ptr<float>() : nullptr,
      reinterpret_cast<__nv_bfloat16*>(x.data_ptr()), static_cast<unsigned>(total), static_cast<int>(S), static_cast<int>(H),
      tok.size(0));
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return x;
}

// tok_grad [V, H] fp32 is added to (null: left out); pos_grad [P, H] fp32 is overwritten, rows past S with zeros
void embed_bwd(at::Tensor dx, at::Tensor ids, c10::optional<at::Tensor> tok_grad, c10::optional<at::Tensor> pos_grad) {
  TORCH_CHECK(dx.is_cuda() && dx.scalar_type() == at::kBFloat16 && dx.dim() == 3 && dx.is_contiguous() && dx.size(2) % 8 == 0 &&
                  reinterpret_cast<uintptr_t>(dx.data_ptr()) % 16 == 0, "embedding backward: bf16 [B, S, H]");
  TORCH_CHECK(ids.is_cuda() && ids.scalar_type() == at::kLong && ids.is_contiguous() && ids.numel() == dx.size(0) * dx.size(1),
              "embedding backward: ids must be int64 [B, S]");
  const int64_t B = dx.size(0), S = dx.size(1), H = dx.size(2);
  if (tok_grad.has_value()) check_vector(*tok_grad, H, "token gradients");
  if (pos_grad.has_value()) {
    check_vector(*pos_grad, H, "position gradients");
    TORCH_CHECK(pos_grad->size(0) >= S, "embedding backward: sequence longer than the position table");
  }
  c10::cuda::CUDAGuard guard(dx.device());
  const int pos_rows = pos_grad.has_value() ? static_cast<int>(pos_grad->size(0)) : 0;
  const long long total = std::max<long long>(S, pos_rows) * (H / 8);
  TORCH_CHECK(total < (1ll << 31), "embedding backward: too large");
  if (total == 0 || B == 0) return;
  // without positions nothing joins the batch entries (as many chunks as a grid takes)
  const int chunk = pos_grad.has_value() ? static_cast<int>(B) : static_cast<int>((B + 65534) / 65535);
  embed_bwd_kernel<<<dim3(static_cast<unsigned>((total + 255) / 256), static_cast<unsigned>((B + chunk - 1) / chunk)), 256, 0,
                     at::cuda::getCurrentCUDAStream()>>>(
      reinterpret_cast<const __nv_bfloat16*>(dx.data_ptr()), reinterpret_cast<const long long*>(ids.data_ptr<int64_t>()),
      tok_grad.has_value() ? tok_grad->data_ptr<float>() : nullptr, pos_grad.has_value() ? pos_grad->data_ptr<float>() : nullptr,
      static_cast<int>(B), static_cast<int>(S), static_cast<int>(H), tok_grad.has_value() ? tok_grad->size(0) : 0, pos_rows, chunk);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
}

}  // namespace dq
