// What surrounds the attention core in a block with one packed projection: qkv [rows, (heads + 2 kv) D].
//
//   rope_qkv_      rotary embedding of the q and k parts in place (the projection's output has no other reader)
//   qkv_grad_pack  dq, dk, dv as the attention backward leaves them -> the packed gradient, with the rotation
//                  undone on the way, or with the projection's bias gradient (column sums) taken on the way
//
// Instead of: a contiguous copy and a rotation of q and of k each way, a concatenation of the three gradients and a
// two-launch column sum (Llama shape, 8192 rows: 2 x 26 + 2 x 9 us forward; GPT-2 shape: 10.7 + 11.3 us backward).
// Bound by memory.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "column_sums.cuh"
#include "norm_kernels.cuh"

namespace dq {
namespace {

using normk::Raw8;
using normk::Vec8;

__device__ __forceinline__ void rotate8(float (&a)[8], float (&b)[8], const float (&c)[8], const float (&s)[8], float sign) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float sk = s[k] * sign, x = a[k], y = b[k];
    a[k] = x * c[k] - y * sk;
    b[k] = y * c[k] + x * sk;
  }
}

// one thread: eight values of the first half of a head and their partners D / 2 further on
template <typename T>
__global__ void __launch_bounds__(256) rope_qkv_kernel(T* __restrict__ qkv, const float* __restrict__ cs,
                                                       const float* __restrict__ sn, unsigned total, int S, int rot_heads,
                                                       int D, int width) {
  const unsigned half = D / 2, groups = half / 8, per_row = rot_heads * groups;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned row = i / per_row, rest = i - row * per_row, head = rest / groups, g = rest - head * groups;
    T* p = qkv + static_cast<size_t>(row) * width + head * D + g * 8;
    const size_t t = static_cast<size_t>(row % S) * half + g * 8;
    float a[8], b[8], c[8], s[8];
    Vec8<T>::load(p, a);
    Vec8<T>::load(p + half, b);
    Vec8<float>::load(cs + t, c);
    Vec8<float>::load(sn + t, s);
    rotate8(a, b, c, s, 1.0f);
    Vec8<T>::store(p, a);
    Vec8<T>::store(p + half, b);
  }
}

// gradients of one operand: [B, heads, S, D] with any strides over the first three dimensions, D contiguous
struct HeadsView {
  const void* p;
  long long sb, sh, ss;
};

template <typename T>
__global__ void __launch_bounds__(256) pack_rope_kernel(HeadsView q, HeadsView k, HeadsView v, const float* __restrict__ cs,
                                                        const float* __restrict__ sn, T* __restrict__ out, unsigned total,
                                                        int S, int nh, int nkv, int D) {
  const unsigned half = D / 2, groups = half / 8, heads = nh + 2 * nkv, per_row = heads * groups;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned row = i / per_row, rest = i - row * per_row, head = rest / groups, g = rest - head * groups;
    const unsigned bi = row / S, si = row - bi * S;
    const HeadsView& w = head < static_cast<unsigned>(nh) ? q : (head < static_cast<unsigned>(nh + nkv) ? k : v);
    const unsigned h = head < static_cast<unsigned>(nh) ? head : (head - nh) % nkv;
    const T* src = static_cast<const T*>(w.p) + bi * w.sb + h * w.sh + si * w.ss + g * 8;
    float a[8], b[8];
    Vec8<T>::load(src, a);
    Vec8<T>::load(src + half, b);
    if (head < static_cast<unsigned>(nh + nkv)) {
      float c[8], s[8];
      const size_t t = static_cast<size_t>(si) * half + g * 8;
      Vec8<float>::load(cs + t, c);
      Vec8<float>::load(sn + t, s);
      rotate8(a, b, c, s, -1.0f);  // the transposed rotation
    }
    T* dst = out + static_cast<size_t>(row) * heads * D + head * D + g * 8;
    Vec8<T>::store(dst, a);
    Vec8<T>::store(dst + half, b);
  }
}

constexpr int kPackWarps = 8, kPackCols = 256;

// a thread keeps its eight columns (one head's) and walks down the rows; part[split][cols]: column sums.  The key part of
// the bias gets exact zeros: a constant added to every key shifts all scores of a query alike, which the softmax does
// not see, so that gradient is zero and its column sums would be rounding noise (which an adaptive optimizer would
// scale up to full steps).
template <typename T>
__global__ void __launch_bounds__(kPackWarps * 32, 5) pack_colsum_kernel(HeadsView q, HeadsView k, HeadsView v,
                                                                         T* __restrict__ out, float* __restrict__ part,
                                                                         int rows, int S, int nh, int nkv, int D,
                                                                         int rows_per_split) {
  constexpr int N = sizeof(T) == 2 ? 4 : 2;  // rows whose loads are in flight together
  __shared__ float sm[kPackWarps][kPackCols];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cols = (nh + 2 * nkv) * D;
  const int c = blockIdx.x * kPackCols + lane * 8;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (c < cols) {
    const int head = c / D;
    const HeadsView& w = head < nh ? q : (head < nh + nkv ? k : v);
    const int h = head < nh ? head : (head - nh) % nkv;
    const bool is_key = head >= nh && head < nh + nkv;
    const T* src = static_cast<const T*>(w.p) + h * w.sh + (c - head * D);
    const int r0 = blockIdx.y * rows_per_split, r1 = min(rows, r0 + rows_per_split);
    for (int r = r0 + warp; r < r1; r += N * kPackWarps) {
      Raw8<T> raw[N];
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const int ru = r + u * kPackWarps, bi = ru / S, si = ru - bi * S;
        if (ru < r1) raw[u].load(src + bi * w.sb + si * w.ss);
      }
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const int ru = r + u * kPackWarps;
        if (ru < r1) {
          float d[8];
          raw[u].get(d);
          if (!is_key) {
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] += d[j];
          }
          Vec8<T>::store(out + static_cast<size_t>(ru) * cols + c, d);
        }
      }
    }
  }
  if (part == nullptr) return;
  Vec8<float>::store(&sm[warp][lane * 8], acc);
  __syncthreads();
  const int col = blockIdx.x * kPackCols + threadIdx.x;
  if (col < cols) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kPackWarps; ++w) s += sm[w][threadIdx.x];
    part[static_cast<size_t>(blockIdx.y) * cols + col] = s;
  }
}

void check_tables(const at::Tensor& cos, const at::Tensor& sin, int64_t S, int64_t D) {
  TORCH_CHECK(cos.is_cuda() && sin.is_cuda() && cos.scalar_type() == at::kFloat && sin.scalar_type() == at::kFloat &&
                  cos.is_contiguous() && sin.is_contiguous() && cos.size(0) >= S && cos.size(1) == D / 2 &&
                  sin.size(0) >= S && sin.size(1) == D / 2, "rope: cos/sin must be fp32 [S, D/2]");
}

HeadsView heads_view(const at::Tensor& t, int64_t B, int64_t heads, int64_t S, int64_t D, const at::Tensor& like) {
  TORCH_CHECK(t.is_cuda() && t.dim() == 4 && t.size(0) == B && t.size(1) == heads && t.size(2) == S && t.size(3) == D &&
                  t.stride(3) == 1 && t.scalar_type() == like.scalar_type() && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 &&
                  t.stride(2) % 8 == 0 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0,
              "qkv_grad_pack: [B, heads, S, D] gradients, D contiguous, 16-byte aligned rows");
  return HeadsView{t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)};
}

int elementwise_grid(long long total) {
  return static_cast<int>(std::min<long long>((total + 255) / 256, device_sms() * 16LL));
}

}  // namespace

// qkv [.., S, (nh + 2 nkv) D], in place
void rope_qkv_(at::Tensor qkv, at::Tensor cos, at::Tensor sin, int64_t nh, int64_t nkv, int64_t D) {
  TORCH_CHECK(qkv.is_cuda() && qkv.is_contiguous() && qkv.dim() >= 2 && qkv.size(-1) == (nh + 2 * nkv) * D && D % 16 == 0 &&
                  (qkv.scalar_type() == at::kBFloat16 || qkv.scalar_type() == at::kFloat) &&
                  reinterpret_cast<uintptr_t>(qkv.data_ptr()) % 16 == 0, "rope_qkv_: contiguous [.., S, (nh + 2 nkv) D]");
  const int S = static_cast<int>(qkv.size(-2));
  check_tables(cos, sin, S, D);
  const long long rows = qkv.numel() / qkv.size(-1), total = rows * (nh + nkv) * (D / 16);
  TORCH_CHECK(total < (1ll << 31), "rope_qkv_: too large");
  if (total == 0) return;
  c10::cuda::CUDAGuard guard(qkv.device());
  auto stream = at::cuda::getCurrentCUDAStream();
#define DQ_CALL(T)                                                                                               \
  rope_qkv_kernel<T><<<elementwise_grid(total), 256, 0, stream>>>(                                               \
      reinterpret_cast<T*>(qkv.data_ptr()), cos.data_ptr<float>(), sin.data_ptr<float>(), static_cast<unsigned>(total), S, \
      static_cast<int>(nh + nkv), static_cast<int>(D), static_cast<int>(qkv.size(-1)))
  if (qkv.scalar_type() == at::kBFloat16) DQ_CALL(__nv_bfloat16); else DQ_CALL(float);
#undef DQ_CALL
  C10_CUDA_KERNEL_LAUNCH_CHECK();
}

// dq [B, nh, S, D], dk / dv [B, nkv, S, D] -> (dqkv [B, S, (nh + 2 nkv) D], dbias); cos / sin: undo the rotation of dq and
// dk; want_bias: fp32 column sums of dqkv (into dbias_out when given), zeros for the key part.  One of the two.
std::tuple<at::Tensor, at::Tensor> qkv_grad_pack(at::Tensor dq, at::Tensor dk, at::Tensor dv, c10::optional<at::Tensor> cos,
                                                 c10::optional<at::Tensor> sin, bool want_bias,
                                                 c10::optional<at::Tensor> dbias_out) {
  TORCH_CHECK(dq.dim() == 4 && (dq.scalar_type() == at::kBFloat16 || dq.scalar_type() == at::kFloat), "qkv_grad_pack: bf16 or fp32 [B, heads, S, D]");
  const int64_t B = dq.size(0), nh = dq.size(1), S = dq.size(2), D = dq.size(3), nkv = dk.size(1);
  TORCH_CHECK(D % 8 == 0 && nkv >= 1, "qkv_grad_pack: head dimension must be a multiple of 8");
  const HeadsView q = heads_view(dq, B, nh, S, D, dq), k = heads_view(dk, B, nkv, S, D, dq), v = heads_view(dv, B, nkv, S, D, dq);
  TORCH_CHECK(!(cos.has_value() && want_bias), "qkv_grad_pack: a rotated projection has no bias");
  c10::cuda::CUDAGuard guard(dq.device());
  const int64_t cols = (nh + 2 * nkv) * D, rows = B * S;
  at::Tensor out = at::empty({B, S, cols}, dq.options());
  auto fopt = dq.options().dtype(at::kFloat);
  at::Tensor dbias = !want_bias ? at::empty({0}, fopt) : (dbias_out.has_value() ? *dbias_out : at::empty({cols}, fopt));
  TORCH_CHECK(!want_bias || (dbias.is_cuda() && dbias.scalar_type() == at::kFloat && dbias.is_contiguous() && dbias.numel() == cols),
              "qkv_grad_pack: dbias must be a contiguous fp32 CUDA vector");
  if (rows == 0) return {out, dbias.zero_()};
  auto stream = at::cuda::getCurrentCUDAStream();
  if (cos.has_value()) {
    TORCH_CHECK(sin.has_value() && D % 16 == 0, "qkv_grad_pack: cos and sin, head dimension a multiple of 16");
    check_tables(*cos, *sin, S, D);
    const long long total = rows * (nh + 2 * nkv) * (D / 16);
    TORCH_CHECK(total < (1ll << 31), "qkv_grad_pack: too large");
#define DQ_CALL(T)                                                                                                     \
  pack_rope_kernel<T><<<elementwise_grid(total), 256, 0, stream>>>(                                                    \
      q, k, v, cos->data_ptr<float>(), sin->data_ptr<float>(), reinterpret_cast<T*>(out.data_ptr()),                   \
      static_cast<unsigned>(total), static_cast<int>(S), static_cast<int>(nh), static_cast<int>(nkv), static_cast<int>(D))
    if (dq.scalar_type() == at::kBFloat16) DQ_CALL(__nv_bfloat16); else DQ_CALL(float);
#undef DQ_CALL
    C10_CUDA_KERNEL_LAUNCH_CHECK();
    return {out, dbias};
  }
  const int tiles = static_cast<int>((cols + kPackCols - 1) / kPackCols);
  int splits = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(device_sms() * 5 / tiles, (rows + 31) / 32)));
  const int per = static_cast<int>((rows + splits - 1) / splits);
  splits = static_cast<int>((rows + per - 1) / per);
  at::Tensor part = at::empty({want_bias ? splits : 0, cols}, fopt);
#define DQ_CALL(T)                                                                                                    \
  pack_colsum_kernel<T><<<dim3(tiles, splits), kPackWarps * 32, 0, stream>>>(                                         \
      q, k, v, reinterpret_cast<T*>(out.data_ptr()), want_bias ? part.data_ptr<float>() : nullptr, static_cast<int>(rows), \
      static_cast<int>(S), static_cast<int>(nh), static_cast<int>(nkv), static_cast<int>(D), per)
  if (dq.scalar_type() == at::kBFloat16) DQ_CALL(__nv_bfloat16); else DQ_CALL(float);
#undef DQ_CALL
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  if (want_bias) {
    reduce_arrays(part.data_ptr<float>(), dbias.data_ptr<float>(), nullptr, nullptr, 1, splits, static_cast<int>(cols), stream);
    C10_CUDA_KERNEL_LAUNCH_CHECK();
  }
  return {out, dbias};
}

}  // namespace dq
