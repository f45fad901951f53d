// Softmax cross-entropy and its gradient in one pass over bf16 logits that nobody else reads.
//
// The forward kernel of loss_ops.cu reads the [N, Vp] logits, its backward kernel reads them again and writes the
// gradient over them: three transfers of 0.8 GB for 8192 x 50304 (231 + 316 us).  Where the logits belong to the loss
// (a model's own head), the gradient for an incoming gradient of 1 can be written as soon as a row's log-sum-exp is
// known: a CTA walks over its row twice, and the second walk finds the row in L2 (two CTAs per SM hold 30 MB of rows
// 50 304 wide, 76 MB of rows 128 256 wide, of 126 MB).  Rows staged in shared memory by bulk copies, in clusters where a
// row does not fit, were slower (359 us; 1.42 ms at 128 256): one row per CTA leaves loads, reductions and stores of a
// CTA behind one another.  Bound by memory next to the exponentials (two per logit at 16 per clock and SM), so everything
// else works on packed pairs: bf16 maxima, fp32x2 multiply-adds, 1 / n folded into the exponent.
//
// Rows to be ignored are only cleared; the label kernel sorts them behind the others so that both kinds are spread
// evenly over the CTAs.  With `colsum` the gradient's sums over the rows - the gradient of a bias on the logits - are kept
// in shared memory, one thread per group of eight columns, instead of in a further pass over the matrix.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <cuda_bf16.h>
#include <torch/extension.h>

#include "column_sums.cuh"
#include "norm_kernels.cuh"

namespace dq {
at::Tensor colsum(at::Tensor x, c10::optional<at::Tensor> out);  // colsum.cu
namespace {

using normk::Vec8;

constexpr float kLog2e = 1.44269504f;

// labels (optionally shifted left by one inside every row of S: position t predicts t + 1, the last is ignored); the
// rows in the order of work: those with a label first, ascending; how many these are
__global__ void __launch_bounds__(1024) ce_labels_kernel(const long long* __restrict__ labels, long long* __restrict__ out,
                                                         int* __restrict__ order, float* __restrict__ n_valid, long long n,
                                                         long long S, int shift, long long ignore) {
  __shared__ int sm[32];
  __shared__ int total;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long per = (n + 1023) / 1024, i0 = tid * per, i1 = min(n, i0 + per);
  auto label = [&](long long i) { return shift ? ((i + 1) % S == 0 ? ignore : labels[i + 1]) : labels[i]; };
  int count = 0;
  for (long long i = i0; i < i1; ++i) {
    const long long v = label(i);
    out[i] = v;
    count += v != ignore;
  }
  int before = count;  // inclusive prefix sum over the threads
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xFFFFFFFFu, before, o);
    if (lane >= o) before += t;
  }
  if (lane == 31) sm[warp] = before;
  __syncthreads();
  if (warp == 0) {
    int t = sm[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xFFFFFFFFu, t, o);
      if (lane >= o) t += u;
    }
    sm[lane] = t;
    if (lane == 31) {
      total = t;
      *n_valid = fmaxf(static_cast<float>(t), 1.0f);
    }
  }
  __syncthreads();
  int at = before - count + (warp > 0 ? sm[warp - 1] : 0);
  long long rest = total + (i0 - at);  // the ignored rows before i0
  for (long long i = i0; i < i1; ++i) {
    if (out[i] != ignore) order[at++] = static_cast<int>(i);
    else order[rest++] = static_cast<int>(i);
  }
}

// loss = sum of the rows' losses / n_valid, in a fixed order
__global__ void __launch_bounds__(1024) ce_mean_kernel(const float* __restrict__ rows, const float* __restrict__ n_valid,
                                                       float* __restrict__ loss, long long n) {
  __shared__ float sm[32];
  float s = 0.f;
  for (long long i = threadIdx.x; i < n; i += 1024) s += rows[i];
  s = normk::warp_sum(s);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = normk::warp_sum(sm[threadIdx.x]);
    if (threadIdx.x == 0) *loss = s / *n_valid;
  }
}

// grad *= *g, nothing when *g is 1 (a loss that is the root of its graph)
__global__ void __launch_bounds__(256) ce_rescale_kernel(__nv_bfloat16* __restrict__ grad, const float* __restrict__ g,
                                                         long long groups) {
  const float f = *g;
  if (f == 1.0f) return;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < groups; i += gridDim.x * 256ll) {
    float v[8];
    Vec8<__nv_bfloat16>::load(grad + 8 * i, v);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] *= f;
    Vec8<__nv_bfloat16>::store(grad + 8 * i, v);
  }
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void merge(float& m, float& s, float m2, float s2) {
  const float mn = fmaxf(m, m2);
  if (mn == -INFINITY) {
    s = 0.f;
    return;
  }
  s = s * ex2((m - mn) * kLog2e) + s2 * ex2((m2 - mn) * kLog2e);
  m = mn;
}

__device__ __forceinline__ float2 bf16_pair(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}

constexpr int kAhead = 4;  // 16-byte loads of a thread that are in flight together

template <int THREADS, bool COLSUM>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) ce_fused_kernel(
    __nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels, const int* __restrict__ order,
    const float* __restrict__ n_valid, float* __restrict__ loss_rows, float* __restrict__ part, int rows, int vocab,
    int stride, long long ignore) {
  extern __shared__ float sums[];  // COLSUM: [stride]
  __shared__ float red_m[32], red_s[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nvec = stride / 8, nfull = vocab / 8;  // groups of eight columns; those without padding
  const float scale = 1.0f / *n_valid, log2_scale = log2f(scale);
  const float2 l2e = make_float2(kLog2e, kLog2e);
  if (COLSUM) {
    for (int i = tid; i < nvec; i += THREADS) {  // every thread clears, adds to and reads its own groups only
      const float zero[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      Vec8<float>::store(sums + 8 * i, zero);
    }
  }
  for (int k = blockIdx.x; k < rows; k += gridDim.x) {
    const int row = order[k];
    const long long label = labels[row];
    uint4* x = reinterpret_cast<uint4*>(logits + static_cast<long long>(row) * stride);
    if (label == ignore) {
      for (int i = tid; i < nvec; i += THREADS) __stcs(x + i, make_uint4(0u, 0u, 0u, 0u));
      if (tid == 0) loss_rows[row] = 0.f;
      continue;
    }
    float m = -INFINITY;
    float2 s2 = make_float2(0.f, 0.f);
    auto add = [&](const uint4& q) {
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(w);
      const __nv_bfloat162 mx = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
      const float lm = fmaxf(__low2float(mx), __high2float(mx));
      if (lm > m) {
        const float f = ex2((m - lm) * kLog2e);
        s2.x *= f, s2.y *= f;
        m = lm;
      }
      const float shift = m == -INFINITY ? 0.f : -m * kLog2e;
      const float2 off = make_float2(shift, shift);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 t = __ffma2_rn(bf16_pair(w[j]), l2e, off);
        s2 = __fadd2_rn(s2, make_float2(ex2(t.x), ex2(t.y)));
      }
    };
    for (int base = 0; base < nfull; base += kAhead * THREADS) {
      uint4 q[kAhead];
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {
        const int i = base + a * THREADS + tid;
        if (i < nfull) q[a] = __ldcg(x + i);
      }
#pragma unroll
      for (int a = 0; a < kAhead; ++a)
        if (base + a * THREADS + tid < nfull) add(q[a]);
    }
    if (nfull < nvec && tid == 0) {  // the group that the padding starts in: padding as -inf
      const uint4 q = __ldcg(x + nfull);
      uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (8 * nfull + j >= vocab) w[j >> 1] = (j & 1) ? ((w[j >> 1] & 0xFFFFu) | 0xFF800000u) : ((w[j >> 1] & 0xFFFF0000u) | 0xFF80u);
      add(make_uint4(w[0], w[1], w[2], w[3]));
    }
    float s = s2.x + s2.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float m2 = __shfl_xor_sync(0xFFFFFFFFu, m, o), t2 = __shfl_xor_sync(0xFFFFFFFFu, s, o);
      merge(m, s, m2, t2);
    }
    __syncthreads();  // the previous row's values have been read
    if (lane == 0) red_m[warp] = m, red_s[warp] = s;
    __syncthreads();
    m = lane < THREADS / 32 ? red_m[lane] : -INFINITY;
    s = lane < THREADS / 32 ? red_s[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float m2 = __shfl_xor_sync(0xFFFFFFFFu, m, o), t2 = __shfl_xor_sync(0xFFFFFFFFu, s, o);
      merge(m, s, m2, t2);
    }
    const float lse = m + logf(s);
    const float neg = log2_scale - lse * kLog2e;  // p / n = 2^(x log2 e + neg)
    const float2 off = make_float2(neg, neg);
    const int label_vec = label >= 0 && label < stride ? static_cast<int>(label / 8) : -1;
    if (tid == 0 && label_vec < 0) loss_rows[row] = NAN;
    for (int base = 0; base < nvec; base += kAhead * THREADS) {
      uint4 q[kAhead];
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {
        const int i = base + a * THREADS + tid;
        if (i < nvec) q[a] = __ldcg(x + i);
      }
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {
        const int i = base + a * THREADS + tid;
        if (i >= nvec) break;
        const uint32_t w[4] = {q[a].x, q[a].y, q[a].z, q[a].w};
        float v[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 t = __ffma2_rn(bf16_pair(w[j]), l2e, off);
          v[2 * j] = ex2(t.x), v[2 * j + 1] = ex2(t.y);
        }
        if (i >= nfull) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (8 * i + j >= vocab) v[j] = 0.f;
        }
        if (i == label_vec) {
          const int at = static_cast<int>(label) & 7;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (j == at) {
              loss_rows[row] = lse - __uint_as_float((j & 1) ? (w[j >> 1] & 0xFFFF0000u) : (w[j >> 1] << 16));
              v[j] -= scale;
            }
          }
        }
        if (COLSUM) {
          float o[8];
          Vec8<float>::load(sums + 8 * i, o);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += v[j];
          Vec8<float>::store(sums + 8 * i, o);
        }
        uint32_t out[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
          out[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        __stcs(x + i, make_uint4(out[0], out[1], out[2], out[3]));  // nothing reads it while rows are still wanted in L2
      }
    }
  }
  if (COLSUM) {
    for (int i = tid; i < nvec; i += THREADS) {
      float o[8];
      Vec8<float>::load(sums + 8 * i, o);
      Vec8<float>::store(part + static_cast<size_t>(blockIdx.x) * stride + 8 * i, o);
    }
  }
}

constexpr int kSumSmem = 220 * 1024;  // widest matrix whose column sums a CTA can hold: 56 320 columns

}  // namespace

// whether ce_fused takes logits of this width
bool ce_fused_fits(int64_t stride) {
  return stride > 0 && stride % 8 == 0 && stride < (1 << 30);
}

// logits [N, stride] bf16: overwritten with d loss / d logits; labels [N] or [B, S] int64, shifted by one position when
// `shift`.  Returns (mean loss [] fp32, colsum fp32 [stride] of the gradient or empty).
std::tuple<at::Tensor, at::Tensor> ce_fused(at::Tensor logits, at::Tensor labels, int64_t vocab, int64_t ignore_index, bool shift,
                                            bool want_colsum) {
  TORCH_CHECK(logits.is_cuda() && logits.dim() == 2 && logits.is_contiguous() && logits.scalar_type() == at::kBFloat16 &&
                  reinterpret_cast<uintptr_t>(logits.data_ptr()) % 16 == 0, "ce_fused: contiguous bf16 [N, Vp] logits");
  const int64_t N = logits.size(0), stride = logits.size(1);
  TORCH_CHECK(ce_fused_fits(stride) && vocab > 0 && vocab <= stride, "ce_fused: width must be a multiple of 8 and >= vocab");
  TORCH_CHECK(labels.is_cuda() && labels.scalar_type() == at::kLong && labels.is_contiguous() && labels.numel() == N &&
                  (!shift || labels.dim() == 2), "ce_fused: labels must be contiguous int64, [B, S] to be shifted");
  c10::cuda::CUDAGuard guard(logits.device());
  auto fopt = logits.options().dtype(at::kFloat);
  TORCH_CHECK(N < (1ll << 31), "ce_fused: too many rows");
  at::Tensor used = at::empty({N}, labels.options()), order = at::empty({N}, labels.options().dtype(at::kInt));
  at::Tensor n_valid = at::empty({1}, fopt), rows = at::empty({N}, fopt);
  at::Tensor loss = at::empty({}, fopt), sums = at::empty({want_colsum ? stride : 0}, fopt);
  if (N == 0) return {loss.zero_(), sums.zero_()};
  auto stream = at::cuda::getCurrentCUDAStream();
  ce_labels_kernel<<<1, 1024, 0, stream>>>(reinterpret_cast<const long long*>(labels.data_ptr<int64_t>()),
                                           reinterpret_cast<long long*>(used.data_ptr<int64_t>()), order.data_ptr<int>(),
                                           n_valid.data_ptr<float>(), N, shift ? labels.size(1) : 1, shift ? 1 : 0, ignore_index);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  const bool in_pass = want_colsum && stride * 4 <= kSumSmem;
  const int sms = device_sms(), per_sm = stride <= 65536 ? 4 : 2;
  // four small CTAs per SM overlap their phases better than two large ones, as long as their rows stay in L2 (78 MB)
  const int grid = static_cast<int>(std::min<int64_t>(N, in_pass ? sms : per_sm * sms));
  at::Tensor part = at::empty({in_pass ? grid : 0, stride}, fopt);
  auto* x = reinterpret_cast<__nv_bfloat16*>(logits.data_ptr());
  const auto* lab = reinterpret_cast<const long long*>(used.data_ptr<int64_t>());
  if (in_pass) {
    C10_CUDA_CHECK(cudaFuncSetAttribute(ce_fused_kernel<1024, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSumSmem));
    ce_fused_kernel<1024, true><<<grid, 1024, stride * 4, stream>>>(
        x, lab, order.data_ptr<int>(), n_valid.data_ptr<float>(), rows.data_ptr<float>(), part.data_ptr<float>(),
        static_cast<int>(N), static_cast<int>(vocab), static_cast<int>(stride), ignore_index);
  } else if (per_sm == 4) {
    ce_fused_kernel<256, false><<<grid, 256, 0, stream>>>(
        x, lab, order.data_ptr<int>(), n_valid.data_ptr<float>(), rows.data_ptr<float>(), nullptr, static_cast<int>(N),
        static_cast<int>(vocab), static_cast<int>(stride), ignore_index);
  } else {
    ce_fused_kernel<512, false><<<grid, 512, 0, stream>>>(
        x, lab, order.data_ptr<int>(), n_valid.data_ptr<float>(), rows.data_ptr<float>(), nullptr, static_cast<int>(N),
        static_cast<int>(vocab), static_cast<int>(stride), ignore_index);
  }
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  ce_mean_kernel<<<1, 1024, 0, stream>>>(rows.data_ptr<float>(), n_valid.data_ptr<float>(), loss.data_ptr<float>(), N);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  if (in_pass) {
    reduce_arrays(part.data_ptr<float>(), sums.data_ptr<float>(), nullptr, nullptr, 1, grid, static_cast<int>(stride), stream);
    C10_CUDA_KERNEL_LAUNCH_CHECK();
  } else if (want_colsum) {
    colsum(logits, sums);
  }
  return {loss, sums};
}

// grad (bf16, in place) *= g (one fp32 value on the device)
void ce_rescale_(at::Tensor grad, at::Tensor g) {
  TORCH_CHECK(grad.is_cuda() && grad.scalar_type() == at::kBFloat16 && grad.is_contiguous() && grad.numel() % 8 == 0 && g.is_cuda() &&
                  g.scalar_type() == at::kFloat && g.numel() == 1, "ce_rescale_: bf16 gradient and an fp32 scalar on the device");
  if (grad.numel() == 0) return;
  c10::cuda::CUDAGuard guard(grad.device());
  const long long groups = grad.numel() / 8;
  ce_rescale_kernel<<<static_cast<int>(std::min<long long>((groups + 255) / 256, device_sms() * 8LL)), 256, 0,
                      at::cuda::getCurrentCUDAStream()>>>(reinterpret_cast<__nv_bfloat16*>(grad.data_ptr()), g.data_ptr<float>(), groups);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
}

}  // namespace dq
