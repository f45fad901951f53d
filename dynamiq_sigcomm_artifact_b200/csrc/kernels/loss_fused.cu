// Softmax cross-entropy and its gradient in one pass over bf16 logits that nobody else reads.
//
// The forward kernel of loss_ops.cu reads the [N, Vp] logits, its backward kernel reads them again and writes the
// gradient over them: three transfers of 0.8 GB for 8192 x 50304 (231 + 316 us).  Where the logits belong to the loss
// (a model's own head), the gradient for an incoming gradient of 1 can be written as soon as a row's log-sum-exp is
// known, while the row is still in shared memory: two transfers.
//
// A cluster of C CTAs owns a row, each CTA a slice of it in shared memory, brought and taken away by bulk (TMA) copies;
// C is the smallest power of two for which two CTAs fit an SM, so that one CTA's copies, reductions and barriers run
// beside another's exponentials.  C = 1 up to 56 000 columns, 4 for 128 256; the CTAs of a cluster exchange their
// (max, sum) through distributed shared memory.  Bound by the exponentials (two per logit at 16 per clock and SM) next
// to memory, so everything else works on packed pairs: bf16 maxima, fp32x2 multiply-adds, 1 / n folded into the exponent.
//
// With `colsum` every thread keeps the gradient's sums over the rows for its own columns in registers - the gradient
// of a bias on the logits - instead of a further pass over the matrix; that takes one CTA per SM, with two buffers.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <torch/extension.h>

#include "../common/tcgen05.cuh"
#include "column_sums.cuh"
#include "norm_kernels.cuh"

namespace dq {
at::Tensor colsum(at::Tensor x, c10::optional<at::Tensor> out);  // colsum.cu
namespace {

namespace cg = cooperative_groups;
using normk::Vec8;

constexpr float kLog2e = 1.44269504f;
constexpr int kSumVecs = 8;  // 8-column groups per thread of the variant with column sums

// labels (optionally shifted left by one inside every row of S: position t predicts t + 1, the last is ignored), and
// how many are not `ignore`
__global__ void __launch_bounds__(1024) ce_labels_kernel(const long long* __restrict__ labels, long long* __restrict__ out,
                                                         float* __restrict__ n_valid, long long n, long long S, int shift,
                                                         long long ignore) {
  __shared__ int sm[32];
  int count = 0;
  for (long long i = threadIdx.x; i < n; i += 1024) {
    const long long v = shift ? ((i + 1) % S == 0 ? ignore : labels[i + 1]) : labels[i];
    out[i] = v;
    count += v != ignore;
  }
  count = __reduce_add_sync(0xFFFFFFFFu, count);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = count;
  __syncthreads();
  if (threadIdx.x < 32) {
    count = __reduce_add_sync(0xFFFFFFFFu, sm[threadIdx.x]);
    if (threadIdx.x == 0) *n_valid = fmaxf(static_cast<float>(count), 1.0f);
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

__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(tc::smem_u32(src)), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

__device__ __forceinline__ float2 bf16_pair(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}

// slice: columns per CTA (a multiple of 8); grid = clusters x C.  COLSUM: two buffers, else one.
constexpr int kCeThreads = 512;
template <bool COLSUM>
__global__ void __launch_bounds__(kCeThreads, COLSUM ? 1 : 2) ce_fused_kernel(
    __nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels, const float* __restrict__ n_valid,
    float* __restrict__ loss_rows, float* __restrict__ part, long long rows, int vocab, int stride, int slice,
    long long ignore) {
  constexpr int NBUF = COLSUM ? 2 : 1;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ float red_m[32], red_s[32], peer_m[2][8], peer_s[2][8];
  __shared__ uint64_t bars[2];
  cg::cluster_group cluster = cg::this_cluster();
  const int C = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lo = rank * slice, n = max(0, min(slice, stride - lo)), nvec = n / 8;  // this CTA's columns [lo, lo + n)
  const int nfull = max(0, min(nvec, (vocab - lo) / 8));                           // groups without padding columns
  const uint32_t bytes = static_cast<uint32_t>(n) * 2;
  if (tid == 0) {
    tc::mbar_init(&bars[0], 1);
    tc::mbar_init(&bars[1], 1);
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  const float scale = 1.0f / *n_valid, log2_scale = log2f(scale);
  const float2 l2e = make_float2(kLog2e, kLog2e);
  float acc[COLSUM ? kSumVecs : 1][8];
  if (COLSUM) {
#pragma unroll
    for (int j = 0; j < kSumVecs; ++j)
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[j][k] = 0.f;
  }
  const long long first = blockIdx.x / C, step = gridDim.x / C;
  if (COLSUM && tid == 0 && bytes > 0 && first < rows) tc::bulk_load(smem, logits + first * stride + lo, bytes, &bars[0]);
  uint32_t parity[2] = {0, 0};
  int turn = 0;
  for (long long row = first; row < rows; row += step, turn ^= 1) {
    const int cur = NBUF == 2 ? turn : 0;
    const long long fetch = NBUF == 2 ? row + step : row;  // two buffers: one row ahead
    const int into = NBUF == 2 ? turn ^ 1 : 0;
    if (tid == 0 && bytes > 0 && fetch < rows) {
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the buffer's previous row has left
      tc::bulk_load(smem + into * 2ll * slice, logits + fetch * stride + lo, bytes, &bars[into]);
    }
    const long long label = labels[row];
    const bool ignored = label == ignore;
    uint4* x = reinterpret_cast<uint4*>(smem + cur * 2ll * slice);
    const bool late = bytes > 0 && !tc::mbar_wait(&bars[cur], parity[cur]);
    if (__syncthreads_or(late)) {  // never landed within the limit: read it directly
      for (int i = tid; i < nvec; i += kCeThreads) x[i] = reinterpret_cast<const uint4*>(logits + row * stride + lo)[i];
      __syncthreads();
    }
    parity[cur] ^= 1u;
    float m = -INFINITY, s = 0.f;
    if (!ignored) {
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
      for (int i = tid; i < nfull; i += kCeThreads) add(x[i]);
      if (nfull < nvec && tid == 0) {  // the group that the padding starts in: padding as -inf
        uint4 q = x[nfull];
        uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (lo + 8 * nfull + k >= vocab)
            w[k >> 1] = (k & 1) ? ((w[k >> 1] & 0xFFFFu) | 0xFF800000u) : ((w[k >> 1] & 0xFFFF0000u) | 0xFF80u);
        add(make_uint4(w[0], w[1], w[2], w[3]));
      }
      s = s2.x + s2.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float m2 = __shfl_xor_sync(0xFFFFFFFFu, m, o), t2 = __shfl_xor_sync(0xFFFFFFFFu, s, o);
      merge(m, s, m2, t2);
    }
    if (lane == 0) red_m[warp] = m, red_s[warp] = s;
    __syncthreads();
    m = lane < kCeThreads / 32 ? red_m[lane] : -INFINITY;
    s = lane < kCeThreads / 32 ? red_s[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float m2 = __shfl_xor_sync(0xFFFFFFFFu, m, o), t2 = __shfl_xor_sync(0xFFFFFFFFu, s, o);
      merge(m, s, m2, t2);
    }
    if (C > 1) {  // every CTA tells every other; the slots alternate, so one barrier per row is enough
      if (tid < C) {
        *cluster.map_shared_rank(&peer_m[turn][rank], tid) = m;
        *cluster.map_shared_rank(&peer_s[turn][rank], tid) = s;
      }
      cluster.sync();
      m = -INFINITY, s = 0.f;
      for (int q = 0; q < C; ++q) merge(m, s, peer_m[turn][q], peer_s[turn][q]);
    }
    const float lse = m + logf(s);
    const float neg = log2_scale - lse * kLog2e;  // p / n = 2^(x log2 e + neg)
    const float2 off = make_float2(neg, neg);
    const int label_vec = !ignored && label >= lo && label < lo + n ? static_cast<int>(label - lo) / 8 : -1;
    if (tid == 0 && rank == 0 && (ignored || label < 0 || label >= stride)) loss_rows[row] = ignored ? 0.f : NAN;
    auto grad = [&](int i, float (&v)[8]) {
      const uint4 q = x[i];
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 t = __ffma2_rn(bf16_pair(w[j]), l2e, off);
        v[2 * j] = ex2(t.x), v[2 * j + 1] = ex2(t.y);
      }
      if (i >= nfull) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (lo + 8 * i + k >= vocab) v[k] = 0.f;
      }
      if (i == label_vec) {
        const int at = static_cast<int>(label - lo) & 7;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (k == at) {
            loss_rows[row] = lse - __uint_as_float((k & 1) ? (w[k >> 1] & 0xFFFF0000u) : (w[k >> 1] << 16));
            v[k] -= scale;
          }
        }
      }
      if (ignored) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = 0.f;
      }
      Vec8<__nv_bfloat16>::store(reinterpret_cast<__nv_bfloat16*>(x + i), v);
    };
    if (COLSUM) {
#pragma unroll
      for (int j = 0; j < kSumVecs; ++j) {
        const int i = tid + j * kCeThreads;
        if (i < nvec) {
          float v[8];
          grad(i, v);
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[j][k] += v[k];
        }
      }
    } else {
      for (int i = tid; i < nvec; i += kCeThreads) {
        float v[8];
        grad(i, v);
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0 && bytes > 0) bulk_store(logits + row * stride + lo, x, bytes);
  }
  if (COLSUM) {
#pragma unroll
    for (int j = 0; j < kSumVecs; ++j) {
      const int i = tid + j * kCeThreads;
      if (i < nvec) Vec8<float>::store(part + static_cast<size_t>(blockIdx.x) * stride + lo + 8 * i, acc[j]);
    }
  }
  if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  if (C > 1) cluster.sync();  // nobody leaves while a peer may still write its slots
}

constexpr int kCeSmem = 111 * 1024;  // a slice: two CTAs per SM

int cluster_size(long long stride, int& slice) {
  for (int c = 1; c <= 8; c *= 2) {
    slice = static_cast<int>(((stride + c - 1) / c + 7) / 8 * 8);
    if (2ll * slice <= kCeSmem) return c;
  }
  return 0;
}

template <bool COLSUM>
int launch_fused(const at::Tensor& logits, const at::Tensor& labels, const at::Tensor& n_valid, at::Tensor& rows_out,
                 at::Tensor& part, int64_t vocab, int64_t ignore, cudaStream_t stream) {
  const long long N = logits.size(0), stride = logits.size(1);
  int slice = 0;
  const int C = cluster_size(stride, slice);
  auto* fn = &ce_fused_kernel<COLSUM>;
  C10_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (COLSUM ? 2 : 1) * kCeSmem));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr, cfg.numAttrs = 1;
  cfg.blockDim = dim3(kCeThreads);
  cfg.dynamicSmemBytes = (COLSUM ? 4ull : 2ull) * slice;
  cfg.stream = stream;
  cfg.gridDim = dim3(C);
  int clusters = 0;
  C10_CUDA_CHECK(cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg));
  clusters = static_cast<int>(std::max<long long>(1, std::min<long long>(N, clusters)));
  cfg.gridDim = dim3(clusters * C);
  if (COLSUM) part = at::empty({clusters, stride}, logits.options().dtype(at::kFloat));
  C10_CUDA_CHECK(cudaLaunchKernelEx(&cfg, fn, reinterpret_cast<__nv_bfloat16*>(logits.data_ptr()),
                                    reinterpret_cast<const long long*>(labels.data_ptr<int64_t>()),
                                    const_cast<const float*>(n_valid.data_ptr<float>()), rows_out.data_ptr<float>(),
                                    COLSUM ? part.data_ptr<float>() : nullptr, N, static_cast<int>(vocab),
                                    static_cast<int>(stride), slice, static_cast<long long>(ignore)));
  return clusters;
}

}  // namespace

// whether ce_fused takes logits of this width
bool ce_fused_fits(int64_t stride) {
  int slice = 0;
  return stride > 0 && stride % 8 == 0 && stride < (1 << 30) && cluster_size(stride, slice) > 0;
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
  at::Tensor used = at::empty({N}, labels.options()), n_valid = at::empty({1}, fopt), rows = at::empty({N}, fopt);
  at::Tensor loss = at::empty({}, fopt), sums = at::empty({want_colsum ? stride : 0}, fopt), part;
  if (N == 0) return {loss.zero_(), sums.zero_()};
  auto stream = at::cuda::getCurrentCUDAStream();
  ce_labels_kernel<<<1, 1024, 0, stream>>>(reinterpret_cast<const long long*>(labels.data_ptr<int64_t>()),
                                           reinterpret_cast<long long*>(used.data_ptr<int64_t>()), n_valid.data_ptr<float>(), N,
                                           shift ? labels.size(1) : 1, shift ? 1 : 0, ignore_index);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  int slice = 0;
  const int C = cluster_size(stride, slice);
  const bool in_pass = want_colsum && C == 1 && slice <= kCeThreads * 8 * kSumVecs;
  int parts = 0;
  if (in_pass) parts = launch_fused<true>(logits, used, n_valid, rows, part, vocab, ignore_index, stream);
  else launch_fused<false>(logits, used, n_valid, rows, part, vocab, ignore_index, stream);
  ce_mean_kernel<<<1, 1024, 0, stream>>>(rows.data_ptr<float>(), n_valid.data_ptr<float>(), loss.data_ptr<float>(), N);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  if (in_pass) {
    reduce_arrays(part.data_ptr<float>(), sums.data_ptr<float>(), nullptr, nullptr, 1, parts, static_cast<int>(stride), stream);
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
