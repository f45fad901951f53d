// EDEN on the GPU: one kernel compresses and one decompresses, a warp per 1024-element block.
//
//   compress    rotate (H_1024, Rademacher signs), ||y||^2, nearest Lloyd-Max level of y / rms, scale
//               ||y||^2 / <y, c>, bit planes of the level indices
//   decompress  bit planes -> level x scale -> inverse rotation
//
// A lane holds 32 coefficients e = (lane & 3) + 4 k + 128 (lane >> 2), so a 32-bit plane word is spread over the four
// lanes that share lane >> 2, eight bits in each; they exchange partial words so that lane l ends with word l and a
// plane of the block is one coalesced store.  Bound by latency at a few MB and by instruction issue above (the level
// search is `bits` dependent shared-memory reads per value).  As a chain of tensor operators this took about 35
// launches, two host synchronisations and six host-to-device copies: 570 us for 2 M values.
//
// Reference counterpart: cuda_kernels/src/srrcomp/srrcomp.py:293-447, csrc/cuda_packing.cu:11-95.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "../common/rht_codec.cuh"
#include "dependent_launch.cuh"

namespace dq {
namespace {

constexpr int kEdenWarps = 8;

__device__ __forceinline__ float sum_of_warp(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFullMask, v, o);
  return v;
}

__device__ __forceinline__ void eden_signs(float* sgn, uint32_t* words, float c, uint32_t step, uint32_t seed_lo,
                                           uint32_t seed_hi) {
  if (threadIdx.x < 32) words[threadIdx.x] = sign_word(threadIdx.x, step, 0u, seed_lo, seed_hi);
  __syncthreads();
  for (int e = threadIdx.x; e < kBlock; e += kEdenWarps * 32) sgn[e] = ((words[e >> 5] >> (e & 31)) & 1u) ? -c : c;
  __syncthreads();
}

// x [n] -> words [BITS, 32 nblocks], scale [nblocks]; levels: 2^BITS centroids, then 2^BITS - 1 boundaries
template <int BITS>
__global__ void __launch_bounds__(kEdenWarps * 32, 2) eden_compress_kernel(
    const float* __restrict__ x, const float* __restrict__ levels, uint32_t* __restrict__ words, float* __restrict__ scale,
    long long n, int nblocks, uint32_t step, uint32_t seed_lo, uint32_t seed_hi) {
  constexpr int L = 1 << BITS;
  __shared__ __align__(16) float tiles[kEdenWarps][kBlock];
  __shared__ __align__(16) float sgn[kBlock];
  __shared__ uint32_t sign_words[32];
  __shared__ float cen[L], bnd[L];
  let_next_start();
  wait_for_previous();
  for (int i = threadIdx.x; i < L; i += kEdenWarps * 32) {
    cen[i] = levels[i];
    bnd[i] = i < L - 1 ? levels[L + i] : INFINITY;
  }
  eden_signs(sgn, sign_words, 1.0f / 32.0f, step, seed_lo, seed_hi);  // also orders the level tables
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool vec_ok = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  const size_t plane = static_cast<size_t>(nblocks) * 32;
  for (int blk = blockIdx.x * kEdenWarps + warp; blk < nblocks; blk += gridDim.x * kEdenWarps) {
    const long long e0 = static_cast<long long>(blk) * kBlock;
    const int valid = static_cast<int>(min(static_cast<long long>(kBlock), n - e0));
    float y[32];
    load_block<float>(x + e0, valid, vec_ok, lane, y);
#pragma unroll
    for (int k = 0; k < 32; ++k) y[k] = sanitize(y[k]);
    rotate_forward(y, sgn, tiles[warp], lane);
    const int first = (lane & 3) + 128 * (lane >> 2);
    if (valid < kBlock) {  // a partial block keeps as many coefficients as it has values
#pragma unroll
      for (int k = 0; k < 32; ++k)
        if (first + 4 * k >= valid) y[k] = 0.0f;
    }
    float norm = 0.0f;
#pragma unroll
    for (int k = 0; k < 32; ++k) norm = fmaf(y[k], y[k], norm);
    norm = sum_of_warp(norm);
    const float unit = rsqrtf(fmaxf(norm, 1e-30f) / static_cast<float>(kBlock));
    float dot = 0.0f;
    uint32_t part[BITS][4];
#pragma unroll
    for (int b = 0; b < BITS; ++b)
#pragma unroll
      for (int q = 0; q < 4; ++q) part[b][q] = 0u;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const float u = y[k] * unit;
      int bin = 0;  // number of boundaries below u
#pragma unroll
      for (int half = L / 2; half > 0; half >>= 1)
        if (bnd[bin + half - 1] < u) bin += half;
      dot = fmaf(y[k], cen[bin], dot);
#pragma unroll
      for (int b = 0; b < BITS; ++b) part[b][k >> 3] |= ((static_cast<uint32_t>(bin) >> b) & 1u) << (4 * (k & 7));
    }
    dot = sum_of_warp(dot);
    if (lane == 0) scale[blk] = __fdiv_rn(norm, fmaxf(dot, 1e-30f));
    const int pos = lane & 3;
#pragma unroll
    for (int b = 0; b < BITS; ++b) {
      // lanes 4 g .. 4 g + 3 hold bits pos, pos + 4, .. of words 4 g .. 4 g + 3; lane 4 g + q collects word q
      uint32_t w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) w[q] = part[b][q] << pos;
      const bool odd = lane & 1, high = lane & 2;
      uint32_t lo = odd ? w[1] : w[0], hi = odd ? w[3] : w[2];
      lo |= __shfl_xor_sync(kFullMask, odd ? w[0] : w[1], 1);
      hi |= __shfl_xor_sync(kFullMask, odd ? w[2] : w[3], 1);
      uint32_t mine = high ? hi : lo;
      mine |= __shfl_xor_sync(kFullMask, high ? lo : hi, 2);
      words[b * plane + static_cast<size_t>(blk) * 32 + lane] = mine;
    }
  }
}

// words [BITS, 32 nblocks], scale [nblocks] -> out [n]
template <int BITS>
__global__ void __launch_bounds__(kEdenWarps * 32, 2) eden_decompress_kernel(
    const uint32_t* __restrict__ words, const float* __restrict__ scale, const float* __restrict__ levels,
    float* __restrict__ out, long long n, int nblocks, int message_blocks, uint32_t step, uint32_t seed_lo, uint32_t seed_hi) {
  constexpr int L = 1 << BITS;
  __shared__ __align__(16) float tiles[kEdenWarps][kBlock];
  __shared__ __align__(16) float sgn[kBlock];
  __shared__ uint32_t sign_words[32];
  __shared__ float cen[L];
  let_next_start();
  wait_for_previous();
  for (int i = threadIdx.x; i < L; i += kEdenWarps * 32) cen[i] = levels[i];
  eden_signs(sgn, sign_words, 1.0f / 32.0f, step, seed_lo, seed_hi);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool vec_ok = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  const size_t plane = static_cast<size_t>(message_blocks) * 32;
  for (int blk = blockIdx.x * kEdenWarps + warp; blk < nblocks; blk += gridDim.x * kEdenWarps) {
    const float s = scale[blk];
    uint32_t mine[BITS];
#pragma unroll
    for (int b = 0; b < BITS; ++b) mine[b] = words[b * plane + static_cast<size_t>(blk) * 32 + lane];
    float y[32];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t w[BITS];
#pragma unroll
      for (int b = 0; b < BITS; ++b) w[b] = __shfl_sync(kFullMask, mine[b], (lane & ~3) | q) >> (lane & 3);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        uint32_t bin = 0;
#pragma unroll
        for (int b = 0; b < BITS; ++b) bin |= ((w[b] >> (4 * j)) & 1u) << b;
        y[8 * q + j] = sanitize(cen[bin] * s);
      }
    }
    rotate_inverse(y, sgn, tiles[warp], lane);
    const long long e0 = static_cast<long long>(blk) * kBlock;
    store_block<float>(out + e0, static_cast<int>(min(static_cast<long long>(kBlock), n - e0)), vec_ok, lane, y);
  }
}

int eden_grid(int nblocks) { return std::min((nblocks + kEdenWarps - 1) / kEdenWarps, 148 * 4); }

void check_levels(const at::Tensor& levels, const at::Tensor& like, int64_t bits) {
  TORCH_CHECK(bits >= 1 && bits <= 8, "EDEN supports 1..8 bits");
  TORCH_CHECK(levels.device() == like.device() && levels.scalar_type() == at::kFloat && levels.is_contiguous() &&
                  levels.numel() == (2 << bits) - 1,
              "eden: levels holds 2^bits centroids and 2^bits - 1 boundaries, fp32, on the input's device");
}

#define DQ_EDEN_SWITCH(CALL)     \
  switch (bits) {                \
    case 1: CALL(1); break;      \
    case 2: CALL(2); break;      \
    case 3: CALL(3); break;      \
    case 4: CALL(4); break;      \
    case 5: CALL(5); break;      \
    case 6: CALL(6); break;      \
    case 7: CALL(7); break;      \
    default: CALL(8); break;     \
  }

}  // namespace

// flat fp32 x -> (words int32 [bits, 32 nb], scale fp32 [nb]), nb = ceil(n / 1024)
std::tuple<at::Tensor, at::Tensor> eden_compress(at::Tensor x, at::Tensor levels, int64_t bits, int64_t seed, int64_t step) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.is_contiguous() && x.dim() == 1, "eden: flat CUDA fp32 tensor");
  check_levels(levels, x, bits);
  c10::cuda::CUDAGuard guard(x.device());
  const long long n = x.numel();
  const int nb = static_cast<int>((n + kBlock - 1) / kBlock);
  at::Tensor words = at::empty({bits, 32ll * nb}, x.options().dtype(at::kInt)), scale = at::empty({nb}, x.options());
  if (nb == 0) return {words, scale};
  const uint64_t s = static_cast<uint64_t>(seed);
  auto stream = at::cuda::getCurrentCUDAStream();
#define DQ_CALL(B)                                                                                                     \
  C10_CUDA_CHECK(launch_dependent(eden_compress_kernel<B>, eden_grid(nb), kEdenWarps * 32, 0, stream,                                               \
      x.data_ptr<float>(), levels.data_ptr<float>(), reinterpret_cast<uint32_t*>(words.data_ptr<int>()),               \
      scale.data_ptr<float>(), n, nb, static_cast<uint32_t>(step), static_cast<uint32_t>(s), static_cast<uint32_t>(s >> 32)))
  DQ_EDEN_SWITCH(DQ_CALL)
#undef DQ_CALL
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return {words, scale};
}

// (words, scale) -> fp32 [n], n <= 1024 nb
at::Tensor eden_decompress(at::Tensor words, at::Tensor scale, at::Tensor levels, int64_t n, int64_t bits, int64_t seed,
                           int64_t step) {
  TORCH_CHECK(scale.is_cuda() && scale.scalar_type() == at::kFloat && scale.is_contiguous(), "eden: fp32 CUDA scales");
  const int nb = static_cast<int>(scale.numel());
  TORCH_CHECK(words.device() == scale.device() && words.scalar_type() == at::kInt && words.is_contiguous() &&
                  words.dim() == 2 && words.size(0) == bits && words.size(1) == 32ll * nb,
              "eden: words must be int32 [bits, 32 x blocks]");
  TORCH_CHECK(n >= 0 && n <= static_cast<int64_t>(nb) * kBlock, "eden: more values than the message holds");
  check_levels(levels, scale, bits);
  c10::cuda::CUDAGuard guard(scale.device());
  at::Tensor out = at::empty({n}, scale.options());
  const int used = static_cast<int>((n + kBlock - 1) / kBlock);
  if (used == 0) return out;
  const uint64_t s = static_cast<uint64_t>(seed);
  auto stream = at::cuda::getCurrentCUDAStream();
#define DQ_CALL(B)                                                                                                     \
  C10_CUDA_CHECK(launch_dependent(eden_decompress_kernel<B>, eden_grid(used), kEdenWarps * 32, 0, stream,                                             \
      reinterpret_cast<const uint32_t*>(words.data_ptr<int>()), scale.data_ptr<float>(), levels.data_ptr<float>(),     \
      out.data_ptr<float>(), n, used, nb, static_cast<uint32_t>(step), static_cast<uint32_t>(s), static_cast<uint32_t>(s >> 32)))
  DQ_EDEN_SWITCH(DQ_CALL)
#undef DQ_CALL
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return out;
}

}  // namespace dq
