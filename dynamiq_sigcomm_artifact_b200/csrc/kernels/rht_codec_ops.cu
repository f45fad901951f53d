// Standalone operators of the rotation codec: encode, hop (decode + add a rotated local block + re-encode), decode.
//
// One warp per 1024-element block, the same device functions as the collective kernel, so the same bytes.  A message
// here has no mailbox: codes and scales are read from and written to the caller's tensors directly, and nothing
// waits for a peer, so the launch is an ordinary one.  (Running them as one-step programs of the collective moved
// every message twice more through the mailbox and cloned the input: 64 us of copies beside 75 us of kernels for
// encode + hop + decode of 16 Mi values.)
//
// Bound by instruction issue (about 790 warp instructions per block for encode) next to HBM: CTAs of eight warps,
// two per SM at 128 registers, each warp with one bulk-copied block in flight ahead of the one it works on.
//
// Reference counterparts: scaling_compress / scaling_dec_comp / scaling_decompress
// (cuda_kernels/src/srrcomp/eden_utils/eden_utils.cpp:133-219).
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "../common/rht_codec.cuh"
#include "../common/tcgen05.cuh"
#include "dependent_launch.cuh"

namespace dq {
namespace {

constexpr int kOpWarps = 8;
enum : int { kOpEncode = 0, kOpHop = 1, kOpDecode = 2 };

struct RhtOpParams {
  void* x;                 // encode / hop: local values (read); decode: result (written)
  const uint32_t* codes_in;
  const float* scales_in;
  uint32_t* codes_out;
  float* scales_out;
  long long n;
  int nblocks;
  uint32_t seed_lo, seed_hi, step, bucket_id, tag;
  float finish_scale;
};

template <int BITS, typename T, int OP>
__global__ void __launch_bounds__(kOpWarps * 32, OP == kOpDecode ? 3 : 2) rht_op_kernel(const __grid_constant__ RhtOpParams p) {
  extern __shared__ __align__(128) uint8_t smem[];  // [tiles][stages][sign table][sign words][barriers]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float* tile = reinterpret_cast<float*>(smem) + warp * kBlock;
  float* stage = reinterpret_cast<float*>(smem) + (kOpWarps + warp) * kBlock;
  float* sgn = reinterpret_cast<float*>(smem) + 2 * kOpWarps * kBlock;
  uint32_t* sign_words = reinterpret_cast<uint32_t*>(sgn + kBlock);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sign_words + 32) + warp;
  if (tid < 32) sign_words[tid] = sign_word(tid, p.step, p.bucket_id, p.seed_lo, p.seed_hi);
  if (lane == 0) tc::mbar_init(bar, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  const float c = OP == kOpDecode ? p.finish_scale : 1.0f;
  for (int e = tid; e < kBlock; e += kOpWarps * 32) sgn[e] = ((sign_words[e >> 5] >> (e & 31)) & 1u) ? -c : c;
  __syncthreads();
  let_next_start();
  wait_for_previous();  // the tables above need no memory

  T* x = static_cast<T*>(p.x);
  const bool vec_ok = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  const int stride = gridDim.x * kOpWarps;
  const int whole = static_cast<int>(p.n / kBlock);  // blocks a bulk copy may fetch
  bool bulk = OP != kOpDecode && vec_ok;
  uint32_t parity = 0;
  int blk = blockIdx.x * kOpWarps + warp;
  if (bulk && blk < whole && lane == 0) tc::bulk_load(stage, x + static_cast<long long>(blk) * kBlock, kBlock * sizeof(T), bar);
  for (; blk < p.nblocks; blk += stride) {
    const long long e0 = static_cast<long long>(blk) * kBlock;
    const int valid = static_cast<int>(min(static_cast<long long>(kBlock), p.n - e0));
    float v[32], scale = 0.f;
    uint32_t w[BITS];
    if (OP != kOpEncode) {
#pragma unroll
      for (int j = 0; j < BITS; ++j) w[j] = __ldcs(p.codes_in + static_cast<size_t>(blk) * (BITS * 32) + j * 32 + lane);
      scale = __ldg(p.scales_in + blk);
    }
    if (OP != kOpDecode) {
      if (bulk && blk < whole && __all_sync(kFullMask, tc::mbar_wait(bar, parity))) {
        parity ^= 1u;
        load_block<T>(reinterpret_cast<const T*>(stage), kBlock, true, lane, v);
        __syncwarp();
      } else {
        if (blk < whole) bulk = false;  // a copy that never landed (or an unaligned input): read directly from here on
        load_block<T>(x + e0, valid, vec_ok, lane, v);
      }
      const int next = blk + stride;
      if (bulk && next < whole && lane == 0) tc::bulk_load(stage, x + static_cast<long long>(next) * kBlock, kBlock * sizeof(T), bar);
      rotate_forward(v, sgn, tile, lane);
      if (OP == kOpHop) dequantize_add_block<BITS>(w, scale, v);
      scale = quantize_block<BITS>(v, w, static_cast<uint32_t>(blk), p.tag, p.step, p.seed_lo, p.seed_hi, lane);
#pragma unroll
      for (int j = 0; j < BITS; ++j) p.codes_out[static_cast<size_t>(blk) * (BITS * 32) + j * 32 + lane] = w[j];
      if (lane == 0) p.scales_out[blk] = scale;
    } else {
      dequantize_block<BITS>(w, scale, v);
      rotate_inverse(v, sgn, tile, lane);
      store_block<T>(x + e0, valid, vec_ok, lane, v);
    }
  }
}

constexpr size_t kOpSmem = (2 * kOpWarps + 1) * kBlock * 4 + 32 * 4 + kOpWarps * 8;

template <int BITS, typename T, int OP>
void launch_op(const RhtOpParams& p, int64_t max_warps, cudaStream_t stream) {
  static const bool configured = [] {
    C10_CUDA_CHECK(cudaFuncSetAttribute(rht_op_kernel<BITS, T, OP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(kOpSmem)));
    return true;
  }();
  (void)configured;
  // a warp per block, at most the warps the caller grants the operator
  const int64_t want = std::min<int64_t>(p.nblocks, std::max<int64_t>(max_warps, kOpWarps));
  C10_CUDA_CHECK(launch_dependent(rht_op_kernel<BITS, T, OP>, static_cast<unsigned>((want + kOpWarps - 1) / kOpWarps), kOpWarps * 32,
                                  kOpSmem, stream, p));
}

template <typename T, int OP>
void launch_bits(int64_t bits, const RhtOpParams& p, int64_t max_warps) {
  cudaStream_t stream = at::cuda::getCurrentCUDAStream();
  switch (bits) {
    case 2: launch_op<2, T, OP>(p, max_warps, stream); break;
    case 3: launch_op<3, T, OP>(p, max_warps, stream); break;
    case 4: launch_op<4, T, OP>(p, max_warps, stream); break;
    case 5: launch_op<5, T, OP>(p, max_warps, stream); break;
    case 6: launch_op<6, T, OP>(p, max_warps, stream); break;
    case 7: launch_op<7, T, OP>(p, max_warps, stream); break;
    case 8: launch_op<8, T, OP>(p, max_warps, stream); break;
    default: TORCH_CHECK(false, "bits must be in 2..8, got ", bits);
  }
}

template <int OP>
void launch(const at::Tensor& x, int64_t bits, const RhtOpParams& p, int64_t max_warps) {
  if (p.nblocks == 0) return;
  if (x.scalar_type() == at::kFloat) launch_bits<float, OP>(bits, p, max_warps);
  else launch_bits<__nv_bfloat16, OP>(bits, p, max_warps);
}

RhtOpParams common(const at::Tensor& x, int64_t seed, int64_t step, int64_t bucket_id) {
  TORCH_CHECK(x.is_cuda() && x.is_contiguous(), "bucket must be a contiguous CUDA tensor");
  TORCH_CHECK(x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16, "bucket must be float32 or bfloat16");
  RhtOpParams p{};
  p.x = x.data_ptr();
  p.n = x.numel();
  p.nblocks = static_cast<int>((p.n + kBlock - 1) / kBlock);
  p.seed_lo = static_cast<uint32_t>(static_cast<uint64_t>(seed) & 0xFFFFFFFFull);
  p.seed_hi = static_cast<uint32_t>(static_cast<uint64_t>(seed) >> 32);
  p.step = static_cast<uint32_t>(step);
  p.bucket_id = static_cast<uint32_t>(bucket_id);
  return p;
}

void take_message(RhtOpParams& p, const at::Tensor& codes, const at::Tensor& scales, int64_t bits, const at::Tensor& like) {
  TORCH_CHECK(codes.device() == like.device() && codes.scalar_type() == at::kInt && codes.is_contiguous() &&
                  codes.numel() >= static_cast<int64_t>(p.nblocks) * bits * 32,
              "codes must be a contiguous int32 CUDA tensor of ", p.nblocks, " x ", bits, " x 32 words");
  TORCH_CHECK(scales.device() == like.device() && scales.scalar_type() == at::kFloat && scales.is_contiguous() &&
                  scales.numel() >= p.nblocks,
              "scales must be a contiguous fp32 CUDA tensor with one value per block");
  p.codes_in = reinterpret_cast<const uint32_t*>(codes.data_ptr<int>());
  p.scales_in = scales.data_ptr<float>();
}

}  // namespace

// x (flat fp32 / bf16) [+ an incoming message] -> (code words int32 [nb, bits, 32], scales fp32 [nb])
std::tuple<at::Tensor, at::Tensor> rht_encode(at::Tensor x, c10::optional<at::Tensor> codes, c10::optional<at::Tensor> scales,
                                              int64_t bits, int64_t seed, int64_t step, int64_t bucket_id, int64_t tag,
                                              int64_t max_warps) {
  c10::cuda::CUDAGuard guard(x.device());
  RhtOpParams p = common(x, seed, step, bucket_id);
  TORCH_CHECK(bits >= 2 && bits <= 8, "bits must be in 2..8, got ", bits);
  p.tag = stream_tag(p.bucket_id, static_cast<uint32_t>(tag));
  at::Tensor c = at::empty({p.nblocks, bits, 32}, x.options().dtype(at::kInt));
  at::Tensor s = at::empty({p.nblocks}, x.options().dtype(at::kFloat));
  p.codes_out = reinterpret_cast<uint32_t*>(c.data_ptr<int>());
  p.scales_out = s.data_ptr<float>();
  if (codes.has_value()) {
    TORCH_CHECK(scales.has_value(), "a message is codes and scales");
    take_message(p, *codes, *scales, bits, x);
    launch<kOpHop>(x, bits, p, max_warps);
  } else {
    launch<kOpEncode>(x, bits, p, max_warps);
  }
  return {c, s};
}

// message -> out (flat fp32 / bf16) = inverse rotation x post_scale
void rht_decode(at::Tensor codes, at::Tensor scales, at::Tensor out, int64_t bits, int64_t seed, int64_t step,
                int64_t bucket_id, double post_scale, int64_t max_warps) {
  c10::cuda::CUDAGuard guard(out.device());
  RhtOpParams p = common(out, seed, step, bucket_id);
  TORCH_CHECK(bits >= 2 && bits <= 8, "bits must be in 2..8, got ", bits);
  p.finish_scale = static_cast<float>(post_scale / 1024.0);
  take_message(p, codes, scales, bits, out);
  launch<kOpDecode>(out, bits, p, max_warps);
}

}  // namespace dq
