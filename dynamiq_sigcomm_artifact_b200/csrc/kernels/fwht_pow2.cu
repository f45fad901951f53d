// Walsh-Hadamard transform (Sylvester order) of a whole vector whose length is a power of two.
//
// A CTA transforms a tile of 8192 values, 13 butterfly levels, in three register rounds of 5 + 5 + 3 levels with two
// exchanges through 32 KB of shared memory.  The first launch takes contiguous tiles (levels 0..12).  Every further
// launch takes up to 10 more levels: its tile is 2^m rows, 2^first values apart, of 2^(13 - m) contiguous columns
// (32 bytes at the least, so no sector is read for nothing), and applies only the levels of the row index.  A vector
// of up to 2^13 values is one launch, up to 2^23 (the longest THC partition) two: the array is read and written twice,
// where tensor-core 1024-blocks followed by radix-32 passes over memory took three or four passes (2^22 values:
// 27 us before, and a status word to clear).  Bound by L2 / HBM traffic and, for short vectors, by latency; plain
// fp32 butterflies, one rounding per addition.
//
// Used by THC's whole-partition rotation (reference: testbed_evaluation/new_comm_hooks/thc_hooks.py:124-149, which
// calls the SIMT Hadamard of cuda_kernels/src/srrcomp/eden_utils/csrc/cuda_hadamard.cu:58-251).
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "dependent_launch.cuh"

namespace dq {
namespace {

constexpr int kTileLog = 13, kTile = 1 << kTileLog, kFwhtThreads = 256;
constexpr int kRowLevels = 10;  // levels of a strided launch: 2^10 rows leave 8 columns

// v[i], v[i + 1] <- sums with v[k], v[k + 1], which become the differences, two values per instruction (the same roundings)
__device__ __forceinline__ void butterfly2(float (&v)[32], int i, int k) {
  asm("{\n\t.reg .b64 a, b, m;\n\t"
      "mov.b64 a, {%0, %1};\n\t"
      "mov.b64 b, {%2, %3};\n\t"
      "mov.b64 m, {%4, %4};\n\t"
      "fma.rn.f32x2 m, b, m, a;\n\t"
      "add.rn.f32x2 a, a, b;\n\t"
      "mov.b64 {%0, %1}, a;\n\t"
      "mov.b64 {%2, %3}, m;\n\t}"
      : "+f"(v[i]), "+f"(v[i + 1]), "+f"(v[k]), "+f"(v[k + 1])
      : "f"(-1.0f));
}

// butterfly on register bit BIT of v, skipped when the level of that bit is not this launch's
template <int BIT>
__device__ __forceinline__ void level(float (&v)[32], bool on) {
  if (!on) return;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    if (i & (1 << BIT)) continue;
    if (BIT == 0) {
      const float a = v[i], b = v[i | 1];
      v[i] = a + b;
      v[i | 1] = a - b;
    } else if ((i & 1) == 0) {
      butterfly2(v, i, i | (1 << BIT));
    }
  }
}

// where value e of the tile lives in shared memory: 16-byte groups of a 128-value row are permuted by bits 7..9, which
// keeps the 16-byte accesses (rounds 1 and 3) and the stride-4 accesses of round 2 free of bank conflicts
__device__ __forceinline__ int place(int e) { return e ^ (((e >> 7) & 7) << 2); }

// levels [lo, hi) of the tile's 13-bit index; row length 2^col_log inside the tile, rows 2^first apart in memory
__global__ void __launch_bounds__(kFwhtThreads, 4) fwht_tile_kernel(const float* in, float* out,
                                                                     long long n, int col_log, int first, int lo, int hi,
                                                                     int clean, float scale) {
  __shared__ __align__(16) float sm[kTile];
  wait_for_previous();
  let_next_start();
  const int tid = threadIdx.x;
  // tile -> (outer block of 2^(first + rows) values, column group)
  const int row_log = kTileLog - col_log;
  long long base;
  if (row_log == 0) {
    base = static_cast<long long>(blockIdx.x) * kTile;
  } else {
    const int groups_log = first - col_log;  // column groups per outer block
    const long long outer = static_cast<long long>(blockIdx.x) >> groups_log;
    const long long group = static_cast<long long>(blockIdx.x) & ((1ll << groups_log) - 1);
    base = (outer << (first + row_log)) + (group << col_log);
  }
  // offset in memory of bit b of the tile index; bits are disjoint, so offsets add up
  auto bit = [&](int b) { return b < col_log ? 1ll << b : 1ll << (first + b - col_log); };
  auto address = [&](int e) {
    return base + (static_cast<long long>(e >> col_log) << first) + (e & ((1 << col_log) - 1));
  };
  float v[32];
  // round 1: registers = bits {0, 1, 10, 11, 12}
  const float* src = in + address(tid * 4);
  const long long s10 = bit(10), s11 = bit(11), s12 = bit(12);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int e = (j << 10) + tid * 4;
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    if (n >= kTile) {
      q = *reinterpret_cast<const float4*>(src + ((j & 1) ? s10 : 0) + ((j & 2) ? s11 : 0) + ((j & 4) ? s12 : 0));
    } else {
      if (e + 0 < n) q.x = in[e];
      if (e + 1 < n) q.y = in[e + 1];
      if (e + 2 < n) q.z = in[e + 2];
      if (e + 3 < n) q.w = in[e + 3];
    }
    v[4 * j] = q.x, v[4 * j + 1] = q.y, v[4 * j + 2] = q.z, v[4 * j + 3] = q.w;
  }
  if (clean) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = fabsf(v[i]) <= 3.402823466e38f ? v[i] : 0.0f;
  }
  auto active = [&](int b) { return b >= lo && b < hi; };
  level<0>(v, active(0));
  level<1>(v, active(1));
  level<2>(v, active(10));
  level<3>(v, active(11));
  level<4>(v, active(12));
#pragma unroll
  for (int j = 0; j < 8; ++j)
    *reinterpret_cast<float4*>(sm + place((j << 10) + tid * 4)) =
        make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  __syncthreads();
  // round 2: registers = bits {2..6}; the lane holds bits {0, 1, 7, 8, 9}, the warp bits {10, 11, 12}
  const int lane = tid & 31, warp = tid >> 5;
  const int e2 = (lane & 3) | ((lane >> 2) << 7) | (warp << 10);
#pragma unroll
  for (int t = 0; t < 32; ++t) v[t] = sm[place(e2 | (t << 2))];
  level<0>(v, active(2));
  level<1>(v, active(3));
  level<2>(v, active(4));
  level<3>(v, active(5));
  level<4>(v, active(6));
#pragma unroll
  for (int t = 0; t < 32; ++t) sm[place(e2 | (t << 2))] = v[t];
  __syncwarp();  // round 3 reads what this warp wrote: bits 10..12 stay with the warp
  // round 3: registers = bits {0, 1, 7, 8, 9}, lanes = bits {2..6}: 512 contiguous bytes per warp and store
  const int e3 = (lane << 2) | (warp << 10);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float4 q = *reinterpret_cast<const float4*>(sm + place(e3 | (j << 7)));
    v[4 * j] = q.x, v[4 * j + 1] = q.y, v[4 * j + 2] = q.z, v[4 * j + 3] = q.w;
  }
  level<2>(v, active(7));
  level<3>(v, active(8));
  level<4>(v, active(9));
  float* dst = out + address(e3);
  const long long s7 = bit(7), s8 = bit(8), s9 = bit(9);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int e = e3 | (j << 7);
    const float4 q = make_float4(v[4 * j] * scale, v[4 * j + 1] * scale, v[4 * j + 2] * scale, v[4 * j + 3] * scale);
    if (n >= kTile) {
      *reinterpret_cast<float4*>(dst + ((j & 1) ? s7 : 0) + ((j & 2) ? s8 : 0) + ((j & 4) ? s9 : 0)) = q;
    } else {
      if (e + 0 < n) out[e] = q.x;
      if (e + 1 < n) out[e + 1] = q.y;
      if (e + 2 < n) out[e + 2] = q.z;
      if (e + 3 < n) out[e + 3] = q.w;
    }
  }
}

}  // namespace

// H x * scale for a flat fp32 tensor whose length is a power of two; `clean`: non-finite inputs count as zeros
at::Tensor fwht_pow2(at::Tensor x, double scale, bool clean) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.is_contiguous() && x.dim() == 1,
              "fwht_pow2: flat contiguous CUDA fp32 tensor");
  const long long n = x.numel();
  TORCH_CHECK(n > 0 && (n & (n - 1)) == 0, "fwht_pow2: length must be a power of two, got ", n);
  c10::cuda::CUDAGuard guard(x.device());
  if (reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 != 0) x = x.clone();
  at::Tensor y = at::empty_like(x);
  int k = 0;
  while ((1ll << k) < n) ++k;
  auto stream = at::cuda::getCurrentCUDAStream();
  const unsigned grid = static_cast<unsigned>(std::max<long long>(1, n >> kTileLog));
  const int contiguous = std::min(k, kTileLog);
  float* out = y.data_ptr<float>();
  C10_CUDA_CHECK(launch_dependent(fwht_tile_kernel, grid, kFwhtThreads, 0, stream, x.data_ptr<float>(), out, n, kTileLog, 0, 0, contiguous, clean ? 1 : 0,
                                                      k <= kTileLog ? static_cast<float>(scale) : 1.0f));
  for (int first = kTileLog; first < k;) {
    const int m = std::min(kRowLevels, k - first);
    C10_CUDA_CHECK(launch_dependent(fwht_tile_kernel, grid, kFwhtThreads, 0, stream, out, out, n, kTileLog - m, first, kTileLog - m, kTileLog, 0,
                                                        first + m == k ? static_cast<float>(scale) : 1.0f));
    first += m;
  }
  return y;
}

}  // namespace dq
