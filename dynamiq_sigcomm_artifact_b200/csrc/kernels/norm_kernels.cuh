// Vector access helpers of the model kernels, and the normalisation backward kernel for rows of up to 2048 columns, shared
// by the operators in residual_norm.cu and the allocation-free C entry point in norm_bwd_noalloc.cu.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace dq {
namespace normk {

constexpr unsigned kFull = 0xFFFFFFFFu;

template <typename T>
struct Vec8;  // 8 elements = 16 bytes for bf16, 32 bytes for float (two float4)
template <>
struct Vec8<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&o)[8]) {
    uint4 q = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[2 * i] = __uint_as_float(w[i] << 16);
      o[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&o)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 h = __floats2bfloat162_rn(o[2 * i], o[2 * i + 1]);
      w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  }
};
template <>
struct Vec8<float> {
  static __device__ __forceinline__ void load(const float* p, float (&o)[8]) {
    float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    o[0] = a.x, o[1] = a.y, o[2] = a.z, o[3] = a.w, o[4] = b.x, o[5] = b.y, o[6] = b.z, o[7] = b.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&o)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(o[4], o[5], o[6], o[7]);
  }
};

__device__ __forceinline__ float to_f(float x) { return x; }
__device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
template <typename P>
__device__ __forceinline__ P from_f(float x);
template <>
__device__ __forceinline__ float from_f<float>(float x) { return x; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

constexpr int kNormWarps = 8;


// eight values as they are in memory: loads of several tensors are in flight before any of them is used
template <typename T>
struct Raw8;
template <>
struct Raw8<__nv_bfloat16> {
  uint4 q;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { q = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ void get(float (&o)[8]) const {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[2 * i] = __uint_as_float(w[i] << 16);
      o[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
  }
};
template <>
struct Raw8<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const float* p) {
    a = *reinterpret_cast<const float4*>(p);
    b = *reinterpret_cast<const float4*>(p + 4);
  }
  __device__ __forceinline__ void get(float (&o)[8]) const {
    o[0] = a.x, o[1] = a.y, o[2] = a.z, o[3] = a.w, o[4] = b.x, o[5] = b.y, o[6] = b.z, o[7] = b.w;
  }
};

// ---- backward of rows with H <= 2048 ----
// A CTA holds several groups of NT threads (a multiple of 32, at least H / 8), one row per group at a time and eight
// columns per thread, so that the column sums of dw, db and dbias are 8 registers each; a group synchronises once a row
// on a barrier of its own.  Every thread brings its own columns of the next rows into its own slots of a shared-memory
// ring with asynchronous copies (no registers, no barrier).  At the end the groups add their sums in a fixed order in
// shared memory and the CTA leaves one partial row: part[arrays][gridDim.x][H], arrays = dw, (db), (dbias).
// `extra` (may be null): a second term of dy, or one of dx.
constexpr int kNormBwdThreads = 384;  // two CTAs per SM at 80 registers
template <typename T>
constexpr int norm_ring() { return sizeof(T) == 2 ? 4 : 2; }  // rows of the ring

inline int norm_group_threads(int H) { return (H / 8 + 31) / 32 * 32; }
inline int norm_groups(int H) { return kNormBwdThreads / norm_group_threads(H) < 8 ? kNormBwdThreads / norm_group_threads(H) : 8; }
// column sums of the groups, then the ring: three tensors x 8 values per thread and row
inline size_t norm_bwd_smem(int H) {
  return static_cast<size_t>(H) * sizeof(float) + static_cast<size_t>(norm_group_threads(H)) * norm_groups(H) * 3 * 64;
}
constexpr int kNormBwdMaxSmem = 2048 * 4 + kNormBwdThreads * 3 * 64;
inline int norm_bwd_grid(int rows, int H, int sms) {
  const int groups = norm_groups(H), want = (rows + groups - 1) / groups;
  const int most = sms * (768 / (groups * norm_group_threads(H)));
  return want < most ? (want > 0 ? want : 1) : most;
}

__device__ __forceinline__ void copy16_async(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem))), "l"(gmem)
               : "memory");
}

template <typename T, bool RMS, bool BIAS>
__global__ void __launch_bounds__(kNormBwdThreads, 2) add_norm_bwd_kernel(
    const T* __restrict__ dy, const T* __restrict__ extra, bool extra_is_dy, const T* __restrict__ s,
    const float* __restrict__ w, const float* __restrict__ mean, const float* __restrict__ rstd, T* __restrict__ dx,
    float* __restrict__ part, int rows, int H, int NT) {
  constexpr int N = norm_ring<T>();
  extern __shared__ __align__(16) float sm[];      // [H], then the ring
  __shared__ float2 red[2][kNormBwdThreads / 32];  // per warp, two rows in turn
  const int groups = blockDim.x / NT, group = threadIdx.x / NT, t = threadIdx.x - group * NT, c = t * 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gw = NT / 32;
  const bool on = c < H;
  const float inv_h = 1.0f / static_cast<float>(H);
  float adw[8], adb[8], abias[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) adw[k] = adb[k] = abias[k] = 0.f;
  T* ring = reinterpret_cast<T*>(sm + H);  // [N][3][blockDim.x][8]
  auto slot = [&](int n, int tensor) { return ring + (static_cast<size_t>(n * 3 + tensor) * blockDim.x + threadIdx.x) * 8; };
  auto fetch = [&](int row, int n) {
    if (on && row < rows) {
      const size_t at = static_cast<size_t>(row) * H + c;
#pragma unroll
      for (int h = 0; h < static_cast<int>(sizeof(T)) / 2; ++h) {  // 16 bytes at a time
        constexpr int V = 16 / sizeof(T);
        copy16_async(slot(n, 0) + h * V, s + at + h * V);
        copy16_async(slot(n, 1) + h * V, dy + at + h * V);
        if (extra != nullptr) copy16_async(slot(n, 2) + h * V, extra + at + h * V);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int step = gridDim.x * groups;
  int row = blockIdx.x * groups + group, turn = 0, n = 0;
#pragma unroll
  for (int i = 0; i < N - 1; ++i) fetch(row + i * step, i);
  float mu = 0.f, rs = 0.f, nmu = 0.f, nrs = 0.f;
  if (row < rows) mu = RMS ? 0.f : mean[row], rs = rstd[row];
  for (; row < rows; row += step, turn ^= 1, n = n + 1 == N ? 0 : n + 1) {
    fetch(row + (N - 1) * step, n == 0 ? N - 1 : n - 1);
    if (row + step < rows) nmu = RMS ? 0.f : mean[row + step], nrs = rstd[row + step];
    asm volatile("cp.async.wait_group %0;" ::"n"(N - 1) : "memory");  // this row's copies, which only this thread reads
    // read before and again after the barrier: fewer registers stay live across it
    auto unpack = [&](float (&v)[8], float (&d)[8], float (&g)[8]) {
      Vec8<T>::load(slot(n, 0), v);
      Vec8<T>::load(slot(n, 1), d);
      if (extra != nullptr && extra_is_dy) {
        float e[8];
        Vec8<T>::load(slot(n, 2), e);
#pragma unroll
        for (int k = 0; k < 8; ++k) d[k] += e[k];
      }
      Vec8<float>::load(w + c, g);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = (v[k] - mu) * rs;  // normalised input
    };
    float s1 = 0.f, s2 = 0.f;
    if (on) {
      float v[8], d[8], g[8];
      unpack(v, d, g);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float gdy = g[k] * d[k];
        s1 += gdy;
        s2 += gdy * v[k];
        adw[k] += d[k] * v[k];
        if (!RMS) adb[k] += d[k];
      }
    }
    if (!RMS) s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (gw > 1) {
      if (lane == 0) red[turn][warp] = make_float2(s1, s2);
      asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(NT) : "memory");
      s1 = s2 = 0.f;
      for (int q = 0; q < gw; ++q) {
        const float2 p = red[turn][group * gw + q];
        s1 += p.x, s2 += p.y;
      }
    }
    if (on) {
      const float m1 = RMS ? 0.f : s1 * inv_h, m2 = s2 * inv_h;
      float o[8], v[8], d[8], g[8];
      unpack(v, d, g);
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = rs * (g[k] * d[k] - m1 - v[k] * m2);
      if (extra != nullptr && !extra_is_dy) {
        float r[8];
        Vec8<T>::load(slot(n, 2), r);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] += r[k];
      }
      if (BIAS) {
#pragma unroll
        for (int k = 0; k < 8; ++k) abias[k] += o[k];
      }
      Vec8<T>::store(dx + static_cast<size_t>(row) * H + c, o);
    }
    mu = nmu, rs = nrs;
  }
  auto combine = [&](float (&acc)[8], int array) {
    for (int q = 0; q < groups; ++q) {
      __syncthreads();
      if (q == group && on) {
        if (q > 0) {
          float o[8];
          Vec8<float>::load(sm + c, o);
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[k] += o[k];
        }
        if (q == groups - 1) Vec8<float>::store(part + (static_cast<size_t>(array) * gridDim.x + blockIdx.x) * H + c, acc);
        else Vec8<float>::store(sm + c, acc);
      }
    }
  };
  combine(adw, 0);
  if constexpr (!RMS) combine(adb, 1);
  if constexpr (BIAS) combine(abias, RMS ? 1 : 2);
}

}  // namespace normk
}  // namespace dq
