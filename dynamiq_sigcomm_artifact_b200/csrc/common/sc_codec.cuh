// Warp-level hierarchical "scaling quantisation" codec (the reference's superchunk format).
//
// A warp owns a block of 1024 values = 4 superchunks of 256 = 16 chunks of 16.  Lane l holds the 32
// consecutive values [32 l, 32 l + 32): two whole chunks of superchunk l / 8, so chunk maxima need
// no shuffles and the superchunk maximum is a 3-step butterfly inside an 8-lane group.
//
// Wire record of a superchunk (byte for byte the reference's layout, eden_utils.cpp:33-40,
// scaling_quantization_algorithm.md:347-388): 16 x [2 b bytes of codes, little end first | 1 byte
// round-up chunk scale] + 2 bytes bf16 scale unit = 16 (2 b + 1) + 2 bytes.  A block's four records are
// contiguous (an 8-byte multiple), are assembled in the warp's shared-memory tile and move with 8-byte
// accesses.
//
// Arithmetic restates parallel/codecs.py::SuperchunkCodec operation by operation (fp32, one rounding
// per operation), which itself restates the reference kernels
// (cuda_hierarchical_mee.cu:203-343 encode, :345-505 decode, :526-696 hop); partial sums stay fp32.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "exact_div.cuh"
#include "philox.cuh"
#include "rht_codec.cuh"

namespace dq {

struct ScParams {
  float lattice_max;  // R for the linear lattice, lattice(R) for the logarithmic one
  float c1, c2;       // (1 + e^2) / (2 e^2) and log2(1 + 2 e^2)
  const float* lut;   // decode levels [2^b], device memory
};

template <int B>
struct ScGeom {
  static constexpr int kChunkBytes = 2 * B + 1;
  static constexpr int kRecordBytes = 16 * kChunkBytes + 2;  // 82 / 146 / 274
  static constexpr int kBlockBytes = 4 * kRecordBytes;       // 328 / 584 / 1096: multiples of 8
};

__device__ __forceinline__ float sc_sanitize(float x) { return (fabsf(x) <= 3.402823466e38f) ? x : 0.0f; }

// lane-contiguous layout: reg k of lane l = element 32 l + k
template <typename T>
__device__ __forceinline__ void sc_load_block(const T* base, int valid, bool vec_ok, int lane, float (&v)[32]) {
  if (valid == 1024 && vec_ok) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      float o[4];
      Elem<T>::load4(base + 32 * lane + 4 * q, o);
#pragma unroll
      for (int k = 0; k < 4; ++k) v[4 * q + k] = o[k];
    }
  } else {
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const int e = 32 * lane + k;
      v[k] = e < valid ? Elem<T>::to_float(base[e]) : 0.0f;
    }
  }
}

template <typename T>
__device__ __forceinline__ void sc_store_block(T* base, int valid, bool vec_ok, int lane, const float (&v)[32]) {
  if (valid == 1024 && vec_ok) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      float o[4] = {v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]};
      Elem<T>::store4(base + 32 * lane + 4 * q, o);
    }
  } else {
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const int e = 32 * lane + k;
      if (e < valid) base[e] = Elem<T>::from_float(v[k]);
    }
  }
}

// The same two moves for whole fp32 blocks with fully coalesced global accesses: the warp reads or writes 512
// contiguous bytes per instruction and the lane-contiguous runs are formed through a warp-private 4 KiB shared
// buffer.  16-byte chunk c (= element / 4) of the block lives at chunk c ^ ((c >> 3) & 7) of the buffer, which
// makes both the linear side (chunk j * 32 + lane) and the per-lane side (chunk lane * 8 + i) free of bank
// conflicts while every register index stays a compile-time constant.
__device__ __forceinline__ void sc_load_block_coalesced(const float* base, float* buf, int lane, float (&v)[32]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = j * 32 + lane;
    const float4 q = *reinterpret_cast<const float4*>(base + 4 * c);
    *reinterpret_cast<float4*>(buf + 4 * (c ^ ((c >> 3) & 7))) = q;
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float4 q = *reinterpret_cast<const float4*>(buf + 4 * ((lane * 8 + i) ^ (lane & 7)));
    v[4 * i] = q.x, v[4 * i + 1] = q.y, v[4 * i + 2] = q.z, v[4 * i + 3] = q.w;
  }
  __syncwarp();
}

__device__ __forceinline__ void sc_store_block_coalesced(float* base, float* buf, int lane, const float (&v)[32]) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
    *reinterpret_cast<float4*>(buf + 4 * ((lane * 8 + i) ^ (lane & 7))) =
        make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = j * 32 + lane;
    *reinterpret_cast<float4*>(base + 4 * c) = *reinterpret_cast<const float4*>(buf + 4 * (c ^ ((c >> 3) & 7)));
  }
  __syncwarp();
}

// ---- a lane's two chunks as one byte stream ----
// A lane's part of a record is [codes of chunk 0][scale][codes of chunk 1][scale]: 4 b + 2 bytes (34 / 18 / 10) at an even
// offset.  It is put together in registers and moved with 32-bit shared-memory accesses (two 16-bit ones where the offset
// is not a multiple of four), instead of byte by byte.

// `B` codes per byte stream of a chunk: four bytes-of-codes words (code 4 j + i in byte i of c[j]) -> B / 2 words
template <int B>
__device__ __forceinline__ void sc_pack16(const uint32_t (&c)[4], uint32_t (&w)[B / 2 > 0 ? B / 2 : 1]) {
  if constexpr (B == 8) {
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = c[j];
  } else if constexpr (B == 4) {
    uint32_t t[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) t[j] = c[j] | (c[j] >> 4);  // bytes 0 and 2 hold two codes each
    w[0] = __byte_perm(t[0], t[1], 0x6420u);
    w[1] = __byte_perm(t[2], t[3], 0x6420u);
  } else {
    uint32_t t[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t p = c[j] | (c[j] >> 6);  // bytes 0 and 2 hold two codes each
      t[j] = p | (p >> 12);                   // byte 0 holds four
    }
    w[0] = __byte_perm(__byte_perm(t[0], t[1], 0x0040u), __byte_perm(t[2], t[3], 0x0040u), 0x5410u);
  }
}

template <int B>
__device__ __forceinline__ void sc_unpack16(const uint32_t (&w)[B / 2 > 0 ? B / 2 : 1], uint32_t (&c)[4]) {
  if constexpr (B == 8) {
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j] = w[j];
  } else if constexpr (B == 4) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t t = __byte_perm(w[j >> 1], 0u, (j & 1) ? 0x4342u : 0x4140u);  // two bytes into bytes 0 and 2
      c[j] = (t | (t << 4)) & 0x0F0F0F0Fu;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t t = __byte_perm(w[0], 0u, 0x4440u + j);
      const uint32_t p = (t | (t << 12)) & 0x000F000Fu;
      c[j] = (p | (p << 6)) & 0x03030303u;
    }
  }
}

// codes of both chunks (as bytes) and their scale bytes -> the lane's stream at `dst` (shared memory, even address)
template <int B>
__device__ __forceinline__ void sc_put_stream(uint8_t* dst, const uint32_t (&c0)[4], const uint32_t (&c1)[4], uint32_t q0,
                                              uint32_t q1) {
  constexpr int W = B / 2;  // code words per chunk: 1, 2, 4
  uint32_t a[W], b[W], w[2 * W + 2];
  sc_pack16<B>(c0, a);
  sc_pack16<B>(c1, b);
#pragma unroll
  for (int j = 0; j < W; ++j) w[j] = a[j];
  w[W] = q0 | (b[0] << 8);
#pragma unroll
  for (int j = 1; j < W; ++j) w[W + j] = __funnelshift_l(b[j - 1], b[j], 8);
  w[2 * W] = (b[W - 1] >> 24) | (q1 << 8);  // 16 bits
  w[2 * W + 1] = 0u;
  const uint32_t odd = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(dst)) & 2u;
  if (odd) *reinterpret_cast<uint16_t*>(dst) = static_cast<uint16_t>(w[0]);
  uint32_t* at = reinterpret_cast<uint32_t*>(dst + odd);
#pragma unroll
  for (int j = 0; j < 2 * W; ++j) at[j] = __funnelshift_r(w[j], w[j + 1], 8 * odd);
  if (!odd) *reinterpret_cast<uint16_t*>(at + 2 * W) = static_cast<uint16_t>(w[2 * W]);
}

template <int B>
__device__ __forceinline__ void sc_get_stream(const uint8_t* src, uint32_t (&c0)[4], uint32_t (&c1)[4], uint32_t& q0,
                                              uint32_t& q1) {
  constexpr int W = B / 2;
  uint32_t r[2 * W + 1], w[2 * W + 1], a[W], b[W];
  const uint32_t odd = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(src)) & 2u;
  const uint32_t* at = reinterpret_cast<const uint32_t*>(src - odd);  // the last word may reach two bytes past the stream:
#pragma unroll                                                       // inside the tile, whose size is a multiple of four
  for (int j = 0; j < 2 * W + 1; ++j) r[j] = at[j];
#pragma unroll
  for (int j = 0; j < 2 * W; ++j) w[j] = __funnelshift_r(r[j], r[j + 1], 8 * odd);
  w[2 * W] = odd ? r[2 * W] >> 16 : r[2 * W];
#pragma unroll
  for (int j = 0; j < W; ++j) a[j] = w[j];
  q0 = w[W] & 0xFFu;
#pragma unroll
  for (int j = 0; j < W; ++j) b[j] = __funnelshift_r(w[W + j], w[W + j + 1], 8);
  q1 = (w[2 * W] >> 8) & 0xFFu;
  sc_unpack16<B>(a, c0);
  sc_unpack16<B>(b, c1);
}

// ---- one lane's 32 values <-> codes (bytes, four per word) and chunk scales ----
// The record's arithmetic with every division done through SharedDivisor: the divisors (chunk scale, lattice constants)
// are shared by 16 values or by all.  A quotient below 1e-20 only has to keep its sign (it ends as level 0 or -1 + 1
// either way), so the general division is needed only where a magnitude exceeds 1e20: the whole warp then takes it.
template <bool MEE>
__device__ __forceinline__ void sc_encode_lane(const float (&v)[32], float lattice_max, float c1, float c2, int R,
                                               uint32_t first_call, uint32_t tag, uint32_t step, uint32_t k0, uint32_t k1,
                                               int lane, uint32_t (&code)[2][4], uint32_t (&scale)[2],
                                               __nv_bfloat16& unit_bf) {
  float x[32], am[2], s[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    am[h] = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      x[16 * h + k] = sc_sanitize(v[16 * h + k]);
      am[h] = fmaxf(am[h], fabsf(x[16 * h + k]));
    }
    s[h] = fmaxf(__fadd_rn(__fdiv_rn(am[h], lattice_max), 1e-7f), 1e-30f);
  }
  float S = fmaxf(s[0], s[1]);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) S = fmaxf(S, __shfl_xor_sync(0xFFFFFFFFu, S, o));
  unit_bf = __float2bfloat16_rn(fmaxf(__fdiv_rn(S, 255.0f), 1e-30f));
  const float unit = fmaxf(__bfloat162float(unit_bf), 1e-30f);
  const bool wide = __any_sync(0xFFFFFFFFu, S > 1e19f);
  const SharedDivisor by_c1(c1), by_c2(c2);
  const float fR = static_cast<float>(R);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float q = fminf(fmaxf(ceilf(__fmul_rn(__fdiv_rn(s[h], S), 255.0f)), 1.0f), 255.0f);
    const float dec = fmaxf(__fmul_rn(q, unit), 1e-30f);
    scale[h] = static_cast<uint32_t>(q);
    float* y = x + 16 * h;
    if (wide) {
#pragma unroll
      for (int k = 0; k < 16; ++k) y[k] = __fdiv_rn(y[k], dec);
    } else {
      const SharedDivisor by_dec(dec);
#pragma unroll
      for (int k = 0; k < 16; ++k) y[k] = by_dec.in_range(y[k]);
    }
    const U4 r = philox4x32<7>(first_call + 2u * static_cast<uint32_t>(lane) + h, 0u, tag, step, k0, k1);
    const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
    uint32_t f[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      float t = y[k];
      if (MEE) {
        const float mag = by_c2.in_range(log2f(__fadd_rn(by_c1.in_range(fabsf(t)), 1.0f)));
        t = t > 0.f ? mag : (t < 0.f ? -mag : 0.f);
      }
      // 2^15 + byte + 0.5 from one byte permute, then (byte + 0.5) / 256: every step exact
      const float u = fmaf(__uint_as_float(__byte_perm(rw[k >> 2], 0x47000080u, 0x7504u | ((k & 3) << 4))), 1.0f / 256.0f, -128.0f);
      const float fl = floorf(t);
      const float c = fl + ((__fsub_rn(t, fl) > u) ? 1.0f : 0.0f);
      f[k] = __float_as_uint(__fadd_rn(fminf(fmaxf(c, -fR), fR), 12582912.0f + fR));  // low byte = c + R
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      code[h][j] = __byte_perm(__byte_perm(f[4 * j], f[4 * j + 1], 0x0040u), __byte_perm(f[4 * j + 2], f[4 * j + 3], 0x0040u), 0x5410u);
  }
}

// `lut`: decode levels in shared memory (MEE)
template <bool MEE, bool ADD>
__device__ __forceinline__ void sc_decode_lane(float (&v)[32], const uint32_t (&code)[2][4], const uint32_t (&scale)[2],
                                               float unit, const float* lut, int R) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float dec = fmaxf(__fmul_rn(static_cast<float>(scale[h]), unit), 1e-30f);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const uint32_t c = (code[h][k >> 2] >> (8 * (k & 3))) & 0xFFu;
      const float level = MEE ? lut[c] : static_cast<float>(static_cast<int>(c) - R);
      const float val = __fmul_rn(level, dec);
      v[16 * h + k] = ADD ? __fadd_rn(v[16 * h + k], val) : val;
    }
  }
}

__device__ __forceinline__ float sc_unit_at(const uint8_t* p) {  // p is even
  return fmaxf(__bfloat162float(__ushort_as_bfloat16(*reinterpret_cast<const unsigned short*>(p))), 1e-30f);
}

// Encode the block held in v into four records in `tile` (shared memory, >= kBlockBytes).
template <int B, bool MEE>
__device__ __forceinline__ void sc_encode_block(const float (&v)[32], uint8_t* tile, const ScParams& sp,
                                                uint32_t first_call, uint32_t tag, uint32_t step, uint32_t k0,
                                                uint32_t k1, int lane) {
  constexpr int R = (1 << (B - 1)) - 1;
  using G = ScGeom<B>;
  uint32_t code[2][4], scale[2];
  __nv_bfloat16 unit;
  sc_encode_lane<MEE>(v, sp.lattice_max, MEE ? sp.c1 : 1.0f, MEE ? sp.c2 : 1.0f, R, first_call, tag, step, k0, k1, lane, code,
                      scale, unit);
  uint8_t* rec = tile + (lane >> 3) * G::kRecordBytes;
  sc_put_stream<B>(rec + 2 * (lane & 7) * G::kChunkBytes, code[0], code[1], scale[0], scale[1]);
  if ((lane & 7) == 0) *reinterpret_cast<__nv_bfloat16*>(rec + 16 * G::kChunkBytes) = unit;
}

// Decode the four records in `tile`; ADD: v <- v + decoded (one rounding each), else v <- decoded.
template <int B, bool MEE, bool ADD>
__device__ __forceinline__ void sc_decode_block(float (&v)[32], const uint8_t* tile, const ScParams& sp, int lane) {
  constexpr int R = (1 << (B - 1)) - 1;
  using G = ScGeom<B>;
  const uint8_t* rec = tile + (lane >> 3) * G::kRecordBytes;
  uint32_t code[2][4], scale[2];
  sc_get_stream<B>(rec + 2 * (lane & 7) * G::kChunkBytes, code[0], code[1], scale[0], scale[1]);
  sc_decode_lane<MEE, ADD>(v, code, scale, sc_unit_at(rec + 16 * G::kChunkBytes), sp.lut, R);
}

// shared-memory tile <-> global record area, 8 bytes per lane per trip
template <int B>
__device__ __forceinline__ void sc_copy_out(uint8_t* dst, const uint8_t* tile, int lane) {
  constexpr int n8 = ScGeom<B>::kBlockBytes / 8;
  for (int i = lane; i < n8; i += 32)
    reinterpret_cast<unsigned long long*>(dst)[i] = reinterpret_cast<const unsigned long long*>(tile)[i];
}
template <int B>
__device__ __forceinline__ void sc_copy_in(uint8_t* tile, const uint8_t* src, int lane) {
  constexpr int n8 = ScGeom<B>::kBlockBytes / 8;
  for (int i = lane; i < n8; i += 32)
    reinterpret_cast<unsigned long long*>(tile)[i] = __ldcg(reinterpret_cast<const unsigned long long*>(src) + i);
}

// ---- mixed widths: every superchunk of a block has its own code width (2, 4 or 8) -----------------
//
// Per block the host side supplies `wpack` (byte j = width of superchunk j) and the block's byte offset
// inside the message (a prefix sum over the blocks' record bytes; any four records add up to a multiple of
// 8 bytes because 82, 146 and 274 are all 2 mod 8).  The arithmetic per superchunk is the fixed-width
// codec's, operation for operation, with the width as a run-time value: a record written here equals the
// record the fixed-width codec of that width writes for the same block, tag and step.
//
// Constant table (fp32, device): [0..2] lattice_max, [4..6] c1, [8..10] c2 for widths 2, 4, 8 (index
// log2(width) - 1); decode levels of width 2 at [16..20), width 4 at [20..36), width 8 at [36..292).
constexpr int kScMixTableFloats = 292;

__device__ __forceinline__ int sc_rec_bytes(int b) { return 16 * (2 * b + 1) + 2; }
__device__ __forceinline__ int sc_mix_block_bytes(uint32_t wpack) {
  return sc_rec_bytes(wpack & 0xFF) + sc_rec_bytes((wpack >> 8) & 0xFF) + sc_rec_bytes((wpack >> 16) & 0xFF) +
         sc_rec_bytes((wpack >> 24) & 0xFF);
}
__device__ __forceinline__ int sc_mix_slot(int b) { return b == 2 ? 0 : (b == 4 ? 1 : 2); }
__device__ __forceinline__ int sc_mix_lut_base(int b) { return b == 2 ? 16 : (b == 4 ? 20 : 36); }

__device__ __forceinline__ int sc_mix_rec_base(uint32_t wpack, int g) {
  int base = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (i < g) base += sc_rec_bytes((wpack >> (8 * i)) & 0xFF);
  return base;
}

// `table` is the constant table, in shared memory
template <bool MEE>
__device__ __forceinline__ void sc_encode_block_mix(const float (&v)[32], uint8_t* tile, const float* table,
                                                    uint32_t wpack, uint32_t first_call, uint32_t tag, uint32_t step,
                                                    uint32_t k0, uint32_t k1, int lane) {
  const int g = lane >> 3;
  const int B = static_cast<int>((wpack >> (8 * g)) & 0xFF);
  const int ti = sc_mix_slot(B), chunk_bytes = 2 * B + 1;
  uint32_t code[2][4], scale[2];
  __nv_bfloat16 unit;
  sc_encode_lane<MEE>(v, table[ti], MEE ? table[4 + ti] : 1.0f, MEE ? table[8 + ti] : 1.0f, (1 << (B - 1)) - 1, first_call,
                      tag, step, k0, k1, lane, code, scale, unit);
  uint8_t* rec = tile + sc_mix_rec_base(wpack, g);
  uint8_t* at = rec + 2 * (lane & 7) * chunk_bytes;
  if (B == 8) sc_put_stream<8>(at, code[0], code[1], scale[0], scale[1]);
  else if (B == 4) sc_put_stream<4>(at, code[0], code[1], scale[0], scale[1]);
  else sc_put_stream<2>(at, code[0], code[1], scale[0], scale[1]);
  if ((lane & 7) == 0) *reinterpret_cast<__nv_bfloat16*>(rec + 16 * chunk_bytes) = unit;
}

template <bool MEE, bool ADD>
__device__ __forceinline__ void sc_decode_block_mix(float (&v)[32], const uint8_t* tile, const float* table,
                                                    uint32_t wpack, int lane) {
  const int g = lane >> 3;
  const int B = static_cast<int>((wpack >> (8 * g)) & 0xFF);
  const int chunk_bytes = 2 * B + 1;
  const uint8_t* rec = tile + sc_mix_rec_base(wpack, g);
  const uint8_t* at = rec + 2 * (lane & 7) * chunk_bytes;
  uint32_t code[2][4], scale[2];
  if (B == 8) sc_get_stream<8>(at, code[0], code[1], scale[0], scale[1]);
  else if (B == 4) sc_get_stream<4>(at, code[0], code[1], scale[0], scale[1]);
  else sc_get_stream<2>(at, code[0], code[1], scale[0], scale[1]);
  sc_decode_lane<MEE, ADD>(v, code, scale, sc_unit_at(rec + 16 * chunk_bytes), table + sc_mix_lut_base(B), (1 << (B - 1)) - 1);
}

__device__ __forceinline__ void sc_copy_out_n(uint8_t* dst, const uint8_t* tile, int n8, int lane) {
  for (int i = lane; i < n8; i += 32)
    reinterpret_cast<unsigned long long*>(dst)[i] = reinterpret_cast<const unsigned long long*>(tile)[i];
}
__device__ __forceinline__ void sc_copy_in_n(uint8_t* tile, const uint8_t* src, int n8, int lane) {
  for (int i = lane; i < n8; i += 32)
    reinterpret_cast<unsigned long long*>(tile)[i] = __ldcg(reinterpret_cast<const unsigned long long*>(src) + i);
}

}  // namespace dq
