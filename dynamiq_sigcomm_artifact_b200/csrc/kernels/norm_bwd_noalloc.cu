// RMSNorm backward without any allocation: the same kernels as torch.ops.dq.norm_bwd, with the
// per-CTA partial sums of dw kept in a fixed device array of this library instead of a tensor
// obtained from the allocator.  Declaration and usage rules: dq_noalloc.h.  There is no
// counterpart of this entry point in the reference implementation.
#include "dq_noalloc.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "column_sums.cuh"
#include "norm_kernels.cuh"

namespace {

// Scratch shared by every call on a device: [DQ_NOALLOC_MAX_PARTS][hidden] floats, fully
// rewritten by add_norm_bwd_kernel before reduce_arrays_kernel reads it.
static __device__ __align__(256) float g_noalloc_scratch[DQ_NOALLOC_MAX_PARTS * DQ_NOALLOC_MAX_HIDDEN];

constexpr int kMaxDevices = 64;
std::mutex g_mu;
float* g_scratch_addr[kMaxDevices] = {nullptr};  // device address of g_noalloc_scratch, per device
thread_local int t_last_cuda_error = 0;

// In host code `g_noalloc_scratch` is only a handle for the symbol; the address a kernel can
// use has to be asked for, once per device, with that device current.
int scratch_for_current_device(float** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    t_last_cuda_error = static_cast<int>(e != cudaSuccess ? e : cudaErrorInvalidDevice);
    return DQ_NOALLOC_CUDA_ERROR;
  }
  std::lock_guard<std::mutex> lk(g_mu);
  if (g_scratch_addr[dev] == nullptr) {
    float* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) {  // a null address with a success code still is a failure to report
      t_last_cuda_error = static_cast<int>(e != cudaSuccess ? e : cudaErrorInvalidSymbol);
      return DQ_NOALLOC_CUDA_ERROR;
    }
    g_scratch_addr[dev] = p;
  }
  *out = g_scratch_addr[dev];
  return DQ_NOALLOC_OK;
}

template <typename T>
void launch_rows(const void* dy, const void* x, const float* w, const float* rstd, void* dx, float* parts, int rows,
                 int hidden, int grid, cudaStream_t stream) {
  using namespace dq::normk;
  const int nt = norm_group_threads(hidden);
  cudaFuncSetAttribute(add_norm_bwd_kernel<T, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kNormBwdMaxSmem);
  add_norm_bwd_kernel<T, true, false><<<grid, nt * norm_groups(hidden), norm_bwd_smem(hidden), stream>>>(
      static_cast<const T*>(dy), nullptr, false, static_cast<const T*>(x), w, nullptr, rstd, static_cast<T*>(dx), parts,
      rows, hidden, nt);
}

bool bad_ptr(const void* p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15u) != 0; }

}  // namespace

extern "C" int dq_rmsnorm_bwd_noalloc(const void* dy, const void* x, const float* w, const float* rstd, void* dx,
                                      float* dw, int rows, int hidden, int is_bf16, void* stream_ptr) {
  using namespace dq::normk;
  if (hidden <= 0 || hidden > DQ_NOALLOC_MAX_HIDDEN || hidden % 8 != 0) return DQ_NOALLOC_BAD_HIDDEN;
  if (rows <= 0) return DQ_NOALLOC_BAD_ROWS;
  if (bad_ptr(dy) || bad_ptr(x) || bad_ptr(w) || bad_ptr(dx) || bad_ptr(dw) || rstd == nullptr)
    return DQ_NOALLOC_BAD_POINTER;
  float* parts = nullptr;
  const int rc = scratch_for_current_device(&parts);
  if (rc != DQ_NOALLOC_OK) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  (void)cudaGetLastError();  // an error left behind by the caller's earlier launches is not this call's
  int grid = norm_bwd_grid(rows, hidden, dq::device_sms());  // one partial row of `hidden` floats per CTA
  if (grid > DQ_NOALLOC_MAX_PARTS) grid = DQ_NOALLOC_MAX_PARTS;
  if (is_bf16) launch_rows<__nv_bfloat16>(dy, x, w, rstd, dx, parts, rows, hidden, grid, stream);
  else launch_rows<float>(dy, x, w, rstd, dx, parts, rows, hidden, grid, stream);
  dq::reduce_arrays(parts, dw, nullptr, nullptr, 1, grid, hidden, stream);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    t_last_cuda_error = static_cast<int>(e);
    return DQ_NOALLOC_CUDA_ERROR;
  }
  return DQ_NOALLOC_OK;
}

extern "C" const char* dq_noalloc_strerror(int code) {
  switch (code) {
    case DQ_NOALLOC_OK: return "ok";
    case DQ_NOALLOC_BAD_HIDDEN: return "hidden size must be a positive multiple of 8 and at most DQ_NOALLOC_MAX_HIDDEN (2048)";
    case DQ_NOALLOC_BAD_ROWS: return "rows must be positive";
    case DQ_NOALLOC_BAD_POINTER: return "a pointer is null or not 16-byte aligned";
    case DQ_NOALLOC_CUDA_ERROR: return "a CUDA call failed (see dq_noalloc_last_cuda_error)";
    default: return "unknown code";
  }
}

extern "C" int dq_noalloc_last_cuda_error(void) { return t_last_cuda_error; }
