// Shared helpers of the TT/TR-SVD kernels (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "ttrsvd.h"

namespace ttr {

// Thread-local error message for tt_last_error().
void set_error(int code, const char* fmt, ...);

#define TT_TRY(expr)                  \
  do {                                \
    int st_ = (expr);                 \
    if (st_ != TT_OK) return st_;     \
  } while (0)

#define TT_CUDA(expr)                                                                     \
  do {                                                                                    \
    cudaError_t e_ = (expr);                                                              \
    if (e_ != cudaSuccess) {                                                              \
      ::ttr::set_error(TT_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__, #expr,            \
                       cudaGetErrorString(e_));                                           \
      return TT_ERR_CUDA;                                                                 \
    }                                                                                     \
  } while (0)

#define TT_LAUNCH_CHECK()                                                                 \
  do {                                                                                    \
    cudaError_t e_ = cudaGetLastError();                                                  \
    if (e_ != cudaSuccess) {                                                              \
      ::ttr::set_error(TT_ERR_CUDA, "%s:%d launch: %s", __FILE__, __LINE__,               \
                       cudaGetErrorString(e_));                                           \
      return TT_ERR_CUDA;                                                                 \
    }                                                                                     \
  } while (0)

// Device status word written by kernels whose work can fail (non-convergence, timeouts).
struct DevStatus {
  int code;     // tt_status of the first failure, 0 if none
  int detail;   // kernel-specific detail (sweeps used, stage index, ...)
  int sweeps;   // largest Jacobi sweep count seen
  int pad;
};

__device__ __forceinline__ void dev_fail(DevStatus* st, int code, int detail) {
  if (st) {
    if (atomicCAS(&st->code, 0, code) == 0) st->detail = detail;
  }
}

inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }
inline long long ceil_div_ll(long long a, long long b) { return (a + b - 1) / b; }

// Current device, its multiprocessor count (cached per device), and a once-per-device raise
// of a kernel's dynamic shared-memory limit (cudaFuncSetAttribute acts on the current device
// only).  smem_optin returns TT_OK or TT_ERR_CUDA with the error message set.
int cur_device();
int dev_sms();
int dev_smem_max();  // opt-in shared memory per block of the current device
int smem_optin(const void* fn, size_t bytes);
template <typename K>
inline int smem_optin_k(K* kernel, size_t bytes) {
  return smem_optin(reinterpret_cast<const void*>(kernel), bytes);
}

// Paired FP32 FMA (fma.rn.f32x2: two lanes of an FP32 pair per issue slot, each rounded like
// fmaf) and the moves in and out of a pair.
__device__ __forceinline__ uint64_t f2_dup(float a) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void ffma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// c += a (8 x 4) * b (4 x 8): lane holds a[lane / 4][lane % 4], b[lane % 4][lane / 4], c[lane / 4][2 (lane % 4) ..].
__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// Launch-count accounting (kernels launched by the current library call).
extern thread_local int g_kernel_launches;
inline void count_launch(int n = 1) { g_kernel_launches += n; }

// Asynchronous global -> shared copies (cp.async): 16-byte, and 16- or 4-byte with zero fill when
// `valid` is false (no byte is read then).
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async16z(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(valid ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

}  // namespace ttr
