// Common definitions for the B200 LES library: complex type, field layout,
// error handling and the device status word.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <string>
#include <stdexcept>

namespace les {

// Sentinel used by the reference for undefined nodes (parameters_IO.f90:49).
constexpr double BOGUS = -1.23456789e20;
constexpr double KVONK = 0.4;

template <typename T>
struct __align__(2 * sizeof(T)) cplx {
  T x, y;
};

template <typename T>
__device__ __forceinline__ cplx<T> cmul(cplx<T> a, cplx<T> b) {
  return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
template <typename T>
__device__ __forceinline__ cplx<T> cmulc(cplx<T> a, cplx<T> b) {  // a * conj(b)
  return {a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y};
}
template <typename T>
__device__ __forceinline__ cplx<T> cadd(cplx<T> a, cplx<T> b) { return {a.x + b.x, a.y + b.y}; }
template <typename T>
__device__ __forceinline__ cplx<T> csub(cplx<T> a, cplx<T> b) { return {a.x - b.x, a.y - b.y}; }
template <typename T>
__device__ __forceinline__ cplx<T> cscale(cplx<T> a, T s) { return {a.x * s, a.y * s}; }
// i * k * a, written as (0 + i k) * (ax + i ay) the way the reference's
// eye*kkx*f_hat evaluates it.
template <typename T>
__device__ __forceinline__ cplx<T> ik_mul(T k, cplx<T> a) {
  return {T(0) * a.x - k * a.y, T(0) * a.y + k * a.x};
}

// Quotient and remainder of non-negative offsets below 2^32 (every field and
// fine-grid buffer of a supported grid; the state checks its sizes when it is
// created) in 32-bit unsigned arithmetic: a 64-bit division is a long
// software sequence on the GPU, and these sit in per-row and per-point paths.
__device__ __forceinline__ int udiv32(long n, long d) { return int(unsigned(n) / unsigned(d)); }
__device__ __forceinline__ int umod32(long n, long d) { return int(unsigned(n) % unsigned(d)); }

// n / d for 0 <= n < 2^31 and a divisor that the host knows, by the multiply,
// add and shift of Granlund and Montgomery (PLDI 1994): a division by a
// run-time divisor is some twenty dependent instructions, and the spectral
// passes do several in a row where a block's other warps wait for the result.
struct FastDiv {
  unsigned m, s;
  __device__ __forceinline__ int operator()(long n) const { return int((__umulhi(unsigned(n), m) + unsigned(n)) >> s); }
};
inline FastDiv fast_div(long d) {
  FastDiv f;
  f.s = 0;
  while ((1l << f.s) < d) ++f.s;
  f.m = unsigned(((1ull << 32) * ((1ull << f.s) - (unsigned long long)d)) / (unsigned long long)d + 1);
  return f;
}

// Device status bits (read back by les_get_status).
enum StatusBits : unsigned {
  ST_NAN = 1u << 0,          // NaN in the velocity (LES_engine.f90:583-616)
  ST_PIVOT = 1u << 1,        // zero pivot in the tridiagonal solve (compute_pressure.f90:411-418)
  ST_MLP_RANGE = 1u << 2,    // learned closure saw inputs outside its training range
  ST_BAD_ARG = 1u << 3,      // kernel argument check failed
  ST_MLP_WAIT = 1u << 4,     // a closure kernel's tensor-core wait ran out
  ST_COPY_WAIT = 1u << 5,    // a spectral pass's bulk-copy wait ran out
};

struct CudaError : std::runtime_error {
  int code;
  CudaError(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

// Status of a failed CUDA call: 3 (the reference's out-of-memory code) for an
// allocation failure, 4 for any other CUDA error.  Errors the CUDA runtime
// marks as sticky (a device fault: illegal address, launch failure, ...)
// leave the context unusable; the message says so.
inline int cuda_status_code(cudaError_t e) { return e == cudaErrorMemoryAllocation ? 3 : 4; }
inline bool cuda_error_is_sticky(cudaError_t e) {
  switch (e) {
    case cudaErrorIllegalAddress: case cudaErrorLaunchFailure: case cudaErrorIllegalInstruction:
    case cudaErrorMisalignedAddress: case cudaErrorInvalidAddressSpace: case cudaErrorInvalidPc:
    case cudaErrorHardwareStackError: case cudaErrorAssert: case cudaErrorLaunchTimeout:
    case cudaErrorECCUncorrectable:
      return true;
    default:
      return false;
  }
}
inline std::string cuda_error_text(const char* call, cudaError_t e) {
  std::string m = std::string(call) + ": " + cudaGetErrorString(e);
  if (cuda_error_is_sticky(e)) m += " (sticky device error: the CUDA context is lost; destroy the states and exit)";
  return m;
}

#define LES_CUDA(call)                                                                          \
  do {                                                                                          \
    cudaError_t e_ = (call);                                                                    \
    if (e_ != cudaSuccess) {                                                                    \
      throw ::les::CudaError(::les::cuda_status_code(e_), ::les::cuda_error_text(#call, e_));   \
    }                                                                                           \
  } while (0)

#define LES_CHECK_LAUNCH() LES_CUDA(cudaGetLastError())

// Dependent launches.  A kernel launched by launch_dep may start as the blocks
// of the kernel in front of it on its stream end, without waiting for the
// whole of it and its memory to settle, and calls dep_wait() before it reads or
// writes anything that another kernel touches.  What stays outside (constant
// tables, shared-memory set-up, the launch itself) overlaps the end of the
// kernel in front; a launch of any other kind waits as usual.  Pointers to
// changing data carry no const __restrict__ in such a kernel: loads through them
// may be moved in front of the wait.  (The x passes' read-only loads, vldg in
// spectral.cuh, are safe: their addresses come from shared memory that is
// filled and synchronised after the wait.)  (Letting the next launch start earlier, as
// soon as all blocks of this one run, slowed large grids: its waiting blocks
// take the room of running ones.)  Per step, us, plain / so / early: 32 x 32 x
// 16 196 / 153 / 175, 64^3 mixed 249 / 207 / 232, 128^3 FP64 1256 / 1215 / 1328,
// 256^3 mixed 3994 / 3912 / 4355.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
inline void launch_dep(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = at;
  c.numAttrs = 1;
  LES_CUDA(cudaLaunchKernelEx(&c, kern, P(args)...));
}

inline int ceil_div(long a, long b) { return int((a + b - 1) / b); }

}  // namespace les
