// Shared helpers for the dionw_b200 CUDA library (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>

#include "../../include/dionw_b200.h"

namespace dionw {

// Records the message returned by dionw_last_error() for the calling thread.
void set_error(const char* fmt, ...);

// Device-side status word: 0 while every bounded wait inside a kernel ended
// normally.  A kernel whose wait ran out stores a non-zero code here and leaves
// through its normal teardown path (no trap, the context stays usable).
int* device_status_word();

inline int check_cuda(cudaError_t err, const char* what) {
  if (err == cudaSuccess) return DIONW_OK;
  set_error("%s: %s", what, cudaGetErrorString(err));
  return DIONW_ERR_CUDA;
}

#define DIONW_CUDA(expr)                                   \
  do {                                                     \
    int _status = ::dionw::check_cuda((expr), #expr);      \
    if (_status != DIONW_OK) return _status;               \
  } while (0)

#define DIONW_REQUIRE(cond, ...)                           \
  do {                                                     \
    if (!(cond)) {                                         \
      ::dionw::set_error(__VA_ARGS__);                     \
      return DIONW_ERR_ARGUMENT;                           \
    }                                                      \
  } while (0)

// Adds one to the library's count of kernel launches (dionw_launch_count()).
void count_launch();

inline int launch_status(const char* what) {
  count_launch();
  return check_cuda(cudaGetLastError(), what);
}

inline int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

// kCount floats, and kCount 2-byte words, as one access each: streamed past the caches.
template <int kCount>
struct Span;
template <>
struct Span<4> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[4]) {
    const float4 q = __ldcs(reinterpret_cast<const float4*>(p));
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[4]) {
    __stcs(reinterpret_cast<float4*>(p), make_float4(v[0], v[1], v[2], v[3]));
  }
  static __device__ __forceinline__ void load(const uint16_t* p, uint32_t (&h)[4]) {
    const uint2 q = __ldcs(reinterpret_cast<const uint2*>(p));
    h[0] = q.x & 0xFFFFu; h[1] = q.x >> 16; h[2] = q.y & 0xFFFFu; h[3] = q.y >> 16;
  }
  static __device__ __forceinline__ void store(uint16_t* p, const uint32_t (&h)[4]) {
    __stcs(reinterpret_cast<uint2*>(p), make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16)));
  }
};
template <>
struct Span<2> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[2]) {
    const float2 q = __ldcs(reinterpret_cast<const float2*>(p));
    v[0] = q.x; v[1] = q.y;
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[2]) {
    __stcs(reinterpret_cast<float2*>(p), make_float2(v[0], v[1]));
  }
  static __device__ __forceinline__ void load(const uint16_t* p, uint32_t (&h)[2]) {
    const uint32_t q = __ldcs(reinterpret_cast<const unsigned int*>(p));
    h[0] = q & 0xFFFFu; h[1] = q >> 16;
  }
  static __device__ __forceinline__ void store(uint16_t* p, const uint32_t (&h)[2]) {
    __stcs(reinterpret_cast<unsigned int*>(p), h[0] | (h[1] << 16));
  }
};
template <>
struct Span<1> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[1]) { v[0] = __ldcs(p); }
  static __device__ __forceinline__ void store(float* p, const float (&v)[1]) { __stcs(p, v[0]); }
  static __device__ __forceinline__ void load(const uint16_t* p, uint32_t (&h)[1]) { h[0] = __ldcs(p); }
  static __device__ __forceinline__ void store(uint16_t* p, const uint32_t (&h)[1]) { __stcs(p, uint16_t(h[0])); }
};

// Elements of one access to rows of `cols` floats and rows of 2-byte words `ld` apart, both from 16-byte (words:
// 8-byte) boundaries on: what divides every row's start.
inline int span_of(long long cols, long long ld) { return cols % 4 == 0 && ld % 4 == 0 ? 4 : cols % 2 == 0 && ld % 2 == 0 ? 2 : 1; }

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <typename T>
__device__ __forceinline__ float to_float(T v);
template <>
__device__ __forceinline__ float to_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

}  // namespace dionw
