// Device helpers of the training-step kernels: 16-byte packets of eight 16-bit floats, warp sums.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

#include "core/core.h"

namespace hl {
namespace train {

template <typename T> struct Half2Of;
template <> struct Half2Of<__nv_bfloat16> {
  using type = __nv_bfloat162;
  static __device__ __forceinline__ float2 up(type v) { return __bfloat1622float2(v); }
  static __device__ __forceinline__ type down(float a, float b) { return __floats2bfloat162_rn(a, b); }
};
template <> struct Half2Of<__half> {
  using type = __half2;
  static __device__ __forceinline__ float2 up(type v) { return __half22float2(v); }
  static __device__ __forceinline__ type down(float a, float b) { return __floats2half2_rn(a, b); }
};

template <typename T> __device__ __forceinline__ void unpack8(const uint4& p, float* f) {
  using H = Half2Of<T>;
  const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = H::up(*reinterpret_cast<const typename H::type*>(&w[i]));
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
  }
}
template <typename T> __device__ __forceinline__ uint4 pack8(const float* f) {
  using H = Half2Of<T>;
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const typename H::type v = H::down(f[2 * i], f[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&v);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ float warpSum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warpMax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Dispatch on the 16-bit element type.
#define HL_HALF_SWITCH(dt, T, ...)                                                        \
  do {                                                                                    \
    if ((dt) == hlBfloat16) { using T = __nv_bfloat16; __VA_ARGS__; }                     \
    else if ((dt) == hlFloat16) { using T = __half; __VA_ARGS__; }                        \
    else return fail(hlUnsupported, "training kernels take fp16 and bf16, not type %d", (int)(dt)); \
  } while (0)

static inline hlResult_t launched(const char* what) {
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? hlSuccess : fail(hlDeviceError, "%s launch: %s", what, cudaGetErrorString(e));
}

}  // namespace train
}  // namespace hl
