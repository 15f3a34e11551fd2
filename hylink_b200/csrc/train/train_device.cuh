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

// Two fp32 operations in one instruction.
__device__ __forceinline__ uint64_t pair(float a, float b) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void unpair(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// gelu in its tanh form. 0.5 (1 + tanh z) = 1 / (1 + exp(-2 z)) =: s, and 1 - s = exp(-2 z) s: two special-function operations and no
// cancellation. (tanhf costs more issue slots than the kernels have at memory speed: 8 x 1280 x 4096 in bf16, forward
// 37.7 us with it and 32.3 without, backward 60.4 and 50.4.) The exponent is capped where s no longer matters, so that exp(-2 z) s stays finite.
// A value's result does not depend on the values beside it. (One reciprocal for four values takes a third off the special-function unit's
// work: products with gelu in the layer of 8192 x 1024 70 us instead of 77, with its gradient and dW2 118 instead of 126. But its rounding
// reaches all four: the slope's mean error grew by 1.4, gelu's last bit came and went with the neighbours, and the strip kernel spilled, 73 us
// for 10240 x 4096 instead of 51.)
struct GeluGate {
  float s, rest;
};
__device__ __forceinline__ GeluGate geluGate(float u) {
  const float e = __expf(fminf(-1.5957691216057308f * (u + 0.044715f * u * u * u), 80.f));
  const float s = __fdividef(1.f, 1.f + e);
  return {s, e * s};
}
// Far below zero the sum 1 + tanh z cancels in fp32; there the plain formula is kept, so that results stay those of torch's own
// kernel bit for bit in bf16 (checked over all values).
constexpr float kGeluFar = -2.5f;
__device__ __forceinline__ float geluFarOf(float u) { return 0.5f * u * (1.f + tanhf(0.7978845608028654f * (u + 0.044715f * u * u * u))); }
__device__ __forceinline__ float gelu(float u) {
  if (u < kGeluFar) return geluFarOf(u);
  return u * geluGate(u).s;
}
// The same for N values with one branch for all of them: where a warp's instructions are the bound, a branch per value costs a quarter.
static __device__ __noinline__ float geluFar(float u) { return geluFarOf(u); }
template <int N>
__device__ __forceinline__ void geluAll(float* f) {
  float out[N], least = f[0];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    out[i] = f[i] * geluGate(f[i]).s;
    least = fminf(least, f[i]);
  }
  if (!(least >= kGeluFar)) {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (f[i] < kGeluFar) out[i] = geluFar(f[i]);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) f[i] = out[i];
}
// gelu'(u): s + u s (1 - s) 2 dz/du
__device__ __forceinline__ float geluSlope(float u) {
  const GeluGate q = geluGate(u);
  const float dz = 1.5957691216057308f * (1.f + 3.f * 0.044715f * u * u);
  return q.s + u * q.s * q.rest * dz;
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
