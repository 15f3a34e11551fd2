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
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
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
__device__ __forceinline__ float exp2Fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float reciprocalFast(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// gelu in its tanh form. 0.5 (1 + tanh z) = 1 / (1 + exp(-2 z)) =: s, and 1 - s = exp(-2 z) s; -2 z log2(e) = u (kGate + kGate3 u^2).
// The special-function unit is what bounds this (8 cycles a warp and operation, where the rest is 9), so four values share one
// reciprocal: 1.25 operations a value instead of 2. tanhf costs more than either: 8 x 1280 x 4096 in bf16, forward
// 37.7 us with it and 32.3 with an exponential and a reciprocal each, backward 60.4 and 50.4. The exponent is capped so that four
// factors of up to 1 + 2^30 stay finite; from kSlopeFar down, where the cap is felt, values go one by one.
constexpr float kGate = -2.302208198f, kGate3 = -0.1029432397f, kGateCap = 30.f, kSlopeFar = -5.25f;
struct GeluGates {
  uint64_t e[2], s[2];   // exp(-2 z) and 1 / (1 + exp(-2 z)) of four values
};
__device__ __forceinline__ GeluGates geluGates(uint64_t u0, uint64_t u1) {
  const uint64_t k1 = pair(kGate, kGate), k3 = pair(kGate3, kGate3), one = pair(1.f, 1.f);
  float a, b, c, d, p, q;
  unpair(mul2(u0, fma2(mul2(u0, u0), k3, k1)), a, b);
  unpair(mul2(u1, fma2(mul2(u1, u1), k3, k1)), c, d);
  GeluGates g;
  g.e[0] = pair(exp2Fast(fminf(a, kGateCap)), exp2Fast(fminf(b, kGateCap)));
  g.e[1] = pair(exp2Fast(fminf(c, kGateCap)), exp2Fast(fminf(d, kGateCap)));
  const uint64_t x0 = add2(g.e[0], one), x1 = add2(g.e[1], one);
  unpair(mul2(x0, x1), p, q);
  const float r = reciprocalFast(p * q);
  const uint64_t inverse = mul2(pair(r, r), pair(q, p));
  g.s[0] = mul2(inverse, x1);
  g.s[1] = mul2(inverse, x0);
  return g;
}
// Far below zero the sum 1 + tanh z cancels in fp32; there the plain formula is kept, so that results stay those of torch's own
// kernel bit for bit in bf16 (checked over all values).
constexpr float kGeluFar = -2.5f;
static __device__ __noinline__ float geluFar(float u) { return 0.5f * u * (1.f + tanhf(0.7978845608028654f * (u + 0.044715f * u * u * u))); }
// f = gelu(f), N a multiple of four. One branch for all of them: a branch per value would have them wait for one another.
template <int N>
__device__ __forceinline__ void geluAll(float* f) {
  float out[N], least = f[0];
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const uint64_t u0 = pair(f[i], f[i + 1]), u1 = pair(f[i + 2], f[i + 3]);
    const GeluGates g = geluGates(u0, u1);
    unpair(mul2(u0, g.s[0]), out[i], out[i + 1]);
    unpair(mul2(u1, g.s[1]), out[i + 2], out[i + 3]);
    least = fminf(least, fminf(fminf(f[i], f[i + 1]), fminf(f[i + 2], f[i + 3])));
  }
  if (!(least >= kGeluFar)) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (f[i] < kGeluFar) out[i] = geluFar(f[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) f[i] = out[i];
}
static __device__ __noinline__ float geluSlopeFar(float u) {
  const float e = exp2Fast(fminf(u * (kGate + kGate3 * u * u), 115.f)), s = reciprocalFast(1.f + e);
  return s + u * s * (e * s) * (1.5957691216f * (1.f + 3.f * 0.044715f * u * u));
}
// d *= gelu'(u): s + u s (1 - s) 2 dz/du. N a multiple of four.
template <int N>
__device__ __forceinline__ void timesGeluSlope(float* d, const float* u) {
  const uint64_t c1 = pair(1.5957691216f, 1.5957691216f), c3 = pair(1.5957691216f * 3.f * 0.044715f, 1.5957691216f * 3.f * 0.044715f);
  float out[N], least = u[0];
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const uint64_t v[2] = {pair(u[i], u[i + 1]), pair(u[i + 2], u[i + 3])};
    const GeluGates g = geluGates(v[0], v[1]);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint64_t slope = fma2(mul2(mul2(v[k], g.s[k]), mul2(g.e[k], g.s[k])), fma2(mul2(v[k], v[k]), c3, c1), g.s[k]);
      unpair(mul2(slope, pair(d[i + 2 * k], d[i + 2 * k + 1])), out[i + 2 * k], out[i + 2 * k + 1]);
    }
    least = fminf(least, fminf(fminf(u[i], u[i + 1]), fminf(u[i + 2], u[i + 3])));
  }
  if (!(least >= kSlopeFar)) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (u[i] < kSlopeFar) out[i] = d[i] * geluSlopeFar(u[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) d[i] = out[i];
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
