// Layer norm backward with the add of the residual gradient, for rows up to kMaxNormWidth wide.
//
// Bound by memory: a warp owns a row, keeps it in registers (lane l holds columns 256 c + 8 l .. + 7 of chunk c, one
// 16-byte packet each) and touches every element once. The residual gradient is added on the way out (separately: two
// tensors read, one written). Three things are summed over the rows: dgamma, dbeta, and dx itself, whose column sums
// are the bias gradient of the linear layer below. The rows of a lane's columns pass through its registers anyway, so
// the sums cost no memory traffic but a partial per CTA.
// 8192 x 1024, bf16, B200: 17.5 us, 20.0 with the column sums of dx; as separate kernels (input gradient, parameter
// gradients, residual add, bias gradient) 17 + 42 + 8 + 8 us.
#include "train/train_device.cuh"
#include "train/train_kernels.h"

namespace hl {
namespace train {

constexpr int kBwdThreads = 384, kBwdWarps = kBwdThreads / 32, kBwdStages = 3;
constexpr int kRowScalars = 2;   // mean, rstd

__device__ __forceinline__ void cpAsync16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cpAsync4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// One CTA of twelve warps per SM. The column sums take 16 or 24 registers per chunk, which leaves no room to hold the
// next rows: they travel through a ring of three rows per warp in shared memory, where a lane reads back exactly what it
// asked for itself, so nothing has to be synchronised. (With the next row in registers and eight warps the kernel had 48
// KB in flight per SM and took 25.8 us for 8192 x 1024.)
template <typename T, int V, bool kResidual, bool kDx>
__global__ void __launch_bounds__(kBwdThreads, 1) kLayerNormBackward(const T* __restrict__ dh, const T* __restrict__ x,
                                                                     const float* __restrict__ mean, const float* __restrict__ rstd,
                                                                     const T* __restrict__ gamma, const T* __restrict__ residual,
                                                                     T* __restrict__ dx, float* __restrict__ partials, int64_t rows, int width) {
  constexpr int kArrays = kResidual ? 3 : 2, kSums = kDx ? 3 : 2;
  constexpr int kPacketsPerStage = kArrays * V * 32;           // of a warp
  extern __shared__ uint4 s_ring[];                            // [warps][stages][arrays][V][32 lanes], then the row scalars
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4* ring = s_ring + warp * kBwdStages * kPacketsPerStage + lane;
  float* scalars = reinterpret_cast<float*>(s_ring + kBwdWarps * kBwdStages * kPacketsPerStage) + warp * kBwdStages * kRowScalars * 32 + lane;
  uint4 pg[V];
  float acc[kSums][V][8];
#pragma unroll
  for (int c = 0; c < V; ++c) {
    if (c * 256 + lane * 8 < width) pg[c] = *reinterpret_cast<const uint4*>(gamma + c * 256 + lane * 8);
#pragma unroll
    for (int k = 0; k < kSums; ++k)
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[k][c][i] = 0.f;
  }
  const int64_t stride = (int64_t)gridDim.x * kBwdWarps, row0 = (int64_t)blockIdx.x * kBwdWarps + warp;
  auto fetch = [&](int64_t at, int stage) {
    if (at < rows) {
      uint4* to = ring + stage * kPacketsPerStage;
#pragma unroll
      for (int c = 0; c < V; ++c) {
        const int col = c * 256 + lane * 8;
        if (col < width) {
          cpAsync16(to + c * 32, dh + at * width + col);
          cpAsync16(to + (V + c) * 32, x + at * width + col);
          if (kResidual) cpAsync16(to + (2 * V + c) * 32, residual + at * width + col);
        }
      }
      cpAsync4(scalars + stage * kRowScalars * 32, mean + at);
      cpAsync4(scalars + stage * kRowScalars * 32 + 32, rstd + at);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int k = 0; k < kBwdStages - 1; ++k) fetch(row0 + k * stride, k);
  int stage = 0;
  for (int64_t row = row0; row < rows; row += stride) {
    fetch(row + (kBwdStages - 1) * stride, stage == 0 ? kBwdStages - 1 : stage - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(kBwdStages - 1) : "memory");
    const uint4* from = ring + stage * kPacketsPerStage;
    const float mu = scalars[stage * kRowScalars * 32], r = scalars[stage * kRowScalars * 32 + 32];
    float c1 = 0.f, c2 = 0.f;
#pragma unroll
    for (int c = 0; c < V; ++c) {
      if (c * 256 + lane * 8 < width) {
        float d[8], f[8], g[8];
        unpack8<T>(from[c * 32], d);
        unpack8<T>(from[(V + c) * 32], f);
        unpack8<T>(pg[c], g);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float xh = (f[i] - mu) * r;
          acc[0][c][i] += d[i] * xh;
          acc[1][c][i] += d[i];
          c1 += d[i] * g[i];
          c2 += d[i] * g[i] * xh;
        }
      }
    }
    c1 = warpSum(c1) / (float)width;
    c2 = warpSum(c2) / (float)width;
#pragma unroll
    for (int c = 0; c < V; ++c) {
      const int col = c * 256 + lane * 8;
      if (col < width) {
        float d[8], f[8], g[8];
        unpack8<T>(from[c * 32], d);
        unpack8<T>(from[(V + c) * 32], f);
        unpack8<T>(pg[c], g);
#pragma unroll
        for (int i = 0; i < 8; ++i) d[i] = r * (d[i] * g[i] - c1 - (f[i] - mu) * r * c2);
        if (kResidual) {
          unpack8<T>(from[(2 * V + c) * 32], f);
#pragma unroll
          for (int i = 0; i < 8; ++i) d[i] += f[i];
        }
        const uint4 p = pack8<T>(d);
        *reinterpret_cast<uint4*>(dx + row * width + col) = p;
        if constexpr (kDx) {
          unpack8<T>(p, d);
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[2][c][i] += d[i];
        }
      }
    }
    stage = stage == kBwdStages - 1 ? 0 : stage + 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                                             // the ring becomes the place where the warps' sums meet
  float* sums = reinterpret_cast<float*>(s_ring);              // [sums][warps][V * 256]
#pragma unroll
  for (int k = 0; k < kSums; ++k)
#pragma unroll
    for (int c = 0; c < V; ++c) {
      float4* p = reinterpret_cast<float4*>(sums + (k * kBwdWarps + warp) * (V * 256) + c * 256 + lane * 8);
      p[0] = make_float4(acc[k][c][0], acc[k][c][1], acc[k][c][2], acc[k][c][3]);
      p[1] = make_float4(acc[k][c][4], acc[k][c][5], acc[k][c][6], acc[k][c][7]);
    }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kSums; ++k) {
    float* dst = partials + ((int64_t)k * gridDim.x + blockIdx.x) * width;
    for (int col = threadIdx.x; col < width; col += kBwdThreads) {
      float t = 0.f;
#pragma unroll
      for (int w = 0; w < kBwdWarps; ++w) t += sums[(k * kBwdWarps + w) * (V * 256) + col];
      dst[col] = t;
    }
  }
}

int layerNormPartials(int64_t rows) {
  const int64_t want = (rows + kBwdWarps - 1) / kBwdWarps;
  return (int)(want < 148 ? (want < 1 ? 1 : want) : 148);
}

hlResult_t layerNormBackward(int dt, const void* dh, const void* x, const float* mean, const float* rstd, const void* gamma,
                             const void* residual, void* dx, bool dx_sums, float* partials, int64_t rows, int width, cudaStream_t s) {
  if (width % 8 || width < 8 || width > kMaxNormWidth) return fail(hlUnsupported, "layer norm: width %d", width);
  if (dx_sums && !residual) return fail(hlInvalidArgument, "layer norm: column sums of dx go with a residual gradient");
  const unsigned blocks = (unsigned)layerNormPartials(rows);
  HL_HALF_SWITCH(dt, T, {
    auto go = [&](auto kern, int V) {
      // ring and scalars; at width 1024 with a residual 225 KB, of which the sums at the end take 144
      const size_t smem = (size_t)kBwdWarps * kBwdStages * ((residual ? 3 : 2) * V * 512 + kRowScalars * 128);
      cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      kern<<<blocks, kBwdThreads, smem, s>>>((const T*)dh, (const T*)x, mean, rstd, (const T*)gamma, (const T*)residual, (T*)dx, partials, rows, width);
    };
    auto chunks = [&](auto v) {
      constexpr int V = decltype(v)::value;
      if (dx_sums) go(kLayerNormBackward<T, V, true, true>, V);
      else if (residual) go(kLayerNormBackward<T, V, true, false>, V);
      else go(kLayerNormBackward<T, V, false, false>, V);
    };
    switch ((width + 255) / 256) {
      case 1: chunks(std::integral_constant<int, 1>()); break;
      case 2: chunks(std::integral_constant<int, 2>()); break;
      case 3: chunks(std::integral_constant<int, 3>()); break;
      default: chunks(std::integral_constant<int, 4>()); break;
    }
  });
  return launched("layer norm backward");
}

}  // namespace train
}  // namespace hl
