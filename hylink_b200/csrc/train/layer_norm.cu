// Layer norm backward with the add of the residual gradient, for rows up to kMaxNormWidth wide.
//
// Bound by memory: a warp owns a row, keeps it in registers (lane l holds columns 256 c + 8 l .. + 7 of chunk c, one
// 16-byte packet each) and touches every element once. The residual gradient is added on the way out (separately: two
// tensors read, one written). Three things are summed over the rows: dgamma, dbeta, and dx itself, whose column sums
// are the bias gradient of the linear layer below. The rows of a lane's columns pass through its registers anyway, so
// the sums cost no memory traffic but a partial per CTA.
// 8192 x 1024, bf16, B200: 25.8 us; as separate kernels (input gradient, parameter gradients, residual add, bias
// gradient) 17 + 42 + 8 + 8 us.
#include "train/train_device.cuh"
#include "train/train_kernels.h"

namespace hl {
namespace train {

constexpr int kBwdThreads = 256;

// One CTA of eight warps per SM, every warp walking its rows with the next row's packets already on their way: the
// three column sums take 24 registers per chunk, so at width 1024 there is room for one such CTA and the loads in
// flight have to come from the look-ahead, not from more warps.
template <typename T, int V, bool kResidual>
__global__ void __launch_bounds__(kBwdThreads, 1) kLayerNormBackward(const T* __restrict__ dh, const T* __restrict__ x,
                                                                     const float* __restrict__ mean, const float* __restrict__ rstd,
                                                                     const T* __restrict__ gamma, const T* __restrict__ residual,
                                                                     T* __restrict__ dx, float* __restrict__ partials, int64_t rows, int width) {
  extern __shared__ float s_sum[];   // [warps][width]
  constexpr int kWarps = kBwdThreads / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float a_gamma[V][8], a_beta[V][8], a_dx[V][8];
#pragma unroll
  for (int c = 0; c < V; ++c)
#pragma unroll
    for (int i = 0; i < 8; ++i) a_gamma[c][i] = a_beta[c][i] = a_dx[c][i] = 0.f;
  const int64_t stride = (int64_t)gridDim.x * kWarps;
  int64_t row = (int64_t)blockIdx.x * kWarps + warp;
  uint4 nd[V], nx[V], nr[V];
  float n_mu = 0.f, n_r = 0.f;
  auto fetch = [&](int64_t at) {
    if (at >= rows) return;
#pragma unroll
    for (int c = 0; c < V; ++c) {
      const int col = c * 256 + lane * 8;
      if (col < width) {
        nd[c] = *reinterpret_cast<const uint4*>(dh + at * width + col);
        nx[c] = *reinterpret_cast<const uint4*>(x + at * width + col);
        if (kResidual) nr[c] = *reinterpret_cast<const uint4*>(residual + at * width + col);
      }
    }
    n_mu = mean[at];
    n_r = rstd[at];
  };
  fetch(row);
  for (; row < rows; row += stride) {
    uint4 pd[V], px[V], pr[V];
#pragma unroll
    for (int c = 0; c < V; ++c) {
      pd[c] = nd[c];
      px[c] = nx[c];
      if (kResidual) pr[c] = nr[c];
    }
    const float mu = n_mu, r = n_r;
    fetch(row + stride);
    float c1 = 0.f, c2 = 0.f;
#pragma unroll
    for (int c = 0; c < V; ++c) {
      const int col = c * 256 + lane * 8;
      if (col < width) {
        float d[8], f[8], g[8];
        unpack8<T>(pd[c], d);
        unpack8<T>(px[c], f);
        unpack8<T>(*reinterpret_cast<const uint4*>(gamma + col), g);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float xh = (f[i] - mu) * r;
          a_gamma[c][i] += d[i] * xh;
          a_beta[c][i] += d[i];
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
        unpack8<T>(pd[c], d);
        unpack8<T>(px[c], f);
        unpack8<T>(*reinterpret_cast<const uint4*>(gamma + col), g);
#pragma unroll
        for (int i = 0; i < 8; ++i) d[i] = r * (d[i] * g[i] - c1 - (f[i] - mu) * r * c2);
        if (kResidual) {
          unpack8<T>(pr[c], f);
#pragma unroll
          for (int i = 0; i < 8; ++i) d[i] += f[i];
        }
        const uint4 p = pack8<T>(d);
        *reinterpret_cast<uint4*>(dx + row * width + col) = p;
        unpack8<T>(p, d);
#pragma unroll
        for (int i = 0; i < 8; ++i) a_dx[c][i] += d[i];
      }
    }
  }
  auto flush = [&](const float(&acc)[V][8], int which) {
    __syncthreads();
#pragma unroll
    for (int c = 0; c < V; ++c) {
      const int col = c * 256 + lane * 8;
      if (col < width) {
        float4* p = reinterpret_cast<float4*>(s_sum + warp * width + col);
        p[0] = make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
        p[1] = make_float4(acc[c][4], acc[c][5], acc[c][6], acc[c][7]);
      }
    }
    __syncthreads();
    float* dst = partials + ((int64_t)which * gridDim.x + blockIdx.x) * width;
    for (int col = threadIdx.x; col < width; col += kBwdThreads) {
      float t = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) t += s_sum[w * width + col];
      dst[col] = t;
    }
  };
  flush(a_gamma, 0);
  flush(a_beta, 1);
  flush(a_dx, 2);
}

int layerNormPartials(int64_t rows) {
  const int64_t want = (rows + kBwdThreads / 32 - 1) / (kBwdThreads / 32);
  return (int)(want < 148 ? (want < 1 ? 1 : want) : 148);
}

hlResult_t layerNormBackward(int dt, const void* dh, const void* x, const float* mean, const float* rstd, const void* gamma,
                             const void* residual, void* dx, float* partials, int64_t rows, int width, cudaStream_t s) {
  if (width % 8 || width < 8 || width > kMaxNormWidth) return fail(hlUnsupported, "layer norm: width %d", width);
  const unsigned blocks = (unsigned)layerNormPartials(rows);
  const size_t smem = (size_t)(kBwdThreads / 32) * width * sizeof(float);   // at most 32 KiB
  HL_HALF_SWITCH(dt, T, {
    auto go = [&](auto kern) {
      kern<<<blocks, kBwdThreads, smem, s>>>((const T*)dh, (const T*)x, mean, rstd, (const T*)gamma, (const T*)residual, (T*)dx, partials, rows, width);
    };
    switch ((width + 255) / 256) {
      case 1: residual ? go(kLayerNormBackward<T, 1, true>) : go(kLayerNormBackward<T, 1, false>); break;
      case 2: residual ? go(kLayerNormBackward<T, 2, true>) : go(kLayerNormBackward<T, 2, false>); break;
      case 3: residual ? go(kLayerNormBackward<T, 3, true>) : go(kLayerNormBackward<T, 3, false>); break;
      default: residual ? go(kLayerNormBackward<T, 4, true>) : go(kLayerNormBackward<T, 4, false>); break;
    }
  });
  return launched("layer norm backward");
}

}  // namespace train
}  // namespace hl
