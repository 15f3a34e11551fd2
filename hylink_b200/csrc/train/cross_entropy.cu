// Mean cross entropy over 16-bit logits, forward and backward, without an fp32 copy of them.
//
// Both directions are bound by memory. Forward reads every logit once: a CTA per row keeps a running maximum and the
// sum of exponentials under it. Backward reads it once more and writes the gradient. The chain of an fp32 copy, a
// log-softmax, the loss and their gradients moves twelve times as much.
// A row starts on a 16-byte boundary (the stride is a multiple of eight elements): the vocabulary is padded for the
// GEMMs on both sides, which run ten times slower on an odd leading dimension.
#include "train/train_device.cuh"
#include "train/train_kernels.h"

namespace hl {
namespace train {

constexpr int kCeThreads = 512;

template <typename T>
__global__ void __launch_bounds__(kCeThreads) kCrossEntropyForward(const T* __restrict__ logits, int64_t stride, const int64_t* __restrict__ targets,
                                                                   int vocab, int64_t ignore_index, float* __restrict__ lse,
                                                                   float* __restrict__ row_loss) {
  __shared__ float s_max[kCeThreads / 32], s_sum[kCeThreads / 32];
  const int64_t row = blockIdx.x;
  const T* p = logits + row * stride;
  const int packets = vocab / 8;
  float m = -INFINITY, s = 0.f;
  auto take = [&](const float* f, int n) {
    float top = f[0];
#pragma unroll
    for (int i = 1; i < 8; ++i)
      if (i < n) top = fmaxf(top, f[i]);
    if (top == -INFINITY) {   // nothing to add, unless one of them is NaN (exp(-inf - -inf) would be, in every case)
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < n && f[i] != -INFINITY) s = NAN;
      return;
    }
    if (top > m) {
      s *= __expf(m - top);
      m = top;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < n) s += __expf(f[i] - m);
  };
  constexpr int U = 4;
  for (int i = threadIdx.x; i < packets; i += kCeThreads * U) {
    uint4 v[U];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (i + k * kCeThreads < packets) v[k] = reinterpret_cast<const uint4*>(p)[i + k * kCeThreads];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (i + k * kCeThreads < packets) {
        float f[8];
        unpack8<T>(v[k], f);
        take(f, 8);
      }
  }
  if (threadIdx.x < vocab - packets * 8) {
    const float f[8] = {(float)p[packets * 8 + threadIdx.x]};
    take(f, 1);
  }
  const float wm = warpMax(m);
  // under a maximum of -inf (no logits, or only -inf and NaN) the sum is zero or NaN already, and inf - inf not to be formed
  s = warpSum(m == -INFINITY ? s : s * __expf(m - wm));
  if ((threadIdx.x & 31) == 0) {
    s_max[threadIdx.x >> 5] = wm;
    s_sum[threadIdx.x >> 5] = s;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const bool in = threadIdx.x < kCeThreads / 32;
    const float wm2 = in ? s_max[threadIdx.x] : -INFINITY;
    const float top = warpMax(wm2);
    const float total = warpSum(!in ? 0.f : (wm2 == -INFINITY ? s_sum[threadIdx.x] : s_sum[threadIdx.x] * __expf(wm2 - top)));
    if (threadIdx.x == 0) {
      const float z = top + logf(total);
      const int64_t t = targets[row];
      lse[row] = z;
      row_loss[row] = t == ignore_index ? 0.f : (t < 0 || t >= vocab ? NAN : z - (float)p[t]);
    }
  }
}

// One CTA: the mean over the rows that count, in a fixed order.
__global__ void __launch_bounds__(1024) kMeanLoss(const float* __restrict__ row_loss, const int64_t* __restrict__ targets, int64_t rows,
                                                  int64_t ignore_index, float* __restrict__ loss) {
  __shared__ float s_sum[32], s_cnt[32];
  float s = 0.f, n = 0.f;
  for (int64_t i = threadIdx.x; i < rows; i += 1024)
    if (targets[i] != ignore_index) {
      s += row_loss[i];
      n += 1.f;
    }
  s = warpSum(s);
  n = warpSum(n);
  if ((threadIdx.x & 31) == 0) {
    s_sum[threadIdx.x >> 5] = s;
    s_cnt[threadIdx.x >> 5] = n;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    s = warpSum(s_sum[threadIdx.x]);
    n = warpSum(s_cnt[threadIdx.x]);
    if (threadIdx.x == 0) {
      loss[0] = s / n;   // no row counts: NaN, as the mean over nothing
      loss[1] = n;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kCeThreads) kCrossEntropyBackward(const T* __restrict__ logits, int64_t stride, const int64_t* __restrict__ targets,
                                                                    int vocab, int64_t ignore_index, const float* __restrict__ lse,
                                                                    const float* __restrict__ loss, const float* __restrict__ grad,
                                                                    T* __restrict__ dlogits) {
  const int64_t row = blockIdx.x;
  const int64_t t = targets[row];
  const float w = t == ignore_index ? 0.f : *grad / loss[1];
  const float z = lse[row];
  const uint4* p = reinterpret_cast<const uint4*>(logits + row * stride);
  uint4* q = reinterpret_cast<uint4*>(dlogits + row * stride);
  const int packets = (int)(stride / 8);
  constexpr int U = 4;
  for (int i = threadIdx.x; i < packets; i += kCeThreads * U) {
    uint4 v[U];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (i + k * kCeThreads < packets) v[k] = p[i + k * kCeThreads];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int j = i + k * kCeThreads;
      if (j < packets) {
        float f[8];
        unpack8<T>(v[k], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          f[e] = w == 0.f ? 0.f : __expf(f[e] - z) * w;
          if (j * 8 + e == t) f[e] -= w;
          if (j * 8 + e >= vocab) f[e] = 0.f;
        }
        q[j] = pack8<T>(f);
      }
    }
  }
}

hlResult_t crossEntropyForward(int dt, const void* logits, int64_t stride, const int64_t* targets, int64_t rows, int vocab, int64_t ignore_index,
                               float* lse, float* row_loss, float* loss, cudaStream_t s) {
  if (stride % 8 || stride < vocab || vocab < 1) return fail(hlInvalidArgument, "cross entropy: stride %lld, vocabulary %d", (long long)stride, vocab);
  if (rows > 0) HL_HALF_SWITCH(dt, T, { kCrossEntropyForward<T><<<(unsigned)rows, kCeThreads, 0, s>>>((const T*)logits, stride, targets, vocab, ignore_index, lse, row_loss); });
  kMeanLoss<<<1, 1024, 0, s>>>(row_loss, targets, rows, ignore_index, loss);
  return launched("cross entropy forward");
}

hlResult_t crossEntropyBackward(int dt, const void* logits, int64_t stride, const int64_t* targets, int64_t rows, int vocab, int64_t ignore_index,
                                const float* lse, const float* loss, const float* grad, void* dlogits, cudaStream_t s) {
  if (stride % 8 || stride < vocab || vocab < 1) return fail(hlInvalidArgument, "cross entropy: stride %lld, vocabulary %d", (long long)stride, vocab);
  if (rows == 0) return hlSuccess;
  HL_HALF_SWITCH(dt, T, {
    kCrossEntropyBackward<T><<<(unsigned)rows, kCeThreads, 0, s>>>((const T*)logits, stride, targets, vocab, ignore_index, lse, loss, grad, (T*)dlogits);
  });
  return launched("cross entropy backward");
}

}  // namespace train
}  // namespace hl
