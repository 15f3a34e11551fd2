// AdamW on this rank's shard of the parameters, one pass.
//
// Bound by memory: with 16-bit weights and an fp32 master copy a parameter costs 28 bytes (gradient in, master and
// both moments in and out, weight out) and fifteen operations. As separate tensor operations the same update reads
// and writes about 120 bytes. A thread owns eight elements: every access is a 16-byte packet, and all seven loads of
// a group are in flight before the first is used.
#include "train/train_device.cuh"
#include "train/train_kernels.h"

namespace hl {
namespace train {

// Eight elements of type T from / to fp32.
template <typename T> struct Group8 {
  static __device__ __forceinline__ void load(const T* p, float* f) { unpack8<T>(*reinterpret_cast<const uint4*>(p), f); }
  static __device__ __forceinline__ void store(T* p, const float* f) { *reinterpret_cast<uint4*>(p) = pack8<T>(f); }
};
template <> struct Group8<float> {
  static __device__ __forceinline__ void load(const float* p, float* f) {
    reinterpret_cast<float4*>(f)[0] = reinterpret_cast<const float4*>(p)[0];
    reinterpret_cast<float4*>(f)[1] = reinterpret_cast<const float4*>(p)[1];
  }
  static __device__ __forceinline__ void store(float* p, const float* f) {
    reinterpret_cast<float4*>(p)[0] = reinterpret_cast<const float4*>(f)[0];
    reinterpret_cast<float4*>(p)[1] = reinterpret_cast<const float4*>(f)[1];
  }
};

template <typename T, bool kMaster>
__global__ void __launch_bounds__(256) kShardedAdamW(const T* __restrict__ grad, T* __restrict__ weight, float* __restrict__ master,
                                                     float* __restrict__ m, float* __restrict__ v, int64_t groups, const AdamWArgs a) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= groups) return;
  alignas(16) float g[8], w[8], fm[8], fv[8];
  Group8<T>::load(grad + i * 8, g);
  if (kMaster) Group8<float>::load(master + i * 8, w);
  else Group8<T>::load(weight + i * 8, w);
  Group8<float>::load(m + i * 8, fm);
  Group8<float>::load(v + i * 8, fv);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float gk = g[k] / a.ranks;
    fm[k] = fm[k] * a.beta1 + a.rest1 * gk;
    fv[k] = fv[k] * a.beta2 + a.rest2 * gk * gk;
    const float denom = sqrtf(fv[k] / a.correction2) + a.eps;
    w[k] = w[k] * a.keep - a.step * (fm[k] / denom);
  }
  Group8<float>::store(m + i * 8, fm);
  Group8<float>::store(v + i * 8, fv);
  if (kMaster) Group8<float>::store(master + i * 8, w);
  Group8<T>::store(weight + i * 8, w);
}

hlResult_t shardedAdamW(int dt, const void* grad, void* weight, float* master, float* m, float* v, int64_t count, const AdamWArgs& a,
                        cudaStream_t s) {
  if (count % 8) return fail(hlInvalidArgument, "sharded AdamW: %lld elements", (long long)count);
  if (count == 0) return hlSuccess;
  const int64_t groups = count / 8;
  const unsigned blocks = (unsigned)((groups + 255) / 256);
  if (dt == hlFloat32) {
    if (master) return fail(hlInvalidArgument, "sharded AdamW: fp32 weights are their own master");
    kShardedAdamW<float, false><<<blocks, 256, 0, s>>>((const float*)grad, (float*)weight, nullptr, m, v, groups, a);
  } else {
    HL_HALF_SWITCH(dt, T, {
      if (master) kShardedAdamW<T, true><<<blocks, 256, 0, s>>>((const T*)grad, (T*)weight, master, m, v, groups, a);
      else kShardedAdamW<T, false><<<blocks, 256, 0, s>>>((const T*)grad, (T*)weight, nullptr, m, v, groups, a);
    });
  }
  return launched("sharded AdamW");
}

}  // namespace train
}  // namespace hl
