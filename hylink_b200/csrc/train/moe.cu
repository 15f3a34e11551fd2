// Routing, dispatch and combine of a top-1 mixture-of-experts layer with a fixed capacity per expert.
//
// moeRoute       a thread per token: the expert with the largest logit and its softmax probability (the gate)
// moeAssign      a CTA per expert: walks the tokens in order, numbers the expert's own by a scan over the CTA; a token's row is expert * capacity + number, or none beyond the capacity. The CTA also writes
//                the inverse map (row -> token), so that everything after it can go by rows: every row of the dispatch
//                buffer is then written exactly once, empty ones with zeros, and nothing needs clearing or atomics.
// moeGather      rows of the dispatch buffer from the tokens
// moeCombine     y = x + gate * row
// moeRowGradient d row = gate * dy; d gate = <dy, row>
// moeTokenGradient  dx = dy + d row + d logits * router; d logits of the gate's softmax
// All of them are bound by memory (16-byte packets, a warp or more per row). As tensor operations the same layer took
// a one-hot matrix, a scan of it along the tokens in 64-bit integers (1.7 ms for 8192 tokens), sorted index updates
// and eleven host round trips for the sizes of boolean selections.
#include "train/train_device.cuh"
#include "train/train_kernels.h"

namespace hl {
namespace train {

template <typename T>
__global__ void __launch_bounds__(128) kMoeRoute(const T* __restrict__ logits, int tokens, int experts, int* __restrict__ expert,
                                                 float* __restrict__ gate) {
  const int t = blockIdx.x * 128 + threadIdx.x;
  if (t >= tokens) return;
  const T* p = logits + (int64_t)t * experts;
  float best = (float)p[0];
  int at = 0;
  for (int e = 1; e < experts; ++e) {
    const float l = (float)p[e];
    if (l > best) {   // the first of equal ones
      best = l;
      at = e;
    }
  }
  float sum = 0.f;
  for (int e = 0; e < experts; ++e) sum += expf((float)p[e] - best);
  expert[t] = at;
  gate[t] = 1.f / sum;
}

constexpr int kAssignThreads = 1024, kAssignTokens = 4;   // four consecutive tokens per thread and sweep
__global__ void __launch_bounds__(kAssignThreads) kMoeAssign(const int* __restrict__ expert, int tokens, int capacity, int* __restrict__ row_of,
                                                             int* __restrict__ token_of) {
  __shared__ int s_count[kAssignThreads / 32];
  const int e = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base = 0;   // tokens of this expert so far
  for (int t0 = 0; t0 < tokens; t0 += kAssignThreads * kAssignTokens) {
    const int t = t0 + threadIdx.x * kAssignTokens;
    bool mine[kAssignTokens];
    int own = 0;
#pragma unroll
    for (int k = 0; k < kAssignTokens; ++k) {
      mine[k] = t + k < tokens && expert[t + k] == e;
      own += mine[k];
    }
    int scan = own;   // tokens of this warp's lanes up to and including this one
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int k = __shfl_up_sync(0xffffffffu, scan, o);
      if (lane >= o) scan += k;
    }
    if (lane == 31) s_count[warp] = scan;
    __syncthreads();
    int all = s_count[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int k = __shfl_up_sync(0xffffffffu, all, o);
      if (lane >= o) all += k;
    }
    const int before = warp ? __shfl_sync(0xffffffffu, all, warp - 1) : 0;
    all = __shfl_sync(0xffffffffu, all, 31);
    int pos = base + before + scan - own;
#pragma unroll
    for (int k = 0; k < kAssignTokens; ++k)
      if (mine[k]) {
        row_of[t + k] = pos < capacity ? e * capacity + pos : -1;
        if (pos < capacity) token_of[e * capacity + pos] = t + k;
        ++pos;
      }
    base += all;
    __syncthreads();
  }
  for (int k = base + threadIdx.x; k < capacity; k += kAssignThreads) token_of[e * capacity + k] = -1;
}

// A warp per row: dst[row] = src[index[row]], zeros where there is none.
template <int U = 4>
__global__ void __launch_bounds__(256) kMoeGather(const uint4* __restrict__ src, const int* __restrict__ index, uint4* __restrict__ dst, int rows,
                                                  int packets) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int from = index[row];
  uint4* d = dst + (int64_t)row * packets;
  const uint4* s = src + (int64_t)(from < 0 ? 0 : from) * packets;
  for (int i = lane; i < packets; i += 32 * U) {
    uint4 v[U];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (i + k * 32 < packets) v[k] = from < 0 ? make_uint4(0u, 0u, 0u, 0u) : s[i + k * 32];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (i + k * 32 < packets) d[i + k * 32] = v[k];
  }
}

template <typename T>
__global__ void __launch_bounds__(256) kMoeCombine(const T* __restrict__ x, const float* __restrict__ gate, const T* __restrict__ rows,
                                                   const int* __restrict__ row_of, T* __restrict__ y, int tokens, int width) {
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= tokens) return;
  const int row = row_of[t];
  const float g = (float)(T)gate[t];
  constexpr int U = 2;
  for (int c = lane * 8; c < width; c += 256 * U) {
    uint4 a[U], b[U];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (c + k * 256 < width) {
        a[k] = *reinterpret_cast<const uint4*>(x + (int64_t)t * width + c + k * 256);
        if (row >= 0) b[k] = *reinterpret_cast<const uint4*>(rows + (int64_t)row * width + c + k * 256);
      }
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (c + k * 256 < width) {
        if (row >= 0) {
          float f[8], h[8];
          unpack8<T>(a[k], f);
          unpack8<T>(b[k], h);
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] += g * h[i];
          a[k] = pack8<T>(f);
        }
        *reinterpret_cast<uint4*>(y + (int64_t)t * width + c + k * 256) = a[k];
      }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) kMoeRowGradient(const T* __restrict__ dy, const float* __restrict__ gate, const T* __restrict__ rows,
                                                       const int* __restrict__ token_of, T* __restrict__ drows, float* __restrict__ dgate, int n_rows,
                                                       int width) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  const int t = token_of[row];
  T* d = drows + (int64_t)row * width;
  if (t < 0) {
    for (int c = lane * 8; c < width; c += 256) *reinterpret_cast<uint4*>(d + c) = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  const float g = (float)(T)gate[t];
  float dot = 0.f;
  constexpr int U = 2;
  for (int c = lane * 8; c < width; c += 256 * U) {
    uint4 a[U], b[U];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (c + k * 256 < width) {
        a[k] = *reinterpret_cast<const uint4*>(dy + (int64_t)t * width + c + k * 256);
        b[k] = *reinterpret_cast<const uint4*>(rows + (int64_t)row * width + c + k * 256);
      }
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (c + k * 256 < width) {
        float f[8], h[8];
        unpack8<T>(a[k], f);
        unpack8<T>(b[k], h);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          dot += f[i] * h[i];
          f[i] *= g;
        }
        *reinterpret_cast<uint4*>(d + c + k * 256) = pack8<T>(f);
      }
  }
  dot = warpSum(dot);
  if (lane == 0) dgate[t] = dot;
}

// A CTA covers all columns (a thread eight of them) and walks tokens. The router's rows lie in shared memory (in
// registers they cost the occupancy that hides the chain row -> packet: 31 us instead of 25 for 8192 x 1024, eight
// experts). E bounds the experts this variant is compiled for; with kRouter false the router's share is left to a GEMM.
template <typename T, int E, bool kRouter>
__global__ void __launch_bounds__(256) kMoeTokenGradient(const T* __restrict__ dy, const T* __restrict__ drows, const int* __restrict__ row_of,
                                                         const T* __restrict__ logits, const float* __restrict__ gate,
                                                         const float* __restrict__ dgate, const T* __restrict__ router, T* __restrict__ dx,
                                                         T* __restrict__ dlogits, int tokens, int width, int experts) {
  extern __shared__ uint4 s_router[];          // [experts][width / 8]
  const int cols = width / 8;                  // threads of one token
  const int per = blockDim.x / cols;           // tokens side by side
  const int sub = threadIdx.x / cols, col = threadIdx.x - sub * cols, c = col * 8;
  if (kRouter) {
    for (int i = threadIdx.x; i < experts * cols; i += blockDim.x) s_router[i] = reinterpret_cast<const uint4*>(router)[i];
    __syncthreads();
  }
  if (sub >= per) return;
  for (int t = blockIdx.x * per + sub; t < tokens; t += gridDim.x * per) {
    const int row = row_of[t];
    const uint4 a = dy ? *reinterpret_cast<const uint4*>(dy + (int64_t)t * width + c) : make_uint4(0u, 0u, 0u, 0u);
    float f[8];
    unpack8<T>(a, f);
    if (row >= 0) {
      float h[8];
      unpack8<T>(*reinterpret_cast<const uint4*>(drows + (int64_t)row * width + c), h);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] += h[i];
    }
    // gate = p_top: d logit_e = d gate * p_top * ([e is top] - p_e), with p_e = exp(l_e - l_top) * p_top. No gradient
    // for a token whose gate was not used.
    const T* l = logits + (int64_t)t * experts;
    const float g = gate[t], dg = row >= 0 ? dgate[t] * g : 0.f;
    if (kRouter) {
      float lv[E], top = -INFINITY;
      int at = 0;
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (e < experts) {
          lv[e] = (float)l[e];
          if (lv[e] > top || e == 0) {
            top = lv[e];
            at = e;
          }
        }
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (e < experts) {
          const T d = (T)(dg * ((e == at ? 1.f : 0.f) - __expf(lv[e] - top) * g));
          if (c == 0) dlogits[(int64_t)t * experts + e] = d;
          float w[8];
          unpack8<T>(s_router[e * cols + col], w);
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] += (float)d * w[i];
        }
    } else if (c == 0) {
      float top = (float)l[0];
      int at = 0;
      for (int e = 1; e < experts; ++e)
        if ((float)l[e] > top) {
          top = (float)l[e];
          at = e;
        }
      for (int e = 0; e < experts; ++e)
        dlogits[(int64_t)t * experts + e] = (T)(dg * ((e == at ? 1.f : 0.f) - __expf((float)l[e] - top) * g));
    }
    *reinterpret_cast<uint4*>(dx + (int64_t)t * width + c) = pack8<T>(f);
  }
}

hlResult_t moeRoute(int dt, const void* logits, int tokens, int experts, int capacity, int* expert, float* gate, int* row_of, int* token_of,
                    cudaStream_t s) {
  if (experts < 1 || capacity < 1 || (int64_t)experts * capacity > 0x7fffffff)
    return fail(hlInvalidArgument, "MoE routing: %d experts of capacity %d", experts, capacity);
  if (tokens > 0) {
    HL_HALF_SWITCH(dt, T, { kMoeRoute<T><<<(tokens + 127) / 128, 128, 0, s>>>((const T*)logits, tokens, experts, expert, gate); });
  }
  kMoeAssign<<<experts, kAssignThreads, 0, s>>>(expert, tokens, capacity, row_of, token_of);
  return launched("MoE routing");
}

hlResult_t moeGather(const void* src, const int* index, void* dst, int rows, int width, cudaStream_t s) {
  if (width % 8) return fail(hlInvalidArgument, "MoE dispatch: width %d", width);
  if (rows > 0) kMoeGather<><<<(rows + 7) / 8, 256, 0, s>>>((const uint4*)src, index, (uint4*)dst, rows, width / 8);
  return launched("MoE dispatch");
}

hlResult_t moeCombine(int dt, const void* x, const float* gate, const void* rows, const int* row_of, void* y, int tokens, int width, cudaStream_t s) {
  if (width % 8) return fail(hlInvalidArgument, "MoE combine: width %d", width);
  if (tokens > 0) {
    HL_HALF_SWITCH(dt, T, { kMoeCombine<T><<<(tokens + 7) / 8, 256, 0, s>>>((const T*)x, gate, (const T*)rows, row_of, (T*)y, tokens, width); });
  }
  return launched("MoE combine");
}

hlResult_t moeRowGradient(int dt, const void* dy, const float* gate, const void* rows, const int* token_of, void* drows, float* dgate, int n_rows,
                          int width, cudaStream_t s) {
  if (width % 8) return fail(hlInvalidArgument, "MoE gradient: width %d", width);
  HL_HALF_SWITCH(dt, T, {
    kMoeRowGradient<T><<<(n_rows + 7) / 8, 256, 0, s>>>((const T*)dy, gate, (const T*)rows, token_of, (T*)drows, dgate, n_rows, width);
  });
  return launched("MoE row gradient");
}

bool moeRouterFits(int experts, int width) { return experts <= 16 && (size_t)experts * width * 2 <= (48u << 10); }

hlResult_t moeTokenGradient(int dt, const void* dy, const void* drows, const int* row_of, const void* logits, const float* gate, const float* dgate,
                            const void* router, void* dx, void* dlogits, int tokens, int width, int experts, cudaStream_t s) {
  if (width % 8 || width > 2048) return fail(hlInvalidArgument, "MoE gradient: width %d", width);
  if (tokens == 0) return hlSuccess;
  const int per = 256 / (width / 8), groups = (tokens + per - 1) / per;
  const unsigned blocks = (unsigned)(groups < 148 * 6 ? groups : 148 * 6);
  const bool fits = moeRouterFits(experts, width);
  const size_t smem = fits ? (size_t)experts * width * 2 : 0;
  HL_HALF_SWITCH(dt, T, {
    auto go = [&](auto kern) {
      kern<<<blocks, 256, smem, s>>>((const T*)dy, (const T*)drows, row_of, (const T*)logits, gate, dgate, (const T*)router, (T*)dx, (T*)dlogits, tokens,
                                     width, experts);
    };
    if (!fits) go(kMoeTokenGradient<T, 1, false>);
    else if (experts <= 8) go(kMoeTokenGradient<T, 8, true>);
    else go(kMoeTokenGradient<T, 16, true>);
  });
  return launched("MoE token gradient");
}

}  // namespace train
}  // namespace hl
