// Routing, dispatch and combine of a top-1 mixture-of-experts layer with a fixed capacity per expert.
//
// moeRoute       a thread per token: the expert with the largest softmax probability, which is the gate
// moeAssign      a CTA per expert: walks the tokens in order, numbers the expert's own by a scan over the CTA; a token's row is expert * capacity + number, or none beyond the capacity. The CTA also writes
//                the inverse map (row -> token), so that everything after it can go by rows: every row of the dispatch
//                buffer is then written exactly once, empty ones with zeros, and nothing needs clearing or atomics.
// moeGather      rows of the dispatch buffer from the tokens
// moeCombine     y = x + gate * row
// moeRowGradient d row = gate * dy; d gate = <dy, row>
// moeTokenGradient  d logits of the gate's softmax; dx = dy + d row + d logits * router
// moeTokensAndRouter  the same, and the router's gradient with it
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
  for (int e = 1; e < experts; ++e) best = fmaxf(best, (float)p[e]);
  float sum = 0.f;
  for (int e = 0; e < experts; ++e) sum += expf((float)p[e] - best);
  // The maximum of the probabilities, as a softmax and a maximum give it: the first of equal ones (logits may differ and
  // their probabilities not), and the first that is NaN (with a NaN or an infinite logit all of them are).
  float top = expf((float)p[0] - best) / sum;
  int at = 0;
  for (int e = 1; e < experts; ++e) {
    const float q = expf((float)p[e] - best) / sum;
    if (q > top) {
      top = q;
      at = e;
    }
  }
  expert[t] = at;
  gate[t] = top;
}

constexpr int kAssignThreads = 1024, kAssignTokens = 4;   // four consecutive tokens per thread and sweep
__global__ void __launch_bounds__(kAssignThreads) kMoeAssign(const int* __restrict__ expert, int tokens, int capacity, int* __restrict__ row_of,
                                                             int* __restrict__ token_of, int* __restrict__ count) {
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
  if (threadIdx.x == 0) count[e] = base < capacity ? base : capacity;
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

// A thread per token. gate = p_top: d logit_e = d gate * p_top * ([e is top] - p_e), with p_e = exp(l_e - l_top) * p_top.
// No gradient for a token whose gate was not used.
template <typename T>
__global__ void __launch_bounds__(128) kMoeLogitGradient(const int* __restrict__ row_of, const T* __restrict__ logits, const int* __restrict__ expert,
                                                         const float* __restrict__ gate, const float* __restrict__ dgate, T* __restrict__ dlogits,
                                                         int tokens, int experts) {
  const int t = blockIdx.x * 128 + threadIdx.x;
  if (t >= tokens) return;
  const T* l = logits + (int64_t)t * experts;
  const int at = expert[t];
  const float g = gate[t], dg = row_of[t] >= 0 ? dgate[t] * g : 0.f, top = (float)l[at];
  for (int e = 0; e < experts; ++e) dlogits[(int64_t)t * experts + e] = (T)(dg * ((e == at ? 1.f : 0.f) - __expf((float)l[e] - top) * g));
}

// dx = dy + d row + d logits * router. A warp takes two tokens, whose gradients of the logits it holds in registers (E
// bounds the experts), so that a packet of the router is loaded once for both. 8192 x 1024, eight experts: 21.6 us, plus
// 3.1 for the logits' gradients above; with four tokens 21.5, with one kernel that walked tokens with the router in
// shared memory 25, and that one was limited to rows of 2048. E = 0: the router's share is left to a GEMM.
constexpr int kTokensPerWarp = 2;
template <typename T, int E>
__global__ void __launch_bounds__(256, 4) kMoeTokenGradient(const T* __restrict__ dy, const T* __restrict__ drows, const int* __restrict__ row_of,
                                                            const T* __restrict__ router, const T* __restrict__ dlogits, T* __restrict__ dx,
                                                            int tokens, int width, int experts) {
  constexpr int K = kTokensPerWarp;
  const int t0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * K, lane = threadIdx.x & 31;
  if (t0 >= tokens) return;
  int row[K];
  T dl[K][E > 0 ? E : 1];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    row[k] = t0 + k < tokens ? row_of[t0 + k] : -1;
#pragma unroll
    for (int e = 0; e < E; ++e) dl[k][e] = e < experts && t0 + k < tokens ? dlogits[(int64_t)(t0 + k) * experts + e] : (T)0.f;
  }
  for (int c = lane * 8; c < width; c += 256) {
    uint4 a[K], b[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      a[k] = dy && t0 + k < tokens ? *reinterpret_cast<const uint4*>(dy + (int64_t)(t0 + k) * width + c) : make_uint4(0u, 0u, 0u, 0u);
      b[k] = row[k] >= 0 ? *reinterpret_cast<const uint4*>(drows + (int64_t)row[k] * width + c) : make_uint4(0u, 0u, 0u, 0u);
    }
    float f[K][8];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      float h[8];
      unpack8<T>(a[k], f[k]);
      unpack8<T>(b[k], h);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[k][i] += h[i];
    }
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (e < experts) {
        float w[8];
        unpack8<T>(__ldg(reinterpret_cast<const uint4*>(router + (int64_t)e * width + c)), w);
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
          for (int i = 0; i < 8; ++i) f[k][i] += (float)dl[k][e] * w[i];
      }
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (t0 + k < tokens) *reinterpret_cast<uint4*>(dx + (int64_t)(t0 + k) * width + c) = pack8<T>(f[k]);
  }
}

// The last three steps of a layer's backward pass in one walk over the tokens, for up to eight experts: the logits' gradients
// (as above), dx = dy + d row + d logits * router, and the sums over the tokens of d logits * x, which are the router's gradient.
// Bound by memory: dy, the rows and x in, dx out. A CTA first works out its tokens' rows and logits' gradients, a thread per token, and
// leaves them in shared memory (each warp for itself, between its loads, took 46 us: a chain of three loads per token). Then a
// warp keeps 256 columns of the router and of the sums in registers and walks tokens, four at a time: twelve packets per
// lane in flight. (128 columns and twice the warps: 37 us.) The warps share out up to 1024 columns and, where the rows are narrower,
// the tokens. Sums go out as one partial per CTA. 8192 x 1024, eight experts: 33 us, and 3.4 to add the partials up; the kernels above 24.3
// + 3.2 and a GEMM over eight rows 15.3, with the gaps between them 50. (What the products before have written leaves L2 meanwhile: 84 MB
// beside the 67 that are moved here.)
constexpr int kSumExperts = 8, kSumThreads = 256, kSumBlock = 1024, kSumTokens = 4;
template <typename T>
__global__ void __launch_bounds__(kSumThreads, 1) kMoeTokensAndRouter(const T* __restrict__ dy, const T* __restrict__ drows, const int* __restrict__ row_of,
                                                                      const T* __restrict__ logits, const int* __restrict__ expert,
                                                                      const float* __restrict__ gate, const float* __restrict__ dgate,
                                                                      const T* __restrict__ router, const T* __restrict__ x, T* __restrict__ dx,
                                                                      float* __restrict__ partials, int tokens, int width, int experts, int shares) {
  constexpr int E = kSumExperts, K = kSumTokens;
  extern __shared__ float s_sums[];                    // [warps][E][256]
  __shared__ __align__(16) float s_dl[kSumThreads][E];
  __shared__ int s_row[kSumThreads];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int share = warp % shares, group = warp / shares, groups = kSumThreads / 32 / shares;   // of the columns, of the tokens
  const int col = blockIdx.y * kSumBlock + share * 256 + lane * 8;
  const bool live = group < groups && col < width;
  uint64_t w[E][4], acc[E][4];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    float f[8];
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (live && e < experts) v = *reinterpret_cast<const uint4*>(router + (int64_t)e * width + col);
    unpack8<T>(v, f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w[e][i] = pair(f[2 * i], f[2 * i + 1]);
      acc[e][i] = 0;
    }
  }
  const int per = (tokens + gridDim.x - 1) / gridDim.x, t0 = blockIdx.x * per, t1 = min(tokens, t0 + per);
  for (int base = t0; base < t1; base += kSumThreads) {
    const int many = min(kSumThreads, t1 - base);
    __syncthreads();
    if ((int)threadIdx.x < many) {
      const int t = base + threadIdx.x, at = expert[t], row = row_of[t];
      const T* l = logits + (int64_t)t * experts;
      const float g = gate[t], dg = row >= 0 ? dgate[t] * g : 0.f, top = (float)l[at];
      s_row[threadIdx.x] = row;
#pragma unroll
      for (int e = 0; e < E; ++e)
        s_dl[threadIdx.x][e] = e < experts ? (float)(T)(dg * ((e == at ? 1.f : 0.f) - __expf((float)l[e] - top) * g)) : 0.f;
    }
    __syncthreads();
    for (int i = group; live && i < many; i += K * groups) {
      uint4 a[K], b[K], c[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const bool here = i + k * groups < many;
        const int row = here ? s_row[i + k * groups] : -1;
        const int64_t at = (int64_t)(base + i + k * groups) * width + col;
        a[k] = here && dy ? *reinterpret_cast<const uint4*>(dy + at) : make_uint4(0u, 0u, 0u, 0u);
        b[k] = row >= 0 ? *reinterpret_cast<const uint4*>(drows + (int64_t)row * width + col) : make_uint4(0u, 0u, 0u, 0u);
        c[k] = here ? *reinterpret_cast<const uint4*>(x + at) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (i + k * groups < many) {
          float f[8], h[8];
          uint64_t sum[4], in[4];
          unpack8<T>(a[k], f);
          unpack8<T>(b[k], h);
#pragma unroll
          for (int j = 0; j < 4; ++j) sum[j] = add2(pair(f[2 * j], f[2 * j + 1]), pair(h[2 * j], h[2 * j + 1]));
          unpack8<T>(c[k], h);
#pragma unroll
          for (int j = 0; j < 4; ++j) in[j] = pair(h[2 * j], h[2 * j + 1]);
#pragma unroll
          for (int q = 0; q < E; q += 4) {
            const float4 d4 = *reinterpret_cast<const float4*>(&s_dl[i + k * groups][q]);
            const float d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (q + e < experts) {
                const uint64_t d2 = pair(d[e], d[e]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  sum[j] = fma2(d2, w[q + e][j], sum[j]);
                  acc[q + e][j] = fma2(d2, in[j], acc[q + e][j]);
                }
              }
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) unpair(sum[j], f[2 * j], f[2 * j + 1]);
          *reinterpret_cast<uint4*>(dx + (int64_t)(base + i + k * groups) * width + col) = pack8<T>(f);
        }
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e)
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<uint64_t*>(s_sums + (warp * E + e) * 256 + lane * 8 + 2 * i) = acc[e][i];
  __syncthreads();
  const int columns = min(kSumBlock, width - (int)blockIdx.y * kSumBlock);
  for (int i = threadIdx.x; i < experts * columns; i += kSumThreads) {
    const int e = i / columns, c = i - e * columns;
    float sum = 0.f;
    for (int g = 0; g < groups; ++g) sum += s_sums[((g * shares + (c >> 8)) * E + e) * 256 + (c & 255)];
    partials[((int64_t)blockIdx.x * experts + e) * width + blockIdx.y * kSumBlock + c] = sum;
  }
}

hlResult_t moeRoute(int dt, const void* logits, int tokens, int experts, int capacity, int* expert, float* gate, int* row_of, int* token_of,
                    int* count, cudaStream_t s) {
  if (experts < 1 || capacity < 1 || (int64_t)experts * capacity > 0x7fffffff)
    return fail(hlInvalidArgument, "MoE routing: %d experts of capacity %d", experts, capacity);
  if (tokens > 0) {
    HL_HALF_SWITCH(dt, T, { kMoeRoute<T><<<(tokens + 127) / 128, 128, 0, s>>>((const T*)logits, tokens, experts, expert, gate); });
  }
  kMoeAssign<<<experts, kAssignThreads, 0, s>>>(expert, tokens, capacity, row_of, token_of, count);
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

bool moeRouterFits(int experts) { return experts <= 16; }

hlResult_t moeTokenGradient(int dt, const void* dy, const void* drows, const int* row_of, const void* logits, const int* expert, const float* gate,
                            const float* dgate, const void* router, void* dx, void* dlogits, int tokens, int width, int experts, cudaStream_t s) {
  if (width % 8) return fail(hlInvalidArgument, "MoE gradient: width %d", width);
  if (tokens == 0) return hlSuccess;
  HL_HALF_SWITCH(dt, T, {
    kMoeLogitGradient<T><<<(tokens + 127) / 128, 128, 0, s>>>(row_of, (const T*)logits, expert, gate, dgate, (T*)dlogits, tokens, experts);
    auto go = [&](auto kern) {
      constexpr int per = 8 * kTokensPerWarp;
      kern<<<(tokens + per - 1) / per, 256, 0, s>>>((const T*)dy, (const T*)drows, row_of, (const T*)router, (const T*)dlogits, (T*)dx, tokens, width, experts);
    };
    if (!moeRouterFits(experts)) go(kMoeTokenGradient<T, 0>);
    else if (experts <= 8) go(kMoeTokenGradient<T, 8>);
    else go(kMoeTokenGradient<T, 16>);
  });
  return launched("MoE token gradient");
}

bool moeTokensAndRouterFits(int experts) { return experts <= kSumExperts; }
int moeRouterPartials(int tokens) { return tokens < 148 ? tokens : 148; }

hlResult_t moeTokensAndRouter(int dt, const void* dy, const void* drows, const int* row_of, const void* logits, const int* expert, const float* gate,
                              const float* dgate, const void* router, const void* x, void* dx, float* partials, int tokens, int width, int experts,
                              cudaStream_t s) {
  if (width % 8 || experts < 1 || experts > kSumExperts || tokens < 1) return fail(hlInvalidArgument, "MoE gradient: %d x %d, %d experts", tokens, width, experts);
  const int blocks = (width + kSumBlock - 1) / kSumBlock, shares = blocks > 1 ? kSumBlock / 256 : (width + 255) / 256;
  const size_t smem = (size_t)(kSumThreads / 32) * kSumExperts * 256 * sizeof(float);
  HL_HALF_SWITCH(dt, T, {
    cudaFuncSetAttribute((const void*)kMoeTokensAndRouter<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kMoeTokensAndRouter<T><<<dim3((unsigned)moeRouterPartials(tokens), (unsigned)blocks), kSumThreads, smem, s>>>(
        (const T*)dy, (const T*)drows, row_of, (const T*)logits, expert, gate, dgate, (const T*)router, (const T*)x, (T*)dx, partials, tokens, width,
        experts, shares);
  });
  return launched("MoE token gradient");
}

}  // namespace train
}  // namespace hl
