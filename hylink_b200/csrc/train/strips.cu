// Element-wise kernels of a transformer block's MLP and attention gradients, with the bias gradients (column sums)
// folded in.
//
// A column sum needs every row of a column; the element-wise pass reads them all anyway. A CTA takes a strip of 256
// columns (one warp reads 512 contiguous bytes of a row) and a range of rows; eight warps walk the rows side by side,
// four rows of each in flight, and add up their columns in registers. One fp32 partial per CTA and column goes out;
// finishColumns adds those of several kernels in one launch. No atomics: the sums have a fixed order.
#include "train/train_device.cuh"
#include "train/train_kernels.h"

namespace hl {
namespace train {

constexpr int kStripThreads = 256, kStripWarps = kStripThreads / 32, kStripUnroll = 4;
constexpr int kStripRows = 128;   // rows of one CTA: 16 per warp; 8192 x 4096 makes 1024 CTAs, 8192 x 1024 256

struct SumOp {   // column sums alone
  const void* src;
};
struct GeluOp {
  const void *dg, *u;
  void* du;
};
struct PackOp {
  Strided4 g[3];
  void* out;
  int64_t seq;
  int head_dim, part_width;   // part_width: heads * head_dim
};

template <typename T, typename Op>
__global__ void __launch_bounds__(kStripThreads, 4) kStrip(const __grid_constant__ Op op, float* __restrict__ partials, int64_t rows, int width) {
  __shared__ float s_sum[kStripWarps][256 + 8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = blockIdx.x * 256 + lane * 8;
  const bool live = col < width;
  const int64_t r0 = (int64_t)blockIdx.y * kStripRows, r1 = r0 + kStripRows < rows ? r0 + kStripRows : rows;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  const T* base0 = nullptr;   // pack: this lane's operand, head and column inside the head are the same for every row
  int64_t sb = 0, st = 0, seq = 1;
  if constexpr (std::is_same<Op, PackOp>::value) {
    if (live) {
      const int part = col / op.part_width, c = col - part * op.part_width;
      const int head = c / op.head_dim;
      base0 = reinterpret_cast<const T*>(op.g[part].p) + head * op.g[part].sh + (c - head * op.head_dim);
      sb = op.g[part].sb;
      st = op.g[part].st;
    }
    seq = op.seq;
  }
  if (live) {
    for (int64_t r = r0 + warp; r < r1; r += kStripWarps * kStripUnroll) {
      uint4 a[kStripUnroll], b[kStripUnroll];
#pragma unroll
      for (int k = 0; k < kStripUnroll; ++k) {
        const int64_t row = r + k * kStripWarps;
        if (row < r1) {
          if constexpr (std::is_same<Op, SumOp>::value) {
            a[k] = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(op.src) + row * width + col);
          } else if constexpr (std::is_same<Op, GeluOp>::value) {
            a[k] = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(op.dg) + row * width + col);
            b[k] = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(op.u) + row * width + col);
          } else {
            const int64_t bi = row / seq;
            a[k] = *reinterpret_cast<const uint4*>(base0 + bi * sb + (row - bi * seq) * st);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < kStripUnroll; ++k) {
        const int64_t row = r + k * kStripWarps;
        if (row < r1) {
          float f[8];
          unpack8<T>(a[k], f);
          if constexpr (std::is_same<Op, GeluOp>::value) {
            float u[8];
            unpack8<T>(b[k], u);
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] *= geluSlope(u[i]);
            const uint4 p = pack8<T>(f);
            *reinterpret_cast<uint4*>(reinterpret_cast<T*>(op.du) + row * width + col) = p;
            unpack8<T>(p, f);   // the bias gradient is the sum of what the GEMMs see
          } else if constexpr (std::is_same<Op, PackOp>::value) {
            *reinterpret_cast<uint4*>(reinterpret_cast<T*>(op.out) + row * width + col) = a[k];
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i] += f[i];
        }
      }
    }
  }
  if (partials == nullptr) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) s_sum[warp][lane * 8 + i] = acc[i];
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c < width) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kStripWarps; ++w) t += s_sum[w][threadIdx.x];
    partials[(int64_t)blockIdx.y * width + c] = t;
  }
}

template <typename T>
__global__ void __launch_bounds__(256) kGeluForward(const uint4* __restrict__ u, uint4* __restrict__ out, int64_t packets) {
  constexpr int U = 4;
  const int64_t i0 = (int64_t)blockIdx.x * (256 * U) + threadIdx.x;
  uint4 v[U];
#pragma unroll
  for (int k = 0; k < U; ++k)
    if (i0 + k * 256 < packets) v[k] = u[i0 + k * 256];
#pragma unroll
  for (int k = 0; k < U; ++k)
    if (i0 + k * 256 < packets) {
      float f[8];
      unpack8<T>(v[k], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = gelu(f[i]);
      out[i0 + k * 256] = pack8<T>(f);
    }
}

struct Segments {
  ColSegment s[kMaxColSegments];
};
template <typename T>
__global__ void __launch_bounds__(256) kFinishColumns(const __grid_constant__ Segments segs) {
  __shared__ float s_sum[8][33];
  const ColSegment g = segs.s[blockIdx.y];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + lane;
  if (blockIdx.x * 32 >= g.width) return;
  float t = 0.f;
  if (col < g.width)
#pragma unroll 8
    for (int r = warp; r < g.rows; r += 8) t += g.src[(int64_t)r * g.width + col];
  s_sum[warp][lane] = t;
  __syncthreads();
  if (warp == 0 && col < g.width) {
    t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += s_sum[w][lane];
    reinterpret_cast<T*>(g.dst)[col] = (T)t;
  }
}

int stripPartials(int64_t rows) { return (int)((rows + kStripRows - 1) / kStripRows); }

template <typename Op>
static hlResult_t strip(int dt, const Op& op, float* partials, int64_t rows, int width, cudaStream_t s) {
  if (width % 8) return fail(hlUnsupported, "strip kernels: width %d", width);
  if (rows == 0) return hlSuccess;
  const dim3 grid((unsigned)((width + 255) / 256), (unsigned)stripPartials(rows));
  static_assert(kMaxRows == 65535LL * kStripRows, "one CTA per range of rows");
  if (rows > kMaxRows) return fail(hlUnsupported, "strip kernels: %lld rows", (long long)rows);
  HL_HALF_SWITCH(dt, T, { kStrip<T, Op><<<grid, kStripThreads, 0, s>>>(op, partials, rows, width); });
  return launched("strip");
}

hlResult_t geluForward(int dt, const void* u, void* out, int64_t count, cudaStream_t s) {
  if (count % 8) return fail(hlUnsupported, "gelu: %lld elements", (long long)count);
  if (count == 0) return hlSuccess;
  const int64_t packets = count / 8;
  HL_HALF_SWITCH(dt, T, { kGeluForward<T><<<(unsigned)((packets + 1023) / 1024), 256, 0, s>>>((const uint4*)u, (uint4*)out, packets); });
  return launched("gelu");
}
hlResult_t geluBackward(int dt, const void* dg, const void* u, void* du, float* partials, int64_t rows, int width, cudaStream_t s) {
  return strip(dt, GeluOp{dg, u, du}, partials, rows, width, s);
}
hlResult_t columnSums(int dt, const void* src, float* partials, int64_t rows, int width, cudaStream_t s) {
  return strip(dt, SumOp{src}, partials, rows, width, s);
}
hlResult_t packQkvGradient(int dt, const Strided4 grads[3], void* dqkv, float* partials, int64_t batch, int64_t seq, int heads, int head_dim,
                           cudaStream_t s) {
  if (head_dim % 8) return fail(hlUnsupported, "attention gradient: head_dim %d", head_dim);
  PackOp op;
  for (int i = 0; i < 3; ++i) op.g[i] = grads[i];
  op.out = dqkv;
  op.seq = seq;
  op.head_dim = head_dim;
  op.part_width = heads * head_dim;
  return strip(dt, op, partials, batch * seq, 3 * heads * head_dim, s);
}
hlResult_t finishColumns(int dt, const ColSegment* segs, int n, cudaStream_t s) {
  if (n < 1 || n > kMaxColSegments) return fail(hlInvalidArgument, "finishColumns: %d segments", n);
  Segments a;
  int widest = 0;
  for (int i = 0; i < n; ++i) {
    a.s[i] = segs[i];
    widest = segs[i].width > widest ? segs[i].width : widest;
  }
  HL_HALF_SWITCH(dt, T, { kFinishColumns<T><<<dim3((unsigned)((widest + 31) / 32), (unsigned)n), 256, 0, s>>>(a); });
  return launched("column sums");
}

}  // namespace train
}  // namespace hl
