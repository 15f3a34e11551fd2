// Matrix products of groups of matrices (a mixture of experts) on the fifth-generation tensor cores.
//
// out[g][n][m] = sum over k of A[g][m][k] B[g][n][k], operands in either major order, with what follows the product in its
// epilogue (gelu, or gelu's gradient). One launch takes up to two products: the two of a backward pass that read the same
// gradient share one set of tiles, so that the last wave of one is filled by the other.
//
// A pair of CTAs computes a 256 x 256 tile: each holds 128 rows of A and half of B's. The accumulator takes half of the tensor memory;
// the other half belongs to the tile before, which the epilogue warps empty meanwhile. Persistent, one pair per two SMs.
//   warp 0      TMA loads, six stages of 64 of k (32 KB per CTA; 8 x 1024 x 1024 x 4096 in bf16: four stages 60 us, five 56.2, six 55.6)
//   warp 1      products, in the pair's first CTA alone
//   warps 4-11  epilogue: chunks of 32 x 32, rounded, transposed by stmatrix through shared memory of the warp's own (two
//               places of 2 KB in turn), and stored as rows of 64 bytes; no warp waits for another. (Chunks of 128 x 32 that leave by TMA, with barriers of 128 threads: 75 us
//               where this takes 67; both with a reciprocal for four of gelu's values.)
// Loads and products run in all lanes of their warps up to the instruction itself, so that its operands are in uniform
// registers: in a branch of one lane the same loops took 86 us instead of 57.
//
// The tokens are n, the weights' rows are m: an expert's last tile is as wide as its tokens need, in steps of 32, where rows of
// tokens as m would come in steps of 256. Where routing is part of the call, the layer's capacity (1.25 times the average in use) costs
// nothing then: tiles and k end at the `counts` that it found, rounded up to 32. Rows between a count and the rounding are zeros.
//
// 8 x 1024 x 1024 x 4096 in bf16, 69 GFLOP a product, every row in use, us here / the library with gelu's passes. Short runs: with gelu 71 / 55 + 26,
// k = 4096 54.6 / 48, gelu's gradient 82 / 55 + 41, the product behind it 52.5 / 48, the gradient with dW2 124 / 55 + 41 + 55, dW1 with dh 99 / 55 + 47.
// Back to back for a second, under the power cap, forward and backward: 95 + 67 + 156 + 119 here, 447 there in eight. So with every row in use
// the two are even; a layer gains by the rows that are not (8192 tokens, 622 -> 510). Bound by power without an epilogue, with one by its
// warps. Tried: pairs of 512 x 256 with one set of accumulators, which read a quarter less (55 us for k = 4096; slower with gelu, whose
// epilogue then has half the time), also with sixteen epilogue warps (58).
// The sums go up k in the order of the library's own kernels: results are theirs, bit for bit (the tests compare the two).
// Every wait is bounded; one that runs out sets the device's status word, which stays set until gemmStatus has reported it: to whoever
// waits for the results (a trainer after its step, replayed from a graph or not), and to every launch until then.
#include <cuda.h>

#include <atomic>
#include <mutex>

#include "hal/cuda_driver.h"
#include "train/tcgen05.cuh"
#include "train/train_device.cuh"
#include "train/train_kernels.h"

namespace hl {
namespace train {

constexpr int kGemmStages = 6, kTile = 256, kKBlock = 64, kStageBytes = 32768, kBoxBytes = 8192, kChunk = 32;
constexpr int kGemmThreads = 384, kEpilogueWarps = 8, kChunkStaging = 2048, kWarpStaging = 2 * kChunkStaging;
constexpr int kGemmShared = kGemmStages * kStageBytes + kEpilogueWarps * kWarpStaging + 1024;
constexpr int kTmemColumns = 512;
constexpr uint64_t kGemmLimitNs = 2000000000ull, kSettleNs = 1000000ull;

struct GemmJob {
  CUtensorMap a, b;
  void *out, *aux;                // [groups][n][m]; aux: the activation (kGemmGelu) or the pre-activation (kGemmGeluGradient)
  int m, n, k, m_tiles;
  int ragged, a_mn, b_mn, epilogue;
  const void* bias;               // [m], or null
  float* columns;                 // [2 (n / 256, rounded up)][m], or null
};
struct GemmArgs {
  GemmJob job[2];
  int jobs, groups;
  const int* counts;
  volatile unsigned* status;
  uint64_t limit_ns;              // of every wait
  int loads;                      // 0: operands never arrive, for tests of the limit
};

struct Tile {
  const GemmJob* job;
  int group, m0, n0, width;       // width: columns that are computed, a multiple of 32
  int k_blocks, last_steps;       // of 64; the last one in steps of 16
};
// The tiles in order: product, group, n, m. Each role of a CTA walks them by itself.
struct Walker {
  int job = 0, group = 0, before = 0;
  __device__ __forceinline__ bool seek(const GemmArgs& g, int t, Tile* o) {
    while (job < g.jobs) {
      const GemmJob& j = g.job[job];
      const int full = j.ragged == kGemmRaggedK ? j.k : j.n;
      int rows = full;
      if (j.ragged != kGemmWhole && g.counts) rows = max(1, min(g.counts[group], full));
      rows = (rows + 31) & ~31;
      const int n = j.ragged == kGemmRaggedK ? (j.n + 31) & ~31 : rows;
      const int tiles = (n + kTile - 1) / kTile * j.m_tiles;
      if (t < before + tiles) {
        const int at = t - before, nt = at / j.m_tiles;
        o->job = &j;
        o->group = group;
        o->m0 = (at - nt * j.m_tiles) * kTile;
        o->n0 = nt * kTile;
        o->width = min(kTile, n - o->n0);
        if (j.b_mn) o->width = (o->width + 127) & ~127;      // each CTA's half in whole groups of 64
        const int k = j.ragged == kGemmRaggedK ? rows : j.k;
        o->k_blocks = (k + kKBlock - 1) / kKBlock;
        o->last_steps = (k - (o->k_blocks - 1) * kKBlock + 15) / 16;
        return true;
      }
      before += tiles;
      if (++group == g.groups) {
        group = 0;
        ++job;
      }
    }
    return false;
  }
};

// 32 x 32 results of a warp, on their way from tensor memory (a lane holds pairs of n) to rows of `out` (a lane holds eight m). Row n,
// eight m from 8 c on lie at 64 n + 16 (c ^ (n / 2 % 4)): neither side has two lanes on the same banks.
__device__ __forceinline__ uint32_t stagedAt(int n, int c) { return (uint32_t)(n * 64 + ((c ^ (n >> 1 & 3)) << 4)); }

template <typename T>
__device__ __forceinline__ void transposeChunk(const float* r, const float* bias, uint32_t staging, int lane) {
  using H = Half2Of<T>;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    uint32_t v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = (i >> 1) * 16 + 4 * g + (i & 1) * 2;
      const typename H::type p = H::down(r[k] + bias[i], r[k + 1] + bias[i]);
      v[i] = *reinterpret_cast<const uint32_t*>(&p);
    }
    tc::storeMatrixT(staging + stagedAt(8 * g + (lane & 7), lane >> 3), v[0], v[1], v[2], v[3]);
  }
}

template <typename T>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1) kExpertGemm(const __grid_constant__ GemmArgs args) {
  extern __shared__ uint8_t s_raw[];
  __shared__ __align__(8) uint64_t s_full[kGemmStages], s_empty[kGemmStages], s_acc_full[2], s_acc_empty[2], s_done;
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_stop;
  const uint32_t stages = (tc::smem(s_raw) + 1023) & ~1023u, staging = stages + kGemmStages * kStageBytes;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // uniform, and known to be
  const uint32_t rank = tc::clusterRank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  if (threadIdx.x == 0) {
    s_stop = 0;
    for (int i = 0; i < kGemmStages; ++i) {
      tc::barInit(tc::smem(&s_full[i]), 1);
      tc::barInit(tc::smem(&s_empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::barInit(tc::smem(&s_acc_full[i]), 1);
      tc::barInit(tc::smem(&s_acc_empty[i]), 2 * kEpilogueWarps);
    }
    tc::barInit(tc::smem(&s_done), 1);
    tc::barInitFence();
  }
  if (warp == 1 && lane == 0)
    for (int i = 0; i < args.jobs; ++i) {
      tc::prefetchMap(&args.job[i].a);
      tc::prefetchMap(&args.job[i].b);
    }
  __syncwarp();
  if (warp == 2) tc::tmemAlloc(tc::smem(&s_tmem), kTmemColumns);
  tc::fenceBefore();
  tc::clusterSync();
  tc::fenceAfter();
  const uint32_t tmem = s_tmem;
  volatile int* const stop = &s_stop;
  Walker walk;
  Tile t;

  if (warp == 0) {                                     // ---- loads
    int s = 0, rounds = 0;
    uint32_t phase = 1;                                // of the wait for a free stage: the first round finds all of them free
    bool go = args.loads != 0;
    const uint32_t full0 = tc::mapToRank(tc::smem(&s_full[0]), 0);
    for (int at = pair; go && walk.seek(args, at, &t); at += pairs) {
      const GemmJob& j = *t.job;
      const int half = t.width / 2;
      const bool two = half > 64;
      const int a0 = t.m0 + (int)rank * 128, b0 = t.n0 + (int)rank * half;
      const uint32_t bytes = two ? 8 * kBoxBytes : 6 * kBoxBytes;
      const bool a_mn = j.a_mn != 0, b_mn = j.b_mn != 0;
      for (int k = 0; k < t.k_blocks * kKBlock; k += kKBlock) {
        go = tc::barWait(tc::smem(&s_empty[s]), phase, stop, args.limit_ns);
        if (!(go = __all_sync(0xffffffffu, go))) break;
        if (tc::elected()) {
          if (rank == 0) tc::barExpect(tc::smem(&s_full[s]), bytes);
          const uint32_t bar = full0 + s * 8, dst = stages + s * kStageBytes;
          tc::loadTilePair(dst, &j.a, a_mn ? a0 : k, a_mn ? k : a0, t.group, bar);
          tc::loadTilePair(dst + kBoxBytes, &j.a, a_mn ? a0 + 64 : k, a_mn ? k : a0 + 64, t.group, bar);
          tc::loadTilePair(dst + 2 * kBoxBytes, &j.b, b_mn ? b0 : k, b_mn ? k : b0, t.group, bar);
          if (two) tc::loadTilePair(dst + 3 * kBoxBytes, &j.b, b_mn ? b0 + 64 : k, b_mn ? k : b0 + 64, t.group, bar);
        }
        __syncwarp();
        if (++s == kGemmStages) {
          s = 0;
          phase ^= 1;
          rounds = 1;
        }
      }
    }
    if (!go && rank == 0)                              // given up: the pair's copies are counted here, those that both have asked for land first
      for (int i = rounds ? 0 : kGemmStages - s; i < kGemmStages; ++i) {
        const int at = (s + i) % kGemmStages;          // oldest first; stages from s on were filled in the round before
        tc::barWait(tc::smem(&s_full[at]), at < s ? phase ^ 1 : phase, nullptr, kSettleNs);
      }
  } else if (warp == 1 && rank == 0) {                 // ---- products
    const uint32_t kind = 1u << 4 | (std::is_same<T, __nv_bfloat16>::value ? 1u << 7 | 1u << 10 : 0u) | (uint32_t)(kTile >> 4) << 24;
    int s = 0, n = 0;
    uint32_t phase = 0;
    bool go = true;
    for (int at = pair; go && walk.seek(args, at, &t); at += pairs, ++n) {
      const GemmJob& j = *t.job;
      const int acc = n & 1;
      go = tc::barWait<true>(tc::smem(&s_acc_empty[acc]), (n >> 1 & 1) ^ 1, stop, args.limit_ns);
      if (!(go = __all_sync(0xffffffffu, go))) break;
      tc::fenceAfter();
      const bool a_mn = j.a_mn != 0, b_mn = j.b_mn != 0;
      const uint32_t idesc = kind | (uint32_t)a_mn << 15 | (uint32_t)b_mn << 16 | (uint32_t)(t.width >> 3) << 17;
      const uint32_t d = tmem + acc * kTile;
      const uint64_t a_step = a_mn ? 2048 >> 4 : 32 >> 4, b_step = b_mn ? 2048 >> 4 : 32 >> 4;   // 16 of k
      const uint64_t a0 = tc::operand(stages, a_mn, kBoxBytes), b0 = tc::operand(stages + 2 * kBoxBytes, b_mn, kBoxBytes);
      for (int kb = 0; kb < t.k_blocks; ++kb) {
        go = tc::barWait(tc::smem(&s_full[s]), phase, stop, args.limit_ns);
        if (!(go = __all_sync(0xffffffffu, go))) break;
        tc::fenceAfter();
        const int steps = kb + 1 < t.k_blocks ? kKBlock / 16 : t.last_steps;
        if (tc::elected()) {
          const uint64_t a = a0 + (uint64_t)(s * (kStageBytes >> 4)), b = b0 + (uint64_t)(s * (kStageBytes >> 4));
#pragma unroll
          for (int i = 0; i < kKBlock / 16; ++i)
            if (i < steps) tc::mma16(d, a + i * a_step, b + i * b_step, idesc, kb > 0 || i > 0);
          tc::commitPair(tc::smem(&s_empty[s]));
          if (kb + 1 == t.k_blocks) tc::commitPair(tc::smem(&s_acc_full[acc]));
        }
        __syncwarp();
        if (++s == kGemmStages) {
          s = 0;
          phase ^= 1;
        }
      }
    }
    if (!go) {                                         // given up: the products that were issued read shared memory until they are done
      if (tc::elected()) tc::commitPair(tc::smem(&s_done));
      __syncwarp();
      tc::barWait(tc::smem(&s_done), 0, nullptr, kSettleNs);
    }
  } else if (warp >= 4) {                              // ---- epilogue
    const int group = (warp - 4) >> 2, q = warp & 3;   // a warp reads the 32 lanes of its place in a group of four
    const uint32_t mine = staging + (warp - 4) * kWarpStaging;
    int n = 0;
    for (int at = pair; walk.seek(args, at, &t); at += pairs, ++n) {
      const GemmJob& j = *t.job;
      const int acc = n & 1, chunks = t.width / kChunk, epilogue = j.epilogue;
      const int m0 = t.m0 + (int)rank * 128 + 32 * q;  // this warp's lanes
      const int mv = m0 + 8 * (lane & 3);              // this lane's eight m of `out`
      const bool live = mv < j.m;
      const int64_t at0 = ((int64_t)t.group * j.n + t.n0) * j.m + mv;
      T* const out = reinterpret_cast<T*>(j.out) + at0;
      T* const aux = reinterpret_cast<T*>(j.aux) + at0;
      const int rows = j.n - t.n0;                     // of the tile that exist
      auto row = [&](int c, int i) { return c * kChunk + 8 * i + (lane >> 2); };
      uint4 pre[4];                                    // pre-activations of the next chunk
      auto fetch = [&](int c, int i) {
        if (live && row(c, i) < rows) pre[i] = __ldcs(reinterpret_cast<const uint4*>(aux + (int64_t)row(c, i) * j.m));
      };
      float bias[4], sums[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {                    // of lane 8 i + lane / 4 of tensor memory
        const int m = m0 + 8 * i + (lane >> 2);
        bias[i] = j.bias && m < j.m ? (float)reinterpret_cast<const T*>(j.bias)[m] : 0.f;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) sums[i] = 0.f;
      if (epilogue == kGemmGeluGradient && group < chunks) {
#pragma unroll
        for (int i = 0; i < 4; ++i) fetch(group, i);
      }
      if (!__all_sync(0xffffffffu, tc::barWait(tc::smem(&s_acc_full[acc]), n >> 1 & 1, stop, args.limit_ns))) break;
      tc::fenceAfter();
      // Chunk c to one of the two places in shared memory; the accumulator is free with the last of them.
      auto stage = [&](int c) {
        float r[32];
        tc::tmemLoad32x32(tmem + ((uint32_t)(q * 32) << 16) + acc * kTile + c * kChunk, r);
        if (c + 2 >= chunks) {
          tc::fenceBefore();
          __syncwarp();
          if (lane == 0) tc::barArriveCluster(tc::mapToRank(tc::smem(&s_acc_empty[acc]), 0));
        }
        transposeChunk<T>(r, bias, mine + (c >> 1 & 1) * kChunkStaging, lane);
      };
      if (group < chunks) stage(group);
      for (int c = group; c < chunks; c += 2) {
        __syncwarp();
        uint4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = tc::loadShared(mine + (c >> 1 & 1) * kChunkStaging + stagedAt(8 * i + (lane >> 2), lane & 3));
        if (c + 2 < chunks) stage(c + 2);              // the next one on its way while this one is worked on
        if (epilogue == kGemmGelu) {
          float f[32];
#pragma unroll
          for (int i = 0; i < 4; ++i) unpack8<T>(v[i], f + 8 * i);
          geluAll<32>(f);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (live && row(c, i) < rows) *reinterpret_cast<uint4*>(aux + (int64_t)row(c, i) * j.m) = pack8<T>(f + 8 * i);
        } else if (epilogue == kGemmGeluGradient) {
#pragma unroll
          for (int i = 0; i < 4; i += 2) {
            float f[16], u[16];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              unpack8<T>(v[i + k], f + 8 * k);
              unpack8<T>(pre[i + k], u + 8 * k);
              if (c + 2 < chunks) fetch(c + 2, i + k);
            }
#pragma unroll
            for (int k = 0; k < 16; ++k) f[k] *= geluSlope(u[k]);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              v[i + k] = pack8<T>(f + 8 * k);
              if (j.columns && row(c, i + k) < rows) { // of what is stored
                float g[8];
                unpack8<T>(v[i + k], g);
#pragma unroll
                for (int l = 0; l < 8; ++l) sums[l] += g[l];
              }
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (live && row(c, i) < rows) *reinterpret_cast<uint4*>(out + (int64_t)row(c, i) * j.m) = v[i];
      }
      if (group >= chunks) {                           // nothing to do here
        tc::fenceBefore();
        __syncwarp();
        if (lane == 0) tc::barArriveCluster(tc::mapToRank(tc::smem(&s_acc_empty[acc]), 0));
      }
      if (j.columns) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
#pragma unroll
          for (int o = 4; o < 32; o <<= 1) sums[i] += __shfl_xor_sync(0xffffffffu, sums[i], o);
        }
        if (lane < 4 && live) {
          float* to = j.columns + (int64_t)(t.n0 / kTile * 2 + group) * j.m + mv;
          *reinterpret_cast<float4*>(to) = make_float4(sums[0], sums[1], sums[2], sums[3]);
          *reinterpret_cast<float4*>(to + 4) = make_float4(sums[4], sums[5], sums[6], sums[7]);
        }
      }
    }
  }
  __syncwarp();
  if (*stop) {                                         // given up: tell. A copy that one CTA alone has asked for ends no phase: it gets the time of many
    *args.status = 1;
    __threadfence_system();
    for (const uint64_t t0 = tc::nowNs(); tc::nowNs() - t0 < kSettleNs;) {
    }
  }
  __syncwarp();
  tc::fenceBefore();
  tc::clusterSync();                                   // the other CTA's operands and barriers are in use until here
  tc::fenceAfter();
  if (warp == 2) tc::tmemFree(tmem, kTmemColumns);
}

namespace {

// A word per device in page-locked memory, set by a kernel whose wait ran out; null where that memory could not be had.
constexpr int kDevices = 64;
std::atomic<unsigned*> g_words{nullptr};
unsigned* statusWords() {
  static std::once_flag once;
  std::call_once(once, [] {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;      // the caller's stream may be recording
    cudaThreadExchangeStreamCaptureMode(&mode);
    void* p = nullptr;
    if (cudaHostAlloc(&p, kDevices * sizeof(unsigned), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
      for (int i = 0; i < kDevices; ++i) ((volatile unsigned*)p)[i] = 0;
      g_words.store((unsigned*)p, std::memory_order_release);
    } else {
      cudaGetLastError();
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
  });
  return g_words.load(std::memory_order_acquire);
}

// Pairs of CTAs that run at once on the current device; 0 where the kernel does not run.
template <typename T>
int residentPairs() {
  static std::atomic<int> known[kDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= kDevices) return 0;
  int have = known[dev].load(std::memory_order_relaxed);
  if (have) return have - 1;
  have = 1;
  int sms = 0, major = 0, most = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
  if (major == 10 && cudaFuncSetAttribute(kExpertGemm<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmShared) == cudaSuccess) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)(sms / 2 * 2));
    c.blockDim = dim3(kGemmThreads);
    c.dynamicSmemBytes = kGemmShared;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&most, kExpertGemm<T>, &c) == cudaSuccess && most > 0) have = 1 + (most < sms / 2 ? most : sms / 2);
  }
  cudaGetLastError();
  known[dev].store(have, std::memory_order_relaxed);
  return have - 1;
}

CUresult encode(const CudaDriver* d, CUtensorMap* m, int dt, const void* p, int64_t inner, int64_t rows, int groups) {
  const cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)rows, (cuuint64_t)groups};
  const cuuint64_t strides[2] = {(cuuint64_t)inner * 2, (cuuint64_t)(inner * rows) * 2};
  const cuuint32_t box[3] = {64, 64, 1}, steps[3] = {1, 1, 1};
  return d->cuTensorMapEncodeTiled(m, dt == hlBfloat16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(p), dims,
                                   strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

}  // namespace

bool gemmRuns(int dt) {
  static const bool wanted = envBool({"HYLINK_OWN_PRODUCTS"}, true);
  const CudaDriver* d = wanted ? CudaDriver::get() : nullptr;
  int dev = 0;
  if (!d || !d->cuTensorMapEncodeTiled || cudaGetDevice(&dev) != cudaSuccess || dev >= kDevices || !statusWords()) return false;
  return dt == hlBfloat16 ? residentPairs<__nv_bfloat16>() > 0 : dt == hlFloat16 && residentPairs<__half>() > 0;
}

// From 2^33 multiplications on the tiles fill the GPU, and the kernels are the faster ones. Smaller layers take the host longer than the GPU,
// and the host has four launches to issue here and eight with the library. Recorded into a graph they take the GPU alone. Whole layers, forward
// and backward, us own / library, issued and (recorded): 64 tokens of 256 x 1024, eight experts 206 / 294 (57 / 51); 200 of 1024 x 4096, eight
// 208 / 262 (170 / 142); 1072 of 768 x 3072, eight 243 / 298 (149 / 136); 2500 of 512 x 2048, eight 207 / 263 (133 / 115); from 2^33 on 2500 of
// 1024 x 4096, four 225 / 266 (205 / 232), 5000 353 / 390 (317 / 338). Below 2^24 nothing is left to win: 31 / 30 for the products.
// (A small layer that is issued behind work that keeps the GPU busy loses those 6 to 20 % too; the host does not know of that.)
bool expertGemmPays(int64_t rows, int64_t width, int64_t hidden, bool captured) {
  return width % 8 == 0 && hidden % 8 == 0 && rows * width * hidden >= (captured ? 1LL << 33 : 1LL << 24);
}
// One product with a bias, which the library's kernels take too: what is gained is the element-wise pass alone, and that once the tiles fill
// the GPU. Training steps, ms own / library: 8192 rows of 1024 x 4096 27.65 / 27.94 (four runs each in turn, which differ by 0.1), 3072 12.93 /
// 12.94, 4096 of 768 x 3072 7.68 / 7.68, 8192 13.36 / 13.36; below the line 1024 rows of 1024 x 4096 9.11 / 9.06, 512 7.71 / 7.53, 256 7.47 / 7.02.
bool mlpGemmPays(int64_t rows, int64_t width, int64_t hidden) {
  return width % 8 == 0 && hidden % 8 == 0 && rows * width * hidden >= (1LL << 33);
}

hlResult_t gemmStatus(int device, bool clear) {
  unsigned* const words = g_words.load(std::memory_order_acquire);
  if (device < 0 && cudaGetDevice(&device) != cudaSuccess) {
    cudaGetLastError();
    return hlSuccess;                                  // no device, no products
  }
  if (!words || device >= kDevices || !((volatile unsigned*)words)[device]) return hlSuccess;
  if (clear) ((volatile unsigned*)words)[device] = 0;
  return fail(hlTimeout, "grouped product: a wait on device %d ran out, results since then are not valid", device);
}

hlResult_t expertGemm(int dt, const GemmSpec* specs, int n, int groups, const int* counts, cudaStream_t s, uint64_t limit_ns, bool loads) {
  const CudaDriver* d = CudaDriver::get();
  if (!d || !d->cuTensorMapEncodeTiled) return fail(hlUnsupported, "grouped product: no driver for tensor maps");
  if (n < 1 || n > 2 || groups < 1) return fail(hlInvalidArgument, "grouped product: %d products of %d groups", n, groups);
  int dev = 0;
  HL_CUDA(cudaGetDevice(&dev));
  HL_CUDA(cudaSetDevice(dev));   // a thread that has made no runtime call yet has no context, which the driver's encoder wants
  unsigned* const words = statusWords();
  if (!words) return fail(hlDeviceError, "grouped product: no page-locked memory");
  if (dev >= kDevices) return fail(hlUnsupported, "grouped product: device %d", dev);
  if (const hlResult_t e = gemmStatus(dev, false)) return e;
  GemmArgs g;
  g.jobs = n;
  g.groups = groups;
  g.counts = counts;
  g.status = words + dev;
  g.limit_ns = limit_ns ? limit_ns : kGemmLimitNs;
  g.loads = loads;
  int64_t tiles = 0;
  for (int i = 0; i < n; ++i) {
    const GemmSpec& x = specs[i];
    GemmJob& j = g.job[i];
    const int a_inner = x.a_mn ? x.m : x.k, b_inner = x.b_mn ? x.n : x.k;
    if (x.m < 1 || x.n < 1 || x.k < 1 || x.m % 8 || a_inner % 8 || b_inner % 8)
      return fail(hlUnsupported, "grouped product: %d x %d x %d", x.m, x.n, x.k);
    for (const void* p : {x.a, x.b, (const void*)x.out, (const void*)x.aux})
      if ((uintptr_t)p & 15) return fail(hlInvalidArgument, "grouped product: an operand starts inside a 16-byte packet");
    CUresult e = encode(d, &j.a, dt, x.a, a_inner, x.a_mn ? x.k : x.m, groups);
    if (e == CUDA_SUCCESS) e = encode(d, &j.b, dt, x.b, b_inner, x.b_mn ? x.k : x.n, groups);
    if (e != CUDA_SUCCESS) return fail(hlDeviceError, "grouped product: tensor maps of %d x %d x %d: %s", x.m, x.n, x.k, d->err(e));
    j.out = x.out;
    j.aux = x.aux;
    j.m = x.m;
    j.n = x.n;
    j.k = x.k;
    j.m_tiles = (x.m + kTile - 1) / kTile;
    j.ragged = x.ragged;
    j.a_mn = x.a_mn;
    j.b_mn = x.b_mn;
    j.epilogue = x.epilogue;
    j.bias = x.bias;
    j.columns = x.columns;
    tiles += (int64_t)groups * j.m_tiles * ((x.n + kTile - 1) / kTile);
  }
  if (tiles > 0x7fffffff / 2) return fail(hlUnsupported, "grouped product: %lld tiles", (long long)tiles);
  HL_HALF_SWITCH(dt, T, {
    const int most = residentPairs<T>();
    if (!most) return fail(hlUnsupported, "grouped product: not on this device");
    kExpertGemm<T><<<2 * (unsigned)(tiles < most ? tiles : most), kGemmThreads, kGemmShared, s>>>(g);
  });
  return launched("grouped product");
}

}  // namespace train
}  // namespace hl
