// Landing reduce, doorbell and warm-up kernels of the PCIe path (sm_100a).
//
// reduceLanding: dst = scale * op(src_0 .. src_{k-1}) (optionally with dst as
// an extra first operand). 16-byte vector accesses, fp32 accumulation for
// fp16/bf16 with one rounding, up to eight sources reduced in ONE pass so that
// a batch of landed chunks is folded with a single read of each. A source may
// be pinned host memory: the kernel then reads the staging buffer over PCIe
// itself, fusing the H2D copy with the reduction.
//
// Parity: replaces D2DReduceTypedKernel<T>, D2DReduceHalfRawKernel and
// D2DReduceBfloat16RawKernel (pcie-ccl-cuda/kernels/wait_kernel.cu:255-360),
// which are scalar two-address grid-stride loops capped at 1024x256 threads;
// the doorbell replaces the 720 named one-thread spin kernels of
// wait_kernel.cu:13-109 with one kernel whose spin is bounded.
#include <cuda_runtime.h>

#include <algorithm>

#include "nvl/nvl_device.cuh"
#include "nvl/nvl_launch.h"

namespace hl {
namespace dev {

constexpr int kRlThreads = 256;

// These kernels are often launched back to back, and a launch that waits for the one before it to drain costs 3 us and
// more: 4.3 us from one small fold to the next, in steps of 2.05 however long the kernel is. So a launch may start while
// its predecessor runs (it lets its own successor do the same at once) and waits here for the predecessor's end, before
// it touches memory: 2.4 us then, which is the host's share, and 26.0 instead of 27.4 for the fold of four times 32 MiB.
// All CTAs of the predecessor have started by then, so it never lacks room to finish. (A CTA must read through the
// coherent path: what it needs is written while it is already resident.)
__device__ __forceinline__ void afterPredecessor() {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// One choice of operator per packet.
template <int N, typename A>
__device__ __forceinline__ void foldPacket(int op, A* acc, const A* b) {
  auto each = [&](auto f) {
#pragma unroll
    for (int e = 0; e < N; ++e) acc[e] = f(acc[e], b[e]);
  };
  switch (op) {
    case hlProd: each([](A x, A y) { return applyOp((int)hlProd, x, y); }); break;
    case hlMax: each([](A x, A y) { return applyOp((int)hlMax, x, y); }); break;
    case hlMin: each([](A x, A y) { return applyOp((int)hlMin, x, y); }); break;
    default: each([](A x, A y) { return applyOp((int)hlSum, x, y); }); break;
  }
}

// Bound by memory. A thread folds U packets: it has the loads of all their operands in flight at once (the operand
// count is compiled in, in classes), adds in a fixed order and stores. The grid covers the message; CTAs that retire
// and start keep more loads in flight than a resident grid whose threads alternate between loading and storing
// (4 x 32 MiB of bf16 into one on B200: 26.8 us = 6.3 TB/s against 28.7; before, with the sources in a run-time loop
// four packets deep and the operator chosen per element, 38.9). With one or two operands a thread that folds a single
// packet is gone before its CTA has cost less than it moved: U is four there, while the CTAs still fill the SMs (28 MB
// copied: 16.3 us with one packet, 12.3 with four). A caller's own block count makes it loop.
// kSum: the operator is known to be an addition; otherwise it is looked up per packet (per element a fold of two 32 MiB
// sources of bf16 took 42.9 us, 12.7 now). The widest class gives up registers for a fourth CTA per SM (five operands of
// 32 MiB, bf16: 51.2 us with two CTAs, 33.7 with four).
template <typename T, int MR, int U, bool kSum>
__global__ void __launch_bounds__(kRlThreads, MR <= 4 ? 0 : (sizeof(T) == 1 ? 3 : 4)) kReduceLanding(const __grid_constant__ nvl::ReduceLandingArgs a,
                                                                                                              const void* const first, int n) {
  afterPredecessor();
  constexpr int N = Packet<T>::N;
  using Acc = typename Wire<T>::Acc;
  const uint64_t tid = (uint64_t)blockIdx.x * kRlThreads + threadIdx.x;
  const uint64_t nthreads = (uint64_t)gridDim.x * kRlThreads;
  // operand 0 is `first` (dst itself when accumulating), operand q > 0 is source q - accumulate
  auto operand = [&](int q) { return q == 0 ? first : a.src[q - (a.accumulate ? 1 : 0)]; };
  bool vec = aligned16(a.dst);
#pragma unroll
  for (int q = 0; q < MR; ++q)
    if (q < n) vec = vec && aligned16(operand(q));
  const uint64_t np = vec ? a.count / N : 0;  // whole packets handled by the vector loop
  T* dst = reinterpret_cast<T*>(a.dst);
  for (uint64_t i0 = (uint64_t)blockIdx.x * (kRlThreads * U) + threadIdx.x; i0 < np; i0 += nthreads * U) {
    uint4 v[U][MR];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int q = 0; q < MR; ++q)
        if (q < n && i0 + u * kRlThreads < np) v[u][q] = reinterpret_cast<const uint4*>(operand(q))[i0 + u * kRlThreads];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * kRlThreads < np) {
        Acc acc[N], b[N];
        Packet<T>::unpack(v[u][0], acc);
#pragma unroll
        for (int q = 1; q < MR; ++q)
          if (q < n) {
            Packet<T>::unpack(v[u][q], b);
            foldPacket<N>(kSum ? (int)hlSum : a.op, acc, b);
          }
        finish<T>(acc, a.scale, 0);
        reinterpret_cast<uint4*>(dst)[i0 + u * kRlThreads] = Packet<T>::pack(acc);
      }
  }
  // ragged tail, or everything when some pointer is not 16-byte aligned
  for (uint64_t e = np * N + tid; e < a.count; e += nthreads) {
    Acc acc = Wire<T>::up(reinterpret_cast<const T*>(first)[e]);
    for (int q = 1; q < n; ++q) acc = applyOp(a.op, acc, Wire<T>::up(reinterpret_cast<const T*>(operand(q))[e]));
    if constexpr (Wire<T>::kFloat) { if (a.scale != 1.0f) acc = (Acc)(acc * (Acc)a.scale); }
    dst[e] = Wire<T>::down(acc);
  }
}

// Plain device-to-device copy of whole 16-byte packets (the one-rank form of every collective). Like the fold, the
// grid covers the message: 128 MiB in 43.1 us (6.2 TB/s) against 46.6 with a resident grid. U packets per thread:
// one while the message leaves SMs idle, four above, where fewer CTAs do.
constexpr int kCopyThreads = 256;
template <int U>
__global__ void __launch_bounds__(kCopyThreads) kCopyPackets(uint4* dst, const uint4* src, uint64_t packets) {
  afterPredecessor();
  const uint64_t i0 = (uint64_t)blockIdx.x * (kCopyThreads * U) + threadIdx.x;
  uint4 v[U];
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (i0 + u * kCopyThreads < packets) v[u] = src[i0 + u * kCopyThreads];
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (i0 + u * kCopyThreads < packets) dst[i0 + u * kCopyThreads] = v[u];
}

__global__ void kWarmup(int* sink) {
  if (sink && threadIdx.x == 0) *sink = 1;
}

// Bounded doorbell: the profile shows `tag` through the launch's NVTX-free
// name argument instead of one symbol per (op, rank, slot).
__global__ void kDoorbell(volatile uint64_t* ready, uint64_t ready_value, volatile uint64_t* complete,
                          uint64_t wait_value, uint64_t timeout_ns, uint64_t* status, const char* tag) {
  (void)tag;
  if (ready) {
    *ready = ready_value;
    __threadfence_system();
  }
  if (!complete) return;
  const uint64_t t0 = globalTimerNs();
  uint32_t spins = 0;
  while (*complete < wait_value) {
    if ((++spins & 15u) == 0) {
      __nanosleep(200);
      if (globalTimerNs() - t0 > timeout_ns) {
        if (status) {
          *reinterpret_cast<volatile uint64_t*>(status) = HL_DEV_TIMEOUT;
          __threadfence_system();
        }
        return;
      }
    }
  }
}

}  // namespace dev

namespace nvl {

// A launch that does not wait for its predecessor in the stream to drain (afterPredecessor).
static cudaError_t launchEarly(const void* fn, unsigned blocks, unsigned threads, void** args, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.stream = stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

// Operand classes: 2 (one source into an accumulator), 4, 9. `packets` of a thread: 1, or what reduceLandingUnroll says.
static int reduceLandingUnroll(int operands) { return operands > 2 ? 1 : 4; }
template <typename T, bool kSum>
static const void* reduceLandingClass(int operands, int packets) {
  using namespace dev;
  if (operands <= 2) return packets == 1 ? (const void*)kReduceLanding<T, 2, 1, kSum> : (const void*)kReduceLanding<T, 2, 4, kSum>;
  if (operands <= 4) return (const void*)kReduceLanding<T, 4, 1, kSum>;
  return (const void*)kReduceLanding<T, 9, 1, kSum>;
}
template <typename T>
static const void* reduceLandingFor(int operands, bool sum, int packets) {
  return sum ? reduceLandingClass<T, true>(operands, packets) : reduceLandingClass<T, false>(operands, packets);
}
static const void* reduceLandingFn(int dt, int operands, bool sum, int packets) {
  switch (dt) {
    case hlInt8: return reduceLandingFor<int8_t>(operands, sum, packets);
    case hlUint8: return reduceLandingFor<uint8_t>(operands, sum, packets);
    case hlInt32: return reduceLandingFor<int32_t>(operands, sum, packets);
    case hlUint32: return reduceLandingFor<uint32_t>(operands, sum, packets);
    case hlInt64: return reduceLandingFor<long long>(operands, sum, packets);
    case hlUint64: return reduceLandingFor<unsigned long long>(operands, sum, packets);
    case hlFloat16: return reduceLandingFor<__half>(operands, sum, packets);
    case hlFloat32: return reduceLandingFor<float>(operands, sum, packets);
    case hlFloat64: return reduceLandingFor<double>(operands, sum, packets);
    case hlBfloat16: return reduceLandingFor<__nv_bfloat16>(operands, sum, packets);
    default: return nullptr;
  }
}

hlResult_t launchReduceLanding(const ReduceLandingArgs& a, int blocks, cudaStream_t stream) {
  if (a.nsrc < 1 || a.nsrc > 8) return fail(hlInvalidArgument, "reduce landing: nsrc %d out of [1,8]", a.nsrc);
  int operands = a.nsrc + (a.accumulate ? 1 : 0);
  const bool sum = a.op == hlSum || a.op == hlAvg || operands == 1;   // one operand: nothing to choose
  const uint64_t packets = (a.count * hlTypeSize((hlDataType_t)a.dtype) + 15) / 16;
  int unroll = reduceLandingUnroll(operands);
  if (packets < (uint64_t)148 * 8 * dev::kRlThreads * unroll) unroll = 1;   // fewer than eight CTAs per SM
  const void* fn = reduceLandingFn(a.dtype, operands, sum, unroll);
  if (!fn) return fail(hlUnsupported, "reduce landing: unsupported dtype %d", a.dtype);
  if (a.count == 0) return hlSuccess;
  const uint64_t per_block = (uint64_t)dev::kRlThreads * unroll;
  if (blocks <= 0) blocks = (int)std::min<uint64_t>((packets + per_block - 1) / per_block, 1u << 30);
  const void* first = a.accumulate ? a.dst : a.src[0];
  void* args[3] = {(void*)&a, (void*)&first, (void*)&operands};
  cudaError_t e = launchEarly(fn, (unsigned)blocks, dev::kRlThreads, args, stream);
  if (e != cudaSuccess) return fail(hlDeviceError, "reduce landing launch: %s", cudaGetErrorString(e));
  return hlSuccess;
}

// dst and src 16-byte aligned, bytes a multiple of 16 (the caller sends anything else through launchReduceLanding).
hlResult_t launchCopy(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  const uint64_t packets = bytes / 16;
  if (!packets) return hlSuccess;
  const int unroll = packets >= (uint64_t)148 * 8 * dev::kCopyThreads * 4 ? 4 : 1;   // from 19 MiB: four packets still fill every SM
  const uint64_t per_block = (uint64_t)dev::kCopyThreads * unroll;
  const unsigned blocks = (unsigned)((packets + per_block - 1) / per_block);
  void* args[3] = {&dst, &src, (void*)&packets};
  cudaError_t e = launchEarly(unroll == 4 ? (const void*)dev::kCopyPackets<4> : (const void*)dev::kCopyPackets<1>, blocks, dev::kCopyThreads, args, stream);
  if (e != cudaSuccess) return fail(hlDeviceError, "copy launch: %s", cudaGetErrorString(e));
  return hlSuccess;
}

hlResult_t prepareReduceLanding() {
  for (int dt = 0; dt < hlNumTypes; ++dt)
    for (int operands : {2, 4, 9})
      for (bool sum : {false, true})
        for (int packets : {1, reduceLandingUnroll(operands)}) {
          cudaFuncAttributes at;
          cudaError_t e = cudaFuncGetAttributes(&at, reduceLandingFn(dt, operands, sum, packets));
          if (e != cudaSuccess) return fail(hlDeviceError, "cudaFuncGetAttributes: %s", cudaGetErrorString(e));
        }
  cudaFuncAttributes at;
  cudaFuncGetAttributes(&at, (const void*)dev::kCopyPackets<1>);
  cudaFuncGetAttributes(&at, (const void*)dev::kCopyPackets<4>);
  cudaFuncGetAttributes(&at, (const void*)dev::kDoorbell);
  cudaFuncGetAttributes(&at, (const void*)dev::kWarmup);
  return hlSuccess;
}

hlResult_t launchWarmup(cudaStream_t stream) {
  dev::kWarmup<<<1, 32, 0, stream>>>(nullptr);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(hlDeviceError, "warm-up launch: %s", cudaGetErrorString(e));
  return hlSuccess;
}

hlResult_t launchDoorbell(volatile uint64_t* ready, uint64_t ready_value, volatile uint64_t* complete,
                          uint64_t wait_value, uint64_t timeout_ns, uint64_t* status, const char* tag,
                          cudaStream_t stream) {
  dev::kDoorbell<<<1, 1, 0, stream>>>(ready, ready_value, complete, wait_value, timeout_ns, status, tag);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(hlDeviceError, "doorbell launch: %s", cudaGetErrorString(e));
  return hlSuccess;
}

}  // namespace nvl
}  // namespace hl
