// Launch side of the dedicated-link kernels (nvl_kernels.cuh): which kernel a call runs and how it is launched.
#include <cuda_runtime.h>

#include <bitset>
#include <mutex>

#include "nvl/nvl_device.cuh"
#include "nvl/nvl_launch.h"

namespace hl {
namespace dev {
constexpr int kPipeWarpGroupThreads = 384;
__global__ void __launch_bounds__(HL_NVL_THREADS) kBarrier(const HlCommDev* comms, HlEmuCalls calls) {
  const HlCommDev& c = comms[blockIdx.y];
  HlCallArgs a = calls.c[blockIdx.y];
  if (!entryOk(c, a)) return;
  blockBarrier(c, a, 1, 1);
  callDone(c, a);
}
}  // namespace dev

namespace nvl {

template <typename W>
const void* pickKernelT(int kind, int nranks);   // nvl_kernels_*.cu
template <typename W>
const void* pickStreamT(int kind, int nranks);   // nvl_stream_*.cu

static bool streamed(int kind) { return kind == kNvlStreamReduceScatter || kind == kNvlStreamAllGather || kind == kNvlStreamAllToAll || kind == kNvlStreamBroadcast; }
template <typename W>
static const void* pick(int kind, int nranks) {
  return streamed(kind) ? pickStreamT<W>(kind, nranks) : pickKernelT<W>(kind, nranks);
}

const void* kernelFor(int kind, int wire_dt, int nranks) {
  if (kind == kNvlBarrier) return (const void*)dev::kBarrier;
  if (kind == kNvlLlAllReduce || kind == kNvlLlReduceScatter || kind == kNvlLlAllGather || kind == kNvlLlAllToAll ||
      kind == kNvlLlBroadcast || kind == kNvlLlAllReduceOneHop)
    return lowLatencyKernelFor(kind, wire_dt);
  switch (wire_dt) {
    case hlInt8: return pick<int8_t>(kind, nranks);
    case hlUint8: return pick<uint8_t>(kind, nranks);
    case hlInt32: return pick<int32_t>(kind, nranks);
    case hlUint32: return pick<uint32_t>(kind, nranks);
    case hlInt64: return pick<long long>(kind, nranks);
    case hlUint64: return pick<unsigned long long>(kind, nranks);
    case hlFloat16: return pick<__half>(kind, nranks);
    case hlFloat32: return pick<float>(kind, nranks);
    case hlFloat64: return pick<double>(kind, nranks);
    case hlBfloat16: return pick<__nv_bfloat16>(kind, nranks);
    default: return nullptr;
  }
}

const char* kernelName(int kind) {
  switch (kind) {
    case kNvlBarrier: return "barrier";
    case kNvlAllReduceOneShot: return "allreduce_oneshot";
    case kNvlAllReduceTwoShot: return "allreduce_twoshot_p2p";
    case kNvlAllReduceNvls: return "allreduce_nvls";
    case kNvlReduceScatter: return "reducescatter_p2p";
    case kNvlReduceScatterNvls: return "reducescatter_nvls";
    case kNvlAllGather: return "allgather_p2p";
    case kNvlBroadcast: return "broadcast_p2p";
    case kNvlAllToAll: return "alltoall_p2p";
    case kNvlAllGatherNvls: return "allgather_nvls";
    case kNvlBroadcastNvls: return "broadcast_nvls";
    case kNvlAllReducePush: return "allreduce_push";
    case kNvlReduceScatterPush: return "reducescatter_push";
    case kNvlAllGatherPush: return "allgather_push";
    case kNvlAllGatherLanes: return "allgather_lanes";
    case kNvlAllReducePipeP2p: return "allreduce_pipelined_p2p";
    case kNvlAllReducePipeNvls: return "allreduce_pipelined_nvls";
    case kNvlReduceScatterPipeP2p: return "reducescatter_pipelined_p2p";
    case kNvlReduceScatterPipeNvls: return "reducescatter_pipelined_nvls";
    case kNvlZcAllReduceNvls: return "allreduce_zerocopy_nvls";
    case kNvlZcAllReduceP2p: return "allreduce_zerocopy_p2p";
    case kNvlZcReduceScatterNvls: return "reducescatter_zerocopy_nvls";
    case kNvlZcReduceScatterP2p: return "reducescatter_zerocopy_p2p";
    case kNvlZcAllGatherNvls: return "allgather_zerocopy_nvls";
    case kNvlZcAllGatherP2p: return "allgather_zerocopy_p2p";
    case kNvlZcBroadcastNvls: return "broadcast_zerocopy_nvls";
    case kNvlZcBroadcastP2p: return "broadcast_zerocopy_p2p";
    case kNvlLlAllReduce: return "allreduce_lowlatency";
    case kNvlLlReduceScatter: return "reducescatter_lowlatency";
    case kNvlLlAllGather: return "allgather_lowlatency";
    case kNvlLlAllToAll: return "alltoall_lowlatency";
    case kNvlLlAllReduceOneHop: return "allreduce_lowlatency_onehop";
    case kNvlLlBroadcast: return "broadcast_lowlatency";
    case kNvlAllToAllPush: return "alltoall_push";
    case kNvlStreamReduceScatter: return "reducescatter_streamed";
    case kNvlStreamAllGather: return "allgather_streamed";
    case kNvlStreamAllToAll: return "alltoall_streamed";
    case kNvlStreamBroadcast: return "broadcast_streamed";
    default: return "?";
  }
}

hlResult_t launch(int kind, int wire_dt, const HlCommDev* dcomms, const HlEmuCalls& calls, int emu_ranks, int blocks,
                  cudaStream_t stream, int nranks, int threads) {
  const void* fn = kernelFor(kind, wire_dt, nranks);
  if (!fn) return fail(hlUnsupported, "no %s kernel for wire type %d", kernelName(kind), wire_dt);
  if (blocks < 1) blocks = 1;
  if (blocks > HL_MAX_BLOCKS) blocks = HL_MAX_BLOCKS;
  dim3 grid((unsigned)blocks, (unsigned)(emu_ranks > 1 ? emu_ranks : 1), 1);
  const bool pipe = kind == kNvlAllReducePipeNvls || kind == kNvlReduceScatterPipeNvls;  // warp-group stages: 384 threads
  if (streamed(kind)) threads = HL_STREAM_WORKERS + 64;
  dim3 block((unsigned)(threads > 0 ? threads : (pipe ? dev::kPipeWarpGroupThreads : HL_NVL_THREADS)), 1, 1);
  void* args[2] = {(void*)&dcomms, (void*)&calls};
  cudaError_t e;
  if (emu_ranks > 1) {
    // The emulated ranks wait on one another: all their blocks must be
    // co-resident, which only a cooperative launch guarantees (it fails
    // cleanly instead of deadlocking when they would not fit).
    e = cudaLaunchCooperativeKernel(fn, grid, block, args, 0, stream);
  } else {
    e = cudaLaunchKernel(fn, grid, block, args, 0, stream);
  }
  if (e != cudaSuccess) return fail(hlDeviceError, "launch of %s failed: %s", kernelName(kind), cudaGetErrorString(e));
  return hlSuccess;
}

hlResult_t prepareKernels() {
  // Resolve every variant once on the init thread: lazy module loading plus
  // concurrent first launches from several threads can deadlock in the driver
  // (same cure as pcie-ccl-cuda/kernels/wait_kernel.cu:216-234,400-432).
  // Once per device: the thousand queries take 1.5 ms, which every later group of the process would wait for.
  static std::mutex mu;
  static std::bitset<64> done;
  int device = 0;
  cudaError_t got = cudaGetDevice(&device);
  if (got != cudaSuccess) return fail(hlDeviceError, "cudaGetDevice: %s", cudaGetErrorString(got));
  std::lock_guard<std::mutex> lock(mu);
  if (device < 64 && done[device]) return hlSuccess;
  static const int kinds[] = {kNvlBarrier, kNvlAllReduceOneShot, kNvlAllReduceTwoShot, kNvlAllReduceNvls,
                              kNvlReduceScatter, kNvlReduceScatterNvls, kNvlAllGather, kNvlBroadcast,
                              kNvlAllToAll, kNvlAllGatherNvls, kNvlBroadcastNvls, kNvlAllReducePipeP2p,
                              kNvlAllReducePipeNvls, kNvlReduceScatterPipeP2p, kNvlReduceScatterPipeNvls, kNvlAllReducePush,
                              kNvlReduceScatterPush, kNvlAllGatherPush, kNvlAllGatherLanes, kNvlZcAllReduceNvls,
                              kNvlZcAllReduceP2p, kNvlZcReduceScatterNvls, kNvlZcReduceScatterP2p, kNvlZcAllGatherNvls,
                              kNvlZcAllGatherP2p, kNvlZcBroadcastNvls, kNvlZcBroadcastP2p, kNvlLlAllReduce,
                              kNvlLlReduceScatter, kNvlLlAllGather, kNvlLlAllToAll, kNvlLlBroadcast, kNvlLlAllReduceOneHop, kNvlAllToAllPush,
                              kNvlStreamReduceScatter, kNvlStreamAllGather, kNvlStreamAllToAll, kNvlStreamBroadcast};
  for (int k : kinds)
    for (int dt = 0; dt < hlNumTypes; ++dt) {
      for (int nr : {2, 4, HL_MAX_RANKS}) {   // rank-count classes (only the pipelined push kernels differ by it)
        const void* fn = kernelFor(k, dt, nr);
        if (!fn) continue;
        cudaFuncAttributes at;
        cudaError_t e = cudaFuncGetAttributes(&at, fn);
        if (e != cudaSuccess) return fail(hlDeviceError, "cudaFuncGetAttributes: %s", cudaGetErrorString(e));
      }
      if (k == kNvlBarrier) break;
    }
  if (device < 64) done.set(device);
  return hlSuccess;
}

}  // namespace nvl
}  // namespace hl
