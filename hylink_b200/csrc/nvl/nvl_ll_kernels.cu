// Low-latency kernels of the dedicated-link path for small messages: all-reduce, reduce-scatter, all-gather,
// all-to-all and broadcast with NO cross-GPU barrier at all.
//
// The barrier-based kernels (nvl_kernels.cuh) pay two flag round trips per call — about 3 to 8 microseconds each
// once the stores in front of them have to be acknowledged — which is most of the time of a message of a few MiB.
// Here every 16-byte store carries its own arrival flag: 8 data bytes and two copies of a 32-bit call tag
// ({d0, tag, d1, tag}, one st.volatile.v4, so each 8-byte half validates itself), written straight into the
// receiver's low-latency region; the receiver spins on the packet itself until all tags match. One network
// traversal per hop, no fence, no second trip. The price is half the link bandwidth, so the host side uses these
// kernels only while latency decides (measured limits in NvlPath::lowLatencyChoice). An all-reduce in the case
// of np < n packets still ends only after some shard owner heard from every rank, which keeps the argument below.
//
// Region (per rank, behind the flag words of the symmetric region): [2 parities][2 phases][HL_MAX_RANKS sources]
// slots of ll_slot_bytes. A call uses the parity of its call index, so the slots it writes were last used two calls
// ago. That reuse is safe without any handshake: in each of these collectives every rank receives from every other
// rank (directly, or through a shard owner that did), so a rank can only FINISH call k+1 after every peer has
// STARTED sending in call k+1, i.e. after every peer has left call k (launches of one communicator are
// stream-ordered); barrier-based kernels in between synchronise all ranks anyway. The tag is
// 2 * call index + 1 (odd: never 0, the value of cleared memory) and differs from the tag that the same slot held two
// calls earlier.
//
// all-to-all:      send segment q to rank q       | receive segment s from rank s into slot s of the output
// all-gather:      send own segment to every peer | receive the others' segments into the output
// reduce-scatter:  send segment q to rank q       | receive n-1 contributions, add in rank order, store
// all-reduce:      reduce-scatter of the n shards (phase 0), then all-gather of the reduced shards (phase 1)
//   in one hop:    all-gather of the whole buffers, added by everybody (the sum order is the same)
// broadcast:       the root sends its buffer to every peer; the others send packet 0 alone, as the sign that they have
//                  started, and everybody waits for all of these (the argument above needs it)
//
// All of this is latency. A call is a chain of L2 round trips (0.3 us each and more): the call's words, the caller's
// data, the packet on its way, the poll that finds it; so whatever a step does not need is out of its way. The first
// column of data is loaded before the call index is known, the abort word and the call index come at addresses that
// are launch arguments, and the count of started CTAs is taken after the sends.
// 8 KiB between ranks of one GPU, us per call before and after: all-gather of 2 ranks 6.1 / 4.1, of 8 6.1 / 4.1;
// all-reduce of 4 ranks 8.2 / 6.1.
// The period of a launch that waits for the one before it comes in steps of 2.05 us on this GPU, whatever the kernel:
// what a call saves shows when it crosses a step.
//
// Buffers: any device memory, any alignment, any element count; no type conversion. Sum order is by rank index on every rank: results are bitwise identical
// across ranks and runs.
//
// The reference has no kernels of its own on this path (it calls the vendor library:
// multipath-orchestrator/libampccl/core/virtual_collective.h:246-252); the protocol is the classic flag-in-data
// scheme of vendor collective libraries, written here from its description.
#include <cuda_runtime.h>

#include "nvl/nvl_device.cuh"
#include "nvl/nvl_launch.h"

namespace hl {
namespace dev {

constexpr int kLlAllReduce = 0, kLlReduceScatter = 1, kLlAllGather = 2, kLlAllToAll = 3, kLlBroadcast = 4, kLlAllReduceOneHop = 5;

__device__ __forceinline__ uint8_t* llSlot(const HlCommDev& c, int owner, int parity, int phase, int src) {
  return c.ll[owner] + ((size_t)((parity * 2 + phase) * HL_MAX_RANKS + src)) * c.ll_slot_bytes;
}

// One 16-byte data packet = two flagged 16-byte stores. Packets are laid out in groups of 32 (one warp): the 32
// first halves side by side (512 bytes), then the 32 second halves, so that each of the two store instructions of
// a warp — and each of the two polling loads — covers 512 contiguous bytes instead of every other 16.
__device__ __forceinline__ uint64_t llOffset(uint64_t j) { return (j >> 5) * 1024 + (j & 31) * 16; }

__device__ __forceinline__ void llSend(uint8_t* slot, uint64_t j, const uint4& v, uint32_t tag) {
  uint8_t* p = slot + llOffset(j);
  asm volatile("st.volatile.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(tag), "r"(v.y), "r"(tag) : "memory");
  asm volatile("st.volatile.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p + 512), "r"(v.z), "r"(tag), "r"(v.w), "r"(tag) : "memory");
}

struct LlWait {
  uint64_t t0;
  bool ok;
};

// Spins until packet j of every source in `pending` (a bit per rank) carries the tag; v[q] becomes the packet of q. The
// polls of all sources are in flight together: one after the other they are a chain of as many memory latencies
// (8 ranks, 64 KiB all-reduce: 12.7 us of kernel, two chains of seven). Bounded: after timeout_ns (or when the
// communicator is poisoned) it records where it gave up, poisons the communicator and returns false; the caller leaves
// the kernel.
__device__ __forceinline__ bool llRecv(const HlCommDev& c, const uint8_t* slots, uint64_t j, uint32_t tag, uint32_t pending, LlWait& w, uint4* v) {
  const uint8_t* p = slots + llOffset(j);
  const uint64_t stride = c.ll_slot_bytes;
  uint32_t spins = 0;
  for (;;) {
    uint4 a[HL_MAX_RANKS], b[HL_MAX_RANKS];
#pragma unroll
    for (int q = 0; q < HL_MAX_RANKS; ++q)
      if (pending >> q & 1u) {
        const uint8_t* s = p + q * stride;
        asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(a[q].x), "=r"(a[q].y), "=r"(a[q].z), "=r"(a[q].w) : "l"(s) : "memory");
        asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(b[q].x), "=r"(b[q].y), "=r"(b[q].z), "=r"(b[q].w) : "l"(s + 512) : "memory");
      }
#pragma unroll
    for (int q = 0; q < HL_MAX_RANKS; ++q)
      if ((pending >> q & 1u) && a[q].y == tag && a[q].w == tag && b[q].y == tag && b[q].w == tag) {
        v[q] = make_uint4(a[q].x, a[q].z, b[q].x, b[q].z);
        pending &= ~(1u << q);
      }
    if (!pending) return true;
    // a late peer (milliseconds, when the call overlaps with compute) must not have thousands of threads hammer L2
    // (an ordinary wait is a handful of polls and never gets here)
    if (++spins > 64) __nanosleep(spins > 1024 ? 400 : 50);
    if ((spins & 63u) == 0) {
      const uint64_t now = globalTimerNs();
      if (w.t0 == 0) w.t0 = now;
      const bool aborted = *reinterpret_cast<volatile uint32_t*>(c.abort_word) != 0;
      if (aborted || now - w.t0 > c.timeout_ns) {
        if (!aborted) {
          volatile uint64_t* st = c.status;
          st[1] = ((uint64_t)8 << 32) | (uint64_t)(__ffs(pending) - 1);   // step 8: a low-latency packet that never arrived
          st[2] = blockIdx.x;
          st[0] = HL_DEV_TIMEOUT;
          *reinterpret_cast<volatile uint32_t*>(c.abort_word) = 1;
          __threadfence_system();
        }
        w.ok = false;
        return false;
      }
    }
  }
}

template <typename W>
__device__ __forceinline__ uint4 llReduce(const uint4* v, int n, int op, float scale, int int_div) {
  constexpr int N = Packet<W>::N;
  typename Wire<W>::Acc acc[N], b[N];
  Packet<W>::unpack(v[0], acc);
  if (op == hlSum || op == hlAvg) {
#pragma unroll
    for (int q = 1; q < HL_MAX_RANKS; ++q)
      if (q < n) {
        Packet<W>::unpack(v[q], b);
#pragma unroll
        for (int i = 0; i < N; ++i) acc[i] = (typename Wire<W>::Acc)(acc[i] + b[i]);
      }
  } else {
#pragma unroll
    for (int q = 1; q < HL_MAX_RANKS; ++q)
      if (q < n) {
        Packet<W>::unpack(v[q], b);
#pragma unroll
        for (int i = 0; i < N; ++i) acc[i] = applyOp(op, acc[i], b[i]);
      }
  }
  finish<W>(acc, scale, int_div);
  return Packet<W>::pack(acc);
}

// `count`: elements of the whole buffer (all-reduce) or of one segment (the others). User buffers may have any
// alignment and any element count: packets are loaded and stored through loadUserPacket / storeUserPacket (vector
// accesses when the segment is 16-byte aligned and the packet whole, element by element otherwise; lanes past the
// end travel as zeros and are never stored). Whether a call takes these kernels therefore depends on sizes and
// types only, which are the same on every rank - never on a pointer, which need not be.
// Every thread keeps the same packet indices in every loop of the kernel, which is what makes the in-place forms
// safe (a location is read by the thread that later overwrites it, earlier in program order).
// All loads of a packet's column are issued before its first send: the stores are volatile, and a load behind one of
// them would wait for its turn.
template <typename W, int kColl>
__global__ void __launch_bounds__(HL_LL_THREADS) kLowLatency(const HlCommDev* comms, HlEmuCalls calls) {
  const HlCommDev& c = comms[blockIdx.y];
  HlCallArgs a = calls.c[blockIdx.y];
  const uint32_t aborted = *reinterpret_cast<volatile uint32_t*>(a.abort_word);
  a.seq = *reinterpret_cast<volatile uint64_t*>(a.seq_words);   // used once the first column has been asked for
  constexpr int N = Packet<W>::N, MR = HL_MAX_RANKS;
  const int n = a.nranks, r = a.rank;
  const uint64_t g0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, gstride = (uint64_t)gridDim.x * blockDim.x;
  const W* in = reinterpret_cast<const W*>(a.in);
  W* out = reinterpret_cast<W*>(a.out);
  const uint64_t cnt = a.count;
  const uint64_t np = (cnt + N - 1) / N;
  // shard q of an all-reduce = packets [q * sp, min(np, (q + 1) * sp)) of the whole buffer; rank q reduces it
  const uint64_t sp = kColl == kLlAllReduce ? (np + n - 1) / n : np;
  // packet j of the segment that starts at element `base` of a buffer
  auto ld = [&](const W* seg, uint64_t j) { return loadUserPacket<W, W>(seg, j * N, cnt, aligned16(seg)); };
  auto st = [&](W* seg, uint64_t j, const uint4& v) { storeUserPacket<W, W>(seg, j * N, cnt, aligned16(seg), v); };
  const uint32_t peers = ((1u << n) - 1u) & ~(1u << r);
  uint4 v[MR];   // indexed by compile-time constants only: stays in registers
  // what this rank has of column j
  auto column = [&](uint64_t j) {
    if constexpr (kColl == kLlAllGather || kColl == kLlAllReduceOneHop) {
      v[0] = ld(in, j);
    } else if constexpr (kColl == kLlBroadcast) {
      v[0] = r == a.root ? ld(in, j) : make_uint4(0u, 0u, 0u, 0u);
    } else {
#pragma unroll
      for (int q = 0; q < MR; ++q)
        if (kColl == kLlAllToAll ? q < n : (peers >> q & 1u)) {
          if constexpr (kColl == kLlAllReduce) {
            if ((uint64_t)q * sp + j < np) v[q] = ld(in, (uint64_t)q * sp + j);
          } else {
            v[q] = ld(in + (uint64_t)q * a.in_seg_stride, j);
          }
        }
    }
  };
  if (g0 < sp) column(g0);

  const uint32_t call = (uint32_t)(a.seq / HL_SEQ_STRIDE);
  const uint32_t tag = 2u * call + 1u;
  const int parity = (int)(call & 1u);
  // the slot of this rank at every peer, and this rank's own slots, by phase
  uint8_t* to[MR];
#pragma unroll
  for (int q = 0; q < MR; ++q)
    if (q < n) to[q] = llSlot(c, q, parity, 0, r);
  const uint64_t phase2 = (uint64_t)HL_MAX_RANKS * c.ll_slot_bytes;   // from a phase-0 slot to its phase-1 counterpart
  const uint8_t* from = llSlot(c, r, parity, 0, 0);
  // the columns of this thread; none on a poisoned communicator (a no-op instead of a second hang candidate)
  const uint64_t end = aborted ? 0 : sp;
  LlWait w;
  w.t0 = 0;
  w.ok = true;
  for (uint64_t j = g0; j < end;) {
#pragma unroll
    for (int q = 0; q < MR; ++q)
      if (peers >> q & 1u) {
        if constexpr (kColl == kLlAllGather || kColl == kLlAllReduceOneHop) llSend(to[q], j, v[0], tag);
        else if constexpr (kColl == kLlBroadcast) {
          if (r == a.root || j == 0) llSend(to[q], j, v[0], tag);
        } else if constexpr (kColl == kLlAllReduce) {
          if ((uint64_t)q * sp + j < np) llSend(to[q], j, v[q], tag);
        } else {
          llSend(to[q], j, v[q], tag);
        }
      }
    if constexpr (kColl == kLlAllGather) st(out + (uint64_t)r * a.out_seg_stride, j, v[0]);
    if constexpr (kColl == kLlBroadcast)
      if (r == a.root && in != out) st(out, j, v[0]);
    if constexpr (kColl == kLlAllToAll) {
#pragma unroll
      for (int q = 0; q < MR; ++q)   // after every read of this thread's column: in place is safe
        if (q == r) st(out + (uint64_t)r * a.out_seg_stride, j, v[q]);
    }
    j += gstride;
    if (j < end) column(j);
  }
  __syncthreads();                   // every thread has its call index
  countEntry(a, 0);
  timelineEntry(c, a);

  if constexpr (kColl == kLlAllGather || kColl == kLlAllToAll) {
    for (uint64_t j = g0; j < end && llRecv(c, from, j, tag, peers, w, v); j += gstride) {
#pragma unroll
      for (int q = 0; q < MR; ++q)
        if (peers >> q & 1u) st(out + (uint64_t)q * a.out_seg_stride, j, v[q]);
    }
  } else if constexpr (kColl == kLlBroadcast) {
    const uint32_t root = peers & (1u << a.root);                  // 0 on the root itself
    for (uint64_t j = g0; j < end; j += gstride) {
      const uint32_t have = j == 0 ? peers : root;
      if (!have || !llRecv(c, from, j, tag, have, w, v)) break;    // the root waits with the thread of packet 0 only
#pragma unroll
      for (int q = 0; q < MR; ++q)
        if (root >> q & 1u) st(out, j, v[q]);
    }
  } else if constexpr (kColl == kLlReduceScatter || kColl == kLlAllReduceOneHop) {
    for (uint64_t j = g0; j < end; j += gstride) {
      const uint4 own = ld(kColl == kLlReduceScatter ? in + (uint64_t)r * a.in_seg_stride : in, j);
      if (!llRecv(c, from, j, tag, peers, w, v)) break;
#pragma unroll
      for (int q = 0; q < MR; ++q)
        if (q == r) v[q] = own;
      st(out, j, llReduce<W>(v, n, a.op, a.scale, a.int_div));
    }
  } else {
    const uint64_t first = (uint64_t)r * sp;
    const uint64_t mine = first >= np || aborted ? 0 : (np - first < sp ? np - first : sp);
    for (uint64_t j = g0; j < mine; j += gstride) {
      const uint4 own = ld(in, first + j);
      if (!llRecv(c, from, j, tag, peers, w, v)) break;
#pragma unroll
      for (int q = 0; q < MR; ++q)
        if (q == r) v[q] = own;
      const uint4 red = llReduce<W>(v, n, a.op, a.scale, a.int_div);
#pragma unroll
      for (int q = 0; q < MR; ++q)
        if (peers >> q & 1u) llSend(to[q] + phase2, j, red, tag);
      st(out, first + j, red);
    }
    for (uint64_t j = g0; j < end && w.ok; j += gstride) {
      uint32_t have = 0;
#pragma unroll
      for (int q = 0; q < MR; ++q)
        if ((peers >> q & 1u) && (uint64_t)q * sp + j < np) have |= 1u << q;
      if (have && !llRecv(c, from + phase2, j, tag, have, w, v)) break;
#pragma unroll
      for (int q = 0; q < MR; ++q)
        if (have >> q & 1u) st(out, (uint64_t)q * sp + j, v[q]);
    }
  }
  // a thread that gave up has poisoned the communicator; the others find the abort word in their own waits
  callDone(c, a);
}

}  // namespace dev

namespace nvl {

template <typename W>
static const void* pickLl(int kind) {
  using namespace dev;
  switch (kind) {
    case kNvlLlAllReduce: return (const void*)kLowLatency<W, kLlAllReduce>;
    case kNvlLlReduceScatter: return (const void*)kLowLatency<W, kLlReduceScatter>;
    case kNvlLlAllGather: return (const void*)kLowLatency<W, kLlAllGather>;
    case kNvlLlAllToAll: return (const void*)kLowLatency<W, kLlAllToAll>;
    case kNvlLlBroadcast: return (const void*)kLowLatency<W, kLlBroadcast>;
    case kNvlLlAllReduceOneHop: return (const void*)kLowLatency<W, kLlAllReduceOneHop>;
    default: return nullptr;
  }
}

const void* lowLatencyKernelFor(int kind, int wire_dt) {
  switch (wire_dt) {
    case hlInt8: return pickLl<int8_t>(kind);
    case hlUint8: return pickLl<uint8_t>(kind);
    case hlInt32: return pickLl<int32_t>(kind);
    case hlUint32: return pickLl<uint32_t>(kind);
    case hlInt64: return pickLl<long long>(kind);
    case hlUint64: return pickLl<unsigned long long>(kind);
    case hlFloat16: return pickLl<__half>(kind);
    case hlFloat32: return pickLl<float>(kind);
    case hlFloat64: return pickLl<double>(kind);
    case hlBfloat16: return pickLl<__nv_bfloat16>(kind);
    default: return nullptr;
  }
}

}  // namespace nvl
}  // namespace hl
