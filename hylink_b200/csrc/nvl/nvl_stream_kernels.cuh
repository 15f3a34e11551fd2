// Streamed kernels: large reduce-scatter, all-gather, all-to-all and broadcast between ranks of ONE GPU.
//
// Between GPUs the link is the bound and staging traffic hides behind it. Between ranks of one GPU the staging IS the
// traffic: a message through slots of its own size moves about 2.2 times the bytes that the caller's buffers hold, all
// of it through HBM. Here the message runs through a ring of small pieces instead, so that staging stays in L2 (a copy
// inside L2 runs at 12 to 13 TB/s, through HBM at 6.2) and HBM sees the caller's buffers alone.
//
// CTA b of every rank owns the same range of packets of every segment and walks it in pieces of P packets. In iteration
// t it
//   pushes piece t to the peers' slots (all-to-all: and copies its own to the output); of an all-gather, where all peers want the
//   same, it stores piece t once, into its own ring, and into the output,
//   folds piece t - L from the landed slots (reduce-scatter), or copies it to the output (the others; of an all-gather
//   from the senders' rings: 4 ranks x 16 MiB of bf16 102 us with a copy of every piece per peer, 98 with one, and 81 with pieces
//   of twice the size, for which the ring has room then),
// and may start once every peer's CTA b has finished iteration t - L. One rule covers arrival and reuse: what is read in
// iteration t was stored by a peer in iteration t - L or earlier, and a ring of R = 2 L pieces is overwritten no sooner
// than L iterations after its last reader. A lockstep (L = 1) waits for stores, flag and poll in every iteration, which
// costs as much as a piece; with a lag they have iterations to travel (4 x 64 MiB reduce-scatter: 110 us with L = 2, 99
// with 3, 102 with 4, whose ring is too large; with the plain kernel 119).
// An all-reduce has a second ring (results) and twice the lag, which no longer fits: 230 us against 125. It stays with
// the plain kernel.
// Broadcast: the root puts piece t into its own ring and into its output, the others copy piece t - L out of the root's
// ring. (With the whole message staged first, the others wait for the root's CTAs, an n-th of the GPU: 64 MiB
// to 8 ranks 249 us, streamed 180 to 200; to 4 ranks 132 and 96. The root's CTAs are the bound: they read once and store twice.)
// Flags are the tile words of the pipelined kernels: [kind 1][CTA][source rank] <- tile base + finished iterations.
//
// Roles: worker warps move data; a poller warp watches the peers' flags and opens iterations; a signaller warp waits
// until all workers are through one and pays for the release store. They meet on shared-memory barriers, one pair
// (open, done) per piece of the ring, and a worker warp waits for nobody but the poller: the warps drift apart by up to
// L iterations, so that some load while others store. (With a CTA barrier per iteration all warps load, then all store:
// 113 us instead of 107 at L = 2.) The caller's data of the next piece is loaded before the wait for it: that load needs
// no permission. (Bulk copies through shared memory by one thread each for the push and the copy-out took 173 us: every
// piece then also passes store completion, and its latency times the rate is more than a ring in L2 can hold.)
// The last wait, for every peer's last iteration, is rule A of nvl_kernels.cuh. Every wait is bounded.
//
// The host takes these kernels only for buffers whose segments all start on 16-byte boundaries; what is not a whole
// packet at the end of a segment goes element by element. Data in the ring is read past L1 (another SM wrote it), and
// the caller's buffers move with streaming hints, which keeps them from displacing the ring.
#pragma once
#include "nvl/nvl_kernels.cuh"

namespace hl {
namespace dev {

enum StreamColl { kStreamReduceScatter = 0, kStreamAllGather = 1, kStreamAllToAll = 2, kStreamBroadcast = 3 };
constexpr int kLag = HL_STREAM_LAG, kStreamRing = 2 * kLag;
constexpr int kWorkWarps = HL_STREAM_WORKERS / 32;

__device__ __forceinline__ uint4 ldRing(const uint4* p) { return __ldcg(p); }

__device__ __forceinline__ uint32_t sharedAddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbInit(uint64_t* b, int arrivals) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sharedAddr(b)), "r"(arrivals) : "memory");
}
__device__ __forceinline__ void mbArrive(uint64_t* b) {   // release at CTA scope
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sharedAddr(b)) : "memory");
}
// Waits for the phase of this parity (acquire at CTA scope); false when `*stop` forbids iteration t or the limit is reached.
__device__ __forceinline__ bool mbWait(uint64_t* b, uint32_t parity, volatile int* stop, int t, uint64_t limit_ns) {
  uint64_t t0 = 0;
  for (uint32_t spins = 0;; ++spins) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(sharedAddr(b)), "r"(parity)
        : "memory");
    if (done) return true;
    if (*stop <= t) return false;
    if ((spins & 15u) == 15u) {
      const uint64_t now = globalTimerNs();
      if (t0 == 0) t0 = now;
      if (now - t0 > limit_ns) return false;
    }
  }
}

template <typename W, int kColl, int MR>
__global__ void __launch_bounds__(HL_STREAM_WORKERS + 64, 1) kStream(const HlCommDev* comms, HlEmuCalls calls) {
  const HlCommDev& c = comms[blockIdx.y];
  HlCallArgs a = calls.c[blockIdx.y];
  constexpr bool kRs = kColl == kStreamReduceScatter, kBc = kColl == kStreamBroadcast;
  constexpr bool kAg = kColl == kStreamAllGather || kBc;       // one input, not one per peer
  constexpr int N = Packet<W>::N, V = (kAg && !kBc ? 16 : 8) / MR;   // packets of every segment per thread
  constexpr uint32_t P = HL_STREAM_WORKERS * V, kStep = HL_STREAM_WORKERS;
  const int n = c.nranks, r = c.rank;
  const uint64_t sp = (a.count + N - 1) / N;
  const uint64_t chunk = (sp + gridDim.x - 1) / gridDim.x;
  const int T = (int)((chunk + P - 1) / P);
  const int I = T + kLag;
  if (!entryOk(c, a, (uint64_t)I)) return;
  __shared__ volatile int s_stop;                     // the first iteration that must not run
  __shared__ __align__(8) uint64_t s_open[kStreamRing], s_done[kStreamRing];
  if (threadIdx.x == 0) {
    s_stop = 0x7fffffff;
    for (int i = 0; i < kStreamRing; ++i) {
      mbInit(&s_open[i], 1);
      mbInit(&s_done[i], kWorkWarps);
    }
  }
  __syncthreads();
  const uint64_t base = a.pipe_seq;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto parity = [](int t) { return (uint32_t)(t / kStreamRing) & 1u; };
  const uint64_t limit = 2 * c.timeout_ns + 1000000000ull;      // inside a CTA: the poller gives up first

  const Parts<W> in(a.in, kAg ? 0 : a.in_seg_stride, a.count, 0), out(a.out, kRs || kBc ? 0 : a.out_seg_stride, a.count, 0);
  const uint64_t c0 = (uint64_t)blockIdx.x * chunk, c1 = c0 + chunk < sp ? c0 + chunk : sp;
  const uint64_t ring0 = (uint64_t)blockIdx.x * kStreamRing * (kAg ? 1 : n) * P;                      // this CTA's ring in a rank's staging
  const uint64_t whole = a.count / N, v1 = c1 < whole ? c1 : whole;                       // vector copies end here
  // packets of piece t: how many are full
  auto first = [&](int t) { return c0 + (uint64_t)t * P; };
  auto full = [&](int t) { return first(t) >= v1 ? 0u : (v1 - first(t) < P ? (uint32_t)(v1 - first(t)) : P); };
  auto ragLoad = [&](const Parts<W>& b, int q, uint64_t j) { return loadUserPacket<W, W>(b.at(q), j * N, a.count, false); };
  auto ragStore = [&](const Parts<W>& b, int q, uint64_t j, const uint4& v) { storeUserPacket<W, W>(b.at(q), j * N, a.count, false, v); };
  // the ragged packet of piece t, if it has one: [ragged0, ragged1)
  auto ragged0 = [&](int t) { return first(t) + full(t); };
  auto ragged1 = [&](int t) { return first(t) + P < c1 ? first(t) + P : c1; };
  const bool own = in.at(kAg ? 0 : r) != out.at(kRs || kBc ? 0 : r);

  if (warp == 0) {                                    // ---- poller
    int gave_up = 0;
    for (int t = 0; t < I + kLag && !gave_up; ++t) {  // t >= I: only the final wait
      if (t >= kLag) {
        const uint64_t need = base + (uint64_t)(t - kLag) + 1;
        if (lane < n) {
          const uint64_t* mine = c.flags[r] + ((size_t)1 * HL_MAX_BLOCKS + blockIdx.x) * HL_MAX_RANKS + lane;
          uint64_t t0 = 0;
          uint32_t spins = 0;
          while (ldAcquire(true, mine) < need) {
            if ((++spins & 31u) == 0) {
              const uint64_t now = globalTimerNs();
              if (t0 == 0) t0 = now;
              const bool aborted = *reinterpret_cast<volatile uint32_t*>(c.abort_word) != 0;
              if (aborted || now - t0 > c.timeout_ns) {
                if (!aborted) {
                  volatile uint64_t* st = c.status;
                  st[1] = ((uint64_t)1 << 32) | (uint64_t)lane;
                  st[2] = blockIdx.x;
                  st[0] = HL_DEV_TIMEOUT;
                  *reinterpret_cast<volatile uint32_t*>(c.abort_word) = 1;
                  __threadfence_system();
                }
                gave_up = 1;
                break;
              }
            }
          }
        }
        gave_up = __any_sync(0xffffffffu, gave_up);
      }
      __syncwarp();                                   // every lane's acquire, before lane 0 lets the workers on (a vote orders no memory)
      if (lane == 0) {
        if (gave_up) s_stop = t;
        else if (t < I) mbArrive(&s_open[t % kStreamRing]);
      }
    }
  } else if (warp == 1) {                             // ---- signaller
    for (int t = 0; t < I; ++t) {
      if (!mbWait(&s_done[t % kStreamRing], parity(t), &s_stop, t, limit)) break;
      if (lane < n) stRelease(true, c.flags[lane] + ((size_t)1 * HL_MAX_BLOCKS + blockIdx.x) * HL_MAX_RANKS + r, base + (uint64_t)t + 1);
    }
  } else {                                            // ---- workers
    const uint32_t tid = threadIdx.x - 64;
    uint4* stage[MR];                                 // of the k-th peer
#pragma unroll
    for (int k = 1; k < MR; ++k)
      if (k < n) stage[k] = reinterpret_cast<uint4*>(c.stage[peerOf(r, k, n)]);
    uint4* const own_ring = reinterpret_cast<uint4*>(c.stage[r]);
    const uint4* mine = own_ring;
    constexpr int kFrom = kColl == kStreamAllToAll ? 0 : 1;      // all-to-all: the own segment travels with the others
    constexpr int kNext = kAg ? 1 : MR;
    uint4 next[V][kNext];                             // the caller's data of the piece to push
    auto fetch = [&](int t) {
      if (t >= T || (kBc && r != a.root)) return;
      const uint32_t cnt = full(t);
      if constexpr (kAg) {
        const uint4* src = reinterpret_cast<const uint4*>(in.at(0)) + first(t);
#pragma unroll
        for (int u = 0; u < V; ++u)
          if (tid + u * kStep < cnt) next[u][0] = __ldcs(src + tid + u * kStep);
      } else {
#pragma unroll
        for (int k = kFrom; k < MR; ++k)
          if (k < n && (k > 0 || own)) {
            const uint4* src = reinterpret_cast<const uint4*>(in.at(peerOf(r, k, n))) + first(t);
#pragma unroll
            for (int u = 0; u < V; ++u)
              if (tid + u * kStep < cnt) next[u][k] = __ldcs(src + tid + u * kStep);
          }
      }
    };
    const uint4* ring = kBc ? reinterpret_cast<const uint4*>(c.stage[a.root]) + ring0 : nullptr;
    fetch(0);
    for (int t = 0; t < I; ++t) {
      if (!mbWait(&s_open[t % kStreamRing], parity(t), &s_stop, t, limit)) break;
      if (kBc) {
        if (r == a.root && t < T) {                   // piece t into the ring and the output
          const uint32_t cnt = full(t);
          uint4* slot = reinterpret_cast<uint4*>(c.stage[r]) + ring0 + (uint64_t)(t % kStreamRing) * P;
          uint4* dst = reinterpret_cast<uint4*>(out.at(0)) + first(t);
#pragma unroll
          for (int u = 0; u < V; ++u)
            if (tid + u * kStep < cnt) slot[tid + u * kStep] = next[u][0];
          if (own) {
#pragma unroll
            for (int u = 0; u < V; ++u)
              if (tid + u * kStep < cnt) __stcs(dst + tid + u * kStep, next[u][0]);
          }
          for (uint64_t j = ragged0(t) + tid; j < ragged1(t); j += kStep) {
            const uint4 v = ragLoad(in, 0, j);
            slot[j - first(t)] = v;
            if (own) ragStore(out, 0, j, v);
          }
          fetch(t + 1);
        } else if (r != a.root && t >= kLag) {        // piece t - L out of it
          const int w = t - kLag;
          const uint32_t cnt = full(w);
          const uint4* landed = ring + (uint64_t)(w % kStreamRing) * P;
          uint4* dst = reinterpret_cast<uint4*>(out.at(0)) + first(w);
          uint4 v[V];
#pragma unroll
          for (int u = 0; u < V; ++u)
            if (tid + u * kStep < cnt) v[u] = ldRing(landed + tid + u * kStep);
#pragma unroll
          for (int u = 0; u < V; ++u)
            if (tid + u * kStep < cnt) __stcs(dst + tid + u * kStep, v[u]);
          for (uint64_t j = ragged0(w) + tid; j < ragged1(w); j += kStep) ragStore(out, 0, j, ldRing(landed + (j - first(w))));
        }
        __syncwarp();
        if (lane == 0) mbArrive(&s_done[t % kStreamRing]);
        continue;
      }
      if (t < T) {                                    // push piece t
        const uint64_t slot = ring0 + (kAg ? (uint64_t)(t % kStreamRing) : (uint64_t)(t % kStreamRing) * n + r) * P;
        const uint32_t cnt = full(t);
        if constexpr (kAg) {
#pragma unroll
          for (int u = 0; u < V; ++u)
            if (tid + u * kStep < cnt) own_ring[slot + tid + u * kStep] = next[u][0];
        } else {
#pragma unroll
          for (int k = 1; k < MR; ++k)
            if (k < n) {
#pragma unroll
              for (int u = 0; u < V; ++u)
                if (tid + u * kStep < cnt) stage[k][slot + tid + u * kStep] = next[u][k];
            }
        }
        if (!kRs && own) {
          uint4* dst = reinterpret_cast<uint4*>(out.at(r)) + first(t);
#pragma unroll
          for (int u = 0; u < V; ++u)
            if (tid + u * kStep < cnt) __stcs(dst + tid + u * kStep, next[u][0]);
        }
        for (uint64_t j = ragged0(t) + tid; j < ragged1(t); j += kStep) {
          if constexpr (kAg) {
            const uint4 v = ragLoad(in, 0, j);
            own_ring[slot + (j - first(t))] = v;
            if (own) ragStore(out, r, j, v);
          } else {
#pragma unroll 1
            for (int k = 0; k < n; ++k) {
              const int q = peerOf(r, k, n);
              if (k == 0 && (kRs || !own)) continue;
              const uint4 v = ragLoad(in, q, j);
              if (k == 0) ragStore(out, r, j, v);
              else reinterpret_cast<uint4*>(c.stage[q])[slot + (j - first(t))] = v;
            }
          }
        }
      }
      uint4 v[V][MR];
      if (kRs && t >= kLag) {                         // fold piece t - L
        const int w = t - kLag;
        const uint64_t p0 = first(w);
        const uint32_t cnt = full(w);
        const uint4* slots = mine + ring0 + (uint64_t)(w % kStreamRing) * n * P;
        const uint4* o = reinterpret_cast<const uint4*>(in.at(r)) + p0;
        uint4* dst = reinterpret_cast<uint4*>(out.at(0)) + p0;
#pragma unroll
        for (int q = 0; q < MR; ++q)                  // ascending rank order: the sum order
          if (q < n) {
#pragma unroll
            for (int u = 0; u < V; ++u)
              if (tid + u * kStep < cnt) v[u][q] = q == r ? __ldcs(o + tid + u * kStep) : ldRing(slots + (uint64_t)q * P + tid + u * kStep);
          }
        fetch(t + 1);
#pragma unroll
        for (int u = 0; u < V; ++u)
          if (tid + u * kStep < cnt) __stcs(dst + tid + u * kStep, reducePackets<W, MR>(v[u], n, a.op, a.scale, a.int_div));
        for (uint64_t j = ragged0(w) + tid; j < ragged1(w); j += kStep) {
          uint4 x[MR];
#pragma unroll
          for (int q = 0; q < MR; ++q)
            if (q < n && q != r) x[q] = ldRing(slots + (uint64_t)q * P + (j - p0));
          const uint4 ov = ragLoad(in, r, j);
#pragma unroll
          for (int q = 0; q < MR; ++q)
            if (q == r) x[q] = ov;
          ragStore(out, 0, j, reducePackets<W, MR>(x, n, a.op, a.scale, a.int_div));
        }
      } else if (!kRs && t >= kLag) {                 // copy piece t - L out
        const int w = t - kLag;
        const uint64_t p0 = first(w);
        const uint32_t cnt = full(w);
        // all-gather: a piece lies in its sender's ring; all-to-all: in the slot of its sender in this rank's
        const uint64_t at = ring0 + (uint64_t)(w % kStreamRing) * (kAg ? 1 : n) * P;
        const uint4* landed = mine + at;
#pragma unroll
        for (int k = 1; k < MR; ++k)
          if (k < n) {
            const uint4* src = kAg ? stage[k] + at : landed + (uint64_t)peerOf(r, k, n) * P;
#pragma unroll
            for (int u = 0; u < V; ++u)
              if (tid + u * kStep < cnt) v[u][k] = ldRing(src + tid + u * kStep);
          }
        fetch(t + 1);
#pragma unroll
        for (int k = 1; k < MR; ++k)
          if (k < n) {
            uint4* dst = reinterpret_cast<uint4*>(out.at(peerOf(r, k, n))) + p0;
#pragma unroll
            for (int u = 0; u < V; ++u)
              if (tid + u * kStep < cnt) __stcs(dst + tid + u * kStep, v[u][k]);
          }
        for (uint64_t j = ragged0(w) + tid; j < ragged1(w); j += kStep)
#pragma unroll 1
          for (int k = 1; k < n; ++k) {
            const int q = peerOf(r, k, n);
            ragStore(out, q, j, ldRing((kAg ? reinterpret_cast<const uint4*>(c.stage[q]) + at : landed + (uint64_t)q * P) + (j - p0)));
          }
      } else {
        fetch(t + 1);
      }
      __syncwarp();                                   // the warp's stores, before its arrival
      if (lane == 0) mbArrive(&s_done[t % kStreamRing]);
    }
  }
  callDone(c, a);
}

}  // namespace dev

namespace nvl {

template <typename W>
const void* pickStreamT(int kind, int nranks) {
  using namespace dev;
#define HL_STREAM_PICK(coll) \
  (nranks <= 2 ? (const void*)kStream<W, coll, 2> : (nranks <= 4 ? (const void*)kStream<W, coll, 4> : (const void*)kStream<W, coll, HL_MAX_RANKS>))
  switch (kind) {
    case kNvlStreamReduceScatter:   // up to four ranks (NvlPath::streamedKind)
      return nranks <= 2 ? (const void*)kStream<W, kStreamReduceScatter, 2> : (nranks <= 4 ? (const void*)kStream<W, kStreamReduceScatter, 4> : nullptr);
    case kNvlStreamAllGather: return HL_STREAM_PICK(kStreamAllGather);
    case kNvlStreamAllToAll: return HL_STREAM_PICK(kStreamAllToAll);
    case kNvlStreamBroadcast: return (const void*)kStream<W, kStreamBroadcast, 1>;
    default: return nullptr;
  }
#undef HL_STREAM_PICK
}

}  // namespace nvl
}  // namespace hl
