// sm_100a building blocks of the matrix kernels: tensor-memory accumulators, fifth-generation tensor-core products over
// pairs of CTAs, TMA tile copies, shared-memory barriers with bounded waits.
#pragma once
#include <cuda.h>
#include <stdint.h>

namespace hl {
namespace tc {

__device__ __forceinline__ uint32_t smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t clusterRank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// This CTA's shared-memory address as CTA `rank` of the cluster has it.
__device__ __forceinline__ uint32_t mapToRank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void clusterSync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint64_t nowNs() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// One lane of a converged warp, the same each time. Code that runs in all lanes up to here keeps its operands in uniform registers, which
// is where copies and products take them from; in a branch of one lane each is moved there first.
__device__ __forceinline__ bool elected() {
  uint32_t one;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(one));
  return one != 0;
}

// ---- barriers in shared memory
__device__ __forceinline__ void barInit(uint32_t bar, int arrivals) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(arrivals) : "memory");
}
__device__ __forceinline__ void barInitFence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void barExpect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void barArriveCluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// `cluster`: the phase is ended by threads of the other CTA. (An acquire at cluster scope costs hundreds of cycles more; what TMA and
// the tensor cores write is ordered by their own arrivals.)
template <bool kCluster>
__device__ __forceinline__ bool barTest(uint32_t bar, uint32_t parity) {
  uint32_t done;
  if constexpr (kCluster)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
  return done != 0;
}
// Waits for the phase of this parity. False once *stop is set, by this wait when `limit_ns` have gone by or by another
// thread of the CTA: then nobody waits any longer. Without `stop` the time alone ends it.
template <bool kCluster = false>
__device__ __forceinline__ bool barWait(uint32_t bar, uint32_t parity, volatile int* stop, uint64_t limit_ns) {
  uint64_t t0 = 0;
  for (uint32_t spins = 0;; ++spins) {
    if (barTest<kCluster>(bar, parity)) return true;
    if ((spins & 63u) == 63u) {
      if (stop && *stop) return false;
      const uint64_t now = nowNs();
      if (t0 == 0) t0 = now;
      if (now - t0 > limit_ns) {
        if (stop) *stop = 1;
        return false;
      }
    }
  }
}
// ---- TMA, three-dimensional tiles
__device__ __forceinline__ void prefetchMap(const CUtensorMap* m) { asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory"); }
// Into this CTA's shared memory; the bytes are counted on `bar`, which may be the barrier of the other CTA of the pair.
__device__ __forceinline__ void loadTilePair(uint32_t dst, const CUtensorMap* m, int x, int y, int z, uint32_t cluster_bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
               "l"(m), "r"(x), "r"(y), "r"(z), "r"(cluster_bar)
               : "memory");
}

// ---- tensor memory and products, CTA pairs
__device__ __forceinline__ void tmemAlloc(uint32_t dst, int columns) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(columns) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmemFree(uint32_t addr, int columns) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(columns) : "memory");
}
__device__ __forceinline__ void fenceBefore() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fenceAfter() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// D[256 x N] (+)= A[256 x 16] B[N x 16]^T; both CTAs of the pair hold one half of A's rows and of B's.
__device__ __forceinline__ void mma16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)add)
      : "memory");
}
// Arrives on the barrier at this address in both CTAs once all products issued so far are done.
__device__ __forceinline__ void commitPair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// 32 lanes x 32 columns of fp32, from lane `addr` on. With t the thread's place in its warp, g < 4, h < 2:
// r[16 h + 4 g + {0, 1}] are columns 8 g + 2 (t mod 4) + {0, 1} of lane 16 h + t / 4, r[16 h + 4 g + {2, 3}] those of lane
// 16 h + t / 4 + 8. (The wait belongs to the same statement: the registers hold nothing before it.)
__device__ __forceinline__ void tmemLoad32x32(uint32_t addr, float* r) {
  uint32_t* u = reinterpret_cast<uint32_t*>(r);
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]), "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]), "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
      : "r"(addr), "r"(addr + (16u << 16))
      : "memory");
}

// Shared-memory operand of 128-byte swizzled tiles (a tile: eight rows or more of 128 bytes, on a 1024-byte boundary).
// K-major: a row is 64 elements of k; MN-major: 64 elements of m or n, with `group` bytes from one 64 to the next.
__device__ __forceinline__ uint64_t operand(uint32_t addr, bool mn_major, uint32_t group) {
  const uint64_t lead = mn_major ? (uint64_t)(group >> 4) : 1ull, stride = 1024 >> 4;
  return (uint64_t)((addr & 0x3ffff) >> 4) | lead << 16 | stride << 32 | 1ull << 46 | 2ull << 61;
}

// Four 8 x 8 matrices of 16-bit elements, transposed on the way; lane l gives the address of row l % 8 of matrix l / 8.
__device__ __forceinline__ void storeMatrixT(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint4 loadShared(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

}  // namespace tc
}  // namespace hl
