// One thread-block cluster as the whole machine of a thin traversal step: its
// CTAs keep their part of the frontier in shared memory and exchange one
// 16-byte record per step (entries queued, edges, flags) that doubles as the
// step's barrier.
//
// A step of a high-diameter traversal has a few hundred to a few thousand
// edges: what it costs is the chain of dependent round trips, not the work.
// Over the whole grid that chain holds a grid barrier (1.2-2.2 us on B200) and
// a queue in L2 (entry, reservation, counters: three more trips of ~0.25 us).
// Inside a cluster the barrier is one st.async of 16 bytes to every CTA, which
// carries the record and completes the receiver's mbarrier (about 0.15 us
// against 0.24 us for barrier.cluster with 512 threads), and the queue is local.
#pragma once
#include "graph_common.cuh"

namespace gsrbg {

constexpr uint32_t kClCtas = 16;      // cluster size
constexpr uint32_t kClThreads = 512;  // threads per CTA (every warp goes through every step: 1024 cost 0.3 us a step more)

struct ClusterLink {
  uint4 tab[2][kClCtas];  // the CTAs' records, by parity of the step
  uint64_t mbar[2];
  uint64_t meet;             // see link_meet
};

__device__ __forceinline__ void st_async_v4(uint32_t caddr, uint4 v, uint32_t cmbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.u32 [%0], {%1,%2,%3,%4}, [%5];"
               ::"r"(caddr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(cmbar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* mbar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(gsrb::ptx::smem_u32(mbar)), "r"(parity) : "memory");
  return ok != 0;
}

// Waits are bounded, and a wait that ran out must not leave a CTA's threads in
// different places: a record that comes at the deadline is seen by some of them.
// So a verdict is a warp's (link_wait, link_meet), and a CTA's warps compare
// theirs at the barrier that ends each step and at one after the loop
// (link_agree): a warp that gave up goes to the latter while the others go
// through the step, and both find out there.  Nothing in between may wait for the
// CTA or, without a bound, for the cluster.
__device__ __forceinline__ bool link_agree(bool ok) { return __syncthreads_or(!ok) == 0; }

// Thread 0 of every CTA; a cluster barrier must follow before the first use.
__device__ __forceinline__ void link_init(ClusterLink& l, uint32_t ncta) {
  gsrb::ptx::mbar_init(&l.mbar[0], 1);
  gsrb::ptx::mbar_init(&l.mbar[1], 1);
  gsrb::ptx::mbar_init(&l.meet, ncta);
  gsrb::ptx::fence_mbar_init();
}
// Thread 0, once per step before it publishes: this step's records to come.
__device__ __forceinline__ void link_expect(ClusterLink& l, uint32_t p, uint32_t ncta) {
  gsrb::ptx::mbar_arrive_expect_tx(&l.mbar[p], 16u * ncta);
}
// One warp: this CTA's record of the step to every CTA of the cluster.
__device__ __forceinline__ void link_publish(ClusterLink& l, uint32_t p, uint4 rec, uint32_t rank, uint32_t ncta) {
  const uint32_t lane = lane_id();
  if (lane < ncta)
    st_async_v4(gsrb::ptx::mapa_shared(gsrb::ptx::smem_u32(&l.tab[p][rank]), lane), rec,
                gsrb::ptx::mapa_shared(gsrb::ptx::smem_u32(&l.mbar[p]), lane));
}
// One warp: the phase has completed before the deadline (the same in every lane).
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* mbar, uint32_t parity, uint64_t timeout_ns) {
  uint64_t t0 = 0;
  bool ok = false;
  for (uint32_t it = 0; !ok; ++it) {
    ok = mbar_try_wait_cluster(mbar, parity);
    if ((it & 63u) == 63u) {
      const uint64_t now = gsrb::ptx::globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > timeout_ns) break;
    }
  }
  return __all_sync(0xffffffffu, ok) != 0;
}
// Every warp: all records of the step are here (bounded by timeout_ns).
// Buffers alternate by the step's parity: a CTA publishes step s + 2 only after
// every CTA published s + 1, that is after it has read the records of s.
__device__ __forceinline__ bool link_wait(ClusterLink& l, uint32_t p, uint32_t& phases, uint64_t timeout_ns) {
  const uint32_t parity = (phases >> p) & 1u;
  phases ^= 1u << p;
  return mbar_wait_cluster(&l.mbar[p], parity, timeout_ns);
}
// Every warp: what the CTAs wrote to their shared memory before their last CTA
// barrier can be read from all of them (bounded; the third bit of `phases` is
// its parity).  barrier.cluster would wait without a bound, and would let a CTA
// that gave up leave while its memory is read.
__device__ __forceinline__ bool link_meet(ClusterLink& l, uint32_t& phases, uint32_t ncta, uint64_t timeout_ns) {
  if (threadIdx.x < ncta) {
    const uint32_t there = gsrb::ptx::mapa_shared(gsrb::ptx::smem_u32(&l.meet), threadIdx.x);
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(there) : "memory");
  }
  __syncwarp();
  const uint32_t parity = (phases >> 2) & 1u;
  phases ^= 4u;
  return mbar_wait_cluster(&l.meet, parity, timeout_ns);
}

__device__ __forceinline__ uint2 ld_cluster_v2(uint32_t caddr) {
  uint2 v;
  asm volatile("ld.shared::cluster.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(caddr) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_cluster_v4(uint32_t caddr) {
  uint4 v;
  asm volatile("ld.shared::cluster.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(caddr) : "memory");
  return v;
}

// A step's totals from its records, the same in every CTA (redux.sync, no
// shuffles).  ALWAYS_Y: y counts in every step, else only beside a w.
struct LinkSum {
  uint32_t x, y, z;  // sums of the first three fields
  bool w;            // some CTA's w is set
  uint32_t own;      // this CTA's x
  uint32_t max_x;
};
template <bool ALWAYS_Y>
__device__ __forceinline__ LinkSum link_sum(const ClusterLink& l, uint32_t p, uint32_t rank, uint32_t ncta) {
  const uint32_t lane = lane_id();
  uint4 t = make_uint4(0, 0, 0, 0);
  if (lane < ncta) t = l.tab[p][lane];
  LinkSum s;
  s.own = l.tab[p][rank].x;
  s.x = __reduce_add_sync(0xffffffffu, t.x);
  s.max_x = __reduce_max_sync(0xffffffffu, t.x);
  s.z = __reduce_add_sync(0xffffffffu, t.z);
  s.w = __any_sync(0xffffffffu, t.w != 0u);
  s.y = ALWAYS_Y || s.w ? __reduce_add_sync(0xffffffffu, t.y) : 0u;
  return s;
}
// Entries a warp takes at a time of n over the CTA's warps (at most 32).
__device__ __forceinline__ uint32_t cl_group(uint32_t n) {
  constexpr uint32_t kWarps = kClThreads / 32;
  return n >= 32u * kWarps ? 32u : max(1u, (n + kWarps - 1) / kWarps);
}
// Entry i of all the CTAs' entries laid end to end: (CTA, index) packed as
// cta << 16 | index.  Warp-synchronous (every lane its own i < s.x).
__device__ __forceinline__ uint32_t link_locate(const ClusterLink& l, uint32_t p, uint32_t ncta, uint32_t i) {
  const uint32_t lane = lane_id();
  const uint32_t x = lane < ncta ? l.tab[p][lane].x : 0u;
  uint32_t inc = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= (uint32_t)o) inc += y;
  }
  const uint32_t excl = inc - x;
  uint32_t c = 0;
#pragma unroll
  for (uint32_t st = 16; st > 0; st >>= 1)
    if (__shfl_sync(0xffffffffu, excl, c + st) <= i) c += st;
  return (c << 16) | (i - __shfl_sync(0xffffffffu, excl, c));
}
// Whether the step is to be redistributed: the fullest CTA holds half as much
// again as an even share.  An SM takes about four cycles an edge, so 250 entries
// of 4 edges on one of 16 CTAs cost 2.0 us beyond the chain; shares drift apart
// over hundreds of steps only.
__device__ __forceinline__ bool link_uneven(const LinkSum& s) {
  const uint32_t share = (s.x + kClCtas - 1) / kClCtas;
  return s.max_x > share + share / 2 + 32u;
}

}  // namespace gsrbg
