// The step loop of the cluster kernels with nothing but its waits: one CTA falls
// silent, leaves a rendezvous out, or publishes a record about when the others'
// waits run out.  Every CTA's threads must leave the loop together, and every
// wait must end.  Prints "ok" or what went wrong.
#include "cluster_link.cuh"

#include <cstdio>
#include <cstdlib>
#include <vector>

using namespace gsrbg;

enum { SILENT = 0, NO_MEET = 1, LATE = 2 };

__global__ void __launch_bounds__(kClThreads, 1)
check_kernel(uint32_t steps, int kind, uint32_t bad_rank, uint32_t bad_step, unsigned long long delay_ns,
             unsigned long long timeout_ns, uint32_t* left) {
  __shared__ ClusterLink link;
  const uint32_t rank = gsrb::ptx::cluster_ctarank(), ncta = gsrb::ptx::cluster_nctarank();
  const uint32_t wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    link_init(link, ncta);
    link_expect(link, 0u, ncta);
  }
  gsrb::ptx::cluster_sync();
  if (wid == 0) link_publish(link, 0u, make_uint4(1u, 0u, 0u, 0u), rank, ncta);
  uint32_t phases = 0, p = 0, step = 0;
  bool ok, agreed = false;
  for (;; ++step) {
    ok = link_wait(link, p, phases, timeout_ns);
    if (!ok || step == steps) break;
    const uint32_t o = p ^ 1u;
    if (threadIdx.x == 0) link_expect(link, o, ncta);
    const bool here = rank == bad_rank && step == bad_step;
    if (step % 3 == 2) ok = kind == NO_MEET && here ? false : link_meet(link, phases, ncta, timeout_ns);
    agreed = true;
    if (!(ok = link_agree(ok))) break;
    agreed = false;
    if (kind == LATE && here && wid == 0) {
      const unsigned long long t0 = gsrb::ptx::globaltimer_ns();
      while (gsrb::ptx::globaltimer_ns() - t0 < delay_ns) {
      }
    }
    if (wid == 0 && !(kind == SILENT && here)) link_publish(link, o, make_uint4(step, 0u, 0u, 0u), rank, ncta);
    p = o;
  }
  if (!agreed) ok = link_agree(ok);
  left[rank * kClThreads + threadIdx.x] = step << 1 | (ok ? 1u : 0u);
  gsrb::ptx::cluster_sync();
}

#define CUDA(x)                                                     \
  do {                                                              \
    cudaError_t e_ = (x);                                           \
    if (e_ != cudaSuccess) {                                        \
      printf("%s: %s\n", #x, cudaGetErrorString(e_));               \
      exit(1);                                                      \
    }                                                               \
  } while (0)

int main() {
  constexpr uint32_t n = kClCtas;
  uint32_t* d = nullptr;
  CUDA(cudaMalloc(&d, n * kClThreads * sizeof(uint32_t)));
  CUDA(cudaFuncSetAttribute(check_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  std::vector<uint32_t> h(n * kClThreads);
  int bad = 0, early = 0;
  // returns whether every CTA got through all steps
  auto run = [&](uint32_t steps, int kind, uint32_t rank, uint32_t step, unsigned long long delay,
                 unsigned long long timeout) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n);
    cfg.blockDim = dim3(kClThreads);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = n;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    CUDA(cudaLaunchKernelEx(&cfg, check_kernel, steps, kind, rank, step, delay, timeout, d));
    CUDA(cudaMemcpy(h.data(), d, h.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    bool all = true;
    for (uint32_t c = 0; c < n; ++c) {
      for (uint32_t i = 1; i < kClThreads; ++i)
        if (h[c * kClThreads + i] != h[c * kClThreads]) {
          if (!bad++) printf("CTA %u: thread %u left at %x, thread 0 at %x\n", c, i, h[c * kClThreads + i], h[c * kClThreads]);
          break;
        }
      all = all && h[c * kClThreads] == (steps << 1 | 1u);
    }
    return all;
  };
  if (!run(300, SILENT, 99, 0, 0, 1000000000ull)) ++bad, printf("a whole loop did not come through\n");
  for (uint32_t s : {0u, 1u, 2u, 7u})
    for (uint32_t r : {0u, 5u, n - 1u})
      if (run(20, SILENT, r, s, 0, 300000)) ++bad, printf("a silent CTA went unnoticed\n");
  for (uint32_t r : {0u, 5u, n - 1u})
    if (run(20, NO_MEET, r, 5, 0, 300000)) ++bad, printf("a CTA missing from a rendezvous went unnoticed\n");
  for (uint32_t i = 0; i < 400; ++i) early += run(6, LATE, i % n, i % 5, 180000 + 200 * i, 200000);
  if (bad) return printf("%d faults\n", bad), 1;
  printf("ok (%d of 400 late records in time)\n", early);
  return 0;
}
