// Helpers of the kernels that split K over a thread-block cluster and add the partial tiles over distributed shared memory.
#pragma once

#include <limits.h>

#include "common.cuh"

namespace qmm {
namespace split {

constexpr int kMaxCluster = 8;

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                               uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Hands a slot of a ring back (one arrival per warp) once what every lane loaded from it is in registers: an arrival that
// merely follows the loads in program order let the refill overtake the last of them (seen with remote shared-memory
// traffic on the same SM).  `dep` combines what all of a lane's loads returned; the vote cannot be taken before the last
// lane has it, and the arrival's address depends on the vote.  `never` is 0, but not to the compiler.
__device__ __forceinline__ void release_slot(uint64_t* empty, uint32_t dep, int never, int lane) {
  const int hit = __any_sync(0xFFFFFFFFu, dep == 0x7FC1FFC1u);
  __syncwarp();
  if (lane == 0) dev::mbar_arrive(empty + (hit & never));
}
// Arrives (release, cluster scope) on the barrier at the same place of CTA `rank`'s shared memory.
__device__ __forceinline__ void arrive_remote(uint64_t* bar, int rank) {
  asm volatile(
      "{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %0, %1;\n\t"
      "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [ra];\n\t}" ::"r"(dev::smem_u32(bar)), "r"(rank)
      : "memory");
}
__device__ __forceinline__ bool try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(dev::smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded, all lanes leave with the same answer.
__device__ __forceinline__ bool wait_cluster_warp(uint64_t* bar, uint32_t parity, int* status, int tag) {
  bool ok = try_wait_cluster(bar, parity);
  if (!ok) {
    const uint64_t t0 = dev::globaltimer_ns();
    while (!(ok = try_wait_cluster(bar, parity)))
      if (dev::globaltimer_ns() - t0 > dev::kWaitLimitNs) break;
    if (!ok && status) atomicExch(status, (tag << 16) | QMM_ERR_TIMEOUT);
  }
  return __all_sync(0xFFFFFFFFu, ok);
}

// Every thread of the cluster: what was written to shared memory before is visible to all of it afterwards.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// *p in the shared memory of CTA `rank`.
__device__ __forceinline__ float2 load_peer(const float2* p, int rank) {
  float2 v;
  asm volatile(
      "{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %2, %3;\n\t"
      "ld.shared::cluster.v2.f32 {%0, %1}, [ra];\n\t}"
      : "=f"(v.x), "=f"(v.y)
      : "r"(dev::smem_u32(p)), "r"(rank)
      : "memory");
  return v;
}
__device__ __forceinline__ float4 load_peer(const float4* p, int rank) {
  float4 v;
  asm volatile(
      "{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %4, %5;\n\t"
      "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [ra];\n\t}"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "r"(dev::smem_u32(p)), "r"(rank)
      : "memory");
  return v;
}

struct Grid {
  int ks, clusters;
};

inline void set_attrs(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[2], int ks) {
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = ks;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
}

// Resident clusters walk the tiles, so a launch takes as many rounds as the busiest cluster has tiles; a round costs its
// stages and the hand-over of the partial tiles (about six stages).  resident(ks): clusters of ks CTAs held at once.
// max_ctas: a caller's limit on the CTAs of the launch.
constexpr int kRoundCost = 6;
template <typename Fn>
inline Grid choose_grid(int tiles, int stages_total, Fn resident, int max_ctas = INT_MAX) {
  Grid best = {1, 1};
  long long best_cost = -1;
  for (int ks = 1; ks <= kMaxCluster && ks <= stages_total && ks <= max_ctas; ++ks) {
    const int held = resident(ks), c = held < max_ctas / ks ? held : max_ctas / ks;
    const int rounds = (tiles + c - 1) / c;
    const long long cost = static_cast<long long>(rounds) * ((stages_total + ks - 1) / ks + kRoundCost);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best.ks = ks;
      best.clusters = tiles < c ? tiles : c;
    }
  }
  return best;
}

// Clusters of `ks` CTAs of a kernel that the current device holds at once; `cache` belongs to the kernel.
template <typename Kern>
inline int resident_clusters(Kern kern, int threads, int smem, int per_sm, int ks, std::atomic<int> (&cache)[kMaxDevices][kMaxCluster + 1]) {
  int dev = 0, n = 0;
  const bool tracked = cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices;
  if (tracked && (n = cache[dev][ks].load(std::memory_order_relaxed)) > 0) return n;
  const int guess = per_sm * num_sms() / ks > 0 ? per_sm * num_sms() / ks : 1;
  if (!tracked) return guess;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(ks, 1024);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  set_attrs(cfg, attr, ks);
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
    (void)cudaGetLastError();
    n = guess;
  }
  cache[dev][ks].store(n, std::memory_order_relaxed);
  return n;
}

}  // namespace split
}  // namespace qmm
