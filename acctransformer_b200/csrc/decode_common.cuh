// What the two decode kernels share: the merge of a slice's parts inside a thread-block cluster, and the launch.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "fa_kernels.cuh"

namespace acct {

__device__ __forceinline__ float decode_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ int cluster_rank() {
  int r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// the word at `p` of this block's shared memory, in the shared memory of block `rank` of the cluster
__device__ __forceinline__ float cluster_load(const float* p, int rank) {
  const uint32_t here = static_cast<uint32_t>(__cvta_generic_to_shared(p));
  uint32_t there;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(here), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(there) : "memory");
  return v;
}

// The parts of one (sequence, cache head) slice are the thread blocks of one cluster.  Each has left its partial result
// in its own shared memory -- acc[head * stride + d], m[head], l[head] -- and block `rank` now forms every `splits`-th
// 128 of the G x D results from all of them.  Against partial results in global memory and a second kernel this takes a
// launch and a pass through L2 off a step whose whole work, for short contexts, is a few microseconds.
template <bool BF16>
__device__ __forceinline__ void cluster_merge(const DecodeParams& p, float* acc, float* m, float* l, int stride, int b,
                                              int h_kv, int threads) {
  cluster_sync();
  const int rank = cluster_rank();
  const int G = p.kv_group, total = G * p.D;
  for (int idx = rank * threads + threadIdx.x; idx < total; idx += threads * p.splits) {
    const int head = idx / p.D, d = idx % p.D;
    float mm[8], ll[8], aa[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      mm[s] = -INFINITY; ll[s] = 0.f; aa[s] = 0.f;
      if (s < p.splits) {
        mm[s] = cluster_load(m + head, s);
        ll[s] = cluster_load(l + head, s);
        aa[s] = cluster_load(acc + head * stride + d, s);
      }
    }
    float big = -INFINITY;
#pragma unroll
    for (int s = 0; s < 8; ++s) big = fmaxf(big, mm[s]);
    float a = 0.f, lsum = 0.f;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const float w = mm[s] == -INFINITY ? 0.f : decode_ex2(mm[s] - big);
      lsum = fmaf(ll[s], w, lsum);
      a = fmaf(aa[s], w, a);
    }
    a *= lsum > 0.f ? 1.0f / lsum : 0.f;
    const int64_t at = (static_cast<int64_t>(b) * p.N + h_kv * G + head) * p.D + d;
    if constexpr (BF16) reinterpret_cast<__nv_bfloat16*>(p.y)[at] = __float2bfloat16(a);
    else reinterpret_cast<__half*>(p.y)[at] = __float2half(a);
  }
  cluster_sync();      // nobody's shared memory goes away while another block still reads it
}

// How many clusters of p.splits blocks of this kernel the device holds at once.  Fewer than its SMs could hold blocks: a
// cluster stays inside one GPC, and what is left over there is too small for another.  Asked once per thread, kernel,
// cluster size and device.
inline cudaError_t resident_clusters(void (*kern)(const DecodeParams), const cudaLaunchConfig_t& cfg, int splits, int* out) {
  struct Seen {
    const void* kernel;
    int splits, dev, n;
  };
  static thread_local Seen seen[16];       // zero-initialised; newest entry overwrites the oldest
  static thread_local unsigned next = 0;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  for (const Seen& s : seen)
    if (s.kernel == reinterpret_cast<const void*>(kern) && s.splits == splits && s.dev == dev) {
      *out = s.n;
      return cudaSuccess;
    }
  e = cudaOccupancyMaxActiveClusters(out, kern, &cfg);
  if (e == cudaSuccess) seen[next++ % 16] = {reinterpret_cast<const void*>(kern), splits, dev, *out};
  return e;
}

// One thread block per part; the parts of a slice form a cluster where p.clustered says so.  With `resident` nothing is
// launched: it receives the number of such clusters that fit at once.
inline cudaError_t launch_parts(void (*kern)(const DecodeParams), const DecodeParams& p, int units, int threads, size_t smem,
                                cudaStream_t stream, int* resident) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.splits, units);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];         // (a cluster of one block is not the same as no cluster: it is scheduled as one)
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.clustered ? 1 : 0;
  if (resident != nullptr) return resident_clusters(kern, cfg, p.splits, resident);
  return cudaLaunchKernelEx(&cfg, kern, p);
}

}  // namespace acct
