// Kernel launches: clusters (rank, barrier, the other CTAs' shared memory) and programmatic dependence.
#pragma once

#include <cstdint>
#include <utility>

#include <cuda_runtime.h>

#include "common.cuh"

namespace dionw {

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t n;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
  return n;
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Address of the same shared-memory object in another CTA of the cluster.
__device__ __forceinline__ uint32_t peer_address(const void* local, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(out)
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(local))), "r"(rank));
  return out;
}

__device__ __forceinline__ uint32_t peer_load(const void* local, uint32_t rank) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer_address(local, rank)) : "memory");
  return v;
}

// Runs whose per-block kernels (row selection, NorMuon scales) share a launch: as many as a plan takes batches.
constexpr int kGroupRuns = 6;

// CTAs that share one block of `rows` rows: one per `rows_per_cta`, at most the portable cluster size.
// (The grid stays below 2^31 CTAs.)
inline unsigned cluster_for(long long blocks, long long rows, long long rows_per_cta) {
  unsigned n = 1;
  while (n < 8 && blocks * n * 2 < (1LL << 31) && rows > n * rows_per_cta) n *= 2;
  return n;
}

// Whether kernels are launched with programmatic dependence: yes, unless DIONW_GEMM_PDL=0 (gemm.cu).
bool use_dependent_launch();

// Programmatic dependent launch: a kernel launched by launch_dependent or launch_clusters may have CTAs
// resident while the kernel before it in the stream still runs, and waits here before it touches global
// memory; the wait returns once that kernel has completed and its writes are visible.  A step of small
// matrices is a chain of 5 to 20 us kernels with 2 to 3 us between them: with
// this the smallest step takes 243 us instead of 257, a 1100-wide encoder's 998 instead of 1059, gpt2-small's
// 1787 instead of 1854.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... Params, typename... Args>
cudaError_t launch_dependent(void (*kernel)(Params...), unsigned grid, unsigned threads, cudaStream_t stream,
                             Args... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(grid);
  config.blockDim = dim3(threads);
  config.stream = stream;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attribute;
  config.numAttrs = use_dependent_launch() ? 1 : 0;
  return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

// blocks x cluster CTAs, `cluster` of them to a cluster.
template <typename... Params, typename... Args>
cudaError_t launch_clusters(void (*kernel)(Params...), unsigned blocks, unsigned cluster, unsigned threads,
                            cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(blocks * cluster);
  config.blockDim = dim3(threads);
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = cluster;
  attributes[0].val.clusterDim.y = 1;
  attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = use_dependent_launch() ? 2 : 1;
  return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

// Calls launch(first run, runs, blocks, cluster) for launches that take all n runs of `runs`, which it puts in the order
// of their clusters (Run::ctas, the CTAs that a block's sums are made by) and whose Run::first_block it fills in.  Every
// block of a launch gets the widest cluster of its runs, whose other CTAs only keep the barriers: narrower runs go along up to
// `per_two_sms` CTAs to two SMs.  A launch against one per run, us, beside 1 x 4096 rows with 1024 selected: selections (an SM holds one CTA) of
// 16 x 128 16 and 26, 228 CTAs 24 and 26, beside 8 x 4096 256 CTAs 28 and 27, 288 36 and 27, beside one 1000 x 128 365 and 85;
// scales (it holds two) 256 CTAs 6.9 and 9.3, 312 9.9 and 9.3, 368 10.4 and 9.2, 520 11.6 and 9.1, 1000 x 128 147 and 25.  (Alone; in a
// step a launch more is one more of some 3 us, so that the scales' line lies past where the two meet: 1100-wide encoder, 304 CTAs, a
// step 736 us with one launch, 739 with two.)
template <typename Run, typename Launch>
int launch_together(Run* runs, int n, int per_two_sms, Launch&& launch) {
  for (int i = 1; i < n; ++i)   // six at most
    for (int j = i; j > 0 && runs[j].ctas > runs[j - 1].ctas; --j) std::swap(runs[j], runs[j - 1]);
  const long long limit = n > 1 ? per_two_sms * sm_count() / 2 : 0;
  for (int first = 0, last = 0; first < n; first = last) {
    const long long widest = runs[first].ctas;
    long long blocks = 0;
    for (; last < n && (runs[last].ctas == widest || (blocks + runs[last].blocks) * widest <= limit); ++last) {
      runs[last].first_block = unsigned(blocks);
      blocks += runs[last].blocks;
    }
    DIONW_REQUIRE(blocks * widest < (1LL << 31), "too many blocks in one launch");
    const int st = launch(runs + first, last - first, unsigned(blocks), unsigned(widest));
    if (st != DIONW_OK) return st;
  }
  return DIONW_OK;
}

}  // namespace dionw
