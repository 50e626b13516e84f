// Shared by the kernels of the small sorted batches (bt_small.cu, and the write
// part in bt_merge.cu): sizes, cluster barrier, launch shape, argument blocks.
#pragma once
#include <cuda_runtime.h>

#include "bt_common.cuh"
#include "bt_internal.h"

namespace bt {

constexpr int kSmallThreads = 1024;
constexpr int kSmallItems = 4;  // requests (and sorted pairs, and new keys) per thread
// most requests per block of a cluster
constexpr uint32_t kSmallPer = kSmallThreads * kSmallItems;
static_assert(kSmallMax == kSmallBlocks * kSmallPer, "the largest small batch fills sixteen blocks");

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// every thread of every block of the cluster; global writes before it are seen after it
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// an empty tree gets a leaf as its root (one thread)
__device__ __forceinline__ void ensure_root_leaf(const DevTree& t) {
  Ctrl* C = t.ctrl;
  if (C->root != kNil) return;
  const uint32_t id = atomicAdd(&C->n_nodes, 1u);
  if (id >= t.cap) {
    atomicOr(&C->error, kErrCapacity);
    return;
  }
  for (int i = 0; i < 31; i++) {
    t.keys[(size_t)id * 32 + i] = kKeyMax;
    t.vals[(size_t)id * 32 + i] = 0;
  }
  t.vals[(size_t)id * 32 + 31] = kKeyMax;
  t.keys[(size_t)id * 32 + 31] = make_hdr(0, 0, 0, C->epoch);
  for (int i = 0; i < 32; i++) t.fp[(size_t)id * 32 + i] = 0;
  t.low[id] = 0;
  C->root = id;
  C->root_level = 0;
}

struct SmallFront {
  BatchCounts* counts;
  uint64_t* tk;
  uint32_t* tv;
  uint32_t* list;
  uint64_t* lk;
  uint64_t *k_a, *k_b;
  uint32_t *v_a, *v_b;
  uint64_t *ukeys, *uvals;
  uint32_t *ins_list, *del_list, *pend;
  void* sums;      // per block: its part of the scan
  uint64_t* edge;  // per block: its first and last key
};

struct SmallRead {
  const BatchCounts* counts;
  const uint32_t* list;
  const uint64_t* lk;
  const uint64_t* ukeys;
  const uint32_t *ins_list, *del_list;
  uint32_t *path, *mleaf, *isnew;
  uint64_t* vpos;
  uint32_t *dleaf, *dslot;
  uint64_t* uans;
  uint8_t* uans_st;
  size_t path_stride;
  int locate_ins;  // 0: the STM kernel inserts
};

// largest cluster of a kernel with `smem` bytes a block that the current device takes (0: none)
unsigned small_largest(const void* kernel, size_t smem);

// at: two attributes, the cluster and the dependent launch
inline void small_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, unsigned C, size_t smem, cudaStream_t s) {
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(kSmallThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
}

}  // namespace bt
