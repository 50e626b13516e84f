// Delete phase of a sorted batch (op code DELETE = 2, src/input-helper.h:16,
// declared by the reference and implemented by none of its versions).
//
// Input: the unique keys whose run ends with a DELETE (w.del_list, ascending
// keys, count on the device), located by locate_kernel (bt_merge.cu: leaf, slot
// or none, the key's pre-batch value as the answer of the run's first request).
// del_apply_kernel removes all of a leaf's found keys at once.
// Leaves shrink in place: no merge with siblings; an emptied leaf stays and
// its separators keep routing (searches in it find nothing, inserts refill
// it).  The apply runs before the insert phase with no other kernel on the
// tree.  HBM traffic per touched leaf: one 512 B row read and written.
#include <cuda_runtime.h>

#include "bt_common.cuh"
#include "bt_delete.cuh"
#include "bt_internal.h"
#include "bt_launch.cuh"
#include "bt_rows.cuh"
#include "bt_search.cuh"

namespace bt {

namespace {

constexpr int kG = 8;
constexpr int kS = 32 / kG;

// One 8-lane group per touched leaf (equal leaves are adjacent because the keys
// ascend), as in the leaf merge: the slots to remove as bits, the kept slots to
// their new places in shared memory, the row written back with 32-byte stores.
// Bound by the chain entry -> leaf -> row and by L1 (72 % of its rate with
// 16-byte accesses and conflicting shared rows, row_at): with a warp per entry, one
// leaf at a time, 2^19 deletes on 2^24 keys took 131 us; groups with such rows 106.
__global__ void __launch_bounds__(256, 5) del_apply_kernel(DevTree t, const uint32_t* n_dev, const uint32_t* dleaf,
                                                        const uint32_t* dslot) {
  after_previous();
  __shared__ __align__(16) uint64_t mk[256 / kG][32];
  __shared__ __align__(16) uint64_t mv[256 / kG][32];
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t g = lane % kG, grp = threadIdx.x / kG;
  const uint32_t gmask = group_mask<kG>(lane);
  const uint32_t n = *n_dev;
  const uint32_t groups = (gridDim.x * blockDim.x) / kG;
  unsigned long long removed = 0;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / kG; i < n; i += groups) {
    const uint32_t leaf = dleaf[i], ahead = i + groups < n ? dleaf[i + groups] : kNil;
    if (ahead != kNil) prefetch_row(t, ahead, g);
    if (leaf == kNil || (i > 0 && dleaf[i - 1] == leaf)) continue;  // not the first entry of its leaf
    uint32_t gone = 0;
    for (uint32_t j = i;; j += kG) {
      const uint32_t x = j + g;
      const bool mine = x < n && dleaf[x] == leaf;
      const uint32_t sl = mine ? dslot[x] : kNoSlot;
      uint32_t bits = sl != kNoSlot ? 1u << sl : 0u;  // slots 0 .. 30
      bits |= mine ? 0u : 0x80000000u;                // bit 31: the leaf's entries end here
#pragma unroll
      for (int o = kG / 2; o >= 1; o >>= 1) bits |= __shfl_xor_sync(gmask, bits, o, kG);
      gone |= bits;
      if (gone >> 31) break;
    }
    gone &= 0x7fffffffu;
    if (!gone) continue;
    const size_t row = (size_t)leaf * 32 + g * kS;
    uint64_t k[kS], v[kS];
    load_row(t.keys + row, k);
    load_row(t.vals + row, v);
    const uint64_t h = __shfl_sync(gmask, k[kS - 1], kG - 1, kG);
    const uint32_t sz = hdr_size(h);
    const uint32_t keep = ((1u << sz) - 1u) & ~gone;  // sz <= 31
    const uint32_t nsz = __popc(keep);
#pragma unroll
    for (int e = 0; e < kS; e++) {
      const uint32_t s = g * kS + e;
      if ((keep >> s) & 1u) {
        const uint32_t pos = __popc(keep & ((1u << s) - 1u));
        mk[grp][row_at(pos, grp)] = k[e];
        mv[grp][row_at(pos, grp)] = v[e];
      }
    }
    __syncwarp(gmask);
    const uint64_t fence = v[kS - 1];  // lane kG - 1's
#pragma unroll
    for (int e = 0; e < kS; e++) {
      const uint32_t s = g * kS + e;
      k[e] = s < nsz ? mk[grp][row_at(s, grp)] : kKeyMax;
      v[e] = s < nsz ? mv[grp][row_at(s, grp)] : 0;
    }
    store_fp4(t, leaf, g, k, -1);
    if (g == kG - 1) {
      k[kS - 1] = make_hdr(nsz, 0, hdr_version(h) + 1, hdr_epoch(h));
      v[kS - 1] = fence;
    }
    store_row(t.keys + row, k);
    store_row(t.vals + row, v);
    __syncwarp(gmask);  // the shared rows are reused by the group's next leaf
    if (g == 0) removed += sz - nsz;
  }
  if (removed) atomicAdd(&t.ctrl->n_keys, (unsigned long long)0 - removed);
}

}  // namespace

// Removes the located DELETE keys (locate_phase; before the batch's inserts).
// n_upper bounds the device count w.counts->n_del.
int delete_apply(Handle* h, size_t n_upper, cudaStream_t s) {
  Work& w = h->w;
  launch_after(del_apply_kernel, (unsigned)min((size_t)h->sm_count * 8, (n_upper * kG + 255) / 256 + 1), 256, 0, s,
               h->tree, &w.counts->n_del, w.d_leaf, w.d_slot);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace bt
