// DELETE apply, shared by del_apply_kernel (bt_delete.cu) and the write part of
// the small batches (bt_merge.cu).
#pragma once
#include "bt_common.cuh"

namespace bt {

constexpr uint32_t kNoSlot = 0xFFFFFFFFu;

// One warp at entry i of the n located DELETE keys: when i is the first of its
// leaf, all of that leaf's found keys are removed (a ballot over the row keeps
// the others in order).  Returns how many.
__device__ __forceinline__ uint32_t del_apply_at(const DevTree& t, const uint32_t* dleaf,
                                                 const uint32_t* dslot, size_t i, size_t n,
                                                 uint32_t lane) {
  const uint32_t leaf = dleaf[i];
  if (leaf == kNil || (i > 0 && dleaf[i - 1] == leaf)) return 0;  // not the first entry of its leaf
  // slots to remove: every found entry of this leaf (entries of a leaf are adjacent)
  uint32_t gone = 0;
  for (size_t j = i;; j += 32) {
    const size_t x = j + lane;
    const bool mine = x < n && dleaf[x] == leaf;
    const uint32_t sl = mine ? dslot[x] : kNoSlot;
    uint32_t bit = (mine && sl != kNoSlot) ? (1u << sl) : 0u;
    bit = __reduce_or_sync(0xffffffffu, bit);
    gone |= bit;
    if (__ballot_sync(0xffffffffu, mine) != 0xffffffffu) break;
  }
  if (!gone) return 0;
  uint64_t* kr = t.keys + (size_t)leaf * 32;
  uint64_t* vr = t.vals + (size_t)leaf * 32;
  const uint64_t k = kr[lane];
  const uint64_t v = vr[lane];
  const uint64_t h = __shfl_sync(0xffffffffu, k, 31);
  const uint32_t sz = hdr_size(h);
  const bool keep = lane < sz && !((gone >> lane) & 1u);
  const uint32_t keepm = __ballot_sync(0xffffffffu, keep);
  const uint32_t nsz = __popc(keepm);
  const uint32_t pos = __popc(keepm & ((1u << lane) - 1u));
  __syncwarp();
  uint8_t* fr = t.fp + (size_t)leaf * 32;
  if (keep) {
    kr[pos] = k;
    vr[pos] = v;
    fr[pos] = slot_fp(k);
  }
  __syncwarp();
  if (lane >= nsz && lane < 31) {
    kr[lane] = kKeyMax;
    vr[lane] = 0;
    fr[lane] = 0;
  }
  if (lane == 31) kr[31] = make_hdr(nsz, 0, hdr_version(h) + 1, hdr_epoch(h));
  return sz - nsz;
}

}  // namespace bt
