// Decoupled look-back over tiles that blocks take in turn (the one-launch scans
// of bt_sort.cu and bt_merge.cu).
//
// status[t] = epoch << 34 | state << 32 | value, state 1 the tile's own sum, 2
// its inclusive prefix; each run's epoch makes the words of earlier runs read
// as not ready, so the array is never cleared.  The epoch is counted on the
// device: as a launch argument it was fixed in a captured launch, and a second
// replay took the first one's words for its own.  ctr[0] hands out tile ids, in
// the order blocks take them (a tile waits only on tiles taken before it), with
// the runs so far in its high half: one atomic gives a block both, where a word
// of its own for the epoch cost a scan 2 us.  ctr[1] counts the blocks that are
// done; the last one starts the ids again and counts the run.  The wait is
// bounded: past kLbSpinLimit it sets kErrSpin in *err and goes on.
#pragma once
#include <cstdint>

#include "bt_common.cuh"

namespace bt {

constexpr uint64_t kLbAgg = 1ull << 32, kLbInc = 2ull << 32;
constexpr uint32_t kLbSpinLimit = 1u << 22;
constexpr uint32_t kLbEpochs = (1u << 30) - 1;  // epochs 1 .. kLbEpochs; zeroed words carry epoch 0
constexpr size_t kLbCtrWords = 2;               // words of ctr, zero before the first run

// a tile (low half) and the run's epoch less one
__device__ __forceinline__ uint64_t take_tile(uint64_t* ctr) {
  return atomicAdd(reinterpret_cast<unsigned long long*>(ctr), 1ull);
}
__device__ __forceinline__ uint32_t tile_epoch(uint64_t ticket) { return (uint32_t)(ticket >> 32) + 1; }

// Publish tile `tile`'s sum and return the sum of the tiles before it; one whole
// warp, all lanes get the result.  32 tiles are read at a time: one after
// another, the walk back to the last prefix bounded a scan of 320 tiles (18 us).
__device__ __forceinline__ uint32_t look_back(uint64_t* status, uint32_t tile, uint32_t sum, uint32_t epoch,
                                              uint32_t* err) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t tag = (uint64_t)epoch << 34;
  if (tile == 0) {
    if (lane == 0) st_release(&status[0], tag | kLbInc | sum);
    return 0;
  }
  if (lane == 0) st_release(&status[tile], tag | kLbAgg | sum);
  uint32_t prefix = 0, spins = 0;
  int64_t t = (int64_t)tile - 1;
  for (;;) {
    const int64_t i = t - lane;
    const uint64_t w = i >= 0 ? ld_acquire(&status[i]) : (tag | kLbInc);  // before tile 0: nothing
    const uint32_t state = (uint32_t)(w >> 34) == epoch ? (uint32_t)(w >> 32) & 3u : 0u;
    const uint32_t done = __ballot_sync(0xffffffffu, state == 2), wait = __ballot_sync(0xffffffffu, state == 0);
    const uint32_t upto = done ? (done & (0u - done)) * 2u - 1u : 0xffffffffu;  // lanes up to the nearest prefix
    if (wait & upto) {
      if (++spins > kLbSpinLimit) {
        if (lane == 0 && err) atomicOr(err, kErrSpin);
        break;
      }
      if (spins > 64) __nanosleep(64);
      continue;
    }
    prefix += __reduce_add_sync(0xffffffffu, (upto >> lane) & 1u ? (uint32_t)w : 0u);
    if (done) break;
    t -= 32;
  }
  if (lane == 0) st_release(&status[tile], tag | kLbInc | (uint64_t)(prefix + sum));
  return prefix;
}

// one thread of every block, at its end
__device__ __forceinline__ void tiles_done(uint64_t* ctr, uint32_t epoch) {
  __threadfence();
  if (atomicAdd(reinterpret_cast<unsigned long long*>(ctr + 1), 1ull) == gridDim.x - 1) {
    ctr[0] = (uint64_t)(epoch % kLbEpochs) << 32;
    ctr[1] = 0;
    __threadfence();
  }
}

}  // namespace bt
