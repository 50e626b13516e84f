// Row access of the kernels that rewrite leaves (bt_merge.cu, bt_delete.cu).
#pragma once
#include "bt_common.cuh"

namespace bt {

// A lane's four slots of a row in one 32-byte access: two of 16 bytes at a stride
// of 32 each touch half of every sector, twice the wavefronts.  Plain accesses,
// in order with the kernel's others: it also writes the rows.
__device__ __forceinline__ void load_row(const uint64_t* p, uint64_t (&x)[4]) {
  asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];"
               : "=l"(x[0]), "=l"(x[1]), "=l"(x[2]), "=l"(x[3])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void store_row(uint64_t* p, const uint64_t (&x)[4]) {
  asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(x[0]), "l"(x[1]), "l"(x[2]), "l"(x[3])
               : "memory");
}

// A lane's share of a row that the group's next turn will read, into L2: the turns
// wait on their rows with DRAM at 35-43 % of its rate (two batches of 2^20 at 50 %
// writes 811 -> 801 us).
__device__ __forceinline__ void prefetch_row(const DevTree& t, uint32_t nd, uint32_t g) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(t.keys + (size_t)nd * 32 + g * 4));
  asm volatile("prefetch.global.L2 [%0];" ::"l"(t.vals + (size_t)nd * 32 + g * 4));
}

// Place of slot s in the shared row of the block's 8-lane group grp, a row
// being 256 bytes.  Lane g holds slots 4g .. 4g + 3; in slot order the lanes'
// e-th slots share four of the sixteen bank pairs and the two groups of a half
// warp the same ones (8 wavefronts an access), here they take all sixteen (2).
__device__ __forceinline__ uint32_t row_at(uint32_t s, uint32_t grp) {
  return ((s & 3u) << 3 | s >> 2) ^ (grp & 1u) << 3;
}

// the fingerprints of a lane's four slots of leaf nd (G = 8); slot 31's byte,
// the split count, is `splits` unless that is negative (then it stays)
__device__ __forceinline__ void store_fp4(const DevTree& t, uint32_t nd, uint32_t g, const uint64_t (&k)[4],
                                          int splits) {
  uint8_t* p = t.fp + (size_t)nd * 32 + g * 4;
  uint32_t w = 0;
#pragma unroll
  for (int i = 0; i < 3; i++) w |= (uint32_t)slot_fp(k[i]) << (8 * i);
  if (g < 7) {
    *reinterpret_cast<uint32_t*>(p) = w | (uint32_t)slot_fp(k[3]) << 24;
  } else if (splits >= 0) {
    *reinterpret_cast<uint32_t*>(p) = w | (uint32_t)splits << 24;
  } else {
    *reinterpret_cast<uint16_t*>(p) = (uint16_t)w;
    p[2] = (uint8_t)(w >> 16);
  }
}

}  // namespace bt
