// Row access of the kernels that rewrite leaves (bt_merge.cu, bt_delete.cu).
#pragma once
#include "bt_common.cuh"

namespace bt {

// S slots of a row that this kernel also writes (plain loads: the read-only
// path must not be used for it)
template <int S>
__device__ __forceinline__ void load_row16(const uint64_t* p, uint64_t (&x)[S]) {
#pragma unroll
  for (int i = 0; i < S; i += 2) {
    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(p + i);
    x[i] = w.x;
    x[i + 1] = w.y;
  }
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

template <int S>
__device__ __forceinline__ void store_row16(uint64_t* p, const uint64_t (&x)[S]) {
#pragma unroll
  for (int i = 0; i < S; i += 2) *reinterpret_cast<ulonglong2*>(p + i) = make_ulonglong2(x[i], x[i + 1]);
}

}  // namespace bt
