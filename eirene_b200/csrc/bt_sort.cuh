// Sort primitives of one block, shared by the small batches (bt_small.cu) and the
// sample sort of the touched requests (bt_sample.cu).  A pair is a key and a
// payload, the request's index above its two-bit op code; pairs are ordered by
// key, then by payload: indices are unique, so every comparison is strict and
// the order is the stable one, and it is the order of one 96-bit number (a
// borrow through three words, where a compare of the key, of its equality and of
// the index in the payload's low bits took 8 instructions).
#pragma once
#include "bt_common.cuh"

namespace bt {

__device__ __forceinline__ uint32_t pair_payload(uint32_t idx, uint32_t op) { return idx << 2 | (op <= 2 ? op : 3u); }
__device__ __forceinline__ uint32_t pair_idx(uint32_t v) { return v >> 2; }
__device__ __forceinline__ uint32_t pair_op(uint32_t v) { return v & 3u; }

// no short-circuit branches: the callers select on the result
__device__ __forceinline__ bool pair_less(uint64_t ka, uint32_t va, uint64_t kb, uint32_t vb) {
  uint32_t borrow;
  asm("{\n\t.reg .u32 t;\n\t"
      "sub.cc.u32 t, %1, %4;\n\t"
      "subc.cc.u32 t, %2, %5;\n\t"
      "subc.cc.u32 t, %3, %6;\n\t"
      "subc.u32 %0, 0, 0;\n\t}"
      : "=r"(borrow)
      : "r"(va), "r"((uint32_t)ka), "r"((uint32_t)(ka >> 32)), "r"(vb), "r"((uint32_t)kb), "r"((uint32_t)(kb >> 32)));
  return borrow != 0;
}

// bitonic exchange of this lane's element i with its partner i ^ j
__device__ __forceinline__ void sort_keep(uint64_t& k, uint32_t& v, uint64_t pk, uint32_t pv, int i, int j, int kk) {
  const bool asc = (i & kk) == 0, lower = (i & j) == 0;
  // (two equal pairs are padding: either outcome is the same)
  const bool take = pair_less(pk, pv, k, v) == (lower == asc);
  k = take ? pk : k;
  v = take ? pv : v;
}

__device__ __forceinline__ void sort_exchange(uint64_t& ka, uint32_t& va, uint64_t& kb, uint32_t& vb, bool asc) {
  const bool sw = pair_less(kb, vb, ka, va) == asc;
  const uint64_t k0 = sw ? kb : ka, k1 = sw ? ka : kb;
  const uint32_t v0 = sw ? vb : va, v1 = sw ? va : vb;
  ka = k0;
  kb = k1;
  va = v0;
  vb = v1;
}

// 128 pairs of a warp, four consecutive ones per lane, in ascending order
__device__ __forceinline__ void warp_sort(uint64_t (&K)[4], uint32_t (&V)[4]) {
  const int base = (threadIdx.x & 31) * 4;
#pragma unroll
  for (int kk = 2; kk <= 128; kk <<= 1) {
#pragma unroll
    for (int j = kk >> 1; j >= 4; j >>= 1) {
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const uint64_t pk = __shfl_xor_sync(0xffffffffu, K[e], j / 4);
        const uint32_t pv = __shfl_xor_sync(0xffffffffu, V[e], j / 4);
        sort_keep(K[e], V[e], pk, pv, base + e, j, kk);
      }
    }
    if (kk >= 4) {
      sort_exchange(K[0], V[0], K[2], V[2], (base & kk) == 0);
      sort_exchange(K[1], V[1], K[3], V[3], ((base + 1) & kk) == 0);
    }
    sort_exchange(K[0], V[0], K[1], V[1], (base & kk) == 0);
    sort_exchange(K[2], V[2], K[3], V[3], ((base + 2) & kk) == 0);
  }
}

// this thread's four outputs [d, d + 4) of the merge of the sorted runs
// (ka, va)[0, la) and (kb, vb)[0, lb) in shared memory
__device__ __forceinline__ void merge4(const uint64_t* ka, const uint32_t* va, int la, const uint64_t* kb,
                                       const uint32_t* vb, int lb, int d, uint64_t (&ok)[4], uint32_t (&ov)[4]) {
  int lo = d > lb ? d - lb : 0, hi = min(d, la);
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (pair_less(ka[mid], va[mid], kb[d - 1 - mid], vb[d - 1 - mid])) lo = mid + 1;
    else hi = mid;
  }
  // the runs' next pairs in registers: one pair read per output, no branches (the
  // rounds wait on these loads; with the 16-byte accesses below, two batches of 2^20
  // at 50 % writes 836 -> 812 us, two Zipf batches of 2^18 336 -> 329)
  int ia = lo, ib = d - lo;
  uint64_t a = ia < la ? ka[ia] : 0, b = ib < lb ? kb[ib] : 0;
  uint32_t x = ia < la ? va[ia] : 0, y = ib < lb ? vb[ib] : 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {  // (past the runs' end: pairs nobody uses)
    const bool take_a = (ib >= lb) | ((ia < la) & pair_less(a, x, b, y));
    ok[j] = take_a ? a : b;
    ov[j] = take_a ? x : y;
    ia += take_a ? 1 : 0;
    ib += take_a ? 0 : 1;
    if (j == 3) break;
    const bool any = take_a ? ia < la : ib < lb;
    const uint64_t* pk = take_a ? ka + ia : kb + ib;
    const uint32_t* pv = take_a ? va + ia : vb + ib;
    const uint64_t nk = any ? *pk : 0;
    const uint32_t nv = any ? *pv : 0;
    a = take_a ? nk : a;
    x = take_a ? nv : x;
    b = take_a ? b : nk;
    y = take_a ? y : nv;
  }
}

// a thread's four pairs [d, d + 4) of a block's arrays (16-byte aligned): 16 bytes
// an access, where four of 8 at a stride of 32 met in four of the sixteen bank pairs
__device__ __forceinline__ void load_pairs(const uint64_t* sk, const uint32_t* sv, int d, uint64_t (&K)[4],
                                           uint32_t (&V)[4]) {
  const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(sk + d), b = *reinterpret_cast<const ulonglong2*>(sk + d + 2);
  const uint4 v = *reinterpret_cast<const uint4*>(sv + d);
  K[0] = a.x;
  K[1] = a.y;
  K[2] = b.x;
  K[3] = b.y;
  V[0] = v.x;
  V[1] = v.y;
  V[2] = v.z;
  V[3] = v.w;
}
__device__ __forceinline__ void store_pairs(uint64_t* sk, uint32_t* sv, int d, const uint64_t (&K)[4],
                                            const uint32_t (&V)[4]) {
  *reinterpret_cast<ulonglong2*>(sk + d) = make_ulonglong2(K[0], K[1]);
  *reinterpret_cast<ulonglong2*>(sk + d + 2) = make_ulonglong2(K[2], K[3]);
  *reinterpret_cast<uint4*>(sv + d) = make_uint4(V[0], V[1], V[2], V[3]);
}

// The first cnt of a block's pairs in shared memory, sorted; the arrays hold cnt
// rounded up to 128, the threads past the count's last run idle.  128-pair runs
// by warp (registers and shuffles), then merged pairwise.  The bitonic network
// over a whole tile of 2048 pairs took 26 us, whatever their count; a search of
// every pair's rank in the other run instead of merge4 made two batches of 2^20
// at 50 % writes 30 us slower.
__device__ __forceinline__ void block_sort(uint64_t* sk, uint32_t* sv, int cnt) {
  const int P = (cnt + 127) & ~127;
  const int d = threadIdx.x * 4;
  uint64_t K[4];
  uint32_t V[4];
  if (d < P) {
    load_pairs(sk, sv, d, K, V);
#pragma unroll
    for (int e = 0; e < 4; e++) {
      if (d + e < cnt) continue;
      K[e] = ~0ull;
      V[e] = 0xFFFFFFFFu;  // behind every request
    }
    warp_sort(K, V);
    store_pairs(sk, sv, d, K, V);
  }
  __syncthreads();
  for (int L = 128; L < P; L <<= 1) {
    const int ps = d & ~(2 * L - 1);
    const int lb = min(L, P - ps - L);
    const bool pair = d < P && lb > 0;  // a last run without a partner stays
    if (pair) merge4(sk + ps, sv + ps, L, sk + ps + L, sv + ps + L, lb, d - ps, K, V);
    __syncthreads();
    if (pair) store_pairs(sk, sv, d, K, V);
    __syncthreads();
  }
}

// elements of A among the first d of merge(A, B), A = k[a0, a0 + na), B = k[b0, b0 + nb)
// in global memory; one warp, 32 candidates per step
__device__ __forceinline__ uint32_t split_of(const uint64_t* k, const uint32_t* v, uint32_t a0, uint32_t na,
                                             uint32_t b0, uint32_t nb, uint32_t d) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t lo = d > nb ? d - nb : 0, hi = min(d, na);
  while (lo < hi) {
    const uint32_t stride = (hi - lo + 31) / 32;
    const uint32_t a = lo + lane * stride;
    bool p = false;
    if (a < hi) {
      const uint32_t b = b0 + d - 1 - a;
      p = pair_less(__ldcg(k + a0 + a), __ldcg(v + a0 + a), __ldcg(k + b), __ldcg(v + b));
    }
    const uint32_t c = __popc(__ballot_sync(0xffffffffu, p));
    if (c == 0) {
      hi = lo;
    } else {
      const uint32_t top = lo + c * stride;
      lo += (c - 1) * stride + 1;
      hi = min(hi, top);
    }
  }
  return lo;
}

}  // namespace bt
