// Hash front end of the sorted-merge batch (the v38 meaning,
// src/gpu-stm-tree-v38/bpt-gpustm-kernel-aux.cuh:16-56).
//
// The meaning only couples requests whose key is written (INSERT or DELETE)
// somewhere in the batch: a request for a key with no write in the batch, or
// one that comes before the first write of its key, sees the pre-batch tree.  So instead
// of sorting the whole batch, the front end
//
//   1. lists the write requests and sizes an open-addressing table for
//      their keys (a power of two >= 4x the count, at least 1024 slots:
//      most lookups ask for a key the table does not hold, and a linear probe
//      for an absent key runs about (1 + 1/(1-a)^2)/2 slots at load a: 1.4
//      at a = 1/4, 5 at a = 2/3),
//   2. records, per written key, the index of its first write,
//   3. classifies every request: "touched" if its op code is invalid or its
//      key has a write at or before it; otherwise it is a plain lookup,
//      and compacts both classes: in one pass over tiles that take their
//      places as they come when the sample sort follows, else in input
//      order (a flag pass, a scan of the per-tile counts, a scatter pass).
//
// The touched requests go through the sort + segmented-scan path (their
// runs all start with a write, so the pre-batch value reaches them from the
// delete or insert phase, which return each key's previous value); the plain lookups
// run on the pre-batch tree, unsorted, writing their answers in place.  For a
// read-mostly batch the sort shrinks to the INSERTs.
//
// HBM traffic per request: gather (1 B op), table insert (the key of a write),
// split (8 B key + 1 B op + the probe, which is L2-resident for small write
// counts, then a 12 B list entry or touched entry); in input order: flag (the
// same reads, then a 1 B flag), scatter (1 B flag, 9 B read, a 12 B entry).
#include <cuda_runtime.h>

#include "bt_block.cuh"
#include "bt_common.cuh"
#include "bt_internal.h"
#include "bt_launch.cuh"
#include "bt_sort.cuh"

namespace bt {

namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr int kThreads = 256;

struct Slot {
  unsigned long long key;  // kKeyMax = empty
  uint32_t first;          // index of the first write of the key
  uint32_t pad;
};

// SplitMix64's finaliser (Steele, Lea, Flood 2014) as the slot hash
__device__ __forceinline__ uint64_t slot_hash(uint64_t x) {
  x ^= x >> 30;
  x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27;
  x *= 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// INSERT or DELETE: the requests that couple the others of their key
__device__ __forceinline__ uint32_t is_write(uint8_t op) { return (op == kOpInsert || op == kOpDelete) ? 1u : 0u; }

__device__ __forceinline__ uint32_t table_cap(uint32_t n_ins, size_t cap_max) {
  uint64_t c = 1024;
  while (c < 4ull * n_ins) c <<= 1;  // load factor at most 1/4 (up to the allocation)
  return (uint32_t)(c < cap_max ? c : cap_max);
}

// The writes (INSERT and DELETE, with a reserved key too) of the batch: their
// number and their request indices, in no order.  16 op codes a thread, one
// atomic a block.  The insert kernel then has only writes before it, with all
// its probes in flight.  Counting, then reading the op codes again and probing
// where there was a write, was 37 us of a 2^22 batch with 5 % writes; a batch is
// 11 us faster with the list, and a 2^18 Zipf batch 7.
constexpr int kGatherItems = 16;

__global__ void __launch_bounds__(kThreads) front_gather_kernel(const uint8_t* ops, size_t n, uint32_t* list,
                                                                BatchCounts* counts) {
  after_previous();
  __shared__ uint32_t wsum[kThreads / 32], at_block;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t i0 = ((size_t)blockIdx.x * kThreads + threadIdx.x) * kGatherItems;
  uint32_t m = 0;
  if (i0 + kGatherItems <= n && ((uintptr_t)ops & 15u) == 0) {
    const uint4 o = *reinterpret_cast<const uint4*>(ops + i0);
    const uint32_t x[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
    for (int j = 0; j < kGatherItems; j++) m |= is_write((uint8_t)(x[j / 4] >> (8 * (j % 4)))) << j;
  } else {
    for (int j = 0; j < kGatherItems; j++)
      if (i0 + j < n) m |= is_write(ops[i0 + j]) << j;
  }
  const uint32_t c = __popc(m);
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
#pragma unroll
    for (int j = 0; j < kThreads / 32; j++) {
      const uint32_t x = wsum[j];
      wsum[j] = t;
      t += x;
    }
    at_block = t ? atomicAdd(&counts->n_ins_req, t) : 0u;
  }
  __syncthreads();
  uint32_t at = at_block + wsum[warp] + incl - c;
  for (; m; m &= m - 1) list[at++] = (uint32_t)i0 + __ffs(m) - 1;
}

__global__ void __launch_bounds__(kThreads) front_clear_kernel(Slot* tab, size_t cap_max, BatchCounts* counts) {
  after_previous();
  const uint32_t cap = table_cap(counts->n_ins_req, cap_max);
  if (blockIdx.x == 0 && threadIdx.x == 0) counts->cap = cap;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += (size_t)gridDim.x * blockDim.x) {
    tab[i].key = kKeyMax;
    tab[i].first = kNone;
    tab[i].pad = 0;
  }
}

// linear probing; the table is at most a quarter full (half, where the allocation
// limits it: table_cap), so a probe ends
__global__ void __launch_bounds__(kThreads) front_insert_kernel(const uint64_t* keys, const uint32_t* list, Slot* tab,
                                                                const BatchCounts* counts) {
  after_previous();
  const uint32_t mask = counts->cap - 1, n = counts->n_ins_req;
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    const uint32_t i = list[q];
    const uint64_t k = keys[i];
    if (k == kKeyMax) continue;
    uint32_t h = (uint32_t)slot_hash(k) & mask;
    for (uint32_t probe = 0; probe <= mask; probe++) {
      const unsigned long long prev = atomicCAS(&tab[h].key, (unsigned long long)kKeyMax, (unsigned long long)k);
      if (prev == kKeyMax || prev == k) {
        atomicMin(&tab[h].first, i);
        break;
      }
      h = (h + 1) & mask;
    }
  }
}

// Classify, then compact, in three launches over tiles of kTile requests:
//   front_flag_kernel     one flag byte per request ("touched": invalid op
//                         code, or its key has a write at or before it) and
//                         the touched count of each tile;
//   front_tile_scan_kernel  exclusive offsets of the tiles (one block) and
//                         the two class counts;
//   front_scatter_kernel  touched requests to (tk, tv), the rest to list and
//                         their keys to lk, both in input order.
// Every launch is fully parallel (no look-back chain between tiles): the
// probes of the flag pass are its only dependent loads, and the scatter
// reads the request's key and op again only when it is touched.
constexpr int kTileThreads = 256;
constexpr int kTileItems = 8;
constexpr int kTile = kTileThreads * kTileItems;  // 2048
constexpr int kTileWarps = kTileThreads / 32;

// The thread's items of a tile (item j: base + j * THREADS + threadIdx.x),
// their keys and op codes, and a bit per item: touched.
template <int THREADS, int ITEMS>
__device__ __forceinline__ uint32_t classify_items(const uint64_t* keys, const uint8_t* ops,
                                                   size_t n, const Slot* tab,
                                                   const BatchCounts* counts, size_t base,
                                                   uint64_t (&k)[ITEMS], uint8_t (&op)[ITEMS]) {
  const uint32_t mask = counts->cap - 1;
  const bool any = counts->n_ins_req != 0;
  uint64_t sk[ITEMS];
  uint32_t sf[ITEMS], sh[ITEMS];
  // loads first, then every item's first probe slot (independent loads in
  // flight), then the rare longer probes
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const size_t i = base + (size_t)j * THREADS + threadIdx.x;
    k[j] = i < n ? keys[i] : kKeyMax;
    op[j] = i < n ? ops[i] : 0;
  }
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    sh[j] = (uint32_t)slot_hash(k[j]) & mask;
    sk[j] = kKeyMax;
    sf[j] = kNone;
    if (any && k[j] != kKeyMax) {
      const ulonglong2 e = *reinterpret_cast<const ulonglong2*>(tab + sh[j]);
      sk[j] = e.x;
      sf[j] = (uint32_t)e.y;
    }
  }
  // the longer probes, all of this thread's unresolved items one slot per
  // round (their loads in flight together), instead of item after item
  uint32_t first[ITEMS];
  uint32_t todo = 0;
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    first[j] = kNone;
    if (sk[j] == k[j] && k[j] != kKeyMax) first[j] = sf[j];
    else if (sk[j] != kKeyMax) todo |= 1u << j;
  }
  for (uint32_t probe = 0; todo && probe < mask; probe++) {
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
      if (!((todo >> j) & 1u)) continue;
      sh[j] = (sh[j] + 1) & mask;
      const ulonglong2 e = *reinterpret_cast<const ulonglong2*>(tab + sh[j]);
      sk[j] = e.x;
      sf[j] = (uint32_t)e.y;
    }
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
      if (!((todo >> j) & 1u)) continue;
      if (sk[j] == k[j]) {
        first[j] = sf[j];
        todo &= ~(1u << j);
      } else if (sk[j] == kKeyMax) {
        todo &= ~(1u << j);
      }
    }
  }
  uint32_t touched = 0;
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const size_t i = base + (size_t)j * THREADS + threadIdx.x;
    if (i < n) {
      bool f = op[j] > 2;  // invalid op codes are rejected on the sorted path
      if (!f && any && k[j] != kKeyMax) f = first[j] != kNone && (uint32_t)i >= first[j];
      touched |= (f ? 1u : 0u) << j;
    }
  }
  return touched;
}

__global__ void __launch_bounds__(kTileThreads) front_flag_kernel(const uint64_t* keys, const uint8_t* ops, size_t n,
                                                                  const Slot* tab, const BatchCounts* counts,
                                                                  uint8_t* flags, uint32_t* tile_cnt) {
  after_previous();
  __shared__ uint32_t wsum[kTileWarps];
  const size_t base = (size_t)blockIdx.x * kTile;
  uint64_t k[kTileItems];
  uint8_t op[kTileItems];
  const uint32_t touched = classify_items<kTileThreads, kTileItems>(keys, ops, n, tab, counts, base, k, op);
#pragma unroll
  for (int j = 0; j < kTileItems; j++) {
    const size_t i = base + (size_t)j * kTileThreads + threadIdx.x;
    if (i < n) flags[i] = (touched >> j) & 1u;
  }
  const uint32_t c = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(touched));
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
#pragma unroll
    for (int w = 0; w < kTileWarps; w++) t += wsum[w];
    tile_cnt[blockIdx.x] = t;
  }
}

// A tile's requests parted in two lists, each in index order: the tile takes its
// places in both with one atomic each, so the tiles come in any order.
// put(item, in the first list, place).  Two requests a thread and every warp slot
// of an SM in use: what bounds these kernels is the latency of the request, its
// hash slot and the places, not the bytes.  With eight a thread (90 registers,
// two blocks an SM) the 2^22 split took 72 us (1.4 TB/s); a batch is 21 us
// shorter with two (four a thread: 14).
constexpr int kSplitThreads = 512;
constexpr int kSplitItems = 2;
constexpr int kSplitTile = kSplitThreads * kSplitItems;
constexpr int kSplitWarps = kSplitThreads / 32;

template <typename Put>
__device__ __forceinline__ void split_tile(uint32_t here, uint32_t first, uint32_t* n_first, uint32_t* n_second,
                                           Put put) {
  constexpr int kCells = kSplitItems * kSplitWarps, kPer = kCells / 32;  // cells of a lane of the scanning warp
  static_assert(kCells % 32 == 0, "whole lanes");
  __shared__ uint32_t cnt[kCells];
  __shared__ uint32_t at_first, at_second;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t bal[kSplitItems];
#pragma unroll
  for (int j = 0; j < kSplitItems; j++) {
    bal[j] = __ballot_sync(0xffffffffu, (first >> j) & 1u);
    if (lane == 0) cnt[j * kSplitWarps + warp] = __popc(bal[j]);
  }
  __syncthreads();
  // exclusive prefix over (item, warp) in index order
  if (warp == 0) {
    uint32_t c[kPer], sum = 0;
#pragma unroll
    for (int x = 0; x < kPer; x++) {
      c[x] = cnt[lane * kPer + x];
      sum += c[x];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    if (lane == 0) at_first = total ? atomicAdd(n_first, total) : 0u;
    if (lane == 1) at_second = here > total ? atomicAdd(n_second, here - total) : 0u;
    uint32_t at = incl - sum;
#pragma unroll
    for (int x = 0; x < kPer; x++) {
      cnt[lane * kPer + x] = at;
      at += c[x];
    }
  }
  __syncthreads();
  const uint32_t f0 = at_first, s0 = at_second;
#pragma unroll
  for (int j = 0; j < kSplitItems; j++) {
    const uint32_t i = (uint32_t)j * kSplitThreads + threadIdx.x;
    if (i >= here) continue;
    const uint32_t p = cnt[j * kSplitWarps + warp] + __popc(bal[j] & ((1u << lane) - 1u));  // first ones before it
    const bool f = (bal[j] >> lane) & 1u;
    put(j, f, f ? f0 + p : s0 + i - p);
  }
}

// Classify and compact in one launch, for the sample sort, which orders equal
// keys by their request index.  `flags`-free: the class is used where it is found.
__global__ void __launch_bounds__(kSplitThreads, 4)
    front_split_kernel(const uint64_t* keys, const uint8_t* ops, size_t n, const Slot* tab, BatchCounts* counts,
                       uint64_t* tk, uint32_t* tv, uint32_t* list, uint64_t* lk) {
  after_previous();
  const size_t base = (size_t)blockIdx.x * kSplitTile;
  uint64_t k[kSplitItems];
  uint8_t op[kSplitItems];
  const uint32_t touched = classify_items<kSplitThreads, kSplitItems>(keys, ops, n, tab, counts, base, k, op);
  split_tile((uint32_t)min((size_t)kSplitTile, n - base), touched, &counts->n_touch, &counts->n_lookup,
             [&](int j, bool touch, uint32_t at) {
               const uint32_t i = (uint32_t)base + (uint32_t)j * kSplitThreads + threadIdx.x;
               if (touch) {
                 tk[at] = k[j];
                 tv[at] = pair_payload(i, op[j]);
               } else {
                 list[at] = i;
                 lk[at] = k[j];
               }
             });
}

// exclusive offsets of n_tiles counts, in place, with one block
__global__ void __launch_bounds__(1024) front_tile_scan_kernel(uint32_t* tile, uint32_t n_tiles, size_t n,
                                                               BatchCounts* counts, uint32_t* hint) {
  after_previous();
  __shared__ uint32_t wtot[32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (uint32_t b = 0; b < n_tiles; b += 1024) {
    const uint32_t i = b + threadIdx.x;
    const uint32_t v = i < n_tiles ? tile[i] : 0u;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) wtot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      uint32_t t = wtot[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= (uint32_t)o) t += y;
      }
      wtot[lane] = t;  // inclusive over warps
    }
    __syncthreads();
    const uint32_t before = warp ? wtot[warp - 1] : 0u;
    if (i < n_tiles) tile[i] = carry + before + incl - v;
    carry += wtot[31];
    __syncthreads();  // wtot is reused by the next chunk
  }
  if (threadIdx.x == 0) {
    counts->n_touch = carry;
    counts->n_lookup = (uint32_t)n - carry;
    if (hint) *reinterpret_cast<volatile uint32_t*>(hint) = carry;  // host memory: a later batch's sort choice
  }
}

__global__ void __launch_bounds__(kTileThreads) front_scatter_kernel(const uint64_t* keys, const uint8_t* ops,
                                                                     size_t n, const uint8_t* flags,
                                                                     const uint32_t* tile_off, uint64_t* tk,
                                                                     uint32_t* tv, uint32_t* list, uint64_t* lk) {
  after_previous();
  __shared__ uint32_t cnt[kTileItems][kTileWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const size_t base = (size_t)blockIdx.x * kTile;
  uint32_t bal[kTileItems];
#pragma unroll
  for (int j = 0; j < kTileItems; j++) {
    const size_t i = base + (size_t)j * kTileThreads + threadIdx.x;
    bal[j] = __ballot_sync(0xffffffffu, i < n && flags[i] != 0);
    if (lane == 0) cnt[j][warp] = __popc(bal[j]);
  }
  __syncthreads();
  // exclusive prefix over (item, warp) in index order
  if (warp == 0) {
    uint32_t carry = 0;
#pragma unroll
    for (int j = 0; j < kTileItems; j++) {
      const uint32_t c = lane < kTileWarps ? cnt[j][lane] : 0u;
      uint32_t incl = c;
#pragma unroll
      for (int o = 1; o < kTileWarps; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane < kTileWarps) cnt[j][lane] = carry + incl - c;
      carry += __shfl_sync(0xffffffffu, incl, kTileWarps - 1);
    }
  }
  __syncthreads();
  const uint32_t excl = tile_off[blockIdx.x];
#pragma unroll
  for (int j = 0; j < kTileItems; j++) {
    const size_t i = base + (size_t)j * kTileThreads + threadIdx.x;
    if (i < n) {
      const uint32_t p = excl + cnt[j][warp] + __popc(bal[j] & lt);  // touched before i
      const uint64_t k = keys[i];
      if ((bal[j] >> lane) & 1u) {
        const uint8_t op = ops[i];
        tk[p] = k;
        tv[p] = (uint32_t)i | ((op <= 2 ? (uint32_t)op : 3u) << 30);
      } else {
        list[i - p] = (uint32_t)i;
        lk[i - p] = k;
      }
    }
  }
}

// Packed INSERT values (bt_execute_batch_host_packed_async): the caller sends
// the values of the batch's INSERTs only, in request order.  Value j belongs
// to the j-th INSERT; two launches around a scan of the per-tile INSERT
// counts put it at that request's slot, so the batch reads vals[r] as usual.
// HBM traffic per request: 2 B of op codes (read twice), plus 16 B per INSERT.
__device__ __forceinline__ uint32_t tile_ballot(const uint8_t* __restrict__ ops, size_t n, size_t i) {
  return __ballot_sync(0xffffffffu, i < n && ops[i] == kOpInsert);
}

__global__ void __launch_bounds__(kTileThreads) pack_count_kernel(const uint8_t* __restrict__ ops, size_t n,
                                                                  uint32_t* __restrict__ tile_cnt) {
  __shared__ uint32_t wsum[kTileWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t base = (size_t)blockIdx.x * kTile;
  uint32_t c = 0;
#pragma unroll
  for (int j = 0; j < kTileItems; j++) c += __popc(tile_ballot(ops, n, base + (size_t)j * kTileThreads + threadIdx.x));
  if (lane == 0) wsum[warp] = c;
  __syncthreads();
  if (warp == 0) {
    uint32_t v = lane < kTileWarps ? wsum[lane] : 0u;
    v = __reduce_add_sync(0xffffffffu, v);
    if (lane == 0) tile_cnt[blockIdx.x] = v;
  }
}

__global__ void __launch_bounds__(kTileThreads) pack_expand_kernel(const uint8_t* __restrict__ ops, size_t n,
                                                                   const uint32_t* __restrict__ tile_off,
                                                                   const uint64_t* __restrict__ packed,
                                                                   size_t n_packed, uint64_t* __restrict__ vals) {
  __shared__ uint32_t cnt[kTileItems][kTileWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const size_t base = (size_t)blockIdx.x * kTile;
  uint32_t bal[kTileItems];
#pragma unroll
  for (int j = 0; j < kTileItems; j++) {
    bal[j] = tile_ballot(ops, n, base + (size_t)j * kTileThreads + threadIdx.x);
    if (lane == 0) cnt[j][warp] = __popc(bal[j]);
  }
  __syncthreads();
  // exclusive prefix over (item, warp) in index order
  if (warp == 0) {
    uint32_t carry = 0;
#pragma unroll
    for (int j = 0; j < kTileItems; j++) {
      const uint32_t c = lane < kTileWarps ? cnt[j][lane] : 0u;
      uint32_t incl = c;
#pragma unroll
      for (int o = 1; o < kTileWarps; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane < kTileWarps) cnt[j][lane] = carry + incl - c;
      carry += __shfl_sync(0xffffffffu, incl, kTileWarps - 1);
    }
  }
  __syncthreads();
  const size_t excl = tile_off[blockIdx.x];
#pragma unroll
  for (int j = 0; j < kTileItems; j++) {
    if ((bal[j] >> lane) & 1u) {
      const size_t p = excl + cnt[j][warp] + __popc(bal[j] & lt);  // INSERTs before this one
      // the host checked the count; the bound keeps a wrong one inside the buffer
      vals[base + (size_t)j * kTileThreads + threadIdx.x] = p < n_packed ? packed[p] : 0;
    }
  }
}

// A count of packed values that differs from the batch's INSERTs: every op
// code becomes invalid, so every request is answered kRejected and nothing
// is applied (the front end reads the op codes after this kernel)
__global__ void __launch_bounds__(kThreads) pack_check_kernel(const uint32_t* __restrict__ total, size_t n_packed,
                                                              uint8_t* __restrict__ ops, size_t n,
                                                              uint32_t* __restrict__ err) {
  const bool bad = (size_t)*total != n_packed;
  if (blockIdx.x == 0 && threadIdx.x == 0) *err = bad ? 1u : 0u;
  if (!bad) return;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    ops[i] = 0xFF;
}

// ---- INSERT combining for BT_MODE_STM batches ----
// Requests of an STM batch are concurrent transactions (the v39 meaning), so
// any serial order of them is a valid outcome.  The INSERTs of one key are
// put in the order in which they reach the key's table slot (an atomic
// exchange on the slot's tail): the first one (the representative) runs in
// the STM kernel and stores the value of the last one; every other INSERT is
// answered at once with the value of the one before it (FOUND), as if the
// key's INSERTs ran back to back at the representative's commit.  A key that
// the batch also DELETEs is not combined.  A slot's `first` holds the tail
// index, and `pad` the representative's index (bit 31: the key has a DELETE).
constexpr uint32_t kDelBit = 1u << 31;

// The requests of an STM batch split in two lists, in no particular order (the
// tiles'): the valid GETs (with their keys, for the lookup kernels) and the rest
// (INSERT, DELETE, invalid op codes and the reserved key, which the STM kernel
// answers).  counts->n_lookup and counts->n_ins_req end as the lists' lengths.
// One atomic a tile and list: one a warp and list, 16,000 on two words, bound a
// 2^20 batch's split (22 us).
__global__ void __launch_bounds__(kSplitThreads, 4)
    stm_split_kernel(const uint64_t* keys, const uint8_t* ops, size_t n, uint32_t* get_list, uint64_t* get_keys,
                     uint32_t* wr_list, BatchCounts* counts) {
  after_previous();
  const size_t base = (size_t)blockIdx.x * kSplitTile;
  uint64_t k[kSplitItems];
  uint32_t gets = 0;
#pragma unroll
  for (int j = 0; j < kSplitItems; j++) {
    const size_t i = base + (size_t)j * kSplitThreads + threadIdx.x;
    k[j] = i < n ? keys[i] : kKeyMax;
    const uint8_t op = i < n ? ops[i] : (uint8_t)kOpGet;
    gets |= (op == kOpGet && k[j] != kKeyMax ? 1u : 0u) << j;
  }
  split_tile((uint32_t)min((size_t)kSplitTile, n - base), gets, &counts->n_lookup, &counts->n_ins_req,
             [&](int j, bool get, uint32_t at) {
               const uint32_t i = (uint32_t)base + (uint32_t)j * kSplitThreads + threadIdx.x;
               if (get) {
                 get_list[at] = i;
                 get_keys[at] = k[j];
               } else {
                 wr_list[at] = i;
               }
             });
}

__global__ void __launch_bounds__(kThreads) combine_arrive_kernel(const uint64_t* keys, const uint8_t* ops,
                                                                  const uint32_t* list, Slot* tab,
                                                                  const BatchCounts* counts, uint32_t* pred,
                                                                  uint32_t* slot_of) {
  after_previous();
  const uint32_t mask = counts->cap - 1;
  const size_t m = counts->n_ins_req;
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < m; q += (size_t)gridDim.x * blockDim.x) {
    const uint32_t i = list[q];
    const uint8_t op = ops[i];
    if (op != kOpInsert && op != kOpDelete) continue;  // an invalid request: the STM kernel rejects it
    const uint64_t k = keys[i];
    if (k == kKeyMax) continue;
    uint32_t h = (uint32_t)slot_hash(k) & mask;
    uint32_t at = kNone;
    for (uint32_t probe = 0; probe <= mask; probe++) {
      const unsigned long long prev = atomicCAS(&tab[h].key, (unsigned long long)kKeyMax, (unsigned long long)k);
      if (prev == kKeyMax || prev == k) {
        at = h;
        break;
      }
      h = (h + 1) & mask;
    }
    if (op == kOpDelete) {
      if (at != kNone) atomicOr(&tab[at].pad, kDelBit);
      continue;
    }
    slot_of[i] = at;
    if (at == kNone) continue;  // no slot (cannot happen below load 1): runs uncombined
    const uint32_t p = atomicExch(&tab[at].first, i);
    pred[i] = p;
    if (p == kNone) atomicOr(&tab[at].pad, i);
  }
}

// per INSERT: its value for the STM kernel, or (combined with an earlier one)
// its answer and a skip mark
__global__ void __launch_bounds__(kThreads) combine_mark_kernel(const uint64_t* keys, const uint64_t* vals,
                                                                const uint8_t* ops, const uint32_t* list,
                                                                const BatchCounts* counts, const Slot* tab,
                                                                const uint32_t* pred, const uint32_t* slot_of,
                                                                uint8_t* skip, uint64_t* cvals, uint64_t* out_vals,
                                                                uint8_t* out_st) {
  after_previous();
  const size_t m = counts->n_ins_req;
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < m; q += (size_t)gridDim.x * blockDim.x) {
    const uint32_t i = list[q];
    if (ops[i] != kOpInsert) continue;
    const uint32_t at = keys[i] != kKeyMax ? slot_of[i] : kNone;
    uint8_t sk = 0;
    if (at == kNone || (tab[at].pad & kDelBit)) {
      cvals[i] = vals[i];
    } else if (pred[i] != kNone) {
      out_vals[i] = vals[pred[i]];
      out_st[i] = kFound;
      sk = 1;
    } else {
      cvals[i] = vals[tab[at].first];  // the last INSERT of the key
    }
    skip[i] = sk;
  }
}

// a representative that did not commit (retry limit, full node pool): the
// INSERTs combined with it report the same status
__global__ void __launch_bounds__(kThreads) combine_fixup_kernel(const uint8_t* ops, const uint32_t* list,
                                                                 const BatchCounts* counts, const uint8_t* skip,
                                                                 const Slot* tab, const uint32_t* slot_of,
                                                                 uint64_t* out_vals, uint8_t* out_st) {
  after_previous();
  const size_t m = counts->n_ins_req;
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < m; q += (size_t)gridDim.x * blockDim.x) {
    const uint32_t i = list[q];
    if (ops[i] != kOpInsert || !skip[i]) continue;
    const uint32_t rep = tab[slot_of[i]].pad & ~kDelBit;
    const uint8_t st = out_st[rep];
    if (st == kRetryExhausted || st == kNoCapacity) {
      out_st[i] = st;
      out_vals[i] = 0;
    }
  }
}

}  // namespace

int stm_split(Handle* h, const uint64_t* keys, const uint8_t* ops, size_t n, cudaStream_t s) {
  Work& w = h->w;
  const unsigned tiles = (unsigned)((n + kSplitTile - 1) / kSplitTile);
  if (cudaMemsetAsync(w.counts, 0, sizeof(BatchCounts), s) != cudaSuccess) return -2;
  launch_after(stm_split_kernel, tiles, kSplitThreads, 0, s, keys, ops, n, w.get_list, w.ukeys, w.ins_list, w.counts);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int stm_combine(Handle* h, const uint64_t* keys, const uint64_t* vals, const uint8_t* ops, size_t n,
                uint64_t* out_vals, uint8_t* out_st, cudaStream_t s, const uint8_t** skip, const uint64_t** cvals) {
  Work& w = h->w;
  BatchCounts* c = w.counts;
  Slot* tab = reinterpret_cast<Slot*>(w.f_tab);
  uint8_t* sk = reinterpret_cast<uint8_t*>(w.f_flags);
  uint64_t* cv = w.f_lk;
  uint32_t* pred = w.f_list;
  uint32_t* slot_of = w.f_pos;
  uint32_t* list = w.ins_list;
  const unsigned g = (unsigned)min((size_t)h->sm_count * 8, (n / 4 + kThreads) / kThreads);
  launch_after(front_clear_kernel, (unsigned)h->sm_count * 4, kThreads, 0, s, tab, w.f_tab_cap, c);
  launch_after(combine_arrive_kernel, g, kThreads, 0, s, keys, ops, list, tab, c, pred, slot_of);
  launch_after(combine_mark_kernel, g, kThreads, 0, s, keys, vals, ops, list, c, tab, pred, slot_of, sk, cv, out_vals,
               out_st);
  count_launch(3);
  *skip = sk;
  *cvals = cv;
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int stm_combine_fixup(Handle* h, const uint8_t* ops, size_t n, uint64_t* out_vals, uint8_t* out_st, cudaStream_t s) {
  Work& w = h->w;
  const unsigned g = (unsigned)min((size_t)h->sm_count * 8, (n / 4 + kThreads) / kThreads);
  launch_after(combine_fixup_kernel, g, kThreads, 0, s, ops, w.ins_list, w.counts,
               reinterpret_cast<const uint8_t*>(w.f_flags), reinterpret_cast<const Slot*>(w.f_tab), w.f_pos, out_vals,
               out_st);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// scratch: tile counts, tile offsets, the INSERT total, the mismatch flag,
// then the scan's own words
size_t pack_scratch_words(size_t n) {
  const size_t tiles = (n + kTile - 1) / kTile;
  return 2 * (tiles + 1) + 2 + scan_scratch_words(tiles);
}

uint32_t* pack_error_word(uint32_t* scratch, size_t n_cap) {
  const size_t tiles = (n_cap + kTile - 1) / kTile;
  return scratch + 2 * (tiles + 1) + 1;
}

cudaError_t pack_check(uint8_t* ops, size_t n, size_t n_packed, uint32_t* scratch, size_t n_cap, int sm_count,
                       cudaStream_t s) {
  const size_t tiles = (n + kTile - 1) / kTile;
  const size_t cap_tiles = (n_cap + kTile - 1) / kTile;
  uint32_t* cnt = scratch;
  uint32_t* off = cnt + cap_tiles + 1;
  uint32_t* total = off + cap_tiles + 1;
  uint32_t* scan = total + 2;
  pack_count_kernel<<<(unsigned)tiles, kTileThreads, 0, s>>>(ops, n, cnt);
  count_launch();
  cudaError_t e = scan_exclusive_u32(cnt, off, tiles, total, scan, s);
  if (e != cudaSuccess) return e;
  pack_check_kernel<<<(unsigned)sm_count * 2, kThreads, 0, s>>>(total, n_packed, ops, n, total + 1);
  count_launch();
  return cudaGetLastError();
}

cudaError_t pack_expand(const uint8_t* ops, size_t n, const uint64_t* packed, size_t n_packed, uint64_t* vals,
                        const uint32_t* scratch, size_t n_cap, cudaStream_t s) {
  if (n == 0 || n_packed == 0) return cudaSuccess;
  const size_t tiles = (n + kTile - 1) / kTile;
  const size_t cap_tiles = (n_cap + kTile - 1) / kTile;
  pack_expand_kernel<<<(unsigned)tiles, kTileThreads, 0, s>>>(ops, n, scratch + cap_tiles + 1, packed, n_packed,
                                                              vals);
  count_launch();
  return cudaGetLastError();
}

// Fills w.f_tk/w.f_tv (touched requests, count counts->n_touch) and
// w.f_list/w.f_lk (plain lookups and their keys, count counts->n_lookup), in
// input order when `ordered`.
int front_classify(Handle* h, const uint64_t* keys, const uint8_t* ops, size_t n, bool ordered, cudaStream_t s) {
  Work& w = h->w;
  BatchCounts* c = w.counts;
  const size_t n_tiles = (n + kTile - 1) / kTile;
  if (cudaMemsetAsync(c, 0, sizeof(BatchCounts), s) != cudaSuccess) return -2;
  const unsigned g = (unsigned)min((size_t)h->sm_count * 8, (n + kThreads - 1) / kThreads);
  Slot* tab = reinterpret_cast<Slot*>(w.f_tab);
  uint8_t* flags = reinterpret_cast<uint8_t*>(w.f_flags);
  uint32_t* tile = w.f_pos;  // per-tile counts, then offsets
  // the writes' list lies in w.f_list until the split, which needs it no more, fills that
  const unsigned gather = (unsigned)((n + kThreads * kGatherItems - 1) / (kThreads * kGatherItems));
  launch_after(front_gather_kernel, gather, kThreads, 0, s, ops, n, w.f_list, c);
  launch_after(front_clear_kernel, (unsigned)h->sm_count * 4, kThreads, 0, s, tab, w.f_tab_cap, c);
  launch_after(front_insert_kernel, g, kThreads, 0, s, keys, w.f_list, tab, c);
  if (!ordered) {
    const unsigned split_tiles = (unsigned)((n + kSplitTile - 1) / kSplitTile);
    launch_after(front_split_kernel, split_tiles, kSplitThreads, 0, s, keys, ops, n, tab, c, w.f_tk, w.f_tv,
                 w.f_list, w.f_lk);
    count_launch(4);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
  }
  launch_after(front_flag_kernel, (unsigned)n_tiles, kTileThreads, 0, s, keys, ops, n, tab, c, flags, tile);
  launch_after(front_tile_scan_kernel, 1, 1024, 0, s, tile, (uint32_t)n_tiles, n, c, h->touch_hint_dev);
  launch_after(front_scatter_kernel, (unsigned)n_tiles, kTileThreads, 0, s, keys, ops, n, flags, tile, w.f_tk, w.f_tv,
               w.f_list, w.f_lk);
  count_launch(6);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace bt
