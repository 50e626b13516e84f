// Sample sort of the hash front end's touched requests, with the first half of
// the batch merge's segmented scan (bt_batch.cu) on the way.
//
// A read-mostly batch of 2^22 has about 2^18 touched requests.  Sorted tile runs
// merged pairwise took a tile kernel of 26 us and seven rounds of 7-9 us, each
// bound by its launch and a dependent search, and the scan three passes more
// (40 us); eight radix passes took 115 us.  Here the pairs cross memory twice
// (us a pass of the batches: 262,145 Zipf requests with 20 % writes, twice, 492 ->
// 376; 2^20 at 50 %, twice, 1248 -> 1157; four host batches of 2^20 1990 -> 1610):
//
//   ss_splitters_kernel  one block: a sorted sample, every k-th pair of it a
//                        splitter (buckets of about 1024-1536 pairs);
//   ss_count_kernel      every pair's bucket by binary search in the splitters,
//                        the tiles' counts added to the buckets';
//   ss_scatter_kernel    the pairs to their buckets;
//   ss_sort_kernel       one block per bucket: sorted on chip, and what the
//                        segmented scan needs of it (BucketSum);
//   ss_resolve_kernel    one block per bucket: the carries of the buckets before
//                        it, then every request's answer or its run's id, and
//                        the unique keys' work lists (merge_pass2 and 3 in one).
//
// Pairs (bt_sort.cuh) are ordered by key, then request, all different, so equal keys spread
// over buckets like any others and a hot key fills no bucket.  The splitters
// come from fixed pseudo-random positions; a bucket that outgrows a block's
// shared memory (more pairs than kSsBuckets is meant for, or an input that beats
// the sample) is sorted in chunks merged through global memory: slower, the
// same result.
#include <cuda_runtime.h>

#include "bt_block.cuh"
#include "bt_common.cuh"
#include "bt_internal.h"
#include "bt_launch.cuh"
#include "bt_sort.cuh"

namespace bt {

struct BucketSum {
  uint32_t agg;    // packed state (below) after the bucket, its first run taken as a continuation
  uint32_t pre;    // ... at the end of the first run, if it ends in the bucket
  uint32_t heads;  // runs after the first
  uint32_t ins, del;  // runs that begin and end inside (neither the first nor the last), by their last write
  uint32_t multi;  // more than one run
  uint32_t pad[2];
};

namespace {

constexpr int kBuckets = (int)kSsBuckets;
constexpr int kCap = 4096;  // pairs that one block sorts on chip
constexpr int kTileThreads = 256;
constexpr int kTileItems = 8;
constexpr int kTile = kTileThreads * kTileItems;

// The "latest write in the current run" state in one word: bit 31 a run head
// occurred; below it the request index of the latest INSERT after the last
// head, or kNoWrite, or kDeleted.
constexpr uint32_t kHead = 0x80000000u, kNoWrite = 0x40000000u, kDeleted = 0x40000001u;
__device__ __forceinline__ uint32_t st_of(uint32_t s) { return s & ~kHead; }
__device__ __forceinline__ uint32_t st_combine(uint32_t a, uint32_t b) {
  const uint32_t bv = st_of(b);
  const uint32_t v = bv != kNoWrite ? bv : (b & kHead) ? kNoWrite : st_of(a);
  return ((a | b) & kHead) | v;
}
__device__ __forceinline__ bool is_ins(uint32_t s) { return st_of(s) < kNoWrite; }
__device__ __forceinline__ bool is_del(uint32_t s) { return st_of(s) == kDeleted; }

// exclusive scan of the state over the block; total: the block's
__device__ __forceinline__ uint32_t blk_exclusive_st(uint32_t x, uint32_t* ws, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t inc = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc = st_combine(y, inc);
  }
  uint32_t ex = __shfl_up_sync(0xffffffffu, inc, 1);
  if (lane == 0) ex = kNoWrite;
  if (lane == 31) ws[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint32_t s = lane < nw ? ws[lane] : kNoWrite;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s = st_combine(y, s);
    }
    if (lane < nw) ws[lane] = s;
  }
  __syncthreads();
  const uint32_t before = warp ? ws[warp - 1] : kNoWrite;
  if (total) *total = ws[nw - 1];
  __syncthreads();
  return st_combine(before, ex);
}

// one request's part of the scan
__device__ __forceinline__ uint32_t item_state(uint64_t k, uint32_t v, bool head) {
  const uint32_t op = pair_op(v);
  uint32_t s = kNoWrite;
  if (k != kKeyMax) s = op == kOpInsert ? pair_idx(v) : op == kOpDelete ? kDeleted : kNoWrite;
  return s | (head ? kHead : 0u);
}

// one bucket per 1024 pairs while every SM has one at most, then whole waves of
// at most 1536 (one per 1024 throughout, with a last wave a fraction full: 2^19
// pairs 8 us more)
__device__ __forceinline__ uint32_t bucket_count(uint32_t m, uint32_t sms) {
  uint32_t p = (m + 1023) / 1024;
  if (p > sms) p = sms * ((m + sms * 1536 - 1) / (sms * 1536));
  return p < 1 ? 1 : p > (uint32_t)kBuckets ? (uint32_t)kBuckets : p;
}

struct SortSmem {
  uint64_t k[kCap];
  uint32_t v[kCap];
  uint32_t ws[32];
  uint32_t split[2];
  uint32_t pre, pre_any;
  uint32_t sum[3];  // heads, ins, del of the bucket
};

__global__ void __launch_bounds__(1024, 1) ss_splitters_kernel(const uint64_t* tk, const uint32_t* tv,
                                                               uint32_t n_upper, const uint32_t* n_dev, uint32_t sms,
                                                               uint64_t* spk, uint32_t* spv, uint32_t* total,
                                                               uint32_t* hint) {
  after_previous();
  extern __shared__ __align__(16) unsigned char raw[];
  SortSmem& S = *reinterpret_cast<SortSmem*>(raw);
  const uint32_t m = min(n_upper, *n_dev);
  const uint32_t p = bucket_count(m, sms);
  if (threadIdx.x < kBuckets) total[threadIdx.x] = 0;
  if (threadIdx.x == 0 && hint) *reinterpret_cast<volatile uint32_t*>(hint) = *n_dev;  // host memory: a later batch's sort choice
  if (p == 1) return;
  // four samples per bucket or more (the largest bucket about 2.5 times the mean),
  // eight when the buckets are more than 3/8 full: this block's sort is the longest
  // step of the splitting (34 us for 4096 samples, half for 2048)
  uint32_t s = 512;
  while (s < (m > p * 1536 ? 8 : 4) * p && s < (uint32_t)kCap) s <<= 1;
  const uint32_t step = m / s;
  for (uint32_t i = threadIdx.x; i < s; i += blockDim.x) {
    const uint32_t at = (uint32_t)((uint64_t)i * m / s) + (i * 0x9E3779B1u >> 8) % (step ? step : 1u);
    S.k[i] = tk[at];
    S.v[i] = tv[at];
  }
  __syncthreads();
  block_sort(S.k, S.v, (int)s);
  for (uint32_t j = threadIdx.x + 1; j < p; j += blockDim.x) {
    const uint32_t at = (uint32_t)((uint64_t)j * s / p);
    spk[j - 1] = S.k[at];
    spv[j - 1] = S.v[at];
  }
}

__global__ void __launch_bounds__(kTileThreads) ss_count_kernel(const uint64_t* tk, const uint32_t* tv,
                                                                uint32_t n_upper, const uint32_t* n_dev, uint32_t sms,
                                                                const uint64_t* spk, const uint32_t* spv,
                                                                uint16_t* ids, uint32_t* off, uint32_t* total) {
  after_previous();
  __shared__ uint64_t sk[kBuckets];
  __shared__ uint32_t sv[kBuckets];
  __shared__ uint32_t hist[kBuckets];
  const uint32_t m = min(n_upper, *n_dev);
  const uint32_t p = bucket_count(m, sms);
  for (uint32_t j = threadIdx.x; j + 1 < p; j += kTileThreads) {
    sk[j] = spk[j];
    sv[j] = spv[j];
  }
  for (uint32_t t = blockIdx.x; (uint64_t)t * kTile < m; t += gridDim.x) {
    for (int j = threadIdx.x; j < kBuckets; j += kTileThreads) hist[j] = 0;
    __syncthreads();
    uint64_t k[kTileItems];
    uint32_t v[kTileItems], lo[kTileItems], hi[kTileItems];
#pragma unroll
    for (int j = 0; j < kTileItems; j++) {
      const uint32_t i = t * kTile + j * kTileThreads + threadIdx.x;
      k[j] = i < m ? tk[i] : 0;
      v[j] = i < m ? tv[i] : 0;
      lo[j] = 0;
      hi[j] = p - 1;
    }
    // splitters not above the pair, all of the thread's searches in step
    for (uint32_t w = p - 1; w > 0; w >>= 1) {
#pragma unroll
      for (int j = 0; j < kTileItems; j++) {
        if (lo[j] < hi[j]) {
          const uint32_t mid = (lo[j] + hi[j]) >> 1;
          if (pair_less(k[j], v[j], sk[mid], sv[mid])) hi[j] = mid;
          else lo[j] = mid + 1;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < kTileItems; j++) {
      const uint32_t i = t * kTile + j * kTileThreads + threadIdx.x;
      if (i < m) {
        ids[i] = (uint16_t)lo[j];
        atomicAdd(&hist[lo[j]], 1u);
      }
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < p; j += kTileThreads)
      if (hist[j]) off[(size_t)t * kBuckets + j] = atomicAdd(total + j, hist[j]);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kTileThreads) ss_scatter_kernel(const uint64_t* tk, const uint32_t* tv,
                                                                  uint32_t n_upper, const uint32_t* n_dev,
                                                                  uint32_t sms, const uint16_t* ids,
                                                                  const uint32_t* off, const uint32_t* total,
                                                                  uint32_t* base, uint64_t* kb, uint32_t* vb) {
  after_previous();
  __shared__ uint32_t ws[32];
  __shared__ uint32_t start[kBuckets], hist[kBuckets];
  const uint32_t m = min(n_upper, *n_dev);
  const uint32_t p = bucket_count(m, sms);
  static_assert(kBuckets == 2 * kTileThreads, "two buckets per thread below");
  const uint32_t b = 2 * threadIdx.x;
  const uint32_t c0 = b < p ? total[b] : 0u, c1 = b + 1 < p ? total[b + 1] : 0u;
  const uint32_t ex = blk_exclusive_sum(c0 + c1, ws, nullptr);
  start[b] = ex;
  start[b + 1] = ex + c0;
  if (blockIdx.x == 0) {
    base[b] = ex;
    base[b + 1] = ex + c0;
    if (threadIdx.x == kTileThreads - 1) base[kBuckets] = m;
  }
  for (uint32_t t = blockIdx.x; (uint64_t)t * kTile < m; t += gridDim.x) {
    __syncthreads();
    for (int j = threadIdx.x; j < kBuckets; j += kTileThreads) hist[j] = 0;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kTileItems; j++) {
      const uint32_t i = t * kTile + j * kTileThreads + threadIdx.x;
      if (i < m) {
        const uint32_t d = ids[i];
        const uint32_t at = start[d] + off[(size_t)t * kBuckets + d] + atomicAdd(&hist[d], 1u);
        kb[at] = tk[i];
        vb[at] = tv[i];
      }
    }
  }
}

// elements of A among the first d of merge(A, B); one warp, 32 candidates per step
__device__ __forceinline__ uint32_t run_split(const uint64_t* k, const uint32_t* v, uint32_t na, uint32_t nb,
                                              uint32_t d) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t lo = d > nb ? d - nb : 0, hi = min(d, na);
  while (lo < hi) {
    const uint32_t stride = (hi - lo + 31) / 32;
    const uint32_t a = lo + lane * stride;
    const uint32_t b = na + d - 1 - a;
    const bool less = a < hi && pair_less(k[a], v[a], k[b], v[b]);
    const uint32_t c = __popc(__ballot_sync(0xffffffffu, less));
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

// a bucket beyond kCap: sorted chunks, then pairs of runs merged through
// (ka, va) and (kb, vb) in turn; the result ends in (ka, va)
__device__ __noinline__ void sort_large(SortSmem& S, uint64_t* ka, uint32_t* va, uint64_t* kb, uint32_t* vb,
                                        uint32_t s) {
  int rounds = 0;
  while (((uint64_t)kCap << rounds) < s) rounds++;
  uint64_t* dk = rounds & 1 ? kb : ka;
  uint32_t* dv = rounds & 1 ? vb : va;
  for (uint32_t c0 = 0; c0 < s; c0 += kCap) {
    const int cnt = (int)min((uint32_t)kCap, s - c0);
    for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
      S.k[i] = kb[c0 + i];
      S.v[i] = vb[c0 + i];
    }
    __syncthreads();
    block_sort(S.k, S.v, cnt);
    for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
      dk[c0 + i] = S.k[i];
      dv[c0 + i] = S.v[i];
    }
    __syncthreads();
  }
  for (int r = 0; r < rounds; r++) {
    const uint64_t* xk = (rounds - r) & 1 ? kb : ka;
    const uint32_t* xv = (rounds - r) & 1 ? vb : va;
    dk = (rounds - r) & 1 ? ka : kb;
    dv = (rounds - r) & 1 ? va : vb;
    const uint64_t L = (uint64_t)kCap << r;
    for (uint32_t o0 = 0; o0 < s; o0 += kCap) {
      const int cnt = (int)min((uint32_t)kCap, s - o0);
      const uint32_t ps = (uint32_t)(o0 / (2 * L) * (2 * L));
      const uint32_t na = (uint32_t)min(L, (uint64_t)(s - ps)), nb = (uint32_t)min(L, (uint64_t)(s - ps - na));
      const uint32_t d0 = o0 - ps;
      if (threadIdx.x < 64) {
        const uint32_t w = threadIdx.x >> 5;
        const uint32_t a = run_split(xk + ps, xv + ps, na, nb, w ? d0 + cnt : d0);
        if ((threadIdx.x & 31) == 0) S.split[w] = a;
      }
      __syncthreads();
      const uint32_t a0 = S.split[0], b0 = d0 - a0;
      const int la = (int)(S.split[1] - a0), lb = cnt - la;
      for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
        const uint32_t at = i < la ? ps + a0 + i : ps + na + b0 + (i - la);
        S.k[i] = xk[at];
        S.v[i] = xv[at];
      }
      __syncthreads();
      const int d = threadIdx.x * 4;
      uint64_t K[4];
      uint32_t V[4];
      if (d < cnt) merge4(S.k, S.v, la, S.k + la, S.v + la, lb, d, K, V);
#pragma unroll
      for (int e = 0; e < 4; e++)
        if (d + e < cnt) {
          dk[o0 + d + e] = K[e];
          dv[o0 + d + e] = V[e];
        }
      __syncthreads();
    }
  }
}

__global__ void __launch_bounds__(1024, 1) ss_sort_kernel(uint32_t n_upper, const uint32_t* n_dev, uint32_t sms,
                                                          const uint32_t* base, uint64_t* ka, uint32_t* va,
                                                          uint64_t* kb, uint32_t* vb, BucketSum* sums) {
  after_previous();
  extern __shared__ __align__(16) unsigned char raw[];
  SortSmem& S = *reinterpret_cast<SortSmem*>(raw);
  const uint32_t m = min(n_upper, *n_dev);
  const uint32_t p = bucket_count(m, sms);
  for (uint32_t b = blockIdx.x; b < p; b += gridDim.x) {
    const uint32_t at = base[b], s = (b + 1 < p ? base[b + 1] : m) - at;
    if (s <= (uint32_t)kCap) {
      for (uint32_t i = threadIdx.x; i < s; i += blockDim.x) {
        S.k[i] = kb[at + i];
        S.v[i] = vb[at + i];
      }
      __syncthreads();
      if (s) block_sort(S.k, S.v, (int)s);
      for (uint32_t i = threadIdx.x; i < s; i += blockDim.x) {
        ka[at + i] = S.k[i];
        va[at + i] = S.v[i];
      }
    } else {
      sort_large(S, ka + at, va + at, kb + at, vb + at, s);
    }
    // the bucket's part of the segmented scan, its first run as a continuation
    // and its last run left open
    uint32_t run = kNoWrite, heads = 0, ins = 0, del = 0;
    if (threadIdx.x == 0) {
      S.pre = kNoWrite;
      S.pre_any = 0;
      S.sum[0] = S.sum[1] = S.sum[2] = 0;
    }
    for (uint32_t c0 = 0; c0 < s; c0 += kCap) {
      const int cnt = (int)min((uint32_t)kCap, s - c0);
      if (s > (uint32_t)kCap) {
        __syncthreads();
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
          S.k[i] = ka[at + c0 + i];
          S.v[i] = va[at + c0 + i];
        }
      }
      __syncthreads();
      const int d = threadIdx.x * 4;
      uint32_t st[4], tail = 0, mine = kNoWrite;
      uint64_t key[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int i = d + e;
        st[e] = kNoWrite;
        key[e] = 0;
        if (i >= cnt) continue;
        key[e] = S.k[i];
        const bool head = i > 0 ? S.k[i - 1] != key[e] : c0 > 0 && ka[at + c0 - 1] != key[e];
        const bool tl = i + 1 < cnt ? S.k[i + 1] != key[e] : c0 + cnt < s && ka[at + c0 + cnt] != key[e];
        st[e] = item_state(key[e], S.v[i], head);
        heads += head ? 1u : 0u;
        tail |= (tl ? 1u : 0u) << e;
        mine = st_combine(mine, st[e]);
      }
      uint32_t all;
      uint32_t x = st_combine(run, blk_exclusive_st(mine, S.ws, &all));
#pragma unroll
      for (int e = 0; e < 4; e++) {
        x = st_combine(x, st[e]);
        if (!((tail >> e) & 1u)) continue;
        if (!(x & kHead)) {  // the end of the first run
          S.pre = x;
          S.pre_any = 1;
        } else if (key[e] != kKeyMax) {
          ins += is_ins(x) ? 1u : 0u;
          del += is_del(x) ? 1u : 0u;
        }
      }
      run = st_combine(run, all);
    }
    // (nothing to add where the loop did not run, so the zeroes above are seen)
    heads = __reduce_add_sync(0xffffffffu, heads);
    ins = __reduce_add_sync(0xffffffffu, ins);
    del = __reduce_add_sync(0xffffffffu, del);
    if ((threadIdx.x & 31) == 0) {
      if (heads) atomicAdd(&S.sum[0], heads);
      if (ins) atomicAdd(&S.sum[1], ins);
      if (del) atomicAdd(&S.sum[2], del);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      BucketSum& o = sums[b];
      o.agg = run;
      o.pre = S.pre;
      o.heads = S.sum[0];
      o.ins = S.sum[1];
      o.del = S.sum[2];
      o.multi = S.pre_any;
    }
    __syncthreads();
  }
}

constexpr int kResThreads = 512;
constexpr int kResItems = 4;  // most buckets in one turn (eight idled two threads of three)
constexpr int kResTile = kResThreads * kResItems;

__global__ void __launch_bounds__(kResThreads) ss_resolve_kernel(
    const uint64_t* sk, const uint32_t* sv, const uint64_t* vals, uint32_t n_upper, const uint32_t* n_dev,
    uint32_t sms, const uint32_t* base, const BucketSum* sums, uint64_t* ukeys, uint64_t* uvals, uint32_t* ins_list,
    uint32_t* del_list, uint32_t* pend, uint64_t* out_vals, uint8_t* out_st, BatchCounts* counts) {
  after_previous();
  __shared__ uint32_t ws[32];
  __shared__ uint32_t carry[kBuckets], hb[kBuckets], ib[kBuckets], db[kBuckets];
  static_assert(kResThreads == kBuckets, "one bucket per thread below");
  const uint32_t m = min(n_upper, *n_dev);
  const uint32_t p = bucket_count(m, sms);
  if (blockIdx.x >= p) return;
  {
    // carries and counts before every bucket (the rules of merge_pass2)
    const uint32_t b = threadIdx.x;
    BucketSum x{};
    x.agg = x.pre = kNoWrite;
    bool any = false, h0 = false, open = true;
    uint64_t first = 0, last = 0;
    if (b < p) {
      const uint32_t a = base[b], e = b + 1 < p ? base[b + 1] : m;
      any = e > a;
      if (any) {
        x = sums[b];
        first = sk[a];
        last = sk[e - 1];
        h0 = a == 0 || sk[a - 1] != first;      // the first run begins here
        open = e < m && sk[e] == last;          // the last run goes on
      }
    }
    const uint32_t self = !any ? kNoWrite : (!x.multi && h0) ? x.agg | kHead : x.agg;
    const uint32_t c = blk_exclusive_st(self, ws, nullptr);
    uint32_t ins = x.ins, del = x.del;
    if (any && x.multi && first != kKeyMax) {  // the first run ends here
      const uint32_t s = h0 ? x.pre : st_combine(c, x.pre);
      ins += is_ins(s) ? 1u : 0u;
      del += is_del(s) ? 1u : 0u;
    }
    if (any && !open && last != kKeyMax) {  // the last run ends here
      const uint32_t s = (x.multi || h0) ? x.agg : st_combine(c, x.agg);
      ins += is_ins(s) ? 1u : 0u;
      del += is_del(s) ? 1u : 0u;
    }
    uint32_t th, ti, td;
    const uint32_t eh = blk_exclusive_sum(any ? x.heads + (h0 ? 1u : 0u) : 0u, ws, &th);
    const uint32_t ei = blk_exclusive_sum(ins, ws, &ti);
    const uint32_t ed = blk_exclusive_sum(del, ws, &td);
    carry[b] = st_of(c);
    hb[b] = eh;
    ib[b] = ei;
    db[b] = ed;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      counts->n_unique = th;
      counts->n_ins = ti;
      counts->n_get = 0;  // every touched run begins with a write or is rejected
      counts->n_del = td;
    }
  }
  __syncthreads();
  for (uint32_t b = blockIdx.x; b < p; b += gridDim.x) {
    const uint32_t a = base[b], e = b + 1 < p ? base[b + 1] : m;
    uint32_t run = carry[b], hpos0 = hb[b], ipos0 = ib[b], dpos0 = db[b];
    for (uint32_t c0 = a; c0 < e; c0 += kResTile) {
      const uint32_t i0 = c0 + threadIdx.x * kResItems;
      uint64_t k[kResItems];
      uint32_t v[kResItems], st[kResItems];
      uint32_t head = 0, tail = 0, valid = 0, mine = kNoWrite, heads = 0;
      const uint64_t prev = i0 > 0 && i0 < e ? sk[i0 - 1] : 0;
#pragma unroll
      for (int j = 0; j < kResItems; j++) {
        const uint32_t i = i0 + j;
        k[j] = i < e ? sk[i] : 0;
        v[j] = i < e ? sv[i] : 0;
        valid |= (i < e ? 1u : 0u) << j;
      }
      const uint64_t next = i0 + kResItems < m ? sk[i0 + kResItems] : 0;
#pragma unroll
      for (int j = 0; j < kResItems; j++) {
        const uint32_t i = i0 + j;
        st[j] = kNoWrite;
        if (i >= e) continue;
        const bool h = i == 0 || (j > 0 ? k[j > 0 ? j - 1 : 0] : prev) != k[j];
        // the pair behind it: in registers, or the next thread's first, or the next bucket's
        const uint64_t nx = j + 1 < kResItems && i + 1 < e ? k[j + 1 < kResItems ? j + 1 : 0]
                            : j + 1 == kResItems ? next : i + 1 < m ? sk[i + 1] : 0;
        const bool tl = i + 1 == m || nx != k[j];
        st[j] = item_state(k[j], v[j], h);
        head |= (h ? 1u : 0u) << j;
        tail |= (tl ? 1u : 0u) << j;
        heads += h ? 1u : 0u;
        mine = st_combine(mine, st[j]);
      }
      uint32_t all;
      uint32_t s = st_combine(run, blk_exclusive_st(mine, ws, &all));
      uint32_t ins = 0, del = 0;
      {
        uint32_t y = s;
#pragma unroll
        for (int j = 0; j < kResItems; j++) {
          y = st_combine(y, st[j]);
          if (((tail >> j) & 1u) && k[j] != kKeyMax) {
            ins += is_ins(y) ? 1u : 0u;
            del += is_del(y) ? 1u : 0u;
          }
        }
      }
      uint32_t th, tw;
      uint32_t hpos = hpos0 + blk_exclusive_sum(heads, ws, &th);
      const uint32_t w = blk_exclusive_sum(ins | (del << 16), ws, &tw);  // at most kResTile of each
      uint32_t ipos = ipos0 + (w & 0xffffu), dpos = dpos0 + (w >> 16);
#pragma unroll
      for (int j = 0; j < kResItems; j++) {
        if (!((valid >> j) & 1u)) break;
        const bool h = (head >> j) & 1u;
        if (h) hpos++;
        const uint32_t u = hpos - 1;  // unique id of this request's run
        const uint32_t r = pair_idx(v[j]);
        uint32_t pd = u;
        if (k[j] == kKeyMax || pair_op(v[j]) > 2u) {
          out_vals[r] = 0;
          out_st[r] = kRejected;
          pd = 0xFFFFFFFFu;
        } else if (!h && st_of(s) != kNoWrite) {  // an earlier write of this same run
          out_vals[r] = is_del(s) ? 0 : vals[st_of(s)];
          out_st[r] = is_del(s) ? kAbsent : kFound;
          pd = 0xFFFFFFFFu;
        }
        pend[i0 + j] = pd;
        s = st_combine(s, st[j]);
        if (((tail >> j) & 1u) && k[j] != kKeyMax) {
          ukeys[u] = k[j];
          if (is_del(s)) {
            del_list[dpos++] = u;
          } else if (is_ins(s)) {
            uvals[u] = vals[st_of(s)];
            ins_list[ipos++] = u;
          }
        }
      }
      run = st_of(st_combine(run, all));
      hpos0 += th;
      ipos0 += tw & 0xffffu;
      dpos0 += tw >> 16;
    }
  }
}

}  // namespace

size_t sample_sum_bytes() { return kSsBuckets * sizeof(BucketSum) + (kSsBuckets + 1) * 4 + 256; }

int sample_prepare() {
  cudaError_t e = cudaFuncSetAttribute(ss_splitters_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(SortSmem));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(ss_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SortSmem));
  return e == cudaSuccess ? 0 : -2;
}

static uint32_t* sum_base(void* sums) {
  return reinterpret_cast<uint32_t*>(static_cast<char*>(sums) + kSsBuckets * sizeof(BucketSum));
}

int sample_sort(Handle* h, size_t n, cudaStream_t s) {
  Work& w = h->w;
  const uint32_t nu = (uint32_t)n, sms = (uint32_t)h->sm_count;
  const uint32_t* m = &w.counts->n_touch;
  uint64_t* spk = w.s_split;
  uint32_t* spv = reinterpret_cast<uint32_t*>(spk + kSsBuckets);
  uint32_t* total = spv + kSsBuckets;
  uint16_t* ids = reinterpret_cast<uint16_t*>(w.f_flags);
  uint32_t* off = w.sort_scratch;
  uint32_t* base = sum_base(w.s_sum);
  BucketSum* sums = reinterpret_cast<BucketSum*>(w.s_sum);
  const unsigned tiles = (unsigned)min((n + kTile - 1) / kTile, (size_t)h->sm_count * 4);
  launch_after(ss_splitters_kernel, 1, 1024, sizeof(SortSmem), s, w.f_tk, w.f_tv, nu, m, sms, spk, spv, total,
               h->touch_hint_dev);
  launch_after(ss_count_kernel, tiles, kTileThreads, 0, s, w.f_tk, w.f_tv, nu, m, sms, spk, spv, ids, off, total);
  launch_after(ss_scatter_kernel, tiles, kTileThreads, 0, s, w.f_tk, w.f_tv, nu, m, sms, ids, off, total, base, w.k_b,
               w.v_b);
  const unsigned buckets = (unsigned)min((n + 1023) / 1024, (size_t)h->sm_count);
  launch_after(ss_sort_kernel, buckets, 1024, sizeof(SortSmem), s, nu, m, sms, base, w.k_a, w.v_a, w.k_b, w.v_b, sums);
  count_launch(4);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int sample_resolve(Handle* h, const uint64_t* vals, uint64_t* out_vals, uint8_t* out_st, size_t n, cudaStream_t s) {
  Work& w = h->w;
  const unsigned buckets = (unsigned)min((n + 1023) / 1024, kSsBuckets);
  launch_after(ss_resolve_kernel, buckets, kResThreads, 0, s, w.k_a, w.v_a, vals, (uint32_t)n, &w.counts->n_touch,
               (uint32_t)h->sm_count, sum_base(w.s_sum), reinterpret_cast<const BucketSum*>(w.s_sum), w.ukeys,
               w.uvals, w.ins_list, w.del_list, w.pend, out_vals, out_st, w.counts);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace bt
