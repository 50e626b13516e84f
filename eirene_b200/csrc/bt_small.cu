// Sorted batches of up to kSmallMax requests.
//
// A batch of a few thousand requests is bound by its launches: the general
// path (bt_front.cu, bt_sort.cu, bt_batch.cu, bt_merge.cu) takes about thirty
// kernels of 2-6 us, most of them with nothing to do for most of the chip, and
// about as many event and stream calls.  Here the same batch takes three
// kernels, in order on the caller's stream:
//
//   small_front_kernel  one thread block cluster: classification by hash, the
//                       sort of the touched requests and the segmented scan
//                       over their runs;
//   small_read_kernel   the whole chip: the plain lookups and the locates of
//                       the unique INSERT and DELETE keys (reads only);
//   small_write_kernel  one cluster (bt_merge.cu): value updates, DELETE
//                       apply, grouping of the new keys by leaf, the leaf
//                       reservation, the write-back, the leaf and inner merge.
//
// The steps inside a kernel are separated by the cluster's hardware barrier
// (no spinning, no cooperative launch).  Meaning, answers and tree are those of
// the general path.  Measured a batch on 2^22 keys, us, here / general path:
// 95/5 batches of 1024: 38 / 143, 16,384: 49 / 159, 65,536: 78 / 190; all
// INSERTs, 1024: 50 / 156, 16,384: 107 / 226, 65,536: 271 / 284.  So the line
// lies at 65,536, where a write-heavy batch begins to be worth launches over
// the whole chip (and a block's shared memory and registers are full).
#include <cuda_runtime.h>

#include "bt_block.cuh"
#include "bt_common.cuh"
#include "bt_internal.h"
#include "bt_launch.cuh"
#include "bt_search.cuh"
#include "bt_small.cuh"
#include "bt_sort.cuh"

namespace bt {

namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kResolved = 0xFFFFFFFFu;
constexpr int kItems = kSmallItems;

struct Slot {
  unsigned long long key;  // kKeyMax = empty
  uint32_t first;          // index of the key's first write
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

struct alignas(16) FrontSum {  // one block's part of the segmented scan (read in 16-byte pieces)
  uint64_t agg_v, pre_v;
  uint32_t agg_f, pre_f;
  uint32_t heads, ins, del;
  uint32_t cont;  // bit 0: a run begun in an earlier block ends here; bit 1: its key is reserved
};

static_assert(sizeof(FrontSum) % 16 == 0, "whole 16-byte pieces");

struct FrontSmem {
  uint64_t k[kSmallThreads * kItems];
  uint32_t v[kSmallThreads * kItems];
  uint64_t wsv[32];
  uint32_t wsf[32], ws[32];
  uint32_t at_touch, at_lookup;
  uint32_t split[2];
  FrontSum sum;    // this block's
  uint64_t cv;     // carry into this block, counts before it
  uint32_t cf, hb, ib, db;
};

__global__ void __launch_bounds__(kSmallThreads, 1)
    small_front_kernel(const uint64_t* keys, const uint64_t* vals, const uint8_t* ops, uint32_t n, Slot* tab,
                       uint32_t mask, SmallFront f, uint64_t* out_vals, uint8_t* out_st, DevTree t, int ensure_root) {
  extern __shared__ __align__(16) unsigned char raw[];
  FrontSmem& S = *reinterpret_cast<FrontSmem*>(raw);
  after_previous();
  const uint32_t rank = cluster_rank(), C = cluster_size();
  const uint32_t nt = C * kSmallThreads, gt = rank * kSmallThreads + threadIdx.x;
  BatchCounts* c = f.counts;
  if (gt == 0) {
    *c = BatchCounts{};
    if (ensure_root) ensure_root_leaf(t);
  }
  // the first write of every written key
  uint64_t k[kItems];
  uint32_t op[kItems], slot[kItems];
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const uint32_t i = j * nt + gt;
    k[j] = i < n ? keys[i] : kKeyMax;
    op[j] = i < n ? ops[i] : (uint32_t)kOpGet;
  }
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    slot[j] = kNone;
    if ((op[j] != kOpInsert && op[j] != kOpDelete) || k[j] == kKeyMax) continue;
    uint32_t h = (uint32_t)slot_hash(k[j]) & mask;
    for (uint32_t probe = 0; probe <= mask; probe++) {
      const unsigned long long prev = atomicCAS(&tab[h].key, (unsigned long long)kKeyMax, (unsigned long long)k[j]);
      if (prev == kKeyMax || prev == k[j]) {
        atomicMin(&tab[h].first, j * nt + gt);
        slot[j] = h;
        break;
      }
      h = (h + 1) & mask;
    }
  }
  cluster_sync();
  // touched: an invalid op code, or a write of the key at or before the request
  uint32_t touched = 0;
  ulonglong2 e[kItems];
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    if (k[j] == kKeyMax) continue;
    const uint32_t h = slot[j] != kNone ? slot[j] : (uint32_t)slot_hash(k[j]) & mask;
    e[j] = __ldcg(reinterpret_cast<const ulonglong2*>(tab + h));
  }
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const uint32_t i = j * nt + gt;
    if (i >= n) continue;
    bool f1 = op[j] > 2;
    if (!f1 && k[j] != kKeyMax) {
      ulonglong2 x = e[j];
      uint32_t h = (uint32_t)slot_hash(k[j]) & mask;
      for (uint32_t probe = 0; x.x != k[j] && x.x != kKeyMax && probe < mask; probe++) {
        h = (h + 1) & mask;
        x = __ldcg(reinterpret_cast<const ulonglong2*>(tab + h));
      }
      f1 = x.x == k[j] && i >= (uint32_t)x.y;
    }
    touched |= (f1 ? 1u : 0u) << j;
  }
  // both classes in lists, in no particular order (the sort key holds the index)
  {
    uint32_t mine = 0;
#pragma unroll
    for (int j = 0; j < kItems; j++)
      if (j * nt + gt < n) mine += (touched >> j) & 1u ? 1u : 0x10000u;
    uint32_t total;
    const uint32_t before = blk_exclusive_sum(mine, S.ws, &total);
    if (threadIdx.x == 0) {
      S.at_touch = (total & 0xffffu) ? atomicAdd(&c->n_touch, total & 0xffffu) : 0u;
      S.at_lookup = (total >> 16) ? atomicAdd(&c->n_lookup, total >> 16) : 0u;
    }
    __syncthreads();
    uint32_t pt = S.at_touch + (before & 0xffffu), pl = S.at_lookup + (before >> 16);
#pragma unroll
    for (int j = 0; j < kItems; j++) {
      const uint32_t i = j * nt + gt;
      if (i >= n) continue;
      if ((touched >> j) & 1u) {
        f.tk[pt] = k[j];
        f.tv[pt++] = pair_payload(i, op[j]);
      } else {
        f.list[pl] = i;
        f.lk[pl++] = k[j];
      }
    }
  }
  cluster_sync();
  // the table is clean again for the next batch
#pragma unroll
  for (int j = 0; j < kItems; j++)
    if (slot[j] != kNone) *reinterpret_cast<uint4*>(tab + slot[j]) = make_uint4(~0u, ~0u, ~0u, ~0u);
  const uint32_t m = __ldcg(&c->n_touch);
  if (m == 0) return;  // uniform over the cluster: no block waits for another below
  // sort: one tile per block, then merge rounds over the tiles
  uint32_t tile = 1024;
  while (tile * C < m) tile <<= 1;
  const uint32_t tiles = (m + tile - 1) / tile;
  int rounds = 0;
  while ((1u << rounds) < tiles) rounds++;
  const uint32_t o0 = rank * tile;
  const int cnt = o0 < m ? (int)min(tile, m - o0) : 0;
  for (int i = threadIdx.x; i < cnt; i += kSmallThreads) {
    S.k[i] = __ldcg(f.tk + o0 + i);
    S.v[i] = __ldcg(f.tv + o0 + i);
  }
  __syncthreads();
  if (cnt) block_sort(S.k, S.v, cnt);
  for (int r = 0; r < rounds; r++) {
    uint64_t* xk = (rounds - r) & 1 ? f.k_b : f.k_a;
    uint32_t* xv = (rounds - r) & 1 ? f.v_b : f.v_a;
    for (int i = threadIdx.x; i < cnt; i += kSmallThreads) {
      xk[o0 + i] = S.k[i];
      xv[o0 + i] = S.v[i];
    }
    cluster_sync();
    const uint32_t L = tile << r;
    const uint32_t ps = o0 / (2 * L) * (2 * L);
    const uint32_t a_end = min(ps + L, m), b_end = min(ps + 2 * L, m);
    if (cnt == 0 || b_end <= a_end) continue;  // no tile, or a run without a partner: it stays as it is
    const uint32_t na = a_end - ps, nb = b_end - a_end, d0 = o0 - ps;
    if (threadIdx.x < 64) {
      const uint32_t w = threadIdx.x >> 5;
      const uint32_t a = split_of(xk, xv, ps, na, a_end, nb, w ? d0 + cnt : d0);
      if ((threadIdx.x & 31) == 0) S.split[w] = a;
    }
    __syncthreads();
    const uint32_t a0 = S.split[0], b0 = d0 - a0;
    const int la = (int)(S.split[1] - a0), lb = cnt - la;
    for (int i = threadIdx.x; i < cnt; i += kSmallThreads) {
      const uint32_t at = i < la ? ps + a0 + i : a_end + b0 + (i - la);
      S.k[i] = __ldcg(xk + at);
      S.v[i] = __ldcg(xv + at);
    }
    __syncthreads();
    uint64_t K[4];
    uint32_t V[4];
    const int d = threadIdx.x * 4;
    if (d < cnt) merge4(S.k, S.v, la, S.k + la, S.v + la, lb, d, K, V);
    __syncthreads();
#pragma unroll
    for (int x = 0; x < 4; x++)
      if (d + x < cnt) {
        S.k[d + x] = K[x];
        S.v[d + x] = V[x];
      }
    __syncthreads();
  }
  // segmented scan over the sorted requests (the rules of merge_pass1 .. 3)
  for (int i = threadIdx.x; i < cnt; i += kSmallThreads) f.v_a[o0 + i] = S.v[i];
  uint64_t k_prev = 0, k_next = 0;
  if (tiles > 1) {  // the neighbours' edge keys
    if (threadIdx.x == 0 && cnt) {
      f.edge[2 * rank] = S.k[0];
      f.edge[2 * rank + 1] = S.k[cnt - 1];
    }
    cluster_sync();
    if (rank > 0 && cnt) k_prev = __ldcg(f.edge + 2 * (rank - 1) + 1);
    if (rank + 1 < tiles) k_next = __ldcg(f.edge + 2 * (rank + 1));
  }
  const int d = threadIdx.x * kItems;
  uint64_t kk[kItems];
  uint32_t r[kItems], o[kItems];
  uint32_t head = 0, tail = 0, valid = 0;
  Seg seg[kItems];
  Seg agg{0, 0};
  uint32_t heads = 0;
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const int i = d + j;
    if (i >= cnt) {
      seg[j] = Seg{0, 0};
      continue;
    }
    valid |= 1u << j;
    kk[j] = S.k[i];
    const uint32_t p = S.v[i];
    r[j] = pair_idx(p);
    o[j] = pair_op(p);
    const bool h = i > 0 ? S.k[i - 1] != kk[j] : (rank == 0 || k_prev != kk[j]);
    const bool tl = i + 1 < cnt ? S.k[i + 1] != kk[j] : (o0 + i + 1 == m || k_next != kk[j]);
    head |= (h ? 1u : 0u) << j;
    tail |= (tl ? 1u : 0u) << j;
    heads += h ? 1u : 0u;
    const bool wr = (o[j] == kOpInsert || o[j] == kOpDelete) && kk[j] != kKeyMax;
    seg[j].f = (h ? 1u : 0u) | (wr ? (o[j] == kOpDelete ? 6u : 2u) : 0u);
    seg[j].v = wr && o[j] == kOpInsert ? vals[r[j]] : 0;
  }
#pragma unroll
  for (int j = 0; j < kItems; j++) agg = seg_combine(agg, seg[j]);
  if (threadIdx.x == 0) S.sum.cont = 0;
  Seg all;
  const Seg st0 = blk_exclusive_seg(agg, Seg{0, 0}, S.wsf, S.wsv, &all);
  if (tiles > 1) {
    uint32_t n_ins = 0, n_del = 0;
    Seg st = st0;
#pragma unroll
    for (int j = 0; j < kItems; j++) {
      st = seg_combine(st, seg[j]);
      if (!((valid & tail) >> j & 1u)) continue;
      if (st.f & 1u) {
        if (kk[j] != kKeyMax) {
          n_del += (st.f & 4u) ? 1u : 0u;
          n_ins += (st.f & 6u) == 2u ? 1u : 0u;
        }
      } else {  // the tail of a run that began in an earlier block
        S.sum.cont = 1u | (kk[j] == kKeyMax ? 2u : 0u);
        S.sum.pre_f = st.f;
        S.sum.pre_v = st.v;
      }
    }
    uint32_t tot;
    blk_exclusive_sum(heads, S.ws, &tot);
    if (threadIdx.x == 0) S.sum.heads = tot;
    blk_exclusive_sum(n_ins | (n_del << 16), S.ws, &tot);
    if (threadIdx.x == 0) {
      S.sum.ins = tot & 0xffffu;
      S.sum.del = tot >> 16;
      S.sum.agg_f = all.f;
      S.sum.agg_v = all.v;
      reinterpret_cast<FrontSum*>(f.sums)[rank] = S.sum;
    }
    cluster_sync();
    if (threadIdx.x < 32) {  // lane x: block x's part; carries and counts before it by shuffles
      const uint32_t lane = threadIdx.x;
      FrontSum x{};
      if (lane < tiles) {
        const uint4* p = reinterpret_cast<const uint4*>(reinterpret_cast<const FrontSum*>(f.sums) + lane);
        uint4* q = reinterpret_cast<uint4*>(&x);
#pragma unroll
        for (int w = 0; w < (int)(sizeof(FrontSum) / 16); w++) q[w] = __ldcg(p + w);
      }
      Seg inc{x.agg_f, x.agg_v};
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        Seg y;
        y.f = __shfl_up_sync(0xffffffffu, inc.f, s);
        y.v = __shfl_up_sync(0xffffffffu, inc.v, s);
        if (lane >= (uint32_t)s) inc = seg_combine(y, inc);
      }
      Seg carry;
      carry.f = __shfl_up_sync(0xffffffffu, inc.f, 1);
      carry.v = __shfl_up_sync(0xffffffffu, inc.v, 1);
      if (lane == 0) carry = Seg{0, 0};
      if ((x.cont & 1u) && !(x.cont & 2u)) {
        const Seg s = seg_combine(carry, Seg{x.pre_f, x.pre_v});
        x.del += (s.f & 4u) ? 1u : 0u;
        x.ins += (s.f & 6u) == 2u ? 1u : 0u;
      }
      uint32_t h = x.heads, ic = x.ins, dc = x.del;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y0 = __shfl_up_sync(0xffffffffu, h, s), y1 = __shfl_up_sync(0xffffffffu, ic, s),
                       y2 = __shfl_up_sync(0xffffffffu, dc, s);
        if (lane >= (uint32_t)s) {
          h += y0;
          ic += y1;
          dc += y2;
        }
      }
      if (lane == rank) {
        S.cf = carry.f;
        S.cv = carry.v;
        S.hb = h - x.heads;
        S.ib = ic - x.ins;
        S.db = dc - x.del;
      }
      if (rank == 0 && lane == 31) {
        c->n_unique = h;
        c->n_ins = ic;
        c->n_del = dc;
      }
    }
  } else if (threadIdx.x == 0) {
    S.cf = 0;
    S.cv = 0;
    S.hb = S.ib = S.db = 0;
  }
  __syncthreads();
  if (cnt == 0) return;  // the block has passed every cluster barrier
  Seg st = seg_combine(Seg{S.cf, S.cv}, st0);
  uint32_t n_ins = 0, n_del = 0;
  {
    Seg s = st;
#pragma unroll
    for (int j = 0; j < kItems; j++) {
      s = seg_combine(s, seg[j]);
      if (((valid & tail) >> j & 1u) && kk[j] != kKeyMax) {
        n_del += (s.f & 4u) ? 1u : 0u;
        n_ins += (s.f & 6u) == 2u ? 1u : 0u;
      }
    }
  }
  uint32_t th, tw;
  uint32_t hpos = blk_exclusive_sum(heads, S.ws, &th) + S.hb;
  const uint32_t wpos = blk_exclusive_sum(n_ins | (n_del << 16), S.ws, &tw);
  uint32_t ipos = (wpos & 0xffffu) + S.ib, dpos = (wpos >> 16) + S.db;
  if (tiles == 1 && threadIdx.x == 0) {
    c->n_unique = th;
    c->n_ins = tw & 0xffffu;
    c->n_del = tw >> 16;
  }
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    if (!((valid >> j) & 1u)) break;
    const bool h = (head >> j) & 1u;
    if (h) hpos++;
    const uint32_t u = hpos - 1;  // unique id of this request's run
    uint32_t pend = u;
    if (kk[j] == kKeyMax || o[j] > 2u) {
      out_vals[r[j]] = 0;
      out_st[r[j]] = kRejected;
      pend = kResolved;
    } else if (!h && (st.f & 2u)) {  // an earlier write of this same run
      const bool gone = (st.f & 4u) != 0;
      out_vals[r[j]] = gone ? 0 : st.v;
      out_st[r[j]] = gone ? kAbsent : kFound;
      pend = kResolved;
    }
    f.pend[o0 + d + j] = pend;
    st = seg_combine(st, seg[j]);
    if (((tail >> j) & 1u) && kk[j] != kKeyMax) {
      f.ukeys[u] = kk[j];
      f.uvals[u] = st.v;
      if (st.f & 4u) f.del_list[dpos++] = u;
      else if (st.f & 2u) f.ins_list[ipos++] = u;
    }
  }
}

// one root-to-leaf descent of an 8-lane group: the leaf's row in k (slot 31
// as padding), the rank of the key in it, the path's node of level g in lane g
template <int G>
__device__ __forceinline__ uint32_t locate_key(const DevTree& t, uint32_t root, uint32_t root_level, uint64_t key,
                                               uint32_t g, uint32_t gmask, int use_pfx, uint64_t (&k)[32 / G],
                                               uint32_t& leaf, uint32_t& path) {
  constexpr int S = 32 / G;
  uint32_t node = root;
  const uint64_t pol = l2_keep();
  for (uint32_t level = root_level; level > 0; level--) {
    if (g == level) path = node;
    const size_t row = (size_t)node * 32 + g * S;
    uint32_t cnt = 0;
    bool full = true;
    if (use_pfx) {
      uint32_t pf[S];
      load_pfx<S>(t.pfx + row, pf, pol);
      const uint32_t x = pfx_rank<G, S>(pf, key, g, gmask);
      cnt = x & 0xffffu;
      full = (x >> 16) != 0;  // a separator shares the key's prefix
    }
    if (full) {
      load_slots<S>(t.keys + row, k);
      if (g == G - 1) k[S - 1] = kKeyMax;
      uint32_t c = 0;
#pragma unroll
      for (int i = 0; i < S; i++) c += (k[i] <= key) ? 1u : 0u;
      cnt = group_sum<G>(c, gmask);
    }
    node = (uint32_t)ldg_hint(t.vals + (size_t)node * 32 + cnt, pol);
  }
  if (g == 0) path = node;
  leaf = node;
  load_slots<S>(t.keys + (size_t)node * 32 + g * S, k);
  if (g == G - 1) k[S - 1] = kKeyMax;
  uint32_t c = 0;
#pragma unroll
  for (int i = 0; i < S; i++) c += (k[i] <= key) ? 1u : 0u;
  return group_sum<G>(c, gmask);
}

constexpr int kReadThreads = 256;
constexpr int kLocG = 8;                                  // lanes per located key
constexpr uint32_t kLocPer = kReadThreads / kLocG;        // keys per block turn
constexpr int kGetG = 4;                                  // lanes per pair of lookups (a few thousand: kWarpLookupMin)
constexpr uint32_t kGetPer = 2 * kReadThreads / kGetG;

// Blocks take turns of three kinds: 32 INSERT keys, 32 DELETE keys, or 128
// plain lookups (kGets: the learned descent's lookups have launches of their
// own).  All of them only read the tree.
template <bool kGets>
__global__ void __launch_bounds__(kReadThreads) small_read_kernel(DevTree t, SmallRead a, int use_pfx,
                                                                  uint64_t* out_vals, uint8_t* out_st) {
  after_previous();
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t n_ins = a.locate_ins ? a.counts->n_ins : 0, n_del = a.counts->n_del;
  const uint32_t n_get = kGets ? a.counts->n_lookup : 0;
  const uint32_t bi = (n_ins + kLocPer - 1) / kLocPer, bd = (n_del + kLocPer - 1) / kLocPer,
                 bg = (n_get + kGetPer - 1) / kGetPer;
  const uint32_t root = t.ctrl->root, root_level = t.ctrl->root_level;
  for (uint32_t b = blockIdx.x; b < bi + bd + bg; b += gridDim.x) {
    if (b < bi + bd) {
      const bool del = b >= bi;
      const uint32_t g = lane % kLocG, gmask = group_mask<kLocG>(lane);
      const uint32_t q = (del ? b - bi : b) * kLocPer + threadIdx.x / kLocG;
      if (q >= (del ? n_del : n_ins)) continue;
      constexpr int S = 32 / kLocG;
      const uint32_t u = del ? a.del_list[q] : a.ins_list[q];
      const uint64_t key = a.ukeys[u];
      // an INSERT needs a root and a path the record holds
      const bool usable = root != kNil && (del || root_level < (uint32_t)kLocG);
      uint32_t leaf = kNil, path = kNil, cnt = 0, slot = 0;
      bool found = false;
      if (usable) {
        uint64_t k[S];
        cnt = locate_key<kLocG>(t, root, root_level, key, g, gmask, use_pfx, k, leaf, path);
        slot = cnt ? cnt - 1 : 0;
        const uint64_t kk = __shfl_sync(gmask, pick<S>(k, slot % S), slot / S, kLocG);
        found = cnt > 0 && kk == key;
        if (!del && g > 0 && g <= root_level) a.path[g * a.path_stride + q] = path;
      }
      if (g == 0) {
        a.uans[u] = found ? t.vals[(size_t)leaf * 32 + slot] : 0;
        a.uans_st[u] = found ? kFound : (del || usable) ? kAbsent : kNoCapacity;
        if (del) {
          a.dleaf[q] = leaf;
          a.dslot[q] = found ? slot : 0xFFFFFFFFu;
        } else {
          a.vpos[q] = found ? (uint64_t)leaf * 32 + slot : ~0ull;
          a.isnew[q] = usable && !found ? 1u : 0u;
          a.mleaf[q] = leaf;
        }
      }
    } else if (kGets) {
      const uint32_t g = lane % kGetG, gmask = group_mask<kGetG>(lane);
      const uint32_t q = (b - bi - bd) * kGetPer + threadIdx.x / kGetG, q2 = q + kGetPer / 2;
      if (q >= n_get) continue;
      const bool two = q2 < n_get;
      const uint32_t ra = a.list[q], rb = two ? a.list[q2] : ra;
      const uint64_t ka = a.lk[q], kb = two ? a.lk[q2] : ka;
      uint8_t sa = kAbsent, sb = kAbsent;
      uint64_t va = 0, vb = 0;
      if (root != kNil)
        group_descend2<kGetG, false, true>(t, root, root_level, ka == kKeyMax ? 0 : ka, kb == kKeyMax ? 0 : kb, g,
                                           gmask, va, sa, vb, sb, use_pfx != 0);
      if (g == 0) {
        out_vals[ra] = ka == kKeyMax ? 0 : va;
        out_st[ra] = ka == kKeyMax ? kRejected : sa;
        if (two) {
          out_vals[rb] = kb == kKeyMax ? 0 : vb;
          out_st[rb] = kb == kKeyMax ? kRejected : sb;
        }
      }
    }
  }
}

}  // namespace

// Blocks of the cluster for n requests: one per 128, up to `most`.  A block's
// leaf merges are what costs in a write-heavy batch, and the barrier of a
// larger cluster costs little (us a batch of 2048 / 4096 all-INSERT requests
// with one block per 4096: 126 / 224, per 1024: 90 / 95, per 128: 59 / 69; a
// 95/5 batch of 4096: 52, 43, 43).
unsigned small_cluster(size_t n, unsigned most) {
  unsigned c = 1;
  while ((size_t)c * 128 < n && c < most) c <<= 1;
  return c;
}

// requests that such clusters take
size_t small_limit(unsigned most) { return (size_t)most * kSmallPer; }

// Sixteen blocks are more than every device has to offer (eight are), and how
// many fit depends on the SMs that a partition leaves each group of them.
unsigned small_largest(const void* kernel, size_t smem) {
  for (unsigned c = kSmallBlocks; c; c >>= 1) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[2];
    small_config(cfg, at, c, smem, nullptr);
    cfg.numAttrs = 1;  // the cluster alone
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) == cudaSuccess && fit > 0) return c;
    cudaGetLastError();
  }
  return 0;
}

unsigned small_blocks(int device) {
  static unsigned known[64] = {};  // one more than the answer
  if (device >= 0 && device < 64 && known[device]) return known[device] - 1;
  const unsigned front = small_largest((const void*)small_front_kernel, sizeof(FrontSmem)), write = small_write_largest();
  const unsigned most = front < write ? front : write;
  if (device >= 0 && device < 64) known[device] = most + 1;
  return most;
}

size_t small_tab_bytes(size_t cap) {
  const size_t nmax = cap < kSmallMax ? cap : kSmallMax;
  size_t slots = 1024;
  while (slots < 4 * nmax) slots <<= 1;
  return slots * sizeof(Slot);
}

size_t small_sum_bytes() { return 16 * sizeof(FrontSum) + 32 * 8; }

int small_prepare() {
  cudaError_t e = cudaFuncSetAttribute(small_front_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(FrontSmem));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(small_front_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e == cudaSuccess ? 0 : -2;
}

int small_front(Handle* h, const uint64_t* keys, const uint64_t* vals, const uint8_t* ops, uint64_t* out_vals,
                uint8_t* out_st, size_t n, bool ensure_root, cudaStream_t s) {
  Work& w = h->w;
  SmallFront f;
  f.counts = w.counts;
  f.tk = w.f_tk;
  f.tv = w.f_tv;
  f.list = w.f_list;
  f.lk = w.f_lk;
  f.k_a = w.k_a;
  f.k_b = w.k_b;
  f.v_a = w.v_a;
  f.v_b = w.v_b;
  f.ukeys = w.ukeys;
  f.uvals = w.uvals;
  f.ins_list = w.ins_list;
  f.del_list = w.del_list;
  f.pend = w.pend;
  f.sums = w.s_sums;
  f.edge = reinterpret_cast<uint64_t*>(static_cast<char*>(w.s_sums) + 16 * sizeof(FrontSum));
  uint32_t slots = 1024;
  while (slots < 4 * n) slots <<= 1;
  const unsigned C = small_cluster(n, h->small_blocks);
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[2];
  small_config(cfg, at, C, sizeof(FrontSmem), s);
  const cudaError_t e =
      cudaLaunchKernelEx(&cfg, small_front_kernel, keys, vals, ops, (uint32_t)n, reinterpret_cast<Slot*>(w.s_tab),
                         slots - 1, f, out_vals, out_st, h->tree, ensure_root ? 1 : 0);
  count_launch();
  return e == cudaSuccess ? 0 : -2;
}

int small_read(Handle* h, bool gets, bool locate_ins, uint64_t* out_vals, uint8_t* out_st, size_t n, cudaStream_t s) {
  Work& w = h->w;
  SmallRead a;
  a.counts = w.counts;
  a.list = w.f_list;
  a.lk = w.f_lk;
  a.ukeys = w.ukeys;
  a.ins_list = w.ins_list;
  a.del_list = w.del_list;
  a.path = w.m_path;
  a.path_stride = w.cap;
  a.mleaf = w.m_leaf;
  a.isnew = w.m_isnew;
  a.vpos = w.m_vpos;
  a.dleaf = w.d_leaf;
  a.dslot = w.d_slot;
  a.uans = w.uans;
  a.uans_st = w.uans_st;
  a.locate_ins = locate_ins ? 1 : 0;
  const int use_pfx = h->use_pfx ? 1 : 0;
  const size_t turns = (n + kLocPer - 1) / kLocPer + 2;
  const unsigned grid = (unsigned)min(turns, (size_t)h->sm_count * 8);
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kReadThreads);
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const cudaError_t e =
      gets ? cudaLaunchKernelEx(&cfg, small_read_kernel<true>, h->tree, a, use_pfx, out_vals, out_st)
           : cudaLaunchKernelEx(&cfg, small_read_kernel<false>, h->tree, a, use_pfx, out_vals, out_st);
  count_launch();
  return e == cudaSuccess ? 0 : -2;
}

}  // namespace bt
