// Segmented leaf merge: the deterministic insert engine of the sorted batch
// (BT_MODE_SORTED | BT_MODE_MERGE_ENGINE).  No counterpart in the reference,
// which inserts one key per warp under STM (src/gpu-stm-tree-v39/
// bpt-gpustm-kernel.cu:14-256); the batch meaning is still v38's.
//
// With the batch's unique INSERT keys in ascending order:
//   locate    a warp descends with 32 keys at a time (warp_descend), records each
//             one's root-to-leaf path, finds it by the leaf's fingerprints,
//             answers the previous value and records where it lies;
//   update    writes the new values of the existing keys in place;
//   group     the new keys, packed, and runs of new keys sharing a leaf (segments);
//   reserve   the new leaves of the segments that split, all or none;
//   leaf      one 8-lane group per touched leaf merges its new keys by rank scatter
//             (each element computes its merged position by binary search in
//             the other sequence); an overflowing leaf becomes
//             p = ceil(m / leaf_fill) leaves of even size, one group per piece;
//             the first keys of pieces 1..p-1 become separator entries for the
//             parent;
//   inner     a cooperative grid applies the entries level by level the same way
//             (children spread evenly over q = ceil((s+1)/(inner_fill+1))
//             nodes, the key between two pieces moves up) and rebuilds an
//             overflowing root with the bulk-load rule.
// Locate only reads the tree, so it may run beside the batch's plain
// lookups (the hash front end does so, and the grouping, which reads no tree);
// the in-place value update, reserve, leaf and inner run after them and alone, so
// no locks are taken.  The rules are
// restated by the CPU oracle (bto_execute_merged with BTO_ENGINE_MERGE) and
// the resulting leaf layout is compared exactly.
#include <cuda_runtime.h>

#include "bt_block.cuh"
#include "bt_common.cuh"
#include "bt_delete.cuh"
#include "bt_internal.h"
#include "bt_launch.cuh"
#include "bt_lookback.cuh"
#include "bt_rows.cuh"
#include "bt_search.cuh"
#include "bt_small.cuh"
#include "bt_sort.cuh"

namespace bt {

struct MergeEntry {
  uint64_t key;
  uint32_t child;
  uint32_t rep;  // index of a new key whose path passes through this piece's parent
};

struct MergeCounts {
  uint32_t n_new;
  uint32_t n_segs;
  uint32_t n_leaf_entries;
  uint32_t node_base;
  uint32_t cap_fail;
  uint32_t root_level;  // of the tree before the inner merge
  uint32_t pad[2];
};

namespace {

constexpr int kPathLevels = 8;
constexpr uint64_t kNoPos = ~0ull;  // locate_kernel: no value to update in place
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ uint32_t ceil_div(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

// piece index and slot of merged position `pos` when m items are spread over p
// pieces (the first m % p pieces hold one more)
__device__ __forceinline__ void piece_of(uint32_t pos, uint32_t m, uint32_t p, uint32_t& c, uint32_t& slot) {
  const uint32_t b = m / p, rem = m % p;
  const uint32_t big = rem * (b + 1);
  if (pos < big) {
    c = pos / (b + 1);
    slot = pos % (b + 1);
  } else {
    const uint32_t q = pos - big;
    c = rem + q / b;
    slot = q % b;
  }
}
__device__ __forceinline__ uint32_t piece_size(uint32_t c, uint32_t m, uint32_t p) {
  return m / p + (c < m % p ? 1u : 0u);
}
__device__ __forceinline__ uint32_t piece_start(uint32_t c, uint32_t m, uint32_t p) {
  const uint32_t b = m / p, rem = m % p;
  return c * b + (c < rem ? c : rem);
}

// number of a[0..n) strictly below key (a ascending)
__device__ __forceinline__ uint32_t count_less(const uint64_t* a, uint32_t n, uint64_t key) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// the same over the n keys of group grp's shared row (row_at)
__device__ __forceinline__ uint32_t count_less_row(const uint64_t* row, uint32_t grp, uint32_t n, uint64_t key) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (row[row_at(mid, grp)] < key) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// ------------------------------------------------------------- root ----
__global__ void merge_ensure_root_kernel(DevTree t) { ensure_root_leaf(t); }

// ------------------------------------------------------------- locate ----
// The batch's unique INSERT and DELETE keys in the pre-batch tree, 32 to a warp
// (warp_descend): the leaf, the slot of a key that is there (by the leaf's
// fingerprints) and its value, and for an INSERT key the inner nodes of its path.
// Reads only.  A run of keys per 8-lane group with path reuse and whole rows took
// 80 us for 2^19 INSERT keys on 2^24 keys and 140 for as many DELETE keys with a
// descent each; this takes 40 for either.
struct LocateArgs {
  const BatchCounts* counts;
  const uint64_t* ukeys;
  const uint32_t *ins_list, *del_list;
  uint32_t *path, *mleaf, *isnew;
  uint64_t* vpos;
  uint32_t *dleaf, *dslot;
  uint64_t* uans;
  uint8_t* uans_st;
  size_t path_stride;
};

__global__ void __launch_bounds__(256) locate_kernel(DevTree t, LocateArgs a, int what) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t n_ins = (what & kLocateIns) ? a.counts->n_ins : 0, n_del = (what & kLocateDel) ? a.counts->n_del : 0;
  const uint32_t ti = ceil_div(n_ins, 32), td = ceil_div(n_del, 32);
  const uint32_t root = t.ctrl->root, root_level = t.ctrl->root_level;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < ti + td; w += warps) {
    const bool del = w >= ti;
    const uint32_t q = (del ? w - ti : w) * 32 + lane;
    const bool live = q < (del ? n_del : n_ins);
    const uint32_t u = live ? (del ? a.del_list : a.ins_list)[q] : 0;
    const uint64_t key = live ? a.ukeys[u] : 0;
    // no root (pool exhausted), or a tree too tall for the path record
    const bool usable = root != kNil && (del || root_level < (uint32_t)kPathLevels);
    uint32_t leaf = kNil, slot = kNoSlot;
    uint64_t val = 0;
    if (usable) {
      leaf = warp_descend(t, root, root_level, key, [&](uint32_t level, uint32_t node) {
        if (live && !del) a.path[level * a.path_stride + q] = node;
      });
      uint64_t row[4];
      ldg32_hint(t.fp + (size_t)leaf * 32, row, l2_keep());
      if (live) leaf_pick(t, leaf, key, fp_match(row, key_fp(key)), l2_stream(), val, slot);
    }
    if (!live) continue;
    const bool found = slot != kNoSlot;
    a.uans[u] = val;
    a.uans_st[u] = found ? kFound : (del || usable) ? kAbsent : kNoCapacity;
    if (del) {
      a.dleaf[q] = leaf;
      a.dslot[q] = slot;
    } else {
      // an existing key's new value goes in later (merge_update_kernel): a plain
      // lookup of it that comes before its first write must still see the old one
      a.vpos[q] = found ? (uint64_t)leaf * 32 + slot : kNoPos;
      a.isnew[q] = usable && !found ? 1u : 0u;
      a.mleaf[q] = leaf;
    }
  }
}

// new values of the keys the batch finds in the tree, in place (keys do not
// move); after the batch's plain lookups, before its DELETE apply
__global__ void merge_update_kernel(DevTree t, const uint64_t* uvals, const uint32_t* ins_list, const uint32_t* n_dev,
                                    const uint64_t* vpos) {
  after_previous();
  const size_t n = *n_dev;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += stride) {
    const uint64_t p = vpos[q];
    if (p != kNoPos) t.vals[p] = uvals[ins_list[q]];
  }
}

// ------------------------------------------------------------- compact ----
// The new keys, packed, and the segments: runs of new keys that share a leaf.
// One launch over tiles of the INSERT keys (the look-back of bt_lookback.cuh
// gives a tile its places): a new key begins a segment when no new key before
// it has its leaf, which the flags and leaves just before it tell (at most 31
// keys of a leaf are in the tree already), so new keys and segments are counted
// in one pass.  It was five launches (scan, compact, flags, scan, starts).
constexpr int kGroupThreads = 1024;
constexpr uint32_t kGroupTile = 2 * kGroupThreads;

__global__ void __launch_bounds__(kGroupThreads)
    merge_group_kernel(MergeCounts* mc, const uint32_t* ins_list, const uint32_t* n_dev, const uint32_t* isnew,
                       const uint64_t* ukeys, const uint64_t* uvals, const uint32_t* mleaf, uint64_t* newk,
                       uint64_t* newv, uint32_t* nq, uint32_t* nleaf, uint32_t* seg_start, uint32_t* seg_leaf,
                       uint64_t* status, uint64_t* status_seg, uint64_t* ctr, uint32_t* err) {
  after_previous();
  __shared__ uint32_t ws[32];
  __shared__ uint32_t s_pre[2];
  __shared__ uint64_t s_ticket;
  uint32_t epoch;
  const uint32_t n = *n_dev, n_tiles = ceil_div(n, kGroupTile);
  for (;;) {
    if (threadIdx.x == 0) s_ticket = take_tile(ctr);
    __syncthreads();
    const uint32_t tile = (uint32_t)s_ticket;
    epoch = tile_epoch(s_ticket);
    __syncthreads();
    if (tile >= n_tiles) {
      if (tile == 0 && threadIdx.x == 0) mc->n_new = mc->n_segs = 0;  // no INSERT
      break;
    }
    const uint32_t q = tile * kGroupTile + 2 * threadIdx.x;
    uint2 is = make_uint2(0, 0), lf = make_uint2(kNil, kNil);
    if (q + 1 < n) {
      is = *reinterpret_cast<const uint2*>(isnew + q);
      lf = *reinterpret_cast<const uint2*>(mleaf + q);
    } else if (q < n) {
      is.x = isnew[q];
      lf.x = mleaf[q];
    }
    uint64_t k[2] = {0, 0}, v[2] = {0, 0};
#pragma unroll
    for (int j = 0; j < 2; j++)
      if (j ? is.y : is.x) {
        const uint32_t u = ins_list[q + j];
        k[j] = ukeys[u];
        v[j] = uvals[u];
      }
    uint32_t head_x = is.x, head_y = is.y;
    if (head_y && is.x && lf.x == lf.y) head_y = 0;
    if (head_x || (head_y && lf.x == lf.y)) {
      bool seen = false;
      for (uint32_t p = q; p > 0 && !seen && mleaf[p - 1] == lf.x; p--) seen = isnew[p - 1] != 0;
      if (seen) {
        head_x = 0;
        if (lf.x == lf.y) head_y = 0;
      }
    }
    // both counts in one sum: at most 2048 of each a tile
    const uint32_t mine = is.x + is.y + ((head_x + head_y) << 16);
    uint32_t tot;
    const uint32_t ex = blk_exclusive_sum(mine, ws, &tot);
    if (threadIdx.x < 64) {
      const bool seg = threadIdx.x >= 32;
      const uint32_t sum = seg ? tot >> 16 : tot & 0xffffu;
      const uint32_t pre = look_back(seg ? status_seg : status, tile, sum, epoch, err);
      if ((threadIdx.x & 31) == 0) {
        s_pre[seg] = pre;
        if (tile == n_tiles - 1) (seg ? mc->n_segs : mc->n_new) = pre + sum;
      }
    }
    __syncthreads();
    uint32_t p = s_pre[0] + (ex & 0xffffu), sg = s_pre[1] + (ex >> 16);
#pragma unroll
    for (int j = 0; j < 2; j++) {
      if (!(j ? is.y : is.x)) continue;
      const uint32_t leaf = j ? lf.y : lf.x;
      newk[p] = k[j];
      newv[p] = v[j];
      nq[p] = q + j;
      nleaf[p] = leaf;
      if (j ? head_y : head_x) {
        seg_start[sg] = p;
        seg_leaf[sg] = leaf;
        sg++;
      }
      p++;
    }
  }
  if (threadIdx.x == 0) tiles_done(ctr, epoch);
}

__device__ __forceinline__ void seg_bounds(const MergeCounts* mc, const uint32_t* seg_start, uint32_t s,
                                           uint32_t& a, uint32_t& b) {
  a = seg_start[s];
  b = (s + 1 < mc->n_segs) ? seg_start[s + 1] : mc->n_new;
}

// reserve the leaf pieces (and headroom for the inner levels) in one step;
// all-or-nothing: on failure no leaf is touched and the new keys report
// kNoCapacity.  entry_cap bounds the separator-entry buffers.
__device__ __forceinline__ void reserve_pieces(const DevTree& t, MergeCounts* mc, uint32_t entry_cap) {
  const uint32_t T = mc->n_leaf_entries;
  // the inner merge's blocks take the level from here: the block that rebuilds
  // the root changes Ctrl::root_level while others may not have read it yet
  mc->root_level = t.ctrl->root_level;
  const uint32_t need = T + T / 4 + 64;
  const uint32_t have = atomicAdd(&t.ctrl->n_nodes, 0u);
  if ((uint64_t)have + need > t.cap || T > entry_cap) {
    mc->cap_fail = 1;
    atomicOr(&t.ctrl->error, kErrCapacity);
    return;
  }
  mc->cap_fail = 0;
  mc->node_base = atomicAdd(&t.ctrl->n_nodes, T);
}

// New leaves per segment (pieces - 1), their places, and the reservation: one
// launch over tiles of the segments; the last tile's block knows the total.  It
// was three launches (count, scan, reserve).
__global__ void __launch_bounds__(kGroupThreads)
    merge_reserve_kernel(DevTree t, uint32_t leaf_fill, uint32_t entry_cap, MergeCounts* mc, const uint32_t* seg_start,
                         const uint32_t* seg_leaf, uint32_t* extra, uint32_t* eoff, uint64_t* status, uint64_t* ctr,
                         uint32_t* err) {
  after_previous();
  __shared__ uint32_t ws[32];
  __shared__ uint32_t s_pre;
  __shared__ uint64_t s_ticket;
  uint32_t epoch;
  const uint32_t n = mc->n_segs, n_tiles = ceil_div(n, (uint32_t)kGroupThreads);
  for (;;) {
    if (threadIdx.x == 0) s_ticket = take_tile(ctr);
    __syncthreads();
    const uint32_t tile = (uint32_t)s_ticket;
    epoch = tile_epoch(s_ticket);
    __syncthreads();
    if (tile >= n_tiles) {
      if (tile == 0 && threadIdx.x == 0) {
        mc->n_leaf_entries = 0;
        reserve_pieces(t, mc, entry_cap);
      }
      break;
    }
    const uint32_t i = tile * kGroupThreads + threadIdx.x;
    uint32_t e = 0;
    if (i < n) {
      uint32_t a, b;
      seg_bounds(mc, seg_start, i, a, b);
      const uint32_t m = hdr_size(t.keys[(size_t)seg_leaf[i] * 32 + 31]) + (b - a);
      e = m <= (uint32_t)kMaxKeys ? 0u : ceil_div(m, leaf_fill) - 1;
    }
    uint32_t tot;
    const uint32_t ex = blk_exclusive_sum(e, ws, &tot);
    if (threadIdx.x < 32) {
      const uint32_t pre = look_back(status, tile, tot, epoch, err);
      if (threadIdx.x == 0) {
        s_pre = pre;
        if (tile == n_tiles - 1) {
          mc->n_leaf_entries = pre + tot;
          reserve_pieces(t, mc, entry_cap);
        }
      }
    }
    __syncthreads();
    if (i < n) {
      extra[i] = e;
      eoff[i] = s_pre + ex;
    }
  }
  if (threadIdx.x == 0) tiles_done(ctr, epoch);
}

// a batch whose pieces did not fit answers kNoCapacity for all its new keys
__global__ void merge_fail_mark_kernel(const MergeCounts* mc, const uint32_t* nq, const uint32_t* ins_list,
                                       uint8_t* uans_st) {
  after_previous();
  if (mc->cap_fail == 0) return;
  const uint32_t n_new = mc->n_new;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_new; i += stride)
    uans_st[ins_list[nq[i]]] = kNoCapacity;
}

// ------------------------------------------------------------- leaf ----
// A touched leaf of sz keys that gets cnt new ones becomes p pieces of even
// size (p = 1 while they fit one leaf).  Piece c holds the merged positions
// [st, st + kc); a group of G lanes builds it whole: every old key's merged
// position by a binary search in the new keys, every new key of the range by
// one in the old row, the row put together in shared memory and written with
// 32-byte stores.  A piece needs nothing of its neighbours: its right fence is
// the key at merged position st + kc.
template <int N>  // groups of the block
struct LeafSmem {
  uint64_t old[N][32];
  __align__(16) uint64_t mk[N][32];
  __align__(16) uint64_t mv[N][32];
};

template <int G, int N>
__device__ __forceinline__ uint64_t leaf_piece(const DevTree& t, LeafSmem<N>& sm, uint32_t grp, uint32_t g,
                                               uint32_t gmask, uint32_t nd, uint32_t c, uint32_t p, uint32_t m,
                                               uint32_t sz, uint64_t hdr, uint64_t fence,
                                               const uint64_t (&ok)[32 / G], const uint64_t (&ov)[32 / G],
                                               const uint64_t* nk, const uint64_t* nv,
                                               uint32_t cnt) {
  constexpr int S = 32 / G;
  const uint32_t st = piece_start(c, m, p), kc = piece_size(c, m, p), end = st + kc;
  uint64_t* mk = sm.mk[grp];
  uint64_t* mv = sm.mv[grp];
  const uint64_t* old = sm.old[grp];
  // old keys of the piece to their slots; how many of them precede its two ends
  uint32_t before = 0;  // old keys at merged positions below st, and (high half) below end
  uint64_t right = 0;   // the key at position end when it is an old one
  bool right_old = false;
#pragma unroll
  for (int i = 0; i < S; i++) {
    const uint32_t slot = g * S + i;
    if (slot < sz) {
      const uint32_t pos = slot + count_less(nk, cnt, ok[i]);
      before += (pos < st ? 1u : 0u) + (pos < end ? 0x10000u : 0u);
      if (pos >= st && pos < end) {
        mk[row_at(pos - st, grp)] = ok[i];
        mv[row_at(pos - st, grp)] = ov[i];
      } else if (pos == end) {
        right = ok[i];
        right_old = true;
      }
    }
  }
  before = group_sum<G>(before, gmask);
  const uint32_t j0 = st - (before & 0xffffu), j1 = end - (before >> 16);
  for (uint32_t j = j0 + g; j < j1; j += G) {
    const uint64_t key = nk[j];
    const uint32_t pos = j + count_less_row(old, grp, sz, key);
    mk[row_at(pos - st, grp)] = key;
    mv[row_at(pos - st, grp)] = nv[j];
  }
  uint64_t rf = fence;
  if (c + 1 < p) {  // the next piece's first key: an old one, or the next new one
    const uint32_t who = __ballot_sync(gmask, right_old) & gmask;
    if (who) rf = __shfl_sync(gmask, right, __ffs(who) - 1);
    else rf = nk[j1];
  }
  __syncwarp(gmask);
  uint64_t wk[S], wv[S];
#pragma unroll
  for (int i = 0; i < S; i++) {
    const uint32_t slot = g * S + i;
    wk[i] = slot < kc ? mk[row_at(slot, grp)] : kKeyMax;
    wv[i] = slot < kc ? mv[row_at(slot, grp)] : 0;
  }
  const uint64_t first = mk[row_at(0, grp)];
  static_assert(G == 8, "four slots per lane");
  int splits = 0;
  if (c == 0 && g == G - 1) {
    splits = t.fp[(size_t)nd * 32 + 31];
    splits = splits < (int)kSplitMany ? splits + 1 : splits;
  }
  store_fp4(t, nd, g, wk, splits);
  if (g == G - 1) {
    wk[S - 1] = make_hdr(kc, 0, c == 0 ? hdr_version(hdr) + 1 : 0, hdr_epoch(hdr));
    wv[S - 1] = rf;
  }
  store_row(t.keys + (size_t)nd * 32 + g * S, wk);
  store_row(t.vals + (size_t)nd * 32 + g * S, wv);
  __syncwarp(gmask);  // the shared rows are reused by the group's next piece
  return first;
}

// a touched leaf's row in registers
template <int G>
__device__ __forceinline__ void leaf_row(const DevTree& t, uint32_t g, uint32_t gmask, uint32_t leaf,
                                         uint64_t (&ok)[32 / G], uint64_t (&ov)[32 / G], uint64_t& hdr,
                                         uint64_t& fence) {
  constexpr int S = 32 / G;
  load_row(t.keys + (size_t)leaf * 32 + g * S, ok);
  load_row(t.vals + (size_t)leaf * 32 + g * S, ov);
  hdr = __shfl_sync(gmask, ok[S - 1], G - 1, G);
  fence = __shfl_sync(gmask, ov[S - 1], G - 1, G);
}

// its keys in shared memory, for searches
template <int G, int N>
__device__ __forceinline__ void leaf_keys(LeafSmem<N>& sm, uint32_t grp, uint32_t g, uint32_t gmask, uint32_t sz,
                                          const uint64_t (&ok)[32 / G]) {
  constexpr int S = 32 / G;
#pragma unroll
  for (int i = 0; i < S; i++) {
    const uint32_t slot = g * S + i;
    sm.old[grp][row_at(slot, grp)] = slot < sz ? ok[i] : kKeyMax;
  }
  __syncwarp(gmask);
}

// Leaf merge: a strided loop of the n_groups groups of G lanes over two kinds of items.
//   segments  a touched leaf whose merged row fits: rewritten in place by its
//             group.  Several leaves per warp keep more row loads in flight
//             than a warp per leaf (the kernel is bound by the dependent chain
//             segment bounds -> leaf id -> row, and by L1: 63 % of its rate with
//             16-byte accesses, conflicting shared rows and a binary search per
//             key).  Most leaves get one to three keys: these are ranked in
//             registers.  With del_apply_kernel's rows the same way, two batches
//             of 2^20 at 50 % writes 863 -> 836 us, four of 2^22 at 5 % 2084 ->
//             2014.
//   entries   one new piece (1 .. p - 1) of a leaf that splits; its segment by a
//             binary search in the entry offsets.  All pieces read the old row,
//             and the group that finishes the leaf's last one (a count down of
//             `extra`, no group waits) writes piece 0 in its place.
// With all the pieces of a leaf in the hands of the leaf's one group, a batch
// that puts 1.3 million keys into a tree of one leaf ran for 75 ms; spread over
// the chip, a tree of 2^23 keys grown by seven such batches takes 6.5 ms, from
// 81.2.  A launch of its own for the pieces cost batches that split nothing 4 %
// (a 50/50 batch of 2^20), and so did 74 registers (three blocks an SM).
template <int G, int N>
__device__ __forceinline__ void leaf_merge(const DevTree& t, uint32_t leaf_fill, const MergeCounts* mc,
                                           const uint32_t* seg_start, const uint32_t* eoff, uint32_t* extra,
                                           const uint64_t* newk, const uint64_t* newv, const uint32_t* nq,
                                           const uint32_t* seg_leaf, MergeEntry* ent, LeafSmem<N>& sm, uint32_t gid,
                                           uint32_t n_groups) {
  constexpr int S = 32 / G;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t g = lane % G;
  const uint32_t grp = threadIdx.x / G;
  const uint32_t gmask = group_mask<G>(lane);
  const uint32_t n_segs = mc->n_segs, n_ent = mc->n_leaf_entries;
  const uint32_t base = mc->node_base;
  unsigned long long added = 0, splits = 0;
  for (uint32_t s = gid; s < n_segs; s += n_groups) {
    uint32_t a, b;
    seg_bounds(mc, seg_start, s, a, b);
    const uint32_t leaf = seg_leaf[s];
    const uint32_t cnt = b - a;
    if (s + n_groups < n_segs) prefetch_row(t, seg_leaf[s + n_groups], g);
    if (g == 0) added += cnt;
    // a leaf that splits (it has entries) is written by their groups
    if (eoff[s] != (s + 1 < n_segs ? eoff[s + 1] : n_ent)) continue;
    uint64_t ok[S], ov[S], hdr, fence;
    leaf_row<G>(t, g, gmask, leaf, ok, ov, hdr, fence);
    const uint32_t sz = hdr_size(hdr), m = sz + cnt;
    if (cnt <= 3) {  // every old key against every new one in registers, the new ones' ranks by one sum
      const uint64_t n0 = newk[a], n1 = cnt > 1 ? newk[a + 1] : kKeyMax, n2 = cnt > 2 ? newk[a + 2] : kKeyMax;
      uint32_t less = 0;  // old keys below n0, n1, n2: a byte each
#pragma unroll
      for (int i = 0; i < S; i++) {
        const uint32_t slot = g * S + i;
        if (slot < sz) {
          const uint32_t b = (n0 < ok[i] ? 1u : 0u) + (n1 < ok[i] ? 0x100u : 0u) + (n2 < ok[i] ? 0x10000u : 0u);
          less += 0x10101u - b;
          const uint32_t at = row_at(slot + (b & 1u) + (b >> 8 & 1u) + (b >> 16), grp);
          sm.mk[grp][at] = ok[i];
          sm.mv[grp][at] = ov[i];
        }
      }
      less = group_sum<G>(less, gmask);
      if (g < cnt) {
        const uint32_t at = row_at(g + (less >> (8 * g) & 0xffu), grp);
        sm.mk[grp][at] = g == 0 ? n0 : g == 1 ? n1 : n2;
        sm.mv[grp][at] = newv[a + g];
      }
    } else {
      leaf_keys<G, N>(sm, grp, g, gmask, sz, ok);
#pragma unroll
      for (int i = 0; i < S; i++) {
        const uint32_t slot = g * S + i;
        if (slot < sz) {
          const uint32_t at = row_at(slot + count_less(newk + a, cnt, ok[i]), grp);
          sm.mk[grp][at] = ok[i];
          sm.mv[grp][at] = ov[i];
        }
      }
      for (uint32_t j = g; j < cnt; j += G) {
        const uint64_t key = newk[a + j];
        const uint32_t at = row_at(j + count_less_row(sm.old[grp], grp, sz, key), grp);
        sm.mk[grp][at] = key;
        sm.mv[grp][at] = newv[a + j];
      }
    }
    __syncwarp(gmask);
    uint64_t wk[S], wv[S];
#pragma unroll
    for (int i = 0; i < S; i++) {
      const uint32_t slot = g * S + i;
      wk[i] = slot < m ? sm.mk[grp][row_at(slot, grp)] : kKeyMax;
      wv[i] = slot < m ? sm.mv[grp][row_at(slot, grp)] : 0;
    }
    store_fp4(t, leaf, g, wk, -1);
    if (g == G - 1) {
      wk[S - 1] = make_hdr(m, 0, hdr_version(hdr) + 1, hdr_epoch(hdr));
      wv[S - 1] = fence;
    }
    store_row(t.keys + (size_t)leaf * 32 + g * S, wk);
    store_row(t.vals + (size_t)leaf * 32 + g * S, wv);
    __syncwarp(gmask);  // the shared rows are reused by the next segment
  }
  for (uint32_t e = gid; e < n_ent; e += n_groups) {
    // the last segment whose entries begin at or before e
    uint32_t lo = 0, hi = n_segs;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (eoff[mid] <= e) lo = mid;
      else hi = mid;
    }
    uint32_t a, b;
    seg_bounds(mc, seg_start, lo, a, b);
    const uint32_t cnt = b - a, leaf = seg_leaf[lo];
    uint64_t ok[S], ov[S], hdr, fence;
    leaf_row<G>(t, g, gmask, leaf, ok, ov, hdr, fence);
    const uint32_t sz = hdr_size(hdr), m = sz + cnt, p = ceil_div(m, leaf_fill);
    leaf_keys<G, N>(sm, grp, g, gmask, sz, ok);
    uint32_t c = e - eoff[lo] + 1, nd = base + e;
    for (;;) {
      const uint64_t first = leaf_piece<G, N>(t, sm, grp, g, gmask, nd, c, p, m, sz, hdr, fence, ok, ov, newk + a,
                                           newv + a, cnt);
      if (c == 0) break;
      uint32_t left = 0;
      if (g == 0) {
        t.low[nd] = first;
        MergeEntry x;
        x.key = first;
        x.child = nd;
        x.rep = nq[a];
        ent[e] = x;
        splits++;
        __threadfence();  // the old row was read before the count says so
        left = atomicSub(extra + lo, 1u);
      }
      if (__shfl_sync(gmask, left, 0, G) != 1u) break;
      c = 0;  // the leaf's other pieces are done: piece 0 takes the leaf's row
      nd = leaf;
    }
  }
  if (g == 0 && (added | splits)) {
    atomicAdd(&t.ctrl->n_keys, added);
    atomicAdd(&t.ctrl->leaf_splits, splits);
  }
}

template <int G>
__global__ void __launch_bounds__(256, 4) merge_leaf_kernel(DevTree t, uint32_t leaf_fill, const MergeCounts* mc,
                                                            const uint32_t* __restrict__ seg_start,
                                                            const uint32_t* __restrict__ eoff,
                                                            uint32_t* __restrict__ extra,
                                                            const uint64_t* __restrict__ newk,
                                                            const uint64_t* __restrict__ newv,
                                                            const uint32_t* __restrict__ nq,
                                                            const uint32_t* __restrict__ seg_leaf,
                                                            MergeEntry* __restrict__ ent) {
  __shared__ LeafSmem<256 / G> sm;
  if (mc->cap_fail) return;  // merge_fail_mark_kernel answered the new keys
  leaf_merge<G, 256 / G>(t, leaf_fill, mc, seg_start, eoff, extra, newk, newv, nq, seg_leaf, ent, sm,
                               (blockIdx.x * blockDim.x + threadIdx.x) / G, (gridDim.x * blockDim.x) / G);
}

// ------------------------------------------------------------- inner ----
// The separator entries are applied level by level by one cooperative grid
// (all blocks resident), with a grid barrier between the steps of a level.
// Entries are in ascending key order; those of one parent are contiguous.
// The barrier's wait is bounded: past kBarrierSpin it sets kErrSpin and every
// block leaves.
constexpr int kInnerThreads = 512;
constexpr uint32_t kBarrierSpin = 1u << 24;

struct InnerSync {
  unsigned count;
  unsigned gen;
  uint32_t fail;
  uint32_t n_groups;
  uint32_t total;  // 1 when the capacity check failed
  uint32_t base;
  uint32_t pad[2];
  uint32_t partial[1024];  // per block
};

__device__ bool grid_sync(InnerSync* gs, uint32_t* err) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned g = ld_acquire32(&gs->gen);
    __threadfence();
    if (atomicAdd(&gs->count, 1u) == gridDim.x - 1) {
      gs->count = 0;
      __threadfence();
      atomicAdd(&gs->gen, 1u);
    } else {
      uint32_t spins = 0;
      while (ld_acquire32(&gs->gen) == g) {
        if (++spins > kBarrierSpin) {
          atomicOr(err, kErrSpin);
          atomicExch(&gs->fail, 1u);
          ok = 0;
          break;
        }
        if (spins > 32) __nanosleep(128);
      }
    }
    __threadfence();
    if (ld_acquire32(&gs->fail)) ok = 0;
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// The blocks that apply the entries: the cooperative grid, or the cluster of a
// small batch (whose hardware barrier cannot fail).
struct GridTeam {
  static constexpr uint32_t kMost = 1024;
  InnerSync* gs;
  uint32_t* err;
  __device__ uint32_t rank() const { return blockIdx.x; }
  __device__ uint32_t size() const { return gridDim.x; }
  __device__ bool sync() const { return grid_sync(gs, err); }
};
struct ClusterTeam {
  static constexpr uint32_t kMost = kSmallBlocks;
  __device__ uint32_t rank() const { return cluster_rank(); }
  __device__ uint32_t size() const { return cluster_size(); }
  __device__ bool sync() const {
    cluster_sync();
    return true;
  }
};

// exclusive scan over the team of f(i), i < n: out[i] and the total.  Each block
// takes one contiguous chunk.  Contains two barriers.
template <int NT, typename Team, typename F>
__device__ bool team_scan(const Team& team, uint32_t n, F f, uint32_t* out, InnerSync* gs, uint32_t* ws,
                          uint32_t* total) {
  const uint32_t chunk = ceil_div(n, team.size());
  const uint32_t c0 = min(n, team.rank() * chunk), c1 = min(n, c0 + chunk);
  uint32_t sum = 0;
  for (uint32_t base = c0; base < c1; base += NT) {
    const uint32_t i = base + threadIdx.x;
    uint32_t tot;
    blk_exclusive_sum(i < c1 ? f(i) : 0u, ws, &tot);
    sum += tot;
  }
  if (threadIdx.x == 0) gs->partial[team.rank()] = sum;
  if (!team.sync()) return false;
  // this block's offset: sum of the lower blocks' partials
  uint32_t off = 0, all = 0;
  for (uint32_t b = threadIdx.x; b < team.size(); b += NT) {
    const uint32_t v = gs->partial[b];
    all += v;
    if (b < team.rank()) off += v;
  }
  uint32_t t0, t1;
  blk_exclusive_sum(off, ws, &t0);
  blk_exclusive_sum(all, ws, &t1);
  uint32_t carry = t0;
  for (uint32_t base = c0; base < c1; base += NT) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < c1 ? f(i) : 0u;
    uint32_t tot;
    const uint32_t ex = blk_exclusive_sum(v, ws, &tot);
    if (i < c1) out[i] = carry + ex;
    carry += tot;
  }
  *total = t1;
  return team.sync();  // out[] complete before anyone reads it
}

template <int NT>
struct InnerSmem {
  uint32_t ws[32];
  uint32_t base;
  uint64_t keys[NT / 32][32];
};

template <int NT, typename Team>
__device__ __forceinline__ void inner_merge(const DevTree& t, uint32_t inner_fill, uint32_t entry_cap,
                                            MergeCounts* mc, InnerSync* gs, MergeEntry* ea, MergeEntry* eb,
                                            const uint32_t* path, size_t path_stride, uint32_t* gstart, uint32_t* goff, uint32_t* kids_a,
                                            uint32_t* kids_b, const Team& team, InnerSmem<NT>& sm) {
  constexpr int NW = NT / 32;
  Ctrl* C = t.ctrl;
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t gw = team.rank() * NW + w, n_warps = team.size() * NW;
  const uint32_t epoch = C->epoch;
  uint32_t n_e = mc->n_leaf_entries;
  MergeEntry* cur = ea;
  MergeEntry* nxt = eb;
  unsigned long long inner_new = 0, roots_new = 0;
  const uint32_t root_level = mc->root_level;
  for (uint32_t lvl = 1; n_e > 0; lvl++) {
    if (lvl > root_level) {
      // the root split: block 0 rebuilds upward from [root, pieces...] with the bulk rule
      if (team.rank() != 0) break;
      uint32_t cnt = n_e + 1;
      if ((uint64_t)C->n_nodes + cnt > t.cap) {
        if (threadIdx.x == 0) atomicOr(&C->error, kErrCapacity);
        return;
      }
      for (uint32_t i = threadIdx.x; i < cnt; i += NT) kids_a[i] = i == 0 ? C->root : cur[i - 1].child;
      __syncthreads();
      uint32_t* ka = kids_a;
      uint32_t* kb = kids_b;
      uint32_t level = lvl;
      while (cnt > 1) {
        const uint32_t per = inner_fill + 1;
        const uint32_t nn = ceil_div(cnt, per);
        if (threadIdx.x == 0) sm.base = atomicAdd(&C->n_nodes, nn);
        __syncthreads();
        const uint32_t nb = sm.base;
        for (uint32_t pidx = w; pidx < nn; pidx += NW) {
          const uint32_t kc = piece_size(pidx, cnt, nn), cs = piece_start(pidx, cnt, nn);
          const uint32_t nd = nb + pidx;
          if (lane < 31) {
            const uint64_t sep = (lane + 1 < kc) ? t.low[ka[cs + lane + 1]] : kKeyMax;
            t.keys[(size_t)nd * 32 + lane] = sep;
            t.pfx[(size_t)nd * 32 + lane] = (uint32_t)(sep >> 32);
          } else {
            t.keys[(size_t)nd * 32 + 31] = make_hdr(kc - 1, level, 0, epoch);
          }
          t.vals[(size_t)nd * 32 + lane] = lane < kc ? (uint64_t)ka[cs + lane] : 0;
          if (lane == 0) {
            t.low[nd] = t.low[ka[cs]];
            kb[pidx] = nd;
          }
        }
        __syncthreads();
        roots_new += nn;
        uint32_t* tmp = ka;
        ka = kb;
        kb = tmp;
        cnt = nn;
        level++;
      }
      if (threadIdx.x == 0) {
        __threadfence();
        C->root = ka[0];
        C->root_level = level - 1;
      }
      __syncthreads();
      break;
    }
    // groups of entries sharing a parent at this level
    auto parent_of = [&](uint32_t i) { return path[lvl * path_stride + cur[i].rep]; };
    auto is_head = [&](uint32_t i) -> uint32_t { return (i == 0 || parent_of(i) != parent_of(i - 1)) ? 1u : 0u; };
    uint32_t ng = 0;
    if (!team_scan<NT>(team, n_e, is_head, goff, gs, sm.ws, &ng)) return;
    for (uint32_t i = team.rank() * NT + threadIdx.x; i < n_e; i += team.size() * NT)
      if (is_head(i)) gstart[goff[i]] = i;
    if (!team.sync()) return;
    // pieces - 1 per group
    auto group_extra = [&](uint32_t gi) -> uint32_t {
      const uint32_t a = gstart[gi], b = gi + 1 < ng ? gstart[gi + 1] : n_e;
      const uint32_t P = parent_of(a);
      const uint32_t tot = hdr_size(t.keys[(size_t)P * 32 + 31]) + (b - a);
      return tot <= (uint32_t)kMaxKeys ? 0u : ceil_div(tot + 1, inner_fill + 1) - 1;
    };
    uint32_t total = 0;
    if (!team_scan<NT>(team, ng, group_extra, goff, gs, sm.ws, &total)) return;
    // one thread checks the capacity and allocates; everyone reads the outcome
    if (team.rank() == 0 && threadIdx.x == 0) {
      if (total > entry_cap || (uint64_t)C->n_nodes + total > t.cap) {
        // cannot happen with inner_fill >= 16 and the headroom reserved
        // above; stop before writing out of bounds and flag the error
        atomicOr(&C->error, kErrCapacity);
        gs->total = 1;
      } else {
        gs->total = 0;
        gs->base = total ? atomicAdd(&C->n_nodes, total) : 0;
      }
    }
    if (!team.sync()) return;
    if (gs->total) return;
    const uint32_t nb = gs->base;
    for (uint32_t gi = gw; gi < ng; gi += n_warps) {
      const uint32_t a = gstart[gi], b = gi + 1 < ng ? gstart[gi + 1] : n_e;
      const uint32_t cnt = b - a;
      const uint32_t P = parent_of(a);
      const uint64_t pk = t.keys[(size_t)P * 32 + lane];
      const uint64_t pv = t.vals[(size_t)P * 32 + lane];
      const uint64_t h = __shfl_sync(kFull, pk, 31);
      const uint32_t sz = hdr_size(h);
      sm.keys[w][lane] = lane < sz ? pk : kKeyMax;
      const uint64_t child0 = __shfl_sync(kFull, pv, 0);
      __syncwarp();
      const uint32_t tot = sz + cnt;
      const uint32_t ch = tot + 1;
      const uint32_t q = tot <= (uint32_t)kMaxKeys ? 1u : ceil_div(ch, inner_fill + 1);
      const uint32_t go = goff[gi];
      auto node_of = [&](uint32_t c) -> uint32_t { return c == 0 ? P : nb + go + c - 1; };
      // separator at merged position x with right child rc: its child index is x + 1
      auto place = [&](uint32_t x, uint64_t key, uint64_t rc) {
        uint32_t c, slot;
        piece_of(x + 1, ch, q, c, slot);
        const uint32_t nd = node_of(c);
        if (slot == 0) {  // first child of piece c >= 1: the separator moves up
          t.vals[(size_t)nd * 32] = rc;
          t.low[nd] = key;
          MergeEntry e;
          e.key = key;
          e.child = nd;
          e.rep = cur[a].rep;
          nxt[go + c - 1] = e;
        } else {
          t.keys[(size_t)nd * 32 + slot - 1] = key;
          t.pfx[(size_t)nd * 32 + slot - 1] = (uint32_t)(key >> 32);
          t.vals[(size_t)nd * 32 + slot] = rc;
        }
      };
      const uint64_t rc_next = __shfl_down_sync(kFull, pv, 1);  // right child of separator `lane`
      if (lane < sz) {
        const uint64_t rc = rc_next;
        uint32_t lo = 0, hi = cnt;
        while (lo < hi) {
          const uint32_t mid = (lo + hi) >> 1;
          if (cur[a + mid].key < pk) lo = mid + 1;
          else hi = mid;
        }
        place(lane + lo, pk, rc);
      }
      __syncwarp();
      for (uint32_t j = lane; j < cnt; j += 32) {
        const MergeEntry e = cur[a + j];
        place(j + count_less(sm.keys[w], sz, e.key), e.key, e.child);
      }
      __syncwarp();
      for (uint32_t c = 0; c < q; c++) {
        const uint32_t nd = node_of(c);
        const uint32_t kc = piece_size(c, ch, q);
        if (c == 0 && lane == 0) t.vals[(size_t)nd * 32] = child0;
        if (lane + 1 >= kc && lane < 31) {
          t.keys[(size_t)nd * 32 + lane] = kKeyMax;
          t.pfx[(size_t)nd * 32 + lane] = 0xffffffffu;
        }
        if (lane >= kc) t.vals[(size_t)nd * 32 + lane] = 0;
        if (lane == 31) t.keys[(size_t)nd * 32 + 31] =
            make_hdr(kc - 1, lvl, c == 0 ? hdr_version(h) + 1 : 0, hdr_epoch(h));
      }
      __syncwarp();
    }
    if (team.rank() == 0) inner_new += total;
    if (!team.sync()) return;  // this level's nodes and the next entries are written
    n_e = total;
    MergeEntry* tmp = cur;
    cur = nxt;
    nxt = tmp;
  }
  if (team.rank() == 0 && threadIdx.x == 0 && (inner_new | roots_new)) {
    atomicAdd(&C->inner_splits, inner_new + roots_new);
    atomicAdd(&C->new_roots, roots_new);
  }
}

__global__ void __launch_bounds__(kInnerThreads) merge_inner_kernel(DevTree t, uint32_t inner_fill, uint32_t entry_cap,
                                                                    MergeCounts* mc, InnerSync* gs,
                                                                    MergeEntry* ea, MergeEntry* eb,
                                                                    const uint32_t* __restrict__ path,
                                                                    size_t path_stride,
                                                                    uint32_t* __restrict__ gstart,
                                                                    uint32_t* __restrict__ goff,
                                                                    uint32_t* __restrict__ kids_a,
                                                                    uint32_t* __restrict__ kids_b) {
  __shared__ InnerSmem<kInnerThreads> sm;
  if (mc->cap_fail) return;
  inner_merge<kInnerThreads>(t, inner_fill, entry_cap, mc, gs, ea, eb, path, path_stride, gstart, goff, kids_a, kids_b,
                             GridTeam{gs, &t.ctrl->error}, sm);
}

// ------------------------------------------------- small batches: write ----
// Everything of a small batch (bt_small.cu) that writes the tree, in one
// cluster: the phases of the general path (merge_update .. merge_fail_mark,
// writeback_kernel, merge_leaf, merge_inner) with a cluster barrier between
// them.  Leaving the leaf and inner merge to their launches over the whole chip
// costs 9 us more a batch up to 4096 requests, and gains only at 65,536 (254
// against 271 us, all INSERTs).
//
// A larger batch takes it when the batch before had few touched requests.  That
// is a guess, and sixteen SMs would take 2.5 us for every further thousand, so
// the batch's own count decides on the device: above the limit the cluster
// returns at once and grid_write_kernel, queued behind it, does the same on
// every SM; at or below it that one finds nothing to do.
struct WriteSmem {
  union {
    LeafSmem<kSmallThreads / 8> leaf;
    InnerSmem<kSmallThreads> inner;
  };
  uint32_t ws[32];
  uint32_t before, total;
};

constexpr uint32_t kWriteTeam = GridTeam::kMost;  // most blocks that write together

struct SmallWrite {
  const BatchCounts* counts;
  MergeCounts* mc;
  InnerSync* gs;
  const uint64_t *ukeys, *uvals, *uans;
  uint8_t* uans_st;
  const uint32_t *ins_list, *pend, *sv, *dleaf, *dslot, *path;
  const uint64_t* vpos;
  uint32_t *isnew, *pos, *leaf, *nq, *nleaf, *seg;
  uint64_t *newk, *newv;
  MergeEntry *ea, *eb;
  uint32_t* sums;  // three sets of kWriteTeam block totals
  uint32_t leaf_fill, inner_fill, entry_cap;
  uint32_t limit;  // touched requests up to which the cluster writes
  size_t path_stride;
};

// exclusive prefix of v over the threads of the team and the total; one
// barrier (sums: a set of its own per use)
template <typename Team>
__device__ __forceinline__ bool team_prefix(const Team& team, uint32_t v, uint32_t* sums, WriteSmem& S,
                                            uint32_t* before, uint32_t* total) {
  uint32_t tot;
  const uint32_t ex = blk_exclusive_sum(v, S.ws, &tot);
  if (threadIdx.x == 0) sums[team.rank()] = tot;
  if (!team.sync()) return false;
  if (threadIdx.x < 32) {
    uint32_t lower = 0, all = 0;
    for (uint32_t b = threadIdx.x; b < team.size(); b += 32) {
      const uint32_t x = __ldcg(sums + b);
      all += x;
      lower += b < team.rank() ? x : 0u;
      if (Team::kMost <= 32) break;
    }
    lower = __reduce_add_sync(kFull, lower);
    all = __reduce_add_sync(kFull, all);
    if (threadIdx.x == 0) {
      S.before = lower;
      S.total = all;
    }
  }
  __syncthreads();
  *before = S.before + ex;
  *total = S.total;
  __syncthreads();
  return true;
}

template <typename Team>
__device__ __forceinline__ void write_part(const DevTree& t, const SmallWrite& a, uint32_t n_ins, uint32_t n_del,
                                           uint32_t n_touch, uint64_t* out_vals, uint8_t* out_st, const Team& team,
                                           WriteSmem& S) {
  const uint32_t rank = team.rank(), C = team.size();
  const uint32_t nt = C * kSmallThreads, gt = rank * kSmallThreads + threadIdx.x;
  MergeCounts* mc = a.mc;
  // new values of the keys found in the tree, then the DELETE keys (which move values)
  for (uint32_t q = gt; q < n_ins; q += nt) {
    const uint64_t p = a.vpos[q];
    if (p != kNoPos) t.vals[p] = a.uvals[a.ins_list[q]];
  }
  if (n_del) {
    if (!team.sync()) return;
    uint32_t removed = 0;
    for (uint32_t i = gt >> 5; i < n_del; i += nt >> 5)
      removed += del_apply_at(t, a.dleaf, a.dslot, i, n_del, threadIdx.x & 31);
    if ((threadIdx.x & 31) == 0 && removed) atomicAdd(&t.ctrl->n_keys, (unsigned long long)0 - removed);
  }
  // this thread's consecutive items of n spread over the team: one while there
  // are threads enough (several would be that many chains of loads in a row)
  auto mine = [&](uint32_t n, uint32_t& i0, uint32_t& i1) {
    const uint32_t each = ceil_div(n, nt);
    i0 = (uint32_t)min((uint64_t)n, (uint64_t)gt * each);
    i1 = min(n, i0 + each);
  };
  uint32_t n_new = 0, n_segs = 0, n_ent = 0;
  if (n_ins) {
    // the new keys, compacted
    uint32_t i0, i1, v = 0;
    mine(n_ins, i0, i1);
    for (uint32_t i = i0; i < i1; i++) v += a.isnew[i];
    uint32_t p;
    if (!team_prefix(team, v, a.sums, S, &p, &n_new)) return;
    for (uint32_t i = i0; i < i1; i++) {
      if (!a.isnew[i]) continue;
      const uint32_t u = a.ins_list[i];
      a.newk[p] = a.ukeys[u];
      a.newv[p] = a.uvals[u];
      a.nq[p] = i;
      a.nleaf[p] = a.leaf[i];
      p++;
    }
  }
  if (n_new) {
    if (!team.sync()) return;
    // runs of new keys that share a leaf
    uint32_t i0, i1, v = 0;
    mine(n_new, i0, i1);
    const uint32_t before = i0 > 0 && i0 < i1 ? __ldcg(a.nleaf + i0 - 1) : kNil;  // kNil: no leaf
    uint32_t prev = before;
    for (uint32_t i = i0; i < i1; i++) {
      const uint32_t lf = __ldcg(a.nleaf + i);
      v += lf != prev ? 1u : 0u;
      prev = lf;
    }
    uint32_t p;
    if (!team_prefix(team, v, a.sums + kWriteTeam, S, &p, &n_segs)) return;
    prev = before;
    for (uint32_t i = i0; i < i1; i++) {
      const uint32_t lf = __ldcg(a.nleaf + i);
      if (lf != prev) {
        a.seg[p] = i;
        a.leaf[p++] = lf;
      }
      prev = lf;
    }
    if (!team.sync()) return;
    // new leaves per run
    mine(n_segs, i0, i1);
    v = 0;
    for (uint32_t i = i0; i < i1; i++) {
      const uint32_t b = __ldcg(a.seg + i), e = i + 1 < n_segs ? __ldcg(a.seg + i + 1) : n_new;
      const uint32_t m = hdr_size(__ldcg(t.keys + (size_t)__ldcg(a.leaf + i) * 32 + 31)) + (e - b);
      const uint32_t x = m <= (uint32_t)kMaxKeys ? 0u : ceil_div(m, a.leaf_fill) - 1;
      a.isnew[i] = x;
      v += x;
    }
    if (!team_prefix(team, v, a.sums + 2 * kWriteTeam, S, &p, &n_ent)) return;
    for (uint32_t i = i0; i < i1; i++) {
      const uint32_t x = a.isnew[i];
      a.pos[i] = p;
      p += x;
    }
  }
  if (gt == 0) {
    mc->n_new = n_new;
    mc->n_segs = n_segs;
    mc->n_leaf_entries = n_ent;
    reserve_pieces(t, mc, a.entry_cap);
  }
  if (!team.sync()) return;
  const bool fail = __ldcg(&mc->cap_fail) != 0;
  if (fail) {  // a full pool: the new keys are answered kNoCapacity
    for (uint32_t i = gt; i < n_new; i += nt) a.uans_st[a.ins_list[a.nq[i]]] = kNoCapacity;
    if (!team.sync()) return;
  }
  for (uint32_t i = gt; i < n_touch; i += nt) {
    const uint32_t u = a.pend[i];
    if (u == 0xFFFFFFFFu) continue;  // answered by the front part
    const uint32_t r = pair_idx(a.sv[i]);
    out_vals[r] = a.uans[u];
    out_st[r] = __ldcg(a.uans_st + u);
  }
  if (fail) return;
  leaf_merge<8, kSmallThreads / 8>(t, a.leaf_fill, mc, a.seg, a.pos, a.isnew, a.newk, a.newv, a.nq, a.leaf,
                                          a.ea, S.leaf, gt / 8, nt / 8);
  if (n_ent == 0) return;
  if (!team.sync()) return;
  inner_merge<kSmallThreads>(t, a.inner_fill, a.entry_cap, mc, a.gs, a.ea, a.eb, a.path, a.path_stride, a.seg, a.nleaf,
                             a.nq, a.pos, team, S.inner);
}

// kGuess: a larger batch's, which may have more touched requests than the limit
template <bool kGuess>
__global__ void __launch_bounds__(kSmallThreads, 1) small_write_kernel(DevTree t, SmallWrite a, uint64_t* out_vals,
                                                                       uint8_t* out_st) {
  extern __shared__ __align__(16) unsigned char raw[];
  after_previous();
  const uint32_t n_ins = a.counts->n_ins, n_del = a.counts->n_del, n_touch = a.counts->n_touch;
  if (kGuess && n_touch > a.limit) {  // for grid_write_kernel, its barrier as new
    if (cluster_rank() == 0 && threadIdx.x == 0) a.gs->count = a.gs->fail = 0;
    return;
  }
  write_part(t, a, n_ins, n_del, n_touch, out_vals, out_st, ClusterTeam{}, *reinterpret_cast<WriteSmem*>(raw));
}

// The same over the chip, one block an SM.  Bound by its ten or so grid barriers, then
// like merge_leaf_kernel by entry -> leaf -> row.  Batches of INSERTs behind a light one
// on 2^23 keys: 100,000 185 us (cluster 305, the general path's launches 210), 2^18 255
// (632, 282), 2^20 565 (1977, 585), 2^21 1040 (general 970), 2^22 2550 (6280, 1740: there
// a thread's 28 consecutive items are as many loads in a row).  Four blocks of 256
// threads an SM: 2^21 1110; one of 256: 1390.
__global__ void __launch_bounds__(kSmallThreads, 1) grid_write_kernel(DevTree t, SmallWrite a, uint64_t* out_vals,
                                                                      uint8_t* out_st) {
  extern __shared__ __align__(16) unsigned char raw[];
  const uint32_t n_touch = a.counts->n_touch;
  if (n_touch <= a.limit) return;  // small_write_kernel wrote it
  write_part(t, a, a.counts->n_ins, a.counts->n_del, n_touch, out_vals, out_st, GridTeam{a.gs, &t.ctrl->error},
             *reinterpret_cast<WriteSmem*>(raw));
}

}  // namespace

// blocks of a cooperative kernel that are resident at once, asked once per device
static unsigned resident_blocks(const Handle* h, const void* kernel, int threads, size_t smem, unsigned (&known)[64]) {
  const int dev = h->device;
  if (dev < 0 || dev >= 64) return (unsigned)h->sm_count;
  if (!known[dev]) {
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem) != cudaSuccess || per < 1) per = 1;
    known[dev] = (unsigned)per * (unsigned)h->sm_count;
  }
  return known[dev];
}

// cooperative launch of merge_inner_kernel: at most the resident blocks
static cudaError_t launch_inner(Handle* h, uint32_t entry_cap, MergeCounts* mc, cudaStream_t s) {
  Work& w = h->w;
  static unsigned resident[64] = {};
  unsigned blocks = resident_blocks(h, (const void*)merge_inner_kernel, kInnerThreads, 0, resident);
  if (blocks > 1024) blocks = 1024;  // InnerSync::partial
  InnerSync* gs = reinterpret_cast<InnerSync*>(w.m_sync);
  cudaError_t e = cudaMemsetAsync(gs, 0, sizeof(InnerSync), s);
  if (e != cudaSuccess) return e;
  DevTree tree = h->tree;
  uint32_t fill = h->inner_fill;
  MergeEntry* ea = reinterpret_cast<MergeEntry*>(w.m_ent_a);
  MergeEntry* eb = reinterpret_cast<MergeEntry*>(w.m_ent_b);
  const uint32_t* path = w.m_path;
  size_t path_stride = w.cap;
  uint32_t* gstart = w.m_seg;
  uint32_t* goff = w.m_nleaf;
  uint32_t* kids_a = w.m_nq;
  uint32_t* kids_b = w.m_pos;
  void* args[] = {&tree, &fill, &entry_cap, &mc, &gs, &ea, &eb, &path, &path_stride, &gstart, &goff, &kids_a, &kids_b};
  e = cudaLaunchCooperativeKernel((const void*)merge_inner_kernel, dim3(blocks), dim3(kInnerThreads), args, 0, s);
  count_launch();
  return e;
}

int locate_phase(Handle* h, int what, size_t n_upper, cudaStream_t s) {
  Work& w = h->w;
  // the INSERT keys need a root; once there is one only a new tree takes it away.
  // A launch that is captured has not run, and its graph may run on a later tree
  // without a root: there it is always part of the batch and says nothing
  bool captured = false;
  if (stream_captured(s, &captured) != cudaSuccess) return -2;
  if ((what & kLocateIns) && (captured || !h->has_root)) {
    merge_ensure_root_kernel<<<1, 1, 0, s>>>(h->tree);
    count_launch();
    h->has_root = h->has_root || !captured;
  }
  LocateArgs a;
  a.counts = w.counts;
  a.ukeys = w.ukeys;
  a.ins_list = w.ins_list;
  a.del_list = w.del_list;
  a.path = w.m_path;
  a.mleaf = w.m_leaf;
  a.isnew = w.m_isnew;
  a.vpos = w.m_vpos;
  a.dleaf = w.d_leaf;
  a.dslot = w.d_slot;
  a.uans = w.uans;
  a.uans_st = w.uans_st;
  a.path_stride = w.cap;
  const unsigned blocks = (unsigned)min((size_t)h->sm_count * 8, (n_upper + 255) / 256 + 1);
  locate_kernel<<<blocks, 256, 0, s>>>(h->tree, a, what);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int merge_update_phase(Handle* h, size_t n_upper, cudaStream_t s) {
  Work& w = h->w;
  const unsigned gb = (unsigned)min((size_t)h->sm_count * 8, (n_upper + 255) / 256);
  launch_after(merge_update_kernel, gb, 256, 0, s, h->tree, w.uvals, w.ins_list, &w.counts->n_ins, w.m_vpos);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// look-back words for a batch of up to n requests: new keys, segments | the
// segments' new leaves reuse the first part
size_t merge_lb_words(size_t n) { return 2 * ((n + kGroupThreads - 1) / kGroupThreads + 1); }

int merge_group_phase(Handle* h, size_t n_upper, cudaStream_t s) {
  Work& w = h->w;
  MergeCounts* mc = reinterpret_cast<MergeCounts*>(w.m_counts);
  const unsigned gb = (unsigned)min((size_t)h->sm_count * 2, (n_upper + kGroupTile - 1) / kGroupTile);
  launch_after(merge_group_kernel, gb, kGroupThreads, 0, s, mc, w.ins_list, &w.counts->n_ins, w.m_isnew, w.ukeys,
               w.uvals, w.m_leaf, w.m_newk, w.m_newv, w.m_nq, w.m_nleaf, w.m_seg, w.m_pos, w.lb_status,
               w.lb_status + merge_lb_words(w.cap) / 2, w.lb_ctr, &h->tree.ctrl->error);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int merge_reserve_phase(Handle* h, size_t n_upper, cudaStream_t s) {
  Work& w = h->w;
  MergeCounts* mc = reinterpret_cast<MergeCounts*>(w.m_counts);
  const unsigned rb = (unsigned)min((size_t)h->sm_count * 2, (n_upper + kGroupThreads - 1) / kGroupThreads);
  launch_after(merge_reserve_kernel, rb, kGroupThreads, 0, s, h->tree, h->leaf_fill, (uint32_t)w.cap, mc, w.m_seg,
               w.m_pos, w.m_isnew, w.m_leaf, w.lb_status, w.lb_ctr, &h->tree.ctrl->error);
  const unsigned gb = (unsigned)min((size_t)h->sm_count * 8, (n_upper + 255) / 256);
  launch_after(merge_fail_mark_kernel, gb, 256, 0, s, mc, w.m_nq, w.ins_list, w.uans_st);
  count_launch(2);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int merge_write_phase(Handle* h, cudaStream_t s) {
  Work& w = h->w;
  MergeCounts* mc = reinterpret_cast<MergeCounts*>(w.m_counts);
  const uint32_t entry_cap = (uint32_t)w.cap;
  merge_leaf_kernel<8><<<(unsigned)((size_t)h->sm_count * 8), 256, 0, s>>>(
      h->tree, h->leaf_fill, mc, w.m_seg, w.m_leaf, w.m_isnew, w.m_newk, w.m_newv, w.m_nq, w.m_pos,
      reinterpret_cast<MergeEntry*>(w.m_ent_a));
  count_launch();
  if (launch_inner(h, entry_cap, mc, s) != cudaSuccess) return -2;
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

size_t small_write_words() { return 3 * kWriteTeam; }

unsigned small_write_largest() { return small_largest((const void*)small_write_kernel<true>, sizeof(WriteSmem)); }

int small_write_prepare() {
  const auto smem = cudaFuncAttributeMaxDynamicSharedMemorySize;
  const auto wide = cudaFuncAttributeNonPortableClusterSizeAllowed;
  const int bytes = (int)sizeof(WriteSmem);
  cudaError_t e = cudaFuncSetAttribute(grid_write_kernel, smem, bytes);
  for (auto k : {small_write_kernel<false>, small_write_kernel<true>}) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, smem, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, wide, 1);
  }
  return e == cudaSuccess ? 0 : -2;
}

int small_write(Handle* h, uint64_t* out_vals, uint8_t* out_st, size_t n, uint32_t limit, cudaStream_t s) {
  Work& w = h->w;
  SmallWrite a;
  a.counts = w.counts;
  a.mc = reinterpret_cast<MergeCounts*>(w.m_counts);
  a.gs = reinterpret_cast<InnerSync*>(w.m_sync);
  a.ukeys = w.ukeys;
  a.uvals = w.uvals;
  a.uans = w.uans;
  a.uans_st = w.uans_st;
  a.ins_list = w.ins_list;
  a.pend = w.pend;
  a.sv = w.v_a;
  a.dleaf = w.d_leaf;
  a.dslot = w.d_slot;
  a.path = w.m_path;
  a.path_stride = w.cap;
  a.vpos = w.m_vpos;
  a.isnew = w.m_isnew;
  a.pos = w.m_pos;
  a.leaf = w.m_leaf;
  a.nq = w.m_nq;
  a.nleaf = w.m_nleaf;
  a.seg = w.m_seg;
  a.newk = w.m_newk;
  a.newv = w.m_newv;
  a.ea = reinterpret_cast<MergeEntry*>(w.m_ent_a);
  a.eb = reinterpret_cast<MergeEntry*>(w.m_ent_b);
  a.sums = w.s_write;
  a.leaf_fill = h->leaf_fill;
  a.inner_fill = h->inner_fill;
  a.entry_cap = (uint32_t)w.cap;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[2];
  small_config(cfg, at, small_cluster(n, h->small_blocks), sizeof(WriteSmem), s);
  a.limit = limit;
  const bool guess = limit < n;
  cudaError_t e =
      cudaLaunchKernelEx(&cfg, guess ? small_write_kernel<true> : small_write_kernel<false>, h->tree, a, out_vals, out_st);
  count_launch();
  if (e == cudaSuccess && guess) {
    static unsigned resident[64] = {};
    void* args[] = {&h->tree, &a, &out_vals, &out_st};
    e = cudaLaunchCooperativeKernel(
        (const void*)grid_write_kernel,
        dim3(min(resident_blocks(h, (const void*)grid_write_kernel, kSmallThreads, sizeof(WriteSmem), resident),
                 kWriteTeam)),
        dim3(kSmallThreads), args, sizeof(WriteSmem), s);
    count_launch();
  }
  return e == cudaSuccess ? 0 : -2;
}

int merge_engine(Handle* h, size_t n_upper, cudaStream_t s) {
  if (locate_phase(h, kLocateIns, n_upper, s) != 0 || merge_update_phase(h, n_upper, s) != 0 ||
      merge_group_phase(h, n_upper, s) != 0 || merge_reserve_phase(h, n_upper, s) != 0)
    return -2;
  return merge_write_phase(h, s);
}

}  // namespace bt
