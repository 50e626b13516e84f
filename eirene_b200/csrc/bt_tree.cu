// Tree construction and the lock-free batched point search.
//
// Search: a group of G lanes serves one request (G = 4, 8, 16 or 32; the
// reference uses a whole warp, one key per lane, src/gpu-stm-tree-v39/
// bpt-gpustm-kernel-tree.cuh:61-118).  Each lane loads 32/G consecutive keys
// of the node with 16-byte vector loads, counts keys <= target, and the group
// sums the counts with xor-shuffles: that sum is the child slot (child i covers
// [key[i-1], key[i]), src/tree.h:7-19).  With G = 8 a warp carries four
// independent descents, four times the memory-level parallelism of the
// reference's warp-per-request layout.  This kernel runs only when no writer
// is active (the batch executor orders it before/after the insert phase), so
// it needs no version checks.
#include <cstdio>
#include <mutex>
#include <cuda_runtime.h>

#include "bt_block.cuh"
#include "bt_common.cuh"
#include "bt_internal.h"
#include "bt_lookback.cuh"
#include "bt_search.cuh"

namespace bt {

namespace {

__global__ void reset_kernel(Ctrl* c, uint32_t epoch) {
  c->root = kNil;
  c->epoch = epoch;
  c->root_lock = 0;
  c->n_nodes = 0;
  c->error = 0;
  c->root_level = 0;
  c->n_keys = 0;
  c->commits = c->aborts = c->leaf_splits = c->inner_splits = c->new_roots = 0;
  c->retry_exhausted = c->learned_hits = c->learned_fallbacks = c->learned_probe_sum = 0;
}

// ---------------------------------------------------------------- build ----
// The bulk loader reads nothing back until its end: how many distinct keys there
// are, whether the last is the reserved one and how many nodes each level takes
// is worked out on the device (BuildGeo), and the grids are sized for n distinct
// keys.
constexpr int kBuildLevels = 30;
struct BuildGeo {
  uint32_t m;       // distinct keys
  uint32_t status;  // 0, or the kBuild* reason why the tree stays empty
  uint32_t height, total;
  uint32_t cnt[kBuildLevels];    // nodes per level, leaves first
  uint32_t first[kBuildLevels];  // id of a level's first node
};
static_assert(sizeof(BuildGeo) <= 256, "the static build's scratch keeps 256 bytes for it");
constexpr uint32_t kBuildCapacity = 4, kBuildReserved = 5;

constexpr int kDedupeThreads = 1024;
constexpr int kDedupeItems = 4;
constexpr int kDedupeTile = kDedupeThreads * kDedupeItems;

// the last pair of every run of equal keys stays (a repeated key's last value wins)
__device__ __forceinline__ uint32_t tails_of(const uint64_t* __restrict__ sk, size_t n, size_t i0,
                                             uint64_t (&k)[kDedupeItems + 1]) {
  uint32_t m = 0;
#pragma unroll
  for (int j = 0; j <= kDedupeItems; j++) k[j] = i0 + j < n ? sk[i0 + j] : 0;
#pragma unroll
  for (int j = 0; j < kDedupeItems; j++)
    if (i0 + j < n && (i0 + j + 1 == n || k[j + 1] != k[j])) m |= 1u << j;
  return m;
}

__global__ void __launch_bounds__(kDedupeThreads) tail_count_kernel(const uint64_t* __restrict__ sk, size_t n,
                                                                    uint32_t* __restrict__ tile) {
  __shared__ uint32_t ws[32];
  uint64_t k[kDedupeItems + 1];
  uint32_t total;
  blk_exclusive_sum(__popc(tails_of(sk, n, (size_t)blockIdx.x * kDedupeTile + threadIdx.x * kDedupeItems, k)), ws,
                    &total);
  if (threadIdx.x == 0) tile[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kDedupeThreads) dedupe_kernel(const uint64_t* __restrict__ sk,
                                                                const uint32_t* __restrict__ sidx,
                                                                const uint64_t* __restrict__ vals, size_t n,
                                                                const uint32_t* __restrict__ tile,
                                                                uint64_t* __restrict__ uk, uint64_t* __restrict__ uv) {
  __shared__ uint32_t ws[32];
  const size_t i0 = (size_t)blockIdx.x * kDedupeTile + threadIdx.x * kDedupeItems;
  uint64_t k[kDedupeItems + 1];
  const uint32_t m = tails_of(sk, n, i0, k);
  uint32_t p = tile[blockIdx.x] + blk_exclusive_sum(__popc(m), ws, nullptr);
#pragma unroll
  for (int j = 0; j < kDedupeItems; j++)
    if ((m >> j) & 1u) {
      uk[p] = k[j];
      uv[p++] = vals[sidx[i0 + j]];
    }
}

__global__ void build_geo_kernel(BuildGeo* g, const uint32_t* m, const uint64_t* last, uint32_t leaf_fill,
                                 uint32_t per, uint32_t cap) {
  g->m = *m;
  uint64_t total = 0;
  uint32_t cnt = (g->m + leaf_fill - 1) / leaf_fill, h = 0;
  for (;; cnt = (cnt + per - 1) / per) {
    g->cnt[h] = cnt;
    g->first[h] = (uint32_t)total;
    total += cnt;
    h++;
    if (cnt == 1 || h == (uint32_t)kBuildLevels) break;
  }
  g->height = h;
  g->total = (uint32_t)total;
  g->status = *last == kKeyMax ? kBuildReserved : (total > cap || cnt != 1) ? kBuildCapacity : 0u;
}

// one warp per leaf; leaves get base or base+1 keys (the first `rem` get one more)
__global__ void __launch_bounds__(256) build_leaves_kernel(DevTree t, const uint64_t* __restrict__ uk,
                                                           const uint64_t* __restrict__ uv,
                                                           const BuildGeo* __restrict__ geo, uint32_t epoch) {
  const uint32_t lane = threadIdx.x & 31;
  const size_t j = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nl = geo->cnt[0];
  if (j >= nl || geo->status) return;
  const uint32_t base = geo->m / nl, rem = geo->m % nl;
  const uint32_t k = base + (j < rem ? 1 : 0);
  const size_t start = j * base + (j < rem ? j : rem);
  const uint64_t key = lane < k ? uk[start + lane] : kKeyMax;
  uint64_t* kr = t.keys + j * 32;
  uint64_t* vr = t.vals + j * 32;
  if (lane < 31) {
    kr[lane] = key;
    vr[lane] = lane < k ? uv[start + lane] : 0;
  } else {
    kr[31] = make_hdr(k, 0, 0, epoch);
    vr[31] = (j + 1 < nl) ? uk[start + k] : kKeyMax;
  }
  t.fp[j * 32 + lane] = lane < k ? slot_fp(key) : (uint8_t)0;
  if (lane == 0) t.low[j] = j == 0 ? 0 : key;
}

// one warp per inner node: node p of the level groups children [c, c + k)
__device__ __forceinline__ void build_inner_node(const DevTree& t, const BuildGeo* geo, uint32_t level, uint32_t p,
                                                 uint32_t lane, uint32_t epoch) {
  const uint32_t n_children = geo->cnt[level - 1], nn = geo->cnt[level];
  const uint32_t base = n_children / nn, rem = n_children % nn;
  const uint32_t k = base + (p < rem ? 1 : 0);
  const uint32_t c = geo->first[level - 1] + p * base + (p < rem ? p : rem);
  const uint32_t id = geo->first[level] + p;
  // key slot i (i < k-1) = low fence of child i+1
  const uint64_t sep = (lane + 1 < k) ? t.low[c + lane + 1] : kKeyMax;
  t.keys[(size_t)id * 32 + lane] = lane < 31 ? sep : make_hdr(k - 1, level, 0, epoch);
  t.pfx[(size_t)id * 32 + lane] = lane < 31 ? (uint32_t)(sep >> 32) : 0xffffffffu;
  t.vals[(size_t)id * 32 + lane] = lane < k ? (uint64_t)(c + lane) : 0;
  if (lane == 0) t.low[id] = t.low[c];
}

__global__ void __launch_bounds__(256) build_inner_kernel(DevTree t, const BuildGeo* __restrict__ geo, uint32_t level,
                                                          uint32_t epoch) {
  const uint32_t p = (uint32_t)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (geo->status || level >= geo->height || p >= geo->cnt[level]) return;
  build_inner_node(t, geo, level, p, threadIdx.x & 31, epoch);
}

// the levels from `level` up (a few hundred nodes at most) and the root, one block
constexpr uint32_t kBuildTopNodes = 512;
__global__ void __launch_bounds__(1024) build_top_kernel(DevTree t, const BuildGeo* geo, uint32_t level,
                                                         uint32_t epoch) {
  if (geo->status) return;
  for (uint32_t l = level; l < geo->height; l++) {
    for (uint32_t p = threadIdx.x >> 5; p < geo->cnt[l]; p += blockDim.x >> 5)
      build_inner_node(t, geo, l, p, threadIdx.x & 31, epoch);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    t.ctrl->root = geo->total - 1;
    t.ctrl->root_level = geo->height - 1;
    t.ctrl->n_nodes = geo->total;
    t.ctrl->n_keys = geo->m;
  }
}

// --------------------------------------------------------------- search ----
template <int G, bool kLeafVals>
__global__ void __launch_bounds__(256) search_kernel(DevTree t, const uint64_t* __restrict__ qkeys,
                                                     const uint32_t* __restrict__ list,
                                                     const uint32_t* __restrict__ n_dev, size_t n_host,
                                                     uint64_t* __restrict__ out_vals, uint8_t* __restrict__ out_st) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t g = lane % G;
  const uint32_t gmask = group_mask<G>(lane);
  const size_t n = n_dev ? (size_t)*n_dev : n_host;
  const uint32_t root = t.ctrl->root;
  const uint32_t root_level = t.ctrl->root_level;
  const size_t stride = ((size_t)gridDim.x * blockDim.x) / G;
  for (size_t q = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / G; q < n; q += stride) {
    const uint32_t r = list ? __ldg(list + q) : (uint32_t)q;
    const uint64_t key = __ldg(qkeys + r);
    uint8_t st = kAbsent;
    uint64_t ans = 0;
    if (key == kKeyMax) st = kRejected;
    else if (root != kNil) st = group_descend<G, kLeafVals>(t, root, root_level, key, g, gmask, ans);
    if (g == 0) {
      out_vals[r] = ans;
      out_st[r] = st;
    }
  }
}

// Two requests per group in lock step (group_descend2): requests q and
// q + stride of the grid-stride loop share a group.
template <int G, bool kLeafVals, bool kChild>
__global__ void __launch_bounds__(256) search2_kernel(DevTree t, const uint64_t* __restrict__ qkeys,
                                                      const uint32_t* __restrict__ list,
                                                      const uint32_t* __restrict__ n_dev, size_t n_host,
                                                      uint64_t* __restrict__ out_vals, uint8_t* __restrict__ out_st,
                                                      int use_pfx, const uint64_t* __restrict__ ckeys) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t g = lane % G;
  const uint32_t gmask = group_mask<G>(lane);
  const size_t n = n_dev ? (size_t)*n_dev : n_host;
  const uint32_t root = t.ctrl->root;
  const uint32_t root_level = t.ctrl->root_level;
  const size_t groups = ((size_t)gridDim.x * blockDim.x) / G;
  for (size_t q = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / G; q < n; q += 2 * groups) {
    const size_t q2 = q + groups;
    const bool two = q2 < n;
    const uint32_t ra = list ? __ldg(list + q) : (uint32_t)q;
    const uint32_t rb = two ? (list ? __ldg(list + q2) : (uint32_t)q2) : ra;
    const uint64_t key_a = ckeys ? __ldg(ckeys + q) : __ldg(qkeys + ra);
    const uint64_t key_b = ckeys ? __ldg(ckeys + (two ? q2 : q)) : __ldg(qkeys + rb);
    uint8_t sa = kAbsent, sb = kAbsent;
    uint64_t aa = 0, ab = 0;
    if (root != kNil) {
      // a reserved key descends as key 0 (keeping the pair in lock step) and is reported as rejected
      group_descend2<G, kLeafVals, kChild>(t, root, root_level, key_a == kKeyMax ? 0 : key_a,
                                   key_b == kKeyMax ? 0 : key_b, g, gmask, aa, sa, ab, sb, use_pfx != 0);
    }
    if (key_a == kKeyMax) {
      sa = kRejected;
      aa = 0;
    }
    if (key_b == kKeyMax) {
      sb = kRejected;
      ab = 0;
    }
    if (g == 0) {
      out_vals[ra] = aa;
      out_st[ra] = sa;
      if (two) {
        out_vals[rb] = ab;
        out_st[rb] = sb;
      }
    }
  }
}

// The default plain lookups (four lanes, child ids): a warp takes 32 requests
// at a time (warp_lookup).  Four lanes to a request with two requests per
// group, shuffles under a mask per group and a 256-byte leaf row issued 63 warp
// instructions a request and took 384 us for 2^22 lookups on 2^24 keys (issue
// 57 %, L1 data pipe 68 %); this form takes 228 us, bound by the L1 data pipe
// (a pass for the row and one for the child id per request and level).
__global__ void __launch_bounds__(256) search_warp_kernel(DevTree t, const uint64_t* __restrict__ qkeys,
                                                          const uint32_t* __restrict__ list,
                                                          const uint32_t* __restrict__ n_dev, size_t n_host,
                                                          uint64_t* __restrict__ out_vals,
                                                          uint8_t* __restrict__ out_st,
                                                          const uint64_t* __restrict__ ckeys) {
  const size_t n = n_dev ? (size_t)*n_dev : n_host;
  const uint32_t root = t.ctrl->root, root_level = t.ctrl->root_level;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  // whole warps: the base index is the warp's
  for (size_t b = (size_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); b < n; b += stride) {
    const size_t q = b + (threadIdx.x & 31u);
    const bool live = q < n;
    const uint32_t r = live && list ? __ldg(list + q) : (uint32_t)q;
    const uint64_t key = live ? (ckeys ? __ldg(ckeys + q) : __ldg(qkeys + r)) : 0;
    uint64_t val;
    const uint8_t st = warp_lookup(t, root, root_level, key, live, val);
    if (live) {
      out_vals[r] = val;
      out_st[r] = st;
    }
  }
}

// Search over keys given in ascending order (the batch executor's unique
// GET list).  Each group walks a contiguous chunk of the list and keeps the
// path of its previous lookup: lane l of the group caches level l's node id
// and the exclusive upper bound of its key range.  A key restarts its descent
// at the lowest cached level whose range still holds it (keys ascend, so only
// the upper bound needs checking); a key in the previous leaf reuses the leaf
// row already in registers.  Requires root_level < G.
template <int G, bool kLeafVals>
__global__ void __launch_bounds__(256) search_sorted_kernel(DevTree t, const uint64_t* __restrict__ qkeys,
                                                            const uint32_t* __restrict__ list,
                                                            const uint32_t* __restrict__ n_dev, size_t n_host,
                                                            uint64_t* __restrict__ out_vals,
                                                            uint8_t* __restrict__ out_st) {
  constexpr int S = 32 / G;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t g = lane % G;
  const uint32_t gmask = group_mask<G>(lane);
  const size_t n = n_dev ? (size_t)*n_dev : n_host;
  const uint32_t root = t.ctrl->root;
  const uint32_t root_level = t.ctrl->root_level;
  const size_t n_groups = ((size_t)gridDim.x * blockDim.x) / G;
  const size_t gid = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
  const size_t chunk = (n + n_groups - 1) / n_groups;
  const size_t q0 = gid * chunk;
  const size_t q1 = min(n, q0 + chunk);
  // path cache (lane g holds level g)
  uint32_t c_node = root;
  uint64_t c_hi = 0;       // exclusive upper bound; 0 with c_valid = false
  bool c_valid = (g == root_level);
  if (c_valid) c_hi = kKeyMax;  // the root covers everything
  uint64_t k[S];
  uint64_t v[S];
  uint32_t leaf = kNil;
  for (size_t q = q0; q < q1; q++) {
    const uint32_t r = list ? __ldg(list + q) : (uint32_t)q;
    const uint64_t key = __ldg(qkeys + r);
    uint8_t st = kAbsent;
    uint64_t ans = 0;
    if (key == kKeyMax) {
      st = kRejected;
    } else if (root != kNil) {
      if (root_level >= (uint32_t)G) {  // tree taller than the cache: plain descent
        st = group_descend<G, false>(t, root, root_level, key, g, gmask, ans);
        if (g == 0) {
          out_vals[r] = ans;
          out_st[r] = st;
        }
        continue;
      }
      // lowest cached level whose range holds the key
      const uint32_t hit = (__ballot_sync(gmask, c_valid && key < c_hi) >> (lane - g)) & ((1u << G) - 1u);
      uint32_t level = hit ? (uint32_t)(__ffs(hit) - 1) : root_level;
      uint32_t node = __shfl_sync(gmask, c_node, level, G);
      uint64_t hi = __shfl_sync(gmask, c_hi, level, G);
      if (!hit) {
        node = root;
        hi = kKeyMax;
      }
      // levels below `level` are now stale
      if (g < level) c_valid = false;
      uint32_t cnt = 0;
      if (level == 0 && node == leaf) {
        uint32_t c = 0;
#pragma unroll
        for (int i = 0; i < S; i++) c += (k[i] <= key) ? 1u : 0u;
        cnt = group_sum<G>(c, gmask);
      } else {
        for (;;) {
          const size_t row = (size_t)node * 32 + g * S;
          load_slots<S>(t.keys + row, k);
          if (level > 0 || kLeafVals) load_slots<S>(t.vals + row, v);
          if (g == G - 1) k[S - 1] = kKeyMax;
          uint32_t c = 0;
#pragma unroll
          for (int i = 0; i < S; i++) c += (k[i] <= key) ? 1u : 0u;
          cnt = group_sum<G>(c, gmask);
          if (level == 0) break;
          // child range upper bound: key[cnt] (padding is UINT64_MAX) capped by ours
          const uint64_t sep = __shfl_sync(gmask, pick<S>(k, cnt % S), cnt / S, G);
          const uint64_t child_hi = sep < hi ? sep : hi;
          node = (uint32_t)__shfl_sync(gmask, pick<S>(v, cnt % S), cnt / S, G);
          hi = child_hi;
          level--;
          if (g == level) {
            c_node = node;
            c_hi = hi;
            c_valid = true;
          }
        }
        leaf = node;
      }
      st = group_leaf_lookup<G, kLeafVals>(t, leaf, key, g, gmask, k, v, cnt, ans);
    }
    if (g == 0) {
      out_vals[r] = ans;
      out_st[r] = st;
    }
  }
}

// ---------------------------------------------------------- enumeration ----
// Levels from the root down, their counts on the device (cnt[l]: nodes of
// level l, leaves at 0).  The top levels, while they have few nodes, by one
// block; each of the others by a count, a scan and a write.
constexpr uint32_t kEnumTop = 512;

__global__ void __launch_bounds__(1024) enum_top_kernel(DevTree t, uint32_t root_level, uint32_t* a, uint32_t* b,
                                                        uint32_t* __restrict__ cnt) {
  __shared__ uint32_t ws[32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t n = 1;
  if (threadIdx.x == 0) {
    a[0] = t.ctrl->root;
    cnt[root_level] = 1;
  }
  __syncthreads();
  __shared__ uint32_t off[kEnumTop];
  for (uint32_t l = root_level; l > 0 && n <= kEnumTop; l--) {
    const uint32_t c = threadIdx.x < n ? hdr_size(t.keys[(size_t)a[threadIdx.x] * 32 + 31]) + 1 : 0u;
    uint32_t total;
    const uint32_t ex = blk_exclusive_sum(c, ws, &total);
    if (threadIdx.x < n) off[threadIdx.x] = ex;
    __syncthreads();
    for (uint32_t i = warp; i < n; i += 32) {
      const uint32_t node = a[i];
      if (lane <= hdr_size(t.keys[(size_t)node * 32 + 31])) b[off[i] + lane] = (uint32_t)t.vals[(size_t)node * 32 + lane];
    }
    __syncthreads();
    n = total;
    if (threadIdx.x == 0) cnt[l - 1] = n;
    uint32_t* x = a;
    a = b;
    b = x;
  }
}

// levels that enum_top_kernel has expanded (a node count up to kEnumTop) are skipped
__device__ __forceinline__ bool enum_done(const uint32_t* cnt, uint32_t level, uint32_t root_level) {
  for (uint32_t l = root_level; l > level; l--)
    if (cnt[l] > kEnumTop) return false;  // the block stopped above this level
  return cnt[level] <= kEnumTop;
}

// children per node of the level (or, `leaf_sizes`, keys per leaf); *n_out: how
// many entries the scan and the write handle (0: done already)
__global__ void __launch_bounds__(256) child_count_kernel(DevTree t, const uint32_t* __restrict__ nodes,
                                                          const uint32_t* __restrict__ cnt, uint32_t level,
                                                          uint32_t root_level, uint32_t* __restrict__ out,
                                                          uint32_t* __restrict__ n_out, int leaf_sizes) {
  const uint32_t n = !leaf_sizes && enum_done(cnt, level, root_level) ? 0u : cnt[level];
  if (blockIdx.x == 0 && threadIdx.x == 0) *n_out = n;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint64_t h = t.keys[(size_t)nodes[i] * 32 + 31];
    out[i] = leaf_sizes ? hdr_size(h) : hdr_size(h) + 1;
  }
}

// the children of the level's nodes in order; total: the scan's
__global__ void __launch_bounds__(256) child_write_kernel(DevTree t, const uint32_t* __restrict__ nodes,
                                                          const uint32_t* __restrict__ n_dev,
                                                          const uint32_t* __restrict__ off,
                                                          const uint32_t* __restrict__ total,
                                                          uint32_t* __restrict__ out, uint32_t* __restrict__ cnt_below) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t n = *n_dev;
  if (n == 0) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) *cnt_below = *total;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const uint32_t node = nodes[i];
    const uint32_t sz = hdr_size(t.keys[(size_t)node * 32 + 31]);
    if (lane <= sz) out[off[i] + lane] = (uint32_t)t.vals[(size_t)node * 32 + lane];
  }
}

// all pairs in order, unless there are more than `cap`
__global__ void __launch_bounds__(256) leaf_dump_kernel(DevTree t, const uint32_t* __restrict__ leaves,
                                                        const uint32_t* __restrict__ n_dev,
                                                        const uint32_t* __restrict__ off,
                                                        const uint32_t* __restrict__ total, size_t cap,
                                                        uint64_t* __restrict__ ok, uint64_t* __restrict__ ov) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t n = *n_dev;
  if (*total > cap) return;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const uint32_t node = leaves[i];
    const uint32_t sz = hdr_size(t.keys[(size_t)node * 32 + 31]);
    if (lane < sz) {
      const size_t o = (size_t)off[i] + lane;
      if (ok) ok[o] = t.keys[(size_t)node * 32 + lane];
      if (ov) ov[o] = t.vals[(size_t)node * 32 + lane];
    }
  }
}

inline unsigned blocks_for(size_t n, int per) { return (unsigned)((n + per - 1) / per); }

// ------------------------------------------------------------ top cache ----
// The upper levels of the tree, copied into shared memory by every block of
// the unsorted search: a request descends them there and continues from
// global memory below.  Built per search launch by one block (breadth-first
// from the root, whole levels while they fit kTopNodes, never the leaf
// level), so it always matches the tree that the search reads.
struct TopNode {
  uint64_t keys[31];   // separators; unused slots hold kKeyMax
  uint32_t child[32];  // next cached level: index into the cache; last cached level: node id
  uint32_t pad[2];
};
static_assert(sizeof(TopNode) == 384, "TopNode layout");

__global__ void __launch_bounds__(256) top_build_kernel(DevTree t, TopNode* __restrict__ top,
                                                       TopInfo* __restrict__ info) {
  __shared__ uint32_t ids[kTopNodes];
  __shared__ uint32_t kids[kTopNodes];  // per node: index of its first child in ids
  __shared__ uint32_t ws[32];
  __shared__ uint32_t s_lvl_start, s_lvl_end, s_levels, s_stop;
  const uint32_t root = t.ctrl->root;
  const uint32_t rl = t.ctrl->root_level;
  if (root == kNil || rl < 1) {
    if (threadIdx.x == 0) info->n_levels = 0;
    return;
  }
  if (threadIdx.x == 0) {
    ids[0] = root;
    s_lvl_start = 0;
    s_lvl_end = 1;
    s_levels = 1;
    s_stop = 0;
  }
  __syncthreads();
  // add whole levels while the next one is still an inner level and fits
  for (uint32_t level = rl; level >= 2; level--) {
    const uint32_t a = s_lvl_start, b = s_lvl_end;
    uint32_t total = 0;
    for (uint32_t base = a; base < b; base += blockDim.x) {
      const uint32_t i = base + threadIdx.x;
      const uint32_t c = i < b ? hdr_size(t.keys[(size_t)ids[i] * 32 + 31]) + 1 : 0u;
      uint32_t tot;
      const uint32_t ex = blk_exclusive_sum(c, ws, &tot);
      if (i < b) kids[i] = b + total + ex;
      total += tot;
    }
    __syncthreads();
    if (b + total > (uint32_t)kTopNodes) break;  // uniform: every thread has the same total
    for (uint32_t i = a + threadIdx.x / 32; i < b; i += blockDim.x / 32) {
      const uint32_t lane = threadIdx.x & 31;
      const uint32_t c = hdr_size(t.keys[(size_t)ids[i] * 32 + 31]) + 1;
      if (lane < c) ids[kids[i] + lane] = (uint32_t)t.vals[(size_t)ids[i] * 32 + lane];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      s_lvl_start = b;
      s_lvl_end = b + total;
      s_levels++;
    }
    __syncthreads();
  }
  const uint32_t n_nodes = s_lvl_end, last = s_lvl_start, n_levels = s_levels;
  // kids[] holds the child offsets of every level except the last cached one
  for (uint32_t i = threadIdx.x / 32; i < n_nodes; i += blockDim.x / 32) {
    const uint32_t lane = threadIdx.x & 31;
    const size_t row = (size_t)ids[i] * 32;
    const uint32_t c = hdr_size(t.keys[row + 31]) + 1;
    if (lane < 31) top[i].keys[lane] = t.keys[row + lane];  // slots past the size hold kKeyMax
    uint32_t ch = kNil;
    if (lane < c) ch = i >= last ? (uint32_t)t.vals[row + lane] : kids[i] + lane;
    top[i].child[lane] = ch;
  }
  if (threadIdx.x == 0) {
    info->n_nodes = n_nodes;
    info->n_levels = n_levels;
    info->below_level = rl - n_levels;
  }
}

template <int G, bool kLeafVals>
__global__ void __launch_bounds__(512) search_top_kernel(DevTree t, const TopNode* __restrict__ top,
                                                        const TopInfo* __restrict__ info,
                                                        const uint64_t* __restrict__ qkeys,
                                                        const uint32_t* __restrict__ list,
                                                        const uint32_t* __restrict__ n_dev, size_t n_host,
                                                        uint64_t* __restrict__ out_vals,
                                                        uint8_t* __restrict__ out_st) {
  constexpr int S = 32 / G;
  extern __shared__ __align__(16) unsigned char top_raw[];
  const TopNode* ts = reinterpret_cast<const TopNode*>(top_raw);
  const uint32_t n_levels = info->n_levels;
  const uint32_t n_nodes = n_levels ? info->n_nodes : 0;
  {
    const uint4* src = reinterpret_cast<const uint4*>(top);
    uint4* dst = reinterpret_cast<uint4*>(top_raw);
    const uint32_t words = n_nodes * (uint32_t)(sizeof(TopNode) / 16);
    for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t g = lane % G;
  const uint32_t gmask = group_mask<G>(lane);
  const size_t n = n_dev ? (size_t)*n_dev : n_host;
  const uint32_t root = t.ctrl->root;
  const uint32_t root_level = t.ctrl->root_level;
  const uint32_t below = info->below_level;
  const size_t stride = ((size_t)gridDim.x * blockDim.x) / G;
  for (size_t q = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / G; q < n; q += stride) {
    const uint32_t r = list ? __ldg(list + q) : (uint32_t)q;
    const uint64_t key = __ldg(qkeys + r);
    uint8_t st = kAbsent;
    uint64_t ans = 0;
    if (key == kKeyMax) {
      st = kRejected;
    } else if (root != kNil) {
      uint32_t node = root, level = root_level;
      if (n_levels) {
        uint32_t idx = 0;
        for (uint32_t l = 0; l < n_levels; l++) {
          const TopNode& tn = ts[idx];
          uint32_t c = 0;
#pragma unroll
          for (int i = 0; i < S; i++) {
            const int slot = g * S + i;
            c += (slot < 31 && tn.keys[slot] <= key) ? 1u : 0u;
          }
          c = group_sum<G>(c, gmask);
          idx = tn.child[c];
        }
        node = idx;
        level = below;
      }
      st = group_descend<G, kLeafVals>(t, node, level, key, g, gmask, ans);
    }
    if (g == 0) {
      out_vals[r] = ans;
      out_st[r] = st;
    }
  }
}

// Range scan, one warp per query.  The descent ends at the parent of the leaf
// that holds `lo`: its separators say which of its children meet [lo, hi] (a
// separator is the next child's low fence), so their rows are read one after
// the other with the next one's loads ahead of the current one's work, and only
// past the parent's last child does a new descent follow, from that leaf's
// right fence.  A lane holds one slot; a ballot compacts the keys in [lo, hi] in
// key order.  Inner levels are ranked by the separators' prefixes.  Read-only;
// runs only when no writer is active.
// kFill: the places past a query's pairs are zeroed, so that the caller need
// not clear 16 bytes a place ahead of a kernel that writes most of them again
// (the same scans, pages of 128: 37.9 -> 32.3 us).
// 20,000 scans of about 100 keys on 2^24 keys, with the zero fill of the
// results: 58.5 us with a descent per leaf (a dependent row and child id per
// level), 42.2 with this at 46 registers, 39.4 at the 36 of seven blocks an SM.
template <bool kFill>
__global__ void __launch_bounds__(256, 7) range_kernel(DevTree t, const uint64_t* __restrict__ lo_keys,
                                                   const uint64_t* __restrict__ hi_keys, size_t n, uint32_t max_per,
                                                   uint64_t* __restrict__ out_keys, uint64_t* __restrict__ out_vals,
                                                   uint32_t* __restrict__ out_counts) {
  constexpr unsigned kAll = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t root = t.ctrl->root;
  const uint32_t root_level = t.ctrl->root_level;
  const uint64_t cap_nodes = t.cap;
  const uint64_t keep = l2_keep(), stream = l2_stream();
  const size_t warps = ((size_t)gridDim.x * blockDim.x) >> 5;
  for (size_t q = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < n; q += warps) {
    const uint64_t lo = __ldg(lo_keys + q), hi = __ldg(hi_keys + q);
    uint32_t count = 0;
    uint64_t from = lo;
    bool more = root != kNil && lo <= hi && lo != kKeyMax;  // UINT64_MAX is never a stored key
    for (uint64_t visited = 0; more && visited <= cap_nodes; visited++) {
      // descend to the parent of the leaf holding `from`
      uint32_t node = root;
      for (uint32_t level = root_level; level > 1; level--) {
        const uint32_t p = __ldg(t.pfx + (size_t)node * 32 + lane), kp = (uint32_t)(from >> 32);
        uint32_t c = __popc(__ballot_sync(kAll, p < kp));
        if (__any_sync(kAll, p == kp)) {  // a separator shares the key's prefix: the full keys
          const uint64_t k = ldg_hint(t.keys + (size_t)node * 32 + lane, keep);
          c = __popc(__ballot_sync(kAll, lane < 31 && k <= from));
        }
        node = (uint32_t)ldg_hint(t.vals + (size_t)node * 32 + c, keep);
      }
      // its children c0 .. c1 meet [from, hi]; a tree of one leaf is its only child
      uint32_t c0 = 0, c1 = 0;
      uint64_t kids = node;
      if (root_level > 0) {
        const uint64_t k = ldg_hint(t.keys + (size_t)node * 32 + lane, keep);
        kids = ldg_hint(t.vals + (size_t)node * 32 + lane, keep);
        c0 = __popc(__ballot_sync(kAll, lane < 31 && k <= from));
        c1 = __popc(__ballot_sync(kAll, lane < 31 && k <= hi && k != kKeyMax));  // slots past the size hold kKeyMax
      }
      uint32_t leaf = (uint32_t)__shfl_sync(kAll, kids, c0);
      uint64_t k = ldg_hint(t.keys + (size_t)leaf * 32 + lane, stream);
      uint64_t v = ldg_hint(t.vals + (size_t)leaf * 32 + lane, stream);
      uint64_t fence = kKeyMax;
      for (uint32_t c = c0; c <= c1; c++) {
        uint64_t k2 = 0, v2 = 0;
        if (c < c1) {
          leaf = (uint32_t)__shfl_sync(kAll, kids, c + 1);
          k2 = ldg_hint(t.keys + (size_t)leaf * 32 + lane, stream);
          v2 = ldg_hint(t.vals + (size_t)leaf * 32 + lane, stream);
        }
        const uint32_t size = hdr_size(__shfl_sync(kAll, k, 31));
        if (c == c1) fence = __shfl_sync(kAll, v, 31);
        const bool in = lane < size && lane < 31 && k >= lo && k <= hi;
        const uint32_t m = __ballot_sync(kAll, in);
        if (in) {
          const uint32_t pos = count + __popc(m & ((1u << lane) - 1u));
          if (pos < max_per) {
            out_keys[q * max_per + pos] = k;
            out_vals[q * max_per + pos] = v;
          }
        }
        count += __popc(m);
        k = k2;
        v = v2;
      }
      // the next leaf starts at the fence; stop when it lies past hi
      more = fence != kKeyMax && fence <= hi && fence > from;
      from = fence;
    }
    if (lane == 0) out_counts[q] = count;
    if (kFill)
      for (uint64_t pos = (uint64_t)count + lane; pos < max_per; pos += 32) {
        out_keys[q * max_per + pos] = 0;
        out_vals[q * max_per + pos] = 0;
      }
  }
}

}  // namespace

int top_alloc(Handle* h) {
  if (h->top) return 0;
  if (cudaMalloc(&h->top, (size_t)kTopNodes * sizeof(TopNode) + 64) != cudaSuccess) return -3;
  h->top_info = reinterpret_cast<TopInfo*>(static_cast<char*>(h->top) + (size_t)kTopNodes * sizeof(TopNode));
  return 0;
}

// unsorted search with the top levels in shared memory
cudaError_t launch_search_top(Handle* h, const uint64_t* qkeys, const uint32_t* list, const uint32_t* n_dev,
                              size_t n, uint64_t* out_vals, uint8_t* out_st, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  if (top_alloc(h) != 0) return cudaErrorMemoryAllocation;
  TopNode* top = reinterpret_cast<TopNode*>(h->top);
  top_build_kernel<<<1, 256, 0, s>>>(h->tree, top, h->top_info);
  count_launch();
  const int threads = 512;
  const size_t smem = (size_t)kTopNodes * sizeof(TopNode);
  const int G = h->search_group;
  static int per_sm[64][5] = {};
  const int gi = G == 4 ? 0 : G == 16 ? 2 : G == 32 ? 3 : G == -8 ? 4 : 1;
  const void* kern;
  switch (gi) {
    case 0: kern = (const void*)search_top_kernel<4, false>; break;
    case 2: kern = (const void*)search_top_kernel<16, false>; break;
    case 3: kern = (const void*)search_top_kernel<32, false>; break;
    case 4: kern = (const void*)search_top_kernel<8, true>; break;
    default: kern = (const void*)search_top_kernel<8, false>; break;
  }
  const int dev = h->device;
  int per = 1;
  if (dev >= 0 && dev < 64 && per_sm[dev][gi]) {
    per = per_sm[dev][gi];
  } else {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return cudaErrorInvalidValue;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem) != cudaSuccess || per < 1) per = 1;
    if (dev >= 0 && dev < 64) per_sm[dev][gi] = per;
  }
  const int lanes = G < 0 ? -G : G;
  size_t blocks = (n * (size_t)lanes + threads - 1) / threads;
  const size_t cap = (size_t)h->sm_count * per;
  if (blocks > cap) blocks = cap;
  if (blocks == 0) blocks = 1;
  DevTree tree = h->tree;
  const TopInfo* info = h->top_info;
  void* args[] = {&tree, &top, &info, (void*)&qkeys, (void*)&list, (void*)&n_dev, &n, &out_vals, &out_st};
  cudaError_t e = cudaLaunchKernel(kern, dim3((unsigned)blocks), dim3(threads), args, smem, s);
  count_launch();
  return e;
}

__global__ void clear_headers_kernel(DevTree t, uint32_t first, uint32_t last) {
  for (size_t i = (size_t)first + (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < last;
       i += (size_t)gridDim.x * blockDim.x)
    t.keys[i * 32 + 31] = 0;
}

cudaError_t clear_headers(Handle* h, uint32_t first, uint32_t last, cudaStream_t s) {
  if (first >= last) return cudaSuccess;
  const size_t n = last - first;
  const unsigned blocks = (unsigned)min((size_t)h->sm_count * 8, (n + 255) / 256);
  clear_headers_kernel<<<blocks, 256, 0, s>>>(h->tree, first, last);
  count_launch();
  return cudaGetLastError();
}

cudaError_t tree_reset(Handle* h, cudaStream_t s) {
  h->has_root = false;
  // The epoch has 15 bits (1 .. 0x7fff; 0 marks never-written rows).  When
  // it comes round to 1 again, rows written by the trees of the last cycle
  // may still carry that number: clear every row's header first, so that a
  // reader which reaches a row without a validated path (the optimistic STM
  // descent, the learned leaf guess) cannot take a row of an older tree for
  // one of the new tree.
  if (h->epoch == 0x7fffu) {
    const cudaError_t e = clear_headers(h, 0, h->tree.cap, s);
    if (e != cudaSuccess) return e;
  }
  h->epoch = (h->epoch % 0x7fffu) + 1;
  reset_kernel<<<1, 1, 0, s>>>(h->tree.ctrl, h->epoch);
  count_launch();
  return cudaGetLastError();
}

// Bulk loader: replaces the contents.  Same packing rule as the oracle
// (bto_bulk_build): ceil(m/leaf_fill) leaves of even size, inner levels of
// inner_fill+1 children per node, leaves first in id order.  The scratch is the
// caller's; nothing is allocated.
int tree_bulk_build_scratch(Handle* h, const uint64_t* keys, const uint64_t* vals, size_t n, cudaStream_t s,
                            const BuildScratch& sc) {
  if (n > sc.cap) return -6;
  if (tree_reset(h, s) != cudaSuccess) return -2;
  if (n == 0) return cudaStreamSynchronize(s) == cudaSuccess ? 0 : -2;
  uint64_t* sk = nullptr;
  uint32_t* si = nullptr;
  if (radix_sort_pairs(keys, nullptr, nullptr, sc.ka, sc.va, sc.kb, sc.vb, n, 0, 64, sc.sort_scratch, s, &sk, &si,
                       &h->tree.ctrl->error) != cudaSuccess)
    return -2;
  uint64_t* uk = (sk == sc.ka) ? sc.kb : sc.ka;
  BuildGeo* geo = reinterpret_cast<BuildGeo*>(sc.tot);
  uint32_t* m = &geo->m;  // the scan's total
  const unsigned tiles = blocks_for(n, kDedupeTile);
  tail_count_kernel<<<tiles, kDedupeThreads, 0, s>>>(sk, n, sc.pos);
  count_launch();
  if (scan_exclusive_u32(sc.pos, sc.pos, tiles, m, sc.sort_scratch, s) != cudaSuccess) return -2;
  dedupe_kernel<<<tiles, kDedupeThreads, 0, s>>>(sk, si, vals, n, sc.pos, uk, sc.uv);
  const uint32_t lf = h->leaf_fill, per = h->inner_fill + 1;
  build_geo_kernel<<<1, 1, 0, s>>>(geo, m, sk + (n - 1), lf, per, h->tree.cap);
  // the grids for n distinct keys
  size_t nodes = (n + lf - 1) / lf;
  build_leaves_kernel<<<blocks_for(nodes * 32, 256), 256, 0, s>>>(h->tree, uk, sc.uv, geo, h->epoch);
  count_launch(3);
  uint32_t level = 1;
  for (nodes = (nodes + per - 1) / per; nodes > kBuildTopNodes; nodes = (nodes + per - 1) / per, level++) {
    build_inner_kernel<<<blocks_for(nodes * 32, 256), 256, 0, s>>>(h->tree, geo, level, h->epoch);
    count_launch();
  }
  build_top_kernel<<<1, 1024, 0, s>>>(h->tree, geo, level, h->epoch);
  count_launch();
  uint32_t* status = h->pin;
  if (cudaGetLastError() != cudaSuccess ||
      cudaMemcpyAsync(status, &geo->status, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return -2;
  h->has_root = *status == 0;
  return *status == kBuildReserved ? -5 : *status == kBuildCapacity ? -4 : 0;
}

// Scratch of the builds of more than max_batch keys: one pool per device, shared
// by its handles, which keeps up to kBuildKeep bytes between builds (a pool that
// gives its memory back at every synchronisation maps and unmaps it per build:
// most of the 1.0 ms that a load of 2^20 keys spent outside its kernels).  With a
// pool for each handle, as many times kBuildKeep stayed mapped as there were large
// trees.  The last handle that used it gives it back; the allocator orders reuse
// between streams and threads.
constexpr uint64_t kBuildKeep = 1ull << 30;
constexpr int kPoolDevices = 64;
struct BuildPool {
  cudaMemPool_t pool = nullptr;
  unsigned users = 0;
};
static std::mutex g_pool_mu;
static BuildPool g_pools[kPoolDevices];

// the handle's share; the device's default pool where there is no table for it
static bool build_pool_take(Handle* h) {
  if (h->build_pool) return true;
  if (h->device < 0 || h->device >= kPoolDevices) return cudaDeviceGetDefaultMemPool(&h->build_pool, h->device) == cudaSuccess;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  BuildPool& p = g_pools[h->device];
  if (p.users == 0) {
    cudaMemPoolProps pp{};
    pp.allocType = cudaMemAllocationTypePinned;
    pp.handleTypes = cudaMemHandleTypeNone;
    pp.location.type = cudaMemLocationTypeDevice;
    pp.location.id = h->device;
    uint64_t keep = kBuildKeep;
    if (cudaMemPoolCreate(&p.pool, &pp) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  p.users++;
  h->build_pool = p.pool;
  return true;
}

void build_pool_drop(Handle* h) {
  if (!h->build_pool || h->device < 0 || h->device >= kPoolDevices) return;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  BuildPool& p = g_pools[h->device];
  h->build_pool = nullptr;
  if (--p.users == 0) {
    cudaMemPoolDestroy(p.pool);
    p.pool = nullptr;
  }
}

// The same with the library's scratch: up to max_batch keys in the batch work
// buffers, more in one block of the device's pool.
int tree_bulk_build(Handle* h, const uint64_t* keys, const uint64_t* vals, size_t n, cudaStream_t s) {
  // the contents are gone in these cases too: a call on another stream may
  // follow at once and has to meet the new tree, not the old one (a captured
  // reset has nothing to wait for)
  auto emptied = [&](int rc) {
    bool captured = false;
    if (tree_reset(h, s) != cudaSuccess || stream_captured(s, &captured) != cudaSuccess) return -2;
    return captured || cudaStreamSynchronize(s) == cudaSuccess ? rc : -2;
  };
  if (n == 0 || n > 0xFFFFFFFFull / 2) return emptied(n ? -1 : 0);
  Work& w = h->w;
  BuildScratch sc;
  sc.tot = h->geo;
  if (n <= w.cap) {
    sc.ka = w.k_a;
    sc.kb = w.k_b;
    sc.va = w.v_a;
    sc.vb = w.v_b;
    sc.sort_scratch = w.sort_scratch;
    sc.pos = w.f_pos;
    sc.uv = w.uvals;
    sc.cap = w.cap;
    return tree_bulk_build_scratch(h, keys, vals, n, s, sc);
  }
  auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t kb = up(n * 8), vb = up(n * 4), pb = up((n / kDedupeTile + 2) * 4);
  char* slab = nullptr;
  if (!build_pool_take(h) ||
      cudaMallocFromPoolAsync((void**)&slab, 3 * kb + 2 * vb + pb + up(sort_scratch_words(n) * 4), h->build_pool, s) !=
      cudaSuccess) {
    cudaGetLastError();
    return emptied(-3);
  }
  char* at = slab;
  auto take = [&](size_t b) {
    char* p = at;
    at += b;
    return p;
  };
  sc.ka = (uint64_t*)take(kb);
  sc.kb = (uint64_t*)take(kb);
  sc.uv = (uint64_t*)take(kb);
  sc.va = (uint32_t*)take(vb);
  sc.vb = (uint32_t*)take(vb);
  sc.pos = (uint32_t*)take(pb);
  sc.sort_scratch = (uint32_t*)at;
  sc.cap = n;
  const int rc = tree_bulk_build_scratch(h, keys, vals, n, s, sc);
  cudaFreeAsync(slab, s);
  return rc;
}

cudaError_t launch_search_sorted(Handle* h, const uint64_t* qkeys, const uint32_t* list, const uint32_t* n_dev,
                                 size_t n, uint64_t* out_vals, uint8_t* out_st, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  // one resident wave of groups; each group takes a contiguous chunk
  const int threads = 256;
  static int per_sm[64][2] = {};
  const int lv = h->sorted_leaf_vals ? 1 : 0;
  if (h->device < 64 && per_sm[h->device][lv] == 0) {
    int b = 0;
    cudaError_t e = lv ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, search_sorted_kernel<8, true>, threads, 0)
                       : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, search_sorted_kernel<8, false>, threads, 0);
    if (e != cudaSuccess || b < 1) b = 4;
    per_sm[h->device][lv] = b;
  }
  const size_t blocks = (size_t)h->sm_count * (h->device < 64 ? per_sm[h->device][lv] : 4);
  if (lv) search_sorted_kernel<8, true><<<(unsigned)blocks, threads, 0, s>>>(h->tree, qkeys, list, n_dev, n, out_vals, out_st);
  else search_sorted_kernel<8, false><<<(unsigned)blocks, threads, 0, s>>>(h->tree, qkeys, list, n_dev, n, out_vals, out_st);
  count_launch();
  return cudaGetLastError();
}

// Prefix rows of the inner nodes and fingerprint rows of the leaves from their
// keys: one warp per 32 nodes reads their headers (one sector each), then
// writes the rows one by one.
__global__ void __launch_bounds__(256) pfx_rebuild_kernel(DevTree t) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t n_nodes = min(t.ctrl->n_nodes, t.cap);
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t b = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; b < n_nodes; b += warps * 32) {
    const uint32_t mine = b + lane;
    const bool inner = mine < n_nodes && hdr_level(t.keys[(size_t)mine * 32 + 31]) > 0;
    const uint32_t inners = __ballot_sync(0xffffffffu, inner);
    const uint32_t m = min(32u, n_nodes - b);
    for (uint32_t i = 0; i < m; i++) {
      const size_t at = (size_t)(b + i) * 32 + lane;
      const uint64_t k = t.keys[at];
      if ((inners >> i) & 1u) t.pfx[at] = lane < 31 ? (uint32_t)(k >> 32) : 0xffffffffu;
      else t.fp[at] = lane < 31 ? slot_fp(k) : (uint8_t)0;
    }
  }
}

cudaError_t rebuild_tables(Handle* h, cudaStream_t s) {
  pfx_rebuild_kernel<<<(unsigned)h->sm_count * 8, 256, 0, s>>>(h->tree);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_search(Handle* h, const uint64_t* qkeys, const uint32_t* list, const uint32_t* n_dev, size_t n,
                          uint64_t* out_vals, uint8_t* out_st, cudaStream_t s, const uint64_t* ckeys) {
  if (n == 0) return cudaSuccess;
  if (h->search_pairs && (h->search_group == 8 || h->search_group == 4 || h->search_group == 16)) {
    const int threads = 256;
    const int G = h->search_group;
    const bool child = h->search_pairs == 2;
    // the separators' prefixes and the leaves' fingerprints (child-id form only)
    const int use_pfx = child && h->use_pfx ? 1 : 0;
    const bool warp = use_pfx && G == 4 && n >= kWarpLookupMin;
    const size_t per_block = warp ? threads : 2 * threads / G;
    size_t blocks = (n + per_block - 1) / per_block;
    size_t cap = (size_t)h->sm_count * 8 * 4;
    if (h->lookup_reserve > 0) {
      // a resident, grid-striding launch that leaves `lookup_reserve` block
      // slots free for kernels running beside it (the overlapped sort)
      static int per_sm[64][4] = {};
      const int gi = warp ? 3 : G == 4 ? 0 : G == 16 ? 2 : 1;
      const int dev = h->device;
      int per = (dev >= 0 && dev < 64) ? per_sm[dev][gi] : 0;
      if (per == 0) {
        const void* k = warp ? (const void*)search_warp_kernel
                        : G == 4 ? (const void*)search2_kernel<4, false, true>
                        : G == 16 ? (const void*)search2_kernel<16, false, true>
                                  : (const void*)search2_kernel<8, false, true>;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, threads, 0) != cudaSuccess || per < 1) per = 1;
        if (dev >= 0 && dev < 64) per_sm[dev][gi] = per;
      }
      const size_t resident = (size_t)h->sm_count * per;
      cap = resident > (size_t)h->lookup_reserve + h->sm_count ? resident - h->lookup_reserve : h->sm_count;
    }
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    if (warp) {
      search_warp_kernel<<<(unsigned)blocks, threads, 0, s>>>(h->tree, qkeys, list, n_dev, n, out_vals, out_st,
                                                              list ? ckeys : nullptr);
      count_launch();
      return cudaGetLastError();
    }
#define BT_S2(GG, CC) search2_kernel<GG, false, CC><<<(unsigned)blocks, threads, 0, s>>>(h->tree, qkeys, list, n_dev, n, out_vals, out_st, use_pfx, list ? ckeys : nullptr)
    if (G == 4) { if (child) BT_S2(4, true); else BT_S2(4, false); }
    else if (G == 16) { if (child) BT_S2(16, true); else BT_S2(16, false); }
    else { if (child) BT_S2(8, true); else BT_S2(8, false); }
#undef BT_S2
    count_launch();
    return cudaGetLastError();
  }
  if (h->top_cache) return launch_search_top(h, qkeys, list, n_dev, n, out_vals, out_st, s);
  const int threads = 256;
  const int G = h->search_group;
  // enough groups to cover the requests, capped at a few waves of resident blocks
  size_t groups_needed = n;
  size_t blocks = (groups_needed * G + threads - 1) / threads;
  size_t cap = (size_t)h->sm_count * 8 * 4;
  if (blocks > cap) blocks = cap;
  if (blocks == 0) blocks = 1;
  switch (G) {
    case 4: search_kernel<4, false><<<(unsigned)blocks, threads, 0, s>>>(h->tree, qkeys, list, n_dev, n, out_vals, out_st); break;
    case 16: search_kernel<16, false><<<(unsigned)blocks, threads, 0, s>>>(h->tree, qkeys, list, n_dev, n, out_vals, out_st); break;
    case 32: search_kernel<32, false><<<(unsigned)blocks, threads, 0, s>>>(h->tree, qkeys, list, n_dev, n, out_vals, out_st); break;
    case -8: search_kernel<8, true><<<(unsigned)blocks, threads, 0, s>>>(h->tree, qkeys, list, n_dev, n, out_vals, out_st); break;
    default: search_kernel<8, false><<<(unsigned)blocks, threads, 0, s>>>(h->tree, qkeys, list, n_dev, n, out_vals, out_st); break;
  }
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_range(Handle* h, const uint64_t* lo, const uint64_t* hi, size_t n, uint32_t max_per,
                         uint64_t* out_keys, uint64_t* out_vals, uint32_t* out_counts, bool fill, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  size_t blocks = (n * 32 + 255) / 256;
  const size_t cap = (size_t)h->sm_count * 16;
  if (blocks > cap) blocks = cap;
  const auto kernel = fill ? range_kernel<true> : range_kernel<false>;
  kernel<<<(unsigned)blocks, 256, 0, s>>>(h->tree, lo, hi, n, max_per, out_keys, out_vals, out_counts);
  count_launch();
  return cudaGetLastError();
}

// grown with a quarter of headroom: the tree grows a little with every batch,
// and a reallocation (cudaFree synchronises the device) on every refit or
// dump stalled the batches queued behind it
static int ensure_enum(Handle* h, size_t n, cudaStream_t s) {
  if (n <= h->enum_cap) return 0;
  n += n / 4 + 4096;
  cudaFree(h->enum_a);
  cudaFree(h->enum_b);
  cudaFree(h->enum_cnt);
  cudaFree(h->enum_lb);
  h->enum_a = h->enum_b = h->enum_cnt = nullptr;
  h->enum_lb = nullptr;
  h->enum_cap = 0;
  const size_t c = n + 64, lb = scan_lb_words(c) + kLbCtrWords;  // the last ones: the scan's counters
  if (cudaMalloc(&h->enum_a, c * 4) != cudaSuccess || cudaMalloc(&h->enum_b, c * 4) != cudaSuccess ||
      cudaMalloc(&h->enum_cnt, c * 4) != cudaSuccess || cudaMalloc(&h->enum_lb, lb * 8) != cudaSuccess ||
      cudaMemsetAsync(h->enum_lb, 0, lb * 8, s) != cudaSuccess)
    return -3;
  h->enum_cap = c;
  h->enum_lb_words = lb;
  return 0;
}

static cudaError_t enum_scan(Handle* h, uint32_t* x, const uint32_t* n_dev, size_t n_upper, uint32_t* total,
                             cudaStream_t s) {
  uint64_t* ctr = h->enum_lb + h->enum_lb_words - kLbCtrWords;
  return scan_exclusive_u32_lb(x, x, n_upper, n_dev, total, h->enum_lb, ctr, &h->tree.ctrl->error, s);
}

// words of the handle's small device block (h->geo) that the enumeration uses
constexpr int kEnumWords = 64;  // [0, 48) counts per level, [48] entries of this level, [49] total

// The leaves' ids in key order in *leaf_ids, their count in cnt[0] on the
// device; one read back (the control block), no other wait.  *root_level < 0:
// an empty tree.  Without `ids` a tree of one leaf needs no kernel.
static int enumerate_queue(Handle* h, cudaStream_t s, uint32_t** leaf_ids, size_t* n_nodes, int* root_level,
                           bool ids = true) {
  Ctrl* c = reinterpret_cast<Ctrl*>(h->pin);
  if (cudaMemcpyAsync(c, h->tree.ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, s) != cudaSuccess) return -2;
  if (cudaStreamSynchronize(s) != cudaSuccess) return -2;
  *leaf_ids = nullptr;
  *root_level = -1;
  *n_nodes = 0;
  h->n_levels = 0;
  if (c->root == kNil) return 0;
  const uint32_t rl = c->root_level;
  if (rl >= 48) return -2;
  const size_t nn = c->n_nodes < h->tree.cap ? c->n_nodes : h->tree.cap;
  h->n_levels = rl + 1;
  if (rl == 0 && !ids) {
    *root_level = 0;
    return 0;
  }
  if (ensure_enum(h, nn + 1, s) != 0) return -3;
  uint32_t* cnt = h->geo;
  uint32_t* cur = h->enum_a;
  uint32_t* nxt = h->enum_b;
  enum_top_kernel<<<1, 1024, 0, s>>>(h->tree, rl, cur, nxt, cnt);
  count_launch();
  const unsigned grid = (unsigned)min((size_t)h->sm_count * 8, nn / 8 + 1);
  for (uint32_t l = rl; l > 0; l--) {
    // levels surely below the block's limit need no launches: every inner node
    // has two children or more (unless the loader ever packed one per node)
    size_t bound = nn;
    for (uint32_t x = 0; x < l && h->inner_min >= 2; x++) bound = (bound + 1) / 2;
    if (bound > kEnumTop) {
      child_count_kernel<<<grid, 256, 0, s>>>(h->tree, cur, cnt, l, rl, h->enum_cnt, cnt + 48, 0);
      count_launch();
      if (enum_scan(h, h->enum_cnt, cnt + 48, bound, cnt + 49, s) != cudaSuccess) return -2;
      child_write_kernel<<<grid, 256, 0, s>>>(h->tree, cur, cnt + 48, h->enum_cnt, cnt + 49, nxt, cnt + l - 1);
      count_launch();
    }
    uint32_t* x = cur;
    cur = nxt;
    nxt = x;
  }
  *leaf_ids = cur;
  *n_nodes = nn;
  *root_level = (int)rl;
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int enumerate_leaves(Handle* h, cudaStream_t s, uint32_t** leaf_ids, size_t* n_leaves) {
  size_t nn = 0;
  int rl = -1;
  *n_leaves = 0;
  uint32_t* none = nullptr;
  const int rc = enumerate_queue(h, s, leaf_ids ? leaf_ids : &none, &nn, &rl, leaf_ids != nullptr);
  if (rc || rl < 0) return rc;
  if (rl == 0) {  // the root is the only leaf: no counts to read
    h->level_counts[0] = 1;
    *n_leaves = 1;
    return 0;
  }
  if (cudaMemcpyAsync(h->pin, h->geo, kEnumWords * 4, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return -2;
  for (int l = 0; l <= rl; l++) h->level_counts[l] = h->pin[l];
  *n_leaves = h->pin[0];
  return 0;
}

cudaError_t leaf_sizes_device(Handle* h, const uint32_t* leaves, size_t n, uint32_t* out, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  child_count_kernel<<<(unsigned)min((size_t)h->sm_count * 8, (n + 255) / 256), 256, 0, s>>>(
      h->tree, leaves, h->geo, 0, 0, out, h->geo + 48, 1);
  count_launch();
  return cudaGetLastError();
}

int tree_dump(Handle* h, uint64_t* out_keys, uint64_t* out_vals, size_t cap, size_t* n_out, cudaStream_t s) {
  uint32_t* leaves = nullptr;
  size_t nn = 0;
  int rl = -1;
  *n_out = 0;
  const int rc = enumerate_queue(h, s, &leaves, &nn, &rl);
  if (rc || rl < 0) return rc;
  uint32_t* cnt = h->geo;
  const unsigned grid = (unsigned)min((size_t)h->sm_count * 8, nn / 8 + 1);
  // the counts per parent are done with: the leaves' sizes take their place
  child_count_kernel<<<grid, 256, 0, s>>>(h->tree, leaves, cnt, 0, 0, h->enum_cnt, cnt + 48, 1);
  count_launch();
  if (enum_scan(h, h->enum_cnt, cnt + 48, nn, cnt + 49, s) != cudaSuccess) return -2;
  leaf_dump_kernel<<<grid, 256, 0, s>>>(h->tree, leaves, cnt + 48, h->enum_cnt, cnt + 49, cap, out_keys, out_vals);
  count_launch();
  if (cudaGetLastError() != cudaSuccess ||
      cudaMemcpyAsync(h->pin, cnt, kEnumWords * 4, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return -2;
  for (int l = 0; l <= rl; l++) h->level_counts[l] = h->pin[l];
  *n_out = h->pin[49];
  return *n_out > cap ? -4 : 0;
}

}  // namespace bt
