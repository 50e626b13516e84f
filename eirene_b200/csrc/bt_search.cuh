// Grouped lock-free descent shared by the plain search kernel and the learned
// search's fallback.  A group of G lanes serves one request; each lane owns
// S = 32/G consecutive slots of a node row and loads them with 16-byte loads.
// Valid only while no writer runs (the batch executor never overlaps this with
// the STM insert phase); the loads are ordinary ones, not ld.global.nc, because
// a kernel may be resident before the one that wrote the rows has ended.
#pragma once
#include "bt_common.cuh"

namespace bt {

template <int G>
__device__ __forceinline__ uint32_t group_mask(uint32_t lane) {
  if constexpr (G == 32) return 0xffffffffu;
  else return ((1u << G) - 1u) << (lane - lane % G);
}

template <int S>
__device__ __forceinline__ void load_slots(const uint64_t* p, uint64_t (&x)[S]) {
  if constexpr (S == 1) {
    x[0] = *p;
  } else {
#pragma unroll
    for (int i = 0; i < S; i += 2) {
      ulonglong2 w = *reinterpret_cast<const ulonglong2*>(p + i);
      x[i] = w.x;
      x[i + 1] = w.y;
    }
  }
}

// L2 eviction priorities for the descent (createpolicy + ld.global with an
// L2 cache hint, PTX ISA 7.4+): inner rows are read by every lookup and
// should stay in L2 (evict_last); a leaf row or value is read once per
// lookup and should not push them out (evict_first).
__device__ __forceinline__ uint64_t l2_keep() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

__device__ __forceinline__ uint64_t l2_stream() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}

__device__ __forceinline__ uint64_t ldg_hint(const uint64_t* p, uint64_t pol) {
  uint64_t r;
  asm("ld.global.L2::cache_hint.u64 %0, [%1], %2;" : "=l"(r) : "l"(p), "l"(pol));
  return r;
}

__device__ __forceinline__ ulonglong2 ldg2_hint(const void* p, uint64_t pol) {
  ulonglong2 r;
  asm("ld.global.L2::cache_hint.v2.u64 {%0, %1}, [%2], %3;" : "=l"(r.x), "=l"(r.y) : "l"(p), "l"(pol));
  return r;
}

template <int S>
__device__ __forceinline__ void load_slots_hint(const uint64_t* p, uint64_t (&x)[S], uint64_t pol) {
  if constexpr (S == 1) {
    x[0] = ldg_hint(p, pol);
  } else {
#pragma unroll
    for (int i = 0; i < S; i += 2)
      asm("ld.global.L2::cache_hint.v2.u64 {%0, %1}, [%2], %3;"
          : "=l"(x[i]), "=l"(x[i + 1])
          : "l"(p + i), "l"(pol));
  }
}

// A row of 32 slots read by a group of G lanes in 16-byte chunks interleaved
// across the lanes: load i of lane g reads chunk i * G + g (slots 2(iG + g)
// and 2(iG + g) + 1), so one warp-wide load instruction covers one contiguous
// 16G-byte piece of each group's row instead of G pieces 64 bytes apart:
// half the 128-byte lines per instruction at G = 4, the unit the L1 data
// pipe works in.  Slot s lives in lane (s / 2) % G, element 2 * (s / 2 / G) +
// s % 2; slot 31 (the header) in lane G - 1, element S - 1.
template <int G>
__device__ __forceinline__ void load_row_il(const uint64_t* row, uint32_t g, uint64_t (&x)[32 / G], uint64_t pol) {
  constexpr int S = 32 / G;
  if constexpr (S == 1) {
    x[0] = ldg_hint(row + g, pol);
  } else {
#pragma unroll
    for (int i = 0; i < S / 2; i++)
      asm("ld.global.L2::cache_hint.v2.u64 {%0, %1}, [%2], %3;"
          : "=l"(x[2 * i]), "=l"(x[2 * i + 1])
          : "l"(row + 2 * (i * G + g)), "l"(pol));
  }
}

// owner lane and element of slot s in an interleaved row
template <int G>
__device__ __forceinline__ uint32_t il_lane(uint32_t s) {
  return G == 32 ? s : (s >> 1) % G;
}
template <int G>
__device__ __forceinline__ uint32_t il_elem(uint32_t s) {
  return G == 32 ? 0 : 2 * ((s >> 1) / G) + (s & 1);
}

// S 32-bit separator prefixes of a row (S = 2, 4 or 8)
template <int S>
__device__ __forceinline__ void load_pfx(const uint32_t* p, uint32_t (&x)[S], uint64_t pol) {
  if constexpr (S == 2) {
    asm("ld.global.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;" : "=r"(x[0]), "=r"(x[1]) : "l"(p), "l"(pol));
  } else {
#pragma unroll
    for (int i = 0; i < S; i += 4)
      asm("ld.global.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
          : "=r"(x[i]), "=r"(x[i + 1]), "=r"(x[i + 2]), "=r"(x[i + 3])
          : "l"(p + i), "l"(pol));
  }
}

template <int S>
__device__ __forceinline__ uint64_t pick(const uint64_t (&x)[S], uint32_t e) {
  uint64_t r = x[0];
#pragma unroll
  for (int i = 1; i < S; i++)
    if (e == (uint32_t)i) r = x[i];
  return r;
}

template <int G>
__device__ __forceinline__ uint32_t group_sum(uint32_t c, uint32_t gmask) {
#pragma unroll
  for (int o = G / 2; o >= 1; o >>= 1) c += __shfl_xor_sync(gmask, c, o, G);
  return c;
}

// Rank of `key` in an inner row from the prefixes: slots whose prefix is
// below the key's count, slots with an equal prefix are counted in bits
// 16.. (the caller then ranks with the full keys); slot 31 is the header.
template <int G, int S>
__device__ __forceinline__ uint32_t pfx_rank(const uint32_t (&p)[S], uint64_t key, uint32_t g, uint32_t gmask) {
  const uint32_t kp = (uint32_t)(key >> 32);
  uint32_t x = 0;
#pragma unroll
  for (int i = 0; i < S; i++)
    if (!(g == (uint32_t)(G - 1) && i == S - 1)) x += p[i] < kp ? 1u : (p[i] == kp ? 0x10000u : 0u);
  return group_sum<G>(x, gmask);
}

// ---- leaf lookup by one thread (DevTree::fp) ----
// 32 bytes in one load
__device__ __forceinline__ void ldg32_hint(const void* p, uint64_t (&x)[4], uint64_t pol) {
  asm("ld.global.L2::cache_hint.v4.u64 {%0, %1, %2, %3}, [%4], %5;"
      : "=l"(x[0]), "=l"(x[1]), "=l"(x[2]), "=l"(x[3])
      : "l"(p), "l"(pol));
}

// the slots of a fingerprint row whose byte equals q, as bits 0 .. 30
__device__ __forceinline__ uint32_t fp_match(const uint64_t (&row)[4], uint32_t q) {
  const uint32_t qq = q * 0x01010101u;
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const uint32_t x = (uint32_t)(row[i >> 1] >> (32 * (i & 1))) ^ qq;
    // a byte's top bit set: the byte is zero (no carry leaves a byte)
    const uint32_t z = ~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x) & 0x80808080u;
    m |= ((z >> 7) * 0x10204080u >> 28) << (4 * i);
  }
  return m & 0x7fffffffu;
}

// The key in the matching slots m of leaf `node`: the first two candidates'
// keys and values are loaded at once (a wrong first one: one lookup in ten;
// a third one: one in 250).
__device__ __forceinline__ bool leaf_pick(const DevTree& t, uint32_t node, uint64_t key, uint32_t m, uint64_t pol,
                                          uint64_t& val, uint32_t& slot) {
  const uint64_t* kr = t.keys + (size_t)node * 32;
  const uint64_t* vr = t.vals + (size_t)node * 32;
  val = 0;
  while (m) {
    const uint32_t s0 = __ffs(m) - 1;
    m &= m - 1;
    const uint32_t s1 = m ? __ffs(m) - 1 : s0;
    const uint64_t k0 = ldg_hint(kr + s0, pol), v0 = ldg_hint(vr + s0, pol);
    uint64_t k1 = k0, v1 = v0;
    if (s1 != s0) {
      k1 = ldg_hint(kr + s1, pol);
      v1 = ldg_hint(vr + s1, pol);
    }
    m &= m - 1;
    if (k0 == key || k1 == key) {
      val = k0 == key ? v0 : v1;
      slot = k0 == key ? s0 : s1;
      return true;
    }
  }
  return false;
}
__device__ __forceinline__ bool leaf_pick(const DevTree& t, uint32_t node, uint64_t key, uint32_t m, uint64_t pol,
                                          uint64_t& val) {
  uint32_t slot;
  return leaf_pick(t, node, key, m, pol, val, slot);
}

// ---- descent of 32 keys by one warp ----
// Lane l owns key l and its node.  At each inner level the warp ranks the keys
// eight at a time, four lanes to a key: a lane compares eight of the row's
// separator prefixes by binary search in registers, the four turns' counts are
// packed into one word (a byte each) and summed over the lanes together, and
// the owner takes its byte and loads its child id.  All lanes stay in step
// (the tree is of one height): full-mask shuffles, no divergence.  A prefix
// equal to a key's (flagged in the byte's upper bits) makes the warp rank that
// level with the full keys.
constexpr uint32_t kEqBit = 0x20u;  // a lane's flag in its byte: four of them still fit

// prefixes below kp among eight ascending ones, kEqBit added if one equals it
__device__ __forceinline__ uint32_t rank8(const uint32_t (&p)[8], uint32_t kp) {
  const bool c1 = p[3] < kp;
  uint32_t ub = c1 ? p[7] : p[3];  // the smallest one seen that is not below kp (or p[7])
  const uint32_t a = c1 ? p[5] : p[1], b0 = c1 ? p[4] : p[0], b1 = c1 ? p[6] : p[2];
  const bool c2 = a < kp;
  ub = c2 ? ub : a;
  const uint32_t b = c2 ? b1 : b0;
  const bool c3 = b < kp;
  ub = c3 ? ub : b;
  return (c1 ? 4u : 0u) + (c2 ? 2u : 0u) + (c3 ? 1u : 0u) + (p[7] < kp ? 1u : 0u) + (ub == kp ? kEqBit : 0u);
}

// every lane of the warp calls it, with any key; returns the lane's leaf;
// visit(level, node): the inner nodes on the lane's way
template <typename F>
__device__ __forceinline__ uint32_t warp_descend(const DevTree& t, uint32_t root, uint32_t root_level, uint64_t key,
                                                 F visit) {
  const uint32_t lane = threadIdx.x & 31, g = lane & 3u;
  const uint64_t keep = l2_keep();
  uint32_t kp[4];
#pragma unroll
  for (int j = 0; j < 4; j++) kp[j] = __shfl_sync(0xffffffffu, (uint32_t)(key >> 32), 8 * j + (lane >> 2));
  uint32_t node = root;
  for (uint32_t level = root_level; level > 0; level--) {
    visit(level, node);
    uint32_t sum = 0;
    uint32_t p[4][8];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t nj = __shfl_sync(0xffffffffu, node, 8 * j + (lane >> 2));
      // 32 bytes a lane: the row's line in one pass of the L1 data pipe (two
      // 16-byte loads would take two)
      uint64_t w[4];
      ldg32_hint(t.pfx + (size_t)nj * 32 + g * 8, w, keep);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        p[j][2 * i] = (uint32_t)w[i];
        p[j][2 * i + 1] = (uint32_t)(w[i] >> 32);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) sum += rank8(p[j], kp[j]) << (8 * j);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    const uint32_t mine = __shfl_sync(0xffffffffu, sum, (lane & 7u) * 4) >> (8 * (lane >> 3)) & 0xffu;
    uint32_t cnt = mine & 31u;
    if (__any_sync(0xffffffffu, mine >= kEqBit)) {
      sum = 0;
#pragma unroll 1
      for (int j = 0; j < 4; j++) {
        const uint32_t nj = __shfl_sync(0xffffffffu, node, 8 * j + (lane >> 2));
        const uint64_t kj = __shfl_sync(0xffffffffu, key, 8 * j + (lane >> 2));
        uint64_t k[8];
        load_row_il<4>(t.keys + (size_t)nj * 32, g, k, keep);
        if (g == 3) k[7] = kKeyMax;  // slot 31 holds the header
        uint32_t c = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) c += (k[i] <= kj) ? 1u : 0u;
        sum += c << (8 * j);
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      cnt = __shfl_sync(0xffffffffu, sum, (lane & 7u) * 4) >> (8 * (lane >> 3)) & 0xffu;
    }
    node = (uint32_t)ldg_hint(t.vals + (size_t)node * 32 + cnt, keep);
  }
  return node;
}

// One lookup per lane, 32 by the warp (every lane calls it; `live` lanes get
// an answer).  Descent as above, then the leaf's fingerprint row and the
// candidates by the owner alone.
__device__ __forceinline__ uint8_t warp_lookup(const DevTree& t, uint32_t root, uint32_t root_level, uint64_t key,
                                               bool live, uint64_t& val) {
  val = 0;
  if (root == kNil) return key == kKeyMax ? kRejected : kAbsent;
  const bool usable = live && key != kKeyMax;
  const uint32_t leaf = warp_descend(t, root, root_level, usable ? key : 0, [](uint32_t, uint32_t) {});
  if (!usable) return kRejected;
  uint64_t row[4];
  ldg32_hint(t.fp + (size_t)leaf * 32, row, l2_keep());
  return leaf_pick(t, leaf, key, fp_match(row, key_fp(key)), l2_stream(), val) ? kFound : kAbsent;
}

// Look `key` up in leaf `node` (slots loaded by the group); returns the status
// and the value (deferred 32 B load of the one matching slot).
template <int G, bool kLeafVals>
__device__ __forceinline__ uint8_t group_leaf_lookup(const DevTree& t, uint32_t node, uint64_t key, uint32_t g,
                                                     uint32_t gmask, const uint64_t (&k)[32 / G],
                                                     const uint64_t (&v)[32 / G], uint32_t cnt, uint64_t& ans) {
  constexpr int S = 32 / G;
  ans = 0;
  if (cnt == 0) return kAbsent;
  const uint32_t slot = cnt - 1;
  const uint32_t owner = slot / S, e = slot % S;
  const uint64_t kk = __shfl_sync(gmask, pick<S>(k, e), owner, G);
  if (kk != key) return kAbsent;
  if (kLeafVals) ans = __shfl_sync(gmask, pick<S>(v, e), owner, G);
  else ans = (g == 0) ? t.vals[(size_t)node * 32 + slot] : 0;
  return kFound;
}

// The same for a leaf row loaded without its values, with the value load
// given L2 eviction policy `pol`.
template <int G>
__device__ __forceinline__ uint8_t group_leaf_lookup_hint(const DevTree& t, uint32_t node, uint64_t key, uint32_t g,
                                                          uint32_t gmask, const uint64_t (&k)[32 / G], uint32_t cnt,
                                                          uint64_t pol, uint64_t& ans) {
  constexpr int S = 32 / G;
  ans = 0;
  if (cnt == 0) return kAbsent;
  const uint32_t slot = cnt - 1;
  const uint64_t kk = __shfl_sync(gmask, pick<S>(k, slot % S), slot / S, G);
  if (kk != key) return kAbsent;
  ans = (g == 0) ? ldg_hint(t.vals + (size_t)node * 32 + slot, pol) : 0;
  return kFound;
}

// Root-to-leaf descent: child slot = number of keys <= target (child i covers
// [key[i-1], key[i]), src/tree.h:7-19).
template <int G, bool kLeafVals>
__device__ __forceinline__ uint8_t group_descend(const DevTree& t, uint32_t node, uint32_t level, uint64_t key,
                                                 uint32_t g, uint32_t gmask, uint64_t& ans) {
  constexpr int S = 32 / G;
  uint64_t k[S];
  uint64_t v[S];
  uint32_t cnt;
  for (;;) {
    const size_t row = (size_t)node * 32 + g * S;
    load_slots<S>(t.keys + row, k);
    if (level > 0 || kLeafVals) load_slots<S>(t.vals + row, v);
    if (g == G - 1) k[S - 1] = kKeyMax;  // slot 31 holds the header
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < S; i++) c += (k[i] <= key) ? 1u : 0u;
    cnt = group_sum<G>(c, gmask);
    if (level == 0) break;
    const uint64_t mine = pick<S>(v, cnt % S);
    node = (uint32_t)__shfl_sync(gmask, mine, cnt / S, G);
    level--;
  }
  return group_leaf_lookup<G, kLeafVals>(t, node, key, g, gmask, k, v, cnt, ans);
}

// Two descents in lock step (same tree, same height): every level issues the
// row loads of both requests before using either, doubling the loads a group
// keeps in flight.  Results as group_descend for each key.
// kChild: at inner levels load only the chosen child id (one 32 B sector)
// after the key comparison instead of the whole 256 B child row with the keys:
// fewer bytes per level, one more dependent load.
// use_pfx (kChild only): inner levels compare the 32-bit separator prefixes
// (half the bytes of the key row) and read the full keys only when a prefix
// equals the key's.
template <int G, bool kLeafVals, bool kChild = false>
__device__ __forceinline__ void group_descend2(const DevTree& t, uint32_t node, uint32_t level, uint64_t key_a,
                                               uint64_t key_b, uint32_t g, uint32_t gmask, uint64_t& ans_a,
                                               uint8_t& st_a, uint64_t& ans_b, uint8_t& st_b,
                                               bool use_pfx = false) {
  constexpr int S = 32 / G;
  uint64_t ka[S], va[S], kb[S], vb[S];
  uint32_t na = node, nb = node;
  uint32_t ca, cb;
  const uint64_t keep = l2_keep(), stream = l2_stream();
  for (;;) {
    const size_t ra = (size_t)na * 32 + g * S, rb = (size_t)nb * 32 + g * S;
    if (kChild && use_pfx && level > 0) {
      uint32_t pa[S], pb[S];
      load_pfx<S>(t.pfx + ra, pa, keep);
      load_pfx<S>(t.pfx + rb, pb, keep);
      const uint32_t xa = pfx_rank<G, S>(pa, key_a, g, gmask), xb = pfx_rank<G, S>(pb, key_b, g, gmask);
      ca = xa & 0xffffu;
      cb = xb & 0xffffu;
      if (xa >> 16) {  // a separator shares the key's prefix: rank with the full keys
        load_slots_hint<S>(t.keys + ra, ka, keep);
        if (g == G - 1) ka[S - 1] = kKeyMax;
        uint32_t c = 0;
#pragma unroll
        for (int i = 0; i < S; i++) c += (ka[i] <= key_a) ? 1u : 0u;
        ca = group_sum<G>(c, gmask);
      }
      if (xb >> 16) {
        load_slots_hint<S>(t.keys + rb, kb, keep);
        if (g == G - 1) kb[S - 1] = kKeyMax;
        uint32_t c = 0;
#pragma unroll
        for (int i = 0; i < S; i++) c += (kb[i] <= key_b) ? 1u : 0u;
        cb = group_sum<G>(c, gmask);
      }
      na = (uint32_t)ldg_hint(t.vals + (size_t)na * 32 + ca, keep);
      nb = (uint32_t)ldg_hint(t.vals + (size_t)nb * 32 + cb, keep);
      level--;
      continue;
    }
    if (kChild) {
      // interleaved 16-byte chunks (load_row_il): the lane counts below do
      // not depend on which slots a lane holds, only the leaf's key pick does
      const uint64_t pol = level > 0 ? keep : stream;
      load_row_il<G>(t.keys + (size_t)na * 32, g, ka, pol);
      load_row_il<G>(t.keys + (size_t)nb * 32, g, kb, pol);
    } else {
      load_slots<S>(t.keys + ra, ka);
      load_slots<S>(t.keys + rb, kb);
    }
    if ((level > 0 && !kChild) || (level == 0 && kLeafVals)) {
      load_slots<S>(t.vals + ra, va);
      load_slots<S>(t.vals + rb, vb);
    }
    if (g == G - 1) {
      ka[S - 1] = kKeyMax;  // slot 31 holds the header
      kb[S - 1] = kKeyMax;
    }
    uint32_t xa = 0, xb = 0;
#pragma unroll
    for (int i = 0; i < S; i++) {
      xa += (ka[i] <= key_a) ? 1u : 0u;
      xb += (kb[i] <= key_b) ? 1u : 0u;
    }
    ca = group_sum<G>(xa, gmask);
    cb = group_sum<G>(xb, gmask);
    if (level == 0) break;
    if (kChild) {
      na = (uint32_t)ldg_hint(t.vals + (size_t)na * 32 + ca, keep);
      nb = (uint32_t)ldg_hint(t.vals + (size_t)nb * 32 + cb, keep);
    } else {
      const uint64_t ma = pick<S>(va, ca % S), mb = pick<S>(vb, cb % S);
      na = (uint32_t)__shfl_sync(gmask, ma, ca / S, G);
      nb = (uint32_t)__shfl_sync(gmask, mb, cb / S, G);
    }
    level--;
  }
  // leaf: find both slots, then issue both value loads together
  const uint32_t sa = ca > 0 ? ca - 1 : 0, sb = cb > 0 ? cb - 1 : 0;
  const uint64_t kka = kChild ? __shfl_sync(gmask, pick<S>(ka, il_elem<G>(sa)), il_lane<G>(sa), G)
                              : __shfl_sync(gmask, pick<S>(ka, sa % S), sa / S, G);
  const uint64_t kkb = kChild ? __shfl_sync(gmask, pick<S>(kb, il_elem<G>(sb)), il_lane<G>(sb), G)
                              : __shfl_sync(gmask, pick<S>(kb, sb % S), sb / S, G);
  const bool fa = ca > 0 && kka == key_a, fb = cb > 0 && kkb == key_b;
  ans_a = 0;
  ans_b = 0;
  if (kLeafVals) {
    const uint64_t xa = __shfl_sync(gmask, pick<S>(va, sa % S), sa / S, G);
    const uint64_t xb = __shfl_sync(gmask, pick<S>(vb, sb % S), sb / S, G);
    ans_a = fa ? xa : 0;
    ans_b = fb ? xb : 0;
  } else if (g == 0) {
    if (fa) ans_a = kChild ? ldg_hint(t.vals + (size_t)na * 32 + sa, stream) : t.vals[(size_t)na * 32 + sa];
    if (fb) ans_b = kChild ? ldg_hint(t.vals + (size_t)nb * 32 + sb, stream) : t.vals[(size_t)nb * 32 + sb];
  }
  st_a = fa ? kFound : kAbsent;
  st_b = fb ? kFound : kAbsent;
}

}  // namespace bt
