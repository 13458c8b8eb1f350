// Local heap queue (LHQ), B200 form.
//
// Reference: src/local_heap_queue.cu.  Each LP owns a binary heap in an array of
// FEL_SIZE items (fel[lp * FEL_SIZE + i], item_count[lp]); queue_insert appends behind
// the heap with atomicAdd (:398-419), queue_post restores the heap with copy_last
// (move the last item to the root after a dequeue, :128-145), heapify_down (:249-267)
// and heapify_up for the new items (:216-233), one thread per LP; queue_peek returns
// the root inside the window (:430-447).
//
// Here the heap is D-ary with D = max(G, 4) children per node stored contiguously, so
// a lane group reads all children of a node with one coalesced access and picks the
// smallest with a shuffle reduction; sift-down therefore takes log_D(n) group steps.
// Children of window s-1 are pushed (sift-up) before the window's safe events are
// popped in key order and staged for the CTA-wide event pass.
//
// The default form gives an LP a whole warp and an eight-ary heap and takes a window's
// items in one piece (lhqw_lp_stage): event by event, a window's time is the pops and
// pushes of its fullest LP one after another, each a chain of dependent levels.
#pragma once

#include "phold_common.cuh"

static constexpr uint32_t kLhqNil = 0xffffffffu;

struct LhqDev {
  gpq_item* items;  // num_lps << cap_log2 items; heap of LP l at items[l << cap_log2]
  uint32_t* size;   // per-LP heap size
  uint32_t cap_log2;
};

struct LhqMeta {
  uint32_t k, n, count;
  unsigned long long csum, ohash;
};

__device__ __forceinline__ LhqMeta lhq_load_meta(const PholdDev& d, const LhqDev& q, const InsDev& ib, uint32_t lp,
                                                 uint32_t prevb) {
  LhqMeta m;
  m.k = ib.cnt[(size_t)prevb * d.L + lp];
  m.n = q.size[lp];
  m.count = d.count[lp];
  m.csum = d.csum[lp];
  m.ohash = d.ohash[lp];
  return m;
}

// Push x into the heap h of n items (sift-up; one lane).
template <int D>
__device__ __forceinline__ void lhq_push(gpq_item* h, uint32_t n, const gpq_item x) {
  const uint64_t kx = gpq_lp_key(x);
  uint32_t pos = n;
  while (pos > 0) {
    const uint32_t parent = (pos - 1) / D;
    const gpq_item p = h[parent];
    if (gpq_lp_key(p) <= kx) break;
    h[pos] = p;
    pos = parent;
  }
  h[pos] = x;
}

// Remove the root of the heap h of n > 0 items (sift-down of the last item with the
// group reading the D children of a node together).  All lanes of the group.
template <int G, int D>
__device__ __forceinline__ void lhq_pop(gpq_item* h, uint32_t n, const LaneGroup<G>& g) {
  const uint32_t last = n - 1;
  if (last == 0) return;
  const gpq_item x = h[last];
  const uint64_t kx = gpq_lp_key(x);
  uint32_t pos = 0;
  for (;;) {
    const uint32_t fc = pos * D + 1;
    if (fc >= last) break;
    uint64_t best = ~0ull;
    uint32_t bidx = kLhqNil;
    gpq_item bit;
#pragma unroll
    for (int j = 0; j < D / G; ++j) {
      const uint32_t c = fc + g.gl + (uint32_t)j * G;
      if (c < last) {
        const gpq_item it = h[c];
        const uint64_t kc = gpq_lp_key(it);
        if (kc < best) { best = kc; bidx = c; bit = it; }
      }
    }
    uint32_t who;
    const uint64_t kmin = g.kmin(best, &who);
    if (kmin >= kx) break;
    const uint32_t cidx = g.shfl(bidx, who);
    if (g.gl == who) h[pos] = bit;
    pos = cidx;
    g.sync();
  }
  if (g.gl == 0) h[pos] = x;
  g.sync();
}

// One LP, one window s, first pass: push the children of window s-1, then pop every
// event with ts < bound and ts < end_time in key order and stage it.  Returns the new
// root's timestamp bits, min'ed with any child processed here.
template <int G>
__device__ __forceinline__ uint32_t lhq_lp_stage(const PholdDev& d, const LhqDev& q, const InsDev& ib, uint32_t lp,
                                                 uint32_t slot, uint32_t s, float bound, const PholdStage& st,
                                                 const LaneGroup<G>& g, uint32_t* err_slot, const LhqMeta& mt) {
  constexpr int D = G >= 4 ? G : 4;
  const uint32_t L = d.L;
  const uint32_t prevb = (s + 1u) & 1u, curb = s & 1u;
  const uint32_t cap = 1u << q.cap_log2;
  gpq_item* h = q.items + ((size_t)lp << q.cap_log2);
  const float T = d.p.end_time;
  uint32_t n = mt.n;
  uint32_t k = mt.k;
  if (k > 0) {
    if (k > ib.ibc) k = ib.ibc;
    if (n + k > cap) {
      if (g.gl == 0) { gpq_set_error(&d.ctrl->err, GPQ_ERR_QUEUE_FULL); atomicOr(err_slot, 1u); }
      k = cap - n;
    }
    const gpq_item* src = ib.buf + ((size_t)prevb * L + lp) * ib.ibc;
    if (g.gl == 0) {
      for (uint32_t j = 0; j < k; ++j) lhq_push<D>(h, n + j, src[j]);
      ib.cnt[(size_t)prevb * L + lp] = 0;
    }
    n += k;
    g.sync();
  }
  if (g.gl == 0) phold_stage_slot_init(st, slot, mt.count, mt.csum, mt.ohash);
  g.sync();
  uint32_t done = 0, cmin = kInfBits, head = kInfBits;
  gpq_item mine;
  bool have = false;
  while (n > 0) {
    const gpq_item top = h[0];
    if (!((top.ts < bound) && (top.ts < T))) { head = gpq_f2u(top.ts); break; }
    if (g.gl == done % G) { mine = top; have = true; }
    lhq_pop<G, D>(h, n, g);
    --n;
    ++done;
    if (done % G == 0) {  // a full batch of G events
      cmin = min(cmin, phold_stage_batch<G>(d, ib, st, g, mine, true, done - G + g.gl, G, slot, curb, err_slot));
      have = false;
    }
  }
  const uint32_t rem = done % G;
  if (rem) cmin = min(cmin, phold_stage_batch<G>(d, ib, st, g, mine, have, done - rem + g.gl, rem, slot, curb, err_slot));
  if (g.gl == 0) {
    q.size[lp] = n;
    st.lp[slot] = done > 0 ? lp : ~0u;
    if (done > 0) d.count[lp] = mt.count + done;
  }
  return min(head, g.umin(cmin));
}

template <int G_>
struct LhqPolicy {
  static constexpr int G = G_;
  using Dev = LhqDev;
  using Meta = LhqMeta;
  struct Smem {};
  __host__ __device__ static size_t group_smem_bytes(uint32_t) { return 0; }
  __device__ static Smem smem(unsigned char*, uint32_t) { return Smem{}; }
  __device__ static Meta load_meta(const PholdDev& d, const Dev& q, const InsDev& ib, uint32_t lp, uint32_t prevb) {
    return lhq_load_meta(d, q, ib, lp, prevb);
  }
  __device__ static uint32_t stage_lp(const PholdDev& d, const Dev& q, const InsDev& ib, uint32_t lp, uint32_t slot,
                                      uint32_t s, float bound, const Smem&, const PholdStage& st,
                                      const LaneGroup<G>& g, uint32_t* err_slot, const Meta& mt) {
    return lhq_lp_stage<G>(d, q, ib, lp, slot, s, bound, st, g, err_slot, mt);
  }
};

// ---- a warp per LP, a window's items in one piece ----
//
// The heap items below the window's end form a subtree at the root: the warp collects them
// level by level, four nodes' children to a step.  New items below the end join them, the
// others take the places of the collected ones from the root down (or are appended, when
// there are more; when there are fewer, the array's last items fill the rest), and heap
// order is restored from the deepest touched level up, four sift-downs of one level at a
// time (eight lanes each; nodes of one level have disjoint subtrees).  More than
// kLhqwMax safe items go through the event-by-event form on the same eight-ary heap.
static constexpr uint32_t kLhqwMax = 128;

struct LhqwSmem {
  uint64_t* key;   // [kLhqwMax] safe items
  uint64_t* sorted;  // [kLhqwMax] in order; before that, flags of the array's last places
  uint16_t* pos;   // [kLhqwMax] places of those from the heap, ascending
};

__host__ __device__ inline size_t lhqw_group_smem_bytes() { return kLhqwMax * (8 + 8 + 2); }

__device__ __forceinline__ LhqwSmem lhqw_smem(unsigned char* base) {
  LhqwSmem s;
  s.key = reinterpret_cast<uint64_t*>(base);
  s.sorted = s.key + kLhqwMax;
  s.pos = reinterpret_cast<uint16_t*>(s.sorted + kLhqwMax);
  return s;
}

// First place of a level of the eight-ary heap (of at most 2^16 items).
__device__ __forceinline__ uint32_t lhqw_level_start(uint32_t level) { return ((1u << (3u * level)) - 1u) / 7u; }

// Sifts down the items at up to four places of one level of the heap h of n items (lanes
// 8i .. 8i + 7 work on place `at` of their lane when `act`).  All lanes.
__device__ __forceinline__ void lhqw_sift(gpq_item* h, uint32_t n, uint32_t at, bool act, uint32_t lane) {
  const uint32_t ch = lane & 7u, shift = lane & 24u;
  uint32_t q = at;
  gpq_item x{};
  uint64_t kx = 0;
  act = act && 8u * q + 1u < n;  // a leaf stays
  if (act) {
    x = h[q];
    kx = gpq_lp_key(x);
  }
  bool moved = false;
  while (__any_sync(GPQ_FULL_MASK, act)) {
    const uint32_t c = 8u * q + 1u + ch;
    gpq_item it{};
    uint64_t kc = ~0ull;
    if (act && c < n) {
      it = h[c];
      kc = gpq_lp_key(it);
    }
    uint32_t mt = (uint32_t)(kc >> 32);  // the smallest timestamp of eight, then its id
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) mt = min(mt, __shfl_xor_sync(GPQ_FULL_MASK, mt, o));
    uint32_t who = (__ballot_sync(GPQ_FULL_MASK, (uint32_t)(kc >> 32) == mt) >> shift) & 0xffu;
    if (__any_sync(GPQ_FULL_MASK, act && (who & (who - 1u)) != 0u)) {
      uint32_t mi = (uint32_t)(kc >> 32) == mt ? (uint32_t)kc : ~0u;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) mi = min(mi, __shfl_xor_sync(GPQ_FULL_MASK, mi, o));
      who = (__ballot_sync(GPQ_FULL_MASK, kc == (((uint64_t)mt << 32) | mi)) >> shift) & 0xffu;
    }
    const uint32_t best = (uint32_t)__ffs((int)who) - 1u;
    const uint64_t m = ((uint64_t)mt << 32) | __shfl_sync(GPQ_FULL_MASK, (uint32_t)kc, (int)(shift + (best & 7u)));
    if (act) {
      if (m < kx) {
        if (ch == best) h[q] = it;
        q = 8u * q + 1u + best;
        moved = true;
        act = 8u * q + 1u < n;
      } else {
        act = false;
      }
      if (!act && moved && ch == 0) h[q] = x;
    }
    __syncwarp();
  }
}

// The c safe items in order when some keys are equal (a caller's population may hold such), by
// their place in the list.  Not inlined, and reached by a test of the ranks' sum: the place
// compared in every step of the rank loop cost 1.9 % of a run of 8,191 LPs x 120, this 0.4 %.
static __device__ __noinline__ void lhqw_rank_equal(const uint64_t* key, uint64_t* sorted, uint32_t c, uint32_t lane) {
  __syncwarp();
  for (uint32_t j = lane; j < c; j += 32u) {
    const uint64_t kj = key[j];
    uint32_t r = 0;
    for (uint32_t i = 0; i < c; ++i) r += key[i] < kj || (key[i] == kj && i < j) ? 1u : 0u;
    sorted[r] = kj;
  }
}

__device__ __forceinline__ uint32_t lhqw_lp_stage(const PholdDev& d, const LhqDev& q, const InsDev& ib, uint32_t lp,
                                                  uint32_t slot, uint32_t s, float bound, const LhqwSmem& sm,
                                                  const PholdStage& st, const LaneGroup<32>& g, uint32_t* err_slot,
                                                  const LhqMeta& mt) {
  const uint32_t lane = g.gl, below = (1u << lane) - 1u;
  const uint32_t prevb = (s + 1u) & 1u, curb = s & 1u;
  const uint32_t cap = 1u << q.cap_log2;
  gpq_item* h = q.items + ((size_t)lp << q.cap_log2);
  const gpq_item* src = ib.buf + ((size_t)prevb * d.L + lp) * ib.ibc;
  const uint64_t lim = (uint64_t)min(gpq_f2u(bound), gpq_f2u(d.p.end_time)) << 32;
  uint32_t n = mt.n;
  uint32_t k = min(mt.k, ib.ibc);
  // the first new items and the root in flight together
  gpq_item nw{};
  if (lane < k) nw = src[lane];
  const uint64_t root = n > 0 ? gpq_lp_key(h[0]) : ~0ull;
  const bool full = n + k > cap;
  if (full) k = cap - n;
  // the heap's safe items
  uint32_t c = 0;
  bool over = false;
  if (root < lim) {
    if (lane == 0) {
      sm.pos[0] = 0;
      sm.key[0] = root;
    }
    c = 1;
  }
  __syncwarp();
  for (uint32_t i = 0; i < c;) {
    const uint32_t m = min(4u, c - i), sub = lane >> 3;
    uint32_t child = 0;
    uint64_t kc = ~0ull;
    if (sub < m) {
      child = 8u * sm.pos[i + sub] + 1u + (lane & 7u);
      if (child < n) kc = gpq_lp_key(h[child]);
    }
    const uint32_t b = __ballot_sync(GPQ_FULL_MASK, kc < lim);
    if (c + (uint32_t)__popc(b) > kLhqwMax) {
      over = true;
      break;
    }
    if (kc < lim) {
      const uint32_t at = c + (uint32_t)__popc(b & below);
      sm.pos[at] = (uint16_t)child;
      sm.key[at] = kc;
    }
    c += (uint32_t)__popc(b);
    i += m;
    __syncwarp();
  }
  const uint32_t holes = c;
  uint32_t safe_new = (uint32_t)__popc(__ballot_sync(GPQ_FULL_MASK, lane < k && gpq_lp_key(nw) < lim));
  for (uint32_t j0 = 32u; j0 < k; j0 += 32u) {
    const uint32_t j = j0 + lane;
    const uint64_t kn = j < k ? gpq_lp_key(src[j]) : ~0ull;
    safe_new += (uint32_t)__popc(__ballot_sync(GPQ_FULL_MASK, kn < lim));
  }
  if (over || c + safe_new > kLhqwMax)
    return lane < 8u ? lhq_lp_stage<8>(d, q, ib, lp, slot, s, bound, st, LaneGroup<8>(), err_slot, mt) : kInfBits;
  if (full && lane == 0) {
    gpq_set_error(&d.ctrl->err, GPQ_ERR_QUEUE_FULL);
    atomicOr(err_slot, 1u);
  }
  // new items: to the safe ones, into the places that became free, or behind the heap
  uint32_t placed = 0;
  for (uint32_t j0 = 0; j0 < k; j0 += 32u) {
    const uint32_t j = j0 + lane;
    const gpq_item it = j0 && j < k ? src[j] : nw;
    const uint64_t kn = j < k ? gpq_lp_key(it) : ~0ull;
    const uint32_t bs = __ballot_sync(GPQ_FULL_MASK, kn < lim), bu = __ballot_sync(GPQ_FULL_MASK, j < k && kn >= lim);
    if (j < k) {
      if (kn < lim) {
        sm.key[c + (uint32_t)__popc(bs & below)] = kn;
      } else {
        const uint32_t u = placed + (uint32_t)__popc(bu & below);
        h[u < holes ? sm.pos[u] : n + (u - holes)] = it;
      }
    }
    c += (uint32_t)__popc(bs);
    placed += (uint32_t)__popc(bu);
  }
  uint32_t lo = 1, hi = 0;  // parents of appended items, places lo .. hi
  uint32_t touched = holes;
  if (placed > holes) {
    const uint32_t n1 = n + (placed - holes);
    if (n1 > 1u) {
      lo = n > 0 ? (n - 1u) >> 3 : 0u;
      hi = (n1 - 2u) >> 3;
    }
    n = n1;
  } else if (placed < holes) {  // the last items into the rest
    const uint32_t r = holes - placed, n1 = n - r;
    uint8_t* gone = reinterpret_cast<uint8_t*>(sm.sorted);  // places n1 + i that are free already
    for (uint32_t i = lane; i < r; i += 32u) gone[i] = 0;
    __syncwarp();
    for (uint32_t i = placed + lane; i < holes; i += 32u)
      if (sm.pos[i] >= n1) gone[sm.pos[i] - n1] = 1;
    __syncwarp();
    uint32_t run = placed;
    for (uint32_t i0 = 0; i0 < r; i0 += 32u) {
      const uint32_t i = i0 + lane;
      const bool mv = i < r && !gone[i];
      const uint32_t b = __ballot_sync(GPQ_FULL_MASK, mv);
      if (mv) h[sm.pos[run + (uint32_t)__popc(b & below)]] = h[n1 + i];
      run += (uint32_t)__popc(b);
    }
    touched = run;
    n = n1;
  }
  __syncwarp();
  // heap order, from the deepest touched level up
  if (touched > 0 || lo <= hi) {
    const uint32_t deepest = max(touched > 0 ? (uint32_t)sm.pos[touched - 1u] : 0u, lo <= hi ? hi : 0u);
    uint32_t level = 0;
    while (lhqw_level_start(level + 1u) <= deepest) ++level;
    uint32_t end = touched;
    for (;; --level) {
      const uint32_t ls = lhqw_level_start(level), ln = 8u * ls + 1u;
      uint32_t first = 0;  // touched places below this level
      for (uint32_t i0 = 0; i0 < end; i0 += 32u)
        first += (uint32_t)__popc(__ballot_sync(GPQ_FULL_MASK, i0 + lane < end && sm.pos[i0 + lane] < ls));
      for (uint32_t i = first; i < end; i += 4u) {
        const uint32_t j = i + (lane >> 3);
        lhqw_sift(h, n, j < end ? sm.pos[j] : 0u, j < end, lane);
      }
      end = first;
      if (lo <= hi && hi >= ls) {  // ancestors of the appended items in this level
        const uint32_t a = max(lo, ls), b = min(hi, ln - 1u);
        for (uint32_t i = a; i <= b; i += 4u) lhqw_sift(h, n, i + (lane >> 3), i + (lane >> 3) <= b, lane);
        if (level == 0) break;
        const uint32_t pa = (a - 1u) >> 3, pb = (b - 1u) >> 3;
        const bool both = lo < ls;  // some of them lie in the level above: all of it then
        hi = both ? ls - 1u : pb;
        lo = both ? lhqw_level_start(level - 1u) : pa;
      }
      if (level == 0) break;
    }
  }
  // the safe items in order
  if (lane == 0) phold_stage_slot_init(st, slot, mt.count, mt.csum, mt.ohash);
  uint32_t ranks = 0;
  for (uint32_t j = lane; j < c; j += 32u) {
    const uint64_t kj = sm.key[j];
    uint32_t r = 0;
    for (uint32_t i = 0; i < c; ++i) r += sm.key[i] < kj ? 1u : 0u;
    sm.sorted[r] = kj;
    ranks += r;
  }
  // equal keys share a rank, which the ranks' sum tells
  if (__reduce_add_sync(GPQ_FULL_MASK, ranks) != c * (c - 1u) / 2u) lhqw_rank_equal(sm.key, sm.sorted, c, lane);
  __syncwarp();
  uint32_t cmin = kInfBits;
  for (uint32_t j0 = 0; j0 < c; j0 += 32u) {
    const uint32_t j = j0 + lane;
    const uint64_t kj = j < c ? sm.sorted[j] : 0ull;
    const gpq_item e{gpq_u2f((uint32_t)(kj >> 32)), lp, (uint32_t)kj, 0u};
    cmin = min(cmin, phold_stage_batch<32>(d, ib, st, g, e, j < c, j, min(32u, c - j0), slot, curb, err_slot));
  }
  const uint32_t head = n > 0 ? gpq_f2u(h[0].ts) : kInfBits;
  if (lane == 0) {
    if (mt.k > 0) ib.cnt[(size_t)prevb * d.L + lp] = 0;
    q.size[lp] = n;
    st.lp[slot] = c > 0 ? lp : ~0u;
    if (c > 0) d.count[lp] = mt.count + c;
  }
  __syncwarp();
  return min(head, g.umin(cmin));
}

struct LhqWarpPolicy {
  static constexpr int G = 32;
  using Dev = LhqDev;
  using Meta = LhqMeta;
  using Smem = LhqwSmem;
  __host__ __device__ static size_t group_smem_bytes(uint32_t) { return lhqw_group_smem_bytes(); }
  __device__ static Smem smem(unsigned char* base, uint32_t) { return lhqw_smem(base); }
  __device__ static Meta load_meta(const PholdDev& d, const Dev& q, const InsDev& ib, uint32_t lp, uint32_t prevb) {
    return lhq_load_meta(d, q, ib, lp, prevb);
  }
  __device__ static uint32_t stage_lp(const PholdDev& d, const Dev& q, const InsDev& ib, uint32_t lp, uint32_t slot,
                                      uint32_t s, float bound, const Smem& sm, const PholdStage& st,
                                      const LaneGroup<32>& g, uint32_t* err_slot, const Meta& mt) {
    return lhqw_lp_stage(d, q, ib, lp, slot, s, bound, sm, st, g, err_slot, mt);
  }
};
