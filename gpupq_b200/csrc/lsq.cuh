// Local splay queue (LSQ), B200 form.
//
// Reference: src/local_splay_queue.cu.  Each LP owns a top-down splay tree (Sleator's
// public-domain code, credited in the reference's header comment) over a per-LP node
// pool of 32-byte nodes with two child pointers (:108-156 splay, :158-202 insert,
// :233-273 delete_min); free nodes are found by scanning the pool (:72-93);
// queue_post inserts the buffered items one by one (:435-454).
//
// Here nodes are pool indices, not pointers: an LP's pool is items[lp << cap_log2 ...]
// (16-byte items) plus a 32-bit link word per node (left << 16 | right, 0xffff = none),
// so a node costs 20 bytes and the structure is relocatable.  Free nodes come from a
// per-LP stack (O(1) instead of a pool scan).  Free pool slots carry lp = 0xffffffff.
//
// A splay tree is a pointer-chasing sequential structure: one lane of a group works on an
// LP's tree, and its time is the chain of dependent loads of the slowest LP.  So
//   * a splay keeps the nodes it stands on in registers (one round trip a level: a node's
//     key and link word are loaded together);
//   * a window's safe events come off in one piece: one splay at the window's end splits
//     the tree, and the left part is taken apart in key order by right rotations, instead
//     of a splay to the minimum per event;
//   * the group's other lanes load the new events and the free nodes ahead of the inserts;
//   * few LPs share a warp while warps are free (lsq_lanes), since lanes on different
//     paths of different trees run one after another.
#pragma once

#include "phold_common.cuh"

static constexpr uint32_t kLsqNil = 0xffffu;
static constexpr uint32_t kLsqHdr = 0x10000u;  // the splay's header node (not in the pool)

struct LsqDev {
  gpq_item* items;   // num_lps << cap_log2 node items
  uint32_t* links;   // num_lps << cap_log2 link words
  uint16_t* freestk; // num_lps << cap_log2 free-node stacks
  uint32_t* root;    // per-LP root index (kLsqNil = empty)
  uint32_t* size;    // per-LP node count
  uint32_t* freetop; // per-LP free-stack height
  uint32_t cap_log2;
};

struct LsqView {
  gpq_item* it;
  uint32_t* ln;
  __device__ __forceinline__ uint64_t key(uint32_t x) const { return gpq_lp_key(it[x]); }
};

// A tree's root in registers: its index, key and link word (which memory holds too).
struct LsqRoot {
  uint32_t t;
  uint32_t ln;
  uint64_t key;
};

__device__ __forceinline__ LsqRoot lsq_load_root(const LsqView& v, uint32_t t) {
  LsqRoot r{t, 0u, 0ull};
  if (t != kLsqNil) {
    r.key = v.key(t);
    r.ln = v.ln[t];
  }
  return r;
}

// Top-down splay of `key` in the tree rooted at `root` (Sleator-Tarjan 1985, top-down
// variant; the tree is not empty): returns the new root, the last node on the search path
// for `key`.  Every node on the path costs one load of its key and link word; a link word
// is stored once, when its last new child is known.  `right_min` gets the smallest key of
// the new root's right subtree when the root's key is below `key` (all ones: none).
__device__ __forceinline__ LsqRoot lsq_splay(const LsqView& v, LsqRoot root, uint64_t key, uint64_t* right_min) {
  uint32_t t = root.t, lt = root.ln;
  uint64_t kt = root.key, kr = ~0ull;
  uint32_t n_left = kLsqNil, n_right = kLsqNil;  // the header's left and right trees
  uint32_t l = kLsqHdr, r = kLsqHdr, ll = 0, lr = 0;
  for (;;) {
    if (key <= kt) {
      uint32_t c = lt >> 16;
      if (c == kLsqNil) break;
      uint64_t kc = v.key(c);
      uint32_t lc = v.ln[c];
      if (key < kc) {  // rotate right
        v.ln[t] = (lt & 0xffffu) | (lc << 16);
        lt = (lc & 0xffff0000u) | t;
        t = c;
        kt = kc;
        c = lt >> 16;
        if (c == kLsqNil) break;
        kc = v.key(c);
        lc = v.ln[c];
      }
      if (r == kLsqHdr) n_left = t; else v.ln[r] = (t << 16) | (lr & 0xffffu);  // link right
      r = t;
      lr = lt;
      kr = kt;
      t = c;
      kt = kc;
      lt = lc;
    } else {
      uint32_t c = lt & 0xffffu;
      if (c == kLsqNil) break;
      uint64_t kc = v.key(c);
      uint32_t lc = v.ln[c];
      if (key > kc) {  // rotate left
        v.ln[t] = (lt & 0xffff0000u) | (lc >> 16);
        lt = (t << 16) | (lc & 0xffffu);
        t = c;
        kt = kc;
        c = lt & 0xffffu;
        if (c == kLsqNil) break;
        kc = v.key(c);
        lc = v.ln[c];
      }
      if (l == kLsqHdr) n_right = t; else v.ln[l] = (ll & 0xffff0000u) | t;  // link left
      l = t;
      ll = lt;
      t = c;
      kt = kc;
      lt = lc;
    }
  }
  const uint32_t tl = lt >> 16, tr = lt & 0xffffu;  // assemble
  if (l == kLsqHdr) n_right = tl; else v.ln[l] = (ll & 0xffff0000u) | tl;
  if (r == kLsqHdr) n_left = tr; else v.ln[r] = (tr << 16) | (lr & 0xffffu);
  lt = (n_right << 16) | n_left;
  v.ln[t] = lt;
  *right_min = kr;
  return LsqRoot{t, lt, kt};
}

// Insert node x of key kx (item already stored) into the tree of `root`; returns the new root.
__device__ __forceinline__ LsqRoot lsq_insert(const LsqView& v, LsqRoot root, uint32_t x, uint64_t kx) {
  uint32_t lx = (kLsqNil << 16) | kLsqNil;
  if (root.t != kLsqNil) {
    uint64_t rm;
    root = lsq_splay(v, root, kx, &rm);
    if (kx <= root.key) {
      lx = (root.ln & 0xffff0000u) | root.t;
      v.ln[root.t] = (kLsqNil << 16) | (root.ln & 0xffffu);
    } else {
      lx = (root.t << 16) | (root.ln & 0xffffu);
      v.ln[root.t] = (root.ln & 0xffff0000u) | kLsqNil;
    }
  }
  v.ln[x] = lx;
  return LsqRoot{x, lx, kx};
}

struct LsqMeta {
  uint32_t k, root, size, freetop, count;
  unsigned long long csum, ohash;
};

__device__ __forceinline__ LsqMeta lsq_load_meta(const PholdDev& d, const LsqDev& q, const InsDev& ib, uint32_t lp,
                                                 uint32_t prevb) {
  LsqMeta m;
  m.k = ib.cnt[(size_t)prevb * d.L + lp];
  m.root = q.root[lp];
  m.size = q.size[lp];
  m.freetop = q.freetop[lp];
  m.count = d.count[lp];
  m.csum = d.csum[lp];
  m.ohash = d.ohash[lp];
  return m;
}

// One LP, one window s: insert the children of window s-1, then take the safe events off
// and stage them.  Returns the new minimum's timestamp bits, min'ed with any child
// processed here.  All lanes of the group call it; lane 0 works on the tree.
template <int G>
__device__ __forceinline__ uint32_t lsq_lp_stage(const PholdDev& d, const LsqDev& q, const InsDev& ib, uint32_t lp,
                                                 uint32_t slot, uint32_t s, float bound, const PholdStage& st,
                                                 const LaneGroup<G>& g, uint32_t* err_slot, const LsqMeta& mt) {
  const uint32_t L = d.L;
  const uint32_t prevb = (s + 1u) & 1u, curb = s & 1u;
  const size_t base = (size_t)lp << q.cap_log2;
  const LsqView v{q.items + base, q.links + base};
  uint16_t* fs = q.freestk + base;
  LsqRoot root = lsq_load_root(v, mt.root);
  uint32_t size = mt.size, ftop = mt.freetop;
  uint32_t k = mt.k;
  if (k > 0) {
    if (k > ib.ibc) k = ib.ibc;
    if (k > ftop) {
      if (g.gl == 0) { gpq_set_error(&d.ctrl->err, GPQ_ERR_QUEUE_FULL); atomicOr(err_slot, 1u); }
      k = ftop;
    }
    const gpq_item* src = ib.buf + ((size_t)prevb * L + lp) * ib.ibc;
    for (uint32_t j0 = 0; j0 < k; j0 += G) {
      const uint32_t j = j0 + g.gl;
      uint32_t x = 0;
      uint64_t kx = 0;
      if (j < k) {
        const gpq_item it = src[j];
        x = fs[ftop - 1u - j];
        v.it[x] = it;
        kx = gpq_lp_key(it);
      }
      g.sync();  // the items before lane 0 walks over them
      const uint32_t m = min((uint32_t)G, k - j0);
      for (uint32_t i = 0; i < m; ++i) {
        const uint32_t xi = g.shfl(x, i);
        const uint64_t ki = ((uint64_t)g.shfl((uint32_t)(kx >> 32), i) << 32) | g.shfl((uint32_t)kx, i);
        if (g.gl == 0) root = lsq_insert(v, root, xi, ki);
      }
    }
    ftop -= k;
    size += k;
    if (g.gl == 0) ib.cnt[(size_t)prevb * L + lp] = 0;
  }
  if (g.gl != 0) return kInfBits;
  const LaneGroup<1> one;
  phold_stage_slot_init(st, slot, mt.count, mt.csum, mt.ohash);
  uint32_t done = 0, cmin = kInfBits, head = kInfBits;
  if (root.t != kLsqNil) {
    // split at the first key that is not safe
    const uint64_t lim = (uint64_t)min(gpq_f2u(bound), gpq_f2u(d.p.end_time)) << 32;
    uint64_t rm;
    root = lsq_splay(v, root, lim, &rm);
    LsqRoot e;  // the safe events' tree
    if (root.key < lim) {
      e = LsqRoot{root.t, (root.ln & 0xffff0000u) | kLsqNil, root.key};
      root.t = root.ln & 0xffffu;
      if (root.t != kLsqNil) head = (uint32_t)(rm >> 32);
    } else {
      e = LsqRoot{root.ln >> 16, 0u, 0ull};
      if (e.t != kLsqNil) {
        v.ln[root.t] = (kLsqNil << 16) | (root.ln & 0xffffu);
        e = lsq_load_root(v, e.t);
      }
      head = (uint32_t)(root.key >> 32);
    }
    while (e.t != kLsqNil) {
      for (uint32_t c = e.ln >> 16; c != kLsqNil; c = e.ln >> 16) {  // rotate right until e is the smallest
        const uint64_t kc = v.key(c);
        const uint32_t lc = v.ln[c];
        v.ln[e.t] = (lc << 16) | (e.ln & 0xffffu);
        e = LsqRoot{c, (lc & 0xffff0000u) | e.t, kc};
      }
      const uint32_t x = e.t;
      const gpq_item ev{gpq_u2f((uint32_t)(e.key >> 32)), lp, (uint32_t)e.key, 0u};
      e = lsq_load_root(v, e.ln & 0xffffu);
      cmin = min(cmin, phold_stage_batch<1>(d, ib, st, one, ev, true, done, 1, slot, curb, err_slot));
      v.it[x].lp = 0xffffffffu;  // free pool slot
      fs[ftop++] = (uint16_t)x;
      ++done;
    }
    size -= done;
  }
  q.root[lp] = root.t;
  q.size[lp] = size;
  q.freetop[lp] = ftop;
  st.lp[slot] = done > 0 ? lp : ~0u;
  if (done > 0) d.count[lp] = mt.count + done;
  return min(head, cmin);
}

template <int G_>
struct LsqPolicy {
  static constexpr int G = G_;
  using Dev = LsqDev;
  using Meta = LsqMeta;
  struct Smem {};
  __host__ __device__ static size_t group_smem_bytes(uint32_t) { return 0; }
  __device__ static Smem smem(unsigned char*, uint32_t) { return Smem{}; }
  __device__ static Meta load_meta(const PholdDev& d, const Dev& q, const InsDev& ib, uint32_t lp, uint32_t prevb) {
    return lsq_load_meta(d, q, ib, lp, prevb);
  }
  __device__ static uint32_t stage_lp(const PholdDev& d, const Dev& q, const InsDev& ib, uint32_t lp, uint32_t slot,
                                      uint32_t s, float bound, const Smem&, const PholdStage& st,
                                      const LaneGroup<G>& g, uint32_t* err_slot, const Meta& mt) {
    return lsq_lp_stage<G>(d, q, ib, lp, slot, s, bound, st, g, err_slot, mt);
  }
};
