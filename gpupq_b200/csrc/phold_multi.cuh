// Many PHOLD instances in one persistent launch (batched and served PHOLD).
//
// The instances share one LP space: instance i owns LPs [lp0_i, lp0_i + L_i) of the
// local array queues (src/local_array_queue.cu as rebuilt in laq.cuh), and every LP
// knows its instance (lp_inst).  All instances advance together, one window per grid
// barrier, but each with its own window: LP lp of instance i drains the events below
// min_i + lookahead_i (and end_time_i), where min_i is instance i's minimum from the
// previous window (src/des.cu:154-214 per instance).  An instance whose minimum reached
// its end time is finished and its LPs are skipped until the host collects it.
//
// A ring's events are in no order (one written in order, by an earlier snapshot or by the
// population, is as good): a window selects the events below its bound, ranks only those,
// and closes their gaps.
#pragma once

#include "laq.cuh"

struct PmInstDev {
  gpq_phold_params p;  // num_lps = L_i
  uint32_t lp0;
  uint32_t per_lp;     // initial events per LP
  uint32_t err;
  uint32_t windows;    // windows this instance took part in
  uint32_t w0;         // its first window; it runs windows [w0, w0 + windows)
  uint32_t aux;        // bucketed sessions: 1 / bucket width of the run (float bits)
};

struct PmCtl {
  uint32_t err;
  uint32_t phase;    // next window
  unsigned long long bar;
};

struct PmDev {
  PmInstDev* inst;
  uint32_t* mins;        // [max_inst][3] window minimum slots (float bits)
  uint32_t* errs;        // [max_inst][3] error seen in the window before (slots like mins)
  const uint8_t* on;     // slot in use
  uint32_t n_inst;       // slots [0, n_inst) may be in use
  uint32_t* lp_inst;     // [n_lps] owning slot, ~0u when free
  uint32_t n_lps;        // LPs [0, n_lps) may be in use
  gpq_item* ring;        // [max_lps << cap_log2]
  uint32_t* rd;
  uint32_t* wr;
  uint32_t cap_log2;
  gpq_item* ibuf;        // [2][max_lps][ibc]
  uint32_t* icnt;        // [2][max_lps]
  uint32_t ibc;
  uint32_t* lmin;        // [max_lps] minimum of the LP's ring (float bits); 0: not known
  uint32_t max_lps;
  uint32_t* count;
  unsigned long long* csum;
  unsigned long long* ohash;
  PmCtl* ctl;
  uint64_t spin_limit;
};

// Instance i runs window s: in use, minimum below its end time, no error in window s - 1.
// Every block decides from the same slots, written before the last grid barrier.
__device__ __forceinline__ bool pm_active(const PmDev& d, uint32_t i, uint32_t s) {
  return d.on[i] && gpq_u2f(ld_relaxed_u32(&d.mins[3 * i + s % 3u])) < d.inst[i].p.end_time &&
         ld_relaxed_u32(&d.errs[3 * i + s % 3u]) == 0u;
}

__device__ __forceinline__ void pm_error(const PmDev& d, uint32_t inst, uint32_t s, uint32_t code) {
  gpq_set_error(&d.inst[inst].err, code);
  atomicOr(&d.errs[3 * inst + (s + 1u) % 3u], 1u);
}

// ---- selection windows -------------------------------------------------------------------
// A warp takes 8 consecutive LPs a turn (4 when the warps outnumber the fours), 8 lanes an LP:
// it streams the LP's ring and its children of the previous window as one sequence of m = n + k
// items, puts the keys of the safe ones into the LP's list in shared memory, and fills the
// ring's first m - safe places: a hole there is a safe item's place, and the items beyond move
// into the holes in order.  Then all 32 lanes rank and process the turn's safe events one per
// lane; each event leaves its two hashes in its list entry, and four lanes an LP add them up.
//
// What bounds it: instructions and the loads' latency (sessions of 48 runs, 256-65,536 LPs x
// 32, lookahead 0.5: 0.28 ms a window of 5.5 M events, 19 G events/s).  Keeping the rings
// sorted (merge the children, drain the prefix; 64 registers, 46.7 warp instructions and
// 135 B of DRAM traffic an event) took 48.2 ms where this takes 29.2; over lookahead
// 0.001-20 and 4-1,000 events an LP it took 1.0-2.4 times as long, most where windows take
// 20 events or more off an LP.  Three blocks an SM: at four the 64 registers put the
// loads in flight into local memory (43-60 ms).  The LPs whose events outgrow a list are
// left to a loop of their own for the same reason: inside the turn their code cost 10 ms.
struct PmSelSmem {
  unsigned long long* key;  // [8][kPmSelStride] safe keys, then the events' hashes
  unsigned long long* oh;   // [8][kPmSelStride] the events' sequence hashes
  uint32_t* at;             // [8][kPmSelStride] where each safe item is; then the events by lane
  uint32_t* beg;            // [12] first event of each LP, in the order of the LPs
  uint32_t* c0;             // [8] the LP's committed count
  uint32_t* inst;           // [8] its run, ~0u: none, or not running
  uint32_t* mn;             // [8] minimum of what it holds
  uint32_t* wide;           // [kPmWides] LPs whose safe events outgrew their list
  uint32_t* par;            // [8][8] the run's model: words 0-6 of its parameters, its first LP
};

static constexpr uint32_t kPmSelLps = 8;
static constexpr uint32_t kPmSelCap = 44;     // safe events of an LP in shared memory
static constexpr uint32_t kPmSelStride = 46;  // 16-byte aligned rows that start in different banks
static constexpr uint32_t kPmWideCap = 2 * kPmSelLps * kPmSelStride - 2;  // keys in the two lists' space
static constexpr uint32_t kPmWides = 32;
static constexpr uint32_t kPmTab = 256;       // runs whose bound a block keeps in shared memory

__host__ __device__ inline size_t pm_sel_warp_bytes() {
  return (size_t)kPmSelLps * kPmSelStride * (8 + 8 + 4) + (12 + 3 * kPmSelLps + 8 * kPmSelLps + kPmWides) * 4;
}

__device__ __forceinline__ PmSelSmem pm_sel_smem(unsigned char* base) {
  PmSelSmem s;
  s.key = reinterpret_cast<unsigned long long*>(base);
  s.oh = s.key + kPmSelLps * kPmSelStride;
  s.at = reinterpret_cast<uint32_t*>(s.oh + kPmSelLps * kPmSelStride);
  s.beg = s.at + kPmSelLps * kPmSelStride;
  s.c0 = s.beg + 12;
  s.inst = s.c0 + kPmSelLps;
  s.mn = s.inst + kPmSelLps;
  s.par = s.mn + kPmSelLps;
  s.wide = s.par + 8 * kPmSelLps;
  return s;
}

// The bound of run i's window s (events below it are safe); negative: it has no selection
// window.
__device__ __forceinline__ float pm_sel_bound(const PmDev& d, uint32_t i, uint32_t s) {
  if (!pm_active(d, i, s)) return -1.f;
  const float m = gpq_u2f(ld_relaxed_u32(&d.mins[3 * i + s % 3u]));
  return fminf(GPQ_FADD(m, d.inst[i].p.lookahead), d.inst[i].p.end_time);
}

// One safe event of LP lp: its hashes, and its child (LP in the session's numbers).
__device__ __forceinline__ gpq_item pm_sel_event(const gpq_phold_params& p, uint32_t lp0, uint32_t lp,
                                                 unsigned long long key, uint64_t seq, uint64_t* h, uint64_t* oh) {
  gpq_item e;
  e.ts = gpq_u2f((uint32_t)(key >> 32));
  e.id = (uint32_t)key;
  e.lp = lp - lp0;
  e.aux = 0;
  *h = gpq_ev_hash(e.id, (uint32_t)(key >> 32));
  *oh = gpq_seq_hash(*h, seq);
  gpq_item ch = gpq_phold_child(p, e);
  ch.lp += lp0;
  return ch;
}

__device__ __forceinline__ void pm_sel_file(const PmDev& d, uint32_t s, uint32_t inst, const gpq_item& ch, uint32_t pos) {
  if (pos < d.ibc) d.ibuf[((size_t)(s & 1u) * d.max_lps + ch.lp) * d.ibc + pos] = ch;
  else pm_error(d, inst, s, GPQ_ERR_INSERT_FULL);
}

// The ranks of a turn's events when some keys of an LP are equal (from a snapshot that holds
// such events, or ids that wrap around), by their place in the list.  All lanes of the warp.
static __device__ __noinline__ void pm_sel_rank_equal(const unsigned long long* key, uint32_t* at, uint32_t total) {
  for (uint32_t y = threadIdx.x & 31u; y < total; y += 32u) {
    const uint32_t seg = (at[y] >> 8) & 0xffu, j = at[y] & 0xffu;
    const unsigned long long kj = key[seg * kPmSelStride + j];
    uint32_t r = at[y] >> 16;
    for (uint32_t t = 0; t < j; ++t) r += key[seg * kPmSelStride + t] == kj ? 1u : 0u;
    at[y] = (r << 16) | (seg << 8) | j;
  }
}

// An LP with more safe events than its list holds, by the whole warp (keys: the lists'
// space): its safe keys side by side, ranked and processed one per lane -- beyond kPmWideCap
// of them, ranked by scanning the LP's items --, then the rest moved down in order.  All
// lanes of the warp.
static __device__ __forceinline__ void pm_select_wide(const PmDev& d, uint32_t s, uint32_t lp, unsigned long long* keys) {
  const uint32_t inst = d.lp_inst[lp], c0 = d.count[lp];
  const float lim = pm_sel_bound(d, inst, s);
  const uint32_t prevb = (s + 1u) & 1u, lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  const uint32_t cap = 1u << d.cap_log2, mask = cap - 1u;
  const uint32_t rd = d.rd[lp], n = d.wr[lp] - rd;
  const uint32_t m = n + min(min(d.icnt[(size_t)prevb * d.max_lps + lp], d.ibc), cap - n);
  gpq_item* ring = d.ring + ((size_t)lp << d.cap_log2);
  const gpq_item* src = d.ibuf + ((size_t)prevb * d.max_lps + lp) * d.ibc;
  auto item = [=](uint32_t i) { return i < n ? ring[(rd + i) & mask] : src[i - n]; };
  uint32_t sc = 0;
  __syncwarp();
#pragma unroll 4
  for (uint32_t i0 = 0; i0 < m; i0 += 32u) {
    gpq_item e;
    bool safe = false;
    if (i0 + lane < m) {
      e = item(i0 + lane);
      safe = e.ts < lim;
    }
    const uint32_t b = __ballot_sync(GPQ_FULL_MASK, safe), pos = sc + (uint32_t)__popc(b & lt);
    if (safe && pos < kPmWideCap) keys[pos] = gpq_lp_key(e);
    sc += (uint32_t)__popc(b);
  }
  const bool fit = sc <= kPmWideCap;
  if (lane == 0 && fit && (sc & 1u)) keys[sc] = ~0ull;  // the rank reads pairs
  __syncwarp();
  const PmInstDev& I = d.inst[inst];
  const uint32_t top = fit ? sc : m;
  uint64_t cs = 0, os = 0;
  uint32_t cmin = kInfBits, ppos = ~0u;
  gpq_item pch;  // the child before, written once its place has come back
  bool pend = false;
  for (uint32_t i = lane; i < top; i += 32u) {
    unsigned long long key;
    uint32_t r = 0;
    if (fit) {  // equal keys by their place: those before the warp's 32 also count when equal
      key = keys[i];
      const uint32_t b = i - lane, e = min(b + 32u, sc);
#pragma unroll 4
      for (uint32_t t = 0; t < b; t += 2u) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(keys + t);
        r += (a.x <= key ? 1u : 0u) + (a.y <= key ? 1u : 0u);
      }
      for (uint32_t t = b; t < e; ++t) r += keys[t] < key || (keys[t] == key && t < i) ? 1u : 0u;
#pragma unroll 4
      for (uint32_t t = b + 32u; t < sc; t += 2u) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(keys + t);
        r += (a.x < key ? 1u : 0u) + (a.y < key ? 1u : 0u);
      }
    } else {
      const gpq_item e = item(i);
      if (!(e.ts < lim)) continue;
      key = gpq_lp_key(e);
      for (uint32_t j = 0; j < m; ++j) {
        const gpq_item o = item(j);
        const unsigned long long ko = gpq_lp_key(o);
        r += o.ts < lim && (ko < key || (ko == key && j < i)) ? 1u : 0u;
      }
    }
    uint64_t h, oh;
    const gpq_item ch = pm_sel_event(I.p, I.lp0, lp, key, (uint64_t)c0 + r, &h, &oh);
    cs += h;
    os += oh;
    cmin = min(cmin, gpq_f2u(ch.ts));
    const uint32_t pos = atomicAdd(&d.icnt[(size_t)(s & 1u) * d.max_lps + ch.lp], 1u);
    if (pend) pm_sel_file(d, s, inst, pch, ppos);
    pch = ch;
    ppos = pos;
    pend = true;
  }
  if (pend) pm_sel_file(d, s, inst, pch, ppos);
  cs = warp_sum_u64(cs);
  os = warp_sum_u64(os);
  __syncwarp();
  uint32_t kept = 0;
  for (uint32_t i0 = 0; i0 < m; i0 += 32u) {
    const uint32_t i = i0 + lane;
    gpq_item e;
    bool stay = false;
    if (i < m) {
      e = item(i);
      stay = !(e.ts < lim);
    }
    const uint32_t b = __ballot_sync(GPQ_FULL_MASK, stay);  // the items are read before any place is written
    if (stay) {
      const uint32_t at = kept + (uint32_t)__popc(b & lt);
      if (at != i || i >= n) ring[(rd + at) & mask] = e;
    }
    kept += (uint32_t)__popc(b);
    __syncwarp();
  }
  if (lane == 0) {
    d.csum[lp] += cs;
    d.ohash[lp] += os;
    d.count[lp] = c0 + sc;
    d.wr[lp] = rd + kept;
    d.lmin[lp] = 0u;
    d.icnt[(size_t)prevb * d.max_lps + lp] = 0u;
  }
  cmin = warp_min_u32(cmin);
  if (lane == 0 && cmin != kInfBits) atomicMin(&d.mins[3 * inst + (s + 1u) % 3u], cmin);
}

// The selection windows of one warp: turns of `lps` LPs (4 or 8), `stride` LPs apart, from
// lp_first until the last LP or until the list of LPs left to pm_select_wide is nearly full.
// Returns the first LP of the next turn.
static __device__ __forceinline__ uint32_t pm_select_turns(const PmDev& d, uint32_t s, uint32_t lp_first, uint32_t lps,
                                                           uint32_t stride, const float* s_bound, const PmSelSmem& sm,
                                                           uint32_t* n_wide) {
  constexpr uint32_t U = 6;  // items in flight per lane
  const uint32_t lane = threadIdx.x & 31u, gl = lane & 7u, grp = lane >> 3, sh = lane & 24u, lt = (1u << gl) - 1u;
  const uint32_t curb = s & 1u, prevb = curb ^ 1u;
  const uint32_t cap = 1u << d.cap_log2, mask = cap - 1u;
  // an LP's words, one per lane: its run, ring counters, children, committed count, minimum
  const uint32_t* mp = gl == 0   ? d.lp_inst
                       : gl == 1 ? d.rd
                       : gl == 2 ? d.wr
                       : gl == 3 ? d.icnt + (size_t)prevb * d.max_lps
                       : gl == 4 ? d.count
                                 : d.lmin;
  auto words = [&](uint32_t lp) { return gl < 6u && lp < d.n_lps ? mp[lp] : ~0u; };
  uint32_t meta = lp_first < d.n_lps ? words(lp_first + grp) : ~0u;
  uint32_t nw = 0, lp0 = lp_first;
  for (; lp0 < d.n_lps && nw <= kPmWides - kPmSelLps; lp0 += stride) {
    for (uint32_t q = 0; q < lps; q += 4u) {
      const uint32_t seg = q + grp, lp = lp0 + seg;
      const uint32_t inst = __shfl_sync(GPQ_FULL_MASK, meta, sh), rd = __shfl_sync(GPQ_FULL_MASK, meta, sh | 1u);
      const uint32_t wr = __shfl_sync(GPQ_FULL_MASK, meta, sh | 2u), kc = __shfl_sync(GPQ_FULL_MASK, meta, sh | 3u);
      const uint32_t c0 = __shfl_sync(GPQ_FULL_MASK, meta, sh | 4u), low = __shfl_sync(GPQ_FULL_MASK, meta, sh | 5u);
      meta = words((q + 4u < lps ? lp0 + q + 4u : lp0 + stride) + grp);  // the next LPs' words
      float lim = -1.f;
      if (inst != ~0u) lim = inst < kPmTab ? s_bound[inst] : pm_sel_bound(d, inst, s);
      const bool run = lim >= 0.f;
      uint32_t par = 0;
      if (run) par = reinterpret_cast<const uint32_t*>(d.inst + inst)[gl < 7u ? gl : 8u];
      const bool idle = run && kc == 0u && low >= gpq_f2u(lim);  // nothing new, nothing safe
      const uint32_t n = run && !idle ? wr - rd : 0u;
      uint32_t k = run ? min(kc, d.ibc) : 0u;  // an overflow was flagged by the inserter
      if (n + k > cap) {
        if (gl == 0) pm_error(d, inst, s, GPQ_ERR_QUEUE_FULL);
        k = cap - n;
      }
      const uint32_t m = n + k;
      gpq_item* ring = d.ring + ((size_t)lp << d.cap_log2);
      const gpq_item* src = d.ibuf + ((size_t)prevb * d.max_lps + lp) * d.ibc;
      unsigned long long* key = sm.key + seg * kPmSelStride;
      uint32_t* at = sm.at + seg * kPmSelStride;
      const uint32_t mmax = __reduce_max_sync(GPQ_FULL_MASK, m);
      uint32_t sc = 0, vmin = idle ? low : kInfBits;
      for (uint32_t b0 = 0; b0 < mmax; b0 += 8u * U) {
        uint32_t t[U], id[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
          const uint32_t i = b0 + u * 8u + gl;
          if (i < m) {
            const gpq_item e = i < n ? ring[(rd + i) & mask] : src[i - n];
            t[u] = gpq_f2u(e.ts);
            id[u] = e.id;
          }
        }
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
          const uint32_t i = b0 + u * 8u + gl;
          const bool safe = i < m && gpq_u2f(t[u]) < lim;
          const uint32_t b = (__ballot_sync(GPQ_FULL_MASK, safe) >> sh) & 0xffu;
          if (safe) {
            const uint32_t pos = sc + (uint32_t)__popc(b & lt);
            if (pos < kPmSelCap) {
              key[pos] = ((unsigned long long)t[u] << 32) | id[u];
              at[pos] = i;
            }
          } else if (i < m) {
            vmin = min(vmin, t[u]);
          }
          sc += (uint32_t)__popc(b);
        }
      }
#pragma unroll
      for (uint32_t o = 4; o > 0; o >>= 1) vmin = min(vmin, __shfl_xor_sync(GPQ_FULL_MASK, vmin, o));
      __syncwarp();
      // the ring's places [0, m - sc)
      const uint32_t n2 = m - sc;
      const bool wide = sc > kPmSelCap;
      const uint32_t hi = wide ? 0u : m;
      uint32_t moved = 0;
      for (uint32_t i = min(n, n2) + gl; __any_sync(GPQ_FULL_MASK, i < hi); i += 8u) {
        gpq_item e;
        bool stay = false;
        if (i < hi) {
          e = i < n ? ring[(rd + i) & mask] : src[i - n];
          stay = !(e.ts < lim);
        }
        const uint32_t b = (__ballot_sync(GPQ_FULL_MASK, stay && i >= n2) >> sh) & 0xffu;
        if (stay) ring[(rd + (i < n2 ? i : at[moved + (uint32_t)__popc(b & lt)])) & mask] = e;
        moved += (uint32_t)__popc(b);
      }
      sm.par[seg * 8u + gl] = par;
      if (gl == 0) {
        sm.beg[1u + seg] = wide ? 0u : sc;
        sm.c0[seg] = c0;
        sm.inst[seg] = run ? inst : ~0u;
        if ((sc & 1u) && !wide) key[sc] = ~0ull;  // the rank reads pairs
        if (run && !wide && !idle) {
          d.lmin[lp] = vmin;
          d.wr[lp] = rd + n2;
          if (kc) d.icnt[(size_t)prevb * d.max_lps + lp] = 0u;
          if (sc) d.count[lp] = c0 + sc;
        }
      }
      const uint32_t wb = __ballot_sync(GPQ_FULL_MASK, wide && gl == 0);
      if (wide && gl == 0) sm.wide[nw + (uint32_t)__popc(wb & ((1u << lane) - 1u))] = lp;
      nw += (uint32_t)__popc(wb);
      if (gl == 0) sm.mn[seg] = vmin;
    }
    if (lps == 4u && lane >= 4u && lane < 8u) {
      sm.beg[1u + lane] = 0u;
      sm.inst[lane] = ~0u;
      sm.mn[lane] = kInfBits;
    }
    __syncwarp();
    // the turn's events in the order of the LPs
    uint32_t incl = lane < kPmSelLps ? sm.beg[1u + lane] : 0u;
#pragma unroll
    for (int o = 1; o < (int)kPmSelLps; o <<= 1) {
      const uint32_t v = __shfl_up_sync(GPQ_FULL_MASK, incl, o);
      if (lane >= (uint32_t)o) incl += v;
    }
    const uint32_t total = __shfl_sync(GPQ_FULL_MASK, incl, kPmSelLps - 1);
    const uint32_t li = lane < kPmSelLps ? sm.inst[lane] : ~0u;
    const uint32_t act = __ballot_sync(GPQ_FULL_MASK, li != ~0u);
    __syncwarp();
    if (lane < kPmSelLps) sm.beg[1u + lane] = incl;
    if (lane == kPmSelLps) sm.beg[0] = 0u;
    if (act == 0u) {
      __syncwarp();
      continue;
    }
    const uint32_t inst0 = __shfl_sync(GPQ_FULL_MASK, li, __ffs(act) - 1);
    const bool one = __all_sync(GPQ_FULL_MASK, li == ~0u || li == inst0);  // all of one run
    __syncwarp();
    uint32_t ranks = 0;
    for (uint32_t y = lane; y < total; y += 32u) {  // rank
      uint32_t seg = 0;
#pragma unroll
      for (uint32_t j = 1; j < kPmSelLps; ++j) seg += y >= sm.beg[j] ? 1u : 0u;
      const uint32_t b = sm.beg[seg], ns = sm.beg[seg + 1u] - b, j = y - b;
      const unsigned long long kj = sm.key[seg * kPmSelStride + j];
      const ulonglong2* kp = reinterpret_cast<const ulonglong2*>(sm.key + seg * kPmSelStride);
      uint32_t r = 0;
#pragma unroll 2
      for (uint32_t t = 0; t < ns; t += 2u) {
        const ulonglong2 a = kp[t >> 1];
        r += (a.x < kj ? 1u : 0u) + (a.y < kj ? 1u : 0u);
      }
      sm.at[y] = (r << 16) | (seg << 8) | j;
      ranks += r;
    }
    {  // equal keys share a rank, which the ranks' sum tells
      const uint32_t ns = lane < kPmSelLps ? sm.beg[lane + 1u] - sm.beg[lane] : 1u;
      if (__reduce_add_sync(GPQ_FULL_MASK, ranks - ns * (ns - 1u) / 2u) != 0u) pm_sel_rank_equal(sm.key, sm.at, total);
    }
    __syncwarp();
    uint32_t cmin = kInfBits;
    gpq_item pch;  // the child before, written once its place has come back
    uint32_t ppos = 0, pin = ~0u;
    for (uint32_t y = lane; y < total; y += 32u) {  // process
      const uint32_t f = sm.at[y], seg = (f >> 8) & 0xffu, w = seg * kPmSelStride + (f & 0xffu);
      const uint4 p0 = reinterpret_cast<const uint4*>(sm.par + seg * 8u)[0], p1 = reinterpret_cast<const uint4*>(sm.par + seg * 8u)[1];
      gpq_phold_params p;
      p.seed = ((uint64_t)p0.y << 32) | p0.x;
      p.num_lps = p0.z;
      p.dest_mode = p0.w;
      p.ring_width = p1.x;
      p.ring_threshold = p1.y;
      p.lookahead = gpq_u2f(p1.z);
      p.end_time = 0.f;  // not read
      uint64_t h, oh;
      const gpq_item ch = pm_sel_event(p, p1.w, lp0 + seg, sm.key[w], (uint64_t)sm.c0[seg] + (f >> 16), &h, &oh);
      sm.key[w] = h;
      sm.oh[w] = oh;
      if (one) cmin = min(cmin, gpq_f2u(ch.ts));
      else atomicMin(&sm.mn[seg], gpq_f2u(ch.ts));
      const uint32_t pos = atomicAdd(&d.icnt[(size_t)curb * d.max_lps + ch.lp], 1u);
      if (pin != ~0u) pm_sel_file(d, s, pin, pch, ppos);
      pch = ch;
      ppos = pos;
      pin = sm.inst[seg];
    }
    if (pin != ~0u) pm_sel_file(d, s, pin, pch, ppos);
    __syncwarp();
    {  // the LPs' sums: two lanes each
      const uint32_t seg = lane >> 2, ns = sm.beg[seg + 1u] - sm.beg[seg];
      const unsigned long long* v = ((lane & 1u) ? sm.oh : sm.key) + seg * kPmSelStride;
      unsigned long long sum = 0;
      for (uint32_t t = (lane >> 1) & 1u; t < ns; t += 2u) sum += v[t];
      sum += __shfl_xor_sync(GPQ_FULL_MASK, sum, 2);
      if (ns && !(lane & 2u)) atomicAdd(((lane & 1u) ? d.ohash : d.csum) + lp0 + seg, sum);
    }
    // one minimum per run
    const uint32_t lm = lane < kPmSelLps ? sm.mn[lane] : kInfBits;
    if (one) {
      const uint32_t v = __reduce_min_sync(GPQ_FULL_MASK, min(lm, cmin));
      if (lane == 0 && v != kInfBits) atomicMin(&d.mins[3 * inst0 + (s + 1u) % 3u], v);
    } else if (li != ~0u && lm != kInfBits) {
      atomicMin(&d.mins[3 * li + (s + 1u) % 3u], lm);
    }
    __syncwarp();
  }
  *n_wide = nw;
  return lp0;
}

// Windows s0, s0 + 1, ... while some instance is running, at most step_windows of them
// (0 = no limit).  Dynamic shared memory: pm_sel_warp_bytes() per warp.
static __global__ void __launch_bounds__(256, 3) pm_persistent_kernel(const __grid_constant__ PmDev d, uint32_t s0, uint32_t step_windows) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_any;
  __shared__ float s_bound[kPmTab];
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
  unsigned long long target = 0;
  uint32_t s = s0;
  for (;; ++s) {
    // every block takes the same decision from the same slots
    if (threadIdx.x == 0) s_any = 0;
    __syncthreads();
    int any = 0;
    for (uint32_t i = threadIdx.x; i < d.n_inst && !any; i += blockDim.x) any = pm_active(d, i, s);
    if (any) s_any = 1;
    __syncthreads();
    if (!s_any || ld_relaxed_u32(&d.ctl->err) != 0u || (step_windows && s - s0 >= step_windows)) break;
    for (uint32_t i = tid; i < d.n_inst; i += nthreads) {
      if (pm_active(d, i, s)) d.inst[i].windows += 1u;
      d.mins[3 * i + (s + 2u) % 3u] = kInfBits;  // slots of window s + 2, last read in window s - 1
      d.errs[3 * i + (s + 2u) % 3u] = 0u;
    }
    for (uint32_t i = threadIdx.x; i < min(d.n_inst, kPmTab); i += blockDim.x) s_bound[i] = pm_sel_bound(d, i, s);
    __syncthreads();
    const uint32_t wpb = blockDim.x >> 5, warps = gridDim.x * wpb, w = blockIdx.x * wpb + (threadIdx.x >> 5);
    const uint32_t lps = d.n_lps > warps * 4u ? kPmSelLps : kPmSelLps / 2;
    const PmSelSmem sm = pm_sel_smem(smem_raw + (size_t)(threadIdx.x >> 5) * pm_sel_warp_bytes());
    for (uint32_t lp = w * lps; lp < d.n_lps;) {
      uint32_t nw;
      lp = pm_select_turns(d, s, lp, lps, warps * lps, s_bound, sm, &nw);
      for (uint32_t j = 0; j < nw; ++j) pm_select_wide(d, s, sm.wide[j], sm.key);
    }
    target += gridDim.x;
    if (!grid_barrier(&d.ctl->bar, target, d.spin_limit, &d.ctl->err)) {
      s += 1u;
      break;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) d.ctl->phase = s;
}

// Initial events of the instances in list[0, n): one warp per LP of each, sorted into
// the ring (ids lp * per_lp + k over local LPs), per-LP outputs zeroed, the instance's
// first minimum into its slot for window s.  blockIdx.y = position in the list.
// Dynamic shared memory: per_lp items and keys per warp.
static __global__ void pm_populate_kernel(PmDev d, const uint32_t* list, uint32_t s) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t inst = list[blockIdx.y];
  const PmInstDev I = d.inst[inst];
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const uint32_t P = I.per_lp;
  gpq_item* s_it = reinterpret_cast<gpq_item*>(smem_raw) + (size_t)wib * P;
  uint64_t* s_key = reinterpret_cast<uint64_t*>(reinterpret_cast<gpq_item*>(smem_raw) + (size_t)wpb * P) + (size_t)wib * P;
  for (uint32_t l = blockIdx.x * wpb + wib; l < I.p.num_lps; l += gridDim.x * wpb) {
    const uint32_t lp = I.lp0 + l;
    gpq_item* ring = d.ring + ((size_t)lp << d.cap_log2);
    uint32_t mn = kInfBits;
    for (uint32_t j = lane; j < P; j += 32) {
      const gpq_item e = gpq_phold_initial(I.p, l, j, P);
      s_it[j] = e;
      s_key[j] = gpq_lp_key(e);
      mn = min(mn, gpq_f2u(e.ts));
    }
    __syncwarp();
    for (uint32_t j = lane; j < P; j += 32) {
      const uint64_t kj = s_key[j];
      uint32_t r = 0;  // rank among the LP's initial events
      for (uint32_t i = 0; i < P; ++i) r += s_key[i] < kj ? 1u : 0u;
      gpq_item e = s_it[j];
      e.lp = lp;
      ring[r] = e;
    }
    __syncwarp();
    mn = warp_min_u32(mn);
    if (lane == 0) {
      d.rd[lp] = 0;
      d.wr[lp] = P;
      d.lmin[lp] = 0;
      d.icnt[lp] = 0;
      d.icnt[(size_t)d.max_lps + lp] = 0;
      d.count[lp] = 0;
      d.csum[lp] = 0;
      d.ohash[lp] = 0;
      d.lp_inst[lp] = inst;
      if (mn != kInfBits) atomicMin(&d.mins[3 * inst + s % 3u], mn);
    }
  }
}

// Results of the finished instances in list[0, n): committed count, pending events (ring
// contents and the unmerged children of the instance's last window), the digest over
// local LP numbers, the pending minimum.  blockIdx.y = position in the list.
struct PmAcc {
  unsigned long long committed, pending, pending_csum, digest;
  uint32_t pending_min;
  uint32_t pad;
};

static __global__ void pm_finalize_kernel(PmDev d, const uint32_t* list, PmAcc* acc) {
  const uint32_t j = blockIdx.y;
  const PmInstDev I = d.inst[list[j]];
  const uint32_t lane = threadIdx.x & 31u, wpb = blockDim.x >> 5;
  const uint32_t s = I.w0 + I.windows;  // the instance's first inactive window
  const uint32_t prevb = (s + 1u) & 1u;
  const uint32_t mask = (1u << d.cap_log2) - 1u;
  uint64_t pend = 0, pcs = 0, dig = 0, com = 0;
  uint32_t pmin = kInfBits;
  for (uint32_t l = blockIdx.x * wpb + (threadIdx.x >> 5); l < I.p.num_lps; l += gridDim.x * wpb) {
    const uint32_t lp = I.lp0 + l;
    const gpq_item* ring = d.ring + ((size_t)lp << d.cap_log2);
    const uint32_t rd = d.rd[lp], n = d.wr[lp] - rd;
    for (uint32_t q = lane; q < n; q += 32) {
      const gpq_item e = ring[(rd + q) & mask];
      pcs += gpq_ev_hash(e.id, gpq_f2u(e.ts));
      pend += 1;
      pmin = min(pmin, gpq_f2u(e.ts));
    }
    const uint32_t k = min(d.icnt[(size_t)prevb * d.max_lps + lp], d.ibc);
    const gpq_item* src = d.ibuf + ((size_t)prevb * d.max_lps + lp) * d.ibc;
    for (uint32_t q = lane; q < k; q += 32) {
      const gpq_item e = src[q];
      pcs += gpq_ev_hash(e.id, gpq_f2u(e.ts));
      pend += 1;
      pmin = min(pmin, gpq_f2u(e.ts));
    }
    if (lane == 0) {
      const uint32_t c = d.count[lp];
      com += c;
      dig += gpq_mix64(gpq_mix64(gpq_mix64(((uint64_t)l << 32) | c) ^ d.csum[lp]) + d.ohash[lp]);
    }
  }
  pend = warp_sum_u64(pend);
  pcs = warp_sum_u64(pcs);
  dig = warp_sum_u64(dig);
  com = warp_sum_u64(com);
  pmin = warp_min_u32(pmin);
  if (lane == 0) {
    atomicAdd(&acc[j].pending, (unsigned long long)pend);
    atomicAdd(&acc[j].pending_csum, (unsigned long long)pcs);
    atomicAdd(&acc[j].digest, (unsigned long long)dig);
    atomicAdd(&acc[j].committed, (unsigned long long)com);
    atomicMin(&acc[j].pending_min, pmin);
  }
}

// Slots in use whose run ended (minimum at or past the end time, or an error) at window s.
static __global__ void pm_done_list_kernel(PmDev d, uint32_t s, uint32_t* out, uint32_t* out_n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < d.n_inst; i += gridDim.x * blockDim.x)
    if (d.on[i] && !pm_active(d, i, s)) out[atomicAdd(out_n, 1u)] = i;
}

// Release the LPs of the instances in list[0, n).
static __global__ void pm_release_kernel(PmDev d, const uint32_t* list) {
  const PmInstDev I = d.inst[list[blockIdx.y]];
  for (uint32_t l = blockIdx.x * blockDim.x + threadIdx.x; l < I.p.num_lps; l += gridDim.x * blockDim.x)
    d.lp_inst[I.lp0 + l] = ~0u;
}
