// A* grid search on the GPU: many instances, each grid cut into square tiles (the
// shards of the open list), one persistent cooperative launch over rounds.
//
// Reference: src/a_star.cu:269-593 runs one best-first search per agent in one CTA,
// popping up to eight open-list minima per round from the agent's queue
// (queue_peek/queue_set_done/queue_insert_or_update, src/queue.cuh:46-70).  Here the
// open list of an instance is sharded by tile, and a round drains every tile's items
// inside the instance's current window f <= bound:
//
//   * phase P: each active tile is taken by one CTA.  Its inbox (items sent by other
//     tiles in the previous round) and, when the window moved, its open array are
//     scanned; stale items (g above the cell's current g) are dropped, items above the
//     instance's best goal cost UB are pruned, items with f <= bound join the CTA's
//     frontier in shared memory and the rest stay in the open array.  The CTA then
//     relaxes the whole tile from them in sweeps (astar_sweep_tile), or -- other tile
//     sides, small CTAs, warps -- expands the frontier level by level: a child whose g
//     improves (atomicMin on the cell's g) goes to the next frontier when it lies in the
//     tile and in the window, to the tile's open array when above the window, or to the
//     owning tile's inbox for the next round.
//   * phase W: an instance whose tiles sent nothing for the next round has drained its
//     window; the window moves to [min f of its open arrays, + delta], or the instance
//     is done when that minimum exceeds UB.  The CTA that makes the instance's last visit
//     of a round decides this, so a round has one grid barrier.
//
// Work items are 8 bytes (y << 16 | x, g); f = g + h(x, y) is recomputed, so the hot loop
// needs no division.  With a consistent
// heuristic every cell with g + h <= C* ends with its exact g, whatever the order of
// expansions, so the outputs (C*, the expanded set, the canonical path) do not depend
// on the schedule; re-expansions only cost time.
#pragma once

#include "common.cuh"
#include "gpq/astar.h"

static constexpr uint32_t kAstarInf = GPQ_ASTAR_INF;

namespace gpq {
// Defaults and limits of the engine knobs (host side, astar.cu).
gpq_status astar_normalize(gpq_astar_config& c);
}  // namespace gpq

struct AstarInstDev {
  gpq_astar_grid g;
  uint64_t cell0;      // first cell in the shared g array and bitmap (a multiple of 32)
  uint32_t tile0;      // first tile
  uint32_t tiles_x, tiles_y;
  uint32_t ub;         // best goal cost found so far
  uint32_t bound;      // window: items with f <= bound are expanded
  uint32_t active[2];  // active tiles of the round with this parity
  uint32_t visited;    // of the current round's active tiles
  uint32_t done;
  uint32_t err;
  uint32_t windows;
  uint32_t delta;      // window width on f
  unsigned long long pops;  // expansions performed (re-expansions included)
  uint32_t gx, gy;     // goal coordinates
};

struct AstarTileDev {
  uint32_t inst;
  uint32_t tx, ty;
  uint32_t in_cnt[2];  // inbox fill per round parity
  uint32_t open_cnt;   // open array fill
  uint32_t open_min;   // min f in the open array (kAstarInf when empty)
  uint32_t queued[2];  // on the active list of the round with this parity
  uint32_t pad[3];
};

// Control words of one launch.
struct AstarCtl {
  uint32_t al_cnt[3];  // active tiles by round mod 3: read in this round, filled for the next, cleared
  uint32_t work[3];    // tiles handed out beyond each worker's first
  uint32_t err;
  uint32_t rounds;
  unsigned long long bar;
  unsigned long long visits;  // tiles processed
};

struct AstarDev {
  AstarInstDev* inst;
  AstarTileDev* tiles;
  uint32_t* gcost;  // [cells]
  const uint32_t* blk;  // blocked bitmap, one bit per cell
  uint8_t* pred;    // [cells + kAstarPredSlack] move to the canonical predecessor (astar_pred_kernel)
  uint2* inbox;     // [2][n_tiles][in_cap] (cell, g)
  uint2* open;      // [n_tiles][open_cap]
  uint32_t* al;     // [2][n_tiles] active tiles per round parity
  AstarCtl* ctl;
  uint32_t n_inst, n_tiles;
  uint32_t in_cap, open_cap;
  uint32_t ts;      // tile side
  uint32_t lts;     // log2(ts)
  uint32_t max_rounds;
  uint32_t frontier_cap;  // per shared frontier buffer
  uint64_t spin_limit;
};

// Bytes after the last cell of the predecessor array: path windows read whole words.
static constexpr uint64_t kAstarPredSlack = 256;

__device__ __forceinline__ uint32_t ldcg_u32(const uint32_t* p) { return __ldcg(p); }

__device__ __forceinline__ bool astar_blocked(const AstarDev& d, const AstarInstDev& I, uint32_t cell) {
  const uint64_t b = I.cell0 + cell;
  return (__ldg(&d.blk[b >> 5]) >> (b & 31u)) & 1u;
}

__device__ __forceinline__ uint32_t astar_tile_of(const AstarDev& d, const AstarInstDev& I, uint32_t cell) {
  const uint32_t x = cell % I.g.width, y = cell / I.g.width;
  return I.tile0 + (y / d.ts) * I.tiles_x + x / d.ts;
}

__device__ __forceinline__ uint32_t astar_hxy(uint32_t conn, int x, int y, int gx, int gy) {
  const uint32_t dx = (uint32_t)abs(x - gx), dy = (uint32_t)abs(y - gy);
  return conn == 4 ? dx + dy : 10u * max(dx, dy) + 4u * min(dx, dy);
}

__device__ __forceinline__ uint32_t astar_pack(int x, int y) { return ((uint32_t)y << 16) | (uint32_t)x; }

// Put tile t on the active list of a round (once per round).
__device__ __forceinline__ void astar_activate(const AstarDev& d, AstarInstDev* Ip, uint32_t t, uint32_t round) {
  const uint32_t par = round & 1u;
  if (atomicExch(&d.tiles[t].queued[par], 1u) == 0u) {
    const uint32_t pos = atomicAdd(&d.ctl->al_cnt[round % 3u], 1u);
    d.al[(size_t)par * d.n_tiles + pos] = t;
    atomicAdd(&Ip->active[par], 1u);
  }
}

// An item into a tile's inbox of a round.
__device__ __forceinline__ void astar_inbox_push(const AstarDev& d, AstarInstDev* Ip, uint32_t t, uint32_t round,
                                                 uint2 it) {
  const uint32_t par = round & 1u;
  const uint32_t pos = atomicAdd(&d.tiles[t].in_cnt[par], 1u);
  if (pos < d.in_cap) {
    d.inbox[((size_t)par * d.n_tiles + t) * d.in_cap + pos] = it;
  } else {
    gpq_set_error(&Ip->err, GPQ_ERR_INSERT_FULL);
  }
  astar_activate(d, Ip, t, round);
}

// Shared state of the CTA working on one tile.  While a CTA holds a tile, the tile's g
// values live in shared memory (gt) and only this CTA changes them; other tiles lower the
// global copy with atomicMin (a filter for their sends) and the holder merges its copy
// back with atomicMin when it lets go of the tile.
struct AstarTileSmem {
  uint2* fa;      // items to expand at the start of the visit; frontier buffer [frontier_cap]
  uint2* fb;      // list walk: second frontier buffer
  uint32_t* gt;   // [ts * ts] g of the tile's cells, local index ly * ts + lx
  uint32_t* blk;  // [ts * ts / 32] blocked bits of the tile
  uint32_t* chg;  // list walk: [ts * ts / 32] cells whose g dropped during this visit
  uint2* ob;      // list walk: [8 * ts] moves into other tiles, sent when the visit ends
  uint16_t* vs;   // sweeps: [ts + 2][astar_sweep_stride] g - g_min of the expanded cells
  uint32_t moved[3];  // sweeps: warps whose cells changed, by barrier mod 3
  uint32_t ob_n;
  uint32_t n[3];  // frontier fill, rotating by level
  uint32_t ub;    // the instance's best goal cost as of this visit (stale values only prune less)
  uint32_t open_min;
  uint32_t open_cnt;
  uint32_t g_min;  // of the items to expand
  uint32_t last;   // this visit was its instance's last of the round
  uint32_t out_n[9], out_base[9];  // sweeps: moves into each neighbour tile, their place in its inbox
  unsigned long long pops;
  uint32_t scan[33];
};

__host__ __device__ inline uint32_t astar_outbox_cap(uint32_t ts) { return 8u * ts; }

// How a visit walks its tile: a CTA with a thread for 8 or for 16 cells sweeps tiles of
// 64 x 64 and 32 x 32 cells (astar_sweep_tile); other tile sides, smaller CTAs, and tiles
// worked by one warp keep frontier lists (astar_expand_warp).  Returns the pairs of cells
// a thread holds (4 or 8), or 0 for lists.
__host__ __device__ inline uint32_t astar_sweep_pairs(uint32_t ts, bool warp, uint32_t block) {
  if (warp || (ts != 64u && ts != 32u)) return 0;
  return block >= ts * ts / 8u ? 4u : block >= ts * ts / 16u ? 8u : 0u;
}

// 16-bit cells of a row in shared memory: 8 in front of the tile's (a 16-byte border, of which
// the last is the left neighbour) and 16 behind.
__host__ __device__ inline uint32_t astar_sweep_stride(uint32_t ts) { return ts + 24u; }

__host__ __device__ inline size_t astar_smem_bytes(uint32_t ts, uint32_t frontier_cap, bool warp, uint32_t block) {
  const size_t cells = (size_t)ts * ts, words = cells / 32;
  if (astar_sweep_pairs(ts, warp, block))
    return (size_t)(ts + 2u) * astar_sweep_stride(ts) * sizeof(uint16_t) + (size_t)frontier_cap * sizeof(uint2) +
           cells * sizeof(uint32_t) + words * sizeof(uint32_t);
  return 2ull * frontier_cap * sizeof(uint2) + (size_t)astar_outbox_cap(ts) * sizeof(uint2) +
         cells * sizeof(uint32_t) + 2ull * words * sizeof(uint32_t);
}

__device__ __forceinline__ void astar_smem_carve(AstarTileSmem& sm, unsigned char* base, uint32_t ts,
                                                 uint32_t frontier_cap, bool warp) {
  const uint32_t words = ts * ts / 32;
  if (astar_sweep_pairs(ts, warp, blockDim.x)) {
    sm.vs = reinterpret_cast<uint16_t*>(base);
    sm.gt = reinterpret_cast<uint32_t*>(sm.vs + (ts + 2u) * astar_sweep_stride(ts));
    sm.fa = reinterpret_cast<uint2*>(sm.gt + ts * ts);
    sm.blk = reinterpret_cast<uint32_t*>(sm.fa + frontier_cap);
    return;
  }
  sm.fa = reinterpret_cast<uint2*>(base);
  sm.fb = sm.fa + frontier_cap;
  sm.ob = sm.fb + frontier_cap;
  sm.gt = reinterpret_cast<uint32_t*>(sm.ob + astar_outbox_cap(ts));
  sm.blk = sm.gt + ts * ts;
  sm.chg = sm.blk + words;
}

// Geometry of the tile being processed.
struct AstarTileGeo {
  uint32_t x0, y0, tw, th, ts;
  __device__ __forceinline__ bool inside(int x, int y) const {
    return x >= (int)x0 && y >= (int)y0 && x < (int)(x0 + tw) && y < (int)(y0 + th);
  }
  uint32_t lts;
  __device__ __forceinline__ uint32_t local(int x, int y) const {
    return (((uint32_t)y - y0) << lts) + ((uint32_t)x - x0);
  }
};

// The threads that process one tile visit: the whole CTA, or one warp (WARP), in which
// case every warp of the CTA works on its own tile with its own slice of shared memory.
template <bool WARP>
struct AstarWorker {
  uint32_t tid;  // thread within the worker
  uint32_t n;    // threads in the worker
  uint32_t id;   // worker within the CTA
  __device__ __forceinline__ AstarWorker() {
    if (WARP) {
      tid = threadIdx.x & 31u;
      n = 32u;
      id = threadIdx.x >> 5;
    } else {
      tid = threadIdx.x;
      n = blockDim.x;
      id = 0;
    }
  }
  __device__ __forceinline__ void sync() const {
    if (WARP) __syncwarp();
    else __syncthreads();
  }
};

// Frontier push: into the shared buffer, or (when it is full) into the tile's own inbox
// for the next round.
__device__ __forceinline__ void astar_frontier_push(const AstarDev& d, AstarInstDev* Ip, AstarTileSmem& sm,
                                                    uint2* buf, uint32_t which, uint32_t t, uint32_t next_round, uint2 it) {
  const uint32_t pos = atomicAdd(&sm.n[which], 1u);
  if (pos < d.frontier_cap) {
    buf[pos] = it;
  } else {
    astar_inbox_push(d, Ip, t, next_round, it);
  }
}

__device__ __forceinline__ void astar_open_push(const AstarDev& d, AstarInstDev* Ip, AstarTileSmem& sm, uint32_t t,
                                                uint2 it, uint32_t f) {
  const uint32_t pos = atomicAdd(&sm.open_cnt, 1u);
  if (pos < d.open_cap) {
    d.open[(size_t)t * d.open_cap + pos] = it;
    atomicMin(&sm.open_min, f);
  } else {
    gpq_set_error(&Ip->err, GPQ_ERR_QUEUE_FULL);
  }
}

__device__ __forceinline__ bool astar_cell_blocked(const AstarDev& d, const AstarInstDev& I, const AstarTileSmem& sm,
                                                   const AstarTileGeo& tg, int x, int y) {
  if (tg.inside(x, y)) {
    const uint32_t l = tg.local(x, y);
    return (sm.blk[l >> 5] >> (l & 31u)) & 1u;
  }
  return astar_blocked(d, I, (uint32_t)y * I.g.width + (uint32_t)x);
}

// A move into another tile: lower the cell's global g (the filter), and when that
// improves it, send the item to the owning tile's inbox for the next round.
__device__ __forceinline__ void astar_send(const AstarDev& d, AstarInstDev* Ip, const AstarInstDev& I, uint2 it,
                                           uint32_t next_round) {
  const int x = (int)(it.x & 0xffffu), y = (int)(it.x >> 16);
  const uint32_t ng = it.y;
  if (ng >= atomicMin(&d.gcost[I.cell0 + (uint32_t)y * I.g.width + (uint32_t)x], ng)) return;
  const uint32_t nf = ng + astar_hxy(I.g.conn, x, y, (int)I.gx, (int)I.gy);
  if (x == (int)I.gx && y == (int)I.gy) atomicMin(&Ip->ub, ng);
  if (nf > ldcg_u32(&Ip->ub)) return;
  const uint32_t nt = I.tile0 + ((uint32_t)y >> d.lts) * I.tiles_x + ((uint32_t)x >> d.lts);
  astar_inbox_push(d, Ip, nt, next_round, it);
}

// Expand frontier items src[ib .. ib + 32 / M) with one warp, one lane per (item, move):
// lane = item * M + move, M = 4 or 8 moves (all lanes call; ib is warp-uniform).  A level
// of few items thus costs the latency of one move, not of M moves in a row.  Children
// are appended with one shared atomic per warp and target: the frontier and the open
// array are the two hot counters of a level.
__device__ __forceinline__ void astar_expand_warp(const AstarDev& d, AstarInstDev* Ip, const AstarInstDev& I,
                                                  AstarTileSmem& sm, const AstarTileGeo& tg, const uint2* src,
                                                  uint32_t ib, uint32_t n, uint2* next, uint32_t which, uint32_t t,
                                                  uint32_t next_round, uint32_t bound, uint32_t* pops) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t conn = I.g.conn;
  const uint32_t M = conn == 4 ? 4u : 8u;
  const uint32_t k = lane & (M - 1u);
  const uint32_t i = ib + lane / M;
  uint32_t kind = 0;  // 1 frontier, 2 open array, 4 outbox (another tile)
  uint2 child = make_uint2(0, 0);
  uint32_t nf = kAstarInf;
  if (i < n) {
    const uint2 it = src[i];
    const int x = (int)(it.x & 0xffffu), y = (int)(it.x >> 16);
    const uint32_t g = it.y;
    if (sm.gt[tg.local(x, y)] == g) {  // else a better path reached the cell meanwhile
      if (k == 0) ++*pops;
      const uint32_t w = I.g.width, h = I.g.height;
      const int nx = x + gpq_astar_dx((int)k), ny = y + gpq_astar_dy((int)k);
      if (nx >= 0 && ny >= 0 && nx < (int)w && ny < (int)h) {
        const bool in = tg.inside(nx, ny);
        const uint32_t l = in ? tg.local(nx, ny) : 0u;
        bool ok = !(in ? ((sm.blk[l >> 5] >> (l & 31u)) & 1u) : astar_blocked(d, I, (uint32_t)ny * w + (uint32_t)nx));
        if (ok && k >= 4) ok = !astar_cell_blocked(d, I, sm, tg, nx, y) && !astar_cell_blocked(d, I, sm, tg, x, ny);
        if (ok) {
          const uint32_t ng = g + gpq_astar_cost(conn, (int)k);
          if (in) {
            ok = ng < atomicMin(&sm.gt[l], ng);
            if (ok) atomicOr(&sm.chg[l >> 5], 1u << (l & 31u));
          } else {
            kind = 4u;  // to the outbox: filtered and sent when the visit ends
            child = make_uint2(astar_pack(nx, ny), ng);
            ok = false;
          }
          if (ok) {
            const int gx = (int)I.gx, gy = (int)I.gy;
            nf = ng + astar_hxy(conn, nx, ny, gx, gy);
            if (nx == gx && ny == gy) {
              atomicMin(&Ip->ub, ng);
              atomicMin(&sm.ub, ng);
            }
            if (nf <= sm.ub) {
              child = make_uint2(astar_pack(nx, ny), ng);
              kind = nf <= bound ? 1u : 2u;
            }
          }
        }
      }
    }
  }
  const uint32_t mf = __ballot_sync(GPQ_FULL_MASK, kind == 1u);
  if (mf) {
    const uint32_t leader = (uint32_t)(__ffs(mf) - 1);
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(&sm.n[which], (uint32_t)__popc(mf));
    base = __shfl_sync(GPQ_FULL_MASK, base, leader);
    if (kind == 1u) {
      const uint32_t pos = base + __popc(mf & lt);
      if (pos < d.frontier_cap) next[pos] = child;
      else astar_inbox_push(d, Ip, t, next_round, child);  // full: the tile's own next round
    }
  }
  const uint32_t mx = __ballot_sync(GPQ_FULL_MASK, kind == 4u);
  if (mx) {
    const uint32_t leader = (uint32_t)(__ffs(mx) - 1);
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(&sm.ob_n, (uint32_t)__popc(mx));
    base = __shfl_sync(GPQ_FULL_MASK, base, leader);
    if (kind == 4u) {
      const uint32_t pos = base + __popc(mx & lt);
      if (pos < astar_outbox_cap(tg.ts)) sm.ob[pos] = child;
      else astar_send(d, Ip, I, child, next_round);  // full: send now
    }
  }
  const uint32_t mo = __ballot_sync(GPQ_FULL_MASK, kind == 2u);
  if (mo) {
    const uint32_t leader = (uint32_t)(__ffs(mo) - 1);
    const uint32_t fmin = __reduce_min_sync(GPQ_FULL_MASK, kind == 2u ? nf : kAstarInf);
    uint32_t base = 0;
    if (lane == leader) {
      base = atomicAdd(&sm.open_cnt, (uint32_t)__popc(mo));
      atomicMin(&sm.open_min, fmin);
    }
    base = __shfl_sync(GPQ_FULL_MASK, base, leader);
    if (kind == 2u) {
      const uint32_t pos = base + __popc(mo & lt);
      if (pos < d.open_cap) d.open[(size_t)t * d.open_cap + pos] = child;
      else gpq_set_error(&Ip->err, GPQ_ERR_QUEUE_FULL);
    }
  }
}

// Block-wide exclusive prefix sum of 0/1 flags; returns this thread's offset and writes
// the total to *total.  All threads call.
__device__ __forceinline__ uint32_t astar_block_scan(uint32_t flag, uint32_t* scratch, uint32_t* total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t bal = __ballot_sync(GPQ_FULL_MASK, flag);
  const uint32_t below = __popc(bal & ((1u << lane) - 1u));
  if (lane == 0) scratch[warp] = __popc(bal);
  __syncthreads();
  if (warp == 0) {
    const uint32_t nw = blockDim.x >> 5;
    uint32_t v = lane < nw ? scratch[lane] : 0u;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(GPQ_FULL_MASK, incl, o);
      if (lane >= (uint32_t)o) incl += u;
    }
    if (lane < nw) scratch[lane] = incl - v;
    if (lane == 31) scratch[32] = incl;
  }
  __syncthreads();
  const uint32_t off = scratch[warp] + below;
  *total = scratch[32];
  __syncthreads();
  return off;
}

template <bool WARP>
__device__ __forceinline__ uint32_t astar_worker_scan(uint32_t flag, uint32_t* scratch, uint32_t* total) {
  if (WARP) {
    const uint32_t bal = __ballot_sync(GPQ_FULL_MASK, flag);
    *total = (uint32_t)__popc(bal);
    return (uint32_t)__popc(bal & ((1u << (threadIdx.x & 31u)) - 1u));
  }
  return astar_block_scan(flag, scratch, total);
}

// ---- sweeps ----
//
// The labels of a visit come from relaxing the whole tile until nothing changes: a thread
// holds 16 cells of a row as 15-bit labels (g - g_min of the visit's items), two to a
// register, and one sweep takes the minimum over a cell's neighbours with the packed
// add-minimum instructions.  A search is a chain of visits -- a round waits for its slowest
// tile -- and a visit's time is its number of steps times the latency of one: a sweep moves
// every wavefront of the tile by one cell in about 250 cycles without lists, atomics or
// per-cell branches, where a level of a frontier list costs a pass through shared-memory
// counters and appends.  Warps whose rows and neighbour rows did not change skip a sweep.
// Measured, search only, against frontier lists: 2048 x 2048 4-connected 8.05 -> 1.95 ms, 500
// 8-connected searches of sides 64 to 1,024 12.0 -> 3.2 ms.
//
// Only cells that this visit labels, and its items, pass their label on, and only inside
// the window (label < K): the others' moves were made when they were labelled.  Labels only
// fall, so a sweep may read a neighbour's label before or after its update.

static constexpr uint32_t kSweepInf = 0x7fffu;        // no label
static constexpr uint32_t kSweepInf2 = 0x7fff7fffu;
static constexpr uint32_t kSweepSpan = 0x7f00u;       // larger labels are not passed on in this visit
// Sweeps of a warp between barriers (fewer when its cells stop changing): with 16 cells a
// thread the 2048 x 2048 search took 3.69 / 3.07 / 2.64 / 2.45 ms with 1 / 2 / 4 / 8.
static constexpr uint32_t kSweepsPerBarrier = 8;
static constexpr uint32_t kSweepMax = 1u << 16;       // sweeps of one visit (at most one per cell is needed)

__device__ __forceinline__ uint32_t astar_pair_perm(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

// The labels v below k, the others as "no label" (both halves; k as (k | 0x8000) - 1).
__device__ __forceinline__ uint32_t astar_pair_below(uint32_t v, uint32_t k1) {
  const uint32_t ok = astar_pair_perm(k1 - v, 0u, 0xbb99u);  // the halves' top bits, spread: v < k
  return v | (~ok & kSweepInf2);
}

// Pairs shifted by one cell along a row of NP pairs p with neighbours a (left) and b (right).
__device__ __forceinline__ uint32_t astar_pair_left(const uint32_t* p, int i, uint32_t a) {
  return astar_pair_perm(i ? p[i ? i - 1 : 0] : a, p[i], 0x5432u);
}
template <int NP>
__device__ __forceinline__ uint32_t astar_pair_right(const uint32_t* p, int i, uint32_t b) {
  return astar_pair_perm(p[i], i < NP - 1 ? p[i < NP - 1 ? i + 1 : 0] : b, 0x5432u);
}

template <int NP>
__device__ __forceinline__ void astar_load_row(const uint16_t* row, uint32_t* p, uint32_t& a, uint32_t& b) {
#pragma unroll
  for (int q = 0; q < NP / 4; ++q) {
    const uint4 u = *reinterpret_cast<const uint4*>(row + 8 * q);
    p[4 * q] = u.x;
    p[4 * q + 1] = u.y;
    p[4 * q + 2] = u.z;
    p[4 * q + 3] = u.w;
  }
  a = *reinterpret_cast<const uint32_t*>(row - 2);
  b = *reinterpret_cast<const uint32_t*>(row + 2 * NP);
}

// Walks the tile from the n items of sm.fa (all threads; sm.g_min is set, sm.vs all "no
// label").  On return sm.vs holds the labels of the expanded cells; changed labels are
// merged into the global g values, labelled cells above the window are in the open array.
// DIAG: 8-connected, costs 10 and 14; else unit moves.  NP: pairs of cells of a thread; a
// warp holds a block of 16 rows x 4 * NP columns, so that a wavefront crossing the tile
// occupies few of them.
template <bool DIAG, int NP>
__device__ __forceinline__ void astar_sweep_tile(const AstarDev& d, AstarInstDev* Ip, const AstarInstDev& I,
                                                 AstarTileSmem& sm, const AstarTileGeo& tg, uint32_t n, uint32_t t,
                                                 uint32_t next_round, uint32_t bound, uint32_t* pops) {
  constexpr uint32_t kStraight = DIAG ? 0x000a000au : 0x00010001u;
  const uint32_t ts = tg.ts, lts = tg.lts, tid = threadIdx.x, stride = astar_sweep_stride(ts);
  const uint32_t warp = tid >> 5, lane = tid & 31u;
  const uint32_t bcols = ts / (4u * NP), brow = warp / bcols, bcol = warp % bcols;  // the warp's block
  const uint32_t y = brow * 16u + (lane >> 1), xs = bcol * (4u * NP) + (lane & 1u) * (2u * NP);
  const bool on = y < ts;
  // blocks whose changes concern this one: itself and its neighbours
  uint32_t near = 0;
  for (int i = -1; i <= 1; ++i)
    for (int j = -1; j <= 1; ++j) {
      const int r = (int)brow + i, c = (int)bcol + j;
      if (r >= 0 && c >= 0 && r < (int)(ts / 16u) && c < (int)bcols) near |= 1u << (r * (int)bcols + c);
    }
  const uint32_t base = sm.g_min, lim = min(bound, sm.ub);
  for (uint32_t i = tid; i < n; i += blockDim.x) {
    const uint2 it = sm.fa[i];
    const int ix = (int)(it.x & 0xffffu), iy = (int)(it.x >> 16);
    if (it.y - base < kSweepSpan) sm.vs[((uint32_t)iy - tg.y0 + 1u) * stride + 8u + (uint32_t)ix - tg.x0] = (uint16_t)(it.y - base);
    else astar_inbox_push(d, Ip, t, next_round, it);  // a later visit starts from its g
  }
  __syncthreads();
  uint16_t* row = sm.vs + ((on ? y : 0u) + 1u) * stride + 8u + xs;
  uint32_t v[NP], k1[NP];                        // labels; min(old label, window) as astar_pair_below takes it
  uint32_t cnw[NP], cne[NP], csw[NP], cse[NP];   // cost of the diagonal move from each neighbour, 0x8000 = none
  uint32_t p[NP], pa, pb;                        // labels passed on
  uint32_t items = 0;                        // the thread's cells that are items
  const int gx = (int)I.gx - (int)(tg.x0 + xs);
  const uint32_t dyg = (uint32_t)abs((int)(tg.y0 + y) - (int)I.gy);
  if (on) {
    astar_load_row<NP>(row, p, pa, pb);
    // blocked bits of columns xs - 1 .. xs + 2 NP of the rows y - 1, y, y + 1 (outside: blocked)
    uint32_t bu = ~0u, bc = ~0u, bd = ~0u;
    auto bits = [&](uint32_t yy) {
      constexpr uint32_t n = 2u * NP;
      const uint32_t l = (yy << lts) + xs;
      uint32_t w = ((sm.blk[l >> 5] >> (l & 31u)) & ((1u << n) - 1u)) << 1;
      const uint32_t room = tg.tw > xs ? tg.tw - xs : 0u;  // columns inside the grid
      if (room < n) w |= ~0u << (room + 1u);
      w |= (xs == 0u) ? 1u : ((sm.blk[(l - 1u) >> 5] >> ((l - 1u) & 31u)) & 1u);
      const bool last = xs + n >= tg.tw;
      w |= (last ? 1u : ((sm.blk[(l + n) >> 5] >> ((l + n) & 31u)) & 1u)) << (n + 1u);
      return w;
    };
    if (y < tg.th) bc = bits(y);
    if (DIAG) {
      if (y > 0 && y - 1u < tg.th) bu = bits(y - 1u);
      if (y + 1u < tg.th) bd = bits(y + 1u);
    }
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      uint32_t vv = 0, kk = 0, c0 = 0, c1 = 0, c2 = 0, c3 = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int x = 2 * i + h;
        const uint32_t src = (p[i] >> (16 * h)) & 0xffffu;
        const bool blocked = (bc >> (x + 1)) & 1u;
        const uint32_t old = sm.gt[(y << lts) + xs + (uint32_t)x];
        // the label that stands: below the items' smallest g nothing improves
        const uint32_t lab = blocked || old < base ? 0u : min(old - base, kSweepInf);
        const uint32_t hh = DIAG ? 10u * max((uint32_t)abs(x - gx), dyg) + 4u * min((uint32_t)abs(x - gx), dyg)
                                 : (uint32_t)abs(x - gx) + dyg;
        const uint32_t win = (lim >= hh && lim - hh >= base) ? min(lim - hh - base + 1u, kSweepSpan) : 0u;
        const bool item = src != kSweepInf && !blocked;
        items |= item ? 1u << x : 0u;
        const uint32_t k = item ? win : min(lab, win);
        vv |= (item ? src : lab) << (16 * h);
        kk |= ((k | 0x8000u) - 1u) << (16 * h);
        if (DIAG) {
          const bool l = !((bc >> x) & 1u), r = !((bc >> (x + 2)) & 1u);
          const bool u = !((bu >> (x + 1)) & 1u), w = !((bd >> (x + 1)) & 1u);
          c0 |= (l && u ? 14u : 0x8000u) << (16 * h);
          c1 |= (r && u ? 14u : 0x8000u) << (16 * h);
          c2 |= (l && w ? 14u : 0x8000u) << (16 * h);
          c3 |= (r && w ? 14u : 0x8000u) << (16 * h);
        }
      }
      v[i] = vv;
      k1[i] = kk;
      cnw[i] = c0;
      cne[i] = c1;
      csw[i] = c2;
      cse[i] = c3;
      // an item whose label no longer lies in the window stays an item: it keeps its label
      p[i] = astar_pair_below(vv, kk);
    }
  }
  uint32_t moved = ~0u;
  for (uint32_t it = 0;; ++it) {
    if (tid == 0) sm.moved[(it + 1u) % 3u] = 0;  // last read before the barrier before this one
    if (on && (moved & near)) {  // the same in a whole warp
      bool any = false;
      for (uint32_t q = 0; q < kSweepsPerBarrier; ++q) {
        uint32_t up[NP], ua, ub2, dn[NP], da, db, np[NP];
        bool changed = false;
        astar_load_row<NP>(row - stride, up, ua, ub2);
        astar_load_row<NP>(row + stride, dn, da, db);
        pa = *reinterpret_cast<const uint32_t*>(row - 2);
        pb = *reinterpret_cast<const uint32_t*>(row + 2 * NP);
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          uint32_t a = v[i];
          a = __viaddmin_u16x2(astar_pair_left(p, i, pa), kStraight, a);
          a = __viaddmin_u16x2(astar_pair_right<NP>(p, i, pb), kStraight, a);
          a = __viaddmin_u16x2(up[i], kStraight, a);
          a = __viaddmin_u16x2(dn[i], kStraight, a);
          if (DIAG) {
            a = __viaddmin_u16x2(astar_pair_left(up, i, ua), cnw[i], a);
            a = __viaddmin_u16x2(astar_pair_right<NP>(up, i, ub2), cne[i], a);
            a = __viaddmin_u16x2(astar_pair_left(dn, i, da), csw[i], a);
            a = __viaddmin_u16x2(astar_pair_right<NP>(dn, i, db), cse[i], a);
          }
          changed |= a != v[i];
          v[i] = a;
          np[i] = astar_pair_below(a, k1[i]);
        }
        if (changed) {
#pragma unroll
          for (int i = 0; i < NP; ++i) p[i] = np[i];
#pragma unroll
          for (int i = 0; i < NP; i += 4)
            *reinterpret_cast<uint4*>(row + 2 * i) = make_uint4(p[i], p[i + 1], p[i + 2], p[i + 3]);
        }
        const bool w = __any_sync(GPQ_FULL_MASK, changed);
        any |= w;
        if (!w) break;
      }
      if (any && lane == 0) atomicOr(&sm.moved[it % 3u], 1u << warp);
    }
    __syncthreads();
    moved = *(volatile uint32_t*)&sm.moved[it % 3u];
    if (moved == 0u) break;
    if (it == kSweepMax) {
      if (tid == 0) gpq_set_error(&Ip->err, GPQ_ERR_TIMEOUT);
      break;
    }
  }
  // changed labels: into the global g values; above the window to the open array
  if (on && y < tg.th) {
    uint32_t* G = d.gcost + I.cell0 + (uint64_t)(tg.y0 + y) * I.g.width + tg.x0 + xs;
    const uint32_t ub = sm.ub;
    uint32_t passed = 0, fell = 0;
#pragma unroll
    for (int x = 0; x < 2 * NP; ++x) {
      const uint32_t lab = (v[x / 2] >> (16 * (x & 1))) & 0xffffu, g = base + lab;
      if (((p[x / 2] >> (16 * (x & 1))) & 0xffffu) != kSweepInf) passed |= 1u << x;
      // no label, and labels that cannot have changed, aside
      if (lab < kSweepInf && lab != 0u && g < sm.gt[(y << lts) + xs + (uint32_t)x]) fell |= 1u << x;
    }
#pragma unroll
    for (int x = 0; x < 2 * NP; ++x)
      if ((fell >> x) & 1u) atomicMin(&G[x], base + ((v[x / 2] >> (16 * (x & 1))) & 0xffffu));
    if (dyg == 0u && gx >= 0 && gx < 2 * NP && ((fell >> gx) & 1u)) {
      uint32_t g = 0;
#pragma unroll
      for (int x = 0; x < 2 * NP; ++x)
        if (x == gx) g = base + ((v[x / 2] >> (16 * (x & 1))) & 0xffffu);
      atomicMin(&Ip->ub, g);
      atomicMin(&sm.ub, g);
    }
    if (fell & ~passed) {
#pragma unroll
      for (int x = 0; x < 2 * NP; ++x) {
        if (!(((fell & ~passed) >> x) & 1u)) continue;
        const uint32_t g = base + ((v[x / 2] >> (16 * (x & 1))) & 0xffffu);
        const uint2 itm = make_uint2(astar_pack((int)(tg.x0 + xs) + x, (int)(tg.y0 + y)), g);
        const uint32_t f = g + astar_hxy(DIAG ? 8 : 4, (int)(tg.x0 + xs) + x, (int)(tg.y0 + y), (int)I.gx, (int)I.gy);
        if (f <= lim) astar_inbox_push(d, Ip, t, next_round, itm);  // beyond the span of this visit's labels
        else if (f <= ub) astar_open_push(d, Ip, sm, t, itm, f);
      }
    }
    *pops += (uint32_t)__popc(passed);
  }
}

// The moves of this visit's expanded cells into other tiles (all threads; a tile's border
// has at most 4 * 64 - 4 cells).  A cell's moves lower the global g values together, then
// the improving ones are counted by neighbour tile, one thread per neighbour reserves their
// place in its inbox, and all are stored: three round trips whatever the number of moves,
// where each move by itself took five one after another.
template <bool DIAG>
__device__ __forceinline__ void astar_send_border(const AstarDev& d, AstarInstDev* Ip, const AstarInstDev& I,
                                                  AstarTileSmem& sm, const AstarTileGeo& tg, uint32_t next_round) {
  constexpr uint32_t M = DIAG ? 8u : 4u;
  const uint32_t w = I.g.width, h = I.g.height, border = 2u * (tg.tw + tg.th);
  const uint32_t npar = next_round & 1u;
  for (uint32_t j0 = 0; j0 < border; j0 += blockDim.x) {
    if (threadIdx.x < 9u) sm.out_n[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t j = j0 + threadIdx.x;
    uint32_t lx, ly;
    bool ok = j < border;
    if (j < 2u * tg.tw) {  // the top and the bottom row, then the sides without their corners
      lx = j >> 1;
      ly = (j & 1u) ? tg.th - 1u : 0u;
      if ((j & 1u) && tg.th == 1u) ok = false;
    } else {
      const uint32_t jj = j - 2u * tg.tw;
      ly = 1u + (jj >> 1);
      lx = (jj & 1u) ? tg.tw - 1u : 0u;
      if (ly + 1u >= tg.th || ((jj & 1u) && tg.tw == 1u)) ok = false;
    }
    const uint32_t lab = ok ? sm.vs[(ly + 1u) * astar_sweep_stride(tg.ts) + 8u + lx] : kSweepInf;
    ok = ok && lab != kSweepInf;
    const int x = (int)(tg.x0 + lx), y = (int)(tg.y0 + ly);
    const uint32_t g = sm.g_min + lab;
    const uint32_t ub = ok ? min(sm.ub, ldcg_u32(&Ip->ub)) : 0u;
    // blocked bits of the eight (four) neighbours: those in other tiles from memory, all in flight
    uint32_t word[M], at[M];
    bool out[M];
#pragma unroll
    for (uint32_t k = 0; k < M; ++k) {
      const int nx = x + gpq_astar_dx((int)k), ny = y + gpq_astar_dy((int)k);
      const bool grid = ok && nx >= 0 && ny >= 0 && nx < (int)w && ny < (int)h;
      out[k] = grid && !tg.inside(nx, ny);
      word[k] = ~0u;  // off the grid: blocked
      at[k] = 0;
      if (grid) {
        const uint32_t c = (uint32_t)ny * w + (uint32_t)nx;
        const uint64_t b = I.cell0 + c;
        const uint32_t l = out[k] ? 0u : tg.local(nx, ny);
        at[k] = out[k] ? (uint32_t)(b & 31u) : l & 31u;
        word[k] = out[k] ? __ldg(&d.blk[b >> 5]) : sm.blk[l >> 5];
      }
    }
    uint32_t open = 0;
#pragma unroll
    for (uint32_t k = 0; k < M; ++k) open |= ((word[k] >> at[k]) & 1u) ? 0u : 1u << k;
    uint32_t old[M];
    bool go[M];
#pragma unroll
    for (uint32_t k = 0; k < M; ++k) {
      go[k] = out[k] && ((open >> k) & 1u);
      if (k >= 4) {  // a diagonal: its two straight neighbours (E 0, W 1, S 2, N 3) are free
        const uint32_t need = (gpq_astar_dx((int)k) > 0 ? 1u : 2u) | (gpq_astar_dy((int)k) > 0 ? 4u : 8u);
        go[k] = go[k] && (open & need) == need;
      }
      old[k] = 0;
      const uint32_t c = (uint32_t)(y + gpq_astar_dy((int)k)) * w + (uint32_t)(x + gpq_astar_dx((int)k));
      if (go[k]) old[k] = atomicMin(&d.gcost[I.cell0 + c], g + gpq_astar_cost(DIAG ? 8 : 4, (int)k));
    }
    uint32_t place[M];  // neighbour tile << 16 | position among the moves into it
#pragma unroll
    for (uint32_t k = 0; k < M; ++k) {
      const int nx = x + gpq_astar_dx((int)k), ny = y + gpq_astar_dy((int)k);
      const uint32_t ng = g + gpq_astar_cost(DIAG ? 8 : 4, (int)k);
      place[k] = ~0u;
      if (!go[k] || ng >= old[k]) continue;
      if (nx == (int)I.gx && ny == (int)I.gy) atomicMin(&Ip->ub, ng);
      if (ng + astar_hxy(I.g.conn, nx, ny, (int)I.gx, (int)I.gy) > ub) continue;
      const uint32_t dir = (nx < (int)tg.x0 ? 0u : nx >= (int)(tg.x0 + tg.ts) ? 2u : 1u) +
                           (ny < (int)tg.y0 ? 0u : ny >= (int)(tg.y0 + tg.ts) ? 6u : 3u);
      place[k] = (dir << 16) | atomicAdd(&sm.out_n[dir], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 9u && sm.out_n[threadIdx.x]) {
      const uint32_t nt = I.tile0 + ((tg.y0 >> tg.lts) + threadIdx.x / 3u - 1u) * I.tiles_x + (tg.x0 >> tg.lts) +
                          threadIdx.x % 3u - 1u;
      sm.out_base[threadIdx.x] = atomicAdd(&d.tiles[nt].in_cnt[npar], sm.out_n[threadIdx.x]);
      astar_activate(d, Ip, nt, next_round);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < M; ++k) {
      if (place[k] == ~0u) continue;
      const int nx = x + gpq_astar_dx((int)k), ny = y + gpq_astar_dy((int)k);
      const uint32_t nt = I.tile0 + ((uint32_t)ny >> tg.lts) * I.tiles_x + ((uint32_t)nx >> tg.lts);
      const uint32_t pos = sm.out_base[place[k] >> 16] + (place[k] & 0xffffu);
      if (pos < d.in_cap)
        d.inbox[((size_t)npar * d.n_tiles + nt) * d.in_cap + pos] =
            make_uint2(astar_pack(nx, ny), g + gpq_astar_cost(DIAG ? 8 : 4, (int)k));
      else
        gpq_set_error(&Ip->err, GPQ_ERR_INSERT_FULL);
    }
    __syncthreads();
  }
}

// Phase W for one instance, by the worker that made the instance's last visit of the round,
// when its tiles sent nothing for the next one: the drained window moves on, or the
// instance ends.  sm.open_min is all ones on entry.
template <bool WARP>
__device__ __forceinline__ void astar_window_step(const AstarDev& d, AstarInstDev* Ip, uint32_t next_round,
                                                  AstarTileSmem& sm, const AstarWorker<WARP>& wk) {
  const uint32_t nt = Ip->tiles_x * Ip->tiles_y, t0 = Ip->tile0;
  uint32_t m = kAstarInf;
  for (uint32_t j = wk.tid; j < nt; j += wk.n) {
    const AstarTileDev* T = d.tiles + t0 + j;
    const uint32_t oc = ldcg_u32(&T->open_cnt), om = ldcg_u32(&T->open_min);
    if (oc) m = min(m, om);
  }
  m = warp_min_u32(m);
  if ((threadIdx.x & 31u) == 0) atomicMin(&sm.open_min, m);
  wk.sync();
  m = sm.open_min;
  const uint32_t ub = ldcg_u32(&Ip->ub);
  if (m == kAstarInf || m > ub) {
    if (wk.tid == 0) Ip->done = 1;
    return;
  }
  uint32_t bound = m + Ip->delta;
  if (bound < m || bound > ub) bound = ub;
  if (wk.tid == 0) {
    Ip->bound = bound;
    Ip->windows += 1;
  }
  for (uint32_t j = wk.tid; j < nt; j += wk.n) {
    const AstarTileDev* T = d.tiles + t0 + j;
    const uint32_t oc = ldcg_u32(&T->open_cnt), om = ldcg_u32(&T->open_min);
    if (oc && om <= bound) astar_activate(d, Ip, t0 + j, next_round);
  }
}

// Process tile t in round s (one worker).
template <bool WARP, int NP>
__device__ void astar_process_tile(const AstarDev& d, uint32_t t, uint32_t s, AstarTileSmem& sm,
                                   const AstarWorker<WARP>& wk) {
  const uint32_t par = s & 1u, next_round = s + 1u;
  AstarTileDev* T = d.tiles + t;
  AstarInstDev* Ip = d.inst + T->inst;
  const AstarInstDev I = *Ip;  // static fields; ub/bound are read through Ip
  uint32_t* G = d.gcost + I.cell0;
  const uint32_t ts = d.ts, words = ts * ts / 32;
  AstarTileGeo tg;
  tg.ts = ts;
  tg.lts = d.lts;
  tg.x0 = T->tx * ts;
  tg.y0 = T->ty * ts;
  tg.tw = min(ts, I.g.width - tg.x0);
  tg.th = min(ts, I.g.height - tg.y0);
  if (wk.tid == 0) {
    sm.n[0] = 0;
    sm.n[1] = 0;
    sm.n[2] = 0;
    sm.ob_n = 0;
    sm.pops = 0;
    sm.open_cnt = T->open_cnt;
    sm.open_min = kAstarInf;
    sm.g_min = kAstarInf;
  }
  wk.sync();
  const uint32_t k_in = min(ldcg_u32(&T->in_cnt[par]), d.in_cap);
  const uint32_t bound = ldcg_u32(&Ip->bound);
  if (ldcg_u32(&Ip->done)) {
    if (wk.tid == 0) {
      T->in_cnt[par] = 0;
      T->queued[par] = 0;
      T->open_cnt = 0;
      T->open_min = kAstarInf;
    }
    wk.sync();
    return;
  }
  const uint32_t ub = ldcg_u32(&Ip->ub);
  if (wk.tid == 0) {
    sm.ub = ub;
    atomicAdd(&d.ctl->visits, 1ull);
  }
  // 0. the tile's g values and blocked bits into shared memory
  constexpr bool sweeps = NP != 0;
  for (uint32_t j = wk.tid; j < words; j += wk.n) {
    sm.blk[j] = 0;
    if (!sweeps) sm.chg[j] = 0;
  }
  if (sweeps) {
    uint4* vs4 = reinterpret_cast<uint4*>(sm.vs);
    const uint4 none = make_uint4(kSweepInf2, kSweepInf2, kSweepInf2, kSweepInf2);
    for (uint32_t j = wk.tid; j < (ts + 2u) * astar_sweep_stride(ts) / 8u; j += wk.n) vs4[j] = none;
    if (wk.tid < 3u) sm.moved[wk.tid] = 0;
  }
  // Several loads of a thread in flight at a time: the copy is a round trip to L2 otherwise
  // repeated.  Fewer where a CTA walks lists, which has 64 registers a thread.
  constexpr uint32_t kFlight = sweeps || WARP ? 16u : 4u;
  for (uint32_t l0 = wk.tid; l0 < ts * ts; l0 += kFlight * wk.n) {
    uint32_t g[kFlight];
#pragma unroll
    for (uint32_t q = 0; q < kFlight; ++q) {
      const uint32_t l = l0 + q * wk.n, lx = l & (ts - 1u), ly = l >> tg.lts;
      g[q] = (l < ts * ts && lx < tg.tw && ly < tg.th) ? ldcg_u32(&G[(tg.y0 + ly) * I.g.width + tg.x0 + lx]) : kAstarInf;
    }
#pragma unroll
    for (uint32_t q = 0; q < kFlight; ++q)
      if (l0 + q * wk.n < ts * ts) sm.gt[l0 + q * wk.n] = g[q];
  }
  wk.sync();
  {
    const uint32_t segw = ts < 32 ? ts : 32u, segs = ts / segw;
    for (uint32_t j = wk.tid; j < tg.th * segs; j += wk.n) {
      const uint32_t ly = j / segs, lx0 = (j % segs) * segw;
      if (lx0 >= tg.tw) continue;
      const uint64_t b0 = I.cell0 + (uint64_t)(tg.y0 + ly) * I.g.width + tg.x0 + lx0;
      uint32_t bits = __funnelshift_r(__ldg(&d.blk[b0 >> 5]), __ldg(&d.blk[(b0 >> 5) + 1]), (uint32_t)(b0 & 31u));
      const uint32_t nb = min(segw, tg.tw - lx0);
      if (nb < 32) bits &= (1u << nb) - 1u;
      const uint32_t l0 = ly * ts + lx0;
      atomicOr(&sm.blk[l0 >> 5], bits << (l0 & 31u));
    }
  }
  wk.sync();
  // 1. the open array, when the window reached it: expand-now items leave, the rest is
  //    compacted in place (a chunk is read completely before any of it is written)
  const uint32_t n_open = sm.open_cnt;
  if (n_open > 0 && ldcg_u32(&T->open_min) <= bound) {
    uint2* O = d.open + (size_t)t * d.open_cap;
    uint32_t kept = 0;
    for (uint32_t c0 = 0; c0 < n_open; c0 += wk.n) {
      const uint32_t i = c0 + wk.tid;
      uint2 it = make_uint2(0, kAstarInf);
      uint32_t keep = 0, f = kAstarInf;
      if (i < n_open) {
        it = O[i];
        const int x = (int)(it.x & 0xffffu), y = (int)(it.x >> 16);
        if (sm.gt[tg.local(x, y)] == it.y) {
          f = it.y + astar_hxy(I.g.conn, x, y, (int)I.gx, (int)I.gy);
          if (f <= ub) {
            if (f <= bound) astar_frontier_push(d, Ip, sm, sm.fa, 0, t, next_round, it);
            else keep = 1;
          }
        }
      }
      uint32_t total;
      const uint32_t off = astar_worker_scan<WARP>(keep, sm.scan, &total);
      if (keep) {
        O[kept + off] = it;
        atomicMin(&sm.open_min, f);
      }
      kept += total;
    }
    if (wk.tid == 0) sm.open_cnt = kept;
    wk.sync();
  } else if (wk.tid == 0) {
    sm.open_min = ldcg_u32(&T->open_min);
  }
  wk.sync();
  // 2. the inbox (senders lowered the global g of these cells before sending)
  {
    const uint2* B = d.inbox + ((size_t)par * d.n_tiles + t) * d.in_cap;
    for (uint32_t i = wk.tid; i < k_in; i += wk.n) {
      const uint2 it = B[i];
      const int x = (int)(it.x & 0xffffu), y = (int)(it.x >> 16);
      if (sm.gt[tg.local(x, y)] != it.y) continue;
      const uint32_t f = it.y + astar_hxy(I.g.conn, x, y, (int)I.gx, (int)I.gy);
      if (f > ub) continue;
      if (f <= bound) astar_frontier_push(d, Ip, sm, sm.fa, 0, t, next_round, it);
      else astar_open_push(d, Ip, sm, t, it, f);
    }
  }
  wk.sync();
  if (wk.tid == 0) {
    T->in_cnt[par] = 0;
    T->queued[par] = 0;
  }
  // 3. sweeps; the border's moves when all labels stand
  uint32_t pops = 0;
  if constexpr (sweeps) {
    const uint32_t n = min(sm.n[0], d.frontier_cap);
    if (n > 0) {  // the same in every thread
      uint32_t lo = kAstarInf;
      for (uint32_t i = wk.tid; i < n; i += wk.n) lo = min(lo, sm.fa[i].y);
      lo = __reduce_min_sync(GPQ_FULL_MASK, lo);
      if ((threadIdx.x & 31u) == 0) atomicMin(&sm.g_min, lo);
      wk.sync();
      if (I.g.conn == 4) {
        astar_sweep_tile<false, NP>(d, Ip, I, sm, tg, n, t, next_round, bound, &pops);
        astar_send_border<false>(d, Ip, I, sm, tg, next_round);
      } else {
        astar_sweep_tile<true, NP>(d, Ip, I, sm, tg, n, t, next_round, bound, &pops);
        astar_send_border<true>(d, Ip, I, sm, tg, next_round);
      }
    }
  } else {
    // list walk: level-by-level expansion of the frontier inside the tile; level i reads
    // buffer i % 2 with fill n[i % 3], fills the other buffer and n[(i + 1) % 3], and clears
    // n[(i + 2) % 3] (read at level i - 1, filled at level i + 1): one barrier a level
    for (uint32_t lv = 0;; ++lv) {
      const uint32_t c3 = lv % 3u;
      const uint32_t n = min(sm.n[c3], d.frontier_cap);
      if (n == 0) break;
      uint2* src = (lv & 1u) ? sm.fb : sm.fa;
      uint2* dst = (lv & 1u) ? sm.fa : sm.fb;
      if (wk.tid == 0) sm.n[(c3 + 2u) % 3u] = 0;
      const uint32_t ipw = I.g.conn == 4 ? 8u : 4u;  // items per warp pass
      for (uint32_t ib = (wk.tid >> 5) * ipw; ib < n; ib += (wk.n >> 5) * ipw)
        astar_expand_warp(d, Ip, I, sm, tg, src, ib, n, dst, (c3 + 1u) % 3u, t, next_round, bound, &pops);
      wk.sync();
    }
    // 4. send the moves into other tiles
    {
      const uint32_t nob = min(sm.ob_n, astar_outbox_cap(ts));
      for (uint32_t i = wk.tid; i < nob; i += wk.n) astar_send(d, Ip, I, sm.ob[i], next_round);
    }
  }
  // 5. list walk: merge the tile's g values back
  if (!sweeps) {
    for (uint32_t l = wk.tid; l < ts * ts; l += wk.n) {
      if ((sm.chg[l >> 5] >> (l & 31u)) & 1u) {
        const uint32_t lx = l & (ts - 1u), ly = l >> tg.lts;
        atomicMin(&G[(tg.y0 + ly) * I.g.width + tg.x0 + lx], sm.gt[l]);
      }
    }
  }
  pops = warp_sum_u32(pops);
  if ((threadIdx.x & 31u) == 0 && pops) atomicAdd(&sm.pops, (unsigned long long)pops);
  wk.sync();
  if (wk.tid == 0) {
    const uint32_t oc = min(sm.open_cnt, d.open_cap);
    T->open_cnt = oc;
    T->open_min = oc ? sm.open_min : kAstarInf;
    if (sm.pops) atomicAdd(&Ip->pops, sm.pops);
    // the instance's last visit of the round: every send and open array of the round stands
    __threadfence();
    const uint32_t last = atomicAdd(&Ip->visited, 1u) + 1u == ldcg_u32(&Ip->active[par]) ? 1u : 0u;
    __threadfence();
    sm.last = last;
    sm.open_min = kAstarInf;
    if (last) {
      Ip->visited = 0;
      Ip->active[par] = 0;
    }
  }
  wk.sync();
  if (sm.last && ldcg_u32(&Ip->active[next_round & 1u]) == 0u) astar_window_step<WARP>(d, Ip, next_round, sm, wk);
  wk.sync();
}

// The persistent search loop over all instances.  Dynamic shared memory: one slice of
// astar_worker_smem_bytes(ts, frontier_cap) per worker (per warp when WARP).
static constexpr uint32_t kAstarMaxWorkers = 8;  // 256 threads / 32

__host__ __device__ inline size_t astar_worker_smem_bytes(uint32_t ts, uint32_t frontier_cap, bool warp, uint32_t block) {
  return (astar_smem_bytes(ts, frontier_cap, warp, block) + 15u) & ~(size_t)15u;
}

// Rounds s0, s0 + 1, ... until every instance is done, or until `step_rounds` rounds ran
// (0 = no limit): a resident session resumes at the next round in its next launch.
// NP: pairs of cells of a thread that sweeps (astar_sweep_pairs), 0: list walk.  With four
// pairs one CTA of 512 threads an SM: a second would halve the registers and spill (2048 x
// 2048 search 1.97 against 2.25 ms, 500 mixed searches 3.16 against 3.29 ms).  CTAs that
// walk lists stay four an SM at 256 threads, since the visits of many searches hide each other's
// chains (at two, with 104 registers: 500 mixed searches in tiles of 16 16.6 against 12.4 ms,
// 2,000 small ones 4.9 / 3.9, in tiles of 8 33 / 21 and 8.6 / 5.8); warps that walk lists gain
// more from loads in flight (tiles of 16: 19.4 ms, 20.5 at four).
template <bool WARP, int NP>
static __global__ void __launch_bounds__(NP == 4 ? 512 : 256, NP == 4 ? 1 : NP == 8 || WARP ? 2 : 4) astar_persistent_kernel(AstarDev d, uint32_t s0, uint32_t step_rounds) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ AstarTileSmem sms[kAstarMaxWorkers];
  __shared__ uint32_t s_t;
  const AstarWorker<WARP> wk;
  AstarTileSmem& sm = sms[wk.id];
  if (wk.tid == 0) {
    astar_smem_carve(sm, smem_raw + (size_t)wk.id * astar_worker_smem_bytes(d.ts, d.frontier_cap, WARP, blockDim.x),
                     d.ts, d.frontier_cap, WARP);
  }
  __syncthreads();
  const unsigned long long nb = gridDim.x;
  unsigned long long bar_target = 0;
  const uint32_t per_cta = WARP ? blockDim.x >> 5 : 1u;
  const uint32_t workers = gridDim.x * per_cta, me = blockIdx.x * per_cta + wk.id;
  for (uint32_t s = s0;; ++s) {
    const uint32_t par = s & 1u, cur = s % 3u, nxt = (s + 1u) % 3u, old = (s + 2u) % 3u;
    const uint32_t n = ldcg_u32(&d.ctl->al_cnt[cur]);
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // last read in round s - 1, filled again in round s + 1
      d.ctl->al_cnt[old] = 0;
      d.ctl->work[old] = 0;
      d.ctl->rounds = s + 1;
    }
    // each worker's first tile goes by its number, later ones from a counter
    for (uint32_t j = me; j < n;) {
      astar_process_tile<WARP, NP>(d, d.al[(size_t)par * d.n_tiles + j], s, sm, wk);
      if (n <= workers) break;
      if (WARP) {
        if (wk.tid == 0) j = workers + atomicAdd(&d.ctl->work[cur], 1u);
        j = __shfl_sync(GPQ_FULL_MASK, j, 0);
      } else {
        if (threadIdx.x == 0) s_t = workers + atomicAdd(&d.ctl->work[cur], 1u);
        __syncthreads();
        j = s_t;
        __syncthreads();
      }
    }
    bar_target += nb;
    if (!grid_barrier(&d.ctl->bar, bar_target, d.spin_limit, &d.ctl->err)) return;
    if (ldcg_u32(&d.ctl->al_cnt[nxt]) == 0 || ldcg_u32(&d.ctl->err) != 0) break;
    if (d.max_rounds && s + 1 >= d.max_rounds) {
      if (blockIdx.x == 0 && threadIdx.x == 0) gpq_set_error(&d.ctl->err, GPQ_ERR_TIMEOUT);
      break;
    }
    if (step_rounds && s + 1 - s0 >= step_rounds) break;
  }
}

// The kernel for a tile side, worker and CTA size (host side).
inline const void* astar_kernel(uint32_t ts, bool warp, uint32_t block) {
  if (warp) return (const void*)astar_persistent_kernel<true, 0>;
  switch (astar_sweep_pairs(ts, false, block)) {
    case 4: return (const void*)astar_persistent_kernel<false, 4>;
    case 8: return (const void*)astar_persistent_kernel<false, 8>;
    default: return (const void*)astar_persistent_kernel<false, 0>;
  }
}

// ---- set-up and results ----

// Blocked bitmap of all instances: one thread per 32-cell word.
static __global__ void astar_bitmap_kernel(const AstarInstDev* inst, uint32_t n_inst, const uint64_t* word0,
                                           uint64_t total_words, uint32_t* blk) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t wi = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; wi < total_words; wi += stride) {
    uint32_t lo = 0, hi = n_inst - 1;  // last instance with word0 <= wi
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (word0[mid] <= wi) lo = mid; else hi = mid - 1;
    }
    const AstarInstDev& I = inst[lo];
    const uint64_t cells = (uint64_t)I.g.width * I.g.height;
    const uint64_t c0 = (wi - word0[lo]) * 32u;
    uint32_t w = 0;
    for (uint32_t b = 0; b < 32; ++b) {
      const uint64_t c = c0 + b;
      if (c < cells && gpq_astar_blocked(&I.g, (uint32_t)c)) w |= 1u << b;
    }
    blk[wi] = w;
  }
}

// Initial state of instances list[0, n) (all instances when list == nullptr): g = inf
// (done by a memset), g[start] = 0, the start item in the start tile's inbox of `round`,
// the start tile on that round's active list.
static __global__ void astar_init_kernel(AstarDev d, const uint32_t* list, uint32_t n, uint32_t round) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const uint32_t i = list ? list[j] : j;
  AstarInstDev& I = d.inst[i];
  d.gcost[I.cell0 + I.g.start] = 0;
  const uint32_t t = astar_tile_of(d, I, I.g.start);
  const uint32_t par = round & 1u;
  d.tiles[t].in_cnt[par] = 1;
  d.inbox[((size_t)par * d.n_tiles + t) * d.in_cap] =
      make_uint2(astar_pack((int)(I.g.start % I.g.width), (int)(I.g.start / I.g.width)), 0);
  astar_activate(d, &I, t, round);
}

// Tile records of instances list[0, n) (all when list == nullptr): one block per instance.
static __global__ void astar_tiles_init_kernel(AstarDev d, const uint32_t* list, uint32_t n) {
  for (uint32_t j = blockIdx.x; j < n; j += gridDim.x) {
    const uint32_t inst = list ? list[j] : j;
    const AstarInstDev& I = d.inst[inst];
    const uint32_t nt = I.tiles_x * I.tiles_y;
    for (uint32_t k = threadIdx.x; k < nt; k += blockDim.x) {
      AstarTileDev T{};
      T.inst = inst;
      T.tx = k % I.tiles_x;
      T.ty = k / I.tiles_x;
      T.open_min = kAstarInf;
      d.tiles[I.tile0 + k] = T;
    }
  }
}

// Blocked bits of instances list[0, n): blockIdx.y = position in the list.  Instance
// cell ranges start on 32-cell boundaries.
static __global__ void astar_bitmap_list_kernel(const AstarInstDev* inst, const uint32_t* list, uint32_t* blk) {
  const AstarInstDev& I = inst[list[blockIdx.y]];
  const uint64_t cells = (uint64_t)I.g.width * I.g.height;
  const uint64_t words = (cells + 31) / 32, w0 = I.cell0 / 32;
  for (uint64_t wi = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; wi < words; wi += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t w = 0;
    for (uint32_t b = 0; b < 32; ++b) {
      const uint64_t c = wi * 32 + b;
      if (c < cells && gpq_astar_blocked(&I.g, (uint32_t)c)) w |= 1u << b;
    }
    blk[w0 + wi] = w;
  }
}

// Slots that are in use (on[slot] != 0) and whose search has ended, appended to out.
static __global__ void astar_done_list_kernel(const AstarInstDev* inst, const uint8_t* on, uint32_t n_slots,
                                              uint32_t* out, uint32_t* out_n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_slots; i += gridDim.x * blockDim.x)
    if (on[i] && inst[i].done) out[atomicAdd(out_n, 1u)] = i;
}

// Move tested l-th (l = 0..7) when looking for a predecessor, numbered as in
// gpq_astar_dx/dy: the neighbours NW, N, NE, W, E, SW, S, SE, which is increasing cell id on
// every grid where two of them exist together.
__device__ __forceinline__ int astar_pred_order(int l) {
  return l == 0 ? 7 : l == 1 ? 3 : l == 2 ? 6 : l == 3 ? 1 : l == 4 ? 0 : l == 5 ? 5 : l == 6 ? 2 : 4;
}

static constexpr uint8_t kAstarNoPred = 0xFF;

// Instances of at least this many cells get predecessor moves from astar_pred_kernel and
// walk their path over them (long walks, few such instances at a time).
static constexpr uint64_t kAstarPredBytesCells = 1ull << 20;

__device__ __forceinline__ bool astar_pred_bytes(const AstarInstDev& I) {
  return (uint64_t)I.g.width * I.g.height >= kAstarPredBytesCells;
}

// The canonical predecessor of cell c (g = g[c], on an optimal path when g + h(c) <= C*):
// the neighbour p with the smallest id that is free (both orthogonal cells free for a
// diagonal), g[p] + c(p, c) == g and g[p] + h(p) <= C*.  Encoded as (dy + 1) << 2 | (dx + 1)
// for the move from c to p; kAstarNoPred when there is none.  Lanes without a cell that
// needs it pass cand = false; the blocked bits and g values of all eight neighbours are
// loaded in one batch and the choice is made in registers, without divergent branches.
__device__ __forceinline__ uint8_t astar_pred_move(const AstarDev& d, const AstarInstDev& I, const uint32_t* G,
                                                   bool cand, uint32_t c, uint32_t g, uint32_t cs) {
  const uint32_t w = I.g.width, h = I.g.height, conn = I.g.conn;
  const int x = (int)(c % w), y = (int)(c / w);
  bool fr[8];
  uint32_t gp[8];
#pragma unroll
  for (int l = 0; l < 8; ++l) {
    const int k = astar_pred_order(l);
    const int nx = x + gpq_astar_dx(k), ny = y + gpq_astar_dy(k);
    const bool in = cand && (conn == 8u || k < 4) && nx >= 0 && ny >= 0 && nx < (int)w && ny < (int)h;
    const uint32_t p = (uint32_t)ny * w + (uint32_t)nx;
    fr[l] = in && !astar_blocked(d, I, p);
    gp[l] = in ? __ldg(&G[p]) : kAstarInf;
  }
  // diagonals (lanes 0 NW, 2 NE, 5 SW, 7 SE) also need their two orthogonal cells free
  const bool diag = conn == 8u;
  const bool ok[8] = {diag && fr[0] && fr[3] && fr[1], fr[1], diag && fr[2] && fr[1] && fr[4], fr[3],
                      fr[4], diag && fr[5] && fr[3] && fr[6], fr[6], diag && fr[7] && fr[4] && fr[6]};
  uint8_t best = kAstarNoPred;
#pragma unroll
  for (int l = 7; l >= 0; --l) {  // the smallest valid l is assigned last
    const int k = astar_pred_order(l);
    const int dx = gpq_astar_dx(k), dy = gpq_astar_dy(k);
    if (ok[l] && gp[l] != kAstarInf && (uint64_t)gp[l] + gpq_astar_cost(conn, k) == g &&
        (uint64_t)gp[l] + astar_hxy(conn, x + dx, y + dy, (int)I.gx, (int)I.gy) <= cs)
      best = (uint8_t)((dy + 1) << 2 | (dx + 1));
  }
  return best;
}

// Per-instance expanded set (g + h <= C*, or every reached cell when the goal is not
// reachable): count and hash.  Block per (instance, chunk): blockIdx.y = instance.
static __global__ void astar_finalize_kernel(AstarDev d, const uint32_t* list, unsigned long long* out /* [n][2] */) {
  const uint32_t j = blockIdx.y;
  const uint32_t i = list ? list[j] : j;
  const AstarInstDev& I = d.inst[i];
  const uint32_t cs = I.ub;
  const uint64_t cells = (uint64_t)I.g.width * I.g.height;
  const uint32_t* G = d.gcost + I.cell0;
  unsigned long long cnt = 0, hs = 0;
  for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < cells;
       c += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t g = G[c];
    if (g == kAstarInf) continue;
    if (cs != kAstarInf && (uint64_t)g + gpq_astar_h(I.g.conn, (uint32_t)c, I.g.goal, I.g.width) > cs) continue;
    ++cnt;
    hs += gpq_astar_cell_hash((uint32_t)c, g);
  }
  cnt = warp_sum_u64(cnt);
  hs = warp_sum_u64(hs);
  if ((threadIdx.x & 31u) == 0 && cnt) {
    atomicAdd(&out[2 * j], cnt);
    atomicAdd(&out[2 * j + 1], hs);
  }
}

// Predecessor move of every expanded cell (g + h <= C*) of the instances in list[0, n)
// that reached their goal and have at least kAstarPredBytesCells cells; the others
// return at once.  Block per (instance, chunk): blockIdx.y = instance.  Whole warps step
// together (blockDim is a multiple of 32), so a warp without expanded cells skips the
// neighbour loads.
static __global__ void astar_pred_kernel(AstarDev d, const uint32_t* list) {
  const uint32_t i = list ? list[blockIdx.y] : blockIdx.y;
  const AstarInstDev& I = d.inst[i];
  const uint32_t cs = I.ub;
  if (cs == kAstarInf || !astar_pred_bytes(I)) return;
  const uint64_t cells = (uint64_t)I.g.width * I.g.height;
  const uint32_t* G = d.gcost + I.cell0;
  const uint32_t lane = threadIdx.x & 31u;
  for (uint64_t base = blockIdx.x * (uint64_t)blockDim.x + (threadIdx.x - lane); base < cells;
       base += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t c = base + lane;
    const uint32_t g = c < cells ? G[c] : kAstarInf;
    const bool exp = g != kAstarInf && (uint64_t)g + gpq_astar_h(I.g.conn, (uint32_t)c, I.g.goal, I.g.width) <= cs;
    if (__any_sync(GPQ_FULL_MASK, exp)) {
      const uint8_t mv = astar_pred_move(d, I, G, exp, (uint32_t)c, g, cs);
      if (exp) d.pred[I.cell0 + c] = mv;
    }
  }
}

// ---- canonical path ----
// From the goal, step to the neighbour p with g[p] + c(p, cell) == g[cell] and
// g[p] + h(p) <= C* that has the smallest id, until the start.  The walk is serial, so
// one CTA per instance keeps everything else off its critical path: all warps stage a
// window of the grid in shared memory, one thread (or warp) walks inside it, and all
// warps hash and store the cells it recorded.  Windows are placed around the current cell
// with most of their room on the side of the start, where the path is heading.  Two forms:
//  - instances of at least kAstarPredBytesCells cells (long walks, few of them at a time)
//    use the predecessor moves that astar_pred_kernel wrote for every expanded cell: staged
//    as 128 x 128 windows that hold each cell's next place, so that a step of the walk is one
//    dependent shared-memory load and nothing else;
//  - smaller instances (many at a time, where a pass over every expanded cell would
//    cost more than it saves) stage 64 x 64 windows of g values and blocked
//    bits, and warp 0 finds each step: lane l tests the l-th neighbour in increasing
//    cell id, and the first lane whose test passes (one ballot) is the step.
static constexpr uint32_t kPathThreads = 512;
static constexpr uint32_t kPathWalkCap = 2048;
static constexpr int kPathWinB = 128;                  // move-byte window side
static constexpr int kPathRowWords = kPathWinB / 4 + 1;  // aligned words that cover 128 bytes
static constexpr uint32_t kPathUnroll = 8;             // steps between two looks at where the walk is
static constexpr int kPathWinC = 64;                   // g-value window side
static constexpr int kPathHalo = kPathWinC + 2;         // plus the cells its moves reach
static constexpr int kPathStageBytes = kPathHalo * kPathHalo * 5 > kPathWinB * kPathWinB * 2
                                           ? kPathHalo * kPathHalo * 5
                                           : kPathWinB * kPathWinB * 2;

// First column (row) of a window of side win around coordinate c on an axis of n cells,
// with the start at coordinate s: 7/8 of the room towards the start.
__device__ __forceinline__ int astar_path_origin(int c, int s, int n, int win) {
  if (n <= win) return 0;
  const int o = s < c ? c - (win - win / 8) : s > c ? c - (win / 8 - 1) : c - win / 2;
  return min(max(o, 0), n - win);
}

struct AstarPathSmem {
  uint32_t* walk;    // [kPathWalkCap] cells recorded in the current window (move-byte form: entries' offsets)
  uint32_t* cur;     // next cell to record
  uint32_t* origin;  // move-byte form: the window's first cell
  uint32_t* nwalk;
  uint32_t* done;  // 0 walking, 1 reached the start, 2 no predecessor
};

// One window of the move-byte form.  Staged: for each cell the byte offset of its
// predecessor's entry; a cell whose walk ends here (the start, no predecessor, a predecessor
// outside the window) points at itself, so the walk needs no test but now and then whether it
// still moves.  Thread 0 then follows the offsets, and a cell of the border that the walk
// cannot leave is the first one of the next window, which lies around it: only the start and
// a cell without a predecessor stop the walk elsewhere.  A 2048^2 grid's 4,095 steps took
// 0.40 ms when a step read a move byte, updated the coordinates and tested them, and take
// 0.23 so.  Ends with a barrier.
__device__ __forceinline__ void astar_path_window_bytes(const AstarDev& d, const AstarInstDev& I, uint16_t* s_next,
                                                        const AstarPathSmem& sm) {
  const uint32_t tid = threadIdx.x;
  const int w = (int)I.g.width, h = (int)I.g.height;
  const uint32_t start = I.g.start, cur = *sm.cur;
  const int sx = (int)(start % (uint32_t)w), sy = (int)(start / (uint32_t)w);
  const int cx = (int)(cur % (uint32_t)w), cy = (int)(cur / (uint32_t)w);
  const int tx0 = astar_path_origin(cx, sx, w, kPathWinB);
  const int ty0 = astar_path_origin(cy, sy, h, kPathWinB);
  const uint32_t* PW = reinterpret_cast<const uint32_t*>(d.pred);
  const int cols = min(kPathWinB, w - tx0), rows = min(kPathWinB, h - ty0);
  // words of four moves, a thread's loads in flight together
  constexpr int kWords = kPathWinB * kPathRowWords, kEach = (kWords + (int)kPathThreads - 1) / (int)kPathThreads;
  uint32_t mv[kEach];
#pragma unroll
  for (int u = 0; u < kEach; ++u) {
    const int k = u * (int)kPathThreads + (int)tid, r = k / kPathRowWords, j = k % kPathRowWords;
    mv[u] = 0u;
    if (r < rows) {
      const uint64_t b0 = I.cell0 + (uint64_t)(ty0 + r) * (uint64_t)w + (uint64_t)tx0;
      if ((int)(4 * j) - (int)(b0 & 3u) < cols) mv[u] = __ldg(&PW[(b0 >> 2) + (uint32_t)j]);
    }
  }
#pragma unroll
  for (int u = 0; u < kEach; ++u) {
    const int k = u * (int)kPathThreads + (int)tid, r = k / kPathRowWords, j = k % kPathRowWords;
    if (r >= rows) continue;
    const int x0 = 4 * j - (int)((I.cell0 + (uint64_t)(ty0 + r) * (uint64_t)w + (uint64_t)tx0) & 3u);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int x = x0 + t;
      if (x < 0 || x >= cols) continue;
      const uint32_t m = (mv[u] >> (8 * t)) & 0xffu;
      const int nx = x + (int)(m & 3u) - 1, ny = r + (int)(m >> 2) - 1;
      const bool stop = m == kAstarNoPred || nx < 0 || ny < 0 || nx >= cols || ny >= rows ||
                        (tx0 + x == sx && ty0 + r == sy);
      s_next[r * kPathWinB + x] = (uint16_t)(2 * (stop ? r * kPathWinB + x : ny * kPathWinB + nx));
    }
  }
  __syncthreads();
  if (tid == 0) {
    const unsigned char* nb = reinterpret_cast<const unsigned char*>(s_next);
    uint32_t at = 2u * (uint32_t)((cy - ty0) * kPathWinB + (cx - tx0)), before = at, q = 0;
    do {
#pragma unroll
      for (uint32_t u = 0; u < kPathUnroll; ++u) {
        sm.walk[q + u] = at;
        before = at;
        at = *reinterpret_cast<const uint16_t*>(nb + at);
      }
      q += kPathUnroll;
    } while (at != before && q + kPathUnroll <= kPathWalkCap);
    uint32_t done = 0;
    const int lx = (int)((at >> 1) % (uint32_t)kPathWinB), ly = (int)((at >> 1) / (uint32_t)kPathWinB);
    const uint32_t c = (uint32_t)(ty0 + ly) * (uint32_t)w + (uint32_t)(tx0 + lx);
    if (at == before) {  // it stays at c: once is enough, and not at all if the next window goes on from it
      while (q > 0 && sm.walk[q - 1] == at) --q;
      const bool edge = lx == 0 || ly == 0 || lx == cols - 1 || ly == rows - 1;
      if (c == start) done = 1;
      else if (!edge || q == 0) done = 2;  // a window lies around its first cell: it could have left
      if (done) sm.walk[q++] = at;
    }
    *sm.cur = c;
    *sm.nwalk = q;
    *sm.done = done;
    *sm.origin = (uint32_t)ty0 * (uint32_t)w + (uint32_t)tx0;
  }
  __syncthreads();
}

// One window of the g-value form: stage g values and blocked bits (one grid row per warp
// and pass), then warp 0 walks.  Ends with a barrier.
__device__ __forceinline__ void astar_path_window_cells(const AstarDev& d, const AstarInstDev& I, uint32_t* s_g,
                                                        uint8_t* s_b, const AstarPathSmem& sm) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t* G = d.gcost + I.cell0;
  const int w = (int)I.g.width, h = (int)I.g.height;
  const uint32_t conn = I.g.conn, start = I.g.start, cs = I.ub, cur = *sm.cur;
  const int cx = (int)(cur % (uint32_t)w), cy = (int)(cur / (uint32_t)w);
  const int tx0 = astar_path_origin(cx, (int)(start % (uint32_t)w), w, kPathWinC);
  const int ty0 = astar_path_origin(cy, (int)(start / (uint32_t)w), h, kPathWinC);
  // the window and its halo, clipped to the grid (moves never leave the grid)
  const int sx0 = max(tx0 - 1, 0), sx1 = min(tx0 + kPathWinC, w - 1);
  const int sy0 = max(ty0 - 1, 0), sy1 = min(ty0 + kPathWinC, h - 1);
  for (int y = sy0 + (int)warp; y <= sy1; y += (int)(kPathThreads / 32)) {
    const uint32_t row = (uint32_t)y * (uint32_t)w;
    const int hrow = (y - ty0 + 1) * kPathHalo - tx0 + 1;  // + x = halo index of (x, y)
    uint32_t gv[3];
    bool bv[3];
#pragma unroll
    for (int u = 0; u < 3; ++u) {  // 3 x 32 >= kPathHalo columns
      const int x = sx0 + (int)lane + 32 * u;
      if (x <= sx1) {
        gv[u] = __ldg(&G[row + (uint32_t)x]);
        bv[u] = astar_blocked(d, I, row + (uint32_t)x);
      }
    }
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      const int x = sx0 + (int)lane + 32 * u;
      if (x <= sx1) {
        s_g[hrow + x] = gv[u];
        s_b[hrow + x] = bv[u] ? 1 : 0;
      }
    }
  }
  __syncthreads();
  if (warp == 0) {
    // this lane's move, offset and cost (lanes 8..31 and the diagonals of 4-conn grids idle)
    const int lk = astar_pred_order((int)(lane & 7u));
    const bool lane_on = lane < 8u && (conn == 8u || lk < 4);
    const int ldx = gpq_astar_dx(lk), ldy = gpq_astar_dy(lk);
    const int loff = ldy * kPathHalo + ldx;
    const uint32_t lcost = gpq_astar_cost(conn, lk);
    uint32_t c = cur, q = 0, done = 0;
    int x = cx, y = cy, lx = cx - tx0, ly = cy - ty0;
    while (lx >= 0 && ly >= 0 && lx < kPathWinC && ly < kPathWinC && q < kPathWalkCap) {
      if (lane == 0) sm.walk[q] = c;
      ++q;
      if (c == start) { done = 1; break; }
      const int hi = (ly + 1) * kPathHalo + (lx + 1);
      bool ok = false;
      if (lane_on) {
        const int nx = x + ldx, ny = y + ldy;
        if (nx >= 0 && ny >= 0 && nx < w && ny < h && !s_b[hi + loff] &&
            (ldx == 0 || ldy == 0 || (!s_b[hi + ldx] && !s_b[hi + ldy * kPathHalo]))) {
          const uint32_t gp = s_g[hi + loff], gc = s_g[hi];
          ok = gp != kAstarInf && (uint64_t)gp + lcost == gc &&
               (uint64_t)gp + astar_hxy(conn, nx, ny, (int)I.gx, (int)I.gy) <= cs;
        }
      }
      const uint32_t m = __ballot_sync(GPQ_FULL_MASK, ok);
      if (m == 0u) { done = 2; break; }
      const int k = astar_pred_order(__ffs(m) - 1);
      const int dx = gpq_astar_dx(k), dy = gpq_astar_dy(k);
      x += dx;
      y += dy;
      lx += dx;
      ly += dy;
      c += (uint32_t)(dy * w + dx);  // modulo 2^32: a step back is a wrapped add
    }
    if (lane == 0) {
      *sm.cur = c;
      *sm.nwalk = q;
      *sm.done = done;
    }
  }
  __syncthreads();
}

// Canonical path of the instances in list[0, n) (list == NULL: instances 0..n-1), one CTA
// per instance.  out[3j..3j+2] = path length, path hash, failure flag; the path of
// instance `want` is written to path[0, cap).
static __global__ void __launch_bounds__(kPathThreads) astar_path_kernel(AstarDev d, const uint32_t* list, uint32_t n,
                                                                         unsigned long long* out, uint32_t want,
                                                                         uint32_t* path, uint32_t cap) {
  __shared__ __align__(16) uint8_t s_stage[kPathStageBytes];
  __shared__ uint32_t s_walk[kPathWalkCap];
  __shared__ uint32_t s_cur, s_len, s_done, s_nwalk, s_origin;
  __shared__ unsigned long long s_hs;
  const uint32_t j = blockIdx.x;
  if (j >= n) return;
  const uint32_t i = list ? list[j] : j;
  const AstarInstDev& I = d.inst[i];
  const uint32_t tid = threadIdx.x;
  if (I.ub == kAstarInf) {
    if (tid == 0) { out[3 * j] = 0; out[3 * j + 1] = 0; out[3 * j + 2] = 0; }
    return;
  }
  const bool bytes = astar_pred_bytes(I);
  const AstarPathSmem sm{s_walk, &s_cur, &s_origin, &s_nwalk, &s_done};
  const uint64_t cells = (uint64_t)I.g.width * I.g.height;
  if (tid == 0) {
    s_cur = I.g.goal;
    s_len = 0;
    s_done = 0;
    s_hs = 0;
  }
  __syncthreads();
  // every window records at least one cell: at most cells + 1 windows
  for (uint64_t it = 0; it <= cells && s_done == 0u; ++it) {
    if (bytes)
      astar_path_window_bytes(d, I, reinterpret_cast<uint16_t*>(s_stage), sm);
    else
      astar_path_window_cells(d, I, reinterpret_cast<uint32_t*>(s_stage), s_stage + kPathHalo * kPathHalo * 4, sm);
    const uint32_t nw = s_nwalk, len0 = s_len;
    unsigned long long part = 0;
    for (uint32_t q = tid; q < nw; q += kPathThreads) {
      uint32_t c = s_walk[q];
      if (bytes) c = s_origin + (c >> 1) / (uint32_t)kPathWinB * I.g.width + (c >> 1) % (uint32_t)kPathWinB;
      part += gpq_astar_path_hash(len0 + q, c);
      if (path && i == want && len0 + q < cap) path[len0 + q] = c;
    }
    part = warp_sum_u64(part);
    if ((tid & 31u) == 0 && part) atomicAdd(&s_hs, part);
    __syncthreads();
    if (tid == 0) s_len = len0 + nw;  // read again only after the next window's barriers
  }
  __syncthreads();
  if (tid == 0) {
    out[3 * j] = s_len;
    out[3 * j + 1] = s_hs;
    out[3 * j + 2] = s_done == 1u ? 0u : 1u;
  }
}
