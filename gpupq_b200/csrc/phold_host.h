// Host-side PHOLD configuration helpers shared by the engine entry points.
#pragma once

#include <algorithm>
#include <cmath>

#include "host_common.h"

namespace gpq {

inline gpq_phold_params phold_params_of(const gpq_phold_config& c) {
  gpq_phold_params p;
  p.seed = c.seed;
  p.num_lps = c.num_lps;
  p.dest_mode = c.dest_mode;
  p.ring_width = c.ring_width;
  p.ring_threshold = c.ring_threshold;
  p.lookahead = c.lookahead;
  p.end_time = c.end_time;
  return p;
}

inline bool is_pow2(uint32_t x) { return x && !(x & (x - 1)); }
inline uint32_t ilog2_ceil(uint32_t x) { uint32_t r = 0; while ((1u << r) < x) ++r; return r; }

// Checks that hold for every queue kind and loop mode.
inline gpq_status validate_phold_config(const gpq_phold_config* c) {
  GPQ_CHECK_ARG(c, "config is NULL");
  GPQ_CHECK_ARG(c->num_lps > 0 && c->num_lps <= (1u << 24), "num_lps must be in [1, 2^24]");
  GPQ_CHECK_ARG(c->events_per_lp > 0, "events_per_lp must be > 0");
  GPQ_CHECK_ARG((uint64_t)c->num_lps * c->events_per_lp <= 0xFFFFFFFFull, "num_lps * events_per_lp must fit 32-bit ids");
  GPQ_CHECK_ARG(c->lookahead > 0.f && c->lookahead < 1e30f, "lookahead must be positive and finite");
  GPQ_CHECK_ARG(c->end_time >= 0.f && c->end_time < 1e30f, "end_time must be finite and >= 0");
  GPQ_CHECK_ARG(c->dest_mode == GPQ_DEST_UNIFORM || c->dest_mode == GPQ_DEST_RING, "dest_mode");
  if (c->dest_mode == GPQ_DEST_RING)
    GPQ_CHECK_ARG(c->ring_width >= 1 && 2ull * c->ring_width < c->num_lps, "ring_width must satisfy 1 <= 2w < num_lps");
  GPQ_CHECK_ARG(c->loop_mode == GPQ_LOOP_PLAIN || c->loop_mode == GPQ_LOOP_PERSISTENT, "loop_mode");
  GPQ_CHECK_ARG(c->queue_kind <= GPQ_QUEUE_LSQ, "queue_kind");
  GPQ_CHECK_ARG(c->laq_mode <= 2 && (c->laq_mode == 0 || c->queue_kind == GPQ_QUEUE_LAQ),
                "laq_mode must be 0, or 1 or 2 with the local array queue");
  return GPQ_OK;
}

// Geometry of the bucketed local array queue (laq_mode 2): bucket width w chosen so that
// about 6 events sit in the front bucket of an LP (the pending events of an LP spread over
// about lookahead + 1 time units, the mean increment), but at least lookahead / 2.5 so
// that a window spans at most 4 buckets; NB buckets (a power of two) covering
// lookahead + 7 time units ahead of the window minimum (an increment beyond lookahead + 7
// has probability e^-7) and at least lookahead / w + 4 buckets, so that one window's
// bucket range never wraps; C slots per bucket, twice the expected front occupancy plus
// 4; spill lists of max(64, C) events.
struct LabGeometry {
  uint32_t nb_log2, c_log2, spill;
  float inv_w;
};

inline uint32_t next_pow2(double x) {
  uint32_t p = 1;
  while ((double)p < x && p < (1u << 30)) p <<= 1;
  return p;
}

inline gpq_status lab_geometry(const gpq_phold_config& c, LabGeometry* g) {
  const double la = c.lookahead, E = c.events_per_lp;
  double w = std::max(6.0 * (la + 1.0) / E, la / 2.5);
  double need = std::max(std::ceil((la + 7.0) / w), std::ceil(la / w) + 4.0);
  if (need > 1024.0) {
    w = std::max((la + 7.0) / 1024.0, la / 1020.0);
    need = 1024.0;
  }
  const uint32_t nb = std::max(16u, next_pow2(need));
  const double occ = E * w / (la + 1.0);
  const uint32_t cs = std::min(1024u, std::max(16u, next_pow2(std::ceil(2.0 * occ + 4.0))));
  g->nb_log2 = ilog2_ceil(nb);
  g->c_log2 = ilog2_ceil(cs);
  g->spill = std::max(64u, cs);
  g->inv_w = (float)(1.0 / w);
  GPQ_CHECK_ARG((double)c.lookahead * g->inv_w + 3.0 <= (double)nb,
                "bucketed local array queue: lookahead too wide for the bucket ring");
  GPQ_CHECK_ARG(((double)c.end_time + la + 20.0) * g->inv_w < 2147483648.0,
                "bucketed local array queue: end_time too large for the bucket width");
  return GPQ_OK;
}

// Lanes per LP of the splay queue: one lane works on a tree, and lanes of a warp on
// different trees take different paths, so they run one after another: an LP gets as wide
// a group as one wave of threads (148 SMs x 1,024) allows.  Measured (16 events per LP,
// lookahead 1, end time 100; ms a run with 1 / 4 / 16 / 32 lanes): 1,024 LPs 13.0 / 4.9 /
// 3.2 / 2.4, 8,191 LPs 14.1 / 5.3 / 5.2 / 6.6; 36,473 LPs to end time 50 7.2 / 4.6 / 8.8 /
// 9.2; 65,536 LPs to end time 30 4.8 / 5.8 (1 / 4 lanes).
inline uint32_t lsq_lanes(uint32_t num_lps) {
  for (uint32_t g = 32; g >= 4; g >>= 1)
    if ((uint64_t)num_lps * g <= 148u * 1024u) return g;
  return 1;
}

// Default lanes per LP of the local array queue, sorted (laq_mode 0) and unordered (1).  A wave
// of CTAs holds 14,208 LPs with 8 lanes each, 7,104 with 16, 3,552 with 32.  In one wave a
// window is one LP's chain of dependent steps, which more lanes shorten when the LP has several
// events; between one and one and a half waves of 8 lanes, three short rounds of 16 beat two
// long ones; otherwise the fixed steps per LP count and 8 lanes cost least.  Where 8 lanes hold
// all LPs at once and 16 do, or nearly do, the unordered arrays, whose events take fewer steps,
// are later to gain from 16.  Measured (us a window, 8 / 16 / 32 lanes; events per LP and
// window), sorted: 1,024 LPs 6.7 / 6.2 / 5.6 (0.8), 10.1 / 7.5 / 6.1 (8); 3,000 6.9 / 6.8 / 7.0
// (0.8), 10.7 / 8.2 / 7.8 (8); 7,000 7.8 / 8.4 (0.8), 9.0 / 8.6 (3), 20.1 / 13.5 (11); 7,500
// 20.3 / 20.8 (11); 21,000 14.8 / 15.8 (3), 18.1 / 17.0 (5), 42.3 / 33.7 (21); 24,000 38.1 /
// 37.0 (11); 40,000 16.8 / 25.1 (0.8), 31.1 / 33.1 (8); 65,536 49.9 / 51.7 (8).  Unordered:
// 1,024 8.1 / 6.4 / 5.1 (0.8), 11.2 / 7.2 / 5.3 (8); 3,000 8.3 / 6.9 / 6.4 (0.8), 11.7 / 7.8 /
// 6.8 (8); 4,096 9.3 / 7.6 (3); 7,000 9.9 / 11.4 (3), 12.7 / 12.9 (8), 24.5 / 21.9 (11); 18,000
// 18.5 / 19.3 (5), 44.8 / 40.4 (11); 21,000 27.5 / 26.1 (8); 40,000 44.5 / 43.3 (8).
inline uint32_t laq_lanes(const gpq_phold_config& c) {
  const uint32_t L = c.num_lps;
  const double events = (double)c.events_per_lp * c.lookahead / (1.0 + c.lookahead);
  const bool unordered = c.laq_mode == 1;
  if (L <= 2048 || (L <= 3552 && events >= 5.0)) return 32;
  if (L <= 4096 || (L <= 7104 && events >= (unordered ? 8.0 : 2.5))) return 16;
  return L > 14208 && L <= 21312 && events >= (unordered ? 8.0 : 5.0) ? 16 : 8;
}

// Whether the local heap queue takes a warp per LP and a window's items in one piece
// (lhqw_lp_stage) where no number of lanes is asked for: with many events per LP and
// window, or, while one wave of warps holds all LPs, from a number of events that grows with
// the LPs on; otherwise the warp's fixed steps cost more than a few single pops.  Measured
// (us a window, 8 lanes / warp; events per LP and window): 64 LPs 5.9 / 6.1 (0.3), 8.6 / 7.3
// (1.5); 1,024 7.2 / 7.0 (0.7), 19.8 / 8.5 (8); 3,000 7.5 / 8.4 (0.7), 11.5 / 10.2 (2); 4,096
// 9.5 / 10.5 (1.3), 14.6 / 12.8 (3); 8,191 39.9 / 29.6 (11); 20,011 24.8 / 39.5 (2) and 58.4 /
// 39.3 (8); 44,123 230 / 121 (21); 65,536 104 / 139 (6) and 112 / 103 (8).
inline bool lhq_warp(const gpq_phold_config& c) {
  const double events = (double)c.events_per_lp * c.lookahead / (1.0 + c.lookahead);
  return events >= 7.5 || (c.num_lps <= 4096 && events >= std::max(0.5, c.num_lps / 2048.0));
}

// Lanes per LP that a run uses: the asked-for number, or by the rules above.  `c` is the
// normalized configuration, which goes into snapshots and keeps 8 (splay queue: 1) for the
// default, so that a run's state goes between handles whatever their lanes.
inline uint32_t run_lanes(const gpq_phold_config& c, uint32_t asked) {
  if (c.queue_kind == GPQ_QUEUE_LSQ) return lsq_lanes(c.num_lps);
  if (c.queue_kind == GPQ_QUEUE_LAQ && c.laq_mode != 2 && asked == 0) return laq_lanes(c);
  return c.lanes_per_lp;
}

// Fills the per-kind defaults (capacity 256, insert capacity 64, 256-thread CTAs,
// 8 lanes per LP; one lane for the splay queue) and checks them.
inline gpq_status normalize_queue_config(gpq_phold_config* c) {
  if (c->capacity == 0) c->capacity = 256;
  if (c->insert_capacity == 0) c->insert_capacity = 64;
  GPQ_CHECK_ARG(is_pow2(c->capacity) && c->capacity >= 32 && c->capacity <= (1u << 16),
                "capacity must be a power of two in [32, 65536]");
  if (c->queue_kind == GPQ_QUEUE_LSQ)
    GPQ_CHECK_ARG(c->capacity <= 32768, "splay queue capacity must be <= 32768");
  GPQ_CHECK_ARG(c->insert_capacity >= 1 && c->insert_capacity <= 1024, "insert_capacity must be in [1, 1024]");
  GPQ_CHECK_ARG(c->events_per_lp <= c->capacity, "events_per_lp must not exceed capacity");
  GPQ_CHECK_ARG(c->events_per_lp <= 8192, "events_per_lp must be <= 8192");
  if (c->block_threads == 0) c->block_threads = 256;
  GPQ_CHECK_ARG(c->block_threads % 32 == 0 && c->block_threads >= 32 && c->block_threads <= 1024,
                "block_threads must be a multiple of 32 in [32, 1024]");
  if (c->queue_kind == GPQ_QUEUE_LSQ) c->lanes_per_lp = 1;
  if (c->lanes_per_lp == 0) c->lanes_per_lp = 8;
  if (c->queue_kind == GPQ_QUEUE_LAQ)
    GPQ_CHECK_ARG(c->lanes_per_lp == 4 || c->lanes_per_lp == 8 || c->lanes_per_lp == 16 || c->lanes_per_lp == 32,
                  "lanes_per_lp must be 4, 8, 16 or 32 for the local array queue");
  if (c->queue_kind == GPQ_QUEUE_LHQ)
    GPQ_CHECK_ARG(c->lanes_per_lp == 1 || c->lanes_per_lp == 4 || c->lanes_per_lp == 8 || c->lanes_per_lp == 16 ||
                      c->lanes_per_lp == 32,
                  "lanes_per_lp must be 1, 4, 8, 16 or 32 for the local heap queue");
  return GPQ_OK;
}

// The LAQ entry points call this name.
inline gpq_status normalize_laq_config(gpq_phold_config* c) { return normalize_queue_config(c); }

// Halves the CTA size until the per-CTA merge scratch (one slice per lane group) fits
// `limit` bytes of shared memory.  Returns false if even one warp does not fit.
inline bool fit_block_to_smem(uint32_t* block, uint32_t group, size_t group_bytes, size_t limit) {
  while ((size_t)(*block / group) * group_bytes > limit && *block > 32) *block /= 2;
  if (*block < 32) *block = 32;
  return (size_t)(*block / group) * group_bytes <= limit;
}

}  // namespace gpq
