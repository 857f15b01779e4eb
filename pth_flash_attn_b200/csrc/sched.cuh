// Work-item schedule of the persistent integer kernel: which (row tile, KV head, split)
// items a launch consists of, how many splits a request gets, and which CTA runs which item.
//
// The host fixes only what a captured CUDA graph may bake in: the number of CTAs and the
// largest split count the workspace holds (num_splits).  Everything that depends on the
// lengths is decided on the device from seq_lens / query_start_loc, by every CTA alike:
//
//   request r     row_tiles(r) = ceil(q_len / bq) row tiles (0 if the launch does not serve
//                 the request), kv_tiles(r) = KV tiles its rows touch together;
//   total work    W = Hkv * sum_r row_tiles(r) * kv_tiles(r)   (KV tiles to read);
//   item size     t* = KV tiles an item should hold: W / (CTAs * m) with m <= 8 items per
//                 CTA, chosen so that t* stays near kItemTilesTarget when there is that much
//                 work, and never below kItemTilesMin;
//   splits        S(r) = round(kv_tiles(r) / t*) clamped to [1, num_splits]: every request is
//                 cut into pieces of about t* tiles, so the items of a launch are about
//                 equally long whatever the mix of context lengths;
//   item order    request-major; inside a request (row tile, split)-major and KV head
//                 fastest, so that the Hkv heads of the same pages are adjacent items;
//   assignment    CTA c runs items c, c + CTAs, c + 2 CTAs, ...: adjacent items (the heads of
//                 one page set) run at the same time on neighbouring CTAs, which lets the
//                 boundary sectors of neighbouring 264-byte cells be served from L2.
//
// That schedule leaves CTAs idle in the last round (mean over longest CTA: 0.83 for a mixed batch of 48
// decode requests, 0.87 for 64 requests of two KV heads, 0.5 - 0.8 for short ragged contexts).  A launch with enough
// work whose caller allows enough pieces (range_sched) is dealt out in RANGES instead: the KV tiles of all
// served row tiles form one sequence, which is cut into equal runs, one for every group of Hkv CTAs; CTA h of a group
// reads KV head h, so the heads of a page are still read at the same time.  The CTAs left over when Hkv does not
// divide their number form a last, smaller group, whose CTAs take several heads one after the other and whose run is
// as much shorter.  A cut closer than `snap` tiles to an end of a row tile moves to that end.
// Measured (equal pieces -> ranges): 32 requests x 4 tokens x 16 to 32 K keys 414 -> 383 us, decode at 64 dims over
// 4 to 12 K keys 184 -> 170, 64 x 8,192 keys 212 -> 205, mixed batch 3,350 -> 3,120.
//
// Splits s >= S(r) of a request hold no keys: their log-sum-exp is set to -inf by the CTA
// that runs split 0 of the same rows, and the combine skips them.
//
// These functions compile for the host too (the schedule is tested without a GPU).
#pragma once

#include <stdint.h>

#include "params.cuh"

#if defined(__CUDACC__)
#define PTHB_HD __host__ __device__ __forceinline__
#else
#define PTHB_HD inline
#endif

namespace pthb200 {

constexpr int kItemTilesTarget = 24;  // KV tiles per item when a CTA has work for several items
constexpr int kItemsPerCtaMax = 8;    // items per CTA the split choice aims for at most
constexpr int kItemTilesMin = 4;      // an item is never planned shorter than this

struct SchedShape {
  int32_t group, num_kv_heads, bq, num_splits, window, causal, row_class, class_rows;
};

PTHB_HD int sched_min(int a, int b) { return a < b ? a : b; }
PTHB_HD int sched_max(int a, int b) { return a > b ? a : b; }

// Inclusive visible key range of query token i of a request (bottom-right aligned).
PTHB_HD void visible_bounds(int window, int causal, int seq_len, int q_len, int i, int* lo, int* hi) {
  const int pos = seq_len - q_len + i;
  *lo = window > 0 ? sched_max(0, pos - window + 1) : 0;
  int h;
  if (causal) {
    h = pos;
  } else if (window > 0) {
    const int64_t far = (int64_t)pos + window - 1;
    h = far > (int64_t)(seq_len - 1) ? seq_len - 1 : (int)far;
  } else {
    h = seq_len - 1;
  }
  *hi = sched_min(h, seq_len - 1);
}

// Row tiles of a request in this launch (0: the launch does not serve it).
PTHB_HD int req_row_tiles(const SchedShape& s, int q_len) {
  if (q_len <= 0) return 0;
  if (s.row_class != 0 && (((int64_t)q_len * s.group <= s.class_rows) != (s.row_class == 1))) return 0;
  return q_len <= s.bq ? 1 : (q_len + s.bq - 1) / s.bq;
}

// KV tiles the rows of a request touch together.
PTHB_HD int req_kv_tiles(const SchedShape& s, int q_len, int seq_len) {
  if (q_len <= 0) return 0;
  int lo0, hi0, lo1, hi1;
  visible_bounds(s.window, s.causal, seq_len, q_len, 0, &lo0, &hi0);
  visible_bounds(s.window, s.causal, seq_len, q_len, q_len - 1, &lo1, &hi1);
  const int rb = lo0, re = sched_max(hi0, hi1) + 1;
  if (re <= rb) return 0;
  return (re + kKvTile - 1) / kKvTile - rb / kKvTile;
}

// t*: KV tiles an item should hold, from the total work and the number of CTAs.
PTHB_HD int item_tiles(unsigned long long total_tiles, int num_ctas) {
  // (divisions of 64-bit numbers are slow, and the first item waits for them)
  const unsigned ctas = num_ctas > 0 ? (unsigned)num_ctas : 1u;
  const unsigned long long per = total_tiles < (1ull << 31) ? ((unsigned)total_tiles + ctas - 1) / ctas : (total_tiles + ctas - 1) / ctas;
  const unsigned per_cta = per > (1ull << 31) ? 1u << 31 : (unsigned)per;  // (far more than a cache holds)
  unsigned m = per_cta / kItemTilesTarget;
  if (m < 1) m = 1;
  if (m > (unsigned)kItemsPerCtaMax) m = kItemsPerCtaMax;
  unsigned t = (per_cta + m - 1) / m;
  if (t < (unsigned)kItemTilesMin) t = kItemTilesMin;
  if (t > (1u << 30)) t = 1u << 30;
  return (int)t;
}

// S(r): splits of a request whose rows touch kv_tiles KV tiles.
PTHB_HD int req_splits(int kv_tiles, int t_star, int num_splits) {
  const unsigned s = ((unsigned)kv_tiles + (unsigned)t_star / 2) / (unsigned)t_star;
  return s < 1 ? 1 : (s > (unsigned)num_splits ? num_splits : (int)s);
}

// KV tiles of a row tile of bq query tokens, as far as the host knows: a row of the block table and the window bound
// them, the window on both sides of a token where the mask is not causal.  (A row that is longer than the stride says, or
// a stride of 0, which says nothing: the CTAs go by the lengths, this only by the time.)
inline int64_t row_tile_bound(int64_t block_table_row_stride, int block_size, int window, int causal, int bq) {
  constexpr int64_t most = 0x7fffffff;
  int64_t tiles = block_table_row_stride > 0 && block_table_row_stride < (1 << 30) ? (block_table_row_stride * block_size + 127) / 128 : most;
  if (window > 0) {
    const int64_t in_window = ((int64_t)window * (causal ? 1 : 2) + bq) / 128 + 2;
    tiles = tiles < in_window ? tiles : in_window;
  }
  return tiles < most ? tiles : most;
}
// Pieces that row tiles of at most `tiles` KV tiles are cut into at most.
inline int pieces_bound(int64_t tiles, int num_splits) {
  const int64_t pieces = (tiles + kItemTilesMin / 2) / kItemTilesMin;
  return pieces < 1 ? 1 : pieces < num_splits ? (int)pieces : num_splits;
}

// Items of a request, and the coordinates of its item `local`.
PTHB_HD int64_t req_items(int row_tiles, int splits, int num_kv_heads) {
  return (int64_t)row_tiles * splits * num_kv_heads;
}
struct ItemCoord {
  int32_t row_tile, split, kvh;
};
PTHB_HD ItemCoord item_coord(int local, int num_kv_heads, int splits) {
  ItemCoord c;
  // (unsigned, and no division for the one row tile that most requests have: the first item waits for it)
  const unsigned rest = (unsigned)local / (unsigned)num_kv_heads;
  c.kvh = (int)((unsigned)local - rest * (unsigned)num_kv_heads);
  c.row_tile = rest < (unsigned)splits ? 0 : (int)(rest / (unsigned)splits);
  c.split = (int)rest - c.row_tile * splits;
  return c;
}

// KV tiles [tile_begin, tile_end) of split `split` out of `splits` for a row tile whose
// rows see the keys [range_begin, range_end) together: whole tiles, sizes differ by <= 1.
PTHB_HD void split_tile_span(int range_begin, int range_end, int split, int splits, int* tile_begin, int* tile_end) {
  if (range_end <= range_begin) {
    *tile_begin = *tile_end = 0;
    return;
  }
  const int t0 = range_begin / kKvTile;
  const int t1 = (range_end + kKvTile - 1) / kKvTile;
  const int n = t1 - t0;
  if (n < (1 << 15) && split < (1 << 16)) {  // (the products fit 32 bits, whose divisions are much faster)
    *tile_begin = t0 + (int)((uint32_t)split * (uint32_t)n / (uint32_t)splits);
    *tile_end = t0 + (int)((uint32_t)(split + 1) * (uint32_t)n / (uint32_t)splits);
  } else {
    *tile_begin = t0 + (int)((int64_t)split * n / splits);
    *tile_end = t0 + (int)((int64_t)(split + 1) * n / splits);
  }
}

// ---- ranges ----
// KV tiles per CTA from which a launch is dealt out in ranges.  Below, a CTA's share is one or two pieces, and cuts that
// ignore the ends of requests make them three.  Equal pieces against ranges: 16 x U[1, 4096] keys of 8 heads (16 tiles
// per CTA) 31.7 and 24.1 us, 16 x U[1, 8192] at 64 dims 48.1 and 34.4, 69 x U[1, 951] at 256 dims (15 tiles) 48.4 and 42.5,
// 8 x 8,192 34.2 and 34.7, 60 x U[1, 988] at 8 rows (14 tiles) 31.9 and 34.1; 8 x U[1, 4096] (8 tiles) 17.7 and 18.5.
constexpr int kRangeTilesMin = 12;
constexpr int kRangeGroupsMax = 160;   // groups a scheduler warp holds the cuts of

struct RangeSched {
  uint32_t work;         // KV tiles of one head; 0: the launch is not dealt out in ranges
  int32_t full;          // groups of num_kv_heads CTAs
  int32_t tail;          // CTAs of the last, smaller group (0: there is none)
  int32_t tail_passes;   // heads each of its CTAs takes one after the other
  int32_t snap;
};

// The run of a group of `tail_passes` times the tail group's length, or a rounding of it: the cut in front of group g
// is at ceil(work * g * passes / (full * passes + 1)) (without a tail group: ceil(work * g / full)).
PTHB_HD int range_groups(const RangeSched& r) { return r.full + (r.tail > 0 ? 1 : 0); }
PTHB_HD uint32_t range_cut(const RangeSched& r, int g) {
  const uint32_t per = r.tail > 0 ? (uint32_t)r.tail_passes : 1u, whole = (uint32_t)r.full * per + (r.tail > 0 ? 1u : 0u);
  if (g >= range_groups(r)) return r.work;
  const unsigned long long num = (unsigned long long)r.work * ((uint32_t)g * per) + (whole - 1);
  if (num <= 0xffffffffull) return (uint32_t)num / whole;
  return (uint32_t)(num / whole);
}
// work: KV tiles of one head over the row tiles of all served requests; longest: of one row tile at most.
PTHB_HD RangeSched range_sched(unsigned long long work, int longest, int num_kv_heads, int num_ctas, int num_splits) {
  RangeSched r;
  r.work = 0;
  r.full = r.tail = r.tail_passes = 0;
  r.snap = 1;
  if (num_splits < 2 || work > (1ull << 30) || work * (unsigned long long)num_kv_heads < (unsigned long long)num_ctas * kRangeTilesMin)
    return r;
  r.full = num_ctas / num_kv_heads;
  r.tail = num_ctas % num_kv_heads;
  r.tail_passes = r.tail > 0 ? (num_kv_heads + r.tail - 1) / r.tail : 0;
  if (range_groups(r) > kRangeGroupsMax) return r;
  const uint32_t per = r.tail > 0 ? (uint32_t)r.tail_passes : 1u, whole = (uint32_t)r.full * per + (r.tail > 0 ? 1u : 0u);
  // the shortest distance of two cuts inside a row tile: a whole group's run
  const unsigned long long run = work * per / whole;
  if (r.full < 1 || run < 4) return r;
  // a row tile of n tiles holds at most ceil((n - 1) / run) cuts, and one piece more than cuts
  const unsigned long long cuts = longest > 1 ? ((unsigned long long)longest - 1 + run - 1) / run : 0;
  if (cuts + 1 > (unsigned long long)num_splits) return r;
  r.snap = run >= 32 ? 2 : 1;
  r.work = (uint32_t)work;
  return r;
}
// Part [*begin, *end) of a row tile that starts at `start` of the sequence and has n KV tiles which belongs to the
// run [lo, hi) of a group; false if there is none.
PTHB_HD bool range_part(const RangeSched& r, uint32_t start, int n, uint32_t lo, uint32_t hi, int* begin, int* end) {
  int b = lo > start ? (int)(lo - start) : 0;
  int e = hi - start < (uint32_t)n ? (int)(hi - start) : n;
  if (b > 0 && b <= r.snap) b = 0;
  else if (b > 0 && n - b <= r.snap) b = n;
  if (e < n && e <= r.snap) e = 0;
  else if (e < n && n - e <= r.snap) e = n;
  *begin = b;
  *end = e;
  return b < e;
}
// Whether a cut of the sequence divides a row tile (rather than moving to one of its ends).
PTHB_HD bool range_divides(const RangeSched& r, uint32_t start, int n, uint32_t cut) {
  return cut > start + (uint32_t)r.snap && cut + (uint32_t)r.snap < start + (uint32_t)n;
}

}  // namespace pthb200
