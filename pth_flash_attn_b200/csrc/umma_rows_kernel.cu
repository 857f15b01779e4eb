// Row-major tcgen05 attention kernel, head size 128: query rows on the MMA M dimension.
//
// For launches with many rows per KV head (prefill chunks, wide verification steps) the
// work per KV tile is dominated by the two contractions and by one exponential per
// (row, key).  This kernel gives every query row of a 128-row tile one softmax thread
// (TMEM lane = row), so the row maximum and sum never leave that thread's registers:
//
//   loader     (1 warp)   TMA page copies of the raw cache cells into a ring of raw half
//                         stages of 64 keys (same scheme as the integer kernel);
//   producers  (8 warps)  thread t of the K set / V set widens key t's int8 K / V bytes
//                         exactly to fp16 into the K image / the V stage (canonical
//                         no-swizzle layout); the K set publishes both scales of the key;
//   MMA issuer (1 warp, one elected lane) S = Q K^T (M = 128 rows, N = 128 keys, fp32 in
//                         TMEM, two buffers: tile i uses buffer i % 2, so S(i + 1) is computed
//                         while the softmax warps work on tile i) and O(g) += P V for each
//                         softmax group g, with P read from TMEM (the A operand) and V from
//                         the V stage as an MN-major B operand;
//   softmax    (2 groups of 4 warps; group g owns keys 64 g .. 64 g + 63 of EVERY tile)
//                         thread r reads the 64 scores of row r and its half once, pass 1
//                         turns them into log2 units (S * k_scale * softmax_scale * log2 e +
//                         log2 v_scale) and finds their maximum, pass 2 writes P as packed
//                         fp16 into TMEM over the columns of S it has read.  The
//                         reference maximum of a (row, half) moves only when the running
//                         maximum outgrows it by 2^4; then the thread rescales its row of
//                         O(g) in TMEM.  In steady state O is never touched by the softmax.
// The two groups' (m, l, O) are merged in the epilogue.  TMEM: S0 S1 O0 O1, 128 columns
// each.  The CTA starts with 96 registers per thread; the producer warpgroups hand part of
// theirs to the softmax warpgroups (setmaxnreg).  Every mbarrier wait is bounded (see
// page_copy.cuh).
#include <cuda.h>

#include <type_traits>

#include "params.cuh"
#include "sched.cuh"
#include "umma_rows.cuh"
#include "page_copy.cuh"
#include "pdl.cuh"

namespace pthb200 {

__device__ unsigned int g_rows_status = 0;

namespace {

constexpr int kRGroup = 128;             // threads of one softmax group = rows of a tile
constexpr int kRSoftmax = 2 * kRGroup;   // warps 0-3, 4-7
constexpr int kRProducers = 256;         // warps 8-11 (K half) and 12-15 (V half)
constexpr int kRMmaWarp = 16, kRLoadWarp = 17;
constexpr int kRThreads = 576;
constexpr int kRNS = 2;                  // V stages
constexpr int kHalfKeys = 64;            // keys of one raw half stage
constexpr int kRawHalfBytes = kHalfKeys * kRawRow;   // 17,408 B
constexpr int kRVStage = kWideBytes;                 // V image
constexpr int kRKsRing = 4;                          // tiles of key scales kept
constexpr int kRQBarrier = kRSoftmax + 32;  // Q image complete: softmax, MMA issuer
// Registers: the CTA starts with 96 per thread (18 warps: five on two of the SM's four schedulers, whose
// 16,384 registers that fills).  The two producer warpgroups hand 32 per thread to the two softmax
// warpgroups, which keep the 64 scores of a row and half tile in registers between the two passes;
// every scheduler has two warps of either kind.
constexpr int kRProducerRegs = 64, kRSoftmaxRegs = 128;
constexpr float kRescaleGap = 4.0f;      // log2 units a row maximum may outgrow its reference

template <int kRNK, int kRNR>  // K images, raw HALF stages (64 keys each)
struct RLayout {
  static constexpr int kimg = 0;
  static constexpr int vst = kimg + kRNK * kWideBytes;
  static constexpr int qimg = vst + kRNS * kRVStage;
  static constexpr int raw = qimg + kQImageBytes;
  static constexpr int ksc = raw + kRNR * kRawHalfBytes;       // KeyScales<128> [kRKsRing]
  static constexpr int park_m = ksc + kRKsRing * (int)sizeof(KeyScales<kTileKeys>); // float [2 groups][128]
  static constexpr int park_l = park_m + 2 * kRGroup * 4;      // float [2 groups][128]
  static constexpr int fix = park_l + 2 * kRGroup * 4;         // float [128], see QueryScale
  static constexpr int stats = fix + kRGroup * 4;              // float [2][128], see merge_pieces
  static constexpr int bars = stats + 2 * kRGroup * 4;         // uint64 [...]
  static constexpr int park = kimg;                            // the K images, idle at the end: [128][128 rows] fp32
  static_assert(kHeadDim * kRGroup * 4 <= kRNK * kWideBytes, "room for a parked accumulator");
  static constexpr int n_bars = kRNS * 2 + 2 * kRNK + 6 + 2 * kRNR;
  static constexpr int misc = bars + n_bars * 8;
  static constexpr int total = misc + 32 + 4 * kRowsItemInts;
};

template <int kRNK, int kRNR>
struct RBars {
  static constexpr int vfull = 0;                      // [NS] V producers -> PV, 128 arrivals
  static constexpr int vempty = kRNS;                  // [NS] PV commit -> V producers
  static constexpr int kempty = 2 * kRNS;              // [NK] QK commit -> K producers
  static constexpr int kfull = 2 * kRNS + kRNK;        // [NK] K producers -> QK, 128 arrivals
  static constexpr int s_ready = 2 * kRNS + 2 * kRNK;  // [2] QK commit -> softmax
  static constexpr int p_ready = s_ready + 2;          // [2] softmax -> PV, 256 arrivals
  static constexpr int pv_done = p_ready + 2;          // [2] PV commit -> QK, softmax
  static constexpr int raw_full = pv_done + 2;         // [NR]
  static constexpr int raw_free = raw_full + kRNR;     // [NR] producers -> loader, 128 arrivals
};

// Key of a tile held by row `r` of its images: with contiguous cells the rows of a half tile
// hold its even keys, then its odd ones (see the producers).
__device__ __forceinline__ int tile_key_rows(int raw_mode, int r) {
  return raw_mode == 2 ? (r & 64) + 2 * (r & 31) + ((r >> 5) & 1) : r;
}

template <int kRNK, int kRNR, bool kClusters>
__global__ void __launch_bounds__(kRThreads, 1)
umma_rows_attention_kernel(const __grid_constant__ KernelParams p, const __grid_constant__ CUtensorMap tmap) {
  using L = RLayout<kRNK, kRNR>;
  using B = RBars<kRNK, kRNR>;
  static_assert(L::raw % 128 == 0 && L::vst % 128 == 0 && L::qimg % 128 == 0, "TMA / image alignment");
  static_assert(L::total <= 227 * 1024, "shared memory of one CTA");
  extern __shared__ __align__(128) uint8_t smem[];
  uint8_t* qimg = smem + L::qimg;
  float* park_m = reinterpret_cast<float*>(smem + L::park_m);
  float* park_l = reinterpret_cast<float*>(smem + L::park_l);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::bars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::misc);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + L::misc + 8);
  KeyScales<kTileKeys>* key_scales = reinterpret_cast<KeyScales<kTileKeys>*>(smem + L::ksc);

  int kvh, tile_index;
  rows_cta<kClusters>(p, &kvh, &tile_index);
  const int split = blockIdx.y;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // Barriers and TMEM are set up by the warps that wait for nothing else.  The CTA of a further piece of the bound, which
  // mostly finds that its request is not cut that often, takes TMEM when it has found work (see launch_row_tiles).
  const bool tmem_ahead = split == 0;
  if (warp == kRLoadWarp) {
    if (lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap)) : "memory");
    if (tmem_ahead) {
      tc::tmem_alloc(tslot, 512);
      tc::tmem_relinquish();
    }
  }
  if (warp == kRMmaWarp && lane == 0) {
    for (int s = 0; s < kRNS; ++s) {
      tc::mbar_init(&bars[B::vfull + s], kRProducers / 2);
      tc::mbar_init(&bars[B::vempty + s], 1);
    }
    for (int s = 0; s < kRNK; ++s) {
      tc::mbar_init(&bars[B::kempty + s], 1);
      tc::mbar_init(&bars[B::kfull + s], kRProducers / 2);
    }
    for (int g = 0; g < 2; ++g) {
      tc::mbar_init(&bars[B::s_ready + g], 1);
      tc::mbar_init(&bars[B::p_ready + g], kRSoftmax);
      tc::mbar_init(&bars[B::pv_done + g], 1);
    }
    for (int s = 0; s < kRNR; ++s) {
      tc::mbar_init(&bars[B::raw_full + s], kHalfKeys >> p.copy_shift);  // page copies of a half stage
      tc::mbar_init(&bars[B::raw_free + s], kRProducers / 2);             // 64 K-set + 64 V-set threads
    }
    *abort_flag = 0;
    tc::mbar_init_fence();
  }
  if (!p.late_wait) pdl_wait();
  // Row tile of this CTA: warp 0 finds it; for longer lists of requests all threads bisect a shared-memory copy of
  // query_start_loc when it fits.
  constexpr int kQslCache = 4096;
  static_assert(kRNR * kRawHalfBytes >= 2 * kQslCache * 4, "the raw ring holds the copies of query_start_loc and seq_lens");
  RowsItem item;
  int* item_s = reinterpret_cast<int*>(smem + L::misc + 32);
  const bool by_warp = p.num_reqs <= kWarpRequests && p.tile_map == 0;
  if (by_warp) {
    if (warp == 0) {
      unsigned long long work = 0;
      const RowTile found = warp_row_tile(p, tile_index, p.num_splits > 1, sched_shape(p), &work);
      item = rows_item<kClusters>(p, found, split, [&] { return warp_sum(work); });
      if (lane == 0) *reinterpret_cast<RowsItem*>(item_s) = item;
    }
  } else {
    RowTile t;
    if (p.tile_map == 0 && p.num_reqs + 1 <= kQslCache) {
      int* qsl_s = reinterpret_cast<int*>(smem + L::raw);
      int* len_s = qsl_s + kQslCache;
      for (int i = tid; i <= p.num_reqs; i += kRThreads) {
        qsl_s[i] = __ldg(p.query_start_loc + i);
        if (i < p.num_reqs) len_s[i] = __ldg(p.seq_lens + i);
      }
      __syncthreads();
      t = resolve_row_tile_with(p, tile_index, [&](int i) { return qsl_s[i]; }, [&](int r) { return len_s[r]; });
      tc::fence_async_smem();  // (page copies write here next, through the other proxy)
      __syncthreads();
    } else {
      t = resolve_row_tile(p, tile_index);
    }
    item = rows_item<kClusters>(p, t, split, [&] { return cta_work<kRThreads>(p, smem + L::misc + 16); });
    if (tid == 0) *reinterpret_cast<RowsItem*>(item_s) = item;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  item = *reinterpret_cast<const RowsItem*>(item_s);
  if (item.state != 1 || (split == 0 && item.nsplits < p.num_splits)) write_empty<kRThreads, kHeadDim>(p, item, kvh, split);
  if (item.state != 1) {
    if (tmem_ahead && warp == kRLoadWarp) tc::tmem_dealloc(*tslot, 512);
    if (p.late_wait) pdl_wait();
    return;
  }
  if (!tmem_ahead) {
    if (warp == kRLoadWarp) {
      tc::tmem_alloc(tslot, 512);
      tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
  }
  const uint32_t tmem_base = *tslot;
  const RowTile& t = item.t;
  const int rows = item.rows;  // <= 128 by construction of bq
  const int tile_begin = item.tile_begin, tile_end = item.tile_end, range_begin = item.range_begin, range_end = item.range_end;

  const int n_tiles = tile_end - tile_begin;
  const uint32_t kimg_s = tc::smem_u32(smem + L::kimg), vst_s = tc::smem_u32(smem + L::vst);
  bool ok = true;

  if (warp >= 8 && warp < kRMmaWarp) {
    // =========================== producers ====================================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRProducerRegs));
    // Warps 8-11 widen the K half of the raw cells into the K image and publish both scales,
    // warps 12-15 the V half into the V stage; thread pt of either set owns key pt of the tile.
    const int pt = tid & 127;
    const bool v_part = warp >= 12;
    const int bs = p.copy_slots;  // slots of one page copy
    const uint8_t* kb = p.k.data + (int64_t)kvh * p.k.stride_head;
    const uint32_t delta = (uint32_t)(reinterpret_cast<uintptr_t>(kb) & 15);
    const int row_pitch = p.raw_mode == 1 ? kRawRow : 2 * kHeadDim + 8;
    // the raw ring is made of half stages of 64 keys: keys 0-63 of tile j are half stage
    // u = 2 j, keys 64-127 are u = 2 j + 1; half stage u sits in slot u % kRNR
    const int half = pt >> 6;
    // Contiguous cells (raw_mode 2) alternate between the two 8-byte alignments: a warp takes the
    // even keys or the odd ones of its half stage, so that it runs one of the two code paths
    // below.  Row pt of the images (and of the scale vectors) then holds key tile_key_rows(pt):
    // the order of the keys inside a tile changes no sum, and the softmax masks by that key.
    const int key = tile_key_rows(p.raw_mode, pt);
    const int my_page = (key & (kHalfKeys - 1)) >> p.copy_shift, my_slot = key & (bs - 1);
    const uint32_t cell_off = my_page * bs * kRawRow + my_slot * row_pitch + delta;  // inside a half stage
    const bool odd = (cell_off & 8u) != 0;
    const float score_mul = p.scale_log2 * query_ungain(p.q_dtype);
#pragma unroll 1
    for (int j = 0; j < n_tiles; ++j) {
      const int u = 2 * j + half;
      const int rs = u % kRNR;
      const int pos = (tile_begin + j) * kTileKeys + key;
      const bool valid = pos >= range_begin && pos < range_end;
      // A raw slot is used by the two halves in turn (kRNR is odd), and a parity wait only
      // tells apart two consecutive phases: this thread must not look at raw_full[rs] while
      // the slot's PREVIOUS half stage (the other half's) is still pending, or it would take
      // the phase before that one for its own, read stale bytes and release the slot early.
      // Page copies can complete out of order, so nothing else rules that out.  Wait first
      // until the previous occupant has been taken out of the slot.
      if (u >= kRNR) ok &= wait_or_abort(&bars[B::raw_free + rs], ((u / kRNR) - 1) & 1, abort_flag);
      ok &= wait_or_abort(&bars[B::raw_full + rs], (u / kRNR) & 1, abort_flag);
      // nine 16-byte chunks: raw words 0..35 (K half, k_scale) or 32..67 (k_scale, V half, v_scale)
      uint32_t w[36];
      if (valid) {
        const uint4* row = reinterpret_cast<const uint4*>(smem + L::raw + rs * kRawHalfBytes + (cell_off & ~15u)) +
                           (v_part ? 8 : 0);
#pragma unroll
        for (int c = 0; c < 9; ++c) {
          const uint4 v = row[c];
          w[4 * c] = v.x;
          w[4 * c + 1] = v.y;
          w[4 * c + 2] = v.z;
          w[4 * c + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int c = 0; c < 36; ++c) w[c] = 0u;
      }
      float v_scale = 1.f;
      if (!v_part && valid)
        v_scale = *reinterpret_cast<const float*>(smem + L::raw + rs * kRawHalfBytes + cell_off + 2 * kHeadDim + 4);
      mbar_arrive(&bars[B::raw_free + rs]);  // the half row is in registers: the stage may be refilled
      const int st = j % kRNS;
      if (!v_part) {
        uint8_t* kdst = smem + L::kimg + (j % kRNK) * kWideBytes + pt * 16;
        if (j >= kRNK) ok &= wait_or_abort(&bars[B::kempty + j % kRNK], ((j / kRNK) - 1) & 1, abort_flag);
        float k_scale;
        if (!odd) {
#pragma unroll
          for (int c = 0; c < kChunks; ++c)
            *reinterpret_cast<uint4*>(kdst + c * kChunkStride) = widen8_f16(make_uint2(w[2 * c], w[2 * c + 1]));
          k_scale = __uint_as_float(w[32]);
        } else {
#pragma unroll
          for (int c = 0; c < kChunks; ++c)
            *reinterpret_cast<uint4*>(kdst + c * kChunkStride) = widen8_f16(make_uint2(w[2 + 2 * c], w[3 + 2 * c]));
          k_scale = __uint_as_float(w[34]);
        }
        KeyScales<kTileKeys>& ks = key_scales[j % kRKsRing];
        const float vs = usable_v_scale(v_scale);
        ks.score[pt] = k_scale * score_mul;
        ks.lv[pt] = __log2f(vs);
        ks.iv[pt] = __fdividef(1.0f, vs);
        tc::fence_async_smem();
        mbar_arrive(&bars[B::kfull + j % kRNK]);
      } else {
        uint8_t* vstage = smem + L::vst + st * kRVStage;
        uint8_t* vdst = vstage + pt * 16;
        if (j >= kRNS) ok &= wait_or_abort(&bars[B::vempty + st], ((j / kRNS) - 1) & 1, abort_flag);
        if (!odd) {
#pragma unroll
          for (int c = 0; c < kChunks; ++c)
            *reinterpret_cast<uint4*>(vdst + c * kChunkStride) = widen8_f16(make_uint2(w[1 + 2 * c], w[2 + 2 * c]));
        } else {
#pragma unroll
          for (int c = 0; c < kChunks; ++c)
            *reinterpret_cast<uint4*>(vdst + c * kChunkStride) = widen8_f16(make_uint2(w[3 + 2 * c], w[4 + 2 * c]));
        }
        tc::fence_async_smem();
        mbar_arrive(&bars[B::vfull + st]);
      }
    }
  } else if (warp == kRLoadWarp) {
    // =========================== loader =======================================
    // One TMA copy per KV page of a tile, issued by lane `page`: a tiled tensor-map box of
    // [block_size slots] x [272 bytes] (raw_mode 1) or one bulk copy of a contiguous page
    // run (raw_mode 2); the next tile's block ids are fetched before waiting for the stage.
    const int pages_per_half = kHalfKeys >> p.copy_shift;
    if (lane < pages_per_half) {
      const int bs = p.copy_slots;
      const int32_t* bt = p.block_table + (int64_t)t.req * p.block_table_row_stride;
      const uint8_t* kb = p.k.data + (int64_t)kvh * p.k.stride_head;
      const uint32_t delta = (uint32_t)(reinterpret_cast<uintptr_t>(kb) & 15);
      const int tma_x = (int)((reinterpret_cast<uintptr_t>(kb) - delta -
                               (reinterpret_cast<uintptr_t>(p.k.data) & ~(uintptr_t)15)) >> 2);
      const uint32_t raw_s = tc::smem_u32(smem + L::raw);
      const int n_halves = 2 * n_tiles;
      // block id of this lane's page of half stage u, -1 if no key of the page is in range
      auto page_block = [&](int u) -> int {
        const int pos0 = tile_begin * kTileKeys + u * kHalfKeys + lane * bs;
        if (u >= n_halves || pos0 >= range_end || pos0 + bs <= range_begin) return -1;
        int page, slot;
        page_and_slot(p, pos0, &page, &slot);
        return __ldg(bt + page);
      };
      // first slot, inside its page, of this lane's copy of half stage u
      auto first_slot = [&](int u) -> int {
        int page, slot;
        page_and_slot(p, tile_begin * kTileKeys + u * kHalfKeys + lane * bs, &page, &slot);
        return slot;
      };
      int blk = page_block(0);
#pragma unroll 1
      for (int u = 0; u < n_halves; ++u) {
        const int blk_next = page_block(u + 1);
        const int rs = u % kRNR;
        if (u >= kRNR) ok &= wait_raw_free(&bars[B::raw_free + rs], ((u / kRNR) - 1) & 1, abort_flag);
        uint64_t* bar = &bars[B::raw_full + rs];
        if (blk >= 0 && ok) {
          const uint32_t dst = raw_s + rs * kRawHalfBytes + lane * bs * kRawRow;
          if (p.raw_mode == 1) {
            mbar_arrive_expect_tx(bar, bs * kRawRow);
            tma_load_3d(dst, &tmap, tma_x, first_slot(u), blk, bar);
          } else {
            const uint32_t bytes = bs * (2 * kHeadDim + 8);  // a multiple of 16, like the run's address
            mbar_arrive_expect_tx(bar, bytes);
            bulk_copy_g2s(dst, kb + (int64_t)blk * p.k.stride_block + (int64_t)first_slot(u) * (2 * kHeadDim + 8), bytes, bar);
          }
        } else {
          mbar_arrive(bar);
        }
        blk = blk_next;
      }
    }
  } else if (warp == kRMmaWarp) {
    // =========================== MMA issuer ===================================
    // ONE thread (the lane elect.sync picks) issues every tcgen05.mma of the CTA, in one fixed
    // order: QK(0), QK(1), then PV(i), QK(i + 2) for i = 0, 1, ...  S has two buffers in TMEM
    // (tile i uses buffer i % 2), so QK(i + 1) runs while the softmax warps work on tile i.
    // P(i) is written over the columns of S(i) it was computed from: QK(i + 2), which
    // overwrites that buffer, waits for PV(i) to have finished reading them - one whole tile
    // of softmax later than it is issued, so the wait is not on the critical path.  PV(i) is
    // two chains: keys 0-63 of the tile into O(0), keys 64-127 into O(1), the accumulators of
    // the two softmax groups.  (Another issuing warp
    // for PV cost the two-row-tile kernel 3 %; polling the barriers and
    // issuing whatever was ready first was slower, too.)  Operand descriptors are kept as register
    // word pairs.
    named_barrier(5, kRQBarrier);  // wait for the Q image
    {
      const RowsDesc qd = rows_desc(tc::smem_u32(qimg), kChunkStride, 128);
      const RowsDesc kd = rows_desc(kimg_s, kChunkStride, 128);
      const RowsDesc vd = rows_desc(vst_s, 128, kChunkStride);
      auto issue_qk = [&](int q) {
        ok &= wait_or_abort(&bars[B::kfull + q % kRNK], (q / kRNK) & 1, abort_flag);
        if (ok && elect_one()) {
          tc::fence_after_sync();
          RowsDesc k = kd;
          k.lo += (uint32_t)(q % kRNK) * (kWideBytes >> 4);
          issue_qk_rows_words(tmem_base + (q & 1) * 128, qd, k);
          tc::mma_commit(&bars[B::s_ready + (q & 1)]);
          tc::mma_commit(&bars[B::kempty + q % kRNK]);
        }
        __syncwarp();
      };
      issue_qk(0);
      if (n_tiles > 1) issue_qk(1);
#pragma unroll 1
      for (int i = 0; i < n_tiles && ok; ++i) {
        const int sb = i & 1;
        ok &= wait_or_abort(&bars[B::p_ready + sb], (i >> 1) & 1, abort_flag);
        // (P says nothing about V: the softmax reads the keys' scales, which the K set publishes)
        ok &= wait_or_abort(&bars[B::vfull + i % kRNS], (i / kRNS) & 1, abort_flag);
        if (ok && elect_one()) {
          tc::fence_after_sync();
          RowsDesc v = vd;
          v.lo += (uint32_t)(i % kRNS) * (kRVStage >> 4);
          issue_pv_halves_words(tmem_base + 256, tmem_base + sb * 128, v, i > 0);
          tc::mma_commit(&bars[B::pv_done + sb]);
          tc::mma_commit(&bars[B::vempty + i % kRNS]);
        }
        __syncwarp();
        if (i + 2 < n_tiles) {
          ok &= wait_or_abort(&bars[B::pv_done + sb], (i >> 1) & 1, abort_flag);
          issue_qk(i + 2);
        }
      }
    }
  } else if (warp < 8) {
    // =========================== softmax ======================================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRSoftmaxRegs));
    // Softmax group h (warps 4 h .. 4 h + 3) owns keys 64 h .. 64 h + 63 of EVERY tile: its thread
    // `row` keeps the running reference maximum and sum of that row over those keys and the
    // accumulator O(h) in TMEM; the two groups' results are merged at the end.  Both groups work
    // on tile i at the same time while the tensor core computes S(i + 1) into the other buffer.
    const int g = warp >> 2;
    const int row = tid & 127;   // row of the tile = TMEM lane
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_half = tmem_base + g * 64 + lane_addr;         // this group's columns of S buffer 0
    const uint32_t o_tmem = tmem_base + 256 + g * 128 + lane_addr;  // O(g)

    // ---- Q image: a warp converts 16 rows ----
    float* fix_s = reinterpret_cast<float*>(smem + L::fix);
    stage_queries<kHeadDim, 16>(p, t, kvh, rows, 16 * warp,
        [&](int n, int block, const uint4& v) { *reinterpret_cast<uint4*>(qimg + block * kChunkStride + n * 16) = v; },
        [&](int n, float fix) { fix_s[n] = fix; });
    tc::fence_async_smem();
    named_barrier(5, kRQBarrier);  // Q image complete; the QK issuer may start
    const float q_fix = fix_s[row];  // what the row's scores are multiplied by (QueryScale)

    int rlo = 0, rhi = -1;  // visible keys of this row (none for a padding row)
    if (row < rows) visible_range(p, t, t.first_idx + row / p.group, &rlo, &rhi);
    int mask_lo, mask_hi, tmp;  // key positions every live row sees: such tiles need no mask
    visible_range(p, t, t.first_idx + t.ntok - 1, &mask_lo, &tmp);
    visible_range(p, t, t.first_idx, &tmp, &mask_hi);
    float m_ref = -INFINITY;  // reference maximum of the row's exponentials (log2 units)
    float l = 0.f;            // 2^kPGain times the sum of exp2(score - m_ref), without v_scale
    // A warp whose 32 rows are all padding (a drafter step fills 64 of the 128 rows, a wide
    // verification step 32) leaves the issue slots to the others; its rows end as rows without
    // keys (m = -inf, l = 0), which the epilogue never writes.
    // (Their loop is a separate one: the live warps' loop carries no trace of the case.)
    if ((row & ~31) >= rows) {
#pragma unroll 1
      for (int i = 0; i < n_tiles; ++i) {
        // the arrival keeps the barrier's count and, behind the wait, its phase: S(i + 2) is not
        // ready before P(i) has been used
        ok &= wait_or_abort(&bars[B::s_ready + (i & 1)], (i >> 1) & 1, abort_flag);
        mbar_arrive(&bars[B::p_ready + (i & 1)]);
      }
    } else {  // warps with live rows (the loop keeps its indentation)
    auto walk_tiles = [&](auto own_power) {  // (one instance for warps without a row of its own power of two)
      constexpr bool kOwnPower = decltype(own_power)::value;
#pragma unroll 1
    for (int i = 0; i < n_tiles; ++i) {
      const KeyScales<kTileKeys>& ks = key_scales[i % kRKsRing];
      const uint32_t s_tmem = s_half + (i & 1) * 128;
      const int pos0 = (tile_begin + i) * kTileKeys;
      const bool interior = pos0 >= mask_lo && pos0 + (kTileKeys - 1) <= mask_hi;
      ok &= wait_or_abort(&bars[B::s_ready + (i & 1)], (i >> 1) & 1, abort_flag);
      tc::fence_after_sync();
      // the 64 scores of this row and half, read once
      uint32_t r[64];
      tc::tmem_ld32(s_tmem, r);
      tc::tmem_ld32(s_tmem + 32, r + 32);
      tc::tmem_ld_wait<64>(r);
      if constexpr (kOwnPower) scale_scores<64>(r, q_fix);

      // ---- pass 1: weighted scores in log2 units (kept in the registers) and their maximum ----
      // (two instances: interior tiles, which every live row sees whole, skip the mask)
      auto all_ready = [] {};
      const float m_t =
          interior ? softmax_pass1<64, false>(r, ks.score + g * 64, ks.lv + g * 64, all_ready, [](int) { return true; })
                   : softmax_pass1<64, true>(r, ks.score + g * 64, ks.lv + g * 64, all_ready, [&](int n) {
                       const int pos = pos0 + tile_key_rows(p.raw_mode, g * 64 + n);  // key held by column g 64 + n
                       return pos >= rlo && pos <= rhi;
                     });
      // ---- move the reference maximum if the row has outgrown it ----
      const float m_new = fmaxf(m_ref, m_t);
      const bool need = m_t > m_ref + kRescaleGap;  // also true when m_ref is still -inf
      if (i == 0) {
        m_ref = m_new;  // nothing accumulated yet
      } else if (__any_sync(0xffffffffu, need)) {
        // O(g) must be at rest: the PV of the previous tile has completed
        ok &= wait_or_abort(&bars[B::pv_done + ((i - 1) & 1)], ((i - 1) >> 1) & 1, abort_flag);
        tc::fence_after_sync();
        const float alpha = need ? ex2f(m_ref - m_new) : 1.0f;  // 0 when m_ref was -inf
#pragma unroll 1
        for (int j = 0; j < 8; ++j) {
          uint32_t o[16];
          tc::tmem_ld16(o_tmem + j * 16, o);
          tc::tmem_ld_wait<16>(o);
#pragma unroll
          for (int n = 0; n < 16; ++n) o[n] = __float_as_uint(__uint_as_float(o[n]) * alpha);
          tc::tmem_st16(o_tmem + j * 16, o);
        }
        tc::tmem_st_wait();
        l *= alpha;
        if (need) m_ref = m_new;
      }
      const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref - kPGain;

      // ---- pass 2: P as packed fp16 over the first columns of this half of S ----
      f32x2 ls[2] = {0ull, 0ull};
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint32_t pk[16];
        softmax_pass2(r + j * 32, ks.iv + g * 64 + j * 32, m_use, ls, pk);
        tc::tmem_st16(s_tmem + j * 16, pk);
      }
      l += sum_pairs(ls);
      tc::tmem_st_wait();
      tc::fence_before_sync();
      mbar_arrive(&bars[B::p_ready + (i & 1)]);  // this group's half of P(i) is complete
    }
    };
    if (__any_sync(0xffffffffu, q_fix != 1.0f)) walk_tiles(std::true_type{}); else walk_tiles(std::false_type{});
    }  // warps with live rows

    // ---- epilogue: merge the two groups' (m, l, O) and write the rows ----
    // (the commit after the last PV covers every MMA issued before it)
    ok &= wait_or_abort(&bars[B::pv_done + ((n_tiles - 1) & 1)], ((n_tiles - 1) >> 1) & 1, abort_flag);
    tc::fence_after_sync();
    // A row's two accumulators are in the same TMEM lane: either group reads both for its half of the columns, and
    // only maximum and sum go through shared memory.
    park_m[g * kRGroup + row] = m_ref;
    park_l[g * kRGroup + row] = l;
    named_barrier(4, kRSoftmax);
    const float m0 = park_m[row], m1 = park_m[kRGroup + row], l0 = park_l[row], l1 = park_l[kRGroup + row];
    const float m = fmaxf(m0, m1);
    const float c0 = m0 == -INFINITY ? 0.f : ex2f(m0 - m);
    const float c1 = m1 == -INFINITY ? 0.f : ex2f(m1 - m);
    const float lsum = l0 * c0 + l1 * c1;
    const float inv = kClusters && item.pieces > 1 ? 1.0f : lsum > 0.f ? 1.0f / lsum : 0.f;  // (pieces are merged as they are)
    if (kClusters && item.pieces > 1 && g == 0) {
      float* stats = reinterpret_cast<float*>(smem + L::stats);
      stats[row] = m;
      stats[kRGroup + row] = lsum;
    }
    // (the Q image is idle: every QK has completed)
    uint8_t* stage = qimg + warp * 4096;
    static_assert(8 * 4096 <= kQImageBytes, "room for every warp's rows");
    const RowsOut dst = rows_out(p, t, kvh, rows, row, split);
    if ((row & ~31) < rows) {
#pragma unroll 1
      for (int j = 2 * g; j < 2 * g + 2; ++j) {
        uint32_t r0[32], r1[32];
        tc::tmem_ld32(tmem_base + 256 + lane_addr + j * 32, r0);
        tc::tmem_ld32(tmem_base + 384 + lane_addr + j * 32, r1);
        tc::tmem_ld_wait<32>(r0);
        tc::tmem_landed<32>(r1);
        float o[32];
#pragma unroll
        for (int n = 0; n < 32; ++n) {
          const float o1 = c1 > 0.f ? __uint_as_float(r1[n]) * c1 : 0.f;
          o[n] = (__uint_as_float(r0[n]) * c0 + o1) * inv;
        }
        if (kClusters && item.pieces > 1) {
          park_row32<kRGroup>(reinterpret_cast<float*>(smem + L::park), j * 32, row, o);
        } else {
          write_rows32(dst, j * 32, stage, o);
        }
      }
    }
    if (g == 0 && row < rows && (!kClusters || item.pieces == 1) && (p.num_splits > 1 || p.lse_out != nullptr)) write_lse(p, t, kvh, row, split, lsum > 0.f ? m - kPGain + log2f(lsum) : -INFINITY);
  }

  if (kClusters && item.pieces > 1) {
    cluster_sync();
    if (warp < 8 && (tid & 127) < rows)
      merge_pieces<kRGroup, 2, kHeadDim>(p, t, kvh, tid & 127, tid >> 7, (int)(blockIdx.x & (uint32_t)(p.cluster - 1)), item.pieces,
                                         reinterpret_cast<const float*>(smem + L::park), reinterpret_cast<const float*>(smem + L::stats),
                                         reinterpret_cast<float*>(smem + L::raw));
    cluster_sync();  // (the others still read this CTA's rows)
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kRLoadWarp) tc::tmem_dealloc(tmem_base, 512);
  if (tid == 0 && *abort_flag) atomicOr(&g_rows_status, 4u);
  if (p.late_wait) pdl_wait();  // (TMEM is free by now: see late_wait)
  (void)ok;
}

}  // namespace

// The row-major kernel reads the cache like the integer kernel (packed cells through TMA
// page copies).
bool umma_rows_supports(const KernelParams& p, const char** why) {
  if (!umma_i8_supports(p, why)) return false;
  // (this file: 128 dims; 256 dims: umma_rows256_kernel.cu; 64 dims: umma_rows2_kernel.cu)
  return true;
}

namespace {
template <int NK, int NR>
cudaError_t launch_rows(const KernelParams& p, const CUtensorMap& map, cudaStream_t stream) {
  return launch_row_tiles<umma_rows_attention_kernel<NK, NR, false>, umma_rows_attention_kernel<NK, NR, true>>(p, map, kRThreads,
                                                                                                              RLayout<NK, NR>::total, stream);
}
}  // namespace

cudaError_t launch_umma_rows_attention(const KernelParams& p_in, cudaStream_t stream) {
  if (p_in.head_size == 256) return launch_umma_rows256_attention(p_in, stream);
  if (p_in.head_size == 64) return launch_umma_rows2_attention(p_in, stream);  // the only row-major kernel for 64 dims
  // Launches whose requests have 256 rows or more on average (prefill chunks) run two row tiles
  // per CTA, which share every widened K / V tile (umma_rows2_kernel.cu); shorter ones (wide
  // verification, drafter steps) would leave its second row tile empty.
  if ((int64_t)p_in.num_tokens * p_in.group >= 256 * (int64_t)p_in.num_reqs) return launch_umma_rows2_attention(p_in, stream);
  KernelParams p = p_in;
  // Row tiles of 128 rows, whatever tile height the caller planned with: the partition of
  // the query tokens into row tiles is internal to a launch.
  set_row_tile(p, 128 / p.group > 0 ? 128 / p.group : 1);
  set_copy_slots(p, kHalfKeys);  // a raw half stage holds whole page copies
  p.raw_mode = raw_mode_for(p);
  p.num_sms = sm_count();
  if (p.num_sms <= 0) return cudaErrorInvalidDevice;
  static const CUtensorMap no_map{};
  const CUtensorMap* mapp = &no_map;
  if (p.raw_mode == 1) {
    mapp = cached_page_map(p);
    if (mapp == nullptr) return cudaErrorInvalidValue;
  }
  const CUtensorMap& map = *mapp;
  // Two K images, so that a tile's keys are widened while the QK of the one in front reads its own, and three raw half
  // stages (64 keys each): all that fits beside them.
  return launch_rows<2, 3>(p, map, stream);
}

// Reads and clears this file's status word (device must be idle).
cudaError_t read_rows_status(unsigned int* v) {
  unsigned int zero = 0;
  cudaError_t err = cudaMemcpyFromSymbol(v, g_rows_status, sizeof(*v));
  if (err != cudaSuccess) return err;
  return cudaMemcpyToSymbol(g_rows_status, &zero, sizeof(zero));
}

}  // namespace pthb200


#include "umma_rows_tile_test.cuh"
