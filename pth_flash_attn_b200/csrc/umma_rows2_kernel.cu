// Row-major tcgen05 attention kernel, head sizes 128 and 64, TWO row tiles per CTA: 256 query rows
// share every widened K / V tile.  (The shapes below are those of 128 dims; at 64 dims the images,
// the accumulators and the contraction steps over the head are half as large.)
//
// In the one-tile kernel (umma_rows_kernel.cu) every row tile of 128 rows widens the int8 keys
// and values of its whole context for itself, and that widening and the shared-memory
// traffic around it - not the tensor core, not the softmax - take most of a tile's time.
// Here a CTA owns 256 rows (two MMA row tiles) and 64-key tiles:
//   TMEM       S(rt, b): 64 columns for row tile rt and buffer b = tile % 2 (256 columns), O(rt):
//              128 columns each (256 columns);
//   MMAs       per KV tile two QK (M 128, N 64, eight steps of 16 dims, Q images in shared
//              memory) on ONE K image and two PV (M 128, N 128, four steps of 16 keys, P from
//              TMEM) on ONE V stage;
//   producers  thread (key, half) of the K set / V set widens 64 of the key's 128 dims to fp16;
//              the K set's upper halves carry both scales of the key to the softmax;
//   softmax    256 threads, one per row: the row's maximum, sum and reference never leave the
//              thread, and there is nothing to merge at the end.
// What bounds it: the softmax's instructions (4.75 per score) and the MMAs they overlap with.  2 x 2,048 tokens
// over 14,336 keys, 64 query heads: 2,175 us; of an earlier 2,268 the kernel without MMAs took 2,004, without
// softmax and widening 1,906.  A tile's MMAs take 637 cycles per row tile (QK 400: both operands in shared
// memory, 6 KB per 32 cycles; PV 272), its softmax about 2,000.
// Raw ring: four units of 64 keys x 272 bytes.  Every mbarrier wait is bounded (page_copy.cuh).
#include <cuda.h>

#include <type_traits>

#include "params.cuh"
#include "sched.cuh"
#include "umma_rows.cuh"
#include "page_copy.cuh"
#include "pdl.cuh"

namespace pthb200 {

__device__ unsigned int g_rows2_status = 0;

namespace {

constexpr int kXKeys = 64;                          // keys of a tile
constexpr int kXRows = 256;                         // rows of a CTA: two MMA row tiles
constexpr int kXChunkStride = kXKeys * 16 + 16;     // 1,040 B: one column block of all keys, padded
constexpr int kXQStride = 128 * 16 + 16;            // 2,064 B: one column block of the 128 rows of a Q image
// Sizes that follow the head size HD (figures for 128).
template <int HD>
struct XG {
  static_assert(HD == 64 || HD == 128, "head size");
  static constexpr int chunks = HD / 8;                    // 16-byte column blocks of a widened row: 8 fp16 each
  static constexpr int image = chunks * kXChunkStride;     // 16,640 B: widened K or V of a tile
  static constexpr int qimage = chunks * kXQStride;        // 33,024 B
  static constexpr int raw_row = raw_row_for(HD);          // 272 B
  static constexpr int raw_unit = kXKeys * raw_row;        // 17,408 B: raw cells of a tile
  static constexpr int piece = HD / 2;                     // bytes of a key a producer thread widens
  static constexpr int piece_chunks = piece / 8;           // column blocks it writes
  static constexpr int load_chunks = piece / 16 + 1;       // 16-byte chunks it reads: the piece, its misalignment, the scale
};
constexpr int kXNK = 2, kXNS = 2, kXNR = 4;         // K images, V stages, raw units
constexpr int kXKsRing = 4;                         // tiles of key scales kept
constexpr int kXSoftmax = 256;                      // warps 0-3 (row tile 0), 4-7 (row tile 1)
constexpr int kXProducers = 256;                    // warps 8-11 (K set) and 12-15 (V set)
constexpr int kXMmaWarp = 16, kXLoadWarp = 17;
constexpr int kXThreads = 576;
constexpr int kXQBarrier = kXSoftmax + 32;  // Q images complete: softmax, MMA issuer
// Registers per thread, of the 96 the CTA starts with.  The softmax, which bounds the kernel by its instructions,
// keeps more of a tile's scales in flight with 136 than with 120; a producer's words fit 56 but for a few.  (Against
// 128 and 64: 4 x 2,048 tokens over 14,336 keys at 64 dims 2,052 us and 2,085; at 128 dims 4 x 2,048 over 30,720
// 9,606 and 9,652, 2 x 1,000 new tokens 54.3 and 55.2, twelve prompts of 37 to 2,500 430 and 434.)
constexpr int kXProducerRegs = 56, kXSoftmaxRegs = 136;
constexpr int kXOCol = 256;                         // TMEM columns: S(rt, b) at (2 rt + b) 64, O(rt) at 256 + 128 rt
constexpr float kXRescaleGap = 4.0f;                // log2 units a row maximum may outgrow its reference (P stays at or below 2^15)

template <int HD>
struct XLayout {
  using G = XG<HD>;
  static constexpr int kimg = 0;
  static constexpr int vst = kimg + kXNK * G::image;
  static constexpr int qimg = vst + kXNS * G::image;                 // [2 row tiles] Q images
  static constexpr int raw = (qimg + 2 * G::qimage + 127) / 128 * 128;
  static constexpr int ksc = raw + kXNR * G::raw_unit;               // KeyScales<64> [kXKsRing]
  static constexpr int fix = ksc + kXKsRing * (int)sizeof(KeyScales<kXKeys>);   // float [256 rows], see QueryScale
  static constexpr int stats = fix + kXRows * 4;                                 // float [2][256 rows], see merge_pieces
  static constexpr int bars = stats + 2 * kXRows * 4;                            // uint64 [...]
  static constexpr int park = kimg;                                              // the images, idle at the end: [HD][256 rows] fp32
  static_assert(HD * kXRows * 4 <= raw, "room for a parked accumulator");
  static_assert(kClusterMax * kXRows * 4 <= kXNR * G::raw_unit, "room for the weights of the pieces, in the idle ring");
  static constexpr int n_bars = 2 * kXNS + 2 * kXNK + 12 + 2 * kXNR;
  static constexpr int misc = bars + n_bars * 8;
  static constexpr int total = misc + 32 + 4 * kRowsItemInts;
};

struct XBars {
  static constexpr int vfull = 0;                      // [NS] V producers -> PV
  static constexpr int vempty = kXNS;                  // [NS] PV commit -> V producers
  static constexpr int kempty = 2 * kXNS;              // [NK] QK commit -> K producers
  static constexpr int kfull = 2 * kXNS + kXNK;        // [NK] K producers -> QK
  static constexpr int s_ready = 2 * kXNS + 2 * kXNK;  // [2 rt][2 b] QK commit -> softmax
  static constexpr int p_ready = s_ready + 4;          // [2 rt][2 b] softmax -> PV
  static constexpr int pv_done = p_ready + 4;          // [2 rt][2 b] PV commit -> QK, softmax
  static constexpr int raw_full = pv_done + 4;         // [NR]
  static constexpr int raw_free = raw_full + kXNR;     // [NR] producers -> loader
};

// Key of a tile held by row `r` of its images: with contiguous cells the even keys, then the odd ones.
__device__ __forceinline__ int tile_key_x(int raw_mode, int r) { return raw_mode == 2 ? 2 * (r & 31) + (r >> 5) : r; }

// S = Q K^T for one row tile: HD / 16 steps of 16 dims = two column blocks of either image each.
template <int HD>
__device__ __forceinline__ void issue_qk_x(uint32_t s_tmem, RowsDesc q, RowsDesc k) {
  constexpr uint32_t idesc = tc::instr_desc(128, kXKeys, tc::kFmtF16, tc::kFmtF16, 0, 0);
  constexpr uint32_t qstep = (2 * kXQStride) >> 4, kstep = (2 * kXChunkStride) >> 4;
  mma_ss_words<false>(s_tmem, q.lo, q.hi, k.lo, k.hi, idesc);
#pragma unroll
  for (int kk = 1; kk < HD / 16; ++kk) mma_ss_words<true>(s_tmem, q.lo + kk * qstep, q.hi, k.lo + kk * kstep, k.hi, idesc);
}
// O += P V for one row tile: P (64 keys, two fp16 per column) in the first 32 columns of its S buffer.
template <int HD>
__device__ __forceinline__ void issue_pv_x(uint32_t o_tmem, uint32_t p_tmem, RowsDesc v, bool accumulate) {
  constexpr uint32_t idesc = tc::instr_desc(128, HD, tc::kFmtF16, tc::kFmtF16, 0, 1);
#pragma unroll
  for (int kk = 0; kk < kXKeys / 16; ++kk) mma_ts_words(o_tmem, p_tmem + kk * 8, v.lo + kk * (256 >> 4), v.hi, idesc, accumulate || kk > 0);
}

template <int HD, bool kClusters>
__global__ void __launch_bounds__(kXThreads, 1)
umma_rows2_attention_kernel(const __grid_constant__ KernelParams p, const __grid_constant__ CUtensorMap tmap) {
  using L = XLayout<HD>;
  using B = XBars;
  using G = XG<HD>;
  constexpr int kXDim = HD, kXImage = G::image, kXVStage = G::image, kXQImage = G::qimage;
  constexpr int kXRawRow = G::raw_row, kXRawUnit = G::raw_unit;
  static_assert(L::raw % 128 == 0 && kXRawUnit % 128 == 0 && (16 * kXRawRow) % 128 == 0, "TMA destinations");
  static_assert(L::vst % 16 == 0 && kXVStage % 16 == 0 && kXImage % 16 == 0 && L::qimg % 16 == 0 && kXQImage % 16 == 0,
                "image alignment");
  static_assert(L::bars % 8 == 0, "mbarriers");
  static_assert(L::total <= 227 * 1024, "shared memory of one CTA");
  extern __shared__ __align__(128) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::bars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::misc);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + L::misc + 8);
  KeyScales<kXKeys>* key_scales = reinterpret_cast<KeyScales<kXKeys>*>(smem + L::ksc);

  int kvh, tile_index;
  rows_cta<kClusters>(p, &kvh, &tile_index);
  const int split = blockIdx.y;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // Barriers and TMEM are set up by the warps that wait for nothing else.  The CTA of a further piece of the bound, which
  // mostly finds that its request is not cut that often, takes TMEM when it has found work (see launch_row_tiles).
  const bool tmem_ahead = split == 0;
  if (warp == kXLoadWarp) {
    if (lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap)) : "memory");
    if (tmem_ahead) {
      tc::tmem_alloc(tslot, 512);
      tc::tmem_relinquish();
    }
  }
  if (warp == kXMmaWarp && lane == 0) {
    for (int s = 0; s < kXNS; ++s) {
      tc::mbar_init(&bars[B::vfull + s], kXProducers / 2);
      tc::mbar_init(&bars[B::vempty + s], 2);  // one commit per row tile's PV
    }
    for (int s = 0; s < kXNK; ++s) {
      tc::mbar_init(&bars[B::kempty + s], 2);  // one commit per row tile's QK
      tc::mbar_init(&bars[B::kfull + s], kXProducers / 2);
    }
    for (int g = 0; g < 4; ++g) {
      tc::mbar_init(&bars[B::s_ready + g], 1);
      tc::mbar_init(&bars[B::p_ready + g], 128);  // the threads of one row tile
      tc::mbar_init(&bars[B::pv_done + g], 1);
    }
    for (int s = 0; s < kXNR; ++s) {
      tc::mbar_init(&bars[B::raw_full + s], kXKeys >> p.copy_shift);  // page copies of a unit
      tc::mbar_init(&bars[B::raw_free + s], kXProducers);             // every producer thread reads every unit
    }
    *abort_flag = 0;
    tc::mbar_init_fence();
  }
  if (!p.late_wait) pdl_wait();
  // Row tile of this CTA: warp 0 finds it; for longer lists of requests all threads bisect a shared-memory copy of
  // query_start_loc when it fits.
  constexpr int kQslCache = 4096;
  static_assert(kXNR * kXRawUnit >= 2 * kQslCache * 4, "the raw ring holds the copies of query_start_loc and seq_lens");
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
      for (int i = tid; i <= p.num_reqs; i += kXThreads) {
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
    item = rows_item<kClusters>(p, t, split, [&] { return cta_work<kXThreads>(p, smem + L::misc + 16); });
    if (tid == 0) *reinterpret_cast<RowsItem*>(item_s) = item;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  item = *reinterpret_cast<const RowsItem*>(item_s);
  if (item.state != 1 || (split == 0 && item.nsplits < p.num_splits)) write_empty<kXThreads, HD>(p, item, kvh, split);
  if (item.state != 1) {
    if (tmem_ahead && warp == kXLoadWarp) tc::tmem_dealloc(*tslot, 512);
    if (p.late_wait) pdl_wait();
    return;
  }
  if (!tmem_ahead) {
    if (warp == kXLoadWarp) {
      tc::tmem_alloc(tslot, 512);
      tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
  }
  const uint32_t tmem_base = *tslot;
  const RowTile& t = item.t;
  const int rows = item.rows;  // <= 256 by construction of bq
  const int tile_begin = item.tile_begin, tile_end = item.tile_end, range_begin = item.range_begin, range_end = item.range_end;

  // the CTA walks its keys in tiles of 64: from the first 128-key tile of its piece to the end
  // of the keys its rows see (or of the piece)
  const int key_begin = tile_begin * 128;
  const int key_end = min(tile_end * 128, range_end);
  const int n_tiles = (key_end - key_begin + kXKeys - 1) / kXKeys;
  // Row tiles with live rows: a CTA of at most 128 rows (the end of a chunk, a short request
  // inside a prefill launch) issues no MMA for its second row tile, whose softmax warps idle.
  const int n_rt = rows > 128 ? 2 : 1;
  const uint32_t kimg_s = tc::smem_u32(smem + L::kimg), vst_s = tc::smem_u32(smem + L::vst);
  bool ok = true;

  if (warp >= 8 && warp < kXMmaWarp) {
    // =========================== producers ====================================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kXProducerRegs));
    // Warps 8-11 widen K, warps 12-15 V.  Thread pt of a set owns row pt % 64 of the images and
    // half of its key's dims (the lower or the upper): HD / 2 bytes of the raw cell, which start 0 or 8 (K) or
    // 4 or 12 (V) bytes after a 16-byte boundary; the K threads of the upper halves find k_scale
    // right behind their bytes.  Contiguous cells (raw_mode 2) alternate between the two
    // 8-byte alignments: a warp takes the even keys or the odd ones (one widening path per warp),
    // so the images hold a tile's even keys, then its odd ones; the softmax masks by that key.
    const int pt = tid & 127;
    const bool v_part = warp >= 12;
    const int img_row = pt & (kXKeys - 1), upper = pt >> 6;
    const int key = tile_key_x(p.raw_mode, img_row);
    const int bs = p.copy_slots;  // slots of one page copy
    const uint8_t* kb = p.k.data + (int64_t)kvh * p.k.stride_head;
    const uint32_t delta = (uint32_t)(reinterpret_cast<uintptr_t>(kb) & 15);
    const int row_pitch = p.raw_mode == 1 ? kXRawRow : 2 * kXDim + 8;
    const int my_page = key >> p.copy_shift, my_slot = key & (bs - 1);
    // first byte of this thread's bytes inside a raw unit
    const uint32_t piece = my_page * bs * kXRawRow + my_slot * row_pitch + delta + (v_part ? kXDim + 4 : 0) + upper * G::piece;
    const int wo = (int)((piece & 15u) >> 2);  // first word of the piece in the 16-byte chunks read: 0 / 2 (K), 1 / 3 (V)
    const float score_mul = p.scale_log2 * query_ungain(p.q_dtype);
#pragma unroll 1
    for (int j = 0; j < n_tiles; ++j) {
      const int rs = j % kXNR;
      const int pos = key_begin + j * kXKeys + key;
      const bool valid = pos >= range_begin && pos < range_end;
      ok &= wait_or_abort(&bars[B::raw_full + rs], (j / kXNR) & 1, abort_flag);
      // the 16-byte chunks from the boundary below the piece: its words and the scale behind them
      uint32_t w[4 * G::load_chunks];
      if (valid) {
        const uint4* row = reinterpret_cast<const uint4*>(smem + L::raw + rs * kXRawUnit + (piece & ~15u));
#pragma unroll
        for (int c = 0; c < G::load_chunks; ++c) {
          const uint4 v = row[c];
          w[4 * c] = v.x;
          w[4 * c + 1] = v.y;
          w[4 * c + 2] = v.z;
          w[4 * c + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int c = 0; c < 4 * G::load_chunks; ++c) w[c] = 0u;
      }
      // (the v_scale of the key, for the threads that publish its scales)
      float v_scale = 1.f;
      if (!v_part && upper && valid)
        v_scale = *reinterpret_cast<const float*>(smem + L::raw + rs * kXRawUnit + my_page * bs * kXRawRow + my_slot * row_pitch +
                                                  delta + 2 * kXDim + 4);
      mbar_arrive(&bars[B::raw_free + rs]);  // the bytes are in registers: the unit may be refilled
      uint8_t* dst;
      if (!v_part) {
        if (j >= kXNK) ok &= wait_or_abort(&bars[B::kempty + j % kXNK], ((j / kXNK) - 1) & 1, abort_flag);
        dst = smem + L::kimg + (j % kXNK) * kXImage;
      } else {
        if (j >= kXNS) ok &= wait_or_abort(&bars[B::vempty + j % kXNS], ((j / kXNS) - 1) & 1, abort_flag);
        dst = smem + L::vst + (j % kXNS) * kXVStage;
      }
      uint8_t* out16 = dst + (upper * G::piece_chunks) * kXChunkStride + img_row * 16;  // this half's column blocks
      uint32_t scale_bits;
      // (one instance per alignment: the words of w must be compile-time indices)
      auto widen_piece = [&](auto first_word) {
        constexpr int kW0 = decltype(first_word)::value;
#pragma unroll
        for (int c = 0; c < G::piece_chunks; ++c) {
          *reinterpret_cast<uint4*>(out16 + c * kXChunkStride) = widen8_f16(make_uint2(w[kW0 + 2 * c], w[kW0 + 2 * c + 1]));
        }
        scale_bits = w[kW0 + G::piece / 4];
      };
      if (wo == 0) widen_piece(std::integral_constant<int, 0>{});
      else if (wo == 1) widen_piece(std::integral_constant<int, 1>{});
      else if (wo == 2) widen_piece(std::integral_constant<int, 2>{});
      else widen_piece(std::integral_constant<int, 3>{});
      if (upper && !v_part) {
        KeyScales<kXKeys>& ks = key_scales[j % kXKsRing];
        const float vs = usable_v_scale(v_scale);
        ks.score[img_row] = __uint_as_float(scale_bits) * score_mul;
        ks.lv[img_row] = __log2f(vs);
        ks.iv[img_row] = __fdividef(1.0f, vs);
      }
      tc::fence_async_smem();
      mbar_arrive(&bars[(v_part ? B::vfull + j % kXNS : B::kfull + j % kXNK)]);
    }
  } else if (warp == kXLoadWarp) {
    // =========================== loader =======================================
    // One TMA copy per run of copy_slots slots of a tile, issued by lane `copy`: a box of the
    // tensor map (raw_mode 1) or a bulk copy of a contiguous run of cells (raw_mode 2); the
    // next tile's block ids are fetched before waiting for the unit.
    const int copies = kXKeys >> p.copy_shift;
    if (lane < copies) {
      const int bs = p.copy_slots;
      const int32_t* bt = p.block_table + (int64_t)t.req * p.block_table_row_stride;
      const uint8_t* kb = p.k.data + (int64_t)kvh * p.k.stride_head;
      const uint32_t delta = (uint32_t)(reinterpret_cast<uintptr_t>(kb) & 15);
      const int tma_x = (int)((reinterpret_cast<uintptr_t>(kb) - delta -
                               (reinterpret_cast<uintptr_t>(p.k.data) & ~(uintptr_t)15)) >> 2);
      const uint32_t raw_s = tc::smem_u32(smem + L::raw);
      auto page_block = [&](int j) -> int {
        const int pos0 = key_begin + j * kXKeys + lane * bs;
        if (j >= n_tiles || pos0 >= range_end || pos0 + bs <= range_begin) return -1;
        int page, slot;
        page_and_slot(p, pos0, &page, &slot);
        return __ldg(bt + page);
      };
      auto first_slot = [&](int j) -> int {
        int page, slot;
        page_and_slot(p, key_begin + j * kXKeys + lane * bs, &page, &slot);
        return slot;
      };
      int blk = page_block(0);
#pragma unroll 1
      for (int j = 0; j < n_tiles; ++j) {
        const int blk_next = page_block(j + 1);
        const int rs = j % kXNR;
        if (j >= kXNR) ok &= wait_raw_free(&bars[B::raw_free + rs], ((j / kXNR) - 1) & 1, abort_flag);
        uint64_t* bar = &bars[B::raw_full + rs];
        if (blk >= 0 && ok) {
          const uint32_t dst = raw_s + rs * kXRawUnit + lane * bs * kXRawRow;
          if (p.raw_mode == 1) {
            mbar_arrive_expect_tx(bar, bs * kXRawRow);
            tma_load_3d(dst, &tmap, tma_x, first_slot(j), blk, bar);
          } else {
            const uint32_t bytes = bs * (2 * kXDim + 8);  // a multiple of 16, like the run's address
            mbar_arrive_expect_tx(bar, bytes);
            bulk_copy_g2s(dst, kb + (int64_t)blk * p.k.stride_block + (int64_t)first_slot(j) * (2 * kXDim + 8), bytes, bar);
          }
        } else {
          mbar_arrive(bar);
        }
        blk = blk_next;
      }
    }
  } else if (warp == kXMmaWarp) {
    // =========================== MMA issuer ===================================
    // ONE elected lane issues every tcgen05.mma of the CTA in one fixed order: the QK pairs of
    // tiles 0 and 1, then for every tile i the two PV(i) and the two QK(i + 2).  Row tile rt's
    // QK(i + 2) overwrites the S buffer its P(i) was written over: it waits for its PV(i) to have
    // finished reading it, a whole tile of softmax after it is issued.
    named_barrier(5, kXQBarrier);  // wait for the Q images
    // (one instance per number of live row tiles: the loops over them unroll as constants)
    auto issue_all = [&](auto live_row_tiles) {
      constexpr int kRowTiles = decltype(live_row_tiles)::value;
      const RowsDesc qd = rows_desc(tc::smem_u32(smem + L::qimg), kXQStride, 128);
      const RowsDesc kd = rows_desc(kimg_s, kXChunkStride, 128);
      const RowsDesc vd = rows_desc(vst_s, 128, kXChunkStride);
      // both row tiles' QK of tile q; after_pv: each first waits for its row tile's PV of tile q - 2
      auto issue_qk_pair = [&](int q, bool after_pv) {
        const int b = q & 1;
        ok &= wait_or_abort(&bars[B::kfull + q % kXNK], (q / kXNK) & 1, abort_flag);
#pragma unroll
        for (int rt = 0; rt < kRowTiles; ++rt) {
          if (after_pv) ok &= wait_or_abort(&bars[B::pv_done + 2 * rt + b], ((q - 2) >> 1) & 1, abort_flag);
          if (ok && elect_one()) {
            tc::fence_after_sync();
            RowsDesc k = kd, qq = qd;
            k.lo += (uint32_t)(q % kXNK) * (kXImage >> 4);
            qq.lo += (uint32_t)rt * (kXQImage >> 4);
            issue_qk_x<HD>(tmem_base + (2 * rt + b) * kXKeys, qq, k);
            tc::mma_commit(&bars[B::s_ready + 2 * rt + b]);
            tc::mma_commit(&bars[B::kempty + q % kXNK]);  // (free once both row tiles' QK have read the K image)
            if constexpr (kRowTiles == 1) tc::mma_commit(&bars[B::kempty + q % kXNK]);
          }
          __syncwarp();
        }
      };
      issue_qk_pair(0, false);
      if (n_tiles > 1) issue_qk_pair(1, false);
#pragma unroll 1
      for (int i = 0; i < n_tiles && ok; ++i) {
        const int b = i & 1;
        ok &= wait_or_abort(&bars[B::vfull + i % kXNS], (i / kXNS) & 1, abort_flag);
#pragma unroll
        for (int rt = 0; rt < kRowTiles; ++rt) {
          ok &= wait_or_abort(&bars[B::p_ready + 2 * rt + b], (i >> 1) & 1, abort_flag);
          if (ok && elect_one()) {
            tc::fence_after_sync();
            RowsDesc v = vd;
            v.lo += (uint32_t)(i % kXNS) * (kXVStage >> 4);
            issue_pv_x<HD>(tmem_base + kXOCol + rt * kXDim, tmem_base + (2 * rt + b) * kXKeys, v, i > 0);
            tc::mma_commit(&bars[B::pv_done + 2 * rt + b]);
            tc::mma_commit(&bars[B::vempty + i % kXNS]);  // (free once both row tiles' PV have read the V stage)
            if constexpr (kRowTiles == 1) tc::mma_commit(&bars[B::vempty + i % kXNS]);
          }
          __syncwarp();
        }
        if (i + 2 < n_tiles) issue_qk_pair(i + 2, true);
      }
    };
    if (n_rt == 2) issue_all(std::integral_constant<int, 2>{}); else issue_all(std::integral_constant<int, 1>{});
  } else if (warp < 8) {
    // =========================== softmax ======================================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kXSoftmaxRegs));
    const int rt = warp >> 2;            // row tile of this thread
    const int row = tid;                 // row of the CTA's 256 (TMEM lane tid % 128 of row tile rt)
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_rt = tmem_base + 2 * rt * kXKeys + lane_addr;          // S(rt, 0)
    const uint32_t o_tmem = tmem_base + kXOCol + rt * kXDim + lane_addr;    // O(rt)

    // ---- Q image of this row tile: a warp converts the 32 rows of its threads ----
    float* fix_s = reinterpret_cast<float*>(smem + L::fix);
    {
      uint8_t* qimg = smem + L::qimg + rt * kXQImage;
      stage_queries<HD, 32>(p, t, kvh, rows, row & ~31,
          [&](int n, int block, const uint4& v) { *reinterpret_cast<uint4*>(qimg + block * kXQStride + (n & 127) * 16) = v; },
          [&](int n, float fix) { fix_s[n] = fix; });
    }
    tc::fence_async_smem();
    named_barrier(5, kXQBarrier);  // Q images complete; the QK issuer may start
    const float q_fix = fix_s[row];  // what the row's scores are multiplied by (QueryScale)

    int rlo = 0, rhi = -1;  // visible keys of this row (none for a padding row)
    if (row < rows) visible_range(p, t, t.first_idx + row / p.group, &rlo, &rhi);
    int mask_lo, mask_hi, tmp;  // key positions every live row sees: such tiles need no mask
    visible_range(p, t, t.first_idx + t.ntok - 1, &mask_lo, &tmp);
    visible_range(p, t, t.first_idx, &tmp, &mask_hi);
    float m_ref = -INFINITY;  // reference maximum of the row's exponentials (log2 units)
    float l = 0.f;            // 2^kPGain times the sum of exp2(score - m_ref), without v_scale
    // A warp whose 32 rows are all padding (the last row tile of a chunk, a short request inside
    // a prefill launch) leaves the issue slots to the others; its rows end as rows without keys
    // (m = -inf, l = 0), which the epilogue never writes.
    // (Their loop is a separate one: the live warps' loop carries no trace of the case.)  A row
    // tile without any live row is never computed: its warps wait for nothing.
    if ((row & ~31) >= rows) {
      if (rt < n_rt) {
#pragma unroll 1
        for (int i = 0; i < n_tiles; ++i) {
          // the arrival keeps the barrier's count and, behind the wait, its phase: S(rt, i + 2) is
          // not ready before P(rt, i) has been used
          ok &= wait_or_abort(&bars[B::s_ready + 2 * rt + (i & 1)], (i >> 1) & 1, abort_flag);
          mbar_arrive(&bars[B::p_ready + 2 * rt + (i & 1)]);
        }
      }
    } else {  // warps with live rows (the loop keeps its indentation)
    auto walk_tiles = [&](auto own_power) {  // (one instance for warps without a row of its own power of two)
      constexpr bool kOwnPower = decltype(own_power)::value;
#pragma unroll 1
    for (int i = 0; i < n_tiles; ++i) {
      const int b = i & 1;
      const KeyScales<kXKeys>& ks = key_scales[i % kXKsRing];
      const uint32_t s_tmem = s_rt + b * kXKeys;
      const int pos0 = key_begin + i * kXKeys;
      const bool interior = pos0 >= mask_lo && pos0 + (kXKeys - 1) <= mask_hi;
      ok &= wait_or_abort(&bars[B::s_ready + 2 * rt + b], (i >> 1) & 1, abort_flag);
      tc::fence_after_sync();
      uint32_t r[kXKeys];  // the row's scores of this tile, read once: the second half arrives while
      tc::tmem_ld32(s_tmem, r);  // pass 1 works on the first
      tc::tmem_ld_wait<32>(r);
      tc::tmem_ld32(s_tmem + 32, r + 32);
      if constexpr (kOwnPower) scale_scores<32>(r, q_fix);

      // ---- pass 1: weighted scores in log2 units (kept in the registers) and their maximum ----
      auto half_ready = [&] {
        tc::tmem_ld_wait<32>(r + 32);
        if constexpr (kOwnPower) scale_scores<32>(r + 32, q_fix);
      };
      const float m_t =
          interior ? softmax_pass1<kXKeys, false>(r, ks.score, ks.lv, half_ready, [](int) { return true; })
                   : softmax_pass1<kXKeys, true>(r, ks.score, ks.lv, half_ready, [&](int n) {
                       const int pos = pos0 + tile_key_x(p.raw_mode, n);  // key held by this column
                       return pos >= rlo && pos <= rhi;
                     });
      // ---- move the reference maximum if the row has outgrown it ----
      const float m_new = fmaxf(m_ref, m_t);
      const bool need = m_t > m_ref + kXRescaleGap;  // also true when m_ref is still -inf
      if (i == 0) {
        m_ref = m_new;  // nothing accumulated yet
      } else if (__any_sync(0xffffffffu, need)) {
        // O(rt) must be at rest: this row tile's PV of the previous tile has completed
        ok &= wait_or_abort(&bars[B::pv_done + 2 * rt + ((i - 1) & 1)], ((i - 1) >> 1) & 1, abort_flag);
        tc::fence_after_sync();
        const float alpha = need ? ex2f(m_ref - m_new) : 1.0f;  // 0 when m_ref was -inf
#pragma unroll 1
        for (int j = 0; j < kXDim / 16; ++j) {
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

      // ---- pass 2: P as packed fp16 over the first 32 columns of S ----
      f32x2 ls[2] = {0ull, 0ull};
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint32_t pk[16];
        softmax_pass2(r + j * 32, ks.iv + j * 32, m_use, ls, pk);
        tc::tmem_st16(s_tmem + j * 16, pk);
      }
      l += sum_pairs(ls);
      tc::tmem_st_wait();
      tc::fence_before_sync();
      mbar_arrive(&bars[B::p_ready + 2 * rt + b]);  // P(rt, i) is complete
    }
    };
    if (__any_sync(0xffffffffu, q_fix != 1.0f)) walk_tiles(std::true_type{}); else walk_tiles(std::false_type{});
    }  // warps with live rows

    // ---- epilogue: the row's output (the commit after the last PV covers every MMA issued before it) ----
    if (rt < n_rt) ok &= wait_or_abort(&bars[B::pv_done + 2 * rt + ((n_tiles - 1) & 1)], ((n_tiles - 1) >> 1) & 1, abort_flag);
    tc::fence_after_sync();
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    // (the Q image of this row tile is idle: every QK that reads it has completed)
    uint8_t* stage = smem + L::qimg + rt * kXQImage + (warp & 3) * 4096;
    if (kClusters && item.pieces > 1) {
      float* stats = reinterpret_cast<float*>(smem + L::stats);
      float* park = reinterpret_cast<float*>(smem + L::park);
      named_barrier(4, kXSoftmax);  // (both row tiles' MMAs are done with the images)
      stats[row] = m_ref;
      stats[kXRows + row] = l;
      if ((row & ~31) < rows) {
#pragma unroll 1
        for (int j = 0; j < kXDim / 32; ++j) {
          float o[32];
          tc::tmem_ld32(o_tmem + j * 32, reinterpret_cast<uint32_t*>(o));
          tc::tmem_ld_wait<32>(reinterpret_cast<uint32_t*>(o));
          park_row32<kXRows>(park, j * 32, row, o);
        }
      }
    } else {
    const RowsOut dst = rows_out(p, t, kvh, rows, row, split);
    if ((row & ~31) < rows) {
#pragma unroll 1
      for (int j = 0; j < kXDim / 32; ++j) {
        uint32_t r[32];
        tc::tmem_ld32(o_tmem + j * 32, r);
        tc::tmem_ld_wait<32>(r);
        float o[32];
#pragma unroll
        for (int n = 0; n < 32; ++n) o[n] = __uint_as_float(r[n]) * inv;
        write_rows32(dst, j * 32, stage, o);
      }
    }
    if (row < rows && (p.num_splits > 1 || p.lse_out != nullptr)) write_lse(p, t, kvh, row, split, l > 0.f ? m_ref - kPGain + log2f(l) : -INFINITY);
    }
  }

  if (kClusters && item.pieces > 1) {
    cluster_sync();
    if (warp < 8 && tid < rows)
      merge_pieces<kXRows, 1, HD>(p, t, kvh, tid, 0, (int)(blockIdx.x & (uint32_t)(p.cluster - 1)), item.pieces,
                                  reinterpret_cast<const float*>(smem + L::park), reinterpret_cast<const float*>(smem + L::stats),
                                  reinterpret_cast<float*>(smem + L::raw));
    cluster_sync();  // (the others still read this CTA's rows)
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kXLoadWarp) tc::tmem_dealloc(tmem_base, 512);
  if (tid == 0 && *abort_flag) atomicOr(&g_rows2_status, 4u);
  if (p.late_wait) pdl_wait();  // (TMEM is free by now: see late_wait)
  (void)ok;
}

}  // namespace

namespace {
template <int HD>
cudaError_t launch_rows2(const KernelParams& p, const CUtensorMap& map, cudaStream_t stream) {
  return launch_row_tiles<umma_rows2_attention_kernel<HD, false>, umma_rows2_attention_kernel<HD, true>>(p, map, kXThreads, XLayout<HD>::total, stream);
}
}  // namespace

cudaError_t launch_umma_rows2_attention(const KernelParams& p_in, cudaStream_t stream) {
  KernelParams p = p_in;
  // Row tiles of 256 rows, whatever tile height the caller planned with.
  set_row_tile(p, kXRows / p.group > 0 ? kXRows / p.group : 1);
  set_copy_slots(p, kXKeys);  // a raw unit (64 keys) holds whole page copies
  p.raw_mode = raw_mode_for(p);
  p.num_sms = sm_count();
  if (p.num_sms <= 0) return cudaErrorInvalidDevice;
  static const CUtensorMap no_map{};
  const CUtensorMap* mapp = &no_map;
  if (p.raw_mode == 1) {
    mapp = cached_page_map(p);
    if (mapp == nullptr) return cudaErrorInvalidValue;
  }
  return p.head_size == 64 ? launch_rows2<64>(p, *mapp, stream) : launch_rows2<128>(p, *mapp, stream);
}

// Reads and clears this kernel's status word (device must be idle).
cudaError_t read_rows2_status(unsigned int* v) {
  unsigned int zero = 0;
  cudaError_t err = cudaMemcpyFromSymbol(v, g_rows2_status, sizeof(*v));
  if (err != cudaSuccess) return err;
  return cudaMemcpyToSymbol(g_rows2_status, &zero, sizeof(zero));
}

}  // namespace pthb200
