// Row-major tcgen05 attention kernel for head size 256: query rows on the MMA M dimension,
// KV tiles of 64 keys.
//
// The 128-dim row-major kernel (umma_rows_kernel.cu) does not stretch to 256 dims: its 16-bit K
// and V images of 128 keys would take 4 x 66 KB.  This kernel keeps the same roles and the
// same exact widening, with other shapes:
//   tile       128 query rows x 64 keys; the split partition stays in units of 128 keys, a
//              CTA walks its range in steps of 64;
//   TMEM       S0 S1 (64 columns each: tile i uses buffer i % 2, so S(i + 1) is computed while
//              the softmax warps work on tile i), ONE accumulator O of 256 columns, and Q (128
//              columns, two fp16 per column): Q is the A operand of QK from TMEM like P is of
//              PV, which takes its 64 KB image out of shared memory;
//   MMAs       S = Q K^T: M 128, N 64, sixteen steps of 16 dims; O += P V: M 128, N 256, four
//              steps of 16 keys;
//   producers  thread (key, half) of the K set / V set widens 128 of the key's 256 dims; the
//              K threads of the upper halves also publish the key's scales;
//   softmax    two groups of 4 warps; group g owns keys 32 g .. 32 g + 31 of EVERY tile and
//              columns 128 g .. 128 g + 127 of O.  The two threads of a row agree on the row's
//              reference maximum tile by tile (through shared memory and one named barrier), which
//              is what lets them share one accumulator; each rescales and finally writes its
//              half of the row's output.
// Raw ring: two units of 64 keys x 528 bytes.  Every mbarrier wait is bounded (page_copy.cuh).
#include <cuda.h>

#include <type_traits>

#include "params.cuh"
#include "sched.cuh"
#include "umma_rows.cuh"
#include "page_copy.cuh"
#include "pdl.cuh"

namespace pthb200 {

__device__ unsigned int g_rows256_status = 0;

namespace {

constexpr int kWDim = 256;                          // head size
constexpr int kWKeys = 64;                          // keys of a tile
constexpr int kWChunks = kWDim / 8;                 // 16-byte column blocks of a widened row: 8 fp16 each
constexpr int kWChunkStride = kWKeys * 16 + 16;     // 1,040 B: one column block of all keys, padded
constexpr int kWImage = kWChunks * kWChunkStride;   // 33,280 B: widened K or V of a tile
constexpr int kWRawRow = raw_row_for(kWDim);        // 528 B
constexpr int kWRawUnit = kWKeys * kWRawRow;        // 33,792 B: raw cells of a tile
constexpr int kWVStage = kWImage;                   // V image
constexpr int kWNK = 2, kWNS = 2, kWNR = 2;         // K images, V stages, raw units
constexpr int kWKsRing = 4;                         // tiles of key scales kept
constexpr int kWGroup = 128;                        // threads of one softmax group = rows of a tile
constexpr int kWSoftmax = 2 * kWGroup;              // warps 0-3, 4-7
constexpr int kWGroupKeys = kWKeys / 2;             // 32 keys of a tile per group
constexpr int kWGroupDims = kWDim / 2;              // 128 columns of O per group
constexpr int kWProducers = 256;                    // warps 8-11 (K set) and 12-15 (V set)
constexpr int kWMmaWarp = 16, kWLoadWarp = 17;
constexpr int kWThreads = 576;
constexpr int kWQBarrier = kWSoftmax + 32;  // Q in TMEM: softmax, MMA issuer
constexpr int kWProducerRegs = 64, kWSoftmaxRegs = 128;  // of the 96 per thread the CTA starts with
constexpr int kWSCol = 0, kWOCol = 128, kWQCol = 384;    // TMEM columns: S buffers at 0 and 64, O, Q
constexpr float kWRescaleGap = 4.0f;                // log2 units a row maximum may outgrow its reference

struct WLayout {
  static constexpr int kimg = 0;
  static constexpr int vst = kimg + kWNK * kWImage;
  static constexpr int raw = (vst + kWNS * kWVStage + 127) / 128 * 128;
  static constexpr int ksc = raw + kWNR * kWRawUnit;                 // KeyScales<64> [kWKsRing]
  static constexpr int tile_max = ksc + kWKsRing * (int)sizeof(KeyScales<kWKeys>);  // float [2 tiles][2 groups][128 rows]
  static constexpr int half_sum = tile_max + 2 * 2 * kWGroup * 4;    // float [2 groups][128 rows]
  static constexpr int qstage = half_sum + 2 * kWGroup * 4;          // [8 warps] 32 dims of 32 rows of Q
  static constexpr int stats = qstage + 8 * 2048;                    // float [2][128 rows], see merge_pieces
  static constexpr int bars = stats + 2 * kWGroup * 4;               // uint64 [...]
  static constexpr int park = kimg;                                  // the images, idle at the end: [256][128 rows] fp32
  static_assert(kWDim * kWGroup * 4 <= raw, "room for a parked accumulator");
  static constexpr int n_bars = kWNS * 2 + 2 * kWNK + 6 + 2 * kWNR;
  static constexpr int misc = bars + n_bars * 8;
  static constexpr int total = misc + 32 + 4 * kRowsItemInts;
};

struct WBars {
  static constexpr int vfull = 0;                      // [NS] V producers -> PV
  static constexpr int vempty = kWNS;                  // [NS] PV commit -> V producers
  static constexpr int kempty = 2 * kWNS;              // [NK] QK commit -> K producers
  static constexpr int kfull = 2 * kWNS + kWNK;        // [NK] K producers -> QK
  static constexpr int s_ready = 2 * kWNS + 2 * kWNK;  // [2] QK commit -> softmax
  static constexpr int p_ready = s_ready + 2;          // [2] softmax -> PV
  static constexpr int pv_done = p_ready + 2;          // [2] PV commit -> QK, softmax
  static constexpr int raw_full = pv_done + 2;         // [NR]
  static constexpr int raw_free = raw_full + kWNR;     // [NR] producers -> loader
};

// Key of a tile held by row `r` of its images: with contiguous cells the even keys, then the odd ones.
__device__ __forceinline__ int tile_key_w(int raw_mode, int r) { return raw_mode == 2 ? 2 * (r & 31) + (r >> 5) : r; }

// S(buffer) = Q K^T with Q in TMEM: 16 steps of 16 dims = two column blocks of the K image each.
__device__ __forceinline__ void issue_qk_w(uint32_t s_tmem, uint32_t q_tmem, RowsDesc k) {
  constexpr uint32_t idesc = tc::instr_desc(128, kWKeys, tc::kFmtF16, tc::kFmtF16, 0, 0);
  constexpr uint32_t step = (2 * kWChunkStride) >> 4;
#pragma unroll
  for (int kk = 0; kk < kWDim / 16; ++kk) mma_ts_words(s_tmem, q_tmem + kk * 8, k.lo + kk * step, k.hi, idesc, kk > 0);
}
// O += P V: P in two pieces (keys 0-31 in columns 0-15 of the S buffer, keys 32-63 in columns
// 32-47: each softmax group writes P over its own half of S), four steps of 16 keys.
__device__ __forceinline__ void issue_pv_w(uint32_t o_tmem, uint32_t s_tmem, RowsDesc v, bool accumulate) {
  constexpr uint32_t idesc = tc::instr_desc(128, kWDim, tc::kFmtF16, tc::kFmtF16, 0, 1);
#pragma unroll
  for (int g = 0; g < 2; ++g)
#pragma unroll
    for (int kk = 0; kk < kWGroupKeys / 16; ++kk)
      mma_ts_words(o_tmem, s_tmem + g * kWGroupKeys + kk * 8, v.lo + (g * (kWGroupKeys / 16) + kk) * (256 >> 4), v.hi, idesc,
                   accumulate || g > 0 || kk > 0);
}

template <bool kClusters>
__global__ void __launch_bounds__(kWThreads, 1)
umma_rows256_attention_kernel(const __grid_constant__ KernelParams p, const __grid_constant__ CUtensorMap tmap) {
  using L = WLayout;
  using B = WBars;
  static_assert(L::raw % 128 == 0 && kWRawUnit % 128 == 0 && (16 * kWRawRow) % 128 == 0, "TMA destinations");
  static_assert(L::vst % 16 == 0 && kWVStage % 16 == 0 && kWImage % 16 == 0, "image alignment");
  static_assert(L::total <= 227 * 1024, "shared memory of one CTA");
  extern __shared__ __align__(128) uint8_t smem[];
  float* tile_max = reinterpret_cast<float*>(smem + L::tile_max);
  float* half_sum = reinterpret_cast<float*>(smem + L::half_sum);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::bars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::misc);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + L::misc + 8);
  KeyScales<kWKeys>* key_scales = reinterpret_cast<KeyScales<kWKeys>*>(smem + L::ksc);

  int kvh, tile_index;
  rows_cta<kClusters>(p, &kvh, &tile_index);
  const int split = blockIdx.y;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // Barriers and TMEM are set up by the warps that wait for nothing else.  The CTA of a further piece of the bound, which
  // mostly finds that its request is not cut that often, takes TMEM when it has found work (see launch_row_tiles).
  const bool tmem_ahead = split == 0;
  if (warp == kWLoadWarp) {
    if (lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap)) : "memory");
    if (tmem_ahead) {
      tc::tmem_alloc(tslot, 512);
      tc::tmem_relinquish();
    }
  }
  if (warp == kWMmaWarp && lane == 0) {
    for (int s = 0; s < kWNS; ++s) {
      tc::mbar_init(&bars[B::vfull + s], kWProducers / 2);
      tc::mbar_init(&bars[B::vempty + s], 1);
    }
    for (int s = 0; s < kWNK; ++s) {
      tc::mbar_init(&bars[B::kempty + s], 1);
      tc::mbar_init(&bars[B::kfull + s], kWProducers / 2);
    }
    for (int g = 0; g < 2; ++g) {
      tc::mbar_init(&bars[B::s_ready + g], 1);
      tc::mbar_init(&bars[B::p_ready + g], kWSoftmax);
      tc::mbar_init(&bars[B::pv_done + g], 1);
    }
    for (int s = 0; s < kWNR; ++s) {
      tc::mbar_init(&bars[B::raw_full + s], kWKeys >> p.copy_shift);  // page copies of a unit
      tc::mbar_init(&bars[B::raw_free + s], kWProducers);             // every producer thread reads every unit
    }
    *abort_flag = 0;
    tc::mbar_init_fence();
  }
  if (!p.late_wait) pdl_wait();
  // Row tile of this CTA: warp 0 finds it; for longer lists of requests all threads bisect a shared-memory copy of
  // query_start_loc when it fits.
  constexpr int kQslCache = 4096;
  static_assert(kWNR * kWRawUnit >= 2 * kQslCache * 4, "the raw ring holds the copies of query_start_loc and seq_lens");
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
      for (int i = tid; i <= p.num_reqs; i += kWThreads) {
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
    item = rows_item<kClusters>(p, t, split, [&] { return cta_work<kWThreads>(p, smem + L::misc + 16); });
    if (tid == 0) *reinterpret_cast<RowsItem*>(item_s) = item;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  item = *reinterpret_cast<const RowsItem*>(item_s);
  if (item.state != 1 || (split == 0 && item.nsplits < p.num_splits)) write_empty<kWThreads, kWDim>(p, item, kvh, split);
  if (item.state != 1) {
    if (tmem_ahead && warp == kWLoadWarp) tc::tmem_dealloc(*tslot, 512);
    if (p.late_wait) pdl_wait();
    return;
  }
  if (!tmem_ahead) {
    if (warp == kWLoadWarp) {
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

  // the CTA walks its keys in tiles of 64: from the first 128-key tile of its piece to the end
  // of the keys its rows see (or of the piece)
  const int key_begin = tile_begin * 128;
  const int key_end = min(tile_end * 128, range_end);
  const int n_tiles = (key_end - key_begin + kWKeys - 1) / kWKeys;
  const uint32_t kimg_s = tc::smem_u32(smem + L::kimg), vst_s = tc::smem_u32(smem + L::vst);
  bool ok = true;

  if (warp >= 8 && warp < kWMmaWarp) {
    // =========================== producers ====================================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kWProducerRegs));
    // Warps 8-11 widen K, warps 12-15 V.  Thread pt of a set owns key pt % 64 and dims
    // 128 (pt / 64) .. + 127 of it: 128 bytes of the raw cell, which start 0 or 8 (K) or 4 or
    // 12 (V) bytes after a 16-byte boundary; the K threads of the upper halves find k_scale
    // right behind their bytes.
    const int pt = tid & 127;
    const bool v_part = warp >= 12;
    // Contiguous cells (raw_mode 2) alternate between the two 8-byte alignments: a warp takes
    // the even keys or the odd ones, so that it runs one instance of the widening below.  Row r
    // of the images (and of the scale vectors) then holds key tile_key_w(r): the order of the
    // keys inside a tile changes no sum, and the softmax masks by that key.
    const int img_row = pt & (kWKeys - 1), upper = pt >> 6;
    const int key = tile_key_w(p.raw_mode, img_row);
    const int bs = p.copy_slots;  // slots of one page copy
    const uint8_t* kb = p.k.data + (int64_t)kvh * p.k.stride_head;
    const uint32_t delta = (uint32_t)(reinterpret_cast<uintptr_t>(kb) & 15);
    const int row_pitch = p.raw_mode == 1 ? kWRawRow : 2 * kWDim + 8;
    const int my_page = key >> p.copy_shift, my_slot = key & (bs - 1);
    // first byte of this thread's 128 bytes inside a raw unit
    const uint32_t piece = my_page * bs * kWRawRow + my_slot * row_pitch + delta + (v_part ? kWDim + 4 : 0) + upper * 128;
    const int wo = (int)((piece & 15u) >> 2);  // first word of the piece in the 16-byte chunks read: 0 / 2 (K), 1 / 3 (V)
    const float score_mul = p.scale_log2 * query_ungain(p.q_dtype);
#pragma unroll 1
    for (int j = 0; j < n_tiles; ++j) {
      const int rs = j % kWNR;
      const int pos = key_begin + j * kWKeys + key;
      const bool valid = pos >= range_begin && pos < range_end;
      ok &= wait_or_abort(&bars[B::raw_full + rs], (j / kWNR) & 1, abort_flag);
      // nine 16-byte chunks from the boundary below the piece: its 32 words and the scale behind them
      uint32_t w[36];
      if (valid) {
        const uint4* row = reinterpret_cast<const uint4*>(smem + L::raw + rs * kWRawUnit + (piece & ~15u));
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
      // (the v_scale of the key, for the threads that publish its scales)
      float v_scale = 1.f;
      if (!v_part && upper && valid)
        v_scale = *reinterpret_cast<const float*>(smem + L::raw + rs * kWRawUnit + my_page * bs * kWRawRow + my_slot * row_pitch +
                                                  delta + 2 * kWDim + 4);
      mbar_arrive(&bars[B::raw_free + rs]);  // the bytes are in registers: the unit may be refilled
      uint8_t* dst;
      if (!v_part) {
        if (j >= kWNK) ok &= wait_or_abort(&bars[B::kempty + j % kWNK], ((j / kWNK) - 1) & 1, abort_flag);
        dst = smem + L::kimg + (j % kWNK) * kWImage;
      } else {
        if (j >= kWNS) ok &= wait_or_abort(&bars[B::vempty + j % kWNS], ((j / kWNS) - 1) & 1, abort_flag);
        dst = smem + L::vst + (j % kWNS) * kWVStage;
      }
      uint8_t* out16 = dst + (upper * 16) * kWChunkStride + img_row * 16;  // column blocks 16 upper .. 16 upper + 15
      uint32_t scale_bits;
      // (one instance per alignment: the words of w must be compile-time indices)
      auto widen_piece = [&](auto first_word) {
        constexpr int kW0 = decltype(first_word)::value;
#pragma unroll
        for (int c = 0; c < 16; ++c)
          *reinterpret_cast<uint4*>(out16 + c * kWChunkStride) = widen8_f16(make_uint2(w[kW0 + 2 * c], w[kW0 + 2 * c + 1]));
        scale_bits = w[kW0 + 32];
      };
      if (wo == 0) widen_piece(std::integral_constant<int, 0>{});
      else if (wo == 1) widen_piece(std::integral_constant<int, 1>{});
      else if (wo == 2) widen_piece(std::integral_constant<int, 2>{});
      else widen_piece(std::integral_constant<int, 3>{});
      if (upper && !v_part) {
        KeyScales<kWKeys>& ks = key_scales[j % kWKsRing];
        const float vs = usable_v_scale(v_scale);
        ks.score[img_row] = __uint_as_float(scale_bits) * score_mul;
        ks.lv[img_row] = __log2f(vs);
        ks.iv[img_row] = __fdividef(1.0f, vs);
      }
      tc::fence_async_smem();
      mbar_arrive(&bars[(v_part ? B::vfull + j % kWNS : B::kfull + j % kWNK)]);
    }
  } else if (warp == kWLoadWarp) {
    // =========================== loader =======================================
    // One TMA copy per run of copy_slots slots of a tile, issued by lane `copy`: a box of the
    // tensor map (raw_mode 1) or a bulk copy of a contiguous run of cells (raw_mode 2); the
    // next tile's block ids are fetched before waiting for the unit.
    const int copies = kWKeys >> p.copy_shift;
    if (lane < copies) {
      const int bs = p.copy_slots;
      const int32_t* bt = p.block_table + (int64_t)t.req * p.block_table_row_stride;
      const uint8_t* kb = p.k.data + (int64_t)kvh * p.k.stride_head;
      const uint32_t delta = (uint32_t)(reinterpret_cast<uintptr_t>(kb) & 15);
      const int tma_x = (int)((reinterpret_cast<uintptr_t>(kb) - delta -
                               (reinterpret_cast<uintptr_t>(p.k.data) & ~(uintptr_t)15)) >> 2);
      const uint32_t raw_s = tc::smem_u32(smem + L::raw);
      auto page_block = [&](int j) -> int {
        const int pos0 = key_begin + j * kWKeys + lane * bs;
        if (j >= n_tiles || pos0 >= range_end || pos0 + bs <= range_begin) return -1;
        int page, slot;
        page_and_slot(p, pos0, &page, &slot);
        return __ldg(bt + page);
      };
      auto first_slot = [&](int j) -> int {
        int page, slot;
        page_and_slot(p, key_begin + j * kWKeys + lane * bs, &page, &slot);
        return slot;
      };
      int blk = page_block(0);
#pragma unroll 1
      for (int j = 0; j < n_tiles; ++j) {
        const int blk_next = page_block(j + 1);
        const int rs = j % kWNR;
        if (j >= kWNR) ok &= wait_raw_free(&bars[B::raw_free + rs], ((j / kWNR) - 1) & 1, abort_flag);
        uint64_t* bar = &bars[B::raw_full + rs];
        if (blk >= 0 && ok) {
          const uint32_t dst = raw_s + rs * kWRawUnit + lane * bs * kWRawRow;
          if (p.raw_mode == 1) {
            mbar_arrive_expect_tx(bar, bs * kWRawRow);
            tma_load_3d(dst, &tmap, tma_x, first_slot(j), blk, bar);
          } else {
            const uint32_t bytes = bs * (2 * kWDim + 8);  // a multiple of 16, like the run's address
            mbar_arrive_expect_tx(bar, bytes);
            bulk_copy_g2s(dst, kb + (int64_t)blk * p.k.stride_block + (int64_t)first_slot(j) * (2 * kWDim + 8), bytes, bar);
          }
        } else {
          mbar_arrive(bar);
        }
        blk = blk_next;
      }
    }
  } else if (warp == kWMmaWarp) {
    // =========================== MMA issuer ===================================
    // ONE elected lane issues every tcgen05.mma of the CTA in one fixed order: QK(0), QK(1),
    // then PV(i), QK(i + 2).  QK(i + 2) overwrites the S buffer P(i) was written over: it
    // waits for PV(i) to have finished reading it, a whole tile of softmax after it is issued.
    named_barrier(5, kWQBarrier);  // wait for Q in TMEM
    tc::fence_after_sync();
    {
      const RowsDesc kd = rows_desc(kimg_s, kWChunkStride, 128);
      const RowsDesc vd = rows_desc(vst_s, 128, kWChunkStride);
      auto issue_qk = [&](int q) {
        ok &= wait_or_abort(&bars[B::kfull + q % kWNK], (q / kWNK) & 1, abort_flag);
        if (ok && elect_one()) {
          tc::fence_after_sync();
          RowsDesc k = kd;
          k.lo += (uint32_t)(q % kWNK) * (kWImage >> 4);
          issue_qk_w(tmem_base + kWSCol + (q & 1) * kWKeys, tmem_base + kWQCol, k);
          tc::mma_commit(&bars[B::s_ready + (q & 1)]);
          tc::mma_commit(&bars[B::kempty + q % kWNK]);
        }
        __syncwarp();
      };
      issue_qk(0);
      if (n_tiles > 1) issue_qk(1);
#pragma unroll 1
      for (int i = 0; i < n_tiles && ok; ++i) {
        const int sb = i & 1;
        ok &= wait_or_abort(&bars[B::p_ready + sb], (i >> 1) & 1, abort_flag);
        ok &= wait_or_abort(&bars[B::vfull + i % kWNS], (i / kWNS) & 1, abort_flag);
        if (ok && elect_one()) {
          tc::fence_after_sync();
          RowsDesc v = vd;
          v.lo += (uint32_t)(i % kWNS) * (kWVStage >> 4);
          issue_pv_w(tmem_base + kWOCol, tmem_base + kWSCol + sb * kWKeys, v, i > 0);
          tc::mma_commit(&bars[B::pv_done + sb]);
          tc::mma_commit(&bars[B::vempty + i % kWNS]);
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
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kWSoftmaxRegs));
    const int g = warp >> 2;
    const int row = tid & 127;   // row of the tile = TMEM lane
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_part = tmem_base + kWSCol + g * kWGroupKeys + lane_addr;   // this group's columns of S buffer 0
    const uint32_t o_part = tmem_base + kWOCol + g * kWGroupDims + lane_addr;   // this group's columns of O

    // ---- Q into TMEM: dims 128 g .. 128 g + 127 of a row through the thread of the row, two fp16 per column.  A warp
    // loads its 32 rows 64 bytes at a time, four lanes a row, and hands them to their threads 32 dims after 32 dims
    // through 2 KB of shared memory.  (Each thread loading its own row: see stage_queries.) ----
    float q_fix = 1.0f;  // what the row's scores are multiplied by (QueryScale)
    {
      const int row0 = row & ~31, c = lane & 3;
      const uint8_t* mine = p.q + row_offset(t, kvh, p.group, 1.0f / (float)p.group, min(row, rows - 1), p.q_stride_token, p.q_stride_head);
      uint8_t* stage = smem + L::qstage + warp * 2048;
      uint4 qv[4][4];  // [32 dims][8 rows]
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int n = row0 + 8 * k + (lane >> 2);
        const uint4* src = reinterpret_cast<const uint4*>(shfl_ptr(mine, 8 * k + (lane >> 2))) + g * (kWGroupDims / 8) + c;
#pragma unroll
        for (int d = 0; d < 4; ++d) qv[d][k] = n < rows ? __ldg(src + 4 * d) : make_uint4(0u, 0u, 0u, 0u);
      }
      if (p.q_dtype == PTH_ATTN_BF16) {
        uint32_t* part = reinterpret_cast<uint32_t*>(tile_max);  // [2 groups][128 rows] (idle until the first tile)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint4 mine[4] = {qv[0][k], qv[1][k], qv[2][k], qv[3][k]};
          uint32_t amax = finite_amax_bf16(mine);
          amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
          amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
          if (c == 0) part[g * kWGroup + row0 + 8 * k + (lane >> 2)] = amax;
        }
        named_barrier(4, kWSoftmax);
        q_fix = query_scale(max(part[row], part[kWGroup + row])).fix;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int n = row0 + 8 * k + (lane >> 2);
          const float scale = query_scale(max(part[n], part[kWGroup + n])).scale;
#pragma unroll
          for (int d = 0; d < 4; ++d) qv[d][k] = queries_to_f16(qv[d][k], scale);
        }
      }
#pragma unroll
      for (int d = 0; d < 4; ++d) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int r = 8 * k + (lane >> 2);
          *reinterpret_cast<uint4*>(stage + r * 64 + ((c ^ ((r >> 1) & 3)) << 4)) = qv[d][k];
        }
        __syncwarp();
        uint32_t qw[16];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint4 v = *reinterpret_cast<const uint4*>(stage + lane * 64 + ((e ^ ((lane >> 1) & 3)) << 4));
          qw[4 * e] = v.x;
          qw[4 * e + 1] = v.y;
          qw[4 * e + 2] = v.z;
          qw[4 * e + 3] = v.w;
        }
        tc::tmem_st16(tmem_base + kWQCol + g * (kWGroupDims / 2) + d * 16 + lane_addr, qw);
        __syncwarp();
      }
      tc::tmem_st_wait();
    }
    tc::fence_before_sync();
    named_barrier(5, kWQBarrier);  // Q complete; the QK issuer may start

    int rlo = 0, rhi = -1;  // visible keys of this row (none for a padding row)
    if (row < rows) visible_range(p, t, t.first_idx + row / p.group, &rlo, &rhi);
    int mask_lo, mask_hi, tmp;  // key positions every live row sees: such tiles need no mask
    visible_range(p, t, t.first_idx + t.ntok - 1, &mask_lo, &tmp);
    visible_range(p, t, t.first_idx, &tmp, &mask_hi);
    float m_ref = -INFINITY;  // reference maximum of the row's exponentials (log2 units)
    float l = 0.f;            // 2^kPGain times the sum of exp2(score - m_ref) over this group's keys, without v_scale
    auto walk_tiles = [&](auto own_power) {  // (one instance for warps without a row of its own power of two)
      constexpr bool kOwnPower = decltype(own_power)::value;
#pragma unroll 1
    for (int i = 0; i < n_tiles; ++i) {
      const KeyScales<kWKeys>& ks = key_scales[i % kWKsRing];
      const uint32_t s_tmem = s_part + (i & 1) * kWKeys;
      const int pos0 = key_begin + i * kWKeys;
      const bool interior = pos0 >= mask_lo && pos0 + (kWKeys - 1) <= mask_hi;
      ok &= wait_or_abort(&bars[B::s_ready + (i & 1)], (i >> 1) & 1, abort_flag);
      tc::fence_after_sync();
      uint32_t r[kWGroupKeys];  // the scores of this row and part, read once
      tc::tmem_ld32(s_tmem, r);
      tc::tmem_ld_wait<kWGroupKeys>(r);
      if constexpr (kOwnPower) scale_scores<kWGroupKeys>(r, q_fix);

      // ---- pass 1: weighted scores in log2 units (kept in the registers) and their maximum ----
      auto all_ready = [] {};
      const int k0 = g * kWGroupKeys;
      float m_t = interior ? softmax_pass1<kWGroupKeys, false>(r, ks.score + k0, ks.lv + k0, all_ready, [](int) { return true; })
                           : softmax_pass1<kWGroupKeys, true>(r, ks.score + k0, ks.lv + k0, all_ready, [&](int n) {
                               const int pos = pos0 + tile_key_w(p.raw_mode, k0 + n);  // key held by this column
                               return pos >= rlo && pos <= rhi;
                             });
      // ---- the row's maximum over the whole tile: the other group has the other keys ----
      float* tm = tile_max + (i & 1) * 2 * kWGroup + row;
      tm[g * kWGroup] = m_t;
      named_barrier(4, kWSoftmax);
      m_t = fmaxf(m_t, tm[(g ^ 1) * kWGroup]);
      // ---- move the reference maximum if the row has outgrown it (both threads of a row decide alike) ----
      const float m_new = fmaxf(m_ref, m_t);
      const bool need = m_t > m_ref + kWRescaleGap;  // also true when m_ref is still -inf
      if (i == 0) {
        m_ref = m_new;  // nothing accumulated yet
      } else if (__any_sync(0xffffffffu, need)) {
        // O must be at rest: the PV of the previous tile has completed
        ok &= wait_or_abort(&bars[B::pv_done + ((i - 1) & 1)], ((i - 1) >> 1) & 1, abort_flag);
        tc::fence_after_sync();
        const float alpha = need ? ex2f(m_ref - m_new) : 1.0f;  // 0 when m_ref was -inf
#pragma unroll 1
        for (int j = 0; j < kWGroupDims / 16; ++j) {
          uint32_t o[16];
          tc::tmem_ld16(o_part + j * 16, o);
          tc::tmem_ld_wait<16>(o);
#pragma unroll
          for (int n = 0; n < 16; ++n) o[n] = __float_as_uint(__uint_as_float(o[n]) * alpha);
          tc::tmem_st16(o_part + j * 16, o);
        }
        tc::tmem_st_wait();
        l *= alpha;
        if (need) m_ref = m_new;
      }
      const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref - kPGain;

      // ---- pass 2: P as packed fp16 over the first columns of this part of S ----
      f32x2 ls[2] = {0ull, 0ull};
      uint32_t pk[16];
      softmax_pass2(r, ks.iv + k0, m_use, ls, pk);
      tc::tmem_st16(s_tmem, pk);
      l += sum_pairs(ls);
      tc::tmem_st_wait();
      tc::fence_before_sync();
      mbar_arrive(&bars[B::p_ready + (i & 1)]);  // this group's part of P(i) is complete
    }
    };
    if (__any_sync(0xffffffffu, q_fix != 1.0f)) walk_tiles(std::true_type{}); else walk_tiles(std::false_type{});

    // ---- epilogue: the row's sum is the two groups' sums; each group writes its half of the dims ----
    // (the commit after the last PV covers every MMA issued before it)
    ok &= wait_or_abort(&bars[B::pv_done + ((n_tiles - 1) & 1)], ((n_tiles - 1) >> 1) & 1, abort_flag);
    tc::fence_after_sync();
    half_sum[g * kWGroup + row] = l;
    named_barrier(4, kWSoftmax);
    const float lsum = half_sum[row] + half_sum[kWGroup + row];  // the same order in both threads
    const float inv = lsum > 0.f ? 1.0f / lsum : 0.f;
    // (the K images are idle: every QK has completed)
    uint8_t* stage = smem + L::kimg + warp * 4096;
    static_assert(8 * 4096 <= kWNK * kWImage, "room for every warp's rows");
    if (kClusters && item.pieces > 1) {
      // (both groups are behind the barrier of the sums, so every MMA is done with the images)
      float* stats = reinterpret_cast<float*>(smem + L::stats);
      float* park = reinterpret_cast<float*>(smem + L::park);
      if (g == 0) {
        stats[row] = m_ref;
        stats[kWGroup + row] = lsum;
      }
      if ((row & ~31) < rows) {
#pragma unroll 1
        for (int j = 0; j < kWGroupDims / 32; ++j) {
          float o[32];
          tc::tmem_ld32(o_part + j * 32, reinterpret_cast<uint32_t*>(o));
          tc::tmem_ld_wait<32>(reinterpret_cast<uint32_t*>(o));
          park_row32<kWGroup>(park, g * kWGroupDims + j * 32, row, o);
        }
      }
    } else {
    const RowsOut dst = rows_out(p, t, kvh, rows, row, split);
    if ((row & ~31) < rows) {
#pragma unroll 1
      for (int j = 0; j < kWGroupDims / 32; ++j) {
        uint32_t r[32];
        tc::tmem_ld32(o_part + j * 32, r);
        tc::tmem_ld_wait<32>(r);
        float o[32];
#pragma unroll
        for (int n = 0; n < 32; ++n) o[n] = __uint_as_float(r[n]) * inv;
        write_rows32(dst, g * kWGroupDims + j * 32, stage, o);
      }
    }
    if (g == 0 && row < rows && (p.num_splits > 1 || p.lse_out != nullptr)) write_lse(p, t, kvh, row, split, lsum > 0.f ? m_ref - kPGain + log2f(lsum) : -INFINITY);
    }
  }

  if (kClusters && item.pieces > 1) {
    cluster_sync();
    if (warp < 8 && (tid & 127) < rows)
      merge_pieces<kWGroup, 2, kWDim>(p, t, kvh, tid & 127, tid >> 7, (int)(blockIdx.x & (uint32_t)(p.cluster - 1)), item.pieces,
                                      reinterpret_cast<const float*>(smem + L::park), reinterpret_cast<const float*>(smem + L::stats),
                                      reinterpret_cast<float*>(smem + L::raw));
    cluster_sync();  // (the others still read this CTA's rows)
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kWLoadWarp) tc::tmem_dealloc(tmem_base, 512);
  if (tid == 0 && *abort_flag) atomicOr(&g_rows256_status, 4u);
  if (p.late_wait) pdl_wait();  // (TMEM is free by now: see late_wait)
  (void)ok;
}

}  // namespace

cudaError_t launch_umma_rows256_attention(const KernelParams& p_in, cudaStream_t stream) {
  KernelParams p = p_in;
  // Row tiles of 128 rows, whatever tile height the caller planned with.
  set_row_tile(p, 128 / p.group > 0 ? 128 / p.group : 1);
  set_copy_slots(p, kWKeys);  // a raw unit (64 keys) holds whole page copies
  p.raw_mode = raw_mode_for(p);
  p.num_sms = sm_count();
  if (p.num_sms <= 0) return cudaErrorInvalidDevice;
  static const CUtensorMap no_map{};
  const CUtensorMap* mapp = &no_map;
  if (p.raw_mode == 1) {
    mapp = cached_page_map(p);
    if (mapp == nullptr) return cudaErrorInvalidValue;
  }
  return launch_row_tiles<umma_rows256_attention_kernel<false>, umma_rows256_attention_kernel<true>>(p, *mapp, kWThreads, WLayout::total, stream);
}

// Reads and clears this kernel's status word (device must be idle).
cudaError_t read_rows256_status(unsigned int* v) {
  unsigned int zero = 0;
  cudaError_t err = cudaMemcpyFromSymbol(v, g_rows256_status, sizeof(*v));
  if (err != cudaSuccess) return err;
  return cudaMemcpyToSymbol(g_rows256_status, &zero, sizeof(zero));
}

}  // namespace pthb200
