// Building blocks of the row-major tcgen05 attention kernels (query rows on the MMA M
// dimension, as a prefill or a wide verification step wants them).
//
//   S[row, key] = sum_d   Q[row, d] * K[key, d]     A = Q image (K-major), B = K tile (K-major)
//   O[row, d]  += sum_key P[row, key] * V[key, d]   A = P in TMEM,         B = V tile (MN-major)
//
// K and V tiles are widened images (chunk c of 8 d, key t at c * kChunkStride + t * 16), which
// serve as B operands unchanged: for K (N = keys, K-major) LBO = chunk stride, SBO = 128; for V
// (N = d, MN-major) LBO = 128 (next 8 keys), SBO = chunk stride (next 8 d).  The Q image has the
// same form with rows in place of keys.  P never touches shared memory: the softmax thread of a
// row writes its probabilities as packed pairs into TMEM (lane = row, 32-bit column j = keys
// 2j, 2j + 1) and the PV MMA reads its A operand from there.
//
// Every operand is fp16, whatever the queries are (both operands of an MMA have one format):
//   K, V   int8 is exact in fp16, and its widening costs 1.25 instructions per value; to bf16,
//          whose 8 bits hold no biased int8, it takes 2;
//   Q      fp16 as it is; bf16 times a power of two that depends on the row alone: 2^7 where the row's
//          largest finite value is in [2^-4, 2^8), and the keys' score factor takes that back, else the one
//          that puts it into [2^14, 2^15), and the row's scores are multiplied by the rest (one
//          more multiplication per score, for warps that hold such a row).  A value is exact down to
//          2^-17 (2^-20 of the row's largest, 2^-31 of it with a power of its own) and off by
//          2^-25 (2^-28 of the largest) at most below.  (One power for the whole CTA let a huge query of one
//          row take the others' bits, and the keys' scales had to wait for it: one bf16 prompt of 100 tokens
//          took 24.3 us against 21.3, two of 1,000 59.5 against 55.1; long chunks, whose loop now has two
//          instances, 2 x 2,048 tokens over 14,336 keys 2,375 against 2,402.)
//   P      2^11 exp2(score + log2(v_scale) - reference): the key's v_scale sits in the exponent, so
//          V needs no multiplication and fp16's range is that of one row, not of the cache.  A
//          weighted score exceeds its reference by at most 4, so P stays at or below 2^15, and
//          with the factor of 2^11 P keeps eight bits (bf16's) down to 2^-28 of the reference and is off by at
//          most 2^-36 of it below: a long context whose mass sits in many small probabilities beside
//          one large one keeps it.  (A reference that scores may exceed by 8, with four bits less below, measured
//          the same within 0.5 %: 3,574 us at 256 dims, 10.21 against 10.26 ms at 128.)  The row
//          sum takes P / v_scale back in fp32.
// Measured against bf16 operands (same launches, one box): 4 x 2,048 tokens over 30,720 keys 10.05 -> 9.80 ms,
// at 256 dims 4.43 -> 3.6 ms, a drafter step 126.5 -> 117.9 us; fp16 queries, which bf16 operands could not
// take, leave the integer kernel's 64-row instance: twelve prompts of 37 to 2,500 tokens 5,754 -> 453 us.
#pragma once

#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "params.cuh"
#include "pdl.cuh"
#include "sched.cuh"
#include "umma_tile.cuh"

namespace pthb200 {

constexpr int kRowsPerTile = 128;                       // MMA M
constexpr int kQImageBytes = kChunks * kChunkStride;    // 33,024 B

namespace tc {

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

}  // namespace tc

// ---- MMA chains, for an issuing thread that keeps its descriptors in registers ----
// (low word = start address in 16-byte units: moving an operand by `bytes` adds bytes / 16)
struct RowsDesc {
  uint32_t lo, hi;
};
__device__ __forceinline__ RowsDesc rows_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  const uint64_t d = tc::smem_desc(saddr, lbo_bytes, sbo_bytes);
  return RowsDesc{(uint32_t)d, (uint32_t)(d >> 32)};
}
template <bool kAccumulate>
__device__ __forceinline__ void mma_ss_words(uint32_t d_tmem, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi,
                                             uint32_t idesc) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc), "n"(kAccumulate ? 1 : 0)
      : "memory");
}
__device__ __forceinline__ void mma_ts_words(uint32_t d_tmem, uint32_t a_tmem, uint32_t blo, uint32_t bhi, uint32_t idesc,
                                             bool accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 db;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "r"(blo), "r"(bhi), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}
// q = rows_desc(Q image, kChunkStride, 128), k = rows_desc(K image, kChunkStride, 128)
__device__ __forceinline__ void issue_qk_rows_words(uint32_t s_tmem, RowsDesc q, RowsDesc k) {
  constexpr uint32_t idesc = tc::instr_desc(kRowsPerTile, kTileKeys, tc::kFmtF16, tc::kFmtF16, 0, 0);
  constexpr uint32_t step = (2 * kChunkStride) >> 4;
  mma_ss_words<false>(s_tmem, q.lo, q.hi, k.lo, k.hi, idesc);
#pragma unroll
  for (int kk = 1; kk < kHeadDim / 16; ++kk)
    mma_ss_words<true>(s_tmem, q.lo + kk * step, q.hi, k.lo + kk * step, k.hi, idesc);
}
// v = rows_desc(V image, 128, kChunkStride).  PV of one tile as two chains: keys 0-63 (P columns 0-31 of the S buffer, V rows 0-63) into the
// accumulator at o_tmem, keys 64-127 (P columns 64-95, V rows 64-127) into the one at o_tmem + 128.
__device__ __forceinline__ void issue_pv_halves_words(uint32_t o_tmem, uint32_t s_tmem, RowsDesc v, bool accumulate) {
  constexpr uint32_t idesc = tc::instr_desc(kRowsPerTile, kHeadDim, tc::kFmtF16, tc::kFmtF16, 0, 1);
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int kk = 0; kk < kTileKeys / 32; ++kk)
      mma_ts_words(o_tmem + h * 128, s_tmem + h * 64 + kk * 8, v.lo + (h * 4 + kk) * (256 >> 4), v.hi, idesc,
                   accumulate || kk > 0);
}

// 4 int8 (one 32-bit word) -> 4 fp16, exactly: with the sign bit flipped a byte is x + 128, the
// fp16 bit pattern 0x6400 | (x + 128) is the integer 1152 + x.
__device__ __forceinline__ void widen4_f16(uint32_t w, uint32_t& out01, uint32_t& out23) {
  const uint32_t b = w ^ 0x80808080u;
  const uint32_t a01 = __byte_perm(b, 0x64646464u, 0x5140);
  const uint32_t a23 = __byte_perm(b, 0x64646464u, 0x7362);
  const __half2 off = __half2half2(__ushort_as_half(0x6480));  // 1152
  const __half2 r01 = __hsub2(*reinterpret_cast<const __half2*>(&a01), off);
  const __half2 r23 = __hsub2(*reinterpret_cast<const __half2*>(&a23), off);
  out01 = *reinterpret_cast<const uint32_t*>(&r01);
  out23 = *reinterpret_cast<const uint32_t*>(&r23);
}
__device__ __forceinline__ uint4 widen8_f16(uint2 raw) {
  uint4 r;
  widen4_f16(raw.x, r.x, r.y);
  widen4_f16(raw.y, r.z, r.w);
  return r;
}
__device__ __forceinline__ uint32_t pack_f16(float a, float b) {
  const __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// KV head and row tile of a CTA: the heads of a row tile side by side, the last row tile of the launch first.
// CTAs start in index order and one fits an SM, so what starts last decides how long the SMs wait for one
// another: under a causal mask those are then the first tiles of the first request, its shortest.  (Row tiles
// in ascending order, head by head: twelve new prompts of 37 to 2,500 tokens ended on the longest tiles of the
// last of them.)
template <bool kClusters>
__device__ __forceinline__ void rows_cta(const KernelParams& p, int* kvh, int* tile_index) {
  const uint32_t x = kClusters ? blockIdx.x >> (__ffs(p.cluster) - 1) : blockIdx.x;
  const uint32_t t = x / (uint32_t)p.num_kv_heads;
  *kvh = (int)(x - t * (uint32_t)p.num_kv_heads);
  *tile_index = p.num_q_tiles - 1 - (int)t;
}

// Row tile x of a padded tile grid (tile_map 0), found by one warp among up to kWarpRequests requests, 32 at a
// time, while others set barriers and TMEM up; its result goes to all threads through shared memory behind the barrier
// that ends the set-up.  (Not from every warp's own shuffles: the compiler then takes the length of the tile loops
// for one per lane, which costs them 4 %.)  *work: the lane's part of the launch's KV tiles per head, if they are wanted.
// (What a CTA does once costs by its instructions, which come from beyond the instruction caches at about ten cycles
// each: so loops stay rolled here, in stage_queries and in write_rows32.  Twelve new prompts of 37 to 2,500 tokens, CTAs of
// a handful of tiles: 425 us with all requests copied to shared memory and bisected by everybody behind two barriers, every
// thread loading and storing its own row of queries and results, 350 with these; with the same unrolled 498.)
constexpr int kWarpRequests = 96;
__device__ __forceinline__ RowTile warp_row_tile(const KernelParams& p, int x, bool want_work, const SchedShape& shape, unsigned long long* work) {
  const int lane = threadIdx.x & 31;
  int owner = 0, q0 = 0, q1 = 0, len = 0;  // the last request whose first tile is not behind x
#pragma unroll 1
  for (int base = 0; base < p.num_reqs; base += 32) {
    const int r = base + lane;
    int a = 0, b = 0, c = 0;
    if (r < p.num_reqs) {
      a = __ldg(p.query_start_loc + r);
      b = __ldg(p.query_start_loc + r + 1);
      c = __ldg(p.seq_lens + r);
    }
    const uint32_t before = __ballot_sync(0xffffffffu, r < p.num_reqs && a / p.bq + r <= x);
    if (before != 0u) {  // (consecutive lanes from 0 on)
      const int src = __popc(before) - 1;
      owner = base + src;
      q0 = __shfl_sync(0xffffffffu, a, src);
      q1 = __shfl_sync(0xffffffffu, b, src);
      len = __shfl_sync(0xffffffffu, c, src);
    } else if (!want_work) {
      break;
    }
    if (want_work && r < p.num_reqs)
      *work += (unsigned long long)req_row_tiles(shape, b - a) * (unsigned long long)req_kv_tiles(shape, b - a, c);
  }
  return finish_row_tile(p, x, owner, q0, q1, len);
}
__device__ __forceinline__ SchedShape sched_shape(const KernelParams& p) {
  SchedShape shape;
  shape.group = p.group;
  shape.num_kv_heads = p.num_kv_heads;
  shape.bq = p.bq;
  shape.num_splits = p.num_splits;
  shape.window = p.window;
  shape.causal = p.causal;
  shape.row_class = p.row_class;
  shape.class_rows = p.class_rows;
  return shape;
}

// ---- clusters ----
// A launch of few row tiles (a chunk or a prompt, few KV heads) leaves SMs idle, and its caller need not have reserved a
// workspace for pieces.  Then the CTAs of a cluster take a row tile together: each walks a run of its keys, leaves maximum,
// sum and accumulator of every row in its shared memory, and then merges and writes a slice of the columns, reading the
// others' through distributed shared memory.  The host takes the largest cluster with which the launch still is one round
// of the SMs (instances of their own: the cluster's code in the others cost twelve short prompts 1.5 %); the CTAs share a
// row tile of 8 tiles of 128 keys or more, at least two tiles each, and those that are not needed leave.  (The host knows the
// lengths no better than the block table's rows: a prompt of 16 tokens takes 9.2 us with a table cut to it, 10.3 with one of
// 131,072 keys a row, whose clusters then have nothing to share.)
// What bounds it: the walk of a piece, then 3 to 4 us for the merge, which reads 128 KB per CTA (at pieces of one tile it
// cost more than it gave: 200 tokens without a cache 17.7 us in two pieces, 13.4 in one).  One CTA per row tile / clusters:
// 200 tokens over 30,000 keys, 1 KV head 569 / 58 us, 8 KV heads over 8,000 162 / 57; 300 over 3,000 at 256 dims 65 / 35,
// two of them at 64 dims, 2 KV heads 68 / 31; 2,000 over 2,000, 1 KV head 86 / 54; 16 over 1,000 17.5 / 14.2.
constexpr int kClusterMax = 16;
__host__ __device__ constexpr int cluster_pieces(int tiles, int cluster) {
  int n = 1;
  while (tiles >= 8 && 2 * n <= cluster && 4 * n <= tiles) n *= 2;
  return n;
}
// (An SM takes one CTA, and the SMs of a cluster come from one group of them: how many of a size fit at once is asked.)
template <auto kKernel>
int clusters_at_once(int size, int threads, int smem) {
  static std::atomic<int> known[64][5];  // by device and log2(size): clusters + 1
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::atomic<int>* slot = dev >= 0 && dev < 64 ? &known[dev][size == 2 ? 1 : size == 4 ? 2 : size == 8 ? 3 : 4] : nullptr;
  if (slot != nullptr && slot->load(std::memory_order_relaxed) != 0) return slot->load(std::memory_order_relaxed) - 1;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)size;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)size);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if ((size > 8 && cudaFuncSetAttribute(kKernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
      cudaOccupancyMaxActiveClusters(&n, kKernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  if (slot != nullptr) slot->store(n + 1, std::memory_order_relaxed);
  return n;
}
inline int64_t tiles_bound(const KernelParams& p) {
  return row_tile_bound(p.block_table_row_stride, p.block_size, p.window, p.causal, p.bq);
}
template <auto kKernel>
int cluster_for(const KernelParams& p, int threads, int smem) {
  if (p.num_splits > 1) return 1;
  const int64_t row_tiles = (int64_t)p.num_q_tiles * p.num_kv_heads;
  const int most = cluster_pieces((int)tiles_bound(p), kClusterMax);
  int c = 1;
  while (2 * c <= most && 2 * c * row_tiles <= p.num_sms && row_tiles <= clusters_at_once<kKernel>(2 * c, threads, smem)) c *= 2;
  return c;
}
// One CTA (kKernel) or one cluster of CTAs (kClustered) per row tile, KV head and piece.
template <auto kKernel, auto kClustered>
cudaError_t launch_row_tiles(const KernelParams& p_in, const CUtensorMap& map, int threads, int smem, cudaStream_t stream) {
  static bool configured[64] = {};
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    err = cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err == cudaSuccess) err = cudaFuncSetAttribute(kClustered, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err != cudaSuccess) return err;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  KernelParams p = p_in;
  p.cluster = last_row_cluster = cluster_for<kClustered>(p, threads, smem);
  const int64_t ctas = (int64_t)p.num_q_tiles * p.num_kv_heads * p.cluster;
  if (ctas > 0x7fffffff) return cudaErrorInvalidConfiguration;
  // Pieces that no request of these lengths is cut into get no CTA (one that finds nothing to do still takes an SM for 1.4 us).
  // That holds as far as the block table is cut to the lengths; an engine's table of the longest context says less.  14 requests
  // of 8 tokens over 2,000 keys at 64 dims, 85 pieces at most: 68 us with a table of 2,000 keys a row, 158 with one of 131,072;
  // 20 of 6 over 1,000, 2 KV heads 19 and 37.  (Those with the wide table while every CTA summed the launch's work up before it
  // asked whether its request has that many pieces 213 and 51, with TMEM taken by every CTA besides 220 and 53.)
  const dim3 grid((unsigned)ctas, (unsigned)pieces_bound(tiles_bound(p), p.num_splits));
  if (p.cluster > 1) return pdl_launch_clusters(p.cluster, kClustered, grid, threads, smem, stream, p, map);
  return pdl_launch(kKernel, grid, threads, smem, stream, p, map);
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_address(uint32_t saddr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
// (between two cluster_sync: nobody writes what is read, so these may be moved among one another)
__device__ __forceinline__ float peer_load(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ float4 peer_load4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
// Columns d0 .. d0 + 31 of row `tile_row` of an accumulator into park: [dim / 4][kRows][4] fp32.
template <int kRows>
__device__ __forceinline__ void park_row32(float* park, int d0, int tile_row, const float (&o)[32]) {
#pragma unroll
  for (int c = 0; c < 8; ++c)
    *reinterpret_cast<float4*>(park + ((d0 / 4 + c) * kRows + tile_row) * 4) = make_float4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
}

// What a CTA computes: the keys of one piece of a row tile.
struct RowsItem {
  RowTile t;
  int rows, nsplits;
  int tile_begin, tile_end, range_begin, range_end;
  int state;   // 0: nothing, 1: keys, 2: rows without keys
  int pieces;  // CTAs of the cluster that share the row tile's keys: this one has piece (rank in the cluster)
};
constexpr int kRowsItemInts = sizeof(RowsItem) / 4;
static_assert(sizeof(RowTile) == 24 && kRowsItemInts == 14, "as the broadcast copies it");
// num_splits is a bound: the pieces a request is cut into are chosen here, from the lengths and the launch's KV tiles
// per head, by the rule of the integer kernel (sched.cuh) - pieces of about equal length over the requests that this launch
// serves.  In a pair launch those are the tall ones alone: two chunks of 136 tiles beside eight verification requests of 256 are
// cut in two pieces each, those in four, whatever decode requests the integer kernel has.
// work(): those tiles, by all threads that call this.  It is asked for only if the request's own tiles allow this piece and more
// than one, whatever the others' are (a piece holds kItemTilesMin tiles on the average at least): most pieces of a generous
// bound are told empty without it, which takes 1.4 us of an SM instead of 2.2.
template <bool kClusters, class Work>
__device__ __forceinline__ RowsItem rows_item(const KernelParams& p, const RowTile& t, int split, Work work) {
  RowsItem it;
  it.t = t;
  it.state = 0;
  it.pieces = 1;
  it.rows = it.nsplits = it.tile_begin = it.tile_end = it.range_begin = it.range_end = 0;
  if (t.req < 0) return it;
  it.rows = t.ntok * p.group;
  it.nsplits = p.num_splits;
  if (p.num_splits > 1) {
    const int kv_tiles = req_kv_tiles(sched_shape(p), t.q_len, t.seq_len);
    const int most = req_splits(kv_tiles, kItemTilesMin, (int)gridDim.y);
    if (split >= most) return it;
    it.nsplits = most == 1 ? 1 : req_splits(kv_tiles, item_tiles(work() * (unsigned long long)p.num_kv_heads, p.num_sms), (int)gridDim.y);
    if (split >= it.nsplits) return it;
  }
  split_tiles(p, t, split, it.nsplits, &it.tile_begin, &it.tile_end, &it.range_begin, &it.range_end);
  it.state = it.tile_begin < it.tile_end ? 1 : 2;
  if constexpr (kClusters) {
    const int rank = (int)(blockIdx.x & (uint32_t)(p.cluster - 1)), n = it.tile_end - it.tile_begin, first = it.tile_begin;
    it.pieces = cluster_pieces(n, p.cluster);
    if (rank >= it.pieces) {
      it.state = 0;
    } else if (it.state == 1) {
      const int log2_pieces = __ffs(it.pieces) - 1;  // (two divisions of 64-bit numbers here: 0.4 us)
      it.tile_begin = first + (int)((int64_t)rank * n >> log2_pieces);
      it.tile_end = first + (int)((int64_t)(rank + 1) * n >> log2_pieces);
    }
  }
  return it;
}
__device__ __forceinline__ unsigned long long warp_sum(unsigned long long w) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
  return w;
}
// The launch's KV tiles per head, summed over the CTA (`scratch`: 8 idle bytes).
template <int kThreads>
__device__ __forceinline__ unsigned long long cta_work(const KernelParams& p, uint8_t* scratch) {
  const SchedShape shape = sched_shape(p);
  unsigned long long* total_s = reinterpret_cast<unsigned long long*>(scratch);
  unsigned long long w = 0;
  for (int r = threadIdx.x; r < p.num_reqs; r += kThreads) {
    const int a = __ldg(p.query_start_loc + r), b = __ldg(p.query_start_loc + r + 1);
    w += (unsigned long long)req_row_tiles(shape, b - a) * (unsigned long long)req_kv_tiles(shape, b - a, __ldg(p.seq_lens + r));
  }
  w = warp_sum(w);
  if (threadIdx.x == 0) *total_s = 0ull;
  __syncthreads();
  if ((threadIdx.x & 31) == 0 && w != 0) atomicAdd(total_s, w);
  __syncthreads();
  return *total_s;
}
// By all threads of the CTA: the CTA of piece 0 marks the pieces that the request does not use as holding no keys; rows
// without keys get a zero output and a log-sum-exp of -inf.
template <int kThreads, int kDim>
__device__ __forceinline__ void write_empty(const KernelParams& p, const RowsItem& it, int kvh, int split) {
  const int tid = threadIdx.x;
  const RowTile& t = it.t;
  if (it.state != 0 && split == 0 && p.num_splits > it.nsplits) {
    for (int i = tid; i < it.rows * (p.num_splits - it.nsplits); i += kThreads) {
      const int token = t.tok0 + (i % it.rows) / p.group, head = kvh * p.group + (i % it.rows) % p.group;
      *reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(p.ws_lse) + (int64_t)(it.nsplits + i / it.rows) * p.ws_lse_stride_split +
                                (int64_t)token * p.ws_lse_stride_token + (int64_t)head * p.ws_lse_stride_head) = -INFINITY;
    }
  }
  if (it.state != 2) return;
  for (int idx = tid; idx < it.rows * kDim; idx += kThreads) {
    const int n = idx / kDim, d = idx % kDim;
    const int token = t.tok0 + n / p.group, head = kvh * p.group + n % p.group;
    if (p.num_splits == 1) {
      store_out_elem(p.out + (int64_t)token * p.out_stride_token + (int64_t)head * p.out_stride_head, d, p.out_dtype, 0.f);
    } else {
      reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(p.ws_o) + (int64_t)split * p.ws_o_stride_split +
                               (int64_t)token * p.ws_o_stride_token + (int64_t)head * p.ws_o_stride_head)[d] = 0.f;
    }
  }
  if (tid < it.rows) {
    const int token = t.tok0 + tid / p.group, head = kvh * p.group + tid % p.group;
    if (p.num_splits > 1) {
      *reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(p.ws_lse) + (int64_t)split * p.ws_lse_stride_split +
                                (int64_t)token * p.ws_lse_stride_token + (int64_t)head * p.ws_lse_stride_head) = -INFINITY;
    } else if (p.lse_out != nullptr) {
      *reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(p.lse_out) + (int64_t)token * p.lse_stride_token +
                                (int64_t)head * p.lse_stride_head) = -INFINITY;
    }
  }
}

// ---- queries ----
constexpr float kQueryGain = 128.0f;
// What the keys' score factor takes back of the queries' power of two.
__device__ __forceinline__ float query_ungain(int q_dtype) { return q_dtype == PTH_ATTN_BF16 ? 1.0f / kQueryGain : 1.0f; }
// Bits of the largest finite magnitude among 8 N bf16 values.  An infinity or a NaN makes its row what it
// makes it anywhere; where one turns up the maximum is taken again without them.
template <int N>
__device__ __forceinline__ uint32_t finite_amax_bf16(const uint4 (&q)[N]) {
  uint32_t m = 0u;
#pragma unroll
  for (int c = 0; c < N; ++c) {
    m = __vimax3_u16x2(m, q[c].x & 0x7fff7fffu, q[c].y & 0x7fff7fffu);
    m = __vimax3_u16x2(m, q[c].z & 0x7fff7fffu, q[c].w & 0x7fff7fffu);
  }
  m = max(m & 0xffffu, m >> 16);
  if (m >= 0x7f80u) {
    m = 0u;
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const uint32_t w[4] = {q[c].x, q[c].y, q[c].z, q[c].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t lo = w[e] & 0x7fffu, hi = (w[e] >> 16) & 0x7fffu;
        m = max(m, max(lo < 0x7f80u ? lo : 0u, hi < 0x7f80u ? hi : 0u));
      }
    }
  }
  return m;
}
// The power of two of a row, and what its scores are multiplied by besides the keys' factor.
struct QueryScale {
  float scale, fix;
};
__device__ __forceinline__ QueryScale query_scale(uint32_t amax_bits) {
  const int e = (int)(amax_bits >> 7) - 127;  // (zero and subnormals: -127)
  if (amax_bits == 0u || (e >= -4 && e < 8)) return QueryScale{kQueryGain, 1.0f};
  const int s = min(14 - e, 126);             // -113 .. 126
  return QueryScale{__uint_as_float((uint32_t)(127 + s) << 23), __uint_as_float((uint32_t)(127 + 7 - s) << 23)};
}
// N scores of a row times what its own power of two leaves.  (In an instance of the tile loop of its own: the
// same multiplications behind a branch cost warps without such a row 1 to 4 %, a rolled loop over
// the scores in TMEM in front of the loads 3 to 5 % at 128 dims.)
template <int N>
__device__ __forceinline__ void scale_scores(uint32_t* r, float fix) {
#pragma unroll
  for (int n = 0; n < N; ++n) r[n] = __float_as_uint(__uint_as_float(r[n]) * fix);
}
// 8 bf16 queries times a power of two -> fp16.
__device__ __forceinline__ uint4 queries_to_f16(uint4 v, float scale) {
  auto two = [&](uint32_t w) { return pack_f16(__uint_as_float(w << 16) * scale, __uint_as_float(w & 0xffff0000u) * scale); };
  return make_uint4(two(v.x), two(v.y), two(v.z), two(v.w));
}

// ---- the softmax's two fp32 lanes per instruction ----
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pair(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpair(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// What the softmax needs of a key, one vector of N floats each: the score factor k_scale *
// softmax_scale * log2 e (/ 2^7 for bf16 queries), log2(v_scale) and 1 / v_scale.
template <int N>
struct KeyScales {
  float score[N], lv[N], iv[N];
};
// log2 of what P is multiplied by (see the head of this file).
constexpr float kPGain = 11.0f;
// v_scale as the softmax uses it: a scale of zero (or one below 2^-90, too small to matter) must not
// turn into 0 * infinity in the row sum, nor the sum of 2^15 / v_scale over a long row into infinity.
__device__ __forceinline__ float usable_v_scale(float v) { return v < 8.1e-28f ? 8.1e-28f : v; }

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Pass 1 of the softmax over N scores of a row (r: bits of S, replaced by score + log2(v_scale) in log2
// units); returns their maximum.  visible(n): whether the row sees the key of column n.
template <int N, bool kMask, class Wait, class Visible>
__device__ __forceinline__ float softmax_pass1(uint32_t (&r)[N], const float* score, const float* lv, Wait half_ready,
                                               Visible visible) {
  float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
  for (int n4 = 0; n4 < N / 4; ++n4) {
    if (n4 == N / 8) half_ready();
    const float4 k4 = reinterpret_cast<const float4*>(score)[n4], l4 = reinterpret_cast<const float4*>(lv)[n4];
    const f32x2 a = fma2(pair(__uint_as_float(r[4 * n4]), __uint_as_float(r[4 * n4 + 1])), pair(k4.x, k4.y), pair(l4.x, l4.y));
    const f32x2 b = fma2(pair(__uint_as_float(r[4 * n4 + 2]), __uint_as_float(r[4 * n4 + 3])), pair(k4.z, k4.w), pair(l4.z, l4.w));
    float t[4];
    unpair(a, t[0], t[1]);
    unpair(b, t[2], t[3]);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if constexpr (kMask) t[e] = visible(4 * n4 + e) ? t[e] : -INFINITY;
      r[4 * n4 + e] = __float_as_uint(t[e]);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) mx[e] = max3(mx[e], t[2 * e], t[2 * e + 1]);
  }
  return fmaxf(mx[0], mx[1]);
}
// Pass 2: probabilities of 32 of the scores as packed fp16 (a masked score is -inf: exp2 gives 0); adds
// p / v_scale to the two pairs of partial row sums.
__device__ __forceinline__ void softmax_pass2(const uint32_t* r, const float* iv, float m_use, f32x2 (&ls)[2], uint32_t (&pk)[16]) {
  const f32x2 neg_m = pair(-m_use, -m_use);
#pragma unroll
  for (int n4 = 0; n4 < 8; ++n4) {
    const float4 i4 = reinterpret_cast<const float4*>(iv)[n4];
    float x[4];
    unpair(add2(pair(__uint_as_float(r[4 * n4]), __uint_as_float(r[4 * n4 + 1])), neg_m), x[0], x[1]);
    unpair(add2(pair(__uint_as_float(r[4 * n4 + 2]), __uint_as_float(r[4 * n4 + 3])), neg_m), x[2], x[3]);
#pragma unroll
    for (int e = 0; e < 4; ++e) x[e] = ex2f(x[e]);
    ls[0] = fma2(pair(x[0], x[1]), pair(i4.x, i4.y), ls[0]);
    ls[1] = fma2(pair(x[2], x[3]), pair(i4.z, i4.w), ls[1]);
    pk[2 * n4] = pack_f16(x[0], x[1]);
    pk[2 * n4 + 1] = pack_f16(x[2], x[3]);
  }
}
__device__ __forceinline__ float sum_pairs(const f32x2 (&ls)[2]) {
  float a, b, c, d;
  unpair(ls[0], a, b);
  unpair(ls[1], c, d);
  return (a + b) + (c + d);
}

// Byte offset of row n of an item in a [token][head] array (rows are token-major).  (n is below 256 and the group at most
// 64: n + 1/2 keeps a distance of 1 / 128 from every multiple of the group.)
__device__ __forceinline__ int64_t row_offset(const RowTile& t, int kvh, int group, float inv_group, int n, int64_t stride_token,
                                              int64_t stride_head) {
  const int tok = (int)(((float)n + 0.5f) * inv_group);
  return (int64_t)(t.tok0 + tok) * stride_token + (int64_t)(kvh * group + (n - tok * group)) * stride_head;
}

__device__ __forceinline__ const uint8_t* shfl_ptr(const uint8_t* ptr, int lane) {
  return reinterpret_cast<const uint8_t*>((uintptr_t)__shfl_sync(0xffffffffu, (unsigned long long)(uintptr_t)ptr, lane));
}

// Queries of kCount rows (row0 .. of the CTA) by one warp: as many lanes per row as it has 16-byte blocks, so that a
// load covers whole rows.  Rows past the live ones are zeros.  Calls
// put(row, block, fp16 block) for every block, and fixed(row, fix) in one lane for every row (QueryScale).
template <int HD, int kCount, class Put, class Fixed>
__device__ __forceinline__ void stage_queries(const KernelParams& p, const RowTile& t, int kvh, int rows, int row0, Put put, Fixed fixed) {
  constexpr int kLanes = HD / 8, kAtOnce = 32 / kLanes, kSteps = kCount / kAtOnce, kBatch = 4;
  static_assert(kLanes <= 32 && kCount <= 32 && kSteps % kBatch == 0, "a warp covers whole rows");
  const int lane = threadIdx.x & 31, block = lane % kLanes, sub = lane / kLanes;
  // (lane l looks row row0 + l up)
  const uint8_t* mine = p.q + row_offset(t, kvh, p.group, 1.0f / (float)p.group, min(row0 + lane, rows - 1), p.q_stride_token, p.q_stride_head);
  const bool bf16 = p.q_dtype == PTH_ATTN_BF16;
  uint4 next[kBatch];
  auto load = [&](int k0) {
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int r = (k0 + k) * kAtOnce + sub;
      const uint8_t* src = shfl_ptr(mine, r);
      next[k] = row0 + r < rows ? __ldg(reinterpret_cast<const uint4*>(src) + block) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  load(0);
#pragma unroll 1
  for (int k0 = 0; k0 < kSteps; k0 += kBatch) {
    uint4 q[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) q[k] = next[k];
    if (k0 + kBatch < kSteps) load(k0 + kBatch);
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int n = row0 + (k0 + k) * kAtOnce + sub;
      float fix = 1.0f;
      if (bf16) {
        const uint4 one[1] = {q[k]};
        uint32_t amax = finite_amax_bf16(one);
#pragma unroll
        for (int o = kLanes / 2; o > 0; o >>= 1) amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        const QueryScale qs = query_scale(amax);
        fix = qs.fix;
        q[k] = queries_to_f16(q[k], qs.scale);
      }
      put(n, block, q[k]);
      if (block == 0) fixed(n, fix);
    }
  }
}

// Where a row's results go (from dim 0 on), and in which type.
struct RowsOut {
  uint8_t* row;   // of this lane's row
  uint32_t live;  // lanes with live rows
  int dtype;
};
__device__ __forceinline__ RowsOut rows_out(const KernelParams& p, const RowTile& t, int kvh, int rows, int row, int split) {
  RowsOut o;
  const float inv_group = 1.0f / (float)p.group;
  o.live = __ballot_sync(0xffffffffu, row < rows);
  if (p.num_splits > 1) {
    o.row = reinterpret_cast<uint8_t*>(p.ws_o) + (int64_t)split * p.ws_o_stride_split +
            row_offset(t, kvh, p.group, inv_group, row, p.ws_o_stride_token, p.ws_o_stride_head);
    o.dtype = PTH_ATTN_F32;
  } else {
    o.row = p.out + row_offset(t, kvh, p.group, inv_group, row, p.out_stride_token, p.out_stride_head);
    o.dtype = p.out_dtype;
  }
  return o;
}
// 32 dims (from d0) of the results of a warp's 32 rows, a row per lane in o: through 4 KB of shared
// memory of the warp's own, so that a store covers whole sectors of a few rows (each thread storing its own row 16 bytes
// at a time, a store touches 32 lines).
__device__ __forceinline__ void write_rows32(const RowsOut& out, int d0, uint8_t* stage, const float (&o)[32]) {
  const int lane = threadIdx.x & 31;
  if (out.dtype == PTH_ATTN_F32) {
#pragma unroll
    for (int c = 0; c < 8; ++c)
      *reinterpret_cast<float4*>(stage + lane * 128 + ((c ^ (lane & 7)) << 4)) = make_float4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
    __syncwarp();
    const int c = lane & 7;
#pragma unroll 2
    for (int k = 0; k < 8; ++k) {
      const int r = 4 * k + (lane >> 3);
      uint8_t* dst = const_cast<uint8_t*>(shfl_ptr(out.row, r)) + d0 * 4 + c * 16;
      const float4 v = *reinterpret_cast<const float4*>(stage + r * 128 + ((c ^ (r & 7)) << 4));
      if (out.live >> r & 1u) *reinterpret_cast<float4*>(dst) = v;
    }
  } else {
    const bool bf16 = out.dtype == PTH_ATTN_BF16;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = bf16 ? pack_bf16(o[8 * c + 2 * e], o[8 * c + 2 * e + 1]) : pack_f16(o[8 * c + 2 * e], o[8 * c + 2 * e + 1]);
      *reinterpret_cast<uint4*>(stage + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    __syncwarp();
    const int c = lane & 3;
#pragma unroll 2
    for (int k = 0; k < 4; ++k) {
      const int r = 8 * k + (lane >> 2);
      uint8_t* dst = const_cast<uint8_t*>(shfl_ptr(out.row, r)) + d0 * 2 + c * 16;
      const uint4 v = *reinterpret_cast<const uint4*>(stage + r * 64 + ((c ^ ((r >> 1) & 3)) << 4));
      if (out.live >> r & 1u) *reinterpret_cast<uint4*>(dst) = v;
    }
  }
  __syncwarp();  // (the stage is written again)
}
// A row's log-sum-exp (log2 units) where the caller wants it.
__device__ __forceinline__ void write_lse(const KernelParams& p, const RowTile& t, int kvh, int row, int split, float lse2) {
  const float inv_group = 1.0f / (float)p.group;
  if (p.num_splits > 1) {
    *reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(p.ws_lse) + (int64_t)split * p.ws_lse_stride_split +
                              row_offset(t, kvh, p.group, inv_group, row, p.ws_lse_stride_token, p.ws_lse_stride_head)) = lse2;
  } else if (p.lse_out != nullptr) {
    *reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(p.lse_out) +
                              row_offset(t, kvh, p.group, inv_group, row, p.lse_stride_token, p.lse_stride_head)) = lse2 * kLn2;
  }
}

// By the kRows * kParts threads of the softmax (`row`, `part`): the rows of a row tile whose keys `pieces` CTAs of the
// cluster have walked (a power of two).  This CTA (`rank`) merges and writes the rank-th run of columns from every CTA's
// parked accumulator (park_row32, relative to the row's maximum there), maxima and sums (stats: [2][kRows]); `weights`:
// idle shared memory, [kClusterMax][kRows].  Each starts with its own piece, so no CTA is read by all at once, and a
// thread has four to eight loads under way: a remote load takes many hundred cycles.
template <int kRows, int kParts, int kDim>
__device__ __forceinline__ void merge_pieces(const KernelParams& p, const RowTile& t, int kvh, int row, int part, int rank, int pieces,
                                             const float* park_own, const float* stats_own, float* weights) {
  const uint32_t park = tc::smem_u32(park_own) + row * 16, stats = tc::smem_u32(stats_own) + row * 4;
  auto peer = [&](int k) { return (rank + k) & (pieces - 1); };
  float m = -INFINITY, l = 0.f;
#pragma unroll 1
  for (int k0 = 0; k0 < pieces; k0 += 2) {
    const float a = peer_load(peer_address(stats, peer(k0))), b = peer_load(peer_address(stats, peer(k0 + 1)));
    m = fmaxf(m, fmaxf(a, b));
  }
#pragma unroll 2
  for (int k = 0; k < pieces; ++k) {
    const uint32_t from = peer_address(stats, peer(k));
    const float v = peer_load(from), sum = peer_load(from + kRows * 4);
    float w = v == -INFINITY ? 0.f : ex2f(v - m);
    if (sum != sum) w = sum;  // (a NaN among a piece's scores makes the row NaN, whatever its weight)
    if (w != 0.f) l = fmaf(w, sum, l);
    weights[k * kRows + row] = w;  // (the same value from every part; read by this thread)
  }
  const float inv = l > 0.f ? 1.0f / l : 0.f;
  uint8_t* dst = p.out + row_offset(t, kvh, p.group, 1.0f / (float)p.group, row, p.out_stride_token, p.out_stride_head);
  const int blocks = kDim / 4 / pieces, first = rank * blocks;  // 4 columns each
  // N blocks of columns from K pieces at once
  auto merge = [&](auto pieces_at_once, auto blocks_at_once) {
    constexpr int K = decltype(pieces_at_once)::value, N = decltype(blocks_at_once)::value;
#pragma unroll 1
    for (int b = part * N; b < blocks; b += kParts * N) {
      float o[N][4] = {};
#pragma unroll 1
      for (int k0 = 0; k0 < pieces; k0 += K) {
        float4 v[K][N];
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const uint32_t from = peer_address(park, peer(k0 + k));
#pragma unroll
          for (int n = 0; n < N; ++n) v[k][n] = peer_load4(from + (first + min(b + n, blocks - 1)) * kRows * 16);
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const float w = weights[(k0 + k) * kRows + row];
          if (w != 0.f) {  // (a NaN counts)
#pragma unroll
            for (int n = 0; n < N; ++n) {
              o[n][0] = fmaf(w, v[k][n].x, o[n][0]);
              o[n][1] = fmaf(w, v[k][n].y, o[n][1]);
              o[n][2] = fmaf(w, v[k][n].z, o[n][2]);
              o[n][3] = fmaf(w, v[k][n].w, o[n][3]);
            }
          }
        }
      }
      const int d = (first + b) * 4;
#pragma unroll
      for (int n = 0; n < N; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] *= inv;
      if (p.out_dtype == PTH_ATTN_F32) {
#pragma unroll
        for (int n = 0; n < N; ++n)
          if (b + n < blocks) *reinterpret_cast<float4*>(dst + (d + 4 * n) * 4) = make_float4(o[n][0], o[n][1], o[n][2], o[n][3]);
      } else {
        const bool bf16 = p.out_dtype == PTH_ATTN_BF16;
#pragma unroll
        for (int n = 0; n < N; n += 2) {
          auto two = [&](float x, float y) { return bf16 ? pack_bf16(x, y) : pack_f16(x, y); };
          const uint2 x = make_uint2(two(o[n][0], o[n][1]), two(o[n][2], o[n][3]));
          if (b + n + 1 < blocks)  // (then d is a multiple of 8)
            *reinterpret_cast<uint4*>(dst + (d + 4 * n) * 2) = make_uint4(x.x, x.y, two(o[n + 1][0], o[n + 1][1]), two(o[n + 1][2], o[n + 1][3]));
          else if (b + n < blocks)
            *reinterpret_cast<uint2*>(dst + (d + 4 * n) * 2) = x;
        }
      }
    }
  };
  if (pieces == 2) merge(std::integral_constant<int, 2>{}, std::integral_constant<int, 2>{});
  else merge(std::integral_constant<int, 4>{}, std::integral_constant<int, 2>{});
  if (rank == 0 && part == 0) write_lse(p, t, kvh, row, 0, l > 0.f ? m - kPGain + log2f(l) : -INFINITY);
}

}  // namespace pthb200
