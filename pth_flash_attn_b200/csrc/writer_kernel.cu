// Quantising KV-cache writer: the step in front of the attention path.
//
// For every new token and KV head it turns one K row and one V row (fp32 / fp16 / bf16) into
// the cache's int8_per_token_head form, with the arithmetic of the writer the cache format
// is defined by, step for step in fp32 so that the bytes are identical:
//   absmax = max |x_d|;   scale = max(absmax / 127, 1e-6);   inv = 1 / scale
//   q_d = clamp(trunc(x_d * inv +- 0.5), -128, 127)          (round half away from zero)
// and stores the D int8 values and the fp32 scale through the same four strided streams the
// attention op reads (K bytes, V bytes, K scales, V scales), at the slot slot_mapping names:
// block = slot / block_size, position = slot % block_size; a negative slot skips the token.
//
// A cell (token, KV head) belongs to one warp: its first 16 lanes take the K row, the others the V
// row.  A row is read 64 elements at a time, four per lane, so that a load is 8 bytes of a 16-bit
// source, the 16 lanes' words leave as one run of 64 bytes whatever the 4-byte alignment of the
// cell, and the row maximum is a reduction over 16 lanes.  The kernel is bound by HBM (it reads
// 2 T Hkv D source elements and writes T Hkv (2 D + 8) bytes) as long as enough loads are in flight:
// a warp issues those of two to four cells before it uses any.
#include <type_traits>

#include "params.cuh"

namespace pthb200 {
namespace {

constexpr int kWriterThreads = 256;

struct WriterParams {
  const uint8_t* key;
  const uint8_t* value;
  int64_t key_stride_token, key_stride_head, value_stride_token, value_stride_head;
  StreamParams k, v, ks, vs;  // data pointers are written through
  const int64_t* slot_mapping;
  int32_t src_dtype, block_size, num_kv_heads, num_tokens;
};

constexpr int kRowLanes = 16;
// Cells a warp has in flight: 2 KB of a 16-bit source up to 128 dims.
__host__ __device__ constexpr int cells_in_flight(int head_size) { return head_size == 256 ? 2 : 4; }

// Four consecutive elements of a source row, as they are in memory.  kVector: 16-bit elements whose rows
// are 8-byte aligned, two per word; otherwise loaded element by element.
template <bool kVector>
struct Four {
  uint32_t w[kVector ? 2 : 4];
  __device__ __forceinline__ void load(const uint8_t* row, int e0, int dtype) {
    if constexpr (kVector) {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(row + e0 * 2));
      w[0] = v.x;
      w[1] = v.y;
    } else if (dtype == PTH_ATTN_F32) {
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = __ldg(reinterpret_cast<const uint32_t*>(row) + e0 + e);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = __ldg(reinterpret_cast<const unsigned short*>(row) + e0 + e);
    }
  }
  __device__ __forceinline__ float get(int e, int dtype) const {
    if (!kVector && dtype == PTH_ATTN_F32) return __uint_as_float(w[e]);
    const uint32_t bits = kVector ? (e & 1 ? w[e >> 1] >> 16 : w[e >> 1] & 0xffffu) : w[e];
    return dtype == PTH_ATTN_BF16 ? __uint_as_float(bits << 16) : __half2float(__ushort_as_half((unsigned short)bits));
  }
};

template <int D, bool kVector>
__global__ void __launch_bounds__(kWriterThreads) kv_writer_kernel(const WriterParams p) {
  constexpr int kCells = cells_in_flight(D);
  constexpr int kRuns = D / (4 * kRowLanes);  // runs of 64 elements per row
  const int lane = threadIdx.x & 31, rl = lane & (kRowLanes - 1);
  const bool is_v = lane >= kRowLanes;
  const int64_t warp = ((int64_t)blockIdx.x * kWriterThreads + threadIdx.x) >> 5;
  const int64_t warps = ((int64_t)gridDim.x * kWriterThreads) >> 5;
  const int64_t cells = (int64_t)p.num_tokens * p.num_kv_heads;
  const uint8_t* src0 = is_v ? p.value : p.key;
  const int64_t src_token = is_v ? p.value_stride_token : p.key_stride_token;
  const int64_t src_head = is_v ? p.value_stride_head : p.key_stride_head;
  const StreamParams& rows = is_v ? p.v : p.k;
  const StreamParams& scales = is_v ? p.vs : p.ks;
  for (int64_t cell0 = warp * kCells; cell0 < cells; cell0 += warps * kCells) {
    int64_t slot[kCells];
    int head[kCells];
    Four<kVector> x[kCells][kRuns];
#pragma unroll
    for (int c = 0; c < kCells; ++c) {
      slot[c] = -1;  // (past the end: treated like a padding token)
      head[c] = 0;
      if (cell0 + c < cells) {
        const int token = cells <= 0x7fffffff ? (int)((uint32_t)(cell0 + c) / (uint32_t)p.num_kv_heads)
                                              : (int)((cell0 + c) / p.num_kv_heads);
        head[c] = (int)(cell0 + c - (int64_t)token * p.num_kv_heads);
        slot[c] = __ldg(p.slot_mapping + token);
        const uint8_t* row = src0 + token * src_token + head[c] * src_head;
#pragma unroll
        for (int r = 0; r < kRuns; ++r) x[c][r].load(row, r * 64 + rl * 4, p.src_dtype);
      }
    }
#pragma unroll
    for (int c = 0; c < kCells; ++c) {
      if (slot[c] < 0) continue;  // (the same for all lanes)
      float f[kRuns][4], amax = 0.f;
#pragma unroll
      for (int r = 0; r < kRuns; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          f[r][e] = x[c][r].get(e, p.src_dtype);
          amax = fmaxf(amax, fabsf(f[r][e]));
        }
#pragma unroll
      for (int o = kRowLanes / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      const float scale = fmaxf(__fdiv_rn(amax, 127.0f), 1e-6f);
      const float inv = __fdiv_rn(1.0f, scale);
      int64_t block, pos;
      if (slot[c] <= 0x7fffffff) {
        block = (uint32_t)slot[c] / (uint32_t)p.block_size;
        pos = (uint32_t)slot[c] - (uint32_t)block * (uint32_t)p.block_size;
      } else {
        block = slot[c] / p.block_size;
        pos = slot[c] - block * p.block_size;
      }
      uint8_t* dst = const_cast<uint8_t*>(rows.data) + block * rows.stride_block + pos * rows.stride_slot + head[c] * rows.stride_head;
#pragma unroll
      for (int r = 0; r < kRuns; ++r) {
        uint32_t word = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float v = __fmul_rn(f[r][e], inv);
          v = v >= 0.f ? __fadd_rn(v, 0.5f) : __fadd_rn(v, -0.5f);
          v = fminf(fmaxf(v, -128.0f), 127.0f);
          word |= (uint32_t)(uint8_t)(int8_t)(int)truncf(v) << (8 * e);
        }
        reinterpret_cast<uint32_t*>(dst)[r * kRowLanes + rl] = word;
      }
      if (rl == 0) {
        *reinterpret_cast<float*>(const_cast<uint8_t*>(scales.data) + block * scales.stride_block +
                                  pos * scales.stride_slot + head[c] * scales.stride_head) = scale;
      }
    }
  }
}

}  // namespace

cudaError_t launch_kv_writer(const PthB200WriteArgs& a, cudaStream_t stream) {
  WriterParams p{};
  p.key = static_cast<const uint8_t*>(a.key);
  p.value = static_cast<const uint8_t*>(a.value);
  p.key_stride_token = a.key_stride_token;
  p.key_stride_head = a.key_stride_head;
  p.value_stride_token = a.value_stride_token;
  p.value_stride_head = a.value_stride_head;
  auto stream_of = [](const PthAttnStream& s) {
    return StreamParams{static_cast<const uint8_t*>(s.data), s.stride_block, s.stride_slot, s.stride_head};
  };
  p.k = stream_of(a.k_cache);
  p.v = stream_of(a.v_cache);
  p.ks = stream_of(a.k_scale);
  p.vs = stream_of(a.v_scale);
  p.slot_mapping = a.slot_mapping;
  p.src_dtype = a.src_dtype;
  p.block_size = a.block_size;
  p.num_kv_heads = a.num_kv_heads;
  p.num_tokens = a.num_tokens;
  const int64_t cells = (int64_t)a.num_tokens * a.num_kv_heads, per_cta = kWriterThreads / 32 * cells_in_flight(a.head_size);
  const int64_t want = (cells + per_cta - 1) / per_cta;
  const unsigned grid = (unsigned)(want > (1 << 30) ? (1 << 30) : want);
  // 8-byte loads need 16-bit rows that start on 8-byte boundaries (D is a multiple of 64)
  auto on8 = [](const void* ptr, int64_t st, int64_t sh) { return (reinterpret_cast<uintptr_t>(ptr) | (uint64_t)st | (uint64_t)sh) % 8 == 0; };
  const bool vector = a.src_dtype != PTH_ATTN_F32 && on8(a.key, a.key_stride_token, a.key_stride_head) &&
                      on8(a.value, a.value_stride_token, a.value_stride_head);
  auto launch = [&](auto head_size) {
    constexpr int D = decltype(head_size)::value;
    if (vector) kv_writer_kernel<D, true><<<grid, kWriterThreads, 0, stream>>>(p);
    else kv_writer_kernel<D, false><<<grid, kWriterThreads, 0, stream>>>(p);
  };
  switch (a.head_size) {
    case 64:
      launch(std::integral_constant<int, 64>{});
      break;
    case 128:
      launch(std::integral_constant<int, 128>{});
      break;
    default:
      launch(std::integral_constant<int, 256>{});
      break;
  }
  return cudaGetLastError();
}

}  // namespace pthb200
