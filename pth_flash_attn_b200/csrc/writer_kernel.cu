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
// cell, and the row maximum is a reduction over 16 lanes.  A warp issues the loads of two to four cells before it
// uses any, which leaves the quantisation's instructions as the bound (2 T Hkv D source elements in, T Hkv (2 D + 8)
// bytes out, at 0.56 of the rate of a copy).
// 8,192 tokens of 8 KV heads x 128 dims in bf16 (51 MB, which the L2 cache holds from call to call): 12.0 us a call back to
// back, 4.2 TB/s.  (One warp per row with
// 2-byte loads, fourteen rows after another: 43 us; with this shape, but maxima and scaling one element at a time, at 77
// registers and as an ordinary launch: 14.5, of which 1.4 were the launch; 40 registers spill: 15.3.)
#include <type_traits>

#include "params.cuh"
#include "pdl.cuh"

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

// Four consecutive elements of a source row, as they are in memory.  kBf16, kF16: rows on 8-byte boundaries,
// one 8-byte load; kAny: any type and alignment, element by element.
enum Source { kBf16, kF16, kAny };
template <Source kSource>
struct Four {
  uint32_t w[kSource == kAny ? 4 : 2];
  __device__ __forceinline__ void load(const uint8_t* row, int e0, int dtype) {
    if constexpr (kSource != kAny) {
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
    if constexpr (kSource == kBf16) return __uint_as_float(e & 1 ? w[e >> 1] & 0xffff0000u : w[e >> 1] << 16);
    else if constexpr (kSource == kF16) return __half2float(__ushort_as_half((unsigned short)(w[e >> 1] >> (16 * (e & 1)))));
    else if (dtype == PTH_ATTN_F32) return __uint_as_float(w[e]);
    else return dtype == PTH_ATTN_BF16 ? __uint_as_float(w[e] << 16) : __half2float(__ushort_as_half((unsigned short)w[e]));
  }
};

// Two fp32 lanes per instruction; each rounds as the instruction for one does.
__device__ __forceinline__ unsigned long long pair(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void mul2(float& a, float& b, float by) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pair(a, b)), "l"(pair(by, by)));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ void add2(float& a, float& b, float x, float y) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pair(a, b)), "l"(pair(x, y)));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}

// Four elements to int8: scaled, rounded half away from zero.  kFinite: all of the row are finite, and with the scale of
// their own maximum none reaches 127.5 by more than its rounding (inv <= 127 (1 + 2^-22) / amax), so nothing clamps
// them; an infinite row has inv = 0 and its infinities turn NaN, which the clamp makes -128 as a NaN is anywhere.
template <bool kFinite, Source kSource>
__device__ __forceinline__ uint32_t quantised(const Four<kSource>& x, float inv, int dtype) {
  int q[4];
#pragma unroll
  for (int e = 0; e < 4; e += 2) {
    float a = x.get(e, dtype), b = x.get(e + 1, dtype);
    mul2(a, b, inv);
    add2(a, b, copysignf(0.5f, a), copysignf(0.5f, b));
    if constexpr (!kFinite) {
      a = fminf(fmaxf(a, -128.0f), 127.0f);
      b = fminf(fmaxf(b, -128.0f), 127.0f);
    }
    q[e] = __float2int_rz(a);
    q[e + 1] = __float2int_rz(b);
  }
  return __byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], q[3], 0x0040), 0x5410);
}

template <int D, Source kSource>
__global__ void __launch_bounds__(kWriterThreads, kSource == kAny ? 1 : 5) kv_writer_kernel(const WriterParams p) {
  constexpr int kCells = cells_in_flight(D);
  constexpr int kRuns = D / (4 * kRowLanes);  // runs of 64 elements per row
  const int lane = threadIdx.x & 31, rl = lane & (kRowLanes - 1);
  const bool is_v = lane >= kRowLanes;
  const int64_t warp = ((int64_t)blockIdx.x * kWriterThreads + threadIdx.x) >> 5;
  const int64_t warps = ((int64_t)gridDim.x * kWriterThreads) >> 5;
  const int64_t cells = (int64_t)p.num_tokens * p.num_kv_heads;
  pdl_wait();
  const uint8_t* src0 = is_v ? p.value : p.key;
  const int64_t src_token = is_v ? p.value_stride_token : p.key_stride_token;
  const int64_t src_head = is_v ? p.value_stride_head : p.key_stride_head;
  const StreamParams& rows = is_v ? p.v : p.k;
  const StreamParams& scales = is_v ? p.vs : p.ks;
  for (int64_t cell0 = warp * kCells; cell0 < cells; cell0 += warps * kCells) {
    // Lane c of each half works out where cell c of its stream comes from and goes to, and its scale; the
    // others fetch that by shuffle.  (Divisions by every lane for every cell were a third of the instructions.)
    const int c_mine = rl & (kCells - 1);
    const int64_t cell = cell0 + c_mine;
    int64_t src_off = 0, slot = -1;  // (past the end: treated like a padding token)
    int head = 0;
    if (cell < cells) {
      const int token = cells <= 0x7fffffff ? (int)((uint32_t)cell / (uint32_t)p.num_kv_heads) : (int)(cell / p.num_kv_heads);
      head = (int)(cell - (int64_t)token * p.num_kv_heads);
      slot = __ldg(p.slot_mapping + token);
      src_off = token * src_token + head * src_head;
    }
    Four<kSource> x[kCells][kRuns] = {};
#pragma unroll
    for (int c = 0; c < kCells; ++c) {
      const uint8_t* row = src0 + __shfl_sync(0xffffffffu, src_off, c, kRowLanes);
      if (cell0 + c < cells) {
#pragma unroll
        for (int r = 0; r < kRuns; ++r) x[c][r].load(row, r * 64 + rl * 4, p.src_dtype);
      }
    }
    int64_t block, pos;
    if (slot <= 0x7fffffff) {
      block = (uint32_t)slot / (uint32_t)p.block_size;
      pos = (uint32_t)slot - (uint32_t)block * (uint32_t)p.block_size;
    } else {
      block = slot / p.block_size;
      pos = slot - block * p.block_size;
    }
    const int64_t dst_off = block * rows.stride_block + pos * rows.stride_slot + head * rows.stride_head;
    const uint32_t skipped = __ballot_sync(0xffffffffu, slot < 0);  // bit c: cell c
    // Largest magnitude of each cell's row.  Of 16-bit values as whole numbers, two at a time; an infinity or a NaN, which
    // does not count here, sends the warp's cells the long way.
    float amax_mine = 0.f;
    bool finite = kSource != kAny;
    if constexpr (kSource != kAny) {
      uint32_t bits_mine = 0u, top = 0u;
#pragma unroll
      for (int c = 0; c < kCells; ++c) {
        uint32_t m = 0u;
#pragma unroll
        for (int r = 0; r < kRuns; ++r) m = __vimax3_u16x2(m, x[c][r].w[0] & 0x7fff7fffu, x[c][r].w[1] & 0x7fff7fffu);
#pragma unroll
        for (int o = kRowLanes / 2; o > 0; o >>= 1) m = __vmaxu2(m, __shfl_xor_sync(0xffffffffu, m, o));
        m = max(m & 0xffffu, m >> 16);
        top = max(top, m);
        if (c_mine == c) bits_mine = m;
      }
      finite = !__any_sync(0xffffffffu, top >= (kSource == kBf16 ? 0x7f80u : 0x7c00u));
      amax_mine = kSource == kBf16 ? __uint_as_float(bits_mine << 16) : __half2float(__ushort_as_half((unsigned short)bits_mine));
    }
    if (!finite) {
#pragma unroll 1
      for (int c = 0; c < kCells; ++c) {
        float amax = 0.f;
#pragma unroll
        for (int k = 0; k < kCells; ++k) {
          if (k != c) continue;
#pragma unroll
          for (int r = 0; r < kRuns; ++r)
#pragma unroll
            for (int e = 0; e < 4; ++e) amax = fmaxf(amax, fabsf(x[k][r].get(e, p.src_dtype)));
        }
#pragma unroll
        for (int o = kRowLanes / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        if (c_mine == c) amax_mine = amax;
      }
    }
    const float scale_mine = fmaxf(__fdiv_rn(amax_mine, 127.0f), 1e-6f);
    const float inv_mine = __fdiv_rn(1.0f, scale_mine);
    if (slot >= 0 && rl < kCells) {
      *reinterpret_cast<float*>(const_cast<uint8_t*>(scales.data) + block * scales.stride_block + pos * scales.stride_slot +
                                head * scales.stride_head) = scale_mine;
    }
#pragma unroll
    for (int c = 0; c < kCells; ++c) {
      const float inv = __shfl_sync(0xffffffffu, inv_mine, c, kRowLanes);
      uint8_t* dst = const_cast<uint8_t*>(rows.data) + __shfl_sync(0xffffffffu, dst_off, c, kRowLanes);
      if (skipped >> c & 1u) continue;  // (the same for all lanes)
#pragma unroll
      for (int r = 0; r < kRuns; ++r)
        reinterpret_cast<uint32_t*>(dst)[r * kRowLanes + rl] =
            finite ? quantised<true>(x[c][r], inv, p.src_dtype) : quantised<false>(x[c][r], inv, p.src_dtype);
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
    if (vector && a.src_dtype == PTH_ATTN_BF16) return pdl_launch(kv_writer_kernel<D, kBf16>, grid, kWriterThreads, 0, stream, p);
    if (vector) return pdl_launch(kv_writer_kernel<D, kF16>, grid, kWriterThreads, 0, stream, p);
    return pdl_launch(kv_writer_kernel<D, kAny>, grid, kWriterThreads, 0, stream, p);
  };
  switch (a.head_size) {
    case 64:
      return launch(std::integral_constant<int, 64>{});
    case 128:
      return launch(std::integral_constant<int, 128>{});
    default:
      return launch(std::integral_constant<int, 256>{});
  }
}

}  // namespace pthb200
