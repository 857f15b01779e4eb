// Split-KV combine: merges the per-split partial outputs of one (token, head)
// row by their log2-sum-exp weights.
//
//   M   = max_s lse_s            (splits with lse_s = -inf hold no keys)
//   w_s = exp2(lse_s - M)
//   out = (sum_s w_s * o_s) / (sum_s w_s)
//
// num_splits is the caller's bound; a row has as many pieces as the attention kernels gave its
// request, one to three mostly.  So a row's log-sum-exps are read once, side by side, and only the
// partials of splits that hold keys are fetched, eight at a time:
//   up to kRowsSplits splits   a warp takes four rows, a lane per (row, split);
//   up to kWarpSplits          a warp takes a row, a lane per split;
//   more                       a CTA of 4 or (beyond kWideSplits) 16 warps takes a row: its live splits form a list,
//                              of which warp w sums the entries w, w + warps, ...; such a launch has few rows, and
//                              one warp walking many partials is pure latency.
// The order of a row's sums depends on its log-sum-exps and the number of splits alone, never on the
// number of rows or on timing.  What bounds it: two round trips to memory, one after the other, then bandwidth.
// (One warp per row reading all of its splits' log-sum-exps twice, one after the other with the token count in front, and
// launched behind the attention kernel's end: mixed batch, 136,000 rows of up to 8 pieces, 97 us, now 46; 768 rows of
// 256 dims and up to 37 pieces 7.6 and 4.0; 8 x U[1, 4096] keys 22.6 us a call, now 17.7.)
//
// A split with lse = -inf is skipped BEFORE its ws_o row is read, so garbage
// (NaN included) in the partial of an empty split never reaches the output.
// Lane j owns output columns 4j..4j+3 (+128, +256 for wider heads) and moves
// them as 16-byte vectors.  A row whose
// splits are all empty gets out = 0 and lse = -inf.  Rows >=
// query_start_loc[num_reqs] are skipped.
#include "params.cuh"
#include "pdl.cuh"

namespace pthb200 {

namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kRowsSplits = 8;
constexpr int kWarpSplits = 32;
constexpr int kWideSplits = 64;
constexpr int kBatch = 8;        // partial rows loaded before their sums start

template <int D>
struct RowSum {
  static constexpr int kCols = (D + 127) / 128;
  float acc[kCols][4];
  float den;
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int c = 0; c < kCols; ++c)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[c][e] = 0.f;
    den = 0.f;
  }
};
template <int D>
struct Partial {
  float4 v[RowSum<D>::kCols];
  __device__ __forceinline__ void load(const uint8_t* o_row, int lane, bool live) {
#pragma unroll
    for (int c = 0; c < RowSum<D>::kCols; ++c) {
      const int d = c * 128 + lane * 4;
      v[c] = live && d < D ? *reinterpret_cast<const float4*>(o_row + (int64_t)d * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  __device__ __forceinline__ void add(float w, RowSum<D>& r) const {
    r.den += w;
#pragma unroll
    for (int c = 0; c < RowSum<D>::kCols; ++c) {
      r.acc[c][0] = fmaf(w, v[c].x, r.acc[c][0]);
      r.acc[c][1] = fmaf(w, v[c].y, r.acc[c][1]);
      r.acc[c][2] = fmaf(w, v[c].z, r.acc[c][2]);
      r.acc[c][3] = fmaf(w, v[c].w, r.acc[c][3]);
    }
  }
};

// (row = token x query head)
struct RowAt {
  int token, head;
  const uint8_t* lse;
  const uint8_t* o;
};
__device__ __forceinline__ RowAt row_at(const CombineParams& p, int64_t row) {
  RowAt r;
  r.token = row <= 0x7fffffff ? (int)((uint32_t)row / (uint32_t)p.num_q_heads) : (int)(row / p.num_q_heads);
  r.head = (int)(row - (int64_t)r.token * p.num_q_heads);
  r.lse = reinterpret_cast<const uint8_t*>(p.ws_lse) + (int64_t)r.token * p.ws_lse_stride_token + (int64_t)r.head * p.ws_lse_stride_head;
  r.o = reinterpret_cast<const uint8_t*>(p.ws_o) + (int64_t)r.token * p.ws_o_stride_token + (int64_t)r.head * p.ws_o_stride_head;
  return r;
}
__device__ __forceinline__ float lse_of(const CombineParams& p, const RowAt& r, int s) {
  return *reinterpret_cast<const float*>(r.lse + (int64_t)s * p.ws_lse_stride_split);
}
// Weight of a split; 0 for one without keys.  (A NaN counts as one; it never raises the maximum either.)
__device__ __forceinline__ float weight_of(float lse, float mx) {
  const float w = lse > -INFINITY ? exp2f(lse - mx) : 0.f;
  return w >= 0.f ? w : 0.f;
}

template <int D>
__device__ __forceinline__ void write_row(const CombineParams& p, const RowAt& at, const RowSum<D>& r, float mx, int lane) {
  const float inv = r.den > 0.f ? 1.f / r.den : 0.f;
  uint8_t* out_row = p.out + (int64_t)at.token * p.out_stride_token + (int64_t)at.head * p.out_stride_head;
#pragma unroll
  for (int c = 0; c < RowSum<D>::kCols; ++c) {
    const int d = c * 128 + lane * 4;
    if (d < D) {
      const float r0 = r.acc[c][0] * inv, r1 = r.acc[c][1] * inv, r2 = r.acc[c][2] * inv, r3 = r.acc[c][3] * inv;
      if (p.out_dtype == PTH_ATTN_BF16) {
        __nv_bfloat162 a = __floats2bfloat162_rn(r0, r1), b = __floats2bfloat162_rn(r2, r3);
        uint2 pk;
        pk.x = *reinterpret_cast<uint32_t*>(&a);
        pk.y = *reinterpret_cast<uint32_t*>(&b);
        *reinterpret_cast<uint2*>(out_row + (int64_t)d * 2) = pk;
      } else if (p.out_dtype == PTH_ATTN_F16) {
        __half2 a = __floats2half2_rn(r0, r1), b = __floats2half2_rn(r2, r3);
        uint2 pk;
        pk.x = *reinterpret_cast<uint32_t*>(&a);
        pk.y = *reinterpret_cast<uint32_t*>(&b);
        *reinterpret_cast<uint2*>(out_row + (int64_t)d * 2) = pk;
      } else {
        *reinterpret_cast<float4*>(out_row + (int64_t)d * 4) = make_float4(r0, r1, r2, r3);
      }
    }
  }
  if (p.lse_out != nullptr && lane == 0) {
    const float lse2 = r.den > 0.f ? mx + log2f(r.den) : -INFINITY;
    *reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(p.lse_out) + (int64_t)at.token * p.lse_stride_token +
                              (int64_t)at.head * p.lse_stride_head) = lse2 * kLn2;
  }
}

// Four rows per warp, lane 8 j + s for split s of row j.
template <int D>
__global__ void __launch_bounds__(kThreads) combine_rows_kernel(const __grid_constant__ CombineParams p) {
  constexpr int kRows = 32 / kRowsSplits;
  const int lane = threadIdx.x & 31;
  const int64_t row0 = ((int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5)) * kRows;
  const int64_t rows = (int64_t)p.num_tokens * p.num_q_heads;
  pdl_wait();
  const int64_t mine = row0 + lane / kRowsSplits;
  const int s_mine = lane % kRowsSplits;
  float lse = -INFINITY;
  if (mine < rows && s_mine < p.num_splits) lse = lse_of(p, row_at(p, mine), s_mine);
  const int64_t valid = (int64_t)min(p.num_tokens, __ldg(p.query_start_loc + p.num_reqs)) * p.num_q_heads;
  float mx = lse > -INFINITY ? lse : -INFINITY;
#pragma unroll
  for (int o = kRowsSplits / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const float w_mine = weight_of(lse, mx);
  const uint32_t live = __ballot_sync(0xffffffffu, w_mine != 0.f && mine < valid);
  RowSum<D> sum[kRows];
  RowAt at[kRows];
  uint32_t left[kRows];  // live splits of the row that are still to be added
#pragma unroll
  for (int j = 0; j < kRows; ++j) {
    sum[j].clear();
    at[j] = row_at(p, row0 + j < rows ? row0 + j : 0);
    left[j] = live >> (kRowsSplits * j) & ((1u << kRowsSplits) - 1);
  }
  // a split of each row, then the next of each: the loads of two steps are in flight together
  while ((left[0] | left[1] | left[2] | left[3]) != 0u) {
    Partial<D> part[2][kRows];
    float w[2][kRows];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int j = 0; j < kRows; ++j) {
        const int s = left[j] != 0u ? __ffs(left[j]) - 1 : 0;
        const float ws = __shfl_sync(0xffffffffu, w_mine, kRowsSplits * j + s);
        w[k][j] = left[j] != 0u ? ws : 0.f;
        part[k][j].load(at[j].o + (int64_t)s * p.ws_o_stride_split, lane, left[j] != 0u);
        left[j] &= left[j] - 1;
      }
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int j = 0; j < kRows; ++j)
        if (w[k][j] != 0.f) part[k][j].add(w[k][j], sum[j]);
  }
#pragma unroll
  for (int j = 0; j < kRows; ++j) {
    const float mx_j = __shfl_sync(0xffffffffu, mx, kRowsSplits * j);
    if (row0 + j < valid) write_row<D>(p, at[j], sum[j], mx_j, lane);
  }
}

// One row per CTA of kRunWarps warps, or, with kRunWarps = 1, one row per warp.
template <int D, int kRunWarps>
__global__ void __launch_bounds__(kRunWarps > 1 ? kRunWarps * 32 : kThreads)
combine_kernel(const __grid_constant__ CombineParams p) {
  constexpr int kCols = RowSum<D>::kCols;
  constexpr int kLanes = kRunWarps * 32;  // splits looked at together
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int run_warp = kRunWarps > 1 ? warp : 0, t = run_warp * 32 + lane;
  const int64_t row = kRunWarps > 1 ? (int64_t)blockIdx.x : (int64_t)blockIdx.x * kWarps + warp;
  pdl_wait();
  if (row >= (int64_t)p.num_tokens * p.num_q_heads) return;  // (the whole CTA with kRunWarps > 1)
  const RowAt at = row_at(p, row);
  const int S = p.num_splits;
  __shared__ float list_w[kRunWarps > 1 ? kLanes : 1];
  __shared__ int list_s[kRunWarps > 1 ? kLanes : 1];
  __shared__ float warp_mx[kRunWarps];
  __shared__ int warp_live[kRunWarps];
  __shared__ float part_s[kRunWarps > 1 ? kRunWarps - 1 : 1][kCols * 4 + 1][32];

  const float first = t < S ? lse_of(p, at, t) : -INFINITY;  // (up to kLanes splits are read once)
  const int valid_tokens = min(p.num_tokens, __ldg(p.query_start_loc + p.num_reqs));
  float mx = first > -INFINITY ? first : -INFINITY;
  for (int s = t + kLanes; s < S; s += kLanes) {
    const float v = lse_of(p, at, s);
    if (v > mx) mx = v;
  }
  if (at.token >= valid_tokens) return;  // (the same for all threads of the row)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if constexpr (kRunWarps > 1) {
    if (lane == 0) warp_mx[warp] = mx;
    __syncthreads();
    mx = warp_mx[0];
#pragma unroll
    for (int w = 1; w < kRunWarps; ++w) mx = fmaxf(mx, warp_mx[w]);
  }
  RowSum<D> r;
  r.clear();
  for (int s0 = 0; s0 < S; s0 += kLanes) {
    const float lse = s0 == 0 ? first : s0 + t < S ? lse_of(p, at, s0 + t) : -INFINITY;
    const float w_mine = weight_of(lse, mx);
    const uint32_t live = __ballot_sync(0xffffffffu, w_mine != 0.f);
    if constexpr (kRunWarps == 1) {
      for (uint32_t left = live; left != 0u;) {
        Partial<D> part[kBatch];
        float w[kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          const int s = left != 0u ? __ffs(left) - 1 : 0;
          const float ws = __shfl_sync(0xffffffffu, w_mine, s);
          w[b] = left != 0u ? ws : 0.f;
          part[b].load(at.o + (int64_t)(s0 + s) * p.ws_o_stride_split, lane, left != 0u);
          left &= left - 1;
        }
#pragma unroll
        for (int b = 0; b < kBatch; ++b)
          if (w[b] != 0.f) part[b].add(w[b], r);
      }
    } else {
      if (lane == 0) warp_live[warp] = __popc(live);
      __syncthreads();
      int at_list = __popc(live & ((1u << lane) - 1)), n = 0;
#pragma unroll
      for (int w = 0; w < kRunWarps; ++w) {
        at_list += w < warp ? warp_live[w] : 0;
        n += warp_live[w];
      }
      if (w_mine != 0.f) {
        list_w[at_list] = w_mine;
        list_s[at_list] = s0 + t;
      }
      __syncthreads();
      for (int i0 = warp; i0 < n; i0 += kBatch * kRunWarps) {
        Partial<D> part[kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          const int i = i0 + b * kRunWarps;
          part[b].load(at.o + (int64_t)(i < n ? list_s[i] : 0) * p.ws_o_stride_split, lane, i < n);
        }
#pragma unroll
        for (int b = 0; b < kBatch; ++b)
          if (i0 + b * kRunWarps < n) part[b].add(list_w[i0 + b * kRunWarps], r);
      }
      if (s0 + kLanes < S) __syncthreads();  // (the list is written anew)
    }
  }
  if constexpr (kRunWarps > 1) {
    if (warp > 0) {
#pragma unroll
      for (int c = 0; c < kCols; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e) part_s[warp - 1][c * 4 + e][lane] = r.acc[c][e];
      part_s[warp - 1][kCols * 4][lane] = r.den;
    }
    __syncthreads();
    if (warp > 0) return;
#pragma unroll
    for (int w = 0; w < kRunWarps - 1; ++w) {
#pragma unroll
      for (int c = 0; c < kCols; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e) r.acc[c][e] += part_s[w][c * 4 + e][lane];
      r.den += part_s[w][kCols * 4][lane];
    }
  }
  write_row<D>(p, at, r, mx, lane);
}

template <int D>
cudaError_t launch_for(const CombineParams& p, cudaStream_t stream) {
  const int64_t rows = (int64_t)p.num_tokens * p.num_q_heads;
  auto grid = [&](int64_t per_cta) { return (unsigned)((rows + per_cta - 1) / per_cta); };
  if (p.num_splits <= kRowsSplits) return pdl_launch(combine_rows_kernel<D>, grid(kWarps * (32 / kRowsSplits)), kThreads, 0, stream, p);
  if (p.num_splits <= kWarpSplits) return pdl_launch(combine_kernel<D, 1>, grid(kWarps), kThreads, 0, stream, p);
  if (p.num_splits <= kWideSplits) return pdl_launch(combine_kernel<D, 4>, grid(1), 4 * 32, 0, stream, p);
  return pdl_launch(combine_kernel<D, 16>, grid(1), 16 * 32, 0, stream, p);
}

}  // namespace

cudaError_t launch_combine_kernel(const CombineParams& p, cudaStream_t stream) {
  switch (p.head_size) {
    case 64:
      return launch_for<64>(p, stream);
    case 128:
      return launch_for<128>(p, stream);
    default:
      return launch_for<256>(p, stream);
  }
}

}  // namespace pthb200
