// Stage 2: per-(request, query head) log-sum-exp merge of the request's partial
// rows (kernel_bench/fasttree.py:482-546).  Memory-bound on the partial buffers;
// those are written by stage 1 just before and are normally still in L2.
//
// stage2_merge_kernel: one warp per (request, head) of head_dim 128 or 256; lanes span
// it in float4 chunks, so a partial row of 128 is one 512-byte coalesced warp load.
// The weights exp(lse_i - max) are computed lane-parallel (32 partial rows at a
// time, running maximum across batches) and broadcast by shuffle, which keeps the
// dependent chain per partial to one FMA.
//
// stage2_piece_kernel: a partial row's heads are adjacent in memory, so a warp takes
// 128 C floats of them at once - lane l the float4s l, l + 32, ..., whatever heads
// they belong to (two heads at head_dim 64, where the other kernel's lanes are half
// idle) - RB rows at a time, and every lane computes the weights of its own heads:
// nothing is exchanged, which is quicker while the rows are few.  SPLIT warps share
// a piece's rows, each its own stretch of them, and merge through shared memory: a
// launch that leaves the SMs nearly empty is bound by the chain of round trips of
// its longest request.
#pragma once

#include "ft_common.cuh"

namespace ft {

// Four columns of an output row.
template <typename T>
__device__ __forceinline__ void store_columns(const Stage2Params& p, int req, int head, int at, const float4& acc, float inv) {
  T* __restrict__ dst = reinterpret_cast<T*>(p.o) + (int64_t)req * p.o_s0 + (int64_t)head * p.o_s1 + at;
  alignas(16) T out[4] = {from_float<T>(acc.x * inv), from_float<T>(acc.y * inv), from_float<T>(acc.z * inv), from_float<T>(acc.w * inv)};
  if (p.o_vec) {  // in one store when the output rows allow it
    if constexpr (sizeof(T) == 2)
      *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(out);
    else
      *reinterpret_cast<float4*>(dst) = *reinterpret_cast<const float4*>(out);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) dst[e] = out[e];
  }
}

// To a new maximum.  A partial row counts only if its weight, relative to the request's largest LSE, is not zero - else
// infinities and NaN in rows that do not count would come into the sum as 0 x Inf.  While rows are still being met the
// largest LSE is not known: a sum of rows that the new maximum leaves nothing of starts anew, whatever it holds.  (What is
// left over: an infinite row of no weight that two steps of the maximum take there, each of which leaves some.  A sum formed
// once more where it did not come out finite has no such case, but the code for it, even where nothing runs it, cost steps
// at head_dim 256 1 to 4 %: 64 requests on 4096 tokens 44.6 -> 46.2 us.)
__device__ __forceinline__ void scale(float4& x, float f) {
  x.x *= f;
  x.y *= f;
  x.z *= f;
  x.w *= f;
  if (f == 0.f) x = make_float4(0.f, 0.f, 0.f, 0.f);
}

// MAXC: float4 chunks per lane (1: head_dim 128, 2: head_dim 256; smaller heads go to the other kernel).  RB: partial rows
// in flight per lane.  A request's merge is a chain of L2 round trips, one per batch of RB rows.  A launch that fits one
// round of CTAs is bound by that chain and runs with RB = 8 at six CTAs per SM; a launch of several rounds is bound by how
// many warps the SM holds and runs with RB = 4 at nine (head_dim 128); at head_dim 256 seven, the next stage 1's first
// CTAs beside them (six, with 78 registers for 72: 256 requests of 30 tokens on 200, 32/8 heads, 31.4 us per step for 30.2).
template <typename T, int MAXC, int RB>
__global__ void __launch_bounds__(128, MAXC == 1 && RB == 4 ? 9 : MAXC == 2 ? 7 : 6) stage2_merge_kernel(Stage2Params p) {
  allow_dependent_launch();  // a following stage-1 launch may set itself up under this kernel's tail
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t pair = (int64_t)blockIdx.x * 4 + warp;
  if (pair >= (int64_t)p.batch * p.heads) return;
  const int req = (int)(pair / p.heads);
  const int head = (int)(pair - (int64_t)req * p.heads);
  const int off = p.r2v_offs[req];
  const int n = p.r2v_lens[req];
  int batch_rows = lane < n ? p.r2v_entries[off + lane] : -1;  // plan data: readable before stage 1 is done
  wait_for_prior_grid();                                       // the partial buffers are complete from here on

  // One pass with a running maximum (as in the online softmax): per batch of up to 32 partial rows the lanes
  // fetch their row's LSE while the first rows of the batch are already being loaded - the row addresses depend
  // on the plan only - so a request with few partials costs one round trip to the partial buffers, not two.
  float mx = -INFINITY;
  float4 acc[MAXC];
#pragma unroll
  for (int c = 0; c < MAXC; ++c) acc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
  float wsum = 0.f;
  for (int base = 0; base < n; base += 32) {
    const int cnt = min(32, n - base);
    int my_row = -1;
    const int row = batch_rows;
    batch_rows = base + 32 + lane < n ? p.r2v_entries[off + base + 32 + lane] : -1;  // the next batch's ids travel under this batch's rows
    if (lane < cnt) {
      if (row >= 0 && row < p.num_partial_rows)
        my_row = row;
      else
        flag_error(FT_DEV_BAD_ROW_INDEX);
    }
    const float my_lse = my_row >= 0 ? __ldcg(p.mid_lse + (int64_t)my_row * p.ml_s0 + head) : -INFINITY;
    float my_w = 0.f;
    for (int i0 = 0; i0 < cnt; i0 += RB) {
      float4 x[RB][MAXC];
      int rows[RB];
#pragma unroll
      for (int r = 0; r < RB; ++r) {
        rows[r] = i0 + r < cnt ? __shfl_sync(0xffffffffu, my_row, (i0 + r) & 31) : -1;
        const float4* __restrict__ src =
            reinterpret_cast<const float4*>(p.mid_o + (int64_t)(rows[r] >= 0 ? rows[r] : 0) * p.mo_s0 + (int64_t)head * p.mo_s1);
#pragma unroll
        for (int c = 0; c < MAXC; ++c) {
          x[r][c] = rows[r] >= 0 ? __ldcg(src + lane + 32 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      if (i0 == 0) {  // the batch's LSEs are needed only now: rescale what has been summed so far to the new maximum
        const float bm = warp_max(my_lse);
        const float new_mx = fmaxf(mx, bm);
        const float corr = new_mx == -INFINITY ? 1.f : expf(mx - new_mx);  // 0 for the first batch
        wsum *= corr;
#pragma unroll
        for (int c = 0; c < MAXC; ++c) {
          scale(acc[c], corr);
        }
        mx = new_mx;
        my_w = my_lse > -INFINITY ? expf(my_lse - mx) : 0.f;  // -inf LSE marks an empty partial
        wsum += my_w;
      }
#pragma unroll
      for (int r = 0; r < RB; ++r) {
        const float w = __shfl_sync(0xffffffffu, my_w, (i0 + r) & 31);
        if (rows[r] < 0 || w == 0.f) continue;
#pragma unroll
        for (int c = 0; c < MAXC; ++c) {
          acc[c].x = fmaf(w, x[r][c].x, acc[c].x);
          acc[c].y = fmaf(w, x[r][c].y, acc[c].y);
          acc[c].z = fmaf(w, x[r][c].z, acc[c].z);
          acc[c].w = fmaf(w, x[r][c].w, acc[c].w);
        }
      }
    }
  }
  wsum = warp_sum(wsum);
  const float inv = wsum > 0.f ? 1.f / wsum : 0.f;
#pragma unroll
  for (int c = 0; c < MAXC; ++c) store_columns<T>(p, req, head, 4 * (lane + 32 * c), acc[c], inv);
  if (p.o_lse != nullptr && lane == 0)
    p.o_lse[(int64_t)req * p.heads + head] = wsum > 0.f ? mx + logf(wsum) : -INFINITY;
}

template <typename T, int C, int RB, int SPLIT>
__global__ void __launch_bounds__(128, RB * C == 4 ? (C == 1 ? 10 : 9) : 1) stage2_piece_kernel(Stage2Params p) {
  static_assert(SPLIT == 1 || SPLIT == 4, "a warp or the whole block per item");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned item = SPLIT == 1 ? blockIdx.x * 4 + warp : blockIdx.x;
  if (item >= p.items) return;
  const int req = (int)(item / p.pieces), piece = (int)(item - req * p.pieces);
  const int off = p.r2v_offs[req], n_all = p.r2v_lens[req];
  // this warp's rows [r0, r1) of the request's
  const int share = (n_all + SPLIT - 1) / SPLIT;
  const int r0 = SPLIT == 1 ? 0 : min(warp * share, n_all), r1 = SPLIT == 1 ? n_all : min(r0 + share, n_all);
  int ids = r0 + lane < r1 ? p.r2v_entries[off + r0 + lane] : -1;  // plan data: readable before stage 1 is done
  const int width = p.heads << p.dim_shift;                        // floats of a partial row
  int head[C], at[C];                                              // (the element's place in its row)
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int f = 4 * (lane + 32 * (c + C * piece));
    head[c] = f < width ? f >> p.dim_shift : -1;
    at[c] = f & (p.head_dim - 1);
  }
  wait_for_prior_grid();  // the partial buffers are complete from here on
  // Only now may a following stage 1 set itself up under this kernel: let in before stage 1 was over, its CTAs were placed
  // around that one's last ones, several to an SM beside idle SMs, and left this kernel's blocks the rest (64 requests on
  // 4096 tokens, 4/1 heads: 15.9 us per step with the earlier permission, 13.2 with this; four requests in fp32 12.6, 10.7).
  allow_dependent_launch();

  // One pass with a running maximum (as in the online softmax)
  float4 acc[C];
  float mx[C], sum[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    acc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
    mx[c] = -INFINITY;
    sum[c] = 0.f;
  }
  auto raise = [&](int c, float top) {  // to the new maximum
    const float corr = top == -INFINITY ? 1.f : expf(mx[c] - top);  // 0 for the first rows
    mx[c] = top;
    sum[c] *= corr;
    scale(acc[c], corr);
  };
  auto weight = [&](float lse, float top) { return lse > -INFINITY ? expf(lse - top) : 0.f; };  // -inf LSE marks an empty partial
  auto add = [&](int c, float w, const float4& x) {
    acc[c].x = fmaf(w, x.x, acc[c].x);
    acc[c].y = fmaf(w, x.y, acc[c].y);
    acc[c].z = fmaf(w, x.z, acc[c].z);
    acc[c].w = fmaf(w, x.w, acc[c].w);
  };
  for (int base = r0; base < r1; base += 32) {
    const int cnt = min(32, r1 - base);
    int my = -1;
    if (lane < cnt) {
      if (ids >= 0 && ids < p.num_partial_rows)
        my = ids;
      else
        flag_error(FT_DEV_BAD_ROW_INDEX);
    }
    ids = base + 32 + lane < r1 ? p.r2v_entries[off + base + 32 + lane] : -1;  // the next 32 travel under these rows
    for (int i0 = 0; i0 < cnt; i0 += RB) {
      float4 x[RB][C];
      float lse[RB][C];
#pragma unroll
      for (int r = 0; r < RB; ++r) {
        const int row = __shfl_sync(0xffffffffu, my, (i0 + r) & 31);
        const bool ok = i0 + r < cnt && row >= 0;
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const bool load = ok && head[c] >= 0;
          const float* src = p.mid_o + (int64_t)row * p.mo_s0 + (int64_t)head[c] * p.mo_s1 + at[c];
          lse[r][c] = load ? __ldcg(p.mid_lse + (int64_t)row * p.ml_s0 + head[c]) : -INFINITY;
          x[r][c] = load ? __ldcg(reinterpret_cast<const float4*>(src)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
#pragma unroll
      for (int c = 0; c < C; ++c) {
        float top = mx[c];
#pragma unroll
        for (int r = 0; r < RB; ++r) top = fmaxf(top, lse[r][c]);
        raise(c, top);
#pragma unroll
        for (int r = 0; r < RB; ++r) {
          const float w = weight(lse[r][c], top);
          sum[c] += w;
          if (w != 0.f) add(c, w, x[r][c]);
        }
      }
    }
  }
  if constexpr (SPLIT > 1) {  // the warps' partial merges, once more the same way
    __shared__ float4 acc_of[SPLIT][32 * C];
    __shared__ float2 mx_sum_of[SPLIT][32 * C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      acc_of[warp][lane + 32 * c] = acc[c];
      mx_sum_of[warp][lane + 32 * c] = make_float2(mx[c], sum[c]);
    }
    __syncthreads();
    if (warp > 0) return;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      float2 part[SPLIT];
      float top = -INFINITY;
#pragma unroll
      for (int w = 0; w < SPLIT; ++w) {
        part[w] = mx_sum_of[w][lane + 32 * c];
        top = fmaxf(top, part[w].x);
      }
      mx[c] = top;
      sum[c] = 0.f;
      acc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < SPLIT; ++w) {
        const float f = weight(part[w].x, top);
        if (f == 0.f) continue;
        sum[c] = fmaf(f, part[w].y, sum[c]);
        add(c, f, acc_of[w][lane + 32 * c]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < C; ++c) {
    if (head[c] < 0) continue;
    const float inv = sum[c] > 0.f ? 1.f / sum[c] : 0.f;
    store_columns<T>(p, req, head[c], at[c], acc[c], inv);
    if (p.o_lse != nullptr && at[c] == 0)
      p.o_lse[(int64_t)req * p.heads + head[c]] = sum[c] > 0.f ? mx[c] + logf(sum[c]) : -INFINITY;
  }
}

}  // namespace ft
