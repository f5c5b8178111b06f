// One packed query row of a task by one warp, in scalar fp32 arithmetic: lanes span the head dimension and the row's
// tokens are walked four per step (their row ids, then their K rows, are independent loads in flight together) with a
// warp-shuffle online softmax.  The scalar kernel is made of it; the tiled kernels fall back to it for single rows.
#pragma once

#include "ft_common.cuh"

namespace ft {

// Row `prow` (request `req`, query head `head`) over the chunk tokens [r_lo, r_hi): writes its partial row and its LSE.
// ids / id_lim: the chunk's row ids; kbase / vbase: the K and V rows of the head's KV head.
template <typename T>
__device__ __forceinline__ void attend_row(const Stage1Params& p, const int32_t* ids, const int id_lim, const T* __restrict__ kbase,
                                           const T* __restrict__ vbase, const int64_t prow, const int req, const int head,
                                           const int r_lo, const int r_hi) {
  constexpr int MAXJ = 8;  // 8 x 32 lanes = head_dim up to 256
  constexpr int TB = 4;    // tokens per step (more in flight per step measured slower: register pressure)
  const int lane = threadIdx.x & 31, D = p.head_dim;
  const T* __restrict__ qp = reinterpret_cast<const T*>(p.q) + (int64_t)req * p.q_s0 + (int64_t)head * p.q_s1;
  float qreg[MAXJ], acc[MAXJ];
#pragma unroll
  for (int j = 0; j < MAXJ; ++j) {
    const int d = lane + 32 * j;
    qreg[j] = d < D ? to_float<T>(qp[d]) : 0.f;
    acc[j] = 0.f;
  }
  float m = -INFINITY, l = 0.f;
  for (int t0 = r_lo; t0 < r_hi; t0 += TB) {
    int rowid[TB];
    float s[TB];
    bool bad = false;  // flagged once after the loads: an atomic between them would serialise them
#pragma unroll
    for (int u = 0; u < TB; ++u) {
      int64_t idx = -1;
      if (t0 + u < r_hi) {
        if (t0 + u < id_lim) idx = ids[t0 + u];
        if (idx < 0 || idx >= p.kv_rows) {
          bad = true;
          idx = -1;
        }
      }
      rowid[u] = (int)idx;
    }
    if (bad && lane == 0) flag_error(FT_DEV_BAD_KV_INDEX);
#pragma unroll
    for (int u = 0; u < TB; ++u) {
      float part = 0.f;
      if (rowid[u] >= 0) {
        const T* __restrict__ kp = kbase + (int64_t)rowid[u] * p.k_s0;
#pragma unroll
        for (int j = 0; j < MAXJ; ++j) {
          const int d = lane + 32 * j;
          if (d < D) part = fmaf(qreg[j], to_float<T>(kp[d]), part);
        }
      }
      s[u] = part;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int u = 0; u < TB; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
    }
    float m_new = m;
#pragma unroll
    for (int u = 0; u < TB; ++u) {
      s[u] = rowid[u] >= 0 ? s[u] * p.sm_scale : -INFINITY;  // scale after the dot, in fp32 (fasttree.py:376)
      m_new = fmaxf(m_new, s[u]);
    }
    if (m_new == -INFINITY) continue;  // nothing valid yet
    const float corr = expf(m - m_new);
    l *= corr;
#pragma unroll
    for (int j = 0; j < MAXJ; ++j) acc[j] *= corr;
#pragma unroll
    for (int u = 0; u < TB; ++u) {
      if (rowid[u] < 0) continue;
      const float pr = expf(s[u] - m_new);
      l += pr;
      // the reference casts the probabilities to V's type before P*V (fasttree.py:391)
      const float pv = to_float<T>(from_float<T>(pr));
      const T* __restrict__ vp = vbase + (int64_t)rowid[u] * p.v_s0;
#pragma unroll
      for (int j = 0; j < MAXJ; ++j) {
        const int d = lane + 32 * j;
        if (d < D) acc[j] = fmaf(pv, to_float<T>(vp[d]), acc[j]);
      }
    }
    m = m_new;
  }
  const float inv = l > 0.f ? 1.f / l : 0.f;
  float* __restrict__ op = p.mid_o + prow * p.mo_s0 + (int64_t)head * p.mo_s1;
#pragma unroll
  for (int j = 0; j < MAXJ; ++j) {
    const int d = lane + 32 * j;
    if (d < D) op[d] = acc[j] * inv;
  }
  if (lane == 0) p.mid_lse[prow * p.ml_s0 + head] = l > 0.f ? logf(l) + m : -INFINITY;
}

// A row that attends to part of its chunk only (a group of short nodes) still has P = 0 multiplied by the other parts' V
// rows in the tiled kernels, and 0 x Inf is NaN: one request's overflowed V row would reach the requests it is grouped
// with.  Such a kernel looks whether a narrowed row came out finite and has those that did not computed here, from their
// own tokens alone, over the partial row it has written.  All lanes of a warp; `row`: packed row of the task.
// The look costs the tcgen05 kernel 16 packed FMAs per 32 columns (its normalisation is packed as well, to pay for them):
// search tree of 1024 requests 127.9 -> 128.1 us, 512 leaves at head_dim 64 36.2 -> 36.4, prefix of 64 requests 27.4 ->
// 27.4; with a second pass over the staged rows 129.2, 36.5 and 27.3.
template <typename T>
__device__ __noinline__ void redo_narrowed_row(const Stage1Params& p, const int kvh, const int q_off, const int kv_off, const int kv_len,
                                               const int row) {
  const int slot = row / p.group;
  const int64_t prow = (int64_t)q_off + slot;
  if (prow < 0 || prow >= p.num_partial_rows) return;
  const int req = p.q_entries[prow];
  if (req < 0 || req >= p.batch) return;
  __syncwarp();  // the warp's own stores to this partial row come first
  attend_row<T>(p, kv_ids_base(p, kv_off), kv_ids_limit(p, kv_off, kv_len),
                reinterpret_cast<const T*>(p.k) + (int64_t)kvh * p.k_s1, reinterpret_cast<const T*>(p.v) + (int64_t)kvh * p.v_s1,
                prow, req, kvh * p.group + row - slot * p.group, max(p.q_ranges[2 * prow], 0), min(p.q_ranges[2 * prow + 1], kv_len));
}

}  // namespace ft
