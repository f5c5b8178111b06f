// Stage 1 for fp32 storage (head_dim 64 or 128): exact fp32 arithmetic on the
// CUDA cores, tiled through shared memory.
//
// One CTA (8 warps) per (vnode, kv head, block of 16 packed query rows).  The KV
// chunk is walked 32 tokens at a time: the tile's K and V rows are gathered by
// row id with 16-byte loads, one tile ahead of the arithmetic (the loads of tile
// t+1 are in flight, in registers, while tile t is computed from shared memory).
//   S[16 x 32]   lane = token, warp w owns rows w and w+8: 2 dot products of length
//                head_dim per thread, Q broadcast from shared memory (two warps per
//                scheduler: the arithmetic of a tile is one dependent chain per warp,
//                and with four warps of four rows a tile took twice as long)
//   softmax      a row's 32 scores sit in the 32 lanes of one warp: shuffles
//   O[16 x D]    thread owns D / 32 adjacent columns of its warp's 2 rows; the
//                probabilities go through shared memory
// Everything in shared memory is read 16 bytes at a time (8 of V at head_dim 64): the K
// tile passes through shared memory once per warp, which bounds a tile's arithmetic, and
// a word at a time the reads' issue did.  With that and the first reads sent off together
// (before: the Q rows, then the row ids, then the K and V rows) stage 1 of 4 requests on
// 512 tokens, 8/2 heads of 128, takes 6.8 us (7.7), of 40 requests of 300 tokens on 500,
// 16/16 heads, 171 (196), of 64 requests of 100 on 1000, 32/8 heads of 64, 66 (79).
// Same conventions as the other stage-1 kernels (kernel_bench/fasttree.py:360-413):
// scores scaled after the dot product, normalised partial output, lse = log(sum) + max;
// optional per-row token ranges; bad indices are skipped and flagged.
#pragma once

#include "ft_common.cuh"
#include "ft_stage1_row.cuh"

namespace ft {

template <int D>
struct F32Cfg {
  static constexpr int ROWS = 16, TILE = 32, THREADS = 256;
  static constexpr int WARPS = THREADS / 32, RPW = ROWS / WARPS;  // rows per warp
  static constexpr int KSTRIDE = D + 4;              // floats between K rows: lane = token 16-byte reads are conflict-free
  static constexpr int Q_FLOATS = ROWS * D, K_FLOATS = TILE * KSTRIDE, V_FLOATS = TILE * D;
  static constexpr int K_OFF = ((Q_FLOATS + 3) / 4) * 4, V_OFF = ((K_OFF + K_FLOATS + 3) / 4) * 4;
  static constexpr int P_OFF = V_OFF + V_FLOATS;     // ROWS x TILE probabilities
  static constexpr int SMEM_BYTES = (P_OFF + ROWS * TILE) * 4;
  static constexpr int C4 = D / 4;                   // float4 chunks per row
  static constexpr int LOADS = TILE * C4 / THREADS;  // float4 loads per thread per operand per tile
};

template <int D>
__global__ void __launch_bounds__(256, D == 64 ? 4 : 3) stage1_f32_kernel(const __grid_constant__ Stage1Params p) {
  using C = F32Cfg<D>;
  allow_dependent_launch();
  wait_for_prior_grid();  // nothing of the preceding kernel's is read or overwritten before this
  extern __shared__ __align__(16) float smem_f32[];
  float* q_s = smem_f32;
  float* k_s = smem_f32 + C::K_OFF;
  float* v_s = smem_f32 + C::V_OFF;
  float* p_s = smem_f32 + C::P_OFF;
  const int vn = blockIdx.x + p.node_offset, kvh = blockIdx.y, row0 = blockIdx.z * C::ROWS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q_off = p.q_offs[vn], q_len = p.q_lens[vn];
  const int kv_off = p.kv_offs[vn], kv_len = max(p.kv_lens[vn], 0);
  const int G = p.group;
  const int rows = min(q_len * G - row0, C::ROWS);
  if (rows <= 0) return;
  // the grid's row blocks come from the caller's request tile: a vnode with more rows than that is a plan error
  if (blockIdx.z == gridDim.z - 1 && q_len * G - row0 > C::ROWS && threadIdx.x == 0) flag_error(FT_DEV_BAD_ROW_INDEX);
  const int32_t* ids = kv_ids_base(p, kv_off);
  const int id_lim = kv_ids_limit(p, kv_off, kv_len);
  const float* kbase = reinterpret_cast<const float*>(p.k) + (int64_t)kvh * p.k_s1;
  const float* vbase = reinterpret_cast<const float*>(p.v) + (int64_t)kvh * p.v_s1;

  // The reads that everything waits for go out together: a thread's row ids of tile 0 and the request ids of its Q rows,
  // then the K, V and Q rows themselves.  (A row's Q float4s: thread tid has number tid % C4 of rows tid / C4 + RPQ u.)
  constexpr int RPQ = C::THREADS / C::C4, QLOADS = C::ROWS / RPQ;
  const int q_c4 = tid % C::C4;
  int q_req[QLOADS];
#pragma unroll
  for (int u = 0; u < QLOADS; ++u) {
    const int r = tid / C::C4 + RPQ * u;
    q_req[u] = -1;
    if (r < rows) {
      const int64_t part = (int64_t)q_off + (row0 + r) / G;
      if (part >= 0 && part < p.num_partial_rows)
        q_req[u] = p.q_entries[part];
      else if (q_c4 == 0)
        flag_error(FT_DEV_BAD_ROW_INDEX);
    }
  }
  // per-thread state: rows warp + WARPS * i
  constexpr int RPW = C::RPW, NW = C::WARPS, CPL = D / 32;  // CPL: columns per lane
  auto load_cols = [](float (&x)[CPL], const float* src) {
    if constexpr (CPL == 4) {
      const float4 y = *reinterpret_cast<const float4*>(src);
      x[0] = y.x, x[1] = y.y, x[2] = y.z, x[3] = y.w;
    } else {
      const float2 y = *reinterpret_cast<const float2*>(src);
      x[0] = y.x, x[1] = y.y;
    }
  };
  float m_run[RPW], l_run[RPW], acc[RPW][CPL];
  int r_lo[RPW], r_hi[RPW];
#pragma unroll
  for (int i = 0; i < RPW; ++i) {
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
#pragma unroll
    for (int j = 0; j < CPL; ++j) acc[i][j] = 0.f;
    r_lo[i] = 0;
    r_hi[i] = kv_len;
    const int r = warp + NW * i;
    if (p.q_ranges != nullptr && r < rows) {
      const int64_t part = (int64_t)q_off + (row0 + r) / G;
      if (part >= 0 && part < p.num_partial_rows) {
        r_lo[i] = max(p.q_ranges[2 * part], 0);
        r_hi[i] = min(p.q_ranges[2 * part + 1], kv_len);
      }
    }
  }

  const int ntiles = (kv_len + C::TILE - 1) / C::TILE;
  float4 kreg[C::LOADS], vreg[C::LOADS];
  // Row ids of tile t (-1: padding), then its rows -> registers (zeros for padding and bad row ids).  A load fetches WPR
  // rows per warp: lane l holds the id of row l % WPR of load l / WPR.  (A register per load, the same in every lane of the
  // row, made the kernel of head_dim 128 spill 28 bytes: 7.2 and 173 us for the first two shapes above.)
  constexpr int WPR = 32 / C::C4;
  int idreg = -1;
  auto fetch_ids = [&](int t) {
    const int pos = t * C::TILE + (lane / WPR) * (C::THREADS / C::C4) + warp * WPR + lane % WPR;
    idreg = lane < WPR * C::LOADS && pos < id_lim ? ids[pos] : -1;
  };
  auto fetch = [&](int t) {
    bool bad = false;
#pragma unroll
    for (int u = 0; u < C::LOADS; ++u) {
      const int i = u * C::THREADS + tid, c4 = i % C::C4;
      const int64_t row = __shfl_sync(0xffffffffu, idreg, u * WPR + lane / C::C4);
      if (row >= 0 && row < p.kv_rows) {
        kreg[u] = __ldg(reinterpret_cast<const float4*>(kbase + row * p.k_s0) + c4);
        vreg[u] = __ldg(reinterpret_cast<const float4*>(vbase + row * p.v_s0) + c4);
      } else {
        bad |= t * C::TILE + i / C::C4 < kv_len;
        kreg[u] = vreg[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    if (bad) flag_error(FT_DEV_BAD_KV_INDEX);
  };
  auto stash = [&]() {
#pragma unroll
    for (int u = 0; u < C::LOADS; ++u) {
      const int i = u * C::THREADS + tid, tok = i / C::C4, c4 = i - tok * C::C4;
      *reinterpret_cast<float4*>(k_s + tok * C::KSTRIDE + 4 * c4) = kreg[u];
      *reinterpret_cast<float4*>(v_s + tok * D + 4 * c4) = vreg[u];
    }
  };

  fetch_ids(0);
  fetch(0);
  if (ntiles > 1) fetch_ids(1);
  // ---- Q rows of this block -> shared memory (zeros for rows past the end or with a bad index)
#pragma unroll
  for (int u = 0; u < QLOADS; ++u) {
    const int r = tid / C::C4 + RPQ * u;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (q_req[u] >= 0 && q_req[u] < p.batch)
      x = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.q) + (int64_t)q_req[u] * p.q_s0 +
                                           (int64_t)(kvh * G + (row0 + r) % G) * p.q_s1 + 4 * q_c4);
    else if (r < rows && q_c4 == 0) {  // a bad row id has been flagged above: no request was read there
      const int64_t part = (int64_t)q_off + (row0 + r) / G;
      if (part >= 0 && part < p.num_partial_rows) flag_error(FT_DEV_BAD_Q_INDEX);
    }
    *reinterpret_cast<float4*>(q_s + r * D + 4 * q_c4) = x;
  }
  for (int t = 0; t < ntiles; ++t) {
    if (t > 0) __syncthreads();  // the previous tile has been consumed
    stash();
    __syncthreads();  // (at t = 0, Q is in place too)
    if (t + 1 < ntiles) {  // in flight during the arithmetic below
      fetch(t + 1);
      if (t + 2 < ntiles) fetch_ids(t + 2);
    }

    // ---- S = Q K^T for this thread's rows and its token
    float s[RPW];
#pragma unroll
    for (int i = 0; i < RPW; ++i) s[i] = 0.f;
    const float4* kr = reinterpret_cast<const float4*>(k_s + lane * C::KSTRIDE);
#pragma unroll 8
    for (int d4 = 0; d4 < C::C4; ++d4) {
      const float4 kv = kr[d4];
#pragma unroll
      for (int i = 0; i < RPW; ++i) {
        const float4 qv = *reinterpret_cast<const float4*>(q_s + (warp + NW * i) * D + 4 * d4);
        s[i] = fmaf(qv.x, kv.x, s[i]);
        s[i] = fmaf(qv.y, kv.y, s[i]);
        s[i] = fmaf(qv.z, kv.z, s[i]);
        s[i] = fmaf(qv.w, kv.w, s[i]);
      }
    }
    // ---- online softmax per row (32 tokens = 32 lanes)
    const int pos = t * C::TILE + lane;
    float pr[RPW];
#pragma unroll
    for (int i = 0; i < RPW; ++i) {
      const bool seen = pos >= r_lo[i] && pos < r_hi[i];
      const float x = seen ? s[i] * p.sm_scale : -INFINITY;
      const float m_new = fmaxf(m_run[i], warp_max(x));
      if (m_new == -INFINITY) {  // nothing valid for this row yet
        pr[i] = 0.f;
        continue;
      }
      const float corr = expf(m_run[i] - m_new);  // 0 while m_run is -inf
      pr[i] = seen ? expf(x - m_new) : 0.f;
      l_run[i] = l_run[i] * corr + warp_sum(pr[i]);
#pragma unroll
      for (int j = 0; j < CPL; ++j) acc[i][j] *= corr;
      m_run[i] = m_new;
    }
    // ---- O += P V
#pragma unroll
    for (int i = 0; i < RPW; ++i) p_s[(warp + NW * i) * C::TILE + lane] = pr[i];
    __syncwarp();
#pragma unroll 2
    for (int t4 = 0; t4 < C::TILE; t4 += 4) {
      float4 w[RPW];
#pragma unroll
      for (int i = 0; i < RPW; ++i) w[i] = *reinterpret_cast<const float4*>(p_s + (warp + NW * i) * C::TILE + t4);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float vv[CPL];
        load_cols(vv, v_s + (t4 + k) * D + CPL * lane);
#pragma unroll
        for (int i = 0; i < RPW; ++i) {
          const float wk = k == 0 ? w[i].x : k == 1 ? w[i].y : k == 2 ? w[i].z : w[i].w;
#pragma unroll
          for (int j = 0; j < CPL; ++j) acc[i][j] = fmaf(wk, vv[j], acc[i][j]);
        }
      }
    }
    __syncwarp();  // before the next tile's probabilities
  }

  // ---- normalise and write the partial rows
  uint32_t todo = 0;
#pragma unroll
  for (int i = 0; i < RPW; ++i) {
    const int r = warp + NW * i;
    if (r >= rows) continue;
    const int prow = row0 + r, slot = prow / G, gg = prow - slot * G;
    const int64_t part = (int64_t)q_off + slot;
    if (part < 0 || part >= p.num_partial_rows) continue;
    const int head = kvh * G + gg;
    const float inv = l_run[i] > 0.f ? 1.f / l_run[i] : 0.f;
    float* op = p.mid_o + part * p.mo_s0 + (int64_t)head * p.mo_s1 + CPL * lane;
    if constexpr (CPL == 4)
      *reinterpret_cast<float4*>(op) = make_float4(acc[i][0] * inv, acc[i][1] * inv, acc[i][2] * inv, acc[i][3] * inv);
    else
      *reinterpret_cast<float2*>(op) = make_float2(acc[i][0] * inv, acc[i][1] * inv);
    if (lane == 0) p.mid_lse[part * p.ml_s0 + head] = l_run[i] > 0.f ? logf(l_run[i]) + m_run[i] : -INFINITY;
    if (r_lo[i] > 0 || r_hi[i] < kv_len) {
      float finite = 0.f;  // 0 x every element: 0, or NaN
#pragma unroll
      for (int j = 0; j < CPL; ++j) finite = fmaf(acc[i][j], 0.f, finite);
      if (__any_sync(0xffffffffu, !(finite == 0.f))) todo |= 1u << i;
    }
  }
#pragma unroll 1
  for (; todo != 0; todo &= todo - 1) redo_narrowed_row<float>(p, kvh, q_off, kv_off, kv_len, row0 + warp + NW * (__ffs(todo) - 1));
}

}  // namespace ft
