// Stage 1 for tasks with few query rows where there are many of them: two tasks
// per CTA.  Same arithmetic as the one-task kernel (ft_stage1_narrow.cuh: tensor
// cores swapped, tokens on the M side), at head_dim 64, 128 and 256.
//
// Four warps run a task (a "body"); a CTA holds two bodies with a task each, or
// one of eight warps.  Warp w owns tokens [16w, 16w+16) of every 64 (128) and
// streams them through a ring of its own: slabs of 16 K rows and 16 V rows in
// turn, NS slabs deep.  Nothing in the token loop is shared between warps, so a
// warp waits for its own copies only; the (max, sum, O) partials are merged
// through shared memory at the end.
//
// Slabs arrive by 16-byte cp.async copies, one commit group each; at head_dim
// 256 slabs of consecutive rows by TMA (boxes of 16 rows), with an mbarrier per
// ring slot.  Both ways were measured at both sizes: 60 leaves of 1500 tokens,
// 16/8 heads of 256, 154 us with copies and 125 with TMA; 64 requests of 256
// tokens on 4096, 32/8 heads of 128, 25.0 with copies and 26.3 with TMA, whose
// test for consecutive rows and barrier arrivals weigh more on the smaller slab.
//
// What bounds a short task is the chain in front of its first slab (table entries
// -> row ids -> rows: three dependent round trips, about 4 us) and its epilogue,
// during which its slot of the SM streams nothing.  Two bodies per CTA put four
// tasks on an SM instead of two, each with half of the shared memory, so that one
// task's start-up runs under the others' streaming.
//
// The price is 128 registers per thread: the two-block body (9 to 16 rows) spills
// at head_dim 128 (72 bytes stored / 172 loaded per thread, 100 / 212 in the fused
// kernel), which is why a plan with many such tasks keeps one per CTA.
#pragma once

#include "ft_async.cuh"
#include "ft_common.cuh"
#include "ft_stage1_mma.cuh"
#include "ft_stage1_narrow.cuh"
#include "ft_stage1_row.cuh"

namespace ft {

template <int D, int NQ, int NS>
struct SlabCfg {
  static constexpr int ROWS = 8 * NQ;               // query rows per pass
  static constexpr int ROWB = D * 2;                // bytes of one Q / K / V row
  static constexpr int CPR = D / 8, RPI = 32 / CPR; // 16-byte chunks per row, rows per warp instruction
  static constexpr int SLAB = 16;                   // tokens of a slab
  static constexpr int SLAB_BYTES = SLAB * ROWB;    // D / 64 blocks of [16 tokens][128 B]
  static constexpr int Q_BYTES = ROWS * ROWB;
  static constexpr int RING_BYTES = NS * SLAB_BYTES;  // of one warp
  static constexpr int OSTRIDE = D + 4;
  static constexpr int bytes(int warps) { return Q_BYTES + warps * (RING_BYTES + NS * 8); }  // Q, rings, their mbarriers
  static constexpr int WAIT_LIMIT = 1 << 16;
  static constexpr bool TMA = D == 256;              // slabs of consecutive rows by TMA
  static_assert(ROWS * OSTRIDE * 4 + 2 * ROWS * 4 <= RING_BYTES, "the partials are staged where the rings were");
  static_assert(Q_BYTES % 1024 == 0 && SLAB_BYTES % 1024 == 0, "swizzled slabs sit on 1024-byte boundaries");
  // the 16-byte chunks of a row are XOR-swizzled by the row: conflict-free for ldmatrix and 16-byte copies
  __device__ static __forceinline__ uint32_t swzq(int row, int chunk) {
    return static_cast<uint32_t>(row * ROWB + ((chunk ^ (row & 7)) << 4));
  }
  __device__ static __forceinline__ uint32_t swz(int row, int chunk) {
    return static_cast<uint32_t>((chunk >> 3) * (SLAB * 128) + row * 128 + (((chunk & 7) ^ (row & 7)) << 4));
  }
};

// Ring depth with two bodies in a CTA: 48 KB of slabs per body at head_dim 64 and 128 (two CTAs per SM), 96 KB at 256 (one)
template <int D>
struct PairCfg {
  static constexpr int NS = D == 64 ? 6 : 3;
  static constexpr int MAX_NQ = D == 256 ? 1 : 2;     // 128 accumulators per thread do not fit: 9 to 16 rows take two passes
  static constexpr int BODY_BYTES = (SlabCfg<D, MAX_NQ, NS>::bytes(4) + 1023) / 1024 * 1024;
  static constexpr int SMEM_BYTES = 2 * BODY_BYTES;
  static_assert(SlabCfg<D, MAX_NQ, NS>::bytes(8) <= SMEM_BYTES, "eight warps on one task");
  static constexpr int THREADS = 256;
  static_assert(SMEM_BYTES <= (D == 256 ? 232448 : 115712), "two CTAs per SM, one at head_dim 256");
};

// Params: SlabParams at head_dim 256, any parameter block below; nw: warps of the body, 4 or 8 (threads tid of 32 nw);
// barrier: a hardware barrier of its own
template <typename T, int D, int NQ, int NS, typename Params>
__device__ __forceinline__ void slab_body(const Params& tp, uint8_t* smem, const int tid, const int nw, const int barrier,
                                            const int kvh, const int q_off, const int q_len, const int kv_off, const int kv_len) {
  using N = SlabCfg<D, NQ, NS>;
  const Stage1Params& p = stage1_of(tp);
  constexpr bool Q_IN_REGS = NQ == 1 && D <= 128;
  const uint32_t q_sm = smem_u32(smem);
  float* epi_o = reinterpret_cast<float*>(smem + N::Q_BYTES);
  float* epi_m = epi_o + nw * N::ROWS * N::OSTRIDE;
  float* epi_l = epi_m + nw * N::ROWS;

  const int warp = tid >> 5, lane = tid & 31;
  const int g8 = lane >> 2, t4 = lane & 3;
  const int G = p.group;
  const int rows = q_len * G;
  if (rows <= 0) return;
  if (tid == 0) FT_TL_MARK(0);
  const float scale2 = p.sm_scale * 1.4426950408889634f;
  const uint32_t ring = q_sm + N::Q_BYTES + warp * N::RING_BYTES;
  auto body_sync = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(barrier), "r"(32 * nw) : "memory"); };

  // the same, and whether any thread of the body says yes
  auto body_any = [&](bool mine) {
    uint32_t any;
    asm volatile("{\n\t.reg .pred a, b;\n\tsetp.ne.u32 a, %1, 0;\n\tbar.red.or.pred b, %2, %3, a;\n\tselp.u32 %0, 1, 0, b;\n\t}\n"
                 : "=r"(any) : "r"((uint32_t)mine), "r"(barrier), "r"(32 * nw) : "memory");
    return any != 0u;
  };

  // row ids past the end of the table are a plan error: flagged once, those tokens become padding
  const int id_lim = kv_ids_limit(p, kv_off, kv_len);
  const int32_t* ids = kv_ids_base(p, kv_off);
  if (id_lim < kv_len && tid == 0) flag_error(FT_DEV_BAD_KV_INDEX);
  const uint32_t row_lim = (uint32_t)(p.kv_rows < 0x7fffffffLL ? p.kv_rows : 0x7fffffffLL);
  const int ld_c = lane % N::CPR, ld_r = lane / N::CPR;
  const T* kbase = reinterpret_cast<const T*>(p.k) + (int64_t)kvh * p.k_s1 + ld_c * 8;
  const T* vbase = reinterpret_cast<const T*>(p.v) + (int64_t)kvh * p.v_s1 + ld_c * 8;
  // this warp's slabs: slab j holds tokens span * j + 16 warp ..
  const int span = 16 * nw;
  const int nslabs = kv_len > 16 * warp ? (kv_len - 16 * warp + span - 1) / span : 0;
  bool bad = false, gathered = false, dead = false;  // (dead: the same in all lanes)
  // one mbarrier per ring slot, one arrival each: lane 0's, with the bytes of a TMA copy or behind the lanes' cp.async copies
  const uint32_t bars = q_sm + N::Q_BYTES + nw * N::RING_BYTES + warp * NS * 8;
  if (N::TMA && lane == 0) {
#pragma unroll
    for (int i = 0; i < NS; ++i) mbar_init(bars + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncwarp();
  // Row ids of slabs 2b and 2b + 1, one per lane; -1 past the end of the chunk (padding).  Loaded two pairs ahead: a plain
  // load next to a full ring of copies returns only after those.
  auto fetch_ids = [&](int b) {
    const int pos = span * (2 * b + (lane >> 4)) + 16 * warp + (lane & 15);
    return pos < id_lim ? __ldg(ids + pos) : -1;
  };
  // units issued and consumed so far: unit u = (slab u / 2, K or V) takes ring slot u % NS for the (u / NS)-th time
  int slot_issue = 0, slot_use = 0, pending = 0;
  uint32_t phase_use = 0;
  auto wait_unit = [&]() {
    if constexpr (!N::TMA) {
      cp_async_wait<NS - 1>();
      __syncwarp();
    } else if (pending > 0) {  // (nothing pending: a wait has run out, nothing is issued any more)
      --pending;
      if (!mbar_wait_warp(bars + 8 * slot_use, phase_use, N::WAIT_LIMIT)) {
        dead = true;
        if (lane == 0) flag_error(FT_DEV_WAIT_TIMEOUT);
      }
    }
    const uint32_t at = ring + slot_use * N::SLAB_BYTES;
    if (++slot_use == NS) {
      slot_use = 0;
      phase_use ^= 1;
    }
    return at;
  };

  for (int row0 = 0; row0 < rows; row0 += N::ROWS) {
    int id_cur = fetch_ids(0), id_nxt = fetch_ids(1);  // the K/V row ids travel while the request ids below are fetched
    // ---- request ids first (independent loads), then the copies
    constexpr int TPP = 128 / N::CPR, QPASSES = (N::ROWS + TPP - 1) / TPP;
    int64_t q_src[QPASSES];
    const int q_c = tid % N::CPR, q_r = tid / N::CPR;
    bool narrowed = false;
#pragma unroll
    for (int ps = 0; ps < QPASSES; ++ps) {
      q_src[ps] = -1;
      const int r = ps * TPP + q_r;
      const int prow = row0 + r;
      if (r < N::ROWS && prow < rows && tid < 128) {
        const int slot = prow / G, gg = prow - slot * G;
        const int64_t part = (int64_t)q_off + slot;
        if (part >= 0 && part < p.num_partial_rows) {
          const int req = p.q_entries[part];
          if (req >= 0 && req < p.batch)
            q_src[ps] = (int64_t)req * p.q_s0 + (int64_t)(kvh * G + gg) * p.q_s1 + q_c * 8;
          else
            flag_error(FT_DEV_BAD_Q_INDEX);
        } else {
          flag_error(FT_DEV_BAD_ROW_INDEX);
        }
      }
    }
    // A row that attends to part of the chunk only: no splitter puts one into a few-row task, so such a pass is left to the
    // scalar routine, row by row (p.q_ranges is the same for all warps, and so is the answer).
    if (p.q_ranges != nullptr) {
      const int row_end = min(rows, row0 + N::ROWS), last_slot = (row_end - 1) / G;
      const int64_t part = (int64_t)q_off + row0 / G + lane;
      if (row0 / G + lane <= last_slot && part >= 0 && part < p.num_partial_rows)
        narrowed = p.q_ranges[2 * part] > 0 || p.q_ranges[2 * part + 1] < kv_len;
      if (__any_sync(0xffffffffu, narrowed)) {
        for (int r = row0 + warp; r < row_end; r += nw) redo_narrowed_row<T>(p, kvh, q_off, kv_off, kv_len, r);
        continue;
      }
    }
#pragma unroll
    for (int ps = 0; ps < QPASSES; ++ps) {
      const int r = ps * TPP + q_r;
      if (r < N::ROWS && tid < 128)
        cp_async16_zfill(q_sm + N::swzq(r, q_c), reinterpret_cast<const T*>(p.q) + (q_src[ps] >= 0 ? q_src[ps] : 0), q_src[ps] >= 0);
    }
    cp_async_commit();
    if (tid == 0) FT_TL_MARK(1);

    int u_issue = 0;
    int first = -1;      // pool row of the lane's slab if its 16 rows are consecutive, else -1
    auto look_at_ids = [&](int b) {  // the pair of slabs in id_cur
      const int pos = span * (2 * b + (lane >> 4)) + 16 * warp + (lane & 15);
      bad |= pos < id_lim && (uint32_t)id_cur >= row_lim;
      if constexpr (N::TMA) {
        first = __shfl_sync(0xffffffffu, id_cur, lane & 16);
        const uint32_t run = __ballot_sync(0xffffffffu, id_cur == first + (lane & 15) && first >= 0 && (uint32_t)first + 16 <= row_lim);
        if (!tp.has_slabs || ((run >> (lane & 16)) & 0xffffu) != 0xffffu) first = -1;
      }
    };
    auto issue = [&]() {
      const int j = u_issue >> 1;
      if (j >= nslabs || dead) {
        if constexpr (!N::TMA) cp_async_commit();  // the groups are counted
        return;
      }
      const bool is_v = (u_issue & 1) != 0;
      const uint32_t dst = ring + slot_issue * N::SLAB_BYTES, full = bars + 8 * slot_issue;
      const int row0_of = N::TMA ? __shfl_sync(0xffffffffu, first, (j & 1) * 16) : -1;
      if (row0_of >= 0) {
        if constexpr (N::TMA) {
          if (lane == 0) {
            mbar_arrive_expect_tx(full, N::SLAB_BYTES);
#pragma unroll
            for (int h = 0; h < D / 64; ++h)
              tma_load_3d(dst + h * (N::SLAB * 128), is_v ? &tp.v_slab_map : &tp.k_slab_map, 64 * h, kvh, row0_of, full);
          }
        }
      } else {
        const T* base = is_v ? vbase : kbase;
        const int64_t stride = is_v ? p.v_s0 : p.k_s0;
#pragma unroll
        for (int i = 0; i < N::SLAB / N::RPI; ++i) {
          const int r = i * N::RPI + ld_r;
          const uint32_t row = (uint32_t)__shfl_sync(0xffffffffu, id_cur, (j & 1) * 16 + r);
          const bool ok = row < row_lim;
          cp_async16_zfill(dst + N::swz(r, ld_c), base + (int64_t)(ok ? row : 0u) * stride, ok);
        }
        if constexpr (N::TMA) {
          mbar_arrive_after_cp_async(full);  // counts itself in before it arrives, so lane 0's arrival below is the one owed
          __syncwarp();
          if (lane == 0) mbar_arrive(full);
          gathered = true;
        }
      }
      if constexpr (!N::TMA) cp_async_commit();
      ++u_issue;
      ++pending;
      slot_issue = slot_issue + 1 == NS ? 0 : slot_issue + 1;
      if ((u_issue & 3) == 0) {  // the next pair of slabs
        id_cur = id_nxt;
        look_at_ids(u_issue >> 2);
        id_nxt = fetch_ids((u_issue >> 2) + 1);
      }
    };
    // refill: every lane has read the slab just used
    auto refill = [&]() {
      if (N::TMA && gathered) proxy_fence();  // a slot last written by plain copies may be taken by a TMA copy
      __syncwarp();
      issue();
    };
    look_at_ids(0);
#pragma unroll
    for (int u = 0; u < NS; ++u) issue();

    float o_acc[D / 16][NQ][4];
#pragma unroll
    for (int mb = 0; mb < D / 16; ++mb)
#pragma unroll
      for (int nq = 0; nq < NQ; ++nq) o_acc[mb][nq][0] = o_acc[mb][nq][1] = o_acc[mb][nq][2] = o_acc[mb][nq][3] = 0.f;
    float m_run[NQ][2], l_run[NQ][2];
#pragma unroll
    for (int nq = 0; nq < NQ; ++nq) {
      m_run[nq][0] = m_run[nq][1] = -INFINITY;
      l_run[nq][0] = l_run[nq][1] = 0.f;
    }
    cp_async_wait<N::TMA ? 0 : NS>();  // Q, the oldest group (with mbarriers the slabs' plain copies are in none)
    body_sync();
    if (tid == 0) FT_TL_MARK(2);
    // Q^T as the "col" operand: row nq*8+g8, d = 16kk + 2*t4 (+8)
    auto q_frag = [&](int nq, int kk, int half) { return lds32(q_sm + N::swzq(nq * 8 + g8, 2 * kk + half) + 4 * t4); };
    uint32_t qb[Q_IN_REGS ? D / 16 : 1][2];
    if constexpr (Q_IN_REGS) {
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        qb[kk][0] = q_frag(0, kk, 0);
        qb[kk][1] = q_frag(0, kk, 1);
      }
    }

    for (int j = 0; j < nslabs; ++j) {
      const uint32_t k_sm = wait_unit();

      // S^T = K Q^T : two interleaved accumulator chains per row block
      float s[2][NQ][4];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int nq = 0; nq < NQ; ++nq) s[h][nq][0] = s[h][nq][1] = s[h][nq][2] = s[h][nq][3] = 0.f;
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        uint32_t ka[4];
        ldmatrix_x4(ka, k_sm + N::swz((lane & 7) + 8 * ((lane >> 3) & 1), 2 * kk + (lane >> 4)));
#pragma unroll
        for (int nq = 0; nq < NQ; ++nq) {
          if constexpr (Q_IN_REGS)
            mma16816<T>(s[kk & 1][nq], ka, qb[kk][0], qb[kk][1]);
          else
            mma16816<T>(s[kk & 1][nq], ka, q_frag(nq, kk, 0), q_frag(nq, kk, 1));
        }
      }
      refill();

      const int pos_lo = span * j + 16 * warp + g8;  // token of c0,c1; c2,c3 are 8 further
      const bool lo_ok = pos_lo < kv_len, hi_ok = pos_lo + 8 < kv_len;
      uint32_t pb[NQ][2];
      bool rescale = false;
      float corr[NQ][2];
#pragma unroll
      for (int nq = 0; nq < NQ; ++nq) {
        float x0 = (s[0][nq][0] + s[1][nq][0]) * scale2, x1 = (s[0][nq][1] + s[1][nq][1]) * scale2;
        float x2 = (s[0][nq][2] + s[1][nq][2]) * scale2, x3 = (s[0][nq][3] + s[1][nq][3]) * scale2;
        if (!lo_ok) x0 = x1 = -INFINITY;
        if (!hi_ok) x2 = x3 = -INFINITY;
        float ma = fmaxf(x0, x2), mb_ = fmaxf(x1, x3);  // rows 2*t4 and 2*t4+1 over this thread's two tokens
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
          ma = fmaxf(ma, __shfl_xor_sync(0xffffffffu, ma, o));
          mb_ = fmaxf(mb_, __shfl_xor_sync(0xffffffffu, mb_, o));
        }
        const float na = fmaxf(m_run[nq][0], ma), nb = fmaxf(m_run[nq][1], mb_);
        const float sa = na == -INFINITY ? 0.f : na, sb = nb == -INFINITY ? 0.f : nb;
        corr[nq][0] = fast_exp2(m_run[nq][0] - sa);
        corr[nq][1] = fast_exp2(m_run[nq][1] - sb);
        rescale |= (na != m_run[nq][0]) | (nb != m_run[nq][1]);
        m_run[nq][0] = na;
        m_run[nq][1] = nb;
        const float p0 = fast_exp2(x0 - sa), p1 = fast_exp2(x1 - sb);
        const float p2 = fast_exp2(x2 - sa), p3 = fast_exp2(x3 - sb);
        l_run[nq][0] = l_run[nq][0] * corr[nq][0] + p0 + p2;
        l_run[nq][1] = l_run[nq][1] * corr[nq][1] + p1 + p3;
        // (token g8 | g8+8 ; rows 2t4,2t4+1) -> (row g8 ; tokens 2t4,2t4+1 | +8): the B operand of P^T
        pb[nq][0] = movmatrix_trans(pack2<T>(p0, p1));
        pb[nq][1] = movmatrix_trans(pack2<T>(p2, p3));
      }
      if (__any_sync(0xffffffffu, rescale)) {
#pragma unroll
        for (int mb = 0; mb < D / 16; ++mb)
#pragma unroll
          for (int nq = 0; nq < NQ; ++nq) {
            o_acc[mb][nq][0] *= corr[nq][0];
            o_acc[mb][nq][1] *= corr[nq][1];
            o_acc[mb][nq][2] *= corr[nq][0];
            o_acc[mb][nq][3] *= corr[nq][1];
          }
      }
      // O^T += V^T P^T
      const uint32_t v_sm = wait_unit();
#pragma unroll
      for (int mb = 0; mb < D / 16; ++mb) {
        uint32_t va[4];
        ldmatrix_x4_trans(va, v_sm + N::swz((lane & 7) + 8 * (lane >> 4), 2 * mb + ((lane >> 3) & 1)));
#pragma unroll
        for (int nq = 0; nq < NQ; ++nq) mma16816<T>(o_acc[mb][nq], va, pb[nq][0], pb[nq][1]);
      }
      refill();
    }
    if constexpr (!N::TMA) {
      cp_async_wait<0>();
      body_sync();
    } else if (body_any(dead)) {
      // A wait ran out: that warp's copies may still arrive, so nothing is staged over the rings.  The rows left come out
      // as if no token had been seen; the status word says why.
      for (int r = row0 + (tid >> 3); r < rows; r += 4 * nw) {
        const int slot = r / G, head = kvh * G + r - slot * G;
        const int64_t part = (int64_t)q_off + slot;
        if (part < 0 || part >= p.num_partial_rows) continue;
        float4* dst = reinterpret_cast<float4*>(p.mid_o + part * p.mo_s0 + (int64_t)head * p.mo_s1);
        for (int i = tid & 7; i < D / 4; i += 8) dst[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if ((tid & 7) == 0) p.mid_lse[part * p.ml_s0 + head] = -INFINITY;
      }
      return;
    }
    // rings idle: reuse them as the staging area
    if (tid == 0) FT_TL_MARK(6);

    // ---- stage this warp's (max, sum, O^T) partial
#pragma unroll
    for (int nq = 0; nq < NQ; ++nq) {
      float la = l_run[nq][0], lb = l_run[nq][1];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        la += __shfl_xor_sync(0xffffffffu, la, o);
        lb += __shfl_xor_sync(0xffffffffu, lb, o);
      }
      const int r = nq * 8 + 2 * t4;
      float* dst = epi_o + (warp * N::ROWS + r) * N::OSTRIDE + g8;
#pragma unroll
      for (int mb = 0; mb < D / 16; ++mb) {
        dst[mb * 16] = o_acc[mb][nq][0];
        dst[N::OSTRIDE + mb * 16] = o_acc[mb][nq][1];
        dst[mb * 16 + 8] = o_acc[mb][nq][2];
        dst[N::OSTRIDE + mb * 16 + 8] = o_acc[mb][nq][3];
      }
      if (g8 == 0) {
        epi_m[warp * N::ROWS + r] = m_run[nq][0];
        epi_m[warp * N::ROWS + r + 1] = m_run[nq][1];
        epi_l[warp * N::ROWS + r] = la;
        epi_l[warp * N::ROWS + r + 1] = lb;
      }
    }
    body_sync();

    // ---- merge the warps, normalise, write the partial rows
    {
      const int r = tid >> 3, seg = tid & 7;
      const int prow = row0 + r;
      if (r < N::ROWS && prow < rows) {  // the first eight threads per row
        const int slot = prow / G, gg = prow - slot * G;
        const int64_t part = (int64_t)q_off + slot;
        if (part >= 0 && part < p.num_partial_rows) {
          float M = -INFINITY;
          for (int w = 0; w < nw; ++w) M = fmaxf(M, epi_m[w * N::ROWS + r]);
          float L = 0.f;
          float4 out[D / 32];
#pragma unroll
          for (int i = 0; i < D / 32; ++i) out[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
          for (int w = 0; w < nw; ++w) {
            const float mw = epi_m[w * N::ROWS + r];
            const float f = mw == -INFINITY ? 0.f : fast_exp2(mw - M);
            L = fmaf(epi_l[w * N::ROWS + r], f, L);
            const float4* src = reinterpret_cast<const float4*>(epi_o + (w * N::ROWS + r) * N::OSTRIDE);
#pragma unroll
            for (int i = 0; i < D / 32; ++i) {
              const float4 x = src[seg + 8 * i];
              out[i].x = fmaf(f, x.x, out[i].x);
              out[i].y = fmaf(f, x.y, out[i].y);
              out[i].z = fmaf(f, x.z, out[i].z);
              out[i].w = fmaf(f, x.w, out[i].w);
            }
          }
          const float inv = L > 0.f ? 1.f / L : 0.f;
          const int head = kvh * G + gg;
          float4* dst = reinterpret_cast<float4*>(p.mid_o + part * p.mo_s0 + (int64_t)head * p.mo_s1);
#pragma unroll
          for (int i = 0; i < D / 32; ++i)
            dst[seg + 8 * i] = make_float4(out[i].x * inv, out[i].y * inv, out[i].z * inv, out[i].w * inv);
          if (seg == 0)
            p.mid_lse[part * p.ml_s0 + head] = L > 0.f ? (M + log2f(L)) * 0.6931471805599453f : -INFINITY;
        }
      }
    }
    if (row0 + N::ROWS < rows) proxy_fence();  // the staged partials come before the next pass's TMA copies
    body_sync();
  }
  if (bad) flag_error(FT_DEV_BAD_KV_INDEX);
}

__device__ __forceinline__ void prefetch_slab_maps(const SlabParams& tp) {
  if (threadIdx.x == 0 && tp.has_slabs) {
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&tp.k_slab_map)) : "memory");
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&tp.v_slab_map)) : "memory");
  }
}

// One few-row CTA.  FEW_PAIR: its two bodies of four warps take tasks `first` and `first` + 1 (of `tasks`, kv head fastest);
// FEW_EIGHT (head_dim 256): all eight warps take task `first`.  Tasks with at most 8 query rows run the one-block body, the
// others the two-block body (which also loops if a task has more than 16 rows).
template <typename T, int D, typename Params>
__device__ __forceinline__ void pair_cta(const Params& tp, uint8_t* smem, const int form, const int first, const int tasks) {
  using P = PairCfg<D>;
  const Stage1Params& p = stage1_of(tp);
  const bool pair = D != 256 || form == FEW_PAIR;
  const int body = pair ? threadIdx.x >> 7 : 0, task = first + body;
  if (task >= tasks) return;
  const int nw = pair ? 4 : 8, tid = threadIdx.x & (32 * nw - 1);
  int vn, kvh;
  task_of_block(p, task, vn, kvh);
  const int q_off = p.q_offs[vn], q_len = p.q_lens[vn], kv_off = p.kv_offs[vn], kv_len = max(p.kv_lens[vn], 0);
  smem += body * P::BODY_BYTES;
  if (q_len * p.group <= 8 || P::MAX_NQ == 1)
    slab_body<T, D, 1, P::NS>(tp, smem, tid, nw, 3 + body, kvh, q_off, q_len, kv_off, kv_len);
  else
    slab_body<T, D, P::MAX_NQ, P::NS>(tp, smem, tid, nw, 3 + body, kvh, q_off, q_len, kv_off, kv_len);
}

// Few-row tasks alone, two to a CTA (head_dim 256 runs them in the fused kernel: its CTAs of both kinds fill an SM each)
template <typename T, int D>
__global__ void __launch_bounds__(PairCfg<D>::THREADS, 2) stage1_pair_kernel(const __grid_constant__ Stage1Params p) {
  static_assert(D <= 128, "at 256 the fused kernel runs them");
  allow_dependent_launch();
  wait_for_prior_grid();  // nothing of the preceding kernel's is read or overwritten before this
  extern __shared__ __align__(1024) uint8_t smem[];
  FT_TL_BEGIN();
  pair_cta<T, D>(p, smem, FEW_PAIR, 2 * (int)blockIdx.x, p.node_count * p.num_kv_heads);
  FT_TL_END(2);
}

}  // namespace ft
