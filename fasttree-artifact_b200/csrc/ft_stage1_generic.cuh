// Stage 1, scalar fp32 kernel: any storage type, any head_dim <= 256.
//
// One CTA per (vnode, kv head), as in the reference launch grid
// (kernel_bench/fasttree.py:448-451), and block of four query rows, one per warp
// (attend_row; packed row = request slot x group member): the rows of a task
// share nothing here, so no step waits for the task that the plan gave the most
// of them.  It is the correctness
// path for unusual head sizes, types and layouts; the 16-bit cases of head_dim
// 64, 128 and 256 go to the tensor-core kernels, fp32 at 64 and 128 to the tiled
// fp32 kernel.
#pragma once

#include "ft_common.cuh"
#include "ft_stage1_row.cuh"

namespace ft {

template <typename T>
__global__ void __launch_bounds__(128) stage1_generic_kernel(Stage1Params p) {
  allow_dependent_launch();
  wait_for_prior_grid();  // nothing of the preceding kernel's is read or overwritten before this
  const int vn = blockIdx.x + p.node_offset;
  const int kvh = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q_off = p.q_offs[vn], q_len = p.q_lens[vn];
  const int kv_off = p.kv_offs[vn], kv_len = p.kv_lens[vn];
  const int G = p.group;
  const int rows = q_len * G;
  const int32_t* ids = kv_ids_base(p, kv_off);
  const int id_lim = kv_ids_limit(p, kv_off, max(kv_len, 0));
  const T* __restrict__ kbase = reinterpret_cast<const T*>(p.k) + (int64_t)kvh * p.k_s1;
  const T* __restrict__ vbase = reinterpret_cast<const T*>(p.v) + (int64_t)kvh * p.v_s1;

  for (int row = warp + 4 * (int)blockIdx.z; row < rows; row += 4 * (int)gridDim.z) {
    const int slot = row / G, g = row - slot * G;
    const int64_t prow = (int64_t)q_off + slot;
    if (prow < 0 || prow >= p.num_partial_rows) {
      if (lane == 0) flag_error(FT_DEV_BAD_ROW_INDEX);
      continue;
    }
    const int req = p.q_entries[prow];
    if (req < 0 || req >= p.batch) {
      if (lane == 0) flag_error(FT_DEV_BAD_Q_INDEX);
      continue;
    }
    const int head = kvh * G + g;
    // the chunk tokens [r_lo, r_hi) this row attends to: the whole chunk unless the plan narrows it
    int r_lo = 0, r_hi = kv_len;
    if (p.q_ranges != nullptr) {
      r_lo = max(p.q_ranges[2 * prow], 0);
      r_hi = min(p.q_ranges[2 * prow + 1], kv_len);
    }
    attend_row<T>(p, ids, id_lim, kbase, vbase, prow, req, head, r_lo, r_hi);
  }
}

}  // namespace ft
