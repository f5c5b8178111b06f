// Asynchronous-copy building blocks shared by the stage-1 kernels: mbarriers, tiled TMA loads, the proxy fence,
// and the kernel-parameter block that carries the TMA descriptors.
#pragma once

#include <cuda.h>

#include "ft_common.cuh"

namespace ft {

// Kernel parameters of the kernels that use TMA: the common ones plus the descriptors of the K and V buffers
// ([rows, kv heads, head_dim], box 64 x 1 x 64 elements, 128-byte swizzle).  has_tma == 0: gather only.
struct alignas(64) TcParams {
  CUtensorMap k_map;
  CUtensorMap v_map;
  CUtensorMap q_map;       // [batch, heads, head_dim], box 64 x q_box_rows x 1: one request
  CUtensorMap q_map_tile;  // same tensor, box 64 x G x 128 / G: a whole Q tile of consecutive requests
  CUtensorMap k_rows_map;  // K and V as [rows, all heads' elements], box 64 x 1: rows picked one by one (tile::gather4)
  CUtensorMap v_rows_map;
  Stage1Params p;
  int has_tma;
  int has_gather4;    // the two row maps are valid
  int q_box_rows;     // 0: gather Q with cp.async (group size above 128, or no descriptor)
  unsigned int* sched;  // persistent kernel: {tasks claimed beyond the first per CTA, CTAs finished}, zero between launches
};

// the same for a launch whose few-row tasks read slabs by TMA (head_dim 256)
struct SlabParams : TcParams {
  CUtensorMap k_slab_map;  // K and V like k_map, box 64 x 1 x 16
  CUtensorMap v_slab_map;
  int has_slabs;
};

// the common parameters of any parameter block
__device__ __forceinline__ const Stage1Params& stage1_of(const Stage1Params& p) { return p; }
__device__ __forceinline__ const Stage1Params& stage1_of(const TcParams& tp) { return tp.p; }

__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
// announces transaction bytes without arriving
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
// the barrier gets one arrival when all earlier cp.async copies of this thread have landed
__device__ __forceinline__ void mbar_arrive_on_cp_async(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
}
// the same for a barrier that does not count on this thread: one more arrival is owed, and made by the copies
__device__ __forceinline__ void mbar_arrive_after_cp_async(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::
          "r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}

// four rows r0..r3 of a 2-D map whose box is one row, 64 elements from column c0, to 4 x 128 bytes at dst (swizzled by address)
__device__ __forceinline__ void tma_gather4(uint32_t dst, const CUtensorMap* map, int c0, int r0, int r1, int r2, int r3, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];\n" ::
          "r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(r0), "r"(r1), "r"(r2), "r"(r3), "r"(bar)
      : "memory");
}

// Bounded wait for the phase of `bar` with the given parity: false after `limit` probes.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int limit) {
  for (int it = 0; it < limit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// The same by a whole warp, with one answer for all lanes: "no" if any lane's probes have run out (a barrier that completes
// at the limit would else split the warp, and its next shuffle would wait for lanes that have left).
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, int limit) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, limit));
}

}  // namespace ft
