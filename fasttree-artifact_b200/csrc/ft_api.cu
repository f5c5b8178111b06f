// C ABI of the tree-attention decode engine: argument validation, kernel
// selection and launches.  Declarations and the mapping to the reference's
// Python entry points are in include/fasttree_b200.h.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <mutex>
#include <utility>
#include <cstdio>
#include <cstring>

#include "fasttree_b200.h"
#include "ft_common.cuh"
#include "ft_stage1_f32.cuh"
#include "ft_stage1_generic.cuh"
#include "ft_stage1_mma.cuh"
#include "ft_stage1_narrow.cuh"
#include "ft_stage1_stream.cuh"
#include "ft_stage1_tc.cuh"
#include "ft_stage2.cuh"

namespace {

thread_local char g_err[512] = "";
std::atomic<int64_t> g_launches{0};
thread_local int64_t t_launches = 0;  // launches issued by this host thread

void count_launch() {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  ++t_launches;
}

// ft_stage1_path_name walks the same selection code as ft_stage1 with launches switched off and collects the
// names of the kernels that would have been launched.
thread_local bool g_dry_run = false;
thread_local char g_kernel_names[160] = "";

bool dry_run(const char* kernel) {
  if (!g_dry_run) return false;
  const size_t used = strlen(g_kernel_names);
  snprintf(g_kernel_names + used, sizeof(g_kernel_names) - used, "%s%s", used ? "+" : "", kernel);
  return true;
}

// Largest dynamic shared memory of a kernel, raised once per device.  Several host threads may make their first
// call at the same time: the flag is atomic and setting the attribute twice is harmless.
struct OncePerDevice {
  std::atomic<bool> done[64];
  OncePerDevice() {
    for (auto& d : done) d.store(false, std::memory_order_relaxed);
  }
};

template <typename Kernel>
cudaError_t raise_smem_limit(OncePerDevice& once, Kernel kernel, int bytes, int* device_out = nullptr) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (device_out != nullptr) *device_out = dev;
  const bool tracked = dev >= 0 && dev < 64;
  if (tracked && once.done[dev].load(std::memory_order_acquire)) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && tracked) once.done[dev].store(true, std::memory_order_release);
  return e;
}

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

#define FT_CUDA_OK(expr)                                                                      \
  do {                                                                                        \
    cudaError_t e_ = (expr);                                                                  \
    if (e_ != cudaSuccess) return fail(FT_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e_)); \
  } while (0)

bool aligned16(const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0; }

int check_common(const ft_decode_args* a) {
  if (a == nullptr) return fail(FT_ERR_INVALID_ARGUMENT, "args is NULL");
  if (a->dtype != FT_F16 && a->dtype != FT_BF16 && a->dtype != FT_F32)
    return fail(FT_ERR_INVALID_ARGUMENT, "dtype %d is not one of FT_F16/FT_BF16/FT_F32", a->dtype);
  if (a->batch < 0 || a->num_qo_heads <= 0 || a->num_kv_heads <= 0 || a->head_dim <= 0)
    return fail(FT_ERR_INVALID_ARGUMENT, "batch/heads/head_dim must be positive (batch %d, hq %d, hkv %d, d %d)",
                a->batch, a->num_qo_heads, a->num_kv_heads, a->head_dim);
  if (a->num_qo_heads % a->num_kv_heads != 0)
    return fail(FT_ERR_INVALID_ARGUMENT, "num_qo_heads %d is not a multiple of num_kv_heads %d", a->num_qo_heads,
                a->num_kv_heads);
  // the reference asserts head_dim in {16,32,64,128,256} (kernel_bench/fasttree.py:439)
  const int d = a->head_dim;
  if (!(d == 16 || d == 32 || d == 64 || d == 128 || d == 256))
    return fail(FT_ERR_UNSUPPORTED, "head_dim %d is not one of 16, 32, 64, 128, 256", d);
  if (a->num_partial_rows < 0) return fail(FT_ERR_INVALID_ARGUMENT, "num_partial_rows is negative");
  if (a->mid_o == nullptr || a->mid_lse == nullptr)
    return fail(FT_ERR_INVALID_ARGUMENT, "mid_o / mid_lse scratch is NULL");
  if (!aligned16(a->mid_o) || a->mid_o_stride0 % 4 != 0 || a->mid_o_stride1 % 4 != 0)
    return fail(FT_ERR_UNSUPPORTED, "mid_o must be 16-byte aligned with strides that are multiples of 4 floats");
  return FT_OK;
}

int check_stage1(const ft_decode_args* a) {
  if (a->q == nullptr || a->k_buffer == nullptr || a->v_buffer == nullptr)
    return fail(FT_ERR_INVALID_ARGUMENT, "q / k_buffer / v_buffer is NULL");
  if (a->kv_rows <= 0) return fail(FT_ERR_INVALID_ARGUMENT, "kv_rows must be positive");
  for (int ph = 0; ph < 2; ++ph)
    if (a->phase_node_nums[ph] < 0 || a->phase_node_offsets[ph] < 0)
      return fail(FT_ERR_INVALID_ARGUMENT, "phase %d: negative vnode count or offset", ph);
  if (a->phase_node_nums[0] + a->phase_node_nums[1] > 0 || a->device_phase_info != nullptr) {
    if (!a->vnode_to_kv_entries || !a->vnode_to_kv_offs || !a->vnode_to_kv_lens || !a->vnode_to_q_entries ||
        !a->vnode_to_q_offs || !a->vnode_to_q_lens)
      return fail(FT_ERR_INVALID_ARGUMENT, "a vnode table pointer is NULL");
    if (a->kv_entries_len <= 0) return fail(FT_ERR_INVALID_ARGUMENT, "kv_entries_len must be positive");
  }
  if (a->num_kv_heads > 65535) return fail(FT_ERR_UNSUPPORTED, "more than 65535 kv heads");
  if (((int64_t)a->phase_node_nums[0] + a->phase_node_nums[1]) * a->num_kv_heads > 0x7fffffffLL)
    return fail(FT_ERR_TOO_LARGE, "vnodes x kv heads exceeds the grid limit");
  return FT_OK;
}

// Can the warp-MMA kernel take these arguments?  Returns a reason or NULL.
const char* mma_obstacle(const ft_decode_args* a) {
  if (a->dtype == FT_F32) return "fp32 inputs";
  if (a->head_dim != 64 && a->head_dim != 128 && a->head_dim != 256) return "head_dim not 64, 128 or 256";
  if (!aligned16(a->q) || !aligned16(a->k_buffer) || !aligned16(a->v_buffer)) return "q/k/v not 16-byte aligned";
  if (a->q_stride0 % 8 || a->q_stride1 % 8 || a->k_stride0 % 8 || a->k_stride1 % 8 || a->v_stride0 % 8 ||
      a->v_stride1 % 8)
    return "a q/k/v stride is not a multiple of 8 elements";
  // partial rows are written 16 bytes at a time
  if (!aligned16(a->mid_o) || a->mid_o_stride0 % 4 || a->mid_o_stride1 % 4) return "mid_o rows not 16-byte aligned";
  return nullptr;
}

int pick_path(const ft_decode_args* a) {
  const char* why = mma_obstacle(a);
  if (a->device_phase_info != nullptr) {  // only the persistent kernel has a grid that does not depend on the plan
    if (a->path != FT_PATH_AUTO && a->path != FT_PATH_PERSIST)
      return fail(FT_ERR_UNSUPPORTED, "device_phase_info needs path AUTO or PERSIST, got %d", a->path);
    if (why != nullptr || a->head_dim != 128)
      return fail(FT_ERR_UNSUPPORTED, "device_phase_info needs the persistent kernel: 16-bit types, head_dim 128, aligned buffers%s%s",
                  why ? "; " : "", why ? why : "");
    return FT_PATH_PERSIST;
  }
  if (a->path == FT_PATH_GENERIC) return FT_PATH_GENERIC;
  if (a->path == FT_PATH_MMA || a->path == FT_PATH_TCGEN05 || a->path == FT_PATH_MMA_WIDE || a->path == FT_PATH_STREAM ||
      a->path == FT_PATH_PERSIST) {
    if (why != nullptr) return fail(FT_ERR_UNSUPPORTED, "tensor-core path unavailable: %s", why);
    if (a->path == FT_PATH_PERSIST && a->head_dim != 128)
      return fail(FT_ERR_UNSUPPORTED, "the persistent kernel needs head_dim 128, got %d", a->head_dim);
    if (a->path != FT_PATH_TCGEN05 && a->head_dim == 256)
      return fail(FT_ERR_UNSUPPORTED, "head_dim 256 runs on paths AUTO, TCGEN05 and GENERIC only");
    return a->path;
  }
  if (a->path != FT_PATH_AUTO) return fail(FT_ERR_INVALID_ARGUMENT, "unknown path %d", a->path);
  return why == nullptr ? FT_PATH_AUTO : FT_PATH_GENERIC;
}

ft::Stage1Params stage1_params(const ft_decode_args* a) {
  ft::Stage1Params p;
  p.q = a->q;
  p.k = a->k_buffer;
  p.v = a->v_buffer;
  p.kv_entries = a->vnode_to_kv_entries;
  p.kv_offs = a->vnode_to_kv_offs;
  p.kv_lens = a->vnode_to_kv_lens;
  p.q_entries = a->vnode_to_q_entries;
  p.q_offs = a->vnode_to_q_offs;
  p.q_lens = a->vnode_to_q_lens;
  p.q_ranges = a->vnode_q_kv_ranges;
  p.dev_phase = a->device_phase_info;
  p.kv_entries_aux = a->vnode_to_kv_entries_aux;
  p.kv_entries_aux_len = a->vnode_to_kv_entries_aux != nullptr ? a->kv_entries_aux_len : 0;
  p.mid_o = a->mid_o;
  p.mid_lse = a->mid_lse;
  p.q_s0 = a->q_stride0;
  p.q_s1 = a->q_stride1;
  p.k_s0 = a->k_stride0;
  p.k_s1 = a->k_stride1;
  p.v_s0 = a->v_stride0;
  p.v_s1 = a->v_stride1;
  p.mo_s0 = a->mid_o_stride0;
  p.mo_s1 = a->mid_o_stride1;
  p.ml_s0 = a->mid_lse_stride0;
  p.kv_rows = a->kv_rows;
  p.kv_entries_len = a->kv_entries_len;
  p.num_partial_rows = a->num_partial_rows;
  p.batch = a->batch;
  p.group = a->num_qo_heads / a->num_kv_heads;
  p.head_dim = a->head_dim;
  p.node_offset = 0;
  p.node_count = 0;
  p.node_split = 0;
  p.lead_wide = 0;
  p.workers = 0;
  p.few_form = ft::FEW_ONE;
  p.num_kv_heads = a->num_kv_heads;
  p.sm_scale = a->sm_scale;
  return p;
}

// Every stage-1 kernel is launched with permission to be scheduled before the preceding kernel of the stream has
// drained (programmatic dependent launch).  The kernels do nothing but on-chip set-up before their
// griddepcontrol.wait, which returns once the preceding kernel has completed and its writes are visible, so the
// permission is safe after any kernel; it pays after kernels that release their dependents early, as both stages of
// this library do: back-to-back decode calls overlap each launch and set-up with the previous kernel's tail.
template <typename... KArgs, typename... Args>
cudaError_t launch_early(void (*kernel)(KArgs...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

template <typename T, int D>
int launch_mma(const ft::Stage1Params& p, int hkv, cudaStream_t st) {
  using C = ft::MmaCfg<D>;
  if (dry_run("stage1_mma_kernel")) return FT_OK;
  static OncePerDevice once;
  FT_CUDA_OK(raise_smem_limit(once, ft::stage1_mma_kernel<T, D>, C::SMEM_BYTES));
  const unsigned grid = (unsigned)p.node_count * (unsigned)hkv;
  FT_CUDA_OK(launch_early(ft::stage1_mma_kernel<T, D>, grid, C::THREADS, C::SMEM_BYTES, st, p));
  count_launch();
  return FT_OK;
}

int sm_count(int dev) {
  static std::atomic<int> sms[64];
  if (dev < 0 || dev >= 64) return 148;
  int n = sms[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    sms[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

// Persistent few-row kernel: two CTAs per SM, each walking its share of the tasks.
template <typename T, int D>
int launch_stream(const ft::TcParams& tp, int hkv, cudaStream_t st) {
  using C = ft::StreamCfg<D>;
  if (dry_run("stage1_stream_kernel")) return FT_OK;
  static OncePerDevice once;
  int dev = 0;
  FT_CUDA_OK(raise_smem_limit(once, ft::stage1_stream_kernel<T, D>, C::SMEM_BYTES, &dev));
  const int64_t tasks = (int64_t)tp.p.node_count * hkv;
  const int64_t slots = 2LL * sm_count(dev);
  const unsigned grid = (unsigned)(tasks < slots ? tasks : slots);
  FT_CUDA_OK(launch_early(ft::stage1_stream_kernel<T, D>, grid, 128, C::SMEM_BYTES, st, tp));
  count_launch();
  return FT_OK;
}

// ---- TMA descriptors of the K / V buffers for the tcgen05 kernel -------------------------------------------
// The driver entry point is looked up through the runtime, so the library has no link-time dependency on libcuda.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<EncodeTiledFn>(f);
  }();
  return fn;
}

struct MapKey {
  const void* base;
  int64_t rows, s0, s1;
  int heads, dtype, box_heads, device;
  bool operator==(const MapKey& o) const {
    return base == o.base && rows == o.rows && s0 == o.s0 && s1 == o.s1 && heads == o.heads && dtype == o.dtype &&
           box_heads == o.box_heads && device == o.device;
  }
};

// Descriptor of a [rows, heads, head_dim] 16-bit tensor (element strides s0, s1), box 64 (head_dim) x box_heads x
// box_rows, 128-byte swizzle; with box_heads 0 the same tensor as [rows, all elements of a row] with a box of 64 x 1,
// the form that gathers rows.  Descriptors are cached by buffer identity (encoding one costs about a microsecond)
// in a hash table of 1024 slots, probed linearly over 8 slots; a full neighbourhood evicts its first slot.  A
// serving process holds four descriptors per layer's K/V buffers (six at head_dim 256) plus two per query shape - a few
// hundred at most.
bool tensor_map(CUtensorMap* out, const void* base, int dtype, int head_dim, int64_t rows, int heads, int64_t s0,
                   int64_t s1, int box_heads, int box_rows) {
  constexpr int SLOTS = 1024, PROBES = 8;
  static std::mutex mu;
  static MapKey keys[SLOTS];
  static CUtensorMap maps[SLOTS];
  static bool used[SLOTS] = {};
  int device = -1;
  if (cudaGetDevice(&device) != cudaSuccess) return false;  // the same address can name different memory on two devices
  const MapKey key{base, rows, s0, s1, heads, dtype + 16 * head_dim, box_heads * 1024 + box_rows, device};
  uint64_t h = reinterpret_cast<uintptr_t>(base) >> 8;
  h = (h ^ (uint64_t)key.box_heads * 0x9E3779B97F4A7C15ull ^ (uint64_t)(device + 1) * 0xC2B2AE3D27D4EB4Full ^
       (uint64_t)rows * 0x165667B19E3779F9ull) * 0xFF51AFD7ED558CCDull;
  const int home = (int)(h >> 40) & (SLOTS - 1);
  std::lock_guard<std::mutex> lock(mu);
  int slot = -1;
  for (int i = 0; i < PROBES; ++i) {
    const int j = (home + i) & (SLOTS - 1);
    if (used[j] && keys[j] == key) {
      *out = maps[j];
      return true;
    }
    if (!used[j] && slot < 0) slot = j;
  }
  if (slot < 0) slot = home;
  EncodeTiledFn enc = encode_tiled_fn();
  if (enc == nullptr || rows <= 0 || rows > 0x7fffffffLL || heads <= 0) return false;
  const bool flat = box_heads == 0;
  const int64_t row_elems = (int64_t)(heads - 1) * s1 + head_dim;
  if (flat && (s1 < 0 || row_elems > s0 || row_elems > 0x7fffffffLL)) return false;  // rows that overlap: no 2-D tensor
  const cuuint64_t dims[3] = {(cuuint64_t)(flat ? row_elems : head_dim), (cuuint64_t)(flat ? rows : heads), (cuuint64_t)rows};
  const cuuint64_t strides[2] = {(cuuint64_t)(flat ? s0 : s1) * 2, (cuuint64_t)s0 * 2};  // bytes, for dimensions 1 and 2
  const cuuint32_t box[3] = {64, (cuuint32_t)(flat ? 1 : box_heads), (cuuint32_t)box_rows};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUtensorMap m;
  const CUresult rc = enc(&m, dtype == FT_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, flat ? 2 : 3,
                          const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) return false;
  keys[slot] = key;
  maps[slot] = m;
  used[slot] = true;
  *out = m;
  return true;
}

ft::TcParams tc_params(const ft::Stage1Params& p, const ft_decode_args* a) {
  ft::TcParams tp;
  memset(&tp, 0, sizeof(tp));
  tp.p = p;
  const int d = a->head_dim;
  tp.has_tma = tensor_map(&tp.k_map, a->k_buffer, a->dtype, d, a->kv_rows, a->num_kv_heads, a->k_stride0,
                             a->k_stride1, 1, 64) &&
               tensor_map(&tp.v_map, a->v_buffer, a->dtype, d, a->kv_rows, a->num_kv_heads, a->v_stride0,
                             a->v_stride1, 1, 64);
  tp.has_gather4 = tp.has_tma &&
                   tensor_map(&tp.k_rows_map, a->k_buffer, a->dtype, d, a->kv_rows, a->num_kv_heads, a->k_stride0,
                                 a->k_stride1, 0, 1) &&
                   tensor_map(&tp.v_rows_map, a->v_buffer, a->dtype, d, a->kv_rows, a->num_kv_heads, a->v_stride0,
                                 a->v_stride1, 0, 1);
  // Q by TMA (tcgen05 kernel): one box per request covering its G heads (at most 8 per box when G is a multiple of 8),
  // or one box for a whole tile of consecutive requests.  Any G up to 128: with 16-byte copies the Q tile arrives later
  // than the first K tile (64 requests on a 4096-token prefix, 24/8 heads: 31.2 us per step with copies, 27.6 with boxes;
  // 28/4 heads: 27.7 and 23.1; on a three-level tree of 256 requests 53.8 and 50.3, 47.5 and 37.0).
  const int g = p.group;
  if (tp.has_tma && g >= 1 && g <= 128) {
    const int box_heads = g % 8 == 0 ? 8 : g;
    if (tensor_map(&tp.q_map, a->q, a->dtype, d, a->batch, a->num_qo_heads, a->q_stride0, a->q_stride1, box_heads, 1) &&
        tensor_map(&tp.q_map_tile, a->q, a->dtype, d, a->batch, a->num_qo_heads, a->q_stride0, a->q_stride1, g, 128 / g))
      tp.q_box_rows = box_heads;
  }
  return tp;
}

// What the plan says of its tasks' sizes; longest 0: nothing is known
struct TaskSizes {
  int64_t few_tokens = 0;
  int64_t few_longest = 0, few_over_8_rows = 0, many_longest = 0;
};

// for a launch whose few-row tasks are phase 1's
TaskSizes task_sizes(const ft_decode_args* a) {
  TaskSizes z;
  if (a->few_tokens > 0 && a->few_longest > 0)
    z = {a->few_tokens, a->few_longest, a->few_over_8_rows, a->many_longest > 0 ? a->many_longest : 0};
  return z;
}

// How the few-row tasks of a launch are run (ft::FEW_*; -1: by the tcgen05 kernel, head_dim 256 only); wide: its many-row CTAs.
// Two tasks per CTA keep an SM streaming while a task starts up, but four then share the SM's copy rate and they are dealt out
// in pairs.  So they pay where the tasks are many for their longest one (their tokens fill 1.5 rounds of it at four tasks per
// SM; 1.25 at head_dim 64), or about even, in enough rounds for their length; where few need the two-block body (more than
// eight rows), which does not fit 128 registers; and where the step does not wait for a many-row chunk, which four neighbours
// slow down (at head_dim 64 sooner: a token's rows are half as long, a many-row tile takes what it takes at 128).  us per step
// with one / two tasks per CTA:
//   head_dim 128  64 leaves of 256 tokens under 4096, 32/8 heads, 27.7 / 25.6, under 16000 40.2 / 37.2; 90 of 400 under 1000
//                 39.1 / 36.7, 74 of 400 33.8 / 35.0; ragged trees: six levels (many for their longest) 577 / 566, four levels
//                 58.6 / 81.2; 26 leaves of 275 under chunks of up to 1181, 32/32 heads, 54.5 / 68.4
//   head_dim 64   448 leaves of 142 under 59, 16/16 heads, 142 / 89; ragged four levels 39.5 / 53.5; 322 leaves of 233 under
//                 chunks of 7998, 64/8 heads, 139 / 188
// Head_dim 256, one CTA per SM: one round on the tcgen05 kernel, whose tile loads are the larger.  Beyond it two at a time if
// none has more than eight rows, which would be two passes over K and V, and they are many for their longest or short (beside
// many-row CTAs, in whose rounds pairs fit worse, shorter); with eight warps each, and those of more than eight rows on the
// tcgen05 body, if they are short or make more than two rounds.  us per step on the tcgen05 kernel / two at a time / eight
// warps each, 16/8 heads: 64 of 256 under 4096 57.1 / 44.9 / 48.1; 60 of 130 under 1000 47.4 / 30.0 / 39.3, 60 of 1500
// 144 / 126 / 129, 16 of 400 (one round) 21.5 / 23.1 / 24.1; 47 of 280 under 930, one task of 15 rows, 24/8 heads, 46.4 /
// 80.4 / 44.8; 29 of 335 under 3 of 127 under 2013, 32/8 heads, 37.0 / 40.4 two at a time; 26 of 314 under 3441 35.2 / 37.1
// with eight warps each; 4 of 60 beside groups of 17 x 60, which the step waits for, 32/32 heads, 33.4 / 35.3 so.
// The bounds are where the ratio of both sides crosses one over 2700 trees drawn from the benchmark's ranges: the rule takes
// two tasks (or eight warps) on 117 of 1030 at head_dim 128, 142 of 1085 at 64 and 124 of 628 at 256, which take 15, 21 and
// 27 % less time for it, and at worst 3, 5 and 0 % more.  Of 1700 trees drawn after
// that it was more than 3 % behind one task per CTA (or the tcgen05 kernel) on one.
int few_rows_form(const TaskSizes& z, int group, int64_t few_nodes, int64_t wide, int hkv, int head_dim, int64_t slots) {
  const int64_t few = few_nodes * hkv, longest = z.few_longest, tokens = z.few_tokens * hkv;
  const int without = head_dim == 256 ? -1 : ft::FEW_ONE;
  if (longest == 0 || group > 8) return without;
  if (head_dim == 256) {
    if (few + wide <= slots) return without;
    const bool alone = 8 * wide <= slots, waits = z.many_longest * slots > 4 * tokens;
    if (z.few_over_8_rows == 0 && !waits && (longest <= (alone ? 400 : 256) || tokens >= 2 * slots * longest))
      return ft::FEW_PAIR;
    const bool brief = longest <= (alone ? 320 : 256) && !waits && 8 * z.few_over_8_rows <= few_nodes && 5 * wide <= 3 * slots;
    return 5 * few > 12 * slots || brief ? ft::FEW_EIGHT : without;
  }
  if (4 * z.few_over_8_rows > few_nodes) return without;
  const bool even = 4 * longest * few_nodes <= 5 * z.few_tokens;
  bool two;
  if (head_dim == 64)
    two = z.many_longest * slots <= tokens && (2 * tokens >= 5 * slots * longest || (even && few >= 2 * slots && longest <= 512));
  else
    two = z.many_longest * slots <= 4 * tokens &&
          (tokens >= 3 * slots * longest || (even && (5 * few >= 12 * slots ? longest <= 640 : 5 * few >= 8 * slots && longest <= 320)));
  return two ? ft::FEW_PAIR : without;
}

// few-row tasks alone, at head_dim 64 or 128
template <typename T, int D>
int launch_narrow(const ft::Stage1Params& p, int hkv, cudaStream_t st, int form) {
  const bool pair = form == ft::FEW_PAIR;
  if (dry_run(pair ? "stage1_pair_kernel" : "stage1_narrow_kernel")) return FT_OK;
  const int64_t tasks = (int64_t)p.node_count * hkv;
  if (pair) {
    using C = ft::PairCfg<D>;
    static OncePerDevice once;
    FT_CUDA_OK(raise_smem_limit(once, ft::stage1_pair_kernel<T, D>, C::SMEM_BYTES));
    FT_CUDA_OK(launch_early(ft::stage1_pair_kernel<T, D>, (unsigned)((tasks + 1) / 2), C::THREADS, C::SMEM_BYTES, st, p));
  } else {
    using C = ft::NarrowCfg<D, 2>;
    static OncePerDevice once;
    FT_CUDA_OK(raise_smem_limit(once, ft::stage1_narrow_kernel<T, D>, C::SMEM_BYTES));
    FT_CUDA_OK(launch_early(ft::stage1_narrow_kernel<T, D>, (unsigned)tasks, 128, C::SMEM_BYTES, st, p));
  }
  count_launch();
  return FT_OK;
}

template <typename T, int D>
int launch_tc(const ft::TcParams& p, int hkv, cudaStream_t st) {
  using C = ft::TcCfg<D>;
  if (dry_run("stage1_tc_kernel")) return FT_OK;
  static OncePerDevice once;
  FT_CUDA_OK(raise_smem_limit(once, ft::stage1_tc_kernel<T, D>, C::SMEM_BYTES));
  const unsigned grid = (unsigned)p.p.node_count * (unsigned)hkv;
  FT_CUDA_OK(launch_early(ft::stage1_tc_kernel<T, D>, grid, C::THREADS, C::SMEM_BYTES, st, p));
  count_launch();
  return FT_OK;
}

// Claim counters of the persistent kernel: 64 pairs used round-robin by successive launches (each launch leaves
// its pair at zero when its last CTA finishes, so a pair is reusable as soon as that launch is over; launches
// 64 apart do not overlap in practice).
static __device__ unsigned int g_sched_counters[64][2];

template <typename T>
int launch_persist(ft::TcParams p, int hkv, cudaStream_t st) {
  using C = ft::TcCfg<128>;
  if (dry_run("stage1_persist_kernel")) return FT_OK;
  static OncePerDevice once;
  int dev = 0;
  FT_CUDA_OK(raise_smem_limit(once, ft::stage1_persist_kernel<T, 128>, C::SMEM_BYTES, &dev));
  if (dev < 0 || dev >= 64) return fail(FT_ERR_UNSUPPORTED, "device ordinal %d outside 0..63", dev);
  static std::atomic<unsigned int*> counters_of_device[64];
  unsigned int* base = counters_of_device[dev].load(std::memory_order_acquire);
  if (base == nullptr) {
    FT_CUDA_OK(cudaGetSymbolAddress(reinterpret_cast<void**>(&base), g_sched_counters));
    counters_of_device[dev].store(base, std::memory_order_release);
  }
  static std::atomic<unsigned int> next_pair{0};
  p.sched = base + 2 * (next_pair.fetch_add(1, std::memory_order_relaxed) % 64u);
  const int64_t slots = 2LL * sm_count(dev);  // two resident CTAs per SM
  int64_t tasks = (int64_t)p.p.node_count * hkv;
  if (p.p.dev_phase != nullptr) tasks = slots;  // the task count is only known on the device: a full grid
  if (tasks <= 0) return FT_OK;
  if (tasks > 0x7fffffffLL) return fail(FT_ERR_TOO_LARGE, "vnodes x kv heads exceeds the task limit");
  const unsigned grid = (unsigned)(tasks < slots ? tasks : slots);
  FT_CUDA_OK(launch_early(ft::stage1_persist_kernel<T, 128>, grid, C::THREADS, C::SMEM_BYTES, st, p));
  count_launch();
  return FT_OK;
}

// Few-row tasks: persistent workers with a task pipeline, or one CTA per task?  The workers hide a short task's start-up
// but deal the tasks out statically; the hardware hands one-CTA tasks to whichever slot is free.  Workers are faster only
// where very many tasks of about a tile each meet few slots.  The host does not see the tasks' lengths: the length of the
// row-id table, of which every few-row chunk has a part of its own, bounds their sum from above, so workers are taken
// where even that bound leaves a mean of at most 80 tokens per few-row node.  The table also holds the many-row phase's
// row ids, and on the serving path it is the whole req_to_token pool: a plan with short few-row tasks beside a long prefix runs one CTA per task although workers would
// be quicker (1024 leaves of 64 tokens under a 32 000-token node).  The splitter groups such leaves; what is left for
// the workers are plans of its reference mode, ungrouped plans and hand-made ones.  Measured per step, one CTA per task /
// workers, 296 slots, leaves under a 1000-token node, 32/8 heads of 128, ungrouped: 1024 leaves of 64 tokens 171 / 140 us,
// of 100 190 / 203, of 300 285 / 314; 512 leaves of 32 84 / 98, of 64 89 / 89, of 130 125 / 155, of 900 324 / 374; a ragged
// tree of 117 tasks x 16 heads, 20 to 1948 tokens, 140 / 247.
bool few_rows_by_workers(int64_t few_nodes, int64_t kv_entries_len, int hkv, int64_t slots) {
  return few_nodes * hkv >= 20 * slots && kv_entries_len <= 80 * few_nodes;
}

template <typename T, int D, bool PAIR>
int launch_fused_as(const ft::FusedParams<D, PAIR>& p, int64_t ctas, cudaStream_t st) {
  constexpr int few_smem = [] {
    if constexpr (PAIR) return ft::PairCfg<D>::SMEM_BYTES;
    else return std::max(ft::StreamCfg<D>::SMEM_BYTES, ft::NarrowCfg<D, 2>::SMEM_BYTES);
  }();
  constexpr int smem = std::max(ft::TcCfg<D>::SMEM_BYTES, few_smem);
  static_assert(smem <= (D == 256 ? 232448 : 115712), "the resident CTAs must fit in one SM's shared memory");
  if (dry_run(!PAIR ? "stage1_fused_kernel" : p.p.few_form == ft::FEW_PAIR ? "stage1_fused_kernel/pair" : "stage1_fused_kernel/eight"))
    return FT_OK;
  if (ctas > 0x7fffffffLL) return fail(FT_ERR_TOO_LARGE, "vnodes x kv heads exceeds the grid limit");
  static OncePerDevice once;
  FT_CUDA_OK(raise_smem_limit(once, ft::stage1_fused_kernel<T, D, PAIR>, smem));
  FT_CUDA_OK(launch_early(ft::stage1_fused_kernel<T, D, PAIR>, (unsigned)ctas, ft::TcCfg<D>::THREADS, smem, st, p));
  count_launch();
  return FT_OK;
}

template <typename T, int D>
int launch_fused(ft::TcParams p, const ft_decode_args* a, const TaskSizes& sizes, int hkv, cudaStream_t st) {
  int dev = 0;
  FT_CUDA_OK(cudaGetDevice(&dev));
  const int64_t wide = (int64_t)p.p.node_split * hkv;
  const int64_t few_nodes = p.p.node_count - p.p.node_split, few = few_nodes * hkv;
  const int64_t slots = (int64_t)ft::TcCfg<D>::CTAS * sm_count(dev);
  p.p.lead_wide = (int)wide;  // many-row CTAs go first
  p.p.few_form = few_rows_form(sizes, p.p.group, few_nodes, wide, hkv, D, slots);
  if constexpr (D <= 128) {
    // Few-row tasks by persistent workers only when the many-row CTAs do not fill the device more than once (the workers
    // take the slots those leave and, as they finish, theirs too).
    if (few_rows_by_workers(few_nodes, p.p.kv_entries_len, hkv, slots) && wide <= slots) {
      p.p.workers = (int)slots;
      return launch_fused_as<T, D, false>(p, wide + slots, st);
    }
    if (p.p.few_form == ft::FEW_ONE) return launch_fused_as<T, D, false>(p, wide + few, st);
  }
  if (p.p.few_form < 0) return launch_tc<T, D>(p, hkv, st);  // the whole range on the tcgen05 kernel
  const int per = ft::few_per_cta(p.p.few_form);
  const int64_t ctas = wide + (few + per - 1) / per;
  if constexpr (D == 256) {
    ft::SlabParams sp;
    memset(&sp, 0, sizeof(sp));
    static_cast<ft::TcParams&>(sp) = p;
    sp.has_slabs = tensor_map(&sp.k_slab_map, a->k_buffer, a->dtype, D, a->kv_rows, hkv, a->k_stride0, a->k_stride1, 1, 16) &&
                   tensor_map(&sp.v_slab_map, a->v_buffer, a->dtype, D, a->kv_rows, hkv, a->v_stride0, a->v_stride1, 1, 16);
    return launch_fused_as<T, D, true>(sp, ctas, st);
  } else {
    return launch_fused_as<T, D, true>(p, ctas, st);
  }
}

// path: AUTO (<= 16 rows: persistent workers or narrow, in the form few_rows_form chooses; above: tcgen05),
// STREAM (like AUTO, always the persistent workers), MMA (narrow / wide), MMA_WIDE (wide for everything),
// TCGEN05 (tcgen05 for everything)
template <typename T, int D>
int launch_tensor(const ft::Stage1Params& p, const ft_decode_args* a, int hkv, cudaStream_t st, int max_rows, int path) {
  const TaskSizes sizes = p.node_offset == a->phase_node_offsets[1] && p.node_count == a->phase_node_nums[1] ? task_sizes(a) : TaskSizes();
  if (path == FT_PATH_TCGEN05 || ((path == FT_PATH_AUTO || path == FT_PATH_STREAM) && max_rows > 16))
    return launch_tc<T, D>(tc_params(p, a), hkv, st);
  int dev = 0;
  FT_CUDA_OK(cudaGetDevice(&dev));
  const int64_t slots = (int64_t)ft::TcCfg<D>::CTAS * sm_count(dev);
  if constexpr (D == 256) {
    return launch_fused<T, D>(tc_params(p, a), a, sizes, hkv, st);  // (no many-row phase)
  } else {
    if (max_rows <= 16) {
      const bool many = few_rows_by_workers(p.node_count, p.kv_entries_len, hkv, slots);
      if (path == FT_PATH_STREAM || (path == FT_PATH_AUTO && many)) return launch_stream<T, D>(tc_params(p, a), hkv, st);
    }
    if (path != FT_PATH_MMA_WIDE && max_rows <= 16)
      return launch_narrow<T, D>(p, hkv, st,
                                 path == FT_PATH_AUTO ? few_rows_form(sizes, p.group, p.node_count, 0, hkv, D, slots) : ft::FEW_ONE);
    return launch_mma<T, D>(p, hkv, st);
  }
}

// fp32 storage at head_dim 64 / 128 with 16-byte aligned rows: the tiled CUDA-core kernel
bool f32_tiled_ok(const ft_decode_args* a) {
  if (a->dtype != FT_F32 || (a->head_dim != 64 && a->head_dim != 128)) return false;
  if (!aligned16(a->q) || !aligned16(a->k_buffer) || !aligned16(a->v_buffer)) return false;
  return a->q_stride0 % 4 == 0 && a->q_stride1 % 4 == 0 && a->k_stride0 % 4 == 0 && a->k_stride1 % 4 == 0 &&
         a->v_stride0 % 4 == 0 && a->v_stride1 % 4 == 0;
}

template <int D>
int launch_f32(const ft::Stage1Params& p, int hkv, cudaStream_t st, int max_rows) {
  using C = ft::F32Cfg<D>;
  if (dry_run("stage1_f32_kernel")) return FT_OK;
  static OncePerDevice once;
  FT_CUDA_OK(raise_smem_limit(once, ft::stage1_f32_kernel<D>, C::SMEM_BYTES));
  const int blocks_z = (max_rows + C::ROWS - 1) / C::ROWS;
  if (blocks_z > 65535) return fail(FT_ERR_TOO_LARGE, "too many query rows per vnode for the fp32 kernel");
  dim3 grid(p.node_count, hkv, blocks_z);
  FT_CUDA_OK(launch_early(ft::stage1_f32_kernel<D>, grid, C::THREADS, C::SMEM_BYTES, st, p));
  count_launch();
  return FT_OK;
}

// Blocks of four rows, one per warp; max_rows only sizes the grid, the kernel strides over whatever rows a task has.
// Measured per step, one block per task / blocks of 32, 16, 8 and 4 rows: fp32, 16/8 heads of 256, 64 requests on 4096
// tokens 66.5 / 24.9, 13.4, 7.3 and 3.8 ms, 256 requests on 2048 tokens 64.8 / 17.7, 10.0, 6.1 and 5.9; fp16, 32/8 heads of
// 32, 40 requests on 500 tokens 795 / 487, 309, 195 and 145 us.
template <typename T>
int launch_generic(const ft::Stage1Params& p, int hkv, cudaStream_t st, int max_rows) {
  if (dry_run("stage1_generic_kernel")) return FT_OK;
  const int blocks_z = max_rows < 256 ? (max_rows + 3) / 4 : 64;
  dim3 grid(p.node_count, hkv, blocks_z);
  FT_CUDA_OK(launch_early(ft::stage1_generic_kernel<T>, grid, 128, 0, st, p));
  count_launch();
  return FT_OK;
}

// max_rows: upper bound on query rows (requests x group) of the tasks in the range
int launch_stage1_range(const ft_decode_args* a, int path, int offset, int count, int max_rows) {
  if (count <= 0) return FT_OK;
  ft::Stage1Params p = stage1_params(a);
  p.node_offset = offset;
  p.node_count = count;
  cudaStream_t st = static_cast<cudaStream_t>(a->stream);
  const int hkv = a->num_kv_heads;
  if (path != FT_PATH_GENERIC) {
    const bool f16 = a->dtype == FT_F16;
    switch (a->head_dim) {
      case 64:
        return f16 ? launch_tensor<__half, 64>(p, a, hkv, st, max_rows, path)
                   : launch_tensor<__nv_bfloat16, 64>(p, a, hkv, st, max_rows, path);
      case 128:
        return f16 ? launch_tensor<__half, 128>(p, a, hkv, st, max_rows, path)
                   : launch_tensor<__nv_bfloat16, 128>(p, a, hkv, st, max_rows, path);
      default:
        return f16 ? launch_tensor<__half, 256>(p, a, hkv, st, max_rows, path)
                   : launch_tensor<__nv_bfloat16, 256>(p, a, hkv, st, max_rows, path);
    }
  }
  // fp32 storage: the tiled kernel when the caller named no path (FT_PATH_GENERIC stays the scalar kernel) and the
  // phase's request tile bounds its rows
  if (a->path == FT_PATH_AUTO && f32_tiled_ok(a) && max_rows > 0 && max_rows < (1 << 20))
    return a->head_dim == 128 ? launch_f32<128>(p, hkv, st, max_rows) : launch_f32<64>(p, hkv, st, max_rows);
  switch (a->dtype) {
    case FT_F16: return launch_generic<__half>(p, hkv, st, max_rows);
    case FT_BF16: return launch_generic<__nv_bfloat16>(p, hkv, st, max_rows);
    default: return launch_generic<float>(p, hkv, st, max_rows);
  }
}

// after_stage1: this launch directly follows a stage-1 launch of the same call on the same stream.  Only then may
// the kernel be scheduled early (programmatic dependent launch): it reads the request tables before it waits for
// the preceding kernel, which is safe after stage 1 (that kernel never writes them) but not after an arbitrary
// kernel of the caller's that may still be building those tables.
int launch_merge(void (*kernel)(ft::Stage2Params), const ft::Stage2Params& p, int64_t blocks, cudaStream_t st, bool after_stage1) {
  if (blocks > 0x7fffffffLL) return fail(FT_ERR_TOO_LARGE, "batch x heads too large for one launch");
  // launched with permission to be scheduled before the preceding kernel (stage 1) has drained; the kernel itself
  // waits for that kernel's completion before it touches the partial buffers
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = after_stage1 ? 1 : 0;
  FT_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, p));
  count_launch();
  return FT_OK;
}

template <typename T, int C, int RB, int SPLIT>
int launch_pieces(ft::Stage2Params p, cudaStream_t st, bool after_stage1) {
  p.pieces = (uint32_t)((((int64_t)p.heads << p.dim_shift) + 128 * C - 1) / (128 * C));
  const int64_t items = (int64_t)p.batch * p.pieces;
  if (items > 0x7fffffffLL) return fail(FT_ERR_TOO_LARGE, "batch x heads too large for one launch");
  p.items = (uint32_t)items;
  return launch_merge(ft::stage2_piece_kernel<T, C, RB, SPLIT>, p, SPLIT == 1 ? (items + 3) / 4 : items, st, after_stage1);
}

// Which merge, by the 128-float pieces of the output and the mean number of partial rows per request (of the plan, where
// the caller states it: its scratch buffers may hold more).  us for the merge alone, replayed from a graph, and per decode step:
//   few pieces, many rows: four warps per piece    160 pieces x 36 rows, one warp per head 5.9 / four 3.9 (step 13.8 / 11.8),
//                                                  32 x 18 4.2 / 2.9 (12.2 / 9.9); 1024 x 9 3.7 / 3.4, 2048 x 9 4.1 / 5.2
//   one round of CTAs with more than four rows, or six rows and more: weights by one lane per row
//                                                  2048 x 7, step, 25.7 (by every lane 26.7); 8192 x 18 11.3 (14.1)
//   fewer rows: weights by every lane              16384 heads of 64 x 3.4 9.0 -> 4.9 (step 37.0 -> 33.1), 8192 x 4 6.1 -> 5.6
//   very many pieces: two of them per warp         65536 x 2 33.8 -> 21.2, 32768 x 3 20.9 -> 17.0 (one piece 18.7)
// At head_dim 64 and below one lane per row would leave half of the lanes and more idle: 8192 pieces x 18 rows 19.3 / 13.8.
// At head_dim 256 a head is two pieces, and weights that every lane computes are computed twice as often as by heads: by pieces
// only where they are few (by pieces / by heads: 1536 x 2 2.57 / 2.71, 2048 x 2 2.74 / 2.78, 4096 x 4 3.61 / 3.27, 8192 x 3
// 4.91 / 3.77, 32000 x 3 13.8 / 10.1; 103 requests of 30 tokens on 200, 32/8 heads, 17.2 / 16.2 per step; 233
// drawn steps of more than 1024 pieces 0.93 to 1.097 of the time by heads, 1.011 in the mean).
template <typename T>
int launch_stage2(const ft::Stage2Params& p, int64_t rows, cudaStream_t st, bool after_stage1) {
  const int64_t pieces = (((int64_t)p.batch * p.heads << p.dim_shift) + 127) / 128, heads = (int64_t)p.batch * p.heads;
  if (pieces == 0) return FT_OK;
  const int64_t batch = p.batch;
  if (pieces <= 1024 && rows >= 6 * batch)
    return rows >= 12 * batch ? launch_pieces<T, 1, 8, 4>(p, st, after_stage1) : launch_pieces<T, 1, 4, 4>(p, st, after_stage1);
  int dev = 0;
  FT_CUDA_OK(cudaGetDevice(&dev));
  const bool one_round = heads <= 24LL * sm_count(dev);
  if (p.head_dim >= 128 && ((one_round && rows > 4 * batch) || rows >= 6 * batch || (p.head_dim > 128 && pieces > 1024))) {
    auto* kernel = p.head_dim > 128 ? ft::stage2_merge_kernel<T, 2, 4> : one_round ? ft::stage2_merge_kernel<T, 1, 8> : ft::stage2_merge_kernel<T, 1, 4>;
    return launch_merge(kernel, p, (heads + 3) / 4, st, after_stage1);
  }
  return pieces <= 16384 ? launch_pieces<T, 1, 4, 1>(p, st, after_stage1) : launch_pieces<T, 2, 2, 1>(p, st, after_stage1);
}

__global__ void bump_kv_lens_kernel(int32_t* kv_lens, const int32_t* last, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const int v = last[i];
    if (v >= 0) atomicAdd(kv_lens + v, 1);
  }
}

}  // namespace

extern "C" {

int ft_version(void) { return 100; }

int ft_decode_args_size(void) { return static_cast<int>(sizeof(ft_decode_args)); }

const char* ft_last_error(void) { return g_err; }

int64_t ft_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

const char* ft_stage1_path_name(const ft_decode_args* args) {
  g_kernel_names[0] = '\0';
  g_dry_run = true;
  const int rc = ft_stage1(args);
  g_dry_run = false;
  if (rc != FT_OK) return nullptr;
  return g_kernel_names;
}

int ft_stage1(const ft_decode_args* a) {
  int rc = check_common(a);
  if (rc != FT_OK) return rc;
  rc = check_stage1(a);
  if (rc != FT_OK) return rc;
  const int path = pick_path(a);
  if (path < 0) return path;
  const int n0 = a->phase_node_nums[0], n1 = a->phase_node_nums[1];
  const int o0 = a->phase_node_offsets[0], o1 = a->phase_node_offsets[1];
  const int group = a->num_qo_heads / a->num_kv_heads;
  // A phase's request tile bounds the query rows of its tasks; a non-positive tile size means "unknown".
  const int64_t r0 = a->phase_q_tile_sizes[0] > 0 ? (int64_t)a->phase_q_tile_sizes[0] * group : 1 << 30;
  const int64_t r1 = a->phase_q_tile_sizes[1] > 0 ? (int64_t)a->phase_q_tile_sizes[1] * group : 1 << 30;
  const int rows0 = (int)(r0 < (1 << 30) ? r0 : (1 << 30)), rows1 = (int)(r1 < (1 << 30) ? r1 : (1 << 30));
  // (head_dim 256: a few-row phase in front of a many-row one runs on the tcgen05 kernel with it)
  const bool same_kernel = path == FT_PATH_GENERIC || path == FT_PATH_MMA_WIDE || path == FT_PATH_TCGEN05 ||
                           a->head_dim == 256 || ((rows0 > 16) == (rows1 > 16));
  // the persistent kernel takes every task of the launch, whatever its row count
  if (path == FT_PATH_PERSIST && a->device_phase_info != nullptr) {
    ft::Stage1Params p = stage1_params(a);  // node_offset / node_count come from the device array
    const ft::TcParams tp = tc_params(p, a);
    cudaStream_t st = static_cast<cudaStream_t>(a->stream);
    return a->dtype == FT_F16 ? launch_persist<__half>(tp, a->num_kv_heads, st)
                              : launch_persist<__nv_bfloat16>(tp, a->num_kv_heads, st);
  }
  if (path == FT_PATH_PERSIST) {
    cudaStream_t st = static_cast<cudaStream_t>(a->stream);
    const bool joined = n0 > 0 && n1 > 0 && o1 == o0 + n0;
    for (int ph = 0; ph < (joined ? 1 : 2); ++ph) {
      ft::Stage1Params p = stage1_params(a);
      p.node_offset = ph == 0 ? o0 : o1;
      p.node_count = joined ? n0 + n1 : (ph == 0 ? n0 : n1);
      p.node_split = ph == 0 ? n0 : 0;
      if (p.node_count <= 0) continue;
      const ft::TcParams tp = tc_params(p, a);
      rc = a->dtype == FT_F16 ? launch_persist<__half>(tp, a->num_kv_heads, st)
                              : launch_persist<__nv_bfloat16>(tp, a->num_kv_heads, st);
      if (rc != FT_OK) return rc;
    }
    return FT_OK;
  }
  // many-row phase followed directly by the few-row phase: one grid with both kernel bodies
  if (path == FT_PATH_AUTO && (a->head_dim == 64 || a->head_dim == 128 || a->head_dim == 256) && n0 > 0 && n1 > 0 && o1 == o0 + n0 && rows0 > 16 && rows1 <= 16) {
    ft::Stage1Params p = stage1_params(a);
    p.node_offset = o0;
    p.node_count = n0 + n1;
    p.node_split = n0;
    cudaStream_t st = static_cast<cudaStream_t>(a->stream);
    const ft::TcParams tp = tc_params(p, a);
    const TaskSizes sizes = task_sizes(a);
    if (a->head_dim == 64)
      return a->dtype == FT_F16 ? launch_fused<__half, 64>(tp, a, sizes, a->num_kv_heads, st)
                                : launch_fused<__nv_bfloat16, 64>(tp, a, sizes, a->num_kv_heads, st);
    if (a->head_dim == 256)
      return a->dtype == FT_F16 ? launch_fused<__half, 256>(tp, a, sizes, a->num_kv_heads, st)
                                : launch_fused<__nv_bfloat16, 256>(tp, a, sizes, a->num_kv_heads, st);
    return a->dtype == FT_F16 ? launch_fused<__half, 128>(tp, a, sizes, a->num_kv_heads, st)
                              : launch_fused<__nv_bfloat16, 128>(tp, a, sizes, a->num_kv_heads, st);
  }
  // Adjacent phases that want the same kernel go out as one grid.
  if (n0 > 0 && n1 > 0 && o1 == o0 + n0 && same_kernel)
    return launch_stage1_range(a, path, o0, n0 + n1, rows0 > rows1 ? rows0 : rows1);
  rc = launch_stage1_range(a, path, o0, n0, rows0);
  if (rc != FT_OK) return rc;
  return launch_stage1_range(a, path, o1, n1, rows1);
}

namespace {
int stage2_impl(const ft_decode_args* a, bool after_stage1) {
  int rc = check_common(a);
  if (rc != FT_OK) return rc;
  if (a->o == nullptr) return fail(FT_ERR_INVALID_ARGUMENT, "o is NULL");
  if (a->batch > 0 && (!a->req_to_vnode_entries || !a->req_to_vnode_offs || !a->req_to_vnode_lens))
    return fail(FT_ERR_INVALID_ARGUMENT, "a request table pointer is NULL");
  ft::Stage2Params p;
  p.r2v_entries = a->req_to_vnode_entries;
  p.r2v_offs = a->req_to_vnode_offs;
  p.r2v_lens = a->req_to_vnode_lens;
  p.mid_o = a->mid_o;
  p.mid_lse = a->mid_lse;
  p.o = a->o;
  p.o_lse = a->o_lse;
  p.mo_s0 = a->mid_o_stride0;
  p.mo_s1 = a->mid_o_stride1;
  p.ml_s0 = a->mid_lse_stride0;
  p.o_s0 = a->o_stride0;
  p.o_s1 = a->o_stride1;
  p.num_partial_rows = a->num_partial_rows;
  p.batch = a->batch;
  p.heads = a->num_qo_heads;
  p.head_dim = a->head_dim;
  for (p.dim_shift = 0; (1 << p.dim_shift) < a->head_dim;) ++p.dim_shift;
  {
    const int64_t esz = a->dtype == FT_F32 ? 4 : 2, vec = 4 * esz;  // bytes of one 4-element store
    p.o_vec = (reinterpret_cast<uintptr_t>(a->o) % vec == 0 && (a->o_stride0 * esz) % vec == 0 &&
               (a->o_stride1 * esz) % vec == 0)
                  ? 1
                  : 0;
  }
  cudaStream_t st = static_cast<cudaStream_t>(a->stream);
  const int64_t rows = a->plan_rows > 0 && a->plan_rows < a->num_partial_rows ? a->plan_rows : a->num_partial_rows;
  switch (a->dtype) {
    case FT_F16: return launch_stage2<__half>(p, rows, st, after_stage1);
    case FT_BF16: return launch_stage2<__nv_bfloat16>(p, rows, st, after_stage1);
    default: return launch_stage2<float>(p, rows, st, after_stage1);
  }
}
}  // namespace

int ft_stage2(const ft_decode_args* a) { return stage2_impl(a, false); }

int ft_decode(const ft_decode_args* a) {
  const int64_t before = t_launches;
  int rc = ft_stage1(a);
  if (rc != FT_OK) return rc;
  // a plan without vnodes launches no stage 1: stage 2 then follows whatever the caller enqueued before
  const bool launched = t_launches != before;
  return stage2_impl(a, launched);
}

namespace {
// Host-to-device copy done by the SMs: 16 bytes per thread from mapped pinned host memory.  For the few hundred
// KiB of a decode step's query this is several microseconds quicker than a copy-engine transfer, whose set-up
// and completion hand-shake dominate at that size.
__global__ void __launch_bounds__(256) host_to_device_kernel(uint4* __restrict__ dst, const uint4* __restrict__ src, size_t n16,
                                                             unsigned char* dst_tail, const unsigned char* src_tail, int tail) {
  // stage 1 may set itself up (barriers, tensor memory) while the query crosses PCIe; it waits for this kernel's
  // completion before it reads anything
  ft::allow_dependent_launch();
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n16) dst[i] = src[i];
  if (i < (size_t)tail) dst_tail[i] = src_tail[i];
}
}  // namespace

int ft_decode_host_io(const ft_decode_args* a, const void* q_host, void* o_host, int wait) {
  if (a == nullptr) return fail(FT_ERR_INVALID_ARGUMENT, "args is NULL");
  if (q_host == nullptr || o_host == nullptr) return fail(FT_ERR_INVALID_ARGUMENT, "q_host / o_host is NULL");
  if (a->q == nullptr || a->o == nullptr) return fail(FT_ERR_INVALID_ARGUMENT, "q / o (device staging buffers) is NULL");
  if (a->batch < 0 || a->num_qo_heads <= 0 || a->head_dim <= 0)
    return fail(FT_ERR_INVALID_ARGUMENT, "batch / num_qo_heads / head_dim must be positive");
  const int64_t row = (int64_t)a->num_qo_heads * a->head_dim;
  if (a->q_stride1 != a->head_dim || a->q_stride0 != row || a->o_stride1 != a->head_dim || a->o_stride0 != row)
    return fail(FT_ERR_UNSUPPORTED, "ft_decode_host_io needs packed [batch, heads, head_dim] device q and o");
  const size_t esz = a->dtype == FT_F32 ? 4 : 2;
  const size_t bytes = (size_t)a->batch * (size_t)row * esz;
  cudaStream_t st = static_cast<cudaStream_t>(a->stream);
  if (bytes == 0) return ft_decode(a);
  // Pinned host memory is mapped into the device's address space: the query is then fetched by a small kernel and
  // stage 2 writes the output rows straight into o_host over PCIe, so no copy-engine transfer sits on the step's
  // critical path.  Memory that is not mapped (pageable, or registered without the mapped flag) takes the copy
  // engine, one cudaMemcpyAsync per buffer.
  void *q_map = nullptr, *o_map = nullptr;
  const bool mapped = cudaHostGetDevicePointer(&q_map, const_cast<void*>(q_host), 0) == cudaSuccess &&
                      cudaHostGetDevicePointer(&o_map, o_host, 0) == cudaSuccess && aligned16(q_map) && aligned16(a->q) &&
                      aligned16(o_map);
  if (!mapped) {
    (void)cudaGetLastError();  // the failed query left an error behind
    FT_CUDA_OK(cudaMemcpyAsync(const_cast<void*>(a->q), q_host, bytes, cudaMemcpyHostToDevice, st));
    const int rc = ft_decode(a);
    if (rc != FT_OK) return rc;
    FT_CUDA_OK(cudaMemcpyAsync(o_host, a->o, bytes, cudaMemcpyDeviceToHost, st));
    if (wait) FT_CUDA_OK(cudaStreamSynchronize(st));
    return FT_OK;
  }
  const size_t n16 = bytes / 16;
  const int tail = (int)(bytes % 16);
  const unsigned blocks = (unsigned)((n16 + (tail ? 1 : 0) + 255) / 256);
  host_to_device_kernel<<<blocks, 256, 0, st>>>(static_cast<uint4*>(const_cast<void*>(a->q)), static_cast<const uint4*>(q_map), n16,
                                                static_cast<unsigned char*>(const_cast<void*>(a->q)) + 16 * n16,
                                                static_cast<const unsigned char*>(q_map) + 16 * n16, tail);
  FT_CUDA_OK(cudaGetLastError());
  count_launch();
  ft_decode_args b = *a;
  b.o = o_map;  // stage 2 writes the merged rows into host memory; the device staging buffer args->o is not used
  const int rc = ft_decode(&b);
  if (rc != FT_OK) return rc;
  if (wait) FT_CUDA_OK(cudaStreamSynchronize(st));
  return FT_OK;
}

// ---- ft_decode_static_scratch: partial-result scratch in a fixed device array owned by the library ----------
//
// The array lives in every CUDA context that loads this library, from load until exit.  In host code its name is
// only a stand-in for the device symbol, so the device address is looked up once per device with
// cudaGetSymbolAddress (that device being current) and that address is what the kernels receive.
#define FT_STATIC_SCRATCH_FLOATS (FT_STATIC_SCRATCH_BYTES / 4u)
static __device__ __align__(256) float g_static_scratch[FT_STATIC_SCRATCH_FLOATS];

int ft_decode_static_scratch(const ft_decode_args* a) {
  if (a == nullptr) return fail(FT_ERR_INVALID_ARGUMENT, "args is NULL");
  if (a->num_partial_rows < 0 || a->num_qo_heads <= 0 || a->head_dim <= 0)
    return fail(FT_ERR_INVALID_ARGUMENT, "num_partial_rows / num_qo_heads / head_dim must be positive");
  const int64_t per_row = (int64_t)a->num_qo_heads * (a->head_dim + 1);
  if (a->num_partial_rows > (int64_t)FT_STATIC_SCRATCH_FLOATS / per_row)
    return fail(FT_ERR_TOO_LARGE,
                "plan needs %lld partial rows x %d heads x (%d+1) floats = %lld bytes of scratch; the built-in array "
                "holds %u bytes - use ft_decode with caller-owned mid_o / mid_lse",
                (long long)a->num_partial_rows, a->num_qo_heads, a->head_dim,
                (long long)(a->num_partial_rows * per_row * 4), (unsigned)(4u * FT_STATIC_SCRATCH_FLOATS));
  static float* scratch_of_device[64] = {};
  int dev = 0;
  FT_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(FT_ERR_UNSUPPORTED, "device ordinal %d outside 0..63", dev);
  if (scratch_of_device[dev] == nullptr) {  // set-up: first call on this device
    float* ptr = nullptr;
    FT_CUDA_OK(cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_static_scratch));
    if (ptr == nullptr) return fail(FT_ERR_CUDA, "cudaGetSymbolAddress returned a null address");
    scratch_of_device[dev] = ptr;
  }
  ft_decode_args b = *a;
  b.mid_o = scratch_of_device[dev];
  b.mid_o_stride0 = (int64_t)a->num_qo_heads * a->head_dim;
  b.mid_o_stride1 = a->head_dim;
  b.mid_lse = b.mid_o + a->num_partial_rows * b.mid_o_stride0;
  b.mid_lse_stride0 = a->num_qo_heads;
  return ft_decode(&b);
}

int ft_bump_kv_lens(int32_t* vnode_to_kv_lens, const int32_t* last_vnodes, int32_t n, void* stream) {
  if (n < 0) return fail(FT_ERR_INVALID_ARGUMENT, "n is negative");
  if (n == 0) return FT_OK;
  if (vnode_to_kv_lens == nullptr || last_vnodes == nullptr)
    return fail(FT_ERR_INVALID_ARGUMENT, "vnode_to_kv_lens / last_vnodes is NULL");
  bump_kv_lens_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(vnode_to_kv_lens, last_vnodes, n);
  FT_CUDA_OK(cudaGetLastError());
  count_launch();
  return FT_OK;
}

namespace {
// one warp per segment of the auxiliary row-id table
__global__ void gather_kv_entries_kernel(const int32_t* __restrict__ src, int64_t src_len, const int32_t* __restrict__ seg_src,
                                         const int32_t* __restrict__ seg_len, const int32_t* __restrict__ seg_dst,
                                         const int32_t* __restrict__ seg_room, int n, int32_t* __restrict__ aux, int64_t aux_len) {
  const int seg = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (seg >= n) return;
  const int64_t from = seg_src[seg], len = seg_len[seg], to = seg_dst[seg], room = seg_room[seg];
  if (len <= 0 || room < 0 || from < 0 || from + len > src_len || to < 0 || to + len + room > aux_len) {
    if (lane == 0 && (len != 0 || room != 0)) ft::flag_error(FT_DEV_BAD_KV_INDEX);
    return;
  }
  for (int64_t i = lane; i < len; i += 32) aux[to + i] = src[from + i];
  const int32_t filler = src[from];
  for (int64_t i = lane; i < room; i += 32) aux[to + len + i] = filler;
}

__global__ void bump_tails_kernel(int32_t* __restrict__ state, int n, int32_t* __restrict__ ranges, int64_t rows,
                                  int32_t* __restrict__ kv_lens, int n_vnodes) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int32_t* st = state + 4 * (int64_t)i;
  const int aux_pos = st[0], index = st[2], room = st[3];
  if (aux_pos < 0) {
    if (index >= 0 && index < n_vnodes) kv_lens[index] += 1;
    else if (index != -1) ft::flag_error(FT_DEV_BAD_ROW_INDEX);  // {-1, x, -1, x}: an unused entry
    return;
  }
  if (room <= 0 || ranges == nullptr || index < 0 || index >= rows) {
    ft::flag_error(FT_DEV_BAD_KV_INDEX);
    return;
  }
  ranges[2 * (int64_t)index + 1] += 1;
  st[0] = aux_pos + 1;
  st[1] += 1;
  st[3] = room - 1;
}

__global__ void refresh_tails_kernel(const int32_t* __restrict__ state, int n, const int32_t* __restrict__ src, int64_t src_len,
                                     int32_t* __restrict__ aux, int64_t aux_len) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t* st = state + 4 * (int64_t)i;
  const int64_t aux_pos = st[0], src_pos = st[1];
  if (aux_pos < 0) return;
  if (aux_pos < 1 || aux_pos > aux_len || src_pos < 1 || src_pos > src_len) {
    ft::flag_error(FT_DEV_BAD_KV_INDEX);
    return;
  }
  aux[aux_pos - 1] = src[src_pos - 1];
}
}  // namespace

int ft_gather_kv_entries(const int32_t* src_table, int64_t src_len, const int32_t* seg_src, const int32_t* seg_len,
                         const int32_t* seg_dst, const int32_t* seg_room, int32_t n_segments, int32_t* aux_table,
                         int64_t aux_len, void* stream) {
  if (n_segments < 0 || src_len < 0 || aux_len < 0) return fail(FT_ERR_INVALID_ARGUMENT, "negative size");
  if (n_segments == 0) return FT_OK;
  if (src_table == nullptr || seg_src == nullptr || seg_len == nullptr || seg_dst == nullptr || seg_room == nullptr ||
      aux_table == nullptr)
    return fail(FT_ERR_INVALID_ARGUMENT, "a table of ft_gather_kv_entries is NULL");
  gather_kv_entries_kernel<<<(n_segments + 7) / 8, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      src_table, src_len, seg_src, seg_len, seg_dst, seg_room, n_segments, aux_table, aux_len);
  FT_CUDA_OK(cudaGetLastError());
  count_launch();
  return FT_OK;
}

int ft_bump_tails(int32_t* tail_state, int32_t n, int32_t* vnode_q_kv_ranges, int64_t num_partial_rows,
                  int32_t* vnode_to_kv_lens, int32_t num_vnodes, void* stream) {
  if (n < 0 || num_partial_rows < 0 || num_vnodes < 0) return fail(FT_ERR_INVALID_ARGUMENT, "negative size");
  if (n == 0) return FT_OK;
  if (tail_state == nullptr || vnode_to_kv_lens == nullptr)
    return fail(FT_ERR_INVALID_ARGUMENT, "tail_state / vnode_to_kv_lens is NULL");
  bump_tails_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      tail_state, n, vnode_q_kv_ranges, num_partial_rows, vnode_to_kv_lens, num_vnodes);
  FT_CUDA_OK(cudaGetLastError());
  count_launch();
  return FT_OK;
}

int ft_refresh_tails(const int32_t* tail_state, int32_t n, const int32_t* src_table, int64_t src_len, int32_t* aux_table,
                     int64_t aux_len, void* stream) {
  if (n < 0 || src_len < 0 || aux_len < 0) return fail(FT_ERR_INVALID_ARGUMENT, "negative size");
  if (n == 0) return FT_OK;
  if (tail_state == nullptr || src_table == nullptr || aux_table == nullptr)
    return fail(FT_ERR_INVALID_ARGUMENT, "tail_state / src_table / aux_table is NULL");
  refresh_tails_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(tail_state, n, src_table, src_len,
                                                                                        aux_table, aux_len);
  FT_CUDA_OK(cudaGetLastError());
  count_launch();
  return FT_OK;
}

namespace {
// One warp waits on an mbarrier that nothing ever arrives at, through the same bounded waits the stage-1 kernels
// use, and on a completed one with too few probes in some lanes.  No copy, no MMA and no tensor memory is involved, so a wait that runs out leaves nothing in flight.
__global__ void bounded_wait_selftest_kernel(int limit, int* result) {
  __shared__ __align__(8) unsigned long long barrier_word[2];
  __shared__ int abort_word;
  const uint32_t bar = ft::smem_u32(barrier_word), done = bar + 8;
  if (threadIdx.x == 0) {
    ft::mbar_init(bar, 1);
    ft::mbar_init(done, 1);
    abort_word = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    ft::mbar_arrive(done);
  }
  __syncthreads();
  // (1) the plain bounded wait of the persistent workers: gives up after `limit` probes
  const bool plain = ft::mbar_wait(bar, 0, limit);
  // (2) the tcgen05 kernel's wait: same limit semantics (its own constant), and it leaves early once a sibling
  // role has raised the CTA's abort flag - raised here by lane 0 before the call
  if (threadIdx.x == 0) abort_word = 1;
  __syncthreads();
  const bool aborted = ft::tc_wait(bar, 0, &abort_word);
  // (3) the few-row bodies' wait by whole warps, on a barrier that has completed: half of the lanes have no probe left,
  // so all lanes must be told that the wait ran out
  const bool split = __any_sync(0xffffffffu, ft::mbar_wait_warp(done, 0, threadIdx.x < 16 ? 0 : limit));
  if (threadIdx.x == 0) {
    if (!plain || !aborted) ft::flag_error(FT_DEV_WAIT_TIMEOUT);  // what the kernels do when a wait runs out
    result[0] = (plain ? 1 : 0) + (split ? 2 : 0);
    result[1] = aborted ? 1 : 0;
  }
}
}  // namespace

int ft_selftest_bounded_wait(int limit, int* result_host, void* stream) {
  if (result_host == nullptr) return fail(FT_ERR_INVALID_ARGUMENT, "result_host is NULL");
  if (limit < 1 || limit > (1 << 20)) return fail(FT_ERR_INVALID_ARGUMENT, "limit must be in [1, 2^20] probes");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int* dev = nullptr;
  FT_CUDA_OK(cudaMalloc(&dev, 2 * sizeof(int)));
  bounded_wait_selftest_kernel<<<1, 32, 0, st>>>(limit, dev);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(result_host, dev, 2 * sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFree(dev);
  if (e != cudaSuccess) return fail(FT_ERR_CUDA, "bounded-wait self-test failed: %s", cudaGetErrorString(e));
  count_launch();
  return FT_OK;
}

#ifdef FT_TIMELINE
// Developer builds only: copies the first n per-CTA records {start ns, end ns, SM id, kind, 12 marks} of the last stage-1 launch.
int ft_debug_timeline(unsigned long long* out, int n) {
  if (out == nullptr || n < 0 || n > ft::FT_TIMELINE_CTAS) return fail(FT_ERR_INVALID_ARGUMENT, "bad timeline request");
  FT_CUDA_OK(cudaDeviceSynchronize());
  FT_CUDA_OK(cudaMemcpyFromSymbol(out, ft::g_timeline, sizeof(unsigned long long) * 16 * (size_t)n));
  return FT_OK;
}
#endif

int ft_read_wait_diagnostics(int32_t* out8) {
  if (out8 == nullptr) return fail(FT_ERR_INVALID_ARGUMENT, "out8 is NULL");
  FT_CUDA_OK(cudaDeviceSynchronize());
  FT_CUDA_OK(cudaMemcpyFromSymbol(out8, ft::g_wait_diag, 8 * sizeof(int)));
  if (out8[0] != 0) {
    const int zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    FT_CUDA_OK(cudaMemcpyToSymbol(ft::g_wait_diag, zero, sizeof(zero)));
  }
  return FT_OK;
}

int ft_read_device_status(void* stream, int32_t* flags) {
  if (flags == nullptr) return fail(FT_ERR_INVALID_ARGUMENT, "flags is NULL");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  FT_CUDA_OK(cudaStreamSynchronize(st));
  int host = 0;
  FT_CUDA_OK(cudaMemcpyFromSymbol(&host, ft::g_device_status, sizeof(int)));
  if (host != 0) {
    const int zero = 0;
    FT_CUDA_OK(cudaMemcpyToSymbol(ft::g_device_status, &zero, sizeof(int)));
  }
  *flags = host;
  return FT_OK;
}

}  // extern "C"
