// The Python call path of the decode entry points: checks the tensors, fills ft_decode_args and calls the C ABI.
//
// A decode step of a few requests is about ten microseconds of GPU work, launched once per layer and step, with a query
// and an output that are new tensors each time.  Done in Python, the checks and the forty-odd argument fields took
// 13.6 us per call (18 us in fp32), so small steps were bound by the host; here they take well under a microsecond beside
// the two launches, which is cheap enough to do for every call: nothing is remembered from one call for the next,
// the argument block lives on the stack, and the GIL is released around the launch.
//
// Built as an extension module of its own (ft_b200/build.py): libfasttree_b200.so stays free of Python and torch.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstring>

#include "fasttree_b200.h"

namespace {

typedef int (*DecodeFn)(const ft_decode_args*);
DecodeFn g_entry[3] = {nullptr, nullptr, nullptr};  // ft_decode, ft_stage1, ft_stage2

struct Refused {};  // a Python error has been set

[[noreturn]] void refuse(const char* fmt, const char* name, const char* more = "") {
  PyErr_Format(PyExc_ValueError, fmt, name, more);
  throw Refused();
}

const at::Tensor& tensor(const char* name, PyObject* o) {
  if (!THPVariable_Check(o)) refuse("%s must be a torch.Tensor", name);
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda())
    refuse("%s is on %s; the engine has no CPU path - tensors must live on a CUDA device", name, t.device().str().c_str());
  return t;
}

const at::Tensor& table(const char* name, PyObject* o) {
  const at::Tensor& t = tensor(name, o);
  if (t.scalar_type() != at::kInt) refuse("%s must be int32, got %s", name, c10::toString(t.scalar_type()));
  if (!t.is_contiguous()) refuse("%s must be contiguous", name);
  return t;
}

void pair(const char* name, PyObject* o, int64_t (&out)[2]) {
  PyObject* seq = PySequence_Fast(o, "expected a pair of integers");
  if (seq == nullptr) throw Refused();
  if (PySequence_Fast_GET_SIZE(seq) != 2) {
    Py_DECREF(seq);
    refuse("%s must have two entries (one per phase)", name);
  }
  for (int i = 0; i < 2; ++i) {
    PyObject* v = PyNumber_Long(PySequence_Fast_GET_ITEM(seq, i));
    out[i] = v != nullptr ? PyLong_AsLongLong(v) : -1;
    Py_XDECREF(v);
    if (PyErr_Occurred()) {
      Py_DECREF(seq);
      throw Refused();
    }
  }
  Py_DECREF(seq);
}

// The task sizes that a plan's vnode_to_kv_lens tensor carries as an attribute (ft_b200.planner.task_sizes), with the plan's
// partial rows behind them where the scratch buffers hold more; without it none are known.
void task_sizes(PyObject* table, ft_decode_args& a) {
  static PyObject* const name = PyUnicode_InternFromString("task_sizes");
  PyObject* sizes = nullptr;
  if (_PyObject_LookupAttr(table, name, &sizes) < 0) throw Refused();
  if (sizes == nullptr) return;
  long long n[5] = {0, 0, 0, 0, 0};
  const int count = PyTuple_Check(sizes) ? (int)PyTuple_GET_SIZE(sizes) : 0;
  for (int i = 0; (count == 4 || count == 5) && i < count; ++i) n[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(sizes, i));
  Py_DECREF(sizes);
  if (PyErr_Occurred()) throw Refused();
  a.few_tokens = n[0];
  a.few_longest = (int32_t)n[1];
  a.few_over_8_rows = (int32_t)n[2];
  a.many_longest = (int32_t)n[3];
  a.plan_rows = (int32_t)n[4];
}

// Positional arguments of the reference's fasttree_decode (kernel_bench/fasttree.py:582-601), in order.
enum { Q, K, V, O, KV_ENTRIES, KV_OFFS, KV_LENS, Q_ENTRIES, Q_OFFS, Q_LENS, R2V_ENTRIES, R2V_OFFS, R2V_LENS, MID_O, MID_LSE,
       NODE_NUMS, NODE_OFFSETS, Q_TILES, KV_TILES, SM_SCALE, N_ARGS };

// (args tuple, logit_cap, path, o_lse | None, row ranges | None, partial rows named by q_entries or -1,
//  phase_info | None, kv_entries_aux | None, stream or -1 for torch's current one)
void fill(PyObject* const* x, ft_decode_args& a, c10::DeviceIndex& device) {
  memset(&a, 0, sizeof(a));
  if (!PyTuple_Check(x[0]) || PyTuple_GET_SIZE(x[0]) != N_ARGS) {
    PyErr_Format(PyExc_TypeError, "expected %d positional arguments", (int)N_ARGS);
    throw Refused();
  }
  auto arg = [&](int i) { return PyTuple_GET_ITEM(x[0], i); };
  const at::Tensor &q = tensor("q", arg(Q)), &k = tensor("k_buffer", arg(K)), &v = tensor("v_buffer", arg(V)),
                   &o = tensor("o", arg(O)), &mid_o = tensor("mid_o", arg(MID_O)), &mid_lse = tensor("mid_lse", arg(MID_LSE));
  if (q.dim() != 3 || o.dim() != 3 || k.dim() != 3 || v.dim() != 3)
    refuse("%s", "q, o must be [batch, heads, head_dim] and k/v buffers [rows, kv_heads, head_dim]");
  const at::ScalarType dtype = q.scalar_type();
  if (dtype != at::kHalf && dtype != at::kBFloat16 && dtype != at::kFloat) refuse("unsupported dtype %s", c10::toString(dtype));
  if (k.scalar_type() != dtype || v.scalar_type() != dtype || o.scalar_type() != dtype)
    refuse("%s", "q, k_buffer, v_buffer and o must share one dtype");
  if (q.size(2) != k.size(2) || q.size(2) != v.size(2)) refuse("%s", "head_dim of q, k_buffer and v_buffer differ");
  if (o.sizes() != q.sizes()) refuse("%s", "o must have the shape of q");
  if (mid_o.scalar_type() != at::kFloat || mid_lse.scalar_type() != at::kFloat) refuse("%s", "mid_o / mid_lse must be float32");
  if (mid_o.dim() != 3 || mid_lse.dim() != 2 || mid_lse.stride(1) != 1)
    refuse("%s", "mid_o must be [rows, heads, head_dim] and mid_lse [rows, heads]");
  const at::Tensor* rows[] = {&q, &k, &v, &o, &mid_o};
  const char* row_names[] = {"q", "k_buffer", "v_buffer", "o", "mid_o"};
  for (int i = 0; i < 5; ++i)
    if (rows[i]->stride(2) != 1) refuse("%s: the head_dim axis must be contiguous", row_names[i]);
  const int64_t batch = q.size(0), heads = q.size(1);
  if (mid_o.size(1) < heads || mid_o.size(2) != q.size(2) || mid_lse.size(1) < heads)
    refuse("%s", "mid_o / mid_lse are too small for the head count of q");
  if (k.sizes() != v.sizes()) refuse("%s", "k_buffer and v_buffer differ in shape");

  static const char* const table_names[] = {"vnode_to_kv_entries", "vnode_to_kv_offs",     "vnode_to_kv_lens",
                                            "vnode_to_q_entries",  "vnode_to_q_offs",      "vnode_to_q_lens",
                                            "req_to_vnode_entries", "req_to_vnode_offs",   "req_to_vnode_lens"};
  const int32_t* tab[9];
  int64_t len[9];
  for (int i = 0; i < 9; ++i) {
    const at::Tensor& t = table(table_names[i], arg(KV_ENTRIES + i));
    tab[i] = static_cast<const int32_t*>(t.data_ptr());
    len[i] = t.numel();
  }
  int64_t nums[2], offs[2], q_tiles[2], kv_tiles[2];
  pair("phase_node_nums", arg(NODE_NUMS), nums);
  task_sizes(arg(KV_LENS), a);
  pair("phase_node_offsets", arg(NODE_OFFSETS), offs);
  pair("phase_q_tile_sizes", arg(Q_TILES), q_tiles);
  pair("phase_kv_tile_sizes", arg(KV_TILES), kv_tiles);
  const bool on_device = x[6] != Py_None;
  if (on_device) {
    const at::Tensor& t = table("phase_info", x[6]);
    if (t.numel() < 4) refuse("%s", "phase_info needs four entries: n0, n1, o0, o1");
    a.device_phase_info = static_cast<const int32_t*>(t.data_ptr());
  }
  if (x[7] != Py_None) {
    const at::Tensor& t = table("kv_entries_aux", x[7]);
    a.vnode_to_kv_entries_aux = static_cast<const int32_t*>(t.data_ptr());
    a.kv_entries_aux_len = t.numel();
  }
  const int64_t vnodes = len[1];
  for (int ph = 0; ph < 2; ++ph)
    if (!on_device && (nums[ph] < 0 || offs[ph] < 0 || offs[ph] + nums[ph] > vnodes))
      refuse("%s", "phase_node_nums / phase_node_offsets do not fit the vnode tables");
  if (std::min({len[2], len[4], len[5]}) < vnodes) refuse("%s", "vnode tables differ in length");
  if (len[7] < batch || len[8] < batch) refuse("%s", "request tables are shorter than the batch");
  if (x[3] != Py_None) {
    const at::Tensor& t = tensor("o_lse", x[3]);
    if (t.scalar_type() != at::kFloat || !t.is_contiguous() || t.numel() < batch * heads)
      refuse("%s", "o_lse must be a contiguous float32 [batch, heads] tensor");
    a.o_lse = static_cast<float*>(t.data_ptr());
  }
  int64_t q_rows = PyLong_AsLongLong(x[5]);
  if (q_rows < 0) q_rows = len[3];
  if (x[4] != Py_None) {
    const at::Tensor& t = table("row ranges", x[4]);
    if (t.numel() < 2 * q_rows) refuse("%s", "the row-range table needs two entries per partial row");
    a.vnode_q_kv_ranges = static_cast<const int32_t*>(t.data_ptr());
  }

  a.q = q.data_ptr();
  a.k_buffer = k.data_ptr();
  a.v_buffer = v.data_ptr();
  a.o = o.data_ptr();
  a.dtype = dtype == at::kHalf ? FT_F16 : dtype == at::kBFloat16 ? FT_BF16 : FT_F32;
  a.batch = (int32_t)batch;
  a.num_qo_heads = (int32_t)heads;
  a.head_dim = (int32_t)q.size(2);
  a.num_kv_heads = (int32_t)k.size(1);
  a.path = (int32_t)PyLong_AsLong(x[2]);
  a.kv_rows = k.size(0);
  a.q_stride0 = q.stride(0), a.q_stride1 = q.stride(1);
  a.k_stride0 = k.stride(0), a.k_stride1 = k.stride(1);
  a.v_stride0 = v.stride(0), a.v_stride1 = v.stride(1);
  a.o_stride0 = o.stride(0), a.o_stride1 = o.stride(1);
  a.vnode_to_kv_entries = tab[0];
  a.vnode_to_kv_offs = tab[1];
  a.vnode_to_kv_lens = const_cast<int32_t*>(tab[2]);
  a.vnode_to_q_entries = tab[3];
  a.vnode_to_q_offs = tab[4];
  a.vnode_to_q_lens = tab[5];
  a.req_to_vnode_entries = tab[6];
  a.req_to_vnode_offs = tab[7];
  a.req_to_vnode_lens = tab[8];
  a.kv_entries_len = len[0];
  a.num_partial_rows = std::min({mid_o.size(0), mid_lse.size(0), q_rows});
  for (int ph = 0; ph < 2; ++ph) {
    a.phase_node_nums[ph] = (int32_t)nums[ph];
    a.phase_node_offsets[ph] = (int32_t)offs[ph];
    a.phase_q_tile_sizes[ph] = (int32_t)q_tiles[ph];
    a.phase_kv_tile_sizes[ph] = (int32_t)kv_tiles[ph];
  }
  a.mid_o = static_cast<float*>(mid_o.data_ptr());
  a.mid_lse = static_cast<float*>(mid_lse.data_ptr());
  a.mid_o_stride0 = mid_o.stride(0), a.mid_o_stride1 = mid_o.stride(1);
  a.mid_lse_stride0 = mid_lse.stride(0);
  a.sm_scale = (float)PyFloat_AsDouble(arg(SM_SCALE));
  a.logit_cap = (float)PyFloat_AsDouble(x[1]);
  const long long stream = PyLong_AsLongLong(x[8]);
  if (PyErr_Occurred()) throw Refused();
  device = q.device().index();
  a.stream = stream != -1 ? reinterpret_cast<void*>(stream) : static_cast<void*>(c10::cuda::getCurrentCUDAStream(device).stream());
}

constexpr int N_FILL = 9;

// args(...) -> bytes of the filled ft_decode_args
PyObject* py_args(PyObject*, PyObject* const* x, Py_ssize_t n) {
  if (n != N_FILL) return PyErr_Format(PyExc_TypeError, "args() takes %d arguments", N_FILL);
  try {
    ft_decode_args a;
    c10::DeviceIndex device;
    fill(x, a, device);
    return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(&a), sizeof(a));
  } catch (const Refused&) {
    return nullptr;
  } catch (const std::exception& e) {
    return PyErr_Format(PyExc_RuntimeError, "%s", e.what());
  }
}

// call(entry, ...as args()) -> status of the C-ABI call, on the device of q
PyObject* py_call(PyObject*, PyObject* const* x, Py_ssize_t n) {
  if (n != 1 + N_FILL) return PyErr_Format(PyExc_TypeError, "call() takes %d arguments", 1 + N_FILL);
  const long entry = PyLong_AsLong(x[0]);
  if (entry < 0 || entry > 2 || g_entry[entry] == nullptr) return PyErr_Format(PyExc_ValueError, "unknown entry");
  try {
    ft_decode_args a;
    c10::DeviceIndex device;
    fill(x + 1, a, device);
    int rc;
    {
      const c10::cuda::CUDAGuard guard(device);
      Py_BEGIN_ALLOW_THREADS
      rc = g_entry[entry](&a);
      Py_END_ALLOW_THREADS
    }
    return PyLong_FromLong(rc);
  } catch (const Refused&) {
    return nullptr;
  } catch (const std::exception& e) {
    return PyErr_Format(PyExc_RuntimeError, "%s", e.what());
  }
}

// bind(address of ft_decode, of ft_stage1, of ft_stage2, sizeof(ft_decode_args) of the library)
PyObject* py_bind(PyObject*, PyObject* const* x, Py_ssize_t n) {
  if (n != 4) return PyErr_Format(PyExc_TypeError, "bind() takes 4 arguments");
  if (PyLong_AsLong(x[3]) != (long)sizeof(ft_decode_args))
    return PyErr_Format(PyExc_RuntimeError, "the library's ft_decode_args differs from the one this module was built with");
  for (int i = 0; i < 3; ++i) g_entry[i] = reinterpret_cast<DecodeFn>(PyLong_AsVoidPtr(x[i]));
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"args", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_args)), METH_FASTCALL, "filled ft_decode_args as bytes"},
    {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_call)), METH_FASTCALL, "check, fill and launch"},
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_bind)), METH_FASTCALL, "addresses of the C ABI"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "ft_call", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit_ft_call(void) { return PyModule_Create(&module); }
