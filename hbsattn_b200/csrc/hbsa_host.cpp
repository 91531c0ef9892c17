// The operators' host path as a CPython extension: argument checks, output and workspace allocation, argument block and
// launch of one call, without the interpreter in between.  What bounds the small calls is this path (a call on the
// example batch spends about 5 us on the GPU); in Python with ctypes it took about 50 us, here it takes about 10.
//
// Every function takes the plain case only - exact torch.Tensors on one CUDA device, int32 contiguous cu_seqlens, consistent
// shapes, no gradient wanted - and returns None for everything else; the callers in hbsa_interface.py and utils.py then go
// through their general code, which converts what can be converted and raises the documented errors.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>
#include <cstring>

#include "../../include/hbsattn_b200.h"

// The torch and the Python of this build; build.py looks for it in the file.
extern "C" __attribute__((used, visibility("default"))) const char hbsa_host_tag[] = HBSA_HOST_TAG;

namespace {

// Entry points of the C ABI library the package has loaded (HBSATTN_B200_LIBRARY may select another build of it).
struct Library {
  decltype(&hbsa_forward) forward;
  decltype(&hbsa_forward_status) forward_status;
  decltype(&hbsa_attention) attention;
  decltype(&hbsa_backward) backward;
  decltype(&hbsa_calculate_blocks_counted) blocks_counted;
  decltype(&hbsa_calculate_blocks) blocks;
  decltype(&hbsa_workspace_bytes) workspace_bytes;
  decltype(&hbsa_backward_workspace_bytes) backward_workspace_bytes;
  decltype(&hbsa_last_error) last_error;
} lib = {};
PyObject* g_state = nullptr;         // hbsa_interface._state: {"impl": ..., "last_workspace": ...}
PyObject *s_impl = nullptr, *s_last_workspace = nullptr;

bool get_int(PyObject* o, int64_t* v) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}

// A plain CUDA tensor on `dev` (or on any device while dev < 0, which it then sets).
const at::Tensor* get_tensor(PyObject* o, int* dev) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || !t.has_storage() || t.layout() != at::kStrided) return nullptr;
  const int d = t.device().index();
  if (*dev < 0) *dev = d;
  return d == *dev ? &t : nullptr;
}

int dtype_code(at::ScalarType t) {
  return t == at::kBFloat16 ? HBSA_DTYPE_BF16 : t == at::kHalf ? HBSA_DTYPE_F16 : t == at::kFloat ? HBSA_DTYPE_F32 : -1;
}

// The `impl` the process has selected with set_kernel_family, or -1.
int selected_impl() {
  PyObject* o = PyDict_GetItem(g_state, s_impl);
  if (!o || !PyUnicode_Check(o)) return -1;
  if (PyUnicode_CompareWithASCIIString(o, "auto") == 0) return HBSA_IMPL_AUTO;
  if (PyUnicode_CompareWithASCIIString(o, "sm100") == 0) return HBSA_IMPL_SM100;
  if (PyUnicode_CompareWithASCIIString(o, "generic") == 0) return HBSA_IMPL_GENERIC;
  return -1;
}

bool validate_wanted() {
  const char* e = std::getenv("HBSATTN_B200_VALIDATE");
  return !e || std::strcmp(e, "0") != 0;
}

void strides3(const at::Tensor& t, int64_t* out) {
  for (int i = 0; i < 3; ++i) out[i] = t.stride(i);
}

// What every operator has in common: q, k, v, cu_q, cu_k, the block mask in one of its two forms, and the options.
struct Call {
  int dev = -1;
  const at::Tensor *q, *k, *v, *cu_q, *cu_k, *mask = nullptr, *row_ptr = nullptr, *col_idx = nullptr;
  int64_t nqb = 0, nkb = 0, qbs, kbs;
  hbsa_forward_args a;

  // o: q, k, v, cu_q, cu_k, mask (None: CSR)
  bool tensors(PyObject* const* o) {
    q = get_tensor(o[0], &dev);
    k = get_tensor(o[1], &dev);
    v = get_tensor(o[2], &dev);
    cu_q = get_tensor(o[3], &dev);
    cu_k = get_tensor(o[4], &dev);
    if (!q || !k || !v || !cu_q || !cu_k) return false;
    if (q->dim() != 3 || k->dim() != 3 || v->dim() != 3 || k->sizes() != v->sizes() || q->size(2) != k->size(2)) return false;
    if (q->scalar_type() != k->scalar_type() || q->scalar_type() != v->scalar_type() || dtype_code(q->scalar_type()) < 0) return false;
    if (q->size(0) <= 0 || q->size(1) <= 0 || k->size(1) <= 0 || q->size(1) % k->size(1) != 0 || q->size(0) > INT32_MAX || k->size(0) > INT32_MAX) return false;
    if (cu_q->dim() != 1 || cu_k->dim() != 1 || cu_q->size(0) != cu_k->size(0) || cu_q->size(0) < 2) return false;
    if (cu_q->scalar_type() != at::kInt || cu_k->scalar_type() != at::kInt || !cu_q->is_contiguous() || !cu_k->is_contiguous()) return false;
    if (o[5] != Py_None) {
      mask = get_tensor(o[5], &dev);
      if (!mask || mask->scalar_type() != at::kBool || mask->dim() != 3 || mask->size(0) != k->size(1)) return false;
      nqb = mask->size(1);
      nkb = mask->size(2);
    }
    return true;
  }
  // o: q_block_size, k_block_size, causal, softmax_scale
  bool options(PyObject* const* o) {
    if (!get_int(o[0], &qbs) || !get_int(o[1], &kbs) || qbs <= 0 || kbs <= 0 || qbs % 16 || kbs % 16 || qbs > INT32_MAX || kbs > INT32_MAX) return false;
    const int causal = PyObject_IsTrue(o[2]);
    if (causal < 0) {
      PyErr_Clear();
      return false;
    }
    std::memset(&a, 0, sizeof(a));
    a.causal = causal;
    a.use_default_scale = o[3] == Py_None;
    if (o[3] != Py_None) {
      if (!PyFloat_CheckExact(o[3])) return false;
      a.softmax_scale = (float)PyFloat_AS_DOUBLE(o[3]);
    }
    return nqb > 0 && nkb > 0 && nqb <= INT32_MAX && nkb <= INT32_MAX;
  }
  void fill(int impl, const at::Tensor& out, const at::Tensor& ws, const at::Tensor* lse) {
    a.struct_bytes = sizeof(a);
    a.q = q->data_ptr();
    a.k = k->data_ptr();
    a.v = v->data_ptr();
    a.o = out.data_ptr();
    strides3(*q, a.q_stride);
    strides3(*k, a.k_stride);
    strides3(*v, a.v_stride);
    strides3(out, a.o_stride);
    a.cu_q_seqlens = static_cast<const int32_t*>(cu_q->data_ptr());
    a.cu_k_seqlens = static_cast<const int32_t*>(cu_k->data_ptr());
    if (mask) {
      a.block_mask = static_cast<const uint8_t*>(mask->data_ptr());
      strides3(*mask, a.mask_stride);                  // bool: one byte per element
    } else {
      a.csr_row_ptr = static_cast<const int32_t*>(row_ptr->data_ptr());
      a.csr_col_idx = static_cast<const int32_t*>(col_idx->data_ptr());
    }
    a.total_q = (int32_t)q->size(0);
    a.total_k = (int32_t)k->size(0);
    a.nhead_q = (int32_t)q->size(1);
    a.nhead_k = (int32_t)k->size(1);
    a.headdim = (int32_t)q->size(2);
    a.batch = (int32_t)cu_q->size(0) - 1;
    a.num_q_block = (int32_t)nqb;
    a.num_k_block = (int32_t)nkb;
    a.q_block_size = (int32_t)qbs;
    a.k_block_size = (int32_t)kbs;
    a.dtype = dtype_code(q->scalar_type());
    a.impl = impl;
    a.workspace = ws.data_ptr();
    a.workspace_bytes = (size_t)ws.numel();
    a.lse = lse ? static_cast<float*>(lse->data_ptr()) : nullptr;
  }
  at::Device device() const { return at::Device(at::kCUDA, (c10::DeviceIndex)dev); }
  at::Tensor empty(at::IntArrayRef size, at::ScalarType t) const { return at::Tensor(at::detail::empty_cuda(size, t, device(), std::nullopt)); }
  at::Tensor workspace() const {
    const int64_t n = (int64_t)lib.workspace_bytes((int)k->size(1), (int)nqb, (int)nkb, (int)cu_q->size(0) - 1);
    return empty({n}, at::kByte);                      // 512-byte aligned, as all of the allocator's blocks
  }
  void* stream() const { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream(); }
};

bool fail(const char* what, int rc) {
  PyErr_Format(PyExc_RuntimeError, "%s failed (%d): %s", what, rc, lib.last_error());
  return false;
}

bool remember(const at::Tensor& ws) {
  PyObject* w = THPVariable_Wrap(ws);
  if (!w) return false;
  const int rc = PyDict_SetItem(g_state, s_last_workspace, w);
  Py_DECREF(w);
  return rc == 0;
}

// One forward; with `validate` it waits for the device status and raises what it says.  False with a Python error set.
bool run_forward(Call& c, int impl, bool validate, const at::Tensor& out, const at::Tensor* lse) {
  at::Tensor ws = c.workspace();
  c.fill(impl, out, ws, lse);
  if (!validate) {
    const int rc = lib.forward(&c.a, c.stream());
    if (rc != 0) return fail("hbsa_forward", rc);
    return remember(ws);
  }
  int32_t status[16];
  int rc;
  void* const stream = c.stream();
  Py_BEGIN_ALLOW_THREADS
  rc = lib.forward_status(&c.a, status, stream);
  Py_END_ALLOW_THREADS
  if (rc != 0) return fail("hbsa_forward", rc);
  if (!remember(ws)) return false;
  if (status[0] == HBSA_STATUS_BLOCK_COUNT_MISMATCH) {
    if (c.mask)
      PyErr_Format(PyExc_AssertionError, "block_mask must be a boolean tensor of shape (nheads_k, num_q_block, num_k_block) = (%lld, %d, %d)",
                   (long long)c.k->size(1), status[1], status[2]);
    else
      PyErr_Format(PyExc_AssertionError, "num_q_block / num_k_block must be (%d, %d) for these cu_seqlens and block sizes", status[1], status[2]);
    return false;
  }
  if (status[0] != HBSA_STATUS_OK) {
    PyErr_Format(PyExc_RuntimeError, "hbsa_forward: device status %d (work item %d)", status[0], status[3]);
    return false;
  }
  return true;
}

// Whether autograd may want to hear of a call with this input: backward mode while gradients are recorded, forward mode always.
bool tracked(const at::Tensor* t) {
  if (t->unsafeGetTensorImpl()->autograd_meta() == nullptr) return false;
  return c10::GradMode::is_enabled() || t->_fw_grad(0).defined();
}
bool modes_active() { return c10::impl::TorchDispatchModeTLS::any_modes_set(); }

// attention(q, k, v, cu_q, cu_k, block_mask, q_block_size, k_block_size, causal, softmax_scale[, tile_mode[, 8 tables]]) -> out
PyObject* py_attention(PyObject*, PyObject* const* o, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n < 10 || n > 19 || modes_active()) Py_RETURN_NONE;
  Call c;
  if (!c.tensors(o) || !c.mask || !c.options(o + 6)) Py_RETURN_NONE;
  if (tracked(c.q) || tracked(c.k) || tracked(c.v)) Py_RETURN_NONE;
  if (n > 10) {
    if (!PyUnicode_Check(o[10])) Py_RETURN_NONE;
    if (PyUnicode_CompareWithASCIIString(o[10], "auto") != 0) {
      if (PyUnicode_CompareWithASCIIString(o[10], "fix") != 0 || (c.qbs & (c.qbs - 1)) || (c.kbs & (c.kbs - 1))) Py_RETURN_NONE;
    }
  }
  bool tables = n == 19;
  for (Py_ssize_t i = 11; i < n; ++i) tables = tables && o[i] != Py_None;
  if (tables) {
    int64_t nqb, nkb;
    if (!get_int(o[11], &nqb) || !get_int(o[15], &nkb) || nqb != c.nqb || nkb != c.nkb) Py_RETURN_NONE;
  }
  const int impl = selected_impl();
  if (impl < 0) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard(c.device());
  at::Tensor out = c.empty(c.q->sizes(), c.q->scalar_type());
  if (!run_forward(c, impl, !tables && validate_wanted(), out, nullptr)) return nullptr;
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// forward(q, k, v, cu_q, cu_k, block_mask | None, q_block_size, k_block_size, causal, softmax_scale, row_ptr, col_idx, num_q_block,
//         num_k_block, want_lse, validate) -> (out, lse | None).  With block_mask the four CSR arguments are None.
PyObject* py_forward(PyObject*, PyObject* const* o, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 16 || modes_active()) Py_RETURN_NONE;
  Call c;
  if (!c.tensors(o)) Py_RETURN_NONE;
  if (!c.mask) {
    c.row_ptr = get_tensor(o[10], &c.dev);
    c.col_idx = get_tensor(o[11], &c.dev);
    if (!c.row_ptr || !c.col_idx || !get_int(o[12], &c.nqb) || !get_int(o[13], &c.nkb)) Py_RETURN_NONE;
    if (c.row_ptr->scalar_type() != at::kInt || c.col_idx->scalar_type() != at::kInt || c.row_ptr->dim() != 1 || c.col_idx->dim() != 1 ||
        !c.row_ptr->is_contiguous() || !c.col_idx->is_contiguous() || c.row_ptr->numel() != c.k->size(1) * c.nqb + 1)
      Py_RETURN_NONE;
    if (c.col_idx->numel() == 0) Py_RETURN_NONE;       // no data pointer
  }
  if (!c.options(o + 6)) Py_RETURN_NONE;
  const int impl = selected_impl();
  if (impl < 0) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard(c.device());
  at::Tensor out = c.empty(c.q->sizes(), c.q->scalar_type()), lse;
  if (o[14] == Py_True) lse = c.empty({c.q->size(0), c.q->size(1)}, at::kFloat);
  if (!run_forward(c, impl, o[15] == Py_True, out, lse.defined() ? &lse : nullptr)) return nullptr;
  PyObject* r = PyTuple_New(2);
  if (!r) return nullptr;
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(out));
  PyTuple_SET_ITEM(r, 1, lse.defined() ? THPVariable_Wrap(lse) : Py_NewRef(Py_None));
  return r;
  END_HANDLE_TH_ERRORS
}

// scheduled(q, k, v, cu_q, cu_k, block_mask, q_block_size, k_block_size, causal, softmax_scale, workspace) -> out
PyObject* py_scheduled(PyObject*, PyObject* const* o, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 11 || modes_active()) Py_RETURN_NONE;
  Call c;
  if (!c.tensors(o) || !c.mask || !c.options(o + 6)) Py_RETURN_NONE;
  const at::Tensor* ws = get_tensor(o[10], &c.dev);
  const int impl = selected_impl();
  if (!ws || impl < 0) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard(c.device());
  at::Tensor out = c.empty(c.q->sizes(), c.q->scalar_type());
  c.fill(impl, out, *ws, nullptr);
  const int rc = lib.attention(&c.a, c.stream());
  if (rc != 0) {
    fail("hbsa_attention", rc);
    return nullptr;
  }
  if (PyDict_SetItem(g_state, s_last_workspace, o[10]) != 0) return nullptr;
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// backward(q, k, v, cu_q, cu_k, block_mask, q_block_size, k_block_size, causal, softmax_scale, out, lse, d_out) -> (dq, dk, dv)
PyObject* py_backward(PyObject*, PyObject* const* o, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 13 || modes_active()) Py_RETURN_NONE;
  Call c;
  if (!c.tensors(o) || !c.mask || !c.options(o + 6)) Py_RETURN_NONE;
  const at::Tensor *out = get_tensor(o[10], &c.dev), *lse = get_tensor(o[11], &c.dev), *g = get_tensor(o[12], &c.dev);
  if (!out || !lse || !g || c.k->size(0) == 0 || out->sizes() != c.q->sizes() || g->sizes() != c.q->sizes()) Py_RETURN_NONE;
  if (out->scalar_type() != c.q->scalar_type() || g->scalar_type() != c.q->scalar_type()) Py_RETURN_NONE;
  if (lse->scalar_type() != at::kFloat || !lse->is_contiguous() || lse->dim() != 2 || lse->size(0) != c.q->size(0) || lse->size(1) != c.q->size(1)) Py_RETURN_NONE;
  const int impl = selected_impl();
  if (!g->is_contiguous() || impl < 0) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard(c.device());
  at::Tensor dq = c.empty(c.q->sizes(), c.q->scalar_type()), dk = c.empty(c.k->sizes(), c.q->scalar_type()), dv = c.empty(c.k->sizes(), c.q->scalar_type());
  at::Tensor ws = c.workspace();
  const int64_t bytes = (int64_t)lib.backward_workspace_bytes(c.q->size(0), c.k->size(0), (int)c.q->size(1), (int)c.k->size(1), (int)c.q->size(2));
  at::Tensor gws = c.empty({bytes}, at::kByte);
  hbsa_backward_args b;
  std::memset(&b, 0, sizeof(b));
  c.fill(impl == HBSA_IMPL_GENERIC ? HBSA_IMPL_GENERIC : HBSA_IMPL_AUTO, *out, ws, lse);
  b.struct_bytes = sizeof(b);
  b.fwd = c.a;
  b.d_o = g->data_ptr();
  strides3(*g, b.do_stride);
  b.dq = dq.data_ptr();
  b.dk = dk.data_ptr();
  b.dv = dv.data_ptr();
  b.grad_workspace = gws.data_ptr();
  b.grad_workspace_bytes = (size_t)bytes;
  const int rc = lib.backward(&b, c.stream());
  if (rc != 0) {
    fail("hbsa_backward", rc);
    return nullptr;
  }
  if (!remember(ws)) return nullptr;
  PyObject* r = PyTuple_New(3);
  if (!r) return nullptr;
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(dq));
  PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(dk));
  PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(dv));
  return r;
  END_HANDLE_TH_ERRORS
}

// calculate_blocks(cu_seqlen, block_size) -> (num_block, cu_block, block_to_batch, cu_num_block).  The tables are allocated for
// `kGuess` blocks, so that one launch and one wait do in the common case, and cut to their size afterwards (16 KB each at most).
PyObject* py_calculate_blocks(PyObject*, PyObject* const* o, Py_ssize_t n) {
  constexpr int64_t kGuess = 4096;
  HANDLE_TH_ERRORS
  int dev = -1;
  int64_t bs;
  if (n != 2 || modes_active()) Py_RETURN_NONE;
  const at::Tensor* cu = get_tensor(o[0], &dev);
  if (!cu || !get_int(o[1], &bs) || bs <= 0 || bs > INT32_MAX || cu->dim() != 1 || cu->size(0) < 2 || cu->scalar_type() != at::kInt || !cu->is_contiguous()) Py_RETURN_NONE;
  const at::Device device(at::kCUDA, (c10::DeviceIndex)dev);
  c10::cuda::CUDAGuard guard(device);
  auto empty = [&](int64_t size) { return at::Tensor(at::detail::empty_cuda({size}, at::kInt, device, std::nullopt)); };
  const int batch = (int)cu->size(0) - 1;
  at::Tensor first = empty(batch + 1), cu_block = empty(kGuess + 1), to_batch = empty(kGuess);
  void* const stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  // sizes and storage: a table that is saved takes its own bytes along, not those of the guess
  auto cut = [](at::Tensor& t, int64_t size) {
    t.unsafeGetTensorImpl()->set_sizes_contiguous({size});
    t.unsafeGetTensorImpl()->unsafe_storage().set_nbytes((size_t)size * sizeof(int32_t));
  };
  auto at_i32 = [](const at::Tensor& t) { return static_cast<int32_t*>(t.data_ptr()); };
  int32_t num = 0;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = lib.blocks_counted(at_i32(*cu), batch, (int)bs, (int)kGuess, at_i32(cu_block), at_i32(to_batch), at_i32(first), &num, stream);
  Py_END_ALLOW_THREADS
  if (rc == 0 && num > kGuess) {
    cu_block = empty(num + 1);
    to_batch = empty(num);
    rc = lib.blocks(at_i32(*cu), batch, (int)bs, num, at_i32(cu_block), at_i32(to_batch), at_i32(first), stream);
  } else if (rc == 0) {
    cut(cu_block, num + 1);
    cut(to_batch, num);
  }
  if (rc != 0) {
    fail("hbsa_calculate_blocks", rc);
    return nullptr;
  }
  PyObject* r = PyTuple_New(4);
  if (!r) return nullptr;
  PyTuple_SET_ITEM(r, 0, PyLong_FromLong(num));
  PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(cu_block));
  PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(to_batch));
  PyTuple_SET_ITEM(r, 3, THPVariable_Wrap(first));
  return r;
  END_HANDLE_TH_ERRORS
}

// setup(state dict, addresses of the library's functions in the order of `Library`)
PyObject* py_setup(PyObject*, PyObject* args) {
  PyObject *state, *addr;
  if (!PyArg_ParseTuple(args, "O!O!", &PyDict_Type, &state, &PyTuple_Type, &addr)) return nullptr;
  void** const slots = reinterpret_cast<void**>(&lib);
  constexpr Py_ssize_t count = sizeof(lib) / sizeof(void*);
  if (PyTuple_GET_SIZE(addr) != count) {
    PyErr_SetString(PyExc_ValueError, "setup: wrong number of function addresses");
    return nullptr;
  }
  for (Py_ssize_t i = 0; i < count; ++i) {
    slots[i] = PyLong_AsVoidPtr(PyTuple_GET_ITEM(addr, i));
    if (PyErr_Occurred()) return nullptr;
  }
  Py_XDECREF(g_state);
  g_state = Py_NewRef(state);
  Py_RETURN_NONE;
}

#define HBSA_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {HBSA_METHOD(attention), HBSA_METHOD(forward), HBSA_METHOD(scheduled), HBSA_METHOD(backward), HBSA_METHOD(calculate_blocks),
                         {"setup", py_setup, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  s_impl = PyUnicode_InternFromString("impl");
  s_last_workspace = PyUnicode_InternFromString("last_workspace");
  return s_impl && s_last_workspace ? PyModule_Create(&module) : nullptr;
}
