// Native call path of the Python entry points (extension module `_native`).
//
// A decode step of a short batch takes the GPU ten to twenty microseconds; the same call made of Python attribute
// accesses, ctypes conversions and context managers took the host 22 us (16 us for a cache write), so small steps ran at
// the speed of the interpreter.  Here the common form of a call is checked, filled into the C ABI's argument block and
// launched from one C function.  Every function returns None (False) without having done anything when the call is
// not of the common form: another layout or dtype, a host tensor, an argument that is wrong.  The Python caller then
// goes through its own checks, which also word the error messages, and through ctypes.
//
// The GIL is let go around allocations and launches: a launch blocks while the stream's queue is full, and what is queued may wait
// for another Python thread (a host callback, say).
//
// The kernels stay behind the C ABI: bind() receives the addresses of its functions from the loaded library, so this
// module works with whichever build of the library was loaded and links against none.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdlib>
#include <string>

#include <ATen/ATen.h>
#include <ATen/core/CachingHostAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/mla_fp4_b200.h"

namespace {

struct Abi {
  decltype(&mla_fp4_decode) decode = nullptr;
  decltype(&mla_fp4_workspace_bytes) workspace_bytes = nullptr;
  decltype(&mla_fp4_cache_write) cache_write = nullptr;
  decltype(&mla_fp4_step_metadata) step_metadata = nullptr;
  decltype(&mla_fp4_last_error) last_error = nullptr;
} abi;

// Without the GIL for as long as it lives.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  NoGil() = default;
  NoGil(const NoGil&) = delete;
  NoGil& operator=(const NoGil&) = delete;
  ~NoGil() { PyEval_RestoreThread(state); }
};

// The exception that the Python binding raises for a status (_cabi.check).
PyObject* raise_status(int rc) {
  const std::string msg = abi.last_error();
  if (rc == MLA_FP4_ERR_BAD_ARG || rc == MLA_FP4_ERR_UNSUPPORTED || rc == MLA_FP4_ERR_WORKSPACE_TOO_SMALL)
    PyErr_SetString(PyExc_ValueError, msg.c_str());
  else
    PyErr_Format(PyExc_RuntimeError, "mla_fp4 error %d: %s", rc, msg.c_str());
  return nullptr;
}

const at::Tensor* tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }
bool on(const at::Tensor& t, const at::Device& d) { return t.is_cuda() && t.device() == d; }
// A number as a double / an integer; anything else (a tensor, say) is left to the Python path.
bool number(PyObject* o, double* v) {
  if (PyFloat_Check(o)) *v = PyFloat_AS_DOUBLE(o);
  else if (PyLong_Check(o)) *v = PyLong_AsDouble(o);
  else return false;
  if (*v == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}
bool integer(PyObject* o, int64_t* v) {
  if (!PyLong_Check(o)) return false;
  int overflow = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}

// bind(decode, workspace_bytes, cache_write, step_metadata, last_error): addresses in the loaded library
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5) return PyErr_Format(PyExc_TypeError, "bind takes 5 addresses");
  void* p[5];
  for (int i = 0; i < 5; ++i) {
    p[i] = PyLong_AsVoidPtr(a[i]);
    if (!p[i]) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "null address");
  }
  abi.decode = reinterpret_cast<decltype(abi.decode)>(p[0]);
  abi.workspace_bytes = reinterpret_cast<decltype(abi.workspace_bytes)>(p[1]);
  abi.cache_write = reinterpret_cast<decltype(abi.cache_write)>(p[2]);
  abi.step_metadata = reinterpret_cast<decltype(abi.step_metadata)>(p[3]);
  abi.last_error = reinterpret_cast<decltype(abi.last_error)>(p[4]);
  Py_RETURN_NONE;
}

// decode(workspace, status, num_heads, page_size, out_code, kernel, num_ctas, pdl, phase_mask, soft_cap, sink, wait_polls,
//        q, kv_cache, block_tables, seq_lens, max_seq_len, softmax_scale, output_scale, out, kv_cache_sf, return_lse, lse_out)
// -> out, (out, lse), or None when the call is not of the common form.
PyObject* decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 23) return PyErr_Format(PyExc_TypeError, "decode takes 23 arguments");
  const at::Tensor *ws = tensor(a[0]), *status = tensor(a[1]), *q = tensor(a[12]), *kv = tensor(a[13]), *bt = tensor(a[14]),
                   *sl = tensor(a[15]), *sf = tensor(a[20]);
  if (!ws || !status || !q || !kv || !bt || !sl || !sf) Py_RETURN_NONE;
  int64_t heads, page, out_code, kernel, ctas, phase, polls, max_len;
  double cap, scale, out_scale;
  if (!integer(a[2], &heads) || !integer(a[3], &page) || !integer(a[4], &out_code) || !integer(a[5], &kernel) || !integer(a[6], &ctas) ||
      !integer(a[8], &phase) || !number(a[9], &cap) || !integer(a[11], &polls) || !integer(a[16], &max_len) || !number(a[17], &scale) ||
      !number(a[18], &out_scale))
    Py_RETURN_NONE;
  const at::Device dev = ws->device();
  if (!on(*q, dev) || !on(*kv, dev) || !on(*bt, dev) || !on(*sl, dev) || !on(*sf, dev) || !on(*status, dev)) Py_RETURN_NONE;
  if (q->dim() != 4 || q->size(2) != heads || q->size(3) != MLA_FP4_LATENT_DIM + MLA_FP4_ROPE_DIM || q->stride(3) != 1 ||
      q->scalar_type() != at::kFloat8_e4m3fn)
    Py_RETURN_NONE;
  const int64_t batch = q->size(0), q_len = q->size(1);
  if (kv->dim() != 3 || kv->scalar_type() != at::kByte || kv->size(1) != page || kv->size(2) != MLA_FP4_ROW_BYTES || !kv->is_contiguous())
    Py_RETURN_NONE;
  if (sf->dim() != 3 || sf->scalar_type() != at::kFloat || sf->size(0) != kv->size(0) || sf->size(1) != page || sf->size(2) != 1 ||
      !sf->is_contiguous())
    Py_RETURN_NONE;
  if (bt->dim() != 2 || bt->scalar_type() != at::kInt || bt->stride(1) != 1 || bt->size(0) != batch) Py_RETURN_NONE;
  if (sl->dim() != 1 || sl->scalar_type() != at::kInt || sl->size(0) != batch || !sl->is_contiguous()) Py_RETURN_NONE;
  if (max_len <= 0 || max_len > bt->size(1) * page) Py_RETURN_NONE;
  const char* validate = std::getenv("MLA_FP4_VALIDATE");
  if (validate && *validate && !(validate[0] == '0' && !validate[1])) Py_RETURN_NONE;  // page ids are checked on the host first
  size_t need = 0;
  if (abi.workspace_bytes(int32_t(batch), int32_t(q_len), int32_t(heads), int32_t(ctas), &need) != MLA_FP4_OK || size_t(ws->numel()) < need)
    Py_RETURN_NONE;
  const at::ScalarType out_type =
      out_code == MLA_FP4_OUT_BF16 ? at::kBFloat16 : (out_code == MLA_FP4_OUT_F32 ? at::kFloat : at::kFloat8_e4m3fn);
  const int64_t shape[4] = {batch, q_len, heads, MLA_FP4_LATENT_DIM};
  const bool given = a[19] != Py_None;
  at::Tensor out;
  if (given) {
    const at::Tensor* o = tensor(a[19]);
    if (!o || !on(*o, dev) || o->scalar_type() != out_type || o->sizes() != at::IntArrayRef(shape, 4) || !o->is_contiguous()) Py_RETURN_NONE;
    out = *o;
  }
  const int want_lse = PyObject_IsTrue(a[21]);
  if (want_lse < 0) return nullptr;
  at::Tensor lse;
  const bool lse_given = want_lse && a[22] != Py_None;
  if (lse_given) {
    const at::Tensor* l = tensor(a[22]);
    if (!l || !on(*l, dev) || l->scalar_type() != at::kFloat || l->sizes() != at::IntArrayRef(shape, 3) || !l->is_contiguous()) Py_RETURN_NONE;
    lse = *l;
  }
  const at::Tensor* sink = a[10] == Py_None ? nullptr : tensor(a[10]);
  if (a[10] != Py_None && !sink) Py_RETURN_NONE;
  const int pdl = PyObject_IsTrue(a[7]);
  if (pdl < 0) return nullptr;

  c10::cuda::CUDAGuard guard(dev);
  MlaFp4DecodeArgs d = {};
  d.q = q->data_ptr();
  d.q_stride_batch = q->stride(0); d.q_stride_qpos = q->stride(1); d.q_stride_head = q->stride(2);
  d.kv_cache = kv->data_ptr();
  d.kv_cache_sf = static_cast<const float*>(sf->data_ptr());
  d.block_tables = static_cast<const int32_t*>(bt->data_ptr());
  d.block_table_stride = bt->stride(0);
  d.seq_lens = static_cast<const int32_t*>(sl->data_ptr());
  d.workspace = ws->data_ptr();
  d.workspace_bytes = size_t(ws->numel());
  d.status = static_cast<int32_t*>(status->data_ptr());
  d.batch = int32_t(batch); d.q_len = int32_t(q_len); d.num_heads = int32_t(heads); d.page_size = int32_t(page);
  d.num_pages = kv->size(0);
  d.softmax_scale = float(scale); d.output_scale = float(out_scale);
  d.out_dtype = int32_t(out_code); d.kernel = int32_t(kernel); d.num_ctas = int32_t(ctas);
  d.enable_pdl = pdl; d.phase_mask = int32_t(phase);
  d.stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  d.max_pages_per_request = int32_t(bt->size(1));
  d.max_seq_len = int32_t(max_len < INT32_MAX ? max_len : INT32_MAX);
  d.wait_polls = int32_t(polls);
  d.logits_soft_cap = float(cap);
  d.sink = sink ? static_cast<const float*>(sink->data_ptr()) : nullptr;
  int rc;
  {
    NoGil released;
    if (!given) out = at::empty(at::IntArrayRef(shape, 4), at::TensorOptions().dtype(out_type).device(dev));
    if (want_lse && !lse_given) lse = at::empty(at::IntArrayRef(shape, 3), at::TensorOptions().dtype(at::kFloat).device(dev));
    d.out = out.data_ptr();
    d.lse = want_lse ? static_cast<float*>(lse.data_ptr()) : nullptr;
    rc = abi.decode(&d);
  }
  if (rc != MLA_FP4_OK) return raise_status(rc);
  PyObject* po = given ? Py_NewRef(a[19]) : THPVariable_Wrap(std::move(out));
  if (!po || !want_lse) return po;
  PyObject* pl = lse_given ? Py_NewRef(a[22]) : THPVariable_Wrap(std::move(lse));
  if (!pl) {
    Py_DECREF(po);
    return nullptr;
  }
  PyObject* both = PyTuple_Pack(2, po, pl);
  Py_DECREF(po);
  Py_DECREF(pl);
  return both;
  END_HANDLE_TH_ERRORS
}

// write_tokens(latent, rope, slot_mapping, kv_cache, kv_cache_sf, token_scale) -> whether it was launched
PyObject* write_tokens(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6) return PyErr_Format(PyExc_TypeError, "write_tokens takes 6 arguments");
  const at::Tensor *lat = tensor(a[0]), *rope = tensor(a[1]), *kv = tensor(a[3]), *sf = tensor(a[4]);
  const at::Tensor *slots = a[2] == Py_None ? nullptr : tensor(a[2]), *ts = a[5] == Py_None ? nullptr : tensor(a[5]);
  if (!lat || !rope || !kv || !sf || (a[2] != Py_None && !slots) || (a[5] != Py_None && !ts)) Py_RETURN_FALSE;
  const at::Device dev = lat->device();
  if (!lat->is_cuda() || !on(*rope, dev) || !on(*kv, dev) || !on(*sf, dev) || (slots && !on(*slots, dev)) || (ts && !on(*ts, dev)))
    Py_RETURN_FALSE;
  if (lat->dim() != 2 || rope->dim() != 2 || lat->size(1) != MLA_FP4_LATENT_DIM || rope->size(1) != MLA_FP4_ROPE_DIM ||
      lat->size(0) != rope->size(0) || lat->stride(1) != 1 || rope->stride(1) != 1 || lat->scalar_type() != rope->scalar_type())
    Py_RETURN_FALSE;
  int in_type;
  if (lat->scalar_type() == at::kBFloat16) in_type = MLA_FP4_IN_BF16;
  else if (lat->scalar_type() == at::kHalf) in_type = MLA_FP4_IN_F16;
  else if (lat->scalar_type() == at::kFloat) in_type = MLA_FP4_IN_F32;
  else Py_RETURN_FALSE;
  const int64_t tokens = lat->size(0);
  if (kv->dim() < 1 || kv->scalar_type() != at::kByte || kv->size(-1) != MLA_FP4_ROW_BYTES || !kv->is_contiguous()) Py_RETURN_FALSE;
  const int64_t num_slots = kv->numel() / MLA_FP4_ROW_BYTES;
  if (sf->scalar_type() != at::kFloat || !sf->is_contiguous() || sf->numel() != num_slots) Py_RETURN_FALSE;
  if (slots && (slots->scalar_type() != at::kLong || slots->numel() != tokens || !slots->is_contiguous())) Py_RETURN_FALSE;
  if (ts && (ts->scalar_type() != at::kFloat || ts->numel() != tokens || !ts->is_contiguous())) Py_RETURN_FALSE;
  c10::cuda::CUDAGuard guard(dev);
  const void *lat_p = lat->data_ptr(), *rope_p = rope->data_ptr();
  const int64_t lat_stride = lat->stride(0), rope_stride = rope->stride(0);
  const float* ts_p = ts ? static_cast<const float*>(ts->data_ptr()) : nullptr;
  const int64_t* slots_p = slots ? static_cast<const int64_t*>(slots->data_ptr()) : nullptr;
  void* kv_p = kv->data_ptr();
  float* sf_p = static_cast<float*>(sf->data_ptr());
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  int rc;
  {
    NoGil released;
    rc = abi.cache_write(lat_p, lat_stride, rope_p, rope_stride, in_type, ts_p, slots_p, tokens, kv_p, sf_p, num_slots, stream);
  }
  if (rc != MLA_FP4_OK) return raise_status(rc);
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// Where the GPU reads a tensor: its device memory, or pinned host memory through its device address; null when it cannot
// (pageable memory).
const void* readable(const at::Tensor& t, const at::Device& dev) {
  if (t.is_cuda()) return t.device() == dev ? t.data_ptr() : nullptr;
  if (!t.is_cpu()) return nullptr;
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, t.data_ptr()) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  return at.type == cudaMemoryTypeHost ? at.devicePointer : nullptr;
}

// Whether the memory that a tensor at p spans meets that of another (neither is empty).
size_t span(const at::Tensor& t) {
  int64_t elements = 1;
  for (int64_t d = 0; d < t.dim(); ++d) elements += (t.size(d) - 1) * t.stride(d);
  return size_t(elements) * t.element_size();
}
bool meets(const void* p, const at::Tensor& t, const at::Tensor& buffer) {
  const auto a = reinterpret_cast<uintptr_t>(p), b = reinterpret_cast<uintptr_t>(buffer.data_ptr());
  return a < b + span(buffer) && b < a + span(t);
}

// step_metadata(block_tables, seq_lens, slot_mapping, dst_block_tables, dst_seq_lens, dst_slot_mapping, page_size, q_len)
// -> whether it was launched
PyObject* step_metadata(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8) return PyErr_Format(PyExc_TypeError, "step_metadata takes 8 arguments");
  const at::Tensor *bt = tensor(a[0]), *sl = tensor(a[1]), *dbt = tensor(a[3]), *dsl = tensor(a[4]), *dsm = tensor(a[5]);
  const at::Tensor* sm = a[2] == Py_None ? nullptr : tensor(a[2]);
  int64_t page, q_len;
  if (!bt || !sl || !dbt || !dsl || !dsm || (a[2] != Py_None && !sm) || !integer(a[6], &page) || !integer(a[7], &q_len)) Py_RETURN_FALSE;
  if (bt->dim() != 2 || bt->scalar_type() != at::kInt || bt->stride(1) != 1 || sl->dim() != 1 || sl->stride(0) != 1 ||
      (sl->scalar_type() != at::kInt && sl->scalar_type() != at::kLong) || bt->numel() == 0)
    Py_RETURN_FALSE;
  if (sm && (sm->scalar_type() != at::kLong || !sm->is_contiguous())) Py_RETURN_FALSE;
  if (!dsl->is_cuda()) Py_RETURN_FALSE;
  const at::Device dev = dsl->device();
  // The buffers are public attributes of the backend: what is not of the form it made them in is the general path's.
  if (!on(*dbt, dev) || dbt->dim() != 2 || dbt->scalar_type() != at::kInt || dbt->stride(1) != 1 || dbt->size(0) < bt->size(0) ||
      dbt->size(1) < bt->size(1) || (dbt->size(0) > 1 && dbt->stride(0) < dbt->size(1)) || dsl->dim() != 1 || dsl->scalar_type() != at::kInt ||
      !dsl->is_contiguous() || dsl->size(0) < sl->size(0) || bt->size(0) != sl->size(0) || !on(*dsm, dev) || dsm->scalar_type() != at::kLong ||
      !dsm->is_contiguous() || q_len <= 0 || dsm->numel() != dsl->size(0) * q_len || (sm && sm->numel() != bt->size(0) * q_len))
    Py_RETURN_FALSE;
  c10::cuda::CUDAGuard guard(dev);
  const void *pbt = readable(*bt, dev), *psl = readable(*sl, dev), *psm = sm ? readable(*sm, dev) : nullptr;
  if (!pbt || !psl || (sm && !psm)) Py_RETURN_FALSE;
  // Sources inside the buffers (a backend's own rows, moved up, say) are the general path's: one kernel would read what it writes.
  if (sl->numel() == 0 || (sm && sm->numel() == 0)) Py_RETURN_FALSE;
  for (const at::Tensor* dst : {dbt, dsl, dsm})
    if (meets(pbt, *bt, *dst) || meets(psl, *sl, *dst) || (sm && meets(psm, *sm, *dst))) Py_RETURN_FALSE;
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(dev.index());
  const int64_t bt_stride = bt->stride(0), dbt_stride = dbt->stride(0);
  const int32_t width = int32_t(bt->size(1)), batch = int32_t(bt->size(0)), max_batch = int32_t(dsl->size(0)), wide = sl->scalar_type() == at::kLong ? 1 : 0;
  int32_t *dbt_p = static_cast<int32_t*>(dbt->data_ptr()), *dsl_p = static_cast<int32_t*>(dsl->data_ptr());
  int64_t* dsm_p = static_cast<int64_t*>(dsm->data_ptr());
  at::Tensor pinned[3];  // kept while they are handed to the allocator
  int n_pinned = 0;
  for (const at::Tensor* t : {bt, sl, sm})
    if (t && !t->is_cuda()) pinned[n_pinned++] = *t;
  int rc;
  {
    NoGil released;
    rc = abi.step_metadata(static_cast<const int32_t*>(pbt), bt_stride, width, psl, wide, static_cast<const int64_t*>(psm), batch, int32_t(page),
                           int32_t(q_len), dbt_p, dbt_stride, dsl_p, dsm_p, max_batch, stream.stream());
    if (rc == MLA_FP4_OK)
      for (int i = 0; i < n_pinned; ++i)  // pinned memory that the caller lets go now is not handed out again before the kernel has read it
        at::getHostAllocator(at::kCUDA)->record_event(pinned[i].data_ptr(), pinned[i].storage().data_ptr().get_context(), stream);
  }
  if (rc != MLA_FP4_OK) return raise_status(rc);
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, nullptr},
    {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(decode)), METH_FASTCALL, nullptr},
    {"write_tokens", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(write_tokens)), METH_FASTCALL, nullptr},
    {"step_metadata", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(step_metadata)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
