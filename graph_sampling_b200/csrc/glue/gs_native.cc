// CPython extension behind graph_sampling_b200/ops.py: one function per operator that checks the tensors, allocates the
// outputs, calls the C ABI on torch's current stream and returns the trimmed tensors.
//
// The operators are a few microseconds of GPU work for an ordinary minibatch, and the same steps written in Python over
// ctypes took 30 - 50 us per call (an object per argument, an allocation through the dispatcher and a view per output).
// Functions take positional arguments only; ops.py keeps the documented signatures.  Every function releases the GIL
// around the C ABI calls, as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <exception>
#include <string>
#include <vector>

#include "../../../include/gsb200.h"

namespace {

using at::Tensor;

PyObject* g_error = nullptr;  // graph_sampling_b200.cabi.GsbError

struct PyErrorSet : std::exception {};  // a Python exception is already set

[[noreturn]] void type_error(const std::string& what) {
  PyErr_SetString(PyExc_TypeError, what.c_str());
  throw PyErrorSet();
}

// An operand: the tensor a pointer was taken from, kept alive (a contiguous copy when the caller's was not contiguous).
struct Arg {
  Tensor hold;
  const Tensor* t = nullptr;
  bool given() const { return t != nullptr; }
  int64_t numel() const { return t->numel(); }
  const int64_t* ids() const { return t ? static_cast<const int64_t*>(t->const_data_ptr()) : nullptr; }
  const float* floats() const { return t ? static_cast<const float*>(t->const_data_ptr()) : nullptr; }
};

Arg operand(PyObject* o, const char* name, bool optional, at::ScalarType dtype, const char* dtype_name) {
  Arg a;
  if (o == Py_None) {
    if (optional) return a;
    type_error(std::string(name) + " is required");
  }
  // device memory, or page-locked host memory that the kernels read in place
  if (!THPVariable_Check(o)) type_error(std::string(name) + " must be " + dtype_name + " CUDA (or pinned host) tensor");
  const Tensor& t = THPVariable_Unpack(o);
  if (t.scalar_type() != dtype || !(t.is_cuda() || t.is_pinned()))
    type_error(std::string(name) + " must be " + dtype_name + " CUDA (or pinned host) tensor");
  if (t.is_contiguous()) {
    a.t = &t;
  } else {
    if (!t.is_cuda()) type_error(std::string(name) + ": a pinned host tensor must be contiguous");
    a.hold = t.contiguous();
    a.t = nullptr;
  }
  return a;
}
// (the address of `hold` is only stable in its final place)
void settle(Arg& a) {
  if (!a.t && a.hold.defined()) a.t = &a.hold;
}
// A tensor the caller provides for the results.
Arg destination(PyObject* o, const char* name) {
  Arg a = operand(o, name, false, at::kFloat, "a float32");
  if (!a.t) type_error(std::string(name) + " must be contiguous");
  return a;
}
#define IDS(var, obj, name) \
  Arg var = operand(obj, name, false, at::kLong, "an int64"); \
  settle(var)
#define IDS_OR_NONE(var, obj, name) \
  Arg var = operand(obj, name, true, at::kLong, "an int64"); \
  settle(var)
#define FLOATS(var, obj, name) \
  Arg var = operand(obj, name, false, at::kFloat, "a float32"); \
  settle(var)
#define FLOATS_OR_NONE(var, obj, name) \
  Arg var = operand(obj, name, true, at::kFloat, "a float32"); \
  settle(var)

int64_t integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyErrorSet();
  return v;
}
uint64_t unsigned_integer(PyObject* o) {
  const unsigned long long v = PyLong_AsUnsignedLongLong(o);
  if (v == (unsigned long long)-1 && PyErr_Occurred()) throw PyErrorSet();
  return v;
}
bool truth(PyObject* o) { return PyObject_IsTrue(o) == 1; }
gsb_ctx* context(PyObject* o) { return reinterpret_cast<gsb_ctx*>(unsigned_integer(o)); }

void* stream() { return static_cast<void*>(c10::cuda::getCurrentCUDAStream().stream()); }

// Results live on the operand's device, or on the current one when the operand is pinned host memory.
c10::Device device_of(const Arg& a) {
  return a.t->is_cuda() ? a.t->device() : c10::Device(c10::kCUDA, c10::cuda::current_device());
}
// Entries of an array in device memory; 0 for one that is read from the host.
int64_t device_entries(const Arg& a) { return a.t->is_cuda() ? a.numel() : 0; }
Tensor empty(int64_t n, c10::Device dev, at::ScalarType dtype = at::kLong) {
  return at::detail::empty_cuda({n}, dtype, dev, c10::nullopt);
}
int64_t* mut(const Tensor& t) { return t.defined() ? static_cast<int64_t*>(t.mutable_data_ptr()) : nullptr; }
float* mutf(const Tensor& t) { return t.defined() ? static_cast<float*>(t.mutable_data_ptr()) : nullptr; }
// The first n elements of a fresh tensor: the tensor itself is shortened, no view is made.
void trim(Tensor& t, int64_t n) {
  if (t.defined() && t.numel() != n) t.unsafeGetTensorImpl()->set_sizes_contiguous({n});
}

void check(gsb_ctx* ctx, int st, const char* where) {
  if (st == GSB_OK) return;
  PyObject* e = PyObject_CallFunction(g_error, "iss", st, where, gsb_last_error_message(ctx));
  if (e) {
    PyErr_SetObject(g_error, e);
    Py_DECREF(e);
  }
  throw PyErrorSet();
}

struct NoGil {
  PyThreadState* state;
  NoGil() : state(PyEval_SaveThread()) {}
  ~NoGil() { PyEval_RestoreThread(state); }
};

PyObject* wrap(Tensor t) {
  if (!t.defined()) Py_RETURN_NONE;
  PyObject* o = THPVariable_Wrap(std::move(t));
  if (!o) throw PyErrorSet();
  return o;
}
template <class... T>
PyObject* tuple_of(T&&... items) {
  PyObject* objs[] = {items...};
  PyObject* out = PyTuple_New(sizeof...(items));
  for (size_t i = 0; i < sizeof...(items); ++i) PyTuple_SET_ITEM(out, (Py_ssize_t)i, objs[i]);
  return out;
}

// Calls `body`, turning C++ exceptions into Python ones.
template <class F>
PyObject* guarded(Py_ssize_t got, Py_ssize_t want, F body) {
  if (got != want) {
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, got);
    return nullptr;
  }
  try {
    return body();
  } catch (const PyErrorSet&) {
    return nullptr;
  } catch (const c10::OutOfMemoryError& e) {
    PyObject* cuda_oom = nullptr;
    if (PyObject* torch = PyImport_ImportModule("torch")) {
      cuda_oom = PyObject_GetAttrString(torch, "OutOfMemoryError");
      Py_DECREF(torch);
    }
    PyErr_SetString(cuda_oom ? cuda_oom : PyExc_RuntimeError, e.what_without_backtrace());
    Py_XDECREF(cuda_oom);
    return nullptr;
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}
#define FUNCTION(name, nargs) \
  PyObject* name##_body(PyObject* const* a); \
  PyObject* name(PyObject*, PyObject* const* a, Py_ssize_t n) { \
    return guarded(n, nargs, [&] { return name##_body(a); }); \
  } \
  PyObject* name##_body(PyObject* const* a)

// ---- column slicing: (ctx, indptr, indices, column_ids | None, with_coo, with_select, data | None, e_ids | None)
//      -> (sub_indptr, coo_col | None, sub_indices, select | None, sliced data | None)
FUNCTION(col_slicing, 8) {
  gsb_ctx* ctx = context(a[0]);
  IDS(indptr, a[1], "indptr");
  IDS(indices, a[2], "indices");
  IDS_OR_NONE(cols, a[3], "column_ids");
  FLOATS_OR_NONE(data, a[6], "data");
  IDS_OR_NONE(e_ids, a[7], "e_ids");
  const c10::Device dev = device_of(indptr);
  const int64_t num_cols = indptr.numel() - 1, S = cols.given() ? cols.numel() : num_cols;
  Tensor sub_indptr = empty(S + 1, dev);
  int64_t nnz = 0;
  int st;
  {
    NoGil free;
    st = gsb_col_slice_count(ctx, stream(), indptr.ids(), num_cols, cols.ids(), S, mut(sub_indptr), &nnz);
  }
  check(ctx, st, "gsb_col_slice_count");
  Tensor sub_indices = empty(nnz, dev), select, coo_col, out_data;
  if (truth(a[5])) select = empty(nnz, dev);
  if (truth(a[4])) coo_col = empty(nnz, dev);
  if (data.given()) out_data = empty(nnz, dev, at::kFloat);
  {
    NoGil free;
    st = gsb_col_slice_fill(ctx, stream(), indptr.ids(), indices.ids(), num_cols, cols.ids(), S, mut(sub_indptr), nnz,
                            mut(sub_indices), mut(select), mut(coo_col), data.floats(), e_ids.ids(), mutf(out_data));
  }
  check(ctx, st, "gsb_col_slice_fill");
  return tuple_of(wrap(std::move(sub_indptr)), wrap(std::move(coo_col)), wrap(std::move(sub_indices)),
                  wrap(std::move(select)), wrap(std::move(out_data)));
}

// ---- uniform / weighted per-column sampling:
// (ctx, indptr, indices, probs | None, column_ids | None, fanout, replace, with_coo, with_select, seed, data | None,
//  e_ids | None) -> (sub_indptr, coo_col | None, sub_indices, select | None, sampled data | None)
FUNCTION(col_sampling, 12) {
  gsb_ctx* ctx = context(a[0]);
  IDS(indptr, a[1], "indptr");
  IDS(indices, a[2], "indices");
  FLOATS_OR_NONE(probs, a[3], "probs");
  IDS_OR_NONE(cols, a[4], "column_ids");
  const int64_t fanout = integer(a[5]);
  const int replace = truth(a[6]) ? 1 : 0;
  const uint64_t seed = unsigned_integer(a[9]);
  FLOATS_OR_NONE(data, a[10], "data");
  IDS_OR_NONE(e_ids, a[11], "e_ids");
  const c10::Device dev = device_of(indptr);
  const int64_t num_cols = indptr.numel() - 1, S = cols.given() ? cols.numel() : num_cols, cap = S * fanout;
  Tensor sub_indptr = empty(S + 1, dev), sub_indices = empty(cap, dev), select, coo_col, out_data;
  if (truth(a[8])) select = empty(cap, dev);
  if (truth(a[7])) coo_col = empty(cap, dev);
  if (data.given()) out_data = empty(cap, dev, at::kFloat);
  int64_t nnz = 0;
  int st;
  {
    NoGil free;
    st = probs.given() ? gsb_sample_weighted(ctx, stream(), indptr.ids(), indices.ids(), num_cols, probs.floats(),
                                             cols.ids(), S, fanout, replace, seed, mut(sub_indptr), mut(sub_indices),
                                             mut(select), mut(coo_col), data.floats(), e_ids.ids(), mutf(out_data), cap,
                                             &nnz)
                       : gsb_sample_uniform_sized(ctx, stream(), indptr.ids(), indices.ids(), num_cols,
                                                  device_entries(indices), cols.ids(), S, fanout, replace, seed,
                                                  mut(sub_indptr), mut(sub_indices), mut(select), mut(coo_col),
                                                  data.floats(), e_ids.ids(), mutf(out_data), cap, &nnz);
  }
  check(ctx, st, probs.given() ? "gsb_sample_weighted" : "gsb_sample_uniform");
  trim(sub_indices, nnz);
  trim(select, nnz);
  trim(coo_col, nnz);
  trim(out_data, nnz);
  return tuple_of(wrap(std::move(sub_indptr)), wrap(std::move(coo_col)), wrap(std::move(sub_indices)),
                  wrap(std::move(select)), wrap(std::move(out_data)));
}

// ---- unique + relabel: (ctx, [item arrays], [arrays to relabel]) -> (unique, [relabelled arrays])
FUNCTION(relabel, 3) {
  gsb_ctx* ctx = context(a[0]);
  const Py_ssize_t ni = PySequence_Size(a[1]), nr = PySequence_Size(a[2]);
  if (ni < 0 || nr < 0) throw PyErrorSet();
  Arg items[GSB_MAX_SEGMENTS], rels[GSB_MAX_SEGMENTS];
  Tensor outs[GSB_MAX_SEGMENTS];
  const int64_t *item_ptr[GSB_MAX_SEGMENTS], *rel_ptr[GSB_MAX_SEGMENTS];
  int64_t item_len[GSB_MAX_SEGMENTS], rel_len[GSB_MAX_SEGMENTS], *out_ptr[GSB_MAX_SEGMENTS], n = 0;
  auto take = [](PyObject* list, Py_ssize_t i, const char* name) {
    PyObject* o = PySequence_GetItem(list, i);  // the list keeps it alive
    if (!o) throw PyErrorSet();
    Py_DECREF(o);
    return operand(o, name, false, at::kLong, "an int64");
  };
  for (Py_ssize_t i = 0; i < ni; ++i) {
    items[i] = take(a[1], i, "mapping tensor");
    settle(items[i]);
    item_len[i] = items[i].numel();
    item_ptr[i] = item_len[i] ? items[i].ids() : nullptr;
    n += item_len[i];
  }
  const c10::Device dev = device_of(items[0]);
  for (Py_ssize_t i = 0; i < nr; ++i) {
    rels[i] = take(a[2], i, "tensor to relabel");
    settle(rels[i]);
    rel_len[i] = rels[i].numel();
    rel_ptr[i] = rel_len[i] ? rels[i].ids() : nullptr;
    outs[i] = empty(rel_len[i], dev);
    if (rels[i].t->dim() != 1) outs[i].unsafeGetTensorImpl()->set_sizes_contiguous(rels[i].t->sizes());
    out_ptr[i] = rel_len[i] ? mut(outs[i]) : nullptr;
  }
  Tensor unique = empty(n, dev);
  int64_t count = 0;
  int st;
  {
    NoGil free;
    st = gsb_unique_relabel(ctx, stream(), item_ptr, item_len, (int)ni, mut(unique), rel_ptr, rel_len, out_ptr, (int)nr,
                            &count);
  }
  check(ctx, st, "gsb_unique_relabel");
  trim(unique, count);
  PyObject* list = PyList_New(nr);
  for (Py_ssize_t i = 0; i < nr; ++i) PyList_SET_ITEM(list, i, wrap(std::move(outs[i])));
  return tuple_of(wrap(std::move(unique)), list);
}

// ---- relabelling of a sampled graph: (ctx, col_ids, rows, cols | None, indptr to copy | None, relabel, id bound)
//      -> (unique, rows | None, cols | None, copy | None, ones | None, whether the bound was refused), or that alone when
//      gsb_graph_relabel does not serve the call
FUNCTION(graph_relabel, 8) {
  gsb_ctx* ctx = context(a[0]);
  IDS(col_ids, a[1], "col_ids");
  IDS(rows, a[2], "rows");
  IDS_OR_NONE(cols, a[3], "cols");
  IDS_OR_NONE(indptr, a[4], "indptr");
  const c10::Device dev = device_of(col_ids);
  const int64_t S = col_ids.numel(), E = rows.numel();
  if (cols.given() && cols.numel() != E) type_error("cols must have one entry per row id");
  Tensor unique = empty(S + E, dev), out_rows, out_cols, copy, ones;
  if (truth(a[7])) ones = empty(E, dev, at::kFloat);
  if (truth(a[5])) out_rows = empty(E, dev);
  const int64_t bound = integer(a[6]);
  if (cols.given()) out_cols = empty(E, dev);
  if (indptr.given()) copy = empty(indptr.numel(), dev);
  int64_t count = 0;
  int st;
  const int64_t refusals = gsb_id_bound_refusals(ctx);
  {
    NoGil free;
    st = gsb_graph_relabel(ctx, stream(), col_ids.ids(), S, rows.ids(), E, cols.ids(), indptr.ids(), mut(copy),
                           indptr.given() ? indptr.numel() : 0, bound, mut(unique), mut(out_rows), mut(out_cols), mutf(ones), &count);
  }
  const long refused = gsb_id_bound_refusals(ctx) != refusals;
  if (st == GSB_ERR_UNSUPPORTED) return PyBool_FromLong(refused);
  check(ctx, st, "gsb_graph_relabel");
  trim(unique, count);
  return tuple_of(wrap(std::move(unique)), wrap(std::move(out_rows)), wrap(std::move(out_cols)), wrap(std::move(copy)),
                  wrap(std::move(ones)), PyBool_FromLong(refused));
}

// ---- random walk: (ctx, indptr, indices, seeds, length, seed, layout, walker_offset) -> trace [W, L + 1]
FUNCTION(random_walk, 8) {
  gsb_ctx* ctx = context(a[0]);
  IDS(indptr, a[1], "indptr");
  IDS(indices, a[2], "indices");
  IDS(seeds, a[3], "seeds");
  const int64_t L = integer(a[4]), W = seeds.numel();
  const uint64_t seed = unsigned_integer(a[5]);
  const int layout = (int)integer(a[6]);
  const int64_t offset = integer(a[7]);
  Tensor out = empty(W * (L + 1), device_of(indptr));
  int st;
  {
    NoGil free;
    st = gsb_random_walk(ctx, stream(), indptr.ids(), indices.ids(), indptr.numel() - 1, seeds.ids(), W, L, seed, layout,
                         offset, mut(out));
  }
  check(ctx, st, "gsb_random_walk");
  out.unsafeGetTensorImpl()->set_sizes_contiguous({W, L + 1});
  return wrap(std::move(out));
}

// ---- column + row slicing: (ctx, indptr, indices, column_ids, row_ids, col_ptr | None, row_ptr | None, encoding_size,
//      with_select, data | None, e_ids | None) -> (sub_indptr, sub_indices, select | None, sliced data | None)
FUNCTION(col_row_slicing, 11) {
  gsb_ctx* ctx = context(a[0]);
  IDS(indptr, a[1], "indptr");
  IDS(indices, a[2], "indices");
  IDS(cols, a[3], "column_ids");
  IDS(rows, a[4], "row_ids");
  IDS_OR_NONE(col_ptr, a[5], "col_ptr");
  IDS_OR_NONE(row_ptr, a[6], "row_ptr");
  const int64_t encoding = integer(a[7]);
  FLOATS_OR_NONE(data, a[9], "data");
  IDS_OR_NONE(e_ids, a[10], "e_ids");
  const c10::Device dev = device_of(indptr);
  const int64_t num_cols = indptr.numel() - 1, S = cols.numel(), R = rows.numel();
  const int64_t G = col_ptr.given() ? col_ptr.numel() - 1 : 1;
  Tensor slice_indptr = empty(S + 1, dev), sub_indptr = empty(S + 1, dev);
  int64_t D = 0, nnz = 0;
  int st;
  {
    NoGil free;
    st = gsb_col_slice_count(ctx, stream(), indptr.ids(), num_cols, cols.ids(), S, mut(slice_indptr), &D);
  }
  check(ctx, st, "gsb_col_slice_count");
  Tensor sub_indices = empty(D, dev), select, out_data;
  if (truth(a[8])) select = empty(D, dev);
  if (data.given()) out_data = empty(D, dev, at::kFloat);
  {
    NoGil free;
    st = gsb_col_row_slice(ctx, stream(), indptr.ids(), indices.ids(), num_cols, cols.ids(), S, mut(slice_indptr), D,
                           rows.ids(), R, col_ptr.ids(), row_ptr.ids(), G, encoding, col_ptr.given() ? 0 : 1,
                           mut(sub_indptr), mut(sub_indices), mut(select), data.floats(), e_ids.ids(), mutf(out_data),
                           &nnz);
  }
  check(ctx, st, "gsb_col_row_slice");
  trim(sub_indices, nnz);
  trim(select, nnz);
  trim(out_data, nnz);
  return tuple_of(wrap(std::move(sub_indptr)), wrap(std::move(sub_indices)), wrap(std::move(select)),
                  wrap(std::move(out_data)));
}

// ---- list sampling: (ctx, data, picks, replace, probs | None, seed) -> (selected data, selected index)
FUNCTION(list_sampling, 6) {
  gsb_ctx* ctx = context(a[0]);
  IDS(data, a[1], "data");
  const int64_t k = integer(a[2]), N = data.numel();
  const bool replace = truth(a[3]);
  FLOATS_OR_NONE(probs, a[4], "probs");
  const uint64_t seed = unsigned_integer(a[5]);
  const int64_t room = !replace && N <= k ? N : k, cap = room > 1 ? room : 1;
  const c10::Device dev = device_of(data);
  Tensor out = empty(cap, dev), index = empty(cap, dev);
  int64_t n = 0;
  int st;
  {
    NoGil free;
    st = gsb_list_sample(ctx, stream(), data.ids(), probs.floats(), N, k, replace ? 1 : 0, seed, mut(out), mut(index), &n);
  }
  check(ctx, st, "gsb_list_sample");
  trim(out, n);
  trim(index, n);
  return tuple_of(wrap(std::move(out)), wrap(std::move(index)));
}

// ---- SDDMM into the caller's tensor: (ctx, op, row, col | None, indptr | None, e_ids | None, lhs | None, rhs | None,
//      out, lhs_target, rhs_target, lhs_len, rhs_len, out_len, reduce_size, lhs_off | None, rhs_off | None)
FUNCTION(sddmm, 17) {
  gsb_ctx* ctx = context(a[0]);
  const int op = (int)integer(a[1]);
  IDS(row, a[2], "row");
  IDS_OR_NONE(col, a[3], "col");
  IDS_OR_NONE(indptr, a[4], "indptr");
  IDS_OR_NONE(e_ids, a[5], "e_ids");
  FLOATS_OR_NONE(lhs, a[6], "lhs");
  FLOATS_OR_NONE(rhs, a[7], "rhs");
  Arg out = destination(a[8], "out");
  const int lt = (int)integer(a[9]), rt = (int)integer(a[10]);
  const int64_t lhs_len = integer(a[11]), rhs_len = integer(a[12]), out_len = integer(a[13]), reduce = integer(a[14]);
  IDS_OR_NONE(lhs_off, a[15], "lhs_off");
  IDS_OR_NONE(rhs_off, a[16], "rhs_off");
  int st;
  {
    NoGil free;
    st = gsb_sddmm(ctx, stream(), op, row.ids(), col.ids(), indptr.ids(), indptr.given() ? indptr.numel() - 1 : 0,
                   e_ids.ids(), row.numel(), lhs.floats(), rhs.floats(), mutf(*out.t), lt, rt, lhs_len, rhs_len, out_len,
                   reduce, lhs_off.ids(), rhs_off.ids());
  }
  check(ctx, st, "gsb_sddmm");
  Py_RETURN_NONE;
}

// ---- segment reductions into the caller's tensor
FUNCTION(segment_sum_csc, 6) {  // (ctx, indptr, e_ids | None, data | None, powk, out)
  gsb_ctx* ctx = context(a[0]);
  IDS(indptr, a[1], "indptr");
  IDS_OR_NONE(e_ids, a[2], "e_ids");
  FLOATS_OR_NONE(data, a[3], "data");
  const int64_t powk = integer(a[4]);
  Arg out = destination(a[5], "out");
  int st;
  {
    NoGil free;
    st = gsb_segment_sum_csc(ctx, stream(), indptr.ids(), indptr.numel() - 1, e_ids.ids(), data.floats(), powk,
                             mutf(*out.t));
  }
  check(ctx, st, "gsb_segment_sum_csc");
  Py_RETURN_NONE;
}

FUNCTION(segment_sum_coo, 7) {  // (ctx, target, e_ids | None, data | None, powk, targets_in_runs, out)
  gsb_ctx* ctx = context(a[0]);
  IDS(target, a[1], "target");
  IDS_OR_NONE(e_ids, a[2], "e_ids");
  FLOATS_OR_NONE(data, a[3], "data");
  const int64_t powk = integer(a[4]);
  const int runs = truth(a[5]) ? 1 : 0;
  Arg out = destination(a[6], "out");
  int st;
  {
    NoGil free;
    st = gsb_segment_sum_coo(ctx, stream(), target.ids(), target.numel(), e_ids.ids(), data.floats(), powk, runs,
                             mutf(*out.t));
  }
  check(ctx, st, "gsb_segment_sum_coo");
  Py_RETURN_NONE;
}

FUNCTION(segment_normalize_csc, 5) {  // (ctx, indptr, e_ids | None, data, out)
  gsb_ctx* ctx = context(a[0]);
  IDS(indptr, a[1], "indptr");
  IDS_OR_NONE(e_ids, a[2], "e_ids");
  FLOATS(data, a[3], "data");
  Arg out = destination(a[4], "out");
  int st;
  {
    NoGil free;
    st = gsb_segment_normalize_csc(ctx, stream(), indptr.ids(), indptr.numel() - 1, e_ids.ids(), data.floats(),
                                   mutf(*out.t));
  }
  check(ctx, st, "gsb_segment_normalize_csc");
  Py_RETURN_NONE;
}

// ---- row slicing
FUNCTION(row_slicing_csc, 5) {  // (ctx, indptr, indices, row_ids, with_coo) -> (indptr, coo_col | None, indices, select)
  gsb_ctx* ctx = context(a[0]);
  IDS(indptr, a[1], "indptr");
  IDS(indices, a[2], "indices");
  IDS(rows, a[3], "row_ids");
  const c10::Device dev = device_of(indptr);
  const int64_t num_cols = indptr.numel() - 1, E = indices.numel();
  Tensor out_indptr = empty(num_cols + 1, dev), out = empty(E, dev), select = empty(E, dev), coo_col;
  if (truth(a[4])) coo_col = empty(E, dev);
  int64_t nnz = 0;
  int st;
  {
    NoGil free;
    st = gsb_row_slice_csc(ctx, stream(), indptr.ids(), indices.ids(), num_cols, E, rows.ids(), rows.numel(),
                           mut(out_indptr), mut(out), mut(select), mut(coo_col), &nnz);
  }
  check(ctx, st, "gsb_row_slice_csc");
  trim(out, nnz);
  trim(select, nnz);
  trim(coo_col, nnz);
  return tuple_of(wrap(std::move(out_indptr)), wrap(std::move(coo_col)), wrap(std::move(out)), wrap(std::move(select)));
}

FUNCTION(row_slicing_coo, 4) {  // (ctx, coo_row, coo_col, row_ids) -> (row, col, select)
  gsb_ctx* ctx = context(a[0]);
  IDS(row, a[1], "coo_row");
  IDS(col, a[2], "coo_col");
  IDS(rows, a[3], "row_ids");
  const c10::Device dev = device_of(row);
  const int64_t E = row.numel();
  Tensor out_row = empty(E, dev), out_col = empty(E, dev), select = empty(E, dev);
  int64_t nnz = 0;
  int st;
  {
    NoGil free;
    st = gsb_row_slice_coo(ctx, stream(), row.ids(), col.ids(), E, rows.ids(), rows.numel(), mut(out_row), mut(out_col),
                           mut(select), &nnz);
  }
  check(ctx, st, "gsb_row_slice_coo");
  trim(out_row, nnz);
  trim(out_col, nnz);
  trim(select, nnz);
  return tuple_of(wrap(std::move(out_row)), wrap(std::move(out_col)), wrap(std::move(select)));
}

// ---- format conversion
FUNCTION(csc2coo, 3) {  // (ctx, indptr, number of edges) -> column of every edge
  gsb_ctx* ctx = context(a[0]);
  IDS(indptr, a[1], "indptr");
  Tensor col = empty(integer(a[2]), device_of(indptr));
  int st;
  {
    NoGil free;
    st = gsb_csc2coo(ctx, stream(), indptr.ids(), indptr.numel() - 1, mut(col));
  }
  check(ctx, st, "gsb_csc2coo");
  return wrap(std::move(col));
}

FUNCTION(coo2csc, 5) {  // (ctx, row, col, num_cols, col_sorted) -> (indptr, row in column order, permutation | None)
  gsb_ctx* ctx = context(a[0]);
  IDS(row, a[1], "row");
  IDS(col, a[2], "col");
  const int64_t num_cols = integer(a[3]), E = row.numel();
  const bool sorted = truth(a[4]);
  const c10::Device dev = device_of(row);
  Tensor indptr = empty(num_cols + 1, dev), out_row = empty(E, dev), perm;
  if (!sorted) perm = empty(E, dev);
  int st;
  {
    NoGil free;
    st = gsb_coo2csc(ctx, stream(), col.ids(), row.ids(), E, num_cols, sorted ? 1 : 0, mut(indptr), mut(out_row),
                     mut(perm));
  }
  check(ctx, st, "gsb_coo2csc");
  return tuple_of(wrap(std::move(indptr)), wrap(std::move(out_row)), wrap(std::move(perm)));
}

// ---- row gather: (ctx, src, index) -> src[index]
FUNCTION(gather_rows, 3) {
  gsb_ctx* ctx = context(a[0]);
  if (!THPVariable_Check(a[1])) type_error("src must be a contiguous float32 tensor");
  const Tensor& src = THPVariable_Unpack(a[1]);
  if (src.scalar_type() != at::kFloat || !src.is_contiguous()) type_error("src must be a contiguous float32 tensor");
  if (!(src.is_cuda() || src.is_pinned())) type_error("src must live on the GPU or in pinned host memory");
  IDS(index, a[2], "index");
  const int64_t num_rows = src.dim() > 0 ? src.size(0) : 0, n = index.numel();
  std::vector<int64_t> shape{n};
  int64_t row_len = 1;
  for (int64_t d = 1; d < src.dim(); ++d) {
    row_len *= src.size(d);
    shape.push_back(src.size(d));
  }
  Tensor out = at::detail::empty_cuda(shape, at::kFloat, device_of(index), c10::nullopt);
  if (row_len == 0) return wrap(std::move(out));
  int st;
  {
    NoGil free;
    st = gsb_gather_rows(ctx, stream(), static_cast<const float*>(src.const_data_ptr()), num_rows, row_len, index.ids(), n,
                         mutf(out));
  }
  check(ctx, st, "gsb_gather_rows");
  return wrap(std::move(out));
}

// ---- super-batch operators
FUNCTION(batch_edge_offsets, 3) {  // (ctx, sub_indptr, seeds_ptr) -> indices_ptr
  gsb_ctx* ctx = context(a[0]);
  IDS(sub_indptr, a[1], "sub_indptr");
  IDS(seeds_ptr, a[2], "seeds_ptr");
  Tensor out = empty(seeds_ptr.numel(), device_of(seeds_ptr));
  int st;
  {
    NoGil free;
    st = gsb_batch_edge_offsets(ctx, stream(), sub_indptr.ids(), seeds_ptr.ids(), seeds_ptr.numel() - 1, mut(out));
  }
  check(ctx, st, "gsb_batch_edge_offsets");
  return wrap(std::move(out));
}

// (ctx, seeds, seeds_ptr, indices, indices_ptr, capacity, sync, num_nodes, seeds_distinct) -> (unique, unique_ptr, relabelled)
FUNCTION(batch_csr_relabel, 9) {
  gsb_ctx* ctx = context(a[0]);
  IDS(seeds, a[1], "seeds");
  IDS(seeds_ptr, a[2], "seeds_ptr");
  IDS(indices, a[3], "indices");
  IDS(indices_ptr, a[4], "indices_ptr");
  const int64_t cap = integer(a[5]), num_nodes = integer(a[7]), G = seeds_ptr.numel() - 1, S = seeds.numel();
  const bool sync = truth(a[6]);
  const int flags = truth(a[8]) ? GSB_SEEDS_DISTINCT : 0;
  const c10::Device dev = device_of(seeds);
  Tensor unique = empty(S + cap, dev), unique_ptr = empty(G + 1, dev), rel = empty(cap, dev);
  int64_t nu = 0, ne = 0;
  int st;
  {
    NoGil free;
    st = gsb_batch_unique_relabel(ctx, stream(), seeds.ids(), seeds_ptr.ids(), S, indices.ids(), indices_ptr.ids(), cap, G,
                                  num_nodes, flags, mut(unique), mut(unique_ptr), mut(rel), sync ? &nu : nullptr,
                                  sync ? &ne : nullptr);
  }
  check(ctx, st, "gsb_batch_unique_relabel");
  if (sync) {
    trim(unique, nu);
    trim(rel, ne);
  }
  return tuple_of(wrap(std::move(unique)), wrap(std::move(unique_ptr)), wrap(std::move(rel)));
}

// One hop of the batched sampler: (ctx, indptr, indices, seeds, seeds_ptr, batch_ids | None, k, edge capacity, replace,
// seed, flags, sync, buffers | None) -> (sub_indptr, indices, select, relabelled, indices_ptr, unique_ptr, unique); `buffers`
// are those seven tensors, at least as large as the results.
FUNCTION(sage_hop, 13) {
  gsb_ctx* ctx = context(a[0]);
  IDS(indptr, a[1], "indptr");
  IDS(indices, a[2], "indices");
  IDS(seeds, a[3], "seeds");
  IDS(seeds_ptr, a[4], "seeds_ptr");
  IDS_OR_NONE(batch_ids, a[5], "batch_ids");
  const int64_t k = integer(a[6]), cap = integer(a[7]), S = seeds.numel(), G = seeds_ptr.numel() - 1;
  const int replace = truth(a[8]) ? 1 : 0;
  const uint64_t seed = unsigned_integer(a[9]);
  const int flags = (int)integer(a[10]);
  const bool sync = truth(a[11]);
  const c10::Device dev = device_of(indptr);
  const int64_t sizes[7] = {S + 1, cap, cap, cap, G + 1, G + 1, S + cap};
  Tensor out[7];
  for (int i = 0; i < 7; ++i) {
    if (a[12] == Py_None) {
      out[i] = empty(sizes[i], dev);
    } else {
      PyObject* o = PyTuple_GetItem(a[12], i);
      if (!o) throw PyErrorSet();
      Arg given = operand(o, "output buffer", false, at::kLong, "an int64");
      if (!given.t || given.numel() < sizes[i]) type_error("an output buffer is too small or not contiguous");
      out[i] = *given.t;
    }
  }
  int64_t nu = 0, ne = 0;
  int st;
  {
    NoGil free;
    st = gsb_sage_hop_sized(ctx, stream(), indptr.ids(), indices.ids(), indptr.numel() - 1, device_entries(indices),
                            seeds.ids(), seeds_ptr.ids(), batch_ids.ids(), G, S, k, cap, replace, seed, flags, mut(out[0]),
                            mut(out[1]), mut(out[2]), mut(out[4]), mut(out[6]), mut(out[5]), mut(out[3]),
                            sync ? &nu : nullptr, sync ? &ne : nullptr);
  }
  check(ctx, st, "gsb_sage_hop");
  if (sync) {
    for (int i = 1; i <= 3; ++i) trim(out[i], ne);
    trim(out[6], nu);
  }
  return tuple_of(wrap(out[0]), wrap(out[1]), wrap(out[2]), wrap(out[3]), wrap(out[4]), wrap(out[5]), wrap(out[6]));
}

PyObject* set_error_class(PyObject*, PyObject* cls) {
  Py_XDECREF(g_error);
  Py_INCREF(cls);
  g_error = cls;
  Py_RETURN_NONE;
}

#define ENTRY(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {ENTRY(col_slicing),        ENTRY(col_sampling),
                         ENTRY(relabel),            ENTRY(graph_relabel),
                         ENTRY(random_walk),
                         ENTRY(col_row_slicing),    ENTRY(list_sampling),
                         ENTRY(sddmm),              ENTRY(segment_sum_csc),
                         ENTRY(segment_sum_coo),    ENTRY(segment_normalize_csc),
                         ENTRY(row_slicing_csc),    ENTRY(row_slicing_coo),
                         ENTRY(csc2coo),            ENTRY(coo2csc),
                         ENTRY(gather_rows),        ENTRY(batch_edge_offsets),
                         ENTRY(batch_csr_relabel),  ENTRY(sage_hop),
                         {"set_error_class", set_error_class, METH_O, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_gsb_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__gsb_native(void) { return PyModule_Create(&module); }
