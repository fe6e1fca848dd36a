// Storage, TensorView and Tensor as CPython types: see engine.h.
#include "engine.h"

#include <algorithm>
#include <cstddef>

namespace eng {

Globals G;

PyObject *raise_status(int status) {
  PyObject *cls = status == NT_ERR_INVALID ? PyExc_ValueError
                  : status == NT_ERR_TYPE  ? PyExc_TypeError
                  : status == NT_ERR_INDEX ? PyExc_IndexError
                                           : PyExc_RuntimeError;
  const char *msg = nt_last_error();
  PyErr_SetString(cls, msg && *msg ? msg : "unknown native error");
  return nullptr;
}

bool named_args(PyObject *const *args, Py_ssize_t n, PyObject *kwnames, std::initializer_list<const char *> names, PyObject **out) {
  const Py_ssize_t want = Py_ssize_t(names.size()), nkw = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
  if (n > want) {
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
    return false;
  }
  for (Py_ssize_t i = 0; i < want; ++i) out[i] = i < n ? args[i] : nullptr;
  for (Py_ssize_t k = 0; k < nkw; ++k) {
    Py_ssize_t at = 0;
    for (const char *name : names) {
      if (PyUnicode_CompareWithASCIIString(PyTuple_GET_ITEM(kwnames, k), name) == 0) break;
      ++at;
    }
    if (at == want || out[at]) {
      PyErr_Format(PyExc_TypeError, "unexpected or repeated keyword argument '%U'", PyTuple_GET_ITEM(kwnames, k));
      return false;
    }
    out[at] = args[n + k];
  }
  for (Py_ssize_t i = 0; i < want; ++i)
    if (!out[i]) {
      PyErr_Format(PyExc_TypeError, "missing argument '%s'", names.begin()[i]);
      return false;
    }
  return true;
}

int parse_dtype(PyObject *o) {
  for (int i = 0; i < 5; ++i)
    if (G.dtypes[i] == o) return i;
  PyErr_Format(PyExc_TypeError, "expected a Dtype, got %s", Py_TYPE(o)->tp_name);
  return -1;
}
int parse_device(PyObject *o) {
  for (int i = 0; i < 2; ++i)
    if (G.devices[i] == o) return i;
  PyErr_Format(PyExc_TypeError, "expected a Device, got %s", Py_TYPE(o)->tp_name);
  return -1;
}

// =============================================================================================
// Storage
PyObject *wrap_storage(nt_storage *s) {
  PyTypeObject *tp = G.storage_type ? G.storage_type : &StorageBase_Type;
  PyObject *o = tp->tp_alloc(tp, 0);
  if (!o) {
    nt_storage_release(s);
    return nullptr;
  }
  reinterpret_cast<StorageObj *>(o)->h = s;
  return o;
}
static nt_storage *handle(PyObject *self) { return reinterpret_cast<StorageObj *>(self)->h; }

static void storage_dealloc(PyObject *self) {
  nt_storage *h = handle(self);
  if (h) nt_storage_release(h);
  Py_TYPE(self)->tp_free(self);
}
static int storage_init(PyObject *, PyObject *, PyObject *) {
  PyErr_SetString(PyExc_TypeError, "Storage: use Storage.allocate or Storage.from_iterable");
  return -1;
}
static PyObject *storage_wrap(PyObject *, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  PyObject *arg;
  if (!named_args(args, n, kwnames, {"handle"}, &arg)) return nullptr;
  void *p = PyLong_AsVoidPtr(arg);
  if (!p) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "null storage");
    return nullptr;
  }
  return wrap_storage(static_cast<nt_storage *>(p));
}
static PyObject *storage_allocate(PyObject *, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  PyObject *a[3];
  if (!named_args(args, n, kwnames, {"n", "dtype", "device"}, a)) return nullptr;
  const long long count = PyLong_AsLongLong(a[0]);
  if (count == -1 && PyErr_Occurred()) return nullptr;
  const int dt = parse_dtype(a[1]);
  if (dt < 0) return nullptr;
  const int dev = parse_device(a[2]);
  if (dev < 0) return nullptr;
  nt_storage *s = nullptr;
  const int rc = nt_storage_allocate(count, dt, dev, &s);
  return rc ? raise_status(rc) : wrap_storage(s);
}
static PyObject *storage_clone(PyObject *self, PyObject *) {
  nt_storage *s = nullptr;
  const int rc = nogil([&] { return nt_storage_clone(handle(self), &s); });
  return rc ? raise_status(rc) : wrap_storage(s);
}
static PyObject *storage_to(PyObject *self, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  PyObject *device;
  if (!named_args(args, n, kwnames, {"device"}, &device)) return nullptr;
  const int dev = parse_device(device);
  if (dev < 0) return nullptr;
  if (dev == handle(self)->device) return own(self);
  nt_storage *s = nullptr;
  const int rc = unlocked([&] { return nt_storage_to(handle(self), dev, &s); });
  return rc ? raise_status(rc) : wrap_storage(s);
}
static PyObject *storage_cast(PyObject *self, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  PyObject *dtype;
  if (!named_args(args, n, kwnames, {"dtype"}, &dtype)) return nullptr;
  const int dt = parse_dtype(dtype);
  if (dt < 0) return nullptr;
  if (dt == handle(self)->dtype) return own(self);
  nt_storage *s = nullptr;
  const int rc = nogil([&] { return nt_storage_cast(handle(self), dt, &s); });
  return rc ? raise_status(rc) : wrap_storage(s);
}
static bool pointer_and_bytes(PyObject *const *args, Py_ssize_t n, PyObject *kwnames, void **p, int64_t *nbytes) {
  PyObject *a[2];
  if (!named_args(args, n, kwnames, {"host_ptr", "nbytes"}, a)) return false;
  *p = PyLong_AsVoidPtr(a[0]);
  if (!*p && PyErr_Occurred()) return false;
  *nbytes = PyLong_AsLongLong(a[1]);
  return !(*nbytes == -1 && PyErr_Occurred());
}
static PyObject *storage_upload(PyObject *self, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  void *p;
  int64_t nbytes;
  if (!pointer_and_bytes(args, n, kwnames, &p, &nbytes)) return nullptr;
  const int rc = unlocked([&] { return nt_storage_upload(handle(self), p, nbytes); });
  if (rc) return raise_status(rc);
  Py_RETURN_NONE;
}
static PyObject *storage_download(PyObject *self, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  void *p;
  int64_t nbytes;
  if (!pointer_and_bytes(args, n, kwnames, &p, &nbytes)) return nullptr;
  const int rc = unlocked([&] { return nt_storage_download(handle(self), p, nbytes); });
  if (rc) return raise_status(rc);
  Py_RETURN_NONE;
}
static PyObject *storage_get_size(PyObject *self, void *) { return PyLong_FromLongLong(handle(self)->n); }
static PyObject *storage_get_itemsize(PyObject *self, void *) {
  return PyLong_FromLongLong(nt_storage_itemsize(handle(self)));
}
static PyObject *storage_get_dtype(PyObject *self, void *) { return own(G.dtypes[handle(self)->dtype]); }
static PyObject *storage_get_device(PyObject *self, void *) { return own(G.devices[handle(self)->device]); }
static PyObject *storage_get_version(PyObject *self, void *) { return PyLong_FromUnsignedLongLong(handle(self)->version); }
static PyObject *storage_get_data_ptr(PyObject *self, void *) { return PyLong_FromVoidPtr(nt_storage_data(handle(self))); }
static PyObject *storage_get_h(PyObject *self, void *) { return PyLong_FromVoidPtr(handle(self)); }

static PyMethodDef storage_methods[] = {
    {"_wrap", fast_kw(storage_wrap), METH_FASTCALL | METH_KEYWORDS | METH_STATIC, "A storage over a native handle (takes its reference)."},
    {"allocate", fast_kw(storage_allocate), METH_FASTCALL | METH_KEYWORDS | METH_STATIC, "allocate(n, dtype, device)"},
    {"clone", storage_clone, METH_NOARGS, nullptr},
    {"to", fast_kw(storage_to), METH_FASTCALL | METH_KEYWORDS, "to(device)"},
    {"cast", fast_kw(storage_cast), METH_FASTCALL | METH_KEYWORDS, "cast(dtype)"},
    {"upload", fast_kw(storage_upload), METH_FASTCALL | METH_KEYWORDS, "upload(host_ptr, nbytes)"},
    {"download", fast_kw(storage_download), METH_FASTCALL | METH_KEYWORDS, "download(host_ptr, nbytes)"},
    {}};
static PyGetSetDef storage_getset[] = {{"size", storage_get_size},       {"itemsize", storage_get_itemsize},
                                       {"dtype", storage_get_dtype},     {"device", storage_get_device},
                                       {"version", storage_get_version}, {"data_ptr", storage_get_data_ptr},
                                       {"_h", storage_get_h},            {}};
PyTypeObject StorageBase_Type = {.ob_base = PyVarObject_HEAD_INIT(nullptr, 0)};

// =============================================================================================
// TensorView
static int view_traverse(PyObject *self, visitproc visit, void *arg) {
  ViewObj *v = reinterpret_cast<ViewObj *>(self);
  Py_VISIT(v->storage);
  return 0;
}
static int view_clear(PyObject *self) {
  Py_CLEAR(reinterpret_cast<ViewObj *>(self)->storage);
  return 0;
}
static void view_dealloc(PyObject *self) {
  PyObject_GC_UnTrack(self);
  ViewObj *v = reinterpret_cast<ViewObj *>(self);
  Py_CLEAR(v->storage);
  Py_CLEAR(v->shape);
  Py_CLEAR(v->strides);
  Py_TYPE(self)->tp_free(self);
}
static int view_init(PyObject *self, PyObject *args, PyObject *kw) {
  static const char *names[] = {"storage", "shape", "strides", "offset", nullptr};
  PyObject *storage = Py_None, *shape = nullptr, *strides = nullptr, *offset = nullptr;
  if (!PyArg_ParseTupleAndKeywords(args, kw, "|OOOO", const_cast<char **>(names), &storage, &shape, &strides, &offset)) return -1;
  ViewObj *v = reinterpret_cast<ViewObj *>(self);
  Ref sh(shape ? PySequence_Tuple(shape) : PyTuple_New(0)), st(strides ? PySequence_Tuple(strides) : PyTuple_New(0));
  if (!sh || !st) return -1;
  int64_t off = 0;
  if (offset) {
    Ref i(PyNumber_Long(offset));
    if (!i) return -1;
    off = PyLong_AsLongLong(i.p);
    if (off == -1 && PyErr_Occurred()) return -1;
  }
  Py_XSETREF(v->storage, own(storage));
  Py_XSETREF(v->shape, sh.release());
  Py_XSETREF(v->strides, st.release());
  v->offset = off;
  return 0;
}
static PyObject *view_get(PyObject *self, void *what) {
  ViewObj *v = reinterpret_cast<ViewObj *>(self);
  switch (reinterpret_cast<intptr_t>(what)) {
  case 0: return own(v->storage ? v->storage : Py_None);
  case 1: return v->shape ? PySequence_List(v->shape) : PyList_New(0);
  case 2: return v->strides ? PySequence_List(v->strides) : PyList_New(0);
  default: return PyLong_FromLongLong(v->offset);
  }
}
static int view_set(PyObject *self, PyObject *value, void *what) {
  ViewObj *v = reinterpret_cast<ViewObj *>(self);
  if (!value) {
    PyErr_SetString(PyExc_AttributeError, "cannot delete a field of a TensorView");
    return -1;
  }
  const intptr_t w = reinterpret_cast<intptr_t>(what);
  if (w == 0) {
    Py_XSETREF(v->storage, own(value));
  } else if (w == 3) {
    Ref i(PyNumber_Long(value));
    if (!i) return -1;
    v->offset = PyLong_AsLongLong(i.p);
    if (v->offset == -1 && PyErr_Occurred()) return -1;
  } else {
    PyObject *t = PySequence_Tuple(value);
    if (!t) return -1;
    if (w == 1) Py_XSETREF(v->shape, t);
    else Py_XSETREF(v->strides, t);
  }
  return 0;
}
static PyGetSetDef view_getset[] = {{"storage", view_get, view_set, nullptr, reinterpret_cast<void *>(0)},
                                    {"shape", view_get, view_set, nullptr, reinterpret_cast<void *>(1)},
                                    {"strides", view_get, view_set, nullptr, reinterpret_cast<void *>(2)},
                                    {"offset", view_get, view_set, nullptr, reinterpret_cast<void *>(3)},
                                    {}};
PyTypeObject View_Type = {.ob_base = PyVarObject_HEAD_INIT(nullptr, 0)};

// The C view of a TensorView argument; false with an exception set.
bool view_arg(PyObject *o, nt_view *out) {
  if (!PyObject_TypeCheck(o, &View_Type)) {
    PyErr_Format(PyExc_TypeError, "expected a TensorView, got %s", Py_TYPE(o)->tp_name);
    return false;
  }
  ViewObj *v = reinterpret_cast<ViewObj *>(o);
  const Py_ssize_t nd = v->shape ? PyTuple_GET_SIZE(v->shape) : 0;
  if ((v->strides ? PyTuple_GET_SIZE(v->strides) : 0) != nd) {
    PyErr_SetString(PyExc_RuntimeError, "TensorView: shape and strides differ in length.");
    return false;
  }
  if (nd > MAXD) {
    PyErr_SetString(PyExc_RuntimeError, "TensorView: more than 8 dimensions are not supported on device.");
    return false;
  }
  if (!v->storage || !is_storage(v->storage)) {
    PyErr_SetString(PyExc_TypeError, "TensorView: storage must be a Storage.");
    return false;
  }
  out->storage = reinterpret_cast<StorageObj *>(v->storage)->h;
  out->ndim = int(nd);
  out->offset = v->offset;
  for (Py_ssize_t i = 0; i < nd; ++i) {
    out->shape[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(v->shape, i));
    if (out->shape[i] == -1 && PyErr_Occurred()) return false;
    out->strides[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(v->strides, i));
    if (out->strides[i] == -1 && PyErr_Occurred()) return false;
  }
  return true;
}

// =============================================================================================
// Tensor
PyObject *dims_tuple(int n, const int64_t *v) {
  PyObject *t = PyTuple_New(n);
  if (!t) return nullptr;
  for (int i = 0; i < n; ++i) {
    PyObject *x = PyLong_FromLongLong(v[i]);
    if (!x) {
      Py_DECREF(t);
      return nullptr;
    }
    PyTuple_SET_ITEM(t, i, x);
  }
  return t;
}
bool parse_dims(PyObject *seq, int64_t *out, int *n) {
  const bool tup = PyTuple_Check(seq);
  if (!tup && !PyList_Check(seq)) return false;
  const Py_ssize_t len = Py_SIZE(seq);
  if (len > MAXD) return false;
  for (Py_ssize_t i = 0; i < len; ++i) {
    PyObject *x = tup ? PyTuple_GET_ITEM(seq, i) : PyList_GET_ITEM(seq, i);
    if (!PyLong_Check(x)) return false;
    int overflow = 0;
    out[i] = PyLong_AsLongLongAndOverflow(x, &overflow);
    if (overflow) return false;
  }
  *n = int(len);
  return true;
}

TensorObj *alloc_tensor() {
  PyTypeObject *tp = G.tensor_type ? G.tensor_type : &TensorBase_Type;
  return reinterpret_cast<TensorObj *>(tp->tp_alloc(tp, 0)); // zero-filled
}
TensorObj *new_tensor(nt_storage *s, int nd, const int64_t *shape) {
  PyObject *so = wrap_storage(s);
  if (!so) return nullptr;
  TensorObj *t = alloc_tensor();
  if (!t) {
    Py_DECREF(so);
    return nullptr;
  }
  t->storage = so;
  t->nd = t->nst = nd;
  int64_t acc = 1;
  for (int d = nd - 1; d >= 0; --d) {
    t->sh[d] = shape[d];
    t->st[d] = acc;
    acc *= shape[d];
  }
  return t;
}
TensorObj *new_view(PyObject *storage, int nd, const int64_t *shape, const int64_t *strides, int64_t offset) {
  TensorObj *t = alloc_tensor();
  if (!t) return nullptr;
  t->storage = own(storage);
  t->nd = t->nst = nd;
  for (int d = 0; d < nd; ++d) {
    t->sh[d] = shape[d];
    t->st[d] = strides[d];
  }
  t->offset = offset;
  return t;
}
bool expand_view(const TensorObj *t, int nd, const int64_t *shape, nt_view *out) {
  const int pad = nd - t->nd;
  if (t->nd < 0 || pad < 0) return false;
  out->storage = storage_of(t);
  out->ndim = nd;
  out->offset = t->offset;
  for (int d = 0; d < nd; ++d) {
    out->shape[d] = shape[d];
    if (d < pad) {
      out->strides[d] = 0;
    } else if (t->sh[d - pad] == shape[d]) {
      out->strides[d] = t->st[d - pad];
    } else if (t->sh[d - pad] == 1) {
      out->strides[d] = 0;
    } else {
      return false;
    }
  }
  return true;
}

static TensorObj *T_(PyObject *o) { return reinterpret_cast<TensorObj *>(o); }

static int tensor_traverse(PyObject *self, visitproc visit, void *arg) {
  TensorObj *t = T_(self);
  Py_VISIT(t->storage);
  Py_VISIT(t->grad);
  Py_VISIT(t->grad_fn);
  Py_VISIT(t->pyvalue);
  return 0;
}
static int tensor_clear(PyObject *self) {
  TensorObj *t = T_(self);
  Py_CLEAR(t->grad);
  Py_CLEAR(t->grad_fn);
  Py_CLEAR(t->pyvalue);
  Py_CLEAR(t->storage);
  return 0;
}
static void tensor_dealloc(PyObject *self) {
  PyObject_GC_UnTrack(self);
  // a long chain of nodes (tensor -> function -> inputs -> ...) must not be freed by recursion
  Py_TRASHCAN_BEGIN(self, tensor_dealloc) TensorObj *t = T_(self);
  Py_CLEAR(t->grad_fn);
  Py_CLEAR(t->grad);
  Py_CLEAR(t->pyvalue);
  Py_CLEAR(t->storage);
  Py_CLEAR(t->shape);
  Py_CLEAR(t->strides);
  Py_TYPE(self)->tp_free(self);
  Py_TRASHCAN_END
}

// ---- shape and strides: tuples on the Python side, arrays here
static PyObject *shape_tuple(TensorObj *t) {
  if (!t->shape) {
    t->shape = dims_tuple(t->nd, t->sh);
    if (!t->shape) return nullptr;
  }
  return own(t->shape);
}
static PyObject *strides_tuple(TensorObj *t) {
  if (!t->strides) {
    t->strides = dims_tuple(t->nst, t->st);
    if (!t->strides) return nullptr;
  }
  return own(t->strides);
}
static PyObject *tensor_get_shape(PyObject *self, void *) { return shape_tuple(T_(self)); }
static PyObject *tensor_get_strides_(PyObject *self, void *) { return strides_tuple(T_(self)); }
static int tensor_set_shape(PyObject *self, PyObject *value, void *) {
  TensorObj *t = T_(self);
  PyObject *tup = value ? PySequence_Tuple(value) : nullptr;
  if (!tup) return -1;
  if (!parse_dims(tup, t->sh, &t->nd)) t->nd = -1;
  Py_XSETREF(t->shape, tup);
  return 0;
}
static int tensor_set_strides(PyObject *self, PyObject *value, void *) {
  TensorObj *t = T_(self);
  PyObject *tup = value ? PySequence_Tuple(value) : nullptr;
  if (!tup) return -1;
  if (!parse_dims(tup, t->st, &t->nst)) t->nd = -1;
  Py_XSETREF(t->strides, tup);
  return 0;
}
static PyObject *tensor_get_strides(PyObject *self, void *) { // Tensor.strides: (strides, offset)
  Ref st(strides_tuple(T_(self)));
  if (!st) return nullptr;
  Ref off(PyLong_FromLongLong(T_(self)->offset));
  return off ? PyTuple_Pack(2, st.p, off.p) : nullptr;
}
static PyObject *tensor_get_offset(PyObject *self, void *) { return PyLong_FromLongLong(T_(self)->offset); }
static int tensor_set_offset(PyObject *self, PyObject *value, void *) {
  if (!value) return -1;
  const long long v = PyLong_AsLongLong(value);
  if (v == -1 && PyErr_Occurred()) return -1;
  T_(self)->offset = v;
  return 0;
}
static PyObject *tensor_get_ndim(PyObject *self, void *) {
  TensorObj *t = T_(self);
  return PyLong_FromSsize_t(t->nd >= 0 ? t->nd : PyTuple_GET_SIZE(t->shape));
}
static PyObject *tensor_get_numel(PyObject *self, void *) {
  TensorObj *t = T_(self);
  if (t->nd >= 0) return PyLong_FromLongLong(numel(t->nd, t->sh));
  Ref n(PyLong_FromLong(1));
  for (Py_ssize_t i = 0; n && i < PyTuple_GET_SIZE(t->shape); ++i) n = Ref(PyNumber_Multiply(n.p, PyTuple_GET_ITEM(t->shape, i)));
  return n.release();
}
static PyObject *tensor_get_is_empty(PyObject *self, void *) {
  Ref n(tensor_get_numel(self, nullptr));
  if (!n) return nullptr;
  const int some = PyObject_IsTrue(n.p);
  return some < 0 ? nullptr : PyBool_FromLong(!some);
}
static Py_ssize_t tensor_len(PyObject *self) {
  TensorObj *t = T_(self);
  if (t->nd >= 0) return t->nd ? Py_ssize_t(t->sh[0]) : 0;
  return PyLong_AsSsize_t(PyTuple_GET_ITEM(t->shape, 0));
}

static PyObject *tensor_storage_attr(PyObject *self, void *name) { // dtype, device, version of the storage
  TensorObj *t = T_(self);
  if (!t->storage) {
    PyErr_SetString(PyExc_AttributeError, "the tensor has no storage");
    return nullptr;
  }
  return PyObject_GetAttrString(t->storage, static_cast<const char *>(name));
}
static PyObject *tensor_get_dtype(PyObject *self, void *name) {
  TensorObj *t = T_(self);
  if (t->storage && is_storage(t->storage)) return own(G.dtypes[storage_of(t)->dtype]);
  return tensor_storage_attr(self, name);
}
static PyObject *tensor_get_device(PyObject *self, void *name) {
  TensorObj *t = T_(self);
  if (t->storage && is_storage(t->storage)) return own(G.devices[storage_of(t)->device]);
  return tensor_storage_attr(self, name);
}
static PyObject *tensor_get_requires_grad(PyObject *self, void *) { return PyBool_FromLong(requires_grad(T_(self))); }
static PyObject *tensor_get_own_requires_grad(PyObject *self, void *) { return PyBool_FromLong(T_(self)->requires_grad); }
static int tensor_set_own_requires_grad(PyObject *self, PyObject *value, void *) {
  const int v = value ? PyObject_IsTrue(value) : 0;
  if (v < 0) return -1;
  T_(self)->requires_grad = char(v);
  return 0;
}
static PyObject *tensor_get_is_leaf(PyObject *self, void *) { return PyBool_FromLong(T_(self)->grad_fn == nullptr); }
static PyObject *tensor_get_field(PyObject *self, void *where) {
  PyObject *o = *reinterpret_cast<PyObject **>(reinterpret_cast<char *>(self) + reinterpret_cast<intptr_t>(where));
  return own(o ? o : Py_None);
}
static int tensor_set_field(PyObject *self, PyObject *value, void *where) {
  PyObject **slot = reinterpret_cast<PyObject **>(reinterpret_cast<char *>(self) + reinterpret_cast<intptr_t>(where));
  PyObject *old = *slot;
  *slot = (value && value != Py_None) ? own(value) : nullptr;
  Py_XDECREF(old);
  return 0;
}
static PyObject *tensor_get_pyvalue(PyObject *self, void *) {
  PyObject *v = pyvalue_of(T_(self));
  return own(v ? v : Py_None);
}
static PyObject *tensor_attach_grad_fn(PyObject *self, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  PyObject *fn;
  if (!named_args(args, n, kwnames, {"grad_fn"}, &fn)) return nullptr;
  tensor_set_field(self, fn, reinterpret_cast<void *>(offsetof(TensorObj, grad_fn)));
  Py_RETURN_NONE;
}
static PyObject *tensor_zero_grad(PyObject *self, PyObject *) {
  Py_CLEAR(T_(self)->grad);
  Py_RETURN_NONE;
}
static PyObject *tensor_enable_grad(PyObject *self, PyObject *) {
  T_(self)->requires_grad = 1;
  Py_RETURN_NONE;
}
static PyObject *tensor_C_view(PyObject *self, void *) {
  TensorObj *t = T_(self);
  Ref sh(shape_tuple(t)), st(strides_tuple(t));
  if (!sh || !st) return nullptr;
  PyObject *o = View_Type.tp_alloc(&View_Type, 0);
  if (!o) return nullptr;
  ViewObj *v = reinterpret_cast<ViewObj *>(o);
  v->storage = own(t->storage ? t->storage : Py_None);
  v->shape = sh.release();
  v->strides = st.release();
  v->offset = t->offset;
  return o;
}
static PyObject *tensor_is_contiguous(PyObject *self, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  TensorObj *t = T_(self);
  const Py_ssize_t total = n + (kwnames ? PyTuple_GET_SIZE(kwnames) : 0);
  const int full = total ? PyObject_IsTrue(args[0]) : 0; // full_span, positional or by name
  if (full < 0) return nullptr;
  bool d;
  int64_t count = 1;
  if (t->nd >= 0) {
    d = dense(t);
    count = numel(t->nd, t->sh);
  } else { // beyond MAXD dims: the same rule over the tuples
    d = true;
    for (Py_ssize_t i = PyTuple_GET_SIZE(t->shape) - 1; i >= 0; --i) {
      if (PyLong_AsLongLong(PyTuple_GET_ITEM(t->strides, i)) != count) d = false;
      count *= PyLong_AsLongLong(PyTuple_GET_ITEM(t->shape, i));
    }
  }
  if (d && full) {
    int64_t size;
    if (is_storage(t->storage)) {
      size = storage_of(t)->n;
    } else {
      Ref s(PyObject_GetAttrString(t->storage, "size"));
      if (!s) return nullptr;
      size = PyLong_AsLongLong(s.p);
    }
    d = t->offset == 0 && count == size;
  }
  return PyBool_FromLong(d);
}
static PyObject *tensor_alias(PyObject *self, PyObject *) {
  TensorObj *t = T_(self);
  if (t->nd >= 0) return reinterpret_cast<PyObject *>(alias_of(t));
  TensorObj *a = alloc_tensor();
  if (!a) return nullptr;
  a->storage = own(t->storage);
  a->shape = own(t->shape);
  a->strides = own(t->strides);
  a->offset = t->offset;
  a->nd = -1;
  return reinterpret_cast<PyObject *>(a);
}

// _new_view(storage, shape, strides or None, offset or None): bounds-checked view, IndexError past the storage
static PyObject *make_view(PyTypeObject *cls, PyObject *storage, PyObject *shape, PyObject *strides, PyObject *offset) {
  Ref sh(PySequence_Tuple(shape));
  if (!sh) return nullptr;
  const Py_ssize_t len = PyTuple_GET_SIZE(sh.p);
  std::vector<int64_t> s(static_cast<size_t>(len)), st(static_cast<size_t>(len));
  int64_t count = 1;
  for (Py_ssize_t i = 0; i < len; ++i) {
    Ref x(PyNumber_Index(PyTuple_GET_ITEM(sh.p, i)));
    if (!x) return nullptr;
    s[i] = PyLong_AsLongLong(x.p);
    if (s[i] == -1 && PyErr_Occurred()) return nullptr;
    count *= s[i];
  }
  if (strides == Py_None) {
    int64_t acc = 1;
    for (Py_ssize_t i = len - 1; i >= 0; --i) {
      st[i] = acc;
      acc *= s[i];
    }
  } else {
    Ref t(PySequence_Tuple(strides));
    if (!t) return nullptr;
    st.resize(size_t(PyTuple_GET_SIZE(t.p)));
    for (size_t i = 0; i < st.size(); ++i) {
      Ref x(PyNumber_Index(PyTuple_GET_ITEM(t.p, Py_ssize_t(i))));
      if (!x) return nullptr;
      st[i] = PyLong_AsLongLong(x.p);
      if (st[i] == -1 && PyErr_Occurred()) return nullptr;
    }
  }
  int64_t off = 0;
  if (offset != Py_None) {
    off = PyLong_AsLongLong(offset);
    if (off == -1 && PyErr_Occurred()) return nullptr;
  }
  if (count > 0) {
    int64_t lo = off, hi = off;
    for (size_t i = 0; i < st.size() && i < s.size(); ++i) (st[i] < 0 ? lo : hi) += (s[i] - 1) * st[i];
    int64_t size;
    if (is_storage(storage)) {
      size = reinterpret_cast<StorageObj *>(storage)->h->n;
    } else {
      Ref n(PyObject_GetAttrString(storage, "size"));
      if (!n) return nullptr;
      size = PyLong_AsLongLong(n.p);
      if (size == -1 && PyErr_Occurred()) return nullptr;
    }
    if (lo < 0 || hi >= size) {
      PyErr_Format(PyExc_IndexError, "View max index %lld exceeds storage capacity %lld.", static_cast<long long>(hi),
                   static_cast<long long>(size));
      return nullptr;
    }
  }
  TensorObj *t = reinterpret_cast<TensorObj *>(cls->tp_alloc(cls, 0));
  if (!t) return nullptr;
  Ref holder(reinterpret_cast<PyObject *>(t));
  t->storage = own(storage);
  t->offset = off;
  if (len <= MAXD && st.size() == size_t(len)) {
    t->nd = t->nst = int(len);
    std::copy(s.begin(), s.end(), t->sh);
    std::copy(st.begin(), st.end(), t->st);
    return holder.release();
  }
  t->nd = -1;
  t->shape = dims_tuple(int(len), s.data());
  t->strides = dims_tuple(int(st.size()), st.data());
  return t->shape && t->strides ? holder.release() : nullptr;
}
static PyObject *tensor_new_view(PyObject *cls, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  PyObject *a[4];
  if (!named_args(args, n, kwnames, {"storage", "shape", "strides", "offset"}, a)) return nullptr;
  return make_view(reinterpret_cast<PyTypeObject *>(cls), a[0], a[1], a[2], a[3]);
}
static PyObject *tensor_new_contiguous(PyObject *cls, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  PyObject *a[2];
  if (!named_args(args, n, kwnames, {"storage", "shape"}, a)) return nullptr;
  return make_view(reinterpret_cast<PyTypeObject *>(cls), a[0], a[1], Py_None, Py_None);
}

// ---- operators: XxxOp.apply(self, totensor(other, anchor=self)), as the reference binds them
static PyObject *op_apply(Op op, PyObject *const *args, Py_ssize_t n, PyObject *kwnames = nullptr) {
  if (!G.op_class[op]) {
    PyErr_SetString(PyExc_RuntimeError, "the op classes are not registered");
    return nullptr;
  }
  return apply(G.op_class[op], args, n, kwnames);
}
static PyObject *binary(Op op, PyObject *a, PyObject *b, bool commutes) {
  if (is_tensor(a)) {
    Ref other(to_operand(b, T_(a)));
    if (!other) return nullptr;
    PyObject *args[2] = {a, other.p};
    return op_apply(op, args, 2);
  }
  Ref other(to_operand(a, T_(b))); // the reflected form
  if (!other) return nullptr;
  PyObject *args[2] = {commutes ? b : other.p, commutes ? other.p : b};
  return op_apply(op, args, 2);
}
static PyObject *nb_add(PyObject *a, PyObject *b) { return binary(OP_ADD, a, b, true); }
static PyObject *nb_sub(PyObject *a, PyObject *b) { return binary(OP_SUB, a, b, false); }
static PyObject *nb_mul(PyObject *a, PyObject *b) { return binary(OP_MUL, a, b, true); }
static PyObject *nb_div(PyObject *a, PyObject *b) { return binary(OP_DIV, a, b, false); }
static PyObject *nb_pow(PyObject *a, PyObject *b, PyObject *modulus) {
  if (modulus != Py_None) Py_RETURN_NOTIMPLEMENTED;
  return binary(OP_POW, a, b, false);
}
static PyObject *nb_matmul(PyObject *a, PyObject *b) {
  if (!is_tensor(a)) Py_RETURN_NOTIMPLEMENTED;
  return binary(OP_MATMUL, a, b, false);
}
static PyObject *nb_neg(PyObject *a) { return op_apply(OP_NEG, &a, 1); }
static PyObject *inplace(Op op, PyObject *a, PyObject *b) {
  static PyObject *names = Py_BuildValue("(s)", "out");
  Ref other(to_operand(b, T_(a)));
  if (!other) return nullptr;
  PyObject *args[3] = {a, other.p, a};
  return op_apply(op, args, 2, names);
}
static PyObject *nb_iadd(PyObject *a, PyObject *b) { return inplace(OP_ADD, a, b); }
static PyObject *nb_isub(PyObject *a, PyObject *b) { return inplace(OP_SUB, a, b); }
static PyObject *nb_imul(PyObject *a, PyObject *b) { return inplace(OP_MUL, a, b); }
static PyObject *nb_idiv(PyObject *a, PyObject *b) { return inplace(OP_DIV, a, b); }

template <Op OP> static PyObject *tensor_unary(PyObject *self, PyObject *) { return op_apply(OP, &self, 1); }
static PyObject *tensor_pow(PyObject *self, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  PyObject *full[2] = {self, nullptr};
  return named_args(args, n, kwnames, {"exponent"}, full + 1) ? op_apply(OP_POW, full, 2) : nullptr;
}
// (axis=None, keepdim=False[, dtype=None]) after self
template <Op OP, int N> static PyObject *tensor_reduce(PyObject *self, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  static const char *const names[3] = {"axis", "keepdim", "dtype"};
  PyObject *full[4] = {self, Py_None, Py_False, Py_None};
  bool given[4] = {};
  if (n > N) {
    PyErr_Format(PyExc_TypeError, "expected at most %d arguments, got %zd", N, n);
    return nullptr;
  }
  for (Py_ssize_t i = 0; i < n; ++i) full[i + 1] = args[i], given[i + 1] = true;
  for (Py_ssize_t k = 0; kwnames && k < PyTuple_GET_SIZE(kwnames); ++k) {
    int at = 0;
    for (int i = 0; i < N; ++i)
      if (PyUnicode_CompareWithASCIIString(PyTuple_GET_ITEM(kwnames, k), names[i]) == 0) at = i + 1;
    if (!at || given[at]) {
      PyErr_Format(PyExc_TypeError, "unexpected or repeated keyword argument '%U'", PyTuple_GET_ITEM(kwnames, k));
      return nullptr;
    }
    full[at] = args[n + k];
    given[at] = true;
  }
  return op_apply(OP, full, 1 + N);
}
// self followed by the given dims
template <Op OP> static PyObject *tensor_dims(PyObject *self, PyObject *const *args, Py_ssize_t n) {
  PyObject *small[16];
  if (n < 16) {
    small[0] = self;
    for (Py_ssize_t i = 0; i < n; ++i) small[i + 1] = args[i];
    return op_apply(OP, small, n + 1);
  }
  std::vector<PyObject *> all(size_t(n) + 1);
  all[0] = self;
  std::copy(args, args + n, all.begin() + 1);
  return op_apply(OP, all.data(), n + 1);
}
static PyObject *tensor_transpose(PyObject *self, PyObject *const *args, Py_ssize_t n, PyObject *kwnames) {
  PyObject *full[3] = {self, nullptr, nullptr};
  return named_args(args, n, kwnames, {"dim0", "dim1"}, full + 1) ? op_apply(OP_TRANSPOSE, full, 3) : nullptr;
}
static PyObject *tensor_get_T(PyObject *self, void *) { return op_apply(OP_T, &self, 1); }

static PyObject *tensor_backward(PyObject *self, PyObject *) {
  TensorObj *t = T_(self);
  if (!requires_grad(t)) {
    PyErr_SetString(PyExc_RuntimeError,
                    "Cannot call .backward() on a tensor that does not require grad and does not have a grad_fn.");
    return nullptr;
  }
  Ref n(tensor_get_numel(self, nullptr));
  if (!n) return nullptr;
  if (PyLong_AsLongLong(n.p) != 1) {
    Ref sh(shape_tuple(t));
    PyErr_Format(PyExc_RuntimeError, "Cannot call .backward() on a non-scalar tensor of shape %R", sh.p);
    return nullptr;
  }
  // the seed: one, in the shape and dtype of the tensor
  Ref seed(PyObject_CallMethod(reinterpret_cast<PyObject *>(Py_TYPE(self)), "_scalar", "dNN", 1.0,
                               PyObject_GetAttrString(self, "dtype"), PyObject_GetAttrString(self, "device")));
  if (!seed) return nullptr;
  if (t->nd != 0) {
    Ref sh(shape_tuple(t));
    Ref storage(own(T_(seed.p)->storage));
    seed = Ref(make_view(Py_TYPE(self), storage.p, sh.p, Py_None, Py_None));
    if (!seed) return nullptr;
  }
  if (!t->grad_fn) { // a leaf's gradient is in memory, like those that leave a sweep
    const int rc = nt_storage_settle(storage_of(T_(seed.p)));
    if (rc) return raise_status(rc);
    Py_XSETREF(t->grad, seed.release());
    Py_RETURN_NONE;
  }
  Py_XSETREF(t->grad, seed.release());
  return run_backward(t);
}

static PyMethodDef tensor_methods[] = {
    {"_new_view", fast_kw(tensor_new_view), METH_FASTCALL | METH_KEYWORDS | METH_CLASS,
     "_new_view(storage, shape, strides or None, offset or None): bounds-checked view of a storage"},
    {"_new_contiguous", fast_kw(tensor_new_contiguous), METH_FASTCALL | METH_KEYWORDS | METH_CLASS,
     "_new_contiguous(storage, shape)"},
    {"_is_contiguous", fast_kw(tensor_is_contiguous), METH_FASTCALL | METH_KEYWORDS,
     "_is_contiguous(full_span=False)"},
    {"_alias", tensor_alias, METH_NOARGS, nullptr},
    {"attach_grad_fn", fast_kw(tensor_attach_grad_fn), METH_FASTCALL | METH_KEYWORDS, "attach_grad_fn(grad_fn)"},
    {"zero_grad", tensor_zero_grad, METH_NOARGS, nullptr},
    {"enable_grad", tensor_enable_grad, METH_NOARGS,
     "Enables gradient tracking after construction.  Unlike the constructor this does not look at the dtype, as in the "
     "reference (src/nanotorch/core.py:536-538; its tests call arange(60, requires_grad=True) on an Int64 range)."},
    {"backward", tensor_backward, METH_NOARGS, "Backpropagate from a one-element tensor through the recorded graph."},
    {"exp", tensor_unary<OP_EXP>, METH_NOARGS, nullptr},
    {"log", tensor_unary<OP_LOG>, METH_NOARGS, nullptr},
    {"sqrt", tensor_unary<OP_SQRT>, METH_NOARGS, nullptr},
    {"tanh", tensor_unary<OP_TANH>, METH_NOARGS, nullptr},
    {"sigmoid", tensor_unary<OP_SIGMOID>, METH_NOARGS, nullptr},
    {"relu", tensor_unary<OP_RELU>, METH_NOARGS, nullptr},
    {"pow", fast_kw(tensor_pow), METH_FASTCALL | METH_KEYWORDS, "pow(exponent)"},
    {"sum", fast_kw(tensor_reduce<OP_SUM, 3>), METH_FASTCALL | METH_KEYWORDS, "sum(axis=None, keepdim=False, dtype=None)"},
    {"mean", fast_kw(tensor_reduce<OP_MEAN, 3>), METH_FASTCALL | METH_KEYWORDS, "mean(axis=None, keepdim=False, dtype=None)"},
    {"max", fast_kw(tensor_reduce<OP_MAX, 2>), METH_FASTCALL | METH_KEYWORDS, "max(axis=None, keepdim=False)"},
    {"min", fast_kw(tensor_reduce<OP_MIN, 2>), METH_FASTCALL | METH_KEYWORDS, "min(axis=None, keepdim=False)"},
    {"reshape", reinterpret_cast<PyCFunction>(tensor_dims<OP_RESHAPE>), METH_FASTCALL, "reshape(*dims)"},
    {"expand", reinterpret_cast<PyCFunction>(tensor_dims<OP_EXPAND>), METH_FASTCALL, "expand(*dims)"},
    {"transpose", fast_kw(tensor_transpose), METH_FASTCALL | METH_KEYWORDS, "transpose(dim0, dim1)"},
    {}};

#define FIELD(name, member, set)                                                                   \
  { name, tensor_get_field, set, nullptr, reinterpret_cast<void *>(offsetof(TensorObj, member)) }
static PyGetSetDef tensor_getset[] = {
    FIELD("_storage", storage, tensor_set_field),
    FIELD("storage", storage, nullptr),
    FIELD("_grad", grad, tensor_set_field),
    FIELD("grad", grad, nullptr),
    FIELD("_grad_fn", grad_fn, tensor_set_field),
    FIELD("grad_fn", grad_fn, nullptr),
    {"_pyvalue", tensor_get_pyvalue, tensor_set_field, nullptr, reinterpret_cast<void *>(offsetof(TensorObj, pyvalue))},
    {"_shape", tensor_get_shape, tensor_set_shape},
    {"shape", tensor_get_shape},
    {"_strides", tensor_get_strides_, tensor_set_strides},
    {"strides", tensor_get_strides},
    {"_offset", tensor_get_offset, tensor_set_offset},
    {"_requires_grad", tensor_get_own_requires_grad, tensor_set_own_requires_grad},
    {"requires_grad", tensor_get_requires_grad},
    {"is_leaf", tensor_get_is_leaf},
    {"ndim", tensor_get_ndim},
    {"numel", tensor_get_numel},
    {"is_empty", tensor_get_is_empty},
    {"dtype", tensor_get_dtype, nullptr, nullptr, const_cast<char *>("dtype")},
    {"device", tensor_get_device, nullptr, nullptr, const_cast<char *>("device")},
    {"version", tensor_storage_attr, nullptr, nullptr, const_cast<char *>("version")},
    {"_C_view", tensor_C_view},
    {"T", tensor_get_T},
    {}};
static PyNumberMethods tensor_number{};
static PySequenceMethods tensor_sequence{};
PyTypeObject TensorBase_Type = {.ob_base = PyVarObject_HEAD_INIT(nullptr, 0)};

bool init_objects(PyObject *m) {
  StorageBase_Type.tp_name = "nanotorch_b200._engine.StorageBase";
  StorageBase_Type.tp_basicsize = sizeof(StorageObj);
  StorageBase_Type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE;
  StorageBase_Type.tp_dealloc = storage_dealloc;
  StorageBase_Type.tp_init = storage_init;
  StorageBase_Type.tp_new = PyType_GenericNew;
  StorageBase_Type.tp_methods = storage_methods;
  StorageBase_Type.tp_getset = storage_getset;

  View_Type.tp_name = "nanotorch_b200._engine.TensorView";
  View_Type.tp_doc = "Strided tensor view handed to the kernels (src/cpp/tensor_view.cuh:10-15, 93-102).";
  View_Type.tp_basicsize = sizeof(ViewObj);
  View_Type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC;
  View_Type.tp_traverse = view_traverse;
  View_Type.tp_clear = view_clear;
  View_Type.tp_dealloc = view_dealloc;
  View_Type.tp_init = view_init;
  View_Type.tp_new = PyType_GenericNew;
  View_Type.tp_getset = view_getset;

  tensor_number.nb_add = nb_add;
  tensor_number.nb_subtract = nb_sub;
  tensor_number.nb_multiply = nb_mul;
  tensor_number.nb_true_divide = nb_div;
  tensor_number.nb_power = nb_pow;
  tensor_number.nb_matrix_multiply = nb_matmul;
  tensor_number.nb_negative = nb_neg;
  tensor_number.nb_inplace_add = nb_iadd;
  tensor_number.nb_inplace_subtract = nb_isub;
  tensor_number.nb_inplace_multiply = nb_imul;
  tensor_number.nb_inplace_true_divide = nb_idiv;
  tensor_sequence.sq_length = tensor_len;
  TensorBase_Type.tp_name = "nanotorch_b200._engine.TensorBase";
  TensorBase_Type.tp_basicsize = sizeof(TensorObj);
  TensorBase_Type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC;
  TensorBase_Type.tp_traverse = tensor_traverse;
  TensorBase_Type.tp_clear = tensor_clear;
  TensorBase_Type.tp_dealloc = tensor_dealloc;
  TensorBase_Type.tp_new = PyType_GenericNew;
  TensorBase_Type.tp_methods = tensor_methods;
  TensorBase_Type.tp_getset = tensor_getset;
  TensorBase_Type.tp_as_number = &tensor_number;
  TensorBase_Type.tp_as_sequence = &tensor_sequence;

  struct {
    const char *name;
    PyTypeObject *type;
  } all[] = {{"StorageBase", &StorageBase_Type}, {"TensorView", &View_Type}, {"TensorBase", &TensorBase_Type}};
  for (auto &t : all) {
    if (PyType_Ready(t.type) < 0) return false;
    if (PyModule_AddObjectRef(m, t.name, reinterpret_cast<PyObject *>(t.type)) < 0) return false;
  }
  return true;
}

} // namespace eng
