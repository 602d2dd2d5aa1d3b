// Python side of the calls that a mini-batch makes: an extension module over the C functions of include/sgl_b200.h.
//
// What it replaces is interpreter time next to kernels of a few microseconds: ctypes converts a call of 30 arguments in 2 - 3 us,
// a tensor from Python costs 1.6 us, a view 0.9 - 1.2, a pointer with its checks 0.2.  A mailbox step of 41 us of kernels took 105.
//
//   sgl_*             the C function of that name: integers, None, tensors (checked as in _C.ptr) as arguments; the interpreter lock is
//                     released; a status that is not 0 raises
//   cut, cuts         views of pieces of one tensor of 8-byte words
//   gather_rows ...   what the functions of the same name in ops.py do between their keyword arguments and their results
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Device.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <stdexcept>
#include <string>
#include <tuple>
#include <type_traits>
#include <vector>

#include "../../include/sgl_b200.h"

namespace {

using Args = PyObject* const*;

PyObject* g_refused = nullptr;           // _C.SglError
PyObject* g_module = nullptr;            // _C: its WORKSPACE is looked up on every call (a captured batch puts its own there)

struct Refused : std::runtime_error {
  using std::runtime_error::runtime_error;
};
struct Raised {};                        // the Python error is set already

template <class F>
PyObject* guarded(F&& f) {
  HANDLE_TH_ERRORS
  try {
    return f();
  } catch (const Refused& e) {
    PyErr_SetString(g_refused, e.what());
  } catch (const Raised&) {
  }
  return nullptr;
  END_HANDLE_TH_ERRORS
}

PyObject* must(PyObject* o) {
  if (o == nullptr) throw Raised();
  return o;
}

struct Unlocked {
  PyThreadState* s = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(s); }
};

void check(int rc) {
  if (rc != SGL_OK) throw Refused("libsgl_b200 error " + std::to_string(rc) + ": " + sgl_last_error());
}

// ---- arguments -----------------------------------------------------------------------------------------------------------
const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "expected a tensor, got %s", Py_TYPE(o)->tp_name);
    throw Raised();
  }
  return THPVariable_Unpack(o);
}

// as _C.ptr
void* ptr(const at::Tensor& t) {
  if (!t.is_cuda() && !t.is_pinned()) throw Refused("expected a CUDA (or pinned host) tensor: the data path has no CPU implementation");
  if (!t.is_contiguous()) throw Refused("expected a contiguous tensor");
  return t.data_ptr();
}

// as ops._i64
at::Tensor i64(PyObject* o) {
  const at::Tensor& t = tensor(o);
  if (t.scalar_type() != at::kLong) throw Refused(std::string("expected int64 tensor, got torch.") + torch::getTHPDtype(t.scalar_type())->name);
  return t.contiguous();
}

uint64_t integer(PyObject* o) {
  if (PyLong_CheckExact(o)) {
    const uint64_t v = PyLong_AsUnsignedLongLongMask(o);
    if (v == (uint64_t)-1 && PyErr_Occurred()) throw Raised();
    return v;
  }
  PyObject* const n = must(PyNumber_Index(o));
  const uint64_t v = PyLong_AsUnsignedLongLongMask(n);
  Py_DECREF(n);
  if (v == (uint64_t)-1 && PyErr_Occurred()) throw Raised();
  return v;
}

// a size: beyond 64 bits it is refused, where an argument of the C functions is taken modulo 2^64 (as ctypes does)
int64_t size(PyObject* o) {
  PyObject* const n = must(PyNumber_Index(o));
  const long long v = PyLong_AsLongLong(n);
  Py_DECREF(n);
  if (v == -1 && PyErr_Occurred()) throw Raised();
  return v;
}

bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw Raised();
  return v != 0;
}

int64_t sum(int64_t a, int64_t b) {
  if (__builtin_add_overflow(a, b, &a)) throw Refused("a size beyond 64 bits");
  return a;
}

int64_t product(int64_t a, int64_t b) {
  if (__builtin_mul_overflow(a, b, &a)) throw Refused("a size beyond 64 bits");
  return a;
}

template <class T>
T argument(PyObject* o) {
  if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) return nullptr;
    return (T)(THPVariable_Check(o) ? ptr(THPVariable_Unpack(o)) : (void*)(uintptr_t)integer(o));
  } else {
    static_assert(std::is_integral_v<T>, "pointers and integers");
    return (T)integer(o);
  }
}

void count(const char* name, Py_ssize_t n, Py_ssize_t want) {
  if (n == want) return;
  PyErr_Format(PyExc_TypeError, "%s: %zd arguments, got %zd", name, want, n);
  throw Raised();
}

template <class T>
T* optional(PyObject* o) {
  return o == Py_None ? nullptr : (T*)ptr(tensor(o));
}

// ---- the C functions as they are -----------------------------------------------------------------------------------------
template <auto F, class = decltype(F)>
struct Plain;
template <auto F, class R, class... A>
struct Plain<F, R (*)(A...)> {
  template <size_t... I>
  static R call(Args a, std::index_sequence<I...>) {
    std::tuple<A...> v{argument<A>(a[I])...};        // (in order, and before the lock is given up)
    Unlocked u;
    return F(std::get<I>(v)...);
  }
  static PyObject* run(PyObject*, Args a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
      count("libsgl_b200", n, sizeof...(A));
      const R r = call(a, std::index_sequence_for<A...>());
      if constexpr (std::is_same_v<R, int>) {
        check(r);
        Py_RETURN_NONE;
      } else {
        return must(std::is_signed_v<R> ? PyLong_FromLongLong((long long)r) : PyLong_FromUnsignedLongLong((unsigned long long)r));
      }
    });
  }
};

// ---- results -------------------------------------------------------------------------------------------------------------
at::Tensor fresh(int64_t n, at::ScalarType type, const at::Device& dev) { return at::empty({n}, at::TensorOptions().dtype(type).device(dev)); }

PyObject* tuple(std::initializer_list<at::Tensor> ts) {      // (an undefined tensor: None)
  PyObject* const out = must(PyTuple_New((Py_ssize_t)ts.size()));
  Py_ssize_t i = 0;
  for (const at::Tensor& t : ts) {
    PyObject* o = Py_None;
    if (t.defined()) o = THPVariable_Wrap(t);
    else Py_INCREF(o);
    if (o == nullptr) {
      Py_DECREF(out);
      throw Raised();
    }
    PyTuple_SET_ITEM(out, i++, o);
  }
  return out;
}

void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }

// _C.WORKSPACE.get(bytes, device, stream); the tensor keeps the scratch of the call
struct Scratch {
  at::Tensor t;
  void* p;
  size_t n;
  Scratch(size_t bytes, const at::Device& dev, void* on) {
    static PyObject *const s_space = PyUnicode_InternFromString("WORKSPACE"), *const s_get = PyUnicode_InternFromString("get");
    PyObject *space = PyObject_GetAttr(g_module, s_space), *n_ = nullptr, *d = nullptr, *s = nullptr, *got = nullptr;
    if (space && (n_ = PyLong_FromSize_t(bytes)) && (d = THPDevice_New(dev)) && (s = PyLong_FromVoidPtr(on)))
      got = PyObject_CallMethodObjArgs(space, s_get, n_, d, s, nullptr);
    Py_XDECREF(space);
    Py_XDECREF(n_);
    Py_XDECREF(d);
    Py_XDECREF(s);
    must(got);
    if (THPVariable_Check(got)) t = THPVariable_Unpack(got);
    Py_DECREF(got);
    if (!t.defined()) throw Refused("the workspace is not a tensor");
    p = t.data_ptr();
    n = (size_t)t.numel();
  }
};

// bytes of a row, and from one to the next (as ops._row_bytes)
struct Rows {
  int64_t bytes, pitch;
  explicit Rows(const at::Tensor& t) {
    const int64_t size = t.element_size();
    bytes = pitch = size;
    if (t.dim() == 1) return;
    if (t.dim() == 0) throw Refused("rows must be contiguous");
    if (t.stride(-1) != 1 && t.size(-1) > 1) throw Refused("rows must be contiguous");
    for (int64_t d = 1; d < t.dim(); ++d) bytes *= t.size(d);
    pitch = t.stride(0) * size;
  }
};

// `size` values of a tensor of 8-byte words from word `at` on; floats: the tensor as fp32, made on first use
at::Tensor piece(const at::Tensor& words, at::Tensor* floats, int64_t at, int64_t size, bool fp32) {
  if (!fp32) return words.as_strided({size}, {1}, at + words.storage_offset());
  if (!floats->defined()) *floats = words.view(at::kFloat);
  return floats->as_strided({size}, {1}, 2 * (at + words.storage_offset()));
}

// (words, at, size, fp32?)
PyObject* cut(PyObject*, Args a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    count("cut", n, 4);
    at::Tensor floats;
    return must(THPVariable_Wrap(piece(tensor(a[0]), &floats, argument<int64_t>(a[1]), argument<int64_t>(a[2]), integer(a[3]) != 0)));
  });
}

// (words, and at, size, fp32? for every piece)
PyObject* cuts(PyObject*, Args a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n < 1 || (n - 1) % 3 != 0) count("cuts", n, 4);
    const at::Tensor& words = tensor(a[0]);
    at::Tensor floats;
    const Py_ssize_t pieces = (n - 1) / 3;
    PyObject* const out = must(PyTuple_New(pieces));
    try {
      for (Py_ssize_t i = 0; i < pieces; ++i)
        PyTuple_SET_ITEM(out, i, must(THPVariable_Wrap(piece(words, &floats, argument<int64_t>(a[1 + 3 * i]), argument<int64_t>(a[2 + 3 * i]),
                                                             integer(a[3 + 3 * i]) != 0))));
    } catch (...) {
      Py_DECREF(out);
      throw;
    }
    return out;
  });
}

// ---- rows ----------------------------------------------------------------------------------------------------------------
// (table, idx, map, d_n, ts_table, mode, out, status)
PyObject* gather_rows(PyObject*, Args a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    count("gather_rows", n_args, 8);
    const at::Tensor &table = tensor(a[0]), idx = i64(a[1]);
    const int64_t n = idx.numel();
    const Rows row(table);
    int64_t dst_pitch = row.bytes;
    at::Tensor out, out_ts;
    if (a[6] == Py_None) {
      at::DimVector shape(table.sizes());
      shape[0] = n;
      out = at::empty(shape, at::TensorOptions().dtype(table.scalar_type()).device(idx.device()));
    } else {
      out = tensor(a[6]);
      if (n) dst_pitch = Rows(out).pitch;
    }
    const bool times = a[4] != Py_None;
    if (times) out_ts = fresh(n, at::kFloat, idx.device());
    const void* const rows = table.numel() ? ptr(table) : nullptr;
    const int64_t *const ids = (const int64_t*)ptr(idx), *const map = optional<int64_t>(a[2]), *const d_n = optional<int64_t>(a[3]);
    const int64_t map_len = a[2] == Py_None ? 0 : tensor(a[2]).numel();
    const float* const ts = optional<float>(a[4]);
    const int mode = argument<int>(a[5]);
    int32_t* const status = argument<int32_t*>(a[7]);
    void* const on = stream();
    int rc;
    {
      Unlocked u;
      rc = sgl_gather_rows(rows, table.size(0), row.bytes, row.pitch, ids, map, map_len, n, d_n, out.numel() ? out.data_ptr() : nullptr,
                           dst_pitch, ts, times ? (float*)out_ts.data_ptr() : nullptr, mode, status, on);
    }
    check(rc);
    return times ? tuple({out, out_ts}) : must(THPVariable_Wrap(out));
  });
}

// (table, idx, rows, map, d_n, ts_table, ts, split_last_col, status)
PyObject* scatter_rows(PyObject*, Args a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    count("scatter_rows", n_args, 9);
    const at::Tensor &table = tensor(a[0]), idx = i64(a[1]), &from = tensor(a[2]);
    const int64_t n = idx.numel();
    const int split = argument<int>(a[7]) != 0;
    const Rows row(table);
    const int64_t src_pitch = n ? Rows(from).pitch : row.bytes + (split ? 4 : 0);
    void* const rows = table.numel() ? ptr(table) : nullptr;
    const int64_t *const ids = (const int64_t*)ptr(idx), *const map = optional<int64_t>(a[3]), *const d_n = optional<int64_t>(a[4]);
    const int64_t map_len = a[3] == Py_None ? 0 : tensor(a[3]).numel();
    float *const ts_table = optional<float>(a[5]), *const ts = optional<float>(a[6]);
    int32_t* const status = argument<int32_t*>(a[8]);
    void* const on = stream();
    int rc;
    {
      Unlocked u;
      rc = sgl_scatter_rows(rows, table.size(0), row.bytes, row.pitch, ids, map, map_len, n, d_n, from.numel() ? from.data_ptr() : nullptr,
                            src_pitch, ts_table, ts, split, status, on);
    }
    check(rc);
    Py_RETURN_NONE;
  });
}

// (cache_rows, hitmap, backing, ids, status)
PyObject* cache_gather(PyObject*, Args a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    count("cache_gather", n_args, 5);
    const at::Tensor &cache = tensor(a[0]), &hitmap = tensor(a[1]), ids = i64(a[3]);
    const int64_t n = ids.numel();
    if (hitmap.scalar_type() != at::kInt) throw Refused("hitmap must be int32");
    const Rows row(cache);
    bool dense = row.pitch == row.bytes;
    if (dense && a[2] != Py_None) {
      const Rows other(tensor(a[2]));
      dense = other.bytes == row.bytes && other.pitch == row.bytes;
    }
    if (!dense) throw Refused("cache and backing rows must be dense and of equal size");
    const at::Device dev = ids.device();
    at::DimVector shape(cache.sizes());
    shape[0] = n;
    at::Tensor out = at::empty(shape, at::TensorOptions().dtype(cache.scalar_type()).device(dev));
    at::Tensor miss_pos = fresh(n > 1 ? n : 1, at::kLong, dev), miss_ids = fresh(n > 1 ? n : 1, at::kLong, dev), counts = fresh(2, at::kLong, dev);
    const void* const rows = ptr(cache);
    const int32_t* const hits = (const int32_t*)ptr(hitmap);
    const void* const backing = optional<void>(a[2]);
    const int64_t* const want = (const int64_t*)ptr(ids);
    int32_t* const status = argument<int32_t*>(a[4]);
    void* const on = stream();
    const Scratch ws(sgl_cache_gather_ws_bytes(n), dev, on);
    int rc;
    {
      Unlocked u;
      rc = sgl_cache_gather(rows, cache.size(0), hits, hitmap.numel(), backing, row.bytes, want, n, n ? out.data_ptr() : nullptr,
                            (int64_t*)miss_pos.data_ptr(), (int64_t*)miss_ids.data_ptr(), (int64_t*)counts.data_ptr(), status, ws.p, ws.n, on);
    }
    check(rc);
    return tuple({out, miss_pos, miss_ids, counts});
  });
}

// ---- mailbox -------------------------------------------------------------------------------------------------------------
// (ids_a, ids_b, ts, num_nodes, segments, want_pos, status, count address, count sequence number)
PyObject* mail_reduce(PyObject*, Args a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    count("mail_reduce", n_args, 9);
    const at::Tensor ids_a = i64(a[0]), ids_b = a[1] == Py_None ? at::Tensor() : i64(a[1]);
    const at::Device dev = ids_a.device();
    const int64_t n_a = ids_a.numel(), n_b = ids_b.defined() ? ids_b.numel() : 0, n = n_a + n_b, cap = n > 1 ? n : 1;
    const at::Tensor& given = tensor(a[2]);
    if (given.scalar_type() != at::kLong && given.scalar_type() != at::kFloat)
      throw Refused(std::string("mail_reduce: timestamps must be int64 or float32, got torch.") + torch::getTHPDtype(given.scalar_type())->name);
    const at::Tensor ts = given.contiguous();
    PyObject* const seq = must(PySequence_Fast(a[4], "mail_reduce: segments are pairs of tables"));
    std::vector<at::Tensor> keep;
    std::vector<const float*> seg_a, seg_b;
    std::vector<int64_t> dims;
    int64_t width = 0;
    try {
      for (Py_ssize_t s = 0; s < PySequence_Fast_GET_SIZE(seq); ++s) {
        PyObject* const pair = must(PySequence_Fast(PySequence_Fast_GET_ITEM(seq, s), "mail_reduce: segments are pairs of tables"));
        at::Tensor ta, tb;
        try {
          if (PySequence_Fast_GET_SIZE(pair) != 2) throw Refused("mail_reduce: segments are pairs of fp32 [rows, dim] tables of equal width");
          ta = tensor(PySequence_Fast_GET_ITEM(pair, 0)).contiguous();
          tb = PySequence_Fast_GET_ITEM(pair, 1) == Py_None ? ta : tensor(PySequence_Fast_GET_ITEM(pair, 1)).contiguous();
        } catch (...) {
          Py_DECREF(pair);
          throw;
        }
        Py_DECREF(pair);
        if (ta.scalar_type() != at::kFloat || tb.scalar_type() != at::kFloat || ta.dim() != 2 || tb.dim() != 2 || ta.size(1) != tb.size(1))
          throw Refused("mail_reduce: segments are pairs of fp32 [rows, dim] tables of equal width");
        if (ta.size(0) < n_a || (n_b && tb.size(0) < n_b)) throw Refused("mail_reduce: a segment table has fewer rows than its entry list");
        keep.push_back(ta);
        keep.push_back(tb);
        seg_a.push_back((const float*)ta.data_ptr());
        seg_b.push_back((const float*)tb.data_ptr());
        dims.push_back(ta.size(1));
        width += ta.size(1);
      }
    } catch (...) {
      Py_DECREF(seq);
      throw;
    }
    Py_DECREF(seq);
    at::Tensor index = fresh(cap, at::kLong, dev), out_ts = fresh(cap, at::kFloat, dev), d_u = fresh(1, at::kLong, dev), pos, mail;
    if (truth(a[5])) pos = fresh(cap, at::kLong, dev);
    if (!dims.empty()) mail = at::empty({cap, width}, at::TensorOptions().dtype(at::kFloat).device(dev));
    const int64_t *const pa = (const int64_t*)ptr(ids_a), *const pb = n_b ? (const int64_t*)ptr(ids_b) : nullptr;
    const void* const times = ptr(ts);
    const int64_t num_nodes = argument<int64_t>(a[3]), seq_no = argument<int64_t>(a[8]);
    int32_t* const status = argument<int32_t*>(a[6]);
    int64_t* const host = argument<int64_t*>(a[7]);
    void* const on = stream();
    const Scratch ws(sgl_mail_reduce_ws_bytes(n), dev, on);
    int rc;
    {
      Unlocked u;
      rc = sgl_mail_reduce_counted(pa, n_a, pb, n_b, num_nodes, times, ts.numel(), ts.scalar_type() == at::kLong ? 1 : 0, (int)dims.size(),
                                   seg_a.data(), seg_b.data(), dims.data(), (int64_t*)index.data_ptr(), pos.defined() ? (int64_t*)pos.data_ptr() : nullptr,
                                   (float*)out_ts.data_ptr(), mail.defined() ? (float*)mail.data_ptr() : nullptr, (int64_t*)d_u.data_ptr(), status, ws.p,
                                   ws.n, host, seq_no, on);
    }
    check(rc);
    return tuple({index, mail, out_ts, pos, d_u});
  });
}

// (index, mail, mail_ts, mailbox, mailbox_ts, next_mail_pos, d_n, advance, status)
PyObject* mailbox_write(PyObject*, Args a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    count("mailbox_write", n_args, 9);
    const at::Tensor index = i64(a[0]), &mail = tensor(a[1]), &mail_ts = tensor(a[2]), &box = tensor(a[3]), &box_ts = tensor(a[4]);
    if (box.dim() != 3 || !box.is_contiguous() || !box_ts.is_contiguous())
      throw Refused("mailbox_write: mailbox must be a contiguous [nodes, slots, width] tensor");
    if (mail.dim() != 2 || mail.size(1) != box.size(2) || mail.scalar_type() != at::kFloat || mail_ts.scalar_type() != at::kFloat)
      throw Refused("mailbox_write: mail rows must be fp32 of the mailbox's width");
    const at::Tensor next = a[5] == Py_None ? at::Tensor() : i64(a[5]);
    const int64_t n = index.numel() < mail.size(0) ? index.numel() : mail.size(0);
    const at::Tensor rows = mail.contiguous(), times = mail_ts.contiguous();
    const int64_t *const ids = (const int64_t*)ptr(index), *const d_n = optional<int64_t>(a[6]);
    const float *const p_rows = (const float*)ptr(rows), *const p_times = (const float*)ptr(times);
    float *const p_box = (float*)ptr(box), *const p_box_ts = (float*)ptr(box_ts);
    int64_t* const p_next = next.defined() ? (int64_t*)ptr(next) : nullptr;
    const bool advance = truth(a[7]);
    int32_t* const status = argument<int32_t*>(a[8]);
    void* const on = stream();
    int rc;
    {
      Unlocked u;
      rc = sgl_mailbox_write(ids, n, d_n, p_rows, p_times, box.size(2), p_box, p_box_ts, p_next, box.size(0), box.size(1), advance ? 1 : 0, status, on);
    }
    check(rc);
    Py_RETURN_NONE;
  });
}

// ---- sampling, T-CSR -----------------------------------------------------------------------------------------------------
// (indptr, nbr, ts, eid, fence, num_nodes, targets, target_ts, fanout, policy, d_n, equal_root_time, allowed_offset, keep_root_time, seed,
//  rng_stream, want_dt_i64, status, count address, count sequence number)
PyObject* sample_layer(PyObject*, Args a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    count("sample_layer", n_args, 20);
    const at::Tensor targets = i64(a[6]), target_ts = i64(a[7]);
    const int64_t n = targets.numel(), fanout = size(a[8]);
    if (target_ts.numel() != n) throw Refused("sample_layer: targets and target_ts differ in length");
    const at::Tensor& indptr = tensor(a[0]);
    const at::Device dev = indptr.device();
    const int64_t edges = product(n, fanout), cap = edges > 1 ? edges : 1;
    at::Tensor nbr = fresh(cap, at::kLong, dev), dst = fresh(cap, at::kLong, dev), ts = fresh(cap, at::kLong, dev), eid = fresh(cap, at::kLong, dev),
               dt = fresh(cap, at::kFloat, dev), offs = fresh(n + 1, at::kLong, dev), dti;
    if (truth(a[16])) dti = fresh(cap, at::kLong, dev);
    const int64_t *const g_ptr = (const int64_t*)ptr(indptr), *const g_nbr = optional<int64_t>(a[1]), *const g_ts = optional<int64_t>(a[2]),
                  *const g_eid = optional<int64_t>(a[3]), *const g_fence = optional<int64_t>(a[4]);
    const int64_t *const t = (const int64_t*)ptr(targets), *const tt = (const int64_t*)ptr(target_ts), *const d_n = optional<int64_t>(a[10]);
    const int64_t num_nodes = argument<int64_t>(a[5]), offset = argument<int64_t>(a[12]), seq_no = argument<int64_t>(a[19]);
    const int policy = argument<int>(a[9]), equal = argument<int>(a[11]), keep = argument<int>(a[13]);
    const uint64_t seed = argument<uint64_t>(a[14]);
    const uint32_t rng = argument<uint32_t>(a[15]);
    int32_t* const status = argument<int32_t*>(a[17]);
    int64_t* const host = argument<int64_t*>(a[18]);
    void* const on = stream();
    const Scratch ws(sgl_sample_ws_bytes(n), dev, on);
    int rc;
    {
      Unlocked u;
      rc = sgl_sample_layer_counted(g_ptr, g_nbr, g_ts, g_eid, g_fence, num_nodes, t, tt, n, d_n, (int)fanout, policy, equal, offset, keep, seed, rng,
                                    (int64_t*)nbr.data_ptr(), (int64_t*)dst.data_ptr(), (int64_t*)ts.data_ptr(), (float*)dt.data_ptr(),
                                    dti.defined() ? (int64_t*)dti.data_ptr() : nullptr, (int64_t*)eid.data_ptr(), (int64_t*)offs.data_ptr(), status,
                                    ws.p, ws.n, host, seq_no, on);
    }
    check(rc);
    return tuple({nbr, dst, ts, dt, eid, offs, dti});
  });
}

// (key, nbr, ts, eid, num_nodes, want_perm, want_fence) -> ((indptr, nbr, ts, eid, perm, fence), smallest time, largest time)
PyObject* tcsr_build(PyObject*, Args a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    count("tcsr_build", n_args, 7);
    const at::Tensor key = i64(a[0]), nbr = i64(a[1]), ts = i64(a[2]), eid = a[3] == Py_None ? at::Tensor() : i64(a[3]);
    const int64_t m = key.numel(), num_nodes = size(a[4]);
    if (nbr.numel() != m || ts.numel() != m || (eid.defined() && eid.numel() != m)) throw Refused("tcsr_build: edge arrays differ in length");
    const at::Device dev = key.device();
    at::Tensor indptr = fresh(sum(num_nodes, 1), at::kLong, dev), o_nbr = fresh(m, at::kLong, dev), o_ts = fresh(m, at::kLong, dev),
               o_eid = fresh(m, at::kLong, dev), perm, fence;
    if (truth(a[5])) perm = fresh(m, at::kLong, dev);
    if (truth(a[6]) && m && num_nodes) fence = fresh(sgl_tcsr_fence_len(num_nodes, m), at::kLong, dev);
    auto words = [](const at::Tensor& t) { return t.defined() ? (int64_t*)ptr(t) : nullptr; };
    const int64_t *const k = words(key), *const p_nbr = words(nbr), *const p_ts = words(ts), *const p_eid = words(eid);
    int64_t *const p_ptr = words(indptr), *const q_nbr = words(o_nbr), *const q_ts = words(o_ts), *const q_eid = words(o_eid), *const q_perm = words(perm),
            *const q_fence = words(fence);
    void* const on = stream();
    const Scratch ws(sgl_tcsr_build_ws_bytes(num_nodes, m), dev, on);
    int64_t range[2] = {0, 0};
    int rc;
    {
      Unlocked u;
      rc = sgl_tcsr_build_fenced(num_nodes, m, k, p_nbr, p_ts, p_eid, p_ptr, q_nbr, q_ts, q_eid, q_perm, q_fence, range, ws.p, ws.n, on);
    }
    check(rc);
    PyObject *const arrays = tuple({indptr, o_nbr, o_ts, o_eid, perm, fence}), *const out = Py_BuildValue("(NLL)", arrays, (long long)range[0], (long long)range[1]);
    return must(out);
  });
}

// ---- whole batches, queries ----------------------------------------------------------------------------------------------
// an array of a graph: where it is (None: nowhere)
int64_t* at_graph(PyObject* o) { return o == Py_None ? nullptr : (int64_t*)tensor(o).data_ptr(); }

// (indptr, nbr, ts, eid, fence, num_nodes, roots, root_ts, fan-outs, hops, policy, equal_root_time, allowed_offset, seed, id_bits, ts_bits,
//  lowest time, places, words of the results (0: the places are addresses), words of the raw arrays (-1: they lie behind the results),
//  words of meta behind the raw arrays (0: meta is given), meta, bytes of scratch, status, host words, early ones, ready one, side stream)
// -> (results or None, raw arrays)
PyObject* build_batch(PyObject*, Args a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    count("build_batch", n_args, 28);
    const at::Device dev = tensor(a[0]).device();
    const at::Tensor roots = i64(a[6]), root_ts = i64(a[7]);
    const int64_t n = roots.numel();
    if (root_ts.numel() != n) throw Refused("build_batch: roots and root_ts differ in length");
    const int64_t words = argument<int64_t>(a[18]), raw_words = argument<int64_t>(a[19]), meta_words = argument<int64_t>(a[20]);
    at::Tensor results, raw;
    if (raw_words < 0) {
      results = raw = fresh(words + meta_words, at::kLong, dev);
    } else {
      raw = fresh(raw_words + meta_words, at::kLong, dev);
      if (words > 0) results = fresh(words, at::kLong, dev);
    }
    int64_t* const other = (int64_t*)raw.data_ptr();
    int64_t* const meta = meta_words ? other + raw.numel() - meta_words : (int64_t*)tensor(a[21]).data_ptr();
    int64_t* const base = results.defined() ? (int64_t*)results.data_ptr() : nullptr;
    const int64_t *const p_roots = (const int64_t*)ptr(roots), *const p_times = (const int64_t*)ptr(root_ts);
    const int64_t *const g_ptr = at_graph(a[0]), *const g_nbr = at_graph(a[1]), *const g_ts = at_graph(a[2]), *const g_eid = at_graph(a[3]),
                  *const g_fence = at_graph(a[4]);
    const int64_t num_nodes = argument<int64_t>(a[5]), offset = argument<int64_t>(a[12]), lowest = argument<int64_t>(a[16]);
    const int32_t* const fan = argument<const int32_t*>(a[8]);
    const int hops = argument<int>(a[9]), policy = argument<int>(a[10]), equal = argument<int>(a[11]), id_bits = argument<int>(a[14]),
              ts_bits = argument<int>(a[15]);
    const uint64_t seed = argument<uint64_t>(a[13]);
    const int64_t* const places = argument<const int64_t*>(a[17]);
    int32_t* const status = argument<int32_t*>(a[23]);
    int64_t *const host = argument<int64_t*>(a[24]), *const early = argument<int64_t*>(a[25]), *const ready = argument<int64_t*>(a[26]);
    void *const side = argument<void*>(a[27]), *const on = stream();
    const Scratch ws(argument<size_t>(a[22]), dev, on);
    int rc;
    {
      Unlocked u;
      rc = sgl_build_batch_ready(g_ptr, g_nbr, g_ts, g_eid, g_fence, num_nodes, p_roots, p_times, n, fan, hops, policy, equal, offset, seed, id_bits,
                                 ts_bits, lowest, places, base, other, meta, status, host, early, ready, ws.p, ws.n, side, on);
    }
    check(rc);
    return tuple({results, raw});
  });
}

// (indptr, nbr, ts, eid, fence, num_nodes, event sources, times, ids, first event, events at most, t_begin, t_end, node_chunk, chunk mask, chunks,
//  negatives, their times, fan-out, hops, policy, equal_root_time, allowed_offset, keep_root_time, id_bits, ts_bits, ts_base, mapper, mask, epoch,
//  restart, next local id, places, words (0: the places are addresses), words of meta or its address, host words, bytes of scratch, producer,
//  and of the graph's stream its id, device index, device type, address) -> arrays or None
PyObject* query(PyObject*, Args a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    count("query", n_args, 42);
    const at::Device dev = tensor(a[0]).device();
    const c10::cuda::CUDAStreamGuard guard(c10::cuda::CUDAStream::unpack3(argument<int64_t>(a[38]), (c10::DeviceIndex)argument<int64_t>(a[39]),
                                                                          (c10::DeviceType)argument<int64_t>(a[40])));
    const int64_t words = argument<int64_t>(a[33]), meta_words = argument<int64_t>(a[34]);
    at::Tensor buf;
    int64_t *base = nullptr, *meta = (int64_t*)(uintptr_t)meta_words;
    if (words > 0) {
      buf = fresh(words + meta_words, at::kLong, dev);
      base = (int64_t*)buf.data_ptr();
      meta = base + words;
    }
    const int64_t n_neg = tensor(a[16]).numel();
    const int64_t *const neg = n_neg ? at_graph(a[16]) : nullptr, *const neg_ts = n_neg ? at_graph(a[17]) : nullptr;
    const int64_t *const g_ptr = at_graph(a[0]), *const g_nbr = at_graph(a[1]), *const g_ts = at_graph(a[2]), *const g_eid = at_graph(a[3]),
                  *const g_fence = at_graph(a[4]), *const e_src = at_graph(a[6]), *const e_ts = at_graph(a[7]), *const e_id = at_graph(a[8]),
                  *const node_chunk = at_graph(a[13]);
    const uint8_t* const chunk_mask = (const uint8_t*)at_graph(a[14]);
    int64_t *const mapper = at_graph(a[27]), *const mask = at_graph(a[28]), *const next = at_graph(a[31]), *const host = argument<int64_t*>(a[35]);
    const int64_t num_nodes = argument<int64_t>(a[5]), first = argument<int64_t>(a[9]), cap = argument<int64_t>(a[10]), t0 = argument<int64_t>(a[11]),
                  t1 = argument<int64_t>(a[12]), chunks = argument<int64_t>(a[15]), offset = argument<int64_t>(a[22]), ts_base = argument<int64_t>(a[26]),
                  epoch = argument<int64_t>(a[29]);
    const int fanout = argument<int>(a[18]), hops = argument<int>(a[19]), policy = argument<int>(a[20]), equal = argument<int>(a[21]),
              keep = argument<int>(a[23]), id_bits = argument<int>(a[24]), ts_bits = argument<int>(a[25]), restart = argument<int>(a[30]);
    const int64_t* const places = argument<const int64_t*>(a[32]);
    void *const producer = argument<void*>(a[37]), *const on = argument<void*>(a[41]);
    const Scratch ws(argument<size_t>(a[36]), dev, on);
    int rc;
    {
      Unlocked u;
      rc = sgl_query_at(g_ptr, g_nbr, g_ts, g_eid, g_fence, num_nodes, e_src, e_ts, e_id, first, cap, t0, t1, node_chunk, chunk_mask, chunks, neg, neg_ts,
                        n_neg, fanout, hops, policy, equal, offset, keep, id_bits, ts_bits, ts_base, mapper, mask, epoch, restart, next, places, base,
                        meta, host, ws.p, ws.n, producer, on);
    }
    check(rc);
    return tuple({buf});
  });
}

// (device index, q_ts, ts_ptr, roots, neg, neg_ts, n_roots, n_pairs, n_queries, and of every hop its nodes, times and count)
// -> per hop (queries, (nodes, times, indices))
PyObject* query_blocks(PyObject*, Args a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args < 9 || (n_args - 9) % 3 != 0) count("query_blocks", n_args, 12);
    const int hops = (int)((n_args - 9) / 3);
    std::vector<const int64_t*> node(hops), ts(hops);
    std::vector<int64_t> n(hops), d(hops);
    const int64_t queries = argument<int64_t>(a[8]);
    int64_t total = 0;
    for (int l = 0; l < hops; ++l) {
      node[l] = argument<const int64_t*>(a[9 + 3 * l]);
      ts[l] = argument<const int64_t*>(a[10 + 3 * l]);
      n[l] = argument<int64_t>(a[11 + 3 * l]);
      d[l] = l ? n[l - 1] : queries;
      total += 2 * (d[l] + n[l]) + n[l];
    }
    at::Tensor out = fresh(total, at::kLong, at::Device(at::kCUDA, (c10::DeviceIndex)argument<int64_t>(a[0])));
    const int64_t *const q_ts = argument<const int64_t*>(a[1]), *const ts_ptr = argument<const int64_t*>(a[2]),
                  *const roots = argument<const int64_t*>(a[3]), *const neg = argument<const int64_t*>(a[4]), *const neg_ts = argument<const int64_t*>(a[5]);
    const int64_t n_roots = argument<int64_t>(a[6]), n_pairs = argument<int64_t>(a[7]);
    void* const on = stream();
    int rc;
    {
      Unlocked u;
      rc = sgl_query_blocks(hops, node.data(), ts.data(), n.data(), q_ts, ts_ptr, roots, neg, neg_ts, n_roots, n_pairs, queries, (int64_t*)out.data_ptr(), on);
    }
    check(rc);
    PyObject* const blocks = must(PyTuple_New(hops));
    try {
      int64_t at = 0;
      for (int l = 0; l < hops; ++l) {
        const int64_t s = d[l] + n[l];
        PyObject *const arrays = tuple({piece(out, nullptr, at, s, false), piece(out, nullptr, at + s, s, false), piece(out, nullptr, at + 2 * s, n[l], false)});
        PyTuple_SET_ITEM(blocks, l, must(Py_BuildValue("(LN)", (long long)d[l], arrays)));
        at += 2 * s + n[l];
      }
    } catch (...) {
      Py_DECREF(blocks);
      throw;
    }
    return blocks;
  });
}

// (SglError, the module that holds WORKSPACE)
PyObject* bind(PyObject*, Args a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    count("bind", n_args, 2);
    Py_INCREF(a[0]);
    Py_INCREF(a[1]);
    g_refused = a[0];
    g_module = a[1];
    Py_RETURN_NONE;
  });
}

#define SGL_METHOD(name, f) {name, (PyCFunction)(void (*)(void))(f), METH_FASTCALL, nullptr}
#define SGL_PLAIN(f) SGL_METHOD(#f, (&Plain<&f>::run))

PyMethodDef methods[] = {
    SGL_METHOD("bind", bind),
    SGL_METHOD("cut", cut),
    SGL_METHOD("cuts", cuts),
    SGL_METHOD("gather_rows", gather_rows),
    SGL_METHOD("scatter_rows", scatter_rows),
    SGL_METHOD("cache_gather", cache_gather),
    SGL_METHOD("mail_reduce", mail_reduce),
    SGL_METHOD("mailbox_write", mailbox_write),
    SGL_METHOD("sample_layer", sample_layer),
    SGL_METHOD("tcsr_build", tcsr_build),
    SGL_METHOD("build_batch", build_batch),
    SGL_METHOD("query", query),
    SGL_METHOD("query_blocks", query_blocks),
    SGL_PLAIN(sgl_wait_word),
    SGL_PLAIN(sgl_prefetch_batch),
    SGL_PLAIN(sgl_plan_routes_ws_bytes),
    SGL_PLAIN(sgl_plan_routes),
    SGL_PLAIN(sgl_export_arrays),
    SGL_PLAIN(sgl_read_back),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_sgl_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__sgl_host() { return PyModule_Create(&module); }
