// Calls of DeviceComm on PyTorch tensors, in native code: a Python module inside the operators' library.  Small operations are
// bound by what the host spends on a call; the addresses, types and checks of up to 8 tensors, the current stream and 21 arguments
// through ctypes cost 10 us of an allreduce's 16 and most of the 55 us of a row exchange.
//
// Every function returns NotImplemented where an argument is not of the plain form that it knows (then aluminum_b200/device.py makes
// the call itself), and raises the package's AlError otherwise.  The interpreter's lock is released around the library's call.
#pragma once
#if __has_include(<Python.h>)
#include <c10/cuda/CUDACachingAllocator.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <typeinfo>
#include <vector>

#include "al/al_c.h"
#include "al/base.hpp"
#include "al/config.hpp"

namespace {
namespace calls {

constexpr Py_ssize_t kRanks = AL_MAX_DEVICE_RANKS;

PyObject* g_error = nullptr;   // AlError

PyObject* not_mine() { Py_RETURN_NOTIMPLEMENTED; }

/** An error of this package (already set), as opposed to one of PyTorch or C++. */
struct Raised {};

[[noreturn]] void raise(const std::string& what) {
  PyErr_SetString(g_error ? g_error : PyExc_RuntimeError, what.c_str());
  throw Raised();
}

void check(int rc) {
  if (rc) raise(al_last_error());
}

template <typename F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const Raised&) {
  } catch (const std::exception& e) {
    if (!PyErr_Occurred()) PyErr_SetString(g_error ? g_error : PyExc_RuntimeError, e.what());
  } catch (...) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "unknown error");
  }
  return nullptr;
}

/** Items of a list or tuple, or one thing on its own. */
struct Items {
  PyObject* const* at = nullptr;
  PyObject* one = nullptr;
  Py_ssize_t n = 0;
  bool list = false;
  explicit Items(PyObject* o) {
    if (PyList_Check(o) || PyTuple_Check(o)) {
      list = true;
      n = PySequence_Fast_GET_SIZE(o);
      at = PySequence_Fast_ITEMS(o);
    } else {
      one = o;
      n = 1;
    }
  }
  PyObject* operator[](Py_ssize_t i) const { return list ? at[i] : one; }
};

/** One entry per local rank: plain tensors, or None (nullptr).  False: something else. */
struct Tensors {
  const at::Tensor* t[kRanks] = {};
  Py_ssize_t n = 0;
  bool take(PyObject* o, Py_ssize_t ranks) {
    n = ranks;
    if (o == Py_None) return true;
    const Items items(o);
    if (items.list && items.n != ranks)
      raise("expected " + std::to_string(ranks) + " tensors (one per local rank), got " + std::to_string(items.n));
    if (!items.list && ranks != 1) raise("an emulated communicator takes a list with one tensor per rank");
    for (Py_ssize_t i = 0; i < ranks; ++i) {
      if (items[i] == Py_None) continue;
      if (!THPVariable_CheckExact(items[i])) return false;
      t[i] = &THPVariable_Unpack(items[i]);
    }
    return true;
  }
  const at::Tensor* first() const {
    for (Py_ssize_t i = 0; i < n; ++i)
      if (t[i]) return t[i];
    return nullptr;
  }
  void pointers(void** out) const {
    for (Py_ssize_t i = 0; i < n; ++i) {
      if (t[i] && !(t[i]->is_cuda() && t[i]->is_contiguous())) raise("device buffers must be contiguous CUDA tensors");
      out[i] = t[i] ? t[i]->data_ptr() : nullptr;
    }
  }
};

int code_of(const at::Tensor& t) {
  using al_t = Al::DType;
  switch (t.scalar_type()) {
    case at::kChar: return (int)al_t::i8;
    case at::kByte: return (int)al_t::u8;
    case at::kShort: return (int)al_t::i16;
    case at::kUInt16: return (int)al_t::u16;
    case at::kInt: return (int)al_t::i32;
    case at::kUInt32: return (int)al_t::u32;
    case at::kLong: return (int)al_t::i64;
    case at::kUInt64: return (int)al_t::u64;
    case at::kHalf: return (int)al_t::f16;
    case at::kBFloat16: return (int)al_t::bf16;
    case at::kFloat: return (int)al_t::f32;
    case at::kDouble: return (int)al_t::f64;
    default: return -1;
  }
}

long long integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw Raised();
  return v;
}

void* address(PyObject* o) {
  void* p = o == Py_None ? nullptr : PyLong_AsVoidPtr(o);
  if (PyErr_Occurred()) throw Raised();
  return p;
}

/** The communicator; a closed one is an error here and not a null pointer in the library. */
void* handle(PyObject* o) {
  void* p = address(o);
  if (!p) raise("the communicator has been closed");
  return p;
}

/** None: PyTorch's current stream. */
void* stream_of(PyObject* o) { return o == Py_None ? (void*)c10::cuda::getCurrentCUDAStream().stream() : address(o); }

/** Run the library's call without the interpreter's lock; the request of a non-blocking one as an integer, else None. */
template <typename F>
PyObject* launch(bool request, F&& call) {
  void* req = nullptr;
  int rc = 0;
  Py_BEGIN_ALLOW_THREADS;
  rc = call(request ? &req : nullptr);
  Py_END_ALLOW_THREADS;
  check(rc);
  if (request) return PyLong_FromVoidPtr(req);
  Py_RETURN_NONE;
}

void need(Py_ssize_t got, Py_ssize_t want) {
  if (got != want) raise("internal error: wrong number of arguments");
}

/** (comm, local ranks, kind, send, recv, count, wire type or -1, op, root, in place, scale, algo, ctas, stream, request wanted) */
PyObject* collective(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 15);
    const Py_ssize_t ranks = integer(a[1]);
    if (ranks < 1 || ranks > kRanks) return not_mine();
    Tensors send, recv;
    if (!send.take(a[3], ranks) || !recv.take(a[4], ranks)) return not_mine();
    const bool inplace = a[9] == Py_True;
    const at::Tensor *first_out = recv.first(), *first_in = inplace ? first_out : send.first();
    const at::Tensor* ref = first_in ? first_in : first_out;
    if (!ref) return not_mine();
    const int in = code_of(*ref);
    int out = first_out ? code_of(*first_out) : -1;
    if (in < 0 || (first_out && out < 0)) return not_mine();   // (the caller's error message names the type)
    if (out == in) out = -1;
    void *sp[kRanks], *rp[kRanks];
    send.pointers(sp);
    recv.pointers(rp);
    void *comm = handle(a[0]), *stream = stream_of(a[13]);
    const int kind = (int)integer(a[2]), wire = (int)integer(a[6]), op = (int)integer(a[7]), root = (int)integer(a[8]), algo = (int)integer(a[11]),
              ctas = (int)integer(a[12]);
    const size_t count = (size_t)integer(a[5]);
    const double scale = PyFloat_AsDouble(a[10]);
    if (PyErr_Occurred()) throw Raised();
    return launch(a[14] == Py_True, [&](void** req) {
      return al_dev_collective(comm, kind, (int)ranks, (const void* const*)sp, rp, count, in, wire, out, op, root, inplace, 0, nullptr, nullptr,
                               nullptr, nullptr, scale, algo, ctas, stream, req);
    });
  });
}

/** One table of a row exchange: a list of one list per local rank (or, for one rank, its list).  False: rows or entries of another kind. */
bool table(PyObject* o, Py_ssize_t ranks, Py_ssize_t size, std::vector<size_t>& out) {
  auto row = [&](const Items& r) {
    for (Py_ssize_t i = 0; i < r.n; ++i) {
      if (!PyLong_Check(r[i])) return false;
      out.push_back((size_t)integer(r[i]));
    }
    return true;
  };
  out.clear();
  const Items rows(o);
  if (!rows.list) return false;
  if (ranks == 1 && (rows.n == 0 || !(PyList_Check(rows[0]) || PyTuple_Check(rows[0])))) {
    if (!row(rows)) return false;
  } else {
    for (Py_ssize_t r = 0; r < rows.n; ++r) {
      const Items one(rows[r]);
      if (!one.list || !row(one)) return false;
    }
  }
  if ((Py_ssize_t)out.size() != ranks * size)
    raise("exchange_rows: tables need " + std::to_string(ranks) + " row(s) of " + std::to_string(size) + " entries");
  return true;
}

/** (comm, local ranks, ranks, send, recv, row bytes, send stride, recv stride, six tables, send index, recv index, stream, request wanted) */
PyObject* exchange_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 18);
    const Py_ssize_t ranks = integer(a[1]), size = integer(a[2]);
    if (ranks < 1 || ranks > kRanks) return not_mine();
    Tensors send, recv, sidx, ridx;
    if (!send.take(a[3], ranks) || !recv.take(a[4], ranks) || !sidx.take(a[14], ranks) || !ridx.take(a[15], ranks)) return not_mine();
    const void* sp[kRanks];
    void* rp[kRanks];
    const long long *si[kRanks], *ri[kRanks];
    size_t sroom[kRanks], rroom[kRanks];
    auto index = [](const at::Tensor* t) -> const long long* {
      if (t && (t->scalar_type() != at::kLong || !t->is_cuda() || !t->is_contiguous()))
        raise("exchange_rows: index tensors must be contiguous CUDA int64 tensors");
      return t ? (const long long*)t->data_ptr() : nullptr;
    };
    auto room = [](const at::Tensor& t) { return t.storage().nbytes() - (size_t)t.storage_offset() * t.element_size(); };
    for (Py_ssize_t r = 0; r < ranks; ++r) {
      if (!send.t[r] || !recv.t[r]) return not_mine();
      sp[r] = send.t[r]->data_ptr();
      rp[r] = recv.t[r]->data_ptr();
      si[r] = index(sidx.t[r]);
      ri[r] = index(ridx.t[r]);
      sroom[r] = room(*send.t[r]);
      rroom[r] = room(*recv.t[r]);
    }
    std::vector<size_t> t[6];
    for (int i = 0; i < 6; ++i) {
      t[i].reserve((size_t)(ranks * size));
      if (!table(a[8 + i], ranks, size, t[i])) return not_mine();
    }
    void *comm = handle(a[0]), *stream = stream_of(a[16]);
    const size_t bytes = (size_t)integer(a[5]), sstride = (size_t)integer(a[6]), rstride = (size_t)integer(a[7]);
    const bool with_s = a[14] != Py_None, with_r = a[15] != Py_None;
    return launch(a[17] == Py_True, [&](void** req) {
      return al_dev_exchange_rows_sized(comm, (int)ranks, sp, rp, with_s ? sroom : nullptr, with_r ? rroom : nullptr, with_s ? si : nullptr,
                                        with_r ? ri : nullptr, bytes, sstride, rstride, t[0].data(), t[1].data(), t[2].data(), t[3].data(),
                                        t[4].data(), t[5].data(), stream, req);
    });
  });
}

/** (comm, default owner, [(is_send, peer, tensor[, owner])], stream, request wanted) */
PyObject* p2p(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 5);
    const Items items(a[2]);
    if (!items.list) return not_mine();
    const size_t count = (size_t)items.n;
    const int me = (int)integer(a[1]);
    std::vector<int> is_send(count), peer(count), owner(count);
    std::vector<void*> buf(count);
    std::vector<size_t> bytes(count);
    for (size_t i = 0; i < count; ++i) {
      PyObject* it = items[(Py_ssize_t)i];
      if (!PyTuple_Check(it) || PyTuple_GET_SIZE(it) < 3 || !THPVariable_CheckExact(PyTuple_GET_ITEM(it, 2))) return not_mine();
      const at::Tensor& t = THPVariable_Unpack(PyTuple_GET_ITEM(it, 2));
      if (PyFloat_Check(PyTuple_GET_ITEM(it, 1)) || (PyTuple_GET_SIZE(it) > 3 && PyFloat_Check(PyTuple_GET_ITEM(it, 3)))) return not_mine();
      const int sends = PyObject_IsTrue(PyTuple_GET_ITEM(it, 0));
      if (sends < 0) throw Raised();
      is_send[i] = sends;
      peer[i] = (int)integer(PyTuple_GET_ITEM(it, 1));
      owner[i] = PyTuple_GET_SIZE(it) > 3 ? (int)integer(PyTuple_GET_ITEM(it, 3)) : me;
      buf[i] = t.data_ptr();
      bytes[i] = (size_t)t.numel() * t.element_size();
    }
    void *comm = handle(a[0]), *stream = stream_of(a[3]);
    return launch(a[4] == Py_True, [&](void** req) {
      return al_dev_p2p(comm, (int)count, is_send.data(), peer.data(), owner.data(), buf.data(), bytes.data(), stream, req);
    });
  });
}

/** (tensors, shapes): a new tensor of shape i like tensor i for every i; one shape (a tuple of ints) serves all. */
PyObject* empties(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 2);
    const Items like(a[0]), shapes(a[1]);
    if (!like.list) return not_mine();
    const bool shared = PyTuple_Check(a[1]);
    if (!shared && shapes.n != like.n) raise("internal error: as many shapes as tensors expected");
    PyObject* out = PyList_New(like.n);
    if (!out) throw Raised();
    try {
      for (Py_ssize_t i = 0; i < like.n; ++i) {
        if (!THPVariable_CheckExact(like[i])) {
          Py_DECREF(out);
          return not_mine();
        }
        const Items shape(shared ? a[1] : shapes[i]);
        c10::SmallVector<int64_t, 5> dims;
        for (Py_ssize_t k = 0; k < shape.n; ++k) dims.push_back(integer(shape[k]));
        const at::Tensor& t = THPVariable_Unpack(like[i]);
        PyObject* made = THPVariable_Wrap(at::empty(dims, at::TensorOptions().dtype(t.scalar_type()).device(t.device())));
        if (!made) throw Raised();
        PyList_SET_ITEM(out, i, made);
      }
    } catch (...) {
      Py_DECREF(out);
      throw;
    }
    return out;
  });
}

/** Parameters, and the views of a flat buffer that hold their gradients. */
struct Gradients {
  Items params, views;
  Gradients(PyObject* p, PyObject* v) : params(p), views(v) {
    if (!params.list || !views.list || params.n != views.n) raise("internal error: as many views as parameters expected");
    for (Py_ssize_t i = 0; i < params.n; ++i)
      if (!THPVariable_Check(params[i]) || !THPVariable_Check(views[i])) raise("internal error: parameters and views are tensors");
  }
  const at::Tensor& param(Py_ssize_t i) const { return THPVariable_Unpack(params[i]); }
  const at::Tensor& view(Py_ssize_t i) const { return THPVariable_Unpack(views[i]); }
};

/** A set of nodes: open addressing, at most half full.  (Some hundred nodes a step: std::unordered_set took half of the walk's time.) */
struct NodeSet {
  std::vector<torch::autograd::Node*> slots = std::vector<torch::autograd::Node*>(2048);
  size_t used = 0;
  /** False: it was there. */
  bool insert(torch::autograd::Node* node) {
    const size_t mask = slots.size() - 1;
    size_t i = ((uintptr_t)node >> 4) * 0x9E3779B97F4A7C15ull >> 20 & mask;
    for (; slots[i]; i = (i + 1) & mask)
      if (slots[i] == node) return false;
    slots[i] = node;
    if (2 * ++used > slots.size()) {
      NodeSet wider;
      wider.slots.assign(slots.size() * 2, nullptr);
      for (torch::autograd::Node* n : slots)
        if (n) wider.insert(n);
      std::swap(slots, wider.slots);
    }
    return true;
  }
};

/**
 * Will a backward from `root` run the framework's nodes (and native ones) alone?  A hook or a function written in Python may look at
 * gradients while it runs: at a parameter's, or at the flat buffer that holds them.
 */
bool unobserved(torch::autograd::Node* root) {
  using torch::autograd::Node;
  const char* const python = "N5torch8autograd6PyNodeE";   // the class of functions written in Python (its type_info is not exported)
  NodeSet seen;
  seen.insert(root);
  std::vector<Node*> todo{root};
  while (!todo.empty()) {
    Node* const node = todo.back();
    todo.pop_back();
    // (the last two are virtual: a parameter's node has the hooks of the parameter)
    if (!node->pre_hooks().empty() || !node->post_hooks().empty() || !node->retains_grad_hooks().empty() || !node->tensor_pre_hooks().empty() ||
        node->tensor_post_acc_grad_hooks() || std::strcmp(typeid(*node).name(), python) == 0)
      return false;
    for (const torch::autograd::Edge& e : node->next_edges())
      if (e.function && seen.insert(e.function.get())) todo.push_back(e.function.get());
  }
  return true;
}

/**
 * (loss, parameters, views): take the views off the parameters, so that backward leaves its gradients as they are instead of adding
 * each to its view.  False, and nothing is changed, if a parameter's gradient is not its view or if anything that the loss's backward
 * runs could tell.  (ResNet-50: about 20 us.)
 */
PyObject* lend_gradients(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 3);
    const Gradients g(a[1], a[2]);
    if (!THPVariable_Check(a[0]) || !THPVariable_Unpack(a[0]).grad_fn() || !unobserved(THPVariable_Unpack(a[0]).grad_fn().get())) Py_RETURN_FALSE;
    for (Py_ssize_t i = 0; i < g.params.n; ++i)
      if (!g.param(i).grad().is_same(g.view(i))) Py_RETURN_FALSE;
    for (Py_ssize_t i = 0; i < g.params.n; ++i) g.param(i).mutable_grad() = at::Tensor();
    Py_RETURN_TRUE;
  });
}

/** The same elements in the same order in memory (strides of dimensions of one element say nothing). */
bool same_layout(const at::Tensor& a, const at::Tensor& b) {
  if (a.sizes() != b.sizes()) return false;
  for (int64_t d = 0; d < a.dim(); ++d)
    if (a.size(d) > 1 && a.stride(d) != b.stride(d)) return false;
  return true;
}

/** Give the views back; what backward left at each parameter besides (undefined: nothing, or what is in the view already). */
std::vector<at::Tensor> taken_back(const Gradients& g) {
  std::vector<at::Tensor> left((size_t)g.params.n);
  for (Py_ssize_t i = 0; i < g.params.n; ++i) {
    at::Tensor grad = g.param(i).grad();
    const at::Tensor& view = g.view(i);
    g.param(i).mutable_grad() = view;
    if (grad.defined() && !(grad.layout() == at::kStrided && grad.is_alias_of(view) && grad.data_ptr() == view.data_ptr())) left[(size_t)i] = std::move(grad);
  }
  return left;
}

/** (parameters, views): give the views back, with what backward left added to them. */
PyObject* return_gradients(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 2);
    const Gradients g(a[0], a[1]);
    const at::NoGradGuard no_grad;
    const std::vector<at::Tensor> left = taken_back(g);
    for (Py_ssize_t i = 0; i < g.params.n; ++i)
      if (left[(size_t)i].defined()) g.view(i).add_(left[(size_t)i]);
    Py_RETURN_NONE;
  });
}

/**
 * (parameters, views, flat parameters, flat momentum, flat gradients, lr, momentum, weight decay, first step): the optimizer step
 * on the gradients that backward left, and the views back in their places, zeroed.  On an error too the views are back, with the
 * gradients added to them.
 */
PyObject* step_on_lent(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 9);
    const Gradients g(a[0], a[1]);
    for (int i = 2; i < 5; ++i)
      if (!THPVariable_Check(a[i])) raise("internal error: flat buffers are tensors");
    const at::Tensor &param = THPVariable_Unpack(a[2]), &momentum = THPVariable_Unpack(a[3]), &flat = THPVariable_Unpack(a[4]);
    float value[3];
    for (int i = 0; i < 3; ++i) value[i] = (float)PyFloat_AsDouble(a[5 + i]);
    const int first = PyObject_IsTrue(a[8]);
    if (PyErr_Occurred()) throw Raised();
    const at::NoGradGuard no_grad;
    const size_t count = (size_t)g.params.n;
    std::vector<at::Tensor> left = taken_back(g);
    try {
      const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream();
      std::vector<const float*> grad(count, nullptr);
      std::vector<size_t> at(count), numel(count);
      for (size_t i = 0; i < count; ++i) {
        const at::Tensor& view = g.view((Py_ssize_t)i);
        at[i] = (size_t)(view.storage_offset() - flat.storage_offset());
        numel[i] = (size_t)view.numel();
        at::Tensor& l = left[i];
        if (!l.defined()) continue;
        if (l.scalar_type() == at::kFloat && l.layout() == at::kStrided && l.device() == view.device() && same_layout(l, view) &&
            l.is_non_overlapping_and_dense() && !l.is_alias_of(flat) && (uintptr_t)l.data_ptr() % 16 == 0) {
          grad[i] = l.data_ptr<float>();
          // (backward may have made it on another stream: its memory stays until this one is past the optimizer)
          c10::cuda::CUDACachingAllocator::recordStream(l.storage().data_ptr(), stream);
        } else {
          g.view((Py_ssize_t)i).add_(l);
          l.reset();
        }
      }
      return launch(false, [&](void**) {
        return al_sgd_momentum_from(param.data_ptr<float>(), momentum.data_ptr<float>(), flat.data_ptr<float>(), grad.data(), at.data(),
                                    numel.data(), (int)count, value[0], value[1], value[2], 1.f, first, (void*)stream.stream());
      });
    } catch (...) {
      for (size_t i = 0; i < count; ++i)
        if (left[i].defined()) g.view((Py_ssize_t)i).add_(left[i]);
      throw;
    }
  });
}

/** The handle of PyTorch's current stream. */
PyObject* current_stream(PyObject*, PyObject*) {
  return guarded([&] { return PyLong_FromVoidPtr((void*)c10::cuda::getCurrentCUDAStream().stream()); });
}

PyObject* set_error(PyObject*, PyObject* type) {
  Py_INCREF(type);
  Py_XSETREF(g_error, type);
  Py_RETURN_NONE;
}

#define AL_FAST(f) {#f, (PyCFunction)(void (*)(void))f, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {AL_FAST(collective), AL_FAST(exchange_rows), AL_FAST(p2p), AL_FAST(empties), AL_FAST(lend_gradients),
                         AL_FAST(return_gradients), AL_FAST(step_on_lent),
                         {"current_stream", current_stream, METH_NOARGS, nullptr},
                         {"set_error", set_error, METH_O, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
#undef AL_FAST
PyModuleDef module = {PyModuleDef_HEAD_INIT, "al_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace calls
}  // namespace

PyMODINIT_FUNC PyInit_al_torch(void) { return PyModule_Create(&calls::module); }
#endif
