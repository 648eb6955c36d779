// The host path between PyTorch tensors and the C ABI (include/nf4ll.h) as a CPython extension: argument checks, output
// allocation, workspace lookup and the call itself without a trip through Python or ctypes. A decode-sized forward is two
// kernel launches of a few microseconds; issued through ctypes its host side (argument conversion, three stream queries,
// four small Python objects per LoRA branch) took 20 us, longer than the kernels.
//
// No kernel lives here and nothing is decided here: every function checks its tensors, allocates what it returns and makes
// one call into libnf4ll.so. Errors of the library are raised by the Python side (_lib.check).
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/torch.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>

#include <vector>

#include "nf4ll.h"

namespace {

constexpr int64_t kRank = 16;
PyObject* g_check = nullptr;       // _lib.check: raises for a status code
PyObject* g_status = nullptr;      // linear.status_word(device)
PyObject* g_memory_error = nullptr;      // torch.OutOfMemoryError

struct PyRaised {};                // a Python exception is set

// A C++ exception rather than a Python one: the backward runs these checks on autograd's thread, without the interpreter lock
[[noreturn]] void value_error(const char* fmt, ...) {
  char buf[256];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  TORCH_CHECK_VALUE(false, buf);
  __builtin_unreachable();
}

void check(int rc) {
  if (rc == 0) return;
  PyObject* r = PyObject_CallFunction(g_check, "i", rc);
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "nf4ll call failed");
  throw PyRaised();
}

const at::Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) value_error("%s must be a tensor", what);
  return THPVariable_Unpack(o);
}
const at::Tensor* optional(PyObject* o, const char* what) { return o == Py_None ? nullptr : &tensor(o, what); }
double number(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyRaised();
  return v;
}
int64_t integer(PyObject* o) {
  int64_t v;
  if (PyLong_Check(o)) {
    v = PyLong_AsLongLong(o);
  } else {                                 // whatever int() takes
    PyObject* n = PyNumber_Long(o);
    if (!n) throw PyRaised();
    v = PyLong_AsLongLong(n);
    Py_DECREF(n);
  }
  if (v == -1 && PyErr_Occurred()) throw PyRaised();
  return v;
}
const nf4ll_mat* mat(PyObject* o) {
  const void* p = PyLong_AsVoidPtr(o);
  if (!p) value_error("not a weight");
  return static_cast<const nf4ll_mat*>(p);
}
void* ptr(const at::Tensor* t) { return t ? t->data_ptr() : nullptr; }

// `rows`: how many the call reads or writes (it may have more)
void check_act(const at::Tensor& t, int64_t cols, const char* what, int64_t rows = 0) {
  if (t.scalar_type() != at::kHalf || t.dim() != 2 || t.size(1) != cols || t.stride(1) != 1 || !t.is_cuda())
    value_error("%s must be a CUDA fp16 matrix [M, %lld] with unit inner stride", what, static_cast<long long>(cols));
  if (t.size(0) < rows) value_error("%s has %lld rows, the call has %lld", what, static_cast<long long>(t.size(0)), static_cast<long long>(rows));
}
// a packed fp32 side array of at least `n` elements
void check_side(const at::Tensor& t, int64_t n, const char* what) {
  if (t.scalar_type() != at::kFloat || !t.is_contiguous() || !t.is_cuda() || t.numel() < n)
    value_error("%s must be contiguous CUDA fp32 with at least %lld elements", what, static_cast<long long>(n));
}
void check_bias(const at::Tensor* b, int64_t N) {
  if (b && (b->scalar_type() != at::kHalf || !b->is_contiguous() || !b->is_cuda() || b->numel() < N))
    value_error("bias must be contiguous CUDA fp16 with %lld elements", static_cast<long long>(N));
}
int64_t ld(const at::Tensor& t) { return t.size(0) == 1 && t.stride(0) < t.size(1) ? t.size(1) : t.stride(0); }

at::Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Tensor& like) {
  return at::detail::empty_cuda(size, type, like.device(), std::nullopt);
}

// Per-thread scratch of eager calls: one workspace per (device, stream), grown on demand, and the device's status word. Both
// end with the thread.
struct Scratch {
  int device;
  cudaStream_t stream;
  at::Tensor ws;
  int64_t refused = 0;                   // bytes that the allocator did not have
  int again = 0;                         // calls until it is asked for them again
};
struct ThreadState {
  std::vector<Scratch> ws;
  std::vector<at::Tensor> status;        // by device
  int tune[3] = {0, 0, 0};
};
ThreadState& state() {
  thread_local ThreadState s;
  return s;
}

struct Call {
  int device;
  cudaStream_t stream;
  explicit Call(const at::Tensor& t) : device(t.get_device()), stream(c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(t.get_device())).stream()) {}
  int32_t* status() const {
    auto& v = state().status;
    if (static_cast<int>(v.size()) <= device) v.resize(device + 1);
    if (!v[device].defined()) {
      PyObject* r = PyObject_CallFunction(g_status, "i", device);
      if (!r) throw PyRaised();
      v[device] = THPVariable_Unpack(r);
      Py_DECREF(r);
    }
    return v[device].data_ptr<int32_t>();
  }
};

// Scratch of a call: fast() is what it runs best with (it may hold an fp16 copy of the weight), least() what it runs with.
struct Need {
  int64_t M, N, K;
  int32_t r;
  int64_t fast() const {
    const int* t = state().tune;
    return t[0] || t[1] || t[2] ? tuned(t) : nf4ll_workspace_bytes_fast(M, N, K, r);
  }
  int64_t least() const {
    const int* t = state().tune;
    return t[0] || t[1] || t[2] ? tuned(t) : nf4ll_workspace_bytes(M, N, K, r);
  }
  int64_t tuned(const int* t) const { return nf4ll_workspace_bytes_tuned(M, N, K, r, t[0], t[1], t[2]); }
};
constexpr int kAskAgain = 256;           // calls on the smaller route after an allocation has failed: every failure empties the allocator's cache

// Where the allocator does not have the memory for a call's fast route, the call takes the route that needs less.
// A captured call has scratch of its own from the graph's memory pool, which lives as long as the graph: the thread's buffer
// is released when it grows, and eager calls write to it while a replay runs.
struct Workspace {
  void* p;
  int64_t bytes;
  at::Tensor own;
  Workspace(const at::Tensor* given, const Call& c, const at::Tensor& like, std::initializer_list<Need> needs) {
    if (given) {
      if (!given->is_cuda()) value_error("workspace must be a CUDA tensor");
      p = given->data_ptr();
      bytes = given->numel();
      return;
    }
    int64_t fast = 0;
    for (const Need& n : needs) fast = std::max(fast, n.fast());
    auto least = [&] {
      int64_t b = 0;
      for (const Need& n : needs) b = std::max(b, n.least());
      return b;
    };
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) {
      own = allocate(fast, least, like);
      use(own);
      return;
    }
    auto& v = state().ws;
    Scratch* s = nullptr;
    for (auto& e : v)
      if (e.device == c.device && e.stream == c.stream) { s = &e; break; }
    if (!s) {
      v.push_back({c.device, c.stream, at::Tensor()});
      s = &v.back();
    }
    const int64_t have = s->ws.defined() ? s->ws.numel() : -1;      // a call that needs none gets one too
    if (have < fast) {
      const bool ask = s->refused == 0 || fast < s->refused || --s->again < 0;
      const int64_t want = ask ? fast : least();
      if (have < want) {
        s->ws = at::Tensor();
        s->ws = allocate(std::max<int64_t>(want, 1 << 20), least, like);
        if (ask) {
          const bool got = s->ws.numel() >= want;
          s->refused = got ? 0 : want;
          s->again = kAskAgain;
        }
      }
    }
    use(s->ws);
  }

 private:
  void use(const at::Tensor& t) {
    p = t.data_ptr();
    bytes = t.numel();
  }
  template <typename F>
  static at::Tensor allocate(int64_t want, F&& least, const at::Tensor& like) {
    try {
      return empty({std::max<int64_t>(want, 1)}, at::kByte, like);
    } catch (const c10::OutOfMemoryError&) {
      const int64_t b = std::max<int64_t>(least(), 1);
      if (b >= want) throw;
      return empty({b}, at::kByte, like);
    }
  }
};

// (A16, B16, scale[, B16t]) or None, mask or None
struct Lora {
  nf4ll_lora c{};
  bool on = false;
  void set(const at::Tensor& A, const at::Tensor& B, double scale, const at::Tensor* Bt, const at::Tensor* mask, double keep_scale) {
    if (Bt && (Bt->scalar_type() != at::kHalf || !Bt->is_contiguous() || Bt->dim() != 2 || Bt->size(0) != A.size(0) || Bt->size(1) != B.size(0)))
      value_error("transposed lora_B shadow must be contiguous fp16 [16, N]");
    if (A.scalar_type() != at::kHalf || B.scalar_type() != at::kHalf) value_error("LoRA shadows must be fp16");
    if (!A.is_contiguous() || !B.is_contiguous()) value_error("LoRA A/B must be contiguous");
    on = true;
    c.A = A.data_ptr();
    c.B = B.data_ptr();
    c.r = static_cast<int32_t>(A.size(0));
    c.scale = static_cast<float>(scale);
    c.Bt = ptr(Bt);
    c.keep_scale = static_cast<float>(keep_scale);
    set_mask(mask);
  }
  void set_mask(const at::Tensor* mask, bool any_byte = false) {
    if (!mask) return;
    const bool type = mask->scalar_type() == at::kByte || mask->scalar_type() == at::kBool || (any_byte && mask->element_size() == 1);
    if (!type || mask->dim() < 1 || mask->stride(-1) != 1)
      value_error("mask must be uint8/bool with unit inner stride");
    c.mask = static_cast<const uint8_t*>(mask->data_ptr());
    c.ld_mask = mask->dim() > 1 ? (mask->size(0) == 1 && mask->stride(0) < mask->size(1) ? mask->size(1) : mask->stride(0)) : mask->size(0);
  }
  void parse(PyObject* lora, PyObject* mask, double keep_scale, int64_t M, int64_t N, int64_t K) {
    if (lora == Py_None) return;
    PyObject* seq = PySequence_Fast(lora, "a LoRA branch is (A16, B16, scale) or (A16, B16, scale, B16t)");
    if (!seq) throw PyRaised();
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
    PyObject** it = PySequence_Fast_ITEMS(seq);
    struct Drop { PyObject* o; ~Drop() { Py_DECREF(o); } } drop{seq};
    if (n < 3) value_error("a LoRA branch is (A16, B16, scale) or (A16, B16, scale, B16t)");
    const at::Tensor &A = tensor(it[0], "lora_A"), &B = tensor(it[1], "lora_B");
    const at::Tensor *Bt = n > 3 ? optional(it[3], "B16t") : nullptr, *m = optional(mask, "mask");
    set(A, B, number(it[2]), Bt, m, keep_scale);
    fit(A, B, Bt, m, M, N, K);
  }
  // the factors and the mask cover a call of M rows on W[N, K]
  void fit(const at::Tensor& A, const at::Tensor& B, const at::Tensor* Bt, const at::Tensor* mask, int64_t M, int64_t N, int64_t K) const {
    if (!A.is_cuda() || !B.is_cuda() || (Bt && !Bt->is_cuda())) value_error("LoRA factors must be CUDA tensors");
    if (A.numel() < c.r * K || B.numel() < N * c.r || (Bt && Bt->numel() < N * c.r))
      value_error("LoRA factors of %lld and %lld elements do not fit W[%lld, %lld]", static_cast<long long>(A.numel()), static_cast<long long>(B.numel()),
                  static_cast<long long>(N), static_cast<long long>(K));
    fit_mask(mask, M, K);
  }
  static void fit_mask(const at::Tensor* mask, int64_t M, int64_t K) {
    if (!mask || M == 0) return;
    if (!mask->is_cuda() || mask->size(-1) < K || (mask->dim() == 1 ? 1 : mask->size(0)) < M)
      value_error("mask must be a CUDA tensor of at least %lld rows of %lld", static_cast<long long>(M), static_cast<long long>(K));
  }
  const nf4ll_lora* get() const { return on ? &c : nullptr; }
};

PyObject* wrap(const at::Tensor& t) { return THPVariable_Wrap(t); }
PyObject* wrap(const at::Tensor* t) {
  if (t && t->defined()) return THPVariable_Wrap(*t);
  Py_RETURN_NONE;
}
// (a, b): b undefined -> None. `keep` (optional): the caller's own object for a.
PyObject* pair(PyObject* a, PyObject* b) {
  PyObject* r = PyTuple_New(2);
  PyTuple_SET_ITEM(r, 0, a);
  PyTuple_SET_ITEM(r, 1, b);
  return r;
}
PyObject* again(PyObject* o) {
  Py_INCREF(o);
  return o;
}

template <typename F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const PyRaised&) {
    return nullptr;
  } catch (python_error& e) {
    e.restore();
    return nullptr;
  } catch (const c10::ValueError& e) {
    PyErr_SetString(PyExc_ValueError, e.what_without_backtrace());
    return nullptr;
  } catch (const c10::Error& e) {
    const bool memory = dynamic_cast<const c10::OutOfMemoryError*>(&e) != nullptr && g_memory_error;
    PyErr_SetString(memory ? g_memory_error : PyExc_RuntimeError, e.what_without_backtrace());
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

#define ARGS(n)                                                                                        \
  if (nargs != (n)) {                                                                                  \
    PyErr_Format(PyExc_TypeError, "%s takes %d arguments, got %zd", __func__, (n), nargs);             \
    return nullptr;                                                                                    \
  }

// forward(mat, x, bias, lora, mask, keep_scale, out, want_t, workspace) -> (y, t)
PyObject* py_forward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(9);
  return guarded([&]() -> PyObject* {
    const nf4ll_mat* w = mat(a[0]);
    const at::Tensor& x = tensor(a[1], "x");
    check_act(x, w->K, "x");
    const at::Tensor* bias = optional(a[2], "bias");
    if (a[4] != Py_None && a[3] == Py_None) value_error("a dropout mask without a LoRA branch has no meaning");
    const int64_t M = x.size(0);
    check_bias(bias, w->N);
    Lora lora;
    lora.parse(a[3], a[4], number(a[5]), M, w->N, w->K);
    at::Tensor y = a[6] == Py_None ? empty({M, w->N}, at::kHalf, x) : tensor(a[6], "out");
    check_act(y, w->N, "out", M);
    at::Tensor t;
    if (lora.on && PyObject_IsTrue(a[7])) t = empty({M, kRank}, at::kFloat, x);
    const Call c(x);
    const Workspace ws(optional(a[8], "workspace"), c, x, {Need{M, w->N, w->K, lora.on ? kRank : 0}});
    check(nf4ll_forward(w, x.data_ptr(), ld(x), ptr(bias), lora.get(), t.defined() ? t.data_ptr() : nullptr, M, y.data_ptr(), ld(y), ws.p, ws.bytes,
                        c.status(), c.stream));
    return pair(a[6] == Py_None ? wrap(y) : again(a[6]), wrap(&t));
  });
}

// forward_multi(mat, x, segments, bias, out, workspace) -> (y, [t])
PyObject* py_forward_multi(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(6);
  return guarded([&]() -> PyObject* {
    const nf4ll_mat* w = mat(a[0]);
    const at::Tensor& x = tensor(a[1], "x");
    check_act(x, w->K, "x");
    const int64_t M = x.size(0);
    at::Tensor y = a[4] == Py_None ? empty({M, w->N}, at::kHalf, x) : tensor(a[4], "out");
    check_act(y, w->N, "out", M);
    const at::Tensor* bias = optional(a[3], "bias");
    check_bias(bias, w->N);
    PyObject* segs = PySequence_Fast(a[2], "segments must be a sequence");
    if (!segs) throw PyRaised();
    struct Drop { PyObject* o; ~Drop() { Py_XDECREF(o); } } drop{segs};
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(segs);
    std::vector<Lora> loras(n);
    std::vector<nf4ll_segment> arr(n);
    Drop ts{PyList_New(n)};
    std::vector<at::Tensor> hold;
    hold.reserve(n);
    for (Py_ssize_t i = 0; i < n; ++i) {
      Drop seg{PySequence_Fast(PySequence_Fast_GET_ITEM(segs, i), "a segment is (rows, lora, mask, keep_scale[, t])")};
      if (!seg.o) throw PyRaised();
      const Py_ssize_t k = PySequence_Fast_GET_SIZE(seg.o);
      PyObject** it = PySequence_Fast_ITEMS(seg.o);
      if (k < 4) value_error("a segment is (rows, lora, mask, keep_scale[, t])");
      if (it[2] != Py_None && it[1] == Py_None) value_error("a dropout mask without a LoRA branch has no meaning");
      arr[i].rows = integer(it[0]);
      loras[i].parse(it[1], it[2], number(it[3]), M, arr[i].rows, w->K);
      arr[i].lora = loras[i].get();
      arr[i].t_out = nullptr;
      arr[i].t_ready = 0;
      PyObject* out = Py_None;
      if (k > 4 && it[4] != Py_None) {
        const at::Tensor& given = tensor(it[4], "t");
        if (!loras[i].on || given.scalar_type() != at::kFloat || given.dim() != 2 || given.size(0) != M || given.size(1) != kRank || !given.is_contiguous())
          value_error("a ready-made rank-16 product must be contiguous fp32 [M, 16] and needs its LoRA branch");
        arr[i].t_out = given.data_ptr();
        arr[i].t_ready = 1;
        out = again(it[4]);
      } else if (loras[i].on) {
        hold.push_back(empty({M, kRank}, at::kFloat, x));
        arr[i].t_out = hold.back().data_ptr();
        out = wrap(hold.back());
      } else {
        Py_INCREF(Py_None);
      }
      PyList_SET_ITEM(ts.o, i, out);
    }
    const Call c(x);
    const Workspace ws(optional(a[5], "workspace"), c, x, {Need{M, w->N, w->K, kRank}});
    check(nf4ll_forward_multi(w, x.data_ptr(), ld(x), ptr(bias), arr.data(), static_cast<int32_t>(n), M, y.data_ptr(), ld(y), ws.p,
                              ws.bytes, c.status(), c.stream));
    return pair(a[4] == Py_None ? wrap(y) : again(a[4]), again(ts.o));
  });
}

// forward_gate_up(mat, x, lora_gate, mask_gate, lora_up, mask_up, keep_scale, workspace) -> (g, u, h, t_gate, t_up)
PyObject* py_forward_gate_up(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(8);
  return guarded([&]() -> PyObject* {
    const nf4ll_mat* w = mat(a[0]);
    const at::Tensor& x = tensor(a[1], "x");
    check_act(x, w->K, "x");
    const int64_t M = x.size(0), I = w->N / 2;
    const double ks = number(a[6]);
    Lora lg, lu;
    lg.parse(a[2], a[3], ks, M, I, w->K);
    lu.parse(a[4], a[5], ks, M, I, w->K);
    at::Tensor gu = empty({M, 2 * I}, at::kHalf, x), g = gu.narrow(1, 0, I), u = gu.narrow(1, I, I), h = empty({M, I}, at::kHalf, x), tg, tu;
    if (lg.on) tg = empty({M, kRank}, at::kFloat, x);
    if (lu.on) tu = empty({M, kRank}, at::kFloat, x);
    const Call c(x);
    const int32_t rank = (lg.on || lu.on) ? kRank : 0;
    const Workspace ws(optional(a[7], "workspace"), c, x, {Need{M, I, w->K, rank}, Need{M, w->N, w->K, rank}});
    check(nf4ll_forward_gate_up(w, x.data_ptr(), ld(x), lg.get(), lu.get(), tg.defined() ? tg.data_ptr() : nullptr, tu.defined() ? tu.data_ptr() : nullptr,
                                M, g.data_ptr(), 2 * I, u.data_ptr(), 2 * I, h.data_ptr(), I, ws.p, ws.bytes, c.status(), c.stream));
    PyObject* r = PyTuple_New(5);
    PyTuple_SET_ITEM(r, 0, wrap(g));
    PyTuple_SET_ITEM(r, 1, wrap(u));
    PyTuple_SET_ITEM(r, 2, wrap(h));
    PyTuple_SET_ITEM(r, 3, wrap(&tg));
    PyTuple_SET_ITEM(r, 4, wrap(&tu));
    return r;
  });
}

// backward_dx(mat, dy, lora, mask, keep_scale, out, accumulate, want_u, workspace) -> (dx, u)
PyObject* py_backward_dx(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(9);
  return guarded([&]() -> PyObject* {
    const nf4ll_mat* w = mat(a[0]);
    const at::Tensor& dy = tensor(a[1], "dy");
    check_act(dy, w->N, "dy");
    const int64_t M = dy.size(0);
    const int accumulate = PyObject_IsTrue(a[6]);
    if (a[5] == Py_None && accumulate) value_error("accumulate needs an existing dx");
    at::Tensor dx = a[5] == Py_None ? empty({M, w->K}, at::kHalf, dy) : tensor(a[5], "dx");
    check_act(dx, w->K, "dx", M);
    Lora lora;
    lora.parse(a[2], a[3], number(a[4]), M, w->N, w->K);
    at::Tensor u;
    if (lora.on && PyObject_IsTrue(a[7])) u = empty({M, kRank}, at::kFloat, dy);
    const Call c(dy);
    const Workspace ws(optional(a[8], "workspace"), c, dy, {Need{M, w->N, w->K, lora.on ? kRank : 0}});
    check(nf4ll_backward_dx(w, dy.data_ptr(), ld(dy), lora.get(), u.defined() ? u.data_ptr() : nullptr, M, dx.data_ptr(), ld(dx), accumulate, ws.p, ws.bytes,
                            c.status(), c.stream));
    return pair(a[5] == Py_None ? wrap(dx) : again(a[5]), wrap(&u));
  });
}

// lora_grads(dy, x, t, u, scale, mask, keep_scale, dA, dB, accumulate) -> (dA, dB)
PyObject* py_lora_grads(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(10);
  return guarded([&]() -> PyObject* {
    const at::Tensor &dy = tensor(a[0], "dy"), &x = tensor(a[1], "x"), &t = tensor(a[2], "t"), &u = tensor(a[3], "u");
    if (x.dim() != 2 || dy.dim() != 2) value_error("x and dy must be matrices");
    const int64_t M = x.size(0), K = x.size(1), N = dy.size(1);
    check_act(x, K, "x");
    check_act(dy, N, "dy", M);
    check_side(t, M * kRank, "t");
    check_side(u, M * kRank, "u");
    Lora m;
    m.set_mask(optional(a[5], "mask"), true);
    Lora::fit_mask(optional(a[5], "mask"), M, K);
    const bool accumulate = PyObject_IsTrue(a[9]);
    at::Tensor dA = a[7] == Py_None ? empty({kRank, K}, at::kFloat, x) : tensor(a[7], "dA");
    at::Tensor dB = a[8] == Py_None ? empty({N, kRank}, at::kFloat, x) : tensor(a[8], "dB");
    check_side(dA, kRank * K, "dA");
    check_side(dB, kRank * N, "dB");
    const int acc_a = accumulate && a[7] != Py_None, acc_b = accumulate && a[8] != Py_None;
    const Call c(x);
    auto call = [&](void* pa, void* pb, int acc) {
      check(nf4ll_lora_grads(dy.data_ptr(), ld(dy), x.data_ptr(), ld(x), m.c.mask, m.c.ld_mask, static_cast<float>(number(a[6])), t.data_ptr(), u.data_ptr(),
                             static_cast<float>(number(a[4])), kRank, M, N, K, pa, pb, acc, c.stream));
    };
    if (acc_a == acc_b) {
      call(dA.data_ptr(), dB.data_ptr(), acc_a);
    } else {
      call(dA.data_ptr(), nullptr, acc_a);
      call(nullptr, dB.data_ptr(), acc_b);
    }
    return pair(a[7] == Py_None ? wrap(dA) : again(a[7]), a[8] == Py_None ? wrap(dB) : again(a[8]));
  });
}

struct Items {                            // the elements of a tuple or list
  PyObject* o;
  explicit Items(PyObject* seq, const char* what) : o(PySequence_Fast(seq, what)) { if (!o) throw PyRaised(); }
  ~Items() { Py_DECREF(o); }
  Py_ssize_t size() const { return PySequence_Fast_GET_SIZE(o); }
  PyObject* operator[](Py_ssize_t i) const { return PySequence_Fast_GET_ITEM(o, i); }
};

// lora_grads_batch(((dy, x, t, u, scale, mask, keep_scale, dA, dB), ...), accumulate)
PyObject* py_lora_grads_batch(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(2);
  return guarded([&]() -> PyObject* {
    const Items list(a[0], "projections must be a sequence");
    if (list.size() < 1) value_error("one projection at least");
    std::vector<nf4ll_grad> grads;
    int64_t M = 0;
    for (Py_ssize_t i = 0; i < list.size(); ++i) {
      const Items it(list[i], "a projection is (dy, x, t, u, scale, mask, keep_scale, dA, dB)");
      if (it.size() != 9) value_error("a projection is (dy, x, t, u, scale, mask, keep_scale, dA, dB)");
      const at::Tensor &dy = tensor(it[0], "dy"), &x = tensor(it[1], "x"), &t = tensor(it[2], "t"), &u = tensor(it[3], "u");
      if (x.dim() != 2 || dy.dim() != 2) value_error("x and dy must be matrices");
      if (i == 0) M = x.size(0);
      const int64_t K = x.size(1), N = dy.size(1);
      if (x.size(0) != M) value_error("the projections of one call have as many rows each");
      check_act(x, K, "x");
      check_act(dy, N, "dy", M);
      check_side(t, M * kRank, "t");
      check_side(u, M * kRank, "u");
      Lora m;
      m.set_mask(optional(it[5], "mask"), true);
      Lora::fit_mask(optional(it[5], "mask"), M, K);
      const at::Tensor *dA = optional(it[7], "dA"), *dB = optional(it[8], "dB");
      if (dA) check_side(*dA, kRank * K, "dA");
      if (dB) check_side(*dB, kRank * N, "dB");
      grads.push_back({dy.data_ptr(), ld(dy), x.data_ptr(), ld(x), m.c.mask, m.c.ld_mask, static_cast<float>(number(it[6])), t.data_ptr(), u.data_ptr(),
                       static_cast<float>(number(it[4])), N, K, ptr(dA), ptr(dB)});
    }
    const Items first(list[0], "a projection");
    check(nf4ll_lora_grads_batch(grads.data(), static_cast<int32_t>(grads.size()), M, PyObject_IsTrue(a[1]), Call(tensor(first[1], "x")).stream));
    Py_RETURN_NONE;
  });
}

// lora_expand(((u, A16, mask, keep_scale), ...), out)
PyObject* py_lora_expand(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(2);
  return guarded([&]() -> PyObject* {
    const at::Tensor& out = tensor(a[1], "out");
    if (out.dim() != 2) value_error("out must be a matrix");
    const int64_t M = out.size(0), K = out.size(1);
    check_act(out, K, "out");
    const Items list(a[0], "branches must be a sequence");
    std::vector<nf4ll_expand> branches;
    for (Py_ssize_t i = 0; i < list.size(); ++i) {
      const Items it(list[i], "a branch is (u, A16, mask, keep_scale)");
      if (it.size() != 4) value_error("a branch is (u, A16, mask, keep_scale)");
      const at::Tensor &u = tensor(it[0], "u"), &A = tensor(it[1], "lora_A");
      check_side(u, M * kRank, "u");
      if (A.scalar_type() != at::kHalf || !A.is_contiguous() || !A.is_cuda() || A.dim() != 2 || A.size(0) != kRank || A.size(1) != K)
        value_error("lora_A shadow must be contiguous CUDA fp16 [16, %lld]", static_cast<long long>(K));
      Lora m;
      m.set_mask(optional(it[2], "mask"));
      Lora::fit_mask(optional(it[2], "mask"), M, K);
      branches.push_back({u.data_ptr(), A.data_ptr(), m.c.mask, m.c.ld_mask, static_cast<float>(number(it[3]))});
    }
    check(nf4ll_lora_expand(branches.data(), static_cast<int32_t>(branches.size()), M, K, out.data_ptr(), ld(out), Call(out).stream));
    Py_RETURN_NONE;
  });
}

// lora_u(dy, B16t, scale) -> u fp32 [M, 16] = scale * dy . B
PyObject* py_lora_u(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(3);
  return guarded([&]() -> PyObject* {
    const at::Tensor &dy = tensor(a[0], "dy"), &Bt = tensor(a[1], "B16t");
    if (dy.dim() != 2) value_error("dy must be a matrix");
    const int64_t M = dy.size(0), N = dy.size(1);
    check_act(dy, N, "dy");
    if (Bt.scalar_type() != at::kHalf || Bt.dim() != 2 || Bt.size(0) != kRank || Bt.size(1) != N || !Bt.is_contiguous())
      value_error("lora_B transposed shadow must be contiguous fp16 [16, N]");
    at::Tensor u = empty({M, kRank}, at::kFloat, dy);
    check(nf4ll_lora_project(dy.data_ptr(), ld(dy), nullptr, 0, 1.0f, Bt.data_ptr(), static_cast<float>(number(a[2])), M, N, u.data_ptr(), Call(dy).stream));
    return wrap(u);
  });
}

// lora_shadow(A, B, A16, B16, B16t): fp16 copies of the fp32 masters, lora_B also transposed
PyObject* py_lora_shadow(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(5);
  return guarded([&]() -> PyObject* {
    const at::Tensor &A = tensor(a[0], "A"), &B = tensor(a[1], "B"), &A16 = tensor(a[2], "A16"), &B16 = tensor(a[3], "B16"), &Bt = tensor(a[4], "B16t");
    if (A.dim() != 2 || B.dim() != 2 || A.size(0) != kRank || B.size(1) != kRank || Bt.dim() != 2 || Bt.size(0) != kRank || Bt.size(1) != B.size(0) ||
        A16.sizes() != A.sizes() || B16.sizes() != B.sizes())
      value_error("lora_A [16, K], lora_B [N, 16] and their shadows do not fit each other");
    for (const auto* t : {&A, &B, &A16, &B16, &Bt})
      if (!t->is_cuda() || !t->is_contiguous() || t->scalar_type() != (t == &A || t == &B ? at::kFloat : at::kHalf))
        value_error("LoRA masters must be contiguous CUDA fp32 and their shadows contiguous CUDA fp16");
    check(nf4ll_lora_shadow(A.data_ptr<float>(), B.data_ptr<float>(), A.size(1), B.size(0), A16.data_ptr(), B16.data_ptr(), Bt.data_ptr(), Call(A).stream));
    Py_RETURN_NONE;
  });
}

// swiglu_forward(g, u, out) -> h
PyObject* py_swiglu_forward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(3);
  return guarded([&]() -> PyObject* {
    const at::Tensor &g = tensor(a[0], "g"), &u = tensor(a[1], "u");
    if (g.dim() != 2) value_error("g must be a matrix");
    const int64_t M = g.size(0), I = g.size(1);
    check_act(g, I, "g");
    check_act(u, I, "u", M);
    at::Tensor h = a[2] == Py_None ? empty({M, I}, at::kHalf, g) : tensor(a[2], "out");
    check_act(h, I, "h", M);
    check(nf4ll_swiglu_forward(g.data_ptr(), ld(g), u.data_ptr(), ld(u), h.data_ptr(), ld(h), M, I, Call(g).stream));
    return a[2] == Py_None ? wrap(h) : again(a[2]);
  });
}

// swiglu_backward(g, u, dh, dg, du)
PyObject* py_swiglu_backward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(5);
  return guarded([&]() -> PyObject* {
    const at::Tensor &g = tensor(a[0], "g"), &u = tensor(a[1], "u"), &dh = tensor(a[2], "dh"), &dg = tensor(a[3], "dg"), &du = tensor(a[4], "du");
    if (g.dim() != 2) value_error("g must be a matrix");
    const int64_t M = g.size(0), I = g.size(1);
    check_act(g, I, "g");
    check_act(u, I, "u", M);
    check_act(dh, I, "dh", M);
    check_act(dg, I, "dg", M);
    check_act(du, I, "du", M);
    check(nf4ll_swiglu_backward(g.data_ptr(), ld(g), u.data_ptr(), ld(u), dh.data_ptr(), ld(dh), dg.data_ptr(), ld(dg), du.data_ptr(), ld(du), M, I,
                                Call(g).stream));
    Py_RETURN_NONE;
  });
}

// gated_backward(g, u, dh, dg, du, mask, keep_scale, t_gate, t_up, u_down, B16t_gate, B16t_up, scale_gate, scale_up, dB_gate, dB_up, dA_down,
//                accumulate) -> (u_gate, u_up), fp32 [M, 16] each
PyObject* py_gated_backward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(18);
  return guarded([&]() -> PyObject* {
    const at::Tensor &g = tensor(a[0], "g"), &u = tensor(a[1], "u"), &dh = tensor(a[2], "dh"), &dg = tensor(a[3], "dg"), &du = tensor(a[4], "du");
    if (g.dim() != 2) value_error("g must be a matrix");
    const int64_t M = g.size(0), I = g.size(1);
    check_act(g, I, "g");
    check_act(u, I, "u", M);
    check_act(dh, I, "dh", M);
    check_act(dg, I, "dg", M);
    check_act(du, I, "du", M);
    Lora m;
    m.set_mask(optional(a[5], "mask"), true);
    Lora::fit_mask(optional(a[5], "mask"), M, I);
    const at::Tensor &tg = tensor(a[7], "t_gate"), &tu = tensor(a[8], "t_up"), &ud = tensor(a[9], "u_down"), &bg = tensor(a[10], "B16t of gate"),
                     &bu = tensor(a[11], "B16t of up"), &dbg = tensor(a[14], "dB of gate"), &dbu = tensor(a[15], "dB of up"), &dad = tensor(a[16], "dA of down");
    for (const auto* t : {&tg, &tu, &ud}) check_side(*t, M * kRank, "t and u");
    for (const auto* t : {&dbg, &dbu, &dad}) check_side(*t, I * kRank, "dA and dB");
    for (const auto* b : {&bg, &bu})
      if (b->scalar_type() != at::kHalf || b->dim() != 2 || b->size(0) != kRank || b->size(1) != I || !b->is_contiguous() || !b->is_cuda())
        value_error("lora_B transposed shadow must be contiguous CUDA fp16 [16, %lld]", static_cast<long long>(I));
    at::Tensor ug = empty({M, kRank}, at::kFloat, g), uu = empty({M, kRank}, at::kFloat, g);
    // where the allocator does not have what all rows at once take, fewer rows at a time
    at::Tensor scratch;
    for (const int64_t rows : {M, std::min<int64_t>(M, 256), std::min<int64_t>(M, 16)}) {
      try {
        scratch = empty({std::max<int64_t>(nf4ll_gated_backward_bytes(rows, I), 1)}, at::kByte, g);
        break;
      } catch (const c10::OutOfMemoryError&) {
        if (rows <= 16) throw;
      }
    }
    const nf4ll_gated p{g.data_ptr(), ld(g), u.data_ptr(), ld(u), dh.data_ptr(), ld(dh), dg.data_ptr(), ld(dg), du.data_ptr(), ld(du), m.c.mask, m.c.ld_mask,
                        static_cast<float>(number(a[6])), tg.data_ptr(), tu.data_ptr(), ud.data_ptr(), bg.data_ptr(), bu.data_ptr(),
                        static_cast<float>(number(a[12])), static_cast<float>(number(a[13])), ug.data_ptr(), uu.data_ptr(), dbg.data_ptr(), dbu.data_ptr(),
                        dad.data_ptr()};
    check(nf4ll_gated_backward(&p, M, I, PyObject_IsTrue(a[17]), scratch.data_ptr(), scratch.numel(), Call(g).stream));
    return pair(wrap(&ug), wrap(&uu));
  });
}

void check_f32(const at::Tensor& t, at::IntArrayRef shape, const char* what) {
  if (t.scalar_type() != at::kFloat || t.sizes() != shape || !t.is_contiguous() || !t.is_cuda()) value_error("%s must be a contiguous CUDA fp32 tensor of the norm's shape", what);
}

struct NormBranch {
  nf4ll_lora c{};
  bool on = false;
  void parse(PyObject* A, PyObject* mask, double keep_scale, int64_t n, int64_t d) {
    if (A == Py_None) return;
    const at::Tensor& t = tensor(A, "lora_A");
    if (t.scalar_type() != at::kHalf || !t.is_contiguous() || !t.is_cuda() || t.dim() != 2 || t.size(0) != kRank || t.numel() < kRank * d)
      value_error("lora_A shadow must be contiguous CUDA fp16 [16, D]");
    Lora m;
    m.set_mask(optional(mask, "mask"));
    Lora::fit_mask(optional(mask, "mask"), n, d);
    on = true;
    c.A = t.data_ptr();
    c.r = kRank;
    c.scale = 1.0f;
    c.mask = m.c.mask;
    c.ld_mask = m.c.ld_mask;
    c.keep_scale = static_cast<float>(keep_scale);
  }
  const nf4ll_lora* get() const { return on ? &c : nullptr; }
};

// rms_forward(x, w, y, rstd, eps, delta, xout, aq, av, tq, tv, mq, mv, keep_scale)
PyObject* py_rms_forward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(14);
  return guarded([&]() -> PyObject* {
    const at::Tensor &x = tensor(a[0], "x"), &w = tensor(a[1], "w"), &rstd = tensor(a[3], "rstd");
    if (x.dim() != 2) value_error("x must be a matrix");
    const int64_t n = x.size(0), d = x.size(1);
    check_f32(x, {n, d}, "x");
    check_f32(w, {d}, "w");
    check_f32(rstd, {n}, "rstd");
    const at::Tensor *y = optional(a[2], "y"), *delta = optional(a[5], "delta"), *xout = optional(a[6], "xout");
    if (xout) check_f32(*xout, {n, d}, "xout");
    if (delta && (delta->scalar_type() != at::kHalf || delta->sizes() != x.sizes() || !delta->is_contiguous())) value_error("delta must be contiguous fp16 [n, d]");
    if (y && (y->scalar_type() != at::kHalf || y->sizes() != x.sizes() || y->stride(1) != 1)) value_error("y must be fp16 [n, d] with unit inner stride");
    const at::Tensor *tq = optional(a[9], "tq"), *tv = optional(a[10], "tv");
    for (int i = 0; i < 2; ++i) {
      const at::Tensor* t = i ? tv : tq;
      if ((a[7 + i] == Py_None) != (t == nullptr)) value_error("the %s branch needs both its lora_A shadow and its [n, 16] output", i ? "v" : "q");
      if (t) check_f32(*t, {n, kRank}, i ? "tv" : "tq");
      if (a[11 + i] != Py_None && a[7 + i] == Py_None) value_error("a dropout mask without its LoRA branch has no meaning");
    }
    NormBranch q, v;
    const double ks = number(a[13]);
    q.parse(a[7], a[11], ks, n, d);
    v.parse(a[8], a[12], ks, n, d);
    check(nf4ll_rms_forward(x.data_ptr<float>(), ptr(delta), static_cast<float*>(ptr(xout)), w.data_ptr<float>(), static_cast<float>(number(a[4])), n, d,
                            ptr(y), y ? ld(*y) : 0, rstd.data_ptr<float>(), q.get(), ptr(tq), v.get(), ptr(tv), Call(x).stream));
    Py_RETURN_NONE;
  });
}

// rms_backward(dy16, gscale, x, w, rstd, out, dres, uq, uv, aq, av, mq, mv, keep_scale, out16, delta)
PyObject* py_rms_backward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(16);
  return guarded([&]() -> PyObject* {
    const at::Tensor &dy = tensor(a[0], "dy16"), &x = tensor(a[2], "x"), &w = tensor(a[3], "w"), &rstd = tensor(a[4], "rstd"), &out = tensor(a[5], "out");
    if (x.dim() != 2) value_error("x must be a matrix");
    const int64_t n = x.size(0), d = x.size(1);
    check_f32(x, {n, d}, "x");
    check_f32(w, {d}, "w");
    check_f32(rstd, {n}, "rstd");
    check_f32(out, {n, d}, "out");
    const at::Tensor *dres = optional(a[6], "dres"), *out16 = optional(a[14], "out16"), *delta = optional(a[15], "delta");
    if (dres) check_f32(*dres, {n, d}, "dres");
    if (dy.scalar_type() != at::kHalf || dy.sizes() != x.sizes() || dy.stride(1) != 1) value_error("dy16 must be fp16 [n, d] with unit inner stride");
    if (out16 && (out16->scalar_type() != at::kHalf || out16->sizes() != x.sizes() || !out16->is_contiguous())) value_error("out16 must be contiguous fp16 [n, d]");
    const at::Tensor *uq = optional(a[7], "uq"), *uv = optional(a[8], "uv");
    for (int i = 0; i < 2; ++i) {
      const at::Tensor* u = i ? uv : uq;
      if ((a[9 + i] == Py_None) != (u == nullptr)) value_error("the %s branch needs both its lora_A shadow and its [n, 16] factor", i ? "v" : "q");
      if (u) check_f32(*u, {n, kRank}, i ? "uv" : "uq");
    }
    NormBranch q, v;
    const double ks = number(a[13]);
    q.parse(a[9], a[11], ks, n, d);
    v.parse(a[10], a[12], ks, n, d);
    check(nf4ll_rms_backward(dy.data_ptr(), ld(dy), static_cast<float>(number(a[1])), x.data_ptr<float>(), ptr(delta), w.data_ptr<float>(),
                             rstd.data_ptr<float>(), dres ? dres->data_ptr<float>() : nullptr, out.data_ptr<float>(), ptr(out16), n, d, q.get(), ptr(uq),
                             v.get(), ptr(uv), Call(x).stream));
    Py_RETURN_NONE;
  });
}

// dequant(packed, qabs, scale2, offset2, code2, n_qblocks, out)
PyObject* py_dequant(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(7);
  return guarded([&]() -> PyObject* {
    const at::Tensor* t[6];
    for (int i = 0; i < 6; ++i) {
      t[i] = &tensor(a[i < 5 ? i : 6], "dequant operand");
    }
    const int64_t n = integer(a[5]);
    const at::Tensor& out = *t[5];
    if (out.scalar_type() != at::kHalf || out.numel() < n * 64) value_error("dequant output must be fp16 with room for every block");
    for (auto* x : t)
      if (!x->is_cuda()) value_error("dequant operands must live on the GPU");
    const int64_t groups = (n + 255) / 256, bytes[5] = {n * 32, n, groups * 4, groups * 4, 256 * 4};
    for (int i = 0; i < 5; ++i)
      if (static_cast<int64_t>(t[i]->nbytes()) < bytes[i]) value_error("dequant operand %d has %lld bytes, the blocks need %lld", i, static_cast<long long>(t[i]->nbytes()), static_cast<long long>(bytes[i]));
    check(nf4ll_dequant(static_cast<const uint8_t*>(t[0]->data_ptr()), static_cast<const uint8_t*>(t[1]->data_ptr()), static_cast<const float*>(t[2]->data_ptr()),
                        static_cast<const float*>(t[3]->data_ptr()), static_cast<const float*>(t[4]->data_ptr()), n, out.data_ptr(), Call(out).stream));
    Py_RETURN_NONE;
  });
}

std::vector<int32_t> lengths(PyObject* o) {
  PyObject* seq = PySequence_Fast(o, "sequence lengths must be a sequence");
  if (!seq) throw PyRaised();
  struct Drop { PyObject* o; ~Drop() { Py_DECREF(o); } } drop{seq};
  std::vector<int32_t> v(PySequence_Fast_GET_SIZE(seq));
  for (size_t i = 0; i < v.size(); ++i) v[i] = static_cast<int32_t>(integer(PySequence_Fast_GET_ITEM(seq, i)));
  return v;
}

// attention_forward(qkv, seq_lens, heads, kv_heads, head_dim, trig) -> (a, roped, lse)
PyObject* py_attention_forward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(6);
  return guarded([&]() -> PyObject* {
    const at::Tensor &qkv = tensor(a[0], "qkv"), &trig = tensor(a[5], "trig");
    const auto lens = lengths(a[1]);
    const int64_t nh = integer(a[2]), nkv = integer(a[3]), hd = integer(a[4]);
    check_act(qkv, (nh + 2 * nkv) * hd, "qkv");
    const int64_t M = qkv.size(0);
    check_f32(trig, {trig.size(0), hd}, "trig");
    for (const int32_t n : lens)
      if (n > trig.size(0)) value_error("the rotary table is shorter than a sequence");
    at::Tensor out = empty({M, nh * hd}, at::kHalf, qkv), roped = empty({M, (nh + nkv) * hd}, at::kHalf, qkv), lse = empty({nh, M}, at::kFloat, qkv);
    check(nf4ll_attention_forward(qkv.data_ptr(), ld(qkv), lens.data(), static_cast<int32_t>(lens.size()), M, nh, nkv, hd, trig.data_ptr(), roped.data_ptr(),
                                  (nh + nkv) * hd, out.data_ptr(), nh * hd, lse.data_ptr<float>(), Call(qkv).stream));
    PyObject* r = PyTuple_New(3);
    PyTuple_SET_ITEM(r, 0, wrap(out));
    PyTuple_SET_ITEM(r, 1, wrap(roped));
    PyTuple_SET_ITEM(r, 2, wrap(lse));
    return r;
  });
}

// attention_backward(qkv, seq_lens, heads, kv_heads, head_dim, trig, roped, a, lse, da) -> dqkv
PyObject* py_attention_backward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(10);
  return guarded([&]() -> PyObject* {
    const at::Tensor &qkv = tensor(a[0], "qkv"), &trig = tensor(a[5], "trig"), &roped = tensor(a[6], "roped"), &out = tensor(a[7], "a"), &lse = tensor(a[8], "lse"),
                     &da = tensor(a[9], "da");
    const auto lens = lengths(a[1]);
    const int64_t nh = integer(a[2]), nkv = integer(a[3]), hd = integer(a[4]), M = qkv.size(0);
    check_act(qkv, (nh + 2 * nkv) * hd, "qkv");
    check_act(roped, (nh + nkv) * hd, "roped", M);
    check_act(out, nh * hd, "a", M);
    check_side(lse, nh * M, "lse");
    check_f32(trig, {trig.size(0), hd}, "trig");
    for (const int32_t n : lens)
      if (n > trig.size(0)) value_error("the rotary table is shorter than a sequence");
    check_act(da, nh * hd, "da");
    if (da.size(0) != M) value_error("da has %lld rows, the forward had %lld", static_cast<long long>(da.size(0)), static_cast<long long>(M));
    at::Tensor dqkv = empty({M, (nh + 2 * nkv) * hd}, at::kHalf, qkv), delta = empty({nh, M}, at::kFloat, qkv);
    check(nf4ll_attention_backward(qkv.data_ptr(), ld(qkv), lens.data(), static_cast<int32_t>(lens.size()), M, nh, nkv, hd, trig.data_ptr(), roped.data_ptr(),
                                   ld(roped), out.data_ptr(), ld(out), lse.data_ptr<float>(), da.data_ptr(), ld(da), delta.data_ptr<float>(), dqkv.data_ptr(),
                                   (nh + 2 * nkv) * hd, Call(qkv).stream));
    return wrap(dqkv);
  });
}

// -------------------------------------------------------------------------------------------------------
// nf4_lora_linear as a C++ autograd node
// -------------------------------------------------------------------------------------------------------
struct WeightRef : torch::CustomClassHolder {      // the Python weight object, for as long as the graph lives
  PyObject* o;
  const nf4ll_mat* m;
  WeightRef(PyObject* w, const nf4ll_mat* mm) : o(w), m(mm) { Py_INCREF(o); }
  ~WeightRef() override {
    if (!Py_IsInitialized()) return;
    PyGILState_STATE s = PyGILState_Ensure();
    Py_DECREF(o);
    PyGILState_Release(s);
  }
};

// f() under the interpreter lock, from a thread that may not hold it; a Python exception travels on as a C++ one
template <typename F>
auto locked(F&& f) {
  struct Gil {
    PyGILState_STATE s = PyGILState_Ensure();
    ~Gil() { PyGILState_Release(s); }
  } gil;
  try {
    return f();
  } catch (const PyRaised&) {
    python_error e;
    e.persist();
    throw e;
  }
}

void check_nogil(int rc) {
  if (rc != 0) locked([&] { check(rc); });
}

int32_t* status_nogil(const Call& c) {
  auto& v = state().status;
  if (static_cast<int>(v.size()) <= c.device || !v[c.device].defined()) return locked([&] { return c.status(); });
  return v[c.device].data_ptr<int32_t>();
}

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct Nf4Linear : torch::autograd::Function<Nf4Linear> {
  // the factors are optional and not undefined tensors, which the autograd machinery does not take for inputs
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& x, const std::optional<at::Tensor>& A, const std::optional<at::Tensor>& B,
                            const c10::intrusive_ptr<WeightRef>& w,
                            const std::optional<at::Tensor>& bias, double scale, const std::optional<at::Tensor>& mask, double keep_scale) {
    const nf4ll_mat* m = w->m;
    at::Tensor x2 = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
    check_act(x2, m->K, "x");
    const int64_t M = x2.size(0);
    at::Tensor m2 = mask ? (mask->dim() == 2 ? *mask : mask->reshape({-1, mask->size(-1)})) : at::Tensor();
    at::Tensor A16, B16, Bt16, t;
    Lora lora;
    const Call c(x2);
    if (A) {
      at::Tensor Ac = A->contiguous(), Bc = B->contiguous();
      if (Ac.scalar_type() == at::kFloat && Bc.scalar_type() == at::kFloat && Ac.dim() == 2 && Bc.dim() == 2 && Ac.size(0) == kRank && Bc.size(1) == kRank &&
          Ac.is_cuda() && Bc.is_cuda() && reinterpret_cast<uintptr_t>(Bc.data_ptr()) % 16 == 0) {
        A16 = empty(Ac.sizes(), at::kHalf, x2);
        B16 = empty(Bc.sizes(), at::kHalf, x2);
        Bt16 = empty({kRank, Bc.size(0)}, at::kHalf, x2);
        check(nf4ll_lora_shadow(Ac.data_ptr<float>(), Bc.data_ptr<float>(), Ac.size(1), Bc.size(0), A16.data_ptr(), B16.data_ptr(), Bt16.data_ptr(), c.stream));
      } else {
        A16 = Ac.to(at::kHalf);
        B16 = Bc.to(at::kHalf);
      }
      lora.set(A16, B16, scale, Bt16.defined() ? &Bt16 : nullptr, m2.defined() ? &m2 : nullptr, keep_scale);
      lora.fit(A16, B16, Bt16.defined() ? &Bt16 : nullptr, m2.defined() ? &m2 : nullptr, M, m->N, m->K);
      t = empty({M, kRank}, at::kFloat, x2);
    } else if (m2.defined()) {
      value_error("a dropout mask without a LoRA branch has no meaning");
    }
    if (bias) check_bias(&*bias, m->N);
    at::Tensor y = empty({M, m->N}, at::kHalf, x2);
    const Workspace ws(nullptr, c, x2, {Need{M, m->N, m->K, lora.on ? kRank : 0}});
    check(nf4ll_forward(m, x2.data_ptr(), ld(x2), bias ? bias->data_ptr() : nullptr, lora.get(), t.defined() ? t.data_ptr() : nullptr, M, y.data_ptr(), m->N,
                        ws.p, ws.bytes, c.status(), c.stream));
    ctx->saved_data["w"] = c10::IValue::make_capsule(w);
    ctx->saved_data["s"] = c10::IValue(c10::List<double>({scale, keep_scale}));
    ctx->saved_data["lead"] = x.sizes().vec();
    // no activations of the graph (saved-tensor hooks do not see them), and the mask may be the caller's reused buffer
    if (lora.on) ctx->saved_data["lora"] = c10::IValue(std::vector<at::Tensor>{A16, B16, Bt16, m2});
    ctx->save_for_backward({x2, t});
    if (x.dim() == 2) return y;
    auto shape = x.sizes().vec();
    shape.back() = m->N;
    return y.view(shape);
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &x2 = saved[0], &t = saved[1];
    at::Tensor A16, B16, Bt16, m2;
    if (const auto it = ctx->saved_data.find("lora"); it != ctx->saved_data.end()) {
      const auto f = it->second.toTensorVector();
      A16 = f[0]; B16 = f[1]; Bt16 = f[2]; m2 = f[3];
    }
    const auto w = c10::static_intrusive_pointer_cast<WeightRef>(ctx->saved_data["w"].toCapsule());
    const auto s = ctx->saved_data["s"].toDoubleVector();
    const nf4ll_mat* m = w->m;
    at::Tensor dy = grads[0];
    if (!dy.defined()) return variable_list(8);
    at::Tensor dy2 = dy.dim() == 2 ? dy : dy.reshape({-1, dy.size(-1)});
    if (dy2.stride(1) != 1) dy2 = dy2.contiguous();
    TORCH_CHECK_VALUE(dy2.scalar_type() == at::kHalf && dy2.size(1) == m->N && dy2.is_cuda(), "dy must be a CUDA fp16 matrix [M, N]");
    const int64_t M = dy2.size(0);
    check_act(x2, m->K, "saved x", M);
    const Call c(dy2);
    at::Tensor dx = empty({M, m->K}, at::kHalf, dy2), u, dA, dB;
    Lora lora;
    if (A16.defined()) {
      lora.set(A16, B16, s[0], Bt16.defined() ? &Bt16 : nullptr, m2.defined() ? &m2 : nullptr, s[1]);
      u = empty({M, kRank}, at::kFloat, dy2);
    }
    const Workspace ws(nullptr, c, dy2, {Need{M, m->N, m->K, lora.on ? kRank : 0}});
    check_nogil(nf4ll_backward_dx(m, dy2.data_ptr(), ld(dy2), lora.get(), u.defined() ? u.data_ptr() : nullptr, M, dx.data_ptr(), m->K, 0, ws.p, ws.bytes,
                                  status_nogil(c), c.stream));
    if (lora.on) {
      // one buffer: the library then clears both gradients with one fill
      at::Tensor flat = empty({kRank * (m->K + m->N)}, at::kFloat, dy2);
      dA = flat.narrow(0, 0, kRank * m->K).view({kRank, m->K});
      dB = flat.narrow(0, kRank * m->K, kRank * m->N).view({m->N, kRank});
      check_nogil(nf4ll_lora_grads(dy2.data_ptr(), ld(dy2), x2.data_ptr(), ld(x2), lora.c.mask, lora.c.ld_mask, static_cast<float>(s[1]), t.data_ptr(),
                                   u.data_ptr(), static_cast<float>(s[0]), kRank, M, m->N, m->K, dA.data_ptr(), dB.data_ptr(), 0, c.stream));
    }
    const auto lead = ctx->saved_data["lead"].toIntVector();
    return {lead.size() == 2 ? dx : dx.view(lead), dA, dB, at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor()};
  }
};

// linear(x, A, B, weight, mat, bias, scale, mask, keep_scale) -> y
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(9);
  return guarded([&]() -> PyObject* {
    const at::Tensor& x = tensor(a[0], "x");
    const at::Tensor *A = optional(a[1], "A"), *B = optional(a[2], "B"), *bias = optional(a[5], "bias"), *mask = optional(a[7], "mask");
    if (x.dim() < 1) value_error("x must have a last dimension");
    auto w = c10::make_intrusive<WeightRef>(a[3], mat(a[4]));
    if (!A != !B) value_error("a LoRA branch needs both of its factors");
    auto given = [](const at::Tensor* t) { return t ? std::optional<at::Tensor>(*t) : std::nullopt; };
    return wrap(Nf4Linear::apply(x, given(A), given(B), w, given(bias), number(a[6]), given(mask), number(a[8])));
  });
}

// set_tune(bm_tiles, bn, splits): what workspaces of this thread's calls are sized for
PyObject* py_set_tune(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(3);
  return guarded([&]() -> PyObject* {
    for (int i = 0; i < 3; ++i) state().tune[i] = static_cast<int>(integer(a[i]));
    Py_RETURN_NONE;
  });
}

// setup(check, status_word, out_of_memory_error)
PyObject* py_setup(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(3);
  g_check = again(a[0]);
  g_status = again(a[1]);
  g_memory_error = again(a[2]);
  Py_RETURN_NONE;
}

#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {METHOD(forward), METHOD(forward_multi), METHOD(forward_gate_up), METHOD(backward_dx), METHOD(lora_grads), METHOD(lora_u), METHOD(lora_shadow),
                         METHOD(lora_grads_batch), METHOD(lora_expand), METHOD(gated_backward),
                         METHOD(swiglu_forward), METHOD(swiglu_backward), METHOD(rms_forward), METHOD(rms_backward), METHOD(dequant),
                         METHOD(attention_forward), METHOD(attention_backward), METHOD(linear), METHOD(set_tune), METHOD(setup), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "host path between PyTorch tensors and libnf4ll.so", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
