// Host side of the hottest calls as a CPython extension: checks of the operands, allocation of the results and the launch.
//
// A small call (a roll-out step of a mesh network, a block on a few thousand points) is bound by its host side: in Python one launch
// took 15 to 50 us (attributes of every tensor, torch.empty, the foreign-function call with up to 40 arguments).  The
// functions do what the Python code did, argument by argument; gradients, dispatch and weight copies stay in Python.  Together with calls
// that skip the autograd function where no gradient is wanted: a message-passing step of 1 885 nodes (three launches) 150 -> 78 us, a Transolver
// block of 4 096 points (eleven) 373 -> 231 us, an AFNO block (twelve) 305 -> 223 us, a U-Net block with attention 601 -> 427 us.
// Where the Python around a launch took longer than the launch, it is native as well: the way from the modules of a message-passing MLP to
// its kernel (mlp3_module), that MLP's backward of eight to fourteen launches (mlp3_bwd), the slice-token calls: the step of 1 885
// nodes 77 -> 52 us, a network of fifteen steps 1 328 -> 1 005 us, a training step of 30 011 nodes 807 -> 660 us, the Transolver block 206 us.
// As there, the interpreter's lock is released not only for the launch but also where memory is allocated or copied (an allocation may wait
// for the device): every function reads its arguments, works in an `Unlocked` scope and wraps its results.
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <cmath>
#include <vector>

#include "pnm_api.h"

namespace {

using at::Tensor;

const Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) throw torch::TypeError(std::string("expected a tensor, got ") + Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
// undefined for None
const Tensor kNone;
const Tensor& optional(PyObject* o) { return o == Py_None ? kNone : tensor(o); }
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
float* fptr(const Tensor& t) { return static_cast<float*>(ptr(t)); }
long long integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v != 0;
}
// what the Python code asserted
struct Refused : torch::PyTorchError {
  using PyTorchError::PyTorchError;
  PyObject* python_type() override { return PyExc_AssertionError; }
};
void require(bool ok, const char* what) {
  if (!ok) throw Refused(what);
}
void need_args(Py_ssize_t got, Py_ssize_t want) {
  if (got != want) throw torch::TypeError("expected " + std::to_string(want) + " arguments, got " + std::to_string(got));
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
// without the interpreter's lock while it lives; an exception that leaves the scope has the lock again
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  Unlocked() = default;
  Unlocked(const Unlocked&) = delete;
  ~Unlocked() { PyEval_RestoreThread(state); }
};
void check(const char* name, int code) {
  if (code != 0) throw std::runtime_error(std::string(name) + " failed with code " + std::to_string(code));
}
uintptr_t address(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()); }
// 2-D view whose last dim is contiguous, whose row stride is a multiple of 8 and that starts on a 16-byte boundary
// (the argument itself or a copy, which `own` holds: a second count on a Python object's tensor goes through the interpreter)
const Tensor& rowmajor2d(const Tensor& in, Tensor& own) {
  require(in.dim() == 2, "expected a matrix");
  const Tensor* t = &in;
  if (t->stride(1) != 1 || t->stride(0) % 8 != 0) t = &(own = in.contiguous());
  if (address(*t) % 16 != 0) t = &(own = t->clone());
  return *t;
}
Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
  return at::empty(sizes, at::TensorOptions().dtype(type).device(like.device()));
}
// fp32 zeros; a memset costs a call 2 us less than the kernel behind at::zeros, and the device 0.5 us
Tensor zeros32(at::IntArrayRef sizes, const Tensor& like) {
  Tensor t = empty(sizes, at::kFloat, like);
  if (t.numel()) check("pnm_zero", pnm_zero(t.data_ptr(), t.numel() * 4, stream()));
  return t;
}
// values of a parameter vector: fp32, contiguous, 16-byte aligned
const Tensor& vector32(const Tensor& in, Tensor& own) {
  if (!in.defined()) return in;
  const Tensor* t = &in;
  if (t->scalar_type() != at::kFloat || !t->is_contiguous()) t = &(own = in.detach().to(at::kFloat).contiguous());
  if (address(*t) % 16 != 0) t = &(own = t->detach().clone());
  return *t;
}
PyObject* tuple_of(std::initializer_list<const Tensor*> tensors) {
  THPObjectPtr result(PyTuple_New(Py_ssize_t(tensors.size())));
  if (!result) throw python_error();
  Py_ssize_t i = 0;
  for (const Tensor* t : tensors) {
    PyObject* o = THPVariable_Wrap(*t);
    if (!o) throw python_error();
    PyTuple_SET_ITEM(result.get(), i++, o);
  }
  return result.release();
}

// gemm_tn(a, b, bias, scale, act, aux, aux_mode, a2, a3, z_out, out, group_out, scale_post, bn, max_ctas) -> out or (out, z)
PyObject* gemm_tn(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 15);
  const Tensor &a0 = tensor(args[0]), &b0 = tensor(args[1]), &bias = optional(args[2]), &scale = optional(args[3]), &aux0 = optional(args[5]),
               &a20 = optional(args[7]), &a30 = optional(args[8]), &given = optional(args[10]), &group_out = optional(args[11]);
  const int act = int(integer(args[4])), aux_mode = int(integer(args[6])), post = truth(args[12]), bn = int(integer(args[13])),
            cap = int(integer(args[14]));
  const bool want_z = truth(args[9]);
  Tensor own[5], made, z;
  const Tensor& out = given.defined() ? given : made;
  {
    const Unlocked unlocked;
    const Tensor &a = rowmajor2d(a0, own[0]), &b = rowmajor2d(b0, own[1]);
    const Tensor &a2 = a20.defined() ? rowmajor2d(a20, own[2]) : kNone, &a3 = a2.defined() && a30.defined() ? rowmajor2d(a30, own[3]) : kNone;
    const int64_t M = a.size(0), K1 = a.size(1), N = b.size(0), K = b.size(1);
    int64_t K2 = K;
    if (a2.defined()) {
      K2 = K1 + a2.size(1);
      if (a3.defined()) {
        require(a3.size(0) == M && K2 + a3.size(1) == K, "the column blocks of A do not match B");
      } else {
        require(a2.size(0) == M && K2 == K, "the column blocks of A do not match B");
      }
    } else {
      require(K1 == K, "A and B have different numbers of columns");
    }
    require(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16, "operands must be bf16");
    if (!given.defined()) made = empty({M, N}, at::kBFloat16, a);
    if (want_z) z = empty({M, N}, at::kBFloat16, a);
    const Tensor& aux = aux0.defined() ? rowmajor2d(aux0, own[4]) : kNone;
    if (aux.defined()) {
      require(aux.size(0) == M && aux.size(1) == N && aux.scalar_type() == at::kBFloat16, "the auxiliary operand must be bf16 [M, N]");
    }
    for (const Tensor* v : {&bias, &scale})
      if (v->defined()) require(v->scalar_type() == at::kFloat && v->numel() == N && v->is_contiguous(), "vectors must be contiguous fp32 [N]");
    auto ld = [](const Tensor& t) { return t.defined() ? int(t.stride(0)) : 0; };
    check("pnm_gemm_tn",
          pnm_gemm_tn(ptr(a), ld(a), ptr(a2), ld(a2), ptr(a3), ld(a3), ptr(b), ld(b), ptr(out), ld(out), ptr(z), ld(z), ptr(aux), ld(aux), int(M),
                      int(N), int(K), int(K1), int(K2), fptr(bias), fptr(scale), fptr(group_out), act, aux_mode, post, bn, cap, stream()));
  }
  return z.defined() ? tuple_of({&out, &z}) : THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// gemm_nt(a, b, colsum, out, colsum_out, max_ctas) -> out or (out, colsum)
PyObject* gemm_nt(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 6);
  const Tensor &a0 = tensor(args[0]), &b0 = tensor(args[1]), &given = optional(args[3]), &given_sums = optional(args[4]);
  const bool want_sums = truth(args[2]);
  const int cap = int(integer(args[5]));
  Tensor own[2], made, made_sums;
  const Tensor &out = given.defined() ? given : made, &sums = given_sums.defined() ? given_sums : made_sums;
  {
    const Unlocked unlocked;
    const Tensor &a = rowmajor2d(a0, own[0]), &b = rowmajor2d(b0, own[1]);
    const int64_t M = a.size(0), Na = a.size(1), Nb = b.size(1);
    require(b.size(0) == M, "operands have different numbers of rows");
    // two buffers: a weight's gradient and its bias' are held, saved and changed one without the other
    if (!given.defined()) made = zeros32({Na, Nb}, a);
    if (!given_sums.defined() && want_sums) made_sums = zeros32({Na}, a);
    check("pnm_gemm_nt", pnm_gemm_nt(ptr(a), int(a.stride(0)), ptr(b), int(b.stride(0)), fptr(out), int(out.stride(0)), fptr(sums), int(M), int(Na),
                                     int(Nb), cap, stream()));
  }
  return sums.defined() ? tuple_of({&out, &sums}) : THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// layernorm_fwd(x [M, C], gamma, beta or None, eps, post or None) -> (y, mean, rstd)
PyObject* layernorm_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 5);
  const Tensor &x = tensor(args[0]), &gamma = tensor(args[1]), &beta = optional(args[2]), &post = optional(args[4]);
  const float eps = float(real(args[3]));
  Tensor y, mean, rstd;
  {
    const Unlocked unlocked;
    require(x.dim() == 2, "expected a matrix");
    const int64_t M = x.size(0), C = x.size(1);
    y = at::empty_like(x); mean = empty({M}, at::kFloat, x); rstd = empty({M}, at::kFloat, x);
    check("pnm_layernorm_fwd", pnm_layernorm_fwd(ptr(x), nullptr, fptr(gamma), fptr(beta), ptr(y), nullptr, fptr(mean), fptr(rstd), ptr(post), M, int(C),
                                                 eps, stream()));
  }
  return tuple_of({&y, &mean, &rstd});
  END_HANDLE_TH_ERRORS
}

// contiguous and 16-byte aligned: the argument or a copy
const Tensor& dense(const Tensor& in, Tensor& own) {
  const Tensor* t = &in;
  if (!t->is_contiguous()) t = &(own = in.contiguous());
  if (address(*t) % 16 != 0) t = &(own = t->clone());
  return *t;
}

constexpr int64_t kWidth = 128, kRows = 128;     // of the one-kernel MLP

// A bf16 table of 128 columns whose rows start on 32-byte boundaries (the kernel moves whole sectors).
bool row_table(PyObject* o) {
  if (Py_TYPE(o) != reinterpret_cast<PyTypeObject*>(THPVariableClass)) return false;     // subclasses dispatch for themselves
  const Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.dim() == 2 && t.size(1) == kWidth && t.size(0) > 0 && t.stride(1) == 1 &&
         t.stride(0) >= kWidth && t.stride(0) % 16 == 0 && address(t) % 32 == 0;
}

// mlp3_operands_ok(tables, weights, biases, gamma, beta): the tables, three 128-wide layers and a LayerNorm fit the one-kernel MLP
PyObject* mlp3_operands_ok(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 5);
  THPObjectPtr tables(PySequence_Fast(args[0], "tables")), weights(PySequence_Fast(args[1], "weights")), biases(PySequence_Fast(args[2], "biases"));
  if (!tables || !weights || !biases) throw python_error();
  const Py_ssize_t nsrc = PySequence_Fast_GET_SIZE(tables.get());
  if (nsrc < 1 || nsrc > 3 || PySequence_Fast_GET_SIZE(weights.get()) != 3 || args[3] == Py_None) Py_RETURN_FALSE;
  for (Py_ssize_t j = 0; j < nsrc; ++j)
    if (!row_table(PySequence_Fast_GET_ITEM(tables.get(), j))) Py_RETURN_FALSE;
  const at::Device dev = THPVariable_Unpack(PySequence_Fast_GET_ITEM(tables.get(), 0)).device();
  auto parameter = [&](PyObject* o) { return THPVariable_CheckExact(o) && THPVariable_Unpack(o).device() == dev; };
  for (int i = 0; i < 3; ++i) {
    PyObject* o = PySequence_Fast_GET_ITEM(weights.get(), i);
    if (!parameter(o)) Py_RETURN_FALSE;
    const Tensor& w = THPVariable_Unpack(o);
    if (w.dim() != 2 || w.size(0) != kWidth || w.size(1) != (i ? kWidth : kWidth * int64_t(nsrc))) Py_RETURN_FALSE;
  }
  auto vector = [&](PyObject* o) { return parameter(o) && THPVariable_Unpack(o).numel() == kWidth; };
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(biases.get()); ++i) {
    PyObject* o = PySequence_Fast_GET_ITEM(biases.get(), i);
    if (o != Py_None && !vector(o)) Py_RETURN_FALSE;
  }
  if (!vector(args[3]) || (args[4] != Py_None && !vector(args[4]))) Py_RETURN_FALSE;
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// mlp3_fwd(tables, row indices (or None each), bf16 weights, (b1, b2, b3, gamma, beta), eps, act, post or None, rows, keep)
//   -> y, or (y, h1, h2, x3, mean, rstd[, z1, z2]) where the backward's needs are kept (z1, z2 not with ReLU)
PyObject* mlp3_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 9);
  THPObjectPtr tables(PySequence_Fast(args[0], "tables")), index(PySequence_Fast(args[1], "indices")), weights(PySequence_Fast(args[2], "weights")),
      vectors(PySequence_Fast(args[3], "vectors"));
  if (!tables || !index || !weights || !vectors) throw python_error();
  const Py_ssize_t nsrc = PySequence_Fast_GET_SIZE(tables.get());
  if (nsrc < 1 || nsrc > 3 || PySequence_Fast_GET_SIZE(index.get()) != nsrc || PySequence_Fast_GET_SIZE(weights.get()) != 3 ||
      PySequence_Fast_GET_SIZE(vectors.get()) != 5)
    throw torch::TypeError("one to three tables, as many indices, three weights, five vectors");
  const void* src[3];
  long long rows[3];
  int ld[3];
  const int* idx[3];
  for (Py_ssize_t j = 0; j < nsrc; ++j) {
    const Tensor& t = tensor(PySequence_Fast_GET_ITEM(tables.get(), j));
    PyObject* i = PySequence_Fast_GET_ITEM(index.get(), j);
    src[j] = t.data_ptr(); rows[j] = t.size(0); ld[j] = int(t.stride(0));
    idx[j] = i == Py_None ? nullptr : static_cast<const int*>(tensor(i).data_ptr());
  }
  const Tensor& table = tensor(PySequence_Fast_GET_ITEM(tables.get(), 0));
  const void* w[3];
  for (int i = 0; i < 3; ++i) w[i] = tensor(PySequence_Fast_GET_ITEM(weights.get(), i)).data_ptr();
  const Tensor* vec[5];
  for (int i = 0; i < 5; ++i) vec[i] = &optional(PySequence_Fast_GET_ITEM(vectors.get(), i));
  const float eps = float(real(args[4]));
  const int act = int(integer(args[5]));
  const Tensor& post = optional(args[6]);
  const int64_t m = integer(args[7]);
  const bool keep = truth(args[8]), relu = act == 3;
  Tensor own[5], y, h1, h2, x3, mean, rstd, z1, z2;
  {
    const Unlocked unlocked;
    for (int i = 0; i < 5; ++i) vec[i] = &vector32(*vec[i], own[i]);
    y = empty({m, kWidth}, at::kBFloat16, table);
    if (keep) {
      const Tensor h = empty({3, m, kWidth}, at::kBFloat16, table), s = empty({2, m}, at::kFloat, table);
      h1 = h.select(0, 0); h2 = h.select(0, 1); x3 = h.select(0, 2);
      mean = s.select(0, 0); rstd = s.select(0, 1);
      if (!relu) {
        const Tensor z = empty({2, (m + kRows - 1) / kRows, kRows * kWidth}, at::kBFloat16, table);     // whole tiles
        z1 = z.select(0, 0); z2 = z.select(0, 1);
      }
    }
    check("pnm_mlp3_ln_fwd",
          pnm_mlp3_ln_fwd(int(nsrc), src, rows, ld, idx, w[0], w[1], w[2], fptr(*vec[0]), fptr(*vec[1]), fptr(*vec[2]), fptr(*vec[3]), fptr(*vec[4]), eps,
                          act, ptr(post), post.defined() ? post.stride(0) : 0, ptr(y), kWidth, ptr(z1), ptr(z2), ptr(h1), ptr(h2), ptr(x3), fptr(mean),
                          fptr(rstd), m, stream()));
  }
  if (!keep) return THPVariable_Wrap(y);
  return relu ? tuple_of({&y, &h1, &h2, &x3, &mean, &rstd}) : tuple_of({&y, &h1, &h2, &x3, &mean, &rstd, &z1, &z2});
  END_HANDLE_TH_ERRORS
}

// Interned names of attributes.
PyObject* name_of(const char* text) {
  PyObject* o = PyUnicode_InternFromString(text);
  if (!o) throw python_error();
  return o;
}
// own attribute, or null (no error set) where there is none
PyObject* attribute(PyObject* o, PyObject* name) {
  PyObject* r = PyObject_GetAttr(o, name);
  if (!r) {
    if (!PyErr_ExceptionMatches(PyExc_AttributeError)) throw python_error();
    PyErr_Clear();
  }
  return r;
}
PyObject* item(PyObject* dict, PyObject* key) {  // borrowed, or null where there is none
  PyObject* r = PyDict_GetItemWithError(dict, key);
  if (!r && PyErr_Occurred()) throw python_error();
  return r;
}
bool same(PyObject* tuple, at::IntArrayRef v) {
  if (!PyTuple_Check(tuple) || PyTuple_GET_SIZE(tuple) != Py_ssize_t(v.size())) return false;
  for (size_t i = 0; i < v.size(); ++i)
    if (integer(PyTuple_GET_ITEM(tuple, i)) != v[i]) return false;
  return true;
}
// The bf16 copy that the weight cache holds of this parameter on this stream (a new reference), as the cache's own look-up finds it
// (ops/gemm.py): an entry is ((version, address, shape, strides), copy, weak reference).  Null where there is none that is valid.
PyObject* kept_copy(PyObject* w, PyObject* cache, PyObject* stream_handle, bool on_default) {
  const Tensor& t = THPVariable_Unpack(w);
  if (t.scalar_type() == at::kBFloat16) {
    if (!t.is_contiguous() || address(t) % 16 != 0) return nullptr;
    Py_INCREF(w);
    return w;
  }
  if (t.is_view() || t.is_inference()) return nullptr;
  THPObjectPtr id(PyLong_FromVoidPtr(w));
  THPObjectPtr key(on_default ? PyTuple_Pack(2, id.get(), Py_False) : PyTuple_Pack(3, id.get(), Py_False, stream_handle));
  if (!key) throw python_error();
  PyObject* hit = item(cache, key.get());
  if (!hit || !PyTuple_Check(hit) || PyTuple_GET_SIZE(hit) != 3) return nullptr;
  PyObject *ver = PyTuple_GET_ITEM(hit, 0), *copy = PyTuple_GET_ITEM(hit, 1);
  THPObjectPtr owner(PyObject_CallNoArgs(PyTuple_GET_ITEM(hit, 2)));
  if (!owner) throw python_error();
  if (owner.get() != w || !PyTuple_Check(ver) || PyTuple_GET_SIZE(ver) != 4 || integer(PyTuple_GET_ITEM(ver, 0)) != int64_t(t._version()) ||
      PyLong_AsUnsignedLongLong(PyTuple_GET_ITEM(ver, 1)) != address(t) || !same(PyTuple_GET_ITEM(ver, 2), t.sizes()) ||
      !same(PyTuple_GET_ITEM(ver, 3), t.strides()) || !THPVariable_Check(copy))
    return nullptr;
  Py_INCREF(copy);
  return copy;
}

// mlp3_module(modules of a Sequential, tables, segment indices (or None each), post or None, weight cache, parameters of captured graphs,
//   stream, (Linear, SiLU, ReLU, GELU, LayerNorm)) -> y, or None where the call has to go the general way.
// The forward of Linear, act, Linear, act, Linear, LayerNorm without gradients: the walk over the modules, the checks of `supported`, the
// look-up of the weights' bf16 copies and the launch.  Anything it does not know (other module types, a weight without a copy that is
// up to date, a capture) is left to the Python code, which decides as before.
PyObject* mlp3_module(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 8);
  static PyObject *const k_parameters = name_of("_parameters"), *const k_weight = name_of("weight"), *const k_bias = name_of("bias"),
                  *const k_eps = name_of("eps"), *const k_approximate = name_of("approximate"), *const k_index = name_of("index32"),
                  *const k_items = name_of("num_items"), *const k_segments = name_of("num_segments");
  PyObject *modules = args[0], *cache = args[4], *kinds = args[7];
  THPObjectPtr tables(PySequence_Fast(args[1], "tables")), segs(PySequence_Fast(args[2], "segment indices"));
  if (!tables || !segs) throw python_error();
  const Py_ssize_t nsrc = PySequence_Fast_GET_SIZE(tables.get());
  if (!PyDict_Check(modules) || PyDict_GET_SIZE(modules) != 6 || !PyDict_Check(cache) || !PyDict_Check(args[5]) || PyDict_GET_SIZE(args[5]) != 0 ||
      !PyTuple_Check(kinds) || PyTuple_GET_SIZE(kinds) != 5 || nsrc < 1 || nsrc > 3 || PySequence_Fast_GET_SIZE(segs.get()) != nsrc)
    Py_RETURN_NONE;
  const long long handle = integer(args[6]);
  if (handle != 0 && c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) Py_RETURN_NONE;

  for (Py_ssize_t j = 0; j < nsrc; ++j)
    if (!row_table(PySequence_Fast_GET_ITEM(tables.get(), j))) Py_RETURN_NONE;
  const Tensor& table = THPVariable_Unpack(PySequence_Fast_GET_ITEM(tables.get(), 0));
  const at::Device dev = table.device();
  auto parameter = [&](PyObject* o) { return o && THPVariable_CheckExact(o) && THPVariable_Unpack(o).device() == dev; };
  // ---- the modules: weights (as kept bf16 copies), vectors (b1, b2, b3, gamma, beta), activation
  THPObjectPtr copies[3], vectors[5];            // owned: another thread may change the modules while this one launches
  int act = 0;
  double eps = 0;
  Py_ssize_t at = 0;
  PyObject *unused, *module;
  for (int i = 0; PyDict_Next(modules, &at, &unused, &module); ++i) {
    PyTypeObject* type = Py_TYPE(module);
    auto is = [&](int k) { return reinterpret_cast<PyObject*>(type) == PyTuple_GET_ITEM(kinds, k); };
    if (i == 1 || i == 3) {
      int code = is(1) ? 2 : is(2) ? 3 : 0;
      if (is(3)) {
        THPObjectPtr form(attribute(module, k_approximate));
        if (form && PyUnicode_Check(form.get()) && PyUnicode_CompareWithASCIIString(form.get(), "none") == 0) code = 1;
      }
      if (!code || (act && act != code)) Py_RETURN_NONE;
      act = code;
      continue;
    }
    if (i == 5 ? !PyType_Check(PyTuple_GET_ITEM(kinds, 4)) || !PyObject_TypeCheck(module, reinterpret_cast<PyTypeObject*>(PyTuple_GET_ITEM(kinds, 4))) : !is(0))
      Py_RETURN_NONE;
    THPObjectPtr own(attribute(module, k_parameters));
    if (!own || !PyDict_Check(own.get())) Py_RETURN_NONE;
    PyObject *w = item(own.get(), k_weight), *b = item(own.get(), k_bias);
    if (!parameter(w) || !b || (b != Py_None && (!parameter(b) || THPVariable_Unpack(b).numel() != kWidth))) Py_RETURN_NONE;
    const Tensor& t = THPVariable_Unpack(w);
    if (i == 5) {
      if (t.numel() != kWidth) Py_RETURN_NONE;
      THPObjectPtr e(attribute(module, k_eps));
      if (!e) Py_RETURN_NONE;
      eps = real(e.get());
      vectors[3] = Py_NewRef(w); vectors[4] = Py_NewRef(b);
    } else {
      if (t.dim() != 2 || t.size(0) != kWidth || t.size(1) != (i ? kWidth : kWidth * int64_t(nsrc))) Py_RETURN_NONE;
      copies[i / 2] = kept_copy(w, cache, args[6], handle == 0);
      if (!copies[i / 2]) Py_RETURN_NONE;
      vectors[i / 2] = Py_NewRef(b);
    }
  }
  // ---- rows
  const void* src[3];
  long long rows[3];
  int ld[3];
  const int* idx[3];
  THPObjectPtr index[3];
  int64_t m = -1;
  Py_ssize_t post_at = -1;
  for (Py_ssize_t j = 0; j < nsrc; ++j) {
    PyObject *o = PySequence_Fast_GET_ITEM(tables.get(), j), *seg = PySequence_Fast_GET_ITEM(segs.get(), j);
    const Tensor& t = THPVariable_Unpack(o);
    int64_t count = t.size(0);
    src[j] = t.data_ptr(); rows[j] = count; ld[j] = int(t.stride(0)); idx[j] = nullptr;
    if (t.device() != dev) Py_RETURN_NONE;
    if (seg != Py_None) {
      THPObjectPtr items(attribute(seg, k_items)), parts(attribute(seg, k_segments));
      index[j] = attribute(seg, k_index);
      if (!items || !parts || !index[j] || integer(parts.get()) != count) Py_RETURN_NONE;
      count = integer(items.get());
      idx[j] = static_cast<const int*>(tensor(index[j].get()).data_ptr());
    } else if (o == args[3] && post_at < 0) {
      post_at = j;
    }
    if (count == 0 || (m >= 0 && m != count)) Py_RETURN_NONE;
    m = count;
  }
  if (args[3] != Py_None && post_at < 0) Py_RETURN_NONE;
  const Tensor& post = args[3] == Py_None ? kNone : THPVariable_Unpack(args[3]);
  const void* w[3];
  for (int i = 0; i < 3; ++i) w[i] = tensor(copies[i].get()).data_ptr();
  const Tensor* vec[5];
  for (int i = 0; i < 5; ++i) vec[i] = &optional(vectors[i].get());
  Tensor own[5], y;
  {
    const Unlocked unlocked;
    for (int i = 0; i < 5; ++i) vec[i] = &vector32(*vec[i], own[i]);
    y = empty({m, kWidth}, at::kBFloat16, table);
    check("pnm_mlp3_ln_fwd",
          pnm_mlp3_ln_fwd(int(nsrc), src, rows, ld, idx, w[0], w[1], w[2], fptr(*vec[0]), fptr(*vec[1]), fptr(*vec[2]), fptr(*vec[3]), fptr(*vec[4]),
                          float(eps), act, ptr(post), post.defined() ? post.stride(0) : 0, ptr(y), kWidth, nullptr, nullptr, nullptr, nullptr, nullptr,
                          nullptr, nullptr, m, stream()));
  }
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

// mlp3_bwd(dy, tables, segment indices (or None each), groups of indexed tables that are one tensor, gradients wanted (per table), post, act,
//   (w1t [128 n, 128], w2t, w3t), gamma, (h1, h2, x3, mean, rstd, z1, z2))
//   -> ([gradient of a table or None], dw1, dw2, dw3, db1, db2, db3, dgamma, dbeta, launches)
// The launches of the backward in their order; see ops/mlp_fused.py for what they compute.
PyObject* mlp3_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 10);
  THPObjectPtr tables(PySequence_Fast(args[1], "tables")), segs(PySequence_Fast(args[2], "segment indices")), groups(PySequence_Fast(args[3], "groups")),
      wanted(PySequence_Fast(args[4], "flags")), weights(PySequence_Fast(args[7], "weights")), kept(PySequence_Fast(args[9], "kept"));
  if (!tables || !segs || !groups || !wanted || !weights || !kept) throw python_error();
  const Py_ssize_t nsrc = PySequence_Fast_GET_SIZE(tables.get());
  if (nsrc < 1 || nsrc > 3 || PySequence_Fast_GET_SIZE(segs.get()) != nsrc || PySequence_Fast_GET_SIZE(wanted.get()) < nsrc ||
      PySequence_Fast_GET_SIZE(weights.get()) != 3 || PySequence_Fast_GET_SIZE(kept.get()) != 7)
    throw torch::TypeError("one to three tables, as many indices and flags, three weights, seven kept tensors");
  const Tensor& dy0 = tensor(args[0]);
  const Py_ssize_t post = args[5] == Py_None ? -1 : Py_ssize_t(integer(args[5]));
  const int act = int(integer(args[6]));
  const Tensor *src[3], *wt[3], *saved[7], &gamma0 = tensor(args[8]);
  bool want[3];
  THPObjectPtr held[3][2];
  const Tensor *perm[3] = {}, *offsets[3] = {};
  static PyObject *const k_perm = name_of("perm"), *const k_offsets = name_of("offsets");
  for (Py_ssize_t j = 0; j < nsrc; ++j) {
    src[j] = &tensor(PySequence_Fast_GET_ITEM(tables.get(), j));
    want[j] = truth(PySequence_Fast_GET_ITEM(wanted.get(), j));
    PyObject* seg = PySequence_Fast_GET_ITEM(segs.get(), j);
    if (seg == Py_None) continue;
    held[j][0] = PyObject_GetAttr(seg, k_perm); held[j][1] = PyObject_GetAttr(seg, k_offsets);
    if (!held[j][0] || !held[j][1]) throw python_error();
    perm[j] = &tensor(held[j][0].get()); offsets[j] = &tensor(held[j][1].get());
  }
  for (int i = 0; i < 3; ++i) wt[i] = &tensor(PySequence_Fast_GET_ITEM(weights.get(), i));
  for (int i = 0; i < 7; ++i) saved[i] = &tensor(PySequence_Fast_GET_ITEM(kept.get(), i));
  std::vector<std::vector<int>> group;
  for (Py_ssize_t k = 0; k < PySequence_Fast_GET_SIZE(groups.get()); ++k) {
    THPObjectPtr members(PySequence_Fast(PySequence_Fast_GET_ITEM(groups.get(), k), "members"));
    if (!members) throw python_error();
    group.emplace_back();
    for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(members.get()); ++i) {
      const long long j = integer(PySequence_Fast_GET_ITEM(members.get(), i));
      if (j < 0 || j >= nsrc || !perm[j]) throw torch::TypeError("groups name indexed tables");
      group.back().push_back(int(j));
    }
  }
  const Tensor &h1 = *saved[0], &h2 = *saved[1], &x3 = *saved[2], &mean = *saved[3], &rstd = *saved[4], &z1 = *saved[5], &z2 = *saved[6];
  Tensor own[2], dsrc[3], dw[3], db[3], dgamma, dbeta;
  int launches = 3;
  {
    const Unlocked unlocked;
    void* const st = stream();
    const int64_t W = kWidth, m = x3.size(0), N = nsrc;
    const Tensor &dy = dense(dy0, own[0]), &gamma = vector32(gamma0, own[1]);
    require(dy.dim() == 2 && dy.size(0) == m && dy.size(1) == W && dy.scalar_type() == at::kBFloat16, "the gradient must be bf16 [rows, 128]");
    // All gradients of parameters in one zeroed buffer, and nothing else: it lives as long as they do.  Before them, in a buffer of its
    // own, the sums against each table's pairs.
    const Tensor grads = zeros32({(N + 2) * W * W + 5 * W}, x3);
    int64_t at = 0;
    auto take = [&](int64_t count) { at += count; return grads.narrow(0, at - count, count); };
    dw[0] = take(N * W * W).view({W, N * W}); dw[1] = take(W * W).view({W, W}); dw[2] = take(W * W).view({W, W});
    for (int i = 0; i < 3; ++i) db[i] = take(W);
    dgamma = take(W); dbeta = take(W);
    const Tensor rows = empty({2, m, W}, at::kBFloat16, x3);
    void *const dx3 = rows.data_ptr(), *const g1 = static_cast<char*>(rows.data_ptr()) + m * W * 2;
    {
      const Tensor scratch = empty({pnm_layernorm_bwd_scratch_floats(m, int(W))}, at::kFloat, x3);
      check("pnm_layernorm_bwd", pnm_layernorm_bwd(ptr(dy), ptr(x3), fptr(gamma), fptr(mean), fptr(rstd), nullptr, dx3, fptr(dgamma), fptr(dbeta),
                                                   fptr(scratch), m, int(W), st));
    }
    check("pnm_mlp3_bwd", pnm_mlp3_bwd(dx3, ptr(z2), ptr(z1), ptr(h2), ptr(h1), ptr(*wt[2]), ptr(*wt[1]), act, g1, fptr(dw[2]), fptr(dw[1]), fptr(db[2]),
                                       fptr(db[1]), m, st));
    float* const dw1 = fptr(dw[0]);
    auto data_gradient = [&](const void* a, int64_t count, int64_t k, const void* b, const Tensor& aux) {
      Tensor out = empty({count, W}, at::kBFloat16, x3);
      check("pnm_gemm_tn", pnm_gemm_tn(a, int(k), nullptr, 0, nullptr, 0, b, int(k), ptr(out), int(W), nullptr, 0, ptr(aux), aux.defined() ? int(W) : 0,
                                       int(count), int(W), int(k), int(k), int(k), nullptr, nullptr, nullptr, 0, aux.defined() ? 1 : 0, 0, 0, 0, st));
      ++launches;
      return out;
    };
    bool summed = false;                         // the bias' gradient: of one source's product
    for (int j = 0; j < N; ++j) {
      if (perm[j]) continue;
      if (want[j]) dsrc[j] = data_gradient(g1, m, W, static_cast<char*>(ptr(*wt[0])) + j * W * W * 2, post == j ? dy : kNone);
      Tensor copy;
      const Tensor& x = rowmajor2d(*src[j], copy);
      check("pnm_gemm_nt", pnm_gemm_nt(g1, int(W), ptr(x), int(x.stride(0)), dw1 + j * W, int(N * W), summed ? nullptr : fptr(db[0]), int(m), int(W), int(W), 0, st));
      ++launches;
      summed = true;
    }
    for (const std::vector<int>& js : group) {
      const int64_t L = js.size(), cols = 2 * W * L;
      Tensor copy;
      const Tensor& x = rowmajor2d(*src[js[0]], copy);
      const int64_t count = offsets[js[0]]->numel() - 1;
      const Tensor pairs = empty({count, cols}, at::kBFloat16, x3);
      for (int k = 0; k < L; ++k) {
        check("pnm_segment_sum_split",
              pnm_segment_sum_split(g1, static_cast<const int*>(ptr(*perm[js[k]])), static_cast<const int*>(ptr(*offsets[js[k]])),
                                    static_cast<char*>(pairs.data_ptr()) + 4 * k * W, cols, count, int(W), st));
        ++launches;
      }
      const Tensor both = zeros32({cols * (W + 1)}, x3);
      check("pnm_gemm_nt", pnm_gemm_nt(ptr(pairs), int(cols), ptr(x), int(x.stride(0)), fptr(both), int(W), summed ? nullptr : fptr(both) + cols * W,
                                       int(count), int(cols), int(W), 0, st));
      ++launches;
      const Tensor halves = both.narrow(0, 0, cols * W).view({L, 2, W, W});
      for (int k = 0; k < L; ++k) {
        Tensor block = dw[0].narrow(1, js[k] * W, W);
        at::add_out(block, halves.select(0, k).select(0, 0), halves.select(0, k).select(0, 1));
      }
      if (!summed) {
        db[0] = both.narrow(0, cols * W, cols).view({L, 2, W}).select(0, 0).sum(0);
        summed = true;
      }
      bool any = false;
      for (int j : js) any = any || want[j];
      if (any) {
        std::vector<Tensor> parts;
        for (int j : js)
          for (int half = 0; half < 2; ++half) parts.push_back(wt[0]->narrow(0, j * W, W));
        const Tensor b = at::cat(parts, 1);
        dsrc[js[0]] = data_gradient(ptr(pairs), count, cols, ptr(b), kNone);
      }
    }
  }
  THPObjectPtr result(PyTuple_New(10)), list(PyList_New(nsrc));
  if (!result || !list) throw python_error();
  for (Py_ssize_t j = 0; j < nsrc; ++j) {
    PyObject* o = dsrc[j].defined() ? THPVariable_Wrap(dsrc[j]) : Py_NewRef(Py_None);
    if (!o) throw python_error();
    PyList_SET_ITEM(list.get(), j, o);
  }
  PyTuple_SET_ITEM(result.get(), 0, list.release());
  const Tensor* out[8] = {&dw[0], &dw[1], &dw[2], &db[0], &db[1], &db[2], &dgamma, &dbeta};
  for (int i = 0; i < 8; ++i) {
    PyObject* o = THPVariable_Wrap(*out[i]);
    if (!o) throw python_error();
    PyTuple_SET_ITEM(result.get(), i + 1, o);
  }
  PyObject* count = PyLong_FromLong(launches);
  if (!count) throw python_error();
  PyTuple_SET_ITEM(result.get(), 9, count);
  return result.release();
  END_HANDLE_TH_ERRORS
}

// segment_sum(x, perm, offsets, segments, accumulate, mean, out or None) -> out
PyObject* segment_sum(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 7);
  const Tensor &x = tensor(args[0]), &perm = tensor(args[1]), &offsets = tensor(args[2]), &given = optional(args[6]);
  const int64_t segments = integer(args[3]);
  const int accumulate = truth(args[4]), mean = truth(args[5]);
  Tensor made;
  const Tensor& out = given.defined() ? given : made;
  {
    const Unlocked unlocked;
    require(x.dim() == 2, "expected a matrix");
    const int64_t C = x.size(1);
    if (!given.defined()) made = empty({segments, C}, at::kBFloat16, x);
    check("pnm_segment_sum",
          pnm_segment_sum(ptr(x), int(x.stride(0)), static_cast<const int*>(ptr(perm)), static_cast<const int*>(ptr(offsets)), ptr(out),
                          int(out.stride(0)), segments, int(C), accumulate, mean, stream()));
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// gather_rows(x, index, scale or None, out or None) -> out
PyObject* gather_rows(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 4);
  const Tensor &x = tensor(args[0]), &index = tensor(args[1]), &scale = optional(args[2]), &given = optional(args[3]);
  Tensor made;
  const Tensor& out = given.defined() ? given : made;
  {
    const Unlocked unlocked;
    require(x.dim() == 2, "expected a matrix");
    const int64_t E = index.numel(), C = x.size(1);
    if (!given.defined()) made = empty({E, C}, at::kBFloat16, x);
    check("pnm_gather_rows", pnm_gather_rows(ptr(x), int(x.stride(0)), static_cast<const int*>(ptr(index)), fptr(scale), ptr(out), int(out.stride(0)), E,
                                             int(C), stream()));
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// conv2d_nhwc(x [n, h, w, cin], packed weight [cout, k k cin], bias fp32 [cout] or None, k, act) -> y [n, h, w, cout]
PyObject* conv2d_nhwc(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 5);
  const Tensor &x = tensor(args[0]), &w = tensor(args[1]), &bias = optional(args[2]);
  const int k = int(integer(args[3])), act = int(integer(args[4]));
  Tensor y;
  {
    const Unlocked unlocked;
    require(x.dim() == 4, "expected an image [n, h, w, c]");
    const int N = int(x.size(0)), H = int(x.size(1)), W = int(x.size(2)), cin = int(x.size(3)), cout = int(w.size(0));
    y = empty({N, H, W, cout}, at::kBFloat16, x);
    check("pnm_conv2d_nhwc", pnm_conv2d_nhwc(ptr(x), ptr(w), ptr(y), N, H, W, cin, cout, k, fptr(bias), act, 0, 0, stream()));
  }
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

// conv_pack_weight(weight [cout, cin, k, k], rows, cols, flip) -> [rows, k k cols] bf16
PyObject* conv_pack_weight(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 4);
  const Tensor& w = tensor(args[0]);
  const int rows = int(integer(args[1])), cols = int(integer(args[2])), flip = truth(args[3]);
  Tensor out;
  {
    const Unlocked unlocked;
    require(w.dim() == 4, "expected a filter [cout, cin, k, k]");
    const int cout = int(w.size(0)), cin = int(w.size(1)), k = int(w.size(2));
    out = empty({rows, int64_t(k) * k * cols}, at::kBFloat16, w);
    check("pnm_conv_pack_weight", pnm_conv_pack_weight(ptr(w), w.scalar_type() == at::kBFloat16, ptr(out), cout, cin, k, rows, cols, flip, stream()));
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// groupnorm_fwd(x, gamma, beta, groups, slices, layout, dtype, silu, eps) -> (y, mean, rstd)
PyObject* groupnorm_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 9);
  const Tensor &x = tensor(args[0]), &gamma = tensor(args[1]), &beta = tensor(args[2]);
  const int G = int(integer(args[3])), S = int(integer(args[4])), layout = int(integer(args[5])), dtype = int(integer(args[6])), silu = truth(args[7]);
  const float eps = float(real(args[8]));
  Tensor y, mean, rstd;
  {
    const Unlocked unlocked;
    require(x.dim() >= 2 && x.numel() > 0, "expected [batch, channels, ...]");
    const int B = int(x.size(0)), C = int(x.size(1));
    const long long hw = x.numel() / (int64_t(B) * C);
    y = at::empty_like(x); mean = empty({int64_t(B) * G}, at::kFloat, x); rstd = empty({int64_t(B) * G}, at::kFloat, x);
    const Tensor scratch = empty({pnm_groupnorm_scratch_floats(B, C, G, S)}, at::kFloat, x);
    check("pnm_groupnorm_fwd", pnm_groupnorm_fwd(ptr(x), fptr(gamma), fptr(beta), ptr(y), fptr(mean), fptr(rstd), fptr(scratch), B, C, hw, G, S, layout,
                                                 dtype, silu, eps, stream()));
  }
  return tuple_of({&y, &mean, &rstd});
  END_HANDLE_TH_ERRORS
}

// pa_prepare_fwd(Wx, bx, Wfx, Ws, bs, temperature, heads, head width) -> (Wc, bc, inv_t, Wfx16, Wback)
PyObject* pa_prepare_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 8);
  const Tensor* p[6];
  for (int i = 0; i < 6; ++i) p[i] = &tensor(args[i]);
  const int64_t H = integer(args[6]), D = integer(args[7]), HS = H * 64, inner = H * D;
  Tensor Wc, bc, inv_t, Wfx16, Wback;
  {
    const Unlocked unlocked;
    const int64_t C = p[0]->size(1);
    Wc = empty({HS, C}, at::kBFloat16, *p[0]); bc = empty({HS}, at::kFloat, *p[0]); inv_t = empty({HS}, at::kFloat, *p[0]);
    Wfx16 = empty({inner, C}, at::kBFloat16, *p[0]); Wback = empty({C, HS + inner}, at::kBFloat16, *p[0]);
    check("pnm_pa_prepare_fwd", pnm_pa_prepare_fwd(fptr(*p[0]), fptr(*p[1]), fptr(*p[2]), fptr(*p[3]), fptr(*p[4]), fptr(*p[5]), ptr(Wc), fptr(bc),
                                                   fptr(inv_t), ptr(Wfx16), ptr(Wback), int(H), int(D), int(C), stream()));
  }
  return tuple_of({&Wc, &bc, &inv_t, &Wfx16, &Wback});
  END_HANDLE_TH_ERRORS
}

// floats of what the forward of the slice-token kernel keeps: token, norm, q, k, v, probabilities, out, Wcomb one after the other
struct TokenParts {
  int64_t count[8], total = 0;
  TokenParts(int64_t H, int64_t D, int64_t cout) : count{H * 64 * D, H * 64, H * 64 * D, H * 64 * D, H * 64 * D, H * 64 * 64, H * 64 * D, cout * H * 64} {
    for (int64_t c : count) total += c;
  }
  void addresses(float* base, void** out) const {
    for (int i = 0; i < 8; base += count[i++]) out[i] = base;
  }
};

// pa_tokens_fwd(address of the token sums, offset of the norms, row length, Wqkv, Wo, heads, head width) -> (Wcomb bf16, kept)
PyObject* pa_tokens_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 7);
  const void* const src = reinterpret_cast<const void*>(uintptr_t(integer(args[0])));
  const long long norm_off = integer(args[1]);
  const int ld = int(integer(args[2])), H = int(integer(args[5])), D = int(integer(args[6]));
  const Tensor &Wqkv = tensor(args[3]), &Wo = tensor(args[4]);
  Tensor wcomb, kept;
  {
    const Unlocked unlocked;
    const int64_t cout = Wo.size(0);
    const TokenParts parts(H, D, cout);
    kept = empty({parts.total}, at::kFloat, Wo);
    wcomb = empty({cout, int64_t(H) * 64}, at::kBFloat16, Wo);
    void* saved[8];
    parts.addresses(fptr(kept), saved);
    check("pnm_pa_tokens_fwd", pnm_pa_tokens_fwd(&src, 1, 0, norm_off, ld, fptr(Wqkv), fptr(Wo), ptr(wcomb), saved, H, D, int(cout),
                                                 float(1.0 / std::sqrt(double(D))), nullptr, 0, 0, 0, 1.0, nullptr, stream()));
  }
  return tuple_of({&wcomb, &kept});
  END_HANDLE_TH_ERRORS
}

// pa_tokens_bwd(address of dWcomb, Wqkv, Wo, kept, heads, head width, share) -> (dWo, dWqkv, d_norm, Bcat, BdT)
PyObject* pa_tokens_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 7);
  const void* const src = reinterpret_cast<const void*>(uintptr_t(integer(args[0])));
  const Tensor &Wqkv = tensor(args[1]), &Wo = tensor(args[2]), &kept = tensor(args[3]);
  const int H = int(integer(args[4])), D = int(integer(args[5]));
  const float share = float(real(args[6]));
  Tensor dWo, dWqkv, d_norm, Bcat, BdT;
  {
    const Unlocked unlocked;
    const int64_t cout = Wo.size(0), inner = int64_t(H) * D, HS = int64_t(H) * 64;
    const TokenParts parts(H, D, cout);
    require(kept.numel() == parts.total && kept.is_contiguous(), "kept values of another layer");
    dWo = empty({cout, inner}, at::kFloat, Wo); dWqkv = zeros32({3 * int64_t(D), D}, Wo); d_norm = empty({HS}, at::kFloat, Wo);
    Bcat = empty({HS, cout + inner}, at::kBFloat16, Wo); BdT = empty({inner, HS}, at::kBFloat16, Wo);
    void* saved[8];
    parts.addresses(fptr(kept), saved);
    check("pnm_pa_tokens_bwd", pnm_pa_tokens_bwd(&src, 1, 0, fptr(Wqkv), fptr(Wo), saved, fptr(dWo), fptr(dWqkv), fptr(d_norm), ptr(Bcat), ptr(BdT), H, D,
                                                 int(cout), float(1.0 / std::sqrt(double(D))), share, nullptr, 0, 0, 0, 1.0, nullptr, stream()));
  }
  return tuple_of({&dWo, &dWqkv, &d_norm, &Bcat, &BdT});
  END_HANDLE_TH_ERRORS
}

// pa_prepare_bwd(dW [64 H + H D, C], db, per-head sums, Wx, bx, Ws, temperature, heads, head width) -> (dWx, dbx, dWfx, dbfx, dWs, dbs, dtemp)
PyObject* pa_prepare_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 9);
  const Tensor* p[7];
  for (int i = 0; i < 7; ++i) p[i] = &tensor(args[i]);
  const int64_t H = integer(args[7]), D = integer(args[8]);
  Tensor dWx, dbx, dWfx, dbfx, dWs, dbs, dtemp;
  {
    const Unlocked unlocked;
    const Tensor& like = *p[3];
    const int64_t C = like.size(1), inner = H * D, rows = H * 64 + inner;
    require(p[0]->numel() == rows * C && p[1]->numel() == rows && p[0]->is_contiguous() && p[1]->is_contiguous(), "gradients of another layer");
    dWx = empty({inner, C}, at::kFloat, like); dbx = empty({inner}, at::kFloat, like); dWfx = empty({inner, C}, at::kFloat, like);
    dbfx = empty({inner}, at::kFloat, like); dWs = empty({64, D}, at::kFloat, like); dbs = empty({64}, at::kFloat, like);
    dtemp = empty({H}, at::kFloat, like);
    check("pnm_pa_prepare_bwd", pnm_pa_prepare_bwd(fptr(*p[0]), fptr(*p[1]), fptr(*p[2]), fptr(*p[3]), fptr(*p[4]), fptr(*p[5]), fptr(*p[6]), fptr(dWx),
                                                   fptr(dbx), fptr(dWfx), fptr(dbfx), fptr(dWs), fptr(dbs), fptr(dtemp), int(H), int(D), int(C), stream()));
  }
  return tuple_of({&dWx, &dbx, &dWfx, &dbfx, &dWs, &dbs, &dtemp});
  END_HANDLE_TH_ERRORS
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(gemm_tn),     FAST(gemm_nt),     FAST(layernorm_fwd),    FAST(mlp3_operands_ok), FAST(mlp3_module),    FAST(mlp3_bwd), FAST(mlp3_fwd),       FAST(segment_sum),
                         FAST(gather_rows), FAST(conv2d_nhwc), FAST(conv_pack_weight), FAST(groupnorm_fwd),    FAST(pa_prepare_fwd), FAST(pa_tokens_fwd),
                         FAST(pa_tokens_bwd), FAST(pa_prepare_bwd),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pnm_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pnm_host() { return PyModule_Create(&module); }
