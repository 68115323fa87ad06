// Host side of the hottest calls as a CPython extension: checks of the operands, allocation of the results and the launch.
//
// A small call (a roll-out step of a mesh network, a block on a few thousand points) is bound by its host side: in Python one launch
// took 15 to 50 us (attributes of every tensor, torch.empty, the foreign-function call with up to 40 arguments).  The
// functions do what the Python code did, argument by argument; gradients, dispatch and weight copies stay in Python.  Together with calls
// that skip the autograd function where no gradient is wanted: a message-passing step of 1 885 nodes (three launches) 150 -> 78 us, a Transolver
// block of 4 096 points (eleven) 373 -> 231 us, an AFNO block (twelve) 305 -> 223 us, a U-Net block with attention 601 -> 427 us.
// As there, the interpreter's lock is released not only for the launch but also where memory is allocated or copied (an allocation may wait
// for the device): every function reads its arguments, works in an `Unlocked` scope and wraps its results.
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

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
    const auto f32 = at::TensorOptions().dtype(at::kFloat).device(a.device());
    if (!given.defined()) made = at::zeros({Na, Nb}, f32);
    if (!given_sums.defined() && want_sums) made_sums = at::zeros({Na}, f32);
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
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(biases.get()); ++i) {
    PyObject* o = PySequence_Fast_GET_ITEM(biases.get(), i);
    if (o != Py_None && !parameter(o)) Py_RETURN_FALSE;
  }
  if (!parameter(args[3]) || THPVariable_Unpack(args[3]).numel() != kWidth || (args[4] != Py_None && !parameter(args[4]))) Py_RETURN_FALSE;
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

// empties(like, is_bf16, shape, shape, ...) -> list of tensors on like's device (many small results of one launch)
PyObject* empties(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n < 2) throw torch::TypeError("expected a tensor, a flag and shapes");
  const Tensor& like = tensor(args[0]);
  const at::ScalarType type = truth(args[1]) ? at::kBFloat16 : at::kFloat;
  std::vector<std::vector<int64_t>> shapes(n - 2);
  for (Py_ssize_t k = 2; k < n; ++k) {
    if (!PyTuple_Check(args[k])) throw torch::TypeError("shapes are tuples of numbers");
    for (Py_ssize_t d = 0; d < PyTuple_GET_SIZE(args[k]); ++d) shapes[k - 2].push_back(integer(PyTuple_GET_ITEM(args[k], d)));
  }
  std::vector<Tensor> tensors;
  {
    const Unlocked unlocked;
    for (const auto& shape : shapes) tensors.push_back(empty(shape, type, like));
  }
  THPObjectPtr result(PyList_New(n - 2));
  if (!result) throw python_error();
  for (Py_ssize_t k = 0; k < n - 2; ++k) {
    PyObject* o = THPVariable_Wrap(tensors[k]);
    if (!o) throw python_error();
    PyList_SET_ITEM(result.get(), k, o);
  }
  return result.release();
  END_HANDLE_TH_ERRORS
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(gemm_tn),     FAST(gemm_nt),     FAST(layernorm_fwd),    FAST(mlp3_operands_ok), FAST(mlp3_fwd),       FAST(segment_sum),
                         FAST(gather_rows), FAST(conv2d_nhwc), FAST(conv_pack_weight), FAST(groupnorm_fwd),    FAST(pa_prepare_fwd), FAST(empties),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pnm_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pnm_host() { return PyModule_Create(&module); }
