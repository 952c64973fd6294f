// The launch path in native code: argument checks, output allocation and the call of the C ABI in one function per operation, for arguments in their plain form
// (CUDA tensors of the current device, contiguous where the kernels need it, the expected types and shapes).  For any other form a function returns None and
// the Python path of fovi_b200/ops.py takes the call, with its conversions and error messages; a status of the C ABI other than 0 is returned as an int.
// What bounds small calls is the host: a sensor call through Python checks, torch.empty and ctypes took 12 us, 5 us of them in the launch and its
// 5 us kernel behind it.
// The C ABI's functions are handed over by address (`connect`), so this module works with whichever build of the library is loaded.
#include <Python.h>

#include <ATen/ATen.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <stdint.h>

#include "../../include/fovi_b200.h"

namespace {

struct Abi {
  decltype(&fovi_sample_forward) sample = nullptr;
  decltype(&fovi_knnconv_forward) conv = nullptr;
  decltype(&fovi_knnconv_forward_f32) conv_f32 = nullptr;
  decltype(&fovi_pack_points) pack_points = nullptr;
  decltype(&fovi_knnconv_pack_weights) pack_weights = nullptr;
  decltype(&fovi_knnconv_pack_weights_transposed) pack_weights_t = nullptr;
  decltype(&fovi_knndw_run) dw_run = nullptr;
  decltype(&fovi_weight_grad_unpack) unpack = nullptr;
  decltype(&fovi_points_to_channels) to_channels = nullptr;
  decltype(&fovi_relu_pool_forward) relu_pool = nullptr;
  decltype(&fovi_norm_block_workspace_bytes) norm_work = nullptr;
  decltype(&fovi_norm_block_backward) norm_back = nullptr;
} abi;

struct Release {      // the interpreter lock is free while a call allocates or launches, as under ctypes
  PyThreadState* state = PyEval_SaveThread();
  ~Release() { PyEval_RestoreThread(state); }
};

// A plain tensor of the current device, or nullptr.
const at::Tensor* plain(PyObject* o, int device) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.has_storage() || !t.is_cuda() || t.get_device() != device || t.layout() != at::kStrided) return nullptr;
  return &t;
}
int code_of(at::ScalarType t) { return t == at::kFloat ? FOVI_F32 : t == at::kBFloat16 ? FOVI_BF16 : t == at::kByte ? FOVI_U8 : -1; }
at::ScalarType type_of(long code) { return code == FOVI_BF16 ? at::kBFloat16 : at::kFloat; }
long num(PyObject* o) { return PyLong_AsLong(o); }
void* handle(PyObject* o) { return o == Py_None ? nullptr : PyLong_AsVoidPtr(o); }
at::Tensor fresh(at::IntArrayRef shape, at::ScalarType type, int device) {
  return at::empty(shape, at::TensorOptions().dtype(type).device(at::Device(at::kCUDA, (c10::DeviceIndex)device)));
}
PyObject* status_or(int rc, const at::Tensor& t) { return rc ? PyLong_FromLong(rc) : THPVariable_Wrap(t); }
// float32 [n] contiguous, or null for None; false: not plain
bool bias_arg(PyObject* o, int device, int64_t n, const float** p) {
  *p = nullptr;
  if (o == Py_None) return true;
  const at::Tensor* t = plain(o, device);
  if (!t || t->scalar_type() != at::kFloat || !t->is_contiguous() || t->numel() != n) return false;
  *p = t->const_data_ptr<float>();
  return true;
}

#define BODY(NAME, COUNT)                                                              \
  PyObject* NAME(PyObject*, PyObject* const* v, Py_ssize_t n) {                        \
    if (n != COUNT) { PyErr_SetString(PyExc_TypeError, #NAME ": wrong number of arguments"); return nullptr; } \
    const int dev = (int)num(v[COUNT - 2]);                                            \
    void* st = handle(v[COUNT - 1]);                                                   \
    if (PyErr_Occurred()) return nullptr;                                              \
    HANDLE_TH_ERRORS
#define END END_HANDLE_TH_ERRORS }
#define GENERAL Py_RETURN_NONE

// plan, points, img, fix_rc, fix_hw, mode, pad, out dtype or -1, layout, channel stride or 0, device, stream
BODY(sample, 12)
  const at::Tensor *img = plain(v[2], dev), *rc = plain(v[3], dev), *hw = plain(v[4], dev);
  if (!img || !rc || !hw || img->dim() != 4 || rc->dim() != 3) GENERAL;
  const int dt = code_of(img->scalar_type());
  const int64_t B = img->size(0), C = img->size(1), H = img->size(2), W = img->size(3), F = rc->size(1), N = num(v[1]);
  if (dt < 0 || rc->scalar_type() != at::kFloat || hw->scalar_type() != at::kFloat || !rc->is_contiguous() || !hw->is_contiguous() || rc->size(0) != B ||
      rc->size(2) != 2 || hw->sizes() != rc->sizes() || B > INT32_MAX || C > INT32_MAX || H > INT32_MAX || W > INT32_MAX || F > INT32_MAX)
    GENERAL;
  const long mode = num(v[5]), pad = num(v[6]), layout = num(v[8]), stride = num(v[9]);
  long od = num(v[7]);
  if (PyErr_Occurred()) return nullptr;
  const bool pairs = layout == FOVI_OUT_FB_PAIRS || layout == FOVI_OUT_BF_PAIRS, nc = layout == FOVI_OUT_BFNC || layout == FOVI_OUT_FBNC;
  const bool f_first = layout == FOVI_OUT_FBCN || layout == FOVI_OUT_FBNC;
  if (od < -1) GENERAL;      // a type the kernels do not write
  if (od < 0) od = dt == FOVI_BF16 ? FOVI_BF16 : FOVI_F32;
  int64_t cp = nc && stride ? stride : C;
  int64_t shape[4] = {f_first ? F : B, f_first ? B : F, nc ? N : C, nc ? cp : N};
  if (pairs) {
    od = FOVI_BF16; cp = 8;
    shape[0] = (B * F + 127) / 128; shape[1] = (N + 1) / 2; shape[2] = 128; shape[3] = 8;
  }
  const int64_t strides[4] = {img->stride(0), img->stride(1), img->stride(2), img->stride(3)};
  at::Tensor out;
  int rcode;
  {
    Release r;
    out = fresh(at::IntArrayRef(shape, 4), type_of(od), dev);
    rcode = abi.sample(static_cast<const fovi_sampler_plan*>(handle(v[0])), img->const_data_ptr(), dt, (int)B, (int)C, (int)H, (int)W, strides,
                       rc->const_data_ptr<float>(), hw->const_data_ptr<float>(), (int)F, (int)mode, (int)pad, out.mutable_data_ptr(), (int)od, (int)layout, (int)cp, st);
  }
  return status_or(rcode, out);
END

// plan, x, wt, bias, relu, out dtype, rows, (x's sizes behind the batch or row tiles) x1, x2, (wt's sizes) w0, w1, w2, pairs, n_out, c_out, device, stream
BODY(conv_forward, 17)
  const at::Tensor *x = plain(v[1], dev), *wt = plain(v[2], dev);
  if (!x || !wt || x->scalar_type() != at::kBFloat16 || wt->scalar_type() != at::kBFloat16 || !x->is_contiguous() || !wt->is_contiguous()) GENERAL;
  const int64_t rows = num(v[6]), x1 = num(v[7]), x2 = num(v[8]), w0 = num(v[9]), w1 = num(v[10]), w2 = num(v[11]), pairs = num(v[12]), n_out = num(v[13]),
                c_out = num(v[14]);
  const long relu = num(v[4]), od = num(v[5]);
  if (PyErr_Occurred()) return nullptr;
  if (od < 0) GENERAL;
  if (pairs) {
    if (x->dim() != 4 || wt->dim() != 4 || x->size(0) != (rows + 127) / 128 || x->size(1) != x1 || x->size(2) != 128 || x->size(3) != 8 || wt->size(0) != w0 ||
        wt->size(2) != w1 || wt->size(3) != w2)
      GENERAL;
  } else if (x->dim() != 3 || wt->dim() != 3 || x->size(0) != rows || x->size(1) != x1 || x->size(2) != x2 || wt->size(0) != w0 || wt->size(1) != w1 ||
             wt->size(2) != w2) {
    GENERAL;
  }
  const float* bias;
  if (rows > INT32_MAX || !bias_arg(v[3], dev, c_out, &bias)) GENERAL;
  at::Tensor out;
  int rcode;
  {
    Release r;
    out = fresh({rows, n_out, c_out}, type_of(od), dev);
    rcode = abi.conv(static_cast<fovi_knnconv_plan*>(handle(v[0])), x->const_data_ptr(), wt->const_data_ptr(), bias, out.mutable_data_ptr(), (int)od, (int)rows,
                     (int)relu, st);
  }
  return status_or(rcode, out);
END

// plan, x [B,c_in,n_in], wt, bias, n_in, c_in, V, cin_packed, n_out, c_out, device, stream
BODY(conv_forward_f32, 12)
  const at::Tensor *x = plain(v[1], dev), *wt = plain(v[2], dev);
  if (!x || !wt || x->dim() != 3 || wt->dim() != 3 || !x->is_contiguous() || wt->scalar_type() != at::kFloat || !wt->is_contiguous()) GENERAL;
  const int dt = code_of(x->scalar_type());
  const int64_t n_in = num(v[4]), c_in = num(v[5]), V = num(v[6]), cp = num(v[7]), n_out = num(v[8]), c_out = num(v[9]), B = x->size(0);
  if (PyErr_Occurred()) return nullptr;
  const float* bias;
  if ((dt != FOVI_F32 && dt != FOVI_BF16) || x->size(1) != c_in || x->size(2) != n_in || wt->size(0) != V || wt->size(1) != c_out || wt->size(2) != cp || B > INT32_MAX ||
      !bias_arg(v[3], dev, c_out, &bias))
    GENERAL;
  at::Tensor out;
  int rcode;
  {
    Release r;
    out = fresh({B, c_out, n_out}, at::kFloat, dev);
    rcode = abi.conv_f32(static_cast<fovi_knnconv_plan*>(handle(v[0])), x->const_data_ptr(), dt, FOVI_ACT_BCN, wt->const_data_ptr<float>(), bias,
                         out.mutable_data_ptr<float>(), FOVI_ACT_BCN, (int)B, 0, st);
  }
  return status_or(rcode, out);
END

// x [B,C,N] contiguous, channels of the packed layout, layout, device, stream
BODY(pack_points, 5)
  const at::Tensor* x = plain(v[0], dev);
  if (!x || x->dim() != 3 || !x->is_contiguous()) GENERAL;
  const int dt = code_of(x->scalar_type());
  const int64_t B = x->size(0), C = x->size(1), N = x->size(2), cp = num(v[1]), layout = num(v[2]);
  if (PyErr_Occurred()) return nullptr;
  if ((dt != FOVI_F32 && dt != FOVI_BF16) || B > INT32_MAX || C > INT32_MAX || N > INT32_MAX) GENERAL;
  at::Tensor out;
  int rcode;
  {
    Release r;
    out = layout == FOVI_X_PAIRS ? fresh({(B + 127) / 128, (N + 1) / 2, 128, 8}, at::kBFloat16, dev) : fresh({B, N, cp}, at::kBFloat16, dev);
    rcode = abi.pack_points(x->const_data_ptr(), dt, (int)B, (int)C, (int)N, out.mutable_data_ptr(), (int)cp, (int)layout, st);
  }
  return status_or(rcode, out);
END

// plan, weight [rows, columns], rows, columns, (slabs) V, c_out, cin_packed, out dtype, transposed, device, stream
BODY(pack_slabs, 11)
  const at::Tensor* w = plain(v[1], dev);
  const int64_t rows = num(v[2]), cols = num(v[3]), V = num(v[4]), c_out = num(v[5]), cp = num(v[6]);
  const long od = num(v[7]), transposed = num(v[8]);
  if (PyErr_Occurred()) return nullptr;
  if (od < 0 || !w || w->dim() != 2 || !w->is_contiguous() || w->size(0) != rows || w->size(1) != cols) GENERAL;
  const int dt = code_of(w->scalar_type());
  if (dt != FOVI_F32 && dt != FOVI_BF16) GENERAL;
  at::Tensor out;
  int rcode;
  {
    Release r;
    out = fresh({V, c_out, cp}, type_of(od), dev);
    auto* p = static_cast<fovi_knnconv_plan*>(handle(v[0]));
    rcode = transposed ? abi.pack_weights_t(p, w->const_data_ptr(), dt, out.mutable_data_ptr(), (int)od, st)
                       : abi.pack_weights(p, w->const_data_ptr(), dt, out.mutable_data_ptr(), (int)od, st);
  }
  return status_or(rcode, out);
END

// plan, p [B,n_p,cp], q [B,n_q,cq], n_p, n_q, V, c_out, c_in, swapped, out dtype, device, stream -> filter gradient [c_out, c_in*V]
BODY(weight_grad, 12)
  const at::Tensor *p = plain(v[1], dev), *q = plain(v[2], dev);
  const int64_t n_p = num(v[3]), n_q = num(v[4]), V = num(v[5]), c_out = num(v[6]), c_in = num(v[7]);
  const long swapped = num(v[8]), od = num(v[9]);
  if (PyErr_Occurred()) return nullptr;
  if (od < 0 || !p || !q || p->dim() != 3 || q->dim() != 3 || p->scalar_type() != at::kBFloat16 || q->scalar_type() != at::kBFloat16 || !p->is_contiguous() ||
      !q->is_contiguous() || p->size(0) != q->size(0) || p->size(1) != n_p || q->size(1) != n_q || p->size(0) > INT32_MAX)
    GENERAL;
  const int64_t cp = p->size(2), cq = q->size(2);
  at::Tensor out;
  int rcode;
  {
    Release r;
    at::Tensor sums = fresh({V, cp, cq}, at::kFloat, dev);
    sums.zero_();
    out = fresh({c_out, c_in * V}, type_of(od), dev);
    rcode = abi.dw_run(static_cast<fovi_knndw_plan*>(handle(v[0])), p->const_data_ptr(), (int)cp, q->const_data_ptr(), (int)cq, (int)p->size(0),
                       sums.mutable_data_ptr<float>(), st);
    if (!rcode)
      rcode = abi.unpack(sums.const_data_ptr<float>(), (int)V, (int)cp, (int)cq, (int)swapped, (int)c_out, (int)c_in, out.mutable_data_ptr(), (int)od, st);
  }
  return status_or(rcode, out);
END

// A training block's forward pass behind its convolution: y [B,N,C], gamma, beta, running mean, running variance, number of batches, momentum, eps, cudnn, relu, pool or None,
// n_out, device, stream -> (mean, rstd, out [B,n_out,C], arg or None)
BODY(block_forward, 14)
  const at::Tensor* t[6];
  for (int i = 0; i < 6; ++i)
    if (!(t[i] = plain(v[i], dev))) GENERAL;
  const at::Tensor& y = *t[0];
  const double momentum = PyFloat_AsDouble(v[6]), eps = PyFloat_AsDouble(v[7]);
  const long cudnn = num(v[8]), relu = num(v[9]);
  const int64_t n_out = num(v[11]);
  void* pool = handle(v[10]);
  if (PyErr_Occurred()) return nullptr;
  if (y.dim() != 3 || y.scalar_type() != at::kFloat || !y.is_contiguous()) GENERAL;
  const int64_t B = y.size(0), N = y.size(1), C = y.size(2);
  at::Tensor mean, rstd, out, arg;
  int rcode;
  {
    Release r;
    at::Tensor yt = fresh({B, C, N}, at::kFloat, dev);
    rcode = abi.to_channels(y.const_data_ptr<float>(), yt.mutable_data_ptr<float>(), (int)B, (int)N, (int)C, st);
    if (!rcode) {
      const_cast<at::Tensor&>(*t[5]).add_(1);
      auto bn = at::_batch_norm_impl_index(yt, *t[1], *t[2], *t[3], *t[4], true, momentum, eps, cudnn != 0);
      mean = std::get<1>(bn); rstd = std::get<2>(bn);
      out = fresh({B, n_out, C}, at::kFloat, dev);
      if (pool) arg = fresh({B, n_out, C}, at::kByte, dev);
      rcode = abi.relu_pool(std::get<0>(bn).const_data_ptr<float>(), (int)B, (int)N, (int)C, (int)relu, static_cast<const fovi_knnpool_plan*>(pool),
                            out.mutable_data_ptr<float>(), pool ? arg.mutable_data_ptr<uint8_t>() : nullptr, st);
    }
  }
  if (rcode) return PyLong_FromLong(rcode);
  PyObject* tuple = PyTuple_New(4);
  if (!tuple) return nullptr;
  PyTuple_SET_ITEM(tuple, 0, THPVariable_Wrap(mean));
  PyTuple_SET_ITEM(tuple, 1, THPVariable_Wrap(rstd));
  PyTuple_SET_ITEM(tuple, 2, THPVariable_Wrap(out));
  if (pool) PyTuple_SET_ITEM(tuple, 3, THPVariable_Wrap(arg));
  else { Py_INCREF(Py_None); PyTuple_SET_ITEM(tuple, 3, Py_None); }
  return tuple;
END

// Its backward pass: y, mean, rstd, gamma, act or None, arg or None, g [B,n_out,C], pool or None, device, stream -> (dy bf16 [B,N,C], dgamma, dbeta)
BODY(block_backward, 10)
  const at::Tensor* t[5];
  PyObject* const need[5] = {v[0], v[1], v[2], v[3], v[6]};
  for (int i = 0; i < 5; ++i)
    if (!(t[i] = plain(need[i], dev)) || t[i]->scalar_type() != at::kFloat || !t[i]->is_contiguous()) GENERAL;
  const at::Tensor *act = nullptr, *arg = nullptr;
  if (v[4] != Py_None && (!(act = plain(v[4], dev)) || act->scalar_type() != at::kFloat || !act->is_contiguous())) GENERAL;
  if (v[5] != Py_None && (!(arg = plain(v[5], dev)) || arg->scalar_type() != at::kByte || !arg->is_contiguous())) GENERAL;
  void* pool = handle(v[7]);
  if (PyErr_Occurred()) return nullptr;
  const at::Tensor &y = *t[0], &g = *t[4];
  if (y.dim() != 3 || g.dim() != 3 || g.size(0) != y.size(0) || g.size(2) != y.size(2) || (act && act->sizes() != y.sizes()) || (arg && arg->sizes() != g.sizes()) ||
      (!pool && g.sizes() != y.sizes()))
    GENERAL;
  const int64_t B = y.size(0), N = y.size(1), C = y.size(2);
  if (t[1]->numel() != C || t[2]->numel() != C || t[3]->numel() != C) GENERAL;
  at::Tensor dx, sums;
  int rcode;
  {
    Release r;
    const int64_t bytes = abi.norm_work((int)B, (int)N, (int)C);
    dx = fresh({B, N, C}, at::kBFloat16, dev);
    sums = fresh({2, C}, at::kFloat, dev);
    at::Tensor work = fresh({bytes}, at::kByte, dev);
    float* d = sums.mutable_data_ptr<float>();
    rcode = abi.norm_back(y.const_data_ptr<float>(), (int)B, (int)N, (int)C, t[1]->const_data_ptr<float>(), t[2]->const_data_ptr<float>(), t[3]->const_data_ptr<float>(),
                          act ? act->const_data_ptr<float>() : nullptr, static_cast<const fovi_knnpool_plan*>(pool), arg ? arg->const_data_ptr<uint8_t>() : nullptr,
                          g.const_data_ptr<float>(), d, d + C, dx.mutable_data_ptr(), work.mutable_data_ptr(), bytes, st);
  }
  if (rcode) return PyLong_FromLong(rcode);
  PyObject* tuple = PyTuple_New(3);
  if (!tuple) return nullptr;
  PyTuple_SET_ITEM(tuple, 0, THPVariable_Wrap(dx));
  PyTuple_SET_ITEM(tuple, 1, THPVariable_Wrap(sums.select(0, 0)));
  PyTuple_SET_ITEM(tuple, 2, THPVariable_Wrap(sums.select(0, 1)));
  return tuple;
END

// {name of the C ABI's function: its address}
PyObject* connect(PyObject*, PyObject* dict) {
  const struct { const char* name; void** at; } want[] = {
      {"fovi_sample_forward", (void**)&abi.sample}, {"fovi_knnconv_forward", (void**)&abi.conv}, {"fovi_knnconv_forward_f32", (void**)&abi.conv_f32},
      {"fovi_pack_points", (void**)&abi.pack_points}, {"fovi_knnconv_pack_weights", (void**)&abi.pack_weights},
      {"fovi_knnconv_pack_weights_transposed", (void**)&abi.pack_weights_t}, {"fovi_knndw_run", (void**)&abi.dw_run},
      {"fovi_weight_grad_unpack", (void**)&abi.unpack}, {"fovi_points_to_channels", (void**)&abi.to_channels},
      {"fovi_relu_pool_forward", (void**)&abi.relu_pool}, {"fovi_norm_block_workspace_bytes", (void**)&abi.norm_work},
      {"fovi_norm_block_backward", (void**)&abi.norm_back}};
  for (const auto& w : want) {
    PyObject* a = PyDict_GetItemString(dict, w.name);
    if (!a) { PyErr_Format(PyExc_KeyError, "%s", w.name); return nullptr; }
    *w.at = PyLong_AsVoidPtr(a);
    if (PyErr_Occurred()) return nullptr;
  }
  Py_RETURN_NONE;
}

#define FAST(NAME) {#NAME, (PyCFunction)(void (*)(void))NAME, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(sample), FAST(conv_forward), FAST(conv_forward_f32), FAST(pack_points), FAST(pack_slabs), FAST(weight_grad), FAST(block_forward),
                         FAST(block_backward), {"connect", connect, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// The module says which torch it was compiled against: its tensors are that one's C++ objects.
PyMODINIT_FUNC PyInit__native() {
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "made_for", FOVI_TORCH_VERSION)) { Py_DECREF(m); return nullptr; }
  return m;
}
