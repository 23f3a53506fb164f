// Host side of the whole-call entries: Python arguments to one C-ABI call without going through Python objects.
//
// A short prompt costs the GPU 20 to 50 us, and a Python wrapper that fills a ctypes descriptor field by field took 55 us
// (zoo cells) to 214 us (the seven launches of a Mamba-2 layer, one wrapper each). Everything a call needs from its
// tensors -- type, extents, pointer, a dense fp32 copy where one is missing -- is read here from the at::Tensor itself,
// outputs and ONE block of scratch come from torch's caching allocator on the current stream, and the GIL is released
// while the kernels are launched. No state survives a call.
//
// Every function returns None when an argument is not in a form it handles (not a tensor, another device, a wrong
// shape): the caller then takes the Python wrappers, which know every conversion and every error. A status of the C ABI
// comes back as an int.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../../include/linquant_b200.h"

namespace {

struct NotPlain {};  // an argument this path does not handle

struct Call {
  std::vector<at::Tensor> keep;  // converted copies the launch reads
  at::Device dev{at::kCUDA, 0};

  static const at::Tensor& tensor(PyObject* o) {
    if (!THPVariable_Check(o)) throw NotPlain{};
    return THPVariable_Unpack(o);
  }
  const at::Tensor& hold(at::Tensor t) {
    keep.push_back(std::move(t));
    return keep.back();
  }
  // dense and on this device, converted to fp32 (and expanded to `shape`) where it is not
  const float* f32(PyObject* o, at::IntArrayRef shape = {}, bool check = false) {
    if (o == nullptr || o == Py_None) return nullptr;
    const at::Tensor& t = tensor(o);
    const bool shaped = shape.empty() || t.sizes() == shape;
    if (check && !shaped) throw NotPlain{};
    if (shaped && t.scalar_type() == at::kFloat && t.device() == dev && t.is_contiguous()) return t.const_data_ptr<float>();
    at::Tensor u = t.to(dev, at::kFloat);
    if (!shaped) u = u.expand(shape);
    return hold(u.contiguous()).const_data_ptr<float>();
  }
  // what f32 gave for `o`, moved to a 16-byte boundary where it is a view that starts elsewhere
  const float* aligned16(const float* p, PyObject* o) {
    if ((reinterpret_cast<uintptr_t>(p) & 15u) == 0) return p;
    return hold(tensor(o).clone(at::MemoryFormat::Contiguous)).const_data_ptr<float>();
  }
  // dense, as it is otherwise; must live on this device
  const at::Tensor& dense(PyObject* o) {
    const at::Tensor& t = tensor(o);
    if (t.device() != dev) throw NotPlain{};
    return t.is_contiguous() ? t : hold(t.contiguous());
  }
};

int act_code(at::ScalarType t) {
  if (t == at::kHalf) return LQ_F16;
  if (t == at::kBFloat16) return LQ_BF16;
  throw NotPlain{};
}
int out_code(at::ScalarType t) { return t == at::kFloat ? LQ_F32 : act_code(t); }

double number(PyObject* o) {
  if (PyFloat_CheckExact(o)) return PyFloat_AS_DOUBLE(o);
  if (!PyLong_CheckExact(o) && !PyFloat_Check(o)) throw NotPlain{};
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    throw NotPlain{};
  }
  return v;
}
int integer(PyObject* o) {
  if (!PyLong_CheckExact(o)) throw NotPlain{};
  const long v = PyLong_AsLong(o);
  if ((v == -1 && PyErr_Occurred()) || v < -(1L << 30) || v > (1L << 30)) {
    PyErr_Clear();
    throw NotPlain{};
  }
  return (int)v;
}

// The per-device status word lives as long as the process in linquant_b200._cabi; its address is looked up once.
int* status_word(at::Device dev) {
  static int* words[64];
  const int i = dev.index();
  if (i < 0 || i >= 64) throw NotPlain{};
  if (words[i] == nullptr) {  // under the GIL
    PyObject* mod = PyImport_ImportModule("linquant_b200._cabi");
    PyObject* t = mod ? PyObject_CallMethod(mod, "status_word", "i", i) : nullptr;
    Py_XDECREF(mod);
    if (t == nullptr) throw python_error();
    words[i] = THPVariable_Unpack(t).data_ptr<int>();
    Py_DECREF(t);
  }
  return words[i];
}

at::Tensor scratch(size_t bytes, at::Device dev) {
  return at::detail::empty_cuda({(int64_t)bytes + 256}, at::kByte, dev, std::nullopt);
}
uint8_t* aligned(const at::Tensor& t) { return (uint8_t*)(((uintptr_t)t.data_ptr() + 255) & ~uintptr_t(255)); }

struct NoGil {
  PyThreadState* s = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(s); }
};

PyObject* none() { Py_RETURN_NONE; }

// ------------------------------------------------------------------------------------------------ zoo cells
// zoo_fwd(cell, q, k, v, g, beta, scales, eta, sigma, tau, scale, chunk, want_state, unrot, bits, out_dtype, signs, dqk,
//         initial_state) -> (o, state or None) | status | None.   cell: 0 simple GLA, 1 GLA, 2 delta, 3 KDA
PyObject* zoo_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    if (n != 19) throw NotPlain{};
    const int cell = integer(a[0]);
    const bool diag = cell & 1, delta = cell & 2;
    Call c;
    const at::Tensor& q0 = Call::tensor(a[1]);
    if (!q0.is_cuda() || q0.dim() != 4 || !PyDict_CheckExact(a[6])) throw NotPlain{};
    c.dev = q0.device();
    c.keep.reserve(24);
    c10::cuda::CUDAGuard guard(c.dev);
    const at::Tensor &q = c.dense(a[1]), &k = c.dense(a[2]), &v = c.dense(a[3]);
    const int64_t B = q.size(0), T = q.size(1), H = q.size(2), K = q.size(3);
    if (v.dim() != 4 || k.sizes() != q.sizes() || k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) throw NotPlain{};
    const int64_t V = v.size(3);
    if (v.size(0) != B || v.size(1) != T || v.size(2) != H) throw NotPlain{};
    const int chunk = integer(a[11]), bits = integer(a[14]);
    if (B * T * H >= (int64_t(1) << 31) || chunk <= 0 || T % chunk != 0 || K > 128 || bits < 2 || bits > 8) throw NotPlain{};

    lq_zoo_problem p;
    std::memset(&p, 0, sizeof p);
    p.B = (int)B; p.T = (int)T; p.H = (int)H; p.K = (int)K; p.V = (int)V; p.chunk = chunk;
    p.act_dtype = act_code(q.scalar_type());
    p.decay = diag ? LQ_DECAY_DIAGONAL : a[4] == Py_None ? LQ_DECAY_NONE : LQ_DECAY_SCALAR;
    p.eta = (float)number(a[7]); p.sigma = (float)number(a[8]); p.tau = (float)number(a[9]);
    p.scale = (float)(a[10] == Py_None ? std::pow((double)K, -0.5) : number(a[10]));
    p.qmax = (float)((1 << (bits - 1)) - 1);
    p.q = q.const_data_ptr(); p.k = k.const_data_ptr(); p.v = v.const_data_ptr();
    if (a[4] != Py_None) p.g = diag ? c.aligned16(c.f32(a[4], {B, T, H, K}, true), a[4]) : c.f32(a[4], {B, T, H}, true);
    if (a[5] != Py_None) p.beta = c.f32(a[5], {B, T, H}, true);
    if (a[16] != Py_None) p.rot_signs = c.f32(a[16], {K}, true);
    if (a[17] != Py_None) p.dqk = c.f32(a[17], {H, K}, true);
    if (a[18] != Py_None) p.initial_state = c.f32(a[18], {B, H, K, V}, true);
    static PyObject* const key_q = PyUnicode_InternFromString("q"), *const key_k = PyUnicode_InternFromString("k"),
        *const key_kw = PyUnicode_InternFromString("kw"), *const key_vl = PyUnicode_InternFromString("vl"),
        *const key_vw = PyUnicode_InternFromString("vw"), *const key_state = PyUnicode_InternFromString("state"),
        *const key_w = PyUnicode_InternFromString("w"), *const key_el = PyUnicode_InternFromString("el"),
        *const key_ew = PyUnicode_InternFromString("ew");
    auto sc = [&](PyObject* key, at::IntArrayRef shape) { return c.f32(PyDict_GetItem(a[6], key), shape, true); };
    p.sq = sc(key_q, {H}); p.sk = sc(key_k, {H}); p.skw = sc(key_kw, {H, K}); p.sstate = sc(key_state, {H, V});
    if (delta) {
      p.sw = sc(key_w, {H}); p.sel = sc(key_el, {H, V}); p.sew = sc(key_ew, {H, V});
    } else {
      p.svl = sc(key_vl, {H, V}); p.svw = sc(key_vw, {H, V});
    }
    if (a[13] != Py_None) {  // the kernels want the fp16 matrix with the input index contiguous
      const at::Tensor& u = Call::tensor(a[13]);
      if (u.dim() != 2 || u.size(0) != V || u.size(1) != V) throw NotPlain{};
      p.unrot_t = c.hold(u.to(c.dev, at::kHalf).t().contiguous()).const_data_ptr();
    }
    const at::ScalarType ot = a[15] == Py_None ? v.scalar_type() : THPDtype_Check(a[15]) ? ((THPDtype*)a[15])->scalar_type : throw NotPlain{};
    p.out_dtype = out_code(ot);
    at::Tensor o = at::detail::empty_cuda(v.sizes(), ot, c.dev, std::nullopt), state;
    p.o = o.data_ptr();
    if (a[12] == Py_True) {
      state = at::detail::empty_cuda({B, H, K, V}, at::kFloat, c.dev, std::nullopt);
      p.final_state = state.data_ptr<float>();
    } else if (a[12] != Py_False) throw NotPlain{};
    p.status = status_word(c.dev);

    const size_t bytes = lq_zoo_workspace_bytes(&p, delta);
    const at::Tensor ws = scratch(bytes, c.dev);
    cudaStream_t st = c10::cuda::getCurrentCUDAStream(c.dev.index()).stream();
    int e;
    {
      NoGil ng;
      static int (*const fwd[4])(const lq_zoo_problem*, void*, size_t, lq_stream) = {lq_simple_gla_fwd, lq_gla_fwd, lq_delta_fwd, lq_kda_fwd};
      e = fwd[cell](&p, aligned(ws), bytes, st);
    }
    if (e != LQ_OK) return PyLong_FromLong(e);
    PyObject* r = PyTuple_New(2);
    PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(o));
    PyTuple_SET_ITEM(r, 1, state.defined() ? THPVariable_Wrap(state) : none());
    return r;
  } catch (const NotPlain&) {
    Py_RETURN_NONE;
  }
  END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------------------------------------ Mamba-2 SSD
// split_rotate(xBC, signs, nheads, ngroups, d_state, headdim, B_inv, C_inv) -> (x, q_B, q_C) | status | None
PyObject* split_rotate(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    if (n != 8) throw NotPlain{};
    Call c;
    const at::Tensor& x0 = Call::tensor(a[0]);
    if (!x0.is_cuda() || x0.dim() != 3) throw NotPlain{};
    c.dev = x0.device();
    c.keep.reserve(8);
    c10::cuda::CUDAGuard guard(c.dev);
    const at::Tensor& x = c.dense(a[0]);
    const int64_t H = integer(a[2]), G = integer(a[3]), N = integer(a[4]), P = integer(a[5]);
    const int64_t B = x.size(0), T = x.size(1), W = x.size(2), d_ssm = H * P;
    if (W != d_ssm + 2 * G * N || G <= 0 || B * T >= (int64_t(1) << 31)) throw NotPlain{};
    const int dt = act_code(x.scalar_type());
    const float* signs = a[1] == Py_None ? nullptr : c.f32(a[1], {G, N}, true);
    const float *ib = c.f32(a[6], {G}, true), *ic = c.f32(a[7], {G}, true);
    at::Tensor qB = at::detail::empty_cuda({B, T, G, N}, at::kChar, c.dev, std::nullopt);
    at::Tensor qC = at::detail::empty_cuda({B, T, G, N}, at::kChar, c.dev, std::nullopt);
    cudaStream_t st = c10::cuda::getCurrentCUDAStream(c.dev.index()).stream();
    int e;
    {
      NoGil ng;
      e = lq_ssd_split_rotate_quant(x.const_data_ptr(), dt, (int)B, (int)T, (int)d_ssm, (int)G, (int)N, signs, ib, ic, nullptr, nullptr,
                                    qB.data_ptr<int8_t>(), qC.data_ptr<int8_t>(), st);
    }
    if (e != LQ_OK) return PyLong_FromLong(e);
    PyObject* r = PyTuple_New(3);
    PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(x.as_strided({B, T, H, P}, {T * W, W, P, 1})));
    PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(qB));
    PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(qC));
    return r;
  } catch (const NotPlain&) {
    Py_RETURN_NONE;
  }
  END_HANDLE_TH_ERRORS
}

// hadamard(x, signs) -> y | status | None
PyObject* hadamard(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    if (n != 2) throw NotPlain{};
    Call c;
    const at::Tensor& x = Call::tensor(a[0]);
    if (!x.is_cuda() || x.dim() != 4) throw NotPlain{};
    c.dev = x.device();
    c10::cuda::CUDAGuard guard(c.dev);
    const int64_t B = x.size(0), T = x.size(1), H = x.size(2), D = x.size(3);
    if (x.stride(3) != 1 || x.stride(2) != D || x.stride(0) != T * x.stride(1) || D < 64 || B * T >= (int64_t(1) << 31)) throw NotPlain{};
    const int dt = act_code(x.scalar_type());
    const float* s = c.f32(a[1], {H, D}, true);
    at::Tensor y = at::detail::empty_cuda({B, T, H, D}, x.scalar_type(), c.dev, std::nullopt);
    cudaStream_t st = c10::cuda::getCurrentCUDAStream(c.dev.index()).stream();
    int e;
    {
      NoGil ng;
      e = lq_kronecker_hadamard(x.const_data_ptr(), y.data_ptr(), dt, (int)B, (int)T, (int)H, (int)D, x.stride(1), s, st);
    }
    return e != LQ_OK ? PyLong_FromLong(e) : THPVariable_Wrap(y);
  } catch (const NotPlain&) {
    Py_RETURN_NONE;
  }
  END_HANDLE_TH_ERRORS
}

// ssd_fwd(x, dt, dt_scale, A_log, A_log_scale, q_B, B_scale, q_C, C_scale, chunk, D, D_scale, dt_bias, dt_softplus, dt_min,
//         dt_max, state_scale, cb_scale, alpha_hp, bscale_g, keyside, x_scale_hp, b_fp, b_gate_scale)
//   -> out | status | None
PyObject* ssd_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    if (n != 24) throw NotPlain{};
    Call c;
    const at::Tensor& x0 = Call::tensor(a[0]);
    if (!x0.is_cuda() || x0.dim() != 4) throw NotPlain{};
    c.dev = x0.device();
    c.keep.reserve(24);
    c10::cuda::CUDAGuard guard(c.dev);
    const bool keyside = a[20] == Py_True;
    if (!keyside && a[20] != Py_False) throw NotPlain{};
    const at::Tensor& x = x0.stride(3) == 1 ? x0 : c.hold(x0.contiguous());
    const at::Tensor &qB = c.dense(a[5]), &qC = c.dense(a[7]);
    const int64_t B = x.size(0), L = x.size(1), H = x.size(2), P = x.size(3);
    if (qB.dim() != 4 || qB.sizes() != qC.sizes() || qB.scalar_type() != at::kChar || qC.scalar_type() != at::kChar) throw NotPlain{};
    const int64_t G = qB.size(2), N = qB.size(3), C = integer(a[9]);
    if (qB.size(0) != B || qB.size(1) != L || C <= 0 || L % C != 0 || B * L * H >= (int64_t(1) << 31)) throw NotPlain{};
    const int64_t NC = L / C;

    lq_ssd_problem p;
    std::memset(&p, 0, sizeof p);
    p.B = (int)B; p.L = (int)L; p.H = (int)H; p.P = (int)P; p.G = (int)G; p.N = (int)N; p.chunk = (int)C;
    p.x = x.const_data_ptr();
    p.x_dtype = act_code(x.scalar_type());
    p.x_stride_b = x.stride(0); p.x_stride_t = x.stride(1); p.x_stride_h = x.stride(2);
    p.dt_in = c.f32(a[1], {B, L, H}, true);
    p.A_log = c.f32(a[3], {H}, true);
    if (a[12] != Py_None) p.dt_bias = c.f32(a[12], {H}, true);
    auto scalar = [&](PyObject* o, float& host, const float*& on_dev) {
      if (!THPVariable_Check(o)) {
        host = (float)number(o);
        return;
      }
      const at::Tensor& t = THPVariable_Unpack(o);
      if (t.scalar_type() != at::kFloat || t.device() != c.dev || t.numel() < 1 || !t.is_contiguous()) throw NotPlain{};
      host = 1.0f;
      on_dev = t.const_data_ptr<float>();
    };
    scalar(a[2], p.dt_scale, p.dt_scale_dev);
    scalar(a[4], p.A_log_scale, p.A_log_scale_dev);
    p.dt_softplus = PyObject_IsTrue(a[13]) == 1;
    p.dt_min = (float)number(a[14]); p.dt_max = (float)number(a[15]);
    p.q_B = qB.const_data_ptr<int8_t>(); p.q_C = qC.const_data_ptr<int8_t>();
    p.B_scale = c.f32(a[6], {G}); p.C_scale = c.f32(a[8], {G});
    p.state_scale = c.f32(a[16], {H, P}); p.cb_scale = c.f32(a[17], {G}, true);
    if (keyside) {
      const at::Tensor& bf = Call::tensor(a[22]);
      if (bf.sizes() != qB.sizes() || bf.device() != c.dev) throw NotPlain{};
      p.b_fp = (bf.scalar_type() == x.scalar_type() && bf.is_contiguous() ? bf : c.hold(bf.to(x.scalar_type()).contiguous())).const_data_ptr();
      if (bf.scalar_type() != x.scalar_type()) throw NotPlain{};  // C.B^T takes b_fp in its own type: the per-op wrappers know how
      p.x_scale_hp = c.f32(a[21], {H, P});
      const at::Tensor& bg0 = Call::tensor(a[23]);
      if (bg0.dim() != 4 || bg0.device() != c.dev) throw NotPlain{};
      const int64_t full[4] = {B, NC, H, N};
      for (int i = 0; i < 4; ++i)
        if (bg0.size(i) != 1 && bg0.size(i) != full[i]) throw NotPlain{};
      const at::Tensor& bg = bg0.scalar_type() == at::kFloat ? bg0 : c.hold(bg0.to(at::kFloat));
      p.b_gate_scale = bg.const_data_ptr<float>();
      for (int i = 0; i < 4; ++i) p.bgs_stride[i] = bg.size(i) > 1 ? bg.stride(i) : 0;
    } else {
      p.alpha_hp = c.f32(a[18], {H, P});
      p.bscale_g = c.f32(a[19], {G}, true);
    }
    if (a[10] != Py_None) {
      const at::Tensor& D = Call::tensor(a[10]);
      if (D.device() != c.dev || !((D.dim() == 1 && D.size(0) == H) || (D.dim() == 2 && D.size(0) == H && D.size(1) == P))) throw NotPlain{};
      if (THPVariable_Check(a[11])) {
        p.D = c.hold((D.to(at::kFloat) * THPVariable_Unpack(a[11]).to(c.dev, at::kFloat)).contiguous()).const_data_ptr<float>();
      } else {
        const double s = number(a[11]);
        p.D = s == 1.0 ? c.f32(a[10]) : c.hold((D.to(at::kFloat) * s).contiguous()).const_data_ptr<float>();
      }
      p.D_has_hdim = D.dim() == 2;
    }
    if (const char* kern = std::getenv("LQ_SCAN_KERNEL"); kern != nullptr && *kern != 0) {  // as chunk_scan_v2 reads it
      if (std::strcmp(kern, "warp_mma") == 0) p.scan_kernel = 1;
      else if (std::strcmp(kern, "tcgen05") == 0) p.scan_kernel = N == 128 && C % 128 == 0 ? 2 : 0;
      else if (std::strcmp(kern, "auto") != 0) throw NotPlain{};
    }
    p.status = status_word(c.dev);

    at::Tensor out = at::detail::empty_cuda({B, L, H, P}, at::kHalf, c.dev, std::nullopt);
    p.out = out.data_ptr();
    const size_t bytes = lq_ssd_combined_workspace_bytes(&p);
    const at::Tensor ws = scratch(bytes, c.dev);
    cudaStream_t st = c10::cuda::getCurrentCUDAStream(c.dev.index()).stream();
    int e;
    {
      NoGil ng;
      e = lq_ssd_combined_fwd(&p, keyside, aligned(ws), bytes, st);
    }
    return e != LQ_OK ? PyLong_FromLong(e) : THPVariable_Wrap(out);
  } catch (const NotPlain&) {
    Py_RETURN_NONE;
  }
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"zoo_fwd", (PyCFunction)(void*)zoo_fwd, METH_FASTCALL, "one chunk call of a zoo cell"},
    {"split_rotate", (PyCFunction)(void*)split_rotate, METH_FASTCALL, "Mamba-2 prologue on xBC"},
    {"hadamard", (PyCFunction)(void*)hadamard, METH_FASTCALL, "Kronecker Hadamard rotation"},
    {"ssd_fwd", (PyCFunction)(void*)ssd_fwd, METH_FASTCALL, "Mamba-2 SSD combined forward"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  PyObject* m = PyModule_Create(&module);
  if (m != nullptr && PyModule_AddStringConstant(m, "built_for", LQ_BUILT_FOR) != 0) Py_CLEAR(m);
  return m;
}
