// Host path of a quantized linear layer: from the Python call to the kernel launches without Python in between.
//
// A decode step launched op by op is bound by the host: going through ctypes with some twenty converted arguments,
// attribute look-ups on the layer and tensor-method calls, one apply() took 26 us for an 8 us launch.  These functions
// read the layer's tensors straight from its dictionaries, check what the Python path checks, allocate the output and
// call the C ABI.  Whatever is not the plain case (tensors to convert or to lay out, wrong devices, errors to report)
// makes them return None: the Python path then does the call, conversions and error messages included.
#include <Python.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>

#include <map>
#include <mutex>
#include <utility>

#include "../../include/polar_b200.h"

namespace {

struct Api {
  decltype(&pe_init) init;
  decltype(&pe_gemv) gemv;
  decltype(&pe_gemv_tiled) gemv_tiled;
  decltype(&pe_gemv_scratch_bytes) gemv_bytes;
  decltype(&pe_gemm) gemm;
  decltype(&pe_gemm_workspace_bytes_splitk) gemm_bytes;
  decltype(&pe_moe_route) moe_route;
  decltype(&pe_moe_plan) moe_plan;
  decltype(&pe_moe_route_plan) moe_route_plan;
  decltype(&pe_moe_combine) moe_combine;
  decltype(&pe_gemv_grouped) grouped;
  decltype(&pe_gemv_grouped_workspace_bytes) grouped_bytes;
  decltype(&pe_gemm_grouped) gemm_grouped;
  decltype(&pe_gemm_grouped_silu_mul) gemm_silu_mul;
  decltype(&pe_gemm_grouped_workspace_bytes) gemm_grouped_bytes;
};
Api api;
bool ready = false;

constexpr int kDecodeRows = 16;  // rows up to which the decode-size kernels run

// ---- scratch ---------------------------------------------------------------------------------------------------
// One grow-only buffer per device, stream and use, shared by the calls on that stream in order.  While a graph is
// captured the buffer comes from the graph's own pool instead, so that it lives as long as the graph replays.  Buffers
// of streams no call has used for a while are given back.
struct Scratch { at::Tensor buf; uint64_t used; };
std::mutex scratch_lock;
std::map<std::pair<int, std::pair<void*, int>>, Scratch> scratch;
uint64_t scratch_clock = 0;
constexpr size_t kScratchBuffers = 64;

at::Tensor take_scratch(const at::Device& dev, cudaStream_t st, int use, size_t bytes, bool zeroed) {
  const auto opts = at::TensorOptions().device(dev).dtype(at::kByte);
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return at::empty({(int64_t)bytes}, opts);
  std::lock_guard<std::mutex> hold(scratch_lock);
  Scratch& s = scratch[{dev.index(), {st, use}}];
  s.used = ++scratch_clock;
  if (!s.buf.defined() || (size_t)s.buf.numel() < bytes) {
    const int64_t n = (int64_t)(bytes + bytes / 4);
    s.buf = zeroed ? at::zeros({n}, opts) : at::empty({n}, opts);  // zero: the status word, which only a time-out writes
  }
  at::Tensor out = s.buf;
  if (scratch.size() > kScratchBuffers) {
    auto old = scratch.begin();
    for (auto it = scratch.begin(); it != scratch.end(); ++it)
      if (it->second.used < old->second.used) old = it;
    scratch.erase(old);
  }
  return out;
}

// ---- small helpers ---------------------------------------------------------------------------------------------
int code_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return PE_F32;
    case at::kHalf: return PE_F16;
    case at::kBFloat16: return PE_BF16;
    default: return -1;
  }
}

const at::Tensor* tensor_or_null(PyObject* o) { return o && THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

bool device_ready(const at::Device& dev) {
  static bool seen[64] = {false};
  const int i = dev.index();
  if (i < 0 || i >= 64 || c10::cuda::current_device() != i) return false;
  if (!seen[i]) {
    if (api.init(i) != PE_OK) return false;
    seen[i] = true;
  }
  return true;
}

struct Matrix {  // a quantized weight
  const at::Tensor *codes, *norms, *ct, *tiles;
  bool packed;
  int out_f, in_f, in_f_padded;
};

bool plain(const Matrix& w, const at::Device& dev) {
  const at::Tensor &c = *w.codes, &n = *w.norms, &t = *w.ct;
  return c.device() == dev && n.device() == dev && t.device() == dev && c.dim() == 2 && c.element_size() == 1 && c.stride(1) == 1 &&
         n.scalar_type() == at::kHalf && n.dim() == 2 && n.size(0) == w.out_f && n.stride(1) == 1 && t.scalar_type() == at::kFloat &&
         t.is_contiguous() && (!w.tiles || w.tiles->device() == dev);
}

// x (rows, in_f or in_f_padded), last dimension contiguous; nullopt-like undefined tensor when not the plain case
at::Tensor multiply(const Matrix& w, const at::Tensor& x, int64_t rows, int64_t ld_x, int kind, at::ScalarType out, const at::Tensor* bias,
                    at::IntArrayRef shape) {
  const at::Device dev = x.device();
  const int xd = code_of(x.scalar_type()), yd = code_of(out);
  if (!dev.is_cuda() || xd < 0 || yd < 0 || rows < 1 || !plain(w, dev) || !device_ready(dev)) return {};
  if (bias && (bias->device() != dev || bias->scalar_type() != at::kHalf || !bias->is_contiguous())) return {};
  at::Tensor y = at::empty(shape, x.options().dtype(out).requires_grad(false));
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const void* b = bias ? bias->const_data_ptr() : nullptr;
  const int levels = (int)w.ct->numel();
  const float* ct = w.ct->const_data_ptr<float>();
  int rc;
  if (rows <= kDecodeRows) {
    const at::Tensor ws = take_scratch(dev, st, 0, api.gemv_bytes((int)rows, w.in_f_padded), true);
    rc = w.tiles ? api.gemv_tiled(w.tiles->const_data_ptr(), w.packed, ct, levels, x.const_data_ptr(), kind, xd, ld_x, w.in_f, y.mutable_data_ptr(),
                                  yd, w.out_f, b, (int)rows, w.out_f, w.in_f_padded, ws.mutable_data_ptr(), ws.numel(), st)
                 : api.gemv(w.codes->const_data_ptr(), w.packed, w.codes->stride(0), w.norms->const_data_ptr(), w.norms->stride(0), ct, levels,
                            x.const_data_ptr(), kind, xd, ld_x, w.in_f, y.mutable_data_ptr(), yd, w.out_f, b, (int)rows, w.out_f, w.in_f_padded,
                            ws.mutable_data_ptr(), ws.numel(), st);
  } else {
    const at::Tensor ws = take_scratch(dev, st, 1, api.gemm_bytes((int)rows, w.out_f, w.in_f_padded), false);
    rc = api.gemm(w.codes->const_data_ptr(), w.packed, w.codes->stride(0), w.norms->const_data_ptr(), w.norms->stride(0), ct, levels,
                  x.const_data_ptr(), kind, xd, ld_x, w.in_f, y.mutable_data_ptr(), yd, w.out_f, b, (int)rows, w.out_f, w.in_f_padded,
                  ws.mutable_data_ptr(), ws.numel(), st);
  }
  return rc == PE_OK ? y : at::Tensor();  // the Python path repeats a refused call and reports why
}

PyObject* wrap_or_none(at::Tensor y) {
  if (!y.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(y));
}

// ---- layer attributes ------------------------------------------------------------------------------------------
struct Names {
  PyObject *dict, *parameters, *buffers, *packed, *codes_packed, *codes, *norms, *ct_scaled, *in_f, *out_f, *in_f_padded;
};
Names names;

struct LayerDicts {
  PyObject *own, *parameters, *buffers;  // borrowed
  PyObject* find(PyObject* name) const {
    PyObject* v = PyDict_GetItem(own, name);
    if (!v && parameters) v = PyDict_GetItem(parameters, name);
    if (!v && buffers) v = PyDict_GetItem(buffers, name);
    return v;
  }
};

bool to_int(PyObject* o, int& out) {
  if (!o || !PyLong_Check(o)) return false;
  const long v = PyLong_AsLong(o);
  out = (int)v;
  return v > 0 && v < (1l << 30);
}

#define PE_GUARD_BEGIN try {
#define PE_GUARD_END                                     \
  }                                                      \
  catch (const std::exception& e) {                      \
    PyErr_SetString(PyExc_RuntimeError, e.what());       \
    return nullptr;                                      \
  }

// apply(layer, x, bias) -> fp16 output, or None
PyObject* host_apply(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) { PyErr_SetString(PyExc_TypeError, "apply takes 3 arguments"); return nullptr; }
  PE_GUARD_BEGIN
  if (!ready) Py_RETURN_NONE;
  PyObject** pd = _PyObject_GetDictPtr(args[0]);
  const at::Tensor* x = tensor_or_null(args[1]);
  if (!pd || !*pd || !x || !x->is_cuda() || x->dim() < 1 || !x->is_contiguous()) Py_RETURN_NONE;
  LayerDicts d = {*pd, PyDict_GetItem(*pd, names.parameters), PyDict_GetItem(*pd, names.buffers)};
  Matrix w = {};
  PyObject* packed = d.find(names.packed);
  w.packed = packed == Py_True;
  w.codes = tensor_or_null(d.find(w.packed ? names.codes_packed : names.codes));
  w.norms = tensor_or_null(d.find(names.norms));
  w.ct = tensor_or_null(d.find(names.ct_scaled));
  if (!w.codes || !w.norms || !w.ct || !to_int(d.find(names.in_f), w.in_f) || !to_int(d.find(names.out_f), w.out_f) ||
      !to_int(d.find(names.in_f_padded), w.in_f_padded) || x->size(-1) != w.in_f)
    Py_RETURN_NONE;
  const at::Tensor* bias = nullptr;
  if (args[2] != Py_None && !(bias = tensor_or_null(args[2]))) Py_RETURN_NONE;
  const int64_t rows = x->numel() / w.in_f;
  at::DimVector shape(x->sizes());
  shape.back() = w.out_f;
  return wrap_or_none(multiply(w, *x, rows, w.in_f, PE_X_RAW, at::kHalf, bias, shape));
  PE_GUARD_END
}

// matmul(codes, packed, norms, ct, x, rotated, out_f, in_f, in_f_padded, out_dtype, bias, tiles) -> output, or None
PyObject* host_matmul(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 12) { PyErr_SetString(PyExc_TypeError, "matmul takes 12 arguments"); return nullptr; }
  PE_GUARD_BEGIN
  if (!ready) Py_RETURN_NONE;
  Matrix w = {};
  w.codes = tensor_or_null(args[0]);
  w.packed = PyObject_IsTrue(args[1]) == 1;
  w.norms = tensor_or_null(args[2]);
  w.ct = tensor_or_null(args[3]);
  const at::Tensor* x = tensor_or_null(args[4]);
  if (!w.codes || !w.norms || !w.ct || !x || !to_int(args[6], w.out_f) || !to_int(args[7], w.in_f) || !to_int(args[8], w.in_f_padded)) Py_RETURN_NONE;
  // rotated, or not; or a PE_X_* number
  int kind = PE_X_RAW;
  if (PyBool_Check(args[5])) kind = args[5] == Py_True ? PE_X_ROTATED : PE_X_RAW;
  else if (!to_int(args[5], kind)) Py_RETURN_NONE;
  const int64_t width = kind == PE_X_ROTATED ? w.in_f_padded : kind == PE_X_SILU_MUL ? 2 * (int64_t)w.in_f : w.in_f;
  if (x->dim() != 2 || x->stride(1) != 1 || x->size(1) != width || !THPDtype_Check(args[9])) Py_RETURN_NONE;
  if (kind == PE_X_SILU_MUL && x->size(0) <= kDecodeRows) Py_RETURN_NONE;
  const at::Tensor* bias = nullptr;
  if (args[10] != Py_None && !(bias = tensor_or_null(args[10]))) Py_RETURN_NONE;
  if (args[11] != Py_None && !(w.tiles = tensor_or_null(args[11]))) Py_RETURN_NONE;
  const at::ScalarType out = reinterpret_cast<THPDtype*>(args[9])->scalar_type;
  return wrap_or_none(multiply(w, *x, x->size(0), x->stride(0), kind, out, bias, {x->size(0), w.out_f}));
  PE_GUARD_END
}

// One projection of every expert over the rows that the plan grouped.
struct Experts {
  const at::Tensor *codes, *norms, *ct;
  bool packed;
};
struct MoePlan {
  int64_t pairs, n_local, max_problems;
  int rows_per_problem, top_k;
  const int32_t *problems, *expert_rows, *pos;
  bool tensor_cores;
};

bool plain_experts(const Experts& w, const at::Device& dev, int64_t rows) {
  return w.codes && w.norms && w.ct && w.codes->device() == dev && w.norms->device() == dev && w.ct->device() == dev && w.codes->dim() == 3 &&
         w.codes->element_size() == 1 && w.codes->is_contiguous() && w.codes->size(1) == rows && w.norms->scalar_type() == at::kHalf &&
         w.norms->dim() == 3 && w.norms->stride(2) == 1 && w.ct->scalar_type() == at::kFloat && w.ct->is_contiguous();
}

int grouped(const Experts& w, const MoePlan& p, const at::Device& dev, cudaStream_t st, const void* x, int kind, int xd, int64_t ld_x, int in_f,
            int in_f_padded, const int32_t* x_rows, bool silu_mul, void* y, int yd, int out_f) {
  const float* ct = w.ct->const_data_ptr<float>();
  const int levels = (int)w.ct->numel();
  if (p.tensor_cores) {
    const at::Tensor ws = take_scratch(dev, st, 1, api.gemm_grouped_bytes((int)p.n_local, (int)p.pairs, out_f, in_f_padded), false);
    if (silu_mul)
      return api.gemm_silu_mul(w.codes->const_data_ptr(), w.packed, w.codes->stride(1), w.codes->stride(0), w.norms->const_data_ptr(),
                               w.norms->stride(1), w.norms->stride(0), ct, levels, x, kind, xd, ld_x, in_f, p.pos, (int)(p.pairs / p.top_k), p.top_k, y,
                               out_f / 2, p.expert_rows,
                               (int)p.n_local, (int)p.pairs, out_f, in_f_padded, ws.mutable_data_ptr(), ws.numel(), st);
    return api.gemm_grouped(w.codes->const_data_ptr(), w.packed, w.codes->stride(1), w.codes->stride(0), w.norms->const_data_ptr(),
                            w.norms->stride(1), w.norms->stride(0), ct, levels, x, kind, xd, ld_x, in_f, x_rows, y, yd, out_f, p.expert_rows,
                            (int)p.n_local, (int)p.pairs, out_f, in_f_padded, ws.mutable_data_ptr(), ws.numel(), st);
  }
  const at::Tensor ws = take_scratch(dev, st, 2, api.grouped_bytes((int)p.max_problems, out_f, in_f_padded), true);
  return api.grouped(w.codes->const_data_ptr(), w.packed, w.codes->stride(1), w.codes->stride(0), w.norms->const_data_ptr(), w.norms->stride(1),
                     w.norms->stride(0), ct, levels, x, kind, xd, ld_x, in_f, x_rows, y, yd, out_f, p.problems, (int)p.max_problems,
                     p.rows_per_problem, out_f, in_f_padded, ws.mutable_data_ptr(), ws.numel(), st);
}

// moe(x, a, b, renormalize, expert_map, (codes, norms, ct, packed) gate/up, (...) down, (hidden, inter, hidden_padded, inter_padded),
//     rows_per_problem, max_problems, tensor_cores) -> fp16 output, or None.  a, b: router logits and top_k, or top-k weights and ids.
PyObject* host_moe(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 11) { PyErr_SetString(PyExc_TypeError, "moe takes 11 arguments"); return nullptr; }
  PE_GUARD_BEGIN
  if (!ready) Py_RETURN_NONE;
  const at::Tensor *x = tensor_or_null(args[0]), *a = tensor_or_null(args[1]), *given = tensor_or_null(args[2]);
  if (!x || !a || !x->is_cuda() || x->dim() < 1 || !x->is_contiguous()) Py_RETURN_NONE;
  const at::Device dev = x->device();
  const at::Tensor* emap = nullptr;
  if (args[4] != Py_None) {
    emap = tensor_or_null(args[4]);
    if (!emap || emap->device() != dev || emap->scalar_type() != at::kLong || !emap->is_contiguous()) Py_RETURN_NONE;
  }
  Experts w[2];
  for (int i = 0; i < 2; ++i) {
    PyObject* t = args[5 + i];
    if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != 4) Py_RETURN_NONE;
    w[i] = {tensor_or_null(PyTuple_GET_ITEM(t, 0)), tensor_or_null(PyTuple_GET_ITEM(t, 1)), tensor_or_null(PyTuple_GET_ITEM(t, 2)),
            PyTuple_GET_ITEM(t, 3) == Py_True};
  }
  int dim[4], rpp, max_problems;
  if (!PyTuple_Check(args[7]) || PyTuple_GET_SIZE(args[7]) != 4) Py_RETURN_NONE;
  for (int i = 0; i < 4; ++i)
    if (!to_int(PyTuple_GET_ITEM(args[7], i), dim[i])) Py_RETURN_NONE;
  if (!to_int(args[8], rpp) || !to_int(args[9], max_problems)) Py_RETURN_NONE;
  const int h = dim[0], inter = dim[1], hp = dim[2], ip = dim[3];
  const int xd = code_of(x->scalar_type());
  if (xd < 0 || x->size(-1) != h || !plain_experts(w[0], dev, 2 * (int64_t)inter) || !plain_experts(w[1], dev, h) || !device_ready(dev)) Py_RETURN_NONE;
  const int64_t tokens = x->numel() / h;
  int top_k = 0;
  const int ad = code_of(a->scalar_type());
  if (given) {
    if (a->device() != dev || given->device() != dev || a->dim() != 2 || given->dim() != 2 || given->scalar_type() != at::kLong ||
        a->scalar_type() != at::kFloat || !a->is_contiguous() || !given->is_contiguous() || given->size(0) != tokens || a->sizes() != given->sizes())
      Py_RETURN_NONE;
    top_k = (int)given->size(1);
  } else if (!to_int(args[2], top_k) || ad < 0 || a->device() != dev || a->dim() != 2 || a->stride(1) != 1 || a->size(0) != tokens ||
             a->size(1) > 1024 || top_k > 32 || top_k > a->size(1)) {
    Py_RETURN_NONE;
  }
  if (tokens < 1) Py_RETURN_NONE;
  MoePlan p = {};
  p.pairs = tokens * top_k;
  p.n_local = w[0].codes->size(0);
  p.max_problems = max_problems;
  p.rows_per_problem = rpp;
  p.tensor_cores = args[10] == Py_True;
  if (p.tensor_cores && w[0].codes->stride(0) != w[0].codes->size(1) * w[0].codes->stride(1)) Py_RETURN_NONE;
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  // the bookkeeping in one buffer: problems, ids, expert rows, weights, tokens of the rows, rows of the pairs
  const auto bytes = x->options().dtype(at::kByte).requires_grad(false);
  const int64_t at_ids = 16 * p.max_problems, at_rows = at_ids + (given ? 0 : 8 * p.pairs), at_w = at_rows + 8 * p.n_local,
                at_tok = at_w + (given ? 0 : 4 * p.pairs), at_pos = at_tok + 4 * p.pairs;
  const at::Tensor book = at::empty({at_pos + 4 * p.pairs}, bytes);
  uint8_t* base = static_cast<uint8_t*>(book.mutable_data_ptr());
  int32_t* problems = reinterpret_cast<int32_t*>(base);
  int32_t *rows = reinterpret_cast<int32_t*>(base + at_rows), *tok = reinterpret_cast<int32_t*>(base + at_tok), *pos = reinterpret_cast<int32_t*>(base + at_pos);
  p.problems = problems;
  p.expert_rows = rows;
  p.pos = pos;
  p.top_k = top_k;
  const float* weights = given ? a->const_data_ptr<float>() : reinterpret_cast<float*>(base + at_w);
  const int64_t* ids = given ? given->const_data_ptr<int64_t>() : reinterpret_cast<int64_t*>(base + at_ids);
  int rc = PE_OK;
  const int64_t* map = emap ? emap->const_data_ptr<int64_t>() : nullptr;
  const int n_global = emap ? (int)emap->numel() : 0;
  float* w_out = reinterpret_cast<float*>(base + at_w);
  int64_t* ids_out = reinterpret_cast<int64_t*>(base + at_ids);
  if (!given && p.pairs <= 1024) {
    rc = api.moe_route_plan(a->const_data_ptr(), ad, a->stride(0), (int)tokens, (int)a->size(1), top_k, PyObject_IsTrue(args[3]) == 1, w_out, ids_out,
                            map, n_global, (int)p.n_local, rpp, max_problems, tok, pos, problems, rows, st);
  } else {
    if (!given)
      rc = api.moe_route(a->const_data_ptr(), ad, a->stride(0), (int)tokens, (int)a->size(1), top_k, PyObject_IsTrue(args[3]) == 1, w_out, ids_out, st);
    if (rc == PE_OK)
      rc = api.moe_plan(ids, map, n_global, (int)p.pairs, top_k, (int)p.n_local, rpp, max_problems, tok, pos, problems, rows, st);
  }
  const auto half = x->options().dtype(at::kHalf).requires_grad(false);
  // tensor cores: the activation function is inside the first launch; else it is computed where the second one's input is prepared
  const int64_t mid = p.tensor_cores ? inter : 2 * (int64_t)inter;
  const at::Tensor gu = at::empty({p.pairs, mid}, half);
  const at::Tensor d = at::empty({p.pairs, h}, half.dtype(at::kFloat));
  if (rc == PE_OK)
    rc = grouped(w[0], p, dev, st, x->const_data_ptr(), PE_X_RAW, xd, h, h, hp, tok, p.tensor_cores, gu.mutable_data_ptr(), PE_F16,
                 2 * inter);
  if (rc == PE_OK)
    rc = grouped(w[1], p, dev, st, gu.const_data_ptr(), p.tensor_cores ? PE_X_RAW : PE_X_SILU_MUL, PE_F16, mid, inter, ip, nullptr, false,
                 d.mutable_data_ptr(), PE_F32, h);
  at::Tensor out = at::empty(x->sizes(), half);
  if (rc == PE_OK)
    rc = api.moe_combine(d.const_data_ptr<float>(), h, pos, weights, (int)tokens, top_k, out.mutable_data_ptr(), PE_F16, h, h, st);
  return wrap_or_none(rc == PE_OK ? out : at::Tensor());
  PE_GUARD_END
}

// setup(library path): the C ABI comes from the library the Python side loaded
PyObject* host_setup(PyObject*, PyObject* arg) {
  const char* path = PyUnicode_AsUTF8(arg);
  if (!path) return nullptr;
  void* lib = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (!lib) { PyErr_SetString(PyExc_RuntimeError, dlerror()); return nullptr; }
#define PE_SYMBOL(member, name)                                                             \
  api.member = reinterpret_cast<decltype(api.member)>(dlsym(lib, #name));                   \
  if (!api.member) { PyErr_SetString(PyExc_RuntimeError, "missing symbol " #name); return nullptr; }
  PE_SYMBOL(init, pe_init)
  PE_SYMBOL(gemv, pe_gemv)
  PE_SYMBOL(gemv_tiled, pe_gemv_tiled)
  PE_SYMBOL(gemv_bytes, pe_gemv_scratch_bytes)
  PE_SYMBOL(gemm, pe_gemm)
  PE_SYMBOL(gemm_bytes, pe_gemm_workspace_bytes_splitk)
  PE_SYMBOL(moe_route, pe_moe_route)
  PE_SYMBOL(moe_plan, pe_moe_plan)
  PE_SYMBOL(moe_route_plan, pe_moe_route_plan)
  PE_SYMBOL(moe_combine, pe_moe_combine)
  PE_SYMBOL(grouped, pe_gemv_grouped)
  PE_SYMBOL(grouped_bytes, pe_gemv_grouped_workspace_bytes)
  PE_SYMBOL(gemm_grouped, pe_gemm_grouped)
  PE_SYMBOL(gemm_silu_mul, pe_gemm_grouped_silu_mul)
  PE_SYMBOL(gemm_grouped_bytes, pe_gemm_grouped_workspace_bytes)
  ready = true;
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"setup", host_setup, METH_O, "bind the C ABI of the library at a path"},
    {"apply", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(host_apply)), METH_FASTCALL, "quantized linear layer, or None"},
    {"matmul", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(host_matmul)), METH_FASTCALL, "quantized matmul, or None"},
    {"moe", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(host_moe)), METH_FASTCALL, "quantized expert layer, or None"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "native host path", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  names.parameters = PyUnicode_InternFromString("_parameters");
  names.buffers = PyUnicode_InternFromString("_buffers");
  names.packed = PyUnicode_InternFromString("packed");
  names.codes_packed = PyUnicode_InternFromString("codes_packed");
  names.codes = PyUnicode_InternFromString("codes");
  names.norms = PyUnicode_InternFromString("norms");
  names.ct_scaled = PyUnicode_InternFromString("ct_scaled");
  names.in_f = PyUnicode_InternFromString("in_f");
  names.out_f = PyUnicode_InternFromString("out_f");
  names.in_f_padded = PyUnicode_InternFromString("in_f_padded");
  return PyModule_Create(&module);
}
