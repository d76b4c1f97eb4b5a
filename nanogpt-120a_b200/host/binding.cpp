// CPython binding of the hot entry points: torch tensors in, one C-ABI call (or one short sequence of them) on the
// current stream, torch tensors out.
//
// Why it exists: at the sizes of a single projection the device work of a call is 5..30 us, and building ctypes
// arguments, filling ctypes structs and allocating each output from Python cost more than that (one quantize + GEMM of
// 16 tokens took 39 us of host time; through this module about 10).  The module holds no state: every buffer is a torch
// tensor, every operation is in libnvfp4_b200.so, and the GIL is released around the C calls as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>

#include "nvfp4_b200.h"

namespace {

PyObject* g_error = nullptr;  // the package's Nvfp4Error

struct Raised {};  // a Python exception is set

[[noreturn]] void raise(PyObject* type, const char* text) {
  PyErr_SetString(type, text);
  throw Raised{};
}

void check(int rc) {
  if (rc == 0) return;
  PyObject* e = PyObject_CallFunction(g_error, "is", rc, nvfp4_last_error());
  if (e) {
    PyErr_SetObject(g_error, e);
    Py_DECREF(e);
  }
  throw Raised{};
}

const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) raise(PyExc_TypeError, "expected a torch.Tensor");
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || !t.is_contiguous())
    raise(PyExc_AssertionError, "tensors crossing the C ABI must be contiguous CUDA tensors");
  return t;
}
template <typename T>
T* ptr(PyObject* o) {
  return o == Py_None ? nullptr : static_cast<T*>(tensor(o).data_ptr());
}
template <typename T>
T* ptr(const at::Tensor& t) {
  return static_cast<T*>(t.data_ptr());
}
uint32_t u32(PyObject* o) {
  const unsigned long v = PyLong_AsUnsignedLongMask(o);
  if (v == static_cast<unsigned long>(-1) && PyErr_Occurred()) throw Raised{};
  return static_cast<uint32_t>(v);
}
float f32(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw Raised{};
  return static_cast<float>(v);
}
bool flag(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw Raised{};
  return v != 0;
}
void* handle(PyObject* o) {
  void* p = PyLong_AsVoidPtr(o);
  if (!p && PyErr_Occurred()) throw Raised{};
  return p;
}

int dtype_code(const at::Tensor& t) {
  if (t.scalar_type() == at::kFloat) return NVFP4_DTYPE_F32;
  if (t.scalar_type() == at::kBFloat16) return NVFP4_DTYPE_BF16;
  raise(PyExc_TypeError, "unsupported dtype; the path takes float32 or bfloat16");
}
at::ScalarType scalar_of(int code) { return code == NVFP4_DTYPE_F32 ? at::kFloat : at::kBFloat16; }

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

struct NoGil {
  PyThreadState* s = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(s); }
};
// Runs without the GIL: `f` may use pointers and at::Tensors taken before, no PyObject.
template <typename F>
void call(F&& f) {
  int rc;
  {
    NoGil g;
    rc = f();
  }
  check(rc);
}

at::Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Device& dev) {
  return at::Tensor(at::detail::empty_cuda(size, type, dev, c10::nullopt));
}
at::Tensor bytes_of(int64_t n, const at::Device& dev) { return empty({n}, at::kByte, dev); }
at::Tensor floats(int64_t n, const at::Device& dev) { return empty({n}, at::kFloat, dev); }

struct Fp4 {
  at::Tensor bytes, scales, globals;
};
Fp4 new_fp4(int64_t rows, int64_t cols, bool packed, int64_t global_scales, const at::Device& dev) {
  return {bytes_of(rows * cols / 2, dev), bytes_of(packed ? (rows + 127) / 128 * (cols / 64) * 512 : rows * cols / 16, dev),
          floats(global_scales, dev)};
}

PyObject* wrap(at::Tensor t) {
  PyObject* o = THPVariable_Wrap(std::move(t));
  if (!o) throw Raised{};
  return o;
}
PyObject* tuple_of(std::initializer_list<PyObject*> items) {  // steals the references
  PyObject* t = PyTuple_New(static_cast<Py_ssize_t>(items.size()));
  Py_ssize_t i = 0;
  for (PyObject* o : items) PyTuple_SET_ITEM(t, i++, o);
  return t;
}
PyObject* none() { return Py_NewRef(Py_None); }

void matrix_shape(const at::Tensor& t, uint32_t& rows, uint32_t& cols) {
  if (t.dim() != 2) raise(PyExc_ValueError, "expected a matrix");
  rows = static_cast<uint32_t>(t.size(0)), cols = static_cast<uint32_t>(t.size(1));
}

// Four-six of a matrix into `q`.  amax null: rowwise takes it in the same pass, a tensor scale from a reduction before it.
void four_six(const at::Tensor& x, const float* amax, bool rowwise, bool packed, const Fp4& q, float* decoded_amax) {
  uint32_t rows, cols;
  matrix_shape(x, rows, cols);
  const int dtype = dtype_code(x), layout = packed ? NVFP4_SCALES_PACKED : NVFP4_SCALES_LOGICAL;
  void* const s = stream();
  uint8_t *b = ptr<uint8_t>(q.bytes), *sc = ptr<uint8_t>(q.scales);
  float* g = ptr<float>(q.globals);
  if (!amax && rowwise) {
    at::Tensor row_amax;
    if (cols > 4096) row_amax = floats(rows, x.device());
    call([&] {
      return nvfp4_quantize_four_six_rowwise_fused(s, x.data_ptr(), dtype, rows, cols, b, sc, layout, g,
                                                   row_amax.defined() ? ptr<float>(row_amax) : nullptr, decoded_amax);
    });
    return;
  }
  if (!amax) {
    const at::Tensor partials = floats(nvfp4_tensor_amax_partials(), x.device());
    call([&] {
      return nvfp4_quantize_four_six_tensor(s, x.data_ptr(), dtype, rows, cols, ptr<float>(partials), b, sc, layout, g);
    });
    return;
  }
  call([&] { return nvfp4_quantize_four_six(s, x.data_ptr(), dtype, amax, rowwise, rows, cols, b, sc, layout, g); });
}

// ---- functions: positional arguments only, checked by the Python callers ------------------------------------------

using Args = PyObject* const*;

// (x, amax | None, rowwise, packed, want_decoded_amax) -> (bytes, scales, global_scales, decoded_amax | None)
PyObject* quantize_new(Args a) {
  const at::Tensor& x = tensor(a[0]);
  const bool rowwise = flag(a[2]), packed = flag(a[3]);
  uint32_t rows, cols;
  matrix_shape(x, rows, cols);
  const Fp4 q = new_fp4(rows, cols, packed, rowwise ? rows : 1, x.device());
  at::Tensor decoded;
  if (flag(a[4])) decoded = floats(1, x.device());
  four_six(x, ptr<float>(a[1]), rowwise, packed, q, decoded.defined() ? ptr<float>(decoded) : nullptr);
  return tuple_of({wrap(q.bytes), wrap(q.scales), wrap(q.globals), decoded.defined() ? wrap(decoded) : none()});
}

// (x, amax | None, rowwise, packed, decoded_amax | None, bytes, scales, global_scales) -> None
PyObject* quantize_into(Args a) {
  const Fp4 q{tensor(a[5]), tensor(a[6]), tensor(a[7])};
  four_six(tensor(a[0]), ptr<float>(a[1]), flag(a[2]), flag(a[3]), q, ptr<float>(a[4]));
  return none();
}

// x f32 [rows, cols], row amax -> (bytes, logical scales, global_scales)
PyObject* four_six_rowwise_f32(Args a) {
  const at::Tensor& x = tensor(a[0]);
  const float* amax = ptr<float>(a[1]);
  uint32_t rows, cols;
  matrix_shape(x, rows, cols);
  const Fp4 q = new_fp4(rows, cols, false, rows, x.device());
  call([&] {
    return nvfp4_fp32_to_nvfp4_four_six_rowwise(stream(), ptr<float>(x), amax, ptr<uint8_t>(q.bytes),
                                                ptr<uint8_t>(q.scales), ptr<float>(q.globals),
                                                static_cast<uint32_t>(static_cast<uint64_t>(rows) * cols / 16), cols);
  });
  return tuple_of({wrap(q.bytes), wrap(q.scales), wrap(q.globals)});
}

// (x, out | None) -> row amax
PyObject* row_amax(Args a) {
  const at::Tensor& x = tensor(a[0]);
  uint32_t rows, cols;
  matrix_shape(x, rows, cols);
  const int dtype = dtype_code(x);
  const at::Tensor out = a[1] == Py_None ? floats(rows, x.device()) : tensor(a[1]);
  call([&] {
    return dtype == NVFP4_DTYPE_F32 ? nvfp4_row_amax_f32(stream(), ptr<float>(x), ptr<float>(out), rows, cols)
                                    : nvfp4_row_amax_bf16(stream(), x.data_ptr(), ptr<float>(out), rows, cols);
  });
  return wrap(out);
}

// (bytes, scales, global_scales, rows, cols, rowwise, transpose) -> f32 matrix
PyObject* decode(Args a) {
  const at::Tensor& b = tensor(a[0]);
  const uint32_t rows = u32(a[3]), cols = u32(a[4]);
  const bool rowwise = flag(a[5]), transpose = flag(a[6]);
  const int64_t r = transpose ? cols : rows, c = transpose ? rows : cols;
  const at::Tensor out = empty({r, c}, at::kFloat, b.device());
  const uint8_t* s = ptr<uint8_t>(a[1]);
  const float* g = ptr<float>(a[2]);
  call([&] {
    if (!transpose) return nvfp4_decode_f32(stream(), ptr<uint8_t>(b), s, g, rowwise, ptr<float>(out), rows, cols);
    return rowwise ? nvfp4_decode_rowwise_transpose_f32(stream(), ptr<uint8_t>(b), s, g, ptr<float>(out), rows, cols)
                   : nvfp4_decode_transpose_f32(stream(), ptr<uint8_t>(b), s, g, ptr<float>(out), rows, cols);
  });
  return wrap(out);
}

// (z, x, beta, packed) -> (bytes, scales, global_scale, amax)
PyObject* materialize(Args a) {
  const at::Tensor &z = tensor(a[0]), &x = tensor(a[1]);
  uint32_t rows, cols;
  matrix_shape(z, rows, cols);
  const float beta = f32(a[2]);
  const bool packed = flag(a[3]);
  const Fp4 q = new_fp4(rows, cols, packed, 1, z.device());
  const at::Tensor amax = floats(1, z.device()), partials = floats(nvfp4_tensor_amax_partials(), z.device());
  // With logical scales the 16-groups run over the flat tensor: its rows need not be whole groups.
  const uint64_t n = static_cast<uint64_t>(rows) * cols;
  if (!packed && cols % 16 != 0 && n <= UINT32_MAX) rows = 1, cols = static_cast<uint32_t>(n);
  call([&] {
    return nvfp4_materialize_schedule_free_partials(stream(), ptr<float>(z), ptr<float>(x), ptr<float>(partials), ptr<float>(amax),
                                                    ptr<uint8_t>(q.bytes), ptr<uint8_t>(q.scales),
                                                    packed ? NVFP4_SCALES_PACKED : NVFP4_SCALES_LOGICAL, ptr<float>(q.globals),
                                                    beta, rows, cols);
  });
  return tuple_of({wrap(q.bytes), wrap(q.scales), wrap(q.globals), wrap(amax)});
}

// (a_bytes, a_scales, a_global, b_bytes, b_scales, b_global, out, aux | None, bias | None, bias_fp4 (3 | None each),
//  m, n, k, ldo, mode, weight_global_scale, epilogue, relu2_row_amax | None) -> None
PyObject* gemm(Args a) {
  nvfp4_gemm_args g;
  std::memset(&g, 0, sizeof(g));
  g.a_bytes = ptr<uint8_t>(a[0]), g.a_scales = ptr<uint8_t>(a[1]), g.a_global = ptr<float>(a[2]);
  g.b_bytes = ptr<uint8_t>(a[3]), g.b_scales = ptr<uint8_t>(a[4]), g.b_global = ptr<float>(a[5]);
  const at::Tensor& out = tensor(a[6]);
  g.out = out.data_ptr(), g.aux = ptr<void>(a[7]), g.bias = ptr<float>(a[8]);
  g.bias_nvfp4_bytes = ptr<uint8_t>(a[9]), g.bias_nvfp4_scales = ptr<uint8_t>(a[10]), g.bias_nvfp4_global = ptr<float>(a[11]);
  g.m = u32(a[12]), g.n = u32(a[13]), g.k = u32(a[14]), g.ldo = u32(a[15]);
  g.global_scale_mode = static_cast<int>(u32(a[16]));
  g.weight_global_scale = f32(a[17]);
  g.epilogue = static_cast<int>(u32(a[18]));
  g.out_dtype = dtype_code(out);
  g.relu2_row_amax = ptr<float>(a[19]);
  call([&] { return nvfp4_gemm(stream(), &g); });
  return none();
}

// (x, rowwise, packed, w_bytes, w_scales, w_global, n, w_k, bias | None, epilogue, out_dtype, out | None) ->
// (y, x bytes, x scales, x global_scales).  The weight's scale plane is packed; x's too unless `packed` is false (a
// packed copy is then made for the GEMM).
PyObject* projection_forward(Args a) {
  const at::Tensor& x = tensor(a[0]);
  const bool rowwise = flag(a[1]), packed = flag(a[2]);
  uint32_t m, k;
  matrix_shape(x, m, k);
  nvfp4_gemm_args g;
  std::memset(&g, 0, sizeof(g));
  g.b_bytes = ptr<uint8_t>(a[3]), g.b_scales = ptr<uint8_t>(a[4]), g.b_global = ptr<float>(a[5]);
  g.m = m, g.n = u32(a[6]), g.k = k, g.ldo = g.n;
  if (u32(a[7]) != k) raise(PyExc_AssertionError, "A and B must share K");
  g.bias = ptr<float>(a[8]);
  g.epilogue = static_cast<int>(u32(a[9]));
  const at::Device dev = x.device();
  const Fp4 q = new_fp4(m, k, packed, rowwise ? m : 1, dev);
  const at::Tensor out = a[11] == Py_None ? empty({m, g.n}, scalar_of(static_cast<int>(u32(a[10]))), dev) : tensor(a[11]);
  four_six(x, nullptr, rowwise, packed, q, nullptr);
  at::Tensor packed_scales = q.scales;
  if (!packed) {
    packed_scales = bytes_of(static_cast<int64_t>(nvfp4_scale_packed_len(m, k)), dev);
    call([&] { return nvfp4_scale_pack(stream(), ptr<uint8_t>(q.scales), ptr<uint8_t>(packed_scales), m, k); });
  }
  g.a_bytes = ptr<uint8_t>(q.bytes), g.a_scales = ptr<uint8_t>(packed_scales), g.a_global = ptr<float>(q.globals);
  g.global_scale_mode = rowwise ? NVFP4_GS_ROWWISE_A : NVFP4_GS_TENSOR;
  g.weight_global_scale = 1.0f;
  g.out = out.data_ptr(), g.out_dtype = dtype_code(out);
  call([&] { return nvfp4_gemm(stream(), &g); });
  return tuple_of({wrap(out), wrap(q.bytes), wrap(q.scales), wrap(q.globals)});
}

// (entry, input bytes, scales, packed, globals, weight bytes, scales, packed, global, bias bytes | None, scales | None,
//  global | None, out | None, pre_activation | None, relu2_row_amax | None, tokens, in, out) -> None
PyObject* projection(Args a) {
  static int (*const entries[])(void*, const nvfp4_projection_args*) = {
      nvfp4_qkv_projection, nvfp4_c_proj,         nvfp4_mlp_up_relu2,      nvfp4_mlp_down_residual,
      nvfp4_lm_head_logits, nvfp4_lm_head_logits_tma, nvfp4_nextlat_projection};
  const uint32_t entry = u32(a[0]);
  if (entry >= sizeof(entries) / sizeof(entries[0])) raise(PyExc_ValueError, "unknown projection entry");
  nvfp4_projection_args p;
  std::memset(&p, 0, sizeof(p));
  const at::Tensor& in = tensor(a[1]);
  p.input_bytes = ptr<uint8_t>(in), p.input_scales = ptr<uint8_t>(a[2]);
  p.input_scale_layout = flag(a[3]) ? NVFP4_SCALES_PACKED : NVFP4_SCALES_LOGICAL;
  p.input_global_scales = ptr<float>(a[4]);
  p.weight_bytes = ptr<uint8_t>(a[5]), p.weight_scales = ptr<uint8_t>(a[6]);
  p.weight_scale_layout = flag(a[7]) ? NVFP4_SCALES_PACKED : NVFP4_SCALES_LOGICAL;
  p.weight_global_scale = ptr<float>(a[8]);
  p.bias_bytes = ptr<uint8_t>(a[9]), p.bias_scales = ptr<uint8_t>(a[10]), p.bias_global_scale = ptr<float>(a[11]);
  p.out = ptr<void>(a[12]), p.pre_activation = ptr<void>(a[13]), p.relu2_row_amax = ptr<float>(a[14]);
  p.out_dtype = dtype_code(tensor(a[12] != Py_None ? a[12] : a[13]));
  p.token_count = u32(a[15]), p.input_dim = u32(a[16]), p.output_dim = u32(a[17]);
  at::Tensor in_scratch, w_scratch;
  if (p.input_scale_layout == NVFP4_SCALES_LOGICAL) {
    in_scratch = bytes_of(static_cast<int64_t>(nvfp4_scale_packed_len(p.token_count, p.input_dim)), in.device());
    p.input_scales_packed_scratch = ptr<uint8_t>(in_scratch);
  }
  if (p.weight_scale_layout == NVFP4_SCALES_LOGICAL) {
    w_scratch = bytes_of(static_cast<int64_t>(nvfp4_scale_packed_len(p.output_dim, p.input_dim)), in.device());
    p.weight_scales_packed_scratch = ptr<uint8_t>(w_scratch);
  }
  call([&] { return entries[entry](stream(), &p); });
  return none();
}

nvfp4_ms_eden_operand operand(PyObject* dict) {
  auto get = [&](const char* key) {
    PyObject* o = PyDict_GetItemString(dict, key);
    if (!o) raise(PyExc_KeyError, key);
    return o;
  };
  nvfp4_ms_eden_operand r;
  r.bytes = ptr<uint8_t>(get("bytes")), r.scales_packed = ptr<uint8_t>(get("scales_packed"));
  r.global_scales = ptr<float>(get("global_scales")), r.global_scale = ptr<float>(get("global_scale"));
  r.chunk_amax = ptr<float>(get("chunk_amax"));
  return r;
}

// (prepare_weight_t_only, e, w bytes, w scales, w packed, w global, x bytes, x scales, x packed, x globals, e_h, e_t_h,
//  weight_t_h, input_t_h (dicts), dinput | None, dweight | None, dbias | None, want_dbias, grad_dtype, tokens, in, out,
//  sign_seed, scale_seed, precomputed_e_amax_chunks, token_offset, e_global_scale | None, x_decoded_amax | None,
//  side stream, fork event, join event (handles, 0 = none), total_token_count, weight_t_prepared)
// -> (dinput, dweight, dbias | None)
PyObject* linear_backward(Args a) {
  nvfp4_linear_backward_args b;
  std::memset(&b, 0, sizeof(b));
  const at::Tensor& e = tensor(a[1]);
  b.e = e.data_ptr(), b.e_dtype = dtype_code(e);
  b.w_bytes = ptr<uint8_t>(a[2]), b.w_scales = ptr<uint8_t>(a[3]);
  b.w_scale_layout = flag(a[4]) ? NVFP4_SCALES_PACKED : NVFP4_SCALES_LOGICAL;
  b.w_global = ptr<float>(a[5]);
  b.x_bytes = ptr<uint8_t>(a[6]), b.x_scales = ptr<uint8_t>(a[7]);
  b.x_scale_layout = flag(a[8]) ? NVFP4_SCALES_PACKED : NVFP4_SCALES_LOGICAL;
  b.x_globals = ptr<float>(a[9]);
  b.e_h = operand(a[10]), b.e_t_h = operand(a[11]), b.weight_t_h = operand(a[12]), b.input_t_h = operand(a[13]);
  const int64_t tokens = u32(a[19]), in_dim = u32(a[20]), out_dim = u32(a[21]);
  const at::ScalarType grad = scalar_of(static_cast<int>(u32(a[18])));
  const at::Device dev = e.device();
  const bool prepare_only = flag(a[0]);
  at::Tensor dinput, dweight, dbias;
  if (!prepare_only) {
    dinput = a[14] == Py_None ? empty({tokens, in_dim}, grad, dev) : tensor(a[14]);
    dweight = a[15] == Py_None ? empty({out_dim, in_dim}, grad, dev) : tensor(a[15]);
    if (flag(a[17])) dbias = a[16] == Py_None ? floats(out_dim, dev) : tensor(a[16]);
    b.dinput = dinput.data_ptr(), b.dinput_dtype = dtype_code(dinput);
    b.dweight = dweight.data_ptr(), b.dweight_dtype = dtype_code(dweight);
    b.dbias = dbias.defined() ? ptr<float>(dbias) : nullptr;
  }
  b.token_count = static_cast<uint32_t>(tokens), b.input_dim = static_cast<uint32_t>(in_dim), b.output_dim = static_cast<uint32_t>(out_dim);
  b.sign_seed = u32(a[22]), b.scale_seed = u32(a[23]), b.precomputed_e_amax_chunks = u32(a[24]), b.token_offset = u32(a[25]);
  b.e_global_scale_override = ptr<float>(a[26]), b.x_decoded_amax = ptr<float>(a[27]);
  b.side_stream = handle(a[28]), b.fork_event = handle(a[29]), b.join_event = handle(a[30]);
  b.total_token_count = u32(a[31]), b.weight_t_prepared = flag(a[32]);
  call([&] { return prepare_only ? nvfp4_linear_backward_prepare_weight_t(stream(), &b) : nvfp4_linear_backward_ms_eden(stream(), &b); });
  if (prepare_only) return none();
  return tuple_of({wrap(dinput), wrap(dweight), dbias.defined() ? wrap(dbias) : none()});
}

// ---- module -------------------------------------------------------------------------------------------------------

template <PyObject* (*kFn)(Args), Py_ssize_t kCount>
PyObject* entry(PyObject*, Args args, Py_ssize_t n) {
  if (n != kCount) {
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", kCount, n);
    return nullptr;
  }
  try {
    return kFn(args);
  } catch (const Raised&) {
  } catch (const c10::OutOfMemoryError& e) {
    PyObject* torch = PyImport_ImportModule("torch");
    PyObject* type = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
    PyErr_SetString(type ? type : PyExc_RuntimeError, e.what_without_backtrace());
    Py_XDECREF(type);
    Py_XDECREF(torch);
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

PyObject* set_error_type(PyObject*, PyObject* type) {
  Py_XSETREF(g_error, Py_NewRef(type));
  return none();
}

#define ENTRY(name, count) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&entry<name, count>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {ENTRY(quantize_new, 5),
                         ENTRY(quantize_into, 8),
                         ENTRY(four_six_rowwise_f32, 2),
                         ENTRY(row_amax, 2),
                         ENTRY(decode, 7),
                         ENTRY(materialize, 4),
                         ENTRY(gemm, 20),
                         ENTRY(projection_forward, 12),
                         ENTRY(projection, 18),
                         ENTRY(linear_backward, 33),
                         {"set_error_type", set_error_type, METH_O, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_nvfp4_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__nvfp4_binding(void) { return PyModule_Create(&module); }
