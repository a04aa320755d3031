// CPython binding of the calls that a program makes per request: argument checks, result and
// workspace allocation and the C ABI call in one native function.  A small layer or pooling node runs
// for two to five microseconds on the GPU; marshalling some twenty arguments through ctypes took twelve
// to sixteen on the host and set the pace.  glow_b200/ops.py holds the Python signatures; this module
// gets the addresses of the library's entry points from the binding table there (setup()).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/empty_like.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <vector>

#include "glow_b200.h"

namespace {

// ---- entry points, by address ----
#define GLOWB200_ENTRY_POINTS(X)                                                                                     \
  X(glowb200_last_error) X(glowb200_slws_workspace_bytes) X(glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum) \
  X(glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum_low_latency)                                         \
  X(glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum_batched_sized)                                       \
  X(glowb200_embedding_bag_byte_rowwise_offsets) X(glowb200_int_nbit_split_embedding_bags)                            \
  X(glowb200_i8_gemm_workspace_bytes) X(glowb200_dynamic_fc_workspace_bytes) X(glowb200_rowwise_quantized_fc_i8_i32)  \
  X(glowb200_fc_i8_i32) X(glowb200_matmul_i8) X(glowb200_dynamic_rowwise_quantized_fc) X(glowb200_dynamic_quantized_fc) \
  X(glowb200_conv2d_workspace_bytes) X(glowb200_channelwise_quantized_conv2d_i8_i32) \
  X(glowb200_channelwise_quantized_conv2d_pair_workspace_bytes) X(glowb200_channelwise_quantized_conv2d_pair_i8_i32) \
  X(glowb200_channelwise_quantized_conv2d_add_i8) X(glowb200_element_add_maxsplat_i8) \
  X(glowb200_element_quantize_i8) X(glowb200_element_dequantize_i8) X(glowb200_max_pool_i8) X(glowb200_avg_pool_i8)    \
  X(glowb200_quantize_transpose_i8) X(glowb200_pairwise_dot_interaction) X(glowb200_device_manager_run_function_io)
struct Entry {
#define X(name) decltype(&::name) name = nullptr;
  GLOWB200_ENTRY_POINTS(X)
#undef X
} fn;
PyObject *error_class = nullptr;   // GlowB200Error(code, message)
PyObject *ndarray = nullptr;       // numpy.ndarray
PyObject *explain = nullptr;       // ops._explain(name, object, dtypes): raises what is wrong with an argument

struct Raised {};  // a Python exception is set

// ---- arguments ----
using at::Tensor;
constexpr unsigned bit(at::ScalarType t) { return 1u << (int)t; }
constexpr unsigned U8 = bit(at::kByte), I8 = bit(at::kChar), I32 = bit(at::kInt), I64 = bit(at::kLong), F16 = bit(at::kHalf),
                   F32 = bit(at::kFloat);

[[noreturn]] void bad_argument(const char *name, PyObject *o, unsigned dtypes) {
  PyObject *r = PyObject_CallFunction(explain, "sOI", name, o, dtypes);
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_Format(PyExc_TypeError, "%s is not a suitable tensor", name);
  throw Raised{};
}

// a contiguous CUDA tensor of one of `dtypes`
const Tensor &cuda_tensor(PyObject *o, const char *name, unsigned dtypes) {
  if (!THPVariable_Check(o)) bad_argument(name, o, dtypes);
  const Tensor &t = THPVariable_Unpack(o);
  if (!t.is_cuda() || !t.is_contiguous() || (dtypes != 0 && !(dtypes >> (int)t.scalar_type() & 1))) bad_argument(name, o, dtypes);
  return t;
}
const Tensor &any_tensor(PyObject *o, const char *name) {
  if (!THPVariable_Check(o)) bad_argument(name, o, 0);
  return THPVariable_Unpack(o);
}
void *address(PyObject *o, const char *name) { return o == Py_None ? nullptr : any_tensor(o, name).data_ptr(); }
int64_t integer(PyObject *o) {
  int64_t v;
  if (PyLong_CheckExact(o)) {
    v = PyLong_AsLongLong(o);
  } else {  // bools, numpy integers, floats: what int() makes of them
    PyObject *i = PyNumber_Long(o);
    if (i == nullptr) throw Raised{};
    v = PyLong_AsLongLong(i);
    Py_DECREF(i);
  }
  if (v == -1 && PyErr_Occurred()) throw Raised{};
  return v;
}
float real(PyObject *o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw Raised{};
  return (float)v;
}
// the items of a list or tuple
template <int N>
struct Items {
  PyObject *seq;
  explicit Items(PyObject *o, const char *what) : seq(PySequence_Fast(o, what)) {
    if (seq == nullptr) throw Raised{};
    if (PySequence_Fast_GET_SIZE(seq) != N) {
      PyErr_Format(PyExc_ValueError, "%s: %d items expected, got %zd", what, N, PySequence_Fast_GET_SIZE(seq));
      Py_DECREF(seq);
      throw Raised{};
    }
  }
  Items(const Items &) = delete;
  ~Items() { Py_DECREF(seq); }
  PyObject *operator[](int i) const { return PySequence_Fast_GET_ITEM(seq, i); }
};
template <int N>
struct Ints {
  int64_t v[N];
  Ints(PyObject *o, const char *what) {
    Items<N> items(o, what);
    for (int i = 0; i < N; i++) v[i] = integer(items[i]);
  }
};

Tensor empty(c10::IntArrayRef sizes, at::ScalarType t, const Tensor &like) {
  return Tensor(at::detail::empty_cuda(sizes, t, like.device(), std::nullopt));
}
// the caller's workspace, or `need` bytes of the caching allocator's
struct Workspace {
  Tensor t;
  Workspace(PyObject *o, size_t need, const Tensor &like)
      : t(o == Py_None ? empty({(int64_t)std::max<size_t>(need, 8)}, at::kByte, like) : cuda_tensor(o, "workspace", 0)) {}
  void *data() const { return t.data_ptr(); }
  size_t bytes() const { return (size_t)t.numel(); }
};
glowb200_stream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

void check(int rc) {
  if (rc == 0) return;
  PyObject *e = PyObject_CallFunction(error_class, "is", rc, fn.glowb200_last_error());
  if (e != nullptr) {
    PyErr_SetObject(error_class, e);
    Py_DECREF(e);
  }
  throw Raised{};
}

// The call itself, other Python threads running meanwhile (a launch may wait for room in its queue).
template <typename... P, typename... A>
void invoke(int (*f)(P...), A... args) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f(static_cast<P>(args)...);
  Py_END_ALLOW_THREADS
  check(rc);
}

PyObject *give(const Tensor &t) { return THPVariable_Wrap(t); }
PyObject *same(PyObject *o) {
  Py_INCREF(o);
  return o;
}

// Every function takes its arguments by position (ops.py fills in defaults) and may throw.
typedef PyObject *(*Body)(PyObject *const *a);
template <Body body, int N>
PyObject *guarded(PyObject *, PyObject *const *a, Py_ssize_t n) {
  if (n != N) {
    PyErr_Format(PyExc_TypeError, "%d arguments expected, got %zd", N, n);
    return nullptr;
  }
  try {
    return body(a);
  } catch (const Raised &) {
    return nullptr;
  } catch (const std::exception &e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

int64_t out_columns(int64_t in_line, int kind) {
  const int64_t payload = in_line - ((kind & 1) ? 4 : 8);
  return kind >= 2 ? payload * 2 : payload;
}

// ---- gather-pool ----
// data, weights, indices, lengths, kind, fp16 accumulation, out, status, workspace, num_indices, out_line, low latency
PyObject *slws(PyObject *const *a) {
  const Tensor &data = cuda_tensor(a[0], "data", U8), &indices = cuda_tensor(a[2], "indices", I32 | I64),
               &lengths = cuda_tensor(a[3], "lengths", I32);
  const int kind = (int)integer(a[4]);
  const int64_t rows = data.size(0), in_line = data.size(1), segments = lengths.size(0);
  const int64_t out_line = a[10] == Py_None ? out_columns(in_line, kind) : integer(a[10]);
  const bool given = a[6] != Py_None;
  const at::ScalarType dt = given ? any_tensor(a[6], "out").scalar_type() : (kind & 1) ? at::kHalf : at::kFloat;
  const Tensor &weights = cuda_tensor(a[1], "weights", bit(dt));
  const bool acc16 = PyObject_IsTrue(a[5]) == 1, low_latency = PyObject_IsTrue(a[11]) == 1;
  if (low_latency && acc16) {
    PyErr_SetString(PyExc_ValueError, "the low-latency form accumulates in fp32");
    throw Raised{};
  }
  const Tensor out = given ? any_tensor(a[6], "out") : empty({segments, out_line}, dt, data);
  const int64_t n = a[9] == Py_None ? indices.size(0) : integer(a[9]);
  const Workspace ws(a[8], fn.glowb200_slws_workspace_bytes(segments, 1), data);
  const int idx64 = indices.scalar_type() == at::kLong, out16 = dt == at::kHalf;
  int32_t *status = (int32_t *)address(a[7], "status");
  if (low_latency)
    invoke(fn.glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum_low_latency, out.data_ptr(), data.data_ptr(), kind,
        rows, weights.data_ptr(), indices.data_ptr(), idx64,
        (const int32_t *)lengths.data_ptr(), segments, n, in_line, out_line, out16, ws.data(), ws.bytes(), status, stream());
  else
    invoke(fn.glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum, out.data_ptr(), data.data_ptr(), kind, rows,
        weights.data_ptr(), indices.data_ptr(), idx64,
        (const int32_t *)lengths.data_ptr(), segments, n, in_line, out_line, out16, acc16, ws.data(), ws.bytes(), status,
        stream());
  return given ? same(a[6]) : give(out);
}

// data, weights, indices, offsets, kind, has end offset, fp16 accumulation, out, status, workspace, num_indices
PyObject *embedding_bag(PyObject *const *a) {
  const Tensor &data = cuda_tensor(a[0], "data", U8), &indices = cuda_tensor(a[2], "indices", I32 | I64),
               &offsets = cuda_tensor(a[3], "offsets", bit(indices.scalar_type()));
  const int kind = (int)integer(a[4]);
  const int64_t rows = data.size(0), in_line = data.size(1), out_line = out_columns(in_line, kind), num_offsets = offsets.size(0);
  const bool given = a[7] != Py_None, end = PyObject_IsTrue(a[5]) == 1;
  const at::ScalarType dt = given ? any_tensor(a[7], "out").scalar_type() : (kind & 1) ? at::kHalf : at::kFloat;
  const Tensor &weights = cuda_tensor(a[1], "weights", bit(dt));
  const int64_t segments = std::max<int64_t>(end ? num_offsets - 1 : num_offsets, 0);
  const Tensor out = given ? any_tensor(a[7], "out") : empty({segments, out_line}, dt, data);
  const int64_t n = a[10] == Py_None ? indices.size(0) : integer(a[10]);
  const Workspace ws(a[9], fn.glowb200_slws_workspace_bytes(segments, 1), data);
  invoke(fn.glowb200_embedding_bag_byte_rowwise_offsets, out.data_ptr(), data.data_ptr(), kind, rows, weights.data_ptr(),
      indices.data_ptr(), offsets.data_ptr(),
      indices.scalar_type() == at::kLong, num_offsets, n, in_line, out_line, end, dt == at::kHalf, PyObject_IsTrue(a[6]) == 1,
          ws.data(),
      ws.bytes(), (int32_t *)address(a[8], "status"), stream());
  return given ? same(a[7]) : give(out);
}

// jobs, count, max_segments, kind, int64 indices, in_line, out_line, fp16 result, fp16 accumulation, workspace, status,
// indices of all jobs
PyObject *slws_batched(PyObject *const *a) {
  const Tensor &ws = any_tensor(a[9], "workspace");
  invoke(fn.glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum_batched_sized, (const glowb200_slws_job *)address(a[0],
      "jobs"), integer(a[1]), integer(a[2]), (int)integer(a[3]), (int)integer(a[4]),
      integer(a[5]), integer(a[6]), (int)integer(a[7]), (int)integer(a[8]), integer(a[11]), ws.data_ptr(), (size_t)ws.numel(),
      (int32_t *)address(a[10], "status"), stream());
  Py_RETURN_NONE;
}

// dev weights, uvm weights, placements, offsets of the tables, types, dim offsets, total dims, indices,
// offsets, pooling mode, indice weights, fp16 result, fp32 scales, row alignment, out, status
PyObject *split_bags(PyObject *const *a) {
  const Tensor &dev = cuda_tensor(a[0], "dev_weights", U8), &uvm = cuda_tensor(a[1], "uvm_weights", U8),
               &placements = cuda_tensor(a[2], "weights_placements", I32), &at_ = cuda_tensor(a[3], "weights_offsets", I32 | I64),
               &tys = cuda_tensor(a[4], "weights_tys", U8), &dims = cuda_tensor(a[5], "dim_offsets", I32),
               &indices = cuda_tensor(a[7], "indices", I32 | I64), &offsets = cuda_tensor(a[8], "offsets",
                   bit(indices.scalar_type()));
  int iw16 = 0;
  if (a[10] != Py_None) iw16 = cuda_tensor(a[10], "indice_weights", F32 | F16).scalar_type() == at::kHalf;
  const int64_t T = dims.size(0) - 1, total = integer(a[6]);
  if (T < 0 || tys.size(0) != T || placements.size(0) != T || at_.size(0) != T) {
    PyErr_SetString(PyExc_ValueError, "table description arrays disagree on the number of tables");
    throw Raised{};
  }
  if (T == 0 || (offsets.size(0) - 1) % T != 0) {
    PyErr_SetString(PyExc_ValueError, "offsets must hold num_tables * bags_per_table + 1 entries");
    throw Raised{};
  }
  const int64_t B = (offsets.size(0) - 1) / T;
  const bool given = a[14] != Py_None;
  const Tensor out = given ? cuda_tensor(a[14], "out", F32 | F16) : empty({B, total},
      PyObject_IsTrue(a[11]) == 1 ? at::kHalf : at::kFloat, indices);
  invoke(fn.glowb200_int_nbit_split_embedding_bags, out.data_ptr(), dev.data_ptr(), dev.numel(), uvm.data_ptr(), uvm.numel(),
      (const int32_t *)placements.data_ptr(), at_.data_ptr(),
      at_.scalar_type() == at::kLong, (const uint8_t *)tys.data_ptr(), (const int32_t *)dims.data_ptr(), T, total,
          indices.data_ptr(),
      offsets.data_ptr(), indices.scalar_type() == at::kLong, indices.size(0), B, (int)integer(a[9]), address(a[10],
          "indice_weights"), iw16,
      out.scalar_type() == at::kHalf, PyObject_IsTrue(a[12]) == 1, (int)integer(a[13]), (int32_t *)address(a[15], "status"),
          stream());
  return given ? same(a[14]) : give(out);
}

// ---- int8 dense layers ----
struct Triples {
  const int32_t *p[3];
  Triples(PyObject *o, bool checked) {
    Items<3> items(o, "requantisation parameters");
    for (int i = 0; i < 3; i++)
      p[i] = (const int32_t *)(checked ? cuda_tensor(items[i], "per-row parameter", I32) : any_tensor(items[i],
          "parameter")).data_ptr();
  }
};

// inp, weights, bias, weight offsets, bias triples, out triples, out offset, in offset, bias offset,
// weight row sums, flags, out, workspace, status
PyObject *rowwise_fc(PyObject *const *a) {
  const Tensor &x = cuda_tensor(a[0], "inp", I8), &w = cuda_tensor(a[1], "weights", I8), &bias = cuda_tensor(a[2], "bias",
      I32 | I8),
               &offs = cuda_tensor(a[3], "per-row parameter", I32);
  const Triples bt(a[4], true), ot(a[5], true);
  const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
  int flags = (int)integer(a[10]);
  if (bias.scalar_type() == at::kChar) flags |= GLOWB200_FC_BIAS_INT8;  // the reference's _i8_i8 form
  const bool given = a[11] != Py_None;
  const Tensor out = given ? any_tensor(a[11], "out") : empty({M, N}, at::kChar, x);
  const Workspace ws(a[12], fn.glowb200_i8_gemm_workspace_bytes(M, K, N), x);
  invoke(fn.glowb200_rowwise_quantized_fc_i8_i32, (int8_t *)out.data_ptr(), (const int8_t *)x.data_ptr(),
      (const int8_t *)w.data_ptr(), (const int32_t *)bias.data_ptr(),
      (const int32_t *)offs.data_ptr(), bt.p[0], bt.p[1], bt.p[2], ot.p[0], ot.p[1], ot.p[2], M, K, N, (int32_t)integer(a[6]),
      (int32_t)integer(a[7]), (int32_t)integer(a[8]), (const int32_t *)address(a[9], "weights_row_sums"), flags, ws.data(),
          ws.bytes(),
      (int32_t *)address(a[13], "status"), stream());
  return given ? same(a[11]) : give(out);
}

// inp, weights, bias, out offset, in offset, weights offset, bias offset, bias triple, out triple,
// weights transposed, flags, out, workspace, status
PyObject *fc_i8(PyObject *const *a) {
  const Tensor &x = any_tensor(a[0], "inp"), &bias = any_tensor(a[2], "bias");
  const int64_t M = x.size(0), K = x.size(1);
  const int64_t N = a[1] != Py_None ? any_tensor(a[1], "weights").size(1) : any_tensor(a[9], "weights_transposed").size(0);
  int flags = (int)integer(a[10]);
  if (bias.scalar_type() == at::kChar) flags |= GLOWB200_FC_BIAS_INT8;
  const Ints<3> bt(a[7], "bias_triple"), ot(a[8], "out_triple");
  const bool given = a[11] != Py_None;
  const Tensor out = given ? any_tensor(a[11], "out") : empty({M, N}, at::kChar, x);
  const Workspace ws(a[12], fn.glowb200_i8_gemm_workspace_bytes(M, K, N), x);
  invoke(fn.glowb200_fc_i8_i32, (int8_t *)out.data_ptr(), (const int8_t *)x.data_ptr(), (const int8_t *)address(a[1],
      "weights"), (const int32_t *)bias.data_ptr(), M,
      K, N, (int32_t)integer(a[3]), (int32_t)integer(a[4]), (int32_t)integer(a[5]), (int32_t)integer(a[6]), (int32_t)bt.v[0],
      (int32_t)bt.v[1], (int32_t)bt.v[2], (int32_t)ot.v[0], (int32_t)ot.v[1], (int32_t)ot.v[2],
      (const int8_t *)address(a[9], "weights_transposed"), flags, ws.data(), ws.bytes(), (int32_t *)address(a[13], "status"),
          stream());
  return given ? same(a[11]) : give(out);
}

// lhs, rhs, out offset, lhs offset, rhs offset, out triple, flags, out, workspace, status
PyObject *matmul(PyObject *const *a) {
  const Tensor &x = any_tensor(a[0], "lhs"), &w = any_tensor(a[1], "rhs");
  const int64_t M = x.size(0), K = x.size(1), N = w.size(1);
  const Ints<3> ot(a[5], "out_triple");
  const bool given = a[7] != Py_None;
  const Tensor out = given ? any_tensor(a[7], "out") : empty({M, N}, at::kChar, x);
  const Workspace ws(a[8], fn.glowb200_i8_gemm_workspace_bytes(M, K, N), x);
  invoke(fn.glowb200_matmul_i8, (int8_t *)out.data_ptr(), (const int8_t *)x.data_ptr(), (const int8_t *)w.data_ptr(), M, K, N,
                              (int32_t)integer(a[2]), (int32_t)integer(a[3]), (int32_t)integer(a[4]), (int32_t)ot.v[0],
                              (int32_t)ot.v[1], (int32_t)ot.v[2], (int)integer(a[6]), ws.data(), ws.bytes(),
                              (int32_t *)address(a[9], "status"), stream());
  return given ? same(a[7]) : give(out);
}

// inp, weights, bias, scales, offsets (tensors, or a float and an integer for the whole of the weights),
// weights transposed, flags, out, workspace, status
template <bool ROWWISE>
PyObject *dynamic_fc(PyObject *const *a) {
  const Tensor &x = cuda_tensor(a[0], "inp", F16), &bias = any_tensor(a[2], "bias");
  const int64_t M = x.size(0), K = x.size(1), N = bias.size(0);
  const bool given = a[7] != Py_None;
  const Tensor out = given ? any_tensor(a[7], "out") : empty({M, N}, at::kHalf, x);
  const Workspace ws(a[8], fn.glowb200_dynamic_fc_workspace_bytes(M, K, N), x);
  const int8_t *w = (const int8_t *)address(a[1], "weights"), *wt = (const int8_t *)address(a[5], "weights_transposed");
  const int flags = (int)integer(a[6]);
  int32_t *status = (int32_t *)address(a[9], "status");
  if constexpr (ROWWISE)
    invoke(fn.glowb200_dynamic_rowwise_quantized_fc, out.data_ptr(), x.data_ptr(), w, (const float *)bias.data_ptr(),
                                                   (const float *)address(a[3], "scales"), (const int32_t *)address(a[4],
                                                       "offsets"), M, K,
                                                   N, wt, flags, ws.data(), ws.bytes(), status, stream());
  else
    invoke(fn.glowb200_dynamic_quantized_fc, out.data_ptr(), x.data_ptr(), w, (const float *)bias.data_ptr(), real(a[3]),
                                           (int32_t)integer(a[4]), M, K, N, wt, flags, ws.data(), ws.bytes(), status, stream());
  return given ? same(a[7]) : give(out);
}

// ---- convolution and glue ----
int64_t conv_out(int64_t in, int64_t k, int64_t s, int64_t pads, int64_t d) {
  const int64_t span = in + pads - ((k - 1) * d + 1);
  return (span >= 0 ? span / s : -((-span + s - 1) / s)) + 1;  // floor division, as Python's
}

// inp, filt, bias, kernels, strides, pads, group, dilation, out offset, in offset, filter offsets, bias
// offsets, bias triples, out triples, activation, its arguments, filter row sums, flags, out, workspace, status
// [, residual, dest offset, lhs offset, residual offset, lhs triple, residual triple, splat]
template <bool ADD>
PyObject *channelwise_conv(PyObject *const *a) {
  const Tensor &x = cuda_tensor(a[0], "inp", I8), &f = cuda_tensor(a[1], "filt", I8);
  const Ints<2> k(a[3], "kernels"), s(a[4], "strides"), d(a[7], "dilation");
  const Ints<4> p(a[5], "pads");
  const int64_t group = integer(a[6]);
  const int64_t in[4] = {x.size(0), x.size(1), x.size(2), x.size(3)}, fd[4] = {f.size(0), f.size(1), f.size(2), f.size(3)};
  const int64_t od[4] = {in[0], conv_out(in[1], k.v[0], s.v[0], p.v[0] + p.v[2], d.v[0]),
                         conv_out(in[2], k.v[1], s.v[1], p.v[1] + p.v[3], d.v[1]), fd[0]};
  const bool given = a[18] != Py_None;
  const Tensor out = given ? any_tensor(a[18], "out") : empty({od[0], od[1], od[2], od[3]}, at::kChar, x);
  const Workspace ws(a[19], a[19] == Py_None ? fn.glowb200_conv2d_workspace_bytes(od, in, fd, k.v, s.v, p.v, group, d.v) : 0, x);
  const Triples bt(a[12], false), ot(a[13], false);
  int32_t act[3] = {0, 0, 0};
  const bool has_args = a[15] != Py_None;
  if (has_args) {
    PyObject *seq = PySequence_Fast(a[15], "act_args");
    if (seq == nullptr) throw Raised{};
    for (Py_ssize_t i = 0; i < std::min<Py_ssize_t>(3, PySequence_Fast_GET_SIZE(seq)); i++) {
      const int64_t v = PyLong_AsLongLong(PySequence_Fast_GET_ITEM(seq, i));
      act[i] = (int32_t)v;
    }
    Py_DECREF(seq);
    if (PyErr_Occurred()) throw Raised{};
  }
  auto with = [&](auto function, auto... add) {
    invoke(function, (int8_t *)out.data_ptr(), (const int8_t *)x.data_ptr(), (const int8_t *)f.data_ptr(),
           (const int32_t *)address(a[2], "bias"), od, in, fd, k.v, s.v, p.v, group, d.v, (int32_t)integer(a[8]),
           (int32_t)integer(a[9]), (const int32_t *)address(a[10], "filter_offsets"), (const int32_t *)address(a[11], "bias_offsets"),
           bt.p[0], bt.p[1], bt.p[2], ot.p[0], ot.p[1], ot.p[2], (int32_t)integer(a[14]), has_args ? act : nullptr,
           (const int32_t *)address(a[16], "filter_row_sums"), (int)integer(a[17]), ws.data(), ws.bytes(),
           (int32_t *)address(a[20], "status"), add..., stream());
  };
  if constexpr (ADD) {
    const Ints<3> lt(a[25], "lhs_triple"), rt(a[26], "residual_triple");
    with(fn.glowb200_channelwise_quantized_conv2d_add_i8, (const int8_t *)cuda_tensor(a[21], "residual", I8).data_ptr(),
         (int32_t)integer(a[22]), (int32_t)integer(a[23]), (int32_t)integer(a[24]), (int32_t)lt.v[0], (int32_t)lt.v[1],
         (int32_t)lt.v[2], (int32_t)rt.v[0], (int32_t)rt.v[1], (int32_t)rt.v[2], (int32_t)integer(a[27]));
  } else {
    with(fn.glowb200_channelwise_quantized_conv2d_i8_i32);
  }
  return given ? same(a[18]) : give(out);
}

// A layer of a pair: filt, bias, kernels, strides, pads, group, dilation, out offset, in offset, filter offsets, bias
// offsets, bias triples, out triples, activation, its arguments, filter row sums, flags
struct ConvLayer {
  const Items<17> a;
  const Tensor &f;
  const Ints<2> k, s, d;
  const Ints<4> p;
  const Triples bt, ot;
  const int64_t fd[4];
  int32_t act[3] = {0, 0, 0};
  glowb200_conv_layer layer;
  ConvLayer(PyObject *o, const char *which)
      : a(o, which), f(cuda_tensor(a[0], "filt", I8)), k(a[2], "kernels"), s(a[3], "strides"), d(a[6], "dilation"), p(a[4], "pads"),
        bt(a[11], false), ot(a[12], false), fd{f.size(0), f.size(1), f.size(2), f.size(3)} {
    if (a[14] != Py_None) {
      const Ints<3> v(a[14], "act_args");
      for (int i = 0; i < 3; i++) act[i] = (int32_t)v.v[i];
    }
    auto ints = [&](int i, const char *name) { return (const int32_t *)address(a[i], name); };
    layer = glowb200_conv_layer{(const int8_t *)f.data_ptr(), ints(1, "bias"), ints(9, "filter_offsets"), ints(10, "bias_offsets"),
                                bt.p[0], bt.p[1], bt.p[2], ot.p[0], ot.p[1], ot.p[2], ints(15, "filter_row_sums"),
                                fd, k.v, s.v, p.v, d.v, integer(a[5]), (int32_t)integer(a[8]), (int32_t)integer(a[7]),
                                (int32_t)integer(a[13]), a[14] != Py_None ? act : nullptr, (int)integer(a[16])};
  }
  // dims of its result over an input of dims `in`
  void result(const int64_t (&in)[4], int64_t (&out)[4]) const {
    out[0] = in[0];
    for (int i = 0; i < 2; i++) out[1 + i] = conv_out(in[1 + i], k.v[i], s.v[i], p.v[i] + p.v[2 + i], d.v[i]);
    out[3] = fd[0];
  }
};

// inp, first layer, second layer, out, workspace, status
PyObject *channelwise_conv_pair(PyObject *const *a) {
  const Tensor &x = cuda_tensor(a[0], "inp", I8);
  const ConvLayer first(a[1], "first"), second(a[2], "second");
  const int64_t in[4] = {x.size(0), x.size(1), x.size(2), x.size(3)};
  int64_t mid[4], od[4];
  first.result(in, mid);
  second.result(mid, od);
  const bool given = a[3] != Py_None;
  const Tensor out = given ? any_tensor(a[3], "out") : empty({od[0], od[1], od[2], od[3]}, at::kChar, x);
  const Workspace ws(a[4], a[4] == Py_None ? fn.glowb200_channelwise_quantized_conv2d_pair_workspace_bytes(in, mid, od, &first.layer,
                                                                                                           &second.layer) : 0, x);
  invoke(fn.glowb200_channelwise_quantized_conv2d_pair_i8_i32, (int8_t *)out.data_ptr(), (const int8_t *)x.data_ptr(), in, mid, od,
         &first.layer, &second.layer, ws.data(), ws.bytes(), (int32_t *)address(a[5], "status"), stream());
  return given ? same(a[3]) : give(out);
}

// lhs, rhs, dest offset, lhs offset, rhs offset, lhs triple, rhs triple, splat, out
PyObject *add_maxsplat(PyObject *const *a) {
  const Tensor &l = any_tensor(a[0], "lhs"), &r = any_tensor(a[1], "rhs");
  const Ints<3> lt(a[5], "lhs_triple"), rt(a[6], "rhs_triple");
  const bool given = a[8] != Py_None;
  const Tensor out = given ? any_tensor(a[8], "out") : l.is_contiguous() ? empty(l.sizes(), l.scalar_type(),
      l) : at::empty_like(l);
  invoke(fn.glowb200_element_add_maxsplat_i8, (int8_t *)out.data_ptr(), (const int8_t *)l.data_ptr(),
      (const int8_t *)r.data_ptr(),
                                            l.numel(), (int32_t)integer(a[2]), (int32_t)integer(a[3]), (int32_t)integer(a[4]),
                                            (int32_t)lt.v[0], (int32_t)lt.v[1], (int32_t)lt.v[2], (int32_t)rt.v[0],
                                                (int32_t)rt.v[1],
                                            (int32_t)rt.v[2], (int32_t)integer(a[7]), stream());
  return given ? same(a[8]) : give(out);
}

// src, scale, offset, out
template <bool QUANTIZE>
PyObject *element_convert(PyObject *const *a) {
  const Tensor &x = any_tensor(a[0], "src");
  const bool given = a[3] != Py_None;
  const Tensor out = given ? any_tensor(a[3], "out") : empty(x.sizes(), QUANTIZE ? at::kChar : at::kFloat, x);
  if constexpr (QUANTIZE)
    invoke(fn.glowb200_element_quantize_i8, (int8_t *)out.data_ptr(), (const float *)x.data_ptr(), x.numel(), real(a[1]),
        (int32_t)integer(a[2]), stream());
  else
    invoke(fn.glowb200_element_dequantize_i8, (float *)out.data_ptr(), (const int8_t *)x.data_ptr(), x.numel(), real(a[1]),
        (int32_t)integer(a[2]), stream());
  return given ? same(a[3]) : give(out);
}

// inp, kernels, strides, pads, out offset, out [, count include pads, in offset, triple]
template <bool AVERAGE>
PyObject *pool(PyObject *const *a) {
  const Tensor &x = any_tensor(a[0], "inp");
  const Ints<2> k(a[1], "kernels"), s(a[2], "strides");
  const Ints<4> p(a[3], "pads");
  const int64_t in[4] = {x.size(0), x.size(1), x.size(2), x.size(3)};
  const bool given = a[5] != Py_None;
  const Tensor out = given ? any_tensor(a[5], "out")
                           : empty({in[0], conv_out(in[1], k.v[0], s.v[0], p.v[0] + p.v[2], 1),
                                    conv_out(in[2], k.v[1], s.v[1], p.v[1] + p.v[3], 1), in[3]}, at::kChar, x);
  const int64_t od[4] = {out.size(0), out.size(1), out.size(2), out.size(3)};
  if constexpr (AVERAGE) {
    const Ints<3> t(a[8], "triple");
    invoke(fn.glowb200_avg_pool_i8, (const int8_t *)x.data_ptr(), (int8_t *)out.data_ptr(), in, od, k.v, s.v, p.v,
        PyObject_IsTrue(a[6]) == 1,
                                  (int32_t)integer(a[4]), (int32_t)integer(a[7]), (int32_t)t.v[0], (int32_t)t.v[1],
                                      (int32_t)t.v[2], stream());
  } else {
    invoke(fn.glowb200_max_pool_i8, (const int8_t *)x.data_ptr(), (int8_t *)out.data_ptr(), in, od, k.v, s.v, p.v,
        (int32_t)integer(a[4]), stream());
  }
  return given ? same(a[5]) : give(out);
}

// src, shuffle, scale, offset, out
PyObject *quantize_transpose(PyObject *const *a) {
  const Tensor &x = cuda_tensor(a[0], "src", F32);
  PyObject *seq = PySequence_Fast(a[1], "shuffle");
  if (seq == nullptr) throw Raised{};
  const int n = (int)PySequence_Fast_GET_SIZE(seq);
  int64_t dims[8] = {}, od[8] = {};
  int32_t sh[8] = {};
  bool ok = n <= 8 && n == x.dim();
  for (int i = 0; ok && i < n; i++) {
    sh[i] = (int32_t)PyLong_AsLongLong(PySequence_Fast_GET_ITEM(seq, i));
    dims[i] = x.size(i);
    ok = sh[i] >= 0 && sh[i] < n;
    if (ok) od[i] = x.size(sh[i]);
  }
  Py_DECREF(seq);
  if (PyErr_Occurred()) throw Raised{};
  if (!ok) {
    PyErr_SetString(PyExc_IndexError, "shuffle does not fit the tensor's dimensions");
    throw Raised{};
  }
  const bool given = a[4] != Py_None;
  const Tensor out = given ? cuda_tensor(a[4], "out", bit(at::kChar)) : empty(c10::IntArrayRef(od, (size_t)n), at::kChar, x);
  invoke(fn.glowb200_quantize_transpose_i8, (int8_t *)out.data_ptr(), (const float *)x.data_ptr(), dims, sh, n, real(a[2]),
      (int32_t)integer(a[3]), stream());
  return given ? same(a[4]) : give(out);
}

// dense, pooled, quantize?, scale, offset, out
PyObject *pairwise_dot(PyObject *const *a) {
  const Tensor &x = cuda_tensor(a[0], "dense", F32), &v = cuda_tensor(a[1], "pooled", F32);
  const int64_t B = x.size(0), D = x.size(1), T = B ? v.numel() / (B * D) : 0, n = T + 1, width = D + n * (n - 1) / 2;
  const bool quant = PyObject_IsTrue(a[2]) == 1, given = a[5] != Py_None;
  const Tensor out = given ? any_tensor(a[5], "out") : empty({B, width}, quant ? at::kChar : at::kFloat, x);
  invoke(fn.glowb200_pairwise_dot_interaction, (const float *)x.data_ptr(), D, (const float *)v.data_ptr(), T * D, B, T, D,
                                             quant ? nullptr : (float *)out.data_ptr(),
                                                 quant ? (int8_t *)out.data_ptr() : nullptr, width,
                                             real(a[3]), (int32_t)integer(a[4]), stream());
  return given ? same(a[5]) : give(out);
}

// ---- device manager ----
// handle, network name, {placeholder name: array}, names of the outputs (None: every array goes in and comes back)
PyObject *run_function(PyObject *const *a) {
  void *dm = PyLong_AsVoidPtr(a[0]);
  const char *name = PyUnicode_AsUTF8(a[1]);
  if (name == nullptr || PyErr_Occurred()) throw Raised{};
  if (!PyDict_Check(a[2])) {
    PyErr_SetString(PyExc_TypeError, "bindings must be a dict of placeholder names and arrays");
    throw Raised{};
  }
  // (a list of its own: the names and arrays stay what they are whatever becomes of the dict during the call)
  struct Items {
    PyObject *list;
    ~Items() { Py_XDECREF(list); }
  } items{PyDict_Items(a[2])};
  if (items.list == nullptr) throw Raised{};
  const size_t n = (size_t)PyList_GET_SIZE(items.list);
  std::vector<const char *> names;
  std::vector<void *> buffers;
  std::vector<size_t> sizes;
  std::vector<int> directions;
  struct Views {
    std::vector<Py_buffer> v;
    ~Views() { for (Py_buffer &b : v) PyBuffer_Release(&b); }
  } views;
  names.reserve(n), buffers.reserve(n), sizes.reserve(n), directions.reserve(n), views.v.reserve(n);
  for (size_t i = 0; i < n; i++) {
    PyObject *item = PyList_GET_ITEM(items.list, (Py_ssize_t)i), *key = PyTuple_GET_ITEM(item, 0), *value = PyTuple_GET_ITEM(item, 1);
    const char *k = PyUnicode_AsUTF8(key);
    if (k == nullptr) throw Raised{};
    Py_buffer b;
    if (!PyObject_TypeCheck(value, reinterpret_cast<PyTypeObject *>(ndarray)) ||
        PyObject_GetBuffer(value, &b, PyBUF_WRITABLE | PyBUF_C_CONTIGUOUS) != 0) {
      PyErr_SetString(PyExc_TypeError, "bindings must be writable C-contiguous numpy arrays");
      throw Raised{};
    }
    views.v.push_back(b);
    names.push_back(k);
    buffers.push_back(b.buf);
    sizes.push_back((size_t)b.len);
    int direction = GLOWB200_BINDING_INPUT | GLOWB200_BINDING_OUTPUT;
    if (a[3] != Py_None) {
      const int is_output = PySequence_Contains(a[3], key);
      if (is_output < 0) throw Raised{};
      direction = is_output ? GLOWB200_BINDING_OUTPUT : GLOWB200_BINDING_INPUT;
    }
    directions.push_back(direction);
  }
  invoke(fn.glowb200_device_manager_run_function_io, static_cast<glowb200_device_manager *>(dm), name, names.data(),
         buffers.data(), sizes.data(), directions.data(), (int)n);
  Py_RETURN_NONE;
}

// setup(addresses by name, error class, explain)
PyObject *setup(PyObject *, PyObject *args) {
  PyObject *table, *error, *why;
  if (!PyArg_ParseTuple(args, "O!OO", &PyDict_Type, &table, &error, &why)) return nullptr;
#define X(name)                                                                        \
  {                                                                                    \
    PyObject *at = PyDict_GetItemString(table, #name);                                 \
    if (at == nullptr) { PyErr_SetString(PyExc_KeyError, #name); return nullptr; }      \
    fn.name = reinterpret_cast<decltype(fn.name)>(PyLong_AsVoidPtr(at));               \
    if (fn.name == nullptr) return nullptr;                                            \
  }
  GLOWB200_ENTRY_POINTS(X)
#undef X
  PyObject *numpy = PyImport_ImportModule("numpy");
  PyObject *array = numpy ? PyObject_GetAttrString(numpy, "ndarray") : nullptr;
  Py_XDECREF(numpy);
  if (array == nullptr) return nullptr;
  Py_XSETREF(ndarray, array);
  Py_INCREF(error);
  Py_INCREF(why);
  Py_XSETREF(error_class, error);
  Py_XSETREF(explain, why);
  Py_RETURN_NONE;
}

#define FAST(name, body, n) \
  {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&guarded<body, n>)), \
   METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"setup", setup, METH_VARARGS, nullptr},
    FAST("slws", slws, 12),
    FAST("embedding_bag", embedding_bag, 11),
    FAST("slws_batched", slws_batched, 12),
    FAST("split_bags", split_bags, 16),
    FAST("rowwise_fc", rowwise_fc, 14),
    FAST("fc_i8", fc_i8, 14),
    FAST("matmul", matmul, 10),
    FAST("dynamic_rowwise_fc", dynamic_fc<true>, 10),
    FAST("dynamic_fc", dynamic_fc<false>, 10),
    FAST("channelwise_conv", channelwise_conv<false>, 21),
    FAST("channelwise_conv_add", channelwise_conv<true>, 28),
    FAST("channelwise_conv_pair", channelwise_conv_pair, 6),
    FAST("add_maxsplat", add_maxsplat, 9),
    FAST("quantize", element_convert<true>, 4),
    FAST("dequantize", element_convert<false>, 4),
    FAST("max_pool", pool<false>, 6),
    FAST("avg_pool", pool<true>, 9),
    FAST("quantize_transpose", quantize_transpose, 5),
    FAST("pairwise_dot", pairwise_dot, 6),
    FAST("run_function", run_function, 4),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding(void) { return PyModule_Create(&module); }
