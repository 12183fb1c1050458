// The host side of a call in native code: reads a GemmParams / ConvParams record as the Python layer
// (cumm_b200/tensorview/gemm.py, _gemm_args and _conv_args) does, and launches.  It answers for the ordinary
// call only -- torch tensors on the current device, a descriptor of this library's kernels, no timer -- and
// returns None for everything else, wrong or merely unusual, before anything has been launched: the Python
// layer then takes the call, with its checks and its errors.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <ATen/core/Tensor.h>
#include <c10/core/impl/DeviceGuardImplInterface.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>

#include "../../include/cumm_b200.h"

namespace {

using RunGemm = int (*)(const cb2_gemm_args *, void *);
using RunConv = int (*)(const cb2_conv_args *, void *);
RunGemm g_run_gemm = nullptr;
RunConv g_run_conv = nullptr;
PyObject *g_gemm_params, *g_gemm_desp, *g_conv_params, *g_conv_desp;  // the record classes

#define CB2_NAMES(X)                                                                                                  \
  X(_a) X(_b) X(_c) X(_d) X(a_inds) X(b_inds) X(c_inds) X(alpha) X(beta) X(act_alpha) X(act_beta) X(act_type)          \
  X(stream) X(timer) X(max_ctas) X(split_k_slices) X(_algo_desp) X(_conv_algo_desp) X(dtype_a) X(dtype_b) X(dtype_c)   \
  X(dacc) X(dcomp) X(trans_a_) X(trans_b_) X(trans_c_) X(tile_shape) X(warp_tile_shape) X(tensorop) X(num_stage)       \
  X(algo) X(shuffle_type) X(element_per_access_a) X(element_per_access_b) X(element_per_access_c) X(input) X(weight)   \
  X(output) X(output_add) X(bias) X(scale) X(indices) X(mask) X(mask_argsort) X(mask_output) X(mask_width)             \
  X(mask_filter) X(reverse_mask) X(verbose) X(op_type) X(ndim) X(mask_sparse) X(dynamic_mask) X(is_int8_inference)     \
  X(split_k_serial_) X(split_k_parallel_) X(padding) X(stride) X(dilation)
#define X(n) PyObject *k_##n;
CB2_NAMES(X)
#undef X

// Not the ordinary call: whoever finds out throws, nothing has been launched yet.  A throw costs 2 us, so what programs
// do in earnest and the Python layer answers for (timers, tensors that are not torch's, other kinds of calls, and
// in run_conv the weight gradient) is found at the start of read_gemm and read_conv, which then return false (0.3 us).
struct Unusual {};
inline void need(bool ok) {
  if (!ok)
    throw Unusual();
}

struct Ref {
  PyObject *p;
  explicit Ref(PyObject *o) : p(o) {}
  Ref(const Ref &) = delete;
  Ref &operator=(const Ref &) = delete;
  ~Ref() { Py_XDECREF(p); }
};

struct Record {
  PyObject *o;
  PyObject *get(PyObject *key) const {
    PyObject *v = PyObject_GetAttr(o, key);
    if (!v)
      PyErr_Clear();
    need(v != nullptr);
    return v;
  }
  long long integer(PyObject *key) const {
    Ref v(get(key));
    need(PyLong_Check(v.p));
    const long long r = PyLong_AsLongLong(v.p);
    if (r == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      throw Unusual();
    }
    return r;
  }
  int small(PyObject *key) const {
    const long long r = integer(key);
    need(r >= -(1ll << 31) && r < (1ll << 31));
    return static_cast<int>(r);
  }
  bool flag(PyObject *key) const {
    Ref v(get(key));
    need(PyBool_Check(v.p));
    return v.p == Py_True;
  }
  float real(PyObject *key) const {
    Ref v(get(key));
    need(PyFloat_CheckExact(v.p) || PyLong_CheckExact(v.p));
    const double r = PyFloat_AsDouble(v.p);
    if (r == -1.0 && PyErr_Occurred()) {
      PyErr_Clear();
      throw Unusual();
    }
    return static_cast<float>(r);
  }
  bool is_tensor(PyObject *key) const {
    Ref v(get(key));
    return THPVariable_CheckExact(v.p);
  }
  bool none(PyObject *key) const {
    Ref v(get(key));
    return v.p == Py_None;
  }
  void triple(PyObject *key, int (&out)[3]) const {
    Ref v(get(key));
    need(PyList_CheckExact(v.p) && PyList_GET_SIZE(v.p) == 3);
    for (int i = 0; i < 3; ++i) {
      PyObject *e = PyList_GET_ITEM(v.p, i);
      need(PyLong_CheckExact(e));
      const long r = PyLong_AsLong(e);
      if (r == -1 && PyErr_Occurred())
        PyErr_Clear();
      need(r > 0 && r < (1 << 20));
      out[i] = static_cast<int>(r);
    }
  }
};

// The types that the Python layer has a code for; a tensor of any other is refused there.
bool has_code(at::ScalarType t) {
  switch (t) {
  case at::kFloat:
  case at::kInt:
  case at::kShort:
  case at::kChar:
  case at::kDouble:
  case at::kBool:
  case at::kByte:
  case at::kHalf:
  case at::kLong:
  case at::kBFloat16:
  case at::kUInt16:
  case at::kUInt32:
  case at::kUInt64:
    return true;
  default:
    return false;
  }
}

// A CUDA tensor with at least one element, or none.
struct View {
  const at::Tensor *t = nullptr;
  int64_t dim(int i) const { return t->size(i); }
  int64_t stride(int i) const { return t->stride(i); }
  int n_dims() const { return static_cast<int>(t->dim()); }
  void *data() const { return t ? t->data_ptr() : nullptr; }
  explicit operator bool() const { return t != nullptr; }
};
View view(const Record &r, PyObject *key, bool may_be_none) {
  Ref v(r.get(key));  // the record holds it for the length of the call
  View w;
  if (v.p == Py_None) {
    need(may_be_none);
    return w;
  }
  need(THPVariable_CheckExact(v.p));
  w.t = &THPVariable_Unpack(v.p);
  need(w.t->is_cuda() && w.t->layout() == at::kStrided && w.t->numel() > 0 && has_code(w.t->scalar_type()));
  return w;
}
int size32(int64_t v) {
  need(v >= 0 && v < (1ll << 31));
  return static_cast<int>(v);
}
int dtype_code(const at::Tensor &t) {
  switch (t.scalar_type()) {
  case at::kHalf:
    return CB2_DTYPE_F16;
  case at::kChar:
    return CB2_DTYPE_I8;
  case at::kFloat:
    return CB2_DTYPE_F32;
  default:
    throw Unusual();
  }
}
void *stream_of(const Record &p) { return reinterpret_cast<void *>(static_cast<intptr_t>(p.integer(k_stream))); }
bool on_current_device(const View &v) {
  return c10::impl::getDeviceGuardImpl(at::kCUDA)->getDevice().index() == v.t->get_device();
}

struct Desp {
  int tile[3];
  int epa[3];
  bool ta, tb, tc;
};
// GemmAlgoDesp.check_valid, and the fields both kinds of call use
Desp read_desp(const Record &d) {
  Desp r;
  const int a = d.small(k_trans_a_), b = d.small(k_trans_b_), c = d.small(k_trans_c_);
  need((a == 0 || a == 1) && (b == 0 || b == 1) && (c == 0 || c == 1));
  r.ta = a, r.tb = b, r.tc = c;
  {
    Ref algo(d.get(k_algo));
    need(PyUnicode_CheckExact(algo.p) && PyUnicode_GET_LENGTH(algo.p) > 0);
  }
  int other[3];
  d.triple(k_tile_shape, r.tile);
  d.triple(k_warp_tile_shape, other);
  d.triple(k_tensorop, other);
  need(d.small(k_dtype_a) != -1 && d.small(k_dtype_b) != -1 && d.small(k_dtype_c) != -1 && d.small(k_dacc) != -1 &&
       d.small(k_dcomp) != -1 && d.small(k_num_stage) > 0);
  r.epa[0] = d.small(k_element_per_access_a);
  r.epa[1] = d.small(k_element_per_access_b);
  r.epa[2] = d.small(k_element_per_access_c);
  need(r.tile[0] == 128);
  return r;
}
bool divides(int epa, long long v) { return epa <= 0 || v % epa == 0; }

// The flat record of a GEMM call whose tensors are on the current device: plain or scattered rows.
bool read_gemm(PyObject *params, cb2_gemm_args &g, bool) {
  if (!g_run_gemm || reinterpret_cast<PyObject *>(Py_TYPE(params)) != g_gemm_params)
    return false;
  const Record p{params};
  if (!p.none(k_timer) || !p.none(k__d) || !p.none(k_b_inds) || !p.is_tensor(k__c))
    return false;
  Ref desp(p.get(k__algo_desp));
  if (reinterpret_cast<PyObject *>(Py_TYPE(desp.p)) != g_gemm_desp)
    return false;
  const Record d{desp.p};
  const int shuffle = d.small(k_shuffle_type);
  if (shuffle != CB2_SHUFFLE_AC && shuffle != CB2_SHUFFLE_NONE)
    return false;
  const Desp ds = read_desp(d);
  need(!ds.ta && !ds.tc);
  need(p.small(k_split_k_slices) == 1);
  const View a = view(p, k__a, false), b = view(p, k__b, false), c = view(p, k__c, false);
  need(a.n_dims() == 2 && b.n_dims() == 2 && c.n_dims() == 2);
  need(a.t->get_device() == c.t->get_device() && b.t->get_device() == c.t->get_device() && on_current_device(c));
  const View ai = view(p, k_a_inds, true), ci = view(p, k_c_inds, shuffle != CB2_SHUFFLE_AC);
  need((!ai || ai.n_dims() > 0) && (!ci || ci.n_dims() > 0));
  g.m = size32(shuffle == CB2_SHUFFLE_AC && ai ? ai.dim(0) : a.dim(0));
  g.k = size32(a.dim(1));
  g.n = size32(b.dim(ds.tb ? 0 : 1));
  need(b.dim(ds.tb ? 1 : 0) == g.k && c.dim(1) == g.n && (shuffle == CB2_SHUFFLE_AC || c.dim(0) == g.m));
  // the leading dimensions GemmAlgoDesp.supported looks at
  need(divides(ds.epa[0], g.k) && divides(ds.epa[1], ds.tb ? g.k : g.n) && divides(ds.epa[2], g.n));
  g.ptr_A = a.data(), g.ptr_B = b.data(), g.ptr_C = c.data();
  g.stride_A = a.stride(0), g.stride_B = b.stride(0), g.stride_C = c.stride(0);
  if (shuffle == CB2_SHUFFLE_AC) {
    g.indiceA = static_cast<const int32_t *>(ai.data());
    g.indiceBorC = static_cast<const int32_t *>(ci.data());
  }
  g.alpha = p.real(k_alpha), g.beta = p.real(k_beta);
  g.act_alpha = p.real(k_act_alpha), g.act_beta = p.real(k_act_beta);
  g.act_type = p.small(k_act_type);
  g.split_k_slices = 1;
  g.dtype_a = d.small(k_dtype_a), g.dtype_b = d.small(k_dtype_b), g.dtype_c = d.small(k_dtype_c);
  g.trans_b = ds.tb;
  g.shuffle_type = shuffle;
  g.rows_A = size32(a.dim(0)), g.rows_B = size32(b.dim(0));
  g.tile_n = ds.tile[1], g.tile_k = ds.tile[2];
  g.max_ctas = p.small(k_max_ctas);
  return true;
}

// What both kinds of convolution calls say about their tensors: rows of channels, and the neighbour tables.
struct ConvTensors {
  View in, w, out, add, ind, mask, order, mask_out;
  int64_t rows_in, rows_out;
  int C, K, kv;
  bool dynamic;  // the descriptor allows more than 32 offsets
};

// The rest of a convolution's record, and its checks.
void fill_conv(const Record &p, const Record &d, const Desp &ds, int op, const ConvTensors &t, cb2_conv_args &g) {
  const bool fwd = op == CB2_CONV_FORWARD, wgrad = op == CB2_CONV_BACKWARD_WEIGHT, int8 = d.flag(k_is_int8_inference);
  g.split_k_slices = p.small(k_split_k_slices);
  need(g.split_k_slices <= 1 || d.small(k_split_k_serial_) == 1 || d.small(k_split_k_parallel_) == 1);
  const View bias = view(p, k_bias, true), scale = view(p, k_scale, true);
  g.K = t.K, g.kernel_volume = t.kv, g.C = t.C;
  need(int8 ? (bias && scale) : !t.add);
  if (t.add)
    need(t.add.t->scalar_type() == t.out.t->scalar_type() && t.add.t->sizes() == t.out.t->sizes());
  const int kv = g.kernel_volume, words = (kv + 31) / 32;
  need(t.ind.n_dims() == 2 && t.ind.dim(0) == kv && kv >= 1 && kv <= 128 && (kv <= 32 || t.dynamic));
  g.N = size32(t.ind.dim(1));
  need(g.N == (fwd || wgrad ? t.rows_out : t.rows_in));
  // what ConvAlgoDesp.supported looks at
  const long long m = wgrad ? g.K : g.N, n = fwd ? g.K : wgrad ? 1ll * g.C * kv : g.C,
                  k = wgrad ? g.N : 1ll * kv * (fwd ? g.C : g.K);
  need(divides(ds.epa[0], ds.ta ? m : k) && divides(ds.epa[1], ds.tb ? k : n) && divides(ds.epa[2], ds.tc ? m : n));
  need(ds.epa[0] != 0 && (fwd ? g.C : g.K) % ds.epa[0] == 0);
  if (wgrad)
    need(ds.epa[1] != 0 && g.C % ds.epa[1] == 0 && g.mask_width > 0 && g.mask_width % ds.tile[2] == 0);
  const View &a = fwd ? t.in : t.out, &b = wgrad ? t.in : t.w, &c = fwd ? t.out : wgrad ? t.w : t.in;
  need(on_current_device(c));
  g.ptr_A = a.data(), g.ptr_B = b.data(), g.ptr_C = c.data();
  g.ptr_D = t.add ? t.add.data() : (int8 || !bias) ? c.data() : bias.data();
  g.d_is_bias = bias && !int8 && !t.add;
  g.bias_pointer = bias.data(), g.scale_pointer = scale.data();
  g.alpha = p.real(k_alpha), g.beta = p.real(k_beta);
  g.act_alpha = p.real(k_act_alpha), g.act_beta = p.real(k_act_beta);
  g.act_type = p.small(k_act_type);
  g.mask_ptr = static_cast<const uint32_t *>(t.mask.data());
  g.mask_out_ptr = static_cast<uint32_t *>(t.mask_out.data());
  g.indice_ptr = static_cast<const int32_t *>(t.ind.data());
  g.mask_argsort_ptr = static_cast<const int32_t *>(t.order.data());
  g.ndim = d.small(k_ndim);
  g.mode = 1;
  g.groups = 1;
  g.op_type = op;
  g.dtype_a = dtype_code(*a.t), g.dtype_b = dtype_code(*b.t), g.dtype_c = dtype_code(*c.t);
  g.is_int8_inference = int8;
  const auto rows = [&](const View &v) { return size32(&v == &t.in ? t.rows_in : &v == &t.out ? t.rows_out : t.K); };
  g.rows_A = rows(a), g.rows_B = rows(b);
  g.mask_words = size32(t.mask.t->numel());
  need(wgrad || g.mask_words >= static_cast<long long>(g.N) * words);
  if (fwd && t.mask_out)
    need(t.mask_out.t->numel() >= (static_cast<long long>(g.N) + 127) / 128 * words);
  g.tile_n = ds.tile[1], g.tile_k = wgrad ? 0 : ds.tile[2];
  g.max_ctas = p.small(k_max_ctas);
}

// The record of a convolution in the ordinary call, its descriptor and its operator; false: some other kind.
bool conv_record(PyObject *params, PyObject *desp) {
  if (!g_run_conv || reinterpret_cast<PyObject *>(Py_TYPE(params)) != g_conv_params ||
      reinterpret_cast<PyObject *>(Py_TYPE(desp)) != g_conv_desp)
    return false;
  const Record p{params};
  return p.none(k_timer) && !p.flag(k_verbose) && p.is_tensor(k_output);
}

// The flat record of a convolution call whose tensors are on the current device.
bool read_conv(PyObject *params, cb2_conv_args &g, bool with_weight_gradient) {
  const Record p{params};
  Ref desp(p.get(k__conv_algo_desp));
  if (!conv_record(params, desp.p))
    return false;
  const Record d{desp.p};
  const int op = d.small(k_op_type);
  if (op < CB2_CONV_FORWARD || op > CB2_CONV_BACKWARD_WEIGHT || (op == CB2_CONV_BACKWARD_WEIGHT && !with_weight_gradient) ||
      !d.flag(k_mask_sparse))
    return false;
  const Desp ds = read_desp(d);
  ConvTensors t;
  t.in = view(p, k_input, false), t.w = view(p, k_weight, false), t.out = view(p, k_output, false);
  need(t.in.n_dims() == 2 && t.out.n_dims() == 2 && t.w.n_dims() == 3);
  need(t.in.t->is_contiguous() && t.w.t->is_contiguous() && t.out.t->is_contiguous());
  t.add = view(p, k_output_add, true);
  t.ind = view(p, k_indices, false), t.mask = view(p, k_mask, false), t.order = view(p, k_mask_argsort, false),
  t.mask_out = view(p, k_mask_output, true);
  t.K = size32(t.w.dim(0)), t.kv = size32(t.w.dim(1)), t.C = size32(t.w.dim(2));
  need(t.in.dim(1) == t.C && t.out.dim(1) == t.K);
  t.rows_in = t.in.dim(0), t.rows_out = t.out.dim(0);
  t.dynamic = t.kv <= 32 || d.flag(k_dynamic_mask);
  g.mask_width = p.small(k_mask_width);
  g.mask_filter = static_cast<uint32_t>(p.integer(k_mask_filter));
  g.reverse_mask = p.flag(k_reverse_mask);
  fill_conv(p, d, ds, op, t, g);
  return true;
}

// ---------------------------------------------------------------- dense convolutions (cumm_b200/dense.py)
// Extents of a dense call, the spatial ones padded to three axes in front; as _geometry there works them out.
struct DenseShape {
  int64_t batch, C, K;
  int64_t in[3], out[3], k[3];
  int pad[3], stride[3], dil[3];
};
void axes(const Record &p, PyObject *key, int ndim, int otherwise, int (&v)[3], int fill) {
  Ref l(p.get(key));
  need(PyList_CheckExact(l.p));
  const Py_ssize_t n = PyList_GET_SIZE(l.p);
  need(n == 0 || n == ndim);
  for (int a = 0; a < 3; ++a)
    v[a] = fill;
  for (int a = 0; a < ndim; ++a) {
    int r = otherwise;
    if (n) {
      PyObject *e = PyList_GET_ITEM(l.p, a);
      need(PyLong_CheckExact(e));
      const long x = PyLong_AsLong(e);
      if (x == -1 && PyErr_Occurred())
        PyErr_Clear();
      need(x >= 0 && x < (1 << 20));
      r = static_cast<int>(x);
    }
    v[3 - ndim + a] = r;
  }
}
// false: not the ordinary dense call
bool dense_shape(const Record &p, const Record &d, DenseShape &s) {
  if (d.flag(k_mask_sparse))
    return false;
  const int ndim = d.small(k_ndim);
  need(ndim >= 1 && ndim <= 3);
  const View in = view(p, k_input, false), w = view(p, k_weight, false), out = view(p, k_output, false);
  need(in.n_dims() == ndim + 2 && w.n_dims() == ndim + 2 && out.n_dims() == ndim + 2);
  need(in.t->is_contiguous() && w.t->is_contiguous() && out.t->is_contiguous() && p.none(k_output_add));
  s.batch = in.dim(0), s.C = in.dim(ndim + 1), s.K = w.dim(0);
  need(w.dim(ndim + 1) == s.C && out.dim(ndim + 1) == s.K && out.dim(0) == s.batch);
  axes(p, k_padding, ndim, 0, s.pad, 0), axes(p, k_stride, ndim, 1, s.stride, 1), axes(p, k_dilation, ndim, 1, s.dil, 1);
  for (int a = 0; a < 3; ++a)
    s.in[a] = s.out[a] = s.k[a] = 1;
  for (int a = 3 - ndim; a < 3; ++a) {
    s.in[a] = in.dim(1 + a - (3 - ndim)), s.k[a] = w.dim(1 + a - (3 - ndim)), s.out[a] = out.dim(1 + a - (3 - ndim));
    const int64_t span = s.in[a] + 2ll * s.pad[a] - s.dil[a] * (s.k[a] - 1) - 1;
    need(s.stride[a] >= 1 && s.dil[a] >= 1 && span >= 0 && s.out[a] == span / s.stride[a] + 1);
  }
  return true;
}
View tensor(PyObject *o) {
  need(THPVariable_CheckExact(o));
  View v;
  v.t = &THPVariable_Unpack(o);
  return v;
}
// `tables`: (indices_fwd, indices_bwd, mask_fwd, mask_bwd, argsort_fwd, argsort_bwd, tile_masks) of the call's shape
bool read_dense(PyObject *params, PyObject *tables, cb2_conv_args &g) {
  Ref desp(Record{params}.get(k__conv_algo_desp));
  if (!conv_record(params, desp.p) || !PyTuple_CheckExact(tables) || PyTuple_GET_SIZE(tables) != 7)
    return false;
  const Record p{params}, d{desp.p};
  DenseShape s;
  if (!dense_shape(p, d, s))
    return false;
  const int op = d.small(k_op_type);
  need(op >= CB2_CONV_FORWARD && op <= CB2_CONV_BACKWARD_WEIGHT);
  const Desp ds = read_desp(d);
  ConvTensors t;
  t.in = view(p, k_input, false), t.w = view(p, k_weight, false), t.out = view(p, k_output, false);
  t.rows_in = s.batch * s.in[0] * s.in[1] * s.in[2], t.rows_out = s.batch * s.out[0] * s.out[1] * s.out[2];
  t.C = size32(s.C), t.K = size32(s.K), t.kv = size32(s.k[0] * s.k[1] * s.k[2]);
  t.dynamic = true;
  const bool bwd = op == CB2_CONV_BACKWARD_INPUT, wgrad = op == CB2_CONV_BACKWARD_WEIGHT;
  t.ind = tensor(PyTuple_GET_ITEM(tables, bwd ? 1 : 0));
  t.mask = tensor(PyTuple_GET_ITEM(tables, wgrad ? 6 : bwd ? 3 : 2));
  t.order = tensor(PyTuple_GET_ITEM(tables, bwd ? 5 : 4));
  g.mask_width = wgrad ? 128 : -1;
  g.mask_filter = 0xffffffffu;
  fill_conv(p, d, ds, op, t, g);
  g.reuse_plan = wgrad ? 0 : 1;  // the grid's tables were whole before the call, and nothing writes them again
  return true;
}

template <class Args, class Run> PyObject *launch(Run run, const Args &a, void *stream) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = run(&a, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

// run_gemm(params), run_conv(params): the call's return code, or None.  The weight gradient needs scratch, which
// the Python layer keeps.
PyObject *run_gemm(PyObject *, PyObject *params) {
  cb2_gemm_args g;
  memset(&g, 0, sizeof(g));
  void *stream;
  try {
    if (!read_gemm(params, g, false))
      Py_RETURN_NONE;
    stream = stream_of(Record{params});
  } catch (...) {
    Py_RETURN_NONE;
  }
  return launch(g_run_gemm, g, stream);
}
PyObject *run_conv(PyObject *, PyObject *params) {
  cb2_conv_args g;
  memset(&g, 0, sizeof(g));
  void *stream;
  try {
    if (!read_conv(params, g, false))
      Py_RETURN_NONE;
    stream = stream_of(Record{params});
  } catch (...) {
    Py_RETURN_NONE;
  }
  return launch(g_run_conv, g, stream);
}

// dense_key(params): what a dense call's tables are found by, or None.
PyObject *dense_key(PyObject *, PyObject *params) {
  try {
    DenseShape s;
    Ref desp(Record{params}.get(k__conv_algo_desp));
    if (!conv_record(params, desp.p) || !dense_shape(Record{params}, Record{desp.p}, s))
      Py_RETURN_NONE;
    Ref out(Record{params}.get(k_output));
    return Py_BuildValue("(iL(LLL)(LLL)(LLL)(iii)(iii)(iii))", static_cast<int>(THPVariable_Unpack(out.p).get_device()),
                         (long long)s.batch, (long long)s.in[0], (long long)s.in[1], (long long)s.in[2], (long long)s.out[0],
                         (long long)s.out[1], (long long)s.out[2], (long long)s.k[0], (long long)s.k[1], (long long)s.k[2],
                         s.stride[0], s.stride[1], s.stride[2], s.pad[0], s.pad[1], s.pad[2], s.dil[0], s.dil[1], s.dil[2]);
  } catch (...) {
    Py_RETURN_NONE;
  }
}
// run_dense(params, tables, address): forward and input gradient are launched (the return code); the weight gradient's
// flat record is left at the address (True).  None: the Python layer takes the call.
PyObject *run_dense(PyObject *, PyObject *args) {
  PyObject *params, *tables;
  unsigned long long address;
  if (!PyArg_ParseTuple(args, "OOK", &params, &tables, &address))
    return nullptr;
  cb2_conv_args g;
  memset(&g, 0, sizeof(g));
  void *stream;
  try {
    if (!read_dense(params, tables, g))
      Py_RETURN_NONE;
    stream = stream_of(Record{params});
  } catch (...) {
    Py_RETURN_NONE;
  }
  if (g.op_type != CB2_CONV_BACKWARD_WEIGHT)
    return launch(g_run_conv, g, stream);
  memcpy(reinterpret_cast<void *>(static_cast<uintptr_t>(address)), &g, sizeof(g));
  Py_RETURN_TRUE;
}

// gemm_args(params, address), conv_args(params, address): fill the flat record there; True, or None.
template <class Args> PyObject *fill(PyObject *args, bool (*read)(PyObject *, Args &, bool)) {
  PyObject *params;
  unsigned long long address;
  if (!PyArg_ParseTuple(args, "OK", &params, &address))
    return nullptr;
  Args g;
  memset(&g, 0, sizeof(g));
  try {
    if (!read(params, g, true))
      Py_RETURN_NONE;
  } catch (...) {
    Py_RETURN_NONE;
  }
  memcpy(reinterpret_cast<void *>(static_cast<uintptr_t>(address)), &g, sizeof(g));
  Py_RETURN_TRUE;
}
PyObject *gemm_args(PyObject *, PyObject *args) { return fill<cb2_gemm_args>(args, read_gemm); }
PyObject *conv_args(PyObject *, PyObject *args) { return fill<cb2_conv_args>(args, read_conv); }

// setup(GemmParams, GemmAlgoDesp, ConvParams, ConvAlgoDesp, address of cb2_gemm_run, of cb2_conv_run)
PyObject *setup(PyObject *, PyObject *args) {
  unsigned long long gemm, conv;
  PyObject *c[4];
  if (!PyArg_ParseTuple(args, "OOOOKK", &c[0], &c[1], &c[2], &c[3], &gemm, &conv))
    return nullptr;
  for (PyObject *o : c)
    Py_INCREF(o);  // for the life of the process
  g_gemm_params = c[0], g_gemm_desp = c[1], g_conv_params = c[2], g_conv_desp = c[3];
  g_run_gemm = reinterpret_cast<RunGemm>(gemm);
  g_run_conv = reinterpret_cast<RunConv>(conv);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"setup", setup, METH_VARARGS, nullptr},
                         {"run_gemm", run_gemm, METH_O, nullptr},
                         {"run_conv", run_conv, METH_O, nullptr},
                         {"gemm_args", gemm_args, METH_VARARGS, nullptr},
                         {"conv_args", conv_args, METH_VARARGS, nullptr},
                         {"dense_key", dense_key, METH_O, nullptr},
                         {"run_dense", run_dense, METH_VARARGS, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__host(void) {
#define X(n)                                                                                                          \
  if (!(k_##n = PyUnicode_InternFromString(#n)))                                                                      \
    return nullptr;
  CB2_NAMES(X)
#undef X
  PyObject *m = PyModule_Create(&module);
#ifdef CB2_HOST_SOURCES  // a digest of this file and the header, by which the Python layer knows its own reader
  if (m && PyModule_AddStringConstant(m, "SOURCES", CB2_HOST_SOURCES) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
#endif
  return m;
}
