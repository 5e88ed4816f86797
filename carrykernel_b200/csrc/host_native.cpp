// The Python surfaces' way into libcarry_gdn.so for calls that need nothing from them: a CPython extension that
// looks a call's tensors over, fills the C ABI's argument block and launches, in one or two microseconds.
//
// What bounded a call at a small batch was the host: at one request a layer's decode kernel takes 5.1 us (6.4 at the
// time) and the Python validation with ctypes took 20 (24 layers: 470 us a step); with this module the host is done
// with a layer in 3.1 us, most of it the CUDA launch, and the kernels bound (127 us).
//
// Every function takes a call only when each condition of the Python validation holds as it stands (plain CUDA
// tensors on one device, the dtypes, shapes and strides that the kernel will index, nothing to convert); it
// then returns its result.  Otherwise -- and when the library returns an error -- it returns None and has done
// nothing, and the Python surface goes through its own checks, which convert, or raise, as they always did.
// No state is kept between calls.  The GIL is released around the launch.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <vector>

#include "../../include/carry_gdn.h"

namespace {

// Entry points of the library the Python side has loaded (it may load a second one, so they come with the call).
struct Table {
  int (*quant_step)(const CarryGdnStepArgs*, void*);
  int (*fp32_step)(const CarryGdnFp32Args*, void*);
  int (*packed_decode)(const CarryGdnPackedArgs*, void*);
  int (*packed_decode_multi)(const CarryGdnPackedMultiArgs*, void*);
  int (*pool_store)(const CarryGdnPoolStoreArgs*, void*);
  int (*pool_load)(const CarryGdnPoolLoadArgs*, void*);
  int (*pool_copy)(const CarryGdnPoolCopyArgs*, void*);
  int (*pool_copy_layers)(const CarryGdnPoolCopyLayersArgs*, void*);
  int (*quant_decode)(const CarryGdnDecodeArgs*, void*);
};
constexpr int kEntries = 9;

const Table* table_of(PyObject* o) { return static_cast<const Table*>(PyLong_AsVoidPtr(o)); }

// A plain torch.Tensor (or Parameter), else null.  A borrowed reference; subclasses go the Python way.
const at::Tensor* plain(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }

int dtype_id(at::ScalarType t) {
  return t == at::kFloat ? CARRY_F32 : t == at::kBFloat16 ? CARRY_BF16 : t == at::kHalf ? CARRY_F16 : -1;
}
bool is(const at::Tensor* t, at::ScalarType dt, int dev) {
  return t && t->scalar_type() == dt && t->is_cuda() && t->get_device() == dev;
}
bool shaped(const at::Tensor& t, std::initializer_list<int64_t> want) {
  return t.sizes() == at::IntArrayRef(want.begin(), want.size());
}
// strides of all dimensions but the first
bool dense_inside(const at::Tensor& t, std::initializer_list<int64_t> want) {
  return t.strides().slice(1) == at::IntArrayRef(want.begin(), want.size());
}
bool fits32(int64_t x) { return x > 0 && x <= 0x7fffffff; }

// the optional status word: false when it is neither absent nor what the kernels may OR into
bool status_of(PyObject* o, int dev, int32_t** out) {
  *out = nullptr;
  if (o == Py_None) return true;
  const at::Tensor* t = plain(o);
  if (!is(t, at::kInt, dev) || t->numel() != 1) return false;
  *out = static_cast<int32_t*>(t->data_ptr());
  return true;
}
bool as_int(PyObject* o, long& v) {
  if (!PyLong_Check(o)) return false;
  v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}

// Launches on the tensors' device and torch's current stream of it.
template <class F>
bool launch(int dev, F&& f) {
  c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(dev));
  void* stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f(stream);
  Py_END_ALLOW_THREADS
  return rc == CARRY_GDN_OK;
}

// A function body that returns a new reference or null for "not taken"; nothing thrown gets out.
template <class F>
PyObject* guarded(F&& f) {
  try {
    if (PyObject* r = f()) return r;
  } catch (...) {
  }
  if (PyErr_Occurred()) PyErr_Clear();
  Py_RETURN_NONE;
}

// ---------------------------------------------------------------------------
// the slot-indexed step, one or several tokens
// ---------------------------------------------------------------------------

// (table, multi, mixed_qkv, a, b, A_log, dt_bias, scale, state_codes, state_scale, resid_codes, resid_scale, out,
//  ssm_state_indices, use_qk_l2norm, resid_fmt, status) -> True
PyObject* packed_decode(PyObject*, PyObject* const* o, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 17) return nullptr;
    const Table* tab = table_of(o[0]);
    const bool multi = o[1] == Py_True;
    const at::Tensor *mixed = plain(o[2]), *a = plain(o[3]), *b = plain(o[4]), *A_log = plain(o[5]), *dt_bias = plain(o[6]);
    const at::Tensor *sc = plain(o[8]), *ss = plain(o[9]), *rc = plain(o[10]), *rs = plain(o[11]), *out = plain(o[12]), *idx = plain(o[13]);
    if (!tab || !mixed || !a || !b || !A_log || !dt_bias || !sc || !ss || !rc || !rs || !out || !idx) return nullptr;
    if (!sc->is_cuda() || sc->dim() != 4) return nullptr;
    const int dev = sc->get_device();
    const int lead = multi ? 3 : 2;                     // [B, W] or [B, T, W]
    const int64_t slots = sc->size(0), HV = sc->size(1), V = sc->size(2), K = sc->size(3);
    if (mixed->dim() != lead || mixed->stride(-1) != 1 || a->dim() != lead || b->dim() != lead) return nullptr;
    const int64_t B = mixed->size(0), T = multi ? mixed->size(1) : 1, W = mixed->size(-1);
    if (!fits32(B) || !fits32(T) || !fits32(HV) || !fits32(V) || !fits32(K) || !fits32(slots)) return nullptr;

    long fmt;
    if (!as_int(o[15], fmt) || (fmt != 0 && fmt != 1)) return nullptr;       // RESID_INT8, RESID_INT4
    const bool int4 = fmt == 1;
    if (int4 && K % 2) return nullptr;
    const int64_t rk = int4 ? K / 2 : K;
    const int rdim = static_cast<int>(rs->dim());
    if (rdim != 2 && rdim != 3) return nullptr;
    if (!is(sc, at::kChar, dev) || !is(rc, at::kChar, dev) || !is(ss, at::kFloat, dev) || !is(rs, at::kFloat, dev) ||
        !is(idx, at::kInt, dev))
      return nullptr;
    if (!shaped(*rc, {slots, HV, V, rk}) || !shaped(*ss, {slots, HV, V})) return nullptr;
    if (rdim == 3 ? !shaped(*rs, {slots, HV, V}) : !shaped(*rs, {slots, HV})) return nullptr;
    if (!dense_inside(*sc, {V * K, K, 1}) || !dense_inside(*rc, {V * rk, rk, 1}) || !dense_inside(*ss, {V, 1})) return nullptr;
    if (rdim == 3 ? !dense_inside(*rs, {V, 1}) : !dense_inside(*rs, {1})) return nullptr;
    if (idx->dim() != 1 || idx->size(0) != B) return nullptr;

    const int64_t qk = W - HV * V;
    if (qk <= 0 || qk % (2 * K)) return nullptr;
    const int64_t H = qk / (2 * K);
    if (H <= 0 || HV % H) return nullptr;
    const int qd = dtype_id(mixed->scalar_type()), ad = dtype_id(a->scalar_type()), od = dtype_id(out->scalar_type());
    const int Ad = dtype_id(A_log->scalar_type()), dd = dtype_id(dt_bias->scalar_type());
    if (qd < 0 || ad < 0 || od < 0 || Ad < 0 || dd < 0) return nullptr;
    if (!is(mixed, mixed->scalar_type(), dev) || !is(a, a->scalar_type(), dev) || !is(b, a->scalar_type(), dev) ||
        !is(out, out->scalar_type(), dev) || !is(A_log, A_log->scalar_type(), dev) || !is(dt_bias, dt_bias->scalar_type(), dev))
      return nullptr;
    if (a->stride(-1) != 1 || b->stride(-1) != 1) return nullptr;
    if (multi ? (!shaped(*a, {B, T, HV}) || !shaped(*b, {B, T, HV})) : (!shaped(*a, {B, HV}) || !shaped(*b, {B, HV}))) return nullptr;
    if (!shaped(*A_log, {HV}) || !shaped(*dt_bias, {HV}) || !A_log->is_contiguous() || !dt_bias->is_contiguous()) return nullptr;
    if (!shaped(*out, {B, T, HV, V}) || !out->is_contiguous()) return nullptr;

    CarryGdnPackedMultiArgs m = {};
    CarryGdnPackedArgs& p = m.step;
    if (!status_of(o[16], dev, &p.status)) return nullptr;
    const double scale = PyFloat_AsDouble(o[7]);
    if (scale == -1.0 && PyErr_Occurred()) return nullptr;
    const int l2 = PyObject_IsTrue(o[14]);
    if (l2 < 0) return nullptr;
    p.mixed_qkv = mixed->data_ptr(); p.stride_mixed_tok = mixed->stride(0); p.qkv_dtype = qd;
    p.a = a->data_ptr(); p.stride_a_tok = a->stride(0);
    p.b = b->data_ptr(); p.stride_b_tok = b->stride(0); p.ab_dtype = ad;
    p.A_log = A_log->data_ptr(); p.A_log_dtype = Ad;
    p.dt_bias = dt_bias->data_ptr(); p.dt_bias_dtype = dd;
    p.scale = static_cast<float>(scale);
    p.state_codes = static_cast<int8_t*>(sc->data_ptr()); p.state_scale = static_cast<float*>(ss->data_ptr());
    p.resid_codes = static_cast<int8_t*>(rc->data_ptr()); p.resid_scale = static_cast<float*>(rs->data_ptr());
    p.stride_state_slot = sc->stride(0); p.stride_resid_slot = rc->stride(0);
    p.stride_sscale_slot = ss->stride(0); p.stride_rscale_slot = rs->stride(0);
    p.out = out->data_ptr(); p.out_dtype = od;
    p.ssm_state_indices = static_cast<const int32_t*>(idx->data_ptr()); p.stride_indices = idx->stride(0);
    p.B = static_cast<int32_t>(B); p.H = static_cast<int32_t>(H); p.HV = static_cast<int32_t>(HV);
    p.K = static_cast<int32_t>(K); p.V = static_cast<int32_t>(V); p.num_slots = static_cast<int32_t>(slots);
    p.use_qk_l2norm = l2;
    p.res_fmt = int4 ? CARRY_RES_INT4 : CARRY_RES_INT8;
    p.resid_scale_mode = rdim == 3 ? CARRY_SCALE_PER_V : CARRY_SCALE_PER_HEAD;
    p.eps_mode = CARRY_EPS_ON_SCALE;
    p.qmax = 127.0f;
    bool ok;
    if (multi) {
      m.T = static_cast<int32_t>(T);
      m.stride_mixed_t = mixed->stride(1); m.stride_a_t = a->stride(1); m.stride_b_t = b->stride(1);
      ok = launch(dev, [&](void* s) { return tab->packed_decode_multi(&m, s); });
    } else {
      ok = launch(dev, [&](void* s) { return tab->packed_decode(&p, s); });
    }
    return ok ? Py_NewRef(Py_True) : nullptr;
  });
}

// ---------------------------------------------------------------------------
// the statequant op
// ---------------------------------------------------------------------------

struct StepShape {
  int dev;
  int64_t B, HV, K, V;
};

// Fills what the step shares between one token and a chain of them; q, k, v, alpha, beta are left to the caller.
bool step_state(const at::Tensor* h, const at::Tensor* scale, const at::Tensor* e, const at::Tensor* es, long bits, long fmt,
                bool resid_per_v, bool state_per_v, StepShape& sh, CarryGdnStepArgs& p) {
  if (!h || !scale || h->dim() != 4 || !h->is_cuda()) return false;
  sh = {h->get_device(), h->size(0), h->size(1), h->size(2), h->size(3)};
  if (!fits32(sh.B) || !fits32(sh.HV) || !fits32(sh.K) || !fits32(sh.V)) return false;
  if (!is(h, at::kChar, sh.dev) || !h->is_contiguous() || !is(scale, at::kFloat, sh.dev) || !scale->is_contiguous()) return false;
  if (state_per_v ? !shaped(*scale, {sh.B, sh.HV, sh.V}) : !shaped(*scale, {sh.B, sh.HV})) return false;
  if (bits < 2 || bits > 8 || fmt < CARRY_RES_FP32 || fmt > CARRY_RES_NONE) return false;
  const bool int_resid = fmt == CARRY_RES_INT8 || fmt == CARRY_RES_INT4;
  if ((fmt == CARRY_RES_NONE) != (e == nullptr) || int_resid != (es != nullptr)) return false;
  if (e) {
    static const at::ScalarType kinds[] = {at::kFloat, at::kHalf, at::kFloat8_e5m2, at::kChar, at::kChar};
    if (fmt == CARRY_RES_INT4 && sh.V % 2) return false;
    if (!is(e, kinds[fmt], sh.dev) || !e->is_contiguous() ||
        !shaped(*e, {sh.B, sh.HV, sh.K, fmt == CARRY_RES_INT4 ? sh.V / 2 : sh.V}))
      return false;
  }
  if (es) {
    if (!is(es, at::kFloat, sh.dev) || !es->is_contiguous()) return false;
    if (resid_per_v ? !shaped(*es, {sh.B, sh.HV, sh.V}) : !shaped(*es, {sh.B, sh.HV})) return false;
  }
  p.h_in = static_cast<const int8_t*>(h->data_ptr());
  p.scale_in = static_cast<const float*>(scale->data_ptr());
  p.e_in = e ? e->data_ptr() : nullptr;
  p.e_scale_in = es ? static_cast<const float*>(es->data_ptr()) : nullptr;
  p.B = static_cast<int32_t>(sh.B); p.HV = static_cast<int32_t>(sh.HV);
  p.K = static_cast<int32_t>(sh.K); p.V = static_cast<int32_t>(sh.V);
  p.o_dtype = CARRY_F32;
  p.qmax = static_cast<float>((1 << (bits - 1)) - 1);
  p.res_fmt = static_cast<int32_t>(fmt);
  p.resid_scale_mode = resid_per_v ? CARRY_SCALE_PER_V : CARRY_SCALE_PER_HEAD;
  p.state_scale_mode = state_per_v ? CARRY_SCALE_PER_V : CARRY_SCALE_PER_HEAD;
  p.eps_mode = CARRY_EPS_ON_AMAX;
  return true;
}

// q, k, v of one element type that the kernels read as it is, alpha and beta fp32, all contiguous
int activations(const at::Tensor* q, const at::Tensor* k, const at::Tensor* v, const at::Tensor* alpha, const at::Tensor* beta, int dev) {
  if (!q || !k || !v) return -1;
  const int d = dtype_id(q->scalar_type());
  if (d < 0 || !is(q, q->scalar_type(), dev) || !is(k, q->scalar_type(), dev) || !is(v, q->scalar_type(), dev) ||
      !is(alpha, at::kFloat, dev) || !is(beta, at::kFloat, dev))
    return -1;
  for (const at::Tensor* t : {q, k, v, alpha, beta})
    if (!t->is_contiguous()) return -1;
  return d;
}

at::Tensor fresh(at::IntArrayRef sizes, at::ScalarType dt, int dev) {
  return at::detail::empty_cuda(sizes, dt, c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(dev)), std::nullopt);
}

PyObject* tuple_of(std::initializer_list<const at::Tensor*> ts) {
  PyObject* r = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
  if (!r) return nullptr;
  Py_ssize_t i = 0;
  for (const at::Tensor* t : ts) {
    PyObject* x = t && t->defined() ? THPVariable_Wrap(*t) : Py_NewRef(Py_None);
    if (!x) { Py_DECREF(r); return nullptr; }
    PyTuple_SET_ITEM(r, i++, x);
  }
  return r;
}

// (table, h_int8, scale, e, e_scale, q, k, v, alpha, beta, bits, res_fmt, resid_per_v, state_per_v)
//   -> (o, h_new, scale_new, e_new, e_scale_new)
PyObject* quant_step(PyObject*, PyObject* const* o, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 14) return nullptr;
    const Table* tab = table_of(o[0]);
    long bits, fmt;
    if (!tab || !as_int(o[10], bits) || !as_int(o[11], fmt)) return nullptr;
    const bool int_resid = fmt == CARRY_RES_INT8 || fmt == CARRY_RES_INT4;
    const at::Tensor *h = plain(o[1]), *scale = plain(o[2]);
    const at::Tensor* e = fmt == CARRY_RES_NONE ? nullptr : plain(o[3]);
    const at::Tensor* es = int_resid ? plain(o[4]) : nullptr;
    if ((int_resid && !es) || (fmt != CARRY_RES_NONE && !e)) return nullptr;
    StepShape sh;
    CarryGdnStepArgs p = {};
    if (!step_state(h, scale, e, es, bits, fmt, o[12] == Py_True, o[13] == Py_True, sh, p)) return nullptr;
    const at::Tensor *q = plain(o[5]), *k = plain(o[6]), *v = plain(o[7]), *alpha = plain(o[8]), *beta = plain(o[9]);
    p.qkv_dtype = activations(q, k, v, alpha, beta, sh.dev);
    if (p.qkv_dtype < 0) return nullptr;
    if (!shaped(*q, {sh.B, sh.HV, sh.K}) || !shaped(*k, {sh.B, sh.HV, sh.K}) || !shaped(*v, {sh.B, sh.HV, sh.V}) ||
        !shaped(*alpha, {sh.B, sh.HV}) || !shaped(*beta, {sh.B, sh.HV}))
      return nullptr;
    p.q = q->data_ptr(); p.k = k->data_ptr(); p.v = v->data_ptr();
    p.alpha = static_cast<const float*>(alpha->data_ptr()); p.beta = static_cast<const float*>(beta->data_ptr());
    const at::Tensor out = fresh({sh.B, sh.HV, sh.V}, at::kFloat, sh.dev), h_new = fresh(h->sizes(), at::kChar, sh.dev);
    const at::Tensor scale_new = fresh(scale->sizes(), at::kFloat, sh.dev);
    at::Tensor e_new, es_new;
    if (e) e_new = fresh(e->sizes(), e->scalar_type(), sh.dev);
    if (es) es_new = fresh(es->sizes(), at::kFloat, sh.dev);
    p.o = out.data_ptr();
    p.h_out = static_cast<int8_t*>(h_new.data_ptr());
    p.scale_out = static_cast<float*>(scale_new.data_ptr());
    p.e_out = e ? e_new.data_ptr() : nullptr;
    p.e_scale_out = es ? static_cast<float*>(es_new.data_ptr()) : nullptr;
    if (!launch(sh.dev, [&](void* s) { return tab->quant_step(&p, s); })) return nullptr;
    return tuple_of({&out, &h_new, &scale_new, &e_new, &es_new});
  });
}

// T chained steps on a state that the caller owns, in place (every kernel reads a tile before it writes it).
// (table, h_int8, scale, e, e_scale, q, k, v, alpha, beta, T, bits, res_fmt, resid_per_v, state_per_v) -> o [T, B, HV, V]
PyObject* quant_decode(PyObject*, PyObject* const* o, Py_ssize_t n) {
  int late = 0;
  PyObject* r = guarded([&]() -> PyObject* {
    if (n != 15) return nullptr;
    const Table* tab = table_of(o[0]);
    long T, bits, fmt;
    if (!tab || !as_int(o[10], T) || !as_int(o[11], bits) || !as_int(o[12], fmt) || T < 1) return nullptr;
    const at::Tensor *h = plain(o[1]), *scale = plain(o[2]);
    const at::Tensor* e = o[3] == Py_None ? nullptr : plain(o[3]);
    const at::Tensor* es = o[4] == Py_None ? nullptr : plain(o[4]);
    StepShape sh;
    CarryGdnStepArgs p = {};
    if (!step_state(h, scale, e, es, bits, fmt, o[13] == Py_True, o[14] == Py_True, sh, p)) return nullptr;
    const at::Tensor *q = plain(o[5]), *k = plain(o[6]), *v = plain(o[7]), *alpha = plain(o[8]), *beta = plain(o[9]);
    p.qkv_dtype = activations(q, k, v, alpha, beta, sh.dev);
    if (p.qkv_dtype < 0) return nullptr;
    if (q->dim() != 4 || k->dim() != 4 || v->dim() != 4 || alpha->dim() != 3 || beta->dim() != 3) return nullptr;
    for (const at::Tensor* t : {q, k, v, alpha, beta})
      if (t->size(0) < T || t->size(1) != sh.B || t->size(2) != sh.HV) return nullptr;
    if (q->size(3) != sh.K || k->size(3) != sh.K || v->size(3) != sh.V) return nullptr;
    const at::Tensor out = fresh({T, sh.B, sh.HV, sh.V}, at::kFloat, sh.dev);
    p.h_out = const_cast<int8_t*>(p.h_in);
    p.scale_out = const_cast<float*>(p.scale_in);
    p.e_out = const_cast<void*>(p.e_in);
    p.e_scale_out = const_cast<float*>(p.e_scale_in);
    const int64_t gates = sh.B * sh.HV, qrow = gates * sh.K, vrow = gates * sh.V, es_ = q->element_size();
    const bool ok = launch(sh.dev, [&](void* s) {
      for (long t = 0; t < T; ++t) {
        p.q = static_cast<const char*>(q->data_ptr()) + t * qrow * es_;
        p.k = static_cast<const char*>(k->data_ptr()) + t * qrow * es_;
        p.v = static_cast<const char*>(v->data_ptr()) + t * vrow * es_;
        p.alpha = static_cast<const float*>(alpha->data_ptr()) + t * gates;
        p.beta = static_cast<const float*>(beta->data_ptr()) + t * gates;
        p.o = static_cast<float*>(out.data_ptr()) + t * vrow;
        // an error at the first step leaves the state as it was; a later one (a launch that the runtime
        // refused) does not, so the call cannot be handed back
        const int rc = tab->quant_step(&p, s);
        if (rc != CARRY_GDN_OK) {
          if (t > 0) late = rc;
          return rc;
        }
      }
      return 0;
    });
    return ok ? THPVariable_Wrap(out) : nullptr;
  });
  if (late) {
    Py_DECREF(r);
    return PyErr_Format(PyExc_RuntimeError, "carry_gdn_quant_step failed in a chain of steps (code %d)", late);
  }
  return r;
}

// The same from a floating-point state, all in one launch, for what the library's chain kernel takes.
// (table, h0, q, k, v, alpha, beta, T, bits, res_fmt) -> (o [T, B, HV, V], h_int8, scale, e)
PyObject* quant_chain(PyObject*, PyObject* const* o, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 10) return nullptr;
    const Table* tab = table_of(o[0]);
    const at::Tensor* h0 = plain(o[1]);
    long T, bits, fmt;
    if (!tab || !as_int(o[7], T) || !as_int(o[8], bits) || !as_int(o[9], fmt) || !fits32(T)) return nullptr;
    if (!h0 || h0->dim() != 4 || !h0->is_cuda() || !h0->is_contiguous() || h0->scalar_type() != at::kFloat) return nullptr;
    // what the kernel takes, looked at before anything is allocated
    if (fmt < CARRY_RES_FP32 || fmt > CARRY_RES_FP8 || bits < 3 || bits > 8 || h0->size(2) != 128 || h0->size(3) != 128) return nullptr;
    const int dev = h0->get_device();
    const int64_t B = h0->size(0), HV = h0->size(1), K = 128, V = 128;
    if (!fits32(B) || !fits32(HV)) return nullptr;
    static const at::ScalarType kinds[] = {at::kFloat, at::kHalf, at::kFloat8_e5m2};
    const at::Tensor *q = plain(o[2]), *k = plain(o[3]), *v = plain(o[4]), *alpha = plain(o[5]), *beta = plain(o[6]);
    CarryGdnDecodeArgs a = {};
    CarryGdnStepArgs& p = a.step;
    p.qkv_dtype = activations(q, k, v, alpha, beta, dev);
    if (p.qkv_dtype < 0 || q->dim() != 4 || k->dim() != 4 || v->dim() != 4 || alpha->dim() != 3 || beta->dim() != 3) return nullptr;
    for (const at::Tensor* t : {q, k, v, alpha, beta})
      if (t->size(0) < T || t->size(1) != B || t->size(2) != HV) return nullptr;
    if (q->size(3) != K || k->size(3) != K || v->size(3) != V) return nullptr;
    const at::Tensor out = fresh({T, B, HV, V}, at::kFloat, dev), h = fresh({B, HV, K, V}, at::kChar, dev);
    const at::Tensor scale = fresh({B, HV, V}, at::kFloat, dev), e = fresh({B, HV, K, V}, kinds[fmt], dev);
    a.h0 = static_cast<const float*>(h0->data_ptr());
    a.T = static_cast<int32_t>(T);
    p.q = q->data_ptr(); p.k = k->data_ptr(); p.v = v->data_ptr();
    p.alpha = static_cast<const float*>(alpha->data_ptr()); p.beta = static_cast<const float*>(beta->data_ptr());
    p.o = out.data_ptr();
    p.h_out = static_cast<int8_t*>(h.data_ptr());
    p.scale_out = static_cast<float*>(scale.data_ptr());
    p.e_out = e.data_ptr();
    p.B = static_cast<int32_t>(B); p.HV = static_cast<int32_t>(HV); p.K = K; p.V = V;
    p.o_dtype = CARRY_F32;
    p.qmax = static_cast<float>((1 << (bits - 1)) - 1);
    p.res_fmt = static_cast<int32_t>(fmt);
    p.resid_scale_mode = p.state_scale_mode = CARRY_SCALE_PER_V;
    p.eps_mode = CARRY_EPS_ON_AMAX;
    if (!launch(dev, [&](void* s) { return tab->quant_decode(&a, s); })) return nullptr;
    return tuple_of({&out, &h, &scale, &e});
  });
}

// (table, h, q, k, v, alpha, beta) -> (h_out, o)
PyObject* fp32_step(PyObject*, PyObject* const* o, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 7) return nullptr;
    const Table* tab = table_of(o[0]);
    const at::Tensor* h = plain(o[1]);
    if (!tab || !h || h->dim() != 4 || !h->is_cuda()) return nullptr;
    const int dev = h->get_device();
    const int64_t B = h->size(0), HV = h->size(1), K = h->size(2), V = h->size(3);
    if (!fits32(B) || !fits32(HV) || !fits32(K) || !fits32(V) || !is(h, at::kFloat, dev) || !h->is_contiguous()) return nullptr;
    const at::Tensor *q = plain(o[2]), *k = plain(o[3]), *v = plain(o[4]), *alpha = plain(o[5]), *beta = plain(o[6]);
    CarryGdnFp32Args p = {};
    p.qkv_dtype = activations(q, k, v, alpha, beta, dev);
    if (p.qkv_dtype < 0) return nullptr;
    if (!shaped(*q, {B, HV, K}) || !shaped(*k, {B, HV, K}) || !shaped(*v, {B, HV, V}) || !shaped(*alpha, {B, HV}) ||
        !shaped(*beta, {B, HV}))
      return nullptr;
    const at::Tensor out = fresh({B, HV, V}, at::kFloat, dev), h_out = fresh(h->sizes(), at::kFloat, dev);
    p.h_in = static_cast<const float*>(h->data_ptr());
    p.q = q->data_ptr(); p.k = k->data_ptr(); p.v = v->data_ptr();
    p.alpha = static_cast<const float*>(alpha->data_ptr()); p.beta = static_cast<const float*>(beta->data_ptr());
    p.o = out.data_ptr();
    p.h_out = static_cast<float*>(h_out.data_ptr());
    p.B = static_cast<int32_t>(B); p.HV = static_cast<int32_t>(HV); p.K = static_cast<int32_t>(K); p.V = static_cast<int32_t>(V);
    p.o_dtype = CARRY_F32;
    if (!launch(dev, [&](void* s) { return tab->fp32_step(&p, s); })) return nullptr;
    return tuple_of({&h_out, &out});
  });
}

// ---------------------------------------------------------------------------
// the slot pool
// ---------------------------------------------------------------------------

// A pool is a tuple or list of four tensors; `dev` is set from the first pool of a call (-1 on entry).
bool pool_of(PyObject* o, long fmt, int& dev, CarryGdnPool& p) {
  if (!PyTuple_CheckExact(o) && !PyList_CheckExact(o)) return false;
  if (PySequence_Fast_GET_SIZE(o) != 4 || (fmt != 0 && fmt != 1)) return false;
  PyObject** it = PySequence_Fast_ITEMS(o);
  const at::Tensor *sc = plain(it[0]), *ss = plain(it[1]), *rc = plain(it[2]), *rs = plain(it[3]);
  if (!sc || !ss || !rc || !rs || sc->dim() != 4 || !sc->is_cuda()) return false;
  if (dev < 0) dev = sc->get_device();
  const int64_t slots = sc->size(0), HV = sc->size(1), V = sc->size(2), K = sc->size(3);
  if (!fits32(slots) || !fits32(HV) || !fits32(V) || !fits32(K) || (fmt == 1 && K % 2)) return false;
  const int64_t rk = fmt == 1 ? K / 2 : K;
  const int rdim = static_cast<int>(rs->dim());
  if (rdim != 2 && rdim != 3) return false;
  if (!is(sc, at::kChar, dev) || !is(rc, at::kChar, dev) || !is(ss, at::kFloat, dev) || !is(rs, at::kFloat, dev)) return false;
  if (!shaped(*rc, {slots, HV, V, rk}) || !shaped(*ss, {slots, HV, V})) return false;
  if (rdim == 3 ? !shaped(*rs, {slots, HV, V}) : !shaped(*rs, {slots, HV})) return false;
  if (!dense_inside(*sc, {V * K, K, 1}) || !dense_inside(*rc, {V * rk, rk, 1}) || !dense_inside(*ss, {V, 1})) return false;
  if (rdim == 3 ? !dense_inside(*rs, {V, 1}) : !dense_inside(*rs, {1})) return false;
  p.state_codes = static_cast<int8_t*>(sc->data_ptr()); p.state_scale = static_cast<float*>(ss->data_ptr());
  p.resid_codes = static_cast<int8_t*>(rc->data_ptr()); p.resid_scale = static_cast<float*>(rs->data_ptr());
  p.stride_state_slot = sc->stride(0); p.stride_resid_slot = rc->stride(0);
  p.stride_sscale_slot = ss->stride(0); p.stride_rscale_slot = rs->stride(0);
  p.num_slots = static_cast<int32_t>(slots); p.HV = static_cast<int32_t>(HV);
  p.V = static_cast<int32_t>(V); p.K = static_cast<int32_t>(K);
  p.res_fmt = fmt == 1 ? CARRY_RES_INT4 : CARRY_RES_INT8;
  p.resid_scale_mode = rdim == 3 ? CARRY_SCALE_PER_V : CARRY_SCALE_PER_HEAD;
  return true;
}
const at::Tensor* ids_of(PyObject* o, int dev) {
  const at::Tensor* t = plain(o);
  return is(t, at::kInt, dev) && t->dim() == 1 && fits32(t->size(0)) ? t : nullptr;
}
bool same_shape(const CarryGdnPool& a, const CarryGdnPool& b) {
  return a.HV == b.HV && a.V == b.V && a.K == b.K && a.res_fmt == b.res_fmt && a.resid_scale_mode == b.resid_scale_mode;
}

// a floating-point state [B, HV, V, K], dense within a request
int state_of(PyObject* o, int64_t B, const CarryGdnPool& p, int dev, const at::Tensor** out) {
  const at::Tensor* h = plain(o);
  if (!h || h->dim() != 4 || !is(h, h->scalar_type(), dev)) return -1;
  if (!shaped(*h, {B, p.HV, p.V, p.K}) || !dense_inside(*h, {static_cast<int64_t>(p.V) * p.K, p.K, 1})) return -1;
  *out = h;
  return dtype_id(h->scalar_type());
}

// (table, store, h, pool, indices, resid_fmt, keep_error / with_residual, status) -> True
PyObject* pool_move(PyObject*, PyObject* const* o, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 8) return nullptr;
    const Table* tab = table_of(o[0]);
    const bool store = o[1] == Py_True;
    long fmt;
    if (!tab || !as_int(o[5], fmt)) return nullptr;
    int dev = -1;
    CarryGdnPool pool = {};
    if (!pool_of(o[3], fmt, dev, pool)) return nullptr;
    const at::Tensor *idx = ids_of(o[4], dev), *h = nullptr;
    if (!idx) return nullptr;
    const int hd = state_of(o[2], idx->size(0), pool, dev, &h);
    const int flag = PyObject_IsTrue(o[6]);
    int32_t* status;
    if (hd < 0 || flag < 0 || !status_of(o[7], dev, &status)) return nullptr;
    const int32_t* slots = static_cast<const int32_t*>(idx->data_ptr());
    const int32_t B = static_cast<int32_t>(idx->size(0));
    bool ok;
    if (store) {
      CarryGdnPoolStoreArgs a = {pool, h->data_ptr(), h->stride(0), hd, slots, idx->stride(0), B, flag, 127.0f, status};
      ok = launch(dev, [&](void* s) { return tab->pool_store(&a, s); });
    } else {
      CarryGdnPoolLoadArgs a = {pool, h->data_ptr(), h->stride(0), hd, slots, idx->stride(0), B, flag, status};
      ok = launch(dev, [&](void* s) { return tab->pool_load(&a, s); });
    }
    return ok ? Py_NewRef(Py_True) : nullptr;
  });
}

// (table, src_pool, dst_pool, src_indices, dst_indices, resid_fmt, status) -> True
PyObject* pool_copy(PyObject*, PyObject* const* o, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 7) return nullptr;
    const Table* tab = table_of(o[0]);
    long fmt;
    if (!tab || !as_int(o[5], fmt)) return nullptr;
    int dev = -1;
    CarryGdnPoolCopyArgs a = {};
    if (!pool_of(o[1], fmt, dev, a.src) || !pool_of(o[2], fmt, dev, a.dst) || !same_shape(a.src, a.dst)) return nullptr;
    const at::Tensor *from = ids_of(o[3], dev), *to = ids_of(o[4], dev);
    if (!from || !to || from->size(0) != to->size(0) || !status_of(o[6], dev, &a.status)) return nullptr;
    a.src_slots = static_cast<const int32_t*>(from->data_ptr()); a.stride_src_slots = from->stride(0);
    a.dst_slots = static_cast<const int32_t*>(to->data_ptr()); a.stride_dst_slots = to->stride(0);
    a.B = static_cast<int32_t>(from->size(0));
    return launch(dev, [&](void* s) { return tab->pool_copy(&a, s); }) ? Py_NewRef(Py_True) : nullptr;
  });
}

// One slot of every layer's pool to a slot of another list of pools (a SlotCache move).
// (table, src_layers, src_slot, dst_layers, dst_slot, resid_fmt) -> True
PyObject* pool_copy_layers(PyObject*, PyObject* const* o, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 6) return nullptr;
    const Table* tab = table_of(o[0]);
    long from, to, fmt;
    if (!tab || !as_int(o[2], from) || !as_int(o[4], to) || !as_int(o[5], fmt)) return nullptr;
    if (!PyList_CheckExact(o[1]) || !PyList_CheckExact(o[3])) return nullptr;
    const Py_ssize_t L = PyList_GET_SIZE(o[1]);
    if (L < 1 || L != PyList_GET_SIZE(o[3])) return nullptr;
    std::vector<CarryGdnPool> pools(static_cast<size_t>(2 * L));
    int dev = -1;
    for (Py_ssize_t i = 0; i < L; ++i) {
      CarryGdnPool &s = pools[static_cast<size_t>(i)], &d = pools[static_cast<size_t>(L + i)];
      if (!pool_of(PyList_GET_ITEM(o[1], i), fmt, dev, s) || !pool_of(PyList_GET_ITEM(o[3], i), fmt, dev, d)) return nullptr;
      if (!same_shape(s, pools[0]) || !same_shape(d, pools[0])) return nullptr;
      if (from <= 0 || from >= s.num_slots || to <= 0 || to >= d.num_slots) return nullptr;
    }
    CarryGdnPoolCopyLayersArgs a = {pools.data(), pools.data() + L, static_cast<int32_t>(L), static_cast<int32_t>(from),
                                    static_cast<int32_t>(to)};
    return launch(dev, [&](void* s) { return tab->pool_copy_layers(&a, s); }) ? Py_NewRef(Py_True) : nullptr;
  });
}

// (address of each entry point, in the order of Table) -> the table's address; it lives as long as the process
PyObject* make_table(PyObject*, PyObject* const* o, Py_ssize_t n) {
  if (n != kEntries) {
    PyErr_SetString(PyExc_ValueError, "make_table: wrong number of entry points");
    return nullptr;
  }
  void* at[kEntries];
  for (int i = 0; i < kEntries; ++i) {
    at[i] = PyLong_AsVoidPtr(o[i]);
    if (!at[i]) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "make_table: null entry point");
      return nullptr;
    }
  }
  static_assert(sizeof(Table) == sizeof(at), "Table is nothing but entry points");
  Table* t = new Table;
  memcpy(t, at, sizeof(at));
  return PyLong_FromVoidPtr(t);
}

#define CARRY_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {CARRY_FAST(make_table), CARRY_FAST(packed_decode), CARRY_FAST(quant_step), CARRY_FAST(quant_decode), CARRY_FAST(quant_chain),
                         CARRY_FAST(fp32_step), CARRY_FAST(pool_move), CARRY_FAST(pool_copy), CARRY_FAST(pool_copy_layers),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Native call path of the Python surfaces.", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
