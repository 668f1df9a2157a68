// CPython extension over the C ABI: the argument marshalling of the hot launchers (kv4.py, kvx.py) in native code.
//
// What bounds it: a decode step of a few microseconds on the GPU is two or three calls from Python.  Building the argument
// structs through ctypes (attribute look-ups, data_ptr() calls, nested Structure constructors, one checked conversion per
// argument) took 8-10 us a call; here a call reads the tensors' C++ objects directly and takes about 1 us beside the launch itself.
// Checks and exception types are those of the Python code it replaces: AssertionError for buffers that do not fit, AttributeError (NotATensor,
// also a TypeError) for what is no tensor, TypeError / ValueError for types and shapes, Kv4Error with the library's message for a rejected
// call, a missing buffer (None) among them where the launcher left that check to the library.  Integers beyond a C int raise OverflowError
// (ctypes cut them off).  The library call itself runs without the interpreter lock, as a ctypes call does.
#include <torch/csrc/autograd/python_variable.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <cstdlib>
#include "../../include/yskn_kv4_abi.h"

namespace {

PyObject *g_kv4_error = nullptr, *g_not_a_tensor = nullptr;
struct Names { PyObject *kq, *kscale, *kzero, *kshadow, *vq, *vscale, *vzero, *hkv, *hd, *max_ctx, *cuda_stream, *maps_ptr, *d_layers, *n, *dev; } N;

struct PyFail {};                                       // a Python exception is set
[[noreturn]] void fail(PyObject* type, const char* msg) { PyErr_SetString(type, msg); throw PyFail{}; }

const at::Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) { PyErr_Format(g_not_a_tensor, "%s: '%s' object is not a tensor", what, Py_TYPE(o)->tp_name); throw PyFail{}; }
  return THPVariable_Unpack(o);
}
void check_dev(const at::Tensor& t, const char* what) {
  if (!t.is_cuda() || !t.is_contiguous()) { PyErr_Format(PyExc_AssertionError, "%s: device buffers must be contiguous CUDA tensors", what); throw PyFail{}; }
}
void* dev_ptr(PyObject* o, const char* what) { const at::Tensor& t = tensor(o, what); check_dev(t, what); return t.data_ptr(); }
void* raw_ptr(PyObject* o, const char* what) { return tensor(o, what).data_ptr(); }
void* opt_dev(PyObject* o, const char* what) { return o == Py_None ? nullptr : dev_ptr(o, what); }
void* opt_raw(PyObject* o, const char* what) { return o == Py_None ? nullptr : raw_ptr(o, what); }

long long_of(PyObject* o) { const long v = PyLong_AsLong(o); if (v == -1 && PyErr_Occurred()) throw PyFail{}; return v; }
int int_of(PyObject* o) {
  const long v = long_of(o);
  if (v != (int)v) fail(PyExc_OverflowError, "an argument does not fit a C int");
  return (int)v;
}
float float_of(PyObject* o) { const double v = PyFloat_AsDouble(o); if (v == -1.0 && PyErr_Occurred()) throw PyFail{}; return (float)v; }
struct Ref { PyObject* p; explicit Ref(PyObject* o) : p(o) { if (!p) throw PyFail{}; } ~Ref() { Py_DECREF(p); } Ref(const Ref&) = delete; };
Ref attr(PyObject* o, PyObject* name) { return Ref(PyObject_GetAttr(o, name)); }

cudaStream_t stream_of(PyObject* o) {
  if (o == Py_None) return c10::cuda::getCurrentCUDAStream().stream();
  return (cudaStream_t)PyLong_AsVoidPtr(attr(o, N.cuda_stream).p);
}
int dtype_code(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kHalf: return YSKN_KV4_F16;
    case at::kBFloat16: return YSKN_KV4_BF16;
    case at::kFloat: return YSKN_KV4_F32;
    default: fail(PyExc_TypeError, "unsupported activation dtype");
  }
}
void need(bool ok, const char* msg) { if (!ok) fail(PyExc_AssertionError, msg); }

struct Layer { yskn_kv_layer s; int hkv, hd, max_ctx; };
Layer layer_of(PyObject* kv) {
  Layer L;
  L.s.kq = (uint8_t*)raw_ptr(attr(kv, N.kq).p, "kq"); L.s.kscale = (uint16_t*)raw_ptr(attr(kv, N.kscale).p, "kscale");
  L.s.kzero = (uint16_t*)raw_ptr(attr(kv, N.kzero).p, "kzero"); L.s.kshadow = (uint16_t*)raw_ptr(attr(kv, N.kshadow).p, "kshadow");
  L.s.vq = (uint8_t*)raw_ptr(attr(kv, N.vq).p, "vq"); L.s.vscale = (uint16_t*)raw_ptr(attr(kv, N.vscale).p, "vscale");
  L.s.vzero = (uint16_t*)raw_ptr(attr(kv, N.vzero).p, "vzero");
  L.hkv = int_of(attr(kv, N.hkv).p); L.hd = int_of(attr(kv, N.hd).p); L.max_ctx = int_of(attr(kv, N.max_ctx).p);
  return L;
}

// The attention arguments shared by the launchers: q16, kv, M, d_pos, splits, pm, pl, pacc, rope, nh, qscale (a[0] .. a[10]).
struct Attn { yskn_attn_g_args a; Layer L; int g, dt; };
Attn attn_of(PyObject* const* v) {
  Attn A;
  const at::Tensor &q = tensor(v[0], "q16"), &dpos = tensor(v[3], "d_pos"), &pm = tensor(v[5], "pm"), &pl = tensor(v[6], "pl"), &pacc = tensor(v[7], "pacc");
  A.L = layer_of(v[1]);
  const int M = int_of(v[2]), splits = int_of(v[4]), nh = int_of(v[9]);
  need(q.is_cuda() && q.is_contiguous() && q.numel() == (int64_t)M * nh * A.L.hd, "q16: a contiguous CUDA tensor [M][nh][hd]");
  need(pm.numel() >= (int64_t)M * splits * nh && pacc.numel() >= (int64_t)M * splits * nh * A.L.hd && dpos.scalar_type() == at::kInt,
       "pm / pacc too small for (M, splits, nh, hd), or d_pos is not int32");
  if (A.L.hkv == 0) fail(PyExc_ZeroDivisionError, "hkv");
  A.g = nh / A.L.hkv; A.dt = dtype_code(q);
  A.a = yskn_attn_g_args{(const uint16_t*)q.data_ptr(), A.L.s, A.L.max_ctx, M, (const int*)dpos.data_ptr(), splits, (float*)pm.data_ptr(), (float*)pl.data_ptr(),
                         (float*)pacc.data_ptr(), (const float*)opt_raw(v[8], "rope"), A.L.hkv, nh, float_of(v[10])};
  return A;
}

// Runs a library call without the interpreter lock; a non-zero code becomes Kv4Error.
template <class F> PyObject* call(const char* what, F f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f();
  Py_END_ALLOW_THREADS
  if (rc) { PyErr_Format(g_kv4_error, "%s failed (code %d): %s", what, rc, yskn_kv4_last_error()); return nullptr; }
  Py_RETURN_NONE;
}
template <class F> PyObject* guarded(Py_ssize_t n, Py_ssize_t want, F f) {
  if (n != want) { PyErr_Format(PyExc_TypeError, "%zd arguments, %zd expected", n, want); return nullptr; }
  try { return f(); } catch (const PyFail&) { return nullptr; } catch (const std::exception& e) { PyErr_SetString(PyExc_RuntimeError, e.what()); return nullptr; }
}

#define FN(name) PyObject* name(PyObject*, PyObject* const* v, Py_ssize_t n)

FN(kv_append) {                                          // kv, k_in, v_in, d_pos, M, stream
  return guarded(n, 6, [&]() -> PyObject* {
    const at::Tensor &k = tensor(v[1], "k_in"), &vv = tensor(v[2], "v_in"), &dpos = tensor(v[3], "d_pos");
    const Layer L = layer_of(v[0]);
    const int M = int_of(v[4]);
    need(k.sizes() == vv.sizes() && k.scalar_type() == vv.scalar_type() && k.numel() == (int64_t)M * L.hkv * L.hd, "k_in, v_in: equal tensors [M][hkv][hd]");
    need(k.is_cuda() && k.is_contiguous() && vv.is_contiguous() && dpos.scalar_type() == at::kInt, "k_in, v_in: contiguous CUDA tensors; d_pos int32");
    const yskn_kv_append_args a{k.data_ptr(), vv.data_ptr(), dtype_code(k), L.s, (const int*)dpos.data_ptr(), M, L.max_ctx, L.hkv, L.hd};
    const cudaStream_t st = stream_of(v[5]);
    return call("yskn_kv4_append", [&] { return yskn_kv4_append(&a, st); });
  });
}

const yskn_kv4_attn_ext* ext_of(PyObject* o, yskn_kv4_attn_ext* out) {       // a ctypes AttnExtC, or None
  if (o == Py_None) return nullptr;
  Py_buffer b;
  if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE)) throw PyFail{};
  const bool ok = b.len == (Py_ssize_t)sizeof(*out);
  if (ok) memcpy(out, b.buf, sizeof(*out));
  PyBuffer_Release(&b);
  if (!ok) fail(PyExc_TypeError, "ext: an AttnExtC is needed");
  return out;
}

FN(attention) {                                          // the eleven of attn_of, rd, stream, ext
  return guarded(n, 14, [&]() -> PyObject* {
    const Attn A = attn_of(v);
    const int rd = int_of(v[11]);
    const cudaStream_t st = stream_of(v[12]);
    yskn_kv4_attn_ext xs;
    const yskn_kv4_attn_ext* x = ext_of(v[13], &xs);
    if (x) return call("yskn_kv4_attention_ex", [&] { return yskn_kv4_attention_ex(&A.a, x, A.g, A.L.hd, rd, A.dt, st); });
    return call("yskn_kv4_attention", [&] { return yskn_kv4_attention(&A.a, A.g, A.L.hd, rd, A.dt, st); });
  });
}

FN(decode) {                                             // the eleven of attn_of, rd, o16, bv, gate, stream, ext
  return guarded(n, 17, [&]() -> PyObject* {
    const Attn A = attn_of(v);
    const int rd = int_of(v[11]);
    const yskn_attn_g_combine_args c{A.a.pm, A.a.pl, A.a.pacc, A.a.splits, A.a.M, (const uint16_t*)opt_raw(v[13], "bv"), (uint16_t*)raw_ptr(v[12], "o16"),
                                     (const uint16_t*)opt_raw(v[14], "gate"), A.a.nh, A.g};
    const cudaStream_t st = stream_of(v[15]);
    yskn_kv4_attn_ext xs;
    const yskn_kv4_attn_ext* x = ext_of(v[16], &xs);
    return call("yskn_kv4_decode", [&] { return yskn_kv4_decode_ex(&A.a, &c, x, A.g, A.L.hd, rd, A.dt, st); });
  });
}

FN(combine) {                                            // pm, pl, pacc, splits, M, o16, nh, g, bv, gate, stream
  return guarded(n, 11, [&]() -> PyObject* {
    const at::Tensor& o = tensor(v[5], "o16");
    const int splits = int_of(v[3]), M = int_of(v[4]), nh = int_of(v[6]), g = int_of(v[7]), dt = dtype_code(o);
    if ((int64_t)M * nh == 0) fail(PyExc_ZeroDivisionError, "M * nh");
    const int hd = (int)(o.numel() / ((int64_t)M * nh));
    const yskn_attn_g_combine_args c{(const float*)raw_ptr(v[0], "pm"), (const float*)raw_ptr(v[1], "pl"), (const float*)raw_ptr(v[2], "pacc"), splits, M,
                                     (const uint16_t*)opt_raw(v[8], "bv"), (uint16_t*)o.data_ptr(), (const uint16_t*)opt_raw(v[9], "gate"), nh, g};
    const cudaStream_t st = stream_of(v[10]);
    return call("yskn_kv4_combine", [&] { return yskn_kv4_combine(&c, hd, dt, st); });
  });
}

FN(attention_ms) {                                       // q16, slots, M, pos, slot, splits, pm, pl, pacc, rope, nh, qscale, rd, stream
  return guarded(n, 14, [&]() -> PyObject* {
    const at::Tensor &q = tensor(v[0], "q16"), &pos = tensor(v[3], "pos"), &slot = tensor(v[4], "slot");
    PyObject* s = v[1];
    const int M = int_of(v[2]), splits = int_of(v[5]), nh = int_of(v[10]), rd = int_of(v[12]);
    need(pos.scalar_type() == at::kInt && slot.scalar_type() == at::kInt && pos.numel() >= M && slot.numel() >= M, "pos, slot: int32 tensors of at least M");
    const int hkv = int_of(attr(s, N.hkv).p), hd = int_of(attr(s, N.hd).p), max_ctx = int_of(attr(s, N.max_ctx).p);
    if (hkv == 0) fail(PyExc_ZeroDivisionError, "hkv");
    const yskn_attn_g_args a{(const uint16_t*)q.data_ptr(), yskn_kv_layer{}, max_ctx, M, nullptr, splits, (float*)raw_ptr(v[6], "pm"), (float*)raw_ptr(v[7], "pl"),
                             (float*)raw_ptr(v[8], "pacc"), (const float*)opt_raw(v[9], "rope"), hkv, nh, float_of(v[11])};
    void* maps = PyLong_AsVoidPtr(attr(s, N.maps_ptr).p);
    const yskn_kv4_ms_rows ms{(const int*)pos.data_ptr(), (const int*)slot.data_ptr(), (const yskn_kv_layer*)raw_ptr(attr(s, N.d_layers).p, "d_layers"), maps,
                              int_of(attr(s, N.n).p)};
    const int dt = dtype_code(q);
    const cudaStream_t st = stream_of(v[13]);
    return call("yskn_kv4_attention_ms", [&] { return yskn_kv4_attention_ms(&a, &ms, nh / hkv, hd, rd, dt, st); });
  });
}

// workspace -> (pointer, length in ELEMENTS: the workspace is a uint8 tensor), as kv4.py passes it
void ws_of(PyObject* o, void** p, size_t* bytes) {
  *p = nullptr; *bytes = 0;
  if (o == Py_None) return;
  *p = dev_ptr(o, "workspace"); *bytes = (size_t)THPVariable_Unpack(o).numel();
}

FN(attention_tc) {                                       // the eleven of attn_of, rd, workspace, valid_tokens, stream
  return guarded(n, 15, [&]() -> PyObject* {
    const Attn A = attn_of(v);
    const int rd = int_of(v[11]), valid = int_of(v[13]);
    void* ws; size_t wb;
    ws_of(v[12], &ws, &wb);
    const cudaStream_t st = stream_of(v[14]);
    return call("yskn_kv4_attention_tc", [&] { return yskn_kv4_attention_tc(&A.a, A.g, A.L.hd, rd, A.dt, ws, wb, valid, st); });
  });
}

FN(prefill_tc) {                                         // the eleven of attn_of, rd, o16, workspace, bv, valid_tokens, stream
  return guarded(n, 17, [&]() -> PyObject* {
    const Attn A = attn_of(v);
    const int rd = int_of(v[11]), valid = int_of(v[15]);
    uint16_t* o16 = (uint16_t*)opt_dev(v[12], "o16");
    const uint16_t* bv = (const uint16_t*)opt_raw(v[14], "bv");
    void* ws; size_t wb;
    ws_of(v[13], &ws, &wb);
    const cudaStream_t st = stream_of(v[16]);
    return call("yskn_kv4_prefill_tc", [&] { return yskn_kv4_prefill_tc(&A.a, A.g, A.L.hd, rd, A.dt, bv, o16, ws, wb, valid, st); });
  });
}

bool is_shape(const at::Tensor& t, int64_t a, int64_t b, int64_t c) { return t.dim() == 3 && t.size(0) == a && t.size(1) == b && t.size(2) == c; }

FN(attn_post) {                                          // q_rows, k_rows, v_rows, qn_w, kn_w, eps, d_pos, rope, rd, q16, gate16, k8, ks, v8, vs, pm, stream
  return guarded(n, 17, [&]() -> PyObject* {
    const at::Tensor &q = tensor(v[0], "q_rows"), &k = tensor(v[1], "k_rows"), &vr = tensor(v[2], "v_rows"), &k8 = tensor(v[11], "k8");
    if (q.dim() < 2 || k8.dim() < 2) fail(PyExc_ValueError, "q_rows [M, nh, 512], k8 [kvh, max_ctx, 256]");
    const int M = (int)q.size(0), nh = (int)q.size(1), kvh = (int)k8.size(0), max_ctx = (int)k8.size(1);
    for (int i : {0, 1, 2, 3, 4, 9, 10})
      if (tensor(v[i], "rows").scalar_type() != at::kBFloat16) fail(PyExc_TypeError, "yskn_kvx_attn_post takes bf16 rows and norm weights");
    if (!is_shape(q, M, nh, 512) || !is_shape(k, M, kvh, 256) || !is_shape(vr, M, kvh, 256)) fail(PyExc_ValueError, "q_rows [M, nh, 512], k_rows / v_rows [M, kvh, 256]");
    auto u16 = [&](int i, const char* w) { return (uint16_t*)dev_ptr(v[i], w); };
    const int pm = PyObject_IsTrue(v[15]);
    if (pm < 0) throw PyFail{};
    const yskn_kvx_attn_post_args a{u16(0, "q_rows"), u16(1, "k_rows"), u16(2, "v_rows"), u16(3, "qn_w"), u16(4, "kn_w"), float_of(v[5]), M,
                                    (const int*)opt_dev(v[6], "d_pos"), (const float*)opt_dev(v[7], "rope"), int_of(v[8]), u16(9, "q16"), u16(10, "gate16"),
                                    (int8_t*)dev_ptr(v[11], "k8"), (int8_t*)opt_dev(v[13], "v8"), (float*)opt_dev(v[12], "ks"), (float*)opt_dev(v[14], "vs"),
                                    max_ctx, nh, kvh, pm};
    const cudaStream_t st = stream_of(v[16]);
    return call("yskn_kvx_attn_post", [&] { return yskn_kvx_attn_post(&a, st); });
  });
}

// Device memory for the work of one call, from torch's caching allocator for the stream the call runs on: given back when the call returns,
// and handed out again only behind this work in that stream.  Straight from the allocator: a tensor would be filled in torch's deterministic mode and
// seen by dispatch modes.  None (the caller's form without it runs) when nothing is asked for, when the stream is being captured (a
// graph outlives the call), when there is no memory, and when torch caches none (every call would wait for the GPU).  Another stream may
// be under capture, in this thread or another: the allocation is no part of it and is made in relaxed mode.
struct Scratch {
  void* p = nullptr;
  size_t bytes = 0;
  Scratch(size_t n, cudaStream_t st) {
    if (!n || getenv("PYTORCH_NO_CUDA_MEMORY_CACHING")) return;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) { (void)cudaGetLastError(); return; }      // the launch itself will tell
    if (cap != cudaStreamCaptureStatusNone) return;
    const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
    try { p = c10::cuda::CUDACachingAllocator::raw_alloc_with_stream(n, st); bytes = n; } catch (const c10::OutOfMemoryError&) {}
  }
  ~Scratch() { if (p) c10::cuda::CUDACachingAllocator::raw_delete(p); }
  Scratch(const Scratch&) = delete;
};

// q16, k8, v8, ks, vs, M, d_pos, splits, pm, pl, pacc, nh, qscale, stream
PyObject* kv8(PyObject* const* v, Py_ssize_t n, const char* who, int (*entry)(const yskn_kv8_attn_args*, int, void*)) {
  return guarded(n, 14, [&]() -> PyObject* {
    const at::Tensor &q = tensor(v[0], "q16"), &k8 = tensor(v[1], "k8");
    if (k8.dim() < 2) fail(PyExc_ValueError, "k8 [kvh, max_ctx, 256]");
    const yskn_kv8_attn_args a{(const uint16_t*)dev_ptr(v[0], "q16"), (const int8_t*)dev_ptr(v[1], "k8"), (const int8_t*)dev_ptr(v[2], "v8"),
                               (const float*)dev_ptr(v[3], "ks"), (const float*)dev_ptr(v[4], "vs"), (int)k8.size(1), int_of(v[5]), (const int*)dev_ptr(v[6], "d_pos"),
                               int_of(v[7]), (float*)dev_ptr(v[8], "pm"), (float*)dev_ptr(v[9], "pl"), (float*)dev_ptr(v[10], "pacc"), (int)k8.size(0),
                               int_of(v[11]), float_of(v[12])};
    const int dt = dtype_code(q);
    const cudaStream_t st = stream_of(v[13]);
    const Scratch ws(yskn_kv8_workspace_bytes(&a), st);
    if (ws.p) return call(who, [&] { return yskn_kv8_attention_ws(&a, dt, ws.p, ws.bytes, st); });
    return call(who, [&] { return entry(&a, dt, st); });
  });
}
FN(kv8_attention) { return kv8(v, n, "yskn_kv8_attention", yskn_kv8_attention); }
FN(kv8_attention_tc) { return kv8(v, n, "yskn_kv8_attention_tc", yskn_kv8_attention_tc); }

FN(kv8_combine) {                                        // pm, pl, pacc, splits, M, nh, o16, gate, inverse_rotate, stream
  return guarded(n, 10, [&]() -> PyObject* {
    const float *pm = (const float*)opt_dev(v[0], "pm"), *pl = (const float*)opt_dev(v[1], "pl"), *pacc = (const float*)opt_dev(v[2], "pacc");
    const int splits = int_of(v[3]), M = int_of(v[4]), nh = int_of(v[5]), inv = PyObject_IsTrue(v[8]);
    if (inv < 0) throw PyFail{};
    void *o16 = dev_ptr(v[6], "o16"), *gate = opt_dev(v[7], "gate");
    const int dt = dtype_code(THPVariable_Unpack(v[6]));
    const cudaStream_t st = stream_of(v[9]);
    return call("yskn_kv8_combine", [&] { return yskn_kv8_combine(pm, pl, pacc, splits, M, nh, gate, o16, dt, inv ? 1 : 0, st); });
  });
}

FN(tb_attention) {  // profile, q16, k_pay, k_side, v_pay, v_side, grp_k, grp_v, M, d_pos, splits, pm, pl, pacc, nh, k_plain, v_plain, qscale, stream
  return guarded(n, 19, [&]() -> PyObject* {
    const at::Tensor& kp = tensor(v[2], "k_pay");
    if (kp.dim() != 3) fail(PyExc_ValueError, "k_pay [kvh, max_ctx, stride]");
    const yskn_tb_attn_args a{(const uint16_t*)dev_ptr(v[1], "q16"), (const uint8_t*)dev_ptr(attr(v[0], N.dev).p, "profile"), (const uint8_t*)dev_ptr(v[2], "k_pay"),
                              (const uint8_t*)opt_dev(v[4], "v_pay"), (int)kp.size(2), (const uint32_t*)opt_dev(v[3], "k_side"), (const uint32_t*)opt_dev(v[5], "v_side"),
                              (const int*)opt_dev(v[6], "grp_k"), (const int*)opt_dev(v[7], "grp_v"), (const float*)opt_dev(v[15], "k_plain"),
                              (const float*)opt_dev(v[16], "v_plain"), (int)kp.size(1), int_of(v[8]), (const int*)opt_dev(v[9], "d_pos"), int_of(v[10]),
                              (float*)opt_dev(v[11], "pm"), (float*)opt_dev(v[12], "pl"), (float*)opt_dev(v[13], "pacc"), (int)kp.size(0), int_of(v[14]), float_of(v[17])};
    const int dt = dtype_code(tensor(v[1], "q16"));
    const cudaStream_t st = stream_of(v[18]);
    return call("yskn_tb_attention", [&] { return yskn_tb_attention(&a, dt, st); });
  });
}

PyObject* library(PyObject*, PyObject* const*, Py_ssize_t) {  // where the library this module calls is loaded
  return PyLong_FromVoidPtr((void*)yskn_kv4_last_error);
}

#define M_(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {M_(kv_append), M_(attention), M_(decode), M_(combine), M_(attention_ms), M_(attention_tc), M_(prefill_tc), M_(attn_post),
                         M_(kv8_attention), M_(kv8_attention_tc), M_(kv8_combine), M_(tb_attention), M_(library), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "argument marshalling of the hot launchers", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
  PyObject* lib = PyImport_ImportModule("yasakani_b200._lib");
  if (!lib) return nullptr;
  g_kv4_error = PyObject_GetAttrString(lib, "Kv4Error");
  g_not_a_tensor = PyObject_GetAttrString(lib, "NotATensor");
  Py_DECREF(lib);
  if (!g_kv4_error || !g_not_a_tensor) return nullptr;
  struct { PyObject** p; const char* s; } names[] = {{&N.kq, "kq"}, {&N.kscale, "kscale"}, {&N.kzero, "kzero"}, {&N.kshadow, "kshadow"}, {&N.vq, "vq"},
      {&N.vscale, "vscale"}, {&N.vzero, "vzero"}, {&N.hkv, "hkv"}, {&N.hd, "hd"}, {&N.max_ctx, "max_ctx"}, {&N.cuda_stream, "cuda_stream"},
      {&N.maps_ptr, "maps_ptr"}, {&N.d_layers, "d_layers"}, {&N.n, "n"}, {&N.dev, "dev"}};
  for (auto& e : names) if (!(*e.p = PyUnicode_InternFromString(e.s))) return nullptr;
  return PyModule_Create(&module_def);
}
