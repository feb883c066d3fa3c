// Python entry points of the hot calls, as a CPython extension over the C interface (include/tq4.h).
//
// A decode step of a small batch takes 15 - 30 us on the GPU; going through ctypes with some fifty
// arguments, and asking every tensor for its pointer, strides and type from Python, took 43 us of host
// time a call and bounded it.  Here the tensors are unpacked, checked and passed on in native code
// (about a tenth of that; what is left is the kernel launches).  The checks, their exceptions and the results are
// those of the Python wrappers in turboquant_vllm/kernels/ops.py, which only forward to this module.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/zeros.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <memory>
#include <stdexcept>
#include <string>
#include <thread>
#include <vector>

#include "tq4.h"

namespace {

constexpr int kMaxDevices = 64;

// thrown with the Python exception already set
struct PyError {};

[[noreturn]] void fail(PyObject* type, const std::string& msg) {
  PyErr_SetString(type, msg.c_str());
  throw PyError{};
}
#define TQ4_ASSERT(cond, msg) \
  do {                        \
    if (!(cond)) fail(PyExc_AssertionError, msg); \
  } while (0)

const at::Tensor& tensor(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, std::string(name) + " must be a torch.Tensor");
  return THPVariable_Unpack(o);
}
const at::Tensor& cuda_tensor(PyObject* o, const char* name) {
  const at::Tensor& t = tensor(o, name);
  if (!t.is_cuda())
    fail(PyExc_RuntimeError, "TQ4 kernels run on CUDA tensors only (sm_100a); got a tensor on " + t.device().str() +
                                 ". There is no CPU fallback in this package.");
  return t;
}
int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return TQ4_F32;
    case at::kHalf: return TQ4_F16;
    case at::kBFloat16: return TQ4_BF16;
    default:
      fail(PyExc_TypeError, std::string("TQ4 kernels support float32/float16/bfloat16, got ") + c10::toString(t));
  }
}
int64_t as_int(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyError{};
  return v;
}
// int(o or 0): None, False and 0 are "none", and whatever int() takes is taken (a float, a NumPy or tensor scalar)
int64_t int_or_zero(PyObject* o) {
  const int truthy = PyObject_IsTrue(o);
  if (truthy < 0) throw PyError{};
  if (!truthy) return 0;
  PyObject* i = PyNumber_Long(o);
  if (!i) throw PyError{};
  const long long v = PyLong_AsLongLong(i);
  Py_DECREF(i);
  if (v == -1 && PyErr_Occurred()) throw PyError{};
  return v;
}
double as_double(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyError{};
  return v;
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PyError{};
  return v != 0;
}
at::ScalarType as_dtype(PyObject* o) {
  if (!THPDtype_Check(o)) fail(PyExc_TypeError, "dtype must be a torch.dtype");
  return reinterpret_cast<THPDtype*>(o)->scalar_type;
}
at::Tensor inner_contiguous(const at::Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }

void check(int status, const char* what) {
  if (status == TQ4_OK) return;
  const std::string msg = std::string(what) + ": " + tq4_status_string(status);
  if (status == TQ4_ERR_UNSUPPORTED) fail(PyExc_NotImplementedError, msg);
  if (status == TQ4_ERR_STATIC_SCRATCH) fail(PyExc_ValueError, msg);
  fail(PyExc_RuntimeError, msg + " (tq4 status " + std::to_string(status) + ")");
}

// Attention scratch of the callers that bring none, grown on demand.  A call is several launches that hand data
// on through it, made without the GIL, so no two calls that can run at a time may share one: it belongs to a
// stream (kernels of two streams overlap) and a thread (launches of two threads interleave).  The last
// kMaxScratch of a device are held.  One that is dropped or outgrown returns to its own stream's pool, so its
// memory is reused behind the kernels that still work on it; a call keeps its tensor until it has launched.
struct Scratch {
  void* stream;
  std::thread::id thread;
  at::Tensor t;
  uint64_t used;
};
constexpr size_t kMaxScratch = 4;
// Per-device error flag and scratch.  Never destroyed: the CUDA context may be gone by the time static objects
// are.  Reached with the GIL held only.
at::Tensor* g_flag[kMaxDevices];
std::vector<Scratch>* g_scratch[kMaxDevices];
uint64_t g_scratch_clock = 0;

int device_index(const at::Tensor& t) {
  const int i = t.get_device();
  if (i < 0 || i >= kMaxDevices) fail(PyExc_RuntimeError, "CUDA device index out of range");
  return i;
}
at::Tensor& flag_of(int dev) {
  if (!g_flag[dev])
    g_flag[dev] = new at::Tensor(at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, dev)));
  return *g_flag[dev];
}
// The device's stream, with the device current for the duration of a call: the C entry points launch on
// the current device.
struct Launch {
  c10::cuda::OptionalCUDAGuard guard;
  void* stream;
  explicit Launch(int dev) {
    guard.set_index((c10::DeviceIndex)dev);
    stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  }
};

at::Tensor workspace_of(int dev, void* stream, int64_t bytes) {
  const auto opts = at::TensorOptions().dtype(at::kByte).device(at::kCUDA, dev);
  // a captured call gets memory of its graph's pool: it is replayed, on any stream, for as long as the graph lives
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return at::empty({bytes}, opts);
  if (!g_scratch[dev]) g_scratch[dev] = new std::vector<Scratch>();
  std::vector<Scratch>& all = *g_scratch[dev];
  const std::thread::id me = std::this_thread::get_id();
  auto it = std::find_if(all.begin(), all.end(), [&](const Scratch& s) { return s.stream == stream && s.thread == me; });
  if (it == all.end()) {
    if (all.size() == kMaxScratch)
      all.erase(std::min_element(all.begin(), all.end(), [](const Scratch& a, const Scratch& b) { return a.used < b.used; }));
    it = all.insert(all.end(), Scratch{stream, me, at::Tensor(), 0});
  }
  it->used = ++g_scratch_clock;
  if (!it->t.defined() || it->t.numel() < bytes) {
    it->t.reset();
    it->t = at::empty({bytes}, opts);
  }
  return it->t;
}

// The GIL given up for the launches of a call; taken back on the way out of an exception, too.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

template <typename F>
PyObject* guarded(F&& body) {
  try {
    return body();
  } catch (const PyError&) {
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

bool expect(const char* name, Py_ssize_t got, Py_ssize_t want) {
  if (got == want) return true;
  PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, want, got);
  return false;
}

// Slot mapping as contiguous int64.
at::Tensor slots64(const at::Tensor& s) {
  at::Tensor t = s.scalar_type() == at::kLong ? s : s.to(at::kLong);
  return t.is_contiguous() ? t : t.contiguous();
}

// attention(q, kv_cache, block_table, seq_lens, k_centroids, v_centroids, rotation, num_kv_heads, block_size,
//           sm_scale, query_start_loc, causal, sliding_window, out, out_dtype, lse_out, out_rotated, workspace,
//           mode, write, max_seq_len)
PyObject* attention(PyObject*, PyObject* const* p, Py_ssize_t n) {
  if (!expect("attention", n, 21)) return nullptr;
  return guarded([&]() -> PyObject* {
    at::Tensor q = cuda_tensor(p[0], "q");
    const at::Tensor& cache = cuda_tensor(p[1], "kv_cache");
    const at::Tensor& bt = cuda_tensor(p[2], "block_table");
    const at::Tensor& lens = cuda_tensor(p[3], "seq_lens");
    const at::Tensor& kc = cuda_tensor(p[4], "k_centroids");
    const at::Tensor& vc = cuda_tensor(p[5], "v_centroids");
    at::Tensor rot = cuda_tensor(p[6], "rotation");
    const int64_t hkv = as_int(p[7]), block = as_int(p[8]);
    TQ4_ASSERT(q.dim() == 3, "q must have three dimensions");
    const int64_t t = q.size(0), hq = q.size(1), d = q.size(2);
    TQ4_ASSERT(hkv > 0 && hq % hkv == 0, "query heads must be a multiple of the KV heads");
    TQ4_ASSERT(cache.scalar_type() == at::kByte && cache.dim() == 3 && cache.stride(2) == 1,
               "kv_cache must be uint8 [blocks, tokens, bytes] with contiguous rows");
    TQ4_ASSERT(bt.scalar_type() == at::kInt && bt.dim() == 2 && bt.stride(1) == 1, "block_table must be int32 with contiguous rows");
    TQ4_ASSERT(lens.scalar_type() == at::kInt && lens.is_contiguous(), "seq_lens must be contiguous int32");
    TQ4_ASSERT(rot.scalar_type() == at::kFloat, "rotation must be float32");
    if (!rot.is_contiguous()) rot = rot.contiguous();  // e.g. the column-major Q factor of a QR
    const at::Tensor* qsl = nullptr;
    if (p[10] != Py_None) {
      qsl = &cuda_tensor(p[10], "query_start_loc");
      TQ4_ASSERT(qsl->scalar_type() == at::kInt && qsl->is_contiguous(), "query_start_loc must be contiguous int32");
    }
    q = inner_contiguous(q);
    const float scale = p[9] == Py_None ? (float)(1.0 / std::sqrt((double)d)) : (float)as_double(p[9]);
    const int dev = device_index(q);
    Launch launch(dev);
    at::Tensor out;
    const bool own_out = p[13] == Py_None;
    if (own_out) {
      const at::ScalarType dt = p[14] == Py_None ? q.scalar_type() : as_dtype(p[14]);
      out = at::empty({t, hq, d}, q.options().dtype(dt).requires_grad(false));
    } else {
      out = cuda_tensor(p[13], "out");
      TQ4_ASSERT(out.dim() == 3 && out.size(0) == t && out.size(1) == hq && out.size(2) == d && out.stride(2) == 1,
                 "out must have q's shape and contiguous rows");
    }
    float* lse = nullptr;
    if (p[15] != Py_None) {
      const at::Tensor& l = cuda_tensor(p[15], "lse_out");
      TQ4_ASSERT(l.scalar_type() == at::kFloat && l.is_contiguous() && l.numel() >= t * hq,
                 "lse_out must be contiguous float32 of rows x heads");
      lse = (float*)l.data_ptr();
    }
    const size_t need = tq4_attention_workspace_bytes(t > 1 ? t : 1, (int)hq, (int)hkv, (int)d);
    if (need == 0)
      fail(PyExc_ValueError, "unsupported attention shape: Hq=" + std::to_string(hq) + ", Hkv=" + std::to_string(hkv) +
                                 ", D=" + std::to_string(d));
    const at::Tensor ws = p[17] == Py_None ? workspace_of(dev, launch.stream, (int64_t)need) : cuda_tensor(p[17], "workspace");
    const size_t have = (size_t)ws.numel() * ws.element_size();
    if (have < need)
      fail(PyExc_ValueError, "workspace has " + std::to_string(have) + " bytes, " + std::to_string(need) + " needed");
    const int causal = truth(p[11]) ? 1 : 0, window = (int)int_or_zero(p[12]);
    // (the width of the table bounds it, too; the stride, which the C interface has, may be a wider one's)
    int64_t max_seq_len = p[20] == Py_None ? 0 : as_int(p[20]);
    if (bt.size(1) > 0 && (max_seq_len <= 0 || max_seq_len > bt.size(1) * block)) max_seq_len = bt.size(1) * block;
    const int rotated = truth(p[16]) ? 1 : 0, mode = (int)as_int(p[18]);
    int* flag = (int*)flag_of(dev).data_ptr();
    const int q_dt = dtype_code(q.scalar_type()), out_dt = dtype_code(out.scalar_type());
    // the new tokens to be written first, if any
    at::Tensor key, value, slots, even, odd, kb, vb;
    int kv_dt = TQ4_F32;
    if (p[19] != Py_None) {
      struct Held {  // any iterable of seven
        PyObject* o;
        ~Held() { Py_XDECREF(o); }
      } seq{PySequence_Tuple(p[19])};
      if (!seq.o) throw PyError{};
      if (PyTuple_GET_SIZE(seq.o) != 7) fail(PyExc_ValueError, "write must hold seven tensors");
      auto item = [&](int i, const char* name) -> const at::Tensor& { return cuda_tensor(PyTuple_GET_ITEM(seq.o, i), name); };
      key = item(0, "key");
      value = item(1, "value");
      slots = slots64(item(2, "slot_mapping"));
      even = item(3, "rotation_T_even");
      odd = item(4, "rotation_T_odd");
      kb = item(5, "k_boundaries");
      vb = item(6, "v_boundaries");
      TQ4_ASSERT(cache.is_contiguous(), "the fused write addresses flat slots: block-major contiguous cache");
      TQ4_ASSERT(key.sizes() == value.sizes() && key.scalar_type() == value.scalar_type() && key.dim() == 3 &&
                     key.size(1) == hkv && key.size(2) == d,
                 "key and value must be [tokens, KV heads, head_dim] of one type");
      key = inner_contiguous(key);
      value = inner_contiguous(value);
      kv_dt = dtype_code(key.scalar_type());
    }
    auto floats = [](const at::Tensor& t) { return t.defined() ? (const float*)t.data_ptr() : nullptr; };
    const bool wr = key.defined();
    int st;
    {
      const NoGil no_gil;
      st = tq4_attention_step(
          wr ? key.data_ptr() : nullptr, wr ? value.data_ptr() : nullptr, kv_dt, wr ? key.size(0) : 0, wr ? key.stride(0) : 0,
          wr ? key.stride(1) : 0, wr ? value.stride(0) : 0, wr ? value.stride(1) : 0,
          wr ? (const int64_t*)slots.data_ptr() : nullptr, wr ? slots.numel() : 0, floats(even), floats(odd), floats(kb),
          wr ? (int)kb.numel() : 0, floats(vb), wr ? (int)vb.numel() : 0, q.data_ptr(), q_dt, t, (int)lens.numel(), (int)hq,
          (int)hkv, (int)d, q.stride(0), q.stride(1), (uint8_t*)cache.data_ptr(), cache.stride(0), cache.stride(1),
          cache.size(0), (int)block, (const int32_t*)bt.data_ptr(), bt.stride(0), (const int32_t*)lens.data_ptr(),
          qsl ? (const int32_t*)qsl->data_ptr() : nullptr, max_seq_len, (const float*)kc.data_ptr(), (int)kc.numel(),
          (const float*)vc.data_ptr(), (int)vc.numel(), (const float*)rot.data_ptr(), scale, causal, window,
          out.data_ptr(), out_dt, out.stride(0), out.stride(1), lse, rotated, ws.data_ptr(), have,
          mode, flag, launch.stream);
    }
    check(st, "paged_tq4_attention");
    if (!own_out) {
      Py_INCREF(p[13]);
      return p[13];
    }
    return THPVariable_Wrap(std::move(out));
  });
}

// write_paged(key, value, kv_cache, slot_mapping, rotation_T_even, rotation_T_odd, k_boundaries, v_boundaries)
PyObject* write_paged(PyObject*, PyObject* const* p, Py_ssize_t n) {
  if (!expect("write_paged", n, 8)) return nullptr;
  return guarded([&]() -> PyObject* {
    at::Tensor key = cuda_tensor(p[0], "key"), value = cuda_tensor(p[1], "value");
    const at::Tensor& cache = cuda_tensor(p[2], "kv_cache");
    const at::Tensor& slot_mapping = cuda_tensor(p[3], "slot_mapping");
    const at::Tensor &even = cuda_tensor(p[4], "rotation_T_even"), &odd = cuda_tensor(p[5], "rotation_T_odd");
    const at::Tensor &kb = cuda_tensor(p[6], "k_boundaries"), &vb = cuda_tensor(p[7], "v_boundaries");
    TQ4_ASSERT(cache.scalar_type() == at::kByte && cache.dim() == 3 && cache.is_contiguous(), "kv_cache must be contiguous uint8");
    TQ4_ASSERT(key.dim() == 3 && key.sizes() == value.sizes() && key.scalar_type() == value.scalar_type(),
               "key and value must be [tokens, KV heads, head_dim] of one type");
    key = inner_contiguous(key);
    value = inner_contiguous(value);
    const at::Tensor slots = slots64(slot_mapping);
    const int dev = device_index(key);
    Launch launch(dev);
    int* flag = (int*)flag_of(dev).data_ptr();
    const int kv_dt = dtype_code(key.scalar_type());
    int st;
    {
      const NoGil no_gil;
      st = tq4_write_paged(key.data_ptr(), value.data_ptr(), kv_dt, key.size(0), (int)key.size(1),
                           (int)key.size(2), key.stride(0), key.stride(1), value.stride(0), value.stride(1),
                           (const int64_t*)slots.data_ptr(), slots.numel(), (const float*)even.data_ptr(),
                           (const float*)odd.data_ptr(), (const float*)kb.data_ptr(), (int)kb.numel(),
                           (const float*)vb.data_ptr(), (int)vb.numel(), (uint8_t*)cache.data_ptr(), cache.size(2),
                           cache.size(0) * cache.size(1), flag, launch.stream);
    }
    check(st, "tq4_write_paged");
    Py_RETURN_NONE;
  });
}

// [batch, heads, tokens, head_dim] K or V of an update, innermost stride 1
struct States {
  at::Tensor t;
  int64_t strides[3];
  States(PyObject* o, const char* name) : t(cuda_tensor(o, name)) {
    TQ4_ASSERT(t.dim() == 4, "key and value must be [batch, heads, tokens, head_dim]");
    t = inner_contiguous(t);
    for (int i = 0; i < 3; ++i) strides[i] = t.stride(i);
  }
};

// attend_rows(q, rows, block_table, len_rows, len, k_centroids, v_centroids, rotation, num_kv_heads, page_tokens,
//             sm_scale, out_dtype): one query row per sequence, q [B, Hq, 1, D], over `len` token rows each
// -> [B, 1, Hq, D].  Everything a generation step needs of `attention`, with no tensor made but the result.
PyObject* attend_rows(PyObject*, PyObject* const* p, Py_ssize_t n) {
  if (!expect("attend_rows", n, 12)) return nullptr;
  return guarded([&]() -> PyObject* {
    const at::Tensor q = inner_contiguous(cuda_tensor(p[0], "q"));
    const at::Tensor &rows = cuda_tensor(p[1], "rows"), &bt = cuda_tensor(p[2], "block_table"), &lens = cuda_tensor(p[3], "len_rows");
    const int64_t len = as_int(p[4]), hkv = as_int(p[8]), page = as_int(p[9]);
    const at::Tensor &kc = cuda_tensor(p[5], "k_centroids"), &vc = cuda_tensor(p[6], "v_centroids");
    at::Tensor rot = cuda_tensor(p[7], "rotation");
    TQ4_ASSERT(q.dim() == 4 && q.size(2) == 1, "q must be [batch, heads, 1, head_dim]");
    const int64_t b = q.size(0), hq = q.size(1), d = q.size(3);
    TQ4_ASSERT(hkv > 0 && hq % hkv == 0, "query heads must be a multiple of the KV heads");
    TQ4_ASSERT(rows.scalar_type() == at::kByte && rows.dim() == 3 && rows.is_contiguous() && rows.size(0) == b && page > 0 &&
                   rows.size(1) % page == 0,
               "rows must be contiguous uint8 [batch, capacity, bytes], whole pages");
    TQ4_ASSERT(bt.scalar_type() == at::kInt && bt.dim() == 2 && bt.size(0) == b && bt.is_contiguous(), "block_table must be contiguous int32");
    TQ4_ASSERT(lens.scalar_type() == at::kInt && lens.dim() == 2 && lens.size(1) == b && lens.is_contiguous() && len >= 0 &&
                   len < lens.size(0),
               "len_rows must be contiguous int32 [capacity + 1, batch]");
    TQ4_ASSERT(rot.scalar_type() == at::kFloat, "rotation must be float32");
    if (!rot.is_contiguous()) rot = rot.contiguous();
    const float scale = p[10] == Py_None ? (float)(1.0 / std::sqrt((double)d)) : (float)as_double(p[10]);
    const int dev = device_index(q);
    Launch launch(dev);
    const at::ScalarType dt = p[11] == Py_None ? q.scalar_type() : as_dtype(p[11]);
    at::Tensor out = at::empty({b, 1, hq, d}, q.options().dtype(dt).requires_grad(false));
    const size_t need = tq4_attention_workspace_bytes(b > 1 ? b : 1, (int)hq, (int)hkv, (int)d);
    if (need == 0)
      fail(PyExc_ValueError, "unsupported attention shape: Hq=" + std::to_string(hq) + ", Hkv=" + std::to_string(hkv) +
                                 ", D=" + std::to_string(d));
    const at::Tensor ws = workspace_of(dev, launch.stream, (int64_t)need);
    int* flag = (int*)flag_of(dev).data_ptr();
    const int q_dt = dtype_code(q.scalar_type()), out_dt = dtype_code(dt);
    int st;
    {
      const NoGil no_gil;
      // (the kernels are chosen by the tokens held, not by the room for more)
      st = tq4_attention_step(
          nullptr, nullptr, q_dt, 0, 0, 0, 0, 0, nullptr, 0, nullptr, nullptr, nullptr, 0, nullptr, 0, q.data_ptr(), q_dt, b, (int)b,
          (int)hq, (int)hkv, (int)d, q.stride(0), q.stride(1), (uint8_t*)rows.data_ptr(), page * rows.size(2), rows.size(2),
          b * (rows.size(1) / page), (int)page, (const int32_t*)bt.data_ptr(), bt.size(1),
          (const int32_t*)lens.data_ptr() + len * b, nullptr, len > 0 ? len : 1, (const float*)kc.data_ptr(), (int)kc.numel(),
          (const float*)vc.data_ptr(), (int)vc.numel(), (const float*)rot.data_ptr(), scale, 0, 0, out.data_ptr(), out_dt,
          out.stride(0), out.stride(2), nullptr, 0, ws.data_ptr(), (size_t)ws.numel() * ws.element_size(), 0, flag, launch.stream);
    }
    check(st, "attend_rows");
    return THPVariable_Wrap(std::move(out));
  });
}

// append_rows(key, value, rows, offset, rotation_T_even, rotation_T_odd, k_boundaries, v_boundaries)
PyObject* append_rows(PyObject*, PyObject* const* p, Py_ssize_t n) {
  if (!expect("append_rows", n, 8)) return nullptr;
  return guarded([&]() -> PyObject* {
    const States k(p[0], "key"), v(p[1], "value");
    const at::Tensor& rows = cuda_tensor(p[2], "rows");
    const int64_t offset = as_int(p[3]);
    const at::Tensor &even = cuda_tensor(p[4], "rotation_T_even"), &odd = cuda_tensor(p[5], "rotation_T_odd");
    const at::Tensor &kb = cuda_tensor(p[6], "k_boundaries"), &vb = cuda_tensor(p[7], "v_boundaries");
    TQ4_ASSERT(k.t.sizes() == v.t.sizes() && k.t.scalar_type() == v.t.scalar_type(), "key and value must be alike");
    TQ4_ASSERT(rows.scalar_type() == at::kByte && rows.dim() == 3 && rows.is_contiguous() && rows.size(0) == k.t.size(0),
               "rows must be contiguous uint8 [batch, capacity, bytes]");
    const int dt = dtype_code(k.t.scalar_type());
    Launch launch(device_index(k.t));
    int st;
    {
      const NoGil no_gil;
      st = tq4_append_rows(k.t.data_ptr(), v.t.data_ptr(), dt, (int)k.t.size(0), (int)k.t.size(2), (int)k.t.size(1), (int)k.t.size(3),
                           k.strides, v.strides, (const float*)even.data_ptr(), (const float*)odd.data_ptr(),
                           (const float*)kb.data_ptr(), (int)kb.numel(), (const float*)vb.data_ptr(), (int)vb.numel(),
                           (uint8_t*)rows.data_ptr(), rows.size(2), rows.size(1), offset, launch.stream);
    }
    check(st, "tq4_append_rows");
    Py_RETURN_NONE;
  });
}

// What an in-place cache update found to fit together: the types and sizes of the states, the device's tables, and the buffers as
// the Python objects that held them (compared by a later step: a buffer that was replaced since is noticed).
struct UpdatePlan {
  int64_t b, h, d, cap, dec_cap;
  at::ScalarType dtype;
  int dev;
  bool k_nib, v_nib;
  at::Tensor prims[7];             // rotation, even, odd, boundaries and centroids of K and V
  std::vector<at::Tensor> out;     // k_idx, k_norms, v_idx, v_norms (and k_dec, v_dec)
  std::vector<PyObject*> held;     // ... as Python objects, and the two quantisers
  ~UpdatePlan() {
    for (PyObject* o : held) Py_XDECREF(o);
  }
};
constexpr const char* kPlanName = "tq4.update_plan";
PyObject *g_buf_name, *g_len_name;  // interned attribute names

// cache_update(key, value, rotation, rotation_T_even, rotation_T_odd, k_boundaries, v_boundaries, k_centroids, v_centroids, k_nibble, v_nibble,
//              k_idx, k_norms, v_idx, v_norms, offset, k_dec, v_dec, dec_offset[, k_quantizer, v_quantizer])
// With the quantisers: returns the plan of the update, for cache_step.
PyObject* cache_update(PyObject*, PyObject* const* p, Py_ssize_t n) {
  if (n != 21 && !expect("cache_update", n, 19)) return nullptr;
  return guarded([&]() -> PyObject* {
    const States k(p[0], "key"), v(p[1], "value");
    const at::Tensor& rot = cuda_tensor(p[2], "rotation");
    const at::Tensor &even = cuda_tensor(p[3], "rotation_T_even"), &odd = cuda_tensor(p[4], "rotation_T_odd");
    const at::Tensor &kb = cuda_tensor(p[5], "k_boundaries"), &vb = cuda_tensor(p[6], "v_boundaries");
    const at::Tensor &kc = cuda_tensor(p[7], "k_centroids"), &vc = cuda_tensor(p[8], "v_centroids");
    const int k_nib = truth(p[9]), v_nib = truth(p[10]);
    const at::Tensor &ki = cuda_tensor(p[11], "k_idx"), &kn = cuda_tensor(p[12], "k_norms");
    const at::Tensor &vi = cuda_tensor(p[13], "v_idx"), &vn = cuda_tensor(p[14], "v_norms");
    const int64_t offset = as_int(p[15]), dec_offset = as_int(p[18]);
    TQ4_ASSERT(k.t.sizes() == v.t.sizes() && k.t.scalar_type() == v.t.scalar_type(), "key and value must be alike");
    const int64_t b = k.t.size(0), h = k.t.size(1), d = k.t.size(3);
    auto buffer = [&](const at::Tensor& t, int64_t width, at::ScalarType type) {
      TQ4_ASSERT(t.dim() == 4 && t.size(0) == b && t.size(1) == h && t.size(3) == width && t.is_contiguous() && t.scalar_type() == type,
                 "buffers must be contiguous [batch, heads, capacity, width]");
      return t.size(2);
    };
    const int64_t cap = buffer(ki, k_nib ? d / 2 : d, at::kByte);
    TQ4_ASSERT(buffer(vi, v_nib ? d / 2 : d, at::kByte) == cap && buffer(kn, 1, at::kFloat) == cap && buffer(vn, 1, at::kFloat) == cap,
               "index and norm buffers must have one capacity");
    void *kd = nullptr, *vd = nullptr;
    int64_t dec_cap = 0;
    if (p[16] != Py_None) {
      const at::Tensor &a = cuda_tensor(p[16], "k_dec"), &c = cuda_tensor(p[17], "v_dec");
      dec_cap = buffer(a, d, k.t.scalar_type());
      TQ4_ASSERT(buffer(c, d, k.t.scalar_type()) == dec_cap, "the two dequantised buffers must have one capacity");
      kd = a.data_ptr();
      vd = c.data_ptr();
    }
    const int dt = dtype_code(k.t.scalar_type());
    Launch launch(device_index(k.t));
    const size_t need = tq4_cache_update_scratch_bytes((int)b, (int)h, (int)k.t.size(2), (int)d);
    at::Tensor scratch;
    if (need) scratch = at::empty({(int64_t)need}, k.t.options().dtype(at::kByte).requires_grad(false));
    int st;
    {
      const NoGil no_gil;
      st = tq4_cache_update(k.t.data_ptr(), v.t.data_ptr(), dt, (int)b, (int)h, (int)k.t.size(2), (int)d, k.strides, v.strides,
                            (const float*)rot.data_ptr(), (const float*)even.data_ptr(), (const float*)odd.data_ptr(),
                            (const float*)kb.data_ptr(), (int)kb.numel(),
                            (const float*)vb.data_ptr(), (int)vb.numel(), (const float*)kc.data_ptr(), (int)kc.numel(),
                            (const float*)vc.data_ptr(), (int)vc.numel(), k_nib, v_nib, (uint8_t*)ki.data_ptr(),
                            (float*)kn.data_ptr(), (uint8_t*)vi.data_ptr(), (float*)vn.data_ptr(), cap, offset, kd, vd, dec_cap,
                            dec_offset, need ? scratch.data_ptr() : nullptr, need, launch.stream);
    }
    check(st, "tq4_cache_update");
    if (n == 19) Py_RETURN_NONE;
    auto plan = std::make_unique<UpdatePlan>();
    plan->b = b; plan->h = h; plan->d = d;
    plan->cap = cap;
    plan->dec_cap = dec_cap;
    plan->dtype = k.t.scalar_type();
    plan->dev = device_index(k.t);
    plan->k_nib = k_nib;
    plan->v_nib = v_nib;
    const at::Tensor* prims[7] = {&rot, &even, &odd, &kb, &vb, &kc, &vc};
    for (int i = 0; i < 7; ++i) plan->prims[i] = *prims[i];
    for (int i : {11, 12, 13, 14, 16, 17}) {
      if (p[i] == Py_None) continue;
      plan->out.push_back(THPVariable_Unpack(p[i]));
      Py_INCREF(p[i]);
      plan->held.push_back(p[i]);
    }
    for (int i : {19, 20}) {
      Py_INCREF(p[i]);
      plan->held.push_back(p[i]);
    }
    PyObject* c = PyCapsule_New(plan.get(), kPlanName, [](PyObject* o) { delete (UpdatePlan*)PyCapsule_GetPointer(o, kPlanName); });
    if (!c) throw PyError{};
    plan.release();
    return c;
  });
}

// cache_step(plan, groups, key, value, k_quantizer, v_quantizer): another update into the plan's buffers, which are the `buf` of the
// groups with `len` tokens each -> (keys, values) of all tokens held, reconstructed, or True without such buffers; None, with nothing changed,
// when the states or the groups are not those of the plan, or there is no room left.
PyObject* cache_step(PyObject*, PyObject* const* p, Py_ssize_t n) {
  if (!expect("cache_step", n, 6)) return nullptr;
  return guarded([&]() -> PyObject* {
    UpdatePlan* plan = (UpdatePlan*)PyCapsule_GetPointer(p[0], kPlanName);
    if (!plan) throw PyError{};
    const size_t n_out = plan->out.size();
    if (!PyTuple_Check(p[1]) || (size_t)PyTuple_GET_SIZE(p[1]) != n_out || plan->held[n_out] != p[4] || plan->held[n_out + 1] != p[5] ||
        !THPVariable_Check(p[2]) || !THPVariable_Check(p[3]))
      Py_RETURN_NONE;
    const at::Tensor &k = THPVariable_Unpack(p[2]), &v = THPVariable_Unpack(p[3]);
    if (k.dim() != 4 || !k.is_cuda() || !v.is_cuda() || k.scalar_type() != plan->dtype || v.scalar_type() != plan->dtype || k.sizes() != v.sizes() ||
        k.get_device() != plan->dev || v.get_device() != plan->dev || k.size(0) != plan->b || k.size(1) != plan->h || k.size(3) != plan->d ||
        k.size(2) == 0)
      Py_RETURN_NONE;
    const int64_t fresh = k.size(2);
    int64_t len[2] = {-1, 0};  // tokens held: compressed, reconstructed
    for (size_t i = 0; i < n_out; ++i) {
      PyObject* g = PyTuple_GET_ITEM(p[1], i);
      PyObject* buf = PyObject_GetAttr(g, g_buf_name);
      if (!buf) throw PyError{};
      const bool same = buf == plan->held[i];
      Py_DECREF(buf);
      if (!same) Py_RETURN_NONE;
      PyObject* l = PyObject_GetAttr(g, g_len_name);
      if (!l) throw PyError{};
      const long long x = PyLong_AsLongLong(l);
      Py_DECREF(l);
      if (x == -1 && PyErr_Occurred()) throw PyError{};
      int64_t& want = len[i < 4 ? 0 : 1];
      if (i == 0 || i == 4) want = x;
      else if (x != want) Py_RETURN_NONE;
    }
    if (len[0] < 0 || len[1] < 0 || len[0] + fresh > plan->cap || (n_out == 6 && len[1] + fresh > plan->dec_cap)) Py_RETURN_NONE;
    const States ks(p[2], "key"), vs(p[3], "value");
    Launch launch(plan->dev);
    const size_t need = tq4_cache_update_scratch_bytes((int)plan->b, (int)plan->h, (int)fresh, (int)plan->d);
    at::Tensor scratch;
    if (need) scratch = at::empty({(int64_t)need}, k.options().dtype(at::kByte).requires_grad(false));
    auto f = [&](int i) { return (const float*)plan->prims[i].data_ptr(); };
    int st;
    {
      const NoGil no_gil;
      st = tq4_cache_update(ks.t.data_ptr(), vs.t.data_ptr(), dtype_code(plan->dtype), (int)plan->b, (int)plan->h, (int)fresh, (int)plan->d,
                            ks.strides, vs.strides, f(0), f(1), f(2), f(3), (int)plan->prims[3].numel(), f(4), (int)plan->prims[4].numel(), f(5),
                            (int)plan->prims[5].numel(), f(6), (int)plan->prims[6].numel(), plan->k_nib, plan->v_nib,
                            (uint8_t*)plan->out[0].data_ptr(), (float*)plan->out[1].data_ptr(), (uint8_t*)plan->out[2].data_ptr(),
                            (float*)plan->out[3].data_ptr(), plan->cap, len[0], n_out == 6 ? plan->out[4].data_ptr() : nullptr,
                            n_out == 6 ? plan->out[5].data_ptr() : nullptr, plan->dec_cap, len[1], need ? scratch.data_ptr() : nullptr, need,
                            launch.stream);
    }
    check(st, "tq4_cache_update");
    for (int part = 0; part < (n_out == 6 ? 2 : 1); ++part) {
      PyObject* l = PyLong_FromLongLong(len[part] + fresh);
      if (!l) throw PyError{};
      for (size_t i = part ? 4 : 0; i < (part ? n_out : 4); ++i)
        if (PyObject_SetAttr(PyTuple_GET_ITEM(p[1], i), g_len_name, l) < 0) {
          Py_DECREF(l);
          throw PyError{};
        }
      Py_DECREF(l);
    }
    if (n_out == 4) Py_RETURN_TRUE;
    PyObject* kv = PyTuple_New(2);
    if (!kv) throw PyError{};
    for (int i = 0; i < 2; ++i) PyTuple_SET_ITEM(kv, i, THPVariable_Wrap(plan->out[4 + i].narrow(2, 0, len[1] + fresh)));
    return kv;
  });
}

// error_flag(device_index) -> the device's int32 flag tensor
PyObject* error_flag(PyObject*, PyObject* const* p, Py_ssize_t n) {
  if (!expect("error_flag", n, 1)) return nullptr;
  return guarded([&]() -> PyObject* {
    const int64_t dev = as_int(p[0]);
    if (dev < 0 || dev >= kMaxDevices) fail(PyExc_RuntimeError, "CUDA device index out of range");
    return THPVariable_Wrap(flag_of((int)dev));
  });
}

PyMethodDef kMethods[] = {
    {"attention", (PyCFunction)(void (*)(void))attention, METH_FASTCALL, "Paged TQ4 attention, optionally with a cache write."},
    {"write_paged", (PyCFunction)(void (*)(void))write_paged, METH_FASTCALL, "Compress K and V into the paged cache."},
    {"attend_rows", (PyCFunction)(void (*)(void))attend_rows, METH_FASTCALL, "Attention of one query row per sequence over token rows."},
    {"append_rows", (PyCFunction)(void (*)(void))append_rows, METH_FASTCALL, "Compress K and V into token rows of a batch."},
    {"cache_update", (PyCFunction)(void (*)(void))cache_update, METH_FASTCALL, "Compress, store and reconstruct an update."},
    {"cache_step", (PyCFunction)(void (*)(void))cache_step, METH_FASTCALL, "An update by a plan."},
    {"error_flag", (PyCFunction)(void (*)(void))error_flag, METH_FASTCALL, "Device error flag."},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_tq4_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__tq4_host(void) {
  g_buf_name = PyUnicode_InternFromString("buf");
  g_len_name = PyUnicode_InternFromString("len");
  if (!g_buf_name || !g_len_name) return nullptr;
  return PyModule_Create(&kModule);
}
