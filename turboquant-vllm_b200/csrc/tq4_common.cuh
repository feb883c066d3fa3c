// Shared device/host helpers for the TQ4 sm_100a kernels.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <mutex>

#include "tq4.h"

#define TQ4_MAX_BOUNDARIES 15
#define TQ4_MAX_CENTROIDS 16

#define TQ4_CHECK_LAUNCH()                                   \
  do {                                                       \
    cudaError_t e__ = cudaGetLastError();                    \
    if (e__ != cudaSuccess) return (int)TQ4_ERR_CUDA;        \
  } while (0)

namespace tq4 {

// per-kernel event timing (tq4_profile.cu); no-ops unless tq4_profile_start() was called
void prof_begin(int kind, cudaStream_t st);
void prof_end(int kind, cudaStream_t st);

// ---- programmatic dependent launch ---------------------------------------------------------------
// The kernels of one decode step (cache write, query rotation + plan, attention, merge) are launched
// back to back.  A kernel that calls pdl_trigger() lets the next launch in the stream start before it
// has finished, if that launch was made with launch_kernel(..., pdl = true); the dependent kernel
// calls pdl_wait() before it reads or writes anything a predecessor touches: after the wait, the
// preceding kernel has completed and its stores are visible.  Rules kept by every kernel here:
//  * the FIRST kernel an entry point launches is a plain stream-ordered launch (pdl = false): its
//    inputs may come from the caller's preceding kernel, which may itself trigger dependents early;
//  * the later kernels of the same entry point are launched with pdl = true; before pdl_wait() they
//    only read caller inputs (which the first kernel's launch has already ordered behind the
//    caller's work) and write shared memory or registers;
//  * a kernel launched with pdl = true calls pdl_wait() on every path before it exits, so its own
//    completion implies the completion of everything before it in the stream.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
bool pdl_enabled();  // false if TQ4_NO_PDL is set in the environment

template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                 cudaStream_t st, bool pdl, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (pdl && pdl_enabled()) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

__host__ __device__ inline bool supported_head_dim(int d) {
  return d == 64 || d == 96 || d == 128 || d == 256;
}

// Bytes of one token row that carry data: [K_idx|K_norm|V_idx|V_norm].
__host__ __device__ inline int row_data_bytes(int num_kv_heads, int head_dim) {
  return num_kv_heads * (head_dim + 8);
}

struct RowLayout {
  int k_idx, k_norm, v_idx, v_norm;  // byte offsets of the four regions in a token row
};
__host__ __device__ inline RowLayout row_layout(int num_kv_heads, int head_dim) {
  RowLayout r;
  r.k_idx = 0;
  r.k_norm = num_kv_heads * (head_dim / 2);
  r.v_idx = r.k_norm + num_kv_heads * 4;
  r.v_norm = r.v_idx + num_kv_heads * (head_dim / 2);
  return r;
}

template <typename T>
__device__ __forceinline__ float to_float(T v);
template <>
__device__ __forceinline__ float to_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T>
__device__ __forceinline__ T from_float(float v);
template <>
__device__ __forceinline__ float from_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Load one element of a typed tensor chosen at run time (cold paths only).
__device__ __forceinline__ float load_as_float(const void* p, int dtype, int64_t i) {
  if (dtype == TQ4_F32) return reinterpret_cast<const float*>(p)[i];
  if (dtype == TQ4_F16) return __half2float(reinterpret_cast<const __half*>(p)[i]);
  return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
}
__device__ __forceinline__ void store_from_float(void* p, int dtype, int64_t i, float v) {
  if (dtype == TQ4_F32) reinterpret_cast<float*>(p)[i] = v;
  else if (dtype == TQ4_F16) reinterpret_cast<__half*>(p)[i] = __float2half_rn(v);
  else reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
}
// four consecutive elements i .. i + 3: one store where the address allows it
__device__ __forceinline__ void store4(void* p, int dtype, int64_t i, const float (&v)[4]) {
  if (dtype == TQ4_F32) {
    float* d = reinterpret_cast<float*>(p) + i;
    if (((uintptr_t)d & 15) == 0) {
      *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
      d[0] = v[0]; d[1] = v[1]; d[2] = v[2]; d[3] = v[3];
    }
    return;
  }
  uint16_t h[4];
#pragma unroll
  for (int e = 0; e < 4; ++e)
    h[e] = dtype == TQ4_F16 ? __half_as_ushort(__float2half_rn(v[e])) : __bfloat16_as_ushort(__float2bfloat16_rn(v[e]));
  uint16_t* d = reinterpret_cast<uint16_t*>(p) + i;
  if (((uintptr_t)d & 7) == 0) {
    *reinterpret_cast<uint2*>(d) = make_uint2(h[0] | ((uint32_t)h[1] << 16), h[2] | ((uint32_t)h[3] << 16));
  } else {
    d[0] = h[0]; d[1] = h[1]; d[2] = h[2]; d[3] = h[3];
  }
}

// four consecutive elements of a typed array as they are, in one load where their address allows it, and as floats: the loads of
// several can be in flight before the first is converted
__device__ __forceinline__ uint4 load4_raw(const void* p, int dtype, int64_t i) {
  uint4 r = make_uint4(0u, 0u, 0u, 0u);
  if (dtype == TQ4_F32) {
    const uint32_t* s = reinterpret_cast<const uint32_t*>(p) + i;
    if (((uintptr_t)s & 15) == 0) return __ldg(reinterpret_cast<const uint4*>(s));
    r.x = __ldg(s); r.y = __ldg(s + 1); r.z = __ldg(s + 2); r.w = __ldg(s + 3);
  } else {
    const uint16_t* s = reinterpret_cast<const uint16_t*>(p) + i;
    if (((uintptr_t)s & 7) == 0) {
      const uint2 t = __ldg(reinterpret_cast<const uint2*>(s));
      r.x = t.x; r.y = t.y;
    } else {
      r.x = __ldg(s) | (uint32_t)__ldg(s + 1) << 16;
      r.y = __ldg(s + 2) | (uint32_t)__ldg(s + 3) << 16;
    }
  }
  return r;
}
__device__ __forceinline__ float4 raw_as_float4(const uint4& r, int dtype) {
  if (dtype == TQ4_F32) return make_float4(__uint_as_float(r.x), __uint_as_float(r.y), __uint_as_float(r.z), __uint_as_float(r.w));
  if (dtype == TQ4_F16) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&r.y));
    return make_float4(a.x, a.y, b.x, b.y);
  }
  return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xFFFF0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xFFFF0000u));
}

// N = 1, 2 or 4 consecutive floats at an address aligned to their size
template <int N>
__device__ __forceinline__ void load_n(const float* p, float (&v)[N]) {
  if constexpr (N == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else if constexpr (N == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x; v[1] = t.y;
  } else {
    v[0] = *p;
  }
}
template <int N>
__device__ __forceinline__ void store_n(float* p, const float (&v)[N]) {
  if constexpr (N == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else if constexpr (N == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  else *p = v[0];
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// idx = #{b : b < y}: the tie rule of torch.bucketize(right=False).  NaN compares false -> 0.
__device__ __forceinline__ int bucketize(float y, const float* __restrict__ b, int nb) {
  int idx = 0;
#pragma unroll
  for (int i = 0; i < TQ4_MAX_BOUNDARIES; ++i)
    if (i < nb) idx += (y > b[i]) ? 1 : 0;
  return idx;
}

// The same count by binary search over ASCENDING boundaries padded to 15 entries with +inf
// (entry 15 is never read): four compares.  NaN compares false at every step -> 0.
__device__ __forceinline__ int bucketize_sorted16(float y, const float* b) {
  int lo = (y > b[7]) ? 8 : 0;
  lo += (y > b[lo + 3]) ? 4 : 0;
  lo += (y > b[lo + 1]) ? 2 : 0;
  lo += (y > b[lo]) ? 1 : 0;
  return lo;
}

// address of element i of an array of dtype-coded elements
__device__ __forceinline__ const void* byte_offset(const void* p, int dtype, int64_t i) {
  return reinterpret_cast<const char*>(p) + i * (dtype == TQ4_F32 ? 4 : 2);
}

// out[i][v] = element 32*i of the strip starting at base[v] (nullptr -> zeros), converted to fp32
template <typename T, int N, int V>
__device__ __forceinline__ void load_strip(const void* const (&base)[V], float (&out)[N][V]) {
#pragma unroll
  for (int v = 0; v < V; ++v)
#pragma unroll
    for (int i = 0; i < N; ++i)
      out[i][v] = base[v] ? to_float<T>(reinterpret_cast<const T*>(base[v])[32 * i]) : 0.f;
}

// ---- per-device host state ---------------------------------------------------------------------
// A process may drive several GPUs (a model spread over devices, one thread per GPU).  Function
// attributes set with cudaFuncSetAttribute and device properties belong to ONE device, so
// everything remembered on the host side is indexed by the ordinal of the current device.
constexpr int kMaxDevices = 64;
inline int device_ordinal() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
  return dev;
}

inline int sm_count() {
  static int n[kMaxDevices];
  const int dev = device_ordinal();
  if (dev < 0) return 148;
  if (n[dev] == 0) {
    cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
    if (n[dev] <= 0) n[dev] = 148;
  }
  return n[dev];
}

// Opt `Kernel` in to `bytes` of dynamic shared memory on the current device (once per device and
// kernel; again if a later call asks for more).  Entry points run without the GIL, so several threads may come
// here for the first time together: the attribute and the record of it change under one lock.
template <auto Kernel>
inline bool ensure_dynamic_smem(int bytes, bool max_carveout = false) {
  static std::atomic<int> set_bytes[kMaxDevices];
  static std::mutex lock;
  const int dev = device_ordinal();
  if (dev < 0) return false;
  if (set_bytes[dev] >= bytes && set_bytes[dev] > 0) return true;
  const std::lock_guard<std::mutex> held(lock);
  if (set_bytes[dev] >= bytes && set_bytes[dev] > 0) return true;
  if (cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
    return false;
  if (max_carveout)
    cudaFuncSetAttribute(Kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  set_bytes[dev] = bytes;
  return true;
}

// The driver's tensor-map encoder (the library does not link to libcuda), looked up once; null if it has none.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);
inline EncodeTiledFn encode_tiled_fn() {
  static const EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    const bool found = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
                       q == cudaDriverEntryPointSuccess;
    return found ? reinterpret_cast<EncodeTiledFn>(p) : nullptr;
  }();
  return fn;
}

// Arguments of the compress / cache-write kernels (tq4_compress.cu) and of the write part of the
// fused prologue kernel (tq4_attention.cu).
struct CompressArgs {
  // sources: [0] = K (or the only tensor), [1] = V (paged write only)
  const void* x[2];
  int64_t token_stride[2], head_stride[2];
  const float* bounds[2];
  int n_bounds[2];
  int64_t n_tokens;
  int num_heads;
  int n_sources;  // 1 or 2
  int x_dtype;    // TQ4_F32 / TQ4_F16 / TQ4_BF16 of both sources (read by the fused prologue kernel)
  const float* rot_even;
  const float* rot_odd;
  // contiguous destination
  uint8_t* packed_out;
  float* norms_out;
  // paged destination (cache != nullptr selects it).  Token t goes to slot_mapping[t], or, with seq > 0, to
  // row (t / seq) * row_capacity + row_offset + t % seq (token rows of a batch, each appended to); batch_stride is
  // then the distance of the sequences in x (with token_stride inside them)
  uint8_t* cache;
  const int64_t* slot_mapping;
  int64_t seq, batch_stride[2], row_capacity, row_offset;
  int64_t n_slots, cache_token_stride, num_cache_slots;
  int* err_flag;
};

__device__ __forceinline__ int64_t write_slot(const CompressArgs& a, int64_t tok) {
  if (a.seq == 0) return a.slot_mapping[tok];
  const unsigned b = (unsigned)tok / (unsigned)a.seq;
  return (int64_t)b * a.row_capacity + a.row_offset + ((unsigned)tok - b * (unsigned)a.seq);
}
// element offset of token `tok` in source `src`
__device__ __forceinline__ int64_t token_offset(const CompressArgs& a, int src, int64_t tok) {
  if (a.seq == 0) return tok * a.token_stride[src];
  const unsigned b = (unsigned)tok / (unsigned)a.seq;
  return (int64_t)b * a.batch_stride[src] + (int64_t)((unsigned)tok - b * (unsigned)a.seq) * a.token_stride[src];
}
// sequences of every source follow one another like tokens (always so without sequences)
inline bool tokens_uniform(const CompressArgs& a) {
  for (int s = 0; s < a.n_sources; ++s)
    if (a.seq > 0 && a.n_tokens > a.seq && a.batch_stride[s] != a.seq * a.token_stride[s]) return false;
  return true;
}

// Which kernel makes a write of so many vectors (B200, back to back, bf16):
//   a block per vector that asks for all of Pi at once up to few_rows(): 8 - 148 vectors of 128 2.8 - 3.0 us against 4.4 of the next one, 296
//     3.4 / 4.6, 444 5.1 / 4.6; of 64 2.2 / 2.7, 592 2.6 / 3.0; of 96 2.7 / 4.4, 444 3.9 / 4.9, 592 5.2 / 5.0; of 256 4.7 / 11.2, 296 8.0 / 11.3
//   a block per vector up to tiny_rows(): a few us plus 1.1 / 1.7 / 2.5 us per 1000 vectors of 64 / 96 / 128, against 8 - 14 us
//     of the tensor-core kernel; at 256 it never pays
//   the tensor-core kernel above tc_rows().  Up to kSmallRows a vector is to have the same bytes however the calls are cut, so
//     there it sums coordinates near a boundary again the FMA kernels' way, within a margin that no sum seen has left
//     (Fmt<T>::kNear; above, at head_dim 128, its bytes are its own).  At 128 that is 2 us for each that a warp has: 15.1 - 17.4 us at
//     4800 - 8192 vectors against 16.5 of the prologue kernel's one wave up to 4736 and 18.5 above.  At 256 the prologue kernel takes 15 us at 800
//   the prologue kernel in between, and up to kSmallRows for what the tensor-core kernel cannot address
constexpr int64_t kSmallRows = 8192;
constexpr int64_t tiny_rows(int head_dim) { return head_dim == 64 ? 6500 : head_dim == 96 ? 3000 : head_dim == 128 ? 4096 : 0; }
inline int64_t few_rows(int head_dim) { return (head_dim == 64 ? 4 : head_dim == 96 ? 3 : 2) * (int64_t)sm_count(); }
constexpr int64_t tc_rows(int head_dim) { return head_dim == 256 ? 1000 : head_dim == 128 ? 4736 : tiny_rows(head_dim); }
int launch_small_write(const CompressArgs& w, int head_dim, cudaStream_t st);
// `fma_bytes`: the bytes of the FMA kernels above kSmallRows, too
int dispatch_compress(const CompressArgs& a, int head_dim, int dtype, cudaStream_t st, bool fma_bytes = false);
// tensor-core (tcgen05) compress kernel for large fp32 or oddly strided inputs at head_dim 128 (tq4_compress_tc.cu)
bool compress_tc_eligible(const CompressArgs& a, int head_dim, int dtype);
int launch_compress_tc(const CompressArgs& a, int dtype, cudaStream_t st);
// pipelined tcgen05 kernel for 16-bit inputs (tq4_compress_tc16.cu)
bool compress_tc16_eligible(const CompressArgs& a, int head_dim, int dtype);
// (fma_bytes: at head_dim 128 the FMA kernels' bytes, too)
int launch_compress_tc16(const CompressArgs& a, int head_dim, int dtype, bool fma_bytes, cudaStream_t st);

}  // namespace tq4
