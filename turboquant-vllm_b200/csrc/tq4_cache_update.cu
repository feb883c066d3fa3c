// One update of a HuggingFace-style cache layer: the new K and V vectors of a step are compressed (indices and
// norms appended to their buffers) and the reconstructed vectors, which the model attends over, appended too.
//
//   norm = |x|, y = x / (norm + 1e-10) * Pi^T, idx = #{boundary < y}          as the compress kernels, bit for bit
//   z = (centroid[idx] * norm) * Pi, rounded to the type of x
//
// Takes the place of a chain of some fifty launches per update (compress, unpack, repack, decompress, a GEMM, casts,
// copies into the buffers), which bounded a step by its host time.  A warp takes four vectors, a lane D / 32
// consecutive coordinates of each; both products read Pi from shared memory (once transposed, once as
// it is; at head_dim 256, where that does not fit, in chunks of 64 rows) and the vectors from a strip per warp.
// A step of a few tokens is latency bound (staging Pi: 128 KB per block), so its vectors are spread over the blocks
// first; a prompt is bound by FMA issue.
// Measured: a generation of 8 tokens behind 4 prompts of 1100, 2 layers of 8 heads of 128, 7800 -> 730 us.
#include <math_constants.h>

#include "tq4_common.cuh"

namespace tq4 {
namespace {

struct UpdateArgs {
  const void* x[2];                    // K and V [B, H, S, D]
  int64_t batch_stride[2], head_stride[2], token_stride[2];
  const float* bounds[2];
  const float* cents[2];
  int n_bounds[2], n_cents[2], nibble[2];
  uint8_t* idx[2];                     // [B, H, cap, D / 2 or D]
  float* norms[2];                     // [B, H, cap]
  void* dec[2];                        // [B, H, dec_cap, D] in x's type, or null
  int64_t cap, dec_cap, offset, dec_offset;
  int batch, heads, n_new, dtype;
  const float* rotation;
};

// two fp32 operations an instruction, each rounded as alone
struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(F2 x, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}

template <int D, int VC_>
struct Cfg {
  static constexpr int WARPS = 8, VC = VC_, NJ = D / 32;
  static constexpr int NCH = D == 256 ? 4 : 1, KC = D / NCH;  // chunks of the reduction, rows of Pi in each
  static constexpr size_t kPi = (size_t)KC * D * 4;
  static constexpr size_t kStrip = (size_t)WARPS * D * VC * 4, kIdx = (size_t)WARPS * VC * D;
  static constexpr size_t kSmem = 2 * kPi + kStrip + kIdx;
};

template <int NJ>
__device__ __forceinline__ void load_row(const float* p, float (&v)[NJ]) {
  if constexpr (NJ == 8) {
    float a[4], b[4];
    load_n<4>(p, a);
    load_n<4>(p + 4, b);
#pragma unroll
    for (int i = 0; i < 4; ++i) { v[i] = a[i]; v[4 + i] = b[i]; }
  } else if constexpr (NJ == 3) {
#pragma unroll
    for (int i = 0; i < 3; ++i) v[i] = p[i];
  } else {
    load_n<NJ>(p, v);
  }
}

// acc[i][j] += (vectors 2 i, 2 i + 1 of the strip's entry) * ps[j]
template <int D, int NJ, int VC>
__device__ __forceinline__ void rank1(const float4* x, const float (&ps)[NJ], F2 (&acc)[VC / 2][NJ]) {
  F2 p2[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) p2[j] = pack2(ps[j], ps[j]);
#pragma unroll
  for (int g = 0; g < VC / 4; ++g) {
    const float4 x4 = x[g * D];
    const F2 lo = pack2(x4.x, x4.y), hi = pack2(x4.z, x4.w);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      acc[2 * g][j] = fma2(lo, p2[j], acc[2 * g][j]);
      acc[2 * g + 1][j] = fma2(hi, p2[j], acc[2 * g + 1][j]);
    }
  }
}

template <int D, int VC>
__global__ void __launch_bounds__(256) cache_update_kernel(const UpdateArgs a) {
  using C = Cfg<D, VC>;
  constexpr int NJ = C::NJ, G = VC / 4, KC = C::KC, NCH = C::NCH, KQ = D / 4, XPL = D / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* s_pit = reinterpret_cast<float*>(smem_raw);           // [KC][D]: Pi[j][k0 + k] at [k][j]
  float* s_pi = s_pit + KC * D;                                // [KC][D]: Pi[k0 + k][j] at [k][j]
  float4* s_x = reinterpret_cast<float4*>(s_pi + KC * D);      // [WARPS][G][D], four vectors per entry
  uint8_t* s_i = reinterpret_cast<uint8_t*>(s_x + C::WARPS * D * G);  // [WARPS][VC][D] indices
  __shared__ float s_b[2][16], s_c[2][16];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < 32) {
    const int src = tid >> 4, i = tid & 15;
    s_b[src][i] = i < a.n_bounds[src] ? a.bounds[src][i] : CUDART_INF_F;
    s_c[src][i] = i < a.n_cents[src] ? a.cents[src][i] : 0.f;
  }
  auto stage_t = [&](int ch) {  // consecutive threads = consecutive rows of Pi: conflict-free stores
    for (int i = tid; i < KC * D / 4; i += 256) {
      const int c4 = i / D, j = i - c4 * D;
      const float4 v = __ldg(reinterpret_cast<const float4*>(a.rotation + (size_t)j * D + ch * KC) + c4);
      float* dst = s_pit + 4 * c4 * D + j;
      dst[0] = v.x; dst[D] = v.y; dst[2 * D] = v.z; dst[3 * D] = v.w;
    }
  };
  auto stage = [&](int ch) {
    for (int i = tid; i < KC * D / 4; i += 256)
      reinterpret_cast<float4*>(s_pi)[i] = __ldg(reinterpret_cast<const float4*>(a.rotation + (size_t)ch * KC * D) + i);
  };
  const int per_src = a.batch * a.heads * a.n_new;
  const int chunks_src = (per_src + VC - 1) / VC, n_chunks = 2 * chunks_src;  // (a chunk holds vectors of one source)
  if (NCH == 1) {
    stage_t(0);
    stage(0);
  }
  __syncthreads();
  float4* gx = s_x + warp * D * G;
  uint8_t* gi = s_i + warp * VC * D;
  const float* pt = s_pit + NJ * lane;
  const float* pp = s_pi + NJ * lane;
  // (every warp of the block makes the same number of passes: the chunked form meets at block barriers)
  const int stride = (int)gridDim.x * C::WARPS;
  for (int base = 0; base < n_chunks; base += stride) {
    const int c = base + warp * (int)gridDim.x + (int)blockIdx.x;
    const bool act = c < n_chunks;
    const int src = act && c >= chunks_src ? 1 : 0, v0 = act ? (c - src * chunks_src) * VC : 0;
    float nrm[VC];
    int64_t at[VC];  // (b * heads + h) and token of the vector
    int tok[VC];
    {
      const void* p[VC];
#pragma unroll
      for (int v = 0; v < VC; ++v) {
        const int vec = v0 + v;
        p[v] = nullptr;
        at[v] = -1;
        tok[v] = 0;
        if (act && vec < per_src) {
          const int bh = vec / a.n_new, s = vec - bh * a.n_new, b = bh / a.heads, h = bh - b * a.heads;
          at[v] = bh;
          tok[v] = s;
          p[v] = byte_offset(a.x[src], a.dtype, (int64_t)b * a.batch_stride[src] + (int64_t)h * a.head_stride[src] +
                                                    (int64_t)s * a.token_stride[src] + lane);
        }
      }
      float xr[XPL][VC];
      if (a.dtype == TQ4_F32) load_strip<float, XPL, VC>(p, xr);
      else if (a.dtype == TQ4_F16) load_strip<__half, XPL, VC>(p, xr);
      else load_strip<__nv_bfloat16, XPL, VC>(p, xr);
#pragma unroll
      for (int v = 0; v < VC; ++v) {
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < XPL; ++i) ss = fmaf(xr[i][v], xr[i][v], ss);
        nrm[v] = sqrtf(warp_sum(ss));
        const float den = nrm[v] + 1e-10f;
#pragma unroll
        for (int i = 0; i < XPL; ++i) xr[i][v] = xr[i][v] / den;
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < XPL; ++i)
#pragma unroll
        for (int g = 0; g < G; ++g)
          gx[g * D + lane + 32 * i] = make_float4(xr[i][4 * g], xr[i][4 * g + 1], xr[i][4 * g + 2], xr[i][4 * g + 3]);
      __syncwarp();
    }
    // ---- rotate: four quarter chains, (s0 + s1) + (s2 + s3) -------------------------------------------
    F2 t[VC / 2][NJ], u[VC / 2][NJ], acc[VC / 2][NJ];
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      if (NCH > 1) {
        __syncthreads();
        stage_t(q);
        __syncthreads();
      }
#pragma unroll
      for (int v = 0; v < VC / 2; ++v)
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[v][j].v = 0;
      const float* pq = pt + (NCH > 1 ? 0 : q * KQ * D);
#pragma unroll 4
      for (int k = 0; k < KQ; ++k) {
        float ps[NJ];
        load_row<NJ>(pq + k * D, ps);
        rank1<D, NJ, VC>(gx + q * KQ + k, ps, acc);
      }
#pragma unroll
      for (int v = 0; v < VC / 2; ++v)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          if (q == 0 || q == 2) u[v][j] = acc[v][j];
          else if (q == 1) t[v][j] = add2(u[v][j], acc[v][j]);
          else t[v][j] = add2(t[v][j], add2(u[v][j], acc[v][j]));
        }
    }
    // ---- indices, norms, and what they stand for --------------------------------------------------------
    __syncwarp();
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      float r[VC], y[VC];
#pragma unroll
      for (int v = 0; v < VC / 2; ++v) unpack2(t[v][j], y[2 * v], y[2 * v + 1]);
#pragma unroll
      for (int v = 0; v < VC; ++v) {
        const int i = bucketize_sorted16(y[v], s_b[src]);
        gi[v * D + NJ * lane + j] = (uint8_t)i;
        r[v] = s_c[src][i] * nrm[v];
      }
#pragma unroll
      for (int g = 0; g < G; ++g) gx[g * D + 32 * j + lane] = make_float4(r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]);
    }
    __syncwarp();
#pragma unroll
    for (int v = 0; v < VC; ++v) {
      if (at[v] < 0) continue;
      const int64_t row = at[v] * a.cap + a.offset + tok[v];
      const uint32_t* gw = reinterpret_cast<const uint32_t*>(gi + v * D);
      if (a.nibble[src]) {  // byte p = index 2 p << 4 | index 2 p + 1
        for (int i = lane; i < D / 8; i += 32) {
          const uint32_t w0 = gw[2 * i], w1 = gw[2 * i + 1];
          const uint32_t lo = ((w0 << 4) & 0x00F000F0u) | ((w0 >> 8) & 0x000F000Fu), hi = ((w1 << 4) & 0x00F000F0u) | ((w1 >> 8) & 0x000F000Fu);
          reinterpret_cast<uint32_t*>(a.idx[src] + row * (D / 2))[i] = __byte_perm(lo, hi, 0x6420);
        }
      } else {
        for (int i = lane; i < D / 4; i += 32) reinterpret_cast<uint32_t*>(a.idx[src] + row * D)[i] = gw[i];
      }
      if (lane == 0) a.norms[src][row] = nrm[v];
    }
    // ---- un-rotate (entry 32 j + l of the strip is coordinate NJ l + j: stored without bank conflicts) ------------------------------------------------------------------------------------------
    if (a.dec[0] == nullptr) continue;
#pragma unroll
    for (int v = 0; v < VC / 2; ++v)
#pragma unroll
      for (int j = 0; j < NJ; ++j) acc[v][j].v = 0;
#pragma unroll 1
    for (int ch = 0; ch < NCH; ++ch) {
      if (NCH > 1) {
        __syncthreads();
        stage(ch);
        __syncthreads();
      }
#pragma unroll 1
      for (int j = 0; j < NJ; ++j)
#pragma unroll 4
        for (int l = 0; l < 32 / NCH; ++l) {
          float ps[NJ];
          load_row<NJ>(pp + (NJ * l + j) * D, ps);
          rank1<D, NJ, VC>(gx + 32 * j + ch * (32 / NCH) + l, ps, acc);
        }
    }
    float z[VC][NJ];
#pragma unroll
    for (int v = 0; v < VC / 2; ++v)
#pragma unroll
      for (int j = 0; j < NJ; ++j) unpack2(acc[v][j], z[2 * v][j], z[2 * v + 1][j]);
#pragma unroll
    for (int v = 0; v < VC; ++v) {
      if (at[v] < 0) continue;
      const int64_t o = (at[v] * a.dec_cap + a.dec_offset + tok[v]) * D + NJ * lane;
      if constexpr (NJ % 4 == 0) {
#pragma unroll
        for (int j = 0; j < NJ; j += 4) {
          const float y[4] = {z[v][j], z[v][j + 1], z[v][j + 2], z[v][j + 3]};
          store4(a.dec[src], a.dtype, o + j, y);
        }
      } else {
#pragma unroll
        for (int j = 0; j < NJ; ++j) store_from_float(a.dec[src], a.dtype, o + j, z[v][j]);
      }
    }
  }
}

template <int D, int VC>
int launch_update(const UpdateArgs& a, cudaStream_t st) {
  using C = Cfg<D, VC>;
  if (!ensure_dynamic_smem<cache_update_kernel<D, VC>>((int)C::kSmem)) return TQ4_ERR_CUDA;
  const int64_t chunks = 2 * (((int64_t)a.batch * a.heads * a.n_new + C::VC - 1) / C::VC);
  const int64_t most = sm_count();
  cache_update_kernel<D, VC><<<(unsigned)(chunks < most ? chunks : most), 256, C::kSmem, st>>>(a);
  TQ4_CHECK_LAUNCH();
  return TQ4_OK;
}

// Eight vectors a warp (half the reads of Pi per FMA) once every warp of the GPU has that many
template <int D>
int launch_update(const UpdateArgs& a, cudaStream_t st) {
  if constexpr (D <= 128)
    if (2 * (int64_t)a.batch * a.heads * a.n_new >= 64 * (int64_t)sm_count()) return launch_update<D, 8>(a, st);
  return launch_update<D, 4>(a, st);
}

}  // namespace
}  // namespace tq4

extern "C" int tq4_cache_update(const void* key, const void* value, int dtype, int batch, int num_heads, int n_new,
                                int head_dim, const int64_t* k_strides, const int64_t* v_strides,
                                const float* rotation, const float* k_boundaries, int n_k_boundaries,
                                const float* v_boundaries, int n_v_boundaries, const float* k_centroids,
                                int n_k_centroids, const float* v_centroids, int n_v_centroids, int k_nibble,
                                int v_nibble, uint8_t* k_idx, float* k_norms, uint8_t* v_idx, float* v_norms,
                                int64_t capacity, int64_t offset, void* k_dec, void* v_dec, int64_t dec_capacity,
                                int64_t dec_offset, void* stream) {
  using namespace tq4;
  if (batch < 0 || num_heads <= 0 || n_new < 0 || offset < 0 || dec_offset < 0) return TQ4_ERR_INVALID_ARG;
  if (!supported_head_dim(head_dim) || dtype < 0 || dtype > 2) return TQ4_ERR_UNSUPPORTED;
  if (n_k_boundaries < 0 || n_k_boundaries > TQ4_MAX_BOUNDARIES || n_v_boundaries < 0 || n_v_boundaries > TQ4_MAX_BOUNDARIES ||
      n_k_centroids <= 0 || n_k_centroids > TQ4_MAX_CENTROIDS || n_v_centroids <= 0 || n_v_centroids > TQ4_MAX_CENTROIDS)
    return TQ4_ERR_UNSUPPORTED;
  if (batch == 0 || n_new == 0) return TQ4_OK;
  if (!key || !value || !k_strides || !v_strides || !rotation || !k_boundaries || !v_boundaries || !k_centroids || !v_centroids ||
      !k_idx || !k_norms || !v_idx || !v_norms || (k_dec == nullptr) != (v_dec == nullptr))
    return TQ4_ERR_INVALID_ARG;
  if (((uintptr_t)rotation & 15) || ((uintptr_t)k_idx & 3) || ((uintptr_t)v_idx & 3) || offset + n_new > capacity ||
      (k_dec && dec_offset + n_new > dec_capacity) || (int64_t)batch * num_heads * n_new > 0x3fffffffll)
    return TQ4_ERR_INVALID_ARG;
  UpdateArgs a{};
  const void* x[2] = {key, value};
  const int64_t* strides[2] = {k_strides, v_strides};
  for (int s = 0; s < 2; ++s) {
    a.x[s] = x[s];
    a.batch_stride[s] = strides[s][0];
    a.head_stride[s] = strides[s][1];
    a.token_stride[s] = strides[s][2];
  }
  a.bounds[0] = k_boundaries; a.n_bounds[0] = n_k_boundaries;
  a.bounds[1] = v_boundaries; a.n_bounds[1] = n_v_boundaries;
  a.cents[0] = k_centroids; a.n_cents[0] = n_k_centroids;
  a.cents[1] = v_centroids; a.n_cents[1] = n_v_centroids;
  a.nibble[0] = k_nibble; a.nibble[1] = v_nibble;
  a.idx[0] = k_idx; a.idx[1] = v_idx;
  a.norms[0] = k_norms; a.norms[1] = v_norms;
  a.dec[0] = k_dec; a.dec[1] = v_dec;
  a.cap = capacity; a.offset = offset;
  a.dec_cap = dec_capacity; a.dec_offset = dec_offset;
  a.batch = batch; a.heads = num_heads; a.n_new = n_new; a.dtype = dtype;
  a.rotation = rotation;
  switch (head_dim) {
    case 64: return launch_update<64>(a, (cudaStream_t)stream);
    case 96: return launch_update<96>(a, (cudaStream_t)stream);
    case 128: return launch_update<128>(a, (cudaStream_t)stream);
    case 256: return launch_update<256>(a, (cudaStream_t)stream);
  }
  return TQ4_ERR_UNSUPPORTED;
}
