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
// A step of a few tokens is bound by latency and has a kernel of its own (cache_update_tiny_kernel); a prompt of 16-bit vectors is
// compressed by the write kernels and restored by the tensor cores (tq4_restore_tc.cu); what is left is bound by FMA issue
// and the reads of Pi.
// The kernels' own times, against the chain's (ncu: cold, serialised; bf16, 8 heads of 128, K4 / V3): a prompt of
// 4 x 1100 tokens 293 us in 26 launches -> 124 in two (16 of them the write kernel's; 36 with the tensor cores restoring), one token
// of each 103 us in 25 launches -> 11 in one.
#include <math_constants.h>

#include "tq4_cache_update.cuh"

namespace tq4 {
namespace {

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

// The same for a step of a few tokens: a block per vector, each warp one quarter of both reductions (head_dim 256: for half
// of the columns) with Pi read through L1 / L2 -- along rows of Pi^T (the even / odd halves) to rotate, along rows of Pi to
// rotate back -- in batches of four rows a lane.  Bound by latency; staging Pi for four vectors a warp, as below,
// cost 18 us for
// a token of four sequences at head_dim 128 and 63 at 256, against 5.5 and 9.
// FEW: for so few vectors that each has an SM to itself: a warp per 32 column pairs, all of its share of Pi^T (head_dim 256: half)
// asked for before anything is known of the vector, and all of Pi before the indices are found.
template <int D, bool FEW>
struct TinyCfg {
  static constexpr int CS = FEW ? (D == 96 ? 1 : D / 64) : D == 256 ? 2 : 1, WARPS = 4 * CS, THREADS = 32 * WARPS;
  static constexpr int HALF = D / 2, NBL = (HALF / CS + 31) / 32, NJ = D / 32 / CS, B = FEW ? (D == 256 ? 32 : D / 4) : 4;
};
template <int D, bool FEW>
__global__ void __launch_bounds__(TinyCfg<D, FEW>::THREADS) cache_update_tiny_kernel(const UpdateArgs a) {
  using C = TinyCfg<D, FEW>;
  constexpr int HALF = C::HALF, NBL = C::NBL, NJ = C::NJ, B = C::B, XPL = D / 32, KQ = D / 4;
  static_assert(KQ % B == 0, "whole batches");
  __shared__ __align__(16) float s_part[4][D];
  __shared__ float s_x[D], s_b[16], s_c[16];
  __shared__ uint8_t s_i[D];
  const int tid = threadIdx.x, lane = tid & 31, q = (tid >> 5) & 3, half = tid >> 7;  // quarter, column half
  const int per_src = a.batch * a.heads * a.n_new;
  const int src = (int)blockIdx.x >= per_src ? 1 : 0, vec = (int)blockIdx.x - src * per_src;
  const int bh = vec / a.n_new, s = vec - bh * a.n_new, b = bh / a.heads, h = bh - b * a.heads;
  const int64_t at = (int64_t)b * a.batch_stride[src] + (int64_t)h * a.head_stride[src] + (int64_t)s * a.token_stride[src];
  const int k0 = q * KQ, p0 = half * (HALF / C::CS) + lane;
  float pe[B][NBL], po[B][NBL];
  auto load_t = [&](int kb) {
#pragma unroll
    for (int u = 0; u < B; ++u)
#pragma unroll
      for (int i = 0; i < NBL; ++i) {
        const int p = p0 + 32 * i, k = k0 + kb + u;
        pe[u][i] = p < HALF ? __ldg(a.rot_even + k * HALF + p) : 0.f;
        po[u][i] = p < HALF ? __ldg(a.rot_odd + k * HALF + p) : 0.f;
      }
  };
  load_t(0);
  if (tid < 16) s_b[tid] = tid < a.n_bounds[src] ? a.bounds[src][tid] : CUDART_INF_F;
  else if (tid < 32) s_c[tid - 16] = tid - 16 < a.n_cents[src] ? a.cents[src][tid - 16] : 0.f;
  float xv[XPL], ss = 0.f;
#pragma unroll
  for (int i = 0; i < XPL; ++i) xv[i] = load_as_float(a.x[src], a.dtype, at + lane + 32 * i);
#pragma unroll
  for (int i = 0; i < XPL; ++i) ss = fmaf(xv[i], xv[i], ss);
  const float norm = sqrtf(warp_sum(ss)), den = norm + 1e-10f;
  if (tid < 32) {
#pragma unroll
    for (int i = 0; i < XPL; ++i) s_x[lane + 32 * i] = xv[i] / den;
  }
  __syncthreads();
  {
    float acc[2 * NBL] = {};
#pragma unroll
    for (int kb = 0; kb < KQ; kb += B) {
      if (kb > 0) load_t(kb);
#pragma unroll
      for (int u = 0; u < B; ++u) {
        const float xk = s_x[k0 + kb + u];
#pragma unroll
        for (int i = 0; i < NBL; ++i) {
          acc[2 * i] = fmaf(xk, pe[u][i], acc[2 * i]);
          acc[2 * i + 1] = fmaf(xk, po[u][i], acc[2 * i + 1]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < NBL; ++i)
      if (p0 + 32 * i < HALF) *reinterpret_cast<float2*>(&s_part[q][2 * (p0 + 32 * i)]) = make_float2(acc[2 * i], acc[2 * i + 1]);
  }
  // the first rows of Pi are on their way while the indices are found
  float pr[B][NJ];
  const int j0 = half * (D / C::CS) + lane;
  auto load_r = [&](int kb) {
#pragma unroll
    for (int u = 0; u < B; ++u)
#pragma unroll
      for (int i = 0; i < NJ; ++i) pr[u][i] = __ldg(a.rotation + (k0 + kb + u) * D + j0 + 32 * i);
  };
  if (a.dec[0] != nullptr) load_r(0);
  __syncthreads();
  for (int j = tid; j < D; j += C::THREADS) {
    const float y = (s_part[0][j] + s_part[1][j]) + (s_part[2][j] + s_part[3][j]);
    const int i = bucketize_sorted16(y, s_b);
    s_i[j] = (uint8_t)i;
    s_x[j] = s_c[i] * norm;
  }
  __syncthreads();
  const int64_t row = (int64_t)bh * a.cap + a.offset + s;
  if (a.nibble[src]) {
    for (int i = tid; i < HALF; i += C::THREADS) a.idx[src][row * HALF + i] = (uint8_t)((s_i[2 * i] << 4) | s_i[2 * i + 1]);
  } else {
    for (int i = tid; i < D; i += C::THREADS) a.idx[src][row * D + i] = s_i[i];
  }
  if (tid == 0) a.norms[src][row] = norm;
  if (a.dec[0] == nullptr) return;
  float acc[NJ] = {};
#pragma unroll
  for (int kb = 0; kb < KQ; kb += B) {
    if (kb > 0) load_r(kb);
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const float xk = s_x[k0 + kb + u];
#pragma unroll
      for (int i = 0; i < NJ; ++i) acc[i] = fmaf(xk, pr[u][i], acc[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < NJ; ++i) s_part[q][j0 + 32 * i] = acc[i];
  __syncthreads();
  const int64_t o = ((int64_t)bh * a.dec_cap + a.dec_offset + s) * D;
  for (int j = tid; j < D; j += C::THREADS)
    store_from_float(a.dec[src], a.dtype, o + j, (s_part[0][j] + s_part[1][j]) + (s_part[2][j] + s_part[3][j]));
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

// DONE: the vectors come compressed
template <int D, int VC, bool DONE>
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
    if (!DONE) stage_t(0);
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
    F2 acc[VC / 2][NJ];
    if constexpr (DONE) {
      static_assert(NJ == 4, "a lane's coordinates are two bytes");
      __syncwarp();
      float r[NJ][VC];
#pragma unroll
      for (int v = 0; v < VC; ++v) {
        const int vec = v0 + v;
        at[v] = -1;
        tok[v] = 0;
        uint32_t w = 0;
        nrm[v] = 0.f;
        if (act && vec < per_src) {
          const int bh = vec / a.n_new, s = vec - bh * a.n_new, b = bh / a.heads, h = bh - b * a.heads;
          at[v] = bh;
          tok[v] = s;
          const int64_t from = src * (int64_t)per_src + ((int64_t)b * a.n_new + s) * a.heads + h;
          w = __ldg(reinterpret_cast<const uint16_t*>(a.packed + from * (D / 2)) + lane);
          nrm[v] = __ldg(a.packed_norms + from);
        }
        // byte p = index 2 p << 4 | index 2 p + 1
        *reinterpret_cast<uint32_t*>(gi + v * D + NJ * lane) = ((w >> 4) & 15u) | (w & 15u) << 8 | ((w >> 12) & 15u) << 16 | ((w >> 8) & 15u) << 24;
        r[0][v] = s_c[src][(w >> 4) & 15] * nrm[v];
        r[1][v] = s_c[src][w & 15] * nrm[v];
        r[2][v] = s_c[src][(w >> 12) & 15] * nrm[v];
        r[3][v] = s_c[src][(w >> 8) & 15] * nrm[v];
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int g = 0; g < G; ++g) gx[g * D + 32 * j + lane] = make_float4(r[j][4 * g], r[j][4 * g + 1], r[j][4 * g + 2], r[j][4 * g + 3]);
    } else {
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
    F2 t[VC / 2][NJ], u[VC / 2][NJ];
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

template <int D, int VC, bool DONE = false>
int launch_update(const UpdateArgs& a, cudaStream_t st) {
  using C = Cfg<D, VC>;
  if (!ensure_dynamic_smem<cache_update_kernel<D, VC, DONE>>((int)C::kSmem)) return TQ4_ERR_CUDA;
  const int64_t chunks = 2 * (((int64_t)a.batch * a.heads * a.n_new + C::VC - 1) / C::VC);
  const int64_t most = sm_count();
  cache_update_kernel<D, VC, DONE><<<(unsigned)(chunks < most ? chunks : most), 256, C::kSmem, st>>>(a);
  TQ4_CHECK_LAUNCH();
  return TQ4_OK;
}

// A block per vector up to kTinyUpdate vectors (B200, bf16; 16 vectors / 1024 / 3000, against four a warp: head_dim 64 3.5 / 4.4 /
// 8.8 and 10.1 us, 96 4.4 / 6.6 / 14.7 and 14.0, 128 5.4 / 8.5 / 19 and 19, 256 8.7 / 27 / 68 and 65).  Eight vectors a warp
// (half the reads of Pi per FMA) once every warp of the GPU has that many.
constexpr int64_t kTinyUpdate = 2800;
// The form with all loads in flight at once up to so many vectors an SM (8 - 64 vectors / 148 / 296 / 592, without and with it: head_dim 64
// 3.5 / 3.5 / 3.6 / 3.8 and 2.7 / 2.8 / 2.9 / 3.2 us, 96 4.5 / 4.9 / 5.0 / 5.5 and 3.2 / 3.3 / 3.8 / 4.7, 128 5.4 / 5.5 / 5.8 / 6.2 and 3.7 / 3.8 / 4.5 /
// 7.1, 256 8.7 / 9.0 / 9.5 / 15.9 and 6.7 / 6.9 / 12.3 / 23.2).
template <int D> constexpr int kFewUpdate = D == 256 ? 1 : D == 128 ? 2 : 4;
template <int D>
int launch_update(const UpdateArgs& a, cudaStream_t st) {
  const int64_t vectors = 2 * (int64_t)a.batch * a.heads * a.n_new;
  if (vectors <= kFewUpdate<D> * (int64_t)sm_count()) {
    cache_update_tiny_kernel<D, true><<<(unsigned)vectors, TinyCfg<D, true>::THREADS, 0, st>>>(a);
    TQ4_CHECK_LAUNCH();
    return TQ4_OK;
  }
  if (vectors <= kTinyUpdate) {
    cache_update_tiny_kernel<D, false><<<(unsigned)vectors, TinyCfg<D, false>::THREADS, 0, st>>>(a);
    TQ4_CHECK_LAUNCH();
    return TQ4_OK;
  }
  if constexpr (D == 128)
    if (a.packed) return launch_update<D, 8, true>(a, st);
  if constexpr (D <= 128)
    if (vectors >= 64 * (int64_t)sm_count()) return launch_update<D, 8>(a, st);
  return launch_update<D, 4>(a, st);
}

// The compression that the tensor cores do for a tensor by itself (dispatch_compress, head_dim 128 above kSmallRows
// vectors) is theirs here, too: the indices are those of tq4_compress of that tensor, and half of the FMAs go away (8 tokens
// behind 4 x 1100, 2 layers: 486 -> 452 us).  A paged write counts K and V together, so between 4097 and 8192 vectors a
// tensor its indices are the tensor cores' and may differ from these, within the write path's bound.
bool compress_first(int batch, int heads, int n_new, int head_dim) {
  return head_dim == 128 && (int64_t)batch * heads * n_new > kSmallRows;
}
// Otherwise it pays where the tensor cores restore, too (restore_tc_kernel): once the FMA kernel would take a second pass (four vectors
// a warp of every SM).  K and V of 8 heads, bf16, FMA kernel / compressed first: 4000 vectors of 128 20.7 / 22.7 us, 6400 35.0 / 22.7,
// 14 400 53 / 24; of 64 12.4 / 12.9, 18.6 / 16.5, 24.7 / 16.6; of 96 16.3 / 20.6, 25.5 / 20.7, 41 / 20.7.  The indices are the FMA
// kernels' (fma_bytes).
bool restore_pays(int batch, int heads, int n_new, int head_dim) {
  return head_dim <= 128 && 2 * (int64_t)batch * heads * n_new > 32 * (int64_t)sm_count();
}
size_t scratch_norms(int batch, int heads, int n_new) { return ((size_t)2 * batch * heads * n_new * sizeof(float) + 15) & ~(size_t)15; }

}  // namespace
}  // namespace tq4

extern "C" size_t tq4_cache_update_scratch_bytes(int batch, int num_heads, int n_new, int head_dim) {
  using namespace tq4;
  if (batch <= 0 || num_heads <= 0 || n_new <= 0) return 0;
  if (!compress_first(batch, num_heads, n_new, head_dim) && !restore_pays(batch, num_heads, n_new, head_dim)) return 0;
  return scratch_norms(batch, num_heads, n_new) + (size_t)2 * batch * num_heads * n_new * (head_dim / 2);
}

extern "C" int tq4_cache_update(const void* key, const void* value, int dtype, int batch, int num_heads, int n_new,
                                int head_dim, const int64_t* k_strides, const int64_t* v_strides,
                                const float* rotation, const float* rot_t_even, const float* rot_t_odd,
                                const float* k_boundaries, int n_k_boundaries,
                                const float* v_boundaries, int n_v_boundaries, const float* k_centroids,
                                int n_k_centroids, const float* v_centroids, int n_v_centroids, int k_nibble,
                                int v_nibble, uint8_t* k_idx, float* k_norms, uint8_t* v_idx, float* v_norms,
                                int64_t capacity, int64_t offset, void* k_dec, void* v_dec, int64_t dec_capacity,
                                int64_t dec_offset, void* scratch, size_t scratch_bytes, void* stream) {
  using namespace tq4;
  if (batch < 0 || num_heads <= 0 || n_new < 0 || offset < 0 || dec_offset < 0) return TQ4_ERR_INVALID_ARG;
  if (!supported_head_dim(head_dim) || dtype < 0 || dtype > 2) return TQ4_ERR_UNSUPPORTED;
  if (n_k_boundaries < 0 || n_k_boundaries > TQ4_MAX_BOUNDARIES || n_v_boundaries < 0 || n_v_boundaries > TQ4_MAX_BOUNDARIES ||
      n_k_centroids <= 0 || n_k_centroids > TQ4_MAX_CENTROIDS || n_v_centroids <= 0 || n_v_centroids > TQ4_MAX_CENTROIDS)
    return TQ4_ERR_UNSUPPORTED;
  if (batch == 0 || n_new == 0) return TQ4_OK;
  if (!key || !value || !k_strides || !v_strides || !rotation || !rot_t_even || !rot_t_odd || !k_boundaries || !v_boundaries || !k_centroids || !v_centroids ||
      !k_idx || !k_norms || !v_idx || !v_norms || (k_dec == nullptr) != (v_dec == nullptr))
    return TQ4_ERR_INVALID_ARG;
  if ((((uintptr_t)rotation | (uintptr_t)rot_t_even | (uintptr_t)rot_t_odd) & 15) || ((uintptr_t)k_idx & 3) || ((uintptr_t)v_idx & 3) || offset + n_new > capacity ||
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
  a.rot_even = rot_t_even;
  a.rot_odd = rot_t_odd;
  const bool must = compress_first(batch, num_heads, n_new, head_dim);
  const bool room = scratch && ((uintptr_t)scratch & 15) == 0 && scratch_bytes >= tq4_cache_update_scratch_bytes(batch, num_heads, n_new, head_dim);
  if (must && !room) return TQ4_ERR_WORKSPACE;
  a.packed = (const uint8_t*)scratch + scratch_norms(batch, num_heads, n_new);
  const bool restore = room && restore_tc_eligible(a, head_dim) && (must || restore_pays(batch, num_heads, n_new, head_dim));
  a.packed = nullptr;
  if (must || restore) {
    CompressArgs c{};
    for (int i = 0; i < 2; ++i) {
      c.x[i] = a.x[i];
      c.batch_stride[i] = a.batch_stride[i];
      c.head_stride[i] = a.head_stride[i];
      c.token_stride[i] = a.token_stride[i];
      c.bounds[i] = a.bounds[i];
      c.n_bounds[i] = a.n_bounds[i];
    }
    c.n_tokens = (int64_t)batch * n_new;
    c.num_heads = num_heads;
    c.n_sources = 2;
    c.x_dtype = dtype;
    c.rot_even = rot_t_even;
    c.rot_odd = rot_t_odd;
    c.seq = n_new;
    for (int i = 0; n_new == 1 && i < 2; ++i) c.token_stride[i] = c.batch_stride[i];  // the sequences are the tokens
    c.norms_out = (float*)scratch;
    c.packed_out = (uint8_t*)scratch + scratch_norms(batch, num_heads, n_new);
    const int rc = dispatch_compress(c, head_dim, dtype, (cudaStream_t)stream, !must);
    if (rc != TQ4_OK) return rc;
    a.packed = c.packed_out;
    a.packed_norms = c.norms_out;
    if (restore) return launch_restore_tc(a, head_dim, (cudaStream_t)stream);
  }
  switch (head_dim) {
    case 64: return launch_update<64>(a, (cudaStream_t)stream);
    case 96: return launch_update<96>(a, (cudaStream_t)stream);
    case 128: return launch_update<128>(a, (cudaStream_t)stream);
    case 256: return launch_update<256>(a, (cudaStream_t)stream);
  }
  return TQ4_ERR_UNSUPPORTED;
}
