// Paged TQ4 attention of a small decode step: one cluster of CTAs per (query row, KV head).
//
// The streaming kernel (tq4_decode_mma.cu) cuts all tiles of a call into equal spans, writes partials and leaves them to a merge
// kernel.  A small call pays for that with its starts: three dependent kernels of one-shot code, the second of which takes whole
// SMs and can start only when the first is gone (1 x 1024 tokens of 28 / 4 heads: prologue 4.8, attention 9, merge 5 us).
// Here the keys of a (row, KV head) are cut over the CTAs of a cluster, each CTA's tiles go round its eight warps, and the
// partials are merged, un-rotated and stored through distributed shared memory by the same kernel.  The byte -> half2 tables are
// built and the first pages looked up while the prologue kernel, which hands the queries over as fp16 terms in the order of the
// MMA fragments, is still running; a call without a write needs no kernel in front (ROT).
//
// The arithmetic is the streaming kernel's (byte -> half2 table, both products on mma.sync with hi / lo split queries and
// probabilities, lazy softmax reference).  A lane loads its own bytes of a tile straight into registers, the next tile's while
// this one is computed: no ring and no copies to wait for, but with one tile a warp in flight a call is bound by latency, and long
// contexts are the streaming kernel's (see decode_step_cluster).
//
// A step with the write of its new tokens, us (before: streaming and merge kernels, a prologue that loaded Pi in steps):
//   1 x 1024, 28 / 4 heads  18.5 -> 12.4      1 x 700, 32 / 8  18.5 -> 10.3      4 x 1000, 32 / 8  21.4 -> 14.4
//   8 x 500, 32 / 8  20.7 -> 14.4      16 x 2000, 4 / 1  24.9 -> 16.2      8 x 1000, 14 / 2 of 64  18.5 -> 12.3
// Of the 12 us about 4 are the prologue, 1 the loads, 1 a tile, 3 the merges and the product with Pi.
#include <math_constants.h>

#include "tq4_mma.cuh"

namespace tq4 {
namespace {

constexpr int kStepWarps = 8, kStepThreads = 32 * kStepWarps;
constexpr int kStepMaxCluster = 8;
constexpr uint32_t kStepTable = 65536;

template <int D, int NB>
struct StepCfg {
  static constexpr int GC = 4 * NB;                                   // query heads of a unit, at most
  static constexpr uint32_t kVec = GC * D * 4;                        // one set of partial outputs
  static_assert(kStepWarps * kVec <= kStepTable, "the warps' partials lie where the table was");
  static constexpr uint32_t smem(int cluster, bool rot) { return kStepTable + (uint32_t)(cluster + 1) * kVec + (rot ? kVec : 0u); }
  // rotation inside (as the prologue kernel's queries, bit for bit): lanes of a row of Pi, rows a warp's load covers, float4 a lane
  static constexpr int RPL = D == 64 ? 2 : 1, GL = 32 / RPL, F4 = D == 256 ? 2 : 1;
};

__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void peer_store4(uint32_t addr, const float4& v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void peer_store2(uint32_t addr, float x, float y) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(x), "f"(y) : "memory");
}

// Sequence and visible keys of query row r (every lane of the warp calls it; raw_len: the length of sequence r, fetched ahead).
__device__ __forceinline__ void step_row_range(const AttnArgs& a, int r, int lane, int raw_len, int& seq, int& start, int& end) {
  const int gr = r + a.sh.row_offset;
  seq = start = end = 0;
  if (a.query_start_loc == nullptr) {
    if (gr >= a.sh.num_seqs) return;
    seq = gr;
    const int len = clamp_seq_len(a, max(0, raw_len));
    end = len;
    start = a.sliding_window > 0 ? max(0, len - a.sliding_window) : 0;
    return;
  }
  int n = 0;  // offsets up to the row's own: the sequence's and those before it
  for (int i = lane; i < ((a.sh.num_seqs + 31) & ~31); i += 32)
    n += __popc(__ballot_sync(0xffffffffu, i < a.sh.num_seqs && __ldg(a.query_start_loc + i) <= gr));
  if (n == 0 || gr >= __ldg(a.query_start_loc + a.sh.num_seqs)) return;
  seq = n - 1;
  const int q0 = __ldg(a.query_start_loc + seq), q1 = __ldg(a.query_start_loc + seq + 1);
  const int len = clamp_seq_len(a, max(0, __ldg(a.seq_lens + seq)));
  const int pos = len - (q1 - q0) + (gr - q0);
  end = max(0, min(a.causal ? pos + 1 : len, len));
  start = min(a.sliding_window > 0 ? max(0, pos + 1 - a.sliding_window) : 0, end);
}

// ROT: no kernel in front (a call without a write); every CTA rotates the queries of its unit
template <int D, int NB, bool ALIGNED, bool ROT>
__global__ void __launch_bounds__(kStepThreads, D * NB <= 128 ? 2 : 1)
decode_step_kernel(const __grid_constant__ AttnArgs a, const int cl_shift) {
  using C = MmaCfg<D, ALIGNED>;
  using S = StepCfg<D, NB>;
  constexpr int GC = S::GC;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ float s_cent[2][TQ4_MAX_CENTROIDS];
  __shared__ float s_m[kStepWarps][GC], s_l[kStepWarps][GC];   // of the warps
  __shared__ __align__(8) float2 s_ml[kStepMaxCluster][GC];    // (m, l) of the cluster's CTAs
  float* s_o = reinterpret_cast<float*>(smem);                 // [warps][GC][D], once the table is no longer read
  float* s_x = reinterpret_cast<float*>(smem + kStepTable);    // [GC][D] merged vectors
  __half* s_q = reinterpret_cast<__half*>(s_x + GC * D);       // ROT: [GC][hi, lo][D]
  float* s_all = s_x + (ROT ? 2 : 1) * GC * D;                 // [cluster][GC][D]
  __shared__ float s_scale[GC];                                // ROT: what the terms lack to the rotated queries
  const AttnShape& sh = a.sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, c = lane & 3;
  const int cl = 1 << cl_shift, rank = (int)blockIdx.x & (cl - 1), unit = (int)blockIdx.x >> cl_shift;
  // (the peers have started once the wait in front of the exchange passes)
  if (cl > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");

  const int n_vh = sh.Hkv * sh.NCH;
  const int r = unit / n_vh, vh = unit - r * n_vh;
  const int kvh = vh / sh.NCH, chunk = vh % sh.NCH;
  const int qh0 = kvh * sh.G + chunk * sh.GC;
  const int gcount = min(sh.GC, sh.G - chunk * sh.GC);
  // ---- ROT: this warp's rows of Pi and the raw queries on their way ---------------------------------------
  constexpr int GL = S::GL, RPL = S::RPL, F4 = S::F4, RB = D == 256 ? 2 : 4;  // (RB row sets ahead)
  constexpr int SETS = D / RPL / kStepWarps;                                  // of a warp
  static_assert(SETS % RB == 0, "whole batches");
  const int l4 = lane % GL;
  const bool lact = l4 < D / 4 / F4;
  float4 pi_r[ROT ? RB : 1][F4], xq[ROT ? GC : 1][F4];
  uint4 raw[ROT ? GC : 1][F4];
  auto load_pi = [&](int set, float4 (&x)[F4]) {
#pragma unroll
    for (int f = 0; f < F4; ++f)
      x[f] = lact ? __ldg(reinterpret_cast<const float4*>(a.rotation + (size_t)(RPL * (warp * SETS + set) + lane / GL) * D) + l4 + GL * f)
                  : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  if constexpr (ROT) {
#pragma unroll
    for (int i = 0; i < RB; ++i) load_pi(i, pi_r[i]);
    const int64_t at = ((int64_t)r + sh.row_offset) * a.q_token_stride + (int64_t)qh0 * a.q_head_stride;
#pragma unroll
    for (int h = 0; h < GC; ++h)
#pragma unroll
      for (int f = 0; f < F4; ++f)
        raw[h][f] = lact && h < gcount ? load4_raw(a.q, a.q_dtype, at + (int64_t)h * a.q_head_stride + 4 * (l4 + GL * f)) : make_uint4(0u, 0u, 0u, 0u);
  }
  const int gr = r + sh.row_offset;
  const int raw_len = a.query_start_loc == nullptr && gr < sh.num_seqs ? __ldg(a.seq_lens + gr) : 0;  // (arrives during the tables)

  // ---- replicated byte -> half2 tables (as the streaming kernel's) -------------------------------------
  if (tid < 2 * TQ4_MAX_CENTROIDS) {
    const int w = tid >> 4, i = tid & 15;
    const float* cent = w ? a.v_centroids : a.k_centroids;
    s_cent[w][i] = i < (w ? a.n_v_centroids : a.n_k_centroids) ? __fmul_rn(w ? a.lut_scale_v : a.lut_scale_k, cent[i]) : 0.f;
  }
  __syncthreads();
  {
    uint4* t = reinterpret_cast<uint4*>(smem);
#pragma unroll 4
    for (int i = tid; i < 256 * 16; i += kStepThreads) {
      const int byte = i >> 4, w = (i >> 3) & 1;
      const uint32_t v = pack_h2(s_cent[w][byte >> 4], s_cent[w][byte & 15]);
      t[i] = make_uint4(v, v, v, v);
    }
  }
  __syncthreads();
  // ---- the CTA's tiles; the first page id arrives during the rotation, or the wait for the kernel in front ------------
  int seq, kv_start, kv_end;
  step_row_range(a, r, lane, raw_len, seq, kv_start, kv_end);
  const int32_t* bt = a.block_table + (int64_t)seq * a.bt_stride;
  const int tile0 = kv_start / kTileTokens;
  const int n_tiles = kv_end > kv_start ? (kv_end + kTileTokens - 1) / kTileTokens - tile0 : 0;
  const int per = (n_tiles + cl - 1) >> cl_shift, p_end = min(n_tiles, (rank + 1) * per);
  int p = rank * per + warp;  // tile of the row
  const int bs_shift = (a.block_size & (a.block_size - 1)) == 0 ? __ffs(a.block_size) - 1 : -1;
  auto page_of = [&](int tile) -> int {
    const int pos = (tile0 + tile) * kTileTokens;
    return __ldg(bt + (bs_shift >= 0 ? pos >> bs_shift : pos / a.block_size));
  };
  int blk = p < p_end ? page_of(p) : 0;

  if constexpr (!ROT) pdl_wait();  // the rotated queries and the written tokens come from the kernel in front

  if constexpr (ROT) {
    // ---- rotate: a row of Pi times the queries, folded over the lanes ---------------------------------------------------
    float sc[GC];
#pragma unroll
    for (int h = 0; h < GC; ++h) {
      float top = 0.f;
#pragma unroll
      for (int f = 0; f < F4; ++f) xq[h][f] = raw_as_float4(raw[h][f], a.q_dtype);
#pragma unroll
      for (int f = 0; f < F4; ++f) top = fmaxf(fmaxf(fmaxf(fabsf(xq[h][f].x), fabsf(xq[h][f].y)), fmaxf(fabsf(xq[h][f].z), fabsf(xq[h][f].w))), top);
#pragma unroll
      for (int o = GL / 2; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      const int e = top > 0.f && top < CUDART_INF_F ? min(max((int)(__float_as_uint(top) >> 23) - 127, -100), 100) : 0;
      sc[h] = __uint_as_float((uint32_t)(127 + 4 - e) << 23);  // (terms of at most 2^5 sqrt(D))
      if (tid == 0) s_scale[h] = __uint_as_float((uint32_t)(127 - 4 + e) << 23);
    }
#pragma unroll 1
    for (int i0 = 0; i0 < SETS; i0 += RB) {
#pragma unroll
      for (int u = 0; u < RB; ++u) {
        float t[GC];
#pragma unroll
        for (int h = 0; h < GC; ++h) {
          t[h] = 0.f;
#pragma unroll
          for (int f = 0; f < F4; ++f)
            t[h] = fmaf(xq[h][f].x, pi_r[u][f].x, fmaf(xq[h][f].y, pi_r[u][f].y, fmaf(xq[h][f].z, pi_r[u][f].z, fmaf(xq[h][f].w, pi_r[u][f].w, t[h]))));
        }
        if (i0 + RB < SETS) load_pi(i0 + RB + u, pi_r[u]);
        int n = 0, o = GL / 2;  // head that the lane ends up with
#pragma unroll
        for (int k = GC / 2; k > 0; k >>= 1) {
          const bool up = lane & o;
#pragma unroll
          for (int h = 0; h < k; ++h) {
            const float mine = up ? t[h + k] : t[h], other = up ? t[h] : t[h + k];
            t[h] = mine + __shfl_xor_sync(0xffffffffu, other, o);
          }
          n += up ? k : 0;
          o >>= 1;
        }
        float y = t[0];
#pragma unroll
        for (; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
        float f = sc[0];
#pragma unroll
        for (int h = 1; h < GC; ++h) f = n == h ? sc[h] : f;
        const float z = y * f;
        const __half hi = __float2half_rn(z), lo = __float2half_rn(z - __half2float(hi));
        if (l4 % (GL / GC) == 0) {  // (GL / GC lanes hold the same)
          __half* to = s_q + 2 * n * D + RPL * (warp * SETS + i0 + u) + lane / GL;
          to[0] = hi;
          to[D] = lo;
        }
      }
    }
  }

  // ---- bytes of a tile: lane-constant offsets from the tile's first row ---------------------------------
  const RowLayout lay = row_layout(sh.Hkv, D);
  const uint32_t ts = (uint32_t)a.cache_token_stride;
  const uint32_t o_k = g * ts + lay.k_idx + kvh * C::HALF + c * C::KBY;
  const uint32_t o_n = g * ts + lay.k_norm + kvh * 4, vn_delta = lay.v_norm - lay.k_norm;
  const uint32_t o_v = 2 * c * ts + lay.v_idx + kvh * C::HALF;
  uint32_t kw[2][C::KW], vw[4][C::VW + C::VH];
  float nrm[4];  // kn(g), kn(g + 8), vn(g), vn(g + 8)
  auto tile_ptr = [&](int tile, int b) -> const uint8_t* {
    const int pos = (tile0 + tile) * kTileTokens;
    const int in = bs_shift >= 0 ? (pos & (a.block_size - 1)) : pos % a.block_size;
    return a.cache + (int64_t)((uint32_t)b < (uint32_t)a.num_blocks ? b : 0) * a.cache_block_stride + (int64_t)in * a.cache_token_stride;
  };
  auto load_k = [&](const uint8_t* t) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int i = 0; i < C::NK; ++i) {
        const uint8_t* q = t + (o_k + 8 * h * ts) + i * C::UK;
        uint32_t* d = kw[h] + i * (C::UK / 4);
        if constexpr (C::UK == 16) {
          const uint4 v = __ldcg(reinterpret_cast<const uint4*>(q));
          d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
        } else if constexpr (C::UK == 8) {
          const uint2 v = __ldcg(reinterpret_cast<const uint2*>(q));
          d[0] = v.x; d[1] = v.y;
        } else {
          d[0] = __ldcg(reinterpret_cast<const uint32_t*>(q));
        }
      }
      nrm[h] = __ldcg(reinterpret_cast<const float*>(t + (o_n + 8 * h * ts)));
      nrm[2 + h] = __ldcg(reinterpret_cast<const float*>(t + (o_n + 8 * h * ts + vn_delta)));
    }
  };
  auto load_v = [&](const uint8_t* t) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // tokens 2c, 2c+1, 2c+8, 2c+9
      const uint8_t* q = t + (o_v + ((j & 1) + 8 * (j >> 1)) * ts);
#pragma unroll
      for (int i = 0; i < C::NV; ++i) {
        const uint8_t* x = q + g * 4 * C::VW + i * C::UV;
        uint32_t* d = vw[j] + i * (C::UV / 4);
        if constexpr (C::UV == 16) {
          const uint4 v = __ldcg(reinterpret_cast<const uint4*>(x));
          d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
        } else if constexpr (C::UV == 8) {
          const uint2 v = __ldcg(reinterpret_cast<const uint2*>(x));
          d[0] = v.x; d[1] = v.y;
        } else {
          d[0] = __ldcg(reinterpret_cast<const uint32_t*>(x));
        }
      }
      if constexpr (C::VH > 0)  // D = 96: the word that holds the thread's last two bytes
        vw[j][C::VW] = __ldcg(reinterpret_cast<const uint32_t*>(q + 32 * C::VW + 4 * (g >> 1)));
    }
  };
  auto page_ok = [&](int b) -> bool {  // (a page out of range is reported and its tile masked)
    const bool ok = (uint32_t)b < (uint32_t)a.num_blocks;
    if (!ok && a.err_flag) atomicOr(a.err_flag, TQ4_DEV_BAD_BLOCK);
    return ok;
  };
  bool okm = true;
  if (p < p_end) {
    const uint8_t* t = tile_ptr(p, blk);
    load_k(t);
    load_v(t);
    okm = page_ok(blk);
    if (p + kStepWarps < p_end) blk = page_of(p + kStepWarps);
  }

  if constexpr (ROT) __syncthreads();  // the terms are there

  // ---- query fragments: column g of n-block nb = head nb*4 + g/2, term g%2 (hi / lo) ------------------
  uint32_t qf[NB][C::KS][2];
  float fscale[NB];
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    const int hh = nb * 4 + (g >> 1);
    const float* terms = ROT ? reinterpret_cast<const float*>(s_q) + hh * D : a.plan.q_rot + ((int64_t)r * sh.Hq + qh0 + hh) * D;
    const uint4* src = reinterpret_cast<const uint4*>(terms + (g & 1) * (D / 2) + c * (C::DPT / 2));
#pragma unroll
    for (int j = 0; j < C::DPT / 8; ++j) {
      const uint4 x = hh >= gcount ? make_uint4(0u, 0u, 0u, 0u) : ROT ? src[j] : __ldcg(src + j);
      qf[nb][2 * j][0] = x.x; qf[nb][2 * j][1] = x.y;
      qf[nb][2 * j + 1][0] = x.z; qf[nb][2 * j + 1][1] = x.w;
    }
    const int hc = nb * 4 + c;  // the head of this lane's scores
    fscale[nb] = (hc >= gcount ? 0.f : ROT ? s_scale[hc] : __ldcg(a.plan.part_l + (int64_t)r * sh.Hq + qh0 + hc)) * (a.scale_log2e / a.lut_scale_k);
  }
  float m[NB], l[NB], acc[C::MB][NB][4];
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    m[nb] = -CUDART_INF_F;
    l[nb] = 0.f;
#pragma unroll
    for (int i = 0; i < C::MB; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][nb][e] = 0.f;
  }
  // one table load per byte: byte B of w into bits 8 - 15 of the offset, the lane's copy below
  const uint32_t lb_k = lane * 4, lb_v = 128 + lane * 4;
  auto lut = [&](uint32_t w, int byte, uint32_t lb) -> uint32_t {
    return *reinterpret_cast<const uint32_t*>(smem + __byte_perm(w, lb, 0x7604 | (byte << 4)));
  };

  for (; p < p_end; p += kStepWarps) {
    const int pos0 = (tile0 + p) * kTileTokens;
    const bool more = p + kStepWarps < p_end;
    // ---- scores ---------------------------------------------------------------------------------------
    float sacc[NB][2][4];  // two independent accumulation chains per n-block
#pragma unroll
    for (int w = 0; w < C::KW; ++w) {
      const uint32_t w0 = kw[0][w], w1 = kw[1][w];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const uint32_t a0 = lut(w0, 2 * s, lb_k), a2 = lut(w0, 2 * s + 1, lb_k);
        const uint32_t a1 = lut(w1, 2 * s, lb_k), a3 = lut(w1, 2 * s + 1, lb_k);
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          if (w == 0) mma16816_zero(sacc[nb][s], a0, a1, a2, a3, qf[nb][s][0], qf[nb][s][1]);
          else mma16816(sacc[nb][s], a0, a1, a2, a3, qf[nb][2 * w + s][0], qf[nb][2 * w + s][1]);
        }
      }
    }
    float kn[2], vn[2], lg[2], bias[2];
    const bool full = pos0 >= kv_start && pos0 + kTileTokens <= kv_end && okm;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int pp = pos0 + g + 8 * h;
      const bool ok = full || (okm && pp >= kv_start && pp < kv_end);  // (first / last tiles of a row, bad page)
      kn[h] = ok ? nrm[h] : 0.f;
      vn[h] = ok ? nrm[2 + h] : 0.f;
      bias[h] = ok ? 0.f : -CUDART_INF_F;
      lg[h] = fmaxf(lg2_approx(vn[h]), -30.f);
    }
    // the next tile's bytes take the place of this one's as soon as these are used
    const uint8_t* t = nullptr;
    if (more) {
      t = tile_ptr(p + kStepWarps, blk);
      okm = page_ok(blk);
      load_k(t);
      if (p + 2 * kStepWarps < p_end) blk = page_of(p + 2 * kStepWarps);
    }
    // ---- online softmax with a lazily updated reference ----------------------------------------------
    float s[NB][2];
    bool need = false;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float dot = (sacc[nb][0][2 * h] + sacc[nb][1][2 * h]) + (sacc[nb][0][2 * h + 1] + sacc[nb][1][2 * h + 1]);
        s[nb][h] = fmaf(dot, fscale[nb] * kn[h], bias[h]);  // masked: -inf
        need |= s[nb][h] + lg[h] > m[nb] + 8.f;
      }
    if (__any_sync(0xffffffffu, need)) {
      asm volatile("" ::: "memory");  // rare path: keep it a real branch
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        float mt = fmaxf(s[nb][0] + lg[0], s[nb][1] + lg[1]);
        mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 4));
        mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 8));
        mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 16));
        if (mt > m[nb] + 8.f) {  // uniform over the 8 lanes that share head c
          const float alpha = m[nb] == -CUDART_INF_F ? 0.f : ex2_approx(m[nb] - mt);
          m[nb] = mt;
          l[nb] *= alpha;
#pragma unroll
          for (int i = 0; i < C::MB; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) asm volatile("mul.f32 %0, %0, %1;" : "+f"(acc[i][nb][e]) : "f"(alpha));
        }
      }
    }
    uint32_t pf[NB][2];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const float m_use = m[nb] == -CUDART_INF_F ? 0.f : m[nb];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float e = ex2_approx(s[nb][h] - m_use);
        l[nb] += e;
        pf[nb][h] = movmatrix_trans(split_h2(e * vn[h]));
      }
    }
    // ---- O^T += V^T * Psplit^T ------------------------------------------------------------------------
#pragma unroll
    for (int w = 0; w < C::VW + C::VH; ++w) {
      uint32_t x0 = vw[0][w], y0 = vw[1][w], x1 = vw[2][w], y1 = vw[3][w];
      if (w == C::VW) {
        const int sft = (g & 1) * 16;
        x0 >>= sft; y0 >>= sft; x1 >>= sft; y1 >>= sft;
      }
      const uint32_t ee0 = (x0 & 0xF0F0F0F0u) | ((y0 >> 4) & 0x0F0F0F0Fu);
      const uint32_t oo0 = ((x0 << 4) & 0xF0F0F0F0u) | (y0 & 0x0F0F0F0Fu);
      const uint32_t ee1 = (x1 & 0xF0F0F0F0u) | ((y1 >> 4) & 0x0F0F0F0Fu);
      const uint32_t oo1 = ((x1 << 4) & 0xF0F0F0F0u) | (y1 & 0x0F0F0F0Fu);
#pragma unroll
      for (int J = 0; J < 4; ++J)
        if (4 * w + J < C::MB) {
          const uint32_t a0 = lut(ee0, J, lb_v), a1 = lut(oo0, J, lb_v), a2 = lut(ee1, J, lb_v), a3 = lut(oo1, J, lb_v);
#pragma unroll
          for (int nb = 0; nb < NB; ++nb) mma16816(acc[4 * w + J][nb], a0, a1, a2, a3, pf[nb][0], pf[nb][1]);
        }
    }
    if (more) load_v(t);
  }

  // ---- the warps' partials, merged to the CTA's ------------------------------------------------------------
  __syncthreads();  // the table has been read
  const float inv_av = 1.f / a.lut_scale_v;
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    float ls = l[nb];
    ls += __shfl_xor_sync(0xffffffffu, ls, 4);
    ls += __shfl_xor_sync(0xffffffffu, ls, 8);
    ls += __shfl_xor_sync(0xffffffffu, ls, 16);
    const int hh = nb * 4 + c;
    if (g == 0) {
      s_m[warp][hh] = m[nb];
      s_l[warp][hh] = ls;
    }
    float* dst = s_o + (warp * GC + hh) * D;
#pragma unroll
    for (int i = 0; i < C::MB; ++i)
      *reinterpret_cast<float2*>(dst + 2 * v_byte_of_mblock<D>(g, i)) =
          make_float2((acc[i][nb][0] + acc[i][nb][1]) * inv_av, (acc[i][nb][2] + acc[i][nb][3]) * inv_av);
  }
  // this CTA's columns of the result and its share of the sum over the rows of Pi
  const int dc = D >> cl_shift, c0 = rank * dc;
  const int jps = (256 / (D == 96 ? 128 : D)) << cl_shift, jn = D / jps;
  const int jp = tid / dc, cc = tid - jp * dc;
  const bool act = jp < jps && !a.out_rotated;
  const float* pi = a.rotation + (int64_t)(jp * jn) * D + c0 + cc;
  constexpr int PB = 8;
  float pr[PB];
#pragma unroll
  for (int i = 0; i < PB; ++i) pr[i] = act && i < jn ? __ldg(pi + i * D) : 0.f;  // in flight during the merge
  __syncthreads();
  if (cl > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  for (int i = tid; i < gcount * (D / 4); i += kStepThreads) {
    const int h = i / (D / 4), d = 4 * (i - h * (D / 4));
    float mw[kStepWarps], M = -CUDART_INF_F, L = 0.f;
#pragma unroll
    for (int w = 0; w < kStepWarps; ++w) {
      mw[w] = s_m[w][h];
      M = fmaxf(M, mw[w]);
    }
    const float m_use = M == -CUDART_INF_F ? 0.f : M;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < kStepWarps; ++w) {
      const float e = ex2_approx(mw[w] - m_use);
      const float4 x = *reinterpret_cast<const float4*>(s_o + (w * GC + h) * D + d);
      L = fmaf(s_l[w][h], e, L);
      o.x = fmaf(x.x, e, o.x); o.y = fmaf(x.y, e, o.y); o.z = fmaf(x.z, e, o.z); o.w = fmaf(x.w, e, o.w);
    }
    if (cl == 1) {
      const float inv = L > 0.f ? 1.f / L : 0.f;
      *reinterpret_cast<float4*>(s_x + h * D + d) = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
      if (d == 0 && a.lse_out)
        a.lse_out[((int64_t)r + sh.row_offset) * sh.Hq + qh0 + h] = L > 0.f ? (M + log2f(L)) * 0.6931471805599453f : -CUDART_INF_F;
    } else {
      const uint32_t at = smem_u32(s_all + (rank * GC + h) * D + d), at_ml = smem_u32(&s_ml[rank][h]);
#pragma unroll 4
      for (int q = 0; q < cl; ++q) {
        peer_store4(peer_addr(at, q), o);
        if (d == 0) peer_store2(peer_addr(at_ml, q), M, L);
      }
    }
  }
  // ---- the CTAs' partials ------------------------------------------------------------------------------
  if (cl > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (int i = tid; i < gcount * (D / 4); i += kStepThreads) {
      const int h = i / (D / 4), d = 4 * (i - h * (D / 4));
      float M = -CUDART_INF_F, L = 0.f;
#pragma unroll
      for (int q = 0; q < kStepMaxCluster; ++q) M = q < cl ? fmaxf(M, s_ml[q][h].x) : M;
      const float m_use = M == -CUDART_INF_F ? 0.f : M;
      float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int q = 0; q < cl; ++q) {
        const float2 ml = s_ml[q][h];
        const float e = ex2_approx(ml.x - m_use);
        const float4 x = *reinterpret_cast<const float4*>(s_all + (q * GC + h) * D + d);
        L = fmaf(ml.y, e, L);
        o.x = fmaf(x.x, e, o.x); o.y = fmaf(x.y, e, o.y); o.z = fmaf(x.z, e, o.z); o.w = fmaf(x.w, e, o.w);
      }
      const float inv = L > 0.f ? 1.f / L : 0.f;
      *reinterpret_cast<float4*>(s_x + h * D + d) = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
      if (d == 0 && rank == 0 && a.lse_out)
        a.lse_out[((int64_t)r + sh.row_offset) * sh.Hq + qh0 + h] = L > 0.f ? (M + log2f(L)) * 0.6931471805599453f : -CUDART_INF_F;
    }
  }
  __syncthreads();
  // ---- un-rotate: out[c] = sum_j x[j] Pi[j][c], the j range cut over jps parts ------------------------------
  const int64_t out0 = ((int64_t)r + sh.row_offset) * a.out_token_stride + (int64_t)qh0 * a.out_head_stride + c0;
  if (a.out_rotated) {
    for (int i = tid; i < gcount * dc; i += kStepThreads) {
      const int h = i / dc, d = i - h * dc;
      store_from_float(a.out, a.out_dtype, out0 + (int64_t)h * a.out_head_stride + d, s_x[h * D + c0 + d]);
    }
    return;
  }
  float y[GC];
#pragma unroll
  for (int h = 0; h < GC; ++h) y[h] = 0.f;
  if (act)
    for (int j = 0; j < jn; j += PB) {
      if (j > 0) {
#pragma unroll
        for (int i = 0; i < PB; ++i) pr[i] = j + i < jn ? __ldg(pi + (j + i) * D) : 0.f;
      }
#pragma unroll
      for (int i = 0; i < PB; ++i)
        if (j + i < jn)
#pragma unroll
          for (int h = 0; h < GC; ++h)
            if (h < gcount) y[h] = fmaf(s_x[h * D + jp * jn + j + i], pr[i], y[h]);
    }
  float* s_red = s_o;  // [jps][GC][dc]
  if (act)
#pragma unroll
    for (int h = 0; h < GC; ++h) s_red[(jp * GC + h) * dc + cc] = y[h];
  __syncthreads();
  for (int i = tid; i < gcount * dc; i += kStepThreads) {
    const int h = i / dc, d = i - h * dc;
    float t = 0.f;
#pragma unroll 8
    for (int q = 0; q < jps; ++q) t += s_red[(q * GC + h) * dc + d];
    store_from_float(a.out, a.out_dtype, out0 + (int64_t)h * a.out_head_stride + d, t);
  }
}

template <int D, int NB, bool ALIGNED, bool ROT>
int launch_step(const AttnArgs& a, int cl_shift, cudaStream_t st) {
  using S = StepCfg<D, NB>;
  constexpr auto kern = decode_step_kernel<D, NB, ALIGNED, ROT>;
  const int cl = 1 << cl_shift;
  if (!ensure_dynamic_smem<kern>((int)S::smem(kStepMaxCluster, ROT), true)) return TQ4_ERR_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(a.sh.rows * a.sh.Hkv * a.sh.NCH) << cl_shift);
  cfg.blockDim = dim3(kStepThreads);
  cfg.dynamicSmemBytes = S::smem(cl > 1 ? cl : 0, ROT);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = !ROT && pdl_enabled() ? 2 : 1;  // (ROT: the entry point's first kernel, a plain stream-ordered launch)
  if (cudaLaunchKernelEx(&cfg, kern, a, cl_shift) != cudaSuccess) return TQ4_ERR_CUDA;
  TQ4_CHECK_LAUNCH();
  return TQ4_OK;
}

template <int D, int NB>
int launch_step_n(const AttnArgs& a, int cl_shift, bool rotate, cudaStream_t st) {
  const bool aligned = cache_aligned(a.sh, a.cache, a.cache_block_stride, a.cache_token_stride);
  if constexpr (D * NB <= 128)
    if (rotate) return aligned ? launch_step<D, NB, true, true>(a, cl_shift, st) : launch_step<D, NB, false, true>(a, cl_shift, st);
  return aligned ? launch_step<D, NB, true, false>(a, cl_shift, st) : launch_step<D, NB, false, false>(a, cl_shift, st);
}
template <int D>
int launch_step_d(const AttnArgs& a, int cl_shift, bool rotate, cudaStream_t st) {
  return a.sh.GC <= 4 ? launch_step_n<D, 1>(a, cl_shift, rotate, st) : launch_step_n<D, 2>(a, cl_shift, rotate, st);
}

}  // namespace

// CTAs that share a (row, KV head), as a power of two; -1: the streaming kernel's call.  As many as leave every cluster at home at
// once (two CTAs fit an SM, one where they take 255 registers; a GPC's SMs are cut into clusters with a remainder), and no more
// keys than the streaming kernel needs its fixed time for: 32 / 8 heads of 128, streaming / here: 1 x 8000 24.1 / 16.6, 1 x 16 000
// 30.8 / 24.9; 2 x 4000 22.5 / 16.8, 2 x 8000 26.0 / 24.5; 4 x 2000 23.9 / 18.3, 4 x 4000 24.6 / 24.6; 8 x 2000 24.7 / 20.5, 8 x 4000
// 29.0 / 33.4; 16 x 1000 28.7 / 22.6, 16 x 2000 31.0 / 36.8 us.  (The lengths are on the device: the longest counts.)
int decode_step_cluster(const AttnArgs& a) {
  if (a.block_size % kTileTokens != 0 || (int64_t)a.sh.rows * a.sh.Hq > tiny_queries(a.sh.D)) return -1;
  const int64_t units = (int64_t)a.sh.rows * a.sh.Hkv * a.sh.NCH;
  const int64_t keys = a.sliding_window > 0 && a.sliding_window < a.max_keys ? a.sliding_window : a.max_keys;
  const bool two = a.sh.D * (a.sh.GC <= 4 ? 1 : 2) <= 128;
  if (units <= 8 && keys <= 8192) return 3;
  if (units <= (two ? 16 : 15) && keys <= 5120) return 3;
  if (units <= (two ? 71 : 33) && keys <= 2560) return 2;
  if (units <= (two ? 148 : 74) && keys <= 1024) return 1;
  return -1;
}

// Where the registers allow two CTAs an SM, the kernel rotates the queries of a call without a write itself, one launch instead of
// two: 1 x 700 keys of 32 / 8 heads of 128 10.3 us either way on the GPU and 2.5 us less of the host's time, 16 x 500 18.5 / 17.0; at
// 28 / 4 heads it would take 14.4 instead of 11.9, at head_dim 256 17.4 instead of 14.5 us.
bool decode_step_rotates(const AttnArgs& a) { return a.sh.D * (a.sh.GC <= 4 ? 1 : 2) <= 128; }

int launch_decode_step(const AttnArgs& a, int cl_shift, bool rotate, cudaStream_t st) {
  switch (a.sh.D) {
    case 64: return launch_step_d<64>(a, cl_shift, rotate, st);
    case 96: return launch_step_d<96>(a, cl_shift, rotate, st);
    case 128: return launch_step_d<128>(a, cl_shift, rotate, st);
    case 256: return launch_step_d<256>(a, cl_shift, rotate, st);
  }
  return TQ4_ERR_UNSUPPORTED;
}

}  // namespace tq4
