// Paged TQ4 attention: planning + query rotation, the fp32 CUDA-core streaming kernel,
// the split merge + un-rotation kernel, and the C entry points.
#include <math_constants.h>

#include <algorithm>
#include <cstdlib>

#include "tq4_attention.cuh"

namespace tq4 {

// ======================================================================================
// 1. Prologue: q_rot = q * Pi^T for every (row, head), and (last block) the tile plan.
// ======================================================================================
// One block.  Phase 1 (inputs only, results in shared memory): per row the visible key range and
// its tile count, an exclusive scan of the tiles, the tiles per CTA, the partial slots per row and
// their scan.  Phase 2, after the preceding kernel has completed: the stores into the plan arrays.
// s_work: 2 * rows ints of dynamic shared memory.
__device__ void build_plan(const AttnArgs& a, int* s_work) {
  const AttnShape& sh = a.sh;
  const AttnPlan& p = a.plan;
  __shared__ int s_part[32];
  __shared__ int s_total;
  __shared__ int s_max_tiles;  // tiles of the longest row
  __shared__ int s_active;     // rows up to the last one that is streamed
  if (threadIdx.x == 0) s_max_tiles = s_active = 0;
  __syncthreads();
  const int rows = sh.rows;
  int* s_tiles = s_work;        // [rows] tile count, then exclusive prefix
  int* s_slots = s_work + rows; // [rows] slot count, then exclusive prefix
  const int per = (rows + blockDim.x - 1) / blockDim.x;
  const int r_lo = min(rows, (int)threadIdx.x * per), r_hi = min(rows, r_lo + per);

  auto row_range = [&](int r, int& seq, int& start, int& end) {
    const int gr = r + sh.row_offset;
    start = 0;
    end = 0;
    if (a.query_start_loc == nullptr) {
      seq = gr;
      if (seq < sh.num_seqs) {
        const int len = clamp_seq_len(a, max(0, a.seq_lens[seq]));
        end = len;
        start = a.sliding_window > 0 ? max(0, len - a.sliding_window) : 0;
      } else {
        seq = 0;
      }
    } else {
      // largest i with qsl[i] <= gr
      int lo = 0, hi = sh.num_seqs;  // qsl has num_seqs + 1 entries
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (a.query_start_loc[mid] <= gr) lo = mid; else hi = mid - 1;
      }
      seq = lo;
      if (seq < sh.num_seqs && gr < a.query_start_loc[sh.num_seqs]) {
        const int q0 = a.query_start_loc[seq], q1 = a.query_start_loc[seq + 1];
        if (a.skip_long > 0 && q1 - q0 >= a.skip_long) {  // (an empty range that no key can have: not merged either)
          end = -1;
          return;
        }
        const int len = clamp_seq_len(a, max(0, a.seq_lens[seq]));
        const int pos = len - (q1 - q0) + (gr - q0);
        end = a.causal ? pos + 1 : len;
        end = max(0, min(end, len));
        start = a.sliding_window > 0 ? max(0, pos + 1 - a.sliding_window) : 0;
        start = min(start, end);
      } else {
        seq = 0;
      }
    }
  };
  // exclusive scan over the block's threads (shuffle scan per warp + scan of the warp totals);
  // s_total receives the sum
  auto block_exclusive_scan = [&](int mine) -> int {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane == 31) s_part[wid] = incl;
    __syncthreads();
    if (wid == 0) {
      const int tot = lane < nw ? s_part[lane] : 0;
      int winc = tot;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, winc, o);
        if (lane >= o) winc += up;
      }
      if (lane < nw) s_part[lane] = winc - tot;  // exclusive warp offsets
      if (lane == 31) s_total = winc;
    }
    __syncthreads();
    const int base = s_part[wid] + incl - mine;
    __syncthreads();
    return base;
  };

  int local = 0, row_max = 0;
  for (int r = r_lo; r < r_hi; ++r) {
    int seq, start, end;
    row_range(r, seq, start, end);
    const int nt = end > start ? (end + kTileTokens - 1) / kTileTokens - start / kTileTokens : 0;
    if (end >= 0) atomicMax(&s_active, r + 1);
    s_tiles[r] = nt;
    local += nt;
    row_max = max(row_max, nt);
  }
  if (row_max > 0) atomicMax(&s_max_tiles, row_max);
  int run = block_exclusive_scan(local);
  for (int r = r_lo; r < r_hi; ++r) {
    const int nt = s_tiles[r];
    s_tiles[r] = run;
    run += nt;
  }
  const int total = s_total;
  const int tps = tiles_per_span(total, sh.span_ctas, s_max_tiles);
  __syncthreads();
  local = 0;
  for (int r = r_lo; r < r_hi; ++r) {
    const int b = s_tiles[r];
    const int e = r + 1 < rows ? s_tiles[r + 1] : total;
    const int n = e > b ? (e - 1) / tps - b / tps + 1 : 0;
    s_slots[r] = n;
    local += n;
  }
  __syncthreads();
  run = block_exclusive_scan(local);
  const int total_slots = s_total;

  for (int r = r_lo; r < r_hi; ++r) {
    int seq, start, end;
    row_range(r, seq, start, end);
    p.kv_start[r] = start;
    p.kv_end[r] = end;
    p.row_seq[r] = seq;
    p.tile_prefix[r] = s_tiles[r];
    p.slot_base[r] = run;
    if (a.plan_records) {
      int4* rec = reinterpret_cast<int4*>(p.row_rec + 8 * (int64_t)r);
      rec[0] = make_int4(s_tiles[r], r + 1 < rows ? s_tiles[r + 1] : total, start, end);
      rec[1] = make_int4(seq, run, 0, 0);
    }
    const int n = s_slots[r];
    s_slots[r] = run;
    run += n;
  }
  if (threadIdx.x == 0) {
    p.tile_prefix[rows] = total;
    p.scalars[0] = total;
    p.scalars[1] = tps;
    p.scalars[2] = s_active;
    p.slot_base[rows] = total_slots;
  }
  __syncthreads();
  for (int s = threadIdx.x; s < sh.span_ctas; s += blockDim.x) {
    const long long T = (long long)s * tps;
    int r = -1;
    if (T < total) {
      int lo = 0, hi = rows - 1;  // the largest r with s_tiles[r] <= T is the row that holds tile T
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_tiles[mid] <= T) lo = mid; else hi = mid - 1;
      }
      r = lo;
    }
    p.span_row[s] = r;
    if (a.plan_records) {
      int4* rec = reinterpret_cast<int4*>(p.span_rec + 12 * (int64_t)s);
      int4 x = make_int4(r, total, tps, 0), y = make_int4(0, 0, 0, 0), z = make_int4(0, 0, 0, 0);
      if (r >= 0) {
        int seq, start, end;
        row_range(r, seq, start, end);
        y = make_int4(s_tiles[r], r + 1 < rows ? s_tiles[r + 1] : total, start, end);
        z.x = seq;
        z.y = s_slots[r];
      }
      rec[0] = x;
      rec[1] = y;
      rec[2] = z;
    }
  }
}

// --------------------------------------------------------------------------------------
// Prologue: ONE launch rotates every query vector of the call and, when the call carries a few new
// tokens, compresses their K and V vectors into the paged cache; block 0 builds the tile plan.  A
// block owns JC output coordinates: its slice of Pi^T sits in shared memory ([d][j]), one WARP takes
// four vectors at a time, and a lane owns NJ consecutive outputs of each, so a step of the reduction
// is one broadcast load of the four vectors' elements and one load of NJ entries of Pi for 4 NJ FMAs.
//
// Latency bound: a decode step waits for this kernel, which is a chain of load Pi, load vectors,
// reduce, store.  While the vectors do not fill the GPU a block therefore takes 32 of the coordinates
// (head_dim 128: 16 KB of Pi to fetch and transpose instead of 64, four times the blocks; kernel time at
// batch 1 11.5 -> 7.8 us, at batch 16 13.4 -> 8.6 us); with many vectors it takes all of them (fewer
// shared-memory reads per FMA).
//
// The write part keeps the arithmetic contract of the compress kernels bit for bit
// (tq4_compress.cu): squared norm by lane-strided FMAs + butterfly reduction, IEEE division by
// (norm + 1e-10), four quarter-length FMA chains in ascending k combined as (s0 + s1) + (s2 + s3).
// --------------------------------------------------------------------------------------
template <int D, int JC>
struct PrologueCfg {
  static constexpr int WARPS = 8;
  static constexpr int THREADS = WARPS * 32;
  static constexpr int VC = 4;                          // vectors per warp per pass
  static constexpr int NJ = JC == 96 ? 4 : JC / 32;     // outputs per lane (JC = 96: lanes 24 .. 31 idle)
  static constexpr int NSPLIT = D / JC;
  static constexpr size_t rot_bytes = ((size_t)D * JC + (size_t)WARPS * D * VC) * sizeof(float);
};

template <int D, int JC>
__global__ void __launch_bounds__(256)
prologue_kernel(const AttnArgs a, const CompressArgs w, const int has_attn, const int has_write) {
  using P = PrologueCfg<D, JC>;
  constexpr int VC = P::VC, NJ = P::NJ, HALF = D / 2, KQ = D / 4, XPL = D / 32;
  static_assert(D % 32 == 0 && KQ % 8 == 0 && D % JC == 0, "head_dim and column block must be multiples of 32");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_trigger();
  if (has_attn && blockIdx.x == 0) {  // the planning block
    build_plan(a, reinterpret_cast<int*>(smem_raw));
    return;
  }
  const int bid = (int)blockIdx.x - (has_attn ? 1 : 0), n_blocks = ((int)gridDim.x - (has_attn ? 1 : 0)) / P::NSPLIT;
  const int j0 = (bid % P::NSPLIT) * JC;
  float* s_pit = reinterpret_cast<float*>(smem_raw);                    // [D][JC]: s_pit[d][j] = Pi[j0 + j][d]
  float4* s_x = reinterpret_cast<float4*>(s_pit + D * JC);              // [WARPS][D] four vectors per entry
  __shared__ float s_bounds[2][16];  // sorted boundaries of K and V, padded with +inf
  __shared__ int s_active;           // rows up to the last one that is streamed (mixed calls)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (has_write && tid < 32) {
    const int src = tid >> 4, i = tid & 15;
    s_bounds[src][i] = (src < w.n_sources && i < w.n_bounds[src]) ? w.bounds[src][i] : CUDART_INF_F;
  }
  if (has_attn && a.skip_long > 0) {
    if (tid == 0) s_active = 0;
    __syncthreads();
    int last = 0;
    for (int s = tid; s < a.sh.num_seqs; s += P::THREADS) {
      const int q0 = a.query_start_loc[s], q1 = a.query_start_loc[s + 1];
      if (q1 > q0 && q1 - q0 < a.skip_long) last = max(last, q1 - a.sh.row_offset);
    }
    if (last > 0) atomicMax(&s_active, min(last, a.sh.rows));
  }

  if (has_attn && a.skip_long > 0) __syncthreads();  // (s_active)
  // vector counts fit 32 bits (rows <= kMaxRowsPerLaunch, writes <= kSmallRows): no 64-bit divisions
  const int n_q = has_attn ? (a.skip_long > 0 ? s_active : a.sh.rows) * a.sh.Hq : 0;
  const int rows_per_src = has_write ? (int)w.n_tokens * w.num_heads : 0;
  const int n_w = rows_per_src * (has_write ? w.n_sources : 0);
  const int cq = (n_q + VC - 1) / VC, cw = (n_w + VC - 1) / VC;
  float4* gx = s_x + warp * D;
  const bool jact = NJ * lane < JC;                     // this lane owns outputs j0 + NJ * lane .. + NJ - 1
  const float* pcol = s_pit + (jact ? NJ * lane : 0);   // + d * JC
  // (source, token, head) of write vector `vec`
  auto w_coords = [&](int vec, int& src, int& tok, int& h) {
    src = vec >= rows_per_src ? 1 : 0;
    const unsigned rem = (unsigned)(vec - src * rows_per_src);
    tok = (int)(rem / (unsigned)w.num_heads);
    h = (int)(rem - (unsigned)tok * (unsigned)w.num_heads);
  };

  // The four vectors of a chunk (lane l: elements l, l + 32, ... of each) and the slots of written ones: fetched before Pi
  // is staged, the next chunk's while this one is multiplied.
  float xr[XPL][VC];
  int64_t slots[VC];
  auto load_chunk = [&](int c) {
    if (c >= cq + cw) return;
    const bool is_w = c >= cq;
    const int v0 = (is_w ? c - cq : c) * VC;
    const int nv = is_w ? n_w : n_q;
    const int dt = is_w ? w.x_dtype : a.q_dtype;
    const void* base[VC];
#pragma unroll
    for (int v = 0; v < VC; ++v) {
      const int vec = v0 + v;
      base[v] = nullptr;
      if (vec < nv) {
        if (!is_w) {
          const unsigned rr = (unsigned)vec / (unsigned)a.sh.Hq;
          const int h = (int)((unsigned)vec - rr * (unsigned)a.sh.Hq);
          base[v] = byte_offset(a.q, dt, ((int64_t)rr + a.sh.row_offset) * a.q_token_stride +
                                             h * a.q_head_stride + lane);
        } else {
          int src, tok, h;
          w_coords(vec, src, tok, h);
          if (w.cache != nullptr) slots[v] = tok < w.n_slots ? write_slot(w, tok) : -1;
          base[v] = byte_offset(w.x[src], dt, token_offset(w, src, tok) + (int64_t)h * w.head_stride[src] + lane);
        }
      }
    }
    if (dt == TQ4_F32) load_strip<float, XPL, VC>(base, xr);
    else if (dt == TQ4_F16) load_strip<__half, XPL, VC>(base, xr);
    else load_strip<__nv_bfloat16, XPL, VC>(base, xr);
  };
  const int first = (bid / P::NSPLIT) * P::WARPS + warp, step = n_blocks * P::WARPS;
  load_chunk(first);

  // ---- stage the slice of Pi^T --------------------------------------------------------------------
  if (has_attn) {
    // thread -> (4 consecutive d of row j), consecutive threads = consecutive j: conflict-free stores
    constexpr int N4 = D * JC / 4, NB = N4 / P::THREADS < 8 ? (N4 + P::THREADS - 1) / P::THREADS : 8;
    for (int i0 = 0; i0 < N4; i0 += P::THREADS * NB) {
      float4 x[NB];
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        const int i = i0 + u * P::THREADS + tid;
        const int c4 = i / JC, jj = i - c4 * JC;
        if (i < N4) x[u] = __ldg(reinterpret_cast<const float4*>(a.rotation + (size_t)(j0 + jj) * D) + c4);
      }
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        const int i = i0 + u * P::THREADS + tid;
        const int c4 = i / JC, jj = i - c4 * JC;
        if (i < N4) {
          float* dst = s_pit + (4 * c4) * JC + jj;
          dst[0] = x[u].x; dst[JC] = x[u].y; dst[2 * JC] = x[u].z; dst[3 * JC] = x[u].w;
        }
      }
    }
  } else {  // write only: the caller gave Pi^T split into even / odd output columns
    constexpr int N = D * JC / 8;  // (row k, four column pairs)
#pragma unroll 4
    for (int i = tid; i < N; i += P::THREADS) {
      const int k = i / (JC / 8), q = i - k * (JC / 8);
      const float4 e = __ldg(reinterpret_cast<const float4*>(w.rot_even + k * HALF + j0 / 2) + q);
      const float4 o = __ldg(reinterpret_cast<const float4*>(w.rot_odd + k * HALF + j0 / 2) + q);
      float4* dst = reinterpret_cast<float4*>(s_pit + k * JC + 8 * q);
      dst[0] = make_float4(e.x, o.x, e.y, o.y);
      dst[1] = make_float4(e.z, o.z, e.w, o.w);
    }
  }
  __syncthreads();

  for (int c = first; c < cq + cw; c += step) {
    const bool is_w = c >= cq;
    const int v0 = (is_w ? c - cq : c) * VC;
    const int nv = is_w ? n_w : n_q;
    float nrm[VC];
    if (is_w) {
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
    }
    __syncwarp();  // the previous pass has finished reading the staging strip
#pragma unroll
    for (int i = 0; i < XPL; ++i) gx[lane + 32 * i] = make_float4(xr[i][0], xr[i][1], xr[i][2], xr[i][3]);
    __syncwarp();
    int64_t slot_of[VC];
#pragma unroll
    for (int v = 0; v < VC; ++v) slot_of[v] = slots[v];
    load_chunk(c + step);

    // ---- y[v][jj] = sum_d x[v][d] * Pi[j0 + NJ*lane + jj][d] as (s0 + s1) + (s2 + s3): the two
    // quarter chains of a half advance together (8 NJ independent accumulators); loops stay rolled,
    // a launch of a few thousand vectors runs this code once per warp and pays for its size
    float y[VC][NJ];
#pragma unroll 1
    for (int hf = 0; hf < 2; ++hf) {
      float sa[VC][NJ], sb[VC][NJ];
#pragma unroll
      for (int v = 0; v < VC; ++v)
#pragma unroll
        for (int jj = 0; jj < NJ; ++jj) sa[v][jj] = sb[v][jj] = 0.f;
      const float* pa = pcol + (2 * hf) * KQ * JC;
      const float4* xa = gx + (2 * hf) * KQ;
#pragma unroll 4
      for (int dd = 0; dd < KQ; ++dd) {
        float ps0[NJ], ps1[NJ];
        load_n<NJ>(pa + dd * JC, ps0);
        load_n<NJ>(pa + (KQ + dd) * JC, ps1);
        const float4 x0 = xa[dd], x1 = xa[KQ + dd];
        const float xs0[VC] = {x0.x, x0.y, x0.z, x0.w};
        const float xs1[VC] = {x1.x, x1.y, x1.z, x1.w};
#pragma unroll
        for (int v = 0; v < VC; ++v)
#pragma unroll
          for (int jj = 0; jj < NJ; ++jj) {
            sa[v][jj] = fmaf(xs0[v], ps0[jj], sa[v][jj]);
            sb[v][jj] = fmaf(xs1[v], ps1[jj], sb[v][jj]);
          }
      }
#pragma unroll
      for (int v = 0; v < VC; ++v)
#pragma unroll
        for (int jj = 0; jj < NJ; ++jj)
          y[v][jj] = hf == 0 ? sa[v][jj] + sb[v][jj] : y[v][jj] + (sa[v][jj] + sb[v][jj]);
    }

    if (!is_w) {
#pragma unroll
      for (int v = 0; v < VC; ++v)
        if (v0 + v < nv && jact) store_n<NJ>(a.plan.q_rot + (int64_t)(v0 + v) * D + j0 + NJ * lane, y[v]);
    } else {
      const RowLayout lay = row_layout(w.num_heads, D);
#pragma unroll
      for (int v = 0; v < VC; ++v) {
        const int vec = v0 + v;
        if (vec >= nv) continue;
        int src, tok, h;
        w_coords(vec, src, tok, h);
        const float* bd = s_bounds[src];
        // eight outputs make a word: the lanes that share it OR their nibbles together
        uint32_t word = 0;
#pragma unroll
        for (int jj = 0; jj < NJ; ++jj) {
          const int p = (NJ * lane + jj) & 7;
          word |= (uint32_t)bucketize_sorted16(y[v][jj], bd) << (8 * (p >> 1) + ((p & 1) ? 0 : 4));
        }
#pragma unroll
        for (int o = 1; o < 8 / NJ; o <<= 1) word |= __shfl_xor_sync(0xffffffffu, word, o);
        uint8_t* dst_idx;
        float* dst_norm;
        if (w.cache != nullptr) {
          const int64_t slot = slot_of[v];
          if (slot < 0) continue;
          if (slot >= w.num_cache_slots) {
            if (lane == 0 && w.err_flag) atomicOr(w.err_flag, TQ4_DEV_BAD_SLOT);
            continue;
          }
          uint8_t* rowp = w.cache + slot * w.cache_token_stride;
          dst_idx = rowp + (src == 0 ? lay.k_idx : lay.v_idx) + h * HALF;
          dst_norm = reinterpret_cast<float*>(rowp + (src == 0 ? lay.k_norm : lay.v_norm) + h * 4);
        } else {
          dst_idx = w.packed_out + (int64_t)vec * HALF;
          dst_norm = w.norms_out + vec;
        }
        const int jo = j0 + NJ * lane;  // (rows start on 4 bytes)
        if (jact && (jo & 7) == 0) *reinterpret_cast<uint32_t*>(dst_idx + jo / 2) = word;
        if (lane == 0 && j0 == 0) *dst_norm = nrm[v];
      }
    }
  }
}

// The same for a step of a few vectors: a block per vector, with all of its Pi (or half, at head_dim 256) asked for before
// anything is known of the vector, so that a load's latency is paid once.
//   A query: lanes along the rows of Pi, so a warp's load is a row (or two), a warp has D / WARPS rows, and their 32 partial sums each are
//     folded over the lanes together.  No staging, no block barrier.
//   A new token's vector: the arithmetic contract of the compress kernels (four quarter chains in ascending k), Pi^T from the
//     caller's even / odd halves, a lane per column pair, warps = quarters x 32 pairs.
// FRAG: for the kernel of small decode steps (tq4_decode_step.cu), which wants a query as fp16 hi and lo terms of y times a power of
// two that follows from the raw vector's largest element.
template <int D>
struct TinyStepCfg {
  static constexpr int HALF = D / 2, CS = (HALF + 31) / 32, WARPS = 4 * CS, THREADS = 32 * WARPS;
  static constexpr int RPL = D == 64 ? 2 : 1;             // rows of Pi a warp's load covers
  static constexpr int F4 = D == 256 ? 2 : 1;             // float4 a lane has of a row
  static constexpr int NV = D / WARPS / RPL;              // rows (row pairs) of a warp
  static constexpr int KQ = D / 4, KB = D == 256 ? 32 : KQ;
};
template <int D, bool WRITE, bool FRAG>
__global__ void __launch_bounds__(TinyStepCfg<D>::THREADS) tiny_prologue_kernel(const AttnArgs a, const CompressArgs w) {
  using C = TinyStepCfg<D>;
  constexpr int HALF = C::HALF, XPL = D / 32, KQ = C::KQ, KB = C::KB, NV = C::NV, F4 = C::F4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float s_x[D];
  __shared__ __align__(16) float s_part[4][D];
  __shared__ float s_b[16];
  pdl_trigger();
  if (!FRAG && blockIdx.x == 0) {  // the planning block
    build_plan(a, reinterpret_cast<int*>(smem_raw));
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n_q = a.sh.rows * a.sh.Hq, vec = (int)blockIdx.x - (FRAG ? 0 : 1);
  if (!WRITE || vec < n_q) {
    // ---- a query ----------------------------------------------------------------------------------------
    constexpr int GL = 32 / C::RPL;                         // lanes of a row
    const int l4 = lane % GL, first = warp * (D / C::WARPS) + lane / GL;
    const bool act = l4 < D / 4 / F4;                       // (head_dim 96: 24 lanes)
    float4 pi[NV][F4];
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
      for (int f = 0; f < F4; ++f)
        pi[i][f] = act ? __ldg(reinterpret_cast<const float4*>(a.rotation + (size_t)(first + C::RPL * i) * D) + l4 + GL * f)
                       : make_float4(0.f, 0.f, 0.f, 0.f);
    const int row = vec / a.sh.Hq;
    const int64_t at = ((int64_t)row + a.sh.row_offset) * a.q_token_stride + (int64_t)(vec - row * a.sh.Hq) * a.q_head_stride;
    uint4 raw[F4];
#pragma unroll
    for (int f = 0; f < F4; ++f) raw[f] = act ? load4_raw(a.q, a.q_dtype, at + 4 * (l4 + GL * f)) : make_uint4(0u, 0u, 0u, 0u);
    float v[NV], top = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = 0.f;
#pragma unroll
    for (int f = 0; f < F4; ++f) {
      const float4 x = raw_as_float4(raw[f], a.q_dtype);
      top = fmaxf(top, fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))));
#pragma unroll
      for (int i = 0; i < NV; ++i)
        v[i] = fmaf(x.x, pi[i][f].x, fmaf(x.y, pi[i][f].y, fmaf(x.z, pi[i][f].z, fmaf(x.w, pi[i][f].w, v[i]))));
    }
    // fold: after the step of `o` lanes a lane has the sums of half as many rows
    int n = 0;  // row of the warp that the lane ends up with (of NV, padded to a power of two)
    constexpr int NP = NV <= 8 ? 8 : 16;
    float t[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) t[i] = i < NV ? v[i] : 0.f;
    int o = GL / 2;
#pragma unroll
    for (int h = NP / 2; h > 0; h >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < h; ++i) {
        const float mine = up ? t[i + h] : t[i], other = up ? t[i] : t[i + h];
        t[i] = mine + __shfl_xor_sync(0xffffffffu, other, o);
      }
      n += up ? h : 0;
      o >>= 1;
    }
    float y = t[0];
#pragma unroll
    for (; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    const bool mine = n < NV && (l4 & (GL / NP - 1)) == 0;  // (the lanes that are left hold the same sum)
    const int j = first + C::RPL * n;
    if constexpr (!FRAG) {
      if (mine) a.plan.q_rot[(int64_t)vec * D + j] = y;
    } else {
#pragma unroll
      for (int s = GL / 2; s > 0; s >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, s));
      const int e = top > 0.f && top < CUDART_INF_F ? min(max((int)(__float_as_uint(top) >> 23) - 127, -100), 100) : 0;
      const float z = y * __uint_as_float((uint32_t)(127 + 4 - e) << 23);  // (at most 2^5 sqrt(D))
      const __half hi = __float2half_rn(z);
      __half* dst = reinterpret_cast<__half*>(a.plan.q_rot + (int64_t)vec * D);
      if (mine) {
        dst[j] = hi;
        dst[D + j] = __float2half_rn(z - __half2float(hi));
      }
      if (threadIdx.x == 0) a.plan.part_l[vec] = __uint_as_float((uint32_t)(127 - 4 + e) << 23);
    }
    return;
  }
  // ---- a vector of a new token --------------------------------------------------------------------------
  const int rows_per_src = (int)w.n_tokens * w.num_heads, r = vec - n_q;
  const int src = r >= rows_per_src ? 1 : 0;
  const unsigned rem = (unsigned)(r - src * rows_per_src);
  const int tok = (int)(rem / (unsigned)w.num_heads), h = (int)(rem - (unsigned)tok * (unsigned)w.num_heads);
  const int q = warp & 3, p = 32 * (warp >> 2) + lane, k0 = q * KQ;
  float pe[KB], po[KB];
  auto load_batch = [&](int kb) {
#pragma unroll
    for (int u = 0; u < KB; ++u) {
      pe[u] = p < HALF ? __ldg(w.rot_even + (k0 + kb + u) * HALF + p) : 0.f;
      po[u] = p < HALF ? __ldg(w.rot_odd + (k0 + kb + u) * HALF + p) : 0.f;
    }
  };
  load_batch(0);
  const int64_t slot = tok < w.n_slots ? write_slot(w, tok) : -1;
  if (threadIdx.x < 16) s_b[threadIdx.x] = threadIdx.x < w.n_bounds[src] ? w.bounds[src][threadIdx.x] : CUDART_INF_F;
  const int64_t at = token_offset(w, src, tok) + (int64_t)h * w.head_stride[src];
  float xv[XPL], ss = 0.f;
#pragma unroll
  for (int i = 0; i < XPL; ++i) xv[i] = load_as_float(w.x[src], w.x_dtype, at + lane + 32 * i);
#pragma unroll
  for (int i = 0; i < XPL; ++i) ss = fmaf(xv[i], xv[i], ss);
  const float norm = sqrtf(warp_sum(ss)), den = norm + 1e-10f;
  if (warp == 0) {
#pragma unroll
    for (int i = 0; i < XPL; ++i) s_x[lane + 32 * i] = xv[i] / den;
  }
  __syncthreads();
  float ae = 0.f, ao = 0.f;
#pragma unroll
  for (int kb = 0; kb < KQ; kb += KB) {
    if (kb > 0) load_batch(kb);
#pragma unroll
    for (int u = 0; u < KB; ++u) {
      const float xk = s_x[k0 + kb + u];
      ae = fmaf(xk, pe[u], ae);
      ao = fmaf(xk, po[u], ao);
    }
  }
  if (p < HALF) *reinterpret_cast<float2*>(&s_part[q][2 * p]) = make_float2(ae, ao);
  __syncthreads();
  if (slot < 0) return;
  if (slot >= w.num_cache_slots) {
    if (threadIdx.x == 0 && w.err_flag) atomicOr(w.err_flag, TQ4_DEV_BAD_SLOT);
    return;
  }
  const RowLayout lay = row_layout(w.num_heads, D);
  uint8_t* rowp = w.cache + slot * w.cache_token_stride;
  uint8_t* dst = rowp + (src == 0 ? lay.k_idx : lay.v_idx) + h * HALF;
  if (threadIdx.x < HALF) {
    const int c = threadIdx.x;
    float y[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) y[e] = (s_part[0][2 * c + e] + s_part[1][2 * c + e]) + (s_part[2][2 * c + e] + s_part[3][2 * c + e]);
    dst[c] = (uint8_t)((bucketize_sorted16(y[0], s_b) << 4) | bucketize_sorted16(y[1], s_b));
  }
  if (threadIdx.x == 0) *reinterpret_cast<float*>(rowp + (src == 0 ? lay.k_norm : lay.v_norm) + h * 4) = norm;
}


template <int D, bool WRITE, bool FRAG>
int launch_tiny_prologue(const AttnArgs& a, const CompressArgs& w, int64_t vectors, cudaStream_t st) {
  const size_t smem = FRAG ? 0 : 2 * (size_t)a.sh.rows * sizeof(int);
  // (first kernel of an entry point: plain stream-ordered launch, see launch_prologue_jc)
  if (launch_kernel(tiny_prologue_kernel<D, WRITE, FRAG>, dim3((unsigned)vectors + (FRAG ? 0 : 1)), dim3(TinyStepCfg<D>::THREADS), smem,
                    st, false, a, w) != cudaSuccess)
    return TQ4_ERR_CUDA;
  TQ4_CHECK_LAUNCH();
  return TQ4_OK;
}

template <int D, int JC>
int launch_prologue_jc(const AttnArgs* a, const CompressArgs* w, cudaStream_t st, int64_t blocks) {
  using P = PrologueCfg<D, JC>;
  const size_t plan = a ? 2 * (size_t)a->sh.rows * sizeof(int) : 0;  // planning block
  const size_t smem = P::rot_bytes > plan ? P::rot_bytes : plan;
  if (!ensure_dynamic_smem<prologue_kernel<D, JC>>((int)smem, true)) return TQ4_ERR_CUDA;
  const int64_t most = 2 * (int64_t)sm_count() / P::NSPLIT;
  if (JC != 32 && blocks > most) blocks = most;
  if (blocks < 1) blocks = 1;
  static const AttnArgs no_attn{};
  static const CompressArgs no_write{};
  // First kernel of an entry point: a plain stream-ordered launch.  It reads tensors the caller's
  // preceding kernel may have produced (q, key, value, seq_lens), so it must not start before that
  // kernel has completed, whatever launch style the caller's kernels use.
  if (launch_kernel(prologue_kernel<D, JC>, dim3((unsigned)(blocks * P::NSPLIT) + (a ? 1 : 0)), dim3(P::THREADS), smem,
                    st, false, a ? *a : no_attn, w ? *w : no_write, a ? 1 : 0, w ? 1 : 0) != cudaSuccess)
    return TQ4_ERR_CUDA;
  TQ4_CHECK_LAUNCH();
  return TQ4_OK;
}

// Column blocks of 32 while they all fit the GPU at once (about three resident blocks an SM), of the
// whole head_dim (64 at head_dim 256: Pi does not fit) above.
template <int D>
int launch_prologue_t(const AttnArgs* a, const CompressArgs* w, cudaStream_t st) {
  constexpr int VC = 4, WARPS = 8;
  const int64_t n_q = a ? (int64_t)a->sh.rows * a->sh.Hq : 0;
  const int64_t n_w = w ? w->n_tokens * w->num_heads * w->n_sources : 0;
  const int64_t chunks = (n_q + VC - 1) / VC + (n_w + VC - 1) / VC;
  const int64_t blocks = (chunks + WARPS - 1) / WARPS;
  if (a && a->skip_long == 0 && n_q <= tiny_queries(D)) {
    static const CompressArgs no_write{};
    if (w && n_w > 2 * tiny_queries(D)) {  // (new vectors: more are left to the write kernels)
      const int rc = dispatch_compress(*w, D, w->x_dtype, st);
      if (rc != TQ4_OK) return rc;
      w = nullptr;
    }
    const int64_t n = n_q + (w ? n_w : 0);
    if (a->no_plan) return w ? launch_tiny_prologue<D, true, true>(*a, *w, n, st) : launch_tiny_prologue<D, false, true>(*a, no_write, n, st);
    return w ? launch_tiny_prologue<D, true, false>(*a, *w, n, st) : launch_tiny_prologue<D, false, false>(*a, no_write, n, st);
  }
  const int64_t wave = 3 * (int64_t)sm_count() / (D / 32);
  if (blocks <= wave) return launch_prologue_jc<D, 32>(a, w, st, blocks);
  // a mixed call streams few of its rows (the kernel finds out how many)
  if (a && a->skip_long > 0) return launch_prologue_jc<D, 32>(a, w, st, wave);
  return launch_prologue_jc<D, (D <= 128 ? D : 64)>(a, w, st, blocks);
}

// ======================================================================================
// 2. fp32 CUDA-core streaming kernel (any supported head_dim, any group size).
// ======================================================================================
template <int D, int GC>
struct Fp32Cfg {
  static constexpr int REPS = (D + 127) / 128;  // 4-dim groups per lane in the V phase
  static constexpr int KW = D / 16;             // 32-bit words of K per lane (half a row)
  static constexpr size_t smem_per_warp =
      (size_t)GC * D * 4 + kTileTokens * GC * 4 + kTileTokens * 8;
};

template <int D, int GC>
__global__ void __launch_bounds__(kMaxWarpsPerCta * 32)
attention_fp32_kernel(const AttnArgs a) {
  using Cfg = Fp32Cfg<D, GC>;
  constexpr int REPS = Cfg::REPS, KW = Cfg::KW, HALF = D / 2;
  const AttnShape& sh = a.sh;
  const AttnPlan& p = a.plan;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float lut_k[TQ4_MAX_CENTROIDS], lut_v[TQ4_MAX_CENTROIDS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* wbase = smem_raw + warp * Cfg::smem_per_warp;
  float* s_q = reinterpret_cast<float*>(wbase);                       // [GC][D]
  float* s_p = s_q + GC * D;                                          // [16][GC]  p * vnorm
  int64_t* s_row = reinterpret_cast<int64_t*>(s_p + kTileTokens * GC);  // [16] row byte offset, -1 = masked

  if (threadIdx.x < TQ4_MAX_CENTROIDS) {
    lut_k[threadIdx.x] = threadIdx.x < a.n_k_centroids ? a.k_centroids[threadIdx.x] : 0.f;
    lut_v[threadIdx.x] = threadIdx.x < a.n_v_centroids ? a.v_centroids[threadIdx.x] : 0.f;
  }
  __syncthreads();
  pdl_trigger();
  pdl_wait();  // plan, rotated queries and cache come from the preceding kernels

  const int c = blockIdx.x % sh.ctas, slice = blockIdx.x / sh.ctas;
  const int vh = slice * sh.HPC + warp % sh.HPC, ts = warp / sh.HPC;
  const int kvh = vh / sh.NCH, chunk = vh % sh.NCH;
  const int qh0 = kvh * sh.G + chunk * sh.GC;
  const int gcount = min(sh.GC, sh.G - chunk * sh.GC);
  const int total = p.scalars[0], tps = p.scalars[1];
  const int t_begin = c * tps, t_end = min(total, t_begin + tps);
  if (t_begin >= t_end) return;
  const RowLayout lay = row_layout(sh.Hkv, D);

  int r = p.span_row[c];
  const int tok = lane & 15, half = lane >> 4;

  int t = t_begin;
  while (t < t_end) {
    const int row_t0 = p.tile_prefix[r], row_t1 = p.tile_prefix[r + 1];
    const int seg_end = min(row_t1, t_end);
    const int kv_start = p.kv_start[r], kv_end = p.kv_end[r];
    const int32_t* bt = a.block_table + (int64_t)p.row_seq[r] * a.bt_stride;
    const int tile0 = kv_start / kTileTokens;  // absolute tile index of the row's first tile

    // q of this row's heads -> smem
    __syncwarp();
    for (int i = lane; i < GC * D; i += 32) {
      const int g = i / D, d = i - g * D;
      s_q[i] = g < gcount ? p.q_rot[((int64_t)r * sh.Hq + qh0 + g) * D + d] : 0.f;
    }
    __syncwarp();

    float m[GC], l[GC], acc[GC][REPS][4];
#pragma unroll
    for (int g = 0; g < GC; ++g) {
      m[g] = -CUDART_INF_F;
      l[g] = 0.f;
#pragma unroll
      for (int rep = 0; rep < REPS; ++rep)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[g][rep][e] = 0.f;
    }

    for (int tt = t + ts; tt < seg_end; tt += sh.TPC) {
      const int pos = (tile0 + (tt - row_t0)) * kTileTokens + tok;
      // ---- K phase: lane = (half, token) -------------------------------------------------
      int64_t row_off = -1;
      if (pos >= kv_start && pos < kv_end) {
        const int blk = bt[pos / a.block_size];
        if (blk < 0 || blk >= a.num_blocks) {
          if (a.err_flag) atomicOr(a.err_flag, TQ4_DEV_BAD_BLOCK);
        } else {
          row_off = (int64_t)blk * a.cache_block_stride +
                    (int64_t)(pos % a.block_size) * a.cache_token_stride;
        }
      }
      float dot[GC];
#pragma unroll
      for (int g = 0; g < GC; ++g) dot[g] = 0.f;
      float knorm = 0.f, vnorm = 0.f;
      if (row_off >= 0) {
        const uint8_t* rowp = a.cache + row_off;
        const uint32_t* kw = reinterpret_cast<const uint32_t*>(rowp + lay.k_idx + kvh * HALF + half * (HALF / 2));
        knorm = *reinterpret_cast<const float*>(rowp + lay.k_norm + kvh * 4);
        vnorm = *reinterpret_cast<const float*>(rowp + lay.v_norm + kvh * 4);
        const int dbase = half * HALF;
#pragma unroll
        for (int w = 0; w < KW; ++w) {
          const uint32_t word = kw[w];
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const uint32_t byte = (word >> (8 * b)) & 0xFFu;
            const float ce = lut_k[byte >> 4], co = lut_k[byte & 0xFu];
            const int d = dbase + w * 8 + b * 2;
#pragma unroll
            for (int g = 0; g < GC; ++g) {
              dot[g] = fmaf(s_q[g * D + d], ce, dot[g]);
              dot[g] = fmaf(s_q[g * D + d + 1], co, dot[g]);
            }
          }
        }
      }
      if (half == 0) s_row[tok] = row_off;
      float pw[GC];
#pragma unroll
      for (int g = 0; g < GC; ++g) {
        float s = dot[g] + __shfl_xor_sync(0xffffffffu, dot[g], 16);
        s = row_off >= 0 ? s * knorm * a.scale_log2e : -CUDART_INF_F;
        float mt = s;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, o));
        const float m_new = fmaxf(m[g], mt);
        const float m_use = m_new == -CUDART_INF_F ? 0.f : m_new;
        const float alpha = exp2f(m[g] - m_use);
        const float pr = exp2f(s - m_use);
        m[g] = m_new;
        l[g] = l[g] * alpha + (half == 0 ? pr : 0.f);
        pw[g] = pr * vnorm;
#pragma unroll
        for (int rep = 0; rep < REPS; ++rep)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[g][rep][e] *= alpha;
      }
      if (half == 0) {
#pragma unroll
        for (int g = 0; g < GC; ++g) s_p[tok * GC + g] = pw[g];
      }
      __syncwarp();
      // ---- V phase: lane = 4 consecutive dims per rep -----------------------------------
#pragma unroll 4
      for (int tk = 0; tk < kTileTokens; ++tk) {
        const int64_t ro = s_row[tk];
        if (ro < 0) continue;
        const uint8_t* vrow = a.cache + ro + lay.v_idx + kvh * HALF;
#pragma unroll
        for (int rep = 0; rep < REPS; ++rep) {
          const int byte0 = 2 * (lane + 32 * rep);
          if (byte0 < HALF) {
            const uint32_t hv = *reinterpret_cast<const uint16_t*>(vrow + byte0);
            const float c0 = lut_v[(hv >> 4) & 0xFu], c1 = lut_v[hv & 0xFu];
            const float c2 = lut_v[(hv >> 12) & 0xFu], c3 = lut_v[(hv >> 8) & 0xFu];
#pragma unroll
            for (int g = 0; g < GC; ++g) {
              const float w = s_p[tk * GC + g];
              acc[g][rep][0] = fmaf(w, c0, acc[g][rep][0]);
              acc[g][rep][1] = fmaf(w, c1, acc[g][rep][1]);
              acc[g][rep][2] = fmaf(w, c2, acc[g][rep][2]);
              acc[g][rep][3] = fmaf(w, c3, acc[g][rep][3]);
            }
          }
        }
      }
      __syncwarp();
    }

    // ---- write this warp's partial for the segment ---------------------------------------
    const int slot = p.slot_base[r] + (c - row_t0 / tps);
    const int64_t pidx = (int64_t)slot * sh.TPC + ts;
#pragma unroll
    for (int g = 0; g < GC; ++g) {
      if (g < gcount) {
        const float lsum = warp_sum(l[g]);
        const int64_t hidx = pidx * sh.Hq + qh0 + g;
        if (lane == 0) {
          p.part_m[hidx] = m[g];
          p.part_l[hidx] = lsum;
        }
#pragma unroll
        for (int rep = 0; rep < REPS; ++rep) {
          const int d = 4 * (lane + 32 * rep);
          if (d < D)
            *reinterpret_cast<float4*>(p.part_o + hidx * D + d) =
                make_float4(acc[g][rep][0], acc[g][rep][1], acc[g][rep][2], acc[g][rep][3]);
        }
      }
    }
    t = seg_end;
    if (t < t_end) {
      ++r;
      while (p.tile_prefix[r + 1] <= t) ++r;
    }
  }
}

template <int D, int GC>
int launch_fp32_t(const AttnArgs& a, cudaStream_t st) {
  using Cfg = Fp32Cfg<D, GC>;
  const size_t smem = Cfg::smem_per_warp * kMaxWarpsPerCta;
  if (!ensure_dynamic_smem<attention_fp32_kernel<D, GC>>((int)smem)) return TQ4_ERR_CUDA;
  const int warps = a.sh.HPC * a.sh.TPC;
  if (launch_kernel(attention_fp32_kernel<D, GC>, dim3(a.sh.ctas * a.sh.n_slices), dim3(warps * 32), smem, st,
                    true, a) != cudaSuccess)
    return TQ4_ERR_CUDA;
  TQ4_CHECK_LAUNCH();
  return TQ4_OK;
}

template <int D>
int launch_fp32_d(const AttnArgs& a, cudaStream_t st) {
  const int gc = a.sh.GC;
  if (gc <= 1) return launch_fp32_t<D, 1>(a, st);
  if (gc <= 2) return launch_fp32_t<D, 2>(a, st);
  if (gc <= 4) return launch_fp32_t<D, 4>(a, st);
  return launch_fp32_t<D, 8>(a, st);
}

int launch_attention_fp32(const AttnArgs& a, cudaStream_t st) {
  switch (a.sh.D) {
    case 64: return launch_fp32_d<64>(a, st);
    case 96: return launch_fp32_d<96>(a, st);
    case 128: return launch_fp32_d<128>(a, st);
    case 256: return launch_fp32_d<256>(a, st);
  }
  return TQ4_ERR_UNSUPPORTED;
}

// ======================================================================================
// 3. Merge the partials of a row, normalise, un-rotate, store.
//    Also serves tq4_combine_partials (cross-GPU shards) through the "dense" mode.
// ======================================================================================
struct CombineArgs {
  const int* active_rows;  // (optional) device count: only the first so many rows are merged ...
  const int* row_end;      // (optional) last visible key of the rows: -1 = a row of the prefill kernel
  int rows_long;           // with row_end: merge the prefill kernel's rows (1) or the others (0)
  // sparse mode (slot_base != null): the partials of row r are slot_base[r]..slot_base[r+1], x TPC
  const int* slot_base;
  int TPC;
  const float* part_o;
  const float* part_m;
  const float* part_l;
  // dense mode (slot_base == null): `world` parts, part index w*rows + r; part_m holds natural-log
  // LSE and part_o is already normalised
  int world;
  int rows, row_offset, Hq;
  const float* rotation;
  void* out;
  int out_dtype;
  int64_t out_token_stride, out_head_stride;
  float* lse_out;
  int out_rotated;
};

// Merge kernel: eight warps, VB = 8 / WPV (row, head) vectors per pass.
//   1. WPV warps merge the partials of one vector: warp w takes partials w, w + WPV, ..., a lane holds
//      the maximum and sum of one of them and four (D = 256: eight) of the accumulator's coordinates, so
//      the loads of eight partials are in flight at a time whatever their number.
//   2. out[v][c] = sum_j x[v][j] * Pi[j][c]: a lane owns 4 columns x 4 vectors, the j range is cut over
//      the warps (JP parts) and summed in shared memory.
// Pi is copied to shared memory while the kernel in front is still running.  At head_dim 256 it does
// not fit: a block owns 64 of the columns and the merge is repeated by the four blocks of a vector.
// Bound by latency (a chain of three memory round trips), so the split follows the number of
// vectors: few vectors get all eight warps each, many share a pass.  Measured on whole decode steps
// against a merge with one thread per coordinate and eight vectors per block: batch 1 x 1024 tokens
// (28 vectors of 64 partials) 73.8 -> 29.7 us, 16 ragged rows 74 -> 50.6 us, batch 64 x 4096 97.6 -> 92.7 us.
template <int D, int WPV>
struct CombineCfg {
  static constexpr int VB = 8 / WPV;                  // vectors per pass
  static constexpr int DC = D == 256 ? 64 : D;        // output columns of a block
  static constexpr int NSPLIT = D / DC;
  static constexpr int LC = DC / 4;                   // lanes that cover the columns
  static constexpr int UPW = 32 / LC;                 // units (column sets) per warp: 2 if 16 lanes cover them
  static constexpr int VPT = VB < 4 ? VB : 4;         // vectors per lane
  static constexpr int NVG = VB / VPT;
  static constexpr int JP = 8 * UPW / NVG;            // parts of the j range
  static constexpr int JN = D / JP;
  static constexpr int XP = D + 4;                    // pitch of a merged vector
  static constexpr size_t kOffX = (size_t)D * DC * 4;
  static constexpr size_t kOffRed = kOffX + (size_t)VB * XP * 4;
  static constexpr size_t kRed = (size_t)JP * VB * DC * 4, kParts = (size_t)8 * D * 4;  // (the two uses of the area)
  static constexpr size_t kSmem = kOffRed + (kRed > kParts ? kRed : kParts);
  static_assert(JN % 4 == 0 && JP * JN == D, "a part of the j range is a multiple of four");
};

template <int D, int WPV>
__global__ void __launch_bounds__(256) combine_kernel(const CombineArgs a) {
  using C = CombineCfg<D, WPV>;
  constexpr int VB = C::VB, R = D == 256 ? 2 : 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* s_pi = reinterpret_cast<float*>(smem_raw);                 // [D][DC]
  float* s_x = reinterpret_cast<float*>(smem_raw + C::kOffX);       // [VB][XP] merged, normalised vectors
  float* s_red = reinterpret_cast<float*>(smem_raw + C::kOffRed);   // [8][D] partial merges, then [JP][VB][DC] partial products
  __shared__ float s_m[8], s_l[8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int split = blockIdx.x % C::NSPLIT;
  int n_vec = a.rows * a.Hq;
  if (!a.out_rotated) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_pi);
    for (int i = tid; i < D * C::LC; i += 256) {
      const int j = i / C::LC, c4 = i - j * C::LC;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 16),
                   "l"(a.rotation + (size_t)j * D + split * C::DC + 4 * c4) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  pdl_wait();  // the partials and the plan come from the kernels before this one
  auto row_mine = [&](int row) { return !a.row_end || (a.row_end[row] < 0) == (a.rows_long != 0); };
  if (a.active_rows) n_vec = min(n_vec, *a.active_rows * a.Hq);
  const bool sparse = a.slot_base != nullptr;
  const float mscale = sparse ? 1.f : 1.4426950408889634f;  // dense partials carry a natural-log LSE
  const int64_t pstride = sparse ? (int64_t)a.Hq : (int64_t)a.rows * a.Hq;  // vectors between two partials

  for (int v0 = (int)(blockIdx.x / C::NSPLIT) * VB; v0 < n_vec; v0 += (int)(gridDim.x / C::NSPLIT) * VB) {
    // ---- merge ------------------------------------------------------------------------------------
    {
      const int v = warp / WPV, sub = warp % WPV, vec = v0 + v;
      float M = -CUDART_INF_F, L = 0.f;
      float o[R][4];
#pragma unroll
      for (int r = 0; r < R; ++r) o[r][0] = o[r][1] = o[r][2] = o[r][3] = 0.f;
      if (vec < n_vec) {
        const int row = vec / a.Hq, head = vec - row * a.Hq;
        const int p0 = sparse ? a.slot_base[row] * a.TPC : 0;
        const int np = sparse ? a.slot_base[row + 1] * a.TPC - p0 : a.world;
        const int64_t first = (sparse ? (int64_t)p0 * a.Hq : (int64_t)row * a.Hq) + head + (int64_t)sub * pstride;
        const int nk = np > sub ? (np - sub + WPV - 1) / WPV : 0;  // partials of this warp
        for (int k0 = 0; k0 < nk; k0 += 32) {
          const int kk = min(32, nk - k0);
          float m = -CUDART_INF_F, l = 0.f;
          if (lane < kk) {
            const int64_t idx = first + (int64_t)(k0 + lane) * WPV * pstride;
            m = __ldg(a.part_m + idx) * mscale;
            l = sparse ? __ldg(a.part_l + idx) : 1.f;
          }
          const float M2 = fmaxf(M, warp_max(m));
          const float m_use = M2 == -CUDART_INF_F ? 0.f : M2;
          const float resc = exp2f(M - m_use);   // (0 the first time)
          const float w = exp2f(m - m_use);      // 0 for empty partials
          L = L * resc + warp_sum(w * l);
          M = M2;
#pragma unroll
          for (int r = 0; r < R; ++r)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[r][e] *= resc;
          const float* po = a.part_o + (first + (int64_t)k0 * WPV * pstride) * D + 4 * lane;
          for (int k = 0; k < kk; k += 8) {  // eight partials in flight
            float4 x[8][R];
            float wk[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              wk[u] = __shfl_sync(0xffffffffu, w, (k + u) & 31);
              const bool use = k + u < kk && wk[u] > 0.f;  // (an empty partial's accumulator is never read)
#pragma unroll
              for (int r = 0; r < R; ++r) {
                x[u][r] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (use && 4 * lane + 128 * r < D)
                  x[u][r] = __ldg(reinterpret_cast<const float4*>(po + (int64_t)(k + u) * WPV * pstride * D + 128 * r));
              }
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
              for (int r = 0; r < R; ++r) {
                o[r][0] = fmaf(x[u][r].x, wk[u], o[r][0]);
                o[r][1] = fmaf(x[u][r].y, wk[u], o[r][1]);
                o[r][2] = fmaf(x[u][r].z, wk[u], o[r][2]);
                o[r][3] = fmaf(x[u][r].w, wk[u], o[r][3]);
              }
          }
        }
      }
      if (WPV > 1) {
        if (lane == 0) { s_m[warp] = M; s_l[warp] = L; }
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (4 * lane + 128 * r < D)
            *reinterpret_cast<float4*>(s_red + warp * D + 4 * lane + 128 * r) = make_float4(o[r][0], o[r][1], o[r][2], o[r][3]);
        __syncthreads();
        M = -CUDART_INF_F;
        L = 0.f;
#pragma unroll
        for (int u = 0; u < WPV; ++u) M = fmaxf(M, s_m[v * WPV + u]);
        const float m_use = M == -CUDART_INF_F ? 0.f : M;
        float wu[WPV];
#pragma unroll
        for (int u = 0; u < WPV; ++u) {
          wu[u] = exp2f(s_m[v * WPV + u] - m_use);
          L = fmaf(s_l[v * WPV + u], wu[u], L);
        }
        const float inv = L > 0.f ? 1.f / L : 0.f;
        // the warps of a vector share its coordinates
        for (int d = sub * 32 + lane; d < D; d += 32 * WPV) {
          float x = 0.f;
#pragma unroll
          for (int u = 0; u < WPV; ++u) x = fmaf(s_red[(v * WPV + u) * D + d], wu[u], x);
          s_x[v * C::XP + d] = x * inv;
        }
      } else {
        const float inv = L > 0.f ? 1.f / L : 0.f;
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (4 * lane + 128 * r < D)
            *reinterpret_cast<float4*>(s_x + v * C::XP + 4 * lane + 128 * r) =
                make_float4(o[r][0] * inv, o[r][1] * inv, o[r][2] * inv, o[r][3] * inv);
      }
      if (a.lse_out && split == 0 && sub == 0 && lane == 0 && vec < n_vec && row_mine(vec / a.Hq))
        a.lse_out[(int64_t)a.row_offset * a.Hq + vec] =
            L > 0.f ? (M + log2f(L)) * 0.6931471805599453f : -CUDART_INF_F;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // ---- un-rotate --------------------------------------------------------------------------------
    if (!a.out_rotated) {
      const int unit = warp * C::UPW + lane / C::LC, cl = lane % C::LC;
      const int vg = unit % C::NVG, jp = unit / C::NVG;
      if (jp < C::JP) {  // (D = 96: lanes 24 .. 31 idle)
        float acc[C::VPT][4];
#pragma unroll
        for (int v = 0; v < C::VPT; ++v) acc[v][0] = acc[v][1] = acc[v][2] = acc[v][3] = 0.f;
        const float4* xp = reinterpret_cast<const float4*>(s_x + vg * C::VPT * C::XP + jp * C::JN);
        const float4* pp = reinterpret_cast<const float4*>(s_pi + (size_t)jp * C::JN * C::DC) + cl;
#pragma unroll 2
        for (int j4 = 0; j4 < C::JN / 4; ++j4) {
          float4 x[C::VPT];
#pragma unroll
          for (int v = 0; v < C::VPT; ++v) x[v] = xp[v * (C::XP / 4) + j4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float4 p = pp[(4 * j4 + e) * C::LC];
#pragma unroll
            for (int v = 0; v < C::VPT; ++v) {
              const float xe = e == 0 ? x[v].x : e == 1 ? x[v].y : e == 2 ? x[v].z : x[v].w;
              acc[v][0] = fmaf(xe, p.x, acc[v][0]);
              acc[v][1] = fmaf(xe, p.y, acc[v][1]);
              acc[v][2] = fmaf(xe, p.z, acc[v][2]);
              acc[v][3] = fmaf(xe, p.w, acc[v][3]);
            }
          }
        }
        if (lane < C::UPW * C::LC)
#pragma unroll
          for (int v = 0; v < C::VPT; ++v)
            *reinterpret_cast<float4*>(s_red + ((size_t)jp * VB + vg * C::VPT + v) * C::DC + 4 * cl) =
                make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
      }
      __syncthreads();
    }
    // ---- sum the parts, cast, store ---------------------------------------------------------------
    for (int i = tid; i < VB * C::LC; i += 256) {
      const int v = i / C::LC, c = 4 * (i - v * C::LC), vec = v0 + v;
      if (vec >= n_vec) continue;
      float y[4] = {0.f, 0.f, 0.f, 0.f};
      if (a.out_rotated) {
        const float4 t = *reinterpret_cast<const float4*>(s_x + v * C::XP + split * C::DC + c);
        y[0] = t.x; y[1] = t.y; y[2] = t.z; y[3] = t.w;
      } else {
#pragma unroll
        for (int jp = 0; jp < C::JP; ++jp) {
          const float4 t = *reinterpret_cast<const float4*>(s_red + ((size_t)jp * VB + v) * C::DC + c);
          y[0] += t.x; y[1] += t.y; y[2] += t.z; y[3] += t.w;
        }
      }
      const int row = vec / a.Hq, head = vec - row * a.Hq;
      if (!row_mine(row)) continue;
      store4(a.out, a.out_dtype, (int64_t)(row + a.row_offset) * a.out_token_stride + (int64_t)head * a.out_head_stride +
                                     split * C::DC + c, y);
    }
    __syncthreads();  // s_x and s_red are rewritten by the next pass
  }
}

template <int D, int WPV>
int launch_combine_w(const CombineArgs& c, cudaStream_t st, bool pdl) {
  using C = CombineCfg<D, WPV>;
  // (same shared-memory carve-out as the attention kernel it follows: no reconfiguration between them)
  if (!ensure_dynamic_smem<combine_kernel<D, WPV>>((int)C::kSmem, true)) return TQ4_ERR_CUDA;
  const int64_t passes = ((int64_t)c.rows * c.Hq + C::VB - 1) / C::VB;
  const int64_t most = 2 * (int64_t)sm_count() / C::NSPLIT;
  if (launch_kernel(combine_kernel<D, WPV>, dim3((unsigned)((passes < most ? passes : most) * C::NSPLIT)), dim3(256),
                    C::kSmem, st, pdl, c) != cudaSuccess)
    return TQ4_ERR_CUDA;
  TQ4_CHECK_LAUNCH();
  return TQ4_OK;
}

// Warps per vector: as many as leave every vector a block of its own in one wave of two blocks per SM
// (the partials of a vector are then read in one round trip), fewer when the vectors fill the GPU anyway.
template <int D>
int launch_combine_t(const CombineArgs& c, cudaStream_t st, bool pdl) {
  const int64_t n_vec = (int64_t)c.rows * c.Hq, wave = 2 * (int64_t)sm_count() / (D == 256 ? 4 : 1);
  if (n_vec <= wave) return launch_combine_w<D, 8>(c, st, pdl);
  if (n_vec <= 4 * wave) return launch_combine_w<D, 2>(c, st, pdl);
  return launch_combine_w<D, 1>(c, st, pdl);
}

// pdl: the launch follows another kernel of the same entry point (false for the stand-alone merge,
// whose partials come from the caller's preceding kernel or collective)
int launch_combine(const CombineArgs& c, int D, cudaStream_t st, bool pdl) {
  if (c.rows == 0) return TQ4_OK;
  switch (D) {
    case 64: return launch_combine_t<64>(c, st, pdl);
    case 96: return launch_combine_t<96>(c, st, pdl);
    case 128: return launch_combine_t<128>(c, st, pdl);
    case 256: return launch_combine_t<256>(c, st, pdl);
  }
  return TQ4_ERR_UNSUPPORTED;
}

// Prologue of an attention call (a != nullptr) and / or cache write of a few new tokens
// (w != nullptr) in one launch; large writes use the compress kernels.
int launch_prologue(const AttnArgs* a, const CompressArgs* w, int head_dim, cudaStream_t st) {
  if (w && w->n_tokens * w->num_heads * w->n_sources > kSmallRows) {
    const int rc = dispatch_compress(*w, head_dim, w->x_dtype, st);
    if (rc != TQ4_OK) return rc;
    w = nullptr;
  }
  if (!a && !w) return TQ4_OK;
  switch (head_dim) {
    case 64: return launch_prologue_t<64>(a, w, st);
    case 96: return launch_prologue_t<96>(a, w, st);
    case 128: return launch_prologue_t<128>(a, w, st);
    case 256: return launch_prologue_t<256>(a, w, st);
  }
  return TQ4_ERR_UNSUPPORTED;
}

int launch_small_write(const CompressArgs& w, int head_dim, cudaStream_t st) { return launch_prologue(nullptr, &w, head_dim, st); }

}  // namespace tq4

// ======================================================================================
// C entry points
// ======================================================================================
extern "C" const char* tq4_version(void) { return "tq4-sm100a 0.1"; }

extern "C" const char* tq4_status_string(int status) {
  switch (status) {
    case TQ4_OK: return "ok";
    case TQ4_ERR_INVALID_ARG: return "invalid argument (null/misaligned pointer or bad size)";
    case TQ4_ERR_UNSUPPORTED: return "unsupported head_dim / head grouping / dtype";
    case TQ4_ERR_CUDA: return "CUDA runtime error at launch";
    case TQ4_ERR_WORKSPACE: return "workspace too small";
    case TQ4_ERR_STATIC_SCRATCH:
      return "request needs more scratch than the built-in static area (TQ4_STATIC_SCRATCH_BYTES); "
             "use tq4_paged_attention with a caller-provided workspace";
  }
  return "unknown status";
}

// What a call of up to so many rows cannot do without.
static size_t workspace_min(int64_t max_query_rows, int num_q_heads, int num_kv_heads, int head_dim) {
  tq4::AttnShape sh{};
  if (max_query_rows <= 0 || !tq4::make_shape(sh, num_q_heads, num_kv_heads, head_dim)) return 0;
  const int64_t rows = max_query_rows < tq4::kMaxRowsPerLaunch ? max_query_rows : tq4::kMaxRowsPerLaunch;
  tq4::AttnPlan p;
  const size_t a = tq4::carve_plan(p, nullptr, rows, num_q_heads, head_dim, sh.TPC);
  tq4::make_shape(sh, num_q_heads, num_kv_heads, head_dim, tq4::kMmaWarpsPerCta);
  const size_t b = tq4::carve_plan(p, nullptr, rows, num_q_heads, head_dim, 1, (int64_t)tq4::kMaxSms * sh.TPC);
  return a > b ? a : b;
}

// ... and room for a prefill call that is cut along the keys: Pi's image and the partials of up to eight parts of the rows,
// as long as these do not fill the GPU.  They lie where the streaming part's partials were (attention_impl), behind
// the plan in a call of both kernels; only calls of few heads or rows need more than the plan has anyway.
extern "C" size_t tq4_attention_workspace_bytes(int64_t max_query_rows, int num_q_heads,
                                                int num_kv_heads, int head_dim) {
  const size_t least = workspace_min(max_query_rows, num_q_heads, num_kv_heads, head_dim);
  if (least == 0) return 0;
  if (max_query_rows < tq4::kPrefillMinRows) return least;
  int64_t vectors = 8 * max_query_rows * num_q_heads;
  if (vectors > tq4::kPrefillSplitVectors) vectors = tq4::kPrefillSplitVectors;
  const int64_t rows = max_query_rows < tq4::kMaxRowsPerLaunch ? max_query_rows : tq4::kMaxRowsPerLaunch;
  tq4::AttnPlan p;
  size_t front = 0;  // (for whichever kernel has more spans)
  constexpr int64_t spans = std::max(tq4::kMaxCtasPerSlice, tq4::kMaxSms * tq4::kMmaWarpsPerCta);
  tq4::carve_plan(p, nullptr, rows, num_q_heads, head_dim, 1, spans, &front);
  // (a vector set of Hq and the alignment of the image on top: prefill_tc_splits counts whole sets)
  const size_t cut = front + 128 + tq4::prefill_tc_image_bytes(head_dim) + (size_t)(vectors + num_q_heads) * (head_dim + 1) * 4;
  return cut > least ? cut : least;
}

// Shared body of the attention entry points: `wr` (optional) is a cache write of new tokens that must land
// before the attention reads the cache.
static int attention_impl(
    const tq4::CompressArgs* wr,
    const void* q, int q_dtype, int64_t num_rows, int num_seqs, int num_q_heads, int num_kv_heads,
    int head_dim, int64_t q_token_stride, int64_t q_head_stride, const uint8_t* cache,
    int64_t cache_block_stride, int64_t cache_token_stride, int64_t num_blocks, int block_size,
    const int32_t* block_table, int64_t bt_stride, const int32_t* seq_lens,
    const int32_t* query_start_loc, int64_t max_seq_len, const float* k_centroids, int n_k_centroids,
    const float* v_centroids, int n_v_centroids, const float* rotation, float sm_scale, int causal,
    int sliding_window, void* out, int out_dtype, int64_t out_token_stride, int64_t out_head_stride,
    float* lse_out, int out_rotated, void* workspace, size_t workspace_bytes, int mode,
    int* err_flag, void* stream) {
  using namespace tq4;
  if (num_rows < 0 || num_seqs < 0 || block_size <= 0 || num_blocks < 0) return TQ4_ERR_INVALID_ARG;
  if (!supported_head_dim(head_dim)) return TQ4_ERR_UNSUPPORTED;
  if (q_dtype < 0 || q_dtype > 2 || out_dtype < 0 || out_dtype > 2) return TQ4_ERR_UNSUPPORTED;
  if (n_k_centroids <= 0 || n_k_centroids > TQ4_MAX_CENTROIDS || n_v_centroids <= 0 ||
      n_v_centroids > TQ4_MAX_CENTROIDS)
    return TQ4_ERR_UNSUPPORTED;
  AttnArgs a{};
  if (!make_shape(a.sh, num_q_heads, num_kv_heads, head_dim)) return TQ4_ERR_UNSUPPORTED;
  if (num_rows == 0) return wr ? launch_prologue(nullptr, wr, head_dim, (cudaStream_t)stream) : TQ4_OK;
  if (!q || !cache || !block_table || !seq_lens || !k_centroids || !v_centroids || !rotation ||
      !out || !workspace)
    return TQ4_ERR_INVALID_ARG;
  if (((uintptr_t)cache & 3) || (cache_token_stride & 3) || (cache_block_stride & 3) ||
      ((uintptr_t)workspace & 15) ||
      cache_token_stride < row_data_bytes(num_kv_heads, head_dim))
    return TQ4_ERR_INVALID_ARG;
  if (query_start_loc == nullptr && num_rows > num_seqs) return TQ4_ERR_INVALID_ARG;
  const bool mma_ok = attention_mma_supported(a.sh, block_size, cache, cache_block_stride,
                                              cache_token_stride);
  if (mode == 2 && !mma_ok) return TQ4_ERR_UNSUPPORTED;
  if (mode < 0 || mode > 4) return TQ4_ERR_INVALID_ARG;
  const bool use_mma = mode == 2 || mode == 3 || mode == 4 || (mode == 0 && mma_ok);
  if (use_mma)
    make_shape(a.sh, num_q_heads, num_kv_heads, head_dim, mma_warps_per_cta(head_dim, a.sh.GC, num_kv_heads, cache_token_stride));
  const int64_t rows_cap = num_rows < kMaxRowsPerLaunch ? num_rows : kMaxRowsPerLaunch;
  // tensor-core kernel: one partial per (row, span), one span per warp phase of every CTA
  const int part_tpc = use_mma ? 1 : a.sh.TPC;
  const int64_t max_spans = use_mma ? (int64_t)kMaxSms * a.sh.TPC : kMaxCtasPerSlice;
  if (workspace_bytes < carve_plan(a.plan, nullptr, rows_cap, num_q_heads, head_dim, part_tpc, max_spans))
    return TQ4_ERR_WORKSPACE;
  carve_plan(a.plan, workspace, rows_cap, num_q_heads, head_dim, part_tpc, max_spans);

  a.sh.num_seqs = num_seqs;
  a.q = q;
  a.q_dtype = q_dtype;
  a.q_token_stride = q_token_stride;
  a.q_head_stride = q_head_stride;
  a.cache = cache;
  a.cache_block_stride = cache_block_stride;
  a.cache_token_stride = cache_token_stride;
  a.num_blocks = num_blocks;
  a.block_size = block_size;
  a.block_table = block_table;
  a.bt_stride = bt_stride;
  a.seq_lens = seq_lens;
  a.query_start_loc = query_start_loc;
  a.max_keys = bt_stride * block_size;
  if (max_seq_len > 0 && max_seq_len < a.max_keys) a.max_keys = max_seq_len;
  a.k_centroids = k_centroids;
  a.v_centroids = v_centroids;
  a.n_k_centroids = n_k_centroids;
  a.n_v_centroids = n_v_centroids;
  a.rotation = rotation;
  a.scale_log2e = sm_scale * 1.4426950408889634f;
  a.lut_scale_k = lut_scale(head_dim, n_k_centroids);
  a.lut_scale_v = lut_scale(head_dim, n_v_centroids);
  a.causal = causal;
  a.sliding_window = sliding_window > 0 ? sliding_window : 0;
  a.out = out;
  a.out_dtype = out_dtype;
  a.out_token_stride = out_token_stride;
  a.out_head_stride = out_head_stride;
  a.lse_out = lse_out;
  a.out_rotated = out_rotated;
  a.err_flag = err_flag;
  a.plan_records = use_mma;

  // Chunked prefill: the tcgen05 kernel takes the sequences with at least kPrefillMinRows new rows (a tile
  // costs it the same for 1 row as for 128 / G, and about as much as the streaming kernel's pass for six of
  // them), the streaming kernel the others.  The lengths are on the device, so a call that may hold both kinds
  // launches both; one sequence, or many rows per sequence (where the odd short one costs less than the
  // streaming kernels' launches), takes one kernel.
  const bool prefill_ok = prefill_tc_supported(a);
  if ((mode == 3 || mode == 4) && !prefill_ok) return TQ4_ERR_UNSUPPORTED;
  const bool all_long = mode == 3 || mode == 4 || (num_seqs == 1 && num_rows >= kPrefillMinRows) || num_rows >= 256 * (int64_t)num_seqs;
  // A call of few rows is the streaming kernel's alone: one pass of launches instead of two, and none of the fixed costs
  // of a prefill tile (Pi's image, rotating and un-rotating 128 rows: 20 us).  45 drawn steps: up to 4096 rows times
  // query heads streaming took 0.43 - 1.0 of the time (34 rows beside 21 running sequences, 28 / 4 heads: 25.9
  // against 49.9 us), above 5000 1.3 - 2.5 times it; head_dim 256, where it reads each row twice: the line is at 2048.
  // And not where long contexts make it re-read more than some 50 us of bytes.  Their length is the caller's
  // max_seq_len: by the width of a server's table (32 768 tokens) 34 rows of at most 26 keys took 66.6 us instead of 25.6,
  // 80 of at most 985 took 87.1 instead of 50.2 (32 / 8 heads of 128).
  const int64_t keys = a.max_keys;
  const bool few = use_mma && num_rows * num_q_heads <= (head_dim == 256 ? 2048 : 4096) &&
                   num_rows * keys * row_data_bytes(num_kv_heads, head_dim) <= (1ll << 28);
  const bool use_prefill = prefill_ok && (mode == 3 || mode == 4 || (mode == 0 && !few && num_rows >= kPrefillMinRows && (num_seqs > 1 || all_long)));
  const bool use_stream = !use_prefill || !all_long;
  a.skip_long = use_prefill && use_stream ? kPrefillMinRows : 0;

  const int sms = sm_count();
  int ctas = (use_mma ? 1 : 4) * sms / a.sh.n_slices;
  if (ctas < 1) ctas = 1;
  if (ctas > kMaxCtasPerSlice) ctas = kMaxCtasPerSlice;
  if (use_mma && ctas > kMaxSms) ctas = kMaxSms;
  a.sh.ctas = ctas;
  a.sh.span_ctas = use_mma ? ctas * a.sh.TPC : ctas;
  a.sh.part_tpc = part_tpc;
  cudaStream_t st = (cudaStream_t)stream;
  // TQ4_FUSED_PROLOGUE=1: decode calls of up to kFusedMaxRows rows plan, rotate and write inside the
  // attention kernel (two launches per step instead of three).  Never faster than the prologue kernel in
  // front (B200, graph replays, 32 / 8 heads, head_dim 128: 86.3 against 81.7 us at 64 x 4096, 92.9 / 92.5 at
  // 128 x 2048, 161.2 / 158.9 at 256 x 2048, 192.2 / 188.9 at 512 x 1024), so only the environment selects it.
  const char* fused_env = getenv("TQ4_FUSED_PROLOGUE");
  const bool want_fused = fused_env != nullptr && atoi(fused_env) != 0;
  a.fused = use_mma && query_start_loc == nullptr && num_rows <= kFusedMaxRows &&
            head_dim <= 128 && want_fused;

  a.sh.rows = (int)rows_cap;
  const int cl_shift = mode == 0 && use_mma && !use_prefill && num_rows <= kMaxRowsPerLaunch && !a.fused ? decode_step_cluster(a) : -1;
  if (cl_shift >= 0) {
    a.no_plan = 1;
    const bool rotate = !wr && decode_step_rotates(a);
    if (!rotate) {
      prof_begin(TQ4_PROF_PROLOGUE, st);
      const int rc = launch_prologue(&a, wr, head_dim, st);
      prof_end(TQ4_PROF_PROLOGUE, st);
      if (rc != TQ4_OK) return rc;
    }
    prof_begin(TQ4_PROF_ATTENTION, st);
    const int rc = launch_decode_step(a, cl_shift, rotate, st);
    prof_end(TQ4_PROF_ATTENTION, st);
    return rc;
  }

  for (int64_t r0 = 0; use_stream && r0 < num_rows; r0 += kMaxRowsPerLaunch) {
    a.sh.rows = (int)((num_rows - r0) < kMaxRowsPerLaunch ? (num_rows - r0) : kMaxRowsPerLaunch);
    a.sh.row_offset = (int)r0;
    int rc;
    if (a.fused) {  // no prologue kernel; a decode step's cache write rides in the attention kernel
      a.fused_write = nullptr;
      if (wr && a.sh.NCH == 1 && wr->n_tokens <= num_rows && getenv("TQ4_NO_FUSED_WRITE") == nullptr) {
        a.fused_write = wr;
      } else if (wr) {
        prof_begin(TQ4_PROF_WRITE, st);
        rc = dispatch_compress(*wr, head_dim, wr->x_dtype, st);
        prof_end(TQ4_PROF_WRITE, st);
        if (rc != TQ4_OK) return rc;
      }
    } else {
      prof_begin(TQ4_PROF_PROLOGUE, st);
      rc = launch_prologue(&a, r0 == 0 ? wr : nullptr, head_dim, st);
      prof_end(TQ4_PROF_PROLOGUE, st);
      if (rc != TQ4_OK) return rc;
    }
    prof_begin(TQ4_PROF_ATTENTION, st);
    rc = use_mma ? launch_attention_mma(a, st) : launch_attention_fp32(a, st);
    prof_end(TQ4_PROF_ATTENTION, st);
    if (rc != TQ4_OK) return rc;
    CombineArgs c{};
    c.slot_base = a.plan.slot_base;
    if (a.skip_long > 0) {
      c.active_rows = a.plan.scalars + 2;
      c.row_end = a.plan.kv_end;
    }
    c.TPC = a.sh.part_tpc;
    c.part_o = a.plan.part_o;
    c.part_m = a.plan.part_m;
    c.part_l = a.plan.part_l;
    c.rows = a.sh.rows;
    c.row_offset = a.sh.row_offset;
    c.Hq = num_q_heads;
    c.rotation = rotation;
    c.out = out;
    c.out_dtype = out_dtype;
    c.out_token_stride = out_token_stride;
    c.out_head_stride = out_head_stride;
    c.lse_out = lse_out;
    c.out_rotated = out_rotated;
    prof_begin(TQ4_PROF_COMBINE, st);
    rc = launch_combine(c, head_dim, st, true);
    prof_end(TQ4_PROF_COMBINE, st);
    if (rc != TQ4_OK) return rc;
  }
  if (!use_prefill) return TQ4_OK;

  // ---- the prefill kernel: all its sequences in one launch; the scratch of the streaming part is free again ----
  a.sh.rows = (int)num_rows;
  a.sh.row_offset = 0;
  if (wr && !use_stream) {
    prof_begin(TQ4_PROF_WRITE, st);
    const int rc = dispatch_compress(*wr, head_dim, wr->x_dtype, st);
    prof_end(TQ4_PROF_WRITE, st);
    if (rc != TQ4_OK) return rc;
  }
  // scratch: Pi's image, then the partials of a call cut along the keys; behind the plan where that is still
  // needed (the merge kernel tells by its ranges which rows are the prefill kernel's)
  const uintptr_t at = use_stream ? (uintptr_t)a.plan.part_o : (uintptr_t)workspace;
  uint8_t* image = reinterpret_cast<uint8_t*>((at + 127) & ~(uintptr_t)127);
  float* part_o = reinterpret_cast<float*>(image + prefill_tc_image_bytes(head_dim));
  const int64_t room = (int64_t)((uintptr_t)workspace + workspace_bytes) - (int64_t)(uintptr_t)part_o;
  const int splits = use_stream && num_rows > kMaxRowsPerLaunch
                         ? 1 : prefill_tc_splits(a, room / ((int64_t)num_q_heads * (head_dim + 1) * 4) - 1);
  const bool to_parts = splits > 1;
  float* part_m = part_o + (size_t)splits * num_rows * num_q_heads * head_dim;
  prof_begin(TQ4_PROF_ATTENTION, st);
  int rc = launch_prefill_tc(a, st, mode == 4, use_stream ? kPrefillMinRows : 1, splits, to_parts, image, part_o, part_m);
  prof_end(TQ4_PROF_ATTENTION, st);
  if (rc != TQ4_OK || !to_parts) return rc;
  CombineArgs c{};
  c.world = splits;
  c.part_o = part_o;
  c.part_m = part_m;
  c.rows = (int)num_rows;
  c.row_end = use_stream ? a.plan.kv_end : nullptr;
  c.rows_long = 1;
  c.Hq = num_q_heads;
  c.rotation = rotation;
  c.out = out;
  c.out_dtype = out_dtype;
  c.out_token_stride = out_token_stride;
  c.out_head_stride = out_head_stride;
  c.lse_out = lse_out;
  c.out_rotated = out_rotated;
  prof_begin(TQ4_PROF_COMBINE, st);
  rc = launch_combine(c, head_dim, st, true);
  prof_end(TQ4_PROF_COMBINE, st);
  return rc;
}

extern "C" int tq4_paged_attention(
    const void* q, int q_dtype, int64_t num_rows, int num_seqs, int num_q_heads, int num_kv_heads,
    int head_dim, int64_t q_token_stride, int64_t q_head_stride, const uint8_t* cache,
    int64_t cache_block_stride, int64_t cache_token_stride, int64_t num_blocks, int block_size,
    const int32_t* block_table, int64_t bt_stride, const int32_t* seq_lens,
    const int32_t* query_start_loc, const float* k_centroids, int n_k_centroids,
    const float* v_centroids, int n_v_centroids, const float* rotation, float sm_scale, int causal,
    int sliding_window, void* out, int out_dtype, int64_t out_token_stride, int64_t out_head_stride,
    float* lse_out, int out_rotated, void* workspace, size_t workspace_bytes, int mode,
    int* err_flag, void* stream) {
  return attention_impl(nullptr, q, q_dtype, num_rows, num_seqs, num_q_heads, num_kv_heads, head_dim,
                        q_token_stride, q_head_stride, cache, cache_block_stride, cache_token_stride,
                        num_blocks, block_size, block_table, bt_stride, seq_lens, query_start_loc, 0,
                        k_centroids, n_k_centroids, v_centroids, n_v_centroids, rotation, sm_scale,
                        causal, sliding_window, out, out_dtype, out_token_stride, out_head_stride,
                        lse_out, out_rotated, workspace, workspace_bytes, mode, err_flag, stream);
}

extern "C" int tq4_attention_step(
    const void* key, const void* value, int kv_dtype, int64_t n_tokens, int64_t k_token_stride,
    int64_t k_head_stride, int64_t v_token_stride, int64_t v_head_stride,
    const int64_t* slot_mapping, int64_t n_slots, const float* rot_t_even, const float* rot_t_odd,
    const float* k_boundaries, int n_k_boundaries, const float* v_boundaries, int n_v_boundaries,
    const void* q, int q_dtype, int64_t num_rows, int num_seqs, int num_q_heads, int num_kv_heads,
    int head_dim, int64_t q_token_stride, int64_t q_head_stride, uint8_t* cache,
    int64_t cache_block_stride, int64_t cache_token_stride, int64_t num_blocks, int block_size,
    const int32_t* block_table, int64_t bt_stride, const int32_t* seq_lens,
    const int32_t* query_start_loc, int64_t max_seq_len, const float* k_centroids, int n_k_centroids,
    const float* v_centroids, int n_v_centroids, const float* rotation, float sm_scale, int causal,
    int sliding_window, void* out, int out_dtype, int64_t out_token_stride, int64_t out_head_stride,
    float* lse_out, int out_rotated, void* workspace, size_t workspace_bytes, int mode,
    int* err_flag, void* stream) {
  using namespace tq4;
  if (n_tokens < 0 || n_slots < 0 || num_kv_heads <= 0 || block_size <= 0 || num_blocks < 0)
    return TQ4_ERR_INVALID_ARG;
  if (!supported_head_dim(head_dim) || kv_dtype < 0 || kv_dtype > 2) return TQ4_ERR_UNSUPPORTED;
  if (n_k_boundaries < 0 || n_k_boundaries > TQ4_MAX_BOUNDARIES || n_v_boundaries < 0 ||
      n_v_boundaries > TQ4_MAX_BOUNDARIES)
    return TQ4_ERR_UNSUPPORTED;
  CompressArgs w{};
  const CompressArgs* wr = nullptr;
  if (n_tokens > 0 && n_slots > 0) {
    if (!key || !value || !slot_mapping || !rot_t_even || !rot_t_odd || !k_boundaries || !v_boundaries ||
        !cache)
      return TQ4_ERR_INVALID_ARG;
    if (((uintptr_t)rot_t_even | (uintptr_t)rot_t_odd) & 15) return TQ4_ERR_INVALID_ARG;
    if (((uintptr_t)cache & 3) || (cache_token_stride & 3) ||
        cache_token_stride < row_data_bytes(num_kv_heads, head_dim) ||
        cache_block_stride != (int64_t)block_size * cache_token_stride)  // flat slots = block-major rows
      return TQ4_ERR_INVALID_ARG;
    w.x[0] = key;
    w.x[1] = value;
    w.token_stride[0] = k_token_stride;
    w.head_stride[0] = k_head_stride;
    w.token_stride[1] = v_token_stride;
    w.head_stride[1] = v_head_stride;
    w.bounds[0] = k_boundaries;
    w.n_bounds[0] = n_k_boundaries;
    w.bounds[1] = v_boundaries;
    w.n_bounds[1] = n_v_boundaries;
    w.n_tokens = n_tokens < n_slots ? n_tokens : n_slots;
    w.num_heads = num_kv_heads;
    w.n_sources = 2;
    w.x_dtype = kv_dtype;
    w.rot_even = rot_t_even;
    w.rot_odd = rot_t_odd;
    w.cache = cache;
    w.slot_mapping = slot_mapping;
    w.n_slots = n_slots;
    w.cache_token_stride = cache_token_stride;
    w.num_cache_slots = num_blocks * block_size;
    w.err_flag = err_flag;
    wr = &w;
  }
  return attention_impl(wr, q, q_dtype, num_rows, num_seqs, num_q_heads, num_kv_heads, head_dim,
                        q_token_stride, q_head_stride, cache, cache_block_stride, cache_token_stride,
                        num_blocks, block_size, block_table, bt_stride, seq_lens, query_start_loc, max_seq_len,
                        k_centroids, n_k_centroids, v_centroids, n_v_centroids, rotation, sm_scale,
                        causal, sliding_window, out, out_dtype, out_token_stride, out_head_stride,
                        lse_out, out_rotated, workspace, workspace_bytes, mode, err_flag, stream);
}

extern "C" int tq4_write_and_attention(
    const void* key, const void* value, int kv_dtype, int64_t n_tokens, int64_t k_token_stride,
    int64_t k_head_stride, int64_t v_token_stride, int64_t v_head_stride,
    const int64_t* slot_mapping, int64_t n_slots, const float* rot_t_even, const float* rot_t_odd,
    const float* k_boundaries, int n_k_boundaries, const float* v_boundaries, int n_v_boundaries,
    const void* q, int q_dtype, int64_t num_rows, int num_seqs, int num_q_heads, int num_kv_heads,
    int head_dim, int64_t q_token_stride, int64_t q_head_stride, uint8_t* cache,
    int64_t cache_block_stride, int64_t cache_token_stride, int64_t num_blocks, int block_size,
    const int32_t* block_table, int64_t bt_stride, const int32_t* seq_lens,
    const int32_t* query_start_loc, const float* k_centroids, int n_k_centroids,
    const float* v_centroids, int n_v_centroids, const float* rotation, float sm_scale, int causal,
    int sliding_window, void* out, int out_dtype, int64_t out_token_stride, int64_t out_head_stride,
    float* lse_out, int out_rotated, void* workspace, size_t workspace_bytes, int mode,
    int* err_flag, void* stream) {
  return tq4_attention_step(key, value, kv_dtype, n_tokens, k_token_stride, k_head_stride, v_token_stride, v_head_stride,
                            slot_mapping, n_slots, rot_t_even, rot_t_odd, k_boundaries, n_k_boundaries, v_boundaries,
                            n_v_boundaries, q, q_dtype, num_rows, num_seqs, num_q_heads, num_kv_heads, head_dim,
                            q_token_stride, q_head_stride, cache, cache_block_stride, cache_token_stride, num_blocks,
                            block_size, block_table, bt_stride, seq_lens, query_start_loc, 0, k_centroids, n_k_centroids,
                            v_centroids, n_v_centroids, rotation, sm_scale, causal, sliding_window, out, out_dtype,
                            out_token_stride, out_head_stride, lse_out, out_rotated, workspace, workspace_bytes, mode,
                            err_flag, stream);
}

extern "C" int tq4_combine_partials(const float* parts_o, const float* parts_lse, int world,
                                    int64_t num_rows, int num_q_heads, int head_dim,
                                    const float* rotation, void* out, int out_dtype,
                                    int64_t out_token_stride, int64_t out_head_stride,
                                    void* stream) {
  using namespace tq4;
  if (world <= 0 || num_rows < 0 || num_q_heads <= 0) return TQ4_ERR_INVALID_ARG;
  if (!supported_head_dim(head_dim) || out_dtype < 0 || out_dtype > 2) return TQ4_ERR_UNSUPPORTED;
  if (num_rows == 0) return TQ4_OK;
  if (!parts_o || !parts_lse || !rotation || !out) return TQ4_ERR_INVALID_ARG;
  if (num_rows > 0x7fffffff) return TQ4_ERR_INVALID_ARG;
  CombineArgs c{};
  c.slot_base = nullptr;
  c.world = world;
  c.part_o = parts_o;
  c.part_m = parts_lse;
  c.rows = (int)num_rows;
  c.row_offset = 0;
  c.Hq = num_q_heads;
  c.rotation = rotation;
  c.out = out;
  c.out_dtype = out_dtype;
  c.out_token_stride = out_token_stride;
  c.out_head_stride = out_head_stride;
  return launch_combine(c, head_dim, (cudaStream_t)stream, false);
}

// ======================================================================================
// Allocation-free variant: the scratch lives in the library image.
// ======================================================================================
// One fixed scratch area per GPU that loads the library, held until the process exits.
static __device__ __align__(256) unsigned char g_static_scratch[TQ4_STATIC_SCRATCH_BYTES];

// Device address of g_static_scratch on the CURRENT device.  In host code the symbol's name is
// only a handle, never a device pointer, so the address is asked for once per device with
// cudaGetSymbolAddress (while that device is current) and remembered.
static int static_scratch_address(void** out) {
  static void* cached[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TQ4_ERR_CUDA;
  if (cached[dev] == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || p == nullptr) return TQ4_ERR_CUDA;
    cached[dev] = p;
  }
  *out = cached[dev];
  return TQ4_OK;
}

extern "C" int tq4_paged_attention_static(
    const void* q, int q_dtype, int64_t num_rows, int num_seqs, int num_q_heads, int num_kv_heads,
    int head_dim, int64_t q_token_stride, int64_t q_head_stride, const uint8_t* cache,
    int64_t cache_block_stride, int64_t cache_token_stride, int64_t num_blocks, int block_size,
    const int32_t* block_table, int64_t bt_stride, const int32_t* seq_lens,
    const int32_t* query_start_loc, const float* k_centroids, int n_k_centroids,
    const float* v_centroids, int n_v_centroids, const float* rotation, float sm_scale, int causal,
    int sliding_window, void* out, int out_dtype, int64_t out_token_stride, int64_t out_head_stride,
    int mode, int* err_flag, void* stream) {
  if (num_rows < 0) return TQ4_ERR_INVALID_ARG;
  if (num_rows == 0) return TQ4_OK;
  const size_t need = workspace_min(num_rows, num_q_heads, num_kv_heads, head_dim);
  if (need == 0) return TQ4_ERR_UNSUPPORTED;
  if (need > (size_t)TQ4_STATIC_SCRATCH_BYTES) return TQ4_ERR_STATIC_SCRATCH;
  void* scratch = nullptr;
  const int rc = static_scratch_address(&scratch);
  if (rc != TQ4_OK) return rc;
  return tq4_paged_attention(q, q_dtype, num_rows, num_seqs, num_q_heads, num_kv_heads, head_dim,
                             q_token_stride, q_head_stride, cache, cache_block_stride,
                             cache_token_stride, num_blocks, block_size, block_table, bt_stride,
                             seq_lens, query_start_loc, k_centroids, n_k_centroids, v_centroids,
                             n_v_centroids, rotation, sm_scale, causal, sliding_window, out, out_dtype,
                             out_token_stride, out_head_stride, nullptr, 0, scratch,
                             (size_t)TQ4_STATIC_SCRATCH_BYTES, mode, err_flag, stream);
}
