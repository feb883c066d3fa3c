// Reconstruction of a prompt's compressed K and V vectors (the second half of a HuggingFace-style cache update) on the
// 5th-generation tensor cores: tiles of 128 vectors, a 128 x D x D GEMM each,
//     z = norm * (centroid[idx] * Pi)          (tcgen05.mma kind::f16, fp32 accumulator in tensor memory)
// with both operands as sums of two fp16 terms (centroids times a power of two, 2^8 Pi: 22 bits each) and all four products,
// the smallest first; z is rounded to the 16-bit type of the cache.
//
// One persistent CTA per SM.  Pi is the B operand, resident as an image whose rows are input coordinates.  The A operand of a
// tile is looked up from its packed bytes (a byte gives two centroids' hi and lo terms in one 8-byte load), while the
// tensor core works on the tile before and that one's predecessor is scaled, rounded and stored; the indices and norms go
// to the cache's buffers on the way.  The 70 400 vectors of 128 of a prompt of 4 x 1100 tokens (8 heads): 97 us by the FMA kernel that
// did this (bound by FMA issue and the reads of Pi), 20 here; what bounds it is the lookups (8192 a tile, and their operand
// stores) and, for few tiles a CTA, the preparation of Pi.
// The FMA kernel's operands had 24 bits, these have 22.  Of the values as rounded to 16 bits so many are not the rounded 64-bit
// result (8000 vectors x 6 rotations, K4/V3 and K2/V4), here / FMA kernel: bf16 1.4 - 2.0 / 1.8 - 2.3 in 10^4 at head_dim 64 and 96, 1.9 - 2.2
// / 2.2 - 2.5 at 128; fp16 0.9 - 1.3 / 1.2 - 1.5 in 10^3 and 1.3 - 1.4 / 1.5 - 1.6; the 2-norm of the error is the same to six figures.
// Waits are bounded: a wait that gives up leaves NaN in the vectors that it should have brought.
#include <math_constants.h>

#include <cstdlib>

#include "tq4_cache_update.cuh"

namespace tq4 {
namespace {

constexpr int kRows = 128;      // vectors per tile
constexpr int kThreads = 512;
constexpr int kCopies = 8;      // of a table entry, against bank conflicts

template <int D>
struct RestoreCfg {
  static constexpr int NC = (D + 63) / 64, NS = D / 32;            // 64-coordinate blocks, 16-byte segments of a packed vector
  static constexpr uint32_t kImgPart = D * 128, kImgTerm = NC * kImgPart;
  static constexpr uint32_t kATerm = NC * kRows * 128, kA = 2 * kATerm;
  static constexpr uint32_t kOffA = 2 * kImgTerm;
  static constexpr uint32_t kOffLut = kOffA + 2 * kA;               // [source][byte][copy] (hi pair, lo pair)
  static constexpr uint32_t kSmem = kOffLut + 2 * 256 * kCopies * 8;
  static constexpr int NIT = (kRows * NS + kThreads - 1) / kThreads;  // segments a thread
  static constexpr int CW = D / 4;                                  // columns an epilogue warp (four share a row quadrant)
  static constexpr int kPitch = D == 64 ? 48 : 80;                  // staged piece of a row, against bank conflicts
  static constexpr uint32_t kCols = 2 * D <= 128 ? 128 : 256;       // two accumulators
  static_assert(16 * 32 * kPitch <= kA, "the rows on their way out lie in an operand buffer");
  static_assert(kSmem <= 227 * 1024 - 1024, "shared memory");
};

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t swz(int row, int c) { return (uint32_t)(row * 128 + ((c ^ (row & 7)) << 4)); }
// operand, 128-byte swizzle, 8-row groups 1024 bytes apart; `lbo`: distance of the 64-element blocks of an MN-major one
__device__ __forceinline__ uint64_t make_desc(uint32_t a, uint32_t lbo) {
  return (uint64_t)((a & 0x3FFFFu) >> 4) | ((uint64_t)(lbo ? lbo >> 4 : 1) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool wait_bounded(uint32_t bar, uint32_t parity) {
  for (int it = 0; it < (1 << 22); ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void tmem_ld8(uint32_t t, uint32_t (&v)[8]) {  // (no wait)
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(t));
}
__device__ __forceinline__ void tmem_ld8_wait(uint32_t (&v)[8]) {  // names the registers: no use of them moves above it
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]));
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// two values -> fp16 hi pair and fp16 pair of what the rounding left
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x0, x1);
  const float2 f = __half22float2(h);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = pack_h2(x0 - f.x, x1 - f.y);
}

template <int D>
__global__ void __launch_bounds__(kThreads, 1) restore_tc_kernel(const UpdateArgs a) {
  using C = RestoreCfg<D>;
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ __align__(8) uint64_t s_bar[3];  // accumulator 0 / 1 complete; drain
  __shared__ uint32_t s_tmem;
  __shared__ float s_cent[2][16], s_unscale[2];
  __shared__ int s_dead;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = saddr(sm);

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&s_tmem)), "r"(C::kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  } else if (warp == 1) {
    // centroids times the power of two that brings the largest into [64, 128): their lo terms stay normal numbers
    const int src = lane >> 4, i = lane & 15;
    const float c = i < a.n_cents[src] ? __ldg(a.cents[src] + i) : 0.f;
    float top = fabsf(c);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    const int e = top > 0.f && top < CUDART_INF_F ? min(max((int)(__float_as_uint(top) >> 23) - 127, -100), 100) : 0;
    s_cent[src][i] = c * __uint_as_float((uint32_t)(127 + 6 - e) << 23);
    if (i == 0) s_unscale[src] = __uint_as_float((uint32_t)(127 - 6 - 8 + e) << 23);  // (and the 2^8 of Pi)
  } else if (warp == 2 && lane == 0) {
    for (int i = 0; i < 3; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(&s_bar[i])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_dead = 0;
  }
  // ---- Pi's image: [term][64-column block][row][128 B, swizzled]; columns past D are zero -----------------------------
  for (int i = tid; i < D * C::NC * 8; i += kThreads) {
    const int r = i / (C::NC * 8), k8 = i - r * (C::NC * 8);
    uint32_t hi[4] = {}, lo[4] = {};
    if (8 * k8 < D) {
      const float4* src = reinterpret_cast<const float4*>(a.rotation + (size_t)r * D + 8 * k8);
      const float4 x = __ldg(src), y = __ldg(src + 1);
      split2(256.f * x.x, 256.f * x.y, hi[0], lo[0]);
      split2(256.f * x.z, 256.f * x.w, hi[1], lo[1]);
      split2(256.f * y.x, 256.f * y.y, hi[2], lo[2]);
      split2(256.f * y.z, 256.f * y.w, hi[3], lo[3]);
    }
    unsigned char* dst = sm + (k8 >> 3) * C::kImgPart + swz(r, k8 & 7);
    *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(dst + C::kImgTerm) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
  __syncthreads();
  for (int i = tid; i < 2 * 256; i += kThreads) {
    const int src = i >> 8, b = i & 255;
    uint2 e;
    split2(s_cent[src][b >> 4], s_cent[src][b & 15], e.x, e.y);
    uint4* dst = reinterpret_cast<uint4*>(sm + C::kOffLut + (size_t)i * kCopies * 8);
#pragma unroll
    for (int c = 0; c < kCopies / 2; ++c) dst[c] = make_uint4(e.x, e.y, e.x, e.y);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;
  pdl_wait();  // the compressed vectors come from the kernel in front

  const int per_src = a.batch * a.heads * a.n_new, tiles_src = (per_src + kRows - 1) / kRows;
  const int my = (2 * tiles_src - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  // tile i of this CTA: its source and first vector (in the order of the cache's buffers: batch, head, token)
  auto tile_of = [&](int i, int& src, int& v0) {
    const int t = (int)blockIdx.x + i * (int)gridDim.x;
    src = t >= tiles_src ? 1 : 0;
    v0 = (t - src * tiles_src) * kRows;
  };
  // (batch * heads + head) and token of a vector, and where the compressed one lies
  auto place = [&](int src, unsigned vec, int& bh, int& s) -> int64_t {
    bh = (int)(vec / (unsigned)a.n_new);
    s = (int)(vec - (unsigned)bh * (unsigned)a.n_new);
    const int b = (int)((unsigned)bh / (unsigned)a.heads), h = bh - b * a.heads;
    return (int64_t)src * per_src + ((int64_t)b * a.n_new + s) * a.heads + h;
  };
  // segment n of this thread: eight lanes take a segment of eight vectors (their operand stores fall into eight bank groups)
  auto item = [&](int n, int& row, int& seg) -> bool {
    const int it = tid + kThreads * n, q = it >> 3;
    seg = q % C::NS;
    row = q / C::NS * 8 + (it & 7);
    return it < kRows * C::NS;
  };
  uint4 w[C::NIT];
  auto fetch = [&](int i) {
    int src, v0;
    tile_of(i, src, v0);
#pragma unroll
    for (int n = 0; n < C::NIT; ++n) {
      int row, seg, bh, s;
      w[n] = make_uint4(0u, 0u, 0u, 0u);
      if (item(n, row, seg) && v0 + row < per_src)
        w[n] = __ldcg(reinterpret_cast<const uint4*>(a.packed + place(src, v0 + row, bh, s) * (D / 2)) + seg);
    }
  };
  if (my > 0) fetch(0);
  bool ok = true;
  for (int i = 0; i <= my; ++i) {
    if (i < my) {
      // ---- indices to the cache, centroid terms into the operand buffer ------------------------------------------
      int src, v0;
      tile_of(i, src, v0);
      unsigned char* ab = sm + C::kOffA + (i & 1) * C::kA;
      const unsigned char* lut = sm + C::kOffLut + src * 256 * kCopies * 8 + (lane & (kCopies - 1)) * 8;
#pragma unroll
      for (int n = 0; n < C::NIT; ++n) {
        int row, seg, bh, s;
        if (!item(n, row, seg)) continue;
        const uint32_t x[4] = {w[n].x, w[n].y, w[n].z, w[n].w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint2 e[4];
#pragma unroll
          for (int b = 0; b < 4; ++b) e[b] = *reinterpret_cast<const uint2*>(lut + ((x[c] >> (8 * b)) & 255u) * (kCopies * 8));
          unsigned char* dst = ab + (seg >> 1) * (kRows * 128) + swz(row, (seg & 1) * 4 + c);
          *reinterpret_cast<uint4*>(dst) = make_uint4(e[0].x, e[1].x, e[2].x, e[3].x);
          *reinterpret_cast<uint4*>(dst + C::kATerm) = make_uint4(e[0].y, e[1].y, e[2].y, e[3].y);
        }
        if (v0 + row >= per_src) continue;
        place(src, v0 + row, bh, s);
        const int64_t at = (int64_t)bh * a.cap + a.offset + s;
        if (a.nibble[src]) {
          *reinterpret_cast<uint4*>(a.idx[src] + at * (D / 2) + 16 * seg) = w[n];
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) {  // byte p = index 2 p << 4 | index 2 p + 1
            const uint32_t hi = (x[c] >> 4) & 0x0F0F0F0Fu, lo = x[c] & 0x0F0F0F0Fu;
            *reinterpret_cast<uint2*>(a.idx[src] + at * D + 32 * seg + 8 * c) = make_uint2(__byte_perm(hi, lo, 0x5140), __byte_perm(hi, lo, 0x7362));
          }
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (i < my && warp == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_one()) {
        constexpr uint32_t idesc = (1u << 4) | (1u << 16) | ((uint32_t)(D >> 3) << 17) | ((128u >> 4) << 24);  // fp16, B MN-major
        const uint32_t d = tmem + (uint32_t)(i & 1) * D, ab = base + C::kOffA + (i & 1) * C::kA;
#pragma unroll 1
        for (int t = 3; t >= 0; --t)  // lo lo, lo hi, hi lo, hi hi
#pragma unroll
          for (int s = 0; s < D / 16; ++s)
            mma(d, make_desc(ab + (t >> 1) * C::kATerm + (s >> 2) * (kRows * 128) + 32u * (s & 3), 0),
                make_desc(base + (t & 1) * C::kImgTerm + 2048u * s, C::kImgPart), idesc, t != 3 || s > 0);
        commit(saddr(&s_bar[i & 1]));
      }
      __syncwarp();
    }
    if (i + 1 < my) fetch(i + 1);
    if (i > 0) {
      // ---- the tile before: scale, round, store (through its operand buffer, so that a row's pieces are stored together) ---
      const int j = i - 1;
      int src, v0;
      tile_of(j, src, v0);
      const int row = 32 * (warp & 3) + lane, cw = warp >> 2;
      const bool live = v0 + row < per_src;
      float f = 0.f;
      int64_t to = -1;  // of this lane's row
      if (live) {
        int bh, s;
        const int64_t from = place(src, v0 + row, bh, s);
        const float norm = __ldcg(a.packed_norms + from);
        f = norm * s_unscale[src];
        if (cw == 0) a.norms[src][(int64_t)bh * a.cap + a.offset + s] = norm;
        to = (((int64_t)bh * a.dec_cap + a.dec_offset + s) * D + C::CW * cw) * 2;
      }
      ok = __all_sync(0xffffffffu, ok && wait_bounded(saddr(&s_bar[j & 1]), (uint32_t)((j >> 1) & 1)));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (!ok) f = __int_as_float(0x7fc00000);
      unsigned char* stage = sm + C::kOffA + (j & 1) * C::kA + warp * 32 * C::kPitch;
#pragma unroll
      for (int q = 0; q < C::CW / 8; ++q) {
        uint32_t v[8], y[4];
        tmem_ld8(tmem + (uint32_t)(j & 1) * D + C::CW * cw + 8 * q + ((uint32_t)(32 * (warp & 3)) << 16), v);
        tmem_ld8_wait(v);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float y0 = __uint_as_float(v[2 * e]) * f, y1 = __uint_as_float(v[2 * e + 1]) * f;
          if (a.dtype == TQ4_F16) {
            y[e] = pack_h2(y0, y1);
          } else {
            const __nv_bfloat162 h = __floats2bfloat162_rn(y0, y1);
            y[e] = *reinterpret_cast<const uint32_t*>(&h);
          }
        }
        *reinterpret_cast<uint4*>(stage + lane * C::kPitch + 16 * q) = make_uint4(y[0], y[1], y[2], y[3]);
      }
      __syncwarp();
      constexpr int PCS = C::CW / 8;
      char* dec = reinterpret_cast<char*>(a.dec[src]);
#pragma unroll
      for (int n = 0; n < PCS; ++n) {
        const int k = lane + 32 * n, r = k / PCS, pc = k - r * PCS;
        const int64_t at = __shfl_sync(0xffffffffu, to, r);
        if (at >= 0) *reinterpret_cast<uint4*>(dec + at + 16 * pc) = *reinterpret_cast<const uint4*>(stage + r * C::kPitch + 16 * pc);
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();  // the buffer and the accumulator may be written again
  }
  if (!ok) s_dead = 1;
  __syncthreads();
  if (warp == 0) {
    if (s_dead) {  // MMAs that have not come home work on memory that the next CTA of the SM is given
      if (elect_one()) {
        commit(saddr(&s_bar[2]));
        wait_bounded(saddr(&s_bar[2]), 0u);
      }
      __syncwarp();
    }
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::kCols) : "memory");
  }
}

template <int D>
int launch_t(const UpdateArgs& a, cudaStream_t st) {
  using C = RestoreCfg<D>;
  // (more than half of an SM: one CTA each, whatever the head_dim)
  constexpr int smem = C::kSmem > 120 * 1024 ? (int)C::kSmem : 120 * 1024;
  if (!ensure_dynamic_smem<restore_tc_kernel<D>>(smem)) return TQ4_ERR_CUDA;
  const int64_t tiles = 2 * (((int64_t)a.batch * a.heads * a.n_new + kRows - 1) / kRows);
  const int64_t most = sm_count();
  if (launch_kernel(restore_tc_kernel<D>, dim3((unsigned)(tiles < most ? tiles : most)), dim3(kThreads), (size_t)smem, st, true, a) != cudaSuccess)
    return TQ4_ERR_CUDA;
  TQ4_CHECK_LAUNCH();
  return TQ4_OK;
}

}  // namespace

bool restore_tc_eligible(const UpdateArgs& a, int head_dim) {
  static const bool disabled = getenv("TQ4_NO_TC") != nullptr;
  if (disabled) return false;
  if ((a.dtype != TQ4_F16 && a.dtype != TQ4_BF16) || head_dim > 128 || a.dec[0] == nullptr || (uintptr_t)a.packed % 16) return false;
  for (int s = 0; s < 2; ++s)
    if ((uintptr_t)a.idx[s] % 16 || (uintptr_t)a.dec[s] % 16) return false;
  return true;
}

int launch_restore_tc(const UpdateArgs& a, int head_dim, cudaStream_t st) {
  switch (head_dim) {
    case 64: return launch_t<64>(a, st);
    case 96: return launch_t<96>(a, st);
    case 128: return launch_t<128>(a, st);
  }
  return TQ4_ERR_UNSUPPORTED;
}

}  // namespace tq4
