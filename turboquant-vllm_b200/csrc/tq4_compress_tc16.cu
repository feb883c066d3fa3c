// TQ4 compress for prefill-sized 16-bit inputs, pipelined on the 5th-generation tensor cores.  The rotation
// of a tile of 128 vectors is a 128 x D x D GEMM
//     Y_raw = X * Pi^T        (tcgen05.mma kind::f16, fp32 accumulator in tensor memory)
// on the RAW input rows: a 16-bit input is exact as an MMA operand, so the A operand needs no
// CUDA-core preparation at all and arrives in shared memory by TMA in the swizzled layout the MMA
// reads.  Pi is the B operand, resident in shared memory as a sum of 16-bit terms (bf16 inputs:
// three bf16 terms = 24 bits; fp16 inputs: 2^8 * Pi as fp16 hi + lo = 22 bits), one MMA per term.
// At head_dim 256 the terms do not fit: a CTA owns 64 of the output coordinates (its rows are read by four
// CTAs, three times from L2).
// The normalisation commutes with the product: y = Y_raw / (norm + 1e-10) is applied to the fp32
// accumulator in the epilogue.  A rotated coordinate therefore differs from the fp32 FMA kernels by
// ~1e-7 absolute, which moves an index only when the coordinate sits that close to a bucket
// boundary (bound 1e-4 of the indices).  Norms are summed in exactly the order of the FMA kernels
// (lane-strided FMAs, butterfly tree), so they are bit-identical to them.
//
// One persistent CTA per SM, warp-specialised, four (head_dim 256: two) input stages and accumulators in flight:
//   warp 0      TMA producer: the 128 rows of a tile as 64-column boxes (128-byte swizzle)
//   warp 1      MMA issuer: D / 16 k-steps x terms of tcgen05.mma, then tcgen05.commit onto the stage's "empty"
//               barrier and the accumulator's "full" barrier
//   warps 2 ..  one epilogue group of four warps per stage; tile i of the CTA belongs to group i % stages and uses
//               that input stage and accumulator, so every barrier is waited on by one group in tile order (a
//               stage shared between groups could show a fast group an older phase).  Thread = row: sum
//               of squares from the staged tile -> release the stage -> wait for the accumulator -> per 32
//               columns: tcgen05.ld, scale, bucketize, nibble-pack, one 16-byte store into the packed output
//               or the paged cache row.
// What bounds it is the epilogue's instruction count, and in it the bucketize.  A search over registers takes 22
// instructions a coordinate.  Here a coordinate is first mapped to one of 32 uniform cells, each of which holds at
// most one boundary (checked when the CTA starts, with a margin for the rounding of the map; codebooks whose
// boundaries are too close for that take the search): two FMAs, two lookups through the warp shuffle
// (lane c holds cell c's boundary and the index below it), one compare, one add.  The comparison is the
// search's own, against the same fp32 boundary, so the indices are the same.  Measured (bf16 cache write, K and
// V): 16384 tokens of 8 heads of 128 48.6 -> 31.1 us (2.7 TB/s), 8208 vectors 24 -> 11.1 us
// against a block per vector, 16384 tokens of 4 heads of 256 894 -> 91 us (62 without the
// second sums below; the 256 columns are split over CTAs:
// one cannot hold Pi and two stages of vectors).
// Every mbarrier wait is bounded; a wait that gives up marks the CTA dead, all roles drain (tiles and MMAs in flight are
// waited for, again within a bound: they work on memory that the next CTA of the SM is given) and the
// kernel reports TQ4_DEV_TIMEOUT.  Tensor memory is released on every path.
#include <math_constants.h>

#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "tq4_common.cuh"

namespace tq4 {
#ifdef TQ4_TRACE
// Tuning builds only (-DTQ4_TRACE): SM clock at points of the tile pipeline of CTA 0 (producer warp,
// MMA warp, first warp of epilogue groups 0 and 1), read back with tq4_compress_trace_read.
__device__ long long g_ctrace[4][32][8];
#define CT_STAMP(role, i, e)                                                                   \
  do {                                                                                         \
    if (blockIdx.x == 0 && (threadIdx.x & 31) == 0 && (i) < 32) g_ctrace[role][i][e] = clock64(); \
  } while (0)
#else
#define CT_STAMP(role, i, e) do {} while (0)
#endif

namespace {

constexpr int kRows = 128;                       // vectors per tile (MMA M, TMEM lanes)
constexpr uint32_t kBlockBytes = kRows * 128;    // one 64-column block of the input tile: 16 KB
constexpr int kMaxTerms = 3;

template <int D>
struct Cfg {
  static constexpr int KB = (D + 63) / 64;                 // 64-column blocks of a vector
  static constexpr int N = D == 256 ? 64 : D;              // output coordinates of a CTA
  static constexpr int NSPLIT = D / N;
  static constexpr int STAGES = D == 256 ? 2 : 4;          // input stages = epilogue groups = accumulators
  static constexpr int THREADS = 64 + STAGES * 128;        // producer, issuer, four warps per group
  static constexpr uint32_t kBBlock = N * 128;             // a 64-column block of a term of Pi
  static constexpr uint32_t kTerm = KB * kBBlock;
  static constexpr uint32_t kTile = KB * kBlockBytes;      // an input stage
  static constexpr uint32_t kOffA = (kMaxTerms * kTerm + 1023) & ~1023u;
  static constexpr uint32_t kSmem = kOffA + STAGES * kTile;
  static constexpr uint32_t kTmemCols = STAGES * N <= 64 ? 64 : STAGES * N <= 128 ? 128 : STAGES * N <= 256 ? 256 : 512;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// byte offset of (row, 16-byte chunk c of the row's 128 bytes) inside a K-block (128-byte swizzle)
__device__ __forceinline__ uint32_t swz(int row, int c) { return (uint32_t)(row * 128 + ((c ^ (row & 7)) << 4)); }
// K-major operand, 128-byte swizzle, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// instruction descriptor: D = F32, A and B of 16-bit format `fmt` (0 = fp16, 1 = bf16), K-major, M = 128
__host__ __device__ constexpr uint32_t instr_desc(uint32_t fmt, uint32_t n) {
  return (1u << 4) | (fmt << 7) | (fmt << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait that also gives up as soon as another role has marked the CTA dead (`dead` null: only at its bound).
__device__ __forceinline__ bool bar_wait_bounded(uint32_t bar, uint32_t parity, const volatile int* dead) {
  for (int it = 0; it < (1 << 22); ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
    if ((it & 1023) == 1023 && dead && *dead) return false;
  }
  return false;
}
__device__ __forceinline__ bool elect_one_sync() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
      "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

template <typename T>
struct Fmt;  // how Pi is split into 16-bit terms for inputs of type T
template <>
struct Fmt<__half> {
  static constexpr int kTerms = 2;
  static constexpr uint32_t kCode = 0;
  static constexpr float kNear = 4e-7f;
  static constexpr float kScale = 256.f;  // keeps the lo term of small entries a normal fp16 number
  static __device__ __forceinline__ uint16_t term(float& rest) {
    const __half h = __float2half_rn(rest);
    rest -= __half2float(h);
    return __half_as_ushort(h);
  }
};
template <>
struct Fmt<__nv_bfloat16> {
  static constexpr int kTerms = 3;
  static constexpr uint32_t kCode = 1;
  static constexpr float kNear = 3.4e-7f;
  static constexpr float kScale = 1.f;
  static __device__ __forceinline__ uint16_t term(float& rest) {
    const __nv_bfloat16 h = __float2bfloat16_rn(rest);
    rest -= __bfloat162float(h);
    return __bfloat16_as_ushort(h);
  }
};

// pairs of fp32 values in one 64-bit register: one instruction does both
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// eight 16-bit elements (one 16-byte chunk) -> fp32 pairs
template <typename T>
__device__ __forceinline__ void chunk_to_pairs(const uint4& v, f2 (&x)[4]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      x[j] = pack2(__uint_as_float(w[j] << 16), __uint_as_float(w[j] & 0xFFFF0000u));
    } else {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
      x[j] = pack2(f.x, f.y);
    }
  }
}

// idx = #{b : b < y} over 15 ascending boundaries (padded with +inf) held in REGISTERS: a four-level
// binary search whose next boundary is picked with selects, so nothing in it touches memory (the
// shared-memory version is a chain of four dependent loads per coordinate, which two epilogue
// warps per scheduler cannot hide).  NaN compares false at every level -> 0.
__device__ __forceinline__ int bucketize_reg(float y, const float (&b)[15]) {
  const bool c1 = y > b[7];
  const bool c2 = y > (c1 ? b[11] : b[3]);
  const float t3 = c2 ? (c1 ? b[13] : b[5]) : (c1 ? b[9] : b[1]);
  const bool c3 = y > t3;
  const float lo4 = c2 ? (c1 ? b[12] : b[4]) : (c1 ? b[8] : b[0]);
  const float hi4 = c2 ? (c1 ? b[14] : b[6]) : (c1 ? b[10] : b[2]);
  const bool c4 = y > (c3 ? hi4 : lo4);
  return (c1 ? 8 : 0) + (c2 ? 4 : 0) + (c3 ? 2 : 0) + (c4 ? 1 : 0);
}

// The two roundings of a coordinate (this kernel's product, the FMA kernels' chains) lie 1 - 2e-8 apart on average; a coordinate
// nearer than Fmt<T>::kNear to a boundary (about 3e-5 of them) is summed again the FMA kernels' way, so that the bytes are theirs.
// That is a margin, not a bound.  Among 2.5e12 coordinates, two thirds of them of vectors that one, two or sixteen coordinates dominate
// (the rounding errors are then as large as the result allows), the largest distance was 3.1e-7 for bf16 and 3.6e-7 for fp16,
// whose Pi has 22 bits; with a margin of 1.5e-7 79 indices differed, from 3.2e-7 on none.  Half a unit a step of the FMA chains and a
// unit an accumulation, at the size of the outermost boundary, would add up to 1.3e-6 at head_dim 128.  With margins of 1.5e-7 / these /
// 1.3e-6 a write of K and V takes, us (bf16): 16384 tokens x 4 heads of 256 82 / 91 / 147, 512 x 8 of 128 15.3 / 17.4 / 20.0 (18.5 by the
// FMA kernels), 4000 x 32 of 96 33.0 / 35.4 / 39.9, 16384 x 2 of 64 14.5 / 14.5 / 16.4.
// (Not in large writes at head_dim 128, which have been the tensor cores' own for longer than there was a choice.)

// The 32-cell map: cell = round(31 * sat(y * s / 31 + 16 / 31)), so y = 0 sits in the middle of cell 16 and
// everything past the ends in the end cells.  `scale` = s / 31; lane c: the boundary inside cell c (+inf: none) and the
// number of boundaries in the cells below.
struct Grid {
  float scale, bound;
  int below;
};
// Grid of 15 ascending boundaries (padded with +inf); false if no scale puts every boundary into a cell of its own, at
// least 1e-3 of a cell away from its edges.  One warp; lane i tries the i-th scale.
__device__ __forceinline__ bool make_grid(const float* b, Grid& g, int lane) {
  float last = 0.f;
  for (int i = 0; i < 15; ++i)
    if (b[i] < CUDART_INF_F) last = fmaxf(last, fabsf(b[i]));
  const float s = last > 0.f ? 15.3f / last * (1.f - 0.01f * lane) : 1.f;
  bool ok = last < CUDART_INF_F;
  float prev = -1.f;
  for (int i = 0; i < 15; ++i) {
    if (!(b[i] < CUDART_INF_F)) continue;
    const float x = fmaf(b[i], s, 16.f), c = rintf(x);
    ok = ok && c > prev && c >= 0.f && c <= 31.f && fabsf(x - c) < 0.499f;
    prev = c;
  }
  const unsigned m = __ballot_sync(0xffffffffu, ok);
  if (m == 0) return false;
  const float best = __shfl_sync(0xffffffffu, s, __ffs(m) - 1);
  g.scale = best / 31.f;
  g.bound = CUDART_INF_F;
  g.below = 0;
  for (int i = 0; i < 15; ++i) {
    if (!(b[i] < CUDART_INF_F)) continue;
    const int c = (int)rintf(fmaf(b[i], best, 16.f));
    if (c == lane) g.bound = b[i];
    if (c < lane) ++g.below;
  }
  return true;
}
__device__ __forceinline__ int bucketize_grid(float y, const Grid& g) {
  const float u = fmaf(__saturatef(fmaf(y, g.scale, 16.f / 31.f)), 31.f, 8388608.f);  // (2^23: the cell in the low bits)
  const int c = __float_as_int(u);  // (the shuffle takes the source lane modulo 32)
  return __shfl_sync(0xffffffffu, g.below, c) + (y > __shfl_sync(0xffffffffu, g.bound, c) ? 1 : 0);
}

// The same, with the distance to the boundary (its sign decides: y - bound is zero only where they are equal)
__device__ __forceinline__ int bucketize_grid(float y, const Grid& g, float& d) {
  const float u = fmaf(__saturatef(fmaf(y, g.scale, 16.f / 31.f)), 31.f, 8388608.f);
  const int c = __float_as_int(u);
  d = y - __shfl_sync(0xffffffffu, g.bound, c);
  return __shfl_sync(0xffffffffu, g.below, c) + (d > 0.f ? 1 : 0);
}

// 32 coordinates of a row that are summed again, later: where they go, the row, 2 * chunk + source
struct Again {
  uint8_t* dst;
  unsigned row, where;
};
template <int D> constexpr int kAgainMax = D == 128 ? 4 : 8;  // a warp's list (what shared memory leaves)

// The chunks on a warp's list by the sums of the FMA kernels: the norm, then lane = coordinate, four quarter chains in
// ascending k, combined as (s0 + s1) + (s2 + s3).  Kept out of the tile loop, whose code has to stay short.
template <typename T, int D>
__device__ __noinline__ void sum_again(const T* x0, const T* x1, const float* even, const float* odd, const CompressArgs* a,
                                       const float (*bounds)[16], const Again* list, int n, int j0, int lane) {
  constexpr int XPL = D / 32, KQ = D / 4, B = 8, STEP = D == 256 ? 32 : B;  // (STEP: from one register of the row)
  static_assert(KQ % STEP == 0, "whole batches");
  for (int m = 0; m < n; ++m) {
    const Again e = list[m];
    const int src = e.where & 1, j = j0 + 32 * (int)(e.where >> 1) + lane;
    const unsigned tok = e.row / (unsigned)a->num_heads, h = e.row - tok * (unsigned)a->num_heads;
    const T* x = (src ? x1 : x0) + token_offset(*a, src, tok) + (int64_t)h * a->head_stride[src];
    const float* pi = ((j & 1) ? odd : even) + (j >> 1);
    float xs[XPL], ss = 0.f;
#pragma unroll
    for (int i = 0; i < XPL; ++i) xs[i] = to_float<T>(x[lane + 32 * i]);
#pragma unroll
    for (int i = 0; i < XPL; ++i) ss = fmaf(xs[i], xs[i], ss);
    const float den = sqrtf(warp_sum(ss)) + 1e-10f;
#pragma unroll
    for (int i = 0; i < XPL; ++i) xs[i] = xs[i] / den;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int o = 0; o < KQ; o += STEP) {  // the four quarters side by side: 32 loads in flight
#pragma unroll 1
      for (int l = 0; l < STEP; l += B) {
        float p[4][B];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int c = 0; c < B; ++c) p[q][c] = __ldg(pi + (q * KQ + o + l + c) * (D / 2));
#pragma unroll
        for (int c = 0; c < B; ++c)
#pragma unroll
          for (int q = 0; q < 4; ++q)
            acc[q] = fmaf(__shfl_sync(0xffffffffu, xs[(q * KQ + o) / 32], (q * KQ + o) % 32 + l + c), p[q][c], acc[q]);
      }
    }
    const float t = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    uint32_t w = (uint32_t)bucketize_sorted16(t, bounds[src]) << (8 * ((lane & 7) >> 1) + ((lane & 1) ? 0 : 4));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) w |= __shfl_xor_sync(0xffffffffu, w, o);
    if ((lane & 7) == 0) reinterpret_cast<uint32_t*>(e.dst)[lane >> 3] = w;
  }
}

struct Bars {
  uint64_t full[4];    // TMA -> consumers: the stage's tile has landed
  uint64_t empty[4];   // consumers -> TMA: MMAs (1 commit) and the norm readers (4 warps) are done with it
  uint64_t tfull[4];   // MMA -> epilogue: the accumulator holds the tile's product
  uint64_t tempty[4];  // epilogue (4 warps) -> MMA: the accumulator has been read
  uint64_t drain;      // a dead CTA's last MMA is complete
};

// AGAIN: a coordinate near a boundary (Fmt<T>::kNear) is summed again
template <typename T, int D, bool AGAIN>
__global__ void __launch_bounds__(Cfg<D>::THREADS, 1)
compress_tc16_kernel(const __grid_constant__ CompressArgs a, const int group_rows, const __grid_constant__ CUtensorMap tm_x0,
                     const __grid_constant__ CUtensorMap tm_x1) {
  using F = Fmt<T>;
  using C = Cfg<D>;
  constexpr int N = C::N, STAGES = C::STAGES;
  constexpr bool kAgain = AGAIN;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) Bars s_bars;
  __shared__ uint32_t s_tmem;
  __shared__ int s_dead;
  __shared__ float s_bounds[2][16];
  __shared__ Again s_again[kAgain ? kAgainMax<D> * (C::THREADS / 32 - 2) : 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_trigger();
  if (warp == 0) CT_STAMP(0, 31, 6);  // kernel entry
  const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;  // swizzle atoms need 1024-byte alignment
  unsigned char* sm = smem_raw + (base - smem_addr(smem_raw));
  volatile int* dead = &s_dead;
  // which output coordinates, and which tiles: CTAs of the same tile stream are neighbours
  const int split = blockIdx.x % C::NSPLIT, stream = blockIdx.x / C::NSPLIT, n_streams = gridDim.x / C::NSPLIT;
  const int j0 = split * N;

  if (tid < 32) {
    const int src = tid >> 4, i = tid & 15;
    s_bounds[src][i] = (src < a.n_sources && i < a.n_bounds[src]) ? a.bounds[src][i] : CUDART_INF_F;
  }
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      bar_init(smem_addr(&s_bars.full[s]), 1);
      bar_init(smem_addr(&s_bars.empty[s]), 1 + 4);
      bar_init(smem_addr(&s_bars.tfull[s]), 1);
      bar_init(smem_addr(&s_bars.tempty[s]), 4);
    }
    bar_init(smem_addr(&s_bars.drain), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    s_dead = 0;
  }
  if (warp == 1) {  // the issuing warp owns the tensor-memory allocation
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                 "r"(C::kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // ---- Pi as the B operand: B[n][k] = Pi[j0 + n][k] in 16-bit terms, K-major, swizzled.  rot_even[k * D/2 + p]
  //      = Pi[2p][k], rot_odd[k * D/2 + p] = Pi[2p + 1][k]; columns past D (D = 96) are zero ---------------------
#pragma unroll 2
  for (int i = tid; i < N * C::KB * 8; i += C::THREADS) {
    const int n = i % N, k8 = i / N, j = j0 + n;  // row n, k = 8 * k8 .. + 7
    const float* src = ((j & 1) ? a.rot_odd : a.rot_even) + (j >> 1);
    float x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = 8 * k8 + e < D ? __ldg(src + (8 * k8 + e) * (D / 2)) * F::kScale : 0.f;
    uint16_t t[kMaxTerms][8];
#pragma unroll
    for (int e = 0; e < 8; ++e)
#pragma unroll
      for (int q = 0; q < F::kTerms; ++q) t[q][e] = F::term(x[e]);
    const uint32_t off = (uint32_t)(k8 >> 3) * C::kBBlock + swz(n, k8 & 7);
#pragma unroll
    for (int q = 0; q < F::kTerms; ++q) {
      uint4 v;
      v.x = t[q][0] | ((uint32_t)t[q][1] << 16);
      v.y = t[q][2] | ((uint32_t)t[q][3] << 16);
      v.z = t[q][4] | ((uint32_t)t[q][5] << 16);
      v.w = t[q][6] | ((uint32_t)t[q][7] << 16);
      *reinterpret_cast<uint4*>(sm + q * C::kTerm + off) = v;
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = s_tmem;
  if (warp == 0) CT_STAMP(0, 31, 7);  // set-up done (Pi converted, tensor memory allocated)

  const int64_t rows_per_src = a.n_tokens * a.num_heads;
  const int64_t tiles_per_src = (rows_per_src + kRows - 1) / kRows;
  const int64_t n_tiles = tiles_per_src * a.n_sources;
  const int64_t my_tiles = stream < n_tiles ? (n_tiles - stream + n_streams - 1) / n_streams : 0;
  bool ok = true;
  int64_t fetched = 0;  // (producer) tiles asked for

  if (warp == 0) {
    // ================= TMA producer =================
    for (int64_t i = 0; i < my_tiles && ok; ++i) {
      const int st = (int)(i % STAGES);
      const uint32_t par = (uint32_t)((i / STAGES) & 1);
      // (passes at once the first time round; warp-uniform so that the election below is well formed)
      ok = __all_sync(0xffffffffu, bar_wait_bounded(smem_addr(&s_bars.empty[st]), par ^ 1u, dead));
      if (!ok) break;
      CT_STAMP(0, i, 0);
      if (elect_one_sync()) {
        const int64_t tile = stream + i * n_streams;
        const int s_ = (int)(tile / tiles_per_src);
        const int y = (int)((tile - (int64_t)s_ * tiles_per_src) * kRows);
        const uint32_t bar = smem_addr(&s_bars.full[st]);
        const uint32_t dst = base + C::kOffA + st * C::kTile;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(C::kTile) : "memory");
        // rows past the end and columns past D are zero-filled
#pragma unroll
        for (int kb = 0; kb < C::KB; ++kb)
          tma_load_3d(dst + kb * kBlockBytes, s_ ? &tm_x1 : &tm_x0, 64 * kb, 0, y / group_rows, bar);
      }
      __syncwarp();
      fetched = i + 1;
    }
  } else if (warp == 1) {
    // ================= MMA issuer =================
    constexpr uint32_t idesc = instr_desc(F::kCode, N);
    for (int64_t i = 0; i < my_tiles && ok; ++i) {
      const int st = (int)(i % STAGES);
      const uint32_t par = (uint32_t)((i / STAGES) & 1);
      ok = __all_sync(0xffffffffu, bar_wait_bounded(smem_addr(&s_bars.full[st]), par, dead) &&
                                       bar_wait_bounded(smem_addr(&s_bars.tempty[st]), par ^ 1u, dead));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      CT_STAMP(1, i, 0);
      if (elect_one_sync()) {
        const uint32_t tmem_d = tmem_base + (uint32_t)st * N;
        const uint32_t a0 = base + C::kOffA + st * C::kTile;
#pragma unroll
        for (int q = F::kTerms - 1; q >= 0; --q) {  // smallest term first
#pragma unroll
          for (int s = 0; s < D / 16; ++s)  // k-steps of 16 columns (32 bytes)
            mma_f16(tmem_d, make_desc(a0 + (s >> 2) * kBlockBytes + 32u * (s & 3)),
                    make_desc(base + q * C::kTerm + (s >> 2) * C::kBBlock + 32u * (s & 3)), idesc,
                    (q != F::kTerms - 1 || s) ? 1u : 0u);
        }
        mma_commit(smem_addr(&s_bars.empty[st]));  // the tensor core has read the stage
        mma_commit(smem_addr(&s_bars.tfull[st]));  // the accumulator is complete
      }
      __syncwarp();
      CT_STAMP(1, i, 1);
    }
  } else {
    // ================= epilogue groups =================
    const int grp = (warp - 2) >> 2;              // tiles i with i % STAGES == grp, accumulator grp
    const int quarter = warp & 3;                 // the 32 TMEM lanes this warp may read
    const int row_in_tile = 32 * quarter + lane;
    const RowLayout lay = row_layout(a.num_heads, D);
    Grid grid[2];
    bool grid_ok = make_grid(s_bounds[0], grid[0], lane);
    grid_ok = make_grid(s_bounds[1], grid[1], lane) && grid_ok;
    [[maybe_unused]] Again* my_again = s_again + (kAgain ? kAgainMax<D> * (warp - 2) : 0);
    [[maybe_unused]] int n_again = 0;
    for (int64_t i = grp; i < my_tiles && ok; i += STAGES) {
      const int st = grp;
      const uint32_t par = (uint32_t)((i / STAGES) & 1);
      const int64_t tile = stream + i * n_streams;
      const int src = (int)(tile / tiles_per_src);
      const int64_t in_src = (tile - (int64_t)src * tiles_per_src) * kRows + row_in_tile;
      const bool live = in_src < rows_per_src;
      // where this row goes (resolved first: the load of its slot overlaps the waits)
      uint8_t* dst_idx = nullptr;
      float* dst_norm = nullptr;
      if (live) {
        const unsigned rem = (unsigned)in_src;
        const unsigned tok = rem / (unsigned)a.num_heads;
        const int h = (int)(rem - tok * (unsigned)a.num_heads);
        if (a.cache != nullptr) {
          const int64_t slot = (int64_t)tok < a.n_slots ? write_slot(a, tok) : -1;
          if (slot >= a.num_cache_slots) {
            if (a.err_flag) atomicOr(a.err_flag, TQ4_DEV_BAD_SLOT);
          } else if (slot >= 0) {
            uint8_t* rowp = a.cache + slot * a.cache_token_stride;
            dst_idx = rowp + (src == 0 ? lay.k_idx : lay.v_idx) + h * (D / 2) + j0 / 2;
            dst_norm = reinterpret_cast<float*>(rowp + (src == 0 ? lay.k_norm : lay.v_norm) + h * 4);
          }
        } else {
          const int64_t row = (int64_t)src * rows_per_src + in_src;
          dst_idx = a.packed_out + row * (D / 2) + j0 / 2;
          dst_norm = a.norms_out + row;
        }
      }
      ok = __all_sync(0xffffffffu, bar_wait_bounded(smem_addr(&s_bars.full[st]), par, dead));
      if (!ok) break;
      if (quarter == 0 && grp < 2) CT_STAMP(2 + grp, i, 0);
      // ---- norm, in the summation order of the FMA kernels: p[l] over k = l, l + 32, ..., then the butterfly
      //      tree 16, 8, 4, 2, 1 (pairs l, l + 1 in one instruction: each lane of it is an ordinary FMA) ------------
      float nrm = 0.f;
      {
        const unsigned char* xt = sm + C::kOffA + st * C::kTile;
        f2 p[16];
#pragma unroll
        for (int l = 0; l < 16; ++l) p[l] = 0ull;
#pragma unroll 1
        for (int q = 0; q < D / 32; ++q) {  // elements [32 q, 32 q + 32) of the row
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) {
            const int chunk = 4 * q + cc;
            const uint4 v = *reinterpret_cast<const uint4*>(xt + (chunk >> 3) * kBlockBytes + swz(row_in_tile, chunk & 7));
            f2 x[4];
            chunk_to_pairs<T>(v, x);
#pragma unroll
            for (int e = 0; e < 4; ++e) p[4 * cc + e] = fma2(x[e], x[e], p[4 * cc + e]);
          }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
          for (int l = 0; l < o; ++l) p[l] = add2(p[l], p[l + o]);
        float p0, p1;
        unpack2(p[0], p0, p1);
        nrm = sqrtf(p0 + p1);
      }
      __syncwarp();
      if (quarter == 0 && grp < 2) CT_STAMP(2 + grp, i, 1);
      if (lane == 0) bar_arrive(smem_addr(&s_bars.empty[st]));  // this warp is done with the staged rows
      // one IEEE division per row; Y_raw * (1 / den) is within an ulp of Y_raw / den
      const float scale = (1.f / (nrm + 1e-10f)) * (1.f / F::kScale);
      const bool wide = dst_idx != nullptr && ((uintptr_t)dst_idx & 15) == 0;  // else rows are 4-byte aligned
      const Grid g = src ? grid[1] : grid[0];

      ok = __all_sync(0xffffffffu, bar_wait_bounded(smem_addr(&s_bars.tfull[st]), par, dead));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (quarter == 0 && grp < 2) CT_STAMP(2 + grp, i, 2);
      // chunks of 32 coordinates -> 16 bytes each; the loop stays rolled so that its body fits the instruction cache
#pragma unroll 1
      for (int q = 0; q < N / 32; ++q) {
        uint32_t v[32];
        tmem_ld32(tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(st * N + 32 * q), v);
        uint32_t word[4];
        [[maybe_unused]] float closest = CUDART_INF_F;  // of the chunk's coordinates to their boundaries
        if (grid_ok) {
#pragma unroll
          for (int w = 0; w < 4; ++w) {  // 8 coordinates -> 4 bytes -> one word
            word[w] = 0;
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
              const float y0 = __uint_as_float(v[8 * w + e]) * scale, y1 = __uint_as_float(v[8 * w + e + 1]) * scale;
              int i0, i1;
              if constexpr (kAgain) {
                float d0, d1;
                i0 = bucketize_grid(y0, g, d0);
                i1 = bucketize_grid(y1, g, d1);
                closest = fminf(closest, fminf(fabsf(d0), fabsf(d1)));
              } else {
                i0 = bucketize_grid(y0, g);
                i1 = bucketize_grid(y1, g);
              }
              word[w] += ((uint32_t)i0 << (4 * e + 4)) + ((uint32_t)i1 << (4 * e));
            }
          }
        } else {
          float b[15];
#pragma unroll
          for (int bi = 0; bi < 15; ++bi) b[bi] = s_bounds[src][bi];
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            word[w] = 0;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float y = __uint_as_float(v[8 * w + e]) * scale;
              const int idx = bucketize_reg(y, b);
              if (kAgain && bucketize_reg(y - F::kNear, b) != bucketize_reg(y + F::kNear, b)) closest = 0.f;
              word[w] += (uint32_t)idx << (8 * (e >> 1) + ((e & 1) ? 0 : 4));
            }
          }
        }
        if (wide) {
          reinterpret_cast<uint4*>(dst_idx)[q] = make_uint4(word[0], word[1], word[2], word[3]);
        } else if (dst_idx) {
#pragma unroll
          for (int w = 0; w < 4; ++w) reinterpret_cast<uint32_t*>(dst_idx)[4 * q + w] = word[w];
        }
        if constexpr (kAgain) {
          // (a zero vector is zero either way)
          uint32_t who = __ballot_sync(0xffffffffu, closest < F::kNear && dst_idx != nullptr && nrm != 0.f);
#pragma unroll 1
          for (; who != 0; who &= who - 1) {
            if (n_again == kAgainMax<D>) {
              __syncwarp();
              sum_again<T, D>(reinterpret_cast<const T*>(a.x[0]), reinterpret_cast<const T*>(a.x[1]), a.rot_even, a.rot_odd, &a,
                              s_bounds, my_again, n_again, j0, lane);
              __syncwarp();
              n_again = 0;
            }
            if (lane == __ffs(who) - 1) my_again[n_again] = Again{dst_idx + 16 * q, (unsigned)in_src, 2u * q + src};
            ++n_again;
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(smem_addr(&s_bars.tempty[st]));  // the accumulator may be overwritten
      if (dst_norm && split == 0) *dst_norm = nrm;
      if (quarter == 0 && grp < 2) CT_STAMP(2 + grp, i, 3);
    }
    if constexpr (kAgain) {
      __syncwarp();
      sum_again<T, D>(reinterpret_cast<const T*>(a.x[0]), reinterpret_cast<const T*>(a.x[1]), a.rot_even, a.rot_odd, &a, s_bounds,
                      my_again, n_again, j0, lane);
    }
  }
  if (!ok) {
    s_dead = 1;
    if (lane == 0 && a.err_flag) atomicOr(a.err_flag, TQ4_DEV_TIMEOUT);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s_dead) {
    if (warp == 0) {
      for (int64_t i = fetched > STAGES ? fetched - STAGES : 0; i < fetched; ++i)
        bar_wait_bounded(smem_addr(&s_bars.full[i % STAGES]), (uint32_t)((i / STAGES) & 1), nullptr);
    } else if (warp == 1) {
      if (elect_one_sync()) {
        mma_commit(smem_addr(&s_bars.drain));
        bar_wait_bounded(smem_addr(&s_bars.drain), 0u, nullptr);
      }
      __syncwarp();
    }
  }
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::kTmemCols) : "memory");
  }
}

// One source as a 3-D tensor [groups][rows of a group][D] of 16-bit elements: a group is a token and its rows the heads
// when the heads divide a tile (any token and head stride), else one row of a dense array.  Box: 128 rows x 64 columns.
bool make_x_map(CUtensorMap* m, const CompressArgs& a, int src, int D, int group_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  const int64_t rows = a.n_tokens * a.num_heads;
  if (!fn || rows <= 0) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)group_rows, (cuuint64_t)(rows / group_rows)};
  const cuuint64_t strides[2] = {(cuuint64_t)(group_rows > 1 ? a.head_stride[src] : D) * 2,
                                 (cuuint64_t)(group_rows > 1 ? a.token_stride[src] : D) * 2};
  const cuuint32_t box[3] = {64, (cuuint32_t)group_rows, (cuuint32_t)(kRows / group_rows)};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void*>(a.x[src]), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// rows that a group of the input map has: the heads of a token, or 1 for a dense array of rows; 0: not covered
int group_of(const CompressArgs& a, int D) {
  bool dense = true;
  for (int s = 0; s < a.n_sources; ++s)
    dense = dense && a.head_stride[s] == D && a.token_stride[s] == (int64_t)a.num_heads * D;
  if (dense) return 1;
  if (a.num_heads > 1 && kRows % a.num_heads == 0) return a.num_heads;
  return 0;
}

template <typename T, int D, bool AGAIN>
int launch_t(const CompressArgs& a, cudaStream_t st) {
  using C = Cfg<D>;
  CUtensorMap m0, m1;
  memset(&m0, 0, sizeof(m0));
  memset(&m1, 0, sizeof(m1));
  const int group = group_of(a, D);
  if (!make_x_map(&m0, a, 0, D, group) || !make_x_map(&m1, a, a.n_sources > 1 ? 1 : 0, D, group)) return TQ4_ERR_CUDA;
  const int smem = (int)C::kSmem + 1024;
  if (!ensure_dynamic_smem<compress_tc16_kernel<T, D, AGAIN>>(smem)) return TQ4_ERR_CUDA;
  int64_t streams = ((a.n_tokens * a.num_heads + kRows - 1) / kRows) * a.n_sources;
  if (streams > sm_count() / C::NSPLIT) streams = sm_count() / C::NSPLIT;
  compress_tc16_kernel<T, D, AGAIN><<<(unsigned)(streams * C::NSPLIT), C::THREADS, smem, st>>>(a, group, m0, m1);
  TQ4_CHECK_LAUNCH();
  return TQ4_OK;
}

template <typename T>
int launch_d(const CompressArgs& a, int head_dim, bool fma_bytes, cudaStream_t st) {
  switch (head_dim) {
    case 64: return launch_t<T, 64, true>(a, st);
    case 96: return launch_t<T, 96, true>(a, st);
    case 128: return fma_bytes ? launch_t<T, 128, true>(a, st) : launch_t<T, 128, false>(a, st);
    case 256: return launch_t<T, 256, true>(a, st);
  }
  return TQ4_ERR_UNSUPPORTED;
}

}  // namespace

// 16-bit inputs whose rows TMA can address: dense arrays, or strided tokens and heads (K and V as views of one
// projection) when the heads divide a tile.  Everything else stays on the kernels in tq4_compress_tc.cu / tq4_compress.cu.
bool compress_tc16_eligible(const CompressArgs& a, int head_dim, int dtype) {
  static const bool disabled = getenv("TQ4_NO_TC") != nullptr || getenv("TQ4_NO_TC16") != nullptr;
  if (disabled || !supported_head_dim(head_dim) || (dtype != TQ4_F16 && dtype != TQ4_BF16)) return false;
  if (a.n_tokens * a.num_heads >= (1ll << 31) || encode_tiled_fn() == nullptr || !tokens_uniform(a)) return false;
  for (int s = 0; s < a.n_sources; ++s)
    if (((uintptr_t)a.x[s] & 15) || a.head_stride[s] <= 0 || a.token_stride[s] <= 0 || a.head_stride[s] % 8 || a.token_stride[s] % 8)
      return false;
  return group_of(a, head_dim) != 0;
}

int launch_compress_tc16(const CompressArgs& a, int head_dim, int dtype, bool fma_bytes, cudaStream_t st) {
  return dtype == TQ4_F16 ? launch_d<__half>(a, head_dim, fma_bytes, st) : launch_d<__nv_bfloat16>(a, head_dim, fma_bytes, st);
}

}  // namespace tq4

#ifdef TQ4_TRACE
extern "C" int tq4_compress_trace_read(long long* out) {
  return cudaMemcpyFromSymbol(out, tq4::g_ctrace, sizeof(long long) * 4 * 32 * 8) == cudaSuccess ? 0 : 1;
}
#endif
