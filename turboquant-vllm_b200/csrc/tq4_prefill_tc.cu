// Chunked-prefill attention over the packed TQ4 cache on the 5th-generation tensor cores, head_dim 64 to
// 256.  A CTA owns one KV head and one or two blocks of 128 / G query rows of a sequence: the M = 128
// rows of the MMAs are the (query row, query head of the GQA group) pairs, so a key/value tile is
// dequantised ONCE per CTA and serves all of them (the streaming kernel dequantises it per query row).
//
// Phases of a CTA:
//   1. rotate the block's queries: raw rows, scaled by a power of two, as fp16 hi (+ lo) in tensor memory
//      times Pi (2^8 Pi as fp16 hi + lo, an operand image in shared memory)         tcgen05.mma
//   2. per 64-token tile
//        packed bytes and norms, prefetched into registers a tile ahead             global loads
//        byte -> half2 table lookups, K~ and V~ into the swizzled operand layouts   dequantising warps
//        S = Qhi K~^T + Qlo K~^T                        (fp32 in tensor memory)     tcgen05.mma
//        x knorm, mask, lazy online softmax, P = p * vnorm as fp16 hi + lo          softmax warps
//        O += Plo V~ + Phi V~                                                       tcgen05.mma
//   3. un-rotate: O / l as fp16 hi + lo times the same image of Pi (read as the other operand major), and
//      store the caller's output.  Nothing but queries, cache and outputs touches global memory.
//
// Why this shape: a tile costs the tensor pipe 2 x 528 cycles per 128 rows (head_dim 128, two terms), the
// softmax about 2 000 cycles of latency-bound CUDA-core work (a thread per row, 64 columns) and the dequantisation
// about 700 + 700 of shared-memory traffic.  Two score buffers a block, sixteen softmax warps, or rows dealt over quads of lanes
// (fewer reads of norms) were each no faster: issue, shared memory and tensor memory are all half busy, and what one of
// these saves the next one takes.  With one row block per CTA these formed one chain of 3 550 cycles a
// tile; with two blocks the tensor pipe works on one while the other is in its softmax, and a dequantised tile
// serves 256 rows: 3 600 cycles for twice the rows, 58 % of them tensor work, which at 8 x 2048 rows on 8192 cached
// tokens (32 / 8 heads) runs into the 1000 W limit.  What bounds it: the chain scores -> softmax -> P -> O and next
// scores of a block (2 150 + 1 450).  Everything meets at mbarriers only: softmax warps (a thread per row; two at
// head_dim 256), eight dequantising warps and one issuing thread.
//   Code that runs once per CTA pays for its instruction fetches (the first version, unrolled, needed 62 000 cycles
//   before its second tile): set-up, rotation, masks and the new-reference path are short loops, a row's largest
//   coordinate is found on its packed bits, the rotated row is split without looking for one, and the outputs leave a row a
//   half-warp.  20 700 -> 15 800 cycles before the loop and 15 600 -> 13 200 after it; with the row factor inside the queries' terms
//   and 16 columns of P a store: 8 x 2048 rows on 8192 (32 / 8 heads) 4815 -> 4690 us, 1531 rows of 28 / 4 heads with their write
//   91 -> 81, 8 x 2048 of 8 / 4 heads of 256 in a window of 4096 1285 -> 1203 (there 5 % by one table for K and V).
//   Tensor memory, per block: [S | P in place][Q hi][Q lo][O]: 64 + 64 + 128 columns at head_dim 128, where
//   Q lo does not fit and sits in shared memory; at head_dim 256 there is one block of 448 columns and the 64 left
//   hold a second S, so that the scores of the next tile are computed during the softmax of this one.
//   P overwrites S in place: the columns of tokens 16 c .. + 15 become P hi and P lo of those tokens.
//
// A block with few CTAs is cut along the keys (gridDim.z): each part leaves its normalised rotated rows and
// their log-sum-exp in the scratch, and the merge kernel folds and un-rotates them.
// Every wait is bounded; a wait that gives up marks the CTA dead, all roles drain, TQ4_DEV_TIMEOUT is raised.  On
// every way out, the empty key parts' and the dead CTA's among them, a CTA first waits for the copies and MMAs it
// issued: they work on its shared and tensor memory, which the next CTA of the SM is given.
#include <math_constants.h>

#include <cstdlib>
#include <type_traits>

#include "tq4_attention.cuh"

namespace tq4 {
#ifdef TQ4_TRACE
// Tuning builds only (-DTQ4_TRACE): the SM clock at points of the tile loop for four warps of one CTA, read
// back with tq4_prefill_trace_read.  Compiled out of the shipped library.
__device__ long long g_ptrace[4][64][8];
#define PF_STAMP(role, j, e)                                                                            \
  do {                                                                                                  \
    if (blockIdx.x == gridDim.x / 2 && blockIdx.z == 0 && (role) >= 0 && (j) < 64)   \
      g_ptrace[(role) & 3][j][e] = clock64();                                                           \
  } while (0)
#else
#define PF_STAMP(role, j, e) do {} while (0)
#endif
namespace {

constexpr int kBN = 64;         // tokens per tile
constexpr int kSmx = 256;       // warps 0-7: softmax, prologue and epilogue of the rows
constexpr int kDeq = 256;       // warps 8-15: dequantisation
constexpr int kThreads = kSmx + kDeq + 32;
constexpr int kIssueWarp = (kSmx + kDeq) / 32;
constexpr int kNormBufs = 4;
constexpr float kHidden = 1e-33f;  // key norm in shared memory of a token whose page id is out of range
constexpr float kQGain = 64.f;     // factor of the queries' terms, its inverse in the key norms: keeps the lo terms normal numbers

template <int D>
struct Cfg {
  static constexpr int NBLK = D == 256 ? 1 : 2;            // row blocks per CTA
  static constexpr int TPR = D == 256 ? 2 : 1;             // softmax threads per row
  static constexpr int CPT = kBN / TPR;                    // score columns per softmax thread
  static constexpr int DPT = D / TPR;                      // coordinates per softmax thread
  static constexpr int NC = (D + 63) / 64;                 // 64-coordinate blocks of a row
  static constexpr int NS = D / 32;                        // 16-byte segments of a packed row
  static constexpr int NKB = 2, NVB = D == 256 ? 1 : 2;    // K~ and V~ buffers
  static constexpr int NIT = (kBN * NS + kDeq - 1) / kDeq;  // segments per dequantising thread
  static constexpr bool QLO_SMEM = D >= 128;               // Q lo in shared memory
  // tensor-memory columns of a block (two S at head_dim 256)
  static constexpr uint32_t kNS = D == 256 ? 2 : 1;
  static constexpr uint32_t kColS = 0, kColQ = 64 * kNS, kColQlo = kColQ + D / 2;
  static constexpr uint32_t kColO = kColQ + (QLO_SMEM ? D / 2 : D);
  static constexpr uint32_t kBlkCols = kColO + D;
  static_assert(NBLK * kBlkCols <= 512, "tensor memory");
  // shared memory, from a 1024-byte boundary
  static constexpr uint32_t kKvBuf = NC * kBN * 128;       // one K~ or V~ buffer
  static constexpr uint32_t kImgPart = (D == 256 ? 64 : D) * 128;  // a column block of one chunk of Pi's image
  static constexpr int kChunks = D == 256 ? 4 : 1;         // chunks of 64 (D = 256) or all of the output coordinates
  static constexpr uint32_t kOffK = 0;
  static constexpr uint32_t kOffV = kOffK + NKB * kKvBuf;
  static constexpr uint32_t kKvEnd = kOffV + NVB * kKvBuf;
  static constexpr uint32_t kImg = 2 * NC * kImgPart;      // the image (chunk) shares the K~ / V~ buffers
  static constexpr uint32_t kOffQlo = kKvEnd > kImg ? kKvEnd : kImg;
  // raw 16-bit query rows on their way in, padded against bank conflicts (the area of Q lo, which is written later)
  static constexpr uint32_t kQPitch = 2 * D + 16;
  static constexpr uint32_t kQStage = NBLK * 128 * kQPitch, kQlo = QLO_SMEM ? NBLK * NC * 128 * 128 : 0;
  static constexpr uint32_t kOffLut = kOffQlo + (((kQStage > kQlo ? kQStage : kQlo) + 1023) & ~1023u);
  // lane copies of a table entry.  (16: room for no more of two tables; every lookup is then a two-way conflict.  K and V of one
  // codebook share a table of 32.)
  static constexpr int kLutCopies = D == 256 ? 16 : 32;
  static constexpr uint32_t kOffNorm = kOffLut + 2 * 256 * kLutCopies * 4;
  static constexpr uint32_t kOffXchg = kOffNorm + kNormBufs * 2 * kBN * 4;
  static constexpr uint32_t kSmem = kOffXchg + (TPR == 2 ? 2 * 2 * 128 * 4 : 0);
  // registers a thread: together the 2 x 96 that the two groups of eight warps are launched with
  static constexpr int kDeqRegs = D == 256 ? 72 : 56, kSmxRegs = 192 - kDeqRegs;
  __host__ __device__ static constexpr uint32_t idesc(uint32_t n, bool b_mn) {  // kind::f16: fp16 operands, fp32 accumulator, M = 128
    return (1u << 4) | (b_mn ? 1u << 16 : 0u) | ((n >> 3) << 17) | ((128u >> 4) << 24);
  }
};

struct PrefillArgs {
  const uint8_t* image;  // Pi's operand image (pi_image_kernel)
  int min_rows;          // sequences with fewer new rows are left to the streaming kernel
  int splits;            // parts of the key range
  int to_parts;          // leave partials for the merge kernel instead of writing the output
  float* part_o;         // [splits][rows][Hq][D] normalised, rotated
  float* part_m;         // [splits][rows][Hq] natural-log LSE
  bool heads_first = false;  // blockIdx.x: KV heads fastest, else row blocks (launch_t)
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16-byte chunk c of row `row` inside a [rows][128 B] block, 128-byte swizzle
__device__ __forceinline__ uint32_t swz(int row, int c) { return (uint32_t)(row * 128 + ((c ^ (row & 7)) << 4)); }
// operand descriptor, 128-byte swizzle, 8-row groups 1024 bytes apart; `lbo`: distance of the 64-element blocks
// of an MN-major operand (K-major: unused)
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo ? lbo >> 4 : 1) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// D (tensor memory) (+)= A * B, A (128 rows x 16 fp16 = 8 columns) from tensor memory
__device__ __forceinline__ void mma_ta(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u), "r"(0u)
      : "memory");
}
// the same with A from shared memory
__device__ __forceinline__ void mma_sa(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u), "r"(0u)
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
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// Bounded wait for another role: also gives up as soon as the CTA is marked dead; marks it itself otherwise.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile int* dead) {
  for (int it = 0; it < (1 << 22); ++it) {
    if (bar_try(bar, parity)) return true;
    if ((it & 1023) == 1023 && *dead) return false;
  }
  *dead = 1;
  return false;
}
// Bounded wait for copies or MMAs in flight, which no other role can hold up: a dead CTA sees them home, too.
__device__ __forceinline__ bool bar_wait_own(uint32_t bar, uint32_t parity, volatile int* dead) {
  for (int it = 0; it < (1 << 22); ++it)
    if (bar_try(bar, parity)) return true;
  *dead = 1;
  return false;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
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
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 32 consecutive 32-bit columns of this thread's tensor-memory lane (with the wait)
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
// 16 columns, without the wait; tmem_ld16_wait names the registers so that no use of them moves above it.  (No
// memory clobber on these: the compiler may move shared-memory loads across them.)
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
      "%14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld16_wait(uint32_t (&v)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                 "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]));
}
// all 32 or 64 columns of a score tile, with the wait
template <int N>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&v)[N]) {
#pragma unroll
  for (int h = 0; h < N / 16; ++h) tmem_ld16_async(taddr + 16 * h, *reinterpret_cast<uint32_t(*)[16]>(v + 16 * h));
#pragma unroll
  for (int h = 0; h < N / 16; ++h) tmem_ld16_wait(*reinterpret_cast<uint32_t(*)[16]>(v + 16 * h));
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {  // (no wait)
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {  // (no wait)
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]));
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float lg2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
// pairs of fp32 values in one 64-bit register: one instruction does both
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
// two values -> fp16 hi pair and fp16 pair of what the rounding left
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x0, x1);
  const float2 f = __half22float2(h);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = pack_h2(x0 - f.x, x1 - f.y);
}
// power of two that brings a value into [1, 2), and its inverse
__device__ __forceinline__ void pow2_scale(float amax, float& sc, float& isc) {
  sc = isc = 1.f;
  if (amax > 0.f && amax < CUDART_INF_F) {
    const int e = min(max((int)((__float_as_uint(amax) >> 23) & 0xFFu) - 127, -100), 100);
    sc = __uint_as_float((uint32_t)(127 - e) << 23);
    isc = __uint_as_float((uint32_t)(127 + e) << 23);
  }
}

// two packed 16-bit values
__device__ __forceinline__ void half_pair(uint32_t w, bool f16, float& x0, float& x1) {
  if (f16) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    x0 = f.x; x1 = f.y;
  } else {
    x0 = __uint_as_float(w << 16); x1 = __uint_as_float(w & 0xFFFF0000u);
  }
}

// 32 consecutive elements i .. i + 31 of a typed tensor
__device__ __forceinline__ void load32(const void* q, int dtype, int64_t i, bool vec_ok, float (&x)[32]) {
  if (!vec_ok) {
#pragma unroll
    for (int e = 0; e < 32; ++e) x[e] = load_as_float(q, dtype, i + e);
    return;
  }
  if (dtype == TQ4_F32) {
    const float4* p = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(q) + i);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float4 v = __ldg(p + e);
      x[4 * e] = v.x; x[4 * e + 1] = v.y; x[4 * e + 2] = v.z; x[4 * e + 3] = v.w;
    }
    return;
  }
  const uint4* p = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(q) + i);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const uint4 v = __ldg(p + e);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (dtype == TQ4_F16) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[k]));
        x[8 * e + 2 * k] = f.x; x[8 * e + 2 * k + 1] = f.y;
      } else {
        x[8 * e + 2 * k] = __uint_as_float(w[k] << 16);
        x[8 * e + 2 * k + 1] = __uint_as_float(w[k] & 0xFFFF0000u);
      }
    }
  }
}

// 32 consecutive outputs
__device__ __forceinline__ void store32(void* p, int dtype, int64_t i, bool vec_ok, const float (&y)[32]) {
  if (dtype != TQ4_F32 && vec_ok) {
    uint4* d = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p) + i);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (dtype == TQ4_F16) {
          w[k] = pack_h2(y[8 * q + 2 * k], y[8 * q + 2 * k + 1]);
        } else {
          const __nv_bfloat162 h = __floats2bfloat162_rn(y[8 * q + 2 * k], y[8 * q + 2 * k + 1]);
          w[k] = *reinterpret_cast<const uint32_t*>(&h);
        }
      }
      d[q] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    return;
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const float t[4] = {y[4 * q], y[4 * q + 1], y[4 * q + 2], y[4 * q + 3]};
    store4(p, dtype, i + 4 * q, t);
  }
}

// Pi's operand image: [term: fp16 hi, lo of 2^8 Pi][64-column block][row of Pi][128 B, swizzled].  As a K-major
// operand its rows are output coordinates (rotation), as an MN-major one they are input coordinates
// (un-rotation).  Columns past head_dim (D = 96) are zero.
template <int D>
__global__ void __launch_bounds__(256) pi_image_kernel(const float* __restrict__ rotation, uint8_t* __restrict__ image) {
  constexpr int NC = (D + 63) / 64;
  pdl_trigger();
  const int i = (int)(blockIdx.x * 256 + threadIdx.x);  // (row, 8-column chunk)
  if (i >= D * NC * 8) return;
  const int r = i / (NC * 8), k8 = i - r * (NC * 8), c = k8 >> 3;
  uint32_t hi[4], lo[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int col = 8 * k8 + 2 * e;
    const float x0 = col < D ? 256.f * __ldg(rotation + (size_t)r * D + col) : 0.f;
    const float x1 = col < D ? 256.f * __ldg(rotation + (size_t)r * D + col + 1) : 0.f;
    split2(x0, x1, hi[e], lo[e]);
  }
  uint8_t* dst = image + (size_t)c * D * 128 + swz(r, k8 & 7);
  *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  *reinterpret_cast<uint4*>(dst + (size_t)NC * D * 128) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}

struct Bars {
  uint64_t kready[2], vready[2];  // dequantising warps -> issuer: K~ / V~ buffer written
  uint64_t kfree[2], vfree[2];    // MMAs -> dequantising warps: buffer read
  uint64_t sready[2];             // MMAs -> softmax: scores of the block (head_dim 256: of the tile's S buffer) complete
  uint64_t pready[2];             // softmax warps -> issuer: P written
  uint64_t pvd;                   // MMAs -> softmax: O updated (head_dim 256; elsewhere sready implies it)
  uint64_t img, cdone;            // image chunk landed / used
  uint64_t aready, rot;           // A operand of a rotation staged / rotation complete
  uint64_t pair[4];               // the two warps of a row quadrant (head_dim 256)
  uint64_t qraw;                  // raw query rows landed
  uint64_t qready, odone;         // queries in place / last MMA of the tile loop complete
  uint64_t drain;                 // a dead CTA's last MMA complete
};

template <int D, bool FAST>
__global__ void __launch_bounds__(kThreads, 1) prefill_tc_kernel(const AttnArgs a, const PrefillArgs pa) {
  using C = Cfg<D>;
  constexpr int NBLK = C::NBLK, TPR = C::TPR, CPT = C::CPT, DPT = C::DPT, NC = C::NC, NKB = C::NKB, NVB = C::NVB, NIT = C::NIT;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) Bars s_bars;
  __shared__ uint32_t s_tmem;
  __shared__ int s_info[5];      // sequence, first row and rows of the CTA; end of the sequence's rows and its length
  __shared__ float s_cent[2][16];  // scaled centroids of K and V
  __shared__ int s_dead, s_bad;  // a wait gave up / some page id is out of range
  const AttnShape& sh = a.sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int inner = pa.heads_first ? sh.Hkv : (int)gridDim.x / sh.Hkv, outer = (int)blockIdx.x / inner, rest = (int)blockIdx.x - outer * inner;
  const int rowblk = pa.heads_first ? outer : rest, kvh = pa.heads_first ? rest : outer, G = sh.G, RB = 128 / G;
  volatile int* dead = &s_dead;
  auto bar = [](const uint64_t& b) { return smem_addr(&b); };
  const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
  unsigned char* sm = smem_raw + (base - smem_addr(smem_raw));

  PF_STAMP(tid == 0 ? 0 : -1, 0, 4);
  // ---- which rows are this CTA's?  Sequences in order, a sequence's last rows (the longest) first --------
  if (warp == 0) {
    int acc = 0, found = -1, first = 0, nrows = 0;
    for (int s0 = 0; s0 < sh.num_seqs && found < 0; s0 += 32) {
      const int s = s0 + lane;
      int q0 = 0, q1 = 0, q_end = 0, seq_len = 0;
      if (s < sh.num_seqs) {
        q0 = max(__ldg(a.query_start_loc + s), 0);
        q_end = __ldg(a.query_start_loc + s + 1);
        seq_len = __ldg(a.seq_lens + s);
        q1 = min(q_end, sh.rows);
      }
      const int n = q1 - q0 >= max(pa.min_rows, 1) ? (q1 - q0 + NBLK * RB - 1) / (NBLK * RB) : 0;
      int incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      const int x = rowblk - acc;
      const unsigned m = __ballot_sync(0xffffffffu, x < incl);
      if (m) {
        const int w = __ffs(m) - 1;
        const int b = n - 1 - (x - (incl - n));  // (lane w: its block, counted from the end)
        found = s0 + w;
        first = __shfl_sync(0xffffffffu, q0 + b * NBLK * RB, w);
        nrows = __shfl_sync(0xffffffffu, min(NBLK * RB, q1 - (q0 + b * NBLK * RB)), w);
        if (lane == w) {
          s_info[3] = q_end;
          s_info[4] = seq_len;
        }
      }
      acc += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) {
      s_info[0] = found;
      s_info[1] = found < 0 ? rowblk - acc : first;  // (without rows: which of the spare CTAs, and how many)
      s_info[2] = found < 0 ? (int)gridDim.x / sh.Hkv - acc : nrows;
      s_dead = 0;
      s_bad = 0;
    }
  }
  if (warp == 1) {
    const int w = lane >> 4, i = lane & 15;
    const float* cent = w ? a.v_centroids : a.k_centroids;
    s_cent[w][i] = i < (w ? a.n_v_centroids : a.n_k_centroids) ? __fmul_rn(w ? a.lut_scale_v : a.lut_scale_k, __ldg(cent + i)) : 0.f;
  }
  if (tid == 64) {
    for (int i = 0; i < 2; ++i) {
      bar_init(bar(s_bars.kready[i]), kDeq / 32);
      bar_init(bar(s_bars.vready[i]), kDeq / 32);
      bar_init(bar(s_bars.kfree[i]), 1);
      bar_init(bar(s_bars.vfree[i]), 1);
      bar_init(bar(s_bars.sready[i]), 1);
      bar_init(bar(s_bars.pready[i]), NBLK == 2 ? 4 : 8);
    }
    for (int i = 0; i < 4; ++i) bar_init(bar(s_bars.pair[i]), 2);
    bar_init(bar(s_bars.pvd), 1);
    bar_init(bar(s_bars.img), 1);
    bar_init(bar(s_bars.cdone), 1);
    bar_init(bar(s_bars.aready), 8);
    bar_init(bar(s_bars.rot), 1);
    bar_init(bar(s_bars.qraw), kSmx);
    bar_init(bar(s_bars.qready), 8);
    bar_init(bar(s_bars.odone), 1);
    bar_init(bar(s_bars.drain), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async();
  }
  __syncthreads();
  const int seq = s_info[0], row0 = s_info[1], nrows = s_info[2];
  if (seq < 0) {  // the grid is an upper bound: ceil(rows / per CTA) + sequences, so at least one CTA is spare
    pdl_trigger();
    pdl_wait();
    // Rows past the last offset belong to no sequence and see no key: zeros, as the streaming kernel writes.  (In a
    // call of both kernels they are the streaming kernel's.)
    const int tail = min(max(a.query_start_loc[sh.num_seqs], 0), sh.rows);
    if (pa.min_rows <= 1) {
      const float zero[4] = {0.f, 0.f, 0.f, 0.f};
      for (int r = tail + row0; r < sh.rows; r += nrows) {
        for (int i = tid; i < G * (D / 4); i += kThreads) {
          const int h = kvh * G + i / (D / 4), d = 4 * (i % (D / 4));
          if (!pa.to_parts)
            store4(a.out, a.out_dtype, (int64_t)r * a.out_token_stride + (int64_t)h * a.out_head_stride + d, zero);
          if (d > 0) continue;
          if (pa.to_parts) pa.part_m[((int64_t)blockIdx.z * sh.rows + r) * sh.Hq + h] = -CUDART_INF_F;
          else if (a.lse_out) a.lse_out[(int64_t)r * sh.Hq + h] = -CUDART_INF_F;
        }
      }
    }
    return;
  }
  // ---- row of a softmax thread (half a row at head_dim 256), and its raw query on the way -------------------
  const int blk = NBLK == 2 ? (warp >> 2) & 1 : 0, part = NBLK == 2 ? 0 : (warp >> 2) & 1;
  const int m = 32 * (warp & 3) + lane, my_r = m / G, my_g = m - my_r * G;
  const int lrow = blk * RB + my_r;                       // row within the CTA
  const bool live = warp < kSmx / 32 && my_r < RB && lrow < nrows;
  const int head = kvh * G + my_g, row = row0 + (live ? lrow : 0);
  const int es = a.q_dtype == TQ4_F32 ? 4 : 2;
  const bool q_vec = ((uintptr_t)a.q % 16 == 0) && (a.q_token_stride * es) % 16 == 0 && (a.q_head_stride * es) % 16 == 0;
  const bool q_staged = q_vec && es == 2;
  const int64_t qi = (int64_t)row * a.q_token_stride + (int64_t)head * a.q_head_stride + part * DPT;
  const uint32_t q_at = C::kOffQlo + (blk * 128 + m) * C::kQPitch + part * DPT * 2;
  if (q_staged && warp < kSmx / 32) {
    if (live) {
      expect_tx(bar(s_bars.qraw), DPT * 2);
      bulk_load(base + q_at, reinterpret_cast<const uint16_t*>(a.q) + qi, DPT * 2, bar(s_bars.qraw));
    } else {
      bar_arrive(bar(s_bars.qraw));
    }
  }
  if (warp == kIssueWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  bool one_table = C::kLutCopies == 16;
  if (one_table)
    for (int i = 0; i < 16; ++i) one_table = one_table && s_cent[0][i] == s_cent[1][i];
  // byte -> half2 tables: (centroid[hi nibble], centroid[lo nibble]) scaled onto the fp16 grid, one copy per lane
  {
    uint4* lut = reinterpret_cast<uint4*>(sm + C::kOffLut);
#pragma unroll 4
    for (int i = tid; i < 512 * C::kLutCopies / 4; i += kThreads) {
      const int e = one_table ? i / 8 : i / (C::kLutCopies / 4), w = e >> 8, b = e & 255;
      const uint32_t v = pack_h2(s_cent[w][b >> 4], s_cent[w][b & 15]);
      lut[i] = make_uint4(v, v, v, v);
    }
  }
  pdl_trigger();
  pdl_wait();  // the operand image of Pi; everything else was complete before the kernel in front started
  fence_before();
  __syncthreads();  // tensor-memory address and tables in place
  fence_after();
  const uint32_t tmem = s_tmem;

  PF_STAMP(tid == 0 ? 0 : -1, 0, 5);
  // ---- keys the CTA needs: rows are in query order, their visible ranges move forward with them -----------
  const int q_end = s_info[3], len = clamp_seq_len(a, max(0, s_info[4]));
  auto row_keys = [&](int row, int& lo, int& hi) {  // visible keys of row `row` of the call
    const int pos = len - (q_end - row);
    hi = max(0, min(a.causal ? pos + 1 : len, len));
    lo = min(a.sliding_window > 0 ? max(0, pos + 1 - a.sliding_window) : 0, hi);
  };
  int blk_lo, blk_hi, t_first = 0, n_tiles = 0;
  {
    int x;
    row_keys(row0, blk_lo, x);
    row_keys(row0 + nrows - 1, x, blk_hi);
    if (blk_hi > blk_lo) {
      t_first = blk_lo / kBN * kBN;
      n_tiles = (blk_hi - t_first + kBN - 1) / kBN;
      const int per = (n_tiles + pa.splits - 1) / pa.splits;  // this part of the key range
      t_first += (int)blockIdx.z * per * kBN;
      n_tiles = max(0, min(per, n_tiles - (int)blockIdx.z * per));
    }
  }
  const int n_blk = nrows > RB ? NBLK : 1;  // row blocks in use

  if (warp == kIssueWarp) {
    // ================= issuing thread =================
    if (n_tiles > 0 && elect_one_sync()) {
      // where a chunk's hi and lo terms go: the K~ / V~ buffers before the tile loop; after it the tables (head_dim
      // 256: the K~ buffer and the tables), which are free before the last values have been multiplied
      const uint32_t img = base + C::kOffK;
      const uint32_t uhi = base + (D == 256 ? C::kOffK : C::kOffLut), ulo = D == 256 ? base + C::kOffLut : uhi + C::kImg / 2;
      uint32_t img_ph = 0, img_n = 0, c_ph = 0;  // image chunks waited for / asked for
      bool ok = true;
      const bool unrotate = !pa.to_parts && !a.out_rotated;
      // chunk ch of the image, as rows (rotation) or as column blocks (un-rotation)
      auto load_chunk = [&](int ch, bool unrot) {
        ++img_n;
        expect_tx(bar(s_bars.img), C::kImg);
        if (C::kChunks == 1) {
          bulk_load(unrot ? uhi : img, pa.image, C::kImg, bar(s_bars.img));
        } else if (unrot) {
          bulk_load(uhi, pa.image + (size_t)ch * D * 128, D * 128, bar(s_bars.img));
          bulk_load(ulo, pa.image + (size_t)(NC + ch) * D * 128, D * 128, bar(s_bars.img));
        } else {
          for (int t = 0; t < 2 * NC; ++t)
            bulk_load(img + t * C::kImgPart, pa.image + (size_t)t * D * 128 + ch * 64 * 128, C::kImgPart, bar(s_bars.img));
        }
      };
      // O = A * B for the blocks in use: A = fp16 hi (and lo) terms at the S and Q columns, B = the image
      auto rotate = [&](bool unrot, bool a_lo) {
        for (int ch = 0; ch < C::kChunks && ok; ++ch) {
          ok = bar_wait_own(bar(s_bars.img), img_ph & 1, dead);
          ++img_ph;
          if (ch == 0) {
            ok = bar_wait(bar(s_bars.aready), unrot ? 1u : 0u, dead) && ok;
            fence_after();
          }
          if (!ok) return;
          constexpr uint32_t N = C::kChunks == 1 ? D : 64;
          const uint32_t idesc = C::idesc(N, unrot);
          const uint32_t hi = unrot ? uhi : img, lo = unrot ? ulo : img + C::kImg / 2;
          for (int b = 0; b < n_blk; ++b) {
            const uint32_t tb = tmem + b * C::kBlkCols, d = tb + C::kColO + 64 * ch;
#pragma unroll 1
            for (int s = 0; s < D / 16; ++s) {
              const uint32_t off = unrot ? 2048u * s : (s >> 2) * C::kImgPart + 32u * (s & 3);
              const uint64_t bh = make_desc(hi + off, unrot ? C::kImgPart : 0), bl = make_desc(lo + off, unrot ? C::kImgPart : 0);
              mma_ta(d, tb + C::kColS + 8 * s, bl, idesc, s > 0);
              if (a_lo) mma_ta(d, tb + C::kColQ + 8 * s, bh, idesc, true);
              mma_ta(d, tb + C::kColS + 8 * s, bh, idesc, true);
            }
          }
          if (ch + 1 < C::kChunks) {
            mma_commit(bar(s_bars.cdone));
            ok = bar_wait(bar(s_bars.cdone), c_ph & 1, dead);
            ++c_ph;
            if (ok) load_chunk(ch + 1, unrot);
          }
        }
        if (ok) mma_commit(bar(s_bars.rot));
      };
      load_chunk(0, false);
      rotate(false, a.q_dtype == TQ4_F32);

      const uint64_t d_k = make_desc(base + C::kOffK, 0), d_v = make_desc(base + C::kOffV, kBN * 128);
      const uint64_t d_qlo = make_desc(base + C::kOffQlo, 0);
      constexpr uint32_t idS = C::idesc(kBN, false), idO = C::idesc(D, true);
      auto issue_s = [&](int b, int j) {  // S = Q K~^T of tile j
        const uint32_t tb = tmem + b * C::kBlkCols, d = tb + C::kColS + (NBLK == 1 ? 64 * (j & 1) : 0);
        const uint64_t dk = d_k + (uint64_t)(((j % NKB) * C::kKvBuf) >> 4);
#pragma unroll
        for (int s = 0; s < D / 16; ++s) {
          const uint64_t db = dk + (uint64_t)(((s >> 2) * (kBN * 128) + 32 * (s & 3)) >> 4);
          if (!FAST) {
            if (C::QLO_SMEM)
              mma_sa(d, d_qlo + (uint64_t)((b * NC * 16384 + (s >> 2) * 16384 + 32 * (s & 3)) >> 4), db, idS, s > 0);
            else
              mma_ta(d, tb + C::kColQlo + 8 * s, db, idS, s > 0);
          }
          mma_ta(d, tb + C::kColQ + 8 * s, db, idS, !FAST || s > 0);
        }
        mma_commit(bar(s_bars.sready[NBLK == 1 ? j & 1 : b]));
      };
      auto issue_pv = [&](int b, int j) {  // O += P V~ of tile j
        const uint32_t tb = tmem + b * C::kBlkCols, p = tb + C::kColS + (NBLK == 1 ? 64 * (j & 1) : 0);
        const uint64_t dv0 = d_v + (uint64_t)(((j % NVB) * C::kKvBuf) >> 4);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const uint64_t dv = dv0 + (uint64_t)((2048 * s) >> 4);
          const uint32_t ph = p + 16 * s;
          if (!FAST) mma_ta(tb + C::kColO, ph + 8, dv, idO, j > 0 || s > 0);
          mma_ta(tb + C::kColO, ph, dv, idO, !FAST || j > 0 || s > 0);
        }
      };
      auto wait_k = [&](int j) { ok = ok && bar_wait(bar(s_bars.kready[j % NKB]), (uint32_t)((j / NKB) & 1), dead); };
      auto wait_v = [&](int j) { ok = ok && bar_wait(bar(s_bars.vready[j % NVB]), (uint32_t)((j / NVB) & 1), dead); };
      auto wait_p = [&](int i, int n) { ok = ok && bar_wait(bar(s_bars.pready[i]), (uint32_t)(n & 1), dead); };

      ok = ok && bar_wait(bar(s_bars.qready), 0u, dead);
      wait_k(0);
      if (ok) {
        fence_after();
        for (int b = 0; b < n_blk; ++b) issue_s(b, 0);
        mma_commit(bar(s_bars.kfree[0]));
      }
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (NBLK == 1) {  // the next tile's scores go into the other S while this tile is in its softmax
          if (j + 1 < n_tiles) {
            wait_k(j + 1);
            if (!ok) break;
            fence_after();
            issue_s(0, j + 1);
            mma_commit(bar(s_bars.kfree[(j + 1) % NKB]));
          }
          PF_STAMP(3, j, 0);
          wait_v(j);
          PF_STAMP(3, j, 1);
          wait_p(j & 1, j >> 1);
          PF_STAMP(3, j, 2);
          if (j == n_tiles - 1 && unrotate) {  // (these scores are complete: this returns at once)
            ok = ok && bar_wait(bar(s_bars.kfree[j % NKB]), (uint32_t)((j / NKB) & 1), dead);
            if (ok) load_chunk(0, true);
          }
          if (!ok) break;
          fence_after();
          issue_pv(0, j);
          mma_commit(bar(s_bars.vfree[j % NVB]));
          mma_commit(bar(s_bars.pvd));
        } else {  // the blocks take turns: while one is in its softmax the other has the tensor pipe
          for (int b = 0; b < n_blk; ++b) {
            if (b == 0) {
              wait_v(j);
              if (j == n_tiles - 1 && unrotate && ok) load_chunk(0, true);
            }
            wait_p(b, j);
            PF_STAMP(3, j, 2 * b);
            if (!ok) break;
            fence_after();
            issue_pv(b, j);
            if (b == n_blk - 1) mma_commit(bar(s_bars.vfree[j % NVB]));
            if (j + 1 < n_tiles) {
              if (b == 0) {
                wait_k(j + 1);
                if (!ok) break;
                fence_after();
              }
              issue_s(b, j + 1);
              if (b == n_blk - 1) mma_commit(bar(s_bars.kfree[(j + 1) % NKB]));
            }
            PF_STAMP(3, j, 2 * b + 1);
          }
        }
      }
      if (ok) {
        mma_commit(bar(s_bars.odone));
        if (unrotate) rotate(true, true);
      }
      if (ok) {  // (as the softmax warps do, unless they have given up)
        bar_wait_own(unrotate ? bar(s_bars.rot) : bar(s_bars.odone), unrotate ? 1u : 0u, dead);
      } else {  // (the CTA is dead)
        if (img_n != img_ph) bar_wait_own(bar(s_bars.img), img_ph & 1, dead);
        mma_commit(bar(s_bars.drain));
        bar_wait_own(bar(s_bars.drain), 0u, dead);
      }
    }
    __syncwarp();
  } else if (warp >= kSmx / 32) {
    // ================= dequantising warps =================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kDeqRegs));
    const int t = tid - kSmx;
    const RowLayout lay = row_layout(sh.Hkv, D);
    const int32_t* bt = a.block_table + (int64_t)seq * a.bt_stride;
    const int bs = a.block_size, shift = (bs & (bs - 1)) == 0 ? __ffs(bs) - 1 : -1;
    const bool al = ((uintptr_t)a.cache | a.cache_block_stride | a.cache_token_stride) % 16 == 0;
    const bool vec = al && lay.v_idx % 16 == 0;  // (K bytes start at a multiple of 16)
    const unsigned n_pages = (unsigned)a.num_blocks;
    // item n of this thread: token and 16-byte segment of the packed row.  Eight lanes take 4 tokens x the 2 segments
    // of one 64-coordinate block: their operand stores (chunk ^ (token & 7)) fall into eight bank groups.
    auto item = [&](int n, int& tok, int& seg) -> bool {
      constexpr int NP = C::NS / 2;
      const int i = t + kDeq * n;
      if (i < 2 * kBN * NP) {
        const int r8 = i & 7, pg = i >> 4, pair = pg % NP, grp = pg / NP;
        tok = grp * 8 + 4 * ((i >> 3) & 1) + (r8 & 3);
        seg = 2 * pair + (r8 >> 2);
        return true;
      }
      tok = i - 2 * kBN * NP;
      seg = C::NS - 1;
      return (C::NS & 1) && tok < kBN;
    };
    // What a thread fetches of a tile: its 16 bytes of K and V and (segment 0) the token's norms.  Page ids are
    // looked up a tile ahead of the rows, the rows a tile ahead of their use.
    struct Item { uint4 k, v; float kn, vn; };
    Item it[NIT] = {};
    int page[NIT] = {}, pos0[NIT];   // page id of the next tile; position in tile 0
    uint32_t k_off[NIT];        // byte offset of the thread's K bytes in a row; its V bytes are v_delta further
    constexpr int kPast = (int)0x80000000;
    const uint32_t v_delta = (uint32_t)(lay.v_idx - lay.k_idx), ts = (uint32_t)a.cache_token_stride;
    const uint32_t kn_off = (uint32_t)(lay.k_norm + 4 * kvh), vn_delta = (uint32_t)(lay.v_norm - lay.k_norm);
    bool has_norm[NIT];
#pragma unroll
    for (int n = 0; n < NIT; ++n) {
      int tok, seg = 0;
      pos0[n] = item(n, tok, seg) ? t_first + tok : 0x3fffffff;
      k_off[n] = (uint32_t)(lay.k_idx + kvh * (D / 2) + 16 * seg);
      has_norm[n] = seg == 0;
    }
    auto look_up = [&](int n, int j) -> int {
      const int pos = pos0[n] + j * kBN;
      if (pos >= blk_hi) return kPast;  // (past the keys of the CTA: masked, whatever is read)
      return __ldg(bt + (shift >= 0 ? pos >> shift : pos / bs));
    };
    auto load16 = [&](const uint8_t* p) -> uint4 {
      if (vec) return __ldg(reinterpret_cast<const uint4*>(p));
      const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
      return make_uint4(__ldg(w), __ldg(w + 1), __ldg(w + 2), __ldg(w + 3));
    };
    auto fetch = [&](int n, int j) {
      const int pg = page[n];
      const bool bad = (unsigned)pg >= n_pages;
      if (bad && pg != kPast) {  // a page id out of range: reported, its tokens hidden
        if (a.err_flag) atomicOr(a.err_flag, TQ4_DEV_BAD_BLOCK);
        s_bad = 1;
      }
      const int pos = pos0[n] + j * kBN;
      const uint32_t in = shift >= 0 ? (uint32_t)(pos & (bs - 1)) : (uint32_t)(pos % bs);
      // (without a valid page: row 0 of the cache, if there is one)
      const uint8_t* row = a.cache + (bad ? 0ull : (unsigned long long)(unsigned)pg * (unsigned long long)a.cache_block_stride + in * ts);
      it[n].kn = pg == kPast ? 1.f : kHidden;
      it[n].vn = 0.f;
      if (n_pages == 0) return;
      it[n].k = load16(row + k_off[n]);
      it[n].v = load16(row + k_off[n] + v_delta);
      if (has_norm[n] && !bad) {
        it[n].kn = __ldg(reinterpret_cast<const float*>(row + kn_off));
        it[n].vn = __ldg(reinterpret_cast<const float*>(row + kn_off + vn_delta));
      }
    };
    // table entry of a byte: sh bits left of it, plus the lane's copy
    const int sh = C::kLutCopies == 32 || one_table ? 7 : 6;
    const uint32_t lut_mask = 255u << sh;
    uint32_t lut_k = base + C::kOffLut + (lane & ((1 << (sh - 2)) - 1)) * 4;
    asm volatile("" : "+r"(lut_k) :: "memory");  // (no lookup before the tables are there)
    const uint32_t lut_v = lut_k + (one_table ? 0u : 256u << sh);
    auto look = [&](uint32_t at) -> uint32_t {
      uint32_t y;
      asm("ld.shared.b32 %0, [%1];" : "=r"(y) : "r"(at));
      return y;
    };
    auto expand = [&](const uint4& pk, uint32_t lut, uint32_t buf, int tok, int seg) {  // 16 bytes -> 32 fp16
      const uint32_t w[4] = {pk.x, pk.y, pk.z, pk.w};
      unsigned char* dst = sm + buf + (seg >> 1) * (kBN * 128);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t x = w[c];
        const uint4 o = make_uint4(look(lut + ((x << sh) & lut_mask)), look(lut + ((x >> (8 - sh)) & lut_mask)),
                                   look(lut + ((x >> (16 - sh)) & lut_mask)), look(lut + ((x >> (24 - sh)) & lut_mask)));
        *reinterpret_cast<uint4*>(dst + swz(tok, (seg & 1) * 4 + c)) = o;
      }
    };
    const int role = tid == kSmx ? 2 : -1;  // (time stamps)
    (void)role;
    bool ok = true;
    auto write_k = [&](int j) {  // K~ and norms of tile j from the registers
      const int b = j % NKB, u = j / NKB;
      if (u > 0) ok = bar_wait(bar(s_bars.kfree[b]), (uint32_t)((u - 1) & 1), dead) && ok;
      if (!ok) return;
      PF_STAMP(role, j, 0);
      float* ns = reinterpret_cast<float*>(sm + C::kOffNorm) + (j % kNormBufs) * 2 * kBN;
#pragma unroll
      for (int n = 0; n < NIT; ++n) {
        int tok, seg;
        if (item(n, tok, seg)) {
          expand(it[n].k, lut_k, C::kOffK + b * C::kKvBuf, tok, seg);
          if (seg == 0) {
            // (positive, so that -inf times it stays -inf)
            ns[tok] = it[n].kn == kHidden ? kHidden : fmaxf(it[n].kn, 1e-30f) * (1.f / kQGain);
            ns[kBN + tok] = it[n].vn;
          }
        }
      }
      fence_async();
      __syncwarp();
      if (lane == 0) bar_arrive(bar(s_bars.kready[b]));
      PF_STAMP(role, j, 1);
    };
    uint4 v_now[NIT], v_next[NIT];
    auto advance = [&](int j) {  // tile j's keys are written: its values step up, tile j + 1 is fetched
#pragma unroll
      for (int n = 0; n < NIT; ++n) {
        v_next[n] = it[n].v;
        if (j + 1 < n_tiles) {
          fetch(n, j + 1);
          page[n] = look_up(n, j + 2);
        }
      }
    };
    auto write_v = [&](int j) {
      const int b = j % NVB, u = j / NVB;
      PF_STAMP(role, j, 2);
      if (u > 0) ok = bar_wait(bar(s_bars.vfree[b]), (uint32_t)((u - 1) & 1), dead) && ok;
      if (!ok) return;
      PF_STAMP(role, j, 3);
#pragma unroll
      for (int n = 0; n < NIT; ++n) {
        int tok, seg;
        if (item(n, tok, seg)) expand(v_now[n], lut_v, C::kOffV + b * C::kKvBuf, tok, seg);
      }
      fence_async();
      __syncwarp();
      if (lane == 0) bar_arrive(bar(s_bars.vready[b]));
      PF_STAMP(role, j, 4);
    };
    if (n_tiles > 0) {
#pragma unroll
      for (int n = 0; n < NIT; ++n) page[n] = look_up(n, 0);
#pragma unroll
      for (int n = 0; n < NIT; ++n) {
        fetch(n, 0);
        page[n] = look_up(n, 1);
      }
      ok = bar_wait(bar(s_bars.rot), 0u, dead);  // the image of Pi has been used
      write_k(0);
      advance(0);
    }
    // The keys run a tile ahead of the values: the scores of tile j + 1 wait for nothing of tile j.  With one V~
    // buffer (head_dim 256) the next keys come before the values, which have to wait for the MMAs of the tile before
    // (5 200 -> 4 000 cycles a tile), and the next fetch after both.
    for (int j = 0; j < n_tiles && ok; ++j) {
#pragma unroll
      for (int n = 0; n < NIT; ++n) v_now[n] = v_next[n];
      if (NVB > 1) write_v(j);
      if (j + 1 < n_tiles && ok) write_k(j + 1);
      if (NVB == 1 && ok) write_v(j);
      if (j + 1 < n_tiles && ok) advance(j + 1);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::kSmxRegs));
    // ================= softmax warps: a row (half a row at head_dim 256) per thread =================
    const uint32_t tb = tmem + blk * C::kBlkCols + ((uint32_t)(32 * (warp & 3)) << 16);
    float* xchg = reinterpret_cast<float*>(sm + C::kOffXchg);
    // maximum (or sum) over the threads of a row
    // (two buffers in turn: a warp that starts exchange n + 2 has seen its partner arrive at n + 1, past reading n)
    uint32_t n_xchg = 0;
    auto row_reduce = [&](float v, auto op) -> float {
      if (TPR == 1) return v;
      float* x = xchg + (n_xchg & 1) * 256;
      x[part * 128 + m] = v;
      __syncwarp();
      if (lane == 0) bar_arrive(bar(s_bars.pair[warp & 3]));
      const bool got = bar_wait(bar(s_bars.pair[warp & 3]), n_xchg & 1, dead);
      ++n_xchg;
      return got ? op(v, x[(part ^ 1) * 128 + m]) : v;
    };
    auto fmax_op = [](float x, float y) { return fmaxf(x, y); };
    auto arrive = [&](uint64_t& b) {  // this warp's share of a hand-over to the issuing thread
      fence_before();
      __syncwarp();
      if (lane == 0) bar_arrive(bar(b));
    };
    bool ok = true;
    const bool use = n_tiles > 0 && blk < n_blk;  // (uniform per warp)
    // the raw queries were asked for, whether this part has keys (then the wait is below) or not.  (One wait for both
    // here, in front of the branch, lengthens a tile by 2 %: 4977 against 4863 us at 8 x 2048 rows on 8192 cached.)
    if (q_staged && n_tiles == 0) bar_wait_own(bar(s_bars.qraw), 0u, dead);

    // ---- rotate the queries -----------------------------------------------------------------------
    float qexp = 1.f;  // what is left between a stored dot product and the score (1 unless the queries are very large or small)
    if (use) {
      // (code that runs once per CTA costs its instruction fetches: short rolled loops)
      if (q_staged) ok = bar_wait_own(bar(s_bars.qraw), 0u, dead);
      float sc = 1.f, isc = 1.f;
      if (q_staged) {  // 16-bit rows in shared memory: the bits without the sign are in the order of the magnitudes
        const uint4* src = reinterpret_cast<const uint4*>(sm + q_at);
        const bool f16 = a.q_dtype == TQ4_F16;
        uint32_t top = 0;
#pragma unroll 4
        for (int i = 0; i < DPT / 8; ++i) {
          const uint4 r = src[i];
          top = __vmaxu2(__vmaxu2(top, r.x & 0x7FFF7FFFu), __vmaxu2(r.y & 0x7FFF7FFFu, __vmaxu2(r.z & 0x7FFF7FFFu, r.w & 0x7FFF7FFFu)));
        }
        float x0, x1;
        half_pair(top, f16, x0, x1);
        pow2_scale(row_reduce(live ? fmaxf(x0, x1) : 0.f, fmax_op), sc, isc);
        if (!live) sc = 0.f;
#pragma unroll 1
        for (int c = 0; c < DPT / 32; ++c) {
          uint32_t h[16];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint4 r = live ? src[4 * c + e] : make_uint4(0u, 0u, 0u, 0u);
            const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              half_pair(w[k], f16, x0, x1);
              h[4 * e + k] = pack_h2(x0 * sc, x1 * sc);
            }
          }
          tmem_st16(tb + C::kColS + (part * DPT) / 2 + 16 * c, h);
        }
      } else {
        float amax = 0.f;
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
#pragma unroll 1
          for (int c = 0; c < DPT / 32; ++c) {
            float x[32];
#pragma unroll
            for (int e = 0; e < 32; ++e) x[e] = 0.f;
            if (live) load32(a.q, a.q_dtype, qi + 32 * c, q_vec, x);
            if (pass == 0) {
#pragma unroll
              for (int e = 0; e < 16; ++e) amax = max3(amax, fabsf(x[2 * e]), fabsf(x[2 * e + 1]));
            } else {
              uint32_t h[16], l[16];
#pragma unroll
              for (int e = 0; e < 16; ++e) split2(x[2 * e] * sc, x[2 * e + 1] * sc, h[e], l[e]);
              tmem_st16(tb + C::kColS + (part * DPT) / 2 + 16 * c, h);
              if (a.q_dtype == TQ4_F32) tmem_st16(tb + C::kColQ + (part * DPT) / 2 + 16 * c, l);
            }
          }
          if (pass == 0) pow2_scale(row_reduce(amax, fmax_op), sc, isc);
        }
      }
      tmem_st_wait();
      arrive(s_bars.aready);
      ok = __all_sync(0xffffffffu, bar_wait(bar(s_bars.rot), 0u, dead));
      fence_after();
      // The rotated row (in tensor memory 2^8 sc times it), times kQGain and what makes its dot products scores in the log2 domain
      // (before the key norm), as fp16 terms.  Its largest coordinate is between isc / sqrt(D) and 2 sqrt(D) isc: no pass looks
      // for it, and where the factor could take the row out of fp16's range, the row keeps a power of two back.
      float f = isc * (a.scale_log2e / a.lut_scale_k);
      const int fe = (int)((__float_as_uint(fabsf(f)) >> 23) & 0xFFu) - 127;
      if (f != 0.f && (fe < -6 || fe > 3)) {
        const int ec = min(max(fe, -126), 126);
        qexp = __uint_as_float((uint32_t)(127 + ec) << 23);
        f *= __uint_as_float((uint32_t)(127 - ec) << 23);
      }
      f *= kQGain / 256.f;
#pragma unroll 1
      for (int c = 0; c < DPT / 32 && ok; ++c) {
        uint32_t v[32], h[16], l[16];
        const int d0 = part * DPT + 32 * c;
        tmem_ld_cols(tb + C::kColO + d0, v);
#pragma unroll
        for (int e = 0; e < 16; ++e) split2(__uint_as_float(v[2 * e]) * f, __uint_as_float(v[2 * e + 1]) * f, h[e], l[e]);
        tmem_st16(tb + C::kColQ + d0 / 2, h);
        if (FAST) continue;
        if (C::QLO_SMEM) {
          unsigned char* dst = sm + C::kOffQlo + blk * (NC * 16384) + (d0 >> 6) * 16384;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<uint4*>(dst + swz(m, ((d0 & 63) >> 3) + i)) = make_uint4(l[4 * i], l[4 * i + 1], l[4 * i + 2], l[4 * i + 3]);
        } else {
          tmem_st16(tb + C::kColQlo + d0 / 2, l);
        }
      }
      tmem_st_wait();
      fence_async();
      arrive(s_bars.qready);
    } else if (n_tiles > 0) {  // a block without rows
      arrive(s_bars.aready);
      arrive(s_bars.qready);
    }

    PF_STAMP(tid == 0 ? 0 : -1, 0, 6);
    // ---- the tile loop --------------------------------------------------------------------------------
    int kv_lo = 0, kv_hi = 0x7fffffff;  // (a row that is not there: zeros, nothing to mask)
    if (live) row_keys(row, kv_lo, kv_hi);
    float m_run = -CUDART_INF_F, l_run = 0.f;
    const int role = tid == 0 ? 0 : tid == 128 ? 1 : -1;  // (time stamps)
    (void)role;
    if (use) {
      for (int j = 0; j < n_tiles && ok; ++j) {
        PF_STAMP(role, j, 0);
        const int t0 = t_first + j * kBN + part * CPT;  // first token of this thread's columns
        const int sb = NBLK == 1 ? j & 1 : blk;
        ok = __all_sync(0xffffffffu, bar_wait(bar(s_bars.sready[sb]), (uint32_t)((NBLK == 1 ? j >> 1 : j) & 1), dead));
        if (!ok) break;
        PF_STAMP(role, j, 1);
        fence_after();
        const uint32_t scol = tb + C::kColS + (NBLK == 1 ? 64 * (j & 1) : 0) + part * CPT;
        const float* ns = reinterpret_cast<const float*>(sm + C::kOffNorm) + (j % kNormBufs) * 2 * kBN + part * CPT;
        // dot x key norm x qscale - reference, exp2, x value norm, split, store in place; two columns per
        // instruction.  Tiles inside the visible range of every row of the warp take the path without
        // per-element masks.  The reference is updated lazily, and looked at only after the fact: when some
        // weight exceeds 2^8 (or the row has no reference yet) the tile is done again from the scores, which stay in
        // registers, with a new one.  That saves the pass over the scores that would find the maximum first.
        const bool inner = __all_sync(0xffffffffu, t0 >= kv_lo && kv_hi - CPT >= t0 && qexp == 1.f) && !*(volatile int*)&s_bad;
        uint32_t v[CPT];
        tmem_ld_cols(scol, v);
        bool seen = true;  // some key of the tile is visible
        if (!inner) {
          // Rows whose queries' factor did not fit: nothing is hidden, so nothing else is to be done.  (As a branch in here; beside `inner`
          // it costs all calls 2 %.)  8 x 2048 rows behind 8192 with every query / one in 64 below the range, us: 5180 / 5080 by the
          // masked path, 4980 / 4790 so, 4635 within it.
          if (__all_sync(0xffffffffu, t0 >= kv_lo && kv_hi - CPT >= t0) && !*(volatile int*)&s_bad) {
#pragma unroll
            for (int i = 0; i < CPT; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * qexp);
          } else {  // hidden columns: a score of -inf (key norms are positive in shared memory)
            int lo = min(max(kv_lo - t0, 0), CPT), hi = min(max(kv_hi - t0, 0), CPT);
            uint32_t vis[CPT / 32];
            seen = false;
#pragma unroll
            for (int w = 0; w < CPT / 32; ++w) {
              const int l = min(max(lo - 32 * w, 0), 32), h = min(max(hi - 32 * w, 0), 32);
              vis[w] = h > l ? (0xFFFFFFFFu >> (32 - (h - l))) << l : 0u;
              if (*(volatile int*)&s_bad)
                for (int i = 0; i < 32; ++i)
                  if (ns[32 * w + i] == kHidden) vis[w] &= ~(1u << i);
              seen = seen || vis[w];
            }
#pragma unroll
            for (int i = 0; i < CPT; ++i)
              v[i] = (vis[i >> 5] >> (i & 31)) & 1u ? __float_as_uint(__uint_as_float(v[i]) * qexp) : 0xFF800000u;
          }
        }
        f2 ls2;
#pragma unroll 1
        for (int attempt = 0;; ++attempt) {
          const float m_neg = m_run == -CUDART_INF_F ? 0.f : -m_run;
          const f2 mn2 = pack2(m_neg, m_neg);
          float wmax = 0.f;
          ls2 = pack2(0.f, 0.f);
          // norms eight columns ahead of their use: a shared-memory read takes hundreds of cycles under this load
          ulonglong2 kn[2][2], vn[2][2];
          auto load_norms = [&](int g) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              kn[g & 1][q] = *reinterpret_cast<const ulonglong2*>(ns + 8 * g + 4 * q);
              vn[g & 1][q] = *reinterpret_cast<const ulonglong2*>(ns + kBN + 8 * g + 4 * q);
            }
          };
          load_norms(0);
          f2 lsb = pack2(0.f, 0.f);
          uint32_t w16[16];  // P of 16 columns: eight words of hi, eight of lo
#pragma unroll
          for (int g = 0; g < CPT / 8; ++g) {
            if (g + 1 < CPT / 8) load_norms(g + 1);
            float x[8];
            f2 e[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
              const int i = 8 * g + 2 * p;
              const f2 k2 = (p & 1) ? kn[g & 1][p >> 1].y : kn[g & 1][p >> 1].x;
              unpack2(fma2(pack2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), k2, mn2), x[2 * p], x[2 * p + 1]);
            }
#pragma unroll
            for (int p = 0; p < 4; ++p) e[p] = pack2(ex2_approx(x[2 * p]), ex2_approx(x[2 * p + 1]));
#pragma unroll
            for (int p = 0; p < 4; ++p) {
              f2& sum = (p & 1) ? lsb : ls2;
              sum = add2(sum, e[p]);
              const f2 v2 = (p & 1) ? vn[g & 1][p >> 1].y : vn[g & 1][p >> 1].x;
              unpack2(mul2(e[p], v2), x[2 * p], x[2 * p + 1]);
            }
            float2 f[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
              wmax = max3(wmax, x[2 * p], x[2 * p + 1]);
              const __half2 h = __floats2half2_rn(x[2 * p], x[2 * p + 1]);
              w16[4 * (g & 1) + p] = *reinterpret_cast<const uint32_t*>(&h);
              f[p] = __half22float2(h);
            }
            if (!FAST) {
#pragma unroll
              for (int p = 0; p < 4; ++p) {
                float r0, r1;
                unpack2(fma2(pack2(f[p].x, f[p].y), pack2(-1.f, -1.f), pack2(x[2 * p], x[2 * p + 1])), r0, r1);
                w16[8 + 4 * (g & 1) + p] = pack_h2(r0, r1);
              }
            }
            if (g & 1) {
              if (FAST) tmem_st8(scol + 8 * (g - 1), *reinterpret_cast<const uint32_t(*)[8]>(w16));
              else tmem_st16(scol + 8 * (g - 1), w16);
            }
          }
          ls2 = add2(ls2, lsb);
          // (sums past 1e30: a value norm of zero hides an overflow from the weights)
          float e0, e1;
          unpack2(ls2, e0, e1);
          bool need = attempt == 0 && (!(wmax <= 256.f) || !(e0 + e1 < 1e30f) || (seen && m_run == -CUDART_INF_F));
          if (TPR == 2) need = row_reduce(need ? 1.f : 0.f, fmax_op) > 0.f;
          if (!__any_sync(0xffffffffu, need)) break;
          // new reference: largest score of the tile, shifted by log2 of its value norm
          float mt = -CUDART_INF_F;
#pragma unroll
          for (int i = 0; i < CPT; i += 4) {
            const float4 kn = *reinterpret_cast<const float4*>(ns + i), vn = *reinterpret_cast<const float4*>(ns + kBN + i);
            mt = max3(mt, fmaf(__uint_as_float(v[i]), kn.x, fmaxf(lg2_approx(vn.x), -30.f)),
                      fmaf(__uint_as_float(v[i + 1]), kn.y, fmaxf(lg2_approx(vn.y), -30.f)));
            mt = max3(mt, fmaf(__uint_as_float(v[i + 2]), kn.z, fmaxf(lg2_approx(vn.z), -30.f)),
                      fmaf(__uint_as_float(v[i + 3]), kn.w, fmaxf(lg2_approx(vn.w), -30.f)));
          }
          mt = row_reduce(mt, fmax_op);
          const bool bump = need && mt > m_run;
          const float alpha = bump ? (m_run == -CUDART_INF_F ? 0.f : ex2_approx(m_run - mt)) : 1.f;
          if (bump) m_run = mt;
          l_run *= alpha;
          if (j > 0) {  // O: no MMA is working on it
            if (NBLK == 1) {
              ok = __all_sync(0xffffffffu, bar_wait(bar(s_bars.pvd), (uint32_t)((j - 1) & 1), dead));
              fence_after();
            }
#pragma unroll 1
            for (int q = 0; q < DPT / 16; ++q) {
              uint32_t o[16];
              tmem_ld16_async(tb + C::kColO + part * DPT + 16 * q, o);
              tmem_ld16_wait(o);
#pragma unroll
              for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              tmem_st16(tb + C::kColO + part * DPT + 16 * q, o);
            }
          }
        }
        tmem_st_wait();
        float s0, s1;
        unpack2(ls2, s0, s1);
        l_run += s0 + s1;
        arrive(s_bars.pready[sb]);
        PF_STAMP(role, j, 3);
      }
    }

    PF_STAMP(tid == 0 ? 0 : -1, 0, 7);
    // ---- normalise, un-rotate, store ------------------------------------------------------------------
    l_run = row_reduce(l_run, [](float x, float y) { return x + y; });
    bool have = use;
    if (use) {
      ok = __all_sync(0xffffffffu, ok && bar_wait(bar(s_bars.odone), 0u, dead));
      fence_after();
      have = ok && l_run > 0.f;
    }
    const float inv = have ? 1.f / (a.lut_scale_v * l_run) : 0.f;
    const float lse = have ? (m_run + lg2_approx(l_run)) * 0.6931471805599453f : -CUDART_INF_F;
    const bool out_vec = (uintptr_t)a.out % 16 == 0 && a.out_token_stride % 8 == 0 && a.out_head_stride % 8 == 0;
    if (pa.to_parts || a.out_rotated) {
      const int64_t vec = ((int64_t)blockIdx.z * sh.rows + row) * sh.Hq + head;
      const int64_t oi = pa.to_parts ? vec * D : (int64_t)row * a.out_token_stride + (int64_t)head * a.out_head_stride;
      void* dst = pa.to_parts ? (void*)pa.part_o : a.out;
      const int dt = pa.to_parts ? TQ4_F32 : a.out_dtype;
#pragma unroll 1
      for (int c = 0; c < DPT / 32; ++c) {
        uint32_t v[32];
        if (use && ok) tmem_ld32(tb + C::kColO + part * DPT + 32 * c, v);
        if (live) {
          float y[32];
#pragma unroll
          for (int e = 0; e < 32; ++e) y[e] = have ? __uint_as_float(v[e]) * inv : 0.f;
          store32(dst, dt, oi + part * DPT + 32 * c, out_vec, y);
        }
      }
      if (live && part == 0 && pa.to_parts) pa.part_m[vec] = lse;
      else if (live && part == 0 && a.lse_out) a.lse_out[(int64_t)row * sh.Hq + head] = lse;
    } else {
      float isc = 0.f;
      if (use) {
        float amax = 0.f, sc = 1.f;
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
#pragma unroll 1
          for (int c = 0; c < DPT / 32 && ok; ++c) {
            uint32_t v[32];
            const int d0 = part * DPT + 32 * c;
            tmem_ld_cols(tb + C::kColO + d0, v);
            if (pass == 0) {
#pragma unroll
              for (int e = 0; e < 16; ++e) amax = max3(amax, fabsf(__uint_as_float(v[2 * e])), fabsf(__uint_as_float(v[2 * e + 1])));
              continue;
            }
            uint32_t h[16], l[16];
#pragma unroll
            for (int e = 0; e < 16; ++e)
              split2(__uint_as_float(v[2 * e]) * inv * sc, __uint_as_float(v[2 * e + 1]) * inv * sc, h[e], l[e]);
            tmem_st16(tb + C::kColS + d0 / 2, h);
            tmem_st16(tb + C::kColQ + d0 / 2, l);
          }
          if (pass == 0) pow2_scale(row_reduce(amax * inv, fmax_op), sc, isc);
        }
        tmem_st_wait();
        arrive(s_bars.aready);
        ok = __all_sync(0xffffffffu, bar_wait(bar(s_bars.rot), 1u, dead)) && ok;
        fence_after();
      } else if (n_tiles > 0) {  // (not before the first rotation is over: its phase wants one arrival per warp)
        bar_wait(bar(s_bars.rot), 0u, dead);
        arrive(s_bars.aready);
      }
      const float f = have && ok ? isc * (1.f / 256.f) : 0.f;
      const int64_t oi = (int64_t)row * a.out_token_stride + (int64_t)head * a.out_head_stride + part * DPT;
      // 16-bit rows go through shared memory (where the raw queries came in), from which a warp stores whole rows: stored from
      // here, its 16-byte pieces would fall into 32 of them
      const bool staged = out_vec && a.out_dtype != TQ4_F32;
#pragma unroll 1
      for (int c = 0; c < DPT / 32; ++c) {
        uint32_t v[32];
        if (use && ok) tmem_ld32(tb + C::kColO + part * DPT + 32 * c, v);
        if (live) {
          float y[32];
#pragma unroll
          for (int e = 0; e < 32; ++e) y[e] = f != 0.f ? __uint_as_float(v[e]) * f : 0.f;
          if (staged) store32(sm + q_at, a.out_dtype, 32 * c, true, y);
          else store32(a.out, a.out_dtype, oi + 32 * c, out_vec, y);
        }
      }
      if (staged) {
        __syncwarp();
        constexpr int PCS = DPT / 8;  // 16-byte pieces of a thread's part of a row
        const unsigned char* rows = sm + C::kOffQlo + (blk * 128 + 32 * (warp & 3)) * C::kQPitch + part * DPT * 2;
        const int64_t to = live ? oi : -1;
#pragma unroll 4
        for (int i = lane; i < 32 * PCS; i += 32) {
          const int r = i / PCS, pc = i - r * PCS;
          const int64_t at = __shfl_sync(0xffffffffu, to, r);
          if (at >= 0)
            *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(a.out) + at + 8 * pc) = *reinterpret_cast<const uint4*>(rows + r * C::kQPitch + 16 * pc);
        }
      }
      if (live && part == 0 && a.lse_out) a.lse_out[(int64_t)row * sh.Hq + head] = lse;
    }
  }
  fence_before();
  __syncthreads();
  PF_STAMP(tid == 0 ? 0 : -1, 1, 4);
  if (s_dead && tid == 0 && a.err_flag) atomicOr(a.err_flag, TQ4_DEV_TIMEOUT);
  if (warp == kIssueWarp) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

template <int D, bool FAST>
int launch_t(const AttnArgs& a, PrefillArgs pa, cudaStream_t st) {
  using C = Cfg<D>;
  constexpr int smem = (int)C::kSmem + 1024;
  static_assert(smem + 2048 <= 227 * 1024, "shared memory");
  static_assert(2 * smem > 227 * 1024 || D < 128, "one CTA per SM: it allocates the whole tensor memory");
  // (head_dim 64 and 96 need less: ask for more than half of the SM so that only one CTA fits)
  constexpr int ask = smem > 120 * 1024 ? smem : 120 * 1024;
  if (!ensure_dynamic_smem<prefill_tc_kernel<D, FAST>>(ask)) return TQ4_ERR_CUDA;
  const int per_cta = C::NBLK * (128 / a.sh.G);
  const unsigned blocks = (unsigned)((a.sh.rows + per_cta - 1) / per_cta + a.sh.num_seqs);  // upper bound
  // More CTAs than fit at once: the KV heads run fastest, so that all heads of a sequence's last rows (the longest) start before any of
  // its first and those left for the end are short.  Rows fastest / heads fastest, us: 2048 rows of 32 / 8 heads of 128 146 / 111, 6000
  // 632 / 572, 4000 of 32 / 32 of 96 362 / 308, 2 x 1500 of 8 / 4 of 256 139 / 113, 8 x 2048 on 8192 4690 / 4605.  One wave: nothing waits, and a
  // head's CTAs next to one another are better off (4 x 500 on 3000, 14 / 2 heads of 64: 129 / 141).  Counted with the spare row blocks
  // of the upper bound, which the SMs go through as well: heads fastest, they come behind all others (480 rows beside 32 running
  // sequences 206 / 201, 256 beside 60, 28 / 4 heads, 145 / 134).  Where only the spare ones make it more than a wave (10 - 64 prompts of
  // 30 - 190 rows on 2000 - 3000, 14 / 2 of 64 and 4 / 1 of 128) the two orders are within 0.6 %.
  const int64_t grid = (int64_t)blocks * a.sh.Hkv;
  if (grid > 0x7fffffff) return TQ4_ERR_UNSUPPORTED;
  pa.heads_first = grid * pa.splits > sm_count();
  if (launch_kernel(prefill_tc_kernel<D, FAST>, dim3((unsigned)grid, 1, (unsigned)pa.splits), dim3(kThreads), (size_t)ask, st, true, a,
                    pa) != cudaSuccess)
    return TQ4_ERR_CUDA;
  TQ4_CHECK_LAUNCH();
  return TQ4_OK;
}

template <int D>
int launch_d(const AttnArgs& a, const PrefillArgs& pa, cudaStream_t st, bool fast, uint8_t* image) {
  constexpr int n = D * ((D + 63) / 64) * 8;
  // first kernel of the prefill part: a plain launch (what the caller and the streaming part wrote is complete)
  if (launch_kernel(pi_image_kernel<D>, dim3((n + 255) / 256), dim3(256), 0, st, false, a.rotation, image) != cudaSuccess)
    return TQ4_ERR_CUDA;
  TQ4_CHECK_LAUNCH();
  return fast ? launch_t<D, true>(a, pa, st) : launch_t<D, false>(a, pa, st);
}

size_t image_bytes(int D) { return (size_t)2 * ((D + 63) / 64) * D * 128; }

}  // namespace

// Every layout of the packed cache is covered (16-byte loads where the rows allow them, 4-byte loads elsewhere).
bool prefill_tc_supported(const AttnArgs& a) {
  static const bool disabled = getenv("TQ4_NO_TC") != nullptr;
  return !disabled && a.query_start_loc != nullptr && a.sh.G <= 128 && a.num_blocks < (1ll << 31) && a.sh.Hkv <= 65535;
}

// Parts of the key range: as many as fill the SMs when the row blocks do not, at least four tiles each; limited
// by the room for their partials (`slots` vectors sets of Hq in the scratch).  The tiles are those of the caller's
// max_seq_len: by the width of a server's table a prompt of 300 tokens (32 / 8 heads of 128) was cut into parts of at
// most two tiles, 52.3 instead of 35.9 us.
int prefill_tc_splits(const AttnArgs& a, int64_t slots) {
  const int per_cta = (a.sh.D == 256 ? 1 : 2) * (128 / a.sh.G);
  const int64_t ctas = (int64_t)((a.sh.rows + per_cta - 1) / per_cta) * a.sh.Hkv;
  int64_t s = sm_count() / (ctas > 0 ? ctas : 1);
  const int64_t tiles = a.max_keys / kBN;
  if (s > tiles / 4) s = tiles / 4;
  if (s > 8) s = 8;
  if (a.sh.rows > 0 && s > slots / a.sh.rows) s = slots / a.sh.rows;
  return s < 1 ? 1 : (int)s;
}
size_t prefill_tc_image_bytes(int D) { return image_bytes(D); }

int launch_prefill_tc(const AttnArgs& a, cudaStream_t st, bool fast, int min_rows, int splits, bool to_parts,
                      uint8_t* image, float* part_o, float* part_m) {
  const PrefillArgs pa{image, min_rows, splits, to_parts ? 1 : 0, part_o, part_m};
  switch (a.sh.D) {
    case 64: return launch_d<64>(a, pa, st, fast, image);
    case 96: return launch_d<96>(a, pa, st, fast, image);
    case 128: return launch_d<128>(a, pa, st, fast, image);
    case 256: return launch_d<256>(a, pa, st, fast, image);
  }
  return TQ4_ERR_UNSUPPORTED;
}

}  // namespace tq4

#ifdef TQ4_TRACE
extern "C" int tq4_prefill_trace_read(long long* out) {
  return cudaMemcpyFromSymbol(out, tq4::g_ptrace, sizeof(long long) * 4 * 64 * 8) == cudaSuccess ? 0 : 1;
}
#endif
