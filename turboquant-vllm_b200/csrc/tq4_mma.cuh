// Pieces that the two streaming attention kernels share (tq4_decode_mma.cu, tq4_decode_step.cu): the MMA on
// registers, the fp16 hi / lo split, and how a tile's bytes are dealt out to the lanes of a warp.
#pragma once
#include "tq4_attention.cuh"

namespace tq4 {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// first MMA of an accumulation chain: C = 0 (no zero-initialised accumulator registers needed)
__device__ __forceinline__ void mma16816_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                              uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

// split x into fp16 hi + fp16 lo and pack (hi, lo) into one register
__device__ __forceinline__ uint32_t split_h2(float x) {
  const __half h = __float2half_rn(x);
  const __half l = __float2half_rn(x - __half2float(h));
  __half2 r = __halves2half2(h, l);
  return *reinterpret_cast<uint32_t*>(&r);
}

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

template <int D, bool ALIGNED>
struct MmaCfg {
  static constexpr int HALF = D / 2;
  static constexpr int KS = D / 16;         // k-steps of the K-side product
  static constexpr int KBY = D / 8;         // K bytes per thread per token
  static constexpr int KW = KBY / 4;        // ... as 32-bit words
  static constexpr int VBY = D / 16;        // V bytes per thread per token
  static constexpr int VW = VBY / 4;        // ... full words
  static constexpr int VH = (VBY % 4) / 2;  // ... plus one half-word (D = 96)
  static constexpr int MB = VBY;            // m-blocks of the V-side product
  static constexpr int DPT = D / 4;         // query dims held per thread
  // cp.async unit sizes (bytes) and counts
  static constexpr int UK = ALIGNED ? (KBY >= 16 ? 16 : KBY) : 4;
  static constexpr int NK = KBY / UK;
  static constexpr int UV = ALIGNED ? (4 * VW >= 16 ? 16 : 4 * VW) : 4;
  static constexpr int NV = (4 * VW) / UV;
  // per-warp bytes of one ring stage: K (2 tokens) + V (4 tokens: words + half-word unit) + norms
  static constexpr int kVTok = 32 * (4 * VW + 4 * VH);
  static constexpr int kOffK1 = 32 * KBY;
  static constexpr int kOffV = 64 * KBY;
  static constexpr int kOffN = kOffV + 4 * kVTok;
  static constexpr int kStageBytes = kOffN + 32 * 16;
  // TMA stage: K tile [16 tok][D/2] | V tile [16 tok][D/2] | K-norm tile [16][16 B] | V-norm tile
  // (VWIDE: the V box starts 0..12 bytes early, on a 16-byte boundary, and is 16 bytes wider)
  static constexpr int kTmaV = 16 * HALF;
  template <bool VWIDE> __host__ __device__ static constexpr int v_pitch() { return VWIDE ? HALF + 16 : HALF; }
  template <bool VWIDE> __host__ __device__ static constexpr int tma_kn() { return 16 * HALF + 16 * v_pitch<VWIDE>(); }
  template <bool VWIDE> __host__ __device__ static constexpr int tma_stage() { return tma_kn<VWIDE>() + 512; }
};

// byte offset (within a head's D/2 V bytes) of this thread's m-block i
template <int D>
__device__ __forceinline__ int v_byte_of_mblock(int g, int i) {
  constexpr int VW = (D / 16) / 4;
  return i < 4 * VW ? g * 4 * VW + i : 32 * VW + 2 * g + (i - 4 * VW);
}

inline bool cache_aligned(const AttnShape& sh, const uint8_t* cache, int64_t bs, int64_t ts) {
  // 16-byte K chunks and 8/16-byte V chunks need the regions of a token row aligned accordingly
  const RowLayout lay = row_layout(sh.Hkv, sh.D);
  const int valign = sh.D >= 256 ? 16 : 8;
  return ((uintptr_t)cache % 16 == 0) && bs % 16 == 0 && ts % 16 == 0 && lay.v_idx % valign == 0 &&
         (sh.D / 2) % valign == 0 && sh.D != 96;
}

}  // namespace tq4
