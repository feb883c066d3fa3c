// Arguments of the kernels of a HuggingFace-style cache update (tq4_cache_update.cu, tq4_restore_tc.cu).
#pragma once
#include "tq4_common.cuh"

namespace tq4 {

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
  const float *rot_even, *rot_odd;  // even / odd columns of Pi^T
  const uint8_t* packed;               // (optional) the vectors compressed already, K then V, [B, S, H, D / 2] and [B, S, H]
  const float* packed_norms;
};

// tensor-core (tcgen05) kernel for 16-bit types: indices, norms and reconstruction of vectors that are compressed already
bool restore_tc_eligible(const UpdateArgs& a, int head_dim);
int launch_restore_tc(const UpdateArgs& a, int head_dim, cudaStream_t st);

}  // namespace tq4
