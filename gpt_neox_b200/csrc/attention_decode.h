// One query row per (batch, head) against its keys: the step of cached generation (attention_decode.cu).
#pragma once
#include "common.h"
#include "ptx.cuh"

namespace nx {

// The log-sum-exp of a row without a usable sum (no visible key, or a NaN among its scores).  Finite and below every
// score: the backward forms exp2(score - lse) with masked scores of -inf, which -inf here would turn into NaN, so that a NaN
// row would reach the gradients of keys it does not see; an unmasked score still gives +inf or NaN.
constexpr float LSE_NONE = -3.0e38f;

struct AttnDecodeParams {
  const h16 *q, *k, *v;
  h16* o;
  float* lse;          // [B, H, 128]: entry 0 of a row is written, the padding behind it set to +inf
  const float* alibi;  // per query head, or null
  int B, H, Hk, Sk, D;
  long long q_sb, q_sh, k_sb, k_sh, k_ss, v_sb, v_sh, v_ss, o_sb, o_sh;
  float scale_log2;
  int key_lo;          // first key the window leaves visible
};

int attn_decode_launch(const AttnDecodeParams& p, cudaStream_t stream);

}  // namespace nx
