// Flash attention backward: what the entry (attention_bwd.cu) and the kernels of one tile per CTA (attention_bwd_tile.cu)
// share.
#pragma once
#include "common.h"
#include "ptx.cuh"

namespace nx {

constexpr int AB = 128;     // rows per resident tile
constexpr float LOG2E = 1.4426950408889634f;

struct AttnBwdParams {
  const float* lse;    // [B,H,Sq_pad] base-2 log-sum-exp, +inf in the padding
  const float* delta;  // [B,H,Sq_pad], 0 in the padding
  const float* alibi;
  h16 *dq, *dk, *dv;
  long long dq_sb, dq_sh, dq_ss, dk_sb, dk_sh, dk_ss, dv_sb, dv_sh, dv_ss;
  int B, H, Hk, Sq, Sk, D, Sq_pad;
  float scale, scale_log2;
  int causal, window;
  int* err;
  // dropout as in the forward (same seed and threshold): dP is masked and scaled before delta is subtracted,
  // and the P^T that feeds dV is the dropped one
  uint32_t drop_thr, seed_lo, seed_hi;
  float drop_rp;
  // block-sparse layout tables of the forward (null = dense): blk_rows[q * blk_nkt + kt] bit j = row q attends to
  // key sub-block j of key tile kt; blk_any[qt * blk_nkt + kt] != 0 = tile (qt, kt) has any live block
  const uint8_t* blk_rows;
  const uint8_t* blk_any;
  int blk_shift, blk_nkt;
};

struct BwdMaps {
  CUtensorMap q, k, v, d_o;      // swizzled boxes of 64 columns and 64 rows, or 128 for the kernels of one CTA per tile
};

// Kernels of one CTA per tile: dQ (dropout, block-sparse layouts and scale 0 included), dK / dV.
int attn_bwd_tile_dq(const BwdMaps& m, const AttnBwdParams& p, cudaStream_t s);
int attn_bwd_tile_dkv(const BwdMaps& m, const AttnBwdParams& p, cudaStream_t s);

}  // namespace nx
