// Flash attention backward, one CTA per tile: the kernels for dropout and for block-sparse layouts, and otherwise for heads of up to
// 64 (dQ: also for larger ones) in calls whose tiles do not fill the SMs often enough (attn_bwd_route in attention_bwd.cu says
// which call takes which and why).  A softmax scale of 0 comes here, too, to the general forms.
//
//   dQ       a CTA per 128 query rows: loops over blocks of 128 keys (longest tiles first)
//   dK / dV  a CTA per 128 keys of a kv head: loops over the query heads of its group and over blocks of 128 query rows
//
// Warp 0 loads (TMA), one thread of warp 1 issues the MMAs, eight element-wise warps take 32 columns of each half of a block.
// Against the persistent kernels a CTA pays its prologue, pipeline fill and stores alone, but its threads have twice the
// registers (dropout there spilled 500 bytes: batch 4, 32 heads, 2048 x 128 causal with dropout 1833 us for the whole
// backward, 953 here), the hardware hands the tiles out as SMs become free (block-sparse tiles are of any length: 1 x 8192, 8
// heads of 128, 731 us persistent, 499 here), and starting takes less (12 heads of 64, 8 x 128 tokens: 19.5 us, 16.3 here).
// Counterpart of the flash-attn 2 backward the reference calls through autograd (megatron/model/transformer.py:573-690).
#include "attention_bwd.h"
#include "ptx.cuh"

namespace nx {

constexpr int TILE_THREADS = 32 * 10;

template <int DP>
struct TileSmem {
  static constexpr int TILE = AB * DP * 2;
  static constexpr int BAR_OFF = 6 * TILE;  // two resident tiles + 2 x 2 streamed tiles
  static constexpr int NBAR = 24;           // (the last: the TMEM base word)
  static constexpr int VEC_OFF = BAR_OFF + NBAR * 8;  // lse / delta staging: 2 stages x 2 x 128 floats
  static constexpr int TOTAL = VEC_OFF + 4 * AB * 4 + 16;
  static constexpr int DYN = TOTAL + 1024;
};

// Loads one [128 x DP] tile (rows contiguous in d) as swizzled boxes of 128 rows x 64 columns.
template <int DP>
__device__ __forceinline__ void tile_load(uint32_t dst, const CUtensorMap* m, uint32_t bar, int row0, int head, int batch) {
#pragma unroll
  for (int c = 0; c < DP / 64; ++c) tma_load_4d(dst + c * (AB * 128), m, bar, c * 64, row0, head, batch);
}
// D[128 x 64] = A[128 x DP] * B[64 x DP]^T, both K-major (head dim contiguous); b points at the first of the 64 rows of a
// 128-row tile.
template <int DP>
__device__ __forceinline__ void tile_mma_nt(uint32_t d_tmem, uint32_t a, uint32_t b) {
  constexpr uint32_t idesc = umma_idesc_bf16(AB, 64, 0, 0);
#pragma unroll
  for (int k = 0; k < DP / 16; ++k) {
    const uint32_t o = (k >> 2) * (AB * 128) + (k & 3) * 32;
    umma_bf16_ss(d_tmem, umma_smem_desc_sw128(a + o, 0, 1024), umma_smem_desc_sw128(b + o, 0, 1024), idesc, k != 0 ? 1u : 0u);
  }
}
// D[128 x DP] (+)= A_tmem[128 x 64 (16 bit)] * B[64 x DP] with B's head dim contiguous (MN-major B operand); b points at the
// first of its rows.  SPLIT: every 16 columns of A (32 rows of B) start 32 columns apart instead of lying back to back.
template <int DP, bool SPLIT>
__device__ __forceinline__ void tile_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b, bool accumulate) {
  constexpr uint32_t idesc = umma_idesc_bf16(AB, DP, 0, 1);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    umma_bf16_ts(d_tmem, a_tmem + (SPLIT ? (k >> 1) * 32 + (k & 1) * 8 : k * 8),
                 umma_smem_desc_sw128(b + k * 2048, AB * 128, 1024), idesc, (accumulate || k != 0) ? 1u : 0u);
}

// ------------------------------------------------------------------------------------------------
// dQ kernel.  smem tiles: 0 = Q, 1 = dO, 2..3 = K ring, 4..5 = V ring.
// TMEM: S [0,128) dP [128,256) dQ [256,256+DP) dS0 [384,448) dS1 [448,512)
// The 128 keys of a block are handled as two halves of 64 with their own S / dP columns (S_h at [64 h, ...), dP_h at
// [128 + 64 h, ...)), dS_h at [384 + 32 h, ...) and their own barriers.  The MMA warp issues S / dP of half u + 1 before it
// waits for dS of half u, so the tensor core computes the next half (and dQ += dS K of the previous one) while the
// element-wise warps work on the current one.
// GEN (this kernel and the next): ALiBi and block-sparse layouts; without them a block that needs a mask differs from one
// that does not by one select per element (batch 4, 32 heads, 2048 x 128 causal: dQ 318 -> 288 us).
// ------------------------------------------------------------------------------------------------
template <int DP, bool DROP, bool GEN>
__global__ void __launch_bounds__(TILE_THREADS, 1)
    attn_bwd_tile_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                            const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                            const AttnBwdParams p) {
  using L = TileSmem<DP>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - smem_u32(smem_raw));
  const uint32_t bar0 = sbase + L::BAR_OFF;
  enum { QDO_FULL = 0, K_FULL = 1, K_EMPTY = 3, V_FULL = 5, V_EMPTY = 7, SDP_FULL = 9, DS_FULL = 11, DQ_DONE = 13, NUSED = 14 };
  auto bar = [&](int which, int idx) { return bar0 + 8u * (which + idx); };
  const uint32_t tmem_slot = bar0 + 8u * 23;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(sgen + L::BAR_OFF + 8 * 23);
  auto tile = [&](int i) { return sbase + i * L::TILE; };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qt = gridDim.x - 1 - blockIdx.x;
  const int head = blockIdx.y, batch = blockIdx.z;
  const int kv_head = head / (p.H / p.Hk);
  const int q0 = qt * AB;
  const int off = p.Sk - p.Sq;
  int kv_end = p.Sk;
  if (p.causal) kv_end = min(p.Sk, q0 + AB + off);
  int kv_begin = 0;
  if (p.window >= 0) kv_begin = max(0, q0 + off - p.window);
  const int jb = kv_begin / AB;
  const int nblk = max((kv_end + AB - 1) / AB - jb, 0);
  // block-sparse layouts: key tiles without a live block for this query tile are skipped by every role; ring
  // stages and barrier phases count the live tiles
  auto tile_live = [&](int kt) { return !GEN || p.blk_any == nullptr || p.blk_any[static_cast<long long>(qt) * p.blk_nkt + kt] != 0; };

  if (threadIdx.x == 0) {
    for (int i = 0; i < NUSED; ++i) mbar_init(bar0 + 8u * i, (i == DS_FULL || i == DS_FULL + 1) ? 8 : 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot_gen;
  const uint32_t T_S = tmem, T_DP = tmem + 128, T_DQ = tmem + 256, T_DS = tmem + 384;
  bool aborted = false;

  if (warp == 0) {
    if (elect_one() && nblk > 0) {
      mbar_expect_tx(bar(QDO_FULL, 0), 2 * L::TILE);
      tile_load<DP>(tile(0), &tmQ, bar(QDO_FULL, 0), q0, head, batch);
      tile_load<DP>(tile(1), &tmDO, bar(QDO_FULL, 0), q0, head, batch);
      for (int t = 0, n = 0; t < nblk; ++t) {
        if (!tile_live(jb + t)) continue;
        const int i = n++;
        const int st = i & 1;
        const uint32_t ph = (i >> 1) & 1;
        const int k0 = (jb + t) * AB;
        if (!mbar_wait(bar(K_EMPTY, st), ph ^ 1, p.err, 31)) { aborted = true; break; }
        mbar_expect_tx(bar(K_FULL, st), L::TILE);
        tile_load<DP>(tile(2 + st), &tmK, bar(K_FULL, st), k0, kv_head, batch);
        if (!mbar_wait(bar(V_EMPTY, st), ph ^ 1, p.err, 32)) { aborted = true; break; }
        mbar_expect_tx(bar(V_FULL, st), L::TILE);
        tile_load<DP>(tile(4 + st), &tmV, bar(V_FULL, st), k0, kv_head, batch);
      }
    }
  } else if (warp == 1) {
    if (elect_one() && nblk > 0) {
      if (!mbar_wait(bar(QDO_FULL, 0), 0, p.err, 34)) aborted = true;
      // sub-step u = 2 i + h of live block i: S_h = Q K_h^T, dP_h = dO V_h^T (64 keys), later dQ += dS_h K_h
      int nl = 0;
      for (int t = 0; t < nblk; ++t) nl += tile_live(jb + t) ? 1 : 0;
      auto issue_m1 = [&](int u) -> bool {
        const int i = u >> 1, h = u & 1, st = i & 1;
        if (h == 0) {
          if (!mbar_wait(bar(K_FULL, st), (i >> 1) & 1, p.err, 35)) return false;
          if (!mbar_wait(bar(V_FULL, st), (i >> 1) & 1, p.err, 36)) return false;
        }
        tc_fence_after_sync();
        tile_mma_nt<DP>(T_S + h * 64, tile(0), tile(2 + st) + h * (64 * 128));
        tile_mma_nt<DP>(T_DP + h * 64, tile(1), tile(4 + st) + h * (64 * 128));
        umma_commit(bar(SDP_FULL, h));
        if (h == 1) umma_commit(bar(V_EMPTY, st));
        return true;
      };
      const int nsub = 2 * nl;
      if (!aborted && nsub > 0 && !issue_m1(0)) aborted = true;
      for (int u = 0; u < nsub && !aborted; ++u) {
        const int i = u >> 1, h = u & 1, st = i & 1;
        if (u + 1 < nsub && !issue_m1(u + 1)) { aborted = true; break; }
        if (!mbar_wait(bar(DS_FULL, h), i & 1, p.err, 33)) { aborted = true; break; }
        tc_fence_after_sync();
        tile_mma_ts<DP, false>(T_DQ, T_DS + h * 32, tile(2 + st) + h * (64 * 128), u != 0);    // dQ += dS_h K_h
        if (h == 1) umma_commit(bar(K_EMPTY, st));
      }
      if (!aborted && nsub > 0) umma_commit(bar(DQ_DONE, 0));
    }
  } else {
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;    // which 32 of a half's 64 key columns (and which half of dQ's columns)
    const int r = quad * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const int qi = q0 + r;
    const int qpos = qi + off;
    const bool row_ok = qi < p.Sq;
    const long long stat_idx = (static_cast<long long>(batch) * p.H + head) * p.Sq_pad + qi;
    const float lse2 = p.lse[stat_idx];     // +inf for rows past Sq -> P = 0
    const float delta = p.delta[stat_idx];
    const float slope2 = GEN && p.alibi != nullptr ? p.alibi[head] * LOG2E : 0.f;
    int nlive = 0;
    for (int t = 0; t < nblk; ++t) {
      if (!tile_live(jb + t)) continue;
      const int i = nlive++;
      const int k0 = (jb + t) * AB;
      uint32_t bits = 0xffffffffu;
      if (GEN && p.blk_rows != nullptr)
        bits = row_ok ? p.blk_rows[static_cast<long long>(qi) * p.blk_nkt + (jb + t)] : 0u;
      const uint32_t full_bits = (1u << (AB >> p.blk_shift)) - 1u;
      const bool blk_partial = GEN && p.blk_rows != nullptr && !__all_sync(0xffffffffu, (bits & full_bits) == full_bits);
      const bool need_mask = (k0 + AB > p.Sk) || (p.causal && k0 + AB - 1 > q0 + quad * 32 + off) ||
                             (p.window >= 0 && k0 < q0 + quad * 32 + 31 + off - p.window) || blk_partial;
      const int rel0 = k0 - qpos;
      int hi = p.Sk - k0 - 1;
      if (p.causal) hi = min(hi, -rel0);
      const int lo = p.window >= 0 ? -rel0 - p.window : -(1 << 30);
      const float bias0 = slope2 * static_cast<float>(rel0) - lse2;  // folded into the exponent
      // pass h = 0, 1 over the block's halves: this warp's chunk in each is c = 2 h + half (block columns 32 c ..), read from
      // the half's own S / dP columns after its own barrier
#pragma unroll 1
      for (int cc = 0; cc < 2; ++cc) {
        const int c = cc * 2 + half;
        if (!mbar_wait(bar(SDP_FULL, cc), i & 1, p.err, 38)) { aborted = true; break; }
        tc_fence_after_sync();
        uint32_t sv[32], dv[32];
        tmem_ld_32x32b_x32(T_S + c * 32 + lane_off, sv);
        tmem_ld_32x32b_x32(T_DP + c * 32 + lane_off, dv);
        tmem_ld_wait();
        if (DROP) {
          // dP of a dropped probability is zero, of a kept one it carries the 1 / (1 - p) factor
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const int kk = k0 + c * 32 + j;
            const uint32_t patch = dropout_patch(p.seed_lo, p.seed_hi, static_cast<uint32_t>(batch * p.H + head),
                                                 static_cast<uint32_t>(qi) >> 1, static_cast<uint32_t>(kk) >> 1);
            dv[j] = dropout_keep(patch, qi, kk, p.drop_thr) ? __float_as_uint(__uint_as_float(dv[j]) * p.drop_rp) : 0u;
            dv[j + 1] = dropout_keep(patch, qi, kk + 1, p.drop_thr)
                            ? __float_as_uint(__uint_as_float(dv[j + 1]) * p.drop_rp) : 0u;
          }
        }
        uint32_t pk[16];
        if (!GEN || (!need_mask && p.alibi == nullptr)) {
          if (!GEN && need_mask) {      // masked scores: -inf, probability 0
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const int idx = c * 32 + j;
              if (idx < lo || idx > hi) sv[j] = __float_as_uint(p.scale_log2 < 0.f ? INFINITY : -INFINITY);
            }
          }
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            // the softmax scale of dS is applied once, to dQ, in the epilogue
            const float p0 = exp2f(fmaf(__uint_as_float(sv[j]), p.scale_log2, -lse2));
            const float p1 = exp2f(fmaf(__uint_as_float(sv[j + 1]), p.scale_log2, -lse2));
            pk[j >> 1] = pack_h16x2(p0 * (__uint_as_float(dv[j]) - delta),
                                     p1 * (__uint_as_float(dv[j + 1]) - delta));
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            float ds[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int idx = c * 32 + j + e;
              float x = fmaf(__uint_as_float(sv[j + e]), p.scale_log2,
                             fmaf(slope2, static_cast<float>(idx), bias0));
              float pr = exp2f(x);
              if (idx < lo || idx > hi || !((bits >> (idx >> p.blk_shift)) & 1u)) pr = 0.f;
              ds[e] = pr * (__uint_as_float(dv[j + e]) - delta);
            }
            pk[j >> 1] = pack_h16x2(ds[0], ds[1]);
          }
        }
        // dS_h sits at [384 + 32 h, ...): the chunk's 16 columns at 16 c (c = 2 h + half)
        tmem_st_32x32b_x16(T_DS + c * 16 + lane_off, pk);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(DS_FULL, cc));
      }
      if (aborted) break;
    }
    if (!aborted && nlive > 0) {
      if (!mbar_wait(bar(DQ_DONE, 0), 0, p.err, 40)) aborted = true;
      tc_fence_after_sync();
    }
    if (!aborted) {
      h16* orow = p.dq + batch * p.dq_sb + head * p.dq_sh + static_cast<long long>(qi) * p.dq_ss;
#pragma unroll 1
      for (int c = half * (DP / 64); c < (half + 1) * (DP / 64); ++c) {   // this warp's dQ columns
        uint32_t ov[32];
        if (nlive > 0) {  // warp-uniform: every lane takes part in the collective TMEM load
          tmem_ld_32x32b_x32(T_DQ + c * 32 + lane_off, ov);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) ov[j] = 0u;
        }
        if (row_ok) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            if (c * 32 + j < p.D) {
              const float sc = p.scale;
              uint4 o4;
              o4.x = pack_h16x2(__uint_as_float(ov[j]) * sc, __uint_as_float(ov[j + 1]) * sc);
              o4.y = pack_h16x2(__uint_as_float(ov[j + 2]) * sc, __uint_as_float(ov[j + 3]) * sc);
              o4.z = pack_h16x2(__uint_as_float(ov[j + 4]) * sc, __uint_as_float(ov[j + 5]) * sc);
              o4.w = pack_h16x2(__uint_as_float(ov[j + 6]) * sc, __uint_as_float(ov[j + 7]) * sc);
              *reinterpret_cast<uint4*>(orow + c * 32 + j) = o4;
            }
          }
        }
      }
    }
  }
  __syncwarp();
  if (aborted) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------------
// dK / dV kernel.  smem tiles: 0 = K, 1 = V, 2..3 = Q ring, 4..5 = dO ring.
// TMEM: S^T [0,128), dP^T [128,256), dK [256,256+DP), dV [384,384+DP)
// A step's 128 query columns are handled as two halves of 64 with their own S^T / dP^T buffers (S^T_h at [64 h, 64 h + 64),
// dP^T_h at [128 + 64 h, ...)) and their own barriers.  The MMA warp issues S^T / dP^T of half u + 1 before it waits for
// P^T / dS^T of half u, so the tensor core works on the next half (and on dV / dK of the previous one) while the
// element-wise warps are busy with the current one.  A warp writes its 16-bit results over the first half of the 32
// columns it read itself (the MMA takes its A operand in pieces of 16 query rows, each with its own column address), so the
// two warps of a quadrant never touch each other's columns and need no barrier between reading and writing.
// ------------------------------------------------------------------------------------------------
template <int DP, bool DROP, bool GEN>
__global__ void __launch_bounds__(TILE_THREADS, 1)
    attn_bwd_tile_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                            const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                            const AttnBwdParams p) {
  using L = TileSmem<DP>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - smem_u32(smem_raw));
  const uint32_t bar0 = sbase + L::BAR_OFF;
  enum { KV_FULL = 0, Q_FULL = 1, Q_EMPTY = 3, ST_FULL = 5, PT_FULL = 7, ACC_DONE = 9, NUSED = 10 };
  auto bar = [&](int which, int idx) { return bar0 + 8u * (which + idx); };
  const uint32_t tmem_slot = bar0 + 8u * 23;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(sgen + L::BAR_OFF + 8 * 23);
  auto tile = [&](int i) { return sbase + i * L::TILE; };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kt = blockIdx.x;
  const int kv_head = blockIdx.y, batch = blockIdx.z;
  const int group = p.H / p.Hk;
  const int k0 = kt * AB;
  const int off = p.Sk - p.Sq;
  // query rows that can see this key block: qpos >= k0 (causal), qpos <= k_last + window
  int q_begin = 0, q_end = p.Sq;
  if (p.causal) q_begin = max(0, k0 - off);
  if (p.window >= 0) q_end = min(p.Sq, k0 + AB - 1 + p.window - off + 1);
  const int ib = q_begin / AB;
  const int nq = max((q_end + AB - 1) / AB - ib, 0);
  const int nsteps = nq * group;
  // block-sparse layouts: query tiles without a live block for this key tile are skipped by every role
  auto step_live = [&](int t) {
    return !GEN || p.blk_any == nullptr || p.blk_any[static_cast<long long>(ib + t % nq) * p.blk_nkt + kt] != 0;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < NUSED; ++i) mbar_init(bar0 + 8u * i, (i == PT_FULL || i == PT_FULL + 1) ? 8 : 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot_gen;
  const uint32_t T_ST = tmem, T_DPT = tmem + 128, T_DK = tmem + 256, T_DV = tmem + 384;
  bool aborted = false;

  if (warp == 0) {
    if (elect_one() && nsteps > 0) {
      mbar_expect_tx(bar(KV_FULL, 0), 2 * L::TILE);
      tile_load<DP>(tile(0), &tmK, bar(KV_FULL, 0), k0, kv_head, batch);
      tile_load<DP>(tile(1), &tmV, bar(KV_FULL, 0), k0, kv_head, batch);
      for (int t = 0, n = 0; t < nsteps; ++t) {
        if (!step_live(t)) continue;
        const int st = n & 1;
        const uint32_t ph = (n >> 1) & 1;
        ++n;
        const int head = kv_head * group + t / nq;
        const int q0 = (ib + t % nq) * AB;
        if (!mbar_wait(bar(Q_EMPTY, st), ph ^ 1, p.err, 51)) { aborted = true; break; }
        mbar_expect_tx(bar(Q_FULL, st), 2 * L::TILE + 2 * AB * 4);
        tile_load<DP>(tile(2 + st), &tmQ, bar(Q_FULL, st), q0, head, batch);
        tile_load<DP>(tile(4 + st), &tmDO, bar(Q_FULL, st), q0, head, batch);
        const long long stat0 = (static_cast<long long>(batch) * p.H + head) * p.Sq_pad + q0;
        bulk_load_1d(sbase + L::VEC_OFF + st * (2 * AB * 4), p.lse + stat0, AB * 4, bar(Q_FULL, st));
        bulk_load_1d(sbase + L::VEC_OFF + st * (2 * AB * 4) + AB * 4, p.delta + stat0, AB * 4,
                     bar(Q_FULL, st));
      }
    }
  } else if (warp == 1) {
    if (elect_one() && nsteps > 0) {
      if (!mbar_wait(bar(KV_FULL, 0), 0, p.err, 52)) aborted = true;
      // sub-step u = 2 t + h of live step t: S^T_h = K Q_h^T, dP^T_h = V dO_h^T (64 query rows), later
      // dV += P^T_h dO_h, dK += dS^T_h Q_h
      int nl = 0;
      for (int tt = 0; tt < nsteps; ++tt) nl += step_live(tt) ? 1 : 0;
      auto issue_m1 = [&](int u) -> bool {
        const int t = u >> 1, h = u & 1, st = t & 1;
        if (h == 0 && !mbar_wait(bar(Q_FULL, st), (t >> 1) & 1, p.err, 53)) return false;
        tc_fence_after_sync();
        tile_mma_nt<DP>(T_ST + h * 64, tile(0), tile(2 + st) + h * (64 * 128));
        tile_mma_nt<DP>(T_DPT + h * 64, tile(1), tile(4 + st) + h * (64 * 128));
        umma_commit(bar(ST_FULL, h));
        return true;
      };
      const int nsub = 2 * nl;
      if (!aborted && nsub > 0 && !issue_m1(0)) aborted = true;
      for (int u = 0; u < nsub && !aborted; ++u) {
        const int t = u >> 1, h = u & 1, st = t & 1;
        if (u + 1 < nsub && !issue_m1(u + 1)) { aborted = true; break; }
        if (!mbar_wait(bar(PT_FULL, h), t & 1, p.err, 54)) { aborted = true; break; }
        tc_fence_after_sync();
        tile_mma_ts<DP, true>(T_DV, T_ST + h * 64, tile(4 + st) + h * (64 * 128), u != 0);    // dV += P^T_h dO_h
        tile_mma_ts<DP, true>(T_DK, T_DPT + h * 64, tile(2 + st) + h * (64 * 128), u != 0);   // dK += dS^T_h Q_h
        if (h == 1) umma_commit(bar(Q_EMPTY, st));
      }
      if (!aborted && nl > 0) umma_commit(bar(ACC_DONE, 0));
    }
  } else {
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;   // which 64 of the 128 query columns of a step (and which half of dK / dV)
    const int r = quad * 32 + lane;  // key row in tile
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const int kcol = k0 + r;
    const bool key_ok = kcol < p.Sk;
    int nlive = 0;
    for (int tt = 0; tt < nsteps; ++tt) {
      if (!step_live(tt)) continue;
      const int t = nlive++;
      const int head = kv_head * group + tt / nq;
      const int q0 = (ib + tt % nq) * AB;
      const float slope2 = GEN && p.alibi != nullptr ? p.alibi[head] * LOG2E : 0.f;
      const int st = t & 1;
      // lse / delta of this query block were bulk-copied next to the Q / dO tiles
      bool ok = mbar_wait(bar(Q_FULL, st), (t >> 1) & 1, p.err, 57);
      const float4* v_lse = reinterpret_cast<const float4*>(sgen + L::VEC_OFF + st * (2 * AB * 4));
      const float4* v_del = v_lse + AB / 4;
      // query columns qq (0..127) of this block are alive for lo <= qq <= hi
      const int rel0 = kcol - q0 - off;  // key position minus position of query column 0
      int lo = p.causal ? rel0 : -(1 << 30);
      int hi = p.window >= 0 ? rel0 + p.window : (1 << 30);
      if (!key_ok) hi = -(1 << 30);
      const bool need_mask = __any_sync(0xffffffffu, lo > 0 || hi < AB - 1) || (GEN && p.blk_rows != nullptr);
      const float bias0 = slope2 * static_cast<float>(rel0);
      const uint32_t kbit = 1u << (r >> p.blk_shift);      // this key row's sub-block within the key tile
      const bool plain = !GEN || (!need_mask && p.alibi == nullptr);   // warp-uniform: no per-element compares in the hot path
      // two passes (the halves of the step), one 32-column chunk per warp and pass, each pass with its own S^T / dP^T buffer
      // and barriers
#pragma unroll 1
      for (int grp = 0; grp < 2; ++grp) {
        const int c = grp * 2 + half;                      // 32 query columns of the step
        const uint32_t at = grp * 64 + half * 32;          // columns of the buffers: read, then overwritten from their first
        if (ok) ok = mbar_wait(bar(ST_FULL, grp), t & 1, p.err, 55);
        if (!__all_sync(0xffffffffu, ok)) { aborted = true; break; }
        tc_fence_after_sync();
        uint32_t pp[16], pd[16];
        uint32_t sv[32], dv[32];
        tmem_ld_32x32b_x32(T_ST + at + lane_off, sv);
        tmem_ld_32x32b_x32(T_DPT + at + lane_off, dv);
        tmem_ld_wait();
        float keepf[32];      // DROP: 0 or 1 / (1 - p) per query column of this chunk (unused otherwise)
        if (DROP) {
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const int qq = q0 + c * 32 + j;
            const uint32_t patch = dropout_patch(p.seed_lo, p.seed_hi, static_cast<uint32_t>(batch * p.H + head),
                                                 static_cast<uint32_t>(qq) >> 1, static_cast<uint32_t>(kcol) >> 1);
            keepf[j] = dropout_keep(patch, qq, kcol, p.drop_thr) ? p.drop_rp : 0.f;
            keepf[j + 1] = dropout_keep(patch, qq + 1, kcol, p.drop_thr) ? p.drop_rp : 0.f;
          }
        }
        if (plain) {
          if (!GEN && need_mask) {      // masked scores: -inf, probability 0
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const int idx = c * 32 + j;
              if (idx < lo || idx > hi) sv[j] = __float_as_uint(p.scale_log2 < 0.f ? INFINITY : -INFINITY);
            }
          }
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 l4 = v_lse[(c * 32 + j) >> 2];
            const float4 d4 = v_del[(c * 32 + j) >> 2];
            const float lq[4] = {l4.x, l4.y, l4.z, l4.w}, dq_[4] = {d4.x, d4.y, d4.z, d4.w};
            float pr[4], ds[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              pr[e] = exp2f(fmaf(__uint_as_float(sv[j + e]), p.scale_log2, -lq[e]));
              const float dpe = DROP ? __uint_as_float(dv[j + e]) * keepf[j + e] : __uint_as_float(dv[j + e]);
              ds[e] = pr[e] * (dpe - dq_[e]);     // softmax scale: once, on dK, in the epilogue
              if (DROP) pr[e] *= keepf[j + e];    // dV takes the dropped probabilities
            }
            pp[j >> 1] = pack_h16x2(pr[0], pr[1]);
            pp[(j >> 1) + 1] = pack_h16x2(pr[2], pr[3]);
            pd[j >> 1] = pack_h16x2(ds[0], ds[1]);
            pd[(j >> 1) + 1] = pack_h16x2(ds[2], ds[3]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 l4 = v_lse[(c * 32 + j) >> 2];
            const float4 d4 = v_del[(c * 32 + j) >> 2];
            const float lq[4] = {l4.x, l4.y, l4.z, l4.w}, dq_[4] = {d4.x, d4.y, d4.z, d4.w};
            float pr[4], ds[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int idx = c * 32 + j + e;
              float x = fmaf(__uint_as_float(sv[j + e]), p.scale_log2, -lq[e]);
              if (p.alibi != nullptr) x += fmaf(-slope2, static_cast<float>(idx), bias0);
              pr[e] = exp2f(x);
              if (idx < lo || idx > hi) pr[e] = 0.f;
              if (p.blk_rows != nullptr) {   // the layout byte of query row q0 + idx (the same for the whole warp)
                const int qq = min(q0 + idx, p.Sq - 1);
                if (!(p.blk_rows[static_cast<long long>(qq) * p.blk_nkt + kt] & kbit)) pr[e] = 0.f;
              }
              const float dpe = DROP ? __uint_as_float(dv[j + e]) * keepf[j + e] : __uint_as_float(dv[j + e]);
              ds[e] = pr[e] * (dpe - dq_[e]);
              if (DROP) pr[e] *= keepf[j + e];
            }
            pp[j >> 1] = pack_h16x2(pr[0], pr[1]);
            pp[(j >> 1) + 1] = pack_h16x2(pr[2], pr[3]);
            pd[j >> 1] = pack_h16x2(ds[0], ds[1]);
            pd[(j >> 1) + 1] = pack_h16x2(ds[2], ds[3]);
          }
        }
        tmem_st_32x32b_x16(T_ST + at + lane_off, pp);
        tmem_st_32x32b_x16(T_DPT + at + lane_off, pd);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(PT_FULL, grp));
      }
      if (aborted) break;
    }
    if (!aborted && nlive > 0) {
      if (!mbar_wait(bar(ACC_DONE, 0), 0, p.err, 56)) aborted = true;
      tc_fence_after_sync();
    }
    if (!aborted) {
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        const uint32_t T = which == 0 ? T_DK : T_DV;
        h16* base = which == 0 ? p.dk : p.dv;
        const long long sb = which == 0 ? p.dk_sb : p.dv_sb, sh = which == 0 ? p.dk_sh : p.dv_sh,
                        ss = which == 0 ? p.dk_ss : p.dv_ss;
        h16* orow = base + batch * sb + kv_head * sh + static_cast<long long>(kcol) * ss;
#pragma unroll 1
        for (int c = half * (DP / 64); c < (half + 1) * (DP / 64); ++c) {   // this warp's columns
          uint32_t ov[32];
          if (nlive > 0) {
            tmem_ld_32x32b_x32(T + c * 32 + lane_off, ov);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) ov[j] = 0u;
          }
          if (key_ok) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              if (c * 32 + j < p.D) {
                const float sc = which == 0 ? p.scale : 1.f;     // dK carries the softmax scale of dS
                uint4 o4;
                o4.x = pack_h16x2(__uint_as_float(ov[j]) * sc, __uint_as_float(ov[j + 1]) * sc);
                o4.y = pack_h16x2(__uint_as_float(ov[j + 2]) * sc, __uint_as_float(ov[j + 3]) * sc);
                o4.z = pack_h16x2(__uint_as_float(ov[j + 4]) * sc, __uint_as_float(ov[j + 5]) * sc);
                o4.w = pack_h16x2(__uint_as_float(ov[j + 6]) * sc, __uint_as_float(ov[j + 7]) * sc);
                *reinterpret_cast<uint4*>(orow + c * 32 + j) = o4;
              }
            }
          }
        }
      }
    }
  }
  __syncwarp();
  if (aborted) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

template <typename K>
static int tile_launch(K kern, int dyn, dim3 grid, const BwdMaps& m, const AttnBwdParams& p, cudaStream_t s) {
  NX_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn));
  kern<<<grid, TILE_THREADS, dyn, s>>>(m.q, m.k, m.v, m.d_o, p);
  NX_LAUNCH_CHECK();
  return NX_OK;
}

// (a zero scale would turn a masked score into NaN)
static bool tile_general(const AttnBwdParams& p) { return p.alibi != nullptr || p.blk_rows != nullptr || p.scale == 0.f; }

template <int DP>
static int tile_dq(const BwdMaps& m, const AttnBwdParams& p, cudaStream_t s) {
  const dim3 grid((p.Sq + AB - 1) / AB, p.H, p.B);
  constexpr int dyn = TileSmem<DP>::DYN;
  if (p.drop_thr > 0u) return tile_launch(attn_bwd_tile_dq_kernel<DP, true, true>, dyn, grid, m, p, s);
  if (tile_general(p)) return tile_launch(attn_bwd_tile_dq_kernel<DP, false, true>, dyn, grid, m, p, s);
  return tile_launch(attn_bwd_tile_dq_kernel<DP, false, false>, dyn, grid, m, p, s);
}
template <int DP>
static int tile_dkv(const BwdMaps& m, const AttnBwdParams& p, cudaStream_t s) {
  const dim3 grid((p.Sk + AB - 1) / AB, p.Hk, p.B);
  constexpr int dyn = TileSmem<DP>::DYN;
  if (p.drop_thr > 0u) return tile_launch(attn_bwd_tile_dkv_kernel<DP, true, true>, dyn, grid, m, p, s);
  if constexpr (DP <= 64) {      // (larger heads without dropout, layout and a scale of 0 are persistent)
    if (!tile_general(p)) return tile_launch(attn_bwd_tile_dkv_kernel<DP, false, false>, dyn, grid, m, p, s);
  }
  return tile_launch(attn_bwd_tile_dkv_kernel<DP, false, true>, dyn, grid, m, p, s);
}

int attn_bwd_tile_dq(const BwdMaps& m, const AttnBwdParams& p, cudaStream_t s) {
  return p.D <= 64 ? tile_dq<64>(m, p, s) : tile_dq<128>(m, p, s);
}
int attn_bwd_tile_dkv(const BwdMaps& m, const AttnBwdParams& p, cudaStream_t s) {
  return p.D <= 64 ? tile_dkv<64>(m, p, s) : tile_dkv<128>(m, p, s);
}

}  // namespace nx
