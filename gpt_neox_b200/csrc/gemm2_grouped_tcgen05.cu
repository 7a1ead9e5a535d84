// Grouped (mixture-of-experts) GEMM on CTA pairs: 256 x 256 tiles of tcgen05.mma.cta_group::2 as in gemm2_tcgen05.cu, over
// expert row segments that start at multiples of 256 rows.  Two forms, both without any read of the routing on the host:
//   rows      : C[rows, N] = epilogue(A[rows, K] * op(B_e)), e the expert of the tile's rows (tiles without one are skipped)
//   reduction : C_e[M, N] (+)= A[rows_e, M]^T * B[rows_e, N], the experts' weight gradients
//
// Why pairs: a lone CTA's 128 x 256 x 64 step reads 48 KB of operands from shared memory while as much arrives, which held
// its tensor pipe at 75 - 78 %; a pair stages half of B each.  Sixteen epilogue warps (four per TMEM lane quadrant, 64
// columns each) hide the chains of the activations and the memory behind the side operands better than eight.
// The bound of the 768-deep GEMMs is the SM's shared memory and L1 together: operands arriving and being read take nearly all
// of its bandwidth at the full MMA rate.  A lane that reads or writes its own row takes a cycle for every 32 bytes; through
// boxes of 64 columns in the 128-byte swizzle it is a quarter of that, at the price of the boxes' room (five operand stages
// instead of six) and of a wait between the two results that share a box.  So a GEMM with a side operand goes through boxes,
// one without stores by itself (us, 32,768 rows, both ways: 768 -> 3072 with GeLU and derivative 146 / 182, product with a
// stored derivative 134 / 150; 3072 -> 768 122 / 113, weight gradients 111 / 107).
// The accumulator goes back to the MMA warp as soon as its last columns are in registers, by an arrival that does not release
// the warp's stores: with one that does, it waited for them (178 -> 160 us on average for the first two).
// 32,768 rows over 8 experts, 768 <-> 3072, us, single-CTA tiles of 128 x 256 / here: GeLU and derivative 174 / 144, second
// GEMM 122 / 116, product 150 / 135, its second GEMM 119 / 117, weight gradients 122 / 108 each.  Layers of 64 - 16,384 tokens,
// 4 - 128 experts, 512 - 1024 wide, forward + backward: 1.09 - 1.44 of the rate, also at 16 rows per expert.
#include <string.h>

#include "common.h"
#include "gemm_pair.cuh"
#include "ptx.cuh"

namespace nx {
namespace g2g {

using namespace g2;

constexpr int BM = 128, BN = 256, BNH = 128, BK = 64, UK = 16;
constexpr int EPI_WARPS = 16, THREADS = 64 + 32 * EPI_WARPS;
constexpr int EPI_COLS = BN / (EPI_WARPS / 4);                  // an epilogue warp's share of a tile: 32 rows x 64 columns
constexpr int MAX_EXPERTS = 256;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BNH * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int BOX_BYTES = 32 * EPI_COLS * 2;
// Shared memory: operand stages; with a side operand a box per epilogue warp; barriers, tensor-memory address, experts' order.
template <int SIDE>
struct Smem {
  static constexpr int STAGES = SIDE != 0 ? 5 : 6, BOXES = SIDE != 0 ? EPI_WARPS : 0;
  static constexpr int BOX_OFFSET = STAGES * STAGE_BYTES, BAR_OFFSET = BOX_OFFSET + BOXES * BOX_BYTES;
  static constexpr int SLOT = 2 * STAGES + 4 + BOXES;           // behind the barriers
  static constexpr int ORDER_OFFSET = BAR_OFFSET + SLOT * 8 + 8;
  static constexpr int DYN_BYTES = ORDER_OFFSET + 2 * MAX_EXPERTS + 1024;       // slack to align by hand
  static_assert(DYN_BYTES <= 232448, "shared memory of one SM");
};

// the bits of gemm_tcgen05.cu's epilogues that grouped GEMMs have here
enum Epi : int { GELU_ERF = 2, GELU_TANH = 4, AUX_OUT = 8, DGELU_ERF = 16, DGELU_TANH = 32, ACCUM = 128, OUT_F32 = 256,
                 AUX_DERIV = 1024, MUL_AUX = 2048 };
constexpr int AUX_IN = DGELU_ERF | DGELU_TANH | MUL_AUX;

struct Params {
  int M, N, K;               // reduction form: M, N of one expert's matrix, K = all rows
  void* C;
  long long ldc, c_stride;   // c_stride: elements between two experts' matrices (reduction form)
  int flags;
  bool wide;                 // the result's rows are 32-byte aligned
  int tiles_m, tiles_n, total_tiles;
  int experts, b_rows;       // b_rows: rows of one expert's matrix in the stacked B (rows form)
  const int* tile_expert;    // [rows / 128]
  const int* row_offsets;    // [experts + 1]
  int* err;
};
struct Maps {
  CUtensorMap a, b, out, aux_out, aux_in;      // out, aux_*: with a side operand
};
struct Tile {
  int m0, n0;                // in C (of the expert)
  int b_off, e, kb0, kb1;
};

// Chunk c (16 bytes) of row r of a box, in the 128-byte swizzle of its tensor map: a warp's 16-byte stores do not collide.
__device__ __forceinline__ uint32_t box_chunk(int r, int c) { return r * 128 + ((c ^ (r & 7)) * 16); }
// The pair's tile of round r; false past the last one.  REDUCE: the experts in `order`, the longest reductions first, and every
// other round backwards, so that the pairs' sums of different lengths come out nearly the same.
template <bool REDUCE>
__device__ __forceinline__ bool tile_of(int r, int pair, int pairs, const Params& p, const uint16_t* order, Tile& t, bool& live) {
  const int at = r * pairs + (REDUCE && (r & 1) ? pairs - 1 - pair : pair);
  if (r * pairs >= p.total_tiles) return false;
  live = false;
  if (at >= p.total_tiles) return true;
  int tm, tn;
  if constexpr (REDUCE) {
    const int per = p.tiles_m * p.tiles_n, k = at / per;
    t.e = order[k];
    tile_coords2(at - k * per, p.tiles_m, p.tiles_n, tm, tn);
    t.b_off = 0;
    t.kb0 = p.row_offsets[t.e] / BK;
    t.kb1 = p.row_offsets[t.e + 1] / BK;
    live = t.kb1 > t.kb0;
  } else {
    tile_coords2(at, p.tiles_m, p.tiles_n, tm, tn);
    t.e = p.tile_expert[2 * tm];
    t.b_off = t.e * p.b_rows;
    t.kb0 = 0;
    t.kb1 = (p.K + BK - 1) / BK;
    live = t.e >= 0;
  }
  t.m0 = tm * 2 * BM;
  t.n0 = tn * BN;
  return true;
}

// SIDE: an epilogue with a side operand to write (1) or to read (2).
template <bool REDUCE, bool B_MN, int SIDE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
    grouped2_kernel(const __grid_constant__ Maps maps, const Params p) {
  constexpr bool A_MN = REDUCE;
  using L = Smem<SIDE>;
  constexpr int STAGES = L::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + L::BAR_OFFSET;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tmem_full_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tmem_empty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  auto aux_bar_of = [&](int w) { return bar_base + 8u * (2 * STAGES + 4 + w); };
  const uint32_t tmem_slot = bar_base + 8u * L::SLOT;
  uint16_t* order = reinterpret_cast<uint16_t*>(smem_gen + L::ORDER_OFFSET);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);               // leader: one expect_tx arrival + the bytes of both CTAs
      mbar_init(empty_bar(s), 1);              // one commit to both CTAs per use
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tmem_full_bar(a), 1);
      mbar_init(tmem_empty_bar(a), 2 * EPI_WARPS);       // leader: the epilogue warps of both CTAs
    }
    for (int w = 0; w < L::BOXES; ++w) mbar_init(aux_bar_of(w), 1);
    fence_barrier_init();
  }
  if (REDUCE && threadIdx.x < p.experts) {
    const int e = threadIdx.x, n = p.row_offsets[e + 1] - p.row_offsets[e];
    int before = 0;
    for (int i = 0; i < p.experts; ++i) {
      const int ni = p.row_offsets[i + 1] - p.row_offsets[i];
      before += ni > n || (ni == n && i < e);
    }
    order[before] = static_cast<uint16_t>(e);
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&maps.a);
    tma_prefetch_desc(&maps.b);
  }
  __syncthreads();
  cluster_sync_all();                          // the peer's barriers exist before anything signals them
  if (warp == 1) {
    tmem_alloc2(tmem_slot, 512);               // two 256-column accumulators
    tmem_relinquish2();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem_gen + L::BAR_OFFSET + 8 * L::SLOT);
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  bool aborted = false, live;
  Tile t;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int r = 0; !aborted && tile_of<REDUCE>(r, pair, pairs, p, order, t, live); ++r) {
        if (!live) continue;
        const int m0 = t.m0 + rank * BM, n0 = t.n0 + rank * BNH;
        for (int kb = t.kb0; kb < t.kb1; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1, p.err, 31)) {
            aborted = true;
            break;
          }
          const uint32_t a_dst = smem_base + stage * STAGE_BYTES, b_dst = a_dst + A_BYTES;
          // completion bytes of both CTAs go to the leader's barrier of this stage
          const uint32_t bar = map_to_cta(full_bar(stage), 0);
          if (leader) mbar_expect_tx(full_bar(stage), 2 * STAGE_BYTES);
          const int k0 = kb * BK;
          if constexpr (!A_MN) {
            tma2_load_2d(a_dst, &maps.a, bar, k0, m0);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma2_load_2d(a_dst + j * (BK * 128), &maps.a, bar, m0 + j * 64, k0);
          }
          if constexpr (!B_MN) {
            tma2_load_2d(b_dst, &maps.b, bar, k0, n0 + t.b_off);
          } else {
#pragma unroll
            for (int j = 0; j < BNH / 64; ++j) tma2_load_2d(b_dst + j * (BK * 128), &maps.b, bar, n0 + j * 64, k0 + t.b_off);
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (leader && elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(2 * BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
      constexpr uint32_t A_LBO = A_MN ? BK * 128 : 0, B_LBO = B_MN ? BK * 128 : 0;
      constexpr uint32_t A_KADV = A_MN ? UK * 128 : UK * 2, B_KADV = B_MN ? UK * 128 : UK * 2;
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      for (int r = 0; !aborted && tile_of<REDUCE>(r, pair, pairs, p, order, t, live); ++r) {
        if (!live) continue;
        if (!mbar_wait(tmem_empty_bar(acc), acc_phase ^ 1, p.err, 32)) {
          aborted = true;
          break;
        }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = t.kb0; kb < t.kb1; ++kb) {
          if (!mbar_wait(full_bar(stage), phase, p.err, 33)) {
            aborted = true;
            break;
          }
          tc_fence_after_sync();
          const uint32_t a_addr = smem_base + stage * STAGE_BYTES, b_addr = a_addr + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UK; ++k) {
            const uint64_t adesc = umma_smem_desc_sw128(a_addr + k * A_KADV, A_LBO, 1024);
            const uint64_t bdesc = umma_smem_desc_sw128(b_addr + k * B_KADV, B_LBO, 1024);
            umma2_bf16_ss(d_tmem, adesc, bdesc, idesc, ((kb - t.kb0) | k) != 0 ? 1u : 0u);
          }
          umma2_commit_both(empty_bar(stage));       // frees this stage in both CTAs
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (aborted) break;
        umma2_commit_both(tmem_full_bar(acc));        // accumulator ready in both CTAs
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
    }
  } else if constexpr (SIDE == 0) {
    // ------------------------------------------------------------------ epilogue: a lane has 64 columns of a row of the tile
    const int quad = warp & 3, c0 = ((warp - 2) >> 2) * EPI_COLS;
    const int flags = p.flags;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int r = 0; !aborted && tile_of<REDUCE>(r, pair, pairs, p, order, t, live); ++r) {
      // (reduction form: an expert without rows gets zeros, unless the call adds)
      const bool zeros = REDUCE && !live && !(flags & ACCUM) &&
                         r * pairs + ((r & 1) ? pairs - 1 - pair : pair) < p.total_tiles;
      if (!live && !zeros) continue;
      const int row = t.m0 + rank * BM + quad * 32 + lane, col0 = t.n0 + c0, left = p.N - col0;
      const bool row_ok = row < p.M;
      if (live) {
        const bool ok = mbar_wait(tmem_full_bar(acc), acc_phase, p.err, 34);
        if (!__all_sync(0xffffffffu, ok)) {
          aborted = true;
          break;
        }
        tc_fence_after_sync();
      }
#pragma unroll
      for (int h = 0; h < EPI_COLS / 32; ++h) {
        float v[32];
        __syncwarp();                    // (lanes without a row come here first; what follows is the whole warp's)
        if (live) {
          uint32_t u[32];
          tmem_ld_32x32b_x32(tmem_base + acc * BN + c0 + h * 32 + (static_cast<uint32_t>(quad * 32) << 16), u);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(u[j]);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0.f;
        }
        if (live && h == EPI_COLS / 32 - 1) {
          // the accumulator has been read: tell the leader's MMA thread
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_read(map_to_cta(tmem_empty_bar(acc), 0));
        }
        const int rest = left - 32 * h;
        if (!row_ok || rest <= 0) continue;
        // (the branch on the activation is taken per 32 columns: per value, the values' chains run one after the other.  With
        // AUX_DERIV the activation is rounded as it is next to a stored derivative.)
        if constexpr (!REDUCE) {
          if (flags & GELU_TANH) {
            float d;
            if (flags & AUX_DERIV) {
#pragma unroll
              for (int j = 0; j < 32; ++j) gelu_tanh_both(v[j], v[j], d);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
            }
          } else if (flags & GELU_ERF) {
            float d0, d1;
            if (flags & AUX_DERIV) {
#pragma unroll
              for (int j = 0; j < 32; j += 2) gelu_erf_both2(v[j], v[j + 1], d0, d1);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = gelu_erf(v[j]);
            }
          }
        }
        const long long at = (REDUCE ? t.e * p.c_stride : 0) + row * p.ldc + col0 + 32 * h;
        if (REDUCE && (flags & OUT_F32)) {
          put_f32(static_cast<float*>(p.C) + at, v, rest, flags & ACCUM, p.wide);
        } else {
          h16* cp = static_cast<h16*>(p.C) + at;
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            if (REDUCE && (flags & ACCUM)) {
              uint4 old[2];
              load16(cp + 16 * k, old[0], old[1], rest - 16 * k, p.wide);
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                const uint32_t ow[4] = {old[i].x, old[i].y, old[i].z, old[i].w};
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                  const float2 a = unpack_h16x2(ow[l]);
                  v[16 * k + 8 * i + 2 * l] += a.x;
                  v[16 * k + 8 * i + 2 * l + 1] += a.y;
                }
              }
            }
            store16(cp + 16 * k, pack8(v + 16 * k), pack8(v + 16 * k + 8), rest - 16 * k, p.wide);
          }
        }
      }
      if (live && ++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue with a side operand: 32 rows x 64 columns of a
    // tile per warp, through a box of shared memory that TMA brings in and sends out
    const int w = warp - 2, quad = warp & 3, c0 = (w >> 2) * EPI_COLS;
    uint8_t* box = smem_gen + L::BOX_OFFSET + w * BOX_BYTES;
    const int flags = p.flags;
    constexpr bool aux_in = SIDE == 2, aux_out = SIDE == 1;
    int acc = 0;
    uint32_t acc_phase = 0, aux_phase = 0;
    const uint32_t aux_bar = aux_bar_of(w);
    // the box is written (every lane fences its writes) and goes out as the columns col0 .. of the rows row0 ..
    auto send = [&](const CUtensorMap* m, int col0, int row0) {
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(m, smem_u32(box), col0, row0);
        tma_store_commit();
      }
    };
    auto box_free = [&] {
      if (lane == 0) tma_store_wait_read<0>();
      __syncwarp();
    };
    // the side operand's share of a tile into the box, which nothing uses
    auto fetch_aux = [&](const Tile& a) {
      if (lane == 0) {
        mbar_expect_tx(aux_bar, BOX_BYTES);
        tma_load_2d(smem_u32(box), &maps.aux_in, aux_bar, a.n0 + c0, a.m0 + rank * BM + quad * 32);
      }
    };
    // the next tile of this pair that has work
    int r = -1;
    auto next_tile = [&](Tile& a, bool& a_live) {
      while (tile_of<REDUCE>(++r, pair, pairs, p, order, a, a_live))
        if (a_live) return true;
      return false;
    };
    Tile nx;
    bool nx_live = false, fetched = false;
    for (bool any = next_tile(t, live), more; any && !aborted; t = nx, live = nx_live, any = more) {
      more = next_tile(nx, nx_live);
      const int row0 = t.m0 + rank * BM + quad * 32, col0 = t.n0 + c0;
      const bool mine = col0 < p.N;
      if (aux_in && mine) {
        if (!fetched) {
          if (lane == 0) tma_store_wait_read<0>();
          fetch_aux(t);
        }
        const bool ok = mbar_wait(aux_bar, aux_phase, p.err, 35);
        if (!__all_sync(0xffffffffu, ok)) {
          aborted = true;
          break;
        }
        aux_phase ^= 1;
        fetched = false;
      }
      const bool ok = mbar_wait(tmem_full_bar(acc), acc_phase, p.err, 34);
      if (!__all_sync(0xffffffffu, ok)) {
        aborted = true;
        break;
      }
      tc_fence_after_sync();
      uint4 keep[8];                     // the activation, while the derivative goes out through the box
      if (mine && !aux_in) box_free();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t u[32];
        tmem_ld_32x32b_x32(tmem_base + acc * BN + c0 + h * 32 + (static_cast<uint32_t>(quad * 32) << 16), u);
        tmem_ld_wait();
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(u[j]);
        if (h == 1) {
          // the accumulator has been read: tell the leader's MMA thread
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_read(map_to_cta(tmem_empty_bar(acc), 0));
        }
        if (!mine) continue;
        // (the branch on the activation is taken per 32 columns: per value, the values' chains run one after the other)
        if constexpr (aux_in) {
          auto times = [&](auto f) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint4 side = *reinterpret_cast<const uint4*>(box + box_chunk(lane, 4 * h + k));
              const uint32_t x[4] = {side.x, side.y, side.z, side.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float2 a = unpack_h16x2(x[i]);
                v[8 * k + 2 * i] *= f(a.x);
                v[8 * k + 2 * i + 1] *= f(a.y);
              }
            }
          };
          if (flags & MUL_AUX) times([](float a) { return a; });
          else if (flags & DGELU_ERF) times([](float a) { return gelu_erf_grad(a); });
          else times([](float a) { return gelu_tanh_grad(a); });
        }
        if constexpr (aux_out) {
          // the derivative goes into the box, the activation takes the pre-activation's place; or the pre-activation goes in
          auto both = [&](auto f) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              float d[8];
              f(v + 8 * k, d);
              *reinterpret_cast<uint4*>(box + box_chunk(lane, 4 * h + k)) = pack8(d);
            }
          };
          if (!(flags & AUX_DERIV))
            both([](float* x, float* d) {
#pragma unroll
              for (int j = 0; j < 8; ++j) d[j] = x[j];
            });
          else if (flags & GELU_TANH)
            both([](float* x, float* d) {
#pragma unroll
              for (int j = 0; j < 8; ++j) gelu_tanh_both(x[j], x[j], d[j]);
            });
          else
            both([](float* x, float* d) {
#pragma unroll
              for (int j = 0; j < 8; j += 2) gelu_erf_both2(x[j], x[j + 1], d[j], d[j + 1]);
            });
        }
        if (aux_out && !(flags & AUX_DERIV)) {
          if (flags & GELU_ERF) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = gelu_erf(v[j]);
          } else if (flags & GELU_TANH) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint4 o = pack8(v + 8 * k);
          if (aux_out) keep[4 * h + k] = o;
          else *reinterpret_cast<uint4*>(box + box_chunk(lane, 4 * h + k)) = o;
        }
      }
      if (mine) {
        if (aux_out) {
          send(&maps.aux_out, col0, row0);
          box_free();
#pragma unroll
          for (int k = 0; k < 8; ++k) *reinterpret_cast<uint4*>(box + box_chunk(lane, k)) = keep[k];
        }
        send(&maps.out, col0, row0);
        if (aux_in && more && nx.n0 + c0 < p.N) {
          // (the fence before the store orders every lane's loads from the box, too, before this copy)
          if (lane == 0) tma_store_wait_read<0>();
          fetch_aux(nx);
          fetched = true;
        }
      }
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
    if (lane == 0) tma_store_wait_read<0>();      // shared memory outlives its last reader
  }

  // ------------------------------------------------------------------ teardown
  __syncwarp();
  if (aborted) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();          // nobody leaves while the peer may still signal this CTA's barriers
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc2(tmem_base, 512);
  }
}

template <bool REDUCE, bool B_MN, int SIDE>
static int launch(const Maps& maps, const Params& p, cudaStream_t stream) {
  auto kern = grouped2_kernel<REDUCE, B_MN, SIDE>;
  static bool configured = false;
  if (!configured) {
    NX_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<SIDE>::DYN_BYTES));
    configured = true;
  }
  const int max_pairs = sm_count() / 2, pairs = p.total_tiles < max_pairs ? p.total_tiles : max_pairs;
  kern<<<2 * pairs, THREADS, Smem<SIDE>::DYN_BYTES, stream>>>(maps, p);               // cluster dims are compiled in
  NX_LAUNCH_CHECK();
  return NX_OK;
}

}  // namespace g2g

// Grouped GEMMs over expert row segments that are aligned to 256 rows (the layout the MoE permute kernel writes).
// mode 1: C[rows, N] = A[rows, K] * op(B_e) with B the experts' matrices stacked ([E*N, K] for transB = 0, [E*K, N] for
// transB = 1) and tile_expert[row / 128] -> expert (or -1).  mode 2: per-expert weight gradient C_e[M, N] (+)=
// A[rows_e, M]^T * B[rows_e, N], rows_e = [row_offsets[e], row_offsets[e+1]), K = all rows; C_e = C + e * c_stride; an expert
// without rows gets zeros, or with ACCUM is left as it is.  All tables live on the device: no host synchronisation on the
// routing result.
NX_API int NX_SYM(nx_gemm_bf16_grouped)(int mode, const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                                 long long ldb, long long ldc, int transB, int experts, const void* tile_expert,
                                 const void* row_offsets, long long c_stride, const void* aux_in, void* aux_out,
                                 long long ld_aux, int flags, void* stream_) {
  using namespace g2g;
  if (M <= 0 || N <= 0) return NX_OK;
  const bool reduce = mode == 2;
  NX_REQUIRE(mode == 1 || mode == 2, "gemm2_grouped: mode %d", mode);
  NX_REQUIRE(K > 0 && experts >= 1 && experts <= MAX_EXPERTS, "gemm2_grouped: K %d, %d experts (max %d)", K, experts, MAX_EXPERTS);
  NX_REQUIRE(N % 8 == 0 && lda % 8 == 0 && ldb % 8 == 0, "gemm2_grouped: N / lda / ldb must be multiples of 8");
  NX_REQUIRE(ldc % ((flags & OUT_F32) ? 4 : 8) == 0 && c_stride % ((flags & OUT_F32) ? 4 : 8) == 0, "gemm2_grouped: ldc alignment");
  NX_REQUIRE((reinterpret_cast<uintptr_t>(C) & 15) == 0, "gemm2_grouped: C must be 16-byte aligned");
  if (reduce) {
    NX_REQUIRE(row_offsets != nullptr && (flags & ~(ACCUM | OUT_F32)) == 0, "gemm2_grouped: reduction mode needs the experts' "
               "row offsets and a plain epilogue");
  } else {
    constexpr int known = GELU_ERF | GELU_TANH | AUX_OUT | AUX_DERIV | AUX_IN;
    NX_REQUIRE(tile_expert != nullptr && M % (2 * BM) == 0, "gemm2_grouped: row mode needs a tile->expert table and M %% %d == 0",
               2 * BM);
    NX_REQUIRE((flags & ~known) == 0 && !((flags & AUX_IN) && (flags & (GELU_ERF | GELU_TANH | AUX_OUT | AUX_DERIV))),
               "gemm2_grouped: epilogue flags %d", flags);
    if (flags & AUX_IN)
      NX_REQUIRE(aux_in != nullptr && ld_aux % 8 == 0 && (reinterpret_cast<uintptr_t>(aux_in) & 15) == 0, "gemm2_grouped: aux_in");
    if (flags & AUX_OUT) NX_REQUIRE(aux_out != nullptr && ld_aux % 8 == 0, "gemm2_grouped: aux_out");
  }
  Maps maps;
  memset(&maps, 0, sizeof(maps));
  bool ok;
  if (reduce) {
    ok = make_tma_2d(&maps.a, A, K, M, lda * 2, BK, 64, 2) && make_tma_2d(&maps.b, B, K, N, ldb * 2, BK, 64, 2);
  } else {
    ok = make_tma_2d(&maps.a, A, M, K, lda * 2, BM, BK, 2);
    const long long eb = experts;
    ok = ok && (transB ? make_tma_2d(&maps.b, B, eb * K, N, ldb * 2, BK, 64, 2) : make_tma_2d(&maps.b, B, eb * N, K, ldb * 2, BNH, BK, 2));
    if (flags & (AUX_OUT | AUX_IN)) ok = ok && make_tma_2d(&maps.out, C, M, N, ldc * 2, 32, EPI_COLS, 2);
    if (flags & AUX_OUT) ok = ok && make_tma_2d(&maps.aux_out, aux_out, M, N, ld_aux * 2, 32, EPI_COLS, 2);
    if (flags & AUX_IN) ok = ok && make_tma_2d(&maps.aux_in, aux_in, M, N, ld_aux * 2, 32, EPI_COLS, 2);
  }
  if (!ok) return NX_ERR_ARG;
  Params p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.N = N; p.K = K;
  p.C = C; p.ldc = ldc; p.c_stride = c_stride;
  p.flags = flags;
  p.wide = (reinterpret_cast<uintptr_t>(C) & 31) == 0 && ldc % (flags & OUT_F32 ? 8 : 16) == 0 &&
           c_stride % (flags & OUT_F32 ? 8 : 16) == 0;
  p.tiles_m = (M + 2 * BM - 1) / (2 * BM);
  p.tiles_n = (N + BN - 1) / BN;
  p.experts = experts;
  p.b_rows = transB ? K : N;
  p.tile_expert = static_cast<const int*>(tile_expert);
  p.row_offsets = static_cast<const int*>(row_offsets);
  const long long tiles = static_cast<long long>(p.tiles_m) * p.tiles_n * (reduce ? experts : 1);
  NX_REQUIRE(tiles < (1ll << 30), "gemm2_grouped: too many tiles");
  p.total_tiles = static_cast<int>(tiles);
  p.err = device_error_word();
  auto s = static_cast<cudaStream_t>(stream_);
  if (reduce) return launch<true, true, 0>(maps, p, s);
  if (flags & AUX_OUT) return transB ? launch<false, true, 1>(maps, p, s) : launch<false, false, 1>(maps, p, s);
  if (flags & AUX_IN) return transB ? launch<false, true, 2>(maps, p, s) : launch<false, false, 2>(maps, p, s);
  return transB ? launch<false, true, 0>(maps, p, s) : launch<false, false, 0>(maps, p, s);
}

}  // namespace nx
