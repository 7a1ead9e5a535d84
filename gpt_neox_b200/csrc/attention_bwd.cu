// Flash attention backward on tcgen05 (causal / sliding window / ALiBi / GQA; dropout, block-sparse layouts and small calls:
// attention_bwd_tile.cu).
//
// Three launches, no atomics, no fp32 scratch for dQ, deterministic:
//   1. attn_delta_kernel    delta[b,h,q] = sum_d O * dO
//   2. attn_bwd_dq_kernel   items of 128 query rows: loops over 128-key blocks, recomputes S = Q K^T and dP = dO V^T on
//                           the tensor cores, forms dS = P o (dP - delta) * scale per row (thread == query row), writes
//                           it as 16-bit values into TMEM and accumulates dQ += dS K  (A operand from TMEM).
//   3. attn_bwd_dkv_kernel  items of 128 keys (per kv head; loops over the query heads of the GQA group and over blocks of
//                           64 query rows): the transposed tiles S^T = K Q^T and dP^T = V dO^T, so that thread == key row,
//                           P^T and dS^T as 16-bit values into TMEM, dV += P^T dO and dK += dS^T Q.
// Recomputing S and dP in both kernels costs 7 tile GEMMs instead of 5 but keeps every accumulator in TMEM from first to
// last block.  Counterpart of the flash-attn 2 backward the reference calls through autograd
// (megatron/model/transformer.py:573-690).
//
// Both kernels are persistent, one CTA per SM that walks its share of the items:
//   warp 0      TMA producer: streamed tiles in rings, the next item's resident tiles as soon as the last scores are issued
//   warps 1, 2  tcgen05.mma issuers, one for the scores (which runs ahead, across items), one for the products
//   warps 4 ..  element-wise: dQ eight warps, 64 of a block's key columns each; dK / dV two sets of eight warps (32 query
//               columns each) that take the blocks in turn, so that one set's waits lie under the other's arithmetic.  They also
//               store a finished item's accumulators (a set dK, the other dV), beside the next item's first block.
// What bounds them (cycle counts of the roles): neither the tensor cores nor the exponentials but the chain scores -> registers
// -> 16-bit results -> products, with about 500 cycles from a commit or an arrival to the warp that waits for it, so a block
// costs dQ 2,250 cycles (MMAs 1,536, exponentials 1,024) and dK / dV 1,650 per 64 queries (MMAs 1,024).  Hence everything that
// lets blocks overlap: issuers apart from each other (one thread issuing all was the bound at 1,700 cycles per 64 rows), scores
// and dP ahead, score buffers given back as soon as they are in registers, the next item's tiles and stores in the shadow of
// the running one.
// Batch 4, 32 heads, 2048 x 128 causal: dQ 290 -> 202 us, dK / dV 324 -> 275 us; 5003 tokens, 32 heads on 8, window of 4096:
// 326 -> 229 us and 435 -> 299 us (before: one CTA per tile).  What was slower: two groups of four warps that write their
// results over their scores (260 / 333 us); before dP had two buffers, dQ by 16 warps with 32 columns each (215 us), dQ with two
// K stages (258 us), one V stage (212 us).
#include "attention_bwd.h"
#include "ptx.cuh"
#include "reduce.cuh"

namespace nx {

constexpr int ABS = 64;     // query rows per block of the dK / dV kernel
constexpr int DQ_THREADS = 32 * 12, DKV_THREADS = 32 * 20;

// delta = rowsum(O * dO), 0 in the padding rows [Sq, Sq_pad).  A group of LPR lanes (D / 16 rounded up to a power of two)
// takes a row, 16 elements of each tensor per lane (one 32-byte load where `wide` says that the rows are aligned so).
// blockIdx.z names the batch.  HEADS: the groups walk over the heads of a query row before the next row, so that what a block
// reads lies together where the heads do; else blockIdx.y names the head.
// Bound by reading O and dO.  134 MB (batch 4, 32 heads, 2048 x 128): 33.4 -> 24.9 us; 82 MB (5003 x 32 heads x 128): 20.8 ->
// 13.7 us (before: a head per block, four rows of 16-byte loads per group; 28.7 and 18.1 us with the heads together only, 25.5
// and 14.7 with two rows per group, 28.3 and 16.9 with four).
template <int LPR, bool HEADS>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const h16* __restrict__ o, const h16* __restrict__ dO, float* __restrict__ delta, int H, int Sq,
                  int Sq_pad, int D, long long o_sb, long long o_sh, long long o_ss, long long d_sb, long long d_sh,
                  long long d_ss, bool wide) {
  const int b = blockIdx.z, c = (threadIdx.x % LPR) * 16;
  const unsigned i = blockIdx.x * (256 / LPR) + threadIdx.x / LPR, row = HEADS ? i / static_cast<unsigned>(H) : i;
  const int q = static_cast<int>(row), h = HEADS ? static_cast<int>(i - row * H) : static_cast<int>(blockIdx.y);
  uint4 a[2], g[2];
  a[0] = a[1] = g[0] = g[1] = make_uint4(0u, 0u, 0u, 0u);
  if (q < Sq) {
    load16(o + b * o_sb + h * o_sh + q * o_ss + c, a[0], a[1], D - c, wide);
    load16(dO + b * d_sb + h * d_sh + q * d_ss + c, g[0], g[1], D - c, wide);
  }
  float s[2];
#pragma unroll
  for (int z = 0; z < 2; ++z) {
    const uint32_t aw[4] = {a[z].x, a[z].y, a[z].z, a[z].w}, gw[4] = {g[z].x, g[z].y, g[z].z, g[z].w};
    s[z] = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 x = unpack_h16x2(aw[k]), y = unpack_h16x2(gw[k]);
      s[z] += x.x * y.x + x.y * y.y;
    }
#pragma unroll
    for (int off = LPR / 2; off > 0; off >>= 1) s[z] += __shfl_xor_sync(0xffffffffu, s[z], off);
  }
  if (c == 0 && q < Sq_pad) delta[(static_cast<long long>(b) * H + h) * Sq_pad + q] = s[0] + s[1];
}

// The same for views whose rows are not 16-byte aligned: one warp per row.
__global__ void __launch_bounds__(256)
attn_delta_any_kernel(const h16* __restrict__ o, const h16* __restrict__ dO, float* __restrict__ delta, int H, int Sq,
                      int Sq_pad, int D, long long o_sb, long long o_sh, long long o_ss, long long d_sb, long long d_sh,
                      long long d_ss) {
  const int h = blockIdx.y, b = blockIdx.z, lane = threadIdx.x & 31;
  const int q = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (q >= Sq_pad) return;
  const h16* op = o + b * o_sb + h * o_sh + q * o_ss;
  const h16* dp = dO + b * d_sb + h * d_sh + q * d_ss;
  float s = 0.f;
  if (q < Sq)
    for (int d = lane; d < D; d += 32) s += h16_to_float(op[d]) * h16_to_float(dp[d]);
  s = warp_sum(s);
  if (lane == 0) delta[(static_cast<long long>(b) * H + h) * Sq_pad + q] = s;
}

// Shared memory, in tiles of 64 rows: the resident pair (128 rows each; dQ: Q, dO; dK / dV: K, V), ten tiles of rings (dQ: K in
// three 128-row stages, V in two; dK / dV: Q and dO in four 64-row stages), the streamed rows' lse / delta (dK / dV), barriers.
template <int DP>
struct BwdSmem {
  static constexpr int T64 = 64 * DP * 2;
  static constexpr int STR_OFF = 4 * T64;
  static constexpr int V_OFF = STR_OFF + 6 * T64;              // dQ
  static constexpr int VEC_OFF = STR_OFF + 8 * T64;            // dK / dV: [BWD_STAGES][lse, delta][64]
  static constexpr int BAR_OFF = STR_OFF + 10 * T64;
  static constexpr int TOTAL = BAR_OFF + 27 * 8;               // 26 barriers and the TMEM base word
  static constexpr int DYN = TOTAL + 1024;
};
constexpr int BWD_STAGES = 4;
static_assert(BwdSmem<128>::DYN <= 232448, "shared memory of one SM");
static_assert(BWD_STAGES * 2 * 64 * 4 <= 2 * BwdSmem<64>::T64, "lse / delta fit behind the ring");

// Barriers.  RES: the two resident tiles; STR / STR2: rings of streamed tiles (STR2: V of the dQ kernel); S: scores of block n
// in buffer n & 1 (dQ: one buffer) written by the tensor core (FULL), in the element-wise warps' registers (EMPTY); DP: dP in
// buffer n & 1 written; P_FULL: the 16-bit results of block n written, in dP's place.  That these are consumed STR_EMPTY
// tells: the products of a block are its stage's last readers.  ACC: an item's accumulators complete / read.
enum { RES_FULL = 0, RES_EMPTY = 2, STR_FULL = 4, STR_EMPTY = 8, STR2_FULL = 12, STR2_EMPTY = 14, S_FULL = 16, S_EMPTY = 18,
       DP_FULL = 20, P_FULL = 22, ACC_FULL = 24, ACC_EMPTY = 25, BWD_NBAR = 26 };
__device__ __forceinline__ void bwd_init_barriers(uint32_t bar0, int element_warps) {
  for (int i = 0; i < BWD_NBAR; ++i) {
    const bool by_warps = i == S_EMPTY || i == S_EMPTY + 1 || i == P_FULL || i == P_FULL + 1;
    // one arrival per element-wise warp that shares a block; of all of them
    mbar_init(bar0 + 8u * i, by_warps ? 8 : i == ACC_EMPTY ? element_warps : 1);
  }
  fence_barrier_init();
}

// Loads ROWS rows (contiguous in d) of one tensor as boxes of 64 rows x 64 columns, swizzled; 64-column panels are ROWS *
// 128 bytes apart.
template <int DP, int ROWS>
__device__ __forceinline__ void load_rows(uint32_t dst, const CUtensorMap* m, uint32_t bar, int row0, int head, int batch) {
#pragma unroll
  for (int c = 0; c < DP / 64; ++c)
#pragma unroll
    for (int r = 0; r < ROWS; r += 64) tma_load_4d(dst + c * (ROWS * 128) + r * 128, m, bar, c * 64, row0 + r, head, batch);
}
// The two issuing warps run converged and only the instructions themselves are predicated on one lane: the descriptors then
// live in uniform registers, where a single diverged lane pays moves for every operand.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, int* err, int where) {
  const bool ok = mbar_wait(bar, parity, err, where);
  return __all_sync(0xffffffffu, ok);
}
// D[128 x N] = A[128 x DP] * B[N x DP]^T, both K-major (head dim contiguous).
template <int DP, int N>
__device__ __forceinline__ void mma_nt(uint32_t leader, uint32_t d_tmem, uint32_t a, uint32_t b) {
  constexpr uint32_t idesc = umma_idesc_bf16(AB, N, 0, 0);
  const uint32_t al = umma_desc_lo(a, 0), bl = umma_desc_lo(b, 0);
#pragma unroll
  for (int k = 0; k < DP / 16; ++k)
    umma_bf16_ss_by(leader, d_tmem, al + ((k >> 2) * (AB * 128) + (k & 3) * 32) / 16,
                    bl + ((k >> 2) * (N * 128) + (k & 3) * 32) / 16, idesc, k != 0 ? 1u : 0u);
}
// D[128 x DP] (+)= A_tmem[128 x KR (16 bit)] * B[KR x DP] with B's head dim contiguous (MN-major B operand).  The KR / 2
// columns of A lie in two halves, `gap` columns from the first of one to the first of the other.
template <int DP, int KR>
__device__ __forceinline__ void mma_ts(uint32_t leader, uint32_t d_tmem, uint32_t a_tmem, int gap, uint32_t b, bool accumulate) {
  constexpr uint32_t idesc = umma_idesc_bf16(AB, DP, 0, 1);
  const uint32_t bl = umma_desc_lo(b, KR * 128);
#pragma unroll
  for (int k = 0; k < KR / 16; ++k)
    umma_bf16_ts_by(leader, d_tmem, a_tmem + (k >= KR / 32 ? gap + (k - KR / 32) * 8 : k * 8), bl + k * (2048 / 16), idesc,
                    (accumulate || k != 0) ? 1u : 0u);
}

// One piece of work: 128 rows of one head and its streamed blocks [j0, j1).
struct BwdItem {
  int tile, head, batch, j0, j1;
  int n_i;      // dK / dV: query blocks per head (block j: query head j / n_i of the group)
  int i0;       // dK / dV: first of them
};

// Which items a CTA takes: the longest first (causal), dealt out forwards and backwards in turn, so that a CTA which got a
// longer item in one round gets a shorter one in the next.
struct BwdOrder {
  int total;
  __device__ __forceinline__ bool next(int& r, int& w) const {
    const int G = gridDim.x, c = blockIdx.x;
    do {
      ++r;
      if (r * G >= total) return false;
      w = r * G + ((r & 1) ? G - 1 - c : c);
    } while (w >= total);
    return true;
  }
};

struct DqWork {
  const AttnBwdParams& p;
  BwdOrder order;
  int nt;
  __device__ __forceinline__ explicit DqWork(const AttnBwdParams& p_) : p(p_) {
    nt = (p.Sq + AB - 1) / AB;
    order.total = nt * p.H * p.B;
  }
  __device__ __forceinline__ bool next(int& r, BwdItem& it) const {
    int w;
    if (!order.next(r, w)) return false;
    const int hb = p.H * p.B, q = w / hb;
    w -= q * hb;
    it.tile = nt - 1 - q;
    it.batch = w / p.H;
    it.head = w - it.batch * p.H;
    const int q0 = it.tile * AB, off = p.Sk - p.Sq;
    const int kv_end = p.causal ? min(p.Sk, q0 + AB + off) : p.Sk;
    const int kv_begin = p.window >= 0 ? max(0, q0 + off - p.window) : 0;
    it.j0 = kv_begin / AB;
    it.j1 = max((kv_end + AB - 1) / AB, it.j0);
    return true;
  }
};
struct DkvWork {
  const AttnBwdParams& p;
  BwdOrder order;
  int group;
  __device__ __forceinline__ explicit DkvWork(const AttnBwdParams& p_) : p(p_) {
    group = p.H / p.Hk;
    order.total = (p.Sk + AB - 1) / AB * p.Hk * p.B;
  }
  __device__ __forceinline__ bool next(int& r, BwdItem& it) const {
    int w;
    if (!order.next(r, w)) return false;
    const int hb = p.Hk * p.B;
    it.tile = w / hb;
    w -= it.tile * hb;
    it.batch = w / p.Hk;
    it.head = w - it.batch * p.Hk;
    const int k0 = it.tile * AB, off = p.Sk - p.Sq;
    // query rows that can see this key tile: qpos >= k0 (causal), qpos <= k_last + window
    const int q_begin = p.causal ? max(0, k0 - off) : 0;
    const int q_end = p.window >= 0 ? min(p.Sq, k0 + AB + p.window - off) : p.Sq;
    it.i0 = q_begin / ABS;
    it.n_i = max((q_end + ABS - 1) / ABS - it.i0, 0);
    it.j0 = 0;
    it.j1 = it.n_i * group;
    return true;
  }
};

// Waits for this warp's TMEM loads; their registers pass through it, so that no use can move in front of it.
__device__ __forceinline__ void tmem_ld_wait_for(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
                 "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
                 "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29])
               :
               : "memory");
  asm volatile("" : "+r"(r[30]), "+r"(r[31]));
}

// A warp's 32 rows x 64 columns of a finished accumulator (zeros where the item had no block): scaled, rounded, transposed in
// pieces of 16 bytes within groups of eight lanes and stored, a group a whole row of 128 bytes.  Written by each lane to its own
// row, every store touched 32 lines, and an item's held up the element-wise warps for 3,800 cycles.
__device__ __forceinline__ void bwd_acc_load(uint32_t tmem_cols, uint32_t (&lo)[32], uint32_t (&hi)[32]) {
  tmem_ld_32x32b_x32(tmem_cols, lo);
  tmem_ld_32x32b_x32(tmem_cols + 32, hi);
  tmem_ld_wait_for(lo);
  tmem_ld_wait_for(hi);
}
__device__ __forceinline__ void bwd_store(h16* base, long long row_stride, const uint32_t (&lo)[32], const uint32_t (&hi)[32],
                                          float sc, int col, int row, int rows, int D) {
  const int lane = threadIdx.x & 31;
  uint32_t w[8][4];
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int e = (c & 3) * 8 + 2 * k;
      const uint32_t x = c < 4 ? lo[e] : hi[e], y = c < 4 ? lo[e + 1] : hi[e + 1];
      w[c][k] = pack_h16x2(__uint_as_float(x) * sc, __uint_as_float(y) * sc);
    }
#pragma unroll
  for (int m = 4; m > 0; m >>= 1) {
    const bool up = lane & m;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (c & m) continue;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? w[c][k] : w[c | m][k], m);
        if (up) w[c][k] = got;
        else w[c | m][k] = got;
      }
    }
  }
  // w[k]: piece lane % 8 of row (lane / 8) * 8 + k
  const int c8 = col + (lane & 7) * 8, r0 = row + (lane & ~7);
  if (c8 < D) {
    h16* o = base + r0 * row_stride + c8;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (r0 + k < rows) *reinterpret_cast<uint4*>(o + k * row_stride) = make_uint4(w[k][0], w[k][1], w[k][2], w[k][3]);
  }
  __syncwarp();
}

// ------------------------------------------------------------------------------------------------
// dQ kernel.  Resident: Q, dO (128 rows).  Streamed: K, V (128 rows).  An element-wise warp has 64 of a block's key columns, in
// two chunks of 32; dS goes over the first half of the dP columns the warp itself has read.
// TMEM: S [0, 128), dP of block n at [128 + 128 (n & 1), ...), dQ [384, 384 + DP).  The single buffer is the scores', which
// are read as soon as they are there: a single one of dP, held from the first chunk's read to the second's, took 206 us (now
// 202; 243 -> 229 with a window, 131 -> 121 with heads of 64; ALiBi 0.97 - 1.04 of the rate).
// Without ALIBI (this kernel and the next) a block that needs a mask differs from one that does not by one select per element.
// ------------------------------------------------------------------------------------------------
template <int DP, bool ALIBI>
__global__ void __launch_bounds__(DQ_THREADS, 1)
    attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                       const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                       const __grid_constant__ AttnBwdParams p) {
  using L = BwdSmem<DP>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - smem_u32(smem_raw));
  const uint32_t bar0 = sbase + L::BAR_OFF;
  auto bar = [&](int which, int idx) { return bar0 + 8u * (which + idx); };
  const uint32_t tmem_slot = bar0 + 8u * BWD_NBAR;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(sgen + L::BAR_OFF + 8 * BWD_NBAR);
  auto res = [&](int which) { return sbase + which * (2 * L::T64); };
  auto kst = [&](int stage) { return sbase + L::STR_OFF + stage * (2 * L::T64); };
  auto vst = [&](int stage) { return sbase + L::V_OFF + stage * (2 * L::T64); };
  constexpr uint32_t T_DP = 128, T_DQ = 384;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int off = p.Sk - p.Sq;
  const DqWork work(p);
  if (threadIdx.x == 0) bwd_init_barriers(bar0, 8);
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot_gen;
  bool aborted = false;

  if (warp == 0) {
    if (elect_one()) {
      int n = 0, t = 0, round = -1, ks = 0;
      uint32_t kph = 0;
      BwdItem it;
      while (!aborted && work.next(round, it)) {
        const int kv_head = it.head / (p.H / p.Hk);
        bool any = false;
        for (int j = it.j0; j < it.j1; ++j) {
          const int vs = n & 1;
          if (!mbar_wait(bar(STR_EMPTY, ks), kph ^ 1, p.err, 32)) { aborted = true; break; }
          mbar_expect_tx(bar(STR_FULL, ks), 2 * L::T64);
          load_rows<DP, AB>(kst(ks), &tmK, bar(STR_FULL, ks), j * AB, kv_head, it.batch);
          if (!any) {
            for (int w = 0; w < 2 && !aborted; ++w) {
              if (!mbar_wait(bar(RES_EMPTY, w), (t & 1) ^ 1, p.err, 31)) { aborted = true; break; }
              mbar_expect_tx(bar(RES_FULL, w), 2 * L::T64);
              load_rows<DP, AB>(res(w), w == 0 ? &tmQ : &tmDO, bar(RES_FULL, w), it.tile * AB, it.head, it.batch);
            }
            any = true;
            ++t;
          }
          if (aborted || !mbar_wait(bar(STR2_EMPTY, vs), ((n >> 1) & 1) ^ 1, p.err, 37)) { aborted = true; break; }
          mbar_expect_tx(bar(STR2_FULL, vs), 2 * L::T64);
          load_rows<DP, AB>(vst(vs), &tmV, bar(STR2_FULL, vs), j * AB, kv_head, it.batch);
          ++n;
          if (++ks == 3) {
            ks = 0;
            kph ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // S = Q K^T, dP = dO V^T
    const uint32_t leader = elect_one() ? 1u : 0u;
    int n = 0, t = 0, round = -1, ks = 0;
    uint32_t kph = 0;
    BwdItem it;
    while (!aborted && work.next(round, it)) {
      bool any = false;
      for (int j = it.j0; j < it.j1; ++j) {
        const bool last = j + 1 == it.j1;
        const int st = n & 1;
        const uint32_t ph = (n >> 1) & 1;
        if ((!any && !warp_wait(bar(RES_FULL, 0), t & 1, p.err, 34)) || !warp_wait(bar(STR_FULL, ks), kph, p.err, 35) ||
            !warp_wait(bar(S_EMPTY, 0), (n & 1) ^ 1, p.err, 43)) {
          aborted = true;
          break;
        }
        tc_fence_after_sync();
        mma_nt<DP, AB>(leader, tmem, res(0), kst(ks));
        umma_commit_by(leader, bar(S_FULL, 0));
        if (last) umma_commit_by(leader, bar(RES_EMPTY, 0));
        // (dP buffer n & 1 is free when dQ has taken dS of block n - 2: its stage is two back in the ring of three)
        if ((!any && !warp_wait(bar(RES_FULL, 1), t & 1, p.err, 45)) || !warp_wait(bar(STR2_FULL, st), ph, p.err, 36) ||
            (n >= 2 && !warp_wait(bar(STR_EMPTY, ks < 2 ? ks + 1 : 0), ks < 2 ? kph ^ 1 : kph, p.err, 39))) {
          aborted = true;
          break;
        }
        tc_fence_after_sync();
        mma_nt<DP, AB>(leader, tmem + T_DP + st * AB, res(1), vst(st));
        umma_commit_by(leader, bar(DP_FULL, st));
        umma_commit_by(leader, bar(STR2_EMPTY, st));
        if (last) umma_commit_by(leader, bar(RES_EMPTY, 1));
        any = true;
        ++n;
        if (++ks == 3) {
          ks = 0;
          kph ^= 1;
        }
      }
      t += any;
    }
  } else if (warp == 2) {
    // dQ += dS K
    const uint32_t leader = elect_one() ? 1u : 0u;
    int n = 0, t = 0, round = -1, ks = 0;
    BwdItem it;
    while (!aborted && work.next(round, it)) {
      bool any = false;
      for (int j = it.j0; j < it.j1; ++j) {
        if ((!any && !warp_wait(bar(ACC_EMPTY, 0), (t & 1) ^ 1, p.err, 33)) ||
            !warp_wait(bar(P_FULL, n & 1), (n >> 1) & 1, p.err, 41)) {
          aborted = true;
          break;
        }
        tc_fence_after_sync();
        mma_ts<DP, AB>(leader, tmem + T_DQ, tmem + T_DP + (n & 1) * AB, 64, kst(ks), any);
        umma_commit_by(leader, bar(STR_EMPTY, ks));
        any = true;
        ++n;
        if (++ks == 3) ks = 0;
      }
      if (any) {
        umma_commit_by(leader, bar(ACC_FULL, 0));
        ++t;
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ element-wise warps
    const int quad = warp & 3, c0 = ((warp - 4) >> 2) * 64;      // first of this warp's 64 key columns of a block
    const int r = quad * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_s = tmem + c0 + lane_off, t_dp = t_s + T_DP;
    int n = 0, round = -1, t = 0;
    BwdItem it;
    bool pending = false;      // `done`: an item whose dQ this warp has still to store
    BwdItem done;
    const bool stores = c0 < DP;      // (64 columns of dQ per warp)
    auto finish = [&](const BwdItem& i, bool live) -> bool {
      uint32_t lo[32], hi[32];
#pragma unroll
      for (int e = 0; e < 32; ++e) lo[e] = hi[e] = 0u;
      if (live) {
        const bool ok = mbar_wait(bar(ACC_FULL, 0), t & 1, p.err, 40);
        if (!__all_sync(0xffffffffu, ok)) return false;
        tc_fence_after_sync();
        if (stores) bwd_acc_load(tmem + T_DQ + c0 + lane_off, lo, hi);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(ACC_EMPTY, 0));
        ++t;
      }
      const int row = i.tile * AB + quad * 32;
      if (stores)
        bwd_store(p.dq + i.batch * p.dq_sb + i.head * p.dq_sh, p.dq_ss, lo, hi, p.scale, c0, row, p.Sq, p.D);
      return true;
    };
    auto stat_of = [&](const BwdItem& i) {
      return (static_cast<long long>(i.batch) * p.H + i.head) * p.Sq_pad + i.tile * AB + r;
    };
    auto wait = [&](int which, int idx, uint32_t parity, int where) -> bool {
      const bool ok = mbar_wait(bar(which, idx), parity, p.err, where);
      const bool all = __all_sync(0xffffffffu, ok);
      tc_fence_after_sync();
      return all;
    };
    bool have = work.next(round, it);
    float lse2 = 0.f, delta = 0.f;     // lse: +inf for rows past Sq -> P = 0
    if (have) {
      lse2 = p.lse[stat_of(it)];
      delta = p.delta[stat_of(it)];
    }
    while (have && !aborted) {
      BwdItem nx;
      const bool have_nx = work.next(round, nx);
      float lse2_nx = 0.f, delta_nx = 0.f;
      if (have_nx) {      // in flight during this item
        lse2_nx = p.lse[stat_of(nx)];
        delta_nx = p.delta[stat_of(nx)];
      }
      const int q0 = it.tile * AB, qi = q0 + r, qpos = qi + off;
      const float slope2 = ALIBI ? p.alibi[it.head] * LOG2E : 0.f;
      // scores of the 32 keys from k0 on -> probabilities, in place
      auto probs = [&](uint32_t (&sv)[32], int k0) {
        const bool need_mask = (k0 + 32 > p.Sk) || (p.causal && k0 + 31 > q0 + quad * 32 + off) ||
                               (p.window >= 0 && k0 < q0 + quad * 32 + 31 + off - p.window);
        // columns e (0..31) are alive for lo <= e <= hi
        const int rel0 = k0 - qpos;
        int hi = p.Sk - k0 - 1;
        if (p.causal) hi = min(hi, -rel0);
        const int lo = p.window >= 0 ? -rel0 - p.window : -(1 << 30);
        if (!ALIBI) {
          if (need_mask) {      // masked scores: -inf, probability 0
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (e < lo || e > hi) sv[e] = __float_as_uint(p.scale_log2 < 0.f ? INFINITY : -INFINITY);
          }
          const float2 sc2 = make_float2(p.scale_log2, p.scale_log2), nl2 = make_float2(-lse2, -lse2);
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const float2 x = ffma2(u2f2(sv[e], sv[e + 1]), sc2, nl2);
            sv[e] = __float_as_uint(exp2f(x.x));
            sv[e + 1] = __float_as_uint(exp2f(x.y));
          }
        } else {
          const float bias0 = slope2 * static_cast<float>(rel0) - lse2;  // folded into the exponent
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const float x = fmaf(__uint_as_float(sv[e]), p.scale_log2, fmaf(slope2, static_cast<float>(e), bias0));
            float pr = exp2f(x);
            if (e < lo || e > hi) pr = 0.f;
            sv[e] = __float_as_uint(pr);
          }
        }
      };
      // probabilities, dP -> dS (16 bit); the softmax scale is applied once, to dQ, when it is stored
      auto grads = [&](const uint32_t (&pr)[32], const uint32_t (&dv)[32], uint32_t (&pk)[16]) {
        const float2 nd2 = make_float2(-delta, -delta);
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const float2 d = fmul2(u2f2(pr[e], pr[e + 1]), fadd2(u2f2(dv[e], dv[e + 1]), nd2));
          pk[e >> 1] = pack_h16x2(d.x, d.y);
        }
      };
      uint32_t sa[32], sb[32], dv[32], pk[16];
      int j = it.j0;
      const bool live = j < it.j1;
      bool first = true;
      while (j < it.j1) {
        const int k0 = j * AB + c0;
        const uint32_t t_dn = t_dp + (n & 1) * AB;
        if (!wait(S_FULL, 0, n & 1, 38)) { aborted = true; break; }
        tmem_ld_32x32b_x32(t_s, sa);
        tmem_ld_32x32b_x32(t_s + 32, sb);
        tmem_ld_wait_for(sa);
        tmem_ld_wait_for(sb);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(S_EMPTY, 0));
        probs(sa, k0);
        if (!wait(DP_FULL, n & 1, (n >> 1) & 1, 44)) { aborted = true; break; }
        tmem_ld_32x32b_x32(t_dn, dv);           // in flight during the second chunk's exponentials
        probs(sb, k0 + 32);
        tmem_ld_wait_for(dv);
        grads(sa, dv, pk);
        tmem_ld_32x32b_x32(t_dn + 32, dv);
        tmem_st_32x32b_x16(t_dn, pk);
        tmem_ld_wait_for(dv);
        grads(sb, dv, pk);
        tmem_st_32x32b_x16(t_dn + 16, pk);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(P_FULL, n & 1));
        ++n;
        ++j;
        // the former item's dQ
        if (first && pending && !finish(done, true)) { aborted = true; break; }
        first = false;
      }
      if (!aborted) {
        if (live) {
          done = it;
          pending = true;
        } else {
          finish(it, false);
        }
      }
      it = nx;
      have = have_nx;
      lse2 = lse2_nx;
      delta = delta_nx;
    }
    if (!aborted && pending && !finish(done, true)) aborted = true;
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
// dK / dV kernel.  Resident: K, V (128 rows).  Streamed: Q, dO (64 rows) with their lse / delta.  Two sets of eight element-wise
// warps (32 query columns each) take the blocks in turn, so that one set's waits lie under the other's arithmetic.
// TMEM: S^T of block n at [64 (n & 1), ...), dP^T [128 + 64 (n & 1), ...), dK [256, 256 + DP), dV [384, 384 + DP).  A warp's P^T and
// dS^T (16 columns each) take the place of its own 32 columns of dP^T, which thus has two buffers as the scores have: with one, and
// one pair for the results, two chains of two handoffs each held a block (294 us, batch 4, 32 heads, 2048 x 128 causal; now 275;
// results in the place of the scores, three buffers of them and one of dP^T 287).  What bounds a block now is the element-wise
// warps: a set is busy for 2,600 cycles of a block of its own, 1,300 per block, at 8 cycles an instruction.
// ------------------------------------------------------------------------------------------------
template <int DP, bool ALIBI>
__global__ void __launch_bounds__(DKV_THREADS, 1)
    attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                        const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                        const __grid_constant__ AttnBwdParams p) {
  using L = BwdSmem<DP>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - smem_u32(smem_raw));
  const uint32_t bar0 = sbase + L::BAR_OFF;
  auto bar = [&](int which, int idx) { return bar0 + 8u * (which + idx); };
  const uint32_t tmem_slot = bar0 + 8u * BWD_NBAR;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(sgen + L::BAR_OFF + 8 * BWD_NBAR);
  auto res = [&](int which) { return sbase + which * (2 * L::T64); };
  auto str = [&](int stage, int which) { return sbase + L::STR_OFF + (stage * 2 + which) * L::T64; };
  constexpr uint32_t T_DP = 128, T_DK = 256, T_DV = 384;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int off = p.Sk - p.Sq;
  const DkvWork work(p);
  if (threadIdx.x == 0) bwd_init_barriers(bar0, 16);
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot_gen;
  bool aborted = false;

  if (warp == 0) {
    if (elect_one()) {
      int st = 0, t = 0, round = -1;
      uint32_t ph = 0;
      BwdItem it;
      while (!aborted && work.next(round, it)) {
        bool any = false;
        int g = 0, ib = it.i0 - 1;
        for (int j = 0; j < it.j1; ++j) {
          if (++ib == it.i0 + it.n_i) {
            ib = it.i0;
            ++g;
          }
          const int q0 = ib * ABS, head = it.head * work.group + g;
          if (!mbar_wait(bar(STR_EMPTY, st), ph ^ 1, p.err, 52)) { aborted = true; break; }
          mbar_expect_tx(bar(STR_FULL, st), 2 * L::T64 + 2 * ABS * 4);
          load_rows<DP, ABS>(str(st, 0), &tmQ, bar(STR_FULL, st), q0, head, it.batch);
          load_rows<DP, ABS>(str(st, 1), &tmDO, bar(STR_FULL, st), q0, head, it.batch);
          const long long stat0 = (static_cast<long long>(it.batch) * p.H + head) * p.Sq_pad + q0;
          const uint32_t vec = sbase + L::VEC_OFF + st * (2 * ABS * 4);
          bulk_load_1d(vec, p.lse + stat0, ABS * 4, bar(STR_FULL, st));
          bulk_load_1d(vec + ABS * 4, p.delta + stat0, ABS * 4, bar(STR_FULL, st));
          if (!any) {
            for (int w = 0; w < 2; ++w) {
              if (!mbar_wait(bar(RES_EMPTY, w), (t & 1) ^ 1, p.err, 51)) { aborted = true; break; }
              mbar_expect_tx(bar(RES_FULL, w), 2 * L::T64);
              load_rows<DP, AB>(res(w), w == 0 ? &tmK : &tmV, bar(RES_FULL, w), it.tile * AB, it.head, it.batch);
            }
            if (aborted) break;
            any = true;
            ++t;
          }
          if (++st == BWD_STAGES) {
            st = 0;
            ph ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // S^T = K Q^T, dP^T = V dO^T
    const uint32_t leader = elect_one() ? 1u : 0u;
    int n = 0, t = 0, round = -1, st = 0;
    uint32_t ph = 0;
    BwdItem it;
    while (!aborted && work.next(round, it)) {
      bool any = false;
      for (int j = 0; j < it.j1; ++j) {
        const bool last = j + 1 == it.j1;
        if ((!any && !warp_wait(bar(RES_FULL, 0), t & 1, p.err, 53)) || !warp_wait(bar(STR_FULL, st), ph, p.err, 54) ||
            !warp_wait(bar(S_EMPTY, n & 1), ((n >> 1) & 1) ^ 1, p.err, 60)) {
          aborted = true;
          break;
        }
        tc_fence_after_sync();
        mma_nt<DP, ABS>(leader, tmem + (n & 1) * ABS, res(0), str(st, 0));
        umma_commit_by(leader, bar(S_FULL, n & 1));
        if (last) umma_commit_by(leader, bar(RES_EMPTY, 0));
        // (the products of block n - 2: its stage, two back in the ring, and the phase of that use)
        if ((!any && !warp_wait(bar(RES_FULL, 1), t & 1, p.err, 64)) ||
            (n >= 2 && !warp_wait(bar(STR_EMPTY, (n - 2) % BWD_STAGES), ((n - 2) / BWD_STAGES) & 1, p.err, 62))) {
          aborted = true;
          break;
        }
        tc_fence_after_sync();
        mma_nt<DP, ABS>(leader, tmem + T_DP + (n & 1) * ABS, res(1), str(st, 1));
        umma_commit_by(leader, bar(DP_FULL, n & 1));
        if (last) umma_commit_by(leader, bar(RES_EMPTY, 1));
        any = true;
        ++n;
        if (++st == BWD_STAGES) {
          st = 0;
          ph ^= 1;
        }
      }
      t += any;
    }
  } else if (warp == 2) {
    // dV += P^T dO, dK += dS^T Q
    const uint32_t leader = elect_one() ? 1u : 0u;
    int n = 0, t = 0, round = -1, st = 0;
    BwdItem it;
    while (!aborted && work.next(round, it)) {
      bool any = false;
      for (int j = 0; j < it.j1; ++j) {
        const uint32_t t_p = tmem + T_DP + (n & 1) * ABS;
        if ((!any && !warp_wait(bar(ACC_EMPTY, 0), (t & 1) ^ 1, p.err, 55)) ||
            !warp_wait(bar(P_FULL, n & 1), (n >> 1) & 1, p.err, 56)) {
          aborted = true;
          break;
        }
        tc_fence_after_sync();
        mma_ts<DP, ABS>(leader, tmem + T_DV, t_p, 32, str(st, 1), any);
        mma_ts<DP, ABS>(leader, tmem + T_DK, t_p + 16, 32, str(st, 0), any);
        umma_commit_by(leader, bar(STR_EMPTY, st));
        any = true;
        ++n;
        if (++st == BWD_STAGES) st = 0;
      }
      if (any) {
        umma_commit_by(leader, bar(ACC_FULL, 0));
        ++t;
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ element-wise sets
    const int quad = warp & 3, h = (warp - 4) >> 3, half = (warp >> 2) & 1;
    const int r = quad * 32 + lane, c0 = half * 32;      // key row in tile; first of this warp's 32 query columns of a block
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_s = tmem + h * ABS + c0 + lane_off, t_dp = t_s + T_DP;
    int n = 0, round = -1, t = 0, st = 0;
    uint32_t ph = 0;
    BwdItem it;
    bool pending = false;      // `done`: an item whose gradients this warp has still to store
    BwdItem done;
    // 64 columns per warp, of dK (set 0; it carries the softmax scale of dS) or of dV (set 1: one set that stored both was the later
    // one, at 11 % of its time)
    const bool stores = half * 64 < DP;
    auto finish = [&](const BwdItem& i, bool live) -> bool {
      uint32_t lo[32], hi[32];
#pragma unroll
      for (int e = 0; e < 32; ++e) lo[e] = hi[e] = 0u;
      if (live) {
        const bool ok = mbar_wait(bar(ACC_FULL, 0), t & 1, p.err, 59);
        if (!__all_sync(0xffffffffu, ok)) return false;
        tc_fence_after_sync();
        if (stores) bwd_acc_load(tmem + (h == 0 ? T_DK : T_DV) + half * 64 + lane_off, lo, hi);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(ACC_EMPTY, 0));
        ++t;
      }
      if (stores) {
        h16* out = h == 0 ? p.dk + i.batch * p.dk_sb + i.head * p.dk_sh : p.dv + i.batch * p.dv_sb + i.head * p.dv_sh;
        bwd_store(out, h == 0 ? p.dk_ss : p.dv_ss, lo, hi, h == 0 ? p.scale : 1.f, half * 64, i.tile * AB + quad * 32, p.Sk, p.D);
      }
      return true;
    };
    auto wait = [&](int which, int idx, uint32_t parity, int where) -> bool {
      const bool ok = mbar_wait(bar(which, idx), parity, p.err, where);
      const bool all = __all_sync(0xffffffffu, ok);
      tc_fence_after_sync();
      return all;
    };
    while (!aborted && work.next(round, it)) {
      const int kcol = it.tile * AB + r;
      const bool key_ok = kcol < p.Sk;
      bool first = true;
      int g = 0, ib = it.i0 - 1;
      for (int j = 0; j < it.j1; ++j) {
        if (++ib == it.i0 + it.n_i) {
          ib = it.i0;
          ++g;
        }
        const int i = n++, cur = st;
        const uint32_t cur_ph = ph;
        if (++st == BWD_STAGES) {
          st = 0;
          ph ^= 1;
        }
        // the former item's gradients: before this item's first block where the other set has it, else after it
        const bool store_former = first && pending;
        first = false;
        if ((i & 1) != h) {
          if (store_former && !finish(done, true)) { aborted = true; break; }
          continue;
        }
        const int q0 = ib * ABS + c0, head = it.head * work.group + g;      // this warp's first query row
        const float slope2 = ALIBI ? p.alibi[head] * LOG2E : 0.f;
        // this warp's query columns e (0..31) are alive for lo <= e <= hi
        const int rel0 = kcol - q0 - off;  // key position minus position of query column 0
        const int lo = p.causal ? rel0 : -(1 << 30);
        int hi = p.window >= 0 ? rel0 + p.window : (1 << 30);
        if (!key_ok) hi = -(1 << 30);
        const bool need_mask = __any_sync(0xffffffffu, lo > 0 || hi < 31);
        const uint32_t par = (i >> 1) & 1;
        // (lse / delta of a query block were bulk-copied next to the Q / dO tiles)
        const float4* v_lse = reinterpret_cast<const float4*>(sgen + L::VEC_OFF + cur * (2 * ABS * 4)) + c0 / 4;
        const float4* v_del = v_lse + ABS / 4;
        uint32_t sv[32], dv[32], pk[16];
        if (!wait(STR_FULL, cur, cur_ph, 57) || !wait(S_FULL, h, par, 58)) { aborted = true; break; }
        tmem_ld_32x32b_x32(t_s, sv);
        tmem_ld_wait_for(sv);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(S_EMPTY, h));
        // probabilities, in place; dV takes them rounded
        if (!ALIBI && need_mask) {      // masked scores: -inf, probability 0
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (e < lo || e > hi) sv[e] = __float_as_uint(p.scale_log2 < 0.f ? INFINITY : -INFINITY);
        }
        auto probs = [&](int first_e) {
          if (!ALIBI) {
            const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
#pragma unroll
            for (int z = 0; z < 16; z += 4) {
              const int e = first_e + z;
              const float4 l4 = v_lse[e >> 2];
              const float2 x0 = ffma2(u2f2(sv[e], sv[e + 1]), sc2, make_float2(-l4.x, -l4.y));
              const float2 x1 = ffma2(u2f2(sv[e + 2], sv[e + 3]), sc2, make_float2(-l4.z, -l4.w));
              const float p0 = exp2f(x0.x), p1 = exp2f(x0.y), p2 = exp2f(x1.x), p3 = exp2f(x1.y);
              pk[e >> 1] = pack_h16x2(p0, p1);
              pk[(e >> 1) + 1] = pack_h16x2(p2, p3);
              sv[e] = __float_as_uint(p0); sv[e + 1] = __float_as_uint(p1);
              sv[e + 2] = __float_as_uint(p2); sv[e + 3] = __float_as_uint(p3);
            }
          } else {
            const float bias0 = slope2 * static_cast<float>(rel0);
#pragma unroll
            for (int z = 0; z < 16; z += 4) {
              const int e0 = first_e + z;
              const float4 l4 = v_lse[e0 >> 2];
              const float lq[4] = {l4.x, l4.y, l4.z, l4.w};
              float kept[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int idx = e0 + e;
                const float x = fmaf(__uint_as_float(sv[idx]), p.scale_log2, -lq[e]) +
                                fmaf(-slope2, static_cast<float>(idx), bias0);
                float pr = exp2f(x);
                if (need_mask && (idx < lo || idx > hi)) pr = 0.f;
                sv[idx] = __float_as_uint(pr);
                kept[e] = pr;
              }
              pk[e0 >> 1] = pack_h16x2(kept[0], kept[1]);
              pk[(e0 >> 1) + 1] = pack_h16x2(kept[2], kept[3]);
            }
          }
        };
        probs(0);
        if (!wait(DP_FULL, h, par, 63)) { aborted = true; break; }
        tmem_ld_32x32b_x32(t_dp, dv);           // in flight during the second half's exponentials
        probs(16);
        tmem_ld_wait_for(dv);
        uint32_t pd[16];
        const float2 m1 = make_float2(-1.f, -1.f);
#pragma unroll
        for (int e = 0; e < 32; e += 4) {      // softmax scale: once, on dK, when it is stored
          const float4 d4 = v_del[e >> 2];
          const float2 s0 = fmul2(u2f2(sv[e], sv[e + 1]), ffma2(make_float2(d4.x, d4.y), m1, u2f2(dv[e], dv[e + 1])));
          const float2 s1 = fmul2(u2f2(sv[e + 2], sv[e + 3]), ffma2(make_float2(d4.z, d4.w), m1, u2f2(dv[e + 2], dv[e + 3])));
          pd[e >> 1] = pack_h16x2(s0.x, s0.y);
          pd[(e >> 1) + 1] = pack_h16x2(s1.x, s1.y);
        }
        tmem_st_32x32b_x16(t_dp, pk);
        tmem_st_32x32b_x16(t_dp + 16, pd);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(P_FULL, h));
        if (store_former && !finish(done, true)) { aborted = true; break; }
      }
      if (!aborted) {
        if (!first) {
          done = it;
          pending = true;
        } else {
          finish(it, false);
        }
      }
    }
    if (!aborted && pending && !finish(done, true)) aborted = true;
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

static bool bwd_map(CUtensorMap* m, const void* base, int B, int Hh, int S, int D, long long sb,
                    long long sh, long long ss, int rows) {
  const uint64_t dims[4] = {(uint64_t)D, (uint64_t)S, (uint64_t)Hh, (uint64_t)B};
  const uint64_t strides[3] = {(uint64_t)ss * 2, (uint64_t)sh * 2, (uint64_t)sb * 2};
  const uint32_t box[4] = {64, (uint32_t)rows, 1, 1};
  return make_tma_4d(m, base, dims, strides, box, 2, true);
}

// Which kernels a call takes: persistent ones or one CTA per tile (attention_bwd_tile.cu).  Persistent CTAs overlap one item
// with the next, so they need more items than SMs; a single item costs them 1 - 4 us more (more roles, barriers and
// threads to set up).  Measured over 64 .. 2048 tokens x 4 .. 1536 heads, time per tile / persistent:
//   dropout      0.5 (registers spill);  block-sparse layouts 0.7 - 1 (a CTA's share is fixed, and tiles are of any length).  A
//                softmax scale of 0, which makes a masked score NaN in the other forms, goes with them
//   dQ, ALiBi    0.93 - 2.7: always persistent
//   dQ, 128      more items than SMs 1.13 - 1.66; fewer, 256 keys and more 0.98 - 1.15, fewer keys 0.86 - 1.17
//   dQ, 64       causal, more items than SMs 1.01 - 1.63; rows of 65 .. 128 keys 0.98 below 2 items per SM, 1.05 - 1.19 above,
//                of 64 keys 0.91 - 0.98 and 1.05 from 9 on; not causal 0.88 - 1.02 up to 4 items per SM, then 0.97 - 1.25
//   dK / dV, 128 and ALiBi  more items than SMs 1.15 - 1.9, fewer 0.98 - 1.2: always persistent
//   dK / dV, 64  fewer items than SMs 0.91 - 1.02, but 1.08 - 1.17 with 300 queries (blocks of 64 queries waste less of a ragged
//                end than tiles of 128); more: causal 1.11 - 1.65; not causal up to 1023 queries 1.06 - 1.41, with more 1.05 -
//                1.11 above 5 items per SM and 0.94 - 1.0 below, 4096 queries 0.98 (queries times the query heads of a key head)
struct BwdRoute {
  long long dq_items, dkv_items;
  bool dq, dkv;      // persistent
};
static BwdRoute attn_bwd_route(const AttnBwdParams& p) {
  BwdRoute r;
  r.dq_items = static_cast<long long>((p.Sq + AB - 1) / AB) * p.H * p.B;
  r.dkv_items = static_cast<long long>((p.Sk + AB - 1) / AB) * p.Hk * p.B;
  r.dq = r.dkv = false;
  if (p.drop_thr > 0u || p.blk_rows != nullptr || p.scale == 0.f) return r;
  const bool alibi = p.alibi != nullptr;
  const int sms = sm_count();
  if (alibi) r.dq = true;
  else if (p.D > 64) r.dq = r.dq_items > sms || p.Sk >= 256;
  else r.dq = r.dq_items > (!p.causal ? 4 : p.Sk > AB ? 1 : p.Sk > ABS ? 2 : 9) * sms;
  const bool many = r.dkv_items > 5 * sms;
  const long long rows = static_cast<long long>(p.Sq) * (p.H / p.Hk);      // an item's queries
  r.dkv = p.D > 64 || alibi || (r.dkv_items > sms && (p.causal || rows < 1024 || (many && rows < 4096)));
  return r;
}

template <typename Smem, typename K>
static int persistent_launch(K kern, int threads, long long items, const BwdMaps& m, const AttnBwdParams& p, cudaStream_t s) {
  NX_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem::DYN));
  kern<<<static_cast<unsigned>(min(items, static_cast<long long>(sm_count()))), threads, Smem::DYN, s>>>(m.q, m.k, m.v, m.d_o, p);
  NX_LAUNCH_CHECK();
  return NX_OK;
}

template <int DP, bool ALIBI>
static int launch_bwd(const BwdMaps (&m)[2], const AttnBwdParams& p, const BwdRoute& r, cudaStream_t s) {
  const int rc = r.dq ? persistent_launch<BwdSmem<DP>>(attn_bwd_dq_kernel<DP, ALIBI>, DQ_THREADS, r.dq_items, m[0], p, s)
                      : attn_bwd_tile_dq(m[1], p, s);
  if (rc != NX_OK) return rc;
  return r.dkv ? persistent_launch<BwdSmem<DP>>(attn_bwd_dkv_kernel<DP, ALIBI>, DKV_THREADS, r.dkv_items, m[0], p, s)
               : attn_bwd_tile_dkv(m[1], p, s);
}

}  // namespace nx

// Views as in nx_flash_attn_fwd (element strides batch, head, seq).  delta: fp32 scratch [B,H,Sq_pad] (Sq rounded up to
// 128) provided by the caller, written whole.  dq/dk/dv: 16-bit strided outputs, fully overwritten.  dropout_p / seed: the
// values the forward was given; blk_rows / blk_any / blk_size: the forward's block-sparse layout tables.
NX_API int NX_SYM(nx_flash_attn_bwd)(const void* q, const void* k, const void* v, const void* o, const void* dO,
                             const void* lse, void* delta, void* dq, void* dk, void* dv,
                             const void* alibi, int B, int H, int Hk, int Sq, int Sk, int D,
                             long long q_sb, long long q_sh, long long q_ss, long long k_sb,
                             long long k_sh, long long k_ss, long long v_sb, long long v_sh,
                             long long v_ss, long long o_sb, long long o_sh, long long o_ss,
                             long long do_sb, long long do_sh, long long do_ss, long long dq_sb,
                             long long dq_sh, long long dq_ss, long long dk_sb, long long dk_sh,
                             long long dk_ss, long long dv_sb, long long dv_sh, long long dv_ss,
                             float scale, int causal, int window, float dropout_p,
                             unsigned long long seed, const void* blk_rows, const void* blk_any, int blk_size,
                             void* stream_) {
  using namespace nx;
  if (B == 0 || H == 0 || Sq == 0 || Sk == 0) return NX_OK;
  NX_REQUIRE((blk_rows == nullptr) == (blk_any == nullptr), "flash_attn_bwd: both block-layout tables or none");
  NX_REQUIRE(blk_rows == nullptr || blk_size == 16 || blk_size == 32 || blk_size == 64 || blk_size == 128,
             "flash_attn_bwd: block-sparse layouts need a block size of 16, 32, 64 or 128 (got %d)", blk_size);
  NX_REQUIRE(dropout_p >= 0.f && dropout_p < 1.f, "flash_attn_bwd: dropout probability %f outside [0, 1)", dropout_p);
  NX_REQUIRE(D % 8 == 0 && D <= 128 && D > 0, "flash_attn_bwd: head dim %d unsupported", D);
  NX_REQUIRE(Hk > 0 && H % Hk == 0, "flash_attn_bwd: H=%d not a multiple of Hk=%d", H, Hk);
  auto aligned = [](const void* ptr, long long a, long long b, long long c) {
    return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0 && a % 8 == 0 && b % 8 == 0 && c % 8 == 0;
  };
  NX_REQUIRE(aligned(dq, dq_sb, dq_sh, dq_ss) && aligned(dk, dk_sb, dk_sh, dk_ss) &&
                 aligned(dv, dv_sb, dv_sh, dv_ss),
             "flash_attn_bwd: gradient views must be 16-byte aligned");
  auto s = (cudaStream_t)stream_;
  {
    const int sq_pad = (Sq + AB - 1) / AB * AB;
    const bool vec = ((o_sb | o_sh | o_ss | do_sb | do_sh | do_ss) % 8) == 0 &&
                     ((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(dO)) & 15) == 0;
    // heads of a query row next to one another in both tensors (the views of attention layers) or not
    const bool heads = o_sh < o_ss && do_sh < do_ss && static_cast<long long>(sq_pad) * H < (1ll << 30);
    auto wide_rows = [](const void* ptr, long long sb, long long sh, long long ss) {
      return (reinterpret_cast<uintptr_t>(ptr) & 31) == 0 && ((sb | sh | ss) % 16) == 0;
    };
    const bool wide = wide_rows(o, o_sb, o_sh, o_ss) && wide_rows(dO, do_sb, do_sh, do_ss);
    auto run = [&](auto kern, bool flat, int rows_per_block, auto... more) {
      kern<<<dim3(((flat ? sq_pad * H : sq_pad) + rows_per_block - 1) / rows_per_block, flat ? 1 : H, B), 256, 0, s>>>(
          (const h16*)o, (const h16*)dO, (float*)delta, H, Sq, sq_pad, D, o_sb, o_sh, o_ss, do_sb, do_sh, do_ss, more...);
    };
    if (!vec) run(attn_delta_any_kernel, false, 8);
    else if (D <= 64 && heads) run(attn_delta_kernel<4, true>, true, 64, wide);
    else if (D <= 64) run(attn_delta_kernel<4, false>, false, 64, wide);
    else if (heads) run(attn_delta_kernel<8, true>, true, 32, wide);
    else run(attn_delta_kernel<8, false>, false, 32, wide);
    NX_LAUNCH_CHECK();
  }
  AttnBwdParams p;
  p.lse = (const float*)lse; p.delta = (const float*)delta; p.alibi = (const float*)alibi;
  p.dq = (h16*)dq; p.dk = (h16*)dk; p.dv = (h16*)dv;
  p.dq_sb = dq_sb; p.dq_sh = dq_sh; p.dq_ss = dq_ss;
  p.dk_sb = dk_sb; p.dk_sh = dk_sh; p.dk_ss = dk_ss;
  p.dv_sb = dv_sb; p.dv_sh = dv_sh; p.dv_ss = dv_ss;
  p.B = B; p.H = H; p.Hk = Hk; p.Sq = Sq; p.Sk = Sk; p.D = D;
  p.Sq_pad = (Sq + AB - 1) / AB * AB;
  p.scale = scale; p.scale_log2 = scale * LOG2E;
  p.causal = causal; p.window = window;
  p.err = device_error_word();
  p.drop_thr = static_cast<uint32_t>(dropout_p * 256.f + 0.5f);
  if (p.drop_thr > 255u) p.drop_thr = 255u;
  p.drop_rp = 256.f / static_cast<float>(256u - p.drop_thr);
  p.seed_lo = static_cast<uint32_t>(seed);
  p.seed_hi = static_cast<uint32_t>(seed >> 32);
  p.blk_rows = static_cast<const uint8_t*>(blk_rows);
  p.blk_any = static_cast<const uint8_t*>(blk_any);
  p.blk_nkt = (Sk + AB - 1) / AB;
  p.blk_shift = blk_size == 16 ? 4 : blk_size == 32 ? 5 : blk_size == 64 ? 6 : 7;
  const BwdRoute route = attn_bwd_route(p);
  BwdMaps m[2];      // for persistent kernels and for one CTA per tile
  for (int t = 0; t < 2; ++t) {
    if (t == 0 ? !route.dq && !route.dkv : route.dq && route.dkv) continue;
    const int rows = t == 0 ? ABS : AB;
    if (!bwd_map(&m[t].q, q, B, H, Sq, D, q_sb, q_sh, q_ss, rows) || !bwd_map(&m[t].k, k, B, Hk, Sk, D, k_sb, k_sh, k_ss, rows) ||
        !bwd_map(&m[t].v, v, B, Hk, Sk, D, v_sb, v_sh, v_ss, rows) ||
        !bwd_map(&m[t].d_o, dO, B, H, Sq, D, do_sb, do_sh, do_ss, rows))
      return NX_ERR_ARG;
  }
  NX_REQUIRE(route.dq_items < (1ll << 30) && route.dkv_items < (1ll << 30), "flash_attn_bwd: too many tiles");
  if (alibi != nullptr) return D <= 64 ? launch_bwd<64, true>(m, p, route, s) : launch_bwd<128, true>(m, p, route, s);
  return D <= 64 ? launch_bwd<64, false>(m, p, route, s) : launch_bwd<128, false>(m, p, route, s);
}
