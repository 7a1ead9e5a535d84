// C[M, N] = epilogue(A[M, K] * W[N, K]^T) for few rows M (generation steps, short prompts) on tcgen05.
//
// Bound by reading W once.  The 128 x 256 tiles of gemm_tcgen05.cu give such a product ceil(N / 256) CTAs, each walking
// the whole reduction: 16 CTAs of 148 SMs for N = 4096.  Here the roles are swapped: W supplies the 128-row operand of
// the MMA and the few rows of A its N operand (NX = M rounded up to 16 .. 128), so no MMA row is padding, and the
// reduction is cut over the CTAs of a cluster until about two CTAs per SM stream W.  The partial tiles (fp32) meet in
// distributed shared memory in rank order: one launch, no workspace, a result that does not depend on timing.
//
// 4 rows x (4096 -> 22016, 11008 -> 4096): 54 us for both, 5.0 TB/s of weights (164 us before, 1.6 TB/s).
//
// 192 threads: warp 0 TMA producer, warp 1 MMA issuer, warps 2..5 epilogue.  A TMEM lane is a row of W, i.e. a column
// of C: the accumulator goes through shared memory and leaves as 4 columns per thread.
#include "gemm_skinny.h"

#include <cooperative_groups.h>

#include <type_traits>

namespace cg = cooperative_groups;

namespace nx {

constexpr int SK_BW = 128;   // rows of W per tile
constexpr int SK_BK = 64;
constexpr int SK_THREADS = 192;
constexpr int SK_MAX_SPLITS = 8;

// the epilogue bits this kernel knows (same values as in gemm_tcgen05.cu)
enum : int {
  SK_BIAS = 1, SK_GELU_ERF = 2, SK_GELU_TANH = 4, SK_AUX_OUT = 8, SK_RESIDUAL = 64, SK_SCALE = 512, SK_AUX_DERIV = 1024
};

template <int NX, int STAGES>
struct SkinnySmem {
  static constexpr int W_BYTES = SK_BW * SK_BK * 2;
  static constexpr int X_BYTES = NX * SK_BK * 2;
  static constexpr int STAGE = W_BYTES + X_BYTES;
  static constexpr int PART = NX * SK_BW * 4;               // the fp32 partial tile, over the drained ring
  static constexpr int RING = STAGES * STAGE > PART ? STAGES * STAGE : PART;
  static constexpr int BAR_OFF = RING;                      // full[STAGES], empty[STAGES], done, TMEM base
  static constexpr int DYN = BAR_OFF + (2 * STAGES + 2) * 8 + 1024;
};

// Four elements of C (row m, columns n .. n + 3) from their accumulator values.
__device__ __forceinline__ void skinny_store4(const SkinnyParams& p, int m, int n, float4 acc, const float (&bias)[4]) {
  float v[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (p.flags & SK_SCALE) v[j] *= p.alpha;
    v[j] += bias[j];
  }
  const long long aux = m * p.ld_aux + n;
  if (p.flags & SK_AUX_OUT) {
    float d[4] = {v[0], v[1], v[2], v[3]};
    if (p.flags & SK_AUX_DERIV) {       // derivative out, activation in place
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (p.flags & SK_GELU_TANH) gelu_tanh_both(v[j], v[j], d[j]);
        else gelu_erf_both(v[j], v[j], d[j]);
      }
    }
    *reinterpret_cast<uint2*>(p.aux_out + aux) = make_uint2(pack_h16x2(d[0], d[1]), pack_h16x2(d[2], d[3]));
  }
  if (p.flags & SK_AUX_DERIV) {
    if (!(p.flags & SK_AUX_OUT)) {        // the same activation without a place for its derivative
      float unused;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (p.flags & SK_GELU_TANH) gelu_tanh_both(v[j], v[j], unused);
        else gelu_erf_both(v[j], v[j], unused);
      }
    }
  } else {
    if (p.flags & SK_GELU_ERF) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = gelu_erf(v[j]);
    } else if (p.flags & SK_GELU_TANH) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = gelu_tanh(v[j]);
    }
  }
  if (p.flags & SK_RESIDUAL) {
    const uint2 r = *reinterpret_cast<const uint2*>(p.residual + aux);
    const float2 a = unpack_h16x2(r.x), b = unpack_h16x2(r.y);
    v[0] += a.x; v[1] += a.y; v[2] += b.x; v[3] += b.y;
  }
  *reinterpret_cast<uint2*>(p.C + m * p.ldc + n) = make_uint2(pack_h16x2(v[0], v[1]), pack_h16x2(v[2], v[3]));
}

// One product, or two side by side: the tiles from first_tiles on are the second one's.  Clusters are as large as the larger
// number of splits; a CTA beyond its product's splits has no part in it.
template <int COUNT>
struct SkinnyArgs {
  CUtensorMap w[COUNT], x[COUNT];
  SkinnyParams p[COUNT];
  int splits[COUNT], first_tiles;
};

template <int NX, int STAGES, int COUNT>
__global__ void __launch_bounds__(SK_THREADS) gemm_skinny_kernel(const __grid_constant__ SkinnyArgs<COUNT> args) {
  using L = SkinnySmem<NX, STAGES>;
  constexpr uint32_t TMEM_COLS = NX < 32 ? 32 : NX;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - smem_u32(smem_raw));
  auto full_bar = [&](int s) { return sbase + L::BAR_OFF + 8u * s; };
  auto empty_bar = [&](int s) { return sbase + L::BAR_OFF + 8u * (STAGES + s); };
  const uint32_t done_bar = sbase + L::BAR_OFF + 8u * (2 * STAGES);
  const uint32_t tmem_slot = done_bar + 8u;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(sgen + L::BAR_OFF + 8 * (2 * STAGES + 1));
  cg::cluster_group cluster = cg::this_cluster();

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int which = COUNT > 1 && static_cast<int>(blockIdx.y) >= args.first_tiles;
  // (one product's parameters are read where they are: copied, 40 - 60 rows took 1 - 3 % longer)
  const std::conditional_t<COUNT == 1, const SkinnyParams&, SkinnyParams> p = args.p[which];
  const CUtensorMap &tmW = args.w[which], &tmX = args.x[which];
  const int nsplit = COUNT > 1 ? args.splits[which] : gridDim.x, split = blockIdx.x;      // the cluster spans the x dimension
  const bool part_of = COUNT == 1 || split < nsplit;
  const int n0 = (blockIdx.y - (which ? args.first_tiles : 0)) * SK_BW;
  const int num_kb = (p.K + SK_BK - 1) / SK_BK;
  const int kb0 = static_cast<int>(static_cast<long long>(num_kb) * split / nsplit);
  const int kb1 = static_cast<int>(static_cast<long long>(num_kb) * (split + 1) / nsplit);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(done_bar, 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  } else if (warp == 0 && part_of && elect_one()) {
    // the first weights on their way into L2 while the kernel before this one ends (which may even be writing them: what is
    // read later is what L2 has then)
    for (int kb = kb0; kb < kb1 && kb < kb0 + STAGES; ++kb) tma_prefetch_l2_2d(&tmW, kb * SK_BK, n0);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot_gen;
  bool aborted = false;
  grid_dependency_wait();

  if (!part_of) {
    // nothing but the barriers below
  } else if (warp == 0) {
    if (elect_one()) {
      for (int kb = kb0; kb < kb1; ++kb) {
        const int i = kb - kb0, st = i % STAGES;
        if (!mbar_wait(empty_bar(st), ((i / STAGES) & 1) ^ 1, p.err, 70)) { aborted = true; break; }
        mbar_expect_tx(full_bar(st), L::STAGE);
        tma_load_2d(sbase + st * L::STAGE, &tmW, full_bar(st), kb * SK_BK, n0);
        tma_load_2d(sbase + st * L::STAGE + L::W_BYTES, &tmX, full_bar(st), kb * SK_BK, 0);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(SK_BW, NX, 0, 0);
      for (int kb = kb0; kb < kb1; ++kb) {
        const int i = kb - kb0, st = i % STAGES;
        if (!mbar_wait(full_bar(st), (i / STAGES) & 1, p.err, 71)) { aborted = true; break; }
        tc_fence_after_sync();
        const uint32_t w = sbase + st * L::STAGE, x = w + L::W_BYTES;
#pragma unroll
        for (int k = 0; k < SK_BK / 16; ++k)
          umma_bf16_ss(tmem, umma_smem_desc_sw128(w + k * 32, 0, 1024), umma_smem_desc_sw128(x + k * 32, 0, 1024), idesc,
                       (i | k) != 0 ? 1u : 0u);
        umma_commit(empty_bar(st));
      }
      if (!aborted) umma_commit(done_bar);
    }
  }
  // ---- epilogue warps: the accumulator to shared memory as [row of A][row of W], then 4 columns of C per thread
  float* part = reinterpret_cast<float*>(sgen);             // [NX][SK_BW], over the drained ring
  if (warp >= 2 && part_of) {
    const int col = (warp & 3) * 32 + lane;                 // row of W in the tile == TMEM lane
    aborted = !__all_sync(0xffffffffu, mbar_wait(done_bar, 0, p.err, 72));
    tc_fence_after_sync();
    if (!aborted) {
#pragma unroll 1
      for (int c = 0; c < NX && c < p.M; c += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(tmem + c + (static_cast<uint32_t>((warp & 3) * 32) << 16), r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) part[(c + j) * SK_BW + col] = __uint_as_float(r[j]);
      }
    }
  }
  __syncwarp();
  if (aborted) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);       // copies in flight land before the shared memory goes away
  }
  // The next kernel's blocks may come now: while the weights streamed they would take the places that come free first, two on
  // one SM and none on another, and their own prefetches part of the bandwidth (1 row, 4096 -> 22016, one call after the
  // other: 33.3 us when they might come at the start, 29.2 so, 30.5 without overlap; 768 -> 768 3.70, 3.58, 4.69).
  allow_dependents();
  if (gridDim.x > 1) cluster.sync();
  else __syncthreads();
  if (warp >= 2 && part_of && !aborted) {
    const int t = threadIdx.x - 64, n = n0 + (t & 31) * 4;
    if (n < p.N) {
      float bias[4] = {0.f, 0.f, 0.f, 0.f};
      if (p.flags & SK_BIAS) {
#pragma unroll
        for (int j = 0; j < 4; ++j) bias[j] = h16_to_float(p.bias[n + j]);
      }
      // the cluster's CTAs take 4 rows each in turn; the partial tiles are added in rank order, their loads issued together
      for (int m = split * 4 + (t >> 5); m < p.M; m += nsplit * 4) {
        const int at = m * SK_BW + (t & 31) * 4;
        float4 v;
        if (nsplit == 1) {
          v = *reinterpret_cast<const float4*>(part + at);
        } else {
          float4 x[SK_MAX_SPLITS];
#pragma unroll
          for (int r = 0; r < SK_MAX_SPLITS; ++r)
            if (r < nsplit) x[r] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(part, r) + at);
          v = x[0];
#pragma unroll
          for (int r = 1; r < SK_MAX_SPLITS; ++r)
            if (r < nsplit) {
              v.x += x[r].x; v.y += x[r].y; v.z += x[r].z; v.w += x[r].w;
            }
        }
        skinny_store4(p, m, n, v, bias);
      }
    }
  }
  if (gridDim.x > 1) cluster.sync();                        // nobody leaves while its partial tile may still be read
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

// splits: until two CTAs per SM are in flight, with at least four 64-wide steps each
static int skinny_splits(int N, int K) {
  const int tiles = (N + SK_BW - 1) / SK_BW, num_kb = (K + SK_BK - 1) / SK_BK;
  int splits = 1;
  while (splits < SK_MAX_SPLITS && tiles * splits * 2 <= 2 * sm_count() && num_kb >= splits * 2 * 4) splits *= 2;
  return splits;
}

template <int NX, int STAGES, int COUNT>
static int launch_skinny(const SkinnyProduct* q, cudaStream_t stream) {
  using L = SkinnySmem<NX, STAGES>;
  auto kern = gemm_skinny_kernel<NX, STAGES, COUNT>;
  static bool configured = false;
  if (!configured) {
    NX_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::DYN));
    configured = true;
  }
  SkinnyArgs<COUNT> a;
  int tiles = 0, splits = 1;
  for (int i = 0; i < COUNT; ++i) {
    const SkinnyParams& p = q[i].p;
    if (!make_tma_2d(&a.w[i], q[i].B, p.N, p.K, q[i].ldb * 2, SK_BW, SK_BK, 2)) return NX_ERR_ARG;
    if (!make_tma_2d(&a.x[i], q[i].A, p.M, p.K, q[i].lda * 2, NX, SK_BK, 2)) return NX_ERR_ARG;
    a.p[i] = p;
    a.splits[i] = skinny_splits(p.N, p.K);
    splits = a.splits[i] > splits ? a.splits[i] : splits;
    tiles += (p.N + SK_BW - 1) / SK_BW;
    if (i == 0) a.first_tiles = tiles;
  }
  // The launch, the set-up and the first weights' way into L2 lie under the kernel before (7B gated MLP, 4 rows, three launches:
  // 74.6 -> 70.5 us; one query row against 1543 keys, whose kernel is launched the same way, 38.7 -> 37.2 us).
  NX_CUDA_CHECK(launch_dependent(kern, dim3(splits, tiles), dim3(SK_THREADS), L::DYN, stream, splits, a));
  return NX_OK;
}

template <int COUNT>
static int launch_skinny_rows(const SkinnyProduct* q, cudaStream_t stream) {
  // ring depths: two CTAs fit an SM's shared memory
  const int M = q[0].p.M;
  if (M <= 16) return launch_skinny<16, 6, COUNT>(q, stream);
  if (M <= 32) return launch_skinny<32, 5, COUNT>(q, stream);
  if (M <= 64) return launch_skinny<64, 4, COUNT>(q, stream);
  return launch_skinny<128, 3, COUNT>(q, stream);
}

int gemm_skinny_launch(const void* A, const void* B, long long lda, long long ldb, const SkinnyParams& p,
                       cudaStream_t stream) {
  const SkinnyProduct q{A, B, lda, ldb, p};
  return launch_skinny_rows<1>(&q, stream);
}

int gemm_skinny_launch_pair(const SkinnyProduct (&q)[2], cudaStream_t stream) { return launch_skinny_rows<2>(q, stream); }

}  // namespace nx
