// Attention of ONE query row per (batch, head) against Sk keys (cached generation; the query is the last position, so
// causality masks nothing and a sliding window only moves the first key).
//
// Bound by the K / V bytes: a query row does 4 flops per 4 bytes it reads, far below the machine's balance, and the
// tiled kernel of attention_fwd.cu spends a 128-row MMA tile, and one CTA for all keys of a head, on one row.
// Here the keys of a head are cut over the CTAs of a cluster and, inside a CTA, over groups of DP / 8 lanes: a lane
// owns 8 head dims (one 16-byte load of a K row, one of a V row) and a group takes UNROLL keys at a time.  The next keys'
// K rows are loaded as soon as the scores of these have been taken, the next V rows after the sums, into the registers
// just freed: loads are in flight throughout.  GT query heads that share a K / V head are done from the same loads.  Every
// group keeps its own running maximum / sum / output in fp32 registers; groups meet through shuffles and shared memory,
// CTAs of a cluster through distributed shared memory in rank order, so there is one launch, no workspace, and the result
// does not depend on timing.  8 sequences, 32 heads of 128, 1543 keys: 35.9 us, 5.6 TB/s (39.7 us with the tiled kernel and its
// fill; 52.6 us with loads only at the head of the loop).
#include "attention_decode.h"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace nx {

constexpr int DEC_THREADS = 128;
constexpr int DEC_WARPS = DEC_THREADS / 32;
constexpr int DEC_MAX_SPLITS = 8;   // portable cluster size

// (not ld.global.nc: this step's key and value row may still be written when the kernel begins)
__device__ __forceinline__ uint4 ld_stream(const h16* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// (m, l, o) of two disjoint key sets -> of their union; a set without keys has m = -inf, l = 0, o = 0.
__device__ __forceinline__ void merge_scale(float m, float m_new, float& a) {
  a = m == -INFINITY ? 0.f : exp2f(m - m_new);
}

// CTAs per SM the register budget allows: the loads in flight, not the arithmetic, set the rate
constexpr int dec_ctas(int gt) { return gt == 1 ? 6 : gt == 2 ? 4 : gt == 4 ? 3 : 2; }

template <int DP, int GT>
__global__ void __launch_bounds__(DEC_THREADS, dec_ctas(GT)) attn_decode_kernel(const AttnDecodeParams p, int keys_per_cta,
                                                                                 bool early) {
  constexpr int LPK = DP / 8;                 // lanes per key
  constexpr int GPW = 32 / LPK;               // key groups per warp
  constexpr int NG = DEC_WARPS * GPW;         // key groups per CTA
  constexpr int UNROLL = GT <= 2 ? 4 : 2;
  __shared__ float s_o[DEC_WARPS][GT][DP];    // after the merge: [0] holds this CTA's o
  __shared__ float s_m[DEC_WARPS][GT], s_l[DEC_WARPS][GT], c_m[GT], c_l[GT];
  cg::cluster_group cluster = cg::this_cluster();
  const int nsplit = gridDim.x, split = blockIdx.x;     // the cluster spans the x dimension
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = warp * GPW + lane / LPK, dl = (lane % LPK) * 8;
  const int G = p.H / p.Hk, per_kv = G / GT;
  const int kvh = blockIdx.y / per_kv, head0 = kvh * G + (blockIdx.y % per_kv) * GT, b = blockIdx.z;
  const bool live = dl < p.D;                 // D below DP: the last lanes of a group hold zeros
  if (early) allow_dependents();
  grid_dependency_wait();

  constexpr bool Q16 = GT >= 4;               // many heads: q stays packed, 4 registers a head
  uint32_t qp[Q16 ? GT : 1][4];
  float2 q[Q16 ? 1 : GT][4], o[GT][4];
  float m[GT], l[GT], slope[GT];
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    uint4 u = make_uint4(0u, 0u, 0u, 0u);
    if (live) u = *reinterpret_cast<const uint4*>(p.q + b * p.q_sb + (head0 + g) * p.q_sh + dl);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (Q16) qp[Q16 ? g : 0][i] = w[i];
      else q[Q16 ? 0 : g][i] = unpack_h16x2(w[i]);
      o[g][i] = make_float2(0.f, 0.f);
    }
    m[g] = -INFINITY;
    l[g] = 0.f;
    slope[g] = p.alibi != nullptr ? p.alibi[head0 + g] * 1.4426950408889634f : 0.f;
  }
  const h16* kp = p.k + b * p.k_sb + kvh * p.k_sh + dl;
  const h16* vp = p.v + b * p.v_sb + kvh * p.v_sh + dl;
  const int lo = p.key_lo + split * keys_per_cta, hi = min(lo + keys_per_cta, p.Sk);

  uint4 ku[UNROLL], vu[UNROLL];
  auto load = [&](uint4 (&r)[UNROLL], const h16* p0, long long stride, int base) {
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int key = base + u * NG;
      r[u] = make_uint4(0u, 0u, 0u, 0u);
      if (live && key < hi) r[u] = ld_stream(p0 + key * stride);
    }
  };
  load(ku, kp, p.k_ss, lo + grp);
  load(vu, vp, p.v_ss, lo + grp);
#pragma unroll 1
  for (int base = lo + grp; base - grp < hi; base += NG * UNROLL) {     // the same trip count for every group
    float s[GT][UNROLL];
#pragma unroll
    for (int g = 0; g < GT; ++g) {
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        auto qv = [&](int i) { return Q16 ? unpack_h16x2(qp[Q16 ? g : 0][i]) : q[Q16 ? 0 : g][i]; };
        float2 a = fmul2(qv(0), unpack_h16x2(ku[u].x));
        a = ffma2(qv(1), unpack_h16x2(ku[u].y), a);
        a = ffma2(qv(2), unpack_h16x2(ku[u].z), a);
        a = ffma2(qv(3), unpack_h16x2(ku[u].w), a);
        float d = a.x + a.y;
#pragma unroll
        for (int x = LPK / 2; x > 0; x >>= 1) d += __shfl_xor_sync(0xffffffffu, d, x);
        const int key = base + u * NG;
        s[g][u] = key < hi ? fmaf(slope[g], static_cast<float>(key - (p.Sk - 1)), d * p.scale_log2) : -INFINITY;
      }
    }
    load(ku, kp, p.k_ss, base + NG * UNROLL);
#pragma unroll
    for (int g = 0; g < GT; ++g) {
      float mx = m[g];
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) mx = fmaxf(mx, s[g][u]);
      const float msub = mx == -INFINITY ? 0.f : mx;
      const float alpha = exp2f(m[g] - msub);           // m = -inf: 0
      m[g] = mx;
      l[g] *= alpha;
      const float2 a2 = make_float2(alpha, alpha);
#pragma unroll
      for (int i = 0; i < 4; ++i) o[g][i] = fmul2(o[g][i], a2);
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const float pr = exp2f(s[g][u] - msub);
        l[g] += pr;
        const float2 p2 = make_float2(pr, pr);
        o[g][0] = ffma2(p2, unpack_h16x2(vu[u].x), o[g][0]);
        o[g][1] = ffma2(p2, unpack_h16x2(vu[u].y), o[g][1]);
        o[g][2] = ffma2(p2, unpack_h16x2(vu[u].z), o[g][2]);
        o[g][3] = ffma2(p2, unpack_h16x2(vu[u].w), o[g][3]);
      }
    }
    load(vu, vp, p.v_ss, base + NG * UNROLL);
  }
  // ---- groups of a warp -> one (m, l, o) per warp, in shared memory
#pragma unroll
  for (int g = 0; g < GT; ++g) {
#pragma unroll
    for (int x = LPK; x < 32; x <<= 1) {
      const float m2 = __shfl_xor_sync(0xffffffffu, m[g], x), l2 = __shfl_xor_sync(0xffffffffu, l[g], x);
      const float mn = fmaxf(m[g], m2);
      float a, c;
      merge_scale(m[g], mn, a);
      merge_scale(m2, mn, c);
      l[g] = l[g] * a + l2 * c;
      m[g] = mn;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        o[g][i].x = o[g][i].x * a + __shfl_xor_sync(0xffffffffu, o[g][i].x, x) * c;
        o[g][i].y = o[g][i].y * a + __shfl_xor_sync(0xffffffffu, o[g][i].y, x) * c;
      }
    }
    if (lane < LPK) {
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<float2*>(&s_o[warp][g][dl + 2 * i]) = o[g][i];
      if (lane == 0) {
        s_m[warp][g] = m[g];
        s_l[warp][g] = l[g];
      }
    }
  }
  __syncthreads();
  // ---- warps -> this CTA's value: o in slot 0 (a thread reads its column of every slot before it writes there), m and l
  // in arrays of their own
  for (int i = threadIdx.x; i < GT * DP; i += DEC_THREADS) {
    const int g = i / DP, d = i % DP;
    float mn = -INFINITY, acc = 0.f, ls = 0.f;
    for (int w = 0; w < DEC_WARPS; ++w) mn = fmaxf(mn, s_m[w][g]);
    for (int w = 0; w < DEC_WARPS; ++w) {
      float a;
      merge_scale(s_m[w][g], mn, a);
      acc += a * s_o[w][g][d];
      ls += a * s_l[w][g];
    }
    s_o[0][g][d] = acc;
    if (d == 0) {
      c_m[g] = mn;
      c_l[g] = ls;
    }
  }
  cluster.sync();
  // ---- CTAs of the cluster: rank r finishes every nsplit-th output
  for (int i = split * DEC_THREADS + threadIdx.x; i < GT * DP; i += nsplit * DEC_THREADS) {
    const int g = i / DP, d = i % DP;
    float mn = -INFINITY, acc = 0.f, ls = 0.f;
    for (int r = 0; r < nsplit; ++r) mn = fmaxf(mn, *cluster.map_shared_rank(&c_m[g], r));
    for (int r = 0; r < nsplit; ++r) {
      float a;
      merge_scale(*cluster.map_shared_rank(&c_m[g], r), mn, a);
      acc += a * *cluster.map_shared_rank(&s_o[0][g][d], r);
      ls += a * *cluster.map_shared_rank(&c_l[g], r);
    }
    // (a NaN sum, from a NaN or +inf score, has to reach the output: only a sum of exactly 0 means a row without keys)
    if (d < p.D) p.o[b * p.o_sb + (head0 + g) * p.o_sh + d] = float_to_h16(ls == 0.f ? 0.f : acc / ls);
    if (d == 0) p.lse[(static_cast<long long>(b) * p.H + head0 + g) * 128] = ls > 0.f ? mn + log2f(ls) : LSE_NONE;
  }
  for (int i = split * DEC_THREADS + threadIdx.x; i < GT * 128; i += nsplit * DEC_THREADS)
    if (i % 128 != 0) p.lse[(static_cast<long long>(b) * p.H + head0 + i / 128) * 128 + i % 128] = INFINITY;
  cluster.sync();     // nobody leaves while its shared memory may still be read
}

static int ceil_div(int a, int b) { return (a + b - 1) / b; }
// splits that leave at least 64 keys to each, below which the merge costs more than the shorter loop saves
static int max_splits(int keys) {
  const int n = ceil_div(keys, 64);
  return n < DEC_MAX_SPLITS ? n : DEC_MAX_SPLITS;
}

// Clusters of 1 .. 8 CTAs that are resident at once.  Fewer than CTAs / size: a cluster lies within one group of SMs.
template <int DP, int GT>
struct ClusterSlots {
  int n[DEC_MAX_SPLITS + 1];
  ClusterSlots() {
    for (int s = 1; s <= DEC_MAX_SPLITS; ++s) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(s);
      cfg.blockDim = dim3(DEC_THREADS);
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = s;
      attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&n[s], attn_decode_kernel<DP, GT>, &cfg) != cudaSuccess || n[s] < 1) {
        (void)cudaGetLastError();
        n[s] = dec_ctas(GT) * sm_count() / s;
      }
    }
  }
};

template <int DP, int GT>
static int launch(const AttnDecodeParams& p, cudaStream_t stream) {
  const int G = p.H / p.Hk, rows = p.Hk * (G / GT);
  const int keys = p.Sk - p.key_lo;
  // Splits: the most whose clusters are resident at once (16 sequences, 24 heads on 3, 4096 keys in eights: 96 us with the 6
  // splits that fit by the number of CTAs, 74 with 4).  Otherwise, where every K / V row is read once (so that DRAM is the
  // bound) and the parts stay long, what wastes least of the last wave: two rounds of thirds instead of one round that
  // fills half of the places (14 x 32 heads of 128, 2048 keys: 89 / 82 us; quarters up to two thirds of the places, 18 x
  // 32, 8192 keys: 395 / 366), halves where a second wave would be nearly empty (32 x 32, 1543 keys: 154 / 137).  The number depends on the batch, and with it the order of the sums: a
  // sequence's last bits are not those it has in another batch.
  static const ClusterSlots<DP, GT> slots;
  const long long clusters = static_cast<long long>(rows) * p.B;
  auto rounds = [&](int s) { return static_cast<int>((clusters + slots.n[s] - 1) / slots.n[s]); };
  int splits = 1;
  for (int s = max_splits(keys); s > 1 && splits == 1; --s)
    if (rounds(s) == 1) splits = s;
  if (splits == 1 && GT == G) {
    const int row = keys / (128 / DP);          // in rows of 128
    if (rounds(1) > 1) {
      if (5 * rounds(2) <= 8 * rounds(1) && row >= 2 * 256) splits = 2;
    } else if (rounds(3) <= 2 && row >= 3 * 256) {
      splits = 3;
    } else if (3 * clusters <= 2 * slots.n[1] && row >= 4 * 1024) {
      splits = 4;
    }
  }
  const int per = (keys + splits - 1) / splits;
  // The next kernel may begin early only beside a short one that leaves places free.  Blocks that wait for a longer one's end
  // sit where places come free first, and if they are a decode kernel's, several on one SM, their sweep is that much
  // longer: one after the other, 1 sequence, 32 heads on 8, 8192 keys 39 us (24 without), 4 sequences 1543 keys 15.0 (11.7);
  // 12 heads of 64, 128 keys 3.0 (3.5).
  const bool early = splits * clusters <= sm_count() && per <= 256;
  NX_CUDA_CHECK(launch_dependent(attn_decode_kernel<DP, GT>, dim3(splits, rows, p.B), dim3(DEC_THREADS), 0, stream, splits, p,
                                 per, early));
  return NX_OK;
}

template <int DP>
static int launch_group(const AttnDecodeParams& p, cudaStream_t stream) {
  const int G = p.H / p.Hk;
  // Heads per CTA: the most whose CTAs, with all the splits that the keys allow, still fill about half of their places (a
  // sweep of 1 - 32 sequences, 1 - 16384 keys, 1 - 32 heads on a K / V head; pairs from a quarter on).  A CTA of
  // eight heads does eight heads' exchanges for every key, so it needs the bytes it saves to be what counts: 1 sequence, 32
  // heads on 4, 64 keys 9.2 us with eight, 3.9 with one (5.4 with the tile kernel); 8 sequences, 16384 keys 140 us with
  // eight, 286 with one.
  auto fits = [&](int gt, float share) {
    return G % gt == 0 && 1.f * p.Hk * (G / gt) * p.B * max_splits(p.Sk - p.key_lo) >= share * dec_ctas(gt) * sm_count();
  };
  if (fits(8, 0.5f)) return launch<DP, 8>(p, stream);
  if (fits(4, 0.5f)) return launch<DP, 4>(p, stream);
  if (fits(2, 0.25f)) return launch<DP, 2>(p, stream);
  return launch<DP, 1>(p, stream);
}

int attn_decode_launch(const AttnDecodeParams& p, cudaStream_t stream) {
  return p.D <= 64 ? launch_group<64>(p, stream) : launch_group<128>(p, stream);
}

}  // namespace nx
