// RWKV-6 WKV recurrence, forward and backward, with no compile-time sequence length.
//
//   y_t[j]   = sum_i r_t[i] * (u[i] * k_t[i] * v_t[j] + S_{t-1}[i][j])
//   S_t[i][j] = d_t[i] * S_{t-1}[i][j] + k_t[i] * v_t[j],      d_t[i] = exp(-exp(w_t[i]))
//
// Counterpart in the reference: megatron/model/rwkv/v6/cuda/wkv6_cuda.cu:6-241 (kernel_forward,
// kernel_backward_111 / _222), which walks the whole sequence in one thread per channel and needs
// the sequence length as a compile-time constant for a per-thread array.
//
// Heads of 64 in bf16 go in blocks of 16 steps as matrix products (second half of this file; wkv_in_blocks).  Heads of 32,
// fp16 and a few short sequences go step by step: one CTA of 2 N threads walks one head's piece of the sequence with the N x N
// state in registers: warp w owns 16 columns j, a lane N / 8 rows i by 4 columns.  Per step a lane reads N / 8 values of each row
// vector and 4 of each column vector from shared memory (column vectors are stored twice side by side, so that the packed fp32 pairs, which run
// over neighbouring rows, need no register moves) and does 3 packed operations per 2 state elements: one for the output
// sum, two for the update.  The u term is taken out of the sums: it is a dot product per step (formed while staging) times
// one value.  Sums over rows / columns leave a lane by transposing exchanges.
//   forward  : one sweep: y (sum over i)
//   backward : a forward sweep: gr (sum over j), then a reverse sweep of the gradient state G = dL/dS with gk (sum over j)
//              and gv (sum over i; a sweep of its own in blocks), which also forms the decay gradient: with
//              Q_t[i] = sum_j G_t[i][j] S_t[i][j] one has Q_{t-1} - Q_t = r_t gr_t - k_t gk_t and
//              dL/d(ew_t) = Q_t - k_t (gk_t - r_t u s_t),  s_t = <gy_t, v_t>,  ew = -exp(w)
// Step by step the shared-memory loads and exchanges of the steps are the bound (32 x 512 tokens, 12 heads of 64, forward +
// backward 788 us).  With the products of a block in their place, and a block's vectors beside the former block's products, 570
// (134 us for column sums, 123 for row sums, 159 for gk with the decay gradient); without bank conflicts on the decays 554 (129, 120,
// 153).  The bound is latency between a block's steps, at 2.6 warps per scheduler (issue slots 48 - 52 % busy, tensor pipe 13 - 24 %,
// shared memory 40 - 49 %, on average over SMs with two and with three CTAs): twice the warps, a group for the vectors beside one
// for the products, took 573 us (80 registers a thread, most warps at a barrier).
//
// The sequence is cut into chunks where that is faster, as a rule when batch x heads leaves the chip idle (wkv_chunk_count): the
// recurrence is linear, so a chunk's end state is  P (.) S_start + S_local  with P[i] = prod_t d_t[i]; local passes start every chunk
// from zero, a fold gives the chunks' start states, and Q at a chunk's end is <G, S> there.
#include <stddef.h>

#include "common.h"
#include "ptx.cuh"
#include "reduce.cuh"

namespace nx {

constexpr int WK_SUB = 16;          // steps staged together
constexpr int WK_MAX_CHUNKS = 32;

enum WkvMode { WK_LOCAL_FWD = 0, WK_LOCAL_REV = 1, WK_Y = 2, WK_GR = 3, WK_G = 4 };

struct WkvParams {
  const h16 *r, *k, *v, *w, *gy;
  long long sb, st;                 // batch / time strides (elements) shared by r, k, v, w, gy
  const float* u;                   // [H, N]
  h16 *y, *o_gr, *o_gk, *o_gv, *o_gw;   // (osb, ost)
  float* gr32;                      // (osb, ost)
  float* gu_part;                   // [B, NC, H, N]: the gradient of u by sequence and chunk
  long long osb, ost;
  float* local;                     // [B, H, NC, N, N] chunk-local end states
  const float* start;               // [B, H, NC, N, N] start states of this sweep; null = zero (one chunk)
  const float* fstart;              // reverse sweep with several chunks: the forward sweep's start states
  float* sumew;                     // [B, H, NC, N]
  int B, T, H, NC, clen;            // clen: steps per chunk, a multiple of WK_SUB
};

// 8 consecutive 16-bit elements (zero where dead): one 16-byte load when VEC, single elements otherwise.
template <bool VEC>
__device__ __forceinline__ uint4 wk_load8(const h16* p, bool ok) {
  uint4 u = make_uint4(0u, 0u, 0u, 0u);
  if (!ok) return u;
  if (VEC) return *reinterpret_cast<const uint4*>(p);
  uint16_t e[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) e[j] = reinterpret_cast<const uint16_t*>(p)[j];
  u.x = e[0] | (uint32_t)e[1] << 16; u.y = e[2] | (uint32_t)e[3] << 16;
  u.z = e[4] | (uint32_t)e[5] << 16; u.w = e[6] | (uint32_t)e[7] << 16;
  return u;
}
__device__ __forceinline__ void wk_unpack8(const uint4& u, float (&f)[8]) {
  const float2 a = unpack_h16x2(u.x), b = unpack_h16x2(u.y), c = unpack_h16x2(u.z), d = unpack_h16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}

// out[i] = <g[i], f[i]> of two states, N / 16 warps: each takes its rows one after the other, a row's values side by side (a thread
// per row, as it was, reads N lines at a time: 16 us of the 25 us of a reverse sweep of one block of steps).
template <int N>
__device__ __forceinline__ void wk_state_dots(const float* g, const float* f, float* out, int warp, int lane) {
#pragma unroll 8
  for (int x = 0; x < 16; ++x) {
    const int i = warp * 16 + x;
    float v = 0.f;
#pragma unroll
    for (int j = lane; j < N; j += 32) v += g[i * N + j] * f[i * N + j];
    v = warp_sum(v);
    if (lane == 0) out[i] = v;
  }
}

template <int N, int MODE>
struct WkvSmem {
  static constexpr bool ROW = MODE == WK_GR || MODE == WK_G, COL = MODE == WK_Y || MODE == WK_G;
  float b[WK_SUB][N], d[WK_SUB][N];             // state update: S = S * d[i] + b[i] * c[j]
  float2 c[WK_SUB][N];                          // (c, c)
  float a[COL ? WK_SUB : 1][N];                 // sum over i of a[i] S[i][j]
  float2 e[ROW ? WK_SUB : 1][N];                // (e, e): sum over j of e[j] S[i][j]
  float ew[WK_SUB][N];
  float colsum[COL ? WK_SUB : 1][N];
  float rowsum[ROW ? N / 16 : 1][ROW ? WK_SUB : 1][N];
  float dot_col[WK_SUB], dot_row[WK_SUB];       // <a, u b> and <e, c>
};

template <int N, int MODE, bool VEC>
__global__ void __launch_bounds__(2 * N) wkv_kernel(const WkvParams p) {
  using Sm = WkvSmem<N, MODE>;
  constexpr bool REV = MODE == WK_LOCAL_REV || MODE == WK_G, ROW = Sm::ROW, COL = Sm::COL;
  constexpr bool LOCAL = MODE == WK_LOCAL_FWD || MODE == WK_LOCAL_REV;
  constexpr int QUADS = N / 32, PAIRS = QUADS * 2;     // a lane's rows: QUADS groups of 4 neighbours
  constexpr int TPR = N / 8;                           // staging threads per step: 2 N threads stage 16 steps
  static_assert(WK_SUB * TPR == 2 * N, "one staging pass");
  extern __shared__ __align__(16) unsigned char wk_raw[];
  Sm& s = *reinterpret_cast<Sm*>(wk_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int jg = lane & 3, ig = lane >> 2;
  const int c = LOCAL && REV ? blockIdx.x + 1 : blockIdx.x, h = blockIdx.y, bi = blockIdx.z;
  const int t_lo = c * p.clen, t_hi = min(t_lo + p.clen, p.T);
  const long long base = ((long long)bi * p.H + h) * p.NC + c;

  float2 S[PAIRS][4];
  auto row_of = [&](int pr) { return (pr >> 1) * 32 + ig * 4 + (pr & 1) * 2; };      // first row of a pair
  auto col_of = [&](int k) { return warp * 16 + (k >> 1) * 8 + jg * 2 + (k & 1); };
#pragma unroll
  for (int pr = 0; pr < PAIRS; ++pr)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      S[pr][k] = make_float2(0.f, 0.f);
      if (!LOCAL && p.start != nullptr) {
        const float* q = p.start + (base * N + row_of(pr)) * N + col_of(k);
        S[pr][k] = make_float2(q[0], q[N]);
      }
    }
  // ---- output role: channel me; of the two threads of a channel the first carries the decay-gradient sum (reverse sweep)
  const int me = threadIdx.x % N, second = threadIdx.x / N;
  float Q = 0.f, gu = 0.f;
  const float u_me = p.u[h * N + me];
  if (MODE == WK_G && p.fstart != nullptr && c + 1 < p.NC) {
    wk_state_dots<N>(p.start + base * N * N, p.fstart + (base + 1) * N * N, &s.colsum[0][0], warp, lane);
    __syncthreads();
    Q = s.colsum[0][me];
  }
  // ---- staging role: step trow, 8 channels from ch8
  const int trow = threadIdx.x / TPR, ch8 = (threadIdx.x % TPR) * 8;
  float u8[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) u8[j] = p.u[h * N + ch8 + j];
  float sew = 0.f;                                     // LOCAL: thread i sums ew of channel i

  const int nsub = (t_hi - t_lo + WK_SUB - 1) / WK_SUB;
  // the next sub-block's inputs are fetched before the steps of this one
  uint4 rw, rb, rc, ra, re;
  auto fetch = [&](int q) {
    const int t = t_lo + (REV ? nsub - 1 - q : q) * WK_SUB + trow;
    const bool ok = t < t_hi;
    const long long o = bi * p.sb + (long long)t * p.st + h * N + ch8;
    rw = wk_load8<VEC>(p.w + o, ok);
    rb = wk_load8<VEC>((REV ? p.r : p.k) + o, ok);
    rc = wk_load8<VEC>((REV ? p.gy : p.v) + o, ok);
    if (COL) ra = wk_load8<VEC>((MODE == WK_Y ? p.r : p.k) + o, ok);
    if (ROW) re = wk_load8<VEC>((MODE == WK_GR ? p.gy : p.v) + o, ok);
  };
  fetch(0);
  for (int q = 0; q < nsub; ++q) {
    const int t0 = t_lo + (REV ? nsub - 1 - q : q) * WK_SUB;
    const int steps = min(WK_SUB, t_hi - t0);
    const long long oo = bi * p.osb + (long long)t0 * p.ost + h * N + me;
    float gr[MODE == WK_G ? WK_SUB : 1];
    if (MODE == WK_G) {
#pragma unroll
      for (int t = 0; t < WK_SUB; ++t) gr[t] = t < steps ? p.gr32[oo + t * p.ost] : 0.f;
    }
    {
      const int t = trow;
      const bool ok = t < steps;
      float x[8], y[8], wv[8];
      wk_unpack8(rw, wv);
      wk_unpack8(rb, x);
      wk_unpack8(rc, y);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float ew = ok ? -__expf(wv[j]) : 0.f;
        s.ew[t][ch8 + j] = ew;
        s.d[t][ch8 + j] = __expf(ew);
        s.b[t][ch8 + j] = x[j];
        s.c[t][ch8 + j] = make_float2(y[j], y[j]);
      }
      if (COL) {
        float a[8], dt = 0.f;
        wk_unpack8(ra, a);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          s.a[t][ch8 + j] = a[j];
          dt += a[j] * u8[j] * x[j];
        }
#pragma unroll
        for (int m = TPR / 2; m > 0; m >>= 1) dt += __shfl_xor_sync(0xffffffffu, dt, m);
        if (ch8 == 0) s.dot_col[t] = dt;
      }
      if (ROW) {
        float e[8], dt = 0.f;
        wk_unpack8(re, e);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          s.e[t][ch8 + j] = make_float2(e[j], e[j]);
          dt += e[j] * y[j];
        }
#pragma unroll
        for (int m = TPR / 2; m > 0; m >>= 1) dt += __shfl_xor_sync(0xffffffffu, dt, m);
        if (ch8 == 0) s.dot_row[t] = dt;
      }
    }
    if (q + 1 < nsub) fetch(q + 1);
    __syncthreads();
#pragma unroll 2
    for (int tq = 0; tq < steps; ++tq) {
      const int t = REV ? steps - 1 - tq : tq;
      float2 dv[PAIRS], bv[PAIRS], av[PAIRS], racc[PAIRS], cacc[4];
#pragma unroll
      for (int g = 0; g < QUADS; ++g) {
        const float4 d4 = *reinterpret_cast<const float4*>(&s.d[t][g * 32 + ig * 4]);
        const float4 b4 = *reinterpret_cast<const float4*>(&s.b[t][g * 32 + ig * 4]);
        dv[2 * g] = make_float2(d4.x, d4.y); dv[2 * g + 1] = make_float2(d4.z, d4.w);
        bv[2 * g] = make_float2(b4.x, b4.y); bv[2 * g + 1] = make_float2(b4.z, b4.w);
        if (COL) {
          const float4 a4 = *reinterpret_cast<const float4*>(&s.a[t][g * 32 + ig * 4]);
          av[2 * g] = make_float2(a4.x, a4.y); av[2 * g + 1] = make_float2(a4.z, a4.w);
        }
      }
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const float4 c4 = *reinterpret_cast<const float4*>(&s.c[t][warp * 16 + m * 8 + jg * 2]);
        float4 e4 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ROW) e4 = *reinterpret_cast<const float4*>(&s.e[t][warp * 16 + m * 8 + jg * 2]);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const int k = 2 * m + x;
          const float2 cc = x ? make_float2(c4.z, c4.w) : make_float2(c4.x, c4.y);
          const float2 ee = x ? make_float2(e4.z, e4.w) : make_float2(e4.x, e4.y);
#pragma unroll
          for (int pr = 0; pr < PAIRS; ++pr) {
            if (COL) cacc[k] = pr == 0 ? fmul2(av[0], S[0][k]) : ffma2(av[pr], S[pr][k], cacc[k]);
            if (ROW) racc[pr] = k == 0 ? fmul2(ee, S[pr][0]) : ffma2(ee, S[pr][k], racc[pr]);
            S[pr][k] = ffma2(S[pr][k], dv[pr], fmul2(bv[pr], cc));
          }
        }
      }
      if (COL) {      // 4 columns over the 8 row groups: lanes ig = 2 k, 2 k + 1 end up with column k
        float v4[4], v2[2];
#pragma unroll
        for (int k = 0; k < 4; ++k) v4[k] = cacc[k].x + cacc[k].y;
        const bool h2 = ig & 4, h1 = ig & 2;
#pragma unroll
        for (int k = 0; k < 2; ++k)
          v2[k] = (h2 ? v4[2 + k] : v4[k]) + __shfl_xor_sync(0xffffffffu, h2 ? v4[k] : v4[2 + k], 16);
        float v = (h1 ? v2[1] : v2[0]) + __shfl_xor_sync(0xffffffffu, h1 ? v2[0] : v2[1], 8);
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        if (!(ig & 1)) s.colsum[t][col_of(ig >> 1)] = v;
      }
      if (ROW) {      // a lane's N / 8 rows over the 4 column groups
        const bool h1 = jg & 2, h0 = jg & 1;
        float2 w2[PAIRS / 2];
#pragma unroll
        for (int k = 0; k < PAIRS / 2; ++k) {
          const float2 keep = h1 ? racc[PAIRS / 2 + k] : racc[k], give = h1 ? racc[k] : racc[PAIRS / 2 + k];
          w2[k].x = keep.x + __shfl_xor_sync(0xffffffffu, give.x, 2);
          w2[k].y = keep.y + __shfl_xor_sync(0xffffffffu, give.y, 2);
        }
        if (PAIRS == 4) {
          const float2 keep = h0 ? w2[PAIRS / 2 - 1] : w2[0], give = h0 ? w2[0] : w2[PAIRS / 2 - 1];
          const float2 o = make_float2(keep.x + __shfl_xor_sync(0xffffffffu, give.x, 1),
                                       keep.y + __shfl_xor_sync(0xffffffffu, give.y, 1));
          *reinterpret_cast<float2*>(&s.rowsum[warp][t][row_of((h1 ? 2 : 0) + (h0 ? 1 : 0))]) = o;
        } else {
          const float o = (h0 ? w2[0].y : w2[0].x) + __shfl_xor_sync(0xffffffffu, h0 ? w2[0].x : w2[0].y, 1);
          s.rowsum[warp][t][row_of(h1 ? 1 : 0) + (h0 ? 1 : 0)] = o;
        }
      }
    }
    __syncthreads();
    if (LOCAL) {
      if (!second)
        for (int t = 0; t < steps; ++t) sew += s.ew[t][me];
    } else if (MODE != WK_G) {
      // the two threads of a channel take half of the steps each
#pragma unroll
      for (int tq = 0; tq < WK_SUB / 2; ++tq) {
        const int t = second * (WK_SUB / 2) + tq;
        if (t >= steps) continue;
        if (MODE == WK_Y) {
          p.y[oo + t * p.ost] = float_to_h16(s.colsum[t][me] + s.c[t][me].x * s.dot_col[t]);
        } else {
          float row = 0.f;
#pragma unroll
          for (int w = 0; w < N / 16; ++w) row += s.rowsum[ROW ? w : 0][ROW ? t : 0][me];
          p.gr32[oo + t * p.ost] = row + u_me * s.b[t][me] * s.dot_row[t];
        }
      }
    } else if (second) {
#pragma unroll
      for (int t = 0; t < WK_SUB; ++t) {
        if (t >= steps) continue;
        p.o_gr[oo + t * p.ost] = float_to_h16(gr[MODE == WK_G ? t : 0]);
        p.o_gv[oo + t * p.ost] = float_to_h16(s.colsum[COL ? t : 0][me] + s.c[t][me].x * s.dot_col[t]);
      }
    } else {
#pragma unroll
      for (int tq = 0; tq < WK_SUB; ++tq) {      // in the sweep's direction
        const int t = WK_SUB - 1 - tq;
        if (t >= steps) continue;
        float row = 0.f;
#pragma unroll
        for (int w = 0; w < N / 16; ++w) row += s.rowsum[ROW ? w : 0][ROW ? t : 0][me];
        const float r_ = s.b[t][me], k_ = s.a[COL ? t : 0][me], st = s.dot_row[t];
        const float gk = row + u_me * r_ * st;
        p.o_gk[oo + t * p.ost] = float_to_h16(gk);
        p.o_gw[oo + t * p.ost] = float_to_h16((Q - k_ * row) * s.ew[t][me]);
        Q += r_ * gr[MODE == WK_G ? t : 0] - k_ * gk;
        gu += r_ * k_ * st;
      }
    }
    __syncthreads();
  }
  if (LOCAL) {
#pragma unroll
    for (int pr = 0; pr < PAIRS; ++pr)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float* o = p.local + (base * N + row_of(pr)) * N + col_of(k);
        o[0] = S[pr][k].x;
        o[N] = S[pr][k].y;
      }
    if (!second) p.sumew[base * N + me] = sew;
  }
  if (MODE == WK_G && !second) p.gu_part[(((long long)bi * p.NC + c) * p.H + h) * N + me] = gu;
}

// ------------------------------------------------------------------------------------------------
// Heads of 64: the same sweeps in blocks of 16 steps, as matrix products.  In the order of a sweep (reverse sweeps run
// backwards in time) let S be the state before a block, d_m the decays, a_t, b_t, c_t, e_t the step's vectors (S += b c^T):
//   column sums   y_t[j]   = sum_i a_t[i] Pre_t[i] S[i][j] + sum_{s < t} A[t][s] c_s[j] + A[t][t] c_t[j]
//   row sums      row_t[i] = Pre_t[i] sum_j e_t[j] S[i][j] + sum_{s < t} (prod_{s < m < t} d_m[i]) b_s[i] M[t][s]
//   state         S[i][j] <- Tot[i] S[i][j] + sum_s Suf_s[i] b_s[i] c_s[j]
// with Pre_t / Suf_t / Tot the products of the decays before / after t / of the block, M[t][s] = <e_t, c_s> and
// A[t][s] = sum_i a_t[i] b_s[i] prod_{s < m < t} d_m[i] (A[t][t]: with u).  Only products of decays between two steps appear,
// never a quotient, so no decay is too strong.  y = column sums forward with (r, k, v); gv the same backwards with (k, r, gy);
// gr = row sums forward with (k, v | gy); gk backwards with (r, gy | v), which also forms the decay gradient.
//
// Four warps; the state is the accumulators of mma.m16n8k16 (warp w: 16 of its rows, a thread 32 values), fp32 throughout.
// What is not a 16-bit input is split into three bf16 parts (24 bits: the products of parts of weight 2^-16 and above are
// all formed; the rest is below fp32's last bit).  The tensor core cuts off what is below the last bit of a sum, always towards
// zero, so a sum that lives long is not its accumulator: a block's products start from zero and are added to the state, and
// to the sums over the state, by rounded additions.  Row sums of 512 steps, error against 64 bits over their norm, decays
// of 1 - 6e-6 | the configured ones | 0.69: 3.4e-7 | 2.8e-7 | 8.3e-8; step by step 1.5e-6 | 1.6e-6 | 9.1e-8, with the
// state as accumulator and the decays of the step-by-step kernel 2.5e-6 | 2.2e-6 | 1.3e-7.
// These products are far too small for tcgen05 (M = 16 rows of steps, operands made in registers between every two of them),
// hence mma.sync.
// Infinity and what bf16 rounds to it have no parts, and a product of two vectors may leave fp32's range where the steps' own
// products do not: a block with such an input or state is done step by step, with the results of the step-by-step kernel.
// ------------------------------------------------------------------------------------------------
constexpr int WM = 16;              // steps per block
constexpr int WN = 64;              // head size
constexpr int WP = WN + 8;          // row pitch of the 16-bit arrays: ldmatrix without bank conflicts
constexpr int WM_THREADS = 128;
#ifdef NX_HALF
constexpr bool WM_BLOCKS = false;
#else
constexpr bool WM_BLOCKS = true;
#endif

__device__ __forceinline__ uint32_t wm_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float2 wm_floats(uint32_t v) {
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
__device__ __forceinline__ void wm_split(float2 x, uint32_t (&p)[3]) {
  const float2 m1 = make_float2(-1.f, -1.f);
  p[0] = wm_bf16x2(x.x, x.y);
  x = ffma2(wm_floats(p[0]), m1, x);
  p[1] = wm_bf16x2(x.x, x.y);
  x = ffma2(wm_floats(p[1]), m1, x);
  p[2] = wm_bf16x2(x.x, x.y);
}
__device__ __forceinline__ void wm_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same on top of zero.
__device__ __forceinline__ void wm_mma0(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// y += A B, with the addition to y rounded (the tensor core drops what is below a sum's last bit).
__device__ __forceinline__ void wm_add(float (&y)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float d[4];
  wm_mma0(d, a, b0, b1);
#pragma unroll
  for (int e = 0; e < 4; ++e) y[e] += d[e];
}
// Four 8 x 8 matrices: (rows r0 .. r0 + 7 | r0 + 8 ..) x (columns c0 .. | c0 + 8 ..) of a 16-bit array.  Plain: registers 0, 1 =
// the first rows' two column groups, 2, 3 = the second rows'; TRANS: each matrix transposed.
template <bool TRANS>
__device__ __forceinline__ void wm_ld4(uint32_t (&r)[4], const uint16_t* base, int r0, int c0, int pitch, bool rows_first) {
  const int lane = threadIdx.x & 31, m = lane >> 3, i = lane & 7;
  // rows_first: matrices in the order (0, 0), (1, 0), (0, 1), (1, 1) of (row group, column group), else (0, 0), (0, 1), ...
  const int rg = rows_first ? m & 1 : m >> 1, cg = rows_first ? m >> 1 : m & 1;
  const uint32_t addr = smem_u32(base + (r0 + rg * 8 + i) * pitch + c0 + cg * 8);
  if (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// exp(x) of x <= 0.  A weak decay stays in the state for many steps, so a bias of its approximation adds up (ex2.approx: an
// error of 1e-6 after 500 steps); near zero the series, whose last addition rounds.
__device__ __forceinline__ float2 wm_decay(float2 x) {
  auto c2 = [](float c) { return make_float2(c, c); };
  float2 p = ffma2(x, c2(1.f / 720), c2(1.f / 120));
  p = ffma2(p, x, c2(1.f / 24));
  p = ffma2(p, x, c2(1.f / 6));
  p = ffma2(p, x, c2(0.5f));
  p = ffma2(p, x, c2(1.f));
  p = ffma2(p, x, c2(1.f));
  return make_float2(x.x > -0.25f ? p.x : __expf(x.x), x.y > -0.25f ? p.y : __expf(x.y));
}

// An input block.
struct WmIn {
  uint16_t raw[WM][WP];
  __device__ __forceinline__ const uint16_t* data() const { return &raw[0][0]; }
  __device__ __forceinline__ void put(int t, int c8, const uint4& u) { *reinterpret_cast<uint4*>(&raw[t][c8]) = u; }
  __device__ __forceinline__ float at(int t, int c) const { return h16_to_float(reinterpret_cast<const h16&>(raw[t][c])); }
  __device__ __forceinline__ float2 pair(int t, int c) const {
    return unpack_h16x2(*reinterpret_cast<const uint32_t*>(&raw[t][c]));
  }
};

// Where channel c stands in a row of 64 fp32 values that is written and read as halves of eight channels: with the halves of the
// upper eights swapped, eight threads' halves lie in different banks.
__device__ __forceinline__ int wm_at(int c) { return c ^ ((c >> 3) & 4); }

// Whether all of eight bf16 inputs are below 2^20 (infinity and NaN are not).  Then no product over a block's vectors
// overflows, and what one loses when it underflows is below 2^-100.
__device__ __forceinline__ bool wm_ordinary(const uint4& u) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
  constexpr uint32_t E = (127u + 20u) << 7;
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 4; ++k) ok = ok && (w[k] & 0x7f80u) < E && ((w[k] >> 16) & 0x7f80u) < E;
  return ok;
}

// Whether this warp's states hold something that three parts do not: infinity, NaN, or a value that bf16 rounds to infinity
// (squares overflow long before; a state above 1e19 is as right step by step).
constexpr float WM_PART_MAX = 3.0e38f;
__device__ __forceinline__ bool wm_odd_state(const float (&S)[8][4]) {
  float2 z[2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float2 x = make_float2(S[n][2 * k], S[n][2 * k + 1]);
      z[k] = ffma2(x, x, z[k]);
    }
  return __any_sync(0xffffffffu, !(z[0].x + z[0].y + (z[1].x + z[1].y) < INFINITY));
}

// Step s of block q in a sweep's order -> time.  Blocks start at the sweep's first step, so that a short one is the last.
template <bool REV>
__device__ __forceinline__ int wm_time(int t_lo, int t_hi, int q, int s) {
  return REV ? t_hi - 1 - (q * WM + s) : t_lo + q * WM + s;
}

struct WmColSmem {
  WmIn a, b;
  float d[WM][WN];
  struct alignas(16) Block {                 // what the products of block q read and give, in slot q & 1
    WmIn c;
    uint16_t ap[3][WM][WP], bp[3][WM][WP];   // parts of a Pre, b Suf
    uint16_t A[3][WM][24];
    uint16_t out[WM][WP];
    float tot[WN];
    int odd_input, odd_A[2];                 // an input / an entry of A (by warp; u is in it) out of the products' range
  } blk[2];
};
static_assert(offsetof(WmColSmem, d) % 16 == 0 && offsetof(WmColSmem, blk) % 16 == 0 && sizeof(WmColSmem::Block) % 16 == 0 &&
                  offsetof(WmColSmem::Block, ap) % 16 == 0 && offsetof(WmColSmem::Block, bp) % 16 == 0 &&
                  offsetof(WmColSmem::Block, A) % 16 == 0 && offsetof(WmColSmem::Block, out) % 16 == 0 &&
                  offsetof(WmColSmem::Block, tot) % 16 == 0,
              "ldmatrix and 16-byte accesses");

// Column sums (y, or gv in reverse), or (LOCAL) only the end state of a chunk from a zero state and the sums of ew.
template <bool REV, bool LOCAL, bool VEC>
__global__ void __launch_bounds__(WM_THREADS, 3) wkv_col_kernel(const WkvParams p) {
  extern __shared__ __align__(16) unsigned char wk_raw[];
  WmColSmem& s = *reinterpret_cast<WmColSmem*>(wk_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ch = LOCAL && REV ? blockIdx.x + 1 : blockIdx.x, h = blockIdx.y, bi = blockIdx.z;
  const int t_lo = ch * p.clen, t_hi = min(t_lo + p.clen, p.T);
  const long long base = ((long long)bi * p.H + h) * p.NC + ch;
  const h16 *ga = REV ? p.k : p.r, *gb = REV ? p.r : p.k, *gc = REV ? p.gy : p.v;
  // S^T: rows j = 16 warp + lane / 4 (+ 8), columns i = 8 n + 2 (lane % 4) (+ 1)
  float S[8][4];
  const int j0 = warp * 16 + (lane >> 2), i0 = (lane & 3) * 2;
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      S[n][e] = 0.f;
      if (!LOCAL && p.start != nullptr) S[n][e] = p.start[(base * WN + 8 * n + i0 + (e & 1)) * WN + j0 + (e >> 1) * 8];
    }
  // the zeros of A (its upper triangle is never written)
  for (int x = tid; x < 3 * WM * 24; x += WM_THREADS) (&s.blk[0].A[0][0][0])[x] = (&s.blk[1].A[0][0][0])[x] = 0;
  const int trow = tid >> 3, ch8 = (tid & 7) * 8;
  float sew[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const int nblk = (t_hi - t_lo + WM - 1) / WM;
  uint4 ra, rb, rc, rw;
  bool live;
  auto fetch = [&](int q) {
    const int t = wm_time<REV>(t_lo, t_hi, q, trow);
    live = t >= t_lo && t < t_hi;
    const long long o = bi * p.sb + (long long)t * p.st + h * WN + ch8;
    if (!LOCAL) ra = wk_load8<VEC>(ga + o, live);
    rb = wk_load8<VEC>(gb + o, live);
    rc = wk_load8<VEC>(gc + o, live);
    rw = wk_load8<VEC>(p.w + o, live);
  };
  fetch(0);
  // Round q: block q is staged, then its vectors (a Pre, b Suf, A) and the products of block q - 1 come between the same two
  // barriers, so that the warps' unequal vector work and the latencies of the two overlap.
  for (int q = 0; q <= nblk; ++q) {
    auto& now = s.blk[q & 1];
    auto& former = s.blk[(q & 1) ^ 1];
    if (q < nblk) {
      if (!LOCAL) s.a.put(trow, ch8, ra);
      s.b.put(trow, ch8, rb);
      now.c.put(trow, ch8, rc);
      float w8[8], d8[8];
      wk_unpack8(rw, w8);
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        const float2 ew = live ? make_float2(-__expf(w8[e]), -__expf(w8[e + 1])) : make_float2(0.f, 0.f);
        const float2 d = wm_decay(ew);
        d8[e] = d.x;
        d8[e + 1] = d.y;
        if (LOCAL) {
          sew[e] += ew.x;
          sew[e + 1] += ew.y;
        }
      }
      *reinterpret_cast<float4*>(&s.d[trow][wm_at(ch8)]) = make_float4(d8[0], d8[1], d8[2], d8[3]);
      *reinterpret_cast<float4*>(&s.d[trow][wm_at(ch8 + 4)]) = make_float4(d8[4], d8[5], d8[6], d8[7]);
    }
    const int odd_input = __syncthreads_or(q < nblk && !(wm_ordinary(rb) && wm_ordinary(rc) && (LOCAL || wm_ordinary(ra))));
    if (tid == 0) now.odd_input = odd_input;
    if (q + 1 < nblk) fetch(q + 1);      // in flight during this round
    if (!LOCAL && q > 1) {               // (the sums of block q - 2, laid out in the last round)
      const int t = wm_time<REV>(t_lo, t_hi, q - 2, trow);
      if (t >= t_lo && t < t_hi)
        *reinterpret_cast<uint4*>((REV ? p.o_gv : p.y) + bi * p.osb + (long long)t * p.ost + h * WN + ch8) =
            *reinterpret_cast<const uint4*>(&now.out[trow][ch8]);
    }
    if (q < nblk && warp == 0) {
      // a Pre, and Tot; two channels per thread
      const int c = lane * 2;
      float2 pre = make_float2(1.f, 1.f);
#pragma unroll 4
      for (int t = 0; t < WM; ++t) {
        const float2 d = *reinterpret_cast<const float2*>(&s.d[t][wm_at(c)]);
        if (!LOCAL) {
          uint32_t x[3];
          wm_split(fmul2(s.a.pair(t, c), pre), x);
#pragma unroll
          for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(&now.ap[k][t][c]) = x[k];
        }
        pre = fmul2(pre, d);
      }
      *reinterpret_cast<float2*>(&now.tot[c]) = pre;
    } else if (q < nblk && warp == 1) {
      const int c = lane * 2;
      float2 suf = make_float2(1.f, 1.f);
#pragma unroll 4
      for (int t = WM - 1; t >= 0; --t) {
        const float2 d = *reinterpret_cast<const float2*>(&s.d[t][wm_at(c)]);
        uint32_t x[3];
        wm_split(fmul2(s.b.pair(t, c), suf), x);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(&now.bp[k][t][c]) = x[k];
        suf = fmul2(suf, d);
      }
    } else if (!LOCAL && q < nblk) {
      // A: eight groups of eight lanes (8 channels each); group g takes columns s = g and s = 15 - g, 15 entries together
      const int g = (tid - 64) >> 3, c = (tid & 7) * 8, turn = WM - 1 - g;
      float2 qv[4];
      auto load_b = [&](int t) {
#pragma unroll
        for (int k = 0; k < 4; ++k) qv[k] = s.b.pair(t, c + 2 * k);
      };
      load_b(g);
      float val[16], diag = 0.f;
#pragma unroll
      for (int it = 0; it < 15; ++it) {
        if (it == turn) load_b(turn);
        const int t = it < turn ? g + 1 + it : turn + 1 + (it - turn);
        float2 acc = make_float2(0.f, 0.f);
        const float4 d0 = *reinterpret_cast<const float4*>(&s.d[t][wm_at(c)]),
                     d1 = *reinterpret_cast<const float4*>(&s.d[t][wm_at(c + 4)]);
        const float2 dd[4] = {{d0.x, d0.y}, {d0.z, d0.w}, {d1.x, d1.y}, {d1.z, d1.w}};
        const uint4 u = *reinterpret_cast<const uint4*>(&s.a.raw[t][c]);
        const uint32_t aw[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          acc = ffma2(unpack_h16x2(aw[k]), qv[k], acc);
          qv[k] = fmul2(qv[k], dd[k]);
        }
        val[it] = acc.x + acc.y;
      }
      // the diagonal entries g (slot 15) and 15 - g
      float dg[2] = {0.f, 0.f};
#pragma unroll
      for (int z = 0; z < 2; ++z)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int t = z == 0 ? g : turn;
          const float2 x = s.a.pair(t, c + 2 * k), y = s.b.pair(t, c + 2 * k);
          dg[z] += x.x * p.u[h * WN + c + 2 * k] * y.x + x.y * p.u[h * WN + c + 2 * k + 1] * y.y;
        }
      val[15] = dg[0];
      diag = dg[1];
#pragma unroll
      for (int m = 4; m > 0; m >>= 1) diag += __shfl_xor_sync(0xffffffffu, diag, m);
      // 16 values over 8 lanes: lane l ends with values 2 l' , 2 l' + 1 of its own order
      const bool h4 = lane & 4, h2 = lane & 2, h1 = lane & 1;
      float v8[8], v4[4], v2[2];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        v8[k] = (h4 ? val[8 + k] : val[k]) + __shfl_xor_sync(0xffffffffu, h4 ? val[k] : val[8 + k], 4);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        v4[k] = (h2 ? v8[4 + k] : v8[k]) + __shfl_xor_sync(0xffffffffu, h2 ? v8[k] : v8[4 + k], 2);
#pragma unroll
      for (int k = 0; k < 2; ++k)
        v2[k] = (h1 ? v4[2 + k] : v4[k]) + __shfl_xor_sync(0xffffffffu, h1 ? v4[k] : v4[2 + k], 1);
      bool odd_A = false;
      auto put_A = [&](int t, int col, float x) {
        odd_A = odd_A || !(fabsf(x) < WM_PART_MAX);
        uint32_t y[3];
        wm_split(make_float2(x, 0.f), y);
#pragma unroll
        for (int k = 0; k < 3; ++k) now.A[k][t][col] = static_cast<uint16_t>(y[k]);
      };
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int it = (h4 ? 8 : 0) + (h2 ? 4 : 0) + (h1 ? 2 : 0) + k;
        if (it == 15) put_A(g, g, v2[k]);
        else if (it < turn) put_A(g + 1 + it, g, v2[k]);
        else put_A(turn + 1 + (it - turn), turn, v2[k]);
      }
      if ((lane & 7) == 0) put_A(turn, turn, diag);
      odd_A = __any_sync(0xffffffffu, odd_A);
      if (lane == 0) now.odd_A[warp - 2] = odd_A;
    }
    if (q > 0 && (former.odd_input || (!LOCAL && (former.odd_A[0] || former.odd_A[1])) || wm_odd_state(S))) {
      // ---- block q - 1 step by step
#pragma unroll 1
      for (int x = 0; x < WM; ++x) {
        const int t = wm_time<REV>(t_lo, t_hi, q - 1, x);
        if (t < t_lo || t >= t_hi) break;
        const long long o = bi * p.sb + (long long)t * p.st + h * WN;
        const float c0 = former.c.at(x, j0), c1 = former.c.at(x, j0 + 8);
        float y0 = 0.f, y1 = 0.f, dot = 0.f;
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int i = 8 * n + i0 + e;
            const float ew = -__expf(h16_to_float(p.w[o + i])), b = h16_to_float(gb[o + i]), d = wm_decay(make_float2(ew, ew)).x;
            if (!LOCAL) {
              const float a = h16_to_float(ga[o + i]);
              y0 += a * S[n][e];
              y1 += a * S[n][2 + e];
              dot += a * p.u[h * WN + i] * b;
            }
            S[n][e] = S[n][e] * d + b * c0;
            S[n][2 + e] = S[n][2 + e] * d + b * c1;
          }
        if (!LOCAL) {
#pragma unroll
          for (int m = 2; m > 0; m >>= 1) {
            y0 += __shfl_xor_sync(0xffffffffu, y0, m);
            y1 += __shfl_xor_sync(0xffffffffu, y1, m);
            dot += __shfl_xor_sync(0xffffffffu, dot, m);
          }
          if ((lane & 3) == 0) {
            const h16 o0 = float_to_h16(y0 + c0 * dot), o1 = float_to_h16(y1 + c1 * dot);
            former.out[x][j0] = reinterpret_cast<const uint16_t&>(o0);
            former.out[x][j0 + 8] = reinterpret_cast<const uint16_t&>(o1);
          }
        }
      }
    } else if (q > 0) {
    // ---- products of block q - 1
    uint32_t cv[4];                      // c^T: 16 rows j of this warp x 16 steps
    wm_ld4<true>(cv, former.c.data(), 0, warp * 16, WP, false);
    if (!LOCAL) {
      float y[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      float z[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};      // the products of lower parts
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        uint32_t sp[3][4];               // S^T[16 j][16 i]
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          uint32_t x[3];
          const float* src = S[2 * ks + (e >> 1)] + (e & 1) * 2;
          wm_split(make_float2(src[0], src[1]), x);
          sp[0][e] = x[0]; sp[1][e] = x[1]; sp[2][e] = x[2];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          uint32_t b[4];
          wm_ld4<false>(b, &former.ap[k][0][0], 0, 16 * ks, WP, false);
#pragma unroll
          for (int m = 2 - k; m >= 0; --m) {
            if (m + k == 0) {
              wm_add(y[0], sp[m], b[0], b[1]);
              wm_add(y[1], sp[m], b[2], b[3]);
            } else {
              wm_mma(z[0], sp[m], b[0], b[1]);
              wm_mma(z[1], sp[m], b[2], b[3]);
            }
          }
        }
      }
#pragma unroll
      for (int k = 2; k >= 0; --k) {
        uint32_t b[4];
        wm_ld4<false>(b, &former.A[k][0][0], 0, 0, 24, false);
        if (k > 0) {
          wm_mma(z[0], cv, b[0], b[1]);
          wm_mma(z[1], cv, b[2], b[3]);
        } else {
          wm_add(y[0], cv, b[0], b[1]);
          wm_add(y[1], cv, b[2], b[3]);
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        y[0][e] += z[0][e];
        y[1][e] += z[1][e];
      }
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const h16 o = float_to_h16(y[n][e]);
          former.out[8 * n + i0 + (e & 1)][j0 + (e >> 1) * 8] = reinterpret_cast<const uint16_t&>(o);
        }
    }
#pragma unroll
    for (int n = 0; n < 8; n += 2) {
      float add[2][4];
#pragma unroll
      for (int k = 2; k >= 0; --k) {
        uint32_t b[4];
        wm_ld4<true>(b, &former.bp[k][0][0], 0, 8 * n, WP, true);
        if (k == 2) {
          wm_mma0(add[0], cv, b[0], b[1]);
          wm_mma0(add[1], cv, b[2], b[3]);
        } else {
          wm_mma(add[0], cv, b[0], b[1]);
          wm_mma(add[1], cv, b[2], b[3]);
        }
      }
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const float2 d = *reinterpret_cast<const float2*>(&former.tot[8 * (n + x) + i0]);
#pragma unroll
        for (int e = 0; e < 4; ++e) S[n + x][e] = fmaf(S[n + x][e], e & 1 ? d.y : d.x, add[x][e]);
      }
    }
    }
    __syncthreads();
  }
  if (!LOCAL) {
    const int t = wm_time<REV>(t_lo, t_hi, nblk - 1, trow);
    if (t >= t_lo && t < t_hi)
      *reinterpret_cast<uint4*>((REV ? p.o_gv : p.y) + bi * p.osb + (long long)t * p.ost + h * WN + ch8) =
          *reinterpret_cast<const uint4*>(&s.blk[(nblk - 1) & 1].out[trow][ch8]);
  }
  if (LOCAL) {
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) p.local[(base * WN + 8 * n + i0 + (e & 1)) * WN + j0 + (e >> 1) * 8] = S[n][e];
    // sums of ew over the 16 staging rows
    float* r = &s.d[0][0];
#pragma unroll
    for (int e = 0; e < 8; ++e) r[trow * WN + ch8 + e] = sew[e];
    __syncthreads();
    if (tid < WN) {
      float a = 0.f;
      for (int t = 0; t < WM; ++t) a += r[t * WN + tid];
      p.sumew[base * WN + tid] = a;
    }
  }
}

struct WmRowSmem {
  float d[WM][WN];
  float M[2][WM][8];                         // <e_t, c_s>: s even | odd
  float inter[WM][WN + 4];
  struct alignas(16) Block {                 // of block q, in slot q & 1
    WmIn b, c, e;
    uint16_t k[WM][WP];                      // gk: the other factor of the decay gradient
    float ew[WM][WN];
    uint16_t bp[3][WM][WP];
    float st[WM];
    float part[2][WM][WN];                   // what a block's own steps add, by the parity of s
    float pre[WM][WN], tot[WN];
    int odd_input;                           // an input out of the products' range
  } blk[2];
};
static_assert(offsetof(WmRowSmem, M) % 16 == 0 && offsetof(WmRowSmem, blk) % 16 == 0 && sizeof(WmRowSmem::Block) % 16 == 0 &&
                  offsetof(WmRowSmem::Block, k) % 16 == 0 && offsetof(WmRowSmem::Block, bp) % 16 == 0,
              "ldmatrix and 16-byte accesses");

// Row sums: gr (fp32 and rounded), or in reverse gk with the decay gradient and the sums for the gradient of u.
template <bool REV, bool VEC>
__global__ void __launch_bounds__(WM_THREADS, 3) wkv_row_kernel(const WkvParams p) {
  extern __shared__ __align__(16) unsigned char wk_raw[];
  WmRowSmem& s = *reinterpret_cast<WmRowSmem*>(wk_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ch = blockIdx.x, h = blockIdx.y, bi = blockIdx.z;
  const int t_lo = ch * p.clen, t_hi = min(t_lo + p.clen, p.T);
  const long long base = ((long long)bi * p.H + h) * p.NC + ch;
  const h16 *gb = REV ? p.r : p.k, *gc = REV ? p.gy : p.v, *ge = REV ? p.v : p.gy;
  // S: rows i = 16 warp + lane / 4 (+ 8), columns j = 8 n + 2 (lane % 4) (+ 1)
  float S[8][4];
  const int r0 = warp * 16 + (lane >> 2), n0 = (lane & 3) * 2;
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      S[n][e] = p.start != nullptr ? p.start[(base * WN + r0 + (e >> 1) * 8) * WN + 8 * n + n0 + (e & 1)] : 0.f;
  const int me = tid & (WN - 1), half = tid >> 6;
  const float u_me = p.u[h * WN + me];
  float Q = 0.f, gu = 0.f;
  if (REV && p.fstart != nullptr && ch + 1 < p.NC) {
    wk_state_dots<WN>(p.start + base * WN * WN, p.fstart + (base + 1) * WN * WN, &s.inter[0][0], warp, lane);
    __syncthreads();
    Q = s.inter[0][me];
  }
  const int trow = tid >> 3, ch8 = (tid & 7) * 8;
  const int nblk = (t_hi - t_lo + WM - 1) / WM;
  uint4 rb, rc, re, rw, rk;
  bool live;
  auto fetch = [&](int q) {
    const int t = wm_time<REV>(t_lo, t_hi, q, trow);
    live = t >= t_lo && t < t_hi;
    const long long o = bi * p.sb + (long long)t * p.st + h * WN + ch8;
    rb = wk_load8<VEC>(gb + o, live);
    rc = wk_load8<VEC>(gc + o, live);
    re = wk_load8<VEC>(ge + o, live);
    rw = wk_load8<VEC>(p.w + o, live);
    if (REV) rk = wk_load8<VEC>(p.k + o, live);
  };
  fetch(0);
  // Round q: block q is staged; M of block q and the products of block q - 1; the results of block q - 1 and what block q's own
  // steps add.  Three barriers a round.
  const long long oo = bi * p.osb + h * WN + me;
  for (int q = 0; q <= nblk; ++q) {
    auto& now = s.blk[q & 1];
    auto& former = s.blk[(q & 1) ^ 1];
    const int steps = min(WM, t_hi - t_lo - (q - 1) * WM);      // of block q - 1
    if (q < nblk) {
    now.b.put(trow, ch8, rb);
    now.c.put(trow, ch8, rc);
    now.e.put(trow, ch8, re);
    if (REV) *reinterpret_cast<uint4*>(&now.k[trow][ch8]) = rk;
    {
      float w8[8];
      wk_unpack8(rw, w8);
#pragma unroll
      for (int e = 0; e < 8; e += 4) {
        float2 ew[2], d[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          ew[k] = live ? make_float2(-__expf(w8[e + 2 * k]), -__expf(w8[e + 2 * k + 1])) : make_float2(0.f, 0.f);
          d[k] = wm_decay(ew[k]);
        }
        *reinterpret_cast<float4*>(&now.ew[trow][wm_at(ch8 + e)]) = make_float4(ew[0].x, ew[0].y, ew[1].x, ew[1].y);
        *reinterpret_cast<float4*>(&s.d[trow][wm_at(ch8 + e)]) = make_float4(d[0].x, d[0].y, d[1].x, d[1].y);
      }
    }
    }
    const int odd_input = __syncthreads_or(q < nblk && !(wm_ordinary(rb) && wm_ordinary(rc) && wm_ordinary(re)));
    if (tid == 0) now.odd_input = odd_input;
    if (q + 1 < nblk) fetch(q + 1);      // in flight during this round
    float gr[REV ? WM : 1];
    if (REV && half == 0 && q > 0) {
#pragma unroll
      for (int t = 0; t < WM; ++t)
        gr[REV ? t : 0] = t < steps ? p.gr32[oo + (long long)(t_hi - 1 - (q - 1) * WM - t) * p.ost] : 0.f;
    }
    // ---- M: warp 0 the first eight s, warp 1 the others
    if (q < nblk && warp < 2) {
      float m4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        uint32_t a[4], b[4];
        wm_ld4<false>(a, now.e.data(), 0, 16 * ks, WP, true);
        wm_ld4<false>(b, now.c.data(), 0, 16 * ks, WP, false);
        wm_add(m4, a, warp == 0 ? b[0] : b[2], warp == 0 ? b[1] : b[3]);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = (lane >> 2) + (e >> 1) * 8, x = warp * 8 + n0 + (e & 1);
        s.M[x & 1][t][x >> 1] = m4[e];
        if (t == x) now.st[t] = m4[e];
      }
    }
    if (q > 0 && (former.odd_input || wm_odd_state(S))) {
      // ---- block q - 1 step by step: whole row sums, in the place of the state's part of them
#pragma unroll 1
      for (int x = 0; x < steps; ++x) {
        const float b0 = former.b.at(x, r0), b1 = former.b.at(x, r0 + 8);
        const float2 d = wm_decay(make_float2(former.ew[x][wm_at(r0)], former.ew[x][wm_at(r0 + 8)]));
        float y0 = 0.f, y1 = 0.f, st = 0.f;
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float c = former.c.at(x, 8 * n + n0 + k), e = former.e.at(x, 8 * n + n0 + k);
            y0 += e * S[n][k];
            y1 += e * S[n][2 + k];
            st += e * c;
            S[n][k] = S[n][k] * d.x + b0 * c;
            S[n][2 + k] = S[n][2 + k] * d.y + b1 * c;
          }
#pragma unroll
        for (int m = 2; m > 0; m >>= 1) {
          y0 += __shfl_xor_sync(0xffffffffu, y0, m);
          y1 += __shfl_xor_sync(0xffffffffu, y1, m);
          st += __shfl_xor_sync(0xffffffffu, st, m);
        }
        if ((lane & 3) == 0) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            s.inter[x][r0 + 8 * k] = k == 0 ? y0 : y1;
            former.pre[x][r0 + 8 * k] = 1.f;
            former.part[0][x][r0 + 8 * k] = former.part[1][x][r0 + 8 * k] = 0.f;
          }
        }
        if (former.odd_input && tid == 0) former.st[x] = st;
      }
    } else if (q > 0) {
    // ---- products
    {
      float y[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      float z[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};      // the products of lower parts
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        uint32_t sp[3][4];               // S[16 i][16 j]
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          uint32_t x[3];
          const float* src = S[2 * ks + (e >> 1)] + (e & 1) * 2;
          wm_split(make_float2(src[0], src[1]), x);
          sp[0][e] = x[0]; sp[1][e] = x[1]; sp[2][e] = x[2];
        }
        uint32_t b[4];
        wm_ld4<false>(b, former.e.data(), 0, 16 * ks, WP, false);
#pragma unroll
        for (int m = 2; m > 0; --m) {
          wm_mma(z[0], sp[m], b[0], b[1]);
          wm_mma(z[1], sp[m], b[2], b[3]);
        }
        wm_add(y[0], sp[0], b[0], b[1]);
        wm_add(y[1], sp[0], b[2], b[3]);
      }
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) s.inter[8 * n + n0 + (e & 1)][r0 + (e >> 1) * 8] = y[n][e] + z[n][e];
      const float t0 = former.tot[r0], t1 = former.tot[r0 + 8];
      uint32_t bt[3][4];                 // (b Suf)^T: 16 rows i x 16 steps
#pragma unroll
      for (int k = 0; k < 3; ++k) wm_ld4<true>(bt[k], &former.bp[k][0][0], 0, warp * 16, WP, false);
#pragma unroll
      for (int n = 0; n < 8; n += 2) {
        uint32_t b[4];
        wm_ld4<true>(b, former.c.data(), 0, 8 * n, WP, true);
        float add[2][4];
        wm_mma0(add[0], bt[2], b[0], b[1]);
        wm_mma0(add[1], bt[2], b[2], b[3]);
#pragma unroll
        for (int k = 1; k >= 0; --k) {
          wm_mma(add[0], bt[k], b[0], b[1]);
          wm_mma(add[1], bt[k], b[2], b[3]);
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[n + x][e] = fmaf(S[n + x][e], e < 2 ? t0 : t1, add[x][e]);
      }
    }
    }
    __syncthreads();
    if (q > 0) {
    // ---- results
    if (!REV) {
#pragma unroll
      for (int x = 0; x < WM / 2; ++x) {
        const int t = half * (WM / 2) + x;
        if (t >= steps) continue;
        const float row = former.pre[t][me] * s.inter[t][me] + (former.part[0][t][me] + former.part[1][t][me]);
        const float gr = row + u_me * former.b.at(t, me) * former.st[t];
        const long long o = oo + (long long)(t_lo + (q - 1) * WM + t) * p.ost;
        p.gr32[o] = gr;
        p.o_gr[o] = float_to_h16(gr);
      }
    } else if (half == 0) {
#pragma unroll
      for (int t = 0; t < WM; ++t) {
        if (t >= steps) continue;
        const float row = former.pre[t][me] * s.inter[t][me] + (former.part[0][t][me] + former.part[1][t][me]);
        const float r_ = former.b.at(t, me), k_ = h16_to_float(reinterpret_cast<const h16&>(former.k[t][me])), st = former.st[t];
        const float gk = row + u_me * r_ * st;
        const long long o = oo + (long long)(t_hi - 1 - (q - 1) * WM - t) * p.ost;
        p.o_gk[o] = float_to_h16(gk);
        p.o_gw[o] = float_to_h16((Q - k_ * row) * former.ew[t][wm_at(me)]);
        Q += r_ * gr[REV ? t : 0] - k_ * gk;
        gu += r_ * k_ * st;
      }
    }
    }
    if (q < nblk) {
    // ---- a block's own steps, for one channel and every second s
    {
      float qv[8], pre = 1.f;
#pragma unroll
      for (int t = 0; t < WM; ++t) {
        const float d = s.d[t][wm_at(me)];
        float acc = 0.f;
        const float4 m0 = *reinterpret_cast<const float4*>(&s.M[half][t][0]), m1 = *reinterpret_cast<const float4*>(&s.M[half][t][4]);
        const float m[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
        // own s: 2 x + half < t; the last of them exists for half 1 only from t on that is even
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          if (2 * x + 1 < t) {
            acc += qv[x] * m[x];
            qv[x] *= d;
          } else if (2 * x < t && half == 0) {
            acc += qv[x] * m[x];
            qv[x] *= d;
          }
        }
        if ((t & 1) == half) qv[t >> 1] = now.b.at(t, me);
        now.part[half][t][me] = acc;
        if (half == 0) {
          now.pre[t][me] = pre;
          pre *= d;
        }
      }
      if (half == 0) now.tot[me] = pre;
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        uint32_t y[3];
        wm_split(make_float2(qv[x], 0.f), y);
#pragma unroll
        for (int k = 0; k < 3; ++k) now.bp[k][2 * x + half][me] = static_cast<uint16_t>(y[k]);
      }
    }
    }
    __syncthreads();
  }
  if (REV && half == 0) p.gu_part[(((long long)bi * p.NC + ch) * p.H + h) * WN + me] = gu;
}

// start[c] for every chunk: forward  start[0] = 0, start[c+1] = P_c start[c] + local[c];
//                           reverse  start[NC-1] = 0, start[c-1] = P_c start[c] + local[c].
// Eight chunks' values are read together: 1 x 512, 12 heads, 16 chunks 6.9 -> 2.9 us (one after the other a chain of loads); with
// many heads the bytes are the bound (8 x 2048, 16 heads, 10 chunks 9.4 -> 7.4 us).
template <int N, bool REV>
__global__ void __launch_bounds__(N) wkv_fold_kernel(const float* __restrict__ local, const float* __restrict__ sumew,
                                                     float* __restrict__ start, int NC) {
  constexpr int AHEAD = 8, STEP = REV ? -1 : 1;
  const long long first = ((static_cast<long long>(blockIdx.z) * gridDim.y + blockIdx.y) * NC + (REV ? NC - 1 : 0)) * N + blockIdx.x;
  local += first * N + threadIdx.x;
  start += first * N + threadIdx.x;
  sumew += first;
  float S = 0.f;
  for (int q0 = 0; q0 < NC; q0 += AHEAD) {
    float l[AHEAD], d[AHEAD];
#pragma unroll
    for (int x = 0; x < AHEAD; ++x)
      if (q0 + x + 1 < NC) {      // (the last chunk's own state is nobody's start)
        d[x] = sumew[x * STEP * N];
        l[x] = local[x * STEP * N * N];
      }
#pragma unroll
    for (int x = 0; x < AHEAD; ++x)
      if (q0 + x < NC) {
        start[x * STEP * N * N] = S;
        if (q0 + x + 1 < NC) S = S * __expf(d[x]) + l[x];
      }
    local += AHEAD * STEP * N * N;
    start += AHEAD * STEP * N * N;
    sumew += AHEAD * STEP * N;
  }
}

// gu[i] = sum of the parts, in an order of its own (no atomics: a backward repeats bit for bit).
constexpr int WK_SUM_X = 32, WK_SUM_Y = 16;
__global__ void __launch_bounds__(WK_SUM_X * WK_SUM_Y) wkv_sum_kernel(const float* part, float* gu, int parts, int n) {
  __shared__ float s[WK_SUM_Y][WK_SUM_X];
  const int i = blockIdx.x * WK_SUM_X + threadIdx.x;
  float a = 0.f;
  if (i < n) {
#pragma unroll 4
    for (int r = threadIdx.y; r < parts; r += WK_SUM_Y) a += part[(long long)r * n + i];
  }
  s[threadIdx.y][threadIdx.x] = a;
  __syncthreads();
  if (threadIdx.y == 0 && i < n) {
#pragma unroll
    for (int y = 1; y < WK_SUM_Y; ++y) a += s[y][threadIdx.x];
    gu[i] = a;
  }
}

template <int N, int MODE>
static int wkv_launch(const WkvParams& p, bool vec, int chunks, cudaStream_t stream) {
  const int smem = (int)sizeof(WkvSmem<N, MODE>);
  static bool attr_set = false;
  if (!attr_set) {
    NX_CUDA_CHECK(cudaFuncSetAttribute(wkv_kernel<N, MODE, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    NX_CUDA_CHECK(cudaFuncSetAttribute(wkv_kernel<N, MODE, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr_set = true;
  }
  const dim3 grid(chunks, p.H, p.B);
  if (vec) wkv_kernel<N, MODE, true><<<grid, 2 * N, smem, stream>>>(p);
  else wkv_kernel<N, MODE, false><<<grid, 2 * N, smem, stream>>>(p);
  NX_LAUNCH_CHECK();
  return NX_OK;
}

// Which calls go in blocks: bf16 (an fp16 input would take two parts, and its products twice to four times as many: 32 x 512, 12
// heads 997 us, step by step 780; 8 x 2048, 16 heads 1,508 against 1,363), and not a few short sequences, where the fourth
// sweep's launch and a block's latency count (forward + backward, step by step / in blocks: 1 x 16, 12 heads 0.89, 8 x 16
// 0.87, 4 x 32 0.95, 1 x 128, 8 heads 0.97; 16 x 16 0.99, 32 x 16 1.11, 8 x 64, 8 heads 1.07, 1 x 200, 16 heads 1.05).
static bool wkv_in_blocks(int B, int T, int H, int N) {
  return WM_BLOCKS && N == WN && (T > 128 || static_cast<long long>(B) * H * T >= 3072);
}

// Chunks the sequence is cut into.  More than one chunk adds the local passes over all chunks but one, the fold's launches and
// chain, and the states' traffic.  In units of a round of 16 steps; `per_sm`: CTAs on an SM in a last round that is not full.
// In blocks: a block of steps takes as long as the SM's CTAs need: latency until it holds WK_CTAS, so with one or two CTAs 2/3 and
// 5/6 of the time with three, which also holds for the CTAs left over by full rounds (40 x 512, 12 heads: 480 CTAs on 444 places
// take 1.62 rounds).  A round: 16.6 us.  Times of forward + backward by the number of chunks, this rule's first: 1 x 512, 12 heads
// 16: 67 us, 32: 67, 8: 78; 4 x 2048 9: 337, 8: 355, 16: 373, 1: 1387; 8 x 2048, 16 heads 10: 850, 3: 877, 1: 1437; 40 x 300, 12
// heads 1: 515, 3: 542, 19: 908 (the choice when only rounds and steps were counted); 40 x 512 4: 823, 1: 860, 8: 900; 16 x 1000, 16
// heads 5: 844, 1: 871; 10 x 400, 12 heads 3: 207, 1: 267.
// Heads of 32: CTAs of two warps, eight on an SM; the local passes are nearly as long as the others.  us, this rule's first, then
// that of the next line, then that of blocks: 8 x 2048, 16 heads 8: 515, 3: 692, 10: 582; 4 x 2048, 24 heads 12: 394, 4: 520, 9: 411; 2 x
// 4096, 32 heads 16: 517, 20: 587, 13: 540; 40 x 512, 12 heads 1: 440, 8: 487, 4: 473; 4 x 300, 24 heads 10: 84, 4: 98; 10 x 400, 24 heads
// 3: 225, 5: 228, 1: 239; 1 x 8192, 24 heads 29: 466, 18: 498, 32: 438; 32 x 512, 24 heads 1: 597.  Of 19 such calls none is more than
// 7 % above its best count's time, and none slower than with the next line's count.
// Heads of 64 step by step (the local passes are as long as the others): whole rounds.
// The count depends on the batch, and the chunks' states are folded in fp32: a sequence's last bits are not those it has in
// another batch.
constexpr int WK_CTAS = 3, WK_CTAS_32 = 8;
static int wkv_chunk_count(int B, int T, int H, int N) {
  const bool blocks = wkv_in_blocks(B, T, H, N);
  const int subs = (T + WK_SUB - 1) / WK_SUB, slots = (N == 32 ? WK_CTAS_32 : WK_CTAS) * sm_count();
  int best = 1;
  float best_cost = 1e30f;
  for (int nc = 1; nc <= WK_MAX_CHUNKS && nc <= subs; ++nc) {
    const int len = (subs + nc - 1) / nc;
    if ((subs + len - 1) / len != nc) continue;
    const long long ctas = static_cast<long long>(B) * H * nc, full = ctas / slots, rest = ctas - full * slots;
    const int per_sm = static_cast<int>((rest + sm_count() - 1) / sm_count());
    float cost;
    if (blocks)
      cost = len * (full + (rest > 0 ? 0.5f + per_sm / 6.f : 0.f)) * (1.f + 0.3f * (nc - 1) / nc) +
             (nc > 1 ? 1.5f + 0.05f * nc + 0.0015f * ctas : 0.f);
    else if (N == 32)
      cost = len * (full + (rest > 0 ? 0.25f + 0.75f * per_sm / WK_CTAS_32 : 0.f)) * (1.f + 0.7f * (nc - 1) / nc) +
             (nc > 1 ? 0.5f + 0.0005f * ctas : 0.f);
    else
      cost = len * (full + (rest > 0)) * (1.f + 0.67f * (nc - 1) / nc) + (nc > 1 ? 0.5f + 0.1f * nc : 0.f);
    if (cost < best_cost) {
      best_cost = cost;
      best = nc;
    }
  }
  return best;
}
static int wkv_chunk_len(int T, int nc) { return ((T + WK_SUB - 1) / WK_SUB + nc - 1) / nc * WK_SUB; }

static bool wkv_vec_ok(const WkvParams& p) {
  auto ok = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  return ok(p.r) && ok(p.k) && ok(p.v) && ok(p.w) && ok(p.gy) && p.sb % 8 == 0 && p.st % 8 == 0;
}

template <typename Smem, typename K>
static int wkv64_launch(K with_vec, K without, const WkvParams& p, bool vec, int chunks, cudaStream_t stream) {
  const K kern = vec ? with_vec : without;
  NX_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem)));
  kern<<<dim3(chunks, p.H, p.B), WM_THREADS, sizeof(Smem), stream>>>(p);
  NX_LAUNCH_CHECK();
  return NX_OK;
}
template <bool REV, bool LOCAL>
static int wkv_col(const WkvParams& p, bool vec, int chunks, cudaStream_t stream) {
  return wkv64_launch<WmColSmem>(wkv_col_kernel<REV, LOCAL, true>, wkv_col_kernel<REV, LOCAL, false>, p, vec, chunks, stream);
}
template <bool REV>
static int wkv_row(const WkvParams& p, bool vec, cudaStream_t stream) {
  return wkv64_launch<WmRowSmem>(wkv_row_kernel<REV, true>, wkv_row_kernel<REV, false>, p, vec, p.NC, stream);
}

// One sweep, in blocks or step by step.
template <int N, int MODE>
static int wkv_sweep(const WkvParams& p, bool vec, int chunks, cudaStream_t stream) {
  if constexpr (N == WN && WM_BLOCKS) {
    if (wkv_in_blocks(p.B, p.T, p.H, N)) {
      if constexpr (MODE == WK_LOCAL_FWD) return wkv_col<false, true>(p, vec, chunks, stream);
      if constexpr (MODE == WK_LOCAL_REV) return wkv_col<true, true>(p, vec, chunks, stream);
      if constexpr (MODE == WK_Y) return wkv_col<false, false>(p, vec, chunks, stream);
      if constexpr (MODE == WK_GR) return wkv_row<false>(p, vec, stream);
      if constexpr (MODE == WK_G) {
        const int rc = wkv_row<true>(p, vec, stream);
        return rc != NX_OK ? rc : wkv_col<true, false>(p, vec, chunks, stream);
      }
    }
  }
  return wkv_launch<N, MODE>(p, vec, chunks, stream);
}

template <int N>
static int wkv_forward(WkvParams p, float* start, cudaStream_t stream) {
  const bool vec = wkv_vec_ok(p);
  if (p.NC > 1) {
    const int rc = wkv_sweep<N, WK_LOCAL_FWD>(p, vec, p.NC - 1, stream);
    if (rc != NX_OK) return rc;
    wkv_fold_kernel<N, false><<<dim3(N, p.H, p.B), N, 0, stream>>>(p.local, p.sumew, start, p.NC);
    NX_LAUNCH_CHECK();
    p.start = start;
  }
  return wkv_sweep<N, WK_Y>(p, vec, p.NC, stream);
}

template <int N>
static int wkv_backward(WkvParams p, const float* fstart, float* rstart, float* gu, cudaStream_t stream) {
  const bool vec = wkv_vec_ok(p);
  p.start = p.NC > 1 ? fstart : nullptr;
  int rc = wkv_sweep<N, WK_GR>(p, vec, p.NC, stream);
  if (rc != NX_OK) return rc;
  p.start = nullptr;
  if (p.NC > 1) {
    rc = wkv_sweep<N, WK_LOCAL_REV>(p, vec, p.NC - 1, stream);
    if (rc != NX_OK) return rc;
    wkv_fold_kernel<N, true><<<dim3(N, p.H, p.B), N, 0, stream>>>(p.local, p.sumew, rstart, p.NC);
    NX_LAUNCH_CHECK();
    p.start = rstart;
    p.fstart = fstart;
  }
  rc = wkv_sweep<N, WK_G>(p, vec, p.NC, stream);
  if (rc != NX_OK) return rc;
  wkv_sum_kernel<<<(p.H * N + WK_SUM_X - 1) / WK_SUM_X, dim3(WK_SUM_X, WK_SUM_Y), 0, stream>>>(p.gu_part, gu, p.B * p.NC,
                                                                                          p.H * N);
  NX_LAUNCH_CHECK();
  return NX_OK;
}

// Chunks for heads of N, and of 64.
NX_API int NX_SYM(nx_wkv6_head_chunks)(int B, int T, int H, int N) { return wkv_chunk_count(B, T, H, N); }
NX_API int NX_SYM(nx_wkv6_chunks)(int B, int T, int H) { return wkv_chunk_count(B, T, H, WN); }
// Kernels a backward launches (two more where there are several chunks).
NX_API int NX_SYM(nx_wkv6_bwd_launches)(int B, int T, int H, int N) { return wkv_in_blocks(B, T, H, N) ? 4 : 3; }

// r, k, v, w: bf16 [B, T, H*N] addressed by (sb, st); u fp32 [H, N]; y bf16 by (osb, ost).  With NC =
// nx_wkv6_head_chunks(B, T, H, N) > 1: local / start fp32 [B, H, NC, N, N] and sumew fp32 [B, H, NC, N] are scratch, and
// `start` is kept for the backward; they may be null for NC = 1.
NX_API int NX_SYM(nx_wkv6_fwd)(const void* r, const void* k, const void* v, const void* w, long long sb, long long st,
                       const void* u, void* y, long long osb, long long ost, void* local, void* start, void* sumew,
                       int B, int T, int H, int N, cudaStream_t stream) {
  NX_REQUIRE(N == 64 || N == 32, "wkv6: head size %d not supported (32 or 64)", N);
  if (B <= 0 || T <= 0 || H <= 0) return NX_OK;
  WkvParams p{};
  p.r = (const h16*)r; p.k = (const h16*)k; p.v = (const h16*)v; p.w = (const h16*)w;
  p.sb = sb; p.st = st; p.u = (const float*)u;
  p.y = (h16*)y; p.osb = osb; p.ost = ost;
  p.local = (float*)local; p.sumew = (float*)sumew;
  p.B = B; p.T = T; p.H = H; p.NC = wkv_chunk_count(B, T, H, N); p.clen = wkv_chunk_len(T, p.NC);
  return N == 64 ? wkv_forward<64>(p, (float*)start, stream) : wkv_forward<32>(p, (float*)start, stream);
}

// gy like r.  gr / gk / gv / gw: bf16 by (osb, ost); gr32: fp32 scratch of the same shape and strides; gu fp32 [H, N];
// gu_part: fp32 scratch [B, NC, H, N].  fstart: the forward's start states; local, rstart, sumew: scratch (all null for
// NC = 1).
NX_API int NX_SYM(nx_wkv6_bwd)(const void* r, const void* k, const void* v, const void* w, const void* gy, long long sb,
                       long long st, const void* u, void* gr, void* gk, void* gv, void* gw, void* gr32, void* gu,
                       void* gu_part, long long osb, long long ost, void* local, const void* fstart, void* rstart, void* sumew,
                       int B, int T, int H, int N, cudaStream_t stream) {
  NX_REQUIRE(N == 64 || N == 32, "wkv6: head size %d not supported (32 or 64)", N);
  if (B <= 0 || T <= 0 || H <= 0) return NX_OK;
  WkvParams p{};
  p.r = (const h16*)r; p.k = (const h16*)k; p.v = (const h16*)v; p.w = (const h16*)w; p.gy = (const h16*)gy;
  p.sb = sb; p.st = st; p.u = (const float*)u;
  p.o_gr = (h16*)gr; p.o_gk = (h16*)gk; p.o_gv = (h16*)gv; p.o_gw = (h16*)gw;
  p.gr32 = (float*)gr32; p.gu_part = (float*)gu_part; p.osb = osb; p.ost = ost;
  p.local = (float*)local; p.sumew = (float*)sumew;
  p.B = B; p.T = T; p.H = H; p.NC = wkv_chunk_count(B, T, H, N); p.clen = wkv_chunk_len(T, p.NC);
  return N == 64 ? wkv_backward<64>(p, (const float*)fstart, (float*)rstart, (float*)gu, stream)
                 : wkv_backward<32>(p, (const float*)fstart, (float*)rstart, (float*)gu, stream);
}

}  // namespace nx
