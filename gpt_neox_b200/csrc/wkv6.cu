// RWKV-6 WKV recurrence, forward and backward, with no compile-time sequence length.
//
//   y_t[j]   = sum_i r_t[i] * (u[i] * k_t[i] * v_t[j] + S_{t-1}[i][j])
//   S_t[i][j] = d_t[i] * S_{t-1}[i][j] + k_t[i] * v_t[j],      d_t[i] = exp(-exp(w_t[i]))
//
// Counterpart in the reference: megatron/model/rwkv/v6/cuda/wkv6_cuda.cu:6-241 (kernel_forward,
// kernel_backward_111 / _222), which walks the whole sequence in one thread per channel and needs
// the sequence length as a compile-time constant for a per-thread array.
//
// One CTA of 2 N threads walks one head's piece of the sequence with the N x N state in registers: warp w owns 16 columns
// j, a lane N / 8 rows i by 4 columns.  Per step a lane reads N / 8 values of each row vector and 4 of each column
// vector from shared memory (column vectors are stored twice side by side, so that the packed fp32 pairs, which run
// over neighbouring rows, need no register moves) and does 3 packed operations per 2 state elements: one for the output
// sum, two for the update.  The former one-column-per-thread mapping read every row vector whole in every thread, which
// used the shared-memory port as fully as the FMA pipe.  The u term is taken out of the sums: it is a dot product per
// step (formed while staging) times one value.  Sums over rows / columns leave a lane by transposing exchanges.
//   forward  : one sweep: y (sum over i)
//   backward : a forward sweep: gr (sum over j), then ONE reverse sweep of the gradient state G = dL/dS with both
//              gk (sum over j) and gv (sum over i), which also forms the decay gradient: with
//              Q_t[i] = sum_j G_t[i][j] S_t[i][j] one has Q_{t-1} - Q_t = r_t gr_t - k_t gk_t and
//              dL/d(ew_t) = Q_t - k_t (gk_t - r_t u s_t),  s_t = <gy_t, v_t>,  ew = -exp(w)
// 3 + 3 + 4 operations per state element and step; at 32 x 512 tokens, 12 heads of 64, the schedulers have 2.6 warps each and
// are bound by the steps' shared-memory loads and exchanges (that pipe 64-74 % busy, issue slots 38-45 %).  Forward +
// backward of that size: 3.03 ms with one column per thread in seven passes, 0.87 ms with 8 columns per lane and half the
// warps, 0.79 ms now.
//
// The sequence is cut into chunks only when batch x heads leaves the chip idle (wkv_chunk_count): the recurrence is
// linear, so a chunk's end state is  P (.) S_start + S_local  with P[i] = prod_t d_t[i]; local passes start every chunk
// from zero, a fold gives the chunks' start states, and Q at a chunk's end is <G, S> there.
#include "common.h"
#include "ptx.cuh"

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
  if (MODE == WK_G && !second && p.fstart != nullptr && c + 1 < p.NC) {
    const float* g = p.start + (base * N + me) * N;
    const float* f = p.fstart + ((base + 1) * N + me) * N;
    for (int j = 0; j < N; ++j) Q += g[j] * f[j];
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

// start[c] for every chunk: forward  start[0] = 0, start[c+1] = P_c start[c] + local[c];
//                           reverse  start[NC-1] = 0, start[c-1] = P_c start[c] + local[c].
template <int N, bool REV>
__global__ void __launch_bounds__(N) wkv_fold_kernel(const float* local, const float* sumew, float* start, int NC) {
  const int j = threadIdx.x, i = blockIdx.x;
  const long long head = (long long)blockIdx.z * gridDim.y + blockIdx.y;
  float S = 0.f;
  for (int q = 0; q < NC; ++q) {
    const int c = REV ? NC - 1 - q : q;
    const long long o = ((head * NC + c) * N + i) * N + j;
    start[o] = S;
    if (q + 1 < NC) S = S * __expf(sumew[(head * NC + c) * N + i]) + local[o];
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

// Chunks the sequence is cut into.  The sweeps are bound by latency until an SM holds WK_CTAS CTAs, so time goes with the
// chunk length times the number of rounds the CTAs take; more than one chunk adds the local pass (2 of the sweep's 3
// operations) over all chunks but one, and the fold.  The count depends on the batch, and the chunks' states are folded in
// fp32: a sequence's last bits are not those it has in another batch.
constexpr int WK_CTAS = 3;
static int wkv_chunk_count(int B, int T, int H) {
  const int subs = (T + WK_SUB - 1) / WK_SUB, slots = WK_CTAS * sm_count();
  int best = 1;
  float best_cost = 1e30f;
  for (int nc = 1; nc <= WK_MAX_CHUNKS && nc <= subs; ++nc) {
    const int len = (subs + nc - 1) / nc;
    if ((subs + len - 1) / len != nc) continue;
    const long long rounds = (static_cast<long long>(B) * H * nc + slots - 1) / slots;
    const float cost = len * rounds * (1.f + 0.67f * (nc - 1) / nc) + (nc > 1 ? 0.5f + 0.1f * nc : 0.f);
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

template <int N>
static int wkv_forward(WkvParams p, float* start, cudaStream_t stream) {
  const bool vec = wkv_vec_ok(p);
  if (p.NC > 1) {
    int rc = wkv_launch<N, WK_LOCAL_FWD>(p, vec, p.NC - 1, stream);
    if (rc != NX_OK) return rc;
    wkv_fold_kernel<N, false><<<dim3(N, p.H, p.B), N, 0, stream>>>(p.local, p.sumew, start, p.NC);
    NX_LAUNCH_CHECK();
    p.start = start;
  }
  return wkv_launch<N, WK_Y>(p, vec, p.NC, stream);
}

template <int N>
static int wkv_backward(WkvParams p, const float* fstart, float* rstart, float* gu, cudaStream_t stream) {
  const bool vec = wkv_vec_ok(p);
  p.start = p.NC > 1 ? fstart : nullptr;
  int rc = wkv_launch<N, WK_GR>(p, vec, p.NC, stream);
  if (rc != NX_OK) return rc;
  p.start = nullptr;
  if (p.NC > 1) {
    rc = wkv_launch<N, WK_LOCAL_REV>(p, vec, p.NC - 1, stream);
    if (rc != NX_OK) return rc;
    wkv_fold_kernel<N, true><<<dim3(N, p.H, p.B), N, 0, stream>>>(p.local, p.sumew, rstart, p.NC);
    NX_LAUNCH_CHECK();
    p.start = rstart;
    p.fstart = fstart;
  }
  rc = wkv_launch<N, WK_G>(p, vec, p.NC, stream);
  if (rc != NX_OK) return rc;
  wkv_sum_kernel<<<(p.H * N + WK_SUM_X - 1) / WK_SUM_X, dim3(WK_SUM_X, WK_SUM_Y), 0, stream>>>(p.gu_part, gu, p.B * p.NC,
                                                                                          p.H * N);
  NX_LAUNCH_CHECK();
  return NX_OK;
}

NX_API int NX_SYM(nx_wkv6_chunks)(int B, int T, int H) { return wkv_chunk_count(B, T, H); }

// r, k, v, w: bf16 [B, T, H*N] addressed by (sb, st); u fp32 [H, N]; y bf16 by (osb, ost).  With NC =
// nx_wkv6_chunks(B, T, H) > 1: local / start fp32 [B, H, NC, N, N] and sumew fp32 [B, H, NC, N] are scratch, and
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
  p.B = B; p.T = T; p.H = H; p.NC = wkv_chunk_count(B, T, H); p.clen = wkv_chunk_len(T, p.NC);
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
  p.B = B; p.T = T; p.H = H; p.NC = wkv_chunk_count(B, T, H); p.clen = wkv_chunk_len(T, p.NC);
  return N == 64 ? wkv_backward<64>(p, (const float*)fstart, (float*)rstart, (float*)gu, stream)
                 : wkv_backward<32>(p, (const float*)fstart, (float*)rstart, (float*)gu, stream);
}

}  // namespace nx
