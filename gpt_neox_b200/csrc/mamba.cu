// Mamba-1 kernels: causal depthwise conv1d (width <= 4) + SiLU, and the S6 selective scan, forward
// and backward, on token-major activations addressed by (batch stride, time stride) so the
// [seq, batch, channel] tensors the projections produce are consumed without a transpose.
//
// Counterparts in the reference: causal_conv1d_fn and selective_scan_fn / selective_scan_ref from
// the external causal_conv1d / mamba_ssm packages, called at megatron/model/mamba/mamba.py:220-247
// and :264-320 (which run on [batch, channel, seq] and need two rearranges per block).
//
// Scan parallelisation: a thread owns 4 of the 16 states of one channel (a quad of lanes per channel), 32 channels per
// CTA, and walks its piece of the sequence in blocks of 32 steps.  The sequence is cut into as few chunks as keep the
// chip busy (scan_chunk_count): one chunk needs one pass; with more, a light pass first runs every chunk from a zero
// state and records its end state and its sum of delta (the chunk's decay is exp(A * sum delta)), and the main pass
// folds the earlier chunks into its start state.  The reverse recurrence of dL/dh is cut the same way.
// The forward keeps the state at the start of every 32-step block for the backward, which recomputes 8 steps at a
// time into registers and walks them in reverse.  Those states take 2 bytes per token and channel from the forward to the
// backward (25 MB for 4 x 2048 x 1536, as much as one more 16-bit activation; 6 MB when a state per 128 steps was kept),
// and the tiles' partial sums of dB and dC 4 bytes during the backward.
// Bound by the shared-memory pipe (78-80 % busy in the main passes: a step's inputs, and the exchanges that sum dB, dC and
// the channel sums over lanes); issue slots 42-50 %, DRAM 6-9 %.  Convolution + scan, forward + backward, 4 x
// 2048 steps of 1536 channels: 1.78 ms with chunks of 128 steps in two passes each way, the states recomputed in three of
// them and scalar staging; 0.98 ms with two (forward three) CTAs an SM; 0.86 ms with the exchanges of dB / dC step by
// step; 0.82 ms now (backward sweep 418 us, 466 before).
#include "common.h"
#include "ptx.cuh"

namespace nx {

// ---------------------------------------------------------------------------------------------
// causal depthwise conv1d + SiLU
// ---------------------------------------------------------------------------------------------
constexpr int CONV_TILE = 64;   // timesteps per thread

__device__ __forceinline__ float ldbf(const h16* p) { return h16_to_float(*p); }

// y[b,t,d] = silu(bias[d] + sum_k w[d,k] * x[b, t-(W-1)+k, d])
__global__ void __launch_bounds__(128)
conv1d_silu_fwd_kernel(const h16* __restrict__ x, long long xsb, long long xst,
                       const h16* __restrict__ w, const h16* __restrict__ bias,
                       h16* __restrict__ y, long long ysb, long long yst, int L, int D, int W) {
  const int d = blockIdx.x * 128 + threadIdx.x;
  if (d >= D) return;
  const int t0 = blockIdx.y * CONV_TILE;
  const int b = blockIdx.z;
  float wk[4] = {0.f, 0.f, 0.f, 0.f};
  for (int k = 0; k < W; ++k) wk[4 - W + k] = ldbf(w + (long long)d * W + k);
  const float bv = bias ? ldbf(bias + d) : 0.f;
  const h16* xp = x + b * xsb + d;
  float win[4];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int t = t0 - 3 + k;
    win[k + 1] = t >= 0 ? ldbf(xp + t * xst) : 0.f;
  }
  const int t1 = min(t0 + CONV_TILE, L);
  for (int t = t0; t < t1; ++t) {
    win[0] = win[1]; win[1] = win[2]; win[2] = win[3];
    win[3] = ldbf(xp + t * xst);
    const float pre = bv + wk[0] * win[0] + wk[1] * win[1] + wk[2] * win[2] + wk[3] * win[3];
    y[b * ysb + t * yst + d] = float_to_h16(silu(pre));
  }
}

// dx[t] = sum_k w[k] * dpre[t + (3-k)];  dw[k] += dpre[t] * x[t-3+k];  dbias += dpre[t]
__global__ void __launch_bounds__(128)
conv1d_silu_bwd_kernel(const h16* __restrict__ x, long long xsb, long long xst,
                       const h16* __restrict__ w, const h16* __restrict__ bias,
                       const h16* __restrict__ dy, long long dsb, long long dst,
                       h16* __restrict__ dx, long long gsb, long long gst,
                       float* __restrict__ dw, float* __restrict__ dbias, int L, int D, int W) {
  const int d = blockIdx.x * 128 + threadIdx.x;
  if (d >= D) return;
  const int t0 = blockIdx.y * CONV_TILE;
  const int b = blockIdx.z;
  float wk[4] = {0.f, 0.f, 0.f, 0.f};
  for (int k = 0; k < W; ++k) wk[4 - W + k] = ldbf(w + (long long)d * W + k);
  const float bv = bias ? ldbf(bias + d) : 0.f;
  const h16* xp = x + b * xsb + d;
  const h16* gp = dy + b * dsb + d;
  float win[4], dp[4] = {0.f, 0.f, 0.f, 0.f};
  float aw[4] = {0.f, 0.f, 0.f, 0.f}, ab = 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int t = t0 - 3 + k;
    win[k + 1] = t >= 0 ? ldbf(xp + t * xst) : 0.f;
  }
  const int t_own = min(t0 + CONV_TILE, L);
  const int t_end = min(t0 + CONV_TILE + 3, L + 3);
  for (int t = t0; t < t_end; ++t) {
    win[0] = win[1]; win[1] = win[2]; win[2] = win[3];
    win[3] = t < L ? ldbf(xp + t * xst) : 0.f;
    float dpre = 0.f;
    if (t < L) {
      const float pre = bv + wk[0] * win[0] + wk[1] * win[1] + wk[2] * win[2] + wk[3] * win[3];
      dpre = ldbf(gp + t * dst) * silu_grad(pre);
    }
    if (t < t_own) {
      aw[0] += dpre * win[0]; aw[1] += dpre * win[1]; aw[2] += dpre * win[2]; aw[3] += dpre * win[3];
      ab += dpre;
    }
    dp[0] = dp[1]; dp[1] = dp[2]; dp[2] = dp[3]; dp[3] = dpre;   // dp[j] = dpre[t-3+j]
    const int to = t - 3;
    if (to >= t0 && to < t_own)
      dx[b * gsb + to * gst + d] =
          float_to_h16(wk[3] * dp[0] + wk[2] * dp[1] + wk[1] * dp[2] + wk[0] * dp[3]);
  }
  for (int k = 0; k < W; ++k) atomicAdd(dw + (long long)d * W + k, aw[4 - W + k]);
  if (dbias) atomicAdd(dbias + d, ab);
}

// Vector forms: a thread owns V neighbouring channels (one V * 2-byte load per step) and CV_T steps; the steps' loads
// are issued before the first use.  The one-channel kernels above keep one 2-byte load in flight per thread and are
// bound by its latency; they remain for channel counts, strides or bases that are not multiples of V elements.
constexpr int CV_X = 32;    // channel groups per block
constexpr int CV_Y = 4;     // time tiles per block
constexpr int CV_T = 16;    // steps per thread
constexpr int CV_FWD_V = 8, CV_BWD_V = 4;

template <int V>
__device__ __forceinline__ void load_vec(const h16* p, float (&f)[V]) {
  uint32_t w[V / 2];
  if constexpr (V == 8) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    w[0] = u.x; w[1] = u.y; w[2] = u.z; w[3] = u.w;
  } else {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    w[0] = u.x; w[1] = u.y;
  }
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {
    const float2 a = unpack_h16x2(w[i]);
    f[2 * i] = a.x;
    f[2 * i + 1] = a.y;
  }
}
template <int V>
__device__ __forceinline__ void store_vec(h16* p, const float (&f)[V]) {
  if constexpr (V == 8)
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_h16x2(f[0], f[1]), pack_h16x2(f[2], f[3]), pack_h16x2(f[4], f[5]),
                                              pack_h16x2(f[6], f[7]));
  else
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_h16x2(f[0], f[1]), pack_h16x2(f[2], f[3]));
}
template <int V>
__device__ __forceinline__ void load_taps(const h16* w, int d, int W, float (&wk)[V][4]) {
#pragma unroll
  for (int c = 0; c < V; ++c)
#pragma unroll
    for (int k = 0; k < 4; ++k) wk[c][k] = k >= 4 - W ? ldbf(w + (long long)(d + c) * W + k - (4 - W)) : 0.f;
}

__global__ void __launch_bounds__(CV_X * CV_Y)
conv1d_silu_fwd_vec_kernel(const h16* __restrict__ x, long long xsb, long long xst, const h16* __restrict__ w,
                           const h16* __restrict__ bias, h16* __restrict__ y, long long ysb, long long yst, int L,
                           int D, int W) {
  constexpr int V = CV_FWD_V;
  const int d = (blockIdx.x * CV_X + threadIdx.x) * V;
  const int t0 = (blockIdx.y * CV_Y + threadIdx.y) * CV_T, b = blockIdx.z;
  if (d >= D || t0 >= L) return;
  float wk[V][4], bv[V], win[3][V];
  load_taps<V>(w, d, W, wk);
  const h16* xp = x + b * xsb + d;
#pragma unroll
  for (int c = 0; c < V; ++c) bv[c] = bias ? ldbf(bias + d + c) : 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int c = 0; c < V; ++c) win[k][c] = 0.f;
    if (t0 - 3 + k >= 0) load_vec<V>(xp + (t0 - 3 + k) * xst, win[k]);
  }
#pragma unroll 1
  for (int s = 0; s < CV_T; s += 8) {
    uint4 raw[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (t0 + s + u < L) raw[u] = *reinterpret_cast<const uint4*>(xp + (t0 + s + u) * xst);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int t = t0 + s + u;
      if (t < L) {
        const uint32_t ww[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
        float o[V];
#pragma unroll
        for (int c = 0; c < V; ++c) {
          const float2 p2 = unpack_h16x2(ww[c / 2]);
          const float cur = (c & 1) ? p2.y : p2.x;
          o[c] = silu(bv[c] + wk[c][0] * win[0][c] + wk[c][1] * win[1][c] + wk[c][2] * win[2][c] + wk[c][3] * cur);
          win[0][c] = win[1][c]; win[1][c] = win[2][c]; win[2][c] = cur;
        }
        store_vec<V>(y + b * ysb + t * yst + d, o);
      }
    }
  }
}

__global__ void __launch_bounds__(CV_X * CV_Y)
conv1d_silu_bwd_vec_kernel(const h16* __restrict__ x, long long xsb, long long xst, const h16* __restrict__ w,
                           const h16* __restrict__ bias, const h16* __restrict__ dy, long long dsb, long long dst,
                           h16* __restrict__ dx, long long gsb, long long gst, float* __restrict__ dw,
                           float* __restrict__ dbias, int L, int D, int W) {
  constexpr int V = CV_BWD_V;
  __shared__ float red[CV_Y][CV_X][V * 5 + 1];
  const int d = (blockIdx.x * CV_X + threadIdx.x) * V;
  const int t0 = (blockIdx.y * CV_Y + threadIdx.y) * CV_T, b = blockIdx.z;
  float aw[V][5];
#pragma unroll
  for (int c = 0; c < V; ++c)
#pragma unroll
    for (int k = 0; k < 5; ++k) aw[c][k] = 0.f;
  if (d < D && t0 < L) {
    float wk[V][4], bv[V], win[3][V], dp[3][V];
    load_taps<V>(w, d, W, wk);
    const h16* xp = x + b * xsb + d;
    const h16* gp = dy + b * dsb + d;
#pragma unroll
    for (int c = 0; c < V; ++c) {
      bv[c] = bias ? ldbf(bias + d + c) : 0.f;
      dp[0][c] = dp[1][c] = dp[2][c] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
#pragma unroll
      for (int c = 0; c < V; ++c) win[k][c] = 0.f;
      if (t0 - 3 + k >= 0) load_vec<V>(xp + (t0 - 3 + k) * xst, win[k]);
    }
    const int t_own = min(t0 + CV_T, L);
    // three steps beyond the tile: their dpre reaches back into it
#pragma unroll 1
    for (int s = 0; s < CV_T + 3; s += 4) {
      uint2 rx[4], rg[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        rx[u] = rg[u] = make_uint2(0u, 0u);
        const int t = t0 + s + u;
        if (t < L && s + u < CV_T + 3) {
          rx[u] = *reinterpret_cast<const uint2*>(xp + t * xst);
          rg[u] = *reinterpret_cast<const uint2*>(gp + t * dst);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int t = t0 + s + u, to = t - 3;
        const float2 x0 = unpack_h16x2(rx[u].x), x1 = unpack_h16x2(rx[u].y);
        const float2 g0 = unpack_h16x2(rg[u].x), g1 = unpack_h16x2(rg[u].y);
        const float xc[4] = {x0.x, x0.y, x1.x, x1.y}, gc[4] = {g0.x, g0.y, g1.x, g1.y};
        float o[V];
#pragma unroll
        for (int c = 0; c < V; ++c) {
          const float pre = bv[c] + wk[c][0] * win[0][c] + wk[c][1] * win[1][c] + wk[c][2] * win[2][c] + wk[c][3] * xc[c];
          const float dpre = gc[c] * silu_grad(pre);      // 0 beyond the sequence: dy was read as 0 there
          if (t < t_own) {
            aw[c][0] += dpre * win[0][c]; aw[c][1] += dpre * win[1][c]; aw[c][2] += dpre * win[2][c];
            aw[c][3] += dpre * xc[c];
            aw[c][4] += dpre;
          }
          o[c] = wk[c][3] * dp[0][c] + wk[c][2] * dp[1][c] + wk[c][1] * dp[2][c] + wk[c][0] * dpre;
          win[0][c] = win[1][c]; win[1][c] = win[2][c]; win[2][c] = xc[c];
          dp[0][c] = dp[1][c]; dp[1][c] = dp[2][c]; dp[2][c] = dpre;
        }
        if (to >= t0 && to < t_own) store_vec<V>(dx + b * gsb + to * gst + d, o);
      }
    }
  }
  // one atomic per block and parameter: the block's time tiles are summed in shared memory first
#pragma unroll
  for (int c = 0; c < V; ++c)
#pragma unroll
    for (int k = 0; k < 5; ++k) red[threadIdx.y][threadIdx.x][c * 5 + k] = aw[c][k];
  __syncthreads();
  for (int i = threadIdx.y * CV_X + threadIdx.x; i < CV_X * V * 5; i += CV_X * CV_Y) {
    const int gx = i / (V * 5), r = i % (V * 5), ch = (blockIdx.x * CV_X + gx) * V + r / 5, k = r % 5;
    if (ch >= D) continue;
    float a = 0.f;
#pragma unroll
    for (int ty = 0; ty < CV_Y; ++ty) a += red[ty][gx][r];
    if (k == 4) {
      if (dbias) atomicAdd(dbias + ch, a);
    } else if (k >= 4 - W) {
      atomicAdd(dw + (long long)ch * W + k - (4 - W), a);
    }
  }
}

static bool vec_ok(const void* p, long long sb, long long st, int V) {
  return (reinterpret_cast<uintptr_t>(p) & (V * 2 - 1)) == 0 && sb % V == 0 && st % V == 0;
}
static dim3 conv_vec_grid(int B, int L, int D, int V) {
  return dim3((D / V + CV_X - 1) / CV_X, (L + CV_T * CV_Y - 1) / (CV_T * CV_Y), B);
}

NX_API int NX_SYM(nx_conv1d_silu_fwd)(const void* x, long long xsb, long long xst, const void* w, const void* bias,
                              void* y, long long ysb, long long yst, int B, int L, int D, int W,
                              cudaStream_t stream) {
  NX_REQUIRE(W >= 1 && W <= 4, "conv1d: kernel width %d not in [1, 4]", W);
  if (D % CV_FWD_V == 0 && vec_ok(x, xsb, xst, CV_FWD_V) && vec_ok(y, ysb, yst, CV_FWD_V)) {
    conv1d_silu_fwd_vec_kernel<<<conv_vec_grid(B, L, D, CV_FWD_V), dim3(CV_X, CV_Y), 0, stream>>>(
        (const h16*)x, xsb, xst, (const h16*)w, (const h16*)bias, (h16*)y, ysb, yst, L, D, W);
    NX_LAUNCH_CHECK();
    return NX_OK;
  }
  dim3 grid((D + 127) / 128, (L + CONV_TILE - 1) / CONV_TILE, B);
  conv1d_silu_fwd_kernel<<<grid, 128, 0, stream>>>((const h16*)x, xsb, xst, (const h16*)w,
                                                   (const h16*)bias, (h16*)y, ysb, yst, L, D, W);
  NX_LAUNCH_CHECK();
  return NX_OK;
}

// dw [D, W] and dbias [D] are fp32 and must be zeroed by the caller.
NX_API int NX_SYM(nx_conv1d_silu_bwd)(const void* x, long long xsb, long long xst, const void* w, const void* bias,
                              const void* dy, long long dsb, long long dst, void* dx, long long gsb,
                              long long gst, void* dw, void* dbias, int B, int L, int D, int W,
                              cudaStream_t stream) {
  NX_REQUIRE(W >= 1 && W <= 4, "conv1d: kernel width %d not in [1, 4]", W);
  if (D % CV_BWD_V == 0 && vec_ok(x, xsb, xst, CV_BWD_V) && vec_ok(dy, dsb, dst, CV_BWD_V) &&
      vec_ok(dx, gsb, gst, CV_BWD_V)) {
    conv1d_silu_bwd_vec_kernel<<<conv_vec_grid(B, L, D, CV_BWD_V), dim3(CV_X, CV_Y), 0, stream>>>(
        (const h16*)x, xsb, xst, (const h16*)w, (const h16*)bias, (const h16*)dy, dsb, dst, (h16*)dx, gsb, gst,
        (float*)dw, (float*)dbias, L, D, W);
    NX_LAUNCH_CHECK();
    return NX_OK;
  }
  dim3 grid((D + 127) / 128, (L + CONV_TILE - 1) / CONV_TILE, B);
  conv1d_silu_bwd_kernel<<<grid, 128, 0, stream>>>(
      (const h16*)x, xsb, xst, (const h16*)w, (const h16*)bias,
      (const h16*)dy, dsb, dst, (h16*)dx, gsb, gst, (float*)dw, (float*)dbias, L, D, W);
  NX_LAUNCH_CHECK();
  return NX_OK;
}


// ---------------------------------------------------------------------------------------------
// selective scan
// ---------------------------------------------------------------------------------------------
constexpr int SC_CH = 32;       // channels per CTA
constexpr int SC_T = 32;        // timesteps per block (staged together; the forward keeps a state per block)
constexpr int SC_REG = 8;       // steps whose states the backward holds in registers
constexpr int SC_THREADS = SC_CH * 4;
constexpr int SC_LD = 40;       // row length of the [step][channel] result arrays: four steps land on distinct banks
constexpr int SC_MAX_CHUNKS = 32;
constexpr int SC_FWD_CTAS = 5, SC_BWD_CTAS = 3;   // CTAs per SM: latency (exponentials, shared memory, exchanges) is hidden
                                                  // by other warps, so registers are bounded for more of them
constexpr float LOG2E = 1.44269504088896340736f, LN2 = 0.69314718055994530942f;

struct ScanParams {
  const h16 *x, *dt, *z, *Bm, *Cm, *dout;
  long long xsb, xst, dsb, dst, zsb, zst, bsb, bst, csb, cst, gsb, gst;
  const float *A, *Dv, *dt_bias;
  h16 *out, *dx, *ddt, *dz;       // [.., D] with strides osb / ost
  long long osb, ost;
  float *chunk_state, *chunk_sumdt;   // [B, NC, D, 16] / [B, NC, D]: end state (or reverse carry) and sum of delta
  float *ckpt;                        // [B, ceil(L / 32), D, 16]: state at the start of every block; null = not kept
  float *partBC;                      // [ceil(D / 32), B, L, 32]
  float *dA, *dD, *dbias;
  int B, L, D, NC, clen;              // clen: steps per chunk, a multiple of SC_T
};

__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(__expf(v)); }
__device__ __forceinline__ float sigmoid_f(float v) { return 1.f / (1.f + __expf(-v)); }

// Sums four values per lane over the quad: lane q returns the total of v[q] (three exchanges instead of eight).
__device__ __forceinline__ float quad_transpose_sum(const float (&v)[4], int q) {
  const bool hi = q & 2, odd = q & 1;
  float a = hi ? v[2] : v[0], b = hi ? v[3] : v[1];
  a += __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 2);
  b += __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 2);
  const float keep = odd ? b : a;
  return keep + __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
}

// The staging role of a thread: step tid / 4 of the block, 8 channels from (tid % 4) * 8.
struct RowOf8 {
  int t, c8, d;     // step in block, first channel in tile, first channel
  int n;            // live channels (0..8)
};
__device__ __forceinline__ RowOf8 row_of8(int d0, int D) {
  RowOf8 r;
  r.t = threadIdx.x >> 2;
  r.c8 = (threadIdx.x & 3) * 8;
  r.d = d0 + r.c8;
  r.n = min(8, max(0, D - r.d));
  return r;
}
// 8 consecutive 16-bit elements (zero where dead): one 16-byte load when VEC, single elements otherwise.
template <bool VEC>
__device__ __forceinline__ uint4 load8(const h16* p, int n) {
  uint4 u = make_uint4(0u, 0u, 0u, 0u);
  if (VEC) {
    if (n > 0) u = *reinterpret_cast<const uint4*>(p);
    return u;
  }
  uint16_t e[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) e[j] = j < n ? reinterpret_cast<const uint16_t*>(p)[j] : 0;
  u.x = e[0] | (uint32_t)e[1] << 16; u.y = e[2] | (uint32_t)e[3] << 16;
  u.z = e[4] | (uint32_t)e[5] << 16; u.w = e[6] | (uint32_t)e[7] << 16;
  return u;
}
template <bool VEC>
__device__ __forceinline__ void store8(h16* p, const float (&f)[8], int n) {
  if (VEC) {
    if (n > 0) store_vec<8>(p, f);
    return;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < n) p[j] = float_to_h16(f[j]);
}
__device__ __forceinline__ void unpack8f(const uint4& u, float (&f)[8]) {
  const float2 a = unpack_h16x2(u.x), b = unpack_h16x2(u.y), c = unpack_h16x2(u.z), d = unpack_h16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ void load_coef(const float* p, const RowOf8& r, float (&f)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = (p != nullptr && j < r.n) ? p[r.d + j] : 0.f;
}

// B or C of a block: 32 steps x 16 states, one column of 4 steps per thread.
// They stay 16-bit in shared memory, so a step reads 4 states of each in 8 bytes and not 16: the pipe of shared memory and
// exchanges bounded the scans (70 - 80 % busy with floats here; its wavefronts are at 49 - 73 % of their rate now, issue
// slots at 48 - 63 %).  4 x 2048 x 1536, fp16,
// us: final forward pass 131 -> 119, its light pass 72.5 -> 70.1, backward light pass 95.9 -> 86.7, backward 413 -> 406.
__device__ __forceinline__ void load_bc(const h16* p, long long st, int t0, int t_end, uint16_t (&v)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int t = (threadIdx.x >> 4) + 8 * k;
    v[k] = t0 + t < t_end ? reinterpret_cast<const uint16_t*>(p)[(t0 + t) * st + (threadIdx.x & 15)] : 0;
  }
}
__device__ __forceinline__ void put_bc(uint16_t (*s)[16], const uint16_t (&v)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) s[(threadIdx.x >> 4) + 8 * k][threadIdx.x & 15] = v[k];
}
__device__ __forceinline__ float4 bc4(const uint16_t* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack_h16x2(u.x), b = unpack_h16x2(u.y);
  return make_float4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ void exp4(float2 a01, float2 a23, float dl, float2 (&a)[2]) {
  const float2 d2 = make_float2(dl, dl);
  const float2 u = fmul2(d2, a01), v = fmul2(d2, a23);
  a[0] = make_float2(exp2f(u.x), exp2f(u.y));
  a[1] = make_float2(exp2f(v.x), exp2f(v.y));
}
__device__ __forceinline__ float4 f4(const float2 (&h)[2]) { return make_float4(h[0].x, h[0].y, h[1].x, h[1].y); }

// FINAL = false: chunks 0 .. NC - 2 from a zero state -> end state and sum of delta.
template <bool FINAL, bool VEC>
__global__ void __launch_bounds__(SC_THREADS, SC_FWD_CTAS)
scan_fwd_kernel(const ScanParams p) {
  __shared__ __align__(16) float2 dd[SC_T][SC_CH];        // (delta, delta * x)
  __shared__ __align__(16) uint16_t Bs[SC_T][16], Cs[FINAL ? SC_T : 1][16];
  __shared__ __align__(16) float ys[FINAL ? SC_T : 1][SC_LD];
  const int ch = threadIdx.x >> 2, q = threadIdx.x & 3;
  const int d0 = blockIdx.x * SC_CH, d = d0 + ch;
  const int c = blockIdx.y, b = blockIdx.z;
  const bool dv_ok = d < p.D;
  const int dd_ = dv_ok ? d : 0;
  const RowOf8 row = row_of8(d0, p.D);
  const float4 Av = *reinterpret_cast<const float4*>(p.A + dd_ * 16 + q * 4);
  const float2 A01 = make_float2(Av.x * LOG2E, Av.y * LOG2E), A23 = make_float2(Av.z * LOG2E, Av.w * LOG2E);
  float2 h[2] = {{0.f, 0.f}, {0.f, 0.f}};
  if (FINAL) {
    for (int cp = 0; cp < c; ++cp) {
      const long long o = ((long long)b * p.NC + cp) * p.D + dd_;
      float2 a[2];
      exp4(A01, A23, p.chunk_sumdt[o], a);
      const float4 e = *reinterpret_cast<const float4*>(p.chunk_state + o * 16 + q * 4);
      h[0] = ffma2(h[0], a[0], make_float2(e.x, e.y));
      h[1] = ffma2(h[1], a[1], make_float2(e.z, e.w));
    }
  }
  const int tc0 = c * p.clen, t_end = min(tc0 + p.clen, p.L);
  const h16 *xp = p.x + b * p.xsb + row.d, *dp = p.dt + b * p.dsb + row.d;
  const h16* zp = p.z != nullptr ? p.z + b * p.zsb + row.d : nullptr;
  const h16 *bp = p.Bm + b * p.bsb, *cp_ = p.Cm + b * p.csb;
  float bias8[8];
  load_coef(p.dt_bias, row, bias8);
  float sdt = 0.f;
  uint4 xu, du, zu = make_uint4(0u, 0u, 0u, 0u);
  uint16_t bv[4], cv[4];
  auto fetch = [&](int t0) {
    const int n = t0 + row.t < t_end ? row.n : 0;
    xu = load8<VEC>(xp + (t0 + row.t) * p.xst, n);
    du = load8<VEC>(dp + (t0 + row.t) * p.dst, n);
    if (FINAL && zp != nullptr) zu = load8<VEC>(zp + (t0 + row.t) * p.zst, n);
    load_bc(bp, p.bst, t0, t_end, bv);
    if (FINAL) load_bc(cp_, p.cst, t0, t_end, cv);
  };
  fetch(tc0);
  for (int t0 = tc0; t0 < t_end; t0 += SC_T) {
    const bool in = t0 + row.t < t_end;
    float xv[8], dv[8];
    unpack8f(xu, xv);
    unpack8f(du, dv);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float dl = in && j < row.n ? softplus_f(dv[j] + bias8[j]) : 0.f;
      dd[row.t][row.c8 + j] = make_float2(dl, dl * xv[j]);
    }
    put_bc(Bs, bv);
    if (FINAL) put_bc(Cs, cv);
    const uint4 zc = zu;
    if (t0 + SC_T < t_end) fetch(t0 + SC_T);      // in flight during the 32 steps
    if (FINAL && p.ckpt != nullptr && dv_ok)
      *reinterpret_cast<float4*>(p.ckpt + (((long long)b * ((p.L + SC_T - 1) / SC_T) + t0 / SC_T) * p.D + d) * 16 + q * 4) =
          f4(h);
    __syncthreads();
    const int live = t_end - t0;                  // (padded steps of the last group of four leave the state as it is)
#pragma unroll 2
    for (int g = 0; g < SC_T && g < live; g += 4) {
      float yp[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int t = g + u;
        const float2 dv2 = dd[t][ch];
        const float4 B4 = bc4(&Bs[t][q * 4]);
        const float2 dx2 = make_float2(dv2.y, dv2.y);
        float2 a[2];
        exp4(A01, A23, dv2.x, a);
        h[0] = ffma2(a[0], h[0], fmul2(dx2, make_float2(B4.x, B4.y)));
        h[1] = ffma2(a[1], h[1], fmul2(dx2, make_float2(B4.z, B4.w)));
        if (FINAL) {
          const float4 C4 = bc4(&Cs[t][q * 4]);
          const float2 y2 = ffma2(h[1], make_float2(C4.z, C4.w), fmul2(h[0], make_float2(C4.x, C4.y)));
          yp[u] = y2.x + y2.y;
        } else {
          sdt += dv2.x;
        }
      }
      if (FINAL) ys[g + q][ch] = quad_transpose_sum(yp, q);
    }
    __syncthreads();
    if (FINAL) {
      if (in) {
        float y8[8], z8[8];
        unpack8f(zc, z8);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float Dj = p.Dv != nullptr && j < row.n ? p.Dv[row.d + j] : 0.f;
          y8[j] = ys[row.t][row.c8 + j] + Dj * xv[j];
          if (zp != nullptr) y8[j] *= silu(z8[j]);
        }
        store8<VEC>(p.out + b * p.osb + (t0 + row.t) * p.ost + row.d, y8, row.n);
      }
    }
  }
  if (!FINAL && dv_ok) {
    const long long o = ((long long)b * p.NC + c) * p.D + d;
    *reinterpret_cast<float4*>(p.chunk_state + o * 16 + q * 4) = f4(h);
    if (q == 0) p.chunk_sumdt[o] = sdt;
  }
}

// Reverse recurrence of chunks 1 .. NC - 1 from a zero carry: chunk_state[c] = what chunk c hands to chunk c - 1.
template <bool VEC>
__global__ void __launch_bounds__(SC_THREADS)
scan_bwd_local_kernel(const ScanParams p) {
  __shared__ __align__(16) float2 dd[SC_T][SC_CH];        // (delta, gradient of the ungated output)
  __shared__ __align__(16) uint16_t Cs[SC_T][16];
  const int ch = threadIdx.x >> 2, q = threadIdx.x & 3;
  const int d0 = blockIdx.x * SC_CH, d = d0 + ch;
  const int c = blockIdx.y + 1, b = blockIdx.z;
  const bool dv_ok = d < p.D;
  const RowOf8 row = row_of8(d0, p.D);
  const float4 Av = *reinterpret_cast<const float4*>(p.A + (dv_ok ? d : 0) * 16 + q * 4);
  const float2 A01 = make_float2(Av.x * LOG2E, Av.y * LOG2E), A23 = make_float2(Av.z * LOG2E, Av.w * LOG2E);
  float2 r[2] = {{0.f, 0.f}, {0.f, 0.f}};
  const int tc0 = c * p.clen, t_end = min(tc0 + p.clen, p.L);
  float bias8[8];
  load_coef(p.dt_bias, row, bias8);
  float sdt = 0.f;
  for (int t0 = tc0 + (t_end - 1 - tc0) / SC_T * SC_T; t0 >= tc0; t0 -= SC_T) {
    const int tt = t0 + row.t;
    const bool in = tt < t_end;
    const int n = in ? row.n : 0;
    const uint4 du = load8<VEC>(p.dt + b * p.dsb + tt * p.dst + row.d, n);
    const uint4 gu = load8<VEC>(p.dout + b * p.gsb + tt * p.gst + row.d, n);
    float dv[8], gv[8], zv[8];
    uint16_t cv[4];
    unpack8f(du, dv);
    unpack8f(gu, gv);
    if (p.z != nullptr) unpack8f(load8<VEC>(p.z + b * p.zsb + tt * p.zst + row.d, n), zv);
    load_bc(p.Cm + b * p.csb, p.cst, t0, t_end, cv);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j)
      dd[row.t][row.c8 + j] = make_float2(in && j < row.n ? softplus_f(dv[j] + bias8[j]) : 0.f,
                                          p.z != nullptr ? gv[j] * silu(zv[j]) : gv[j]);
    put_bc(Cs, cv);
    __syncthreads();
#pragma unroll
    for (int t = SC_T - 1; t >= 0; --t) {
      const float2 v = dd[t][ch];
      const float4 C4 = bc4(&Cs[t][q * 4]);
      const float2 g2 = make_float2(v.y, v.y);
      float2 a[2];
      exp4(A01, A23, v.x, a);
      r[0] = fmul2(a[0], ffma2(make_float2(C4.x, C4.y), g2, r[0]));
      r[1] = fmul2(a[1], ffma2(make_float2(C4.z, C4.w), g2, r[1]));
      sdt += v.x;
    }
  }
  if (dv_ok) {
    const long long o = ((long long)b * p.NC + c) * p.D + d;
    *reinterpret_cast<float4*>(p.chunk_state + o * 16 + q * 4) = f4(r);
    if (q == 0) p.chunk_sumdt[o] = sdt;
  }
}

struct ScanBwdSmem {
  float4 dd[SC_T][SC_CH];                     // delta, delta * x, gradient of the ungated output, sigmoid(dt)
  uint16_t Bs[SC_T][16], Cs[SC_T][16];
  float dzf[SC_T][SC_LD];                     // d out / d z without the scan value
  float s_gb[SC_T][SC_LD], s_da[SC_T][SC_LD], s_hc[SC_T][SC_LD];   // sums over the 16 states
  float4 ck[SC_T / SC_REG][SC_THREADS];       // states at the starts of the block's quarters
  float acc[SC_THREADS][17];                  // dD and dbias of a staging thread's 8 channels
  float bc[SC_THREADS / 32][SC_T][32];
};

template <bool VEC>
__global__ void __launch_bounds__(SC_THREADS, SC_BWD_CTAS)
scan_bwd_kernel(const ScanParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ScanBwdSmem& s = *reinterpret_cast<ScanBwdSmem*>(smem_raw);
  const int ch = threadIdx.x >> 2, q = threadIdx.x & 3;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int d0 = blockIdx.x * SC_CH, d = d0 + ch;
  const int c = blockIdx.y, b = blockIdx.z;
  const bool dv_ok = d < p.D;
  const int dd_ = dv_ok ? d : 0;
  const RowOf8 row = row_of8(d0, p.D);
  const float4 Av = *reinterpret_cast<const float4*>(p.A + dd_ * 16 + q * 4);
  const float2 A01 = make_float2(Av.x * LOG2E, Av.y * LOG2E), A23 = make_float2(Av.z * LOG2E, Av.w * LOG2E);
  float2 r[2] = {{0.f, 0.f}, {0.f, 0.f}}, dA[2] = {{0.f, 0.f}, {0.f, 0.f}};
  for (int cp = p.NC - 1; cp > c; --cp) {
    const long long o = ((long long)b * p.NC + cp) * p.D + dd_;
    float2 a[2];
    exp4(A01, A23, p.chunk_sumdt[o], a);
    const float4 e = *reinterpret_cast<const float4*>(p.chunk_state + o * 16 + q * 4);
    r[0] = ffma2(a[0], r[0], make_float2(e.x, e.y));
    r[1] = ffma2(a[1], r[1], make_float2(e.z, e.w));
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) s.acc[threadIdx.x][j] = 0.f;
  const int tc0 = c * p.clen, t_end = min(tc0 + p.clen, p.L);
  // which of the quad's 8 values (dB of 4 states, dC of 4 states) this lane ends up with after the exchange over channels
  const bool b2 = lane & 4, b3 = lane & 8, b4 = lane & 16;
  const int idx = (b2 ? 4 : 0) + (b3 ? 2 : 0) + (b4 ? 1 : 0);
  const int col = idx < 4 ? q * 4 + idx : 16 + q * 4 + (idx - 4);
  uint4 xu, du, gu, zu = make_uint4(0u, 0u, 0u, 0u);
  uint16_t bv[4], cv[4];
  float4 hc;                                  // state at the start of the block
  auto fetch = [&](int t0) {
    const int tt = t0 + row.t, n = tt < t_end ? row.n : 0;
    xu = load8<VEC>(p.x + b * p.xsb + tt * p.xst + row.d, n);
    du = load8<VEC>(p.dt + b * p.dsb + tt * p.dst + row.d, n);
    gu = load8<VEC>(p.dout + b * p.gsb + tt * p.gst + row.d, n);
    if (p.z != nullptr) zu = load8<VEC>(p.z + b * p.zsb + tt * p.zst + row.d, n);
    load_bc(p.Bm + b * p.bsb, p.bst, t0, t_end, bv);
    load_bc(p.Cm + b * p.csb, p.cst, t0, t_end, cv);
    hc = *reinterpret_cast<const float4*>(
        p.ckpt + (((long long)b * ((p.L + SC_T - 1) / SC_T) + t0 / SC_T) * p.D + dd_) * 16 + q * 4);
  };
  int t0 = tc0 + (t_end - 1 - tc0) / SC_T * SC_T;
  fetch(t0);
  for (; t0 >= tc0; t0 -= SC_T) {
    const bool in = t0 + row.t < t_end;
    const uint4 xc = xu;
    {
      float xv[8], dv[8], gv[8], zv[8];
      unpack8f(xu, xv);
      unpack8f(du, dv);
      unpack8f(gu, gv);
      unpack8f(zu, zv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float dl = 0.f, sg = 0.f, dys = gv[j], dzf = 0.f;
        if (in && j < row.n) {
          const float raw = dv[j] + p.dt_bias[row.d + j], e = __expf(raw);
          dl = raw > 20.f ? raw : log1pf(e);
          sg = raw > 20.f ? 1.f : e / (1.f + e);
        }
        if (p.z != nullptr) {
          const float sz = sigmoid_f(zv[j]);
          dys = gv[j] * (zv[j] * sz);
          dzf = gv[j] * (sz * (1.f + zv[j] * (1.f - sz)));
        }
        s.dd[row.t][row.c8 + j] = make_float4(dl, dl * xv[j], dys, sg);
        s.dzf[row.t][row.c8 + j] = dzf;
      }
    }
    put_bc(s.Bs, bv);
    put_bc(s.Cs, cv);
    __syncthreads();
    // the states at the starts of the quarters (read back by the thread that wrote them)
    const int quarters = min(SC_T / SC_REG, (t_end - t0 + SC_REG - 1) / SC_REG);
    {
      float2 h[2] = {{hc.x, hc.y}, {hc.z, hc.w}};
      s.ck[0][threadIdx.x] = f4(h);
#pragma unroll 1
      for (int quarter = 1; quarter < quarters; ++quarter) {
#pragma unroll
        for (int k = 0; k < SC_REG; ++k) {
          const int t = (quarter - 1) * SC_REG + k;
          const float4 v = s.dd[t][ch];
          const float4 B4 = bc4(&s.Bs[t][q * 4]);
          const float2 dx2 = make_float2(v.y, v.y);
          float2 a[2];
          exp4(A01, A23, v.x, a);
          h[0] = ffma2(a[0], h[0], fmul2(dx2, make_float2(B4.x, B4.y)));
          h[1] = ffma2(a[1], h[1], fmul2(dx2, make_float2(B4.z, B4.w)));
        }
        s.ck[quarter][threadIdx.x] = f4(h);
      }
    }
    if (t0 - SC_T >= tc0) fetch(t0 - SC_T);       // in flight during this block
#pragma unroll 1
    for (int quarter = quarters - 1; quarter >= 0; --quarter) {
      const int tb = quarter * SC_REG;
      float2 hs[SC_REG + 1][2], as[SC_REG][2];    // hs[t + 1]: state after step t
      const float4 h0 = s.ck[quarter][threadIdx.x];
      hs[0][0] = make_float2(h0.x, h0.y);
      hs[0][1] = make_float2(h0.z, h0.w);
#pragma unroll
      for (int t = 0; t < SC_REG; ++t) {
        const float4 v = s.dd[tb + t][ch];
        const float4 B4 = bc4(&s.Bs[tb + t][q * 4]);
        const float2 dx2 = make_float2(v.y, v.y);
        exp4(A01, A23, v.x, as[t]);
        hs[t + 1][0] = ffma2(as[t][0], hs[t][0], fmul2(dx2, make_float2(B4.x, B4.y)));
        hs[t + 1][1] = ffma2(as[t][1], hs[t][1], fmul2(dx2, make_float2(B4.z, B4.w)));
      }
#pragma unroll
      for (int g = SC_REG - 4; g >= 0; g -= 4) {
        float v_gb[4], v_da[4], v_hc[4], vB[4][4], vC[4][4];
#pragma unroll
        for (int u = 3; u >= 0; --u) {
          const int t = g + u;
          const float4 v = s.dd[tb + t][ch];
          const float4 B4 = bc4(&s.Bs[tb + t][q * 4]);
          const float4 C4 = bc4(&s.Cs[tb + t][q * 4]);
          const float2 dl2 = make_float2(v.x, v.x), dx2 = make_float2(v.y, v.y), dy2 = make_float2(v.z, v.z);
          const float2 g0 = ffma2(make_float2(C4.x, C4.y), dy2, r[0]), g1 = ffma2(make_float2(C4.z, C4.w), dy2, r[1]);
          r[0] = fmul2(as[t][0], g0);
          r[1] = fmul2(as[t][1], g1);
          const float2 e0 = fmul2(r[0], hs[t][0]), e1 = fmul2(r[1], hs[t][1]);     // g * a * h_{t-1}
          dA[0] = ffma2(e0, dl2, dA[0]);
          dA[1] = ffma2(e1, dl2, dA[1]);
          const float2 da = ffma2(e1, A23, fmul2(e0, A01));
          const float2 gb = ffma2(g1, make_float2(B4.z, B4.w), fmul2(g0, make_float2(B4.x, B4.y)));
          const float2 hcv = ffma2(hs[t + 1][1], make_float2(C4.z, C4.w), fmul2(hs[t + 1][0], make_float2(C4.x, C4.y)));
          v_da[u] = da.x + da.y;
          v_gb[u] = gb.x + gb.y;
          v_hc[u] = hcv.x + hcv.y;
          const float2 b0 = fmul2(g0, dx2), b1 = fmul2(g1, dx2);                   // dB
          const float2 c0 = fmul2(hs[t + 1][0], dy2), c1 = fmul2(hs[t + 1][1], dy2);   // dC
          vB[u][0] = b0.x; vB[u][1] = b0.y; vB[u][2] = b1.x; vB[u][3] = b1.y;
          vC[u][0] = c0.x; vC[u][1] = c0.y; vC[u][2] = c1.x; vC[u][3] = c1.y;
        }
        // sum dB / dC over the 8 channels of the warp, halving the value set at every exchange; four steps together, so
        // that their exchanges overlap
        float w4[4][4], w2[4][2];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            w4[u][j] = (b2 ? vC[u][j] : vB[u][j]) + __shfl_xor_sync(0xffffffffu, b2 ? vB[u][j] : vC[u][j], 4);
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            w2[u][j] = (b3 ? w4[u][2 + j] : w4[u][j]) + __shfl_xor_sync(0xffffffffu, b3 ? w4[u][j] : w4[u][2 + j], 8);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          s.bc[warp][tb + g + u][col] =
              (b4 ? w2[u][1] : w2[u][0]) + __shfl_xor_sync(0xffffffffu, b4 ? w2[u][0] : w2[u][1], 16);
        s.s_da[tb + g + q][ch] = quad_transpose_sum(v_da, q);
        s.s_gb[tb + g + q][ch] = quad_transpose_sum(v_gb, q);
        s.s_hc[tb + g + q][ch] = quad_transpose_sum(v_hc, q);
      }
    }
    __syncthreads();
    if (in && row.n > 0) {
      float xv[8], ox[8], ot[8], oz[8];
      unpack8f(xc, xv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 v = s.dd[row.t][row.c8 + j];
        const float Dj = p.Dv != nullptr && j < row.n ? p.Dv[row.d + j] : 0.f;
        const float gb = s.s_gb[row.t][row.c8 + j];
        ox[j] = v.x * gb + Dj * v.z;
        ot[j] = (LN2 * s.s_da[row.t][row.c8 + j] + xv[j] * gb) * v.w;              // A was scaled by log2(e)
        oz[j] = s.dzf[row.t][row.c8 + j] * (s.s_hc[row.t][row.c8 + j] + Dj * xv[j]);
        s.acc[threadIdx.x][j] += v.z * xv[j];
        s.acc[threadIdx.x][8 + j] += ot[j];
      }
      const long long o = b * p.osb + (t0 + row.t) * p.ost + row.d;
      store8<VEC>(p.dx + o, ox, row.n);
      store8<VEC>(p.ddt + o, ot, row.n);
      if (p.dz != nullptr) store8<VEC>(p.dz + o, oz, row.n);
    }
    for (int i = threadIdx.x; i < SC_T * 8; i += SC_THREADS) {
      const int t = i >> 3, c4 = (i & 7) * 4;
      if (t0 + t < t_end) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < SC_THREADS / 32; ++w) {
          const float4 v = *reinterpret_cast<const float4*>(&s.bc[w][t][c4]);
          a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
        }
        *reinterpret_cast<float4*>(p.partBC + (((long long)blockIdx.x * p.B + b) * p.L + t0 + t) * 32 + c4) = a;
      }
    }
    __syncthreads();
  }
  if (dv_ok) {
    float* o = p.dA + d * 16 + q * 4;
    atomicAdd(o, dA[0].x);
    atomicAdd(o + 1, dA[0].y);
    atomicAdd(o + 2, dA[1].x);
    atomicAdd(o + 3, dA[1].y);
  }
  if (threadIdx.x < 2 * SC_CH) {                  // 32 steps' staging threads -> one value per channel
    const int cc = threadIdx.x % SC_CH, which = threadIdx.x / SC_CH;
    float a = 0.f;
    for (int t = 0; t < SC_T; ++t) a += s.acc[t * 4 + cc / 8][which * 8 + cc % 8];
    if (d0 + cc < p.D) {
      if (which == 1) atomicAdd(p.dbias + d0 + cc, a);
      else if (p.dD != nullptr) atomicAdd(p.dD + d0 + cc, a);
    }
  }
}

// dB and dC of every (batch, step): the channel tiles' partial sums, rounded once.
__global__ void __launch_bounds__(256)
scan_bc_reduce_kernel(const float* __restrict__ part, int ntiles, long long rows, h16* __restrict__ dB,
                      h16* __restrict__ dC) {
  const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;    // 4 of a row's 32 values
  if (i >= rows * 8) return;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int k = 0; k < ntiles; ++k) {
    const float4 v = *reinterpret_cast<const float4*>(part + (k * rows * 8 + i) * 4);
    a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
  }
  const int c4 = static_cast<int>(i & 7) * 4;
  h16* o = (c4 < 16 ? dB : dC) + (i >> 3) * 16 + (c4 & 15);
  *reinterpret_cast<uint2*>(o) = make_uint2(pack_h16x2(a.x, a.y), pack_h16x2(a.z, a.w));
}

// Chunks the sequence is cut into.  The kernels are bound by latency until an SM holds its `ctas` CTAs, so time goes with
// the chunk length times the number of rounds the CTAs take; more than one chunk adds the light pass over all chunks but
// one (about `light` of the main pass).  The count depends on the batch and the channels, and the chunks' states are folded
// in fp32: a sequence's last bits are not those it has in another batch.
static int scan_chunk_count(int B, int L, int D, int ctas, float light) {
  const int tiles = (D + SC_CH - 1) / SC_CH * B, blocks = (L + SC_T - 1) / SC_T, slots = ctas * sm_count();
  int best = 1;
  float best_cost = 1e30f;
  for (int nc = 1; nc <= SC_MAX_CHUNKS && nc <= blocks; ++nc) {
    const int len = (blocks + nc - 1) / nc, real = (blocks + len - 1) / len;
    if (real != nc) continue;
    const int rounds = static_cast<int>((static_cast<long long>(tiles) * nc + slots - 1) / slots);
    const float cost = len * rounds * (1.f + light * (nc - 1) / nc) + 0.02f * blocks * (nc > 1);
    if (cost < best_cost) {
      best_cost = cost;
      best = nc;
    }
  }
  return best;
}
constexpr float LIGHT_FWD = 0.6f, LIGHT_BWD = 0.25f;

NX_API int NX_SYM(nx_scan_chunks)(int B, int L, int D, int backward) {
  return scan_chunk_count(B, L, D, backward ? SC_BWD_CTAS : SC_FWD_CTAS, backward ? LIGHT_BWD : LIGHT_FWD);
}
NX_API int NX_SYM(nx_scan_channel_blocks)(int D) { return (D + SC_CH - 1) / SC_CH; }
NX_API int NX_SYM(nx_scan_blocks)(int L) { return (L + SC_T - 1) / SC_T; }

static void scan_common(ScanParams& p, int B, int L, int D, int ctas, float light) {
  p.B = B; p.L = L; p.D = D;
  p.NC = scan_chunk_count(B, L, D, ctas, light);
  p.clen = ((L + SC_T - 1) / SC_T + p.NC - 1) / p.NC * SC_T;
}

// A [D,16] fp32 (negative), Dv [D] fp32 or null, dt_bias [D] fp32; x/dt/z/out bf16 addressed by
// (batch stride, time stride); Bm/Cm bf16 [.., 16]. Scratch (fp32), NC = nx_scan_chunks(B, L, D, 0): chunk_state
// [B, NC, D, 16], chunk_sumdt [B, NC, D] (unused for NC = 1).  ckpt fp32 [B, nx_scan_blocks(L), D, 16] for the
// backward, or null.
NX_API int NX_SYM(nx_selective_scan_fwd)(const void* x, long long xsb, long long xst, const void* dt, long long dsb,
                                 long long dst, const void* z, long long zsb, long long zst, const void* Bm,
                                 long long bsb, long long bst, const void* Cm, long long csb, long long cst,
                                 const void* A, const void* Dv, const void* dt_bias, void* out, long long osb,
                                 long long ost, void* chunk_state, void* chunk_sumdt, void* ckpt, int B,
                                 int L, int D, cudaStream_t stream) {
  ScanParams p{};
  p.x = (const h16*)x; p.xsb = xsb; p.xst = xst;
  p.dt = (const h16*)dt; p.dsb = dsb; p.dst = dst;
  p.z = (const h16*)z; p.zsb = zsb; p.zst = zst;
  p.Bm = (const h16*)Bm; p.bsb = bsb; p.bst = bst;
  p.Cm = (const h16*)Cm; p.csb = csb; p.cst = cst;
  p.A = (const float*)A; p.Dv = (const float*)Dv; p.dt_bias = (const float*)dt_bias;
  p.out = (h16*)out; p.osb = osb; p.ost = ost;
  p.chunk_state = (float*)chunk_state; p.chunk_sumdt = (float*)chunk_sumdt; p.ckpt = (float*)ckpt;
  if (B <= 0 || L <= 0 || D <= 0) return NX_OK;
  scan_common(p, B, L, D, SC_FWD_CTAS, LIGHT_FWD);
  const bool vec = D % 8 == 0 && vec_ok(x, xsb, xst, 8) && vec_ok(dt, dsb, dst, 8) && vec_ok(z, zsb, zst, 8) &&
                   vec_ok(out, osb, ost, 8);
  const dim3 grid((D + SC_CH - 1) / SC_CH, p.NC, B);
  if (p.NC > 1) {
    const dim3 light(grid.x, p.NC - 1, B);
    if (vec) scan_fwd_kernel<false, true><<<light, SC_THREADS, 0, stream>>>(p);
    else scan_fwd_kernel<false, false><<<light, SC_THREADS, 0, stream>>>(p);
    NX_LAUNCH_CHECK();
  }
  if (vec) scan_fwd_kernel<true, true><<<grid, SC_THREADS, 0, stream>>>(p);
  else scan_fwd_kernel<true, false><<<grid, SC_THREADS, 0, stream>>>(p);
  NX_LAUNCH_CHECK();
  return NX_OK;
}

// dx / ddt / dz: bf16 with strides (osb, ost). dB / dC: bf16 [B, L, 16] contiguous.  dA [D,16], dD [D], dbias [D] fp32,
// zeroed by the caller.  ckpt from the forward.  Scratch (fp32): partBC [nx_scan_channel_blocks(D), B, L, 32],
// chunk_state / chunk_sumdt as in the forward with NC = nx_scan_chunks(B, L, D, 1).
NX_API int NX_SYM(nx_selective_scan_bwd)(const void* x, long long xsb, long long xst, const void* dt, long long dsb,
                                 long long dst, const void* z, long long zsb, long long zst, const void* Bm,
                                 long long bsb, long long bst, const void* Cm, long long csb, long long cst,
                                 const void* A, const void* Dv, const void* dt_bias, const void* dout,
                                 long long gsb, long long gst, void* dx, void* ddt, void* dz, long long osb,
                                 long long ost, void* dB, void* dC, void* partBC, void* dA, void* dD, void* dbias,
                                 void* ckpt, void* chunk_state, void* chunk_sumdt, int B, int L, int D,
                                 cudaStream_t stream) {
  ScanParams p{};
  p.x = (const h16*)x; p.xsb = xsb; p.xst = xst;
  p.dt = (const h16*)dt; p.dsb = dsb; p.dst = dst;
  p.z = (const h16*)z; p.zsb = zsb; p.zst = zst;
  p.Bm = (const h16*)Bm; p.bsb = bsb; p.bst = bst;
  p.Cm = (const h16*)Cm; p.csb = csb; p.cst = cst;
  p.dout = (const h16*)dout; p.gsb = gsb; p.gst = gst;
  p.A = (const float*)A; p.Dv = (const float*)Dv; p.dt_bias = (const float*)dt_bias;
  p.dx = (h16*)dx; p.ddt = (h16*)ddt; p.dz = (h16*)dz; p.osb = osb; p.ost = ost;
  p.partBC = (float*)partBC; p.dA = (float*)dA; p.dD = (float*)dD; p.dbias = (float*)dbias;
  p.ckpt = (float*)ckpt; p.chunk_state = (float*)chunk_state; p.chunk_sumdt = (float*)chunk_sumdt;
  if (B <= 0 || L <= 0 || D <= 0) return NX_OK;
  scan_common(p, B, L, D, SC_BWD_CTAS, LIGHT_BWD);
  const bool vec = D % 8 == 0 && vec_ok(x, xsb, xst, 8) && vec_ok(dt, dsb, dst, 8) && vec_ok(z, zsb, zst, 8) &&
                   vec_ok(dout, gsb, gst, 8) && vec_ok(dx, osb, ost, 8) && vec_ok(ddt, osb, ost, 8) &&
                   vec_ok(dz, osb, ost, 8);
  const dim3 grid((D + SC_CH - 1) / SC_CH, p.NC, B);
  const int smem = (int)sizeof(ScanBwdSmem);
  static bool attr_set = false;
  if (!attr_set) {
    NX_CUDA_CHECK(cudaFuncSetAttribute(scan_bwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    NX_CUDA_CHECK(cudaFuncSetAttribute(scan_bwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr_set = true;
  }
  if (p.NC > 1) {
    const dim3 light(grid.x, p.NC - 1, B);
    if (vec) scan_bwd_local_kernel<true><<<light, SC_THREADS, 0, stream>>>(p);
    else scan_bwd_local_kernel<false><<<light, SC_THREADS, 0, stream>>>(p);
    NX_LAUNCH_CHECK();
  }
  if (vec) scan_bwd_kernel<true><<<grid, SC_THREADS, smem, stream>>>(p);
  else scan_bwd_kernel<false><<<grid, SC_THREADS, smem, stream>>>(p);
  NX_LAUNCH_CHECK();
  const long long rows = static_cast<long long>(B) * L;
  scan_bc_reduce_kernel<<<static_cast<unsigned>((rows * 8 + 255) / 256), 256, 0, stream>>>(
      (const float*)partBC, (int)grid.x, rows, (h16*)dB, (h16*)dC);
  NX_LAUNCH_CHECK();
  return NX_OK;
}

}  // namespace nx
