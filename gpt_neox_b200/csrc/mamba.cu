// Mamba-1 kernels: causal depthwise conv1d (width <= 4) + SiLU, and the S6 selective scan, forward
// and backward, on token-major activations addressed by (batch stride, time stride) so the
// [seq, batch, channel] tensors the projections produce are consumed without a transpose.
//
// Counterparts in the reference: causal_conv1d_fn and selective_scan_fn / selective_scan_ref from
// the external causal_conv1d / mamba_ssm packages, called at megatron/model/mamba/mamba.py:220-247
// and :264-320 (which run on [batch, channel, seq] and need two rearranges per block).
//
// Scan parallelisation: a lane owns 4 of the 16 states of two neighbouring channels (a quad of lanes per pair; of one channel where
// there are so few that the chip would be idle), a warp 16 (8) channels, and walks its piece of the sequence in blocks of 32
// steps, cut into segments of four: lane q of a quad reads, prepares and finishes step q of a segment, so the forward sweeps and the
// light reverse sweep need no barrier but the warp's.  The sequence is cut into as few chunks as keep the chip busy (scan_plan): one
// chunk needs one pass; with more, a light pass first runs every chunk from a zero state and records its end state and its sum
// of delta (the chunk's decay is exp(A * sum delta)), and the main pass folds the other chunks into its start state.  The reverse
// recurrence of dL/dh is cut the same way.
// The forward keeps the state at the start of every 32-step block for the backward, which recomputes the states at the
// starts of the segments, then four steps at a time into registers, and walks them in reverse; dB and dC are added over a
// lane's channels before lanes and warps exchange them, and the next block's segment is staged where the walked one
// was.  Those states take 2 bytes per token and channel from the forward to the backward (25 MB for 4 x 2048 x 1536, as
// much as one more 16-bit activation), and the tiles' partial sums of dB and dC 2 bytes during the backward.
// Bound by: light sweeps, the unit of exponentials (16 per step and channel; 81 and 70 % busy); forward, that unit 66 %, shared
// memory 68 % and issue slots 63 % together; backward, issue slots (60 % with 3 warps per scheduler; shared memory 52 %),
// where a step and channel costs 500 lane operations for 16 states.  DRAM 8-14 %.
// Convolution + scan, forward + backward, 4 x 2048 steps of 1536 channels, fp16: 785 us with one channel per quad, inputs staged
// by the whole CTA and dB / dC exchanged per channel (final forward sweep 119, light ones 70 and 86, backward 407 us); 583 us
// now (91, 60 and 74, 277).  Calls of few channels and steps are latency, us, forward / forward + backward, that kernel and this
// one: 2 x 31 x 768 4.9 / 20.0, 5.2 / 18.1; 1 x 64 x 768 8.7 / 27.1, 8.1 / 25.6; 1 x 128 x 768 9.0 / 28.6, 10.1 / 29.1; 1 x 128 x 1536 9.9 / 37.7,
// 10.9 / 32.3; 1 x 256 x 1536 13.1 / 45.7, 13.4 / 39.6; 4 x 128 x 1536 18.5 / 66.3, 14.9 / 48.3.
// Tried for the backward: states packed per channel pair instead of per state pair (B and C twice in shared memory, no copies
// of a step's scalars): shared memory 62 % busy, 305 - 330 us; inputs staged per block with its loads waited for: 290 - 320.  For the
// forward: the next segment prepared beside the walk of this one: 3 - 5 % more time, with one channel or two.
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

// Vector forms: a thread owns four neighbouring channels (an 8-byte load per step, packed pairs) and `steps` steps (conv_steps), in
// groups whose loads are asked for together, in the forward one group ahead (the backward has no registers left for that: 54
// us).  The one-channel kernels above keep one 2-byte load in flight per thread and are bound by its latency; they remain for
// channel counts, strides or bases that are not multiples of four elements.  The backward walks three steps more than it owns,
// whose gradient reaches back into its tile: 5, 13 and 21 + 3 are whole groups.
// Bound by latency at 28 and 16 warps an SM and by issue slots; calls that leave the chip idle by the chain of a thread's steps.
// 4 x 2048 x 1536 / 16 x 512 x 2048, fp16, us: forward 19.8 / 26.5 with eight channels a thread and no pairs (142 registers), 12.8 /
// 15.2 now; backward 37.3 / 47.2 with 16 steps a thread, 32.1 / 39.1.  bf16 the same since conv_loaded: its backward took 56.
constexpr int CV_X = 32;    // channel groups per block
constexpr int CV_Y = 4;     // time tiles per block
constexpr int CV_V = 4;     // channels per thread
constexpr int CV_G = 4;     // steps per group
struct Conv4 { float2 a, b; };      // four channels
__device__ __forceinline__ Conv4 conv_unpack(const uint2& u) { return {unpack_h16x2(u.x), unpack_h16x2(u.y)}; }
__device__ __forceinline__ uint2 conv_pack(const Conv4& v) { return make_uint2(pack_h16x2(v.a.x, v.a.y), pack_h16x2(v.b.x, v.b.y)); }
__device__ __forceinline__ Conv4 conv_fma(const Conv4& x, const Conv4& y, const Conv4& z) { return {ffma2(x.a, y.a, z.a), ffma2(x.b, y.b, z.b)}; }
__device__ __forceinline__ Conv4 conv_mul(const Conv4& x, const Conv4& y) { return {fmul2(x.a, y.a), fmul2(x.b, y.b)}; }
__device__ __forceinline__ Conv4 conv_sigmoid(const Conv4& x) {
  auto f = [](float v) { return __fdividef(1.f, 1.f + __expf(-v)); };
  return {make_float2(f(x.a.x), f(x.a.y)), make_float2(f(x.b.x), f(x.b.y))};
}
// The loads of a group stay together in front of their first use: without this the bf16 build, whose conversions are plain
// integer operations, moves them into the branches of the single loads, which then wait for one another.
__device__ __forceinline__ void conv_loaded(uint2 (&u)[CV_G]) {
#pragma unroll
  for (int k = 0; k < CV_G; ++k) asm volatile("" : "+r"(u[k].x), "+r"(u[k].y));
}
// wk[k]: the tap on step t - 3 + k (zeros in front of a shorter kernel), and the bias
__device__ __forceinline__ void conv_taps(const h16* w, const h16* bias, int d, int W, Conv4 (&wk)[4], Conv4& bv) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float t[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) t[c] = k >= 4 - W ? ldbf(w + (long long)(d + c) * W + k - (4 - W)) : 0.f;
    wk[k] = {make_float2(t[0], t[1]), make_float2(t[2], t[3])};
  }
  bv = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
  if (bias != nullptr) bv = {make_float2(ldbf(bias + d), ldbf(bias + d + 1)), make_float2(ldbf(bias + d + 2), ldbf(bias + d + 3))};
}
__device__ __forceinline__ Conv4 conv_pre(const Conv4 (&wk)[4], const Conv4& bv, const Conv4 (&win)[3], const Conv4& cur) {
  return conv_fma(wk[3], cur, conv_fma(wk[2], win[2], conv_fma(wk[1], win[1], conv_fma(wk[0], win[0], bv))));
}

__global__ void __launch_bounds__(CV_X * CV_Y)
conv1d_silu_fwd_vec_kernel(const h16* __restrict__ x, long long xsb, long long xst, const h16* __restrict__ w,
                           const h16* __restrict__ bias, h16* __restrict__ y, long long ysb, long long yst, int L,
                           int D, int W, int steps) {
  const int d = (blockIdx.x * CV_X + threadIdx.x) * CV_V;
  const int t0 = (blockIdx.y * CV_Y + threadIdx.y) * steps, b = blockIdx.z;
  if (d >= D || t0 >= L) return;
  const int t1 = min(t0 + steps, L);
  const h16* xp = x + b * xsb + d;
  uint2 now[CV_G], next[CV_G];
  auto fetch = [&](int t, uint2 (&u)[CV_G]) {
#pragma unroll
    for (int k = 0; k < CV_G; ++k) {
      u[k] = make_uint2(0u, 0u);
      if (t + k < t1) u[k] = *reinterpret_cast<const uint2*>(xp + (t + k) * xst);
    }
  };
  fetch(t0, now);
  Conv4 wk[4], bv, win[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    uint2 u = make_uint2(0u, 0u);
    if (t0 - 3 + k >= 0) u = *reinterpret_cast<const uint2*>(xp + (t0 - 3 + k) * xst);
    win[k] = conv_unpack(u);
  }
  conv_taps(w, bias, d, W, wk, bv);
  h16* yp = y + b * ysb + t0 * yst + d;
#pragma unroll 1
  for (int t = t0; t < t1; t += CV_G) {
#ifndef NX_HALF
    conv_loaded(now);      // (fp16: 0.7 us more)
#endif
    fetch(t + CV_G, next);
#pragma unroll
    for (int k = 0; k < CV_G; ++k) {
      const Conv4 cur = conv_unpack(now[k]), pre = conv_pre(wk, bv, win, cur);
      if (t + k < t1) *reinterpret_cast<uint2*>(yp) = conv_pack(conv_mul(pre, conv_sigmoid(pre)));
      yp += yst;
      win[0] = win[1]; win[1] = win[2]; win[2] = cur;
    }
#pragma unroll
    for (int k = 0; k < CV_G; ++k) now[k] = next[k];
  }
}

template <int STEPS>      // (a number that the kernel is called with takes 4 - 7 % longer)
__global__ void __launch_bounds__(CV_X * CV_Y, 4)
conv1d_silu_bwd_vec_kernel(const h16* __restrict__ x, long long xsb, long long xst, const h16* __restrict__ w,
                           const h16* __restrict__ bias, const h16* __restrict__ dy, long long dsb, long long dst,
                           h16* __restrict__ dx, long long gsb, long long gst, float* __restrict__ dw,
                           float* __restrict__ dbias, int L, int D, int W) {
  __shared__ float red[CV_Y][CV_X][CV_V * 5 + 1];
  const int d = (blockIdx.x * CV_X + threadIdx.x) * CV_V;
  const int t0 = (blockIdx.y * CV_Y + threadIdx.y) * STEPS, b = blockIdx.z;
  Conv4 aw[5] = {};                       // gradients of the four taps and the bias
  if (d < D && t0 < L) {
    const h16* xp = x + b * xsb + d;
    const h16* gp = dy + b * dsb + d;
    const int t_own = min(t0 + STEPS, L), t_end = min(t0 + STEPS + 3, L);
    uint2 rx[CV_G], rg[CV_G];
    auto fetch = [&](int t, uint2 (&u)[CV_G], uint2 (&g)[CV_G]) {
#pragma unroll
      for (int k = 0; k < CV_G; ++k) {
        u[k] = g[k] = make_uint2(0u, 0u);
        if (t + k < t_end) {
          u[k] = *reinterpret_cast<const uint2*>(xp + (t + k) * xst);
          g[k] = *reinterpret_cast<const uint2*>(gp + (t + k) * dst);
        }
      }
      conv_loaded(u);
      conv_loaded(g);
    };
    Conv4 wk[4], bv, win[3], dp[3] = {};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      uint2 u = make_uint2(0u, 0u);
      if (t0 - 3 + k >= 0) u = *reinterpret_cast<const uint2*>(xp + (t0 - 3 + k) * xst);
      win[k] = conv_unpack(u);
    }
    conv_taps(w, bias, d, W, wk, bv);
#pragma unroll 1
    for (int s = 0; s < STEPS + 3; s += CV_G) {
      fetch(t0 + s, rx, rg);
#pragma unroll
      for (int k = 0; k < CV_G; ++k) {
        const int t = t0 + s + k, to = t - 3;
        const Conv4 cur = conv_unpack(rx[k]), pre = conv_pre(wk, bv, win, cur), sg = conv_sigmoid(pre);
        // silu' = s (1 + x (1 - s)); 0 beyond the sequence: dy was read as 0 there
        auto grad = [](float2 xx, float2 ss) {
          return fmul2(ss, ffma2(xx, ffma2(ss, make_float2(-1.f, -1.f), make_float2(1.f, 1.f)), make_float2(1.f, 1.f)));
        };
        const Conv4 dpre = conv_mul(conv_unpack(rg[k]), {grad(pre.a, sg.a), grad(pre.b, sg.b)});
        if (t < t_own) {
#pragma unroll
          for (int c = 0; c < 3; ++c) aw[c] = conv_fma(dpre, win[c], aw[c]);
          aw[3] = conv_fma(dpre, cur, aw[3]);
          aw[4] = {fadd2(aw[4].a, dpre.a), fadd2(aw[4].b, dpre.b)};
        }
        if (to >= t0 && to < t_own)
          *reinterpret_cast<uint2*>(dx + b * gsb + to * gst + d) =
              conv_pack(conv_fma(wk[0], dpre, conv_fma(wk[1], dp[2], conv_fma(wk[2], dp[1], conv_mul(wk[3], dp[0])))));
        win[0] = win[1]; win[1] = win[2]; win[2] = cur;
        dp[0] = dp[1]; dp[1] = dp[2]; dp[2] = dpre;
      }
    }
  }
  // one atomic per block and parameter: the block's time tiles are summed in shared memory first
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    float* r = red[threadIdx.y][threadIdx.x] + k;
    r[0] = aw[k].a.x; r[5] = aw[k].a.y; r[10] = aw[k].b.x; r[15] = aw[k].b.y;
  }
  __syncthreads();
  for (int i = threadIdx.y * CV_X + threadIdx.x; i < CV_X * CV_V * 5; i += CV_X * CV_Y) {
    const int gx = i / (CV_V * 5), r = i % (CV_V * 5), ch = (blockIdx.x * CV_X + gx) * CV_V + r / 5, k = r % 5;
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
// Steps per thread, by the work per SM (in steps of four channels): as few as still leave every SM enough threads, since a thread's
// steps are a chain; more where the three steps in front of a tile (backward: behind it), which are read again, count.  us,
// forward, 4 / 8 / 16 / 32 steps: 1 x 128 x 1536 (330 per SM) 2.3, 2.7, 3.5, 5.2; 4 x 128 x 1536 (1,330) 3.3, 3.3, 3.6, 5.2; 4 x 512 x
// 1536 (5,300) 7.1, 5.9, 5.6, 6.3; 4 x 2048 x 1536 (21,000) 19.5, 14.2, 12.8, 13.5; 16 x 512 x 2048 (28,000) 25.4, 17.8, 15.5, 15.2.
// Backward with its forward, 5 / 13 / 21 steps: 14.8, 16.4, 18.1; 16.4, 16.5, 18.1; 25.2, 21.7, 22.6; 66, 51, 52; 83, 65, 62.
static int conv_steps(int B, int L, int D, bool backward) {
  const long long per_sm = static_cast<long long>(B) * L * (D / CV_V) / sm_count();
  if (backward) return per_sm <= 1800 ? 5 : per_sm <= 6800 ? 13 : 21;
  return per_sm <= 450 ? 4 : per_sm <= 1800 ? 8 : per_sm <= 24000 ? 16 : 32;
}
static dim3 conv_vec_grid(int B, int L, int D, int steps) {
  return dim3((D / CV_V + CV_X - 1) / CV_X, (L + steps * CV_Y - 1) / (steps * CV_Y), B);
}

NX_API int NX_SYM(nx_conv1d_silu_fwd)(const void* x, long long xsb, long long xst, const void* w, const void* bias,
                              void* y, long long ysb, long long yst, int B, int L, int D, int W,
                              cudaStream_t stream) {
  NX_REQUIRE(W >= 1 && W <= 4, "conv1d: kernel width %d not in [1, 4]", W);
  if (D % CV_V == 0 && vec_ok(x, xsb, xst, CV_V) && vec_ok(y, ysb, yst, CV_V)) {
    const int steps = conv_steps(B, L, D, false);
    conv1d_silu_fwd_vec_kernel<<<conv_vec_grid(B, L, D, steps), dim3(CV_X, CV_Y), 0, stream>>>(
        (const h16*)x, xsb, xst, (const h16*)w, (const h16*)bias, (h16*)y, ysb, yst, L, D, W, steps);
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
  if (D % CV_V == 0 && vec_ok(x, xsb, xst, CV_V) && vec_ok(dy, dsb, dst, CV_V) && vec_ok(dx, gsb, gst, CV_V)) {
    const int steps = conv_steps(B, L, D, true);
    auto run = [&](auto kern) {
      kern<<<conv_vec_grid(B, L, D, steps), dim3(CV_X, CV_Y), 0, stream>>>(
          (const h16*)x, xsb, xst, (const h16*)w, (const h16*)bias, (const h16*)dy, dsb, dst, (h16*)dx, gsb, gst,
          (float*)dw, (float*)dbias, L, D, W);
    };
    if (steps == 5) run(conv1d_silu_bwd_vec_kernel<5>);
    else if (steps == 13) run(conv1d_silu_bwd_vec_kernel<13>);
    else run(conv1d_silu_bwd_vec_kernel<21>);
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
constexpr int SC_T = 32;        // steps per block (the forward keeps a state per block for the backward)
constexpr int SC_SEG = 4;       // steps per segment: lane q of a quad reads, and writes the results of, step q of it
constexpr int SC_SEGS = SC_T / SC_SEG;
constexpr int SC_WARPS = 4, SC_THREADS = SC_WARPS * 32;
// C, the channels of a quad of lanes: two neighbouring ones, or one where that leaves the chip idle (scan_plan)
constexpr int scan_channels(int C) { return SC_WARPS * 8 * C; }      // of a CTA
constexpr int SC_MAX_CHUNKS = 64;
constexpr int SC_FWD_CTAS = 5, SC_BWD_CTAS = 3;   // CTAs per SM: registers are bounded for so many of them
constexpr float LOG2E = 1.44269504088896340736f, LN2 = 0.69314718055994530942f;

struct ScanParams {
  const h16 *x, *dt, *z, *Bm, *Cm, *dout;
  long long xsb, xst, dsb, dst, zsb, zst, bsb, bst, csb, cst, gsb, gst;
  const float *A, *Dv, *dt_bias;
  h16 *out, *dx, *ddt, *dz;       // [.., D] with strides osb / ost
  long long osb, ost;
  float *chunk_state, *chunk_sumdt;   // [B, NC, D, 16] / [B, NC, D]: end state (or reverse carry) and sum of delta
  float *ckpt;                        // [B, ceil(L / 32), D, 16]: state at the start of every block; null = not kept
  float *partBC;                      // [ceil(D / 64), B, L, 32]
  float *dA, *dD, *dbias;
  int B, L, D, NC, clen;              // clen: steps per chunk, a multiple of SC_T
  bool bc_vec;                        // four neighbouring values of B (and of C) can be read as 8 bytes
};

__device__ __forceinline__ float sigmoid_f(float v) { return __fdividef(1.f, 1.f + __expf(-v)); }
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
// log(1 + exp(v)) = max(v, 0) + log(1 + e) with e = exp(-|v|) <= 1, and log(1 + e) = e + e^2 p(e), p of degree 9: no branch, no
// division, and right for small e, infinities and NaN.  p's coefficients are least-squares fits of the largest error relative to
// the result (1e-9), rounded one after the other with the rest fitted again: rounded together they leave a bias of 2e-8.
// `e` goes out too.
__device__ __forceinline__ float2 softplus2(float2 v, float2& e) {
  constexpr float P[] = {0.00208493182f, -0.0136934891f, 0.0421184078f, -0.0832427964f, 0.124797717f,
                         -0.161352605f, 0.19899641f, -0.249888659f, 0.333327144f, -0.499999881f};
  e = make_float2(exp2f(-fabsf(v.x) * LOG2E), exp2f(-fabsf(v.y) * LOG2E));
  float2 p = both(P[0]);
#pragma unroll
  for (int i = 1; i < 10; ++i) p = ffma2(e, p, both(P[i]));
  return fadd2(ffma2(fmul2(e, e), p, e), make_float2(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f)));
}

// Sums four values per lane over the quad: lane q returns the total of v[q] (three exchanges instead of eight).
__device__ __forceinline__ float quad_transpose_sum(float v0, float v1, float v2, float v3, int q) {
  const bool hi = q & 2, odd = q & 1;
  float a = hi ? v2 : v0, b = hi ? v3 : v1;
  a += __shfl_xor_sync(0xffffffffu, hi ? v0 : v2, 2);
  b += __shfl_xor_sync(0xffffffffu, hi ? v1 : v3, 2);
  const float keep = odd ? b : a;
  return keep + __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
}
__device__ __forceinline__ float quad_transpose_sum(const float (&v)[SC_SEG], int q) {
  return quad_transpose_sum(v[0], v[1], v[2], v[3], q);
}
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// A lane's place: states 4 q .. 4 q + 3 of the channels d .. d + C - 1.
struct ScanLane {
  int lane, warp, j, q, d, n;       // n: live channels of the quad's
};
template <int C>
__device__ __forceinline__ ScanLane scan_lane(int D) {
  ScanLane s;
  s.lane = threadIdx.x & 31;
  s.warp = threadIdx.x >> 5;
  s.j = s.lane >> 2;
  s.q = s.lane & 3;
  s.d = blockIdx.x * scan_channels(C) + (s.warp * 8 + s.j) * C;
  s.n = min(C, max(0, D - s.d));
  return s;
}
// Two neighbouring 16-bit elements (zero where dead): one 4-byte access when VEC, single elements otherwise.
template <bool VEC>
__device__ __forceinline__ uint32_t load2(const h16* p, int n) {
  if (VEC) return n > 0 ? *reinterpret_cast<const uint32_t*>(p) : 0u;
  const uint16_t* e = reinterpret_cast<const uint16_t*>(p);
  return (n > 0 ? e[0] : 0u) | (n > 1 ? static_cast<uint32_t>(e[1]) << 16 : 0u);
}
template <bool VEC>
__device__ __forceinline__ void store2(h16* p, float2 v, int n) {
  if (VEC) {
    if (n > 0) *reinterpret_cast<uint32_t*>(p) = pack_h16x2(v.x, v.y);
    return;
  }
  if (n > 0) p[0] = float_to_h16(v.x);
  if (n > 1) p[1] = float_to_h16(v.y);
}
__device__ __forceinline__ float2 coef2(const float* p, const ScanLane& s) {
  return make_float2(p != nullptr && s.n > 0 ? p[s.d] : 0.f, p != nullptr && s.n > 1 ? p[s.d + 1] : 0.f);
}
// A lane's states: [channel of the quad][pair of states].  In memory [channel][16] floats from the channel d on; zero where dead.
__device__ __forceinline__ void get4(const float4& v, float2 (&h)[2]) {
  h[0] = make_float2(v.x, v.y);
  h[1] = make_float2(v.z, v.w);
}
__device__ __forceinline__ float4 put4(const float2 (&h)[2]) { return make_float4(h[0].x, h[0].y, h[1].x, h[1].y); }
template <int C>
__device__ __forceinline__ void load_states(const float* p, const ScanLane& s, float2 (&h)[C][2]) {
#pragma unroll
  for (int i = 0; i < C; ++i) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < s.n) v = *reinterpret_cast<const float4*>(p + i * 16 + s.q * 4);
    get4(v, h[i]);
  }
}
template <int C>
__device__ __forceinline__ void store_states(float* p, const ScanLane& s, const float2 (&h)[C][2]) {
#pragma unroll
  for (int i = 0; i < C; ++i)
    if (i < s.n) *reinterpret_cast<float4*>(p + i * 16 + s.q * 4) = put4(h[i]);
}
// The states' decay rates times log2(e).
template <int C>
__device__ __forceinline__ void load_A(const float* A, const ScanLane& s, float2 (&a)[C][2]) {
  load_states(A + static_cast<long long>(s.d) * 16, s, a);
#pragma unroll
  for (int i = 0; i < C; ++i)
#pragma unroll
    for (int k = 0; k < 2; ++k) a[i][k] = fmul2(a[i][k], both(LOG2E));
}
// Four neighbouring values of a row of B or C.
__device__ __forceinline__ uint2 load_bc4(const h16* p, bool vec) {
  if (vec) return *reinterpret_cast<const uint2*>(p);
  const uint16_t* e = reinterpret_cast<const uint16_t*>(p);
  return make_uint2(e[0] | static_cast<uint32_t>(e[1]) << 16, e[2] | static_cast<uint32_t>(e[3]) << 16);
}
__device__ __forceinline__ float4 bc4(const uint2& u) {
  const float2 a = unpack_h16x2(u.x), b = unpack_h16x2(u.y);
  return make_float4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ float2 exp2_2(float2 v) { return make_float2(exp2f(v.x), exp2f(v.y)); }
__device__ __forceinline__ void decay(const float2 (&A)[2], float dl, float2 (&a)[2]) {
  a[0] = exp2_2(fmul2(both(dl), A[0]));
  a[1] = exp2_2(fmul2(both(dl), A[1]));
}
// One step of a channel's four states: h1 = a h0 + dx B, with a = exp(delta A).
__device__ __forceinline__ void scan_step(const float2 (&A)[2], float dl, float dx, const float4& B, float2 (&a)[2],
                                          const float2 (&h0)[2], float2 (&h1)[2]) {
  decay(A, dl, a);
  h1[0] = ffma2(a[0], h0[0], fmul2(both(dx), make_float2(B.x, B.y)));
  h1[1] = ffma2(a[1], h0[1], fmul2(both(dx), make_float2(B.z, B.w)));
}
__device__ __forceinline__ float dot4(const float2 (&a)[2], const float4& b) {
  const float2 v = ffma2(a[1], make_float2(b.z, b.w), fmul2(a[0], make_float2(b.x, b.y)));
  return v.x + v.y;
}
// The state after the chunk c, whose walk from a zero state ended in chunk_state.
template <int C>
__device__ __forceinline__ void fold_chunk(const ScanParams& p, const ScanLane& s, const float2 (&A)[C][2], int b, int c,
                                           float2 (&h)[C][2]) {
  const long long o = (static_cast<long long>(b) * p.NC + c) * p.D + s.d;
  float2 e[C][2];
  load_states(p.chunk_state + o * 16, s, e);
#pragma unroll
  for (int i = 0; i < C; ++i) {
    float2 a[2];
    decay(A[i], i < s.n ? p.chunk_sumdt[o + i] : 0.f, a);
    h[i][0] = ffma2(a[0], h[i][0], e[i][0]);
    h[i][1] = ffma2(a[1], h[i][1], e[i][1]);
  }
}
template <int C>
__device__ __forceinline__ void put_chunk(const ScanParams& p, const ScanLane& s, int b, int c, const float2 (&h)[C][2],
                                          float2 sdt) {
  const long long o = (static_cast<long long>(b) * p.NC + c) * p.D + s.d;
  store_states(p.chunk_state + o * 16, s, h);
  sdt = make_float2(quad_sum(sdt.x), quad_sum(sdt.y));
  if (s.q < s.n) p.chunk_sumdt[o + s.q] = s.q == 0 ? sdt.x : sdt.y;
}

// FINAL = false: chunks 0 .. NC - 2 from a zero state -> end state and sum of delta.
template <bool FINAL, int C, bool VEC>
__global__ void __launch_bounds__(SC_THREADS, SC_FWD_CTAS)
scan_fwd_kernel(const ScanParams p) {
  // per warp and for two segments in turn: delta and delta * x of a quad's channels; B and C of the segment's steps
  __shared__ float4 dd[SC_WARPS][2][SC_SEG][8], bc[SC_WARPS][2][SC_SEG][FINAL ? 8 : 4];
  const ScanLane s = scan_lane<C>(p.D);
  const int c = blockIdx.y, b = blockIdx.z, q = s.q;
  float2 A[C][2], h[C][2] = {};
  load_A(p.A, s, A);
  if (FINAL) {
#pragma unroll 4
    for (int cp = 0; cp < c; ++cp) fold_chunk(p, s, A, b, cp, h);     // (four chunks' loads in flight)
  }
  const int tc0 = c * p.clen, t_end = min(tc0 + p.clen, p.L);
  // the lane's next segment: step q of it of x, dt and z, and four values of B or C of step lane / 8
  const int bt = s.lane >> 3, bn = (s.lane & 7) * 4;
  const bool isC = bn >= 16;
  const h16 *xp = p.x + b * p.xsb + (tc0 + q) * p.xst + s.d, *dp = p.dt + b * p.dsb + (tc0 + q) * p.dst + s.d;
  const h16* zp = FINAL && p.z != nullptr ? p.z + b * p.zsb + (tc0 + q) * p.zst + s.d : nullptr;
  const h16* bcp = isC ? p.Cm + b * p.csb + (tc0 + bt) * p.cst + bn - 16 : p.Bm + b * p.bsb + (tc0 + bt) * p.bst + bn;
  h16* op = FINAL ? p.out + b * p.osb + (tc0 + q) * p.ost + s.d : nullptr;
  const float2 bias = coef2(p.dt_bias, s), Dv = FINAL ? coef2(p.Dv, s) : both(0.f);
  float2 sdt = both(0.f);
  struct Raw { uint32_t x, d, z; uint2 bc; } raw[2];
  auto fetch = [&](int t0, Raw& r) {              // called for the segments one after the other
    const int n = t0 + q < t_end ? s.n : 0;
    r.x = load2<VEC>(xp, n);
    r.d = load2<VEC>(dp, n);
    xp += SC_SEG * p.xst;
    dp += SC_SEG * p.dst;
    r.z = 0u;
    if (FINAL && zp != nullptr) {
      r.z = load2<VEC>(zp, n);
      zp += SC_SEG * p.zst;
    }
    r.bc = make_uint2(0u, 0u);
    if (t0 + bt < t_end && (FINAL || !isC)) r.bc = load_bc4(bcp, p.bc_vec);
    bcp += SC_SEG * (isC ? p.cst : p.bst);
  };
  fetch(tc0, raw[0]);
  fetch(tc0 + SC_SEG, raw[1]);
  for (int tb = tc0; tb < t_end; tb += 2 * SC_SEG) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int t0 = tb + k * SC_SEG;
      if (t0 >= t_end) break;
      const bool in = t0 + q < t_end;
      const float2 xv = unpack_h16x2(raw[k].x), zv = unpack_h16x2(raw[k].z);
      float2 e, dl = softplus2(fadd2(unpack_h16x2(raw[k].d), bias), e);
      if (!in) dl = both(0.f);                    // (a step beyond the end leaves the state as it is)
      const float2 dx = fmul2(dl, xv);
      dd[s.warp][k][q][s.j ^ (2 * q)] = make_float4(dl.x, dx.x, dl.y, dx.y);   // (neither writers nor readers collide)
      if (!FINAL) sdt = fadd2(sdt, dl);
      if (FINAL || !isC) bc[s.warp][k][bt][s.lane & 7] = bc4(raw[k].bc);
      fetch(t0 + 2 * SC_SEG, raw[k]);             // in flight during two segments
      if (FINAL && p.ckpt != nullptr && (t0 & (SC_T - 1)) == 0)
        store_states(p.ckpt + ((static_cast<long long>(b) * ((p.L + SC_T - 1) / SC_T) + t0 / SC_T) * p.D + s.d) * 16, s, h);
      __syncwarp();        // (this buffer's last readers have passed the other one's)
      float yp[C][SC_SEG];
#pragma unroll
      for (int t = 0; t < SC_SEG; ++t) {
        const float4 v = dd[s.warp][k][t][s.j ^ (2 * t)], B4 = bc[s.warp][k][t][q];
        float2 a[2];
#pragma unroll
        for (int i = 0; i < C; ++i) scan_step(A[i], i == 0 ? v.x : v.z, i == 0 ? v.y : v.w, B4, a, h[i], h[i]);
        if (FINAL) {
          const float4 C4 = bc[s.warp][k][t][4 + q];
#pragma unroll
          for (int i = 0; i < C; ++i) yp[i][t] = dot4(h[i], C4);
        }
      }
      if (FINAL) {
        float2 y = ffma2(Dv, xv, make_float2(quad_transpose_sum(yp[0], q), C > 1 ? quad_transpose_sum(yp[C - 1], q) : 0.f));
        if (p.z != nullptr) y = make_float2(y.x * silu(zv.x), y.y * silu(zv.y));
        if (in) store2<VEC>(op, y, s.n);
        op += SC_SEG * p.ost;
      }
    }
  }
  if (!FINAL) put_chunk(p, s, b, c, h, sdt);
}

// Reverse recurrence of chunks 1 .. NC - 1 from a zero carry: chunk_state[c] = what chunk c hands to chunk c - 1.
template <int C, bool VEC>
__global__ void __launch_bounds__(SC_THREADS, SC_FWD_CTAS)
scan_bwd_local_kernel(const ScanParams p) {
  // as in the forward: delta and the gradient of the ungated output of a quad's channels; C
  __shared__ float4 dd[SC_WARPS][2][SC_SEG][8], cs[SC_WARPS][2][SC_SEG][4];
  const ScanLane s = scan_lane<C>(p.D);
  const int c = blockIdx.y + 1, b = blockIdx.z, q = s.q;
  float2 A[C][2], r[C][2] = {};
  load_A(p.A, s, A);
  const int tc0 = c * p.clen, t_end = min(tc0 + p.clen, p.L);
  const int last = tc0 + (t_end - 1 - tc0) / SC_SEG * SC_SEG, bt = s.j & 3;
  const h16 *dp = p.dt + b * p.dsb + (last + q) * p.dst + s.d, *gp = p.dout + b * p.gsb + (last + q) * p.gst + s.d;
  const h16* zp = p.z != nullptr ? p.z + b * p.zsb + (last + q) * p.zst + s.d : nullptr;
  const h16* cp = p.Cm + b * p.csb + (last + bt) * p.cst + q * 4;
  const float2 bias = coef2(p.dt_bias, s);
  float2 sdt = both(0.f);
  struct Raw { uint32_t d, g, z; uint2 c; } raw[2];
  auto fetch = [&](int t0, Raw& u) {              // called for the segments one before the other
    const int n = t0 >= tc0 && t0 + q < t_end ? s.n : 0;
    u.d = load2<VEC>(dp, n);
    u.g = load2<VEC>(gp, n);
    dp -= SC_SEG * p.dst;
    gp -= SC_SEG * p.gst;
    u.z = 0u;
    if (zp != nullptr) {
      u.z = load2<VEC>(zp, n);
      zp -= SC_SEG * p.zst;
    }
    u.c = make_uint2(0u, 0u);
    if (t0 >= tc0 && t0 + bt < t_end) u.c = load_bc4(cp, p.bc_vec);
    cp -= SC_SEG * p.cst;
  };
  fetch(last, raw[0]);
  fetch(last - SC_SEG, raw[1]);
  for (int tb = last; tb >= tc0; tb -= 2 * SC_SEG) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int t0 = tb - k * SC_SEG;
      if (t0 < tc0) break;
      float2 e, dl = softplus2(fadd2(unpack_h16x2(raw[k].d), bias), e), g = unpack_h16x2(raw[k].g);
      if (t0 + q >= t_end) dl = both(0.f);
      if (p.z != nullptr) {
        const float2 zv = unpack_h16x2(raw[k].z);
        g = fmul2(g, make_float2(silu(zv.x), silu(zv.y)));
      }
      dd[s.warp][k][q][s.j ^ (2 * q)] = make_float4(dl.x, g.x, dl.y, g.y);
      sdt = fadd2(sdt, dl);
      if (s.j < SC_SEG) cs[s.warp][k][bt][q] = bc4(raw[k].c);
      fetch(t0 - 2 * SC_SEG, raw[k]);
      __syncwarp();
#pragma unroll
      for (int t = SC_SEG - 1; t >= 0; --t) {
        const float4 v = dd[s.warp][k][t][s.j ^ (2 * t)], C4 = cs[s.warp][k][t][q];
#pragma unroll
        for (int i = 0; i < C; ++i) {
          const float2 g2 = both(i == 0 ? v.y : v.w);
          float2 a[2];
          decay(A[i], i == 0 ? v.x : v.z, a);
          r[i][0] = fmul2(a[0], ffma2(make_float2(C4.x, C4.y), g2, r[i][0]));
          r[i][1] = fmul2(a[1], ffma2(make_float2(C4.z, C4.w), g2, r[i][1]));
        }
      }
    }
  }
  put_chunk(p, s, b, c, r, sdt);
}

// With one channel there are no second halves of a segment's states (see ScanBwdWarp): room of its own.
template <int C>
struct ScanBwdRoom { float4 own[3][32]; };
template <>
struct ScanBwdRoom<2> {};
template <int C>
struct ScanBwdWarp : ScanBwdRoom<C> {
  float4 dd[SC_T][8 * C];             // delta, x, gradient of the ungated output, sigmoid(dt) of the warp's channels
  float4 ck[SC_SEGS - 1][C][32];      // a lane's states at the starts of the segments 1 .., per channel
  float2 dzf[SC_SEGS][32];            // d out / d z without the scan value, of the lane that writes it
  // A segment's states make room, once used: the first half for the sums over the warp's channels, dB and dC as [step][32]
  // (segment 0 has no states here, its sums go to the second half of segment 5), the second halves of the last two for the
  // state at the block's start, and of segments 3 and 4 for that of the next block to be walked.
  __device__ __forceinline__ float* sums(int sg) {
    if (sg > 0) return reinterpret_cast<float*>(ck[sg - 1][0]);
    if constexpr (C > 1) return reinterpret_cast<float*>(ck[4][1]);
    else return reinterpret_cast<float*>(this->own[0]);
  }
  __device__ __forceinline__ float4* start(int i, int lane) {
    if constexpr (C > 1) return &ck[5 + i][1][lane];
    else return &this->own[1][lane];
  }
  __device__ __forceinline__ float4* next_start(int i, int lane) {
    if constexpr (C > 1) return &ck[2 + i][1][lane];
    else return &this->own[2][lane];
  }
  // a step's channels, placed so that neither a segment's writers (a step per lane of a quad) nor a step's readers collide
  static __device__ __forceinline__ int slot(int t, int j, int i) { return i * 8 + (j ^ (2 * (t & 3))); }
};
template <int C>
struct ScanBwdSmem {
  ScanBwdWarp<C> w[SC_WARPS];
  float bc[SC_T][32];                 // B | C
};
// 16 bytes to shared memory behind the thread's back (zeros where dead); waited for by the thread that asked.
__device__ __forceinline__ void copy16_async(float4* dst, const float* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(live ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int C, bool VEC>
__global__ void __launch_bounds__(SC_THREADS, SC_BWD_CTAS)
scan_bwd_kernel(const ScanParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ScanBwdSmem<C>& sm = *reinterpret_cast<ScanBwdSmem<C>*>(smem_raw);
  const ScanLane s = scan_lane<C>(p.D);
  ScanBwdWarp<C>& w = sm.w[s.warp];
  const int c = blockIdx.y, b = blockIdx.z, q = s.q, lane = s.lane;
  float2 A[C][2], r[C][2] = {}, dA[C][2] = {};
  load_A(p.A, s, A);
#pragma unroll 4
  for (int cp = p.NC - 1; cp > c; --cp) fold_chunk(p, s, A, b, cp, r);
  const int tc0 = c * p.clen, t_end = min(tc0 + p.clen, p.L);
  // which of the quad's 8 values (dB of 4 states, dC of 4 states) this lane ends up with after the exchange over channels
  const bool b2 = lane & 4, b3 = lane & 8, b4 = lane & 16;
  const int idx = (b2 ? 4 : 0) + (b3 ? 2 : 0) + (b4 ? 1 : 0);
  const int col = idx < 4 ? q * 4 + idx : 16 + q * 4 + (idx - 4);
  const float2 bias = coef2(p.dt_bias, s), Dv = coef2(p.Dv, s);
  float2 sumD = both(0.f), sumb = both(0.f);
  const float* ckpt = p.ckpt + (static_cast<long long>(b) * ((p.L + SC_T - 1) / SC_T) * p.D + s.d) * 16 + q * 4;
  const int last = tc0 + (t_end - 1 - tc0) / SC_T * SC_T;
  struct Raw { uint32_t x, d, g, z; };
  auto fetch = [&](int t, Raw& u) {               // the lane's channels of step t
    const int n = t < t_end ? s.n : 0;
    u.x = load2<VEC>(p.x + b * p.xsb + t * p.xst + s.d, n);
    u.d = load2<VEC>(p.dt + b * p.dsb + t * p.dst + s.d, n);
    u.g = load2<VEC>(p.dout + b * p.gsb + t * p.gst + s.d, n);
    u.z = p.z != nullptr ? load2<VEC>(p.z + b * p.zsb + t * p.zst + s.d, n) : 0u;
  };
  auto stage = [&](int sg, const Raw& u, bool in) {
    const float2 xv = unpack_h16x2(u.x), v = fadd2(unpack_h16x2(u.d), bias);
    float2 e, dl = softplus2(v, e), sd, dys = unpack_h16x2(u.g), dzf = both(0.f);
    sd = make_float2(__fdividef(v.x >= 0.f ? 1.f : e.x, 1.f + e.x), __fdividef(v.y >= 0.f ? 1.f : e.y, 1.f + e.y));
    if (!in) dl = sd = both(0.f);
    if (p.z != nullptr) {
      const float2 z = unpack_h16x2(u.z), sz = make_float2(sigmoid_f(z.x), sigmoid_f(z.y)), zs = fmul2(z, sz);
      // silu' = sz (1 + z (1 - sz)) = sz + z sz (1 - sz)
      dzf = fmul2(dys, ffma2(zs, fadd2(both(1.f), make_float2(-sz.x, -sz.y)), sz));
      dys = fmul2(dys, zs);
    }
    w.dd[sg * SC_SEG + q][w.slot(q, s.j, 0)] = make_float4(dl.x, xv.x, dys.x, sd.x);
    if (C > 1) w.dd[sg * SC_SEG + q][w.slot(q, s.j, C - 1)] = make_float4(dl.y, xv.y, dys.y, sd.y);
    w.dzf[sg][lane] = dzf;
  };
  auto fetch_start = [&](int t0, float4* a, float4* b, bool any) {        // the state at the start of a block
    if (any) {
      const float* src = ckpt + static_cast<long long>(t0 / SC_T) * p.D * 16;
      copy16_async(a, s.n > 0 ? src : p.ckpt, s.n > 0);
      if (C > 1) copy16_async(b, s.n > 1 ? src + 16 : p.ckpt, s.n > 1);
    }
    copy_async_commit();
  };
  // Blocks from the last one back, before it a turn that only brings it in: while a block's segment is walked, the same
  // segment of the block to be walked next is on its way from memory, and takes its place afterwards.
  for (int t0 = last + SC_T;; t0 -= SC_T) {
    const bool more = t0 > tc0;
    const int segs = t0 <= last ? min(SC_SEGS, (t_end - t0 + SC_SEG - 1) / SC_SEG) : 0, tn = t0 - SC_T;
    if (segs == 0) {
      Raw u[SC_SEGS];
#pragma unroll
      for (int sg = 0; sg < SC_SEGS; ++sg) fetch(tn + sg * SC_SEG + q, u[sg]);
      fetch_start(tn, w.next_start(0, lane), w.next_start(1, lane), true);
#pragma unroll
      for (int sg = 0; sg < SC_SEGS; ++sg) stage(sg, u[sg], tn + sg * SC_SEG + q < t_end);
    }
#pragma unroll 1
    for (int sg = segs > 0 ? SC_SEGS - 1 : -1; sg >= 0; --sg) {
      const int tb = sg * SC_SEG;
      Raw raw = {};
      if (more) fetch(tn + tb + q, raw);          // (a full block: only the last one walked first may be short)
      if (sg == 1) fetch_start(t0, w.start(0, lane), w.start(1, lane), true);
      if (sg == 0) {
        fetch_start(tn, w.next_start(0, lane), w.next_start(1, lane), more);
        copy_async_wait<1>();
      }
      if (sg < segs) {
        float2 aB[SC_SEG][2], aC[SC_SEG][2];        // dB and dC of the quad's channels
        float ox[2] = {}, ot[2] = {}, oz[2] = {};
        const bool in = t0 + tb + q < t_end;
        const float2 dzf = w.dzf[sg][lane];
#pragma unroll
        for (int i = 0; i < C; ++i) {
          float2 hs[SC_SEG + 1][2], as[SC_SEG][2];  // hs[t + 1]: state after step t
          float4 v[SC_SEG];
          float dx[SC_SEG];
          get4(sg > 0 ? w.ck[sg - 1][i][lane] : *w.start(i, lane), hs[0]);
#pragma unroll
          for (int t = 0; t < SC_SEG; ++t) {
            v[t] = w.dd[tb + t][w.slot(t, s.j, i)];
            dx[t] = v[t].x * v[t].y;
            scan_step(A[i], v[t].x, dx[t], *reinterpret_cast<const float4*>(&sm.bc[tb + t][q * 4]), as[t], hs[t], hs[t + 1]);
          }
          float v_gb[SC_SEG], v_da[SC_SEG], v_hc[SC_SEG];
#pragma unroll
          for (int t = SC_SEG - 1; t >= 0; --t) {
            const float4 B4 = *reinterpret_cast<const float4*>(&sm.bc[tb + t][q * 4]);
            const float4 C4 = *reinterpret_cast<const float4*>(&sm.bc[tb + t][16 + q * 4]);
            const float2 dl2 = both(v[t].x), dx2 = both(dx[t]), dy2 = both(v[t].z);
            const float2 g[2] = {ffma2(make_float2(C4.x, C4.y), dy2, r[i][0]), ffma2(make_float2(C4.z, C4.w), dy2, r[i][1])};
            r[i][0] = fmul2(as[t][0], g[0]);
            r[i][1] = fmul2(as[t][1], g[1]);
            const float2 e0 = fmul2(r[i][0], hs[t][0]), e1 = fmul2(r[i][1], hs[t][1]);     // g * a * h_{t-1}
            dA[i][0] = ffma2(e0, dl2, dA[i][0]);
            dA[i][1] = ffma2(e1, dl2, dA[i][1]);
            const float2 da = ffma2(e1, A[i][1], fmul2(e0, A[i][0]));
            v_da[t] = da.x + da.y;
            v_gb[t] = dot4(g, B4);
            v_hc[t] = dot4(hs[t + 1], C4);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              aB[t][k] = i == 0 ? fmul2(g[k], dx2) : ffma2(g[k], dx2, aB[t][k]);
              aC[t][k] = i == 0 ? fmul2(hs[t + 1][k], dy2) : ffma2(hs[t + 1][k], dy2, aC[t][k]);
            }
          }
          const float da = quad_transpose_sum(v_da, q), gb = quad_transpose_sum(v_gb, q), hc = quad_transpose_sum(v_hc, q);
          const float4 m = w.dd[tb + q][w.slot(q, s.j, i)];
          const float Di = i == 0 ? Dv.x : Dv.y;
          ox[i] = m.x * gb + Di * m.z;
          ot[i] = (LN2 * da + m.y * gb) * m.w;                                             // A was scaled by log2(e)
          oz[i] = (i == 0 ? dzf.x : dzf.y) * (hc + Di * m.y);
          if (in) {
            (i == 0 ? sumD.x : sumD.y) += m.z * m.y;
            (i == 0 ? sumb.x : sumb.y) += ot[i];
          }
        }
        if (in) {
          const long long o = b * p.osb + (t0 + tb + q) * p.ost + s.d;
          store2<VEC>(p.dx + o, make_float2(ox[0], ox[1]), s.n);
          store2<VEC>(p.ddt + o, make_float2(ot[0], ot[1]), s.n);
          if (p.dz != nullptr) store2<VEC>(p.dz + o, make_float2(oz[0], oz[1]), s.n);
        }
        // sum dB / dC over the 8 quads of the warp, halving the value set at every exchange; four steps together, so
        // that their exchanges overlap
        float w4[SC_SEG][4], w2[SC_SEG][2];
#pragma unroll
        for (int t = 0; t < SC_SEG; ++t) {
          const float vB[4] = {aB[t][0].x, aB[t][0].y, aB[t][1].x, aB[t][1].y};
          const float vC[4] = {aC[t][0].x, aC[t][0].y, aC[t][1].x, aC[t][1].y};
#pragma unroll
          for (int k = 0; k < 4; ++k) w4[t][k] = (b2 ? vC[k] : vB[k]) + __shfl_xor_sync(0xffffffffu, b2 ? vB[k] : vC[k], 4);
        }
#pragma unroll
        for (int t = 0; t < SC_SEG; ++t)
#pragma unroll
          for (int k = 0; k < 2; ++k)
            w2[t][k] = (b3 ? w4[t][2 + k] : w4[t][k]) + __shfl_xor_sync(0xffffffffu, b3 ? w4[t][k] : w4[t][2 + k], 8);
        __syncwarp();                   // every lane has read its states of this segment, and the segment's inputs
        float* sums = w.sums(sg);
#pragma unroll
        for (int t = 0; t < SC_SEG; ++t)
          sums[t * 32 + col] = (b4 ? w2[t][1] : w2[t][0]) + __shfl_xor_sync(0xffffffffu, b4 ? w2[t][0] : w2[t][1], 16);
      }
      if (more) stage(sg, raw, true);
    }
    uint2 bcu[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int t = tn + (threadIdx.x >> 3) + 16 * k, n4 = (threadIdx.x & 7) * 4;
      bcu[k] = make_uint2(0u, 0u);
      if (more && t < t_end)
        bcu[k] = load_bc4(n4 < 16 ? p.Bm + b * p.bsb + t * p.bst + n4 : p.Cm + b * p.csb + t * p.cst + n4 - 16, p.bc_vec);
    }
    __syncthreads();                  // the warps' sums of the block are there, and B and C have been used
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int t = (threadIdx.x >> 3) + 16 * k, c4 = (threadIdx.x & 7) * 4;
      if (segs > 0 && t0 + t < t_end) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int ww = 0; ww < SC_WARPS; ++ww) {
          const float4 u = *reinterpret_cast<const float4*>(sm.w[ww].sums(t / SC_SEG) + (t & (SC_SEG - 1)) * 32 + c4);
          a.x += u.x; a.y += u.y; a.z += u.z; a.w += u.w;
        }
        *reinterpret_cast<float4*>(p.partBC + ((static_cast<long long>(blockIdx.x) * p.B + b) * p.L + t0 + t) * 32 + c4) = a;
      }
      *reinterpret_cast<float4*>(&sm.bc[t][c4]) = bc4(bcu[k]);
    }
    if (!more) break;
    copy_async_wait<0>();
    float2 h[C][2];
#pragma unroll
    for (int i = 0; i < C; ++i) get4(*w.next_start(i, lane), h[i]);
    __syncthreads();                  // B and C of the next block are there, and the sums have been read
    // the states at the starts of its segments (read back by the lane that wrote them)
    const int next_segs = min(SC_SEGS, (t_end - tn + SC_SEG - 1) / SC_SEG);
#pragma unroll 1
    for (int sg = 0; sg < next_segs - 1; ++sg) {
#pragma unroll
      for (int t = 0; t < SC_SEG; ++t) {
        const float4 B4 = *reinterpret_cast<const float4*>(&sm.bc[sg * SC_SEG + t][q * 4]);
#pragma unroll
        for (int i = 0; i < C; ++i) {
          const float2 v = *reinterpret_cast<const float2*>(&w.dd[sg * SC_SEG + t][w.slot(t, s.j, i)]);
          float2 a[2];
          scan_step(A[i], v.x, v.x * v.y, B4, a, h[i], h[i]);
        }
      }
#pragma unroll
      for (int i = 0; i < C; ++i) w.ck[sg][i][lane] = put4(h[i]);
    }
  }
  sumD = make_float2(quad_sum(sumD.x), quad_sum(sumD.y));
  sumb = make_float2(quad_sum(sumb.x), quad_sum(sumb.y));
#pragma unroll
  for (int i = 0; i < C; ++i)
    if (i < s.n) {
      float* o = p.dA + (s.d + i) * 16 + q * 4;
      atomicAdd(o, dA[i][0].x);
      atomicAdd(o + 1, dA[i][0].y);
      atomicAdd(o + 2, dA[i][1].x);
      atomicAdd(o + 3, dA[i][1].y);
      if (q == 0) atomicAdd(p.dbias + s.d + i, i == 0 ? sumb.x : sumb.y);
      if (q == 1 && p.dD != nullptr) atomicAdd(p.dD + s.d + i, i == 0 ? sumD.x : sumD.y);
    }
}

// dB and dC of every (batch, step): the channel tiles' partial sums, rounded once.  Four groups of eight lanes share a row's tiles,
// so that few rows with many tiles are a short chain of loads.
__global__ void __launch_bounds__(256)
scan_bc_reduce_kernel(const float* __restrict__ part, int ntiles, long long rows, h16* __restrict__ dB,
                      h16* __restrict__ dC) {
  const long long row = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);    // a warp per row
  if (row >= rows) return;
  const int c4 = (threadIdx.x & 7) * 4;                                                 // 4 of its 32 values
  part += row * 32 + c4;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int k = (threadIdx.x >> 3) & 3; k < ntiles; k += 4) {
    const float4 v = *reinterpret_cast<const float4*>(part + k * rows * 32);
    a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
  }
#pragma unroll
  for (int m = 8; m < 32; m *= 2) {
    a.x += __shfl_xor_sync(0xffffffffu, a.x, m);
    a.y += __shfl_xor_sync(0xffffffffu, a.y, m);
    a.z += __shfl_xor_sync(0xffffffffu, a.z, m);
    a.w += __shfl_xor_sync(0xffffffffu, a.w, m);
  }
  if (threadIdx.x & 24) return;
  h16* o = (c4 < 16 ? dB : dC) + row * 16 + (c4 & 15);
  *reinterpret_cast<uint2*>(o) = make_uint2(pack_h16x2(a.x, a.y), pack_h16x2(a.z, a.w));
}

static int scan_tiles(int D, int C) { return (D + scan_channels(C) - 1) / scan_channels(C); }
// Channels of a quad and chunks the sequence is cut into.  Time goes with the blocks of a chunk times the rounds that the CTAs take; a
// last round that leaves an SM only some of its CTAs is shorter (measured, time of a block with 1, 2, 3 CTAs on every SM: backward
// 0.57, 0.77, 1; forward, 1 .. 5: 0.48, 0.54, 0.66, 0.85, 1).  More than one chunk adds the light pass over all chunks but one, whose
// block takes `light` of the main pass's (forward 7.2 of 10 us, backward 9 of 18.5, with every SM full), and its launch.  us, forward +
// backward, fp16, with 1, 4, 8, 16, 22 and 32 chunks: 4 x 2048 x 1536: 980, 568, 530, 506, 502, 514 (the rule: 22 and 16);
// 16 x 512 x 1536: 413, 446, 444, 473 (1 and 1); 1 x 4096 x 1536: 1808, 683, 466, 312, 315, 311 (43 and 43).
// With one channel a quad a block takes `one` of the time with two, and there are twice the CTAs: shorter where CTAs are few.  us,
// forward / backward, two channels and one, at the better count of chunks: 2 x 31 x 768 6.2, 5.3 / 16.0, 12.8; 1 x 64 x 768 10.1, 7.9 /
// 21.4, 17.9; 1 x 128 x 1536 11.5, 10.9 / 22.7, 21.5; 1 x 512 x 768 15.1, 13.9 / 27.8, 26.2; 4 x 128 x 1536 14.8, 17.5 / 32.9, 40.0; 4 x
// 2048 x 1536 144, 186 / 356, 465.
// Both depend on the batch and the channels, and the chunks' states are folded in fp32: a sequence's last bits are not those it has
// in another batch.
static float scan_rounds(long long ctas, int per_sm) {
  const int sms = sm_count();
  const long long slots = static_cast<long long>(per_sm) * sms, rest = ctas % slots;
  return static_cast<float>(ctas / slots) + (rest > 0 ? 0.35f + 0.65f * static_cast<float>((rest + sms - 1) / sms) / per_sm : 0.f);
}
struct ScanPlan { int C, NC; };      // channels of a quad, chunks
static ScanPlan scan_plan(int B, int L, int D, bool backward) {
  const int ctas = backward ? SC_BWD_CTAS : SC_FWD_CTAS, blocks = (L + SC_T - 1) / SC_T;
  const float light = backward ? 0.48f : 0.7f, one = backward ? 0.67f : 0.74f, launch = backward ? 0.11f : 0.2f;
  ScanPlan best{2, 1};
  float best_cost = 1e30f;
  for (int C = 2; C >= 1; --C) {
    const long long tiles = static_cast<long long>(scan_tiles(D, C)) * B;
    const float unit = C == 1 ? one : 1.f;
    for (int nc = 1; nc <= SC_MAX_CHUNKS && nc <= blocks; ++nc) {
      const int len = (blocks + nc - 1) / nc, real = (blocks + len - 1) / len;
      if (real != nc) continue;
      // (a tenth of a block to begin a chunk, and its fold of the other chunks' states)
      float cost = unit * (len + 0.1f + 0.002f * nc) * scan_rounds(tiles * nc, ctas);
      if (nc > 1) cost += unit * light * (len + 0.1f) * scan_rounds(tiles * (nc - 1), SC_FWD_CTAS) + launch;
      if (cost < best_cost) {
        best_cost = cost;
        best = {C, nc};
      }
    }
  }
  return best;
}

NX_API int NX_SYM(nx_scan_chunks)(int B, int L, int D, int backward) { return scan_plan(B, L, D, backward != 0).NC; }
NX_API int NX_SYM(nx_scan_tiles)(int B, int L, int D) { return scan_tiles(D, scan_plan(B, L, D, true).C); }
NX_API int NX_SYM(nx_scan_blocks)(int L) { return (L + SC_T - 1) / SC_T; }

// -> channels of a quad
static int scan_common(ScanParams& p, int B, int L, int D, bool backward) {
  const ScanPlan plan = scan_plan(B, L, D, backward);
  p.B = B; p.L = L; p.D = D;
  p.NC = plan.NC;
  p.clen = ((L + SC_T - 1) / SC_T + p.NC - 1) / p.NC * SC_T;
  p.bc_vec = vec_ok(p.Bm, p.bsb, p.bst, 4) && vec_ok(p.Cm, p.csb, p.cst, 4);
  return plan.C;
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
  const int C = scan_common(p, B, L, D, false);
  const bool vec = D % 2 == 0 && vec_ok(x, xsb, xst, 2) && vec_ok(dt, dsb, dst, 2) && vec_ok(z, zsb, zst, 2) &&
                   vec_ok(out, osb, ost, 2);
  const dim3 grid(scan_tiles(D, C), p.NC, B), light(grid.x, p.NC - 1, B);
  auto run = [&](auto local, auto final) {
    if (p.NC > 1) {
      local<<<light, SC_THREADS, 0, stream>>>(p);
      NX_LAUNCH_CHECK();
    }
    final<<<grid, SC_THREADS, 0, stream>>>(p);
    NX_LAUNCH_CHECK();
    return NX_OK;
  };
  if (C == 1) return run(scan_fwd_kernel<false, 1, false>, scan_fwd_kernel<true, 1, false>);
  if (vec) return run(scan_fwd_kernel<false, 2, true>, scan_fwd_kernel<true, 2, true>);
  return run(scan_fwd_kernel<false, 2, false>, scan_fwd_kernel<true, 2, false>);
}

// dx / ddt / dz: bf16 with strides (osb, ost). dB / dC: bf16 [B, L, 16] contiguous.  dA [D,16], dD [D], dbias [D] fp32,
// zeroed by the caller.  ckpt from the forward.  Scratch (fp32): partBC [nx_scan_tiles(B, L, D), B, L, 32],
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
  const int C = scan_common(p, B, L, D, true);
  const bool vec = D % 2 == 0 && vec_ok(x, xsb, xst, 2) && vec_ok(dt, dsb, dst, 2) && vec_ok(z, zsb, zst, 2) &&
                   vec_ok(dout, gsb, gst, 2) && vec_ok(dx, osb, ost, 2) && vec_ok(ddt, osb, ost, 2) &&
                   vec_ok(dz, osb, ost, 2);
  const dim3 grid(scan_tiles(D, C), p.NC, B), light(grid.x, p.NC - 1, B);
  constexpr int smem1 = sizeof(ScanBwdSmem<1>), smem2 = sizeof(ScanBwdSmem<2>);
  static bool attr_set = false;
  if (!attr_set) {
    NX_CUDA_CHECK(cudaFuncSetAttribute(scan_bwd_kernel<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem1));
    NX_CUDA_CHECK(cudaFuncSetAttribute(scan_bwd_kernel<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem2));
    NX_CUDA_CHECK(cudaFuncSetAttribute(scan_bwd_kernel<2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem2));
    attr_set = true;
  }
  auto run = [&](auto local, auto kern, int smem) {
    if (p.NC > 1) {
      local<<<light, SC_THREADS, 0, stream>>>(p);
      NX_LAUNCH_CHECK();
    }
    kern<<<grid, SC_THREADS, smem, stream>>>(p);
    NX_LAUNCH_CHECK();
    return NX_OK;
  };
  const int rc = C == 1 ? run(scan_bwd_local_kernel<1, false>, scan_bwd_kernel<1, false>, smem1)
                 : vec  ? run(scan_bwd_local_kernel<2, true>, scan_bwd_kernel<2, true>, smem2)
                        : run(scan_bwd_local_kernel<2, false>, scan_bwd_kernel<2, false>, smem2);
  if (rc != NX_OK) return rc;
  const long long rows = static_cast<long long>(B) * L;
  scan_bc_reduce_kernel<<<static_cast<unsigned>((rows + 7) / 8), 256, 0, stream>>>(
      (const float*)partBC, (int)grid.x, rows, (h16*)dB, (h16*)dC);
  NX_LAUNCH_CHECK();
  return NX_OK;
}

}  // namespace nx
