// One parallel-residual transformer layer of a generation step, without autograd: every launch of the layer from one
// call.  x + attention(ln1(x)) + mlp(ln2(x)) with the keys and values of this step written into the layer's cache.
//
// A step of a few tokens keeps the GPU busy for 30 us per layer; issued op by op the eight launches cost several
// times that on the host.  The kernels and their arguments are those of the op-by-op path
// (models/transformer.py, ParallelTransformerLayer.forward with `use_cache`), so both give the same bits: the branches
// are what the two modules return, rounded at their own size, and meet the residual stream in fp32 in the last kernel.
// With few rows the two branches' first products go in one launch, and their second ones: a step is a chain of short kernels,
// which it makes shorter by two (a captured step of 12 layers of 768, batch 4: 400 us with eight launches per layer, 327 with
// six).
#include <cstddef>

#include "common.h"
#include "gemm_skinny.h"

NX_API int NX_SYM(nx_norm_fwd)(int kind, const void* x, const void* g1, const void* b1, void* y1, const void* g2,
                       const void* b2, void* y2, void* mean, void* rstd, long long rows, int H, float eps, void* stream_);
NX_API int NX_SYM(nx_gemm_bf16)(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                        long long ldc, int transA, int transB, const void* bias, const void* aux_in, void* aux_out,
                        const void* residual, long long ld_aux, int flags, float alpha, void* stream_);
NX_API int NX_SYM(nx_gemm2_bf16)(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                         long long ldc, int transA, int transB, const void* bias, const void* aux_in, void* aux_out,
                         const void* residual, long long ld_aux, int flags, float alpha, void* stream_);
NX_API int NX_SYM(nx_branch_sum)(const void* x, const void* a, const void* ba, const void* m, const void* bm, void* out,
                         long long rows, int cols, void* stream_);
NX_API int NX_SYM(nx_rope_qk)(const void* q, const void* k, const void* v, void* qd, void* kd, void* vd, const void* cos,
                      const void* sin, int S, int B, int NQ, int NK, int D, int R, const long long* strides, int pos0,
                      int inverse, void* stream_);
NX_API int NX_SYM(nx_flash_attn_fwd)(const void* q, const void* k, const void* v, void* o, void* lse, const void* alibi,
                             int B, int H, int Hk, int Sq, int Sk, int D, long long q_sb, long long q_sh,
                             long long q_ss, long long k_sb, long long k_sh, long long k_ss, long long v_sb,
                             long long v_sh, long long v_ss, long long o_sb, long long o_sh, long long o_ss,
                             float scale, int causal, int window, float dropout_p, unsigned long long seed,
                             const void* blk_rows, const void* blk_any, int blk_size, void* stream_);

extern "C" {
// Everything contiguous; 16-bit tensors of one type.  Layouts: x / out [s, b, h]; wqkv [(np + 2 kvp) hn, h] with the rows
// of the fused projection (per head q | k | v for np == kvp, else Q | K | V); cache: the front of [2, room, b, kvp, hn],
// rows [past, past + s) written here.
struct nx_layer_infer_args {
  const void *x, *ln1_w, *ln1_b, *ln2_w, *ln2_b, *w_qkv, *b_qkv, *w_dense, *b_dense, *w1, *b1, *w2, *b2;
  long long bytes;                      // of this block, as the caller packs it
  const void *cos, *sin;
  // scratch: work, 16-bit: x1, x2, the attention branch (rows x h each), qkv, context, the MLP's hidden
  // layer; stats, fp32: mean and rstd of every row, the log-sum-exp of the attention [b, np, s rounded up to 128]
  void *cache, *work, *stats, *out;
  long long cache_kv_stride;            // elements between the key and the value part of the cache
  int s, b, h, np, kvp, hn, ffn, past, rot, window, act, pair_gemm;     // act: the GeLU's EPI_* bits (gemm_tcgen05.cu)
  float eps, scale;
};
}
// (packed by ops/layer_infer.py: 13 addresses, the size, and behind it no gap)
static_assert(offsetof(nx_layer_infer_args, bytes) == 13 * 8 && offsetof(nx_layer_infer_args, cache_kv_stride) == 20 * 8 &&
              offsetof(nx_layer_infer_args, eps) == 21 * 8 + 12 * 4 && sizeof(nx_layer_infer_args) == 22 * 8 + 12 * 4);

// An error, or minus the number of launches.
NX_API int NX_SYM(nx_layer_infer)(const nx_layer_infer_args* a, void* stream) {
  using namespace nx;
  enum { BIAS = 1 };
  NX_REQUIRE(a->bytes == sizeof(*a), "layer_infer: a block of %lld bytes, not %zu", a->bytes, sizeof(*a));
  const long long rows = static_cast<long long>(a->s) * a->b;
  if (rows == 0) return NX_OK;
  NX_REQUIRE(rows < (1ll << 31), "layer_infer: too many rows");
  NX_REQUIRE(a->h % 8 == 0 && a->hn % 8 == 0 && a->ffn % 8 == 0 && a->rot % 16 == 0 && a->rot > 0,
             "layer_infer: sizes must be multiples of 8 (rotary dims of 16)");
  const int M = static_cast<int>(rows), qkv_n = (a->np + 2 * a->kvp) * a->hn, ctx_n = a->np * a->hn, hn = a->hn;
  uint16_t* w = static_cast<uint16_t*>(a->work);
  uint16_t *x1 = w, *x2 = x1 + rows * a->h, *t = x2 + rows * a->h, *qkv = t + rows * a->h, *ctx = qkv + rows * qkv_n,
           *mid = ctx + rows * ctx_n;
  float *mean = static_cast<float*>(a->stats), *rstd = mean + rows, *lse = rstd + rows;
  auto gemm = [&](const void* A, const void* W, void* C, int N, int K, const void* bias, int act) {
    auto fn = a->pair_gemm && M >= 256 && N >= 256 ? NX_SYM(nx_gemm2_bf16) : NX_SYM(nx_gemm_bf16);
    return fn(A, W, C, M, N, K, K, K, N, 0, 0, bias, nullptr, nullptr, nullptr, 0, act | (bias != nullptr ? BIAS : 0), 1.f,
              stream);
  };
  // both products in one launch where each would go to the few-rows kernel
  struct Product {
    const void *A, *W;
    void* C;
    int N, K;
    const void* bias;
    int act;
  };
  int launches = 6;
  auto gemms = [&](const Product& x, const Product& y) {
    const Product* both[2] = {&x, &y};
    SkinnyProduct q[2];
    bool few = true;
    for (int i = 0; i < 2; ++i) {
      const Product& g = *both[i];
      const int flags = g.act | (g.bias != nullptr ? BIAS : 0);
      few = few && skinny_better(M, g.N, g.K, 0, 0, flags);
      q[i] = SkinnyProduct{g.A, g.W, g.K, g.K,
                           SkinnyParams{M, g.N, g.K, static_cast<h16*>(g.C), g.N, static_cast<const h16*>(g.bias), nullptr, nullptr, 0,
                                        flags, 1.f, device_error_word()}};
    }
    if (few) return gemm_skinny_launch_pair(q, static_cast<cudaStream_t>(stream));
    ++launches;
    const int rc = gemm(x.A, x.W, x.C, x.N, x.K, x.bias, x.act);
    return rc != NX_OK ? rc : gemm(y.A, y.W, y.C, y.N, y.K, y.bias, y.act);
  };
#define NX_TRY(expr)                  \
  do {                                \
    const int rc_ = (expr);           \
    if (rc_ != NX_OK) return rc_;     \
  } while (0)
  NX_TRY(NX_SYM(nx_norm_fwd)(0, a->x, a->ln1_w, a->ln1_b, x1, a->ln2_w, a->ln2_b, x2, mean, rstd, rows, a->h, a->eps,
                             stream));
  NX_TRY(gemms({x1, a->w_qkv, qkv, qkv_n, a->h, a->b_qkv, 0}, {x2, a->w1, mid, a->ffn, a->h, a->b1, a->act}));
  // q, k and v inside the projection's rows
  const bool mha = a->np == a->kvp;
  const long long ss = static_cast<long long>(a->b) * qkv_n, sb = qkv_n, sh = mha ? 3 * hn : hn;
  uint16_t *q = qkv, *k = qkv + (mha ? hn : ctx_n), *v = qkv + (mha ? 2 * hn : ctx_n + a->kvp * hn);
  const long long cs = static_cast<long long>(a->b) * a->kvp * hn, cb = static_cast<long long>(a->kvp) * hn;
  uint16_t *kc = static_cast<uint16_t*>(a->cache), *vc = kc + a->cache_kv_stride;
  const long long strides[18] = {ss, sb, sh, ss, sb, sh, ss, sb, sh, ss, sb, sh, cs, cb, hn, cs, cb, hn};
  NX_TRY(NX_SYM(nx_rope_qk)(q, k, v, q, kc + a->past * cs, vc + a->past * cs, a->cos, a->sin, a->s, a->b, a->np, a->kvp, hn,
                            a->rot, strides, a->past, 0, stream));
  // the context as [b, s, heads, hn] memory is what the op-by-op path writes; here it goes straight to [s, b, heads, hn]
  NX_TRY(NX_SYM(nx_flash_attn_fwd)(q, kc, vc, ctx, lse, nullptr, a->b, a->np, a->kvp, a->s, a->past + a->s, hn, sb, sh, ss,
                                   cb, hn, cs, cb, hn, cs, ctx_n, hn, static_cast<long long>(a->b) * ctx_n, a->scale, 1,
                                   a->window, 0.f, 0, nullptr, nullptr, 0, stream));
  NX_TRY(gemms({ctx, a->w_dense, t, a->h, ctx_n, nullptr, 0}, {mid, a->w2, a->out, a->h, a->ffn, nullptr, 0}));
  NX_TRY(NX_SYM(nx_branch_sum)(a->x, t, a->b_dense, a->out, a->b2, a->out, rows, a->h, stream));
#undef NX_TRY
  return -launches;
}
