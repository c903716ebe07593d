// The layer loops of the two transformer engines in native code.
//
// A decoder token is ~35 short launches and an encoder forward ~350; issued one by one from the host language each costs
// 7-9 us of interpreter, foreign-function and handle work around ~4 us of C, more than most of the kernels take.  These
// entry points issue the same members in the same order (src/engines/asr-whisper/raw-whisper-decoder.js:108-140,
// src/engines/asr-parakeet/raw-encoder.js:240-386), so that the host calls once per layer stack or block.  Nothing here
// launches a kernel of its own and no handle is kept, views included.
#include "fa_internal.cuh"

namespace {

// Closes the arena on every way out; what the caller keeps is pinned out of it first.
struct ArenaScope {
  fa_ctx *ctx;
  int id = -1;
  explicit ArenaScope(fa_ctx *c) : ctx(c) {}
  int open() { return fa_push_arena(ctx, &id); }
  ~ArenaScope() {
    if (id >= 0) {
      const std::string msg = ctx->err;
      fa_pop_arena(ctx, id);
      ctx->err = msg;
    }
  }
};

int linear(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *g, const fa_tensor *b, const fa_linear &w, int act, const fa_tensor *add,
           fa_tensor **out) {
  return fa_linear_step(ctx, x, g, b, 1e-5f, w.scale ? nullptr : (fa_tensor *)w.w, w.scale ? (fa_bytes *)w.w : nullptr, w.scale, w.N,
                        w.K, w.bias, act, add, out);
}

// Views of one layer.  No arena owns a view, so they are freed here on every way out, before the arena frees what they look at.
struct Views {
  fa_ctx *ctx;
  fa_tensor *v[6];
  int n = 0;
  explicit Views(fa_ctx *c) : ctx(c) {}
  int add(int rc, fa_tensor **t) {
    if (rc == FA_OK) v[n++] = *t;
    return rc;
  }
  int reshape(fa_tensor *t, int rows, int cols, fa_tensor **out) { return add(fa_reshape_view(ctx, t, rows, cols, out), out); }
  int rows(fa_tensor *t, int rows, fa_tensor **out) { return add(fa_rows_view(ctx, t, rows, out), out); }
  ~Views() {
    const std::string msg = ctx->err;
    for (int i = 0; i < n; i++) fa_free_tensor(ctx, v[i]);
    ctx->err = msg;
  }
};

// raw-whisper-decoder.js:112-124 from the separate members, for shapes the one-pass attention declines
int self_attention_ops(fa_ctx *ctx, Views &views, const fa_tensor *qkv, fa_tensor *ck, fa_tensor *cv, int n, int NH, int HD, fa_tensor **out) {
  const int S = qkv->rows, D = NH * HD;
  fa_tensor *part[3], *flat[3], *K, *V, *sc, *pr, *att;
  for (int i = 0; i < 3; i++) {
    FA_TRY(fa_slice_cols(ctx, qkv, i * D, D, &part[i]));
    FA_TRY(views.reshape(part[i], 1, S * D, &flat[i]));
  }
  FA_TRY(fa_copy_rows(ctx, ck, flat[1], n));
  FA_TRY(fa_copy_rows(ctx, cv, flat[2], n));
  FA_TRY(views.rows(ck, n + 1, &K));
  FA_TRY(views.rows(cv, n + 1, &V));
  FA_TRY(fa_bmm_qk(ctx, flat[0], K, nullptr, S * NH, HD, 1, 0, &sc));
  FA_TRY(fa_softmax(ctx, sc, &pr));
  FA_TRY(fa_bmm_pv(ctx, pr, V, S * NH, HD, 1, &att));
  return views.reshape(att, S, D, out);
}

int decoder_layer(fa_ctx *ctx, const fa_decoder_layer &w, const fa_tensor *x, const fa_tensor *kk, const fa_tensor *kv, fa_tensor *ck,
                  fa_tensor *cv, int n, int NH, int HD, fa_tensor **out) {
  const int S = x->rows;
  fa_tensor *qkv, *att = nullptr, *x1, *cq, *x2, *h;
  Views views(ctx);
  FA_TRY(linear(ctx, x, w.ln1_w, w.ln1_b, w.sqkv, FA_ACT_NONE, nullptr, &qkv));
  FA_TRY(fa_attn_step_append(ctx, qkv, ck, cv, n, NH, HD, &att));
  if (!att) FA_TRY(self_attention_ops(ctx, views, qkv, ck, cv, n, NH, HD, &att));
  FA_TRY(linear(ctx, att, nullptr, nullptr, w.so, FA_ACT_NONE, x, &x1));
  FA_TRY(linear(ctx, x1, w.ln2_w, w.ln2_b, w.cq, FA_ACT_NONE, nullptr, &cq));
  FA_TRY(fa_attn_step(ctx, cq, kk, kv, NH, HD, S, &att));
  if (!att) {
    fa_tensor *sc, *pr;
    FA_TRY(fa_bmm_qk(ctx, cq, kk, nullptr, NH, HD, S, 0, &sc));
    FA_TRY(fa_softmax(ctx, sc, &pr));
    FA_TRY(fa_bmm_pv(ctx, pr, kv, NH, HD, S, &att));
  }
  FA_TRY(linear(ctx, att, nullptr, nullptr, w.co, FA_ACT_NONE, x1, &x2));
  FA_TRY(linear(ctx, x2, w.ln3_w, w.ln3_b, w.f1, FA_ACT_GELU_ERF, nullptr, &h));
  return linear(ctx, h, nullptr, nullptr, w.f2, FA_ACT_NONE, x2, out);
}

}  // namespace

extern "C" int fa_decoder_step(fa_ctx *ctx, const fa_decoder_layer *layers, int n_layers, const fa_tensor *x, fa_tensor *const *cross_k,
                               fa_tensor *const *cross_v, fa_tensor *const *self_k, fa_tensor *const *self_v, int n, int NH, int HD,
                               const fa_tensor *lnf_w, const fa_tensor *lnf_b, const fa_linear *logits, fa_tensor **out) {
  if (!ctx || !out || !layers || !cross_k || !cross_v || !self_k || !self_v || !logits)
    return fa_fail(ctx, FA_ERR_INVALID, "decoderStep: NULL argument");
  FA_REQUIRE(ctx, fa_valid(ctx, x) && n_layers > 0, "decoderStep: unknown handle");
  ArenaScope scope(ctx);
  FA_TRY(scope.open());
  fa_tensor *cur = nullptr, *y = nullptr;
  for (int l = 0; l < n_layers; l++)
    FA_TRY(decoder_layer(ctx, layers[l], cur ? cur : x, cross_k[l], cross_v[l], self_k[l], self_v[l], n, NH, HD, &cur));
  FA_TRY(linear(ctx, cur, lnf_w, lnf_b, *logits, FA_ACT_NONE, nullptr, &y));
  FA_TRY(fa_pin(ctx, y, 1));
  *out = y;
  return FA_OK;
}

extern "C" int fa_conformer_block(fa_ctx *ctx, const fa_conformer_layer *w, const fa_tensor *x, const fa_tensor *x_ff, const fa_tensor *pos,
                                  int pos_projected, int H, int HD, int W, int dw_k, const fa_tensor *next_w, const fa_tensor *next_b,
                                  fa_tensor **out, fa_tensor **out_ff) {
  if (!ctx || !w || !out || !out_ff) return fa_fail(ctx, FA_ERR_INVALID, "conformerBlock: NULL argument");
  FA_REQUIRE(ctx, fa_valid(ctx, x) && fa_valid(ctx, pos) && W >= 1 && x->rows % W == 0, "conformerBlock: bad operands");
  ArenaScope scope(ctx);
  FA_TRY(scope.open());
  const float eps = 1e-5f;
  const int T = x->rows / W, S = H * HD;
  auto ff = [&](const fa_tensor *in, const fa_tensor *normed, const fa_feed_forward &f, fa_tensor **y) {
    fa_tensor *xn = nullptr, *h;
    if (!normed) FA_TRY(fa_layernorm_operand(ctx, in, f.ln_w, f.ln_b, eps, &xn));
    FA_TRY(fa_matmul(ctx, normed ? normed : xn, f.w1, f.b1, FA_ACT_SILU, nullptr, &h));
    return fa_matmul(ctx, h, f.w2, f.b2, FA_ACT_NONE, in, y);
  };
  fa_tensor *x1, *xln, *qkv, *q = nullptr, *k = nullptr, *v = nullptr, *p = nullptr, *att = nullptr, *x2, *x3, *x4, *xn, *pre, *dwo;
  FA_TRY(ff(x, x_ff, w->ff1, &x1));
  FA_TRY(fa_layernorm_operand(ctx, x1, w->lnatt_w, w->lnatt_b, eps, &xln));
  // q | k | v as one projection where the one-kernel attention reads it; from 256 rows on as the packed operand alone
  const bool fused = w->qkv && T >= 16 && T <= 192;
  if (fused) {
    if (x->rows >= 256) FA_TRY(fa_matmul_operand(ctx, xln, w->qkv, w->qkvb, FA_ACT_NONE, &qkv));
    else FA_TRY(fa_matmul(ctx, xln, w->qkv, w->qkvb, FA_ACT_NONE, nullptr, &qkv));
  } else {
    FA_TRY(fa_matmul(ctx, xln, w->q, w->qb, FA_ACT_NONE, nullptr, &q));
    FA_TRY(fa_matmul(ctx, xln, w->k, w->kb, FA_ACT_NONE, nullptr, &k));
    FA_TRY(fa_matmul(ctx, xln, w->v, w->vb, FA_ACT_NONE, nullptr, &v));
  }
  if (!pos_projected) FA_TRY(fa_matmul(ctx, pos, w->pos, nullptr, FA_ACT_NONE, nullptr, &p));
  const fa_tensor *pp = pos_projected ? pos : p;
  if (fused) {
    FA_TRY(fa_attn_fused_qkv(ctx, qkv, pp, w->pbu, w->pbv, H, HD, W, &att));
    if (!att) {  // declined: cut the columns apart and carry on with the separate members
      FA_TRY(fa_slice_cols(ctx, qkv, 0, S, &q));
      FA_TRY(fa_slice_cols(ctx, qkv, S, S, &k));
      FA_TRY(fa_slice_cols(ctx, qkv, 2 * S, S, &v));
    }
  }
  if (!att) FA_TRY(fa_attn_fused(ctx, q, k, v, pp, w->pbu, w->pbv, H, HD, W, &att));
  if (!att) {
    fa_tensor *ac, *bq, *bd, *sum, *pr;
    FA_TRY(fa_bmm_qk(ctx, q, k, w->pbu, H, HD, W, 0, &ac));
    FA_TRY(fa_bmm_qk(ctx, q, pp, w->pbv, H, HD, W, 1, &bq));
    FA_TRY(fa_rel_shift_b(ctx, bq, W * H, &bd));
    FA_TRY(fa_ewise(ctx, ac, bd, 0, &sum));
    FA_TRY(fa_softmax(ctx, sum, &pr));
    FA_TRY(fa_bmm_pv(ctx, pr, v, H, HD, W, &att));
  }
  FA_TRY(fa_matmul(ctx, att, w->out, w->outb, FA_ACT_NONE, x1, &x2));
  FA_TRY(fa_layernorm_operand(ctx, x2, w->lnconv_w, w->lnconv_b, eps, &xn));
  FA_TRY(fa_matmul(ctx, xn, w->pw1, w->pw1b, FA_ACT_NONE, nullptr, &pre));
  const int pad = (dw_k - 1) >> 1;
  FA_TRY(fa_glu_dwconv_tm(ctx, pre, w->dw, w->dwb, dw_k, pad, pad, FA_ACT_SILU, W, &dwo));
  FA_TRY(fa_matmul(ctx, dwo, w->pw2, w->pw2b, FA_ACT_NONE, x2, &x3));
  FA_TRY(ff(x3, nullptr, w->ff2, &x4));
  fa_tensor *y = nullptr, *y_ff = nullptr;
  if (next_w) {  // this block's last layernorm and the next block's first one in one pass over the rows
    FA_TRY(fa_layernorm_chain(ctx, x4, w->lnout_w, w->lnout_b, next_w, next_b, eps, &y, &y_ff));
    FA_TRY(fa_pin(ctx, y_ff, 1));
  } else {
    FA_TRY(fa_layernorm(ctx, x4, w->lnout_w, w->lnout_b, eps, &y));
  }
  FA_TRY(fa_pin(ctx, y, 1));
  *out = y;
  *out_ff = y_ff;
  return FA_OK;
}
