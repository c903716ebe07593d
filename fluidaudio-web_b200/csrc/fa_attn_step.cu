// Attention of ONE query per stream (token-by-token decoding) as one pass over the keys and values.
//
// The op sequence is bmmQK -> softmax -> bmmPV with T = 1 (src/engines/asr-whisper/raw-whisper-decoder.js:118-131), and
// for self-attention the two copyRows that append the token's key and value to the cache in front of it (:113-116).  As
// separate kernels the scores travel through memory twice, the value pass of one stream runs on as many blocks as there
// are 128-column strips (10 of 148 SMs at D = 1280), and every boundary costs a launch.  Here a block reads the same
// rows of K and of V and keeps a running (maximum, sum, weighted sum) per head, the softmax being rescaled when the
// maximum moves, so that the cache is read once and nothing in between is stored.
//
// What bounds it: HBM, the cache is read once (983 MB per layer for 64 streams x 1500 keys x 1280 columns).
// Layout: a warp owns 128 consecutive columns (32 lanes x float4, HD / 4 lanes per head) and takes U = 8 rows of K and
// the same rows of V at a time, all 16 loads of a lane in flight together (8 KB per warp, 128 KB per SM with two blocks
// of 8 warps); the 8 warps of a block take rows round-robin.  gridDim.y splits the keys so that a single stream fills
// the GPU too; the splits' partial results meet in the block that takes the last ticket, in split order (nothing waits).
// All arithmetic is f32.
// Measured in whole decoder passes of 16 tokens (4 layers, 20 heads of 64, 1500 keys), the separate ops before and this
// kernel after: one stream, int8 weights 12.64 -> 8.24 ms (a value pass on 10 blocks took 44 us), 64 streams, f16 weights
// 21.15 -> 19.06 ms (77 us of scores + 16 us of softmax + 78 us of values per layer, against the 150 us of one reading).
#include "fa_internal.cuh"

namespace {

constexpr int kWarps = 8, kThreads = kWarps * 32, kU = 8;

struct StepParams {
  const float *q;            // query of column c in window w: q + w*q_win + (c / D)*ldq + c % D
  const float *k, *v;        // row j of window w: k + w*kv_win + j*ld
  const float *knew, *vnew;  // APPEND: the row `Tk - 1`, addressed like q; the kernel also stores it into the caches
  float *kc, *vc;            // APPEND: the caches
  float *out;                // [W][C]
  __half *y16;               // packed f16 row operand of out seen as [R][D] (value plane, then residue plane), or NULL
  float *pacc, *pml;         // splits > 1: partial sums [W][splits][C] and (maximum, sum) [W][splits][C/4][2]
  int *tickets;              // [W][strips]
  long long q_win, kv_win, ld, lo_off;
  int ldq, D, C, R, Tk, lph, kper;
};

// exp(m - M) for M >= m, 1 where the two are the same infinity
__device__ __forceinline__ float step_scale(float m, float M) { return m == M ? 1.0f : expf(m - M); }

struct Running {
  float m, l;
  float4 a;
};
__device__ __forceinline__ void merge(Running &r, float m, float l, const float4 &a) {
  const float M = fmaxf(r.m, m), f0 = step_scale(r.m, M), f1 = step_scale(m, M);
  r.l = r.l * f0 + l * f1;
  r.a.x = r.a.x * f0 + a.x * f1, r.a.y = r.a.y * f0 + a.y * f1;
  r.a.z = r.a.z * f0 + a.z * f1, r.a.w = r.a.w * f0 + a.w * f1;
  r.m = M;
}

// The block's 8 running results into warp 0's, in warp order.
__device__ __forceinline__ void merge_block(Running &r, int warp, int lane, float4 (*sa)[32], float2 (*sml)[32]) {
  sa[warp][lane] = r.a;
  sml[warp][lane] = make_float2(r.m, r.l);
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int i = 1; i < kWarps; i++) merge(r, sml[i][lane].x, sml[i][lane].y, sa[i][lane]);
  }
}

template <bool APPEND>
__global__ void __launch_bounds__(kThreads, 2) k_attn_step(const StepParams p) {
  __shared__ float4 sa[kWarps][32];
  __shared__ float2 sml[kWarps][32];
  __shared__ int last;
  fa_grid_dep_sync();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, w = blockIdx.z, split = blockIdx.y;
  const int c = blockIdx.x * 128 + lane * 4;
  const bool live = c < p.C;
  const int cc = live ? c : 0, row = cc / p.D, col = cc - row * p.D;
  const size_t qoff = (size_t)w * p.q_win + (size_t)row * p.ldq + col;
  const float4 qv = *(const float4 *)(p.q + qoff);
  const float *kb = p.k + (size_t)w * p.kv_win + cc, *vb = p.v + (size_t)w * p.kv_win + cc;
  const int k0 = split * p.kper, k1 = min(p.Tk, k0 + p.kper);
  Running r{-INFINITY, 0.0f, make_float4(0.f, 0.f, 0.f, 0.f)};
  for (int j0 = k0 + warp * kU; j0 < k1; j0 += kWarps * kU) {
    float4 kx[kU], vx[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int j = j0 + u;
      kx[u] = vx[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j < k1) {
        if (APPEND) {
          const bool fresh = j == p.Tk - 1;
          kx[u] = *(const float4 *)(fresh ? p.knew + qoff : kb + (size_t)j * p.ld);
          vx[u] = *(const float4 *)(fresh ? p.vnew + qoff : vb + (size_t)j * p.ld);
        } else {
          kx[u] = __ldcs((const float4 *)(kb + (size_t)j * p.ld));
          vx[u] = __ldcs((const float4 *)(vb + (size_t)j * p.ld));
        }
      }
    }
    float d[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) d[u] = fmaf(qv.x, kx[u].x, fmaf(qv.y, kx[u].y, fmaf(qv.z, kx[u].z, qv.w * kx[u].w)));
    for (int o = p.lph >> 1; o > 0; o >>= 1) {
#pragma unroll
      for (int u = 0; u < kU; u++) d[u] += __shfl_xor_sync(0xffffffffu, d[u], o);
    }
    float nm = r.m;
#pragma unroll
    for (int u = 0; u < kU; u++)
      if (j0 + u < k1) nm = fmaxf(nm, d[u]);
    const float f = step_scale(r.m, nm);
    r.m = nm, r.l *= f, r.a.x *= f, r.a.y *= f, r.a.z *= f, r.a.w *= f;
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const float e = j0 + u < k1 && d[u] != -INFINITY ? expf(d[u] - nm) : 0.0f;  // (a NaN score stays one)
      r.l += e;
      r.a.x = fmaf(e, vx[u].x, r.a.x), r.a.y = fmaf(e, vx[u].y, r.a.y);
      r.a.z = fmaf(e, vx[u].z, r.a.z), r.a.w = fmaf(e, vx[u].w, r.a.w);
    }
    if (APPEND) {
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (j0 + u == p.Tk - 1 && live) {  // read by nobody in this launch: every lane above took the fresh row
          *(float4 *)(p.kc + (size_t)(j0 + u) * p.ld + c) = kx[u];
          *(float4 *)(p.vc + (size_t)(j0 + u) * p.ld + c) = vx[u];
        }
    }
  }
  merge_block(r, warp, lane, sa, sml);
  if (gridDim.y > 1) {
    if (warp == 0) {
      if (live) {
        const size_t o = ((size_t)w * gridDim.y + split) * p.C + c;
        *(float4 *)(p.pacc + o) = r.a;
        *(float2 *)(p.pml + o / 2) = make_float2(r.m, r.l);
        __threadfence();
      }
      __syncwarp();
      if (lane == 0) {
        int *t = p.tickets + (size_t)w * gridDim.x + blockIdx.x;
        last = atomicAdd(t, 1) == (int)gridDim.y - 1;
        if (last) *t = 0;  // ready for the next launch on this stream
      }
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    r = Running{-INFINITY, 0.0f, make_float4(0.f, 0.f, 0.f, 0.f)};
    for (int s = warp; s < (int)gridDim.y; s += kWarps) {
      const size_t o = ((size_t)w * gridDim.y + s) * p.C + cc;
      const float4 a = __ldcg((const float4 *)(p.pacc + o));
      const float2 ml = __ldcg((const float2 *)(p.pml + o / 2));
      merge(r, ml.x, ml.y, a);
    }
    merge_block(r, warp, lane, sa, sml);
  }
  if (warp == 0 && live) {
    const float inv = 1.0f / r.l;
    const float4 t = make_float4(r.a.x * inv, r.a.y * inv, r.a.z * inv, r.a.w * inv);
    *(float4 *)(p.out + (size_t)w * p.C + c) = t;
    if (p.y16) {
      const int orow = w * (p.C / p.D) + row;
      __half2 *d16 = (__half2 *)(p.y16 + ((size_t)(col >> 6) * p.R + orow) * 64 + (col & 63));
      const __half2 h0 = __floats2half2_rn(t.x, t.y), h1 = __floats2half2_rn(t.z, t.w);
      d16[0] = h0, d16[1] = h1;
      if (p.lo_off) {
        const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
        __half2 *l16 = (__half2 *)((__half *)d16 + p.lo_off);
        l16[0] = __floats2half2_rn(t.x - f0.x, t.y - f0.y);
        l16[1] = __floats2half2_rn(t.z - f1.x, t.w - f1.y);
      }
    }
  }
}

bool step_shape_ok(int HD) { return HD >= 4 && HD <= 128 && (HD & (HD - 1)) == 0; }
bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

// Launches over W windows of C = p.C columns and p.Tk keys; the result is [R][D].
int step_launch(fa_ctx *ctx, StepParams &p, int W, int HD, bool append, fa_tensor **out) {
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, p.R, p.D, FA_F32, true, &y));
  p.out = (float *)y->dptr;
  p.lph = HD / 4;
  if ((p.D & 63) == 0 && fa_tc_available(ctx)) {  // the product that follows reads the packed operand
    if (p.R <= ctx->f16_hilo_rows) {
      if ((p.y16 = fa_shadow_hilo_block(ctx, y)) != nullptr) p.lo_off = (long long)(p.D >> 6) * p.R * 64;
    } else {
      p.y16 = fa_shadow_block(ctx, y);
    }
    if (p.y16) y->a16_valid = true;
  }
  // Keys are split until about 8 blocks per SM exist (two are resident), with at least one row octet per warp in each:
  // below that a single stream leaves most SMs idle, above it the partial results cost more than the even tail gives.
  const int strips = ceil_div(p.C, 128);
  long long splits = ((long long)ctx->sm_count * 8 + (long long)strips * W - 1) / ((long long)strips * W);
  if (splits > ceil_div(p.Tk, kWarps * kU)) splits = ceil_div(p.Tk, kWarps * kU);
  if ((long long)strips * W > ctx->gemv_ticket_count || splits < 1) splits = 1;
  p.kper = ceil_div(ceil_div(p.Tk, (int)splits), kWarps * kU) * kWarps * kU;
  splits = ceil_div(p.Tk, p.kper);
  void *scratch = nullptr;
  size_t bytes = 0;
  int rc = FA_OK;
  if (splits > 1) {
    const size_t n = (size_t)W * splits * p.C;
    rc = fa_block_acquire(ctx, n * 4 + n * 2, &scratch, &bytes);
    p.pacc = (float *)scratch, p.pml = (float *)scratch + n, p.tickets = ctx->gemv_tickets;
  }
  if (rc == FA_OK) {
    LaunchScope ls(ctx, append ? "attn_step_append" : "attn_step");
    const cudaError_t e = fa_launch_dep(ctx, append ? k_attn_step<true> : k_attn_step<false>, dim3(strips, (unsigned)splits, W),
                                        dim3(kThreads), 0, p);
    if (e != cudaSuccess) rc = fa_fail(ctx, FA_ERR_CUDA, "launch attn_step: %s", cudaGetErrorString(e));
  }
  if (scratch) fa_block_release(ctx, scratch);
  if (rc != FA_OK) {
    fa_free_tensor(ctx, y);
    return rc;
  }
  *out = y;
  return FA_OK;
}

int step_operand(fa_ctx *ctx, const fa_tensor *t, const char *op) {
  FA_REQUIRE(ctx, fa_valid(ctx, t), "%s: unknown tensor handle", op);
  FA_REQUIRE(ctx, t->storage == FA_F32, "%s: operand must be f32 storage", op);
  return fa_touch_f32(ctx, t);
}

}  // namespace

extern "C" int fa_attn_step(fa_ctx *ctx, const fa_tensor *q, const fa_tensor *k, const fa_tensor *v, int H, int HD, int W,
                            fa_tensor **out) {
  if (!ctx || !out) return fa_fail(ctx, FA_ERR_INVALID, "attnStep: NULL argument");
  *out = nullptr;
  FA_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
  FA_TRY(step_operand(ctx, q, "attnStep"));
  FA_TRY(step_operand(ctx, k, "attnStep"));
  FA_TRY(step_operand(ctx, v, "attnStep"));
  FA_REQUIRE(ctx, H > 0 && HD > 0 && W > 0 && (long long)H * HD == q->cols && k->cols == q->cols && v->cols == q->cols,
             "attnStep: q/k/v need %lld columns", (long long)H * HD);
  FA_REQUIRE(ctx, q->rows % W == 0 && k->rows % W == 0 && v->rows == k->rows, "attnStep: rows not divisible by W=%d", W);
  if (q->rows != W || k->rows == 0 || W > 65535 || !step_shape_ok(HD) || !aligned16(q->dptr) || !aligned16(k->dptr) || !aligned16(v->dptr))
    return FA_OK;  // not this kernel's shape: the caller takes the separate ops
  StepParams p{};
  p.q = (const float *)q->dptr, p.k = (const float *)k->dptr, p.v = (const float *)v->dptr;
  p.C = p.D = q->cols, p.R = W, p.Tk = k->rows / W;
  p.q_win = p.C, p.ld = p.C, p.kv_win = (long long)p.Tk * p.C;
  return step_launch(ctx, p, W, HD, false, out);
}

extern "C" int fa_attn_step_append(fa_ctx *ctx, const fa_tensor *qkv, fa_tensor *cache_k, fa_tensor *cache_v, int n, int NH, int HD,
                                   fa_tensor **out) {
  if (!ctx || !out) return fa_fail(ctx, FA_ERR_INVALID, "attnStepAppend: NULL argument");
  *out = nullptr;
  FA_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
  FA_TRY(step_operand(ctx, qkv, "attnStepAppend"));
  FA_TRY(step_operand(ctx, cache_k, "attnStepAppend"));
  FA_TRY(step_operand(ctx, cache_v, "attnStepAppend"));
  const long long D = (long long)NH * HD, S = qkv->rows;
  FA_REQUIRE(ctx, NH > 0 && HD > 0 && qkv->cols == 3 * D, "attnStepAppend: qkv has %d columns, expected %lld", qkv->cols, 3 * D);
  FA_REQUIRE(ctx, cache_k != cache_v && cache_k->cols == S * D && cache_v->cols == S * D && n >= 0 && n < cache_k->rows && n < cache_v->rows,
             "attnStepAppend: caches need %lld columns and a row %d", S * D, n);
  if (S == 0 || !step_shape_ok(HD) || !aligned16(qkv->dptr) || !aligned16(cache_k->dptr) || !aligned16(cache_v->dptr))
    return FA_OK;
  StepParams p{};
  p.q = (const float *)qkv->dptr, p.knew = p.q + D, p.vnew = p.q + 2 * D;
  p.k = (const float *)cache_k->dptr, p.v = (const float *)cache_v->dptr;
  p.kc = (float *)cache_k->dptr, p.vc = (float *)cache_v->dptr;
  p.C = (int)(S * D), p.D = (int)D, p.R = (int)S, p.Tk = n + 1, p.ldq = (int)(3 * D), p.ld = p.C;
  fa_shadow_drop(cache_k);
  fa_shadow_drop(cache_v);
  return step_launch(ctx, p, 1, HD, true, out);
}
