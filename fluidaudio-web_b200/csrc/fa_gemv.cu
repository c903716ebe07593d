// Decode-size products (M <= 4 activation rows) on the CUDA cores: pure streams over the weights in the
// layouts the reference uploads them in (no repack, no packing prepass, no TMEM or cluster set-up), with
// 128-bit coalesced loads, in-register dequantisation and f32 / exact-integer accumulation.
//
//   k_gemv_nbits  matmulNBits (rust/wasm-kernels/src/lib.rs:169-203): bq [N][nblk][16] nibbles, K-contiguous.
//                 One warp per output column; a lane takes whole 32-weight blocks (one 16-byte load each).
//                 The activation row is split, inside the kernel, into two int8 digits of its own maximum,
//                 stored in the even/odd order the nibbles unpack to, so a block is 16 dp4a per digit pair
//                 and its sum is an exact integer; zero-point and scale are applied once per block:
//                 y = s_m * sum_blk scale[n,blk] * ((S1 - zp*A1) + (S2 - zp*A2) / 128).
//                 Arithmetic budget: ~1 lane-op per weight at M = 1 (an f32 unpack-and-FMA needs 4).
//   k_gemv_kn     matmul with f16-storage B [K][N] (lib.rs:59-94) and matmulInt8 with wq [K][N]
//                 (lib.rs:143-162) at M = 1: N-contiguous rows.  A block owns 128 or 64 consecutive columns, its 8
//                 warps take rows k round-robin, K is split over the ranks of a cluster; activations stay f32 (exact),
//                 and a layernorm of the row can run in front of the product.  Sums meet in a fixed order.
#include <cuda_fp16.h>

#include <type_traits>

#include "fa_internal.cuh"

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---- int4 ---------------------------------------------------------------------------------------

// One 32-weight block of R weight rows against the digits of every activation row.
template <int M, int R>
__device__ __forceinline__ void nbits_block(const uint4 (&wv)[R], const float (&sc)[R], const int (&z)[R], int b, int K, int nblk,
                                            const int8_t *dig, const int *SA, float (&acc)[R][M]) {
  int lo[R][4], hi[R][4];
#pragma unroll
  for (int r = 0; r < R; r++) {
    lo[r][0] = (int)(wv[r].x & 0x0F0F0F0Fu), hi[r][0] = (int)((wv[r].x >> 4) & 0x0F0F0F0Fu);
    lo[r][1] = (int)(wv[r].y & 0x0F0F0F0Fu), hi[r][1] = (int)((wv[r].y >> 4) & 0x0F0F0F0Fu);
    lo[r][2] = (int)(wv[r].z & 0x0F0F0F0Fu), hi[r][2] = (int)((wv[r].z >> 4) & 0x0F0F0F0Fu);
    lo[r][3] = (int)(wv[r].w & 0x0F0F0F0Fu), hi[r][3] = (int)((wv[r].w >> 4) & 0x0F0F0F0Fu);
  }
#pragma unroll
  for (int m = 0; m < M; m++) {
    const int4 e1 = *(const int4 *)(dig + (size_t)(m * 2 + 0) * K + b * 16);
    const int4 o1 = *(const int4 *)(dig + (size_t)(m * 2 + 0) * K + (K >> 1) + b * 16);
    const int4 e2 = *(const int4 *)(dig + (size_t)(m * 2 + 1) * K + b * 16);
    const int4 o2 = *(const int4 *)(dig + (size_t)(m * 2 + 1) * K + (K >> 1) + b * 16);
    const int a1 = SA[(m * 2 + 0) * nblk + b], a2 = SA[(m * 2 + 1) * nblk + b];
#pragma unroll
    for (int r = 0; r < R; r++) {
      int s1 = 0, s2 = 0;
      s1 = __dp4a(lo[r][0], e1.x, s1), s1 = __dp4a(hi[r][0], o1.x, s1);
      s1 = __dp4a(lo[r][1], e1.y, s1), s1 = __dp4a(hi[r][1], o1.y, s1);
      s1 = __dp4a(lo[r][2], e1.z, s1), s1 = __dp4a(hi[r][2], o1.z, s1);
      s1 = __dp4a(lo[r][3], e1.w, s1), s1 = __dp4a(hi[r][3], o1.w, s1);
      s2 = __dp4a(lo[r][0], e2.x, s2), s2 = __dp4a(hi[r][0], o2.x, s2);
      s2 = __dp4a(lo[r][1], e2.y, s2), s2 = __dp4a(hi[r][1], o2.y, s2);
      s2 = __dp4a(lo[r][2], e2.z, s2), s2 = __dp4a(hi[r][2], o2.z, s2);
      s2 = __dp4a(lo[r][3], e2.w, s2), s2 = __dp4a(hi[r][3], o2.w, s2);
      const float f = fmaf((float)(s2 - z[r] * a2), 1.0f / 128.0f, (float)(s1 - z[r] * a1));
      acc[r][m] = fmaf(sc[r], f, acc[r][m]);
    }
  }
}

// The kernel is one pass: a warp's first (for the benchmark shapes: only) group of R weight rows is requested
// from HBM BEFORE the activation digits are made - before the kernel even waits for its predecessor in the stream:
// the packed weights of a PackedBytes handle are only ever written by an upload, never by a kernel, so reading them
// early is safe, while scales, zero-points and activations (tensors a kernel may have produced) are read after the
// wait.  The stream over the weights - the whole cost of the product - thus runs under the predecessor's tail and
// the prologue instead of after them (measured before the change: ~4 us of a 5.5 us launch had no weight byte in
// flight, against 1.6 us of streaming).  PRE blocks per lane and column are requested early, PRE * R the same for every
// R: few columns on long rows (N = 2048, K = 8192) keep as many bytes in flight as many on short ones, see launch_nbits.
// Prologue: a thread owns 8 consecutive k of one row, which is exactly one 32-bit word of the even-k digit plane and
// one of the odd-k plane, so digits go to shared memory as whole words and the per-block digit sums are two shuffles.
template <int M, int R, int PRE>
__global__ void __launch_bounds__(kThreads, 2) k_gemv_nbits(const float *__restrict__ a, const uint8_t *__restrict__ bq,
                                                            const float *__restrict__ scales, const uint8_t *__restrict__ zp,
                                                            float *__restrict__ y, int N, int K, int nblk, int zpb) {
  extern __shared__ __align__(16) unsigned char smem[];
  int8_t *dig = (int8_t *)smem;                     // [M][2] planes of K bytes: even-k words of every block (16 B
                                                    // each, so 8 lanes read 128 consecutive bytes), then odd-k words
  int *SA = (int *)(smem + (size_t)M * 2 * K);      // [M][2][nblk] digit sums per block
  float *red = (float *)(SA + M * 2 * nblk);        // [8][M] per-warp row maxima
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint4 *bq4 = (const uint4 *)bq;
  const int n_first = (blockIdx.x * 8 + warp) * R, n_stride = gridDim.x * 8 * R;

  // ---- early requests: the first group's weights --------------------------------------------------------------
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  uint4 pw[PRE][R];
#pragma unroll
  for (int i = 0; i < PRE; i++) {
    const int b = lane + 32 * i;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int n = n_first + r < N ? n_first + r : N - 1;
      pw[i][r] = (b < nblk && n_first < N) ? __ldcs(bq4 + (size_t)n * nblk + b) : make_uint4(0u, 0u, 0u, 0u);
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  float psc[PRE][R];
  unsigned pzb[PRE][R];
#pragma unroll
  for (int i = 0; i < PRE; i++) {
    const int b = lane + 32 * i;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int n = n_first + r < N ? n_first + r : N - 1;
      const bool ok = b < nblk && n_first < N;
      psc[i][r] = ok ? __ldg(scales + (size_t)n * nblk + b) : 0.f;
      pzb[i][r] = ok ? (unsigned)__ldg(zp + (size_t)n * zpb + (b >> 1)) : 0u;
    }
  }

  // ---- activation digits: q1 = rint(a/s), q2 = rint((a/s - q1) * 128) with s = max|row| / 127 --------------------
  // The warps split the rows between them (8 / M warps per row), so the code below handles ONE row per thread and
  // its register need does not grow with M; the second sweep re-reads the row (a few KB, L1-resident).
  constexpr int WPR = 8 / M;                       // warps per row (M = 3: two warps idle here)
  const int row = warp % M, wr = warp / M;
  const bool prow = wr < WPR;
  const float *arow = a + (size_t)row * K;
  float mx = 0.f;
  if (prow)
    for (int k0 = (wr * 32 + lane) * 8; k0 < K; k0 += WPR * 256) {
      const float4 x0 = __ldg((const float4 *)(arow + k0)), x1 = __ldg((const float4 *)(arow + k0 + 4));
      mx = fmaxf(mx, fmaxf(fmaxf(fabsf(x0.x), fabsf(x0.y)), fmaxf(fabsf(x0.z), fabsf(x0.w))));
      mx = fmaxf(mx, fmaxf(fmaxf(fabsf(x1.x), fabsf(x1.y)), fmaxf(fabsf(x1.z), fabsf(x1.w))));
    }
  mx = warp_max_f(mx);
  if (lane == 0) red[warp] = mx;
  __syncthreads();
  float rs[M];
#pragma unroll
  for (int m = 0; m < M; m++) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < WPR; w++) t = fmaxf(t, red[w * M + m]);
    rs[m] = t > 0.f ? t / 127.0f : 1.0f;
  }
  if (prow) {
    float inv = 1.0f;
#pragma unroll
    for (int m = 0; m < M; m++)
      if (m == row) inv = 1.0f / rs[m];
    const int kend = ((K + WPR * 256 - 1) / (WPR * 256)) * (WPR * 256);  // whole warps stay together for the shuffles
    for (int k0 = (wr * 32 + lane) * 8; k0 < kend; k0 += WPR * 256) {
      const bool in = k0 < K;
      const int b = k0 >> 5, wi = (k0 & 31) >> 3;
      float x[8];
      if (in) {
        const float4 x0 = __ldg((const float4 *)(arow + k0)), x1 = __ldg((const float4 *)(arow + k0 + 4));
        x[0] = x0.x, x[1] = x0.y, x[2] = x0.z, x[3] = x0.w, x[4] = x1.x, x[5] = x1.y, x[6] = x1.z, x[7] = x1.w;
      } else {
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = 0.f;
      }
      int q1[8], q2[8], s1 = 0, s2 = 0;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const float t = x[i] * inv;
        const float f1 = rintf(t);
        q1[i] = (int)f1;
        q2[i] = (int)rintf((t - f1) * 128.0f);
        s1 += q1[i];
        s2 += q2[i];
      }
      // digit words: bytes = k 0,2,4,6 (even plane) and 1,3,5,7 (odd plane) of this thread's 8
      auto pack = [](int b0, int b1, int b2, int b3) {
        return (unsigned)(b0 & 0xFF) | ((unsigned)(b1 & 0xFF) << 8) | ((unsigned)(b2 & 0xFF) << 16) | ((unsigned)(b3 & 0xFF) << 24);
      };
      if (in) {
        *(unsigned *)(dig + (size_t)(row * 2 + 0) * K + b * 16 + wi * 4) = pack(q1[0], q1[2], q1[4], q1[6]);
        *(unsigned *)(dig + (size_t)(row * 2 + 0) * K + (K >> 1) + b * 16 + wi * 4) = pack(q1[1], q1[3], q1[5], q1[7]);
        *(unsigned *)(dig + (size_t)(row * 2 + 1) * K + b * 16 + wi * 4) = pack(q2[0], q2[2], q2[4], q2[6]);
        *(unsigned *)(dig + (size_t)(row * 2 + 1) * K + (K >> 1) + b * 16 + wi * 4) = pack(q2[1], q2[3], q2[5], q2[7]);
      }
      // the 4 lanes of a 32-weight block
      s1 += __shfl_xor_sync(0xffffffffu, s1, 1), s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
      s2 += __shfl_xor_sync(0xffffffffu, s2, 1), s2 += __shfl_xor_sync(0xffffffffu, s2, 2);
      if (in && (lane & 3) == 0) {
        SA[(row * 2 + 0) * nblk + b] = s1;
        SA[(row * 2 + 1) * nblk + b] = s2;
      }
    }
  }
  __syncthreads();

  for (int n0 = n_first; n0 < N; n0 += n_stride) {
    float acc[R][M];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int m = 0; m < M; m++) acc[r][m] = 0.f;
    const bool early = n0 == n_first;
#pragma unroll
    for (int i = 0; i < PRE; i++) {
      const int b = lane + 32 * i;
      if (b >= nblk) break;
      uint4 wv[R];
      float sc[R];
      int z[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        unsigned zb;
        if (early) {
          wv[r] = pw[i][r], sc[r] = psc[i][r], zb = pzb[i][r];
        } else {
          const int n = n0 + r < N ? n0 + r : N - 1;
          wv[r] = __ldcs(bq4 + (size_t)n * nblk + b);
          sc[r] = scales[(size_t)n * nblk + b];
          zb = zp[(size_t)n * zpb + (b >> 1)];
        }
        z[r] = (b & 1) ? (int)(zb >> 4) : (int)(zb & 15u);
      }
      nbits_block<M, R>(wv, sc, z, b, K, nblk, dig, SA, acc);
    }
    for (int b = lane + 32 * PRE; b < nblk; b += 32) {
      uint4 wv[R];
      float sc[R];
      int z[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int n = n0 + r < N ? n0 + r : N - 1;
        wv[r] = __ldcs(bq4 + (size_t)n * nblk + b);
        sc[r] = scales[(size_t)n * nblk + b];
        const unsigned zb = zp[(size_t)n * zpb + (b >> 1)];
        z[r] = (b & 1) ? (int)(zb >> 4) : (int)(zb & 15u);
      }
      nbits_block<M, R>(wv, sc, z, b, K, nblk, dig, SA, acc);
    }
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int m = 0; m < M; m++) {
        const float t = warp_sum_f(acc[r][m]);
        if (lane == 0 && n0 + r < N) y[(size_t)m * N + n0 + r] = t * rs[m];
      }
  }
}

// ---- f16 / int8 weights, N-contiguous ---------------------------------------------------------------

struct GemvEp {
  const float *colscale, *bias, *add;
  int act;
};

__device__ __forceinline__ float gemv_finish(float acc, int m, int n, int N, const GemvEp &ep) {
  float v = acc;
  if (ep.colscale) v *= ep.colscale[n];
  if (ep.bias) v += ep.bias[n];
  v = fa_actf(v, ep.act);
  if (ep.add) v += ep.add[(size_t)m * N + n];
  return v;
}

// Four consecutive weights of a row as loaded: 4 bytes of int8, 8 of f16.
template <bool I8>
struct RawRow {
  using type = typename std::conditional<I8, unsigned, uint2>::type;
};
// Two f32 values in a register pair, and the packed add and multiply-add on them (each half rounded like the scalar one).
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// The four weights as f32 pairs of columns (0, 1) and (2, 3).
__device__ __forceinline__ void widen(unsigned v, uint64_t &w01, uint64_t &w23) {
  // byte b of (q + 128) into the mantissa of 2^23: the float 8388608 + q + 128, then back to q
  const unsigned x = v ^ 0x80808080u;
  const uint64_t off = pack2(-8388736.0f, -8388736.0f);
  w01 = add2(pack2(__uint_as_float(__byte_perm(x, 0x4B000000u, 0x7650)), __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7651))), off);
  w23 = add2(pack2(__uint_as_float(__byte_perm(x, 0x4B000000u, 0x7652)), __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7653))), off);
}
__device__ __forceinline__ void widen(uint2 v, uint64_t &w01, uint64_t &w23) {
  const __half2 *h = (const __half2 *)&v;
  const float2 a = __half22float2(h[0]), b = __half22float2(h[1]);
  w01 = pack2(a.x, a.y), w23 = pack2(b.x, b.y);
}

__device__ __forceinline__ float block_sum(float v, float *red, int lane, int warp) {
  v = warp_sum_f(v);
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = red[0];
#pragma unroll
  for (int i = 1; i < kThreads / 32; i++) t += red[i];
  __syncthreads();
  return t;
}

// y[n] = act(sum_k x[k] * w[k][n] * colscale[n] + bias[n]) + add[n] for ONE row x [K]; with NORM, x is first replaced by
// its layernorm (gamma, beta: two-pass mean and variance as in k_layernorm_reg).
//
// What bounds it: the instructions of the inner loop and the weight stream for the large matrices, latency for the others:
// 1.6 MB are 0.3 us of HBM time, so the launch is a chain of load -> row sum -> exchange between K slices.
// Layout: a block owns 128 columns (one 4-byte int8 or 8-byte f16 load per lane and row; 64 columns, two rows per warp, where
// 128 with the widest K split would not give every SM a block) and a K slice, its 8 warps take rows round-robin with two
// batches of U loads per lane in flight, the first ones requested before the launch waits for its predecessor where the
// weights can only have been written by an upload (int8 payloads).  K slices are the ranks of a cluster: their sums meet in
// rank 0's shared memory, in rank order, after one cluster barrier.
// A whole batch is loaded without a bound per row (rows past the end meet a zero activation instead), an activation lies in
// shared memory twice so that one 8-byte read is the operand of two packed multiply-adds, and U and the resident blocks are
// chosen together: 16 loads of int8 (8 where two batches of 8 cover the slice) and 8 of f16, at three blocks per SM, or at
// four in 64 registers where the grid needs them.  With 16 loads of f16 (112 registers, two blocks per SM), a bound per row and
// scalar arithmetic the wide products took, us at one row -> now: f16 1280 x 5120 10.6 -> 5.8, 1280 x 51868 47.9 -> 23.3 (5.7
// TB/s), 5120 x 10240 47.0 -> 20.0; int8 1280 x 20484 14.8 -> 10.0, 1280 x 51868 26.7 -> 15.7 (4.2 TB/s), 5120 x 10244 27.3 ->
// 16.3; small ones 1280 x 1280 3.9 -> 3.3 (int8), 4.6 -> 3.3 (f16).  The same int8 products as a digit pass and a tensor-core
// product of two int8 digits: 1280 x 51868 16.0, 1280 x 20484 10.3, 5120 x 10244 16.3.
// In a decoder step the launch stands for a layernorm, a product and a residual add: 1280 x 51868 int8 with its layernorm 16.0 us
// against 3.8 + 2.6 + 12.5.
constexpr int kKnCols = 128, kKnSlice = 2048;  // most columns per block, rows of x held at a time
constexpr int kKnNormMax = 4096;               // longest row that the layernorm prologue holds in registers

struct KnParams {
  const float *x, *gamma, *beta;
  const void *w;
  float *y;
  int K, N, kslice;
  float eps;
  GemvEp ep;
};

template <bool I8, bool NORM, int COLS, int U, int BLOCKS>
__global__ void __launch_bounds__(kThreads, BLOCKS) k_gemv_kn(const KnParams p) {
  constexpr int RPW = kKnCols / COLS, kStride = 8 * RPW;  // rows a warp reads at once, rows of a block's 8 warps
  constexpr int B = kStride * U;                          // rows of a batch
  static_assert(kKnSlice % (2 * B) == 0, "a slice is whole pairs of batches, but for the last");
  __shared__ __align__(16) float2 xs[kKnSlice];  // each activation twice, zeros up to the end of a pair of batches
  __shared__ __align__(16) float4 red[kThreads / 32][COLS / 4];
  __shared__ float cred[8][COLS];  // rank 0: the K slices' sums
  __shared__ float stat[kThreads / 32];
  using Raw = typename RawRow<I8>::type;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.y, ks = gridDim.y, N = p.N, K = p.K;
  const int k0 = min(K, rank * p.kslice), k1 = min(K, k0 + p.kslice);
  const int c0 = blockIdx.x * COLS + (lane % (COLS / 4)) * 4;
  const bool live = c0 < N;  // N % 4 == 0: a live lane owns four whole columns
  const int cc = live ? c0 : 0;
  const int below = RPW - 1 - lane / (COLS / 4);  // a warp's last row of a step lies this far below the lane's
  const size_t elem = I8 ? 1 : 2, step = (size_t)kStride * N * elem;
  Raw ra[U], rb[U];
  auto fetch = [&](Raw(&raw)[U], int kk) {
    const char *q = (const char *)p.w + ((size_t)kk * N + cc) * elem;
    if (kk + below + (U - 1) * kStride < k1) {
#pragma unroll
      for (int u = 0; u < U; u++, q += step) raw[u] = __ldcs((const Raw *)q);
    } else {
#pragma unroll
      for (int u = 0; u < U; u++, q += step) {
        raw[u] = Raw{};
        if (kk + u * kStride < k1) raw[u] = __ldcs((const Raw *)q);
      }
    }
  };
  int kk = k0 + warp * RPW + lane / (COLS / 4);  // rows kk, kk + kStride, ...
  if (I8) fetch(ra, kk), fetch(rb, kk + B);
  if (ks > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // every rank runs before a remote store
  fa_grid_dep_sync();
  if (!I8) fetch(ra, kk), fetch(rb, kk + B);
  auto padded = [](int rows) { return (rows + 2 * B - 1) / (2 * B) * (2 * B); };
  if (NORM) {
    float4 v[kKnNormMax / 4 / kThreads];
    const int k4 = K >> 2;
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < kKnNormMax / 4 / kThreads; u++) {
      const int q = tid + u * kThreads;
      v[u] = q < k4 ? ((const float4 *)p.x)[q] : make_float4(0.f, 0.f, 0.f, 0.f);
      s += (v[u].x + v[u].y) + (v[u].z + v[u].w);
    }
    const float mean = block_sum(s, stat, lane, warp) / (float)K;
    float vs = 0.f;
#pragma unroll
    for (int u = 0; u < kKnNormMax / 4 / kThreads; u++)
      if (tid + u * kThreads < k4) {
        const float a = v[u].x - mean, b = v[u].y - mean, c = v[u].z - mean, d = v[u].w - mean;
        vs += (a * a + b * b) + (c * c + d * d);
      }
    const float inv = 1.0f / sqrtf(block_sum(vs, stat, lane, warp) / (float)K + p.eps);
#pragma unroll
    for (int u = 0; u < kKnNormMax / 4 / kThreads; u++) {
      const int q = tid + u * kThreads, k = q * 4;
      if (q < k4 && k >= k0 && k < k1) {  // kslice % 8 == 0: a quad lies in one slice; the slice fits xs (host check)
        const float4 g = ((const float4 *)p.gamma)[q], b = ((const float4 *)p.beta)[q];
        const float4 t = make_float4((v[u].x - mean) * inv * g.x + b.x, (v[u].y - mean) * inv * g.y + b.y,
                                     (v[u].z - mean) * inv * g.z + b.z, (v[u].w - mean) * inv * g.w + b.w);
        float4 *d = (float4 *)(xs + (k - k0));
        d[0] = make_float4(t.x, t.x, t.y, t.y), d[1] = make_float4(t.z, t.z, t.w, t.w);
      }
    }
    for (int i = k1 - k0 + tid; i < padded(k1 - k0); i += kThreads) xs[i] = make_float2(0.f, 0.f);
    __syncthreads();
  }
  auto load_x = [&](int base, int end) {
    for (int i = tid; i < padded(end - base); i += kThreads) {
      const float x = base + i < end ? p.x[base + i] : 0.0f;
      xs[i] = make_float2(x, x);
    }
    __syncthreads();
  };
  if (!NORM) load_x(k0, min(k1, k0 + kKnSlice));
  uint64_t a01 = 0, a23 = 0;  // sums of columns (0, 1) and (2, 3)
#pragma unroll 1
  for (int base = k0; base < k1; base += kKnSlice) {
    const int end = min(k1, base + kKnSlice);
    if (!NORM && base > k0) __syncthreads(), load_x(base, end);
    auto consume = [&](const Raw(&raw)[U], int kk) {
      const uint64_t *x = (const uint64_t *)xs + (kk - base);
#pragma unroll
      for (int u = 0; u < U; u++) {
        uint64_t w01, w23;
        widen(raw[u], w01, w23);
        const uint64_t a = x[u * kStride];
        a01 = fma2(a, w01, a01), a23 = fma2(a, w23, a23);
      }
    };
#pragma unroll 1
    for (; kk < end; kk += 2 * B) {
      consume(ra, kk);
      if (kk + 2 * B < k1) fetch(ra, kk + 2 * B);
      consume(rb, kk + B);
      if (kk + 3 * B < k1) fetch(rb, kk + 3 * B);
    }
  }
  const float2 s01 = unpack2(a01), s23 = unpack2(a23);
  float4 acc = make_float4(s01.x, s01.y, s23.x, s23.y);
  if (RPW == 2) {
    __syncwarp();
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, 16), acc.y += __shfl_xor_sync(0xffffffffu, acc.y, 16);
    acc.z += __shfl_xor_sync(0xffffffffu, acc.z, 16), acc.w += __shfl_xor_sync(0xffffffffu, acc.w, 16);
  }
  if (lane < COLS / 4) red[warp][lane] = acc;
  __syncthreads();
  float sum = 0.f;
  if (tid < COLS) {
    const float *r = (const float *)red;
    sum = r[tid];
#pragma unroll
    for (int i = 1; i < kThreads / 32; i++) sum += r[i * COLS + tid];
  }
  if (ks > 1) {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (tid < COLS) {
      uint32_t remote;
      const uint32_t local = (uint32_t)__cvta_generic_to_shared(&cred[rank][tid]);
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(0));
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(sum) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (rank != 0) return;
    if (tid < COLS) {
      sum = cred[0][tid];
      for (int i = 1; i < ks; i++) sum += cred[i][tid];
    }
  }
  const int n = blockIdx.x * COLS + tid;
  if (tid < COLS && n < N) p.y[n] = gemv_finish(sum, 0, n, N, p.ep);
}

constexpr size_t kNbitsSmemMax = 97 * 1024;  // fa_gemv_nbits_ok keeps every launch below

template <int M, int R, int PRE>
int launch_nbits_r(fa_ctx *ctx, const float *a, const uint8_t *bq, const float *scales, const uint8_t *zp, float *y, int N,
                   int K, int nblk, int zpb) {
  const size_t smem = (size_t)M * 2 * K + (size_t)M * 2 * nblk * 4 + 8 * M * 4;
  auto kern = k_gemv_nbits<M, R, PRE>;
  static SmemLimit limit;
  FA_CHECK_CUDA(ctx, limit.raise(ctx, kern, kNbitsSmemMax));
  // one resident wave: every CTA pays the digit prologue once and a second wave would pay it twice
  int per_sm = 0;
  FA_CHECK_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem));
  if (per_sm < 1) per_sm = 1;
  if (per_sm > ctx->gemv_ctas_per_sm) per_sm = ctx->gemv_ctas_per_sm;
  int grid = ceil_div(N, 8 * R);
  if (grid > ctx->sm_count * per_sm) grid = ctx->sm_count * per_sm;
  {
    LaunchScope ls(ctx, "gemv_nbits");
    fa_launch_dep(ctx, kern, dim3(grid), dim3(kThreads), smem, a, bq, scales, zp, y, N, K, nblk, zpb);
  }
  FA_LAUNCH_CHECK(ctx, "gemv_nbits");
  return FA_OK;
}

// Output columns per warp pass (each digit load is shared between R rows of weights): 4 for one activation row - with two
// resident CTAs per SM (register cap 128) one wave then covers 148 * 2 * 8 * 4 = 9472 columns - and 2 for more rows,
// where 4 would not fit the registers next to the early-requested weights; fewer while the CTAs would not cover the SMs, on
// rows longer than the two blocks per lane that the wide form requests early (K > 2048).
// Measured at one row, K = 8192, N = 2048 in a recorded chain: 64 CTAs of 4 columns per warp 11.5 us, 256 of 1 column
// 6.7 us (11 MB: 1.6 us of HBM time); N = 8192, K = 2048 keeps its 4 columns (4.2 us).  On short rows more CTAs only repeat
// the digit prologue: N = 2048, K = 2048 2.8 us at 4 columns, 3.2 at 1; four rows, N = 512, K = 2048 4.6 us at 2, 5.1 at 1.
template <int M>
int launch_nbits(fa_ctx *ctx, const float *a, const uint8_t *bq, const float *scales, const uint8_t *zp, float *y, int N,
                 int K, int nblk, int zpb) {
  const bool is_short = nblk <= 64;
  if constexpr (M == 1) {
    if (is_short || ceil_div(N, 8 * 4) >= ctx->sm_count) return launch_nbits_r<1, 4, 2>(ctx, a, bq, scales, zp, y, N, K, nblk, zpb);
    if (ceil_div(N, 8 * 2) >= ctx->sm_count) return launch_nbits_r<1, 2, 4>(ctx, a, bq, scales, zp, y, N, K, nblk, zpb);
    return launch_nbits_r<1, 1, 8>(ctx, a, bq, scales, zp, y, N, K, nblk, zpb);
  } else {
    if (is_short || ceil_div(N, 8 * 2) >= ctx->sm_count) return launch_nbits_r<M, 2, 2>(ctx, a, bq, scales, zp, y, N, K, nblk, zpb);
    return launch_nbits_r<M, 1, 4>(ctx, a, bq, scales, zp, y, N, K, nblk, zpb);
  }
}

}  // namespace

bool fa_gemv_nbits_ok(int M, int N, int K, int block_size) {
  return M >= 1 && M <= kGemvMaxRows && block_size == 32 && (K & 31) == 0 && K >= 32 && N >= 1 &&
         (size_t)M * 2 * K + (size_t)M * (K / 32) * 8 + 64 <= 96 * 1024;
}

int fa_gemv_nbits(fa_ctx *ctx, const float *a, const uint8_t *bq, const float *scales, const uint8_t *zp, float *y, int M,
                  int N, int K, int nblk, int zpb) {
  switch (M) {
    case 1: return launch_nbits<1>(ctx, a, bq, scales, zp, y, N, K, nblk, zpb);
    case 2: return launch_nbits<2>(ctx, a, bq, scales, zp, y, N, K, nblk, zpb);
    case 3: return launch_nbits<3>(ctx, a, bq, scales, zp, y, N, K, nblk, zpb);
    default: return launch_nbits<4>(ctx, a, bq, scales, zp, y, N, K, nblk, zpb);
  }
}

namespace {

// ---- int4, 5..16 activation rows: weights streamed once as uploaded, widened in registers, mma.sync -------------------
// The tensor-core GEMM serves these shapes from a dequantised f16 copy of the weights: four times the bytes, a packing
// prepass and a split-K hand-off for ~0.5 GFLOP of work, and weights (q - zp) * scale rounded to f16.  Here the 4-bit
// weights are read once, in the layout they were uploaded in, and the block scale multiplies the block's f32 sum, so that
// the weights stay exact.
//
// What bounds it: instruction issue.  A warp owns ONE quad of 32-weight blocks (16 warps x 4 blocks = the 2048 k that the
// activation planes of 16 rows leave room for in shared memory; on shorter slices several warps share a quad's columns) and walks up to G groups of 8 output columns with it:
//   - a lane loads one whole block per group (16 bytes; the 4 lanes of a column read 64 consecutive bytes), all groups up
//     front, before the launch waits for its predecessor (the payload is only ever written by an upload);
//   - a 4 x 4 transpose between the 4 lanes of a column (4 shuffles) gives each lane word j of all four blocks, so that
//     one mma.sync.m16n8k16 works inside ONE block and the scale can wait for its result;
//   - a nibble pair (k, k + 4) becomes two f16 `1024 + q` with one mask, minus 1024 + zp: exact.  Which k sits in which of
//     the instruction's slots does not matter for a sum; rows r and r + 8 lie in shared memory interleaved in the same order,
//     so that one 16-byte load IS a lane's A operand (four registers in a row: put together from two loads it cost a move per
//     register, group and block), and are read once per block for all groups (pitch = 64 mod 128 bytes: conflict-free);
//   - per block and group: 4 mma (value and residue plane of the activations), then 4 multiply-adds with the scale.
// The 16 warps' sums meet in shared memory in warp order; from K = 2048 on K is split over the four ranks of a cluster, whose
// sums meet in rank 0's shared memory in rank order.
// Measured, 16 rows, recorded blocks: 13.2 us on average for K = 2048, N = 8192 and K = 8192, N = 2048, against 14.1 and 20.0 us
// (digit pass included) for the f16 copy on the tensor cores, which read 33.5 MB where this reads 10.5.  What is left is the
// chain of one launch: its 512 threads of 128 registers cannot start beside the block before them.
constexpr int kMmaWarps = 16, kMmaThreads = kMmaWarps * 32;
constexpr int kMmaSliceBlk = kMmaWarps * 4;  // 32-weight blocks per K slice
constexpr int kMmaMaxSlices = 4;
__host__ __device__ constexpr int mma_row_pitch(int blks) { return blks * 128 + 64; }  // rows r and r + 8 together

__device__ __forceinline__ void mma16816_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The same from a zero accumulator.
__device__ __forceinline__ void mma16816_f16_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}

struct MmaParams {
  const float *a;
  const uint8_t *bq;
  const float *scales;
  const uint8_t *zp;
  float *y;
  int M, N, K, nblk, zpb;
  int slice;  // blocks per K slice (a multiple of 4, at most kMmaSliceBlk)
  int lq;     // log2 of the quads per slice that have warps of their own (16, 8 or 4): 16 >> lq warps share a quad's columns
  int gper;   // column groups per thread block
};

// Lane j of 4 holds words 0..3 of block j; afterwards word j of blocks 0..3.
__device__ __forceinline__ void transpose4(uint4 &w, int lane) {
  const bool o1 = lane & 1, o2 = lane & 2;
  unsigned t = __shfl_xor_sync(0xffffffffu, o1 ? w.x : w.y, 1);
  if (o1) w.x = t; else w.y = t;
  t = __shfl_xor_sync(0xffffffffu, o1 ? w.z : w.w, 1);
  if (o1) w.z = t; else w.w = t;
  t = __shfl_xor_sync(0xffffffffu, o2 ? w.x : w.z, 2);
  if (o2) w.x = t; else w.z = t;
  t = __shfl_xor_sync(0xffffffffu, o2 ? w.y : w.w, 2);
  if (o2) w.y = t; else w.w = t;
}

template <bool HILO, int G>
__global__ void __launch_bounds__(kMmaThreads, 1) k_nbits_mma(const MmaParams p) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g4 = lane >> 2, j4 = lane & 3;
  const int rank = blockIdx.y, slices = gridDim.y, b0 = rank * p.slice, nb = min(p.slice, p.nblk - b0);  // blocks of this slice
  const int pitch = mma_row_pitch(p.slice);
  unsigned char *ap = smem;                                                     // [planes][8 row pairs][pitch]
  float4 *red = (float4 *)(smem + (size_t)(HILO ? 2 : 1) * 8 * pitch);         // [quads][gall][32]
  const int gw = kMmaWarps >> p.lq, gall = G * gw;                              // warps per quad, groups of a pass
  float4 *cred = red + kMmaWarps * G * 32;                                      // rank 0: [2][slices][gall][32]
  const int quad = warp & ((1 << p.lq) - 1), goff = (warp >> p.lq) * G;         // the warp's quad and first group of a pass
  const int qb = b0 + quad * 4;         // first block of the quad
  const int qn = min(4, b0 + nb - qb);  // its blocks (<= 0: none)
  const int groups = p.N >> 3, gfirst = blockIdx.x * p.gper, gend = min(groups, gfirst + p.gper);
  const uint4 *bq4 = (const uint4 *)p.bq;

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  uint4 w[G];
  auto fetch = [&](int g0) {
#pragma unroll
    for (int g = 0; g < G; g++) {
      w[g] = make_uint4(0u, 0u, 0u, 0u);
      if (g0 + goff + g < gend && j4 < qn) w[g] = __ldcs(bq4 + (size_t)((g0 + goff + g) * 8 + g4) * p.nblk + qb + j4);
    }
  };
  fetch(gfirst);
  if (slices > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // every rank runs before a remote store
  asm volatile("griddepcontrol.wait;" ::: "memory");

  float sc[G];     // lane: block j4 of column g4
  unsigned z4[G];  // column g4: zero-points of the quad's blocks, a nibble each
  auto fetch_scales = [&](int g0) {
#pragma unroll
    for (int g = 0; g < G; g++) {
      sc[g] = 0.f, z4[g] = 0u;
      if (g0 + goff + g < gend && qn > 0) {
        const int n = (g0 + goff + g) * 8 + g4;
        if (j4 < qn) sc[g] = __ldg(p.scales + (size_t)n * p.nblk + qb + j4);
        const uint8_t *z = p.zp + (size_t)n * p.zpb + (qb >> 1);  // qb is a multiple of 4
        z4[g] = __ldg(z);
        if (qn > 2) z4[g] |= (unsigned)__ldg(z + 1) << 8;
      }
    }
  };
  fetch_scales(gfirst);  // (a kernel may have made them: not before the wait)

  // activation rows of this K slice: 8 consecutive k of rows r and r + 8 per step, as the two A operands {r: k0,k4 | r+8: k0,k4 |
  // r: k1,k5 | r+8: k1,k5} and the same of k2,k6 and k3,k7, 64 bytes apart; a thread requests two steps before it converts
  // the first
  const bool quads = (p.K & 3) == 0;
  const int octs = p.slice * 4;
  for (int i0 = tid; i0 < 8 * octs; i0 += 2 * kMmaThreads) {
    float x[2][2][8];
    int r[2], oct[2];
#pragma unroll
    for (int s = 0; s < 2; s++) {
      const int i = i0 + s * kMmaThreads;
      r[s] = i / octs, oct[s] = i - r[s] * octs;
      const int k = b0 * 32 + oct[s] * 8;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int m = r[s] + 8 * h;
#pragma unroll
        for (int u = 0; u < 8; u++) x[s][h][u] = 0.f;
        if (r[s] < 8 && m < p.M) {
          const float *row = p.a + (size_t)m * p.K;
          if (quads && k + 8 <= p.K) {
            const float4 x0 = *(const float4 *)(row + k), x1 = *(const float4 *)(row + k + 4);
            x[s][h][0] = x0.x, x[s][h][1] = x0.y, x[s][h][2] = x0.z, x[s][h][3] = x0.w;
            x[s][h][4] = x1.x, x[s][h][5] = x1.y, x[s][h][6] = x1.z, x[s][h][7] = x1.w;
          } else {
#pragma unroll
            for (int u = 0; u < 8; u++)
              if (k + u < p.K) x[s][h][u] = row[k + u];
          }
        }
      }
    }
#pragma unroll
    for (int s = 0; s < 2; s++) {
      if (r[s] >= 8) break;
      __half2 hi[4][2], lo[4][2];  // [pair (k_u, k_u+4)][row r, row r + 8]
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          hi[u][h] = __floats2half2_rn(x[s][h][u], x[s][h][u + 4]);
          const float2 f = __half22float2(hi[u][h]);
          lo[u][h] = __floats2half2_rn(x[s][h][u] - f.x, x[s][h][u + 4] - f.y);
        }
      unsigned char *dst = ap + (size_t)r[s] * pitch + (oct[s] >> 2) * 128 + (oct[s] & 3) * 16;
      *(uint4 *)dst = *(const uint4 *)hi[0];
      *(uint4 *)(dst + 64) = *(const uint4 *)hi[2];
      if (HILO) {
        *(uint4 *)(dst + (size_t)8 * pitch) = *(const uint4 *)lo[0];
        *(uint4 *)(dst + (size_t)8 * pitch + 64) = *(const uint4 *)lo[2];
      }
    }
  }
  __syncthreads();
  if (slices > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");

  int pass = 0;
  for (int g0 = gfirst; g0 < gend; g0 += gall, pass++) {
    if (g0 > gfirst) fetch(g0), fetch_scales(g0);
    float acc[G][4];
#pragma unroll
    for (int g = 0; g < G; g++) {
      transpose4(w[g], lane);
#pragma unroll
      for (int c = 0; c < 4; c++) acc[g][c] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (i >= qn) break;  // warp-uniform
      const unsigned char *src = ap + (size_t)g4 * pitch + (quad * 4 + i) * 128 + j4 * 16;
      const uint4 h0 = *(const uint4 *)src, h1 = *(const uint4 *)(src + 64);
      uint4 l0, l1;
      if (HILO) l0 = *(const uint4 *)(src + (size_t)8 * pitch), l1 = *(const uint4 *)(src + (size_t)8 * pitch + 64);
#pragma unroll
      for (int g = 0; g < G; g++) {
        if (g0 + goff + g >= gend) break;
        const unsigned x = i == 0 ? w[g].x : (i == 1 ? w[g].y : (i == 2 ? w[g].z : w[g].w));
        const unsigned zz = 0x6400u + ((z4[g] >> (4 * i)) & 15u), z2 = zz | (zz << 16);  // 1024 + zp, twice
        uint32_t b[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const unsigned q = ((x >> (4 * u)) & 0x000F000Fu) | 0x64006400u;
          const __half2 d = __hsub2(*(const __half2 *)&q, *(const __half2 *)&z2);
          b[u] = *(const uint32_t *)&d;
        }
        float c[4];
        mma16816_f16_first(c, h0.x, h0.y, h0.z, h0.w, b[0], b[1]);
        mma16816_f16(c, h1.x, h1.y, h1.z, h1.w, b[2], b[3]);
        if (HILO) {
          mma16816_f16(c, l0.x, l0.y, l0.z, l0.w, b[0], b[1]);
          mma16816_f16(c, l1.x, l1.y, l1.z, l1.w, b[2], b[3]);
        }
        const float s0 = __shfl_sync(0xffffffffu, sc[g], j4 * 8 + i), s1 = __shfl_sync(0xffffffffu, sc[g], j4 * 8 + 4 + i);
        acc[g][0] = fmaf(s0, c[0], acc[g][0]), acc[g][1] = fmaf(s1, c[1], acc[g][1]);
        acc[g][2] = fmaf(s0, c[2], acc[g][2]), acc[g][3] = fmaf(s1, c[3], acc[g][3]);
      }
    }
    if (pass > 0) __syncthreads();  // the sums of the pass before have been read
#pragma unroll
    for (int g = 0; g < G; g++) red[(quad * gall + goff + g) * 32 + lane] = make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
    __syncthreads();
    // two buffers: a rank stores pass n + 2 only after the barrier of pass n + 1, which rank 0 reaches when it has read n
    float4 *buf = cred + (size_t)(pass & 1) * slices * gall * 32;
    auto store = [&](int e, const float4 &t) {  // e = group of the pass * 32 + lane of the accumulator tile
      const int g = g0 + (e >> 5), row = (e & 31) >> 2, n = g * 8 + (e & 3) * 2;
      if (g >= gend) return;
      if (row < p.M) *(float2 *)(p.y + (size_t)row * p.N + n) = make_float2(t.x, t.y);
      if (row + 8 < p.M) *(float2 *)(p.y + (size_t)(row + 8) * p.N + n) = make_float2(t.z, t.w);
    };
    for (int e = tid; e < gall * 32; e += kMmaThreads) {
      float4 t = red[e];
      for (int v = 1; v < (1 << p.lq); v++) {
        const float4 o = red[v * gall * 32 + e];
        t.x += o.x, t.y += o.y, t.z += o.z, t.w += o.w;
      }
      if (slices > 1) {
        uint32_t remote;
        const uint32_t local = (uint32_t)__cvta_generic_to_shared(buf + rank * gall * 32 + e);
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(0));
        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(remote), "f"(t.x), "f"(t.y), "f"(t.z), "f"(t.w) : "memory");
      } else {
        store(e, t);
      }
    }
    if (slices > 1) {
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      if (rank == 0)
        for (int e = tid; e < gall * 32; e += kMmaThreads) {
          float4 t = buf[e];
          for (int v = 1; v < slices; v++) {
            const float4 o = buf[v * gall * 32 + e];
            t.x += o.x, t.y += o.y, t.z += o.z, t.w += o.w;
          }
          store(e, t);
        }
    }
  }
}

size_t mma_smem(bool hilo, int G, int slice, int slices, int lq) {
  return (size_t)(hilo ? 2 : 1) * 8 * mma_row_pitch(slice) + (size_t)G * 32 * 16 * (kMmaWarps + (slices > 1 ? 2 * slices * (kMmaWarps >> lq) : 0));
}
// K slices (a power of two: clusters of 3 place badly) and blocks per slice, a multiple of 4.  Four slices from K = 2048 on:
// every block of the grid converts all rows of its K slice before it starts, so four times the columns on a quarter of K
// cost a quarter of that for one cluster hand-over (K = 2048, N = 8192 and back, 16 rows: 129.5 us in one slice per 2048,
// 127.6 us so, 121.1 us with whole A operands in shared memory).
void mma_slices(int nblk, int &slices, int &slice, int &lq) {
  slices = nblk >= kMmaSliceBlk ? kMmaMaxSlices : 1;
  slice = ceil_div(ceil_div(nblk, slices), 4) * 4;
  lq = slice > 32 ? 4 : (slice > 16 ? 3 : 2);
}

template <bool HILO, int G>
cudaError_t launch_mma(fa_ctx *ctx, cudaLaunchConfig_t &cfg, const MmaParams &p) {
  cfg.dynamicSmemBytes = mma_smem(HILO, G, p.slice, (int)cfg.gridDim.y, p.lq);
  static SmemLimit limit;
  const cudaError_t e = limit.raise(ctx, k_nbits_mma<HILO, G>, 227 * 1024);
  return e != cudaSuccess ? e : cudaLaunchKernelEx(&cfg, k_nbits_mma<HILO, G>, p);
}

}  // namespace

// int4 products with up to 16 activation rows on k_nbits_mma.  hilo: the rows enter as value + residue f16 planes.
bool fa_nbits_mma_ok(int M, int N, int K, int block_size) {
  return M >= 1 && M <= 16 && block_size == 32 && K >= 32 && K <= kMmaMaxSlices * kMmaSliceBlk * 32 && N >= 8 && (N & 7) == 0;
}

// Column groups per thread block: as many as leave one wave of blocks (clusters of K slices do not tile every GPC, so an eighth
// of the SMs is left out of the count there).
static int mma_groups(const fa_ctx *ctx, int N, int slices) {
  const int room = slices == 1 ? ctx->sm_count : ctx->sm_count * 7 / 8 / slices;
  return ceil_div(N / 8, room < 1 ? 1 : room);
}

// A block walks its column groups one after another, `pw` of them a warp (in steps of 2, 4 or 8 at a time), so the time grows
// with the columns; the product on the f16 copy of the weights reads four times the bytes, but at the tensor cores' and the
// HBM's rate.  12 rows, us, here / f16 copy:
//   K = 512   N = 8192 4.1 / 6.8, 16384 (pw 4) 6.0 / 6.5, 24576 (6) 9.1 / 8.7, 51200 18.2 / 11.9
//   K = 1024  N = 4096 4.9 / 7.2, 8192 (4) 6.4 / 8.9, 10240 (5) 9.0 / 7.6, 32768 20.2 / 13.6
//   K = 1536  N = 4096 6.7 / 8.7, 8192 (7) 9.6 / 10.3, 10240 (9) 12.9 / 9.5, 51200 49.4 / 28.0
//   K = 2048  N = 2048 5.2 / 12.5, 4096 (4) 7.5 / 9.5, 5120 (5) 10.9 / 10.2, 8192 (8) 12.8 / 11.4, 10240 20.1 / 11.0, 51200 79.5 / 36.0
//   K = 2560  N = 2048 (4) 7.2 / 13.2, 2560 (5) 10.1 / 8.9, 4096 (8) 11.3 / 10.1, 6144 (12) 18.7 / 11.4
//   K = 4096  N = 2048 (4) 7.6 / 16.3, 2560 (5) 10.4 / 10.1, 4096 (8) 12.1 / 11.8, 5120 17.5 / 13.5
//   K = 5120  N = 2048 (8) 10.7 / 17.2, 2304 (9) 13.9 / 17.5, 2560 (10) 14.6 / 11.0
//   K = 8192  N = 1536 (6) 11.6 / 11.4, 2048 (8) 13.6 / 19.9, 2304 (9) 17.2 / 20.1, 2560 (10) 18.1 / 13.3, 4096 23.8 / 16.4
// On one slice of K: four groups a warp where warps share a quad, one pass of eight where none do.  With K over a cluster: the same
// one pass of eight, and on up to 4096 of K as many groups as stay within a quarter of the copy's time or near it, for the sake
// of the weights, which the copy rounds to f16 (4e-4 of a result against 4e-7 here).  And up to two passes where the copy's
// product splits K over clusters of eight that are not all resident at once (13 to 18 column tiles).
bool fa_nbits_mma_worth(fa_ctx *ctx, int N, int K) {
  int slices, slice, lq;
  mma_slices(ceil_div(K, 32), slices, slice, lq);
  const int gper = mma_groups(ctx, N, slices), gw = kMmaWarps >> lq, pw = ceil_div(gper, gw);
  if (slices == 1) return pw <= (gw == 1 ? 8 : 4);
  const int eighths = ceil_div(N, 128) * 8, chunks = ceil_div(K, 64);
  if (eighths > ctx->sm_count * 2 / 3 && eighths <= ctx->sm_count && 7 * ceil_div(chunks, 8) < chunks) return pw <= 16;
  return gw == 1 ? pw <= 8 : gper * slice <= (gw == 4 ? 512 : 420);
}

int fa_nbits_mma(fa_ctx *ctx, const float *a, const uint8_t *bq, const float *scales, const uint8_t *zp, float *y, int M, int N,
                 int K, int nblk, int zpb, bool hilo) {
  MmaParams p{a, bq, scales, zp, y, M, N, K, nblk, zpb, 0, 0, 0};
  int slices;
  mma_slices(nblk, slices, p.slice, p.lq);
  const int gw = kMmaWarps >> p.lq;  // warps that share a quad's columns
  const int groups = N / 8;
  p.gper = mma_groups(ctx, N, slices);  // walked 8, 4 or 2 at a time by each of the gw warps of a quad
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(ceil_div(groups, p.gper), slices);
  cfg.blockDim = dim3(kMmaThreads);
  cfg.stream = ctx->stream;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see fa_launch_dep
  attr[0].val.programmaticStreamSerializationAllowed = ctx->pdl ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = slices;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = slices > 1 ? 2 : 1;
  cudaError_t e;
  {
    LaunchScope ls(ctx, "nbits_mma");
    if (p.gper <= 2 * gw) e = hilo ? launch_mma<true, 2>(ctx, cfg, p) : launch_mma<false, 2>(ctx, cfg, p);
    else if (p.gper <= 4 * gw) e = hilo ? launch_mma<true, 4>(ctx, cfg, p) : launch_mma<false, 4>(ctx, cfg, p);
    else e = hilo ? launch_mma<true, 8>(ctx, cfg, p) : launch_mma<false, 8>(ctx, cfg, p);
  }
  if (e != cudaSuccess) return fa_fail(ctx, FA_ERR_CUDA, "launch nbits_mma: %s", cudaGetErrorString(e));
  return FA_OK;
}

// N-contiguous weights: one activation row only.  From two rows on, the tensor-core kernel (which shares each
// weight tile between all rows for free) is at least as fast as this one; measured on 1280 x 1280 f16 at
// M = 4: 10.6 us here against 7.3 us there.
bool fa_gemv_kn_ok(int M, int N, int K) { return M == 1 && K >= 1 && N >= 4 && (N & 3) == 0; }

// The layernorm prologue holds the row in registers and a K slice of it in shared memory, in whole quads.
bool fa_gemv_kn_norm_ok(int K) { return K >= 4 && (K & 3) == 0 && K <= kKnNormMax; }

// w: f16 [K][N] (i8 = false) or int8 [K][N]; y = act(acc * colscale[n] + bias[n]) + add[n]; gamma != NULL: layernorm first.
int fa_gemv_kn(fa_ctx *ctx, const float *x, const float *gamma, const float *beta, float eps, const void *w, bool i8,
               const float *colscale, const float *bias, int act, const float *add, float *y, int N, int K) {
  KnParams p{x, gamma, beta, w, y, K, N, 0, eps, GemvEp{colscale, bias, add, act}};
  // K slices = ranks of a cluster, as many (1, 2, 4, 8) as leave at most four blocks per SM and 64 rows to each; the layernorm
  // form needs its slice in shared memory whole.  More blocks than are resident start in a second wave, clusters last (int8
  // 1280 x 30724: 482 blocks 12.1 us, 964 15.9, 241 16.2), and blocks that leave an SM with one of them run at half its rate.
  const bool narrow = ceil_div(N, kKnCols) * 8 < ctx->sm_count;
  const int strips = ceil_div(N, narrow ? kKnCols / 2 : kKnCols);
  int ks = 1;
  while (ks < 8 && (long long)strips * ks * 2 <= 4ll * ctx->sm_count && K >= 64 * ks * 2) ks *= 2;
  while (gamma && ks < 8 && ceil_div(K, ks) > kKnSlice) ks *= 2;
  p.kslice = (ceil_div(K, ks) + 7) / 8 * 8;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(strips, ks);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = ctx->stream;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see fa_launch_dep
  attr[0].val.programmaticStreamSerializationAllowed = ctx->pdl ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = ks;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ks > 1 ? 2 : 1;
  cudaError_t e;
  {
    LaunchScope ls(ctx, i8 ? "gemv_i8" : "gemv_f16");
    // three resident blocks leave the registers for all loads of both batches, four are needed from 3 x the SMs on: int8 1280 x
    // 51868 (406 blocks) 15.7 us at three, 19.0 at four; 1280 x 30724 (482 blocks) 16.0 and 12.1
    const bool four = !gamma && !narrow && (long long)strips * ks > 3ll * ctx->sm_count;
    const bool shallow = p.kslice <= 2 * 8 * (narrow ? 16 : 8);  // two batches of 8 cover the slice
    auto form = [&](auto i8_tag, auto u_tag, auto blocks_tag) {
      constexpr bool I8 = decltype(i8_tag)::value;
      constexpr int U = decltype(u_tag)::value, BL = decltype(blocks_tag)::value;
      return gamma ? (narrow ? k_gemv_kn<I8, true, 64, U, BL> : k_gemv_kn<I8, true, 128, U, BL>)
                   : (narrow ? k_gemv_kn<I8, false, 64, U, BL> : k_gemv_kn<I8, false, 128, U, BL>);
    };
    using True = std::true_type;
    using False = std::false_type;
    using Eight = std::integral_constant<int, 8>;
    using Sixteen = std::integral_constant<int, 16>;
    using Three = std::integral_constant<int, 3>;
    using Four = std::integral_constant<int, 4>;
    auto kern = i8 ? (shallow ? form(True{}, Eight{}, Four{}) : (four ? k_gemv_kn<true, false, 128, 16, 4> : form(True{}, Sixteen{}, Three{})))
                   : (four ? k_gemv_kn<false, false, 128, 8, 4> : form(False{}, Eight{}, Three{}));
    e = cudaLaunchKernelEx(&cfg, kern, p);
  }
  if (e != cudaSuccess) return fa_fail(ctx, FA_ERR_CUDA, "launch gemv_kn: %s", cudaGetErrorString(e));
  return FA_OK;
}
