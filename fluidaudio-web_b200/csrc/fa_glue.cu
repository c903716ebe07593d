// Glue ops the encoder/decoder forwards call between GEMMs.  Each follows the arithmetic of the
// reference's CPU twin (src/gpu/wasm-context.js:308-685) and the grid shape idea of its WGSL kernel
// (src/gpu/kernels/{normalization,attention,convolution,tensor-ops}.js); all are f32.
#include "fa_internal.cuh"

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// One CTA (256 threads) per row; two-pass mean/variance (wasm-context.js:308-326).
__global__ void __launch_bounds__(256) k_layernorm(const float *__restrict__ x, const float *__restrict__ g,
                                                   const float *__restrict__ b, float *__restrict__ y,
                                                   __half *__restrict__ y16, int R, int C, float eps) {
  fa_grid_dep_sync();
  __shared__ float red[8];
  __shared__ float stat;
  for (int r = blockIdx.x; r < R; r += gridDim.x) {
    const float *row = x + (size_t)r * C;
    float s = 0.f;
    for (int j = threadIdx.x; j < C; j += 256) s += row[j];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      float t = 0.f;
      for (int w = 0; w < 8; w++) t += red[w];
      stat = t / (float)C;
    }
    __syncthreads();
    const float mean = stat;
    float v = 0.f;
    for (int j = threadIdx.x; j < C; j += 256) {
      float d = row[j] - mean;
      v += d * d;
    }
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      float t = 0.f;
      for (int w = 0; w < 8; w++) t += red[w];
      stat = 1.0f / sqrtf(t / (float)C + eps);
    }
    __syncthreads();
    const float inv = stat;
    for (int j = threadIdx.x; j < C; j += 256) {
      const float o = (row[j] - mean) * inv * g[j] + b[j];
      y[(size_t)r * C + j] = o;
      // normalised rows feed linear layers: also emit them as the packed f16 row operand Ap[j/64][r][j%64]
      if (y16) y16[((size_t)(j >> 6) * R + r) * 64 + (j & 63)] = __float2half_rn(o);
    }
    __syncthreads();
  }
}

// Row held in registers (C % 4 == 0, C <= 4096): one global read, one write.  Same two-pass
// mean / variance arithmetic as above.
template <int V4>  // float4 per thread
__global__ void __launch_bounds__(256) k_layernorm_reg(const float *__restrict__ x, const float *__restrict__ g,
                                                       const float *__restrict__ b, float *__restrict__ y,
                                                       __half *__restrict__ y16, size_t lo_off, int R, int C,
                                                       float eps) {
  fa_grid_dep_sync();
  __shared__ float red[8];
  __shared__ float stat;
  const int r = blockIdx.x, c4 = C >> 2;
  const float4 *row = (const float4 *)(x + (size_t)r * C);
  float4 v[V4];
  float s = 0.f;
#pragma unroll
  for (int u = 0; u < V4; u++) {
    const int q = threadIdx.x + u * 256;
    v[u] = q < c4 ? row[q] : make_float4(0.f, 0.f, 0.f, 0.f);
    s += (v[u].x + v[u].y) + (v[u].z + v[u].w);
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < 8; w++) t += red[w];
    stat = t / (float)C;
  }
  __syncthreads();
  const float mean = stat;
  float vs = 0.f;
#pragma unroll
  for (int u = 0; u < V4; u++) {
    const int q = threadIdx.x + u * 256;
    if (q < c4) {
      const float a = v[u].x - mean, bb = v[u].y - mean, c = v[u].z - mean, d = v[u].w - mean;
      vs += (a * a + bb * bb) + (c * c + d * d);
    }
  }
  vs = warp_sum(vs);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = vs;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < 8; w++) t += red[w];
    stat = 1.0f / sqrtf(t / (float)C + eps);
  }
  __syncthreads();
  const float inv = stat;
#pragma unroll
  for (int u = 0; u < V4; u++) {
    const int q = threadIdx.x + u * 256;
    if (q < c4) {
      const float4 gg = ((const float4 *)g)[q], bb = ((const float4 *)b)[q];
      float4 o;
      o.x = (v[u].x - mean) * inv * gg.x + bb.x;
      o.y = (v[u].y - mean) * inv * gg.y + bb.y;
      o.z = (v[u].z - mean) * inv * gg.z + bb.z;
      o.w = (v[u].w - mean) * inv * gg.w + bb.w;
      ((float4 *)(y + (size_t)r * C))[q] = o;
      if (y16) {
        const int j = q * 4;
        __half2 *d16 = (__half2 *)(y16 + ((size_t)(j >> 6) * R + r) * 64 + (j & 63));
        const __half2 h0 = __floats2half2_rn(o.x, o.y), h1 = __floats2half2_rn(o.z, o.w);
        d16[0] = h0;
        d16[1] = h1;
        if (lo_off) {  // second plane: what the f16 rounding dropped
          const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
          __half2 *l16 = (__half2 *)((__half *)d16 + lo_off);
          l16[0] = __floats2half2_rn(o.x - f0.x, o.y - f0.y);
          l16[1] = __floats2half2_rn(o.z - f1.x, o.w - f1.y);
        }
      }
    }
  }
}

// One warp per row (C % 4 == 0, C <= 1024): the row lives in the warp's registers, both reductions are
// shuffles, no block barrier; 8 rows per CTA.  Same two-pass mean / variance arithmetic as above.
// EARLY: gamma and beta are requested together with the row instead of after the two reductions.  That costs V4 * 8
// registers and with them resident blocks, so it is for the launches that do not fill the GPU anyway (few rows), where the
// kernel is nothing but its chain of latencies.  Measured: 512 x 1024 6.1 -> 4.1 us, 937 x 1024 6.7 -> 4.6 us.
template <int V4, bool EARLY>  // float4 per lane: C <= 128 * V4
__global__ void __launch_bounds__(256) k_layernorm_warp(const float *__restrict__ x, const float *__restrict__ g,
                                                        const float *__restrict__ b, float *__restrict__ y,
                                                        __half *__restrict__ y16, size_t lo_off, int R, int C, float eps) {
  fa_grid_dep_sync();
  const int lane = threadIdx.x & 31, r = blockIdx.x * 8 + (threadIdx.x >> 5), c4 = C >> 2;
  if (r >= R) return;
  const float4 *row = (const float4 *)(x + (size_t)r * C);
  float4 v[V4];
  float s = 0.f;
#pragma unroll
  for (int u = 0; u < V4; u++) {
    const int q = lane + u * 32;
    v[u] = q < c4 ? row[q] : make_float4(0.f, 0.f, 0.f, 0.f);
    s += (v[u].x + v[u].y) + (v[u].z + v[u].w);
  }
  float4 ge[EARLY ? V4 : 1], be[EARLY ? V4 : 1];
  if (EARLY) {
#pragma unroll
    for (int u = 0; u < V4; u++) {
      const int q = lane + u * 32;
      if (q < c4) ge[u] = ((const float4 *)g)[q], be[u] = ((const float4 *)b)[q];
    }
  }
  const float mean = warp_sum(s) / (float)C;
  float vs = 0.f;
#pragma unroll
  for (int u = 0; u < V4; u++) {
    if (lane + u * 32 < c4) {
      const float a = v[u].x - mean, bb = v[u].y - mean, c = v[u].z - mean, d = v[u].w - mean;
      vs += (a * a + bb * bb) + (c * c + d * d);
    }
  }
  const float inv = 1.0f / sqrtf(warp_sum(vs) / (float)C + eps);
#pragma unroll
  for (int u = 0; u < V4; u++) {
    const int q = lane + u * 32;
    if (q < c4) {
      const float4 gg = EARLY ? ge[EARLY ? u : 0] : ((const float4 *)g)[q], bb = EARLY ? be[EARLY ? u : 0] : ((const float4 *)b)[q];
      float4 o;
      o.x = (v[u].x - mean) * inv * gg.x + bb.x;
      o.y = (v[u].y - mean) * inv * gg.y + bb.y;
      o.z = (v[u].z - mean) * inv * gg.z + bb.z;
      o.w = (v[u].w - mean) * inv * gg.w + bb.w;
      if (y) ((float4 *)(y + (size_t)r * C))[q] = o;  // y == nullptr: the result exists only as the packed operand
      if (y16) {
        const int j = q * 4;
        __half2 *d16 = (__half2 *)(y16 + ((size_t)(j >> 6) * R + r) * 64 + (j & 63));
        const __half2 h0 = __floats2half2_rn(o.x, o.y), h1 = __floats2half2_rn(o.z, o.w);
        d16[0] = h0;
        d16[1] = h1;
        if (lo_off) {
          const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
          __half2 *l16 = (__half2 *)((__half *)d16 + lo_off);
          l16[0] = __floats2half2_rn(o.x - f0.x, o.y - f0.y);
          l16[1] = __floats2half2_rn(o.z - f1.x, o.w - f1.y);
        }
      }
    }
  }
}

// Two layernorms back to back on the same rows (the last one of a conformer block, then the first of the next
// block, which only feeds a product): y = LN1(x) leaves as f32, z = LN2(y) as the packed f16 row operand alone.
// The row never leaves the warp's registers in between, so z is bit-identical to layernorm of the stored y.
// EARLY as in k_layernorm_warp, for both layernorms' gamma and beta.  Measured: 804 x 1024 in
// an encoder pass 11.3 us a block before; six windows of 134 frames 3.51 -> 3.38 ms a pass.
template <int V4, bool EARLY>
__global__ void __launch_bounds__(256) k_layernorm_chain(const float *__restrict__ x, const float *__restrict__ g1,
                                                         const float *__restrict__ b1, const float *__restrict__ g2,
                                                         const float *__restrict__ b2, float *__restrict__ y,
                                                         __half *__restrict__ z16, int R, int C, float eps) {
  fa_grid_dep_sync();
  const int lane = threadIdx.x & 31, r = blockIdx.x * 8 + (threadIdx.x >> 5), c4 = C >> 2;
  if (r >= R) return;
  const float4 *row = (const float4 *)(x + (size_t)r * C);
  float4 v[V4];
#pragma unroll
  for (int u = 0; u < V4; u++) {
    const int q = lane + u * 32;
    v[u] = q < c4 ? row[q] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float4 ge[2][EARLY ? V4 : 1], be[2][EARLY ? V4 : 1];
  if (EARLY) {
#pragma unroll
    for (int pass = 0; pass < 2; pass++)
#pragma unroll
      for (int u = 0; u < V4; u++) {
        const int q = lane + u * 32;
        if (q < c4) ge[pass][u] = ((const float4 *)(pass ? g2 : g1))[q], be[pass][u] = ((const float4 *)(pass ? b2 : b1))[q];
      }
  }
#pragma unroll
  for (int pass = 0; pass < 2; pass++) {
    const float *g = pass ? g2 : g1, *b = pass ? b2 : b1;
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < V4; u++) s += (v[u].x + v[u].y) + (v[u].z + v[u].w);  // (lanes past the row hold zeros)
    const float mean = warp_sum(s) / (float)C;
    float vs = 0.f;
#pragma unroll
    for (int u = 0; u < V4; u++) {
      if (lane + u * 32 < c4) {
        const float a = v[u].x - mean, bb = v[u].y - mean, c = v[u].z - mean, d = v[u].w - mean;
        vs += (a * a + bb * bb) + (c * c + d * d);
      }
    }
    const float inv = 1.0f / sqrtf(warp_sum(vs) / (float)C + eps);
#pragma unroll
    for (int u = 0; u < V4; u++) {
      const int q = lane + u * 32;
      if (q < c4) {
        const float4 gg = EARLY ? ge[pass][EARLY ? u : 0] : ((const float4 *)g)[q], bb = EARLY ? be[pass][EARLY ? u : 0] : ((const float4 *)b)[q];
        float4 o;
        o.x = (v[u].x - mean) * inv * gg.x + bb.x;
        o.y = (v[u].y - mean) * inv * gg.y + bb.y;
        o.z = (v[u].z - mean) * inv * gg.z + bb.z;
        o.w = (v[u].w - mean) * inv * gg.w + bb.w;
        v[u] = o;
        if (pass == 0) {
          ((float4 *)(y + (size_t)r * C))[q] = o;
        } else {
          const int j = q * 4;
          __half2 *d16 = (__half2 *)(z16 + ((size_t)(j >> 6) * R + r) * 64 + (j & 63));
          d16[0] = __floats2half2_rn(o.x, o.y);
          d16[1] = __floats2half2_rn(o.z, o.w);
        }
      }
    }
  }
}

// One warp per row (wasm-context.js:327-343).
__global__ void k_softmax(const float *__restrict__ x, float *__restrict__ y, int R, int C) {
  fa_grid_dep_sync();
  const int warps = (blockDim.x >> 5);
  const int lane = threadIdx.x & 31;
  for (int r = blockIdx.x * warps + (threadIdx.x >> 5); r < R; r += gridDim.x * warps) {
    const float *row = x + (size_t)r * C;
    float mx = -INFINITY;
    for (int j = lane; j < C; j += 32) mx = fmaxf(mx, row[j]);
    mx = warp_max(mx);
    float s = 0.f;
    for (int j = lane; j < C; j += 32) s += expf(row[j] - mx);
    s = warp_sum(s);
    const float inv = 1.0f / s;
    for (int j = lane; j < C; j += 32) y[(size_t)r * C + j] = expf(row[j] - mx) * inv;
  }
}

// Rows of up to 256 columns: the row lives in registers (8 values per lane), one read and one write.
__global__ void k_softmax_reg(const float *__restrict__ x, float *__restrict__ y, int R, int C) {
  fa_grid_dep_sync();
  const int warps = blockDim.x >> 5, lane = threadIdx.x & 31;
  for (int r = blockIdx.x * warps + (threadIdx.x >> 5); r < R; r += gridDim.x * warps) {
    const float *row = x + (size_t)r * C;
    float v[8];
    float mx = -INFINITY;
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int j = lane + 32 * u;
      v[u] = j < C ? row[j] : -INFINITY;
      mx = fmaxf(mx, v[u]);
    }
    mx = warp_max(mx);
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < 8; u++) {
      v[u] = lane + 32 * u < C ? expf(v[u] - mx) : 0.f;
      s += v[u];
    }
    s = warp_sum(s);
    const float inv = 1.0f / s;
#pragma unroll
    for (int u = 0; u < 8; u++)
      if (lane + 32 * u < C) y[(size_t)r * C + lane + 32 * u] = v[u] * inv;
  }
}

// float4 forms of the elementwise family (n % 4 == 0, 16-byte aligned operands)
__global__ void k_ewise4(const float4 *__restrict__ a, const float4 *__restrict__ b, float4 *__restrict__ y, unsigned n4,
                         int mul) {
  fa_grid_dep_sync();
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += gridDim.x * blockDim.x) {
    const float4 p = a[i], q = b[i];
    y[i] = mul ? make_float4(p.x * q.x, p.y * q.y, p.z * q.z, p.w * q.w) : make_float4(p.x + q.x, p.y + q.y, p.z + q.z, p.w + q.w);
  }
}
__global__ void k_glu4(const float4 *__restrict__ x, float4 *__restrict__ y, unsigned n4) {
  fa_grid_dep_sync();
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += gridDim.x * blockDim.x) {
    const float4 p = x[i], q = x[i + n4];
    y[i] = make_float4(p.x * (1.0f / (1.0f + expf(-q.x))), p.y * (1.0f / (1.0f + expf(-q.y))),
                       p.z * (1.0f / (1.0f + expf(-q.z))), p.w * (1.0f / (1.0f + expf(-q.w))));
  }
}

__global__ void k_ewise(const float *__restrict__ a, const float *__restrict__ b, float *__restrict__ y, size_t n, int C,
                        int bcast, int mul) {
  fa_grid_dep_sync();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    float bv = bcast ? b[i % C] : b[i];
    y[i] = mul ? a[i] * bv : a[i] + bv;
  }
}
__global__ void k_scale(const float *__restrict__ x, float *__restrict__ y, size_t n, float s) {
  fa_grid_dep_sync();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = x[i] * s;
}
__global__ void k_unary(const float *__restrict__ x, float *__restrict__ y, size_t n, int act) {
  fa_grid_dep_sync();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = fa_actf(x[i], act);
}
// x[2C,T] -> x[c,t] * sigmoid(x[c+C,t]) (wasm-context.js:428-434)
__global__ void k_glu(const float *__restrict__ x, float *__restrict__ y, int C, int T) {
  fa_grid_dep_sync();
  size_t n = (size_t)C * T;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = x[i] * (1.0f / (1.0f + expf(-x[i + n])));
}
__global__ void k_transpose(const float *__restrict__ x, float *__restrict__ y, int R, int C) {
  fa_grid_dep_sync();
  __shared__ float t[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    int r = r0 + i, c = c0 + threadIdx.x;
    if (r < R && c < C) t[i][threadIdx.x] = x[(size_t)r * C + c];
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    int c = c0 + i, r = r0 + threadIdx.x;
    if (r < R && c < C) y[(size_t)c * R + r] = t[threadIdx.x][i];
  }
}
// dst[r, dcol0 + j] = src[r, scol0 + j] for j < width
__global__ void k_copy_cols(const float *__restrict__ src, int scols, int scol0, float *__restrict__ dst, int dcols,
                            int dcol0, int rows, int width) {
  fa_grid_dep_sync();
  size_t n = (size_t)rows * width;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    int r = (int)(i / width), j = (int)(i % width);
    dst[(size_t)r * dcols + dcol0 + j] = src[(size_t)r * scols + scol0 + j];
  }
}
// [C, Tsub*F] -> [Tsub, C*F] (wasm-context.js:552-563)
// blockIdx.y = window: window b reads x + b*xstride and writes rows [b*Tsub, (b+1)*Tsub).
__global__ void k_sub_reshape(const float *__restrict__ x, float *__restrict__ y, int C, int Tsub, int F, size_t xstride) {
  fa_grid_dep_sync();
  size_t n = (size_t)Tsub * C * F;
  int CF = C * F;
  x += (size_t)blockIdx.y * xstride;
  y += (size_t)blockIdx.y * n;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    int ho = (int)(i / CF), rem = (int)(i % CF), c = rem / F, wo = rem % F;
    y[i] = x[(size_t)c * Tsub * F + (size_t)ho * F + wo];
  }
}
// The same move four columns at a time (F % 4 == 0), also emitting the result as the packed f16 row operand
// Ap[k/64][m][k%64] of the product that follows (m = window*Tsub + frame, k = c*F + f); y may be NULL when only
// that operand is wanted.  Thread = one float4 of one output row; consecutive threads walk the output row.
__global__ void __launch_bounds__(256) k_sub_reshape4(const float *__restrict__ x, float *__restrict__ y,
                                                      __half *__restrict__ y16, int C, int Tsub, int F, size_t xstride,
                                                      int rows) {
  fa_grid_dep_sync();
  const int CF4 = (C * F) >> 2, F4 = F >> 2;
  const int m = blockIdx.y, wdw = m / Tsub, ho = m - wdw * Tsub;
  const float *xw = x + (size_t)wdw * xstride + (size_t)ho * F;
  for (int q = blockIdx.x * 256 + threadIdx.x; q < CF4; q += gridDim.x * 256) {
    const int c = q / F4, f4 = q - c * F4;
    const float4 v = __ldg((const float4 *)(xw + (size_t)c * Tsub * F) + f4);
    if (y) ((float4 *)(y + (size_t)m * C * F))[q] = v;
    if (y16) {
      const int k = q * 4;
      const __half2 h0 = __floats2half2_rn(v.x, v.y), h1 = __floats2half2_rn(v.z, v.w);
      uint2 o;
      o.x = *(const uint32_t *)&h0;
      o.y = *(const uint32_t *)&h1;
      *(uint2 *)(y16 + ((size_t)(k >> 6) * rows + m) * 64 + (k & 63)) = o;
    }
  }
}

// Batched rel_shift (wasm-context.js:525-538): x[H*t, 2t-1] -> [H*t, t].  With f = t + i*(2t-1) + j the
// reference reads row f / 2t, column f % 2t - 1; for 0 <= i, j < t that is row i, column t-1-i+j (never
// the zero column), so every output row is one contiguous run of its input row.
__global__ void k_rel_shift_b(const float *__restrict__ x, float *__restrict__ y, int rows, int t) {
  fa_grid_dep_sync();
  const int p = 2 * t - 1;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const int i = r % t;
    const float *src = x + (size_t)r * p + (t - 1 - i);
    float *dst = y + (size_t)r * t;
    for (int j = threadIdx.x; j < t; j += blockDim.x) dst[j] = src[j];
  }
}

// Batched QK^T (wasm-context.js:462-482): one (w,h) per blockIdx.z, 64x64 output tile per CTA,
// 4x4 outputs per thread, HD consumed in slices of 16 through shared memory.
// out[((w*H+h)*T+i)*Tb + j] = sum_d (q[(w*T+i)*S + h*HD + d] + qb[h*HD+d]) * b[brow(j)*S + h*HD + d]
__global__ void __launch_bounds__(256) k_bmm_qk(const float *__restrict__ q, const float *__restrict__ b,
                                                const float *__restrict__ qb, float *__restrict__ out, int T, int Tb,
                                                int H, int HD, int bShared) {
  fa_grid_dep_sync();
  __shared__ __align__(16) float Qs[16][68], Bs[16][68];
  const int w = blockIdx.z / H, h = blockIdx.z % H, S = H * HD;
  const int i0 = blockIdx.y * 64, j0 = blockIdx.x * 64;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const float *qbase = q + (size_t)w * T * S + h * HD;
  const float *bbase = b + (size_t)(bShared ? 0 : w) * Tb * S + h * HD;
  float acc[4][4] = {};
  for (int d0 = 0; d0 < HD; d0 += 16) {
#pragma unroll
    for (int s = 0; s < 4; s++) {
      const int e = threadIdx.x + 256 * s, r = e >> 4, dd = e & 15, d = d0 + dd;
      float qv = 0.f, bv = 0.f;
      if (d < HD) {
        if (i0 + r < T) qv = qbase[(size_t)(i0 + r) * S + d] + (qb ? qb[h * HD + d] : 0.f);
        if (j0 + r < Tb) bv = bbase[(size_t)(j0 + r) * S + d];
      }
      Qs[dd][r] = qv;
      Bs[dd][r] = bv;
    }
    __syncthreads();
#pragma unroll
    for (int d = 0; d < 16; d++) {
      const float4 a4 = *(const float4 *)&Qs[d][ty * 4];
      const float4 b4 = *(const float4 *)&Bs[d][tx * 4];
      const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) acc[u][v] = fmaf(av[u], bv[v], acc[u][v]);
    }
    __syncthreads();
  }
  float *obase = out + ((size_t)w * H + h) * T * Tb;
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int i = i0 + ty * 4 + u;
    if (i >= T) continue;
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const int j = j0 + tx * 4 + v;
      if (j < Tb) obase[(size_t)i * Tb + j] = acc[u][v];
    }
  }
}

// Single-query forms of the two attention products (token-by-token decoding: T = 1 per window).  Both are
// streams over the key / value cache, so they are laid out for full-line loads: a warp owns 128 consecutive
// columns (32 lanes x float4) of one cache row at a time, 8 warps take rows round-robin, U rows in flight each.
// LPH = lanes per head = HD / 4 (a power of two <= 32).
template <int U>
__global__ void __launch_bounds__(256) k_bmm_qk_t1(const float *__restrict__ q, const float *__restrict__ b,
                                                    const float *__restrict__ qb, float *__restrict__ out, int Tb, int H,
                                                    int HD, int bShared, int lph) {
  fa_grid_dep_sync();
  const int S = H * HD, w = blockIdx.z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 128 + lane * 4;
  const bool live = c < S;
  float4 qv = make_float4(0.f, 0.f, 0.f, 0.f);
  if (live) {
    qv = *(const float4 *)(q + (size_t)w * S + c);
    if (qb) {
      const float4 t = *(const float4 *)(qb + c);
      qv.x += t.x, qv.y += t.y, qv.z += t.z, qv.w += t.w;
    }
  }
  const float *bbase = b + (size_t)(bShared ? 0 : w) * Tb * S + (live ? c : 0);
  const int h = (live ? c : 0) / HD;
  float *orow = out + ((size_t)w * H + h) * Tb;
  const bool writer = live && (lane & (lph - 1)) == 0;
  const bool vec = (Tb & 3) == 0 && (((uintptr_t)out) & 15) == 0;
  const int jstep = gridDim.y * 8 * U;
  for (int j0 = (blockIdx.y * 8 + warp) * U; j0 < Tb; j0 += jstep) {
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int j = j0 + u < Tb ? j0 + u : Tb - 1;
      v[u] = __ldcs((const float4 *)(bbase + (size_t)j * S));
    }
    float d[U];
#pragma unroll
    for (int u = 0; u < U; u++) d[u] = fmaf(qv.x, v[u].x, fmaf(qv.y, v[u].y, fmaf(qv.z, v[u].z, qv.w * v[u].w)));
    for (int o = lph >> 1; o > 0; o >>= 1) {
#pragma unroll
      for (int u = 0; u < U; u++) d[u] += __shfl_xor_sync(0xffffffffu, d[u], o);
    }
    if (writer) {
      if (vec && j0 + U <= Tb) {  // U consecutive scores of one head: whole 16-byte stores
#pragma unroll
        for (int u = 0; u < U; u += 4) *(float4 *)(orow + j0 + u) = make_float4(d[u], d[u + 1], d[u + 2], d[u + 3]);
      } else {
#pragma unroll
        for (int u = 0; u < U; u++)
          if (j0 + u < Tb) orow[j0 + u] = d[u];
      }
    }
  }
}

template <int U>
__global__ void __launch_bounds__(256) k_bmm_pv_t1(const float *__restrict__ p, const float *__restrict__ v,
                                                    float *__restrict__ out, __half *__restrict__ y16, size_t lo_off,
                                                    int Tk, int H, int HD) {
  fa_grid_dep_sync();
  __shared__ float4 part[8][32];
  const int S = H * HD, w = blockIdx.z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 128 + lane * 4;
  const bool live = c < S;
  const int cc = live ? c : 0, h = cc / HD;
  const float *prow = p + ((size_t)w * H + h) * Tk;
  const float *vbase = v + (size_t)w * Tk * S + cc;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j0 = warp * U; j0 < Tk; j0 += 8 * U) {
    float4 x[U];
    float pr[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int j = j0 + u < Tk ? j0 + u : Tk - 1;
      x[u] = __ldcs((const float4 *)(vbase + (size_t)j * S));
      pr[u] = j0 + u < Tk ? prow[j] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      acc.x = fmaf(pr[u], x[u].x, acc.x);
      acc.y = fmaf(pr[u], x[u].y, acc.y);
      acc.z = fmaf(pr[u], x[u].z, acc.z);
      acc.w = fmaf(pr[u], x[u].w, acc.w);
    }
  }
  part[warp][lane] = acc;
  __syncthreads();
  if (warp == 0 && live) {
    float4 t = part[0][lane];
#pragma unroll
    for (int i = 1; i < 8; i++) {
      const float4 o = part[i][lane];
      t.x += o.x, t.y += o.y, t.z += o.z, t.w += o.w;
    }
    *(float4 *)(out + (size_t)w * S + c) = t;
    if (y16) {  // packed f16 row operand of the product that follows (value plane, then residue plane)
      __half2 *d16 = (__half2 *)(y16 + ((size_t)(c >> 6) * gridDim.z + w) * 64 + (c & 63));
      const __half2 h0 = __floats2half2_rn(t.x, t.y), h1 = __floats2half2_rn(t.z, t.w);
      d16[0] = h0;
      d16[1] = h1;
      if (lo_off) {
        const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
        __half2 *l16 = (__half2 *)((__half *)d16 + lo_off);
        l16[0] = __floats2half2_rn(t.x - f0.x, t.y - f0.y);
        l16[1] = __floats2half2_rn(t.z - f1.x, t.w - f1.y);
      }
    }
  }
}

// Batched P@V (wasm-context.js:484-500), 64 (rows i) x 64 (head dims d) per CTA, keys in slices of 16:
// out[(w*Tq+i)*S + h*HD + d] = sum_j p[((w*H+h)*Tq+i)*Tk + j] * v[(w*Tk+j)*S + h*HD + d]
__global__ void __launch_bounds__(256) k_bmm_pv(const float *__restrict__ p, const float *__restrict__ v,
                                                float *__restrict__ out, int Tq, int Tk, int H, int HD) {
  fa_grid_dep_sync();
  __shared__ __align__(16) float Ps[16][68], Vs[16][68];
  const int w = blockIdx.z / H, h = blockIdx.z % H, S = H * HD;
  const int i0 = blockIdx.y * 64, d0 = blockIdx.x * 64;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const float *pbase = p + ((size_t)w * H + h) * Tq * Tk;
  const float *vbase = v + (size_t)w * Tk * S + h * HD;
  float acc[4][4] = {};
  for (int j0 = 0; j0 < Tk; j0 += 16) {
#pragma unroll
    for (int s = 0; s < 4; s++) {
      const int e = threadIdx.x + 256 * s;
      {  // P tile: 64 rows x 16 keys, keys fastest in memory
        const int r = e >> 4, jj = e & 15;
        Ps[jj][r] = (i0 + r < Tq && j0 + jj < Tk) ? pbase[(size_t)(i0 + r) * Tk + j0 + jj] : 0.f;
      }
      {  // V tile: 16 keys x 64 dims, dims fastest in memory
        const int jj = e >> 6, dd = e & 63;
        Vs[jj][dd] = (j0 + jj < Tk && d0 + dd < HD) ? vbase[(size_t)(j0 + jj) * S + d0 + dd] : 0.f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 16; j++) {
      const float4 a4 = *(const float4 *)&Ps[j][ty * 4];
      const float4 b4 = *(const float4 *)&Vs[j][tx * 4];
      const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[u][c] = fmaf(av[u], bv[c], acc[u][c]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int i = i0 + ty * 4 + u;
    if (i >= Tq) continue;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int d = d0 + tx * 4 + c;
      if (d < HD) out[((size_t)w * Tq + i) * S + h * HD + d] = acc[u][c];
    }
  }
}

// Direct grouped 1-D conv (rust/wasm-kernels/src/lib.rs:99-138): one thread per output sample.
// With `Lw` < L the columns are independent windows of Lw samples each (stride 1, same-length
// output): taps never cross a window seam, which is the per-window loop of
// src/engines/asr-parakeet/raw-encoder.js:343-351 done in one launch.
__global__ void k_conv1d(const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ bias,
                         float *__restrict__ y, int cout, int cin, int L, int Lout, int Lw, int k, int stride, int padl,
                         int dil, int groups, int act) {
  fa_grid_dep_sync();
  const int cin_g = cin / groups, cout_g = cout / groups;
  const unsigned n = (unsigned)cout * (unsigned)Lout;
  for (unsigned idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += gridDim.x * blockDim.x) {
    const int co = (int)(idx / (unsigned)Lout), t = (int)(idx % (unsigned)Lout), g = co / cout_g;
    const int wbase = Lw < L ? (t / Lw) * Lw : 0;   // first column of this sample's window
    const int tl = t - wbase;
    float acc = 0.f;
    for (int cig = 0; cig < cin_g; cig++) {
      const float *xr = x + (size_t)(g * cin_g + cig) * L + wbase;
      const float *wr = w + ((size_t)co * cin_g + cig) * k;
      for (int kk = 0; kk < k; kk++) {
        const int xi = tl * stride + kk * dil - padl;
        if (xi >= 0 && xi < Lw) acc = fmaf(xr[xi], wr[kk], acc);
      }
    }
    if (bias) acc += bias[co];
    y[idx] = fa_actf(acc, act);
  }
}

// Depthwise forms (one filter per channel): channel = blockIdx.y, threads walk the output row/plane, so
// the only integer division left is the window / row split.
__global__ void __launch_bounds__(256) k_dwconv1d(const float *__restrict__ x, const float *__restrict__ w,
                                                  const float *__restrict__ bias, float *__restrict__ y, int L, int Lw,
                                                  int k, int padl, int dil, int act) {
  fa_grid_dep_sync();
  const int c = blockIdx.y, t = blockIdx.x * 256 + threadIdx.x;
  if (t >= L) return;
  const int wbase = (t / Lw) * Lw, tl = t - wbase;
  const float *xr = x + (size_t)c * L + wbase;
  const float *wr = w + (size_t)c * k;
  float acc = 0.f;
  for (int kk = 0; kk < k; kk++) {
    const int xi = tl + kk * dil - padl;
    if (xi >= 0 && xi < Lw) acc = fmaf(xr[xi], __ldg(wr + kk), acc);
  }
  if (bias) acc += bias[c];
  y[(size_t)c * L + t] = fa_actf(acc, act);
}

__global__ void __launch_bounds__(256) k_dwconv2d_3x3(const float *__restrict__ x, const float *__restrict__ w,
                                                      const float *__restrict__ bias, float *__restrict__ y, int h, int W,
                                                      int sh, int sw, int pt, int pl, int Ho, int Wo, int act,
                                                      size_t xstride, size_t ystride) {
  fa_grid_dep_sync();
  // One thread = 4 consecutive outputs of one row of one channel (Wo4 = ceil(Wo/4) groups per row): the three input
  // rows it needs are loaded once, all loads issued before any arithmetic (addresses clamped, taps outside the image
  // zeroed afterwards), and the four results leave as one 16-byte store when the row allows it.
  const int c = blockIdx.y, Wo4 = (Wo + 3) >> 2;
  const unsigned grp = blockIdx.x * 256 + threadIdx.x;
  if (grp >= (unsigned)(Ho * Wo4)) return;
  x += (size_t)blockIdx.z * xstride;  // blockIdx.z = window
  y += (size_t)blockIdx.z * ystride;
  const int ho = (int)(grp / (unsigned)Wo4), wo0 = (int)(grp % (unsigned)Wo4) * 4;
  const float *xp = x + (size_t)c * h * W;
  float wk[9];
#pragma unroll
  for (int t = 0; t < 9; t++) wk[t] = __ldg(w + (size_t)c * 9 + t);
  const float b = bias ? bias[c] : 0.f;
  if (sw == 2) {
    float in[3][9];  // input columns 2*wo0 - pl .. + 8
    if (pl == 1 && (W & 3) == 0 && 2 * wo0 + 8 <= W && ((((uintptr_t)xp) & 15) == 0)) {
      // the 9 columns 2*wo0-1 .. 2*wo0+7 sit inside three aligned 16-byte groups starting at 2*wo0-4: three vector
      // loads per row instead of nine scalar ones (the scalar form kept the L1 90 % busy)
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const int hi = ho * sh + a - pt, hc = min(max(hi, 0), h - 1);
        const float4 *r4 = (const float4 *)(xp + (size_t)hc * W + 2 * wo0);
        const float4 m = r4[0], n = r4[1];
        const float lft = wo0 > 0 ? xp[(size_t)hc * W + 2 * wo0 - 1] : 0.f;
        in[a][0] = lft;
        in[a][1] = m.x, in[a][2] = m.y, in[a][3] = m.z, in[a][4] = m.w;
        in[a][5] = n.x, in[a][6] = n.y, in[a][7] = n.z, in[a][8] = n.w;
      }
    } else {
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int hi = ho * sh + a - pt, hc = min(max(hi, 0), h - 1);
#pragma unroll
      for (int j = 0; j < 9; j++) {
        const int wi = wo0 * 2 + j - pl, wc = min(max(wi, 0), W - 1);
        in[a][j] = xp[(size_t)hc * W + wc];
      }
    }
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int hi = ho * sh + a - pt;
#pragma unroll
      for (int j = 0; j < 9; j++) {
        const int wi = wo0 * 2 + j - pl;
        if (hi < 0 || hi >= h || wi < 0 || wi >= W) in[a][j] = 0.f;
      }
    }
    float o[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      float acc = b;
#pragma unroll
      for (int a = 0; a < 3; a++)
#pragma unroll
        for (int bb = 0; bb < 3; bb++) acc = fmaf(in[a][2 * q + bb], wk[a * 3 + bb], acc);
      o[q] = fa_actf(acc, act);
    }
    float *dst = y + (size_t)c * Ho * Wo + (size_t)ho * Wo + wo0;
    if ((Wo & 3) == 0 && ((ystride | ((size_t)Ho * Wo)) & 3) == 0 && (((uintptr_t)y) & 15) == 0) {
      *(float4 *)dst = make_float4(o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (wo0 + q < Wo) dst[q] = o[q];
    }
    return;
  }
  for (int q = 0; q < 4 && wo0 + q < Wo; q++) {  // other strides: one output at a time
    const int wo = wo0 + q;
    float acc = b;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int hi = ho * sh + a - pt;
      if (hi < 0 || hi >= h) continue;
#pragma unroll
      for (int bb = 0; bb < 3; bb++) {
        const int wi = wo * sw + bb - pl;
        if (wi >= 0 && wi < W) acc = fmaf(xp[(size_t)hi * W + wi], wk[a * 3 + bb], acc);
      }
    }
    y[(size_t)c * Ho * Wo + (size_t)ho * Wo + wo] = fa_actf(acc, act);
  }
}

// First two layers of the 8x subsampling stem in one pass, for 128-column images (128 mel bins):
//   c1 = relu(conv 1->C, 3x3, stride 2, pad 1)   [C][H1][64]      (never stored)
//   d  = depthwise 3x3, stride 2, pad 1 of c1     [C][H2][32]
// written straight into the packed f16 layout Wp[n/128][k/64][n%128][k%64] (n = pixel y*32 + x, k = channel)
// that the pointwise product after it streams as its [cin, H2*W2] operand.  Same accumulation order as
// k_conv2d_c1_3x3 and k_dwconv2d_3x3 and the same f16 rounding as k_pack_w_f16, so the result is bit-identical
// to running the three kernels; what disappears is the store and re-load of c1 (the largest tensor of the
// forward) and of d.
// CTA = 8 rows of d (two 128-pixel blocks) x 64 channels x one window.  The 35 input rows those need sit in shared
// memory, zero padded; a lane owns a channel (its 20 weights stay in registers), a warp walks a 4-pixel-wide
// column strip downwards, so every input read is a 16-byte shared-memory broadcast and each c1 row is evaluated
// once per strip (the row shared by consecutive d rows is kept in registers).
constexpr int kStemRows = 8, kStemInRows = 4 * kStemRows + 3, kStemLd = 132;
__global__ void __launch_bounds__(256, 3) k_stem_c1_dw_pack(const float *__restrict__ x, const float *__restrict__ w0,
                                                            const float *__restrict__ b0, const float *__restrict__ w1,
                                                            const float *__restrict__ b1, __half *__restrict__ out, int H,
                                                            int H1, int H2, int nblocks, int nch, size_t xstride,
                                                            size_t slab) {
  fa_grid_dep_sync();
  extern __shared__ __align__(16) unsigned char stem_smem[];
  float(*in_s)[kStemLd] = (float(*)[kStemLd])stem_smem;                                 // [35][4 zeros + 128]
  __half *o_s = (__half *)(stem_smem + sizeof(float) * kStemInRows * kStemLd);          // [2][128][64]
  const int y0 = blockIdx.x * kStemRows, cq = blockIdx.y, win = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  x += (size_t)win * xstride;
  const int in_row0 = 4 * y0 - 3;
  for (int e = threadIdx.x; e < kStemInRows * (kStemLd / 4); e += 256) {
    const int r = e / (kStemLd / 4), q = e - r * (kStemLd / 4), hi = in_row0 + r;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (q > 0 && hi >= 0 && hi < H) v = __ldg((const float4 *)(x + (size_t)hi * 128) + (q - 1));
    *(float4 *)&in_s[r][q * 4] = v;
  }
  const int cl = (warp & 1) * 32 + lane, c = cq * 64 + cl;
  float wa[9], wb[9];
#pragma unroll
  for (int t = 0; t < 9; t++) {
    wa[t] = __ldg(w0 + (size_t)c * 9 + t);
    wb[t] = __ldg(w1 + (size_t)c * 9 + t);
  }
  const float ba = b0 ? __ldg(b0 + c) : 0.f, bb = b1 ? __ldg(b1 + c) : 0.f;
  __syncthreads();

  // one c1 row (9 columns 2*x0-1 .. 2*x0+7) of this lane's channel; rows outside the c1 image are the zero
  // padding of the depthwise layer, and so is column -1
  auto c1_row = [&](int r, int x0, float(&o)[9]) {
    if (r < 0 || r >= H1) {
#pragma unroll
      for (int j = 0; j < 9; j++) o[j] = 0.f;
      return;
    }
#pragma unroll
    for (int j = 0; j < 9; j++) o[j] = ba;
    const int sr = 2 * r - 1 - in_row0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      float v[20];  // input columns 4*x0-4 .. 4*x0+15
      const float4 *src = (const float4 *)&in_s[sr + a][4 * x0];
#pragma unroll
      for (int q = 0; q < 5; q++) {
        const float4 t = src[q];
        v[4 * q] = t.x, v[4 * q + 1] = t.y, v[4 * q + 2] = t.z, v[4 * q + 3] = t.w;
      }
#pragma unroll
      for (int j = 0; j < 9; j++)
#pragma unroll
        for (int t = 0; t < 3; t++) o[j] = fmaf(v[1 + 2 * j + t], wa[a * 3 + t], o[j]);
    }
#pragma unroll
    for (int j = 0; j < 9; j++) o[j] = fmaxf(o[j], 0.0f);
    if (x0 == 0) o[0] = 0.f;
  };

  for (int task = 0; task < 2; task++) {
    const int x0 = ((warp >> 1) + task * 4) * 4;  // first d column of the strip
    float prev[9], ra[9], rb[9];
    c1_row(2 * y0 - 1, x0, prev);
    for (int yl = 0; yl < kStemRows; yl++) {
      const int y2 = y0 + yl;
      __half *dst = o_s + ((size_t)(yl >> 2) * 128 + (yl & 3) * 32 + x0) * 64 + cl;
      if (y2 >= H2) {  // rows past the image: the zero fill of the packed block
#pragma unroll
        for (int q = 0; q < 4; q++) dst[q * 64] = __float2half_rn(0.f);
        continue;
      }
      c1_row(2 * y2, x0, ra);
      c1_row(2 * y2 + 1, x0, rb);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        float acc = bb;
#pragma unroll
        for (int t = 0; t < 3; t++) acc = fmaf(prev[2 * q + t], wb[t], acc);
#pragma unroll
        for (int t = 0; t < 3; t++) acc = fmaf(ra[2 * q + t], wb[3 + t], acc);
#pragma unroll
        for (int t = 0; t < 3; t++) acc = fmaf(rb[2 * q + t], wb[6 + t], acc);
        dst[q * 64] = __float2half_rn(acc);
      }
#pragma unroll
      for (int j = 0; j < 9; j++) prev[j] = rb[j];
    }
  }
  __syncthreads();
  out += (size_t)win * slab;
  for (int half = 0; half < 2; half++) {
    const int nb = (y0 >> 2) + half;
    if (nb >= nblocks) break;
    uint4 *dst = (uint4 *)(out + ((size_t)nb * nch + cq) * 128 * 64);
    const uint4 *src = (const uint4 *)(o_s + (size_t)half * 128 * 64);
    for (int e = threadIdx.x; e < 128 * 64 / 8; e += 256) dst[e] = src[e];
  }
}

// Depthwise 3x3, stride 2, pad 1 over 32-column feature maps [C][H][32] -> [C][H2][16], written straight into the
// packed f16 layout Wp[n/128][k/64][n%128][k%64] (n = pixel y*16 + x, k = channel) of the pointwise product that
// follows: the stem's fourth layer without its f32 result and without the separate pack pass.  Same accumulation
// order as k_dwconv2d_3x3, same rounding as k_pack_w_f16.  CTA = 8 output rows (one 128-pixel block) x 64 channels
// x one window; a half-warp owns a channel, a lane one output column: it loads its two input columns of each of
// the 17 rows as one 8-byte word (a half-warp reads one 128-byte row) and gets the left neighbour by one shuffle.
constexpr int kDwPitch = 72;  // halves per pixel row of the staging tile: 144 B keeps 16-byte alignment, spreads banks
__global__ void __launch_bounds__(256) k_dw_s2_pack(const float *__restrict__ x, const float *__restrict__ w1,
                                                    const float *__restrict__ b1, __half *__restrict__ out, int C, int H,
                                                    int H2, int nblocks, int nch, size_t xstride, size_t slab) {
  fa_grid_dep_sync();
  __shared__ __align__(16) __half o_s[128 * kDwPitch];
  const int y0 = blockIdx.x * 8, cq = blockIdx.y, win = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, x2 = lane & 15;
  x += (size_t)win * xstride;
#pragma unroll 1
  for (int ci = 0; ci < 4; ci++) {
    const int cl = warp * 8 + ci * 2 + (lane >> 4), c = cq * 64 + cl;
    const float2 *xc = (const float2 *)(x + (size_t)c * H * 32) + x2;
    float2 v[17];
#pragma unroll
    for (int r = 0; r < 17; r++) {
      const int row = 2 * y0 - 1 + r;
      v[r] = (row >= 0 && row < H) ? __ldg(xc + (size_t)row * 16) : make_float2(0.f, 0.f);
    }
    float wk[9];
#pragma unroll
    for (int t = 0; t < 9; t++) wk[t] = __ldg(w1 + (size_t)c * 9 + t);
    const float bb = b1 ? __ldg(b1 + c) : 0.f;
    float lf[17];
#pragma unroll
    for (int r = 0; r < 17; r++) {
      lf[r] = __shfl_up_sync(0xffffffffu, v[r].y, 1);
      if (x2 == 0) lf[r] = 0.f;  // column -1 is padding (and lane 16 must not see the other channel)
    }
#pragma unroll
    for (int yl = 0; yl < 8; yl++) {
      float acc = bb;
#pragma unroll
      for (int a = 0; a < 3; a++) {
        acc = fmaf(lf[2 * yl + a], wk[a * 3], acc);
        acc = fmaf(v[2 * yl + a].x, wk[a * 3 + 1], acc);
        acc = fmaf(v[2 * yl + a].y, wk[a * 3 + 2], acc);
      }
      o_s[(yl * 16 + x2) * kDwPitch + cl] = __float2half_rn(y0 + yl < H2 ? acc : 0.f);
    }
  }
  __syncthreads();
  if ((int)blockIdx.x < nblocks) {
    uint4 *dst = (uint4 *)(out + (size_t)win * slab + ((size_t)blockIdx.x * nch + cq) * 128 * 64);
    for (int e = threadIdx.x; e < 128 * 8; e += 256) dst[e] = *(const uint4 *)(o_s + (e >> 3) * kDwPitch + (e & 7) * 8);
  }
}

// The conformer conv module between its two pointwise projections, in the time-major layout the
// projections use (src/engines/asr-parakeet/raw-encoder.js:340-362 does it as transpose -> glu ->
// per-window depthwise conv1d(+act) -> transpose): x [W*T, 2D] -> y [W*T, D],
//   y[t][c] = act( bias[c] + sum_k w[c][k] * g[t + k - padl][c] ),  g[t][c] = x[t][c] * sigmoid(x[t][c + D]),
// taps outside the window of t read zero.  Lanes walk channels, so every access is coalesced; the result is
// also emitted as the packed f16 row operand of the projection that follows.
__global__ void __launch_bounds__(256) k_glu_dwconv_tm(const float *__restrict__ x, const float *__restrict__ w,
                                                       const float *__restrict__ bias, float *__restrict__ y,
                                                       __half *__restrict__ y16, int rows, int Tw, int D, int k, int padl,
                                                       int act) {
  fa_grid_dep_sync();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= D) return;
  float wk[16];
#pragma unroll
  for (int kk = 0; kk < 16; kk++) wk[kk] = kk < k ? w[(size_t)c * k + kk] : 0.f;
  const float b = bias ? bias[c] : 0.f;
  const int t0 = blockIdx.y * 16;  // 16 consecutive frames per CTA row block
  for (int t = t0; t < t0 + 16 && t < rows; t++) {
    const int wbase = (t / Tw) * Tw, tl = t - wbase;
    float acc = b;
#pragma unroll
    for (int kk = 0; kk < 16; kk++) {
      if (kk >= k) break;
      const int tt = tl + kk - padl;
      if (tt >= 0 && tt < Tw) {
        const float *xr = x + (size_t)(wbase + tt) * (2 * D);
        acc = fmaf(wk[kk], xr[c] * (1.0f / (1.0f + expf(-xr[c + D]))), acc);
      }
    }
    const float o = fa_actf(acc, act);
    y[(size_t)t * D + c] = o;
    if (y16) y16[((size_t)(c >> 6) * rows + t) * 64 + (c & 63)] = __float2half_rn(o);
  }
}

// Same operation with the tap count known at compile time: a thread owns one channel and 16 consecutive
// frames, evaluates the gated values of the 16+K-1 frames it needs once (one exp each) and slides the
// filter over them in registers.
template <int K>
__global__ void __launch_bounds__(256) k_glu_dwconv_tm_k(const float *__restrict__ x, const float *__restrict__ w,
                                                         const float *__restrict__ bias, float *__restrict__ y,
                                                         __half *__restrict__ y16, int rows, int Tw, int D, int padl,
                                                         int act, int chunks) {
  fa_grid_dep_sync();
  // blockIdx.y = (window, chunk of 16 frames inside it): every frame a CTA touches that belongs to its window
  // takes part, everything else is a zero tap, so the filter loop needs no per-tap window test.
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= D) return;
  const int wdw = blockIdx.y / chunks, ch = blockIdx.y - wdw * chunks;
  const int lo = wdw * Tw, hi = lo + Tw;          // frames of this window
  const int t0 = lo + ch * 16, nt = min(16, hi - t0);
  float wk[K];
#pragma unroll
  for (int kk = 0; kk < K; kk++) wk[kk] = w[(size_t)c * K + kk];
  const float b = bias ? bias[c] : 0.f;
  float g[16 + K - 1], gate[16 + K - 1];
  const size_t ld = 2 * (size_t)D;
  // a chunk whose 16 + K - 1 frames all lie inside the window (all but the first and last chunk of a window) needs
  // no clamping, no zero taps and no ragged tail: one base address and constant strides
  const bool interior = t0 - padl >= lo && t0 - padl + 16 + K - 1 <= hi;
  if (interior) {
    const float *xr = x + (size_t)(t0 - padl) * ld + c;
#pragma unroll
    for (int j = 0; j < 16 + K - 1; j++) {
      g[j] = __ldg(xr + j * ld);
      gate[j] = __ldg(xr + j * ld + D);
    }
#pragma unroll
    for (int j = 0; j < 16 + K - 1; j++) g[j] *= fa_sigmoid_fast(gate[j]);
  } else {
    // all loads first (addresses clamped into the window so none is conditional), then the gating math
#pragma unroll
    for (int j = 0; j < 16 + K - 1; j++) {
      const int tg = t0 - padl + j, tc = min(max(tg, lo), hi - 1);
      const float *xr = x + (size_t)tc * ld;
      g[j] = __ldg(xr + c);
      gate[j] = __ldg(xr + c + D);
    }
#pragma unroll
    for (int j = 0; j < 16 + K - 1; j++) {
      const int tg = t0 - padl + j;
      g[j] = (tg >= lo && tg < hi) ? g[j] * fa_sigmoid_fast(gate[j]) : 0.f;
    }
  }
  float *yr = y ? y + (size_t)t0 * D + c : nullptr;  // y == nullptr: the result exists only as the packed operand
  __half *y16r = y16 ? y16 + ((size_t)(c >> 6) * rows + t0) * 64 + (c & 63) : nullptr;
  const bool silu = act == FA_ACT_SILU;
#pragma unroll
  for (int i = 0; i < 16; i++) {
    if (!interior && i >= nt) break;
    float acc = b;
#pragma unroll
    for (int kk = 0; kk < K; kk++) acc = fmaf(wk[kk], g[i + kk], acc);
    const float o = silu ? fa_silu_fast(acc) : fa_actf(acc, act);
    if (yr) yr[(size_t)i * D] = o;
    if (y16r) y16r[i * 64] = __float2half_rn(o);
  }
}

// Direct 2-D conv, batch 1 (wasm-context.js:632-685): one thread per output element.
__global__ void k_conv2d(const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ bias,
                         float *__restrict__ y, int cout, int cin, int h, int W, int kh, int kw, int sh, int sw, int pt,
                         int pl, int Ho, int Wo, int groups, int act) {
  fa_grid_dep_sync();
  const int cinG = cin / groups, coutG = cout / groups;
  const unsigned plane = (unsigned)Ho * (unsigned)Wo, n = (unsigned)cout * plane;
  for (unsigned idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += gridDim.x * blockDim.x) {
    const int co = (int)(idx / plane);
    const unsigned rem = idx - (unsigned)co * plane;
    const int ho = (int)(rem / (unsigned)Wo), wo = (int)(rem % (unsigned)Wo);
    const int g = co / coutG;
    float acc = bias ? bias[co] : 0.f;
    for (int ci = 0; ci < cinG; ci++) {
      const float *xp = x + (size_t)(g * cinG + ci) * h * W;
      const float *wp = w + ((size_t)co * cinG + ci) * kh * kw;
      for (int a = 0; a < kh; a++) {
        const int hi = ho * sh + a - pt;
        if (hi < 0 || hi >= h) continue;
        for (int b = 0; b < kw; b++) {
          const int wi = wo * sw + b - pl;
          if (wi < 0 || wi >= W) continue;
          acc = fmaf(xp[(size_t)hi * W + wi], wp[a * kw + b], acc);
        }
      }
    }
    y[idx] = fa_actf(acc, act);
  }
}

// Single-input-channel 3x3 conv (the first subsampling layer; the reference has the same special
// case, src/gpu/kernels/convolution.js:112-147): a thread reads its 9 taps once and produces 32
// output channels, lanes walking consecutive output positions so every channel's store is coalesced.
template <int SW>
__global__ void __launch_bounds__(256, 4) k_conv2d_c1_3x3(const float *__restrict__ x, const float *__restrict__ w,
                                                       const float *__restrict__ bias, float *__restrict__ y, int cout,
                                                       int h, int W, int sh, int sw, int pt, int pl, int Ho, int Wo,
                                                       int act, size_t xstride, size_t ystride) {
  fa_grid_dep_sync();
  // One thread = 4 consecutive output positions of one row, all 32 channels of its channel group: the 3 x 9 input
  // patch is loaded once, each channel's 9 weights are read from shared memory once per 4 outputs (read per output
  // they made the kernel load/store-unit bound), and every channel's 4 results leave as one 16-byte store.
  __shared__ float ws[32][9], bs[32];
  const int co0 = blockIdx.y * 32;
  x += (size_t)blockIdx.z * xstride;  // blockIdx.z = window
  y += (size_t)blockIdx.z * ystride;
  for (int e = threadIdx.x; e < 32 * 9; e += 256) {
    const int c = e / 9;
    ws[c][e % 9] = co0 + c < cout ? w[(size_t)(co0 + c) * 9 + e % 9] : 0.f;
  }
  if (threadIdx.x < 32) bs[threadIdx.x] = (bias && co0 + threadIdx.x < cout) ? bias[co0 + threadIdx.x] : 0.f;
  __syncthreads();
  const unsigned plane = (unsigned)Ho * (unsigned)Wo;
  const int Wo4 = (Wo + 3) >> 2;
  const unsigned groups = (unsigned)Ho * (unsigned)Wo4;
  const bool vec = (Wo & 3) == 0 && ((ystride | plane) & 3) == 0 && (((uintptr_t)y) & 15) == 0;
  for (unsigned grp = blockIdx.x * 256 + threadIdx.x; grp < groups; grp += gridDim.x * 256) {
    const int ho = (int)(grp / (unsigned)Wo4), wo0 = (int)(grp % (unsigned)Wo4) * 4;
    constexpr int NCOL = 3 * SW + 3;  // input columns wo0*SW - pl .. that 4 outputs touch
    float in[3][NCOL];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int hi = ho * sh + a - pt;
#pragma unroll
      for (int j = 0; j < NCOL; j++) {
        const int wi = wo0 * SW + j - pl;
        in[a][j] = (hi >= 0 && hi < h && wi >= 0 && wi < W) ? x[(size_t)hi * W + wi] : 0.f;
      }
    }
#pragma unroll 2
    for (int c = 0; c < 32; c++) {
      if (co0 + c >= cout) break;
      float wk[9];
#pragma unroll
      for (int t = 0; t < 9; t++) wk[t] = ws[c][t];
      float o[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        float acc = bs[c];
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
          for (int bb = 0; bb < 3; bb++) {
            acc = fmaf(in[a][SW * q + bb], wk[a * 3 + bb], acc);  // tap bb of output q sits in column q*SW + bb
          }
        o[q] = fa_actf(acc, act);
      }
      float *dst = y + (size_t)(co0 + c) * plane + (size_t)ho * Wo + wo0;
      if (vec) {
        *(float4 *)dst = make_float4(o[0], o[1], o[2], o[3]);
      } else {
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (wo0 + q < Wo) dst[q] = o[q];
      }
    }
  }
}

// Per-row argmax: out[r] = {index, value}; ties resolve to the lowest index like the host loop
// of src/engines/asr-whisper/index.ts:80-97.  One block per row, bound by the latency of its loads: a long row takes 32 warps
// with eight loads of a thread in flight, a short one, or one of so many that the blocks fill the GPU several times, 8 warps
// with one load each, eight blocks to an SM.  Measured, us, 8 warps / 32 warps: 64 rows of 51866 columns 9.5 / 6.9, of 16384 3.8
// / 3.3, of 8192 2.6 / 2.6, of 1000 2.0 / 2.5; 512 rows of 8192 4.9 / 4.9, of 4096 3.3 / 4.6; 2048 rows of 16384 27.5 / 26.6,
// of 8192 11.6 / 14.6, of 1000 4.9 / 14.1.  So 32 warps from 16384 columns on, and from 8192 up to four rows per SM.
template <int kArgThreads, int kArgBatch>
__global__ void __launch_bounds__(kArgThreads) k_argmax_rows(const float *__restrict__ x, float *__restrict__ out, int R, int ld,
                                                             int C) {
  fa_grid_dep_sync();
  __shared__ float bv[kArgThreads / 32];
  __shared__ int bi[kArgThreads / 32];
  auto better = [](float v, int j, float best, int idx) { return v > best || (v == best && j < idx); };
  for (int r = blockIdx.x; r < R; r += gridDim.x) {
    const float *row = x + (size_t)r * ld;
    float best = -INFINITY;
    int idx = 0x7fffffff;
    for (int j0 = threadIdx.x; j0 < C; j0 += kArgThreads * kArgBatch) {
      float v[kArgBatch];
#pragma unroll
      for (int u = 0; u < kArgBatch; u++) {
        const int j = j0 + u * kArgThreads;
        v[u] = j < C ? row[j] : -INFINITY;
      }
#pragma unroll
      for (int u = 0; u < kArgBatch; u++) {
        const int j = j0 + u * kArgThreads;
        if (j < C && better(v[u], j, best, idx)) { best = v[u]; idx = j; }
      }
    }
    auto warp_best = [&]() {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (better(ov, oi, best, idx)) { best = ov; idx = oi; }
      }
    };
    warp_best();
    if ((threadIdx.x & 31) == 0) { bv[threadIdx.x >> 5] = best; bi[threadIdx.x >> 5] = idx; }
    __syncthreads();
    if (threadIdx.x < 32) {
      const int w = threadIdx.x < kArgThreads / 32 ? threadIdx.x : 0;  // (a repeated warp changes nothing)
      best = bv[w], idx = bi[w];
      warp_best();
      if (threadIdx.x == 0) {
        out[(size_t)r * 2] = (float)idx;
        out[(size_t)r * 2 + 1] = best;
      }
    }
    __syncthreads();
  }
}

// Token embedding + position for one decoding step, on the device: out[s][:] = table[idx[s*stride]][:] + pos[n][:].
// idx holds token ids as floats (an argmax_rows result, stride 2, or a [S,1] tensor, stride 1); ids outside
// [0, V) select row 0 and set word 3 of the context's status block (reported by the next sync) instead of reading out of bounds.
__global__ void __launch_bounds__(256) k_embed_rows(const float *__restrict__ table, const float *__restrict__ pos,
                                                     const float *__restrict__ idx, int stride, int V, int D, int n,
                                                     float *__restrict__ out, int *status) {
  fa_grid_dep_sync();
  const int s = blockIdx.x;
  int t = (int)idx[(size_t)s * stride];
  if (t < 0 || t >= V) {
    if (threadIdx.x == 0) atomicOr(status + 3, 1);
    t = 0;
  }
  const float *row = table + (size_t)t * D, *pr = pos + (size_t)n * D;
  for (int d = threadIdx.x; d < D; d += 256) out[(size_t)s * D + d] = row[d] + pr[d];
}

int grid1d(fa_ctx *ctx, size_t n, int block) {
  size_t g = (n + block - 1) / block, cap = (size_t)ctx->sm_count * 16;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

int need_f32(fa_ctx *ctx, const fa_tensor *t, const char *op) {
  FA_REQUIRE(ctx, fa_valid(ctx, t), "%s: unknown tensor handle", op);
  FA_REQUIRE(ctx, t->storage == FA_F32, "%s: operand must be f32 storage", op);
  return fa_touch_f32(ctx, t);
}

}  // namespace

#define GLUE_PROLOGUE(name)                                                         \
  if (!ctx || !out) return fa_fail(ctx, FA_ERR_INVALID, name ": NULL argument");    \
  FA_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));

// operand_only: the caller promises the result is read as a matmul row operand.  When the packed f16 shadow can
// carry it (single plane, warp-per-row kernel), the f32 store is skipped and the tensor is marked lazy: anything
// else that reads it gets the f32 storage filled from the shadow first (values rounded to f16).
static int layernorm_impl(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *gamma, const fa_tensor *beta, float eps,
                          bool operand_only, fa_tensor **out) {
  GLUE_PROLOGUE("layernorm");
  FA_TRY(need_f32(ctx, x, "layernorm"));
  FA_TRY(need_f32(ctx, gamma, "layernorm"));
  FA_TRY(need_f32(ctx, beta, "layernorm"));
  FA_REQUIRE(ctx, gamma->rows * gamma->cols >= x->cols && beta->rows * beta->cols >= x->cols,
             "layernorm: gamma/beta shorter than %d columns", x->cols);
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, x->rows, x->cols, FA_F32, true, &y));
  if (x->rows && x->cols) {
    int grid = x->rows < ctx->sm_count * 8 ? x->rows : ctx->sm_count * 8;
    {
      LaunchScope ls(ctx, "layernorm");
      __half *y16 = nullptr;
      size_t lo_off = 0;
      const float *xp = (const float *)x->dptr, *gp = (const float *)gamma->dptr, *bp = (const float *)beta->dptr;
      const bool al = (((uintptr_t)xp | (uintptr_t)gp | (uintptr_t)bp | (uintptr_t)y->dptr) & 15) == 0;
      const bool reg = (x->cols & 3) == 0 && x->cols <= 4096 && al;
      if ((x->cols & 63) == 0 && fa_tc_available(ctx)) {
        if (x->rows <= ctx->f16_hilo_rows) {  // few rows: the consumer wants value + residue planes
          if (reg && (y16 = fa_shadow_hilo_block(ctx, y)) != nullptr) {
            y->a16_valid = true;
            lo_off = (size_t)(x->cols >> 6) * x->rows * 64;
          }
        } else if (x->rows >= 16 && (y16 = fa_shadow_block(ctx, y)) != nullptr) {
          y->a16_valid = true;
        }
      }
      float *yp = (float *)y->dptr;
      if (operand_only && fa_operand_only_ok(ctx, x->rows, x->cols) && y16 && !lo_off && (x->cols & 3) == 0 && x->cols <= 1024 && al) {
        yp = nullptr;
        y->f32_lazy = true;
        y->lazy_sticky = ctx->capturing != nullptr;
      }
      const bool few = ceil_div(x->rows, 8) <= ctx->sm_count;  // one block per SM at most: see k_layernorm_warp
      if ((x->cols & 3) == 0 && x->cols <= 512 && al)
        fa_launch_dep(ctx, few ? k_layernorm_warp<4, true> : k_layernorm_warp<4, false>, dim3(ceil_div(x->rows, 8)), dim3(256), 0, xp, gp, bp, yp, y16, lo_off, x->rows,
                                                                          x->cols, eps);
      else if ((x->cols & 3) == 0 && x->cols <= 1024 && al)
        fa_launch_dep(ctx, few ? k_layernorm_warp<8, true> : k_layernorm_warp<8, false>, dim3(ceil_div(x->rows, 8)), dim3(256), 0, xp, gp, bp, yp, y16, lo_off, x->rows,
                                                                          x->cols, eps);
      else if (reg)
        fa_launch_dep(ctx, k_layernorm_reg<4>, dim3(x->rows), dim3(256), 0, xp, gp, bp, (float *)y->dptr, y16, lo_off, x->rows, x->cols, eps);
      else
        fa_launch_dep(ctx, k_layernorm, dim3(grid), dim3(256), 0, xp, gp, bp, (float *)y->dptr, y16, x->rows, x->cols, eps);
    }
    FA_LAUNCH_CHECK(ctx, "layernorm");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_layernorm(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *gamma, const fa_tensor *beta, float eps,
                            fa_tensor **out) {
  return layernorm_impl(ctx, x, gamma, beta, eps, false, out);
}
extern "C" int fa_layernorm_operand(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *gamma, const fa_tensor *beta,
                                    float eps, fa_tensor **out) {
  return layernorm_impl(ctx, x, gamma, beta, eps, true, out);
}

// y = layernorm(x, g1, b1); z = layernormOperand(y, g2, b2) - in one pass over the rows when z can be kept as the
// packed operand alone, as the two calls otherwise.
extern "C" int fa_layernorm_chain(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *g1, const fa_tensor *b1,
                                  const fa_tensor *g2, const fa_tensor *b2, float eps, fa_tensor **out_y, fa_tensor **out) {
  GLUE_PROLOGUE("layernormChain");
  if (!out_y) return fa_fail(ctx, FA_ERR_INVALID, "layernormChain: NULL argument");
  const fa_tensor *ts[5] = {x, g1, b1, g2, b2};
  for (int i = 0; i < 5; i++) FA_TRY(need_f32(ctx, ts[i], "layernormChain"));
  for (int i = 1; i < 5; i++)
    FA_REQUIRE(ctx, ts[i]->rows * ts[i]->cols >= x->cols, "layernormChain: gamma/beta shorter than %d columns", x->cols);
  const bool al = ((((uintptr_t)x->dptr) | ((uintptr_t)g1->dptr) | ((uintptr_t)b1->dptr) | ((uintptr_t)g2->dptr) |
                    ((uintptr_t)b2->dptr)) & 15) == 0;
  if (!(al && (x->cols & 63) == 0 && x->cols <= 1024 && fa_tc_available(ctx) && fa_operand_only_ok(ctx, x->rows, x->cols))) {
    FA_TRY(layernorm_impl(ctx, x, g1, b1, eps, false, out_y));
    int rc = layernorm_impl(ctx, *out_y, g2, b2, eps, true, out);
    if (rc != FA_OK) fa_free_tensor(ctx, *out_y);
    return rc;
  }
  fa_tensor *y = nullptr, *z = nullptr;
  FA_TRY(fa_tensor_new(ctx, x->rows, x->cols, FA_F32, true, &y));
  int rc = fa_tensor_new(ctx, x->rows, x->cols, FA_F32, true, &z);
  __half *z16 = rc == FA_OK ? fa_shadow_block(ctx, z) : nullptr;
  if (rc != FA_OK || !z16 || ((((uintptr_t)y->dptr)) & 15)) {
    if (z) fa_free_tensor(ctx, z);
    fa_free_tensor(ctx, y);
    return rc != FA_OK ? rc : fa_fail(ctx, FA_ERR_OOM, "layernormChain: no block for the packed operand");
  }
  z->a16_valid = true;
  z->f32_lazy = true;
  z->lazy_sticky = ctx->capturing != nullptr;
  {
    LaunchScope ls(ctx, "layernorm");
    const float *xp = (const float *)x->dptr;
    const bool few = ceil_div(x->rows, 8) <= ctx->sm_count;
    if (x->cols <= 512)
      fa_launch_dep(ctx, few ? k_layernorm_chain<4, true> : k_layernorm_chain<4, false>, dim3(ceil_div(x->rows, 8)), dim3(256), 0, xp, (const float *)g1->dptr,
                    (const float *)b1->dptr, (const float *)g2->dptr, (const float *)b2->dptr, (float *)y->dptr, z16, x->rows,
                    x->cols, eps);
    else
      fa_launch_dep(ctx, few ? k_layernorm_chain<8, true> : k_layernorm_chain<8, false>, dim3(ceil_div(x->rows, 8)), dim3(256), 0, xp, (const float *)g1->dptr,
                    (const float *)b1->dptr, (const float *)g2->dptr, (const float *)b2->dptr, (float *)y->dptr, z16, x->rows,
                    x->cols, eps);
  }
  FA_LAUNCH_CHECK(ctx, "layernorm");
  *out_y = y;
  *out = z;
  return FA_OK;
}

extern "C" int fa_softmax(fa_ctx *ctx, const fa_tensor *x, fa_tensor **out) {
  GLUE_PROLOGUE("softmax");
  FA_TRY(need_f32(ctx, x, "softmax"));
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, x->rows, x->cols, FA_F32, true, &y));
  if (x->rows && x->cols) {
    int grid = ceil_div(x->rows, 8);
    if (grid > ctx->sm_count * 16) grid = ctx->sm_count * 16;
    {
      LaunchScope ls(ctx, "softmax");
      if (x->cols <= 256)
        fa_launch_dep(ctx, k_softmax_reg, dim3(grid), dim3(256), 0, (const float *)x->dptr, (float *)y->dptr, x->rows, x->cols);
      else
        fa_launch_dep(ctx, k_softmax, dim3(grid), dim3(256), 0, (const float *)x->dptr, (float *)y->dptr, x->rows, x->cols);
    }
    FA_LAUNCH_CHECK(ctx, "softmax");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_ewise(fa_ctx *ctx, const fa_tensor *a, const fa_tensor *b, int op_mul, fa_tensor **out) {
  GLUE_PROLOGUE("ewise");
  FA_TRY(need_f32(ctx, a, "ewise"));
  FA_TRY(need_f32(ctx, b, "ewise"));
  const bool bcast = b->rows == 1 && a->rows != 1;
  FA_REQUIRE(ctx, b->cols == a->cols && (bcast || b->rows == a->rows), "ewise: a is [%d,%d], b is [%d,%d]", a->rows,
             a->cols, b->rows, b->cols);
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, a->rows, a->cols, FA_F32, true, &y));
  size_t n = (size_t)a->rows * a->cols;
  if (n) {
    {
      LaunchScope ls(ctx, "ewise");
      if (!bcast && (n & 3) == 0 && n / 4 < (1ull << 32))
        fa_launch_dep(ctx, k_ewise4, dim3(grid1d(ctx, n / 4, 256)), dim3(256), 0, (const float4 *)a->dptr, (const float4 *)b->dptr,
                                                                   (float4 *)y->dptr, (unsigned)(n / 4), op_mul);
      else
        fa_launch_dep(ctx, k_ewise, dim3(grid1d(ctx, n, 256)), dim3(256), 0, (const float *)a->dptr, (const float *)b->dptr,
                                                              (float *)y->dptr, n, a->cols, bcast ? 1 : 0, op_mul);
    }
    FA_LAUNCH_CHECK(ctx, "ewise");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_scale(fa_ctx *ctx, const fa_tensor *x, float s, fa_tensor **out) {
  GLUE_PROLOGUE("scale");
  FA_TRY(need_f32(ctx, x, "scale"));
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, x->rows, x->cols, FA_F32, true, &y));
  size_t n = (size_t)x->rows * x->cols;
  if (n) {
    {
      LaunchScope ls(ctx, "scale");
      fa_launch_dep(ctx, k_scale, dim3(grid1d(ctx, n, 256)), dim3(256), 0, (const float *)x->dptr, (float *)y->dptr, n, s);
    }
    FA_LAUNCH_CHECK(ctx, "scale");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_unary(fa_ctx *ctx, const fa_tensor *x, int act, fa_tensor **out) {
  GLUE_PROLOGUE("unary");
  FA_TRY(need_f32(ctx, x, "unary"));
  FA_REQUIRE(ctx, act >= 0 && act <= 5, "unary: unknown activation code %d", act);
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, x->rows, x->cols, FA_F32, true, &y));
  size_t n = (size_t)x->rows * x->cols;
  if (n) {
    {
      LaunchScope ls(ctx, "unary");
      fa_launch_dep(ctx, k_unary, dim3(grid1d(ctx, n, 256)), dim3(256), 0, (const float *)x->dptr, (float *)y->dptr, n, act);
    }
    FA_LAUNCH_CHECK(ctx, "unary");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_glu(fa_ctx *ctx, const fa_tensor *x, fa_tensor **out) {
  GLUE_PROLOGUE("glu");
  FA_TRY(need_f32(ctx, x, "glu"));
  FA_REQUIRE(ctx, x->rows % 2 == 0, "glu: %d rows is not even", x->rows);
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, x->rows / 2, x->cols, FA_F32, true, &y));
  size_t n = (size_t)(x->rows / 2) * x->cols;
  if (n) {
    {
      LaunchScope ls(ctx, "glu");
      if ((n & 3) == 0 && n / 4 < (1ull << 31))
        fa_launch_dep(ctx, k_glu4, dim3(grid1d(ctx, n / 4, 256)), dim3(256), 0, (const float4 *)x->dptr, (float4 *)y->dptr, (unsigned)(n / 4));
      else
        fa_launch_dep(ctx, k_glu, dim3(grid1d(ctx, n, 256)), dim3(256), 0, (const float *)x->dptr, (float *)y->dptr, x->rows / 2, x->cols);
    }
    FA_LAUNCH_CHECK(ctx, "glu");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_transpose(fa_ctx *ctx, const fa_tensor *x, fa_tensor **out) {
  GLUE_PROLOGUE("transpose");
  FA_TRY(need_f32(ctx, x, "transpose"));
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, x->cols, x->rows, FA_F32, true, &y));
  if (x->rows && x->cols) {
    dim3 grid(ceil_div(x->cols, 32), ceil_div(x->rows, 32)), block(32, 8);
    FA_REQUIRE(ctx, grid.y <= 65535, "transpose: %d rows is too many", x->rows);
    {
      LaunchScope ls(ctx, "transpose");
      fa_launch_dep(ctx, k_transpose, dim3(grid), dim3(block), 0, (const float *)x->dptr, (float *)y->dptr, x->rows, x->cols);
    }
    FA_LAUNCH_CHECK(ctx, "transpose");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_slice_cols(fa_ctx *ctx, const fa_tensor *x, int col0, int width, fa_tensor **out) {
  GLUE_PROLOGUE("sliceCols");
  FA_TRY(need_f32(ctx, x, "sliceCols"));
  FA_REQUIRE(ctx, col0 >= 0 && width >= 0 && col0 + width <= x->cols, "sliceCols: [%d,%d) of %d columns", col0,
             col0 + width, x->cols);
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, x->rows, width, FA_F32, true, &y));
  size_t n = (size_t)x->rows * width;
  if (n) {
    {
      LaunchScope ls(ctx, "slice_cols");
      fa_launch_dep(ctx, k_copy_cols, dim3(grid1d(ctx, n, 256)), dim3(256), 0, (const float *)x->dptr, x->cols, col0, (float *)y->dptr,
                                                                width, 0, x->rows, width);
    }
    FA_LAUNCH_CHECK(ctx, "slice_cols");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_set_cols(fa_ctx *ctx, fa_tensor *dst, const fa_tensor *src, int col0) {
  if (!ctx) return fa_fail(ctx, FA_ERR_INVALID, "setCols: NULL context");
  FA_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
  FA_TRY(need_f32(ctx, dst, "setCols"));
  FA_TRY(need_f32(ctx, src, "setCols"));
  FA_REQUIRE(ctx, col0 >= 0 && col0 + src->cols <= dst->cols && src->rows <= dst->rows,
             "setCols: src [%d,%d] at column %d does not fit dst [%d,%d]", src->rows, src->cols, col0, dst->rows, dst->cols);
  fa_shadow_drop(dst);
  size_t n = (size_t)src->rows * src->cols;
  if (n) {
    {
      LaunchScope ls(ctx, "set_cols");
      fa_launch_dep(ctx, k_copy_cols, dim3(grid1d(ctx, n, 256)), dim3(256), 0, (const float *)src->dptr, src->cols, 0,
                                                                (float *)dst->dptr, dst->cols, col0, src->rows, src->cols);
    }
    FA_LAUNCH_CHECK(ctx, "set_cols");
  }
  return FA_OK;
}

// Column shards stacked along rows, g [world*M][Ns] (what an all-gather of per-rank [M][Ns] results
// leaves), into the row-major product out [M][world*Ns]: out[m][r*Ns + j] = g[r*M + m][j].
__global__ void __launch_bounds__(256) k_unshard_cols(const float4 *__restrict__ g, float4 *__restrict__ out, int M,
                                                      int ns4, int world) {
  fa_grid_dep_sync();
  const size_t total = (size_t)world * M * ns4;
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (size_t)gridDim.x * 256) {
    const int j = (int)(i % ns4);
    const size_t rm = i / ns4;
    const int m = (int)(rm % M), r = (int)(rm / M);
    out[((size_t)m * world + r) * ns4 + j] = g[i];
  }
}

extern "C" int fa_unshard_cols(fa_ctx *ctx, const fa_tensor *gathered, int world, fa_tensor **out) {
  GLUE_PROLOGUE("unshardCols");
  FA_TRY(need_f32(ctx, gathered, "unshardCols"));
  FA_REQUIRE(ctx, world >= 1 && gathered->rows % world == 0, "unshardCols: %d rows do not split into %d shards",
             gathered->rows, world);
  FA_REQUIRE(ctx, (gathered->cols & 3) == 0, "unshardCols: shard width %d is not a multiple of 4", gathered->cols);
  const int M = gathered->rows / world, ns = gathered->cols;
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, M, world * ns, FA_F32, true, &y));
  const size_t n4 = (size_t)gathered->rows * (ns / 4);
  if (n4) {
    {
      LaunchScope ls(ctx, "unshard_cols");
      fa_launch_dep(ctx, k_unshard_cols, dim3(grid1d(ctx, n4, 256)), dim3(256), 0, (const float4 *)gathered->dptr, (float4 *)y->dptr, M,
                                                                    ns / 4, world);
    }
    FA_LAUNCH_CHECK(ctx, "unshard_cols");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_slice_rows(fa_ctx *ctx, const fa_tensor *x, int row0, int count, fa_tensor **out) {
  GLUE_PROLOGUE("sliceRows");
  FA_TRY(need_f32(ctx, x, "sliceRows"));
  FA_REQUIRE(ctx, row0 >= 0 && count >= 0 && row0 + count <= x->rows, "sliceRows: [%d,%d) of %d rows", row0, row0 + count,
             x->rows);
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, count, x->cols, FA_F32, true, &y));
  size_t bytes = (size_t)count * x->cols * 4;
  if (bytes)
    FA_CHECK_CUDA(ctx, cudaMemcpyAsync(y->dptr, (const float *)x->dptr + (size_t)row0 * x->cols, bytes,
                                       cudaMemcpyDeviceToDevice, ctx->stream));
  *out = y;
  return FA_OK;
}

extern "C" int fa_copy_rows(fa_ctx *ctx, fa_tensor *dst, const fa_tensor *src, int row_offset) {
  if (!ctx) return fa_fail(ctx, FA_ERR_INVALID, "copyRows: NULL context");
  FA_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
  FA_TRY(need_f32(ctx, dst, "copyRows"));
  FA_TRY(need_f32(ctx, src, "copyRows"));
  FA_REQUIRE(ctx, src->cols == dst->cols && row_offset >= 0 && row_offset + src->rows <= dst->rows,
             "copyRows: src [%d,%d] at row %d does not fit dst [%d,%d]", src->rows, src->cols, row_offset, dst->rows,
             dst->cols);
  fa_shadow_drop(dst);
  size_t bytes = (size_t)src->rows * src->cols * 4;
  if (bytes)
    FA_CHECK_CUDA(ctx, cudaMemcpyAsync((float *)dst->dptr + (size_t)row_offset * dst->cols, src->dptr, bytes,
                                       cudaMemcpyDeviceToDevice, ctx->stream));
  return FA_OK;
}

extern "C" int fa_concat_rows(fa_ctx *ctx, const fa_tensor *const *tensors, int count, fa_tensor **out) {
  GLUE_PROLOGUE("concatRows");
  FA_REQUIRE(ctx, tensors && count > 0, "concatRows: empty list");
  int rows = 0, cols = 0;
  for (int i = 0; i < count; i++) {
    FA_TRY(need_f32(ctx, tensors[i], "concatRows"));
    if (i == 0) cols = tensors[i]->cols;
    FA_REQUIRE(ctx, tensors[i]->cols == cols, "concatRows: tensor %d has %d columns, expected %d", i, tensors[i]->cols, cols);
    rows += tensors[i]->rows;
  }
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, rows, cols, FA_F32, true, &y));
  size_t off = 0;
  for (int i = 0; i < count; i++) {
    size_t bytes = (size_t)tensors[i]->rows * cols * 4;
    if (bytes)
      FA_CHECK_CUDA(ctx, cudaMemcpyAsync((char *)y->dptr + off, tensors[i]->dptr, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    off += bytes;
  }
  *out = y;
  return FA_OK;
}

static int sub_reshape_impl(fa_ctx *ctx, const fa_tensor *x, int C, int Tsub, int F, int windows, fa_tensor **out) {
  GLUE_PROLOGUE("subReshape");
  FA_TRY(need_f32(ctx, x, "subReshape"));
  FA_REQUIRE(ctx, C > 0 && Tsub > 0 && F > 0 && windows > 0 && windows <= 65535, "subReshape: bad geometry");
  if (windows == 1)
    FA_REQUIRE(ctx, (long long)x->rows * x->cols >= (long long)C * Tsub * F,
               "subReshape: x has %d elements, need %d*%d*%d", x->rows * x->cols, C, Tsub, F);
  else
    FA_REQUIRE(ctx, x->rows == windows && (long long)x->cols >= (long long)C * Tsub * F,
               "subReshapeWindows: x is [%d,%d], need [%d, >= %d*%d*%d]", x->rows, x->cols, windows, C, Tsub, F);
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, windows * Tsub, C * F, FA_F32, true, &y));
  size_t n = (size_t)Tsub * C * F;
  const int rows = windows * Tsub;
  if ((F & 3) == 0 && rows <= 65535 && (x->cols & 3) == 0 && ((size_t)Tsub * F & 3) == 0 &&
      ((((uintptr_t)x->dptr) | ((uintptr_t)y->dptr)) & 15) == 0) {
    // the result is the row operand of the stem's linear layer: emit it as that (and, when the product is sure to
    // read only that, as nothing else)
    __half *y16 = nullptr;
    float *yp = (float *)y->dptr;
    if (((C * F) & 63) == 0 && fa_tc_available(ctx) && rows >= 16 && (y16 = fa_shadow_block(ctx, y)) != nullptr) {
      y->a16_valid = true;
      if (fa_operand_only_ok(ctx, rows, C * F)) {
        yp = nullptr;
        y->f32_lazy = true;
        y->lazy_sticky = ctx->capturing != nullptr;
      }
    }
    {
      LaunchScope ls(ctx, "sub_reshape");
      const int gx = ceil_div((C * F) >> 2, 256);
      fa_launch_dep(ctx, k_sub_reshape4, dim3(gx < 8 ? gx : 8, rows), dim3(256), 0, (const float *)x->dptr, yp, y16, C, Tsub, F,
                    windows == 1 ? (size_t)0 : (size_t)x->cols, rows);
    }
    FA_LAUNCH_CHECK(ctx, "sub_reshape");
    *out = y;
    return FA_OK;
  }
  {
    LaunchScope ls(ctx, "sub_reshape");
    fa_launch_dep(ctx, k_sub_reshape, dim3(dim3(grid1d(ctx, n, 256), windows)), dim3(256), 0, (const float *)x->dptr, (float *)y->dptr, C,
                                                                              Tsub, F, (size_t)x->cols);
  }
  FA_LAUNCH_CHECK(ctx, "sub_reshape");
  *out = y;
  return FA_OK;
}

extern "C" int fa_sub_reshape(fa_ctx *ctx, const fa_tensor *x, int C, int Tsub, int F, fa_tensor **out) {
  return sub_reshape_impl(ctx, x, C, Tsub, F, 1, out);
}
extern "C" int fa_sub_reshape_windows(fa_ctx *ctx, const fa_tensor *x, int C, int Tsub, int F, int windows,
                                      fa_tensor **out) {
  return sub_reshape_impl(ctx, x, C, Tsub, F, windows, out);
}

extern "C" int fa_rel_shift_b(fa_ctx *ctx, const fa_tensor *x, int H, fa_tensor **out) {
  GLUE_PROLOGUE("relShiftB");
  FA_TRY(need_f32(ctx, x, "relShiftB"));
  FA_REQUIRE(ctx, H > 0 && x->rows % H == 0, "relShiftB: %d rows not divisible by H=%d", x->rows, H);
  const int t = x->rows / H;
  FA_REQUIRE(ctx, x->cols == 2 * t - 1, "relShiftB: x is [%d,%d], expected %d columns", x->rows, x->cols, 2 * t - 1);
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, H * t, t, FA_F32, true, &y));
  size_t n = (size_t)H * t * t;
  if (n) {
    {
      LaunchScope ls(ctx, "rel_shift_b");
      const int rows = H * t, rgrid = rows < ctx->sm_count * 32 ? rows : ctx->sm_count * 32;
      fa_launch_dep(ctx, k_rel_shift_b, dim3(rgrid), dim3(t >= 128 ? 128 : 64), 0, (const float *)x->dptr, (float *)y->dptr, rows, t);
    }
    FA_LAUNCH_CHECK(ctx, "rel_shift_b");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_bmm_qk(fa_ctx *ctx, const fa_tensor *q, const fa_tensor *b, const fa_tensor *qb, int H, int HD, int W,
                         int b_shared, fa_tensor **out) {
  GLUE_PROLOGUE("bmmQK");
  FA_TRY(need_f32(ctx, q, "bmmQK"));
  FA_TRY(need_f32(ctx, b, "bmmQK"));
  if (qb) FA_TRY(need_f32(ctx, qb, "bmmQK"));
  FA_REQUIRE(ctx, H > 0 && HD > 0 && W > 0 && q->cols == H * HD && b->cols == H * HD, "bmmQK: q/b need %d columns", H * HD);
  FA_REQUIRE(ctx, q->rows % W == 0 && (b_shared || b->rows % W == 0), "bmmQK: rows not divisible by W=%d", W);
  if (qb) FA_REQUIRE(ctx, qb->rows * qb->cols >= H * HD, "bmmQK: qb shorter than %d", H * HD);
  const int T = q->rows / W, Tb = b_shared ? b->rows : b->rows / W;
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, W * H * T, Tb, FA_F32, true, &y));
  bool on_tc = false;
  const int lph = HD / 4;
  if (T == 1 && Tb && (HD & 3) == 0 && lph <= 32 && (lph & (lph - 1)) == 0 && W <= 65535) {
    const int strips = ceil_div(H * HD, 128);
    const int U = Tb >= 256 ? 8 : 4;  // rows in flight per warp: 8 on long caches (measured 77 vs 81 us), 4 on short ones
    int gy = ceil_div(ctx->sm_count * 8, strips * W);
    const int gy_max = ceil_div(Tb, 8 * U);
    if (gy > gy_max) gy = gy_max;
    if (gy < 1) gy = 1;
    {
      LaunchScope ls(ctx, "bmm_qk_t1");
      auto kern = U == 8 ? k_bmm_qk_t1<8> : k_bmm_qk_t1<4>;
      fa_launch_dep(ctx, kern, dim3(dim3(strips, gy, W)), dim3(256), 0, (const float *)q->dptr, (const float *)b->dptr,
                                                        qb ? (const float *)qb->dptr : nullptr, (float *)y->dptr, Tb, H,
                                                        HD, b_shared, lph);
    }
    FA_LAUNCH_CHECK(ctx, "bmm_qk_t1");
    *out = y;
    return FA_OK;
  }
  if (T && Tb)
    FA_TRY(fa_tc_bmm_qk(ctx, (const float *)q->dptr, (const float *)b->dptr, b_shared ? const_cast<fa_tensor *>(b) : nullptr,
                        qb ? (const float *)qb->dptr : nullptr, (float *)y->dptr, T, Tb, H, HD, W, b_shared, &on_tc));
  if (T && Tb && !on_tc) {
    dim3 grid(ceil_div(Tb, 64), ceil_div(T, 64), W * H);
    FA_REQUIRE(ctx, grid.z <= 65535 && grid.y <= 65535, "bmmQK: batch too large");
    {
      LaunchScope ls(ctx, "bmm_qk");
      fa_launch_dep(ctx, k_bmm_qk, dim3(grid), dim3(256), 0, (const float *)q->dptr, (const float *)b->dptr,
                                              qb ? (const float *)qb->dptr : nullptr, (float *)y->dptr, T, Tb, H, HD,
                                              b_shared);
    }
    FA_LAUNCH_CHECK(ctx, "bmm_qk");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_bmm_pv(fa_ctx *ctx, const fa_tensor *p, const fa_tensor *v, int H, int HD, int W, fa_tensor **out) {
  GLUE_PROLOGUE("bmmPV");
  FA_TRY(need_f32(ctx, p, "bmmPV"));
  FA_TRY(need_f32(ctx, v, "bmmPV"));
  FA_REQUIRE(ctx, H > 0 && HD > 0 && W > 0 && v->cols == H * HD, "bmmPV: v needs %d columns", H * HD);
  FA_REQUIRE(ctx, v->rows % W == 0 && p->rows % (W * H) == 0, "bmmPV: rows not divisible by W*H");
  const int Tk = v->rows / W, Tq = p->rows / (W * H);
  FA_REQUIRE(ctx, p->cols == Tk, "bmmPV: p has %d columns, v has %d rows per window", p->cols, Tk);
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, W * Tq, H * HD, FA_F32, true, &y));
  bool on_tc = false;
  if (Tq == 1 && Tk && (HD & 3) == 0 && W <= 65535) {
    {
      LaunchScope ls(ctx, "bmm_pv_t1");
      __half *y16 = nullptr;
      size_t lo_off = 0;
      if (((H * HD) & 63) == 0 && fa_tc_available(ctx)) {
        if (W <= ctx->f16_hilo_rows) {
          if ((y16 = fa_shadow_hilo_block(ctx, y)) != nullptr) lo_off = (size_t)((H * HD) >> 6) * W * 64;
        } else {
          y16 = fa_shadow_block(ctx, y);
        }
        if (y16) y->a16_valid = true;
      }
      auto kern = Tk >= 256 ? k_bmm_pv_t1<8> : k_bmm_pv_t1<4>;  // 8 rows in flight: 74 us vs 105 us on 491 MB
      fa_launch_dep(ctx, kern, dim3(dim3(ceil_div(H * HD, 128), 1, W)), dim3(256), 0, (const float *)p->dptr, (const float *)v->dptr,
                                                                      (float *)y->dptr, y16, lo_off, Tk, H, HD);
    }
    FA_LAUNCH_CHECK(ctx, "bmm_pv_t1");
    *out = y;
    return FA_OK;
  }
  if (Tq && Tk)
  {
    __half *y16 = ((H * HD) & 63) == 0 && (HD & 31) == 0 ? fa_shadow_block(ctx, y) : nullptr;
    FA_TRY(fa_tc_bmm_pv(ctx, (const float *)p->dptr, (const float *)v->dptr, (float *)y->dptr, y16, Tq, Tk, H, HD, W, &on_tc));
    if (on_tc && y16) y->a16_valid = true;
  }
  if (Tq && Tk && !on_tc) {
    dim3 grid(ceil_div(HD, 64), ceil_div(Tq, 64), W * H);
    FA_REQUIRE(ctx, grid.z <= 65535 && grid.y <= 65535, "bmmPV: batch too large");
    {
      LaunchScope ls(ctx, "bmm_pv");
      fa_launch_dep(ctx, k_bmm_pv, dim3(grid), dim3(256), 0, (const float *)p->dptr, (const float *)v->dptr, (float *)y->dptr, Tq, Tk, H, HD);
    }
    FA_LAUNCH_CHECK(ctx, "bmm_pv");
  }
  *out = y;
  return FA_OK;
}

static int conv1d_impl(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *w, const fa_tensor *bias, int cout, int k,
                       int stride, int pad_left, int pad_right, int dilation, int groups, int act, int windows,
                       fa_tensor **out) {
  if (!ctx || !out) return fa_fail(ctx, FA_ERR_INVALID, "conv1d: NULL argument");
  FA_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
  FA_TRY(need_f32(ctx, x, "conv1d"));
  FA_TRY(need_f32(ctx, w, "conv1d"));
  if (bias) FA_TRY(need_f32(ctx, bias, "conv1d"));
  const int cin = x->rows, L = x->cols;
  FA_REQUIRE(ctx, cout > 0 && k > 0 && stride > 0 && dilation > 0 && groups > 0 && cin % groups == 0 && cout % groups == 0,
             "conv1d: bad geometry cout=%d k=%d stride=%d dilation=%d groups=%d cin=%d", cout, k, stride, dilation, groups, cin);
  FA_REQUIRE(ctx, (long long)w->rows * w->cols >= (long long)cout * (cin / groups) * k, "conv1d: weight tensor too small");
  if (bias) FA_REQUIRE(ctx, bias->rows * bias->cols >= cout, "conv1d: bias shorter than cout");
  FA_REQUIRE(ctx, windows >= 1 && L % windows == 0, "conv1d: %d columns do not split into %d windows", L, windows);
  const int Lw = L / windows;
  const int Lout_w = (Lw + pad_left + pad_right - dilation * (k - 1) - 1) / stride + 1;
  FA_REQUIRE(ctx, Lout_w > 0, "conv1d: empty output (L=%d)", Lw);
  if (windows > 1)
    FA_REQUIRE(ctx, stride == 1 && Lout_w == Lw, "conv1d: the windowed form needs stride 1 and same-length output");
  const int Lout = Lout_w * windows;
  FA_REQUIRE(ctx, (long long)cout * Lout < (1ll << 31), "conv1d: output too large");
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, cout, Lout, FA_F32, true, &y));
  size_t n = (size_t)cout * Lout;
  if (groups == cin && cout == cin && stride == 1 && Lout == L && cout <= 65535) {
    {
      LaunchScope ls(ctx, "dwconv1d");
      fa_launch_dep(ctx, k_dwconv1d, dim3(dim3(ceil_div(L, 256), cout)), dim3(256), 0, (const float *)x->dptr, (const float *)w->dptr,
                                                                       bias ? (const float *)bias->dptr : nullptr,
                                                                       (float *)y->dptr, L, Lw, k, pad_left, dilation, act);
    }
    FA_LAUNCH_CHECK(ctx, "dwconv1d");
    *out = y;
    return FA_OK;
  }
  {
    LaunchScope ls(ctx, windows > 1 ? "conv1d_windows" : "conv1d");
    fa_launch_dep(ctx, k_conv1d, dim3(grid1d(ctx, n, 128)), dim3(128), 0, (const float *)x->dptr, (const float *)w->dptr,
                                                           bias ? (const float *)bias->dptr : nullptr, (float *)y->dptr,
                                                           cout, cin, L, Lout, Lw, k, stride, pad_left, dilation, groups, act);
  }
  FA_LAUNCH_CHECK(ctx, "conv1d");
  *out = y;
  return FA_OK;
}

extern "C" int fa_attn_fused(fa_ctx *ctx, const fa_tensor *q, const fa_tensor *k, const fa_tensor *v, const fa_tensor *pos,
                             const fa_tensor *pbu, const fa_tensor *pbv, int H, int HD, int W, fa_tensor **out) {
  GLUE_PROLOGUE("attnFused");
  *out = nullptr;
  const fa_tensor *ts[6] = {q, k, v, pos, pbu, pbv};
  for (int i = 0; i < 6; i++) FA_TRY(need_f32(ctx, ts[i], "attnFused"));
  FA_REQUIRE(ctx, H > 0 && HD > 0 && W > 0 && q->rows % W == 0, "attnFused: bad geometry");
  const int T = q->rows / W, S = H * HD;
  FA_REQUIRE(ctx, q->cols == S && k->cols == S && v->cols == S && pos->cols == S && k->rows == q->rows && v->rows == q->rows &&
                      pos->rows == 2 * T - 1 && pbu->rows * pbu->cols >= S && pbv->rows * pbv->cols >= S,
             "attnFused: operand shapes do not match T=%d H=%d HD=%d W=%d", T, H, HD, W);
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, W * T, S, FA_F32, true, &y));
  __half *y16 = (S & 63) == 0 && (HD & 31) == 0 ? fa_shadow_block(ctx, y) : nullptr;
  if (ctx->attn_one_kernel && fa_attn_rel_shape_ok(T, H, HD, W)) {
    // the result feeds the output projection: above the hi/lo row limit its packed operand is all that is written
    float *yp = (float *)y->dptr;
    if (y16 && fa_operand_only_ok(ctx, W * T, S)) {
      yp = nullptr;
      y->f32_lazy = true;
      y->lazy_sticky = ctx->capturing != nullptr;
    }
    int rc1 = fa_attn_rel(ctx, (const float *)q->dptr, (const float *)k->dptr, (const float *)v->dptr, (const float *)pos->dptr,
                          const_cast<fa_tensor *>(pos), (const float *)pbu->dptr, (const float *)pbv->dptr, yp, y16, T, H, HD, W, S);
    if (rc1 != FA_OK) {
      fa_free_tensor(ctx, y);
      return rc1;
    }
    if (y16) y->a16_valid = true;
    *out = y;
    return FA_OK;
  }
  bool done = false;
  int rc = fa_tc_attn_fused(ctx, (const float *)q->dptr, (const float *)k->dptr, (const float *)v->dptr,
                            (const float *)pos->dptr, const_cast<fa_tensor *>(pos), (const float *)pbu->dptr,
                            (const float *)pbv->dptr, (float *)y->dptr, y16, T, H, HD, W, &done);
  if (rc != FA_OK || !done) {  // not this shape: the caller falls back to the separate ops (may return null)
    fa_free_tensor(ctx, y);
    return rc;
  }
  if (y16) y->a16_valid = true;
  *out = y;
  return FA_OK;
}

// attnFused over the columns of ONE fused projection qkv [W*T, 3*H*HD] (q | k | v side by side): the three
// projections of the attention block as one product with the weights concatenated at load time.  One-kernel form
// only; *out stays NULL when the shape is outside its range.
extern "C" int fa_attn_fused_qkv(fa_ctx *ctx, const fa_tensor *qkv, const fa_tensor *pos, const fa_tensor *pbu,
                                 const fa_tensor *pbv, int H, int HD, int W, fa_tensor **out) {
  GLUE_PROLOGUE("attnFusedQKV");
  *out = nullptr;
  FA_REQUIRE(ctx, fa_valid(ctx, qkv) && qkv->storage == FA_F32, "attnFusedQKV: qkv must be an f32-storage tensor");
  // a projection that exists only as its packed f16 operand (matmul with the operand hint) is read as that
  const bool packed = qkv->f32_lazy && qkv->a16_valid && !qkv->a16_hilo && qkv->a16 && !qkv->view;
  if (!packed) FA_TRY(need_f32(ctx, qkv, "attnFusedQKV"));
  const fa_tensor *ts[3] = {pos, pbu, pbv};
  for (int i = 0; i < 3; i++) FA_TRY(need_f32(ctx, ts[i], "attnFusedQKV"));
  FA_REQUIRE(ctx, H > 0 && HD > 0 && W > 0 && qkv->rows % W == 0, "attnFusedQKV: bad geometry");
  const int T = qkv->rows / W, S = H * HD;
  FA_REQUIRE(ctx, qkv->cols == 3 * S && pos->cols == S && pos->rows == 2 * T - 1 && pbu->rows * pbu->cols >= S &&
                      pbv->rows * pbv->cols >= S,
             "attnFusedQKV: operand shapes do not match T=%d H=%d HD=%d W=%d", T, H, HD, W);
  if (!ctx->attn_one_kernel || !fa_attn_rel_shape_ok(T, H, HD, W)) return FA_OK;  // declined
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, W * T, S, FA_F32, true, &y));
  __half *y16 = (S & 63) == 0 ? fa_shadow_block(ctx, y) : nullptr;
  float *yp = (float *)y->dptr;
  if (y16 && fa_operand_only_ok(ctx, W * T, S)) {
    yp = nullptr;
    y->f32_lazy = true;
    y->lazy_sticky = ctx->capturing != nullptr;
  }
  const float *base = packed ? (const float *)qkv->a16 : (const float *)qkv->dptr;
  int rc = fa_attn_rel(ctx, base, base + S, base + 2 * S, (const float *)pos->dptr, const_cast<fa_tensor *>(pos),
                       (const float *)pbu->dptr, (const float *)pbv->dptr, yp, y16, T, H, HD, W, packed ? 0 : 3 * S);
  if (rc != FA_OK) {
    fa_free_tensor(ctx, y);
    return rc;
  }
  if (y16) y->a16_valid = true;
  *out = y;
  return FA_OK;
}

extern "C" int fa_glu_dwconv_tm(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *w, const fa_tensor *bias, int k,
                                int pad_left, int pad_right, int act, int windows, fa_tensor **out) {
  GLUE_PROLOGUE("gluDwConvTimeMajor");
  FA_TRY(need_f32(ctx, x, "gluDwConvTimeMajor"));
  FA_TRY(need_f32(ctx, w, "gluDwConvTimeMajor"));
  if (bias) FA_TRY(need_f32(ctx, bias, "gluDwConvTimeMajor"));
  FA_REQUIRE(ctx, x->cols % 2 == 0 && windows >= 1 && x->rows % windows == 0, "gluDwConvTimeMajor: x is [%d,%d], %d windows",
             x->rows, x->cols, windows);
  const int D = x->cols / 2, rows = x->rows, Tw = rows / windows;
  FA_REQUIRE(ctx, k >= 1 && k <= 16 && pad_left + pad_right == k - 1, "gluDwConvTimeMajor: k=%d pads %d+%d (same-length only)", k,
             pad_left, pad_right);
  FA_REQUIRE(ctx, (long long)w->rows * w->cols >= (long long)D * k, "gluDwConvTimeMajor: weight tensor too small");
  if (bias) FA_REQUIRE(ctx, bias->rows * bias->cols >= D, "gluDwConvTimeMajor: bias shorter than D");
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, rows, D, FA_F32, true, &y));
  if (rows && D) {
    __half *y16 = nullptr;
    if ((D & 63) == 0 && rows >= 16 && fa_tc_available(ctx) && (y16 = fa_shadow_block(ctx, y)) != nullptr) y->a16_valid = true;
    dim3 grid(ceil_div(D, 256), ceil_div(rows, 16));
    FA_REQUIRE(ctx, grid.y <= 65535, "gluDwConvTimeMajor: too many rows");
    {
      LaunchScope ls(ctx, "glu_dwconv_tm");
      const float *bp = bias ? (const float *)bias->dptr : nullptr;
      const int chunks = ceil_div(Tw, 16);
      if (k == 9 && (long long)windows * chunks <= 65535) {
        // the module's next step is a product: above the hi/lo row limit the packed operand is all it reads, so
        // the f32 result stays unwritten until something else asks for it
        float *yp = (float *)y->dptr;
        if (y16 && fa_operand_only_ok(ctx, rows, D)) {
          yp = nullptr;
          y->f32_lazy = true;
          y->lazy_sticky = ctx->capturing != nullptr;
        }
        fa_launch_dep(ctx, k_glu_dwconv_tm_k<9>, dim3(dim3(ceil_div(D, 256), windows * chunks)), dim3(256), 0,
            (const float *)x->dptr, (const float *)w->dptr, bp, yp, y16, rows, Tw, D, pad_left, act, chunks);
      }
      else
        fa_launch_dep(ctx, k_glu_dwconv_tm, dim3(grid), dim3(256), 0, (const float *)x->dptr, (const float *)w->dptr, bp, (float *)y->dptr,
                                                       y16, rows, Tw, D, k, pad_left, act);
    }
    FA_LAUNCH_CHECK(ctx, "glu_dwconv_tm");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_conv1d(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *w, const fa_tensor *bias, int cout, int k,
                         int stride, int pad_left, int pad_right, int dilation, int groups, int act, fa_tensor **out) {
  return conv1d_impl(ctx, x, w, bias, cout, k, stride, pad_left, pad_right, dilation, groups, act, 1, out);
}

extern "C" int fa_conv1d_windows(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *w, const fa_tensor *bias, int cout,
                                 int k, int pad_left, int pad_right, int dilation, int groups, int act, int windows,
                                 fa_tensor **out) {
  return conv1d_impl(ctx, x, w, bias, cout, k, 1, pad_left, pad_right, dilation, groups, act, windows, out);
}

// windows == 1: x holds one image [cin*h*w] (any [rows, cols] with that many elements), out [cout, Ho*Wo].
// windows > 1: x [windows, cin*h*w], one image per row; out [windows, cout*Ho*Wo]; one launch for all of them.
static int conv2d_impl(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *w, const fa_tensor *bias, int cout, int cin,
                       int h, int w_, int kh, int kw, int stride_h, int stride_w, int pad_top, int pad_bottom,
                       int pad_left, int pad_right, int groups, int act, int windows, fa_tensor **out) {
  GLUE_PROLOGUE("conv2d");
  FA_TRY(need_f32(ctx, x, "conv2d"));
  FA_TRY(need_f32(ctx, w, "conv2d"));
  if (bias) FA_TRY(need_f32(ctx, bias, "conv2d"));
  FA_REQUIRE(ctx, cout > 0 && cin > 0 && groups > 0 && cin % groups == 0 && cout % groups == 0 && stride_h > 0 && stride_w > 0,
             "conv2d: bad geometry");
  FA_REQUIRE(ctx, windows >= 1 && windows <= 65535, "conv2d: %d windows", windows);
  if (windows == 1)
    FA_REQUIRE(ctx, (long long)x->rows * x->cols >= (long long)cin * h * w_, "conv2d: input smaller than cin*h*w");
  else
    FA_REQUIRE(ctx, x->rows == windows && (long long)x->cols >= (long long)cin * h * w_,
               "conv2dWindows: x is [%d,%d], need [%d, >= %d]", x->rows, x->cols, windows, cin * h * w_);
  const size_t xstride = windows == 1 ? 0 : (size_t)x->cols;
  FA_REQUIRE(ctx, (long long)w->rows * w->cols >= (long long)cout * (cin / groups) * kh * kw, "conv2d: weight tensor too small");
  const int Ho = (h + pad_top + pad_bottom - kh) / stride_h + 1, Wo = (w_ + pad_left + pad_right - kw) / stride_w + 1;
  FA_REQUIRE(ctx, Ho > 0 && Wo > 0, "conv2d: empty output");
  fa_tensor *y = nullptr;
  if (windows == 1)
    FA_TRY(fa_tensor_new(ctx, cout, Ho * Wo, FA_F32, true, &y));
  else
    FA_TRY(fa_tensor_new(ctx, windows, cout * Ho * Wo, FA_F32, true, &y));
  size_t n = (size_t)cout * Ho * Wo;
  const size_t ystride = n;
  // A pointwise convolution is the product W[cout,cin] @ x[cin, H*W] (the reference routes it to its GEMM
  // plus a per-row bias pass, src/gpu/compute.js:551-555,804-810): run it on the tensor cores with the
  // feature map as the streamed operand and the output-channel bias applied per row in the epilogue.
  const int P = h * w_;
  if (kh == 1 && kw == 1 && stride_h == 1 && stride_w == 1 && groups == 1 && pad_top == 0 && pad_bottom == 0 &&
      pad_left == 0 && pad_right == 0 && fa_tc_available(ctx) && cin >= 64 && P >= 64 &&
      (long long)cout * cin * P >= (1ll << 21)) {
    void *xa = nullptr, *wa = nullptr;
    size_t xb = 0, wb = 0;
    const size_t slab = fa_tc_weight_bytes(P, cin, 2);
    int rc = fa_block_acquire(ctx, slab * windows, &xa, &xb);
    if (rc == FA_OK) rc = fa_block_acquire(ctx, fa_tc_act_bytes(cout, cin, 2, 1), &wa, &wb);
    if (rc == FA_OK) rc = fa_pack_w_f16_batched(ctx, x->dptr, cin, P, windows, xstride, (__half *)xa);
    if (rc == FA_OK) rc = fa_prep_a_f16(ctx, (const float *)w->dptr, cout, cin, (__half *)wa);
    if (rc == FA_OK) {
      TcEpilogue ep;
      ep.rowbias = bias ? (const float *)bias->dptr : nullptr;
      ep.act = act;
      if (windows > 1) {  // one feature map per window against the shared filter bank
        ep.batches = windows;
        ep.a_shared = true;
        ep.o_div = 1;
        ep.o_hi = (long long)ystride;
        ep.ldc = P;
      }
      rc = fa_tc_gemm_f16(ctx, (const __half *)wa, (const __half *)xa, (float *)y->dptr, cout, P, cin, ep);
    }
    if (xa) fa_block_release(ctx, xa);
    if (wa) fa_block_release(ctx, wa);
    if (rc != FA_OK) {
      fa_free_tensor(ctx, y);
      return rc;
    }
    *out = y;
    return FA_OK;
  }
  FA_REQUIRE(ctx, n < (1ull << 31), "conv2d: output too large");
  if (cin == 1 && groups == 1 && kh == 3 && kw == 3 && stride_w <= 3) {
    const unsigned groups4 = (unsigned)Ho * ((Wo + 3) / 4);  // threads: 4 output positions each
    dim3 grid((groups4 + 255) / 256 < (unsigned)ctx->sm_count * 4 ? (groups4 + 255) / 256 : ctx->sm_count * 4,
              ceil_div(cout, 32), windows);
    {
      LaunchScope ls(ctx, "conv2d_c1_3x3");
      auto kern = stride_w == 1 ? k_conv2d_c1_3x3<1> : (stride_w == 2 ? k_conv2d_c1_3x3<2> : k_conv2d_c1_3x3<3>);
      fa_launch_dep(ctx, kern, dim3(grid), dim3(256), 0, (const float *)x->dptr, (const float *)w->dptr,
                                                     bias ? (const float *)bias->dptr : nullptr, (float *)y->dptr, cout, h,
                                                     w_, stride_h, stride_w, pad_top, pad_left, Ho, Wo, act, xstride, ystride);
    }
    FA_LAUNCH_CHECK(ctx, "conv2d_c1_3x3");
    *out = y;
    return FA_OK;
  }
  if (groups == cin && cout == cin && kh == 3 && kw == 3 && cout <= 65535) {
    {
      LaunchScope ls(ctx, "dwconv2d_3x3");
      fa_launch_dep(ctx, k_dwconv2d_3x3, dim3(ceil_div(Ho * ((Wo + 3) / 4), 256), cout, windows), dim3(256), 0,
          (const float *)x->dptr, (const float *)w->dptr, bias ? (const float *)bias->dptr : nullptr, (float *)y->dptr, h,
          w_, stride_h, stride_w, pad_top, pad_left, Ho, Wo, act, xstride, ystride);
    }
    FA_LAUNCH_CHECK(ctx, "dwconv2d_3x3");
    *out = y;
    return FA_OK;
  }
  for (int b = 0; b < windows; b++) {  // general geometry: one launch per window
    LaunchScope ls(ctx, "conv2d");
    fa_launch_dep(ctx, k_conv2d, dim3(grid1d(ctx, n, 128)), dim3(128), 0, (const float *)x->dptr + b * xstride, (const float *)w->dptr,
                                                           bias ? (const float *)bias->dptr : nullptr,
                                                           (float *)y->dptr + b * ystride, cout, cin, h, w_, kh, kw, stride_h,
                                                           stride_w, pad_top, pad_left, Ho, Wo, groups, act);
  }
  FA_LAUNCH_CHECK(ctx, "conv2d");
  *out = y;
  return FA_OK;
}

// conv(1->C, 3x3, s2, p1, relu) -> depthwise(3x3, s2, p1) -> pointwise(C->C, relu): the head of the subsampling
// stem as one member.  The first two layers run fused into the packed operand of the third (k_stem_c1_dw_pack),
// which is the same tensor-core product conv2d_impl makes of a pointwise layer.  *out stays NULL when the
// geometry is not the fused kernel's (image width 128, C a multiple of 64): the caller runs the three members.
extern "C" int fa_conv_stem_windows(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *w0, const fa_tensor *b0,
                                    const fa_tensor *w1, const fa_tensor *b1, const fa_tensor *w2, const fa_tensor *b2,
                                    int C, int h, int w_, int windows, fa_tensor **out) {
  GLUE_PROLOGUE("convStemWindows");
  *out = nullptr;
  FA_TRY(need_f32(ctx, x, "convStemWindows"));
  FA_TRY(need_f32(ctx, w0, "convStemWindows"));
  FA_TRY(need_f32(ctx, w1, "convStemWindows"));
  FA_TRY(need_f32(ctx, w2, "convStemWindows"));
  if (b0) FA_TRY(need_f32(ctx, b0, "convStemWindows"));
  if (b1) FA_TRY(need_f32(ctx, b1, "convStemWindows"));
  if (b2) FA_TRY(need_f32(ctx, b2, "convStemWindows"));
  FA_REQUIRE(ctx, C > 0 && h > 0 && w_ > 0 && windows >= 1 && windows <= 65535, "convStemWindows: bad geometry");
  FA_REQUIRE(ctx, x->rows == windows && (long long)x->cols >= (long long)h * w_, "convStemWindows: x is [%d,%d], need [%d, >= %d]",
             x->rows, x->cols, windows, h * w_);
  FA_REQUIRE(ctx, (long long)w0->rows * w0->cols >= (long long)C * 9 && (long long)w1->rows * w1->cols >= (long long)C * 9 &&
                      (long long)w2->rows * w2->cols >= (long long)C * C,
             "convStemWindows: weight tensor too small");
  FA_REQUIRE(ctx, (!b0 || b0->rows * b0->cols >= C) && (!b1 || b1->rows * b1->cols >= C) && (!b2 || b2->rows * b2->cols >= C),
             "convStemWindows: bias shorter than %d", C);
  const int H1 = (h - 1) / 2 + 1, H2 = (H1 - 1) / 2 + 1, W2 = 32, P = H2 * W2;
  const bool al = ((((uintptr_t)x->dptr) & 15) == 0) && (x->cols & 3) == 0;
  // declined unless conv2d would also run the pointwise layer as the tensor-core product (same size rule)
  if (w_ != 128 || (C & 63) || !fa_tc_available(ctx) || !al || ceil_div(H2, kStemRows) > 65535 || (C >> 6) > 65535 ||
      P < 64 || (long long)C * C * P < (1ll << 21))
    return FA_OK;
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, windows, C * P, FA_F32, true, &y));
  void *xa = nullptr, *wa = nullptr;
  size_t xb = 0, wb = 0;
  const size_t slab = fa_tc_weight_bytes(P, C, 2);
  int rc = fa_block_acquire(ctx, slab * windows, &xa, &xb);
  if (rc == FA_OK) rc = fa_block_acquire(ctx, fa_tc_act_bytes(C, C, 2, 1), &wa, &wb);
  if (rc == FA_OK) {
    static bool attr_set[64] = {false};
    const size_t smem = sizeof(float) * kStemInRows * kStemLd + sizeof(__half) * 2 * 128 * 64;
    if (!attr_set[ctx->device & 63]) {
      cudaFuncSetAttribute(k_stem_c1_dw_pack, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      attr_set[ctx->device & 63] = true;
    }
    {
      LaunchScope ls(ctx, "stem_c1_dw_pack");
      fa_launch_dep(ctx, k_stem_c1_dw_pack, dim3(ceil_div(H2, kStemRows), C >> 6, windows), dim3(256), smem,
                    (const float *)x->dptr, (const float *)w0->dptr, b0 ? (const float *)b0->dptr : nullptr,
                    (const float *)w1->dptr, b1 ? (const float *)b1->dptr : nullptr, (__half *)xa, h, H1, H2,
                    ceil_div(P, 128), fa_tc_chunks(C, 2), (size_t)x->cols, slab / sizeof(__half));
    }
    if (cudaGetLastError() != cudaSuccess) rc = fa_fail(ctx, FA_ERR_CUDA, "stem_c1_dw_pack: launch failed");
  }
  if (rc == FA_OK) rc = fa_prep_a_f16(ctx, (const float *)w2->dptr, C, C, (__half *)wa);
  if (rc == FA_OK) {
    TcEpilogue ep;
    ep.rowbias = b2 ? (const float *)b2->dptr : nullptr;
    ep.act = FA_ACT_RELU;
    ep.batches = windows;
    ep.a_shared = true;
    ep.o_div = 1;
    ep.o_hi = (long long)C * P;
    ep.ldc = P;
    rc = fa_tc_gemm_f16(ctx, (const __half *)wa, (const __half *)xa, (float *)y->dptr, C, P, C, ep);
  }
  if (xa) fa_block_release(ctx, xa);
  if (wa) fa_block_release(ctx, wa);
  if (rc != FA_OK) {
    fa_free_tensor(ctx, y);
    return rc;
  }
  *out = y;
  return FA_OK;
}

// depthwise(3x3, s2, p1) -> pointwise(C->C, relu) over 32-column feature maps x [windows, C*h*32]: the stem's fourth
// and fifth layers as one member (k_dw_s2_pack + the tensor-core product of the pointwise layer).  *out stays NULL
// when the geometry is not the fused kernel's: the caller runs the two members.
extern "C" int fa_conv_dw_pw_windows(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *w1, const fa_tensor *b1,
                                     const fa_tensor *w2, const fa_tensor *b2, int C, int h, int w_, int windows,
                                     fa_tensor **out) {
  GLUE_PROLOGUE("convDwPwWindows");
  *out = nullptr;
  FA_TRY(need_f32(ctx, x, "convDwPwWindows"));
  FA_TRY(need_f32(ctx, w1, "convDwPwWindows"));
  FA_TRY(need_f32(ctx, w2, "convDwPwWindows"));
  if (b1) FA_TRY(need_f32(ctx, b1, "convDwPwWindows"));
  if (b2) FA_TRY(need_f32(ctx, b2, "convDwPwWindows"));
  FA_REQUIRE(ctx, C > 0 && h > 0 && w_ > 0 && windows >= 1 && windows <= 65535, "convDwPwWindows: bad geometry");
  FA_REQUIRE(ctx, (long long)x->rows * x->cols >= (long long)windows * C * h * w_ && (windows == 1 || x->rows == windows),
             "convDwPwWindows: x is [%d,%d], need %d windows of %d*%d*%d", x->rows, x->cols, windows, C, h, w_);
  FA_REQUIRE(ctx, (long long)w1->rows * w1->cols >= (long long)C * 9 && (long long)w2->rows * w2->cols >= (long long)C * C,
             "convDwPwWindows: weight tensor too small");
  FA_REQUIRE(ctx, (!b1 || b1->rows * b1->cols >= C) && (!b2 || b2->rows * b2->cols >= C), "convDwPwWindows: bias shorter than %d", C);
  const int H2 = (h - 1) / 2 + 1, W2 = 16, P = H2 * W2;
  // declined unless conv2d would also run the pointwise layer as the tensor-core product (same size rule)
  if (w_ != 32 || (C & 63) || !fa_tc_available(ctx) || ceil_div(H2, 8) > 65535 || (C >> 6) > 65535 || P < 64 ||
      (long long)C * C * P < (1ll << 21))
    return FA_OK;
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, windows, C * P, FA_F32, true, &y));
  void *xa = nullptr, *wa = nullptr;
  size_t xb = 0, wb = 0;
  const size_t slab = fa_tc_weight_bytes(P, C, 2);
  int rc = fa_block_acquire(ctx, slab * windows, &xa, &xb);
  if (rc == FA_OK) rc = fa_block_acquire(ctx, fa_tc_act_bytes(C, C, 2, 1), &wa, &wb);
  if (rc == FA_OK) {
    {
      LaunchScope ls(ctx, "dw_s2_pack");
      fa_launch_dep(ctx, k_dw_s2_pack, dim3(ceil_div(H2, 8), C >> 6, windows), dim3(256), 0, (const float *)x->dptr,
                    (const float *)w1->dptr, b1 ? (const float *)b1->dptr : nullptr, (__half *)xa, C, h, H2, ceil_div(P, 128),
                    fa_tc_chunks(C, 2), windows == 1 ? (size_t)0 : (size_t)x->cols, slab / sizeof(__half));
    }
    if (cudaGetLastError() != cudaSuccess) rc = fa_fail(ctx, FA_ERR_CUDA, "dw_s2_pack: launch failed");
  }
  if (rc == FA_OK) rc = fa_prep_a_f16(ctx, (const float *)w2->dptr, C, C, (__half *)wa);
  if (rc == FA_OK) {
    TcEpilogue ep;
    ep.rowbias = b2 ? (const float *)b2->dptr : nullptr;
    ep.act = FA_ACT_RELU;
    ep.batches = windows;
    ep.a_shared = true;
    ep.o_div = 1;
    ep.o_hi = (long long)C * P;
    ep.ldc = P;
    rc = fa_tc_gemm_f16(ctx, (const __half *)wa, (const __half *)xa, (float *)y->dptr, C, P, C, ep);
  }
  if (xa) fa_block_release(ctx, xa);
  if (wa) fa_block_release(ctx, wa);
  if (rc != FA_OK) {
    fa_free_tensor(ctx, y);
    return rc;
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_conv2d(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *w, const fa_tensor *bias, int cout, int cin,
                         int h, int w_, int kh, int kw, int stride_h, int stride_w, int pad_top, int pad_bottom,
                         int pad_left, int pad_right, int groups, int act, fa_tensor **out) {
  return conv2d_impl(ctx, x, w, bias, cout, cin, h, w_, kh, kw, stride_h, stride_w, pad_top, pad_bottom, pad_left,
                     pad_right, groups, act, 1, out);
}
extern "C" int fa_conv2d_windows(fa_ctx *ctx, const fa_tensor *x, const fa_tensor *w, const fa_tensor *bias, int cout,
                                 int cin, int h, int w_, int kh, int kw, int stride_h, int stride_w, int pad_top,
                                 int pad_bottom, int pad_left, int pad_right, int groups, int act, int windows,
                                 fa_tensor **out) {
  return conv2d_impl(ctx, x, w, bias, cout, cin, h, w_, kh, kw, stride_h, stride_w, pad_top, pad_bottom, pad_left,
                     pad_right, groups, act, windows, out);
}

extern "C" int fa_embed_rows(fa_ctx *ctx, const fa_tensor *table, const fa_tensor *pos, const fa_tensor *idx, int n,
                             fa_tensor **out) {
  GLUE_PROLOGUE("embedRows");
  FA_TRY(need_f32(ctx, table, "embedRows"));
  FA_TRY(need_f32(ctx, pos, "embedRows"));
  FA_TRY(need_f32(ctx, idx, "embedRows"));
  FA_REQUIRE(ctx, pos->cols == table->cols, "embedRows: table has %d columns, pos has %d", table->cols, pos->cols);
  FA_REQUIRE(ctx, n >= 0 && n < pos->rows, "embedRows: position %d outside [0,%d)", n, pos->rows);
  FA_REQUIRE(ctx, idx->cols >= 1, "embedRows: empty index tensor");
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, idx->rows, table->cols, FA_F32, true, &y));
  if (idx->rows) {
    {
      LaunchScope ls(ctx, "embed_rows");
      fa_launch_dep(ctx, k_embed_rows, dim3(idx->rows), dim3(256), 0, (const float *)table->dptr, (const float *)pos->dptr,
                                                       (const float *)idx->dptr, idx->cols, table->rows, table->cols, n,
                                                       (float *)y->dptr, ctx->dev_status);
    }
    FA_LAUNCH_CHECK(ctx, "embed_rows");
  }
  *out = y;
  return FA_OK;
}

extern "C" int fa_argmax_rows(fa_ctx *ctx, const fa_tensor *x, int ncols, fa_tensor **out) {
  GLUE_PROLOGUE("argmaxRows");
  FA_TRY(need_f32(ctx, x, "argmaxRows"));
  FA_REQUIRE(ctx, x->cols > 0, "argmaxRows: no columns");
  FA_REQUIRE(ctx, ncols <= x->cols, "argmaxRows: %d of %d columns", ncols, x->cols);
  if (ncols <= 0) ncols = x->cols;
  fa_tensor *y = nullptr;
  FA_TRY(fa_tensor_new(ctx, x->rows, 2, FA_F32, true, &y));
  if (x->rows) {
    int grid = x->rows < ctx->sm_count * 8 ? x->rows : ctx->sm_count * 8;
    {
      LaunchScope ls(ctx, "argmax_rows");
      const bool wide = ncols >= 16384 || (ncols >= 8192 && x->rows <= 4 * ctx->sm_count);  // see the kernel
      fa_launch_dep(ctx, wide ? k_argmax_rows<1024, 8> : k_argmax_rows<256, 1>, dim3(grid), dim3(wide ? 1024 : 256), 0, (const float *)x->dptr, (float *)y->dptr, x->rows, x->cols, ncols);
    }
    FA_LAUNCH_CHECK(ctx, "argmax_rows");
  }
  *out = y;
  return FA_OK;
}
