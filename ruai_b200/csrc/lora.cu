// LoRA on a quantized base and the input gradient of the quantized matmul: what the reference's
// QLoRA-style fine-tuning runs on top of the same packed weights.
//
//   Linear::forward with an adapter (src/nn/modules/layers.rs:169-190, add_lora 84-97):
//       y = matmul_int8/int4(x)        (frozen quantized base)
//       y = y + (x @ A @ B) * scale    (A [k, r], B [r, n], scale = alpha / r)
//       y = y + bias
//   Backward of Tensor::matmul_int8 / matmul_int4 (src/nn/ops.rs:705-709, 731-734): the weights are frozen, the
//   only gradient is dx = g @ dequant(W)^T.  The reference materialises the f32 [k, n] weight for it; here tiles of
//   the packed weight are dequantised in shared memory.
// All in f32.
#include "common.cuh"

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = 0.0f;
  for (int i = 0; i < kThreads / 32; ++i) t += red[i];  // fixed order
  return t;
}

// dx[i, rows of chunk c] = sum_j g[i, j] * scale * q[row, j]; chunk layout (pack.cu): few rows, each reading the packed weight
// once for itself.  grid (chunks, m).
template <int BITS>
__global__ void __launch_bounds__(kThreads) grad_input_chunk_kernel(const uint4* __restrict__ w, const float* __restrict__ scale, const float* __restrict__ g,
                                                                    uint32_t k, uint32_t n, float* __restrict__ dx) {
  constexpr int R = BITS == 4 ? 32 : 16;
  __shared__ float red[kThreads / 32];
  const uint32_t c = blockIdx.x, i = blockIdx.y;
  float acc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = 0.0f;
  for (uint32_t j = threadIdx.x; j < n; j += kThreads) {
    const uint4 q = w[(size_t)c * n + j];
    const float v = g[(size_t)i * n + j] * (BITS == 4 ? scale[(size_t)c * n + j] : scale[j]);
    const uint32_t words[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int wi = 0; wi < 4; ++wi) {
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const uint32_t byte = (words[wi] >> (8 * b)) & 0xFFu;
        if (BITS == 4) {  // low nibble: row 4 wi + b, high nibble: row 16 + 4 wi + b, stored value + 8
          acc[4 * wi + b] = fmaf(v, (float)((int)(byte & 0xFu) - 8), acc[4 * wi + b]);
          acc[16 + 4 * wi + b] = fmaf(v, (float)((int)(byte >> 4) - 8), acc[16 + 4 * wi + b]);
        } else {
          acc[4 * wi + b] = fmaf(v, (float)(int)(int8_t)byte, acc[4 * wi + b]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float t = block_sum(acc[r], red);
    const uint32_t row = c * R + r;
    if (threadIdx.x == 0 && row < k) dx[(size_t)i * k + row] = t;
  }
}

// dx[i, r] = sum_j g[i, j] * scale * q[r, j] for the chunk layout (pack.cu): an f32 matrix product on tiles of 64 rows of g x 64 rows of
// W, 16 columns of W at a time through two shared-memory buffers; W is dequantised once per tile instead of once per row of g.  A thread
// owns 8 x 4 results; g is kept twice side by side, so that packed multiply-adds (two f32 in one instruction, each rounded like fmaf)
// need no shuffling: five 16-byte reads from shared memory per 16 of them.  The columns are shared out over gridDim.z CTAs for about
// four CTAs per SM; the shares are added in a fixed order by sum_shares_kernel.  Bound by f32 multiply-adds and their operands'
// reads: 256 x 2048 x 2048 int4 116 us (a row of g at a time: 344 us).  The sums' additions are a fifth of the multiply-adds and
// within what the reads leave free: four CTAs per SM (128 registers) 116 us, three with 158 registers 123.
// Up to here a row at a time is as fast or faster, taken together (us, rows | tiles): 16 rows, 2048 x 2048 int4 28.7 | 28.8, int8 22.6 |
// 28.8, 4096 x 4096 79 | 84 and 64 | 82; 20 rows 33.8 | 29.0, 27.4 | 28.8, 98 | 86, 78 | 84.  Small weights favour the rows for longer
// (512 x 512 int4, 24 rows: 10.3 | 12.4), flat ones the tiles sooner (k 2048, n 512 int4, 14 rows: 17.4 | 14.4).
constexpr uint32_t kGradFewRows = 18;
constexpr int kGradTile = 64, kGradCols = 16, kGradThreads = 128, kGradPad = kGradTile + 4;

__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(0xBF800000BF800000ull), "l"(a));
  return r;
}

template <int BITS>
__global__ void __launch_bounds__(kGradThreads, 4) grad_input_kernel(const uint4* __restrict__ w, const float* __restrict__ scale, const float* __restrict__ g,
                                                                  uint32_t m, uint32_t k, uint32_t n, uint32_t chunks, uint32_t cols_per_share, float* __restrict__ out) {
  constexpr int kChunkRows = BITS == 4 ? 32 : 16, kTileChunks = kGradTile / kChunkRows;
  constexpr int kLoads = kTileChunks * kGradCols / kGradThreads > 0 ? kTileChunks * kGradCols / kGradThreads : 1;  // chunks per thread and step
  constexpr uint32_t kGHalf = kGradCols / 2;
  __shared__ __align__(16) float2 gs[2][kGradCols][kGradTile];
  __shared__ __align__(16) float ws[2][kGradCols][kGradPad];
  const uint32_t tid = threadIdx.x, c0 = blockIdx.x * kTileChunks, i0 = blockIdx.y * kGradTile;
  const uint32_t j_begin = blockIdx.z * cols_per_share, j_end = min(n, j_begin + cols_per_share);
  const uint32_t wj = tid % kGradCols, wc = tid / kGradCols;  // this thread's column and first chunk of a step
  const uint32_t gi = tid / 2, gj = (tid % 2) * kGHalf;       // its row of g and the first of its columns
  uint4 q[kLoads];
  float sc[kLoads], gv[kGHalf];
  auto load = [&](uint32_t j0) {
#pragma unroll
    for (int l = 0; l < kLoads; ++l) {
      const uint32_t c = c0 + wc + l * (kGradThreads / kGradCols), j = j0 + wj;
      const bool in = wc < (uint32_t)kTileChunks && c < chunks && j < j_end;
      q[l] = in ? __ldg(&w[(size_t)c * n + j]) : make_uint4(0, 0, 0, 0);
      sc[l] = in ? __ldg(&scale[BITS == 4 ? (size_t)c * n + j : (size_t)j]) : 0.0f;
    }
#pragma unroll
    for (uint32_t t = 0; t < kGHalf; ++t) gv[t] = i0 + gi < m && j0 + gj + t < j_end ? __ldg(&g[(size_t)(i0 + gi) * n + j0 + gj + t]) : 0.0f;
  };
  auto store = [&](int b) {
    if (wc < (uint32_t)kTileChunks) {
#pragma unroll
      for (int l = 0; l < kLoads; ++l) {
        float* dst = &ws[b][wj][(wc + l * (kGradThreads / kGradCols)) * kChunkRows];
        const uint32_t words[4] = {q[l].x, q[l].y, q[l].z, q[l].w};
#pragma unroll
        for (int wi = 0; wi < 4; ++wi) {
          float lo[4], hi[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const uint32_t byte = (words[wi] >> (8 * t)) & 0xFFu;
            if (BITS == 4) {  // low nibble: row 4 wi + t, high nibble: row 16 + 4 wi + t, stored value + 8
              lo[t] = sc[l] * (float)((int)(byte & 0xFu) - 8);
              hi[t] = sc[l] * (float)((int)(byte >> 4) - 8);
            } else {
              lo[t] = sc[l] * (float)(int)(int8_t)byte;
            }
          }
          *reinterpret_cast<float4*>(dst + 4 * wi) = make_float4(lo[0], lo[1], lo[2], lo[3]);
          if (BITS == 4) *reinterpret_cast<float4*>(dst + 16 + 4 * wi) = make_float4(hi[0], hi[1], hi[2], hi[3]);
        }
      }
    }
#pragma unroll
    for (uint32_t t = 0; t < kGHalf; ++t) gs[b][gj + t][gi] = make_float2(gv[t], gv[t]);
  };
  const uint32_t tr = (tid / 16) * 8, tk = (tid % 16) * 4;  // this thread's 8 rows of g x 4 rows of W
  // Sums of a step's 16 columns, added up; what an addition leaves out (exactly, where the sum so far is the larger) starts the next step's
  // sum, so that the rounding error is that of a chain of 16 however long the share is.  An infinite sum leaves a NaN out: where a sum is
  // not finite in the end, the CTA starts over without.
  unsigned long long acc[8][2], sum[8][2];
  for (bool plain = false;; plain = true) {
#pragma unroll
    for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = sum[r][0] = sum[r][1] = 0ull;
    if (j_begin < j_end) {
      load(j_begin);
      store(0);
    }
    __syncthreads();
    int b = 0;
    for (uint32_t j0 = j_begin; j0 < j_end; j0 += kGradCols, b ^= 1) {
      const bool more = j0 + kGradCols < j_end;
      if (more) load(j0 + kGradCols);
#pragma unroll 8
      for (int j = 0; j < kGradCols; ++j) {
        const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(&ws[b][j][tk]);
#pragma unroll
        for (int r = 0; r < 8; r += 2) {
          const ulonglong2 gp = *reinterpret_cast<const ulonglong2*>(&gs[b][j][tr + r]);
          fma2(acc[r][0], gp.x, wv.x); fma2(acc[r][1], gp.x, wv.y);
          fma2(acc[r + 1][0], gp.y, wv.x); fma2(acc[r + 1][1], gp.y, wv.y);
        }
      }
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const unsigned long long now = add2(sum[r][t], acc[r][t]);
          acc[r][t] = plain ? 0ull : sub2(acc[r][t], sub2(now, sum[r][t]));
          sum[r][t] = now;
        }
      if (more) store(b ^ 1);
      __syncthreads();
    }
    bool finite = true;
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        sum[r][t] = add2(sum[r][t], acc[r][t]);
        finite = finite && isfinite(__uint_as_float((uint32_t)sum[r][t])) && isfinite(__uint_as_float((uint32_t)(sum[r][t] >> 32)));
      }
    if (plain || !__syncthreads_or(!finite)) break;
  }
  float* dst = out + (size_t)blockIdx.z * m * k;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const uint32_t row = i0 + tr + r;
    if (row >= m) break;
#pragma unroll
    for (uint32_t t = 0; t < 4; ++t) {
      const uint32_t kk = c0 * kChunkRows + tk + t;
      if (kk < k) dst[(size_t)row * k + kk] = __uint_as_float((uint32_t)(sum[r][t / 2] >> (32 * (t & 1))));
    }
  }
}

__global__ void __launch_bounds__(kThreads) sum_shares_kernel(const float* __restrict__ part, size_t count, uint32_t shares, float* __restrict__ out) {
  const size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x;
  if (i >= count) return;
  float v = 0.0f, low = 0.0f;  // low: what the additions leave out
  for (uint32_t s0 = 0; s0 < shares; s0 += 8) {
    float a[8];  // requested together
#pragma unroll
    for (uint32_t t = 0; t < 8; ++t) a[t] = s0 + t < shares ? __ldcg(part + (size_t)(s0 + t) * count + i) : 0.0f;
#pragma unroll
    for (uint32_t t = 0; t < 8; ++t) {
      const float now = __fadd_rn(v, a[t]);
      low += __fsub_rn(a[t], __fsub_rn(now, v));
      v = now;
    }
  }
  out[i] = isfinite(low) ? v + low : v;  // an infinite sum leaves no number out
}

// dx for int4 weights kept in the reference layout (groups other than 32): one packed row (two rows of k)
// per block.  grid (k / 2, m).
__global__ void __launch_bounds__(kThreads) grad_input_ref4_kernel(const int8_t* __restrict__ q, const float* __restrict__ scale, const float* __restrict__ g,
                                                                   uint32_t k, uint32_t n, uint32_t group, float* __restrict__ dx) {
  __shared__ float red[kThreads / 32];
  const uint32_t r = blockIdx.x, i = blockIdx.y;
  const float* s0 = scale + (size_t)((2 * r) / group) * n;
  const float* s1 = scale + (size_t)((2 * r + 1) / group) * n;
  float a0 = 0.0f, a1 = 0.0f;
  for (uint32_t j = threadIdx.x; j < n; j += kThreads) {
    const uint8_t b = (uint8_t)q[(size_t)r * n + j];
    const float gv = g[(size_t)i * n + j];
    a0 = fmaf(gv * s0[j], (float)int4_of(b, false), a0);
    a1 = fmaf(gv * s1[j], (float)int4_of(b, true), a1);
  }
  const float t0 = block_sum(a0, red), t1 = block_sum(a1, red);
  if (threadIdx.x == 0) { dx[(size_t)i * k + 2 * r] = t0; dx[(size_t)i * k + 2 * r + 1] = t1; }
}

// t[i, r0 .. r0+7] = sum_p x[i, p] * A[p, r] for kXaRows rows of x, which read A once between them; grid (ceil(m / kXaRows), ceil(rank / 8)).
constexpr int kXaRows = 4;
__global__ void __launch_bounds__(kThreads) lora_xa_kernel(const float* __restrict__ x, const float* __restrict__ a, uint32_t m, uint32_t k, uint32_t rank,
                                                           float* __restrict__ t) {
  __shared__ float red[kThreads / 32][8 * kXaRows];
  const uint32_t i0 = blockIdx.x * kXaRows, r0 = blockIdx.y * 8, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float acc[kXaRows][8];
#pragma unroll
  for (int i = 0; i < kXaRows; ++i)
#pragma unroll
    for (int u = 0; u < 8; ++u) acc[i][u] = 0.0f;
  for (uint32_t p = threadIdx.x; p < k; p += kThreads) {
    float av[8];
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) av[u] = r0 + u < rank ? a[(size_t)p * rank + r0 + u] : 0.0f;
#pragma unroll
    for (int i = 0; i < kXaRows; ++i) {
      const float xv = i0 + i < m ? x[(size_t)(i0 + i) * k + p] : 0.0f;
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[i][u] = fmaf(xv, av[u], acc[i][u]);
    }
  }
#pragma unroll
  for (int i = 0; i < kXaRows; ++i)
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      float v = acc[i][u];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
      if (lane == 0) red[warp][8 * i + u] = v;
    }
  __syncthreads();
  if (threadIdx.x < 8 * kXaRows) {
    const uint32_t i = i0 + threadIdx.x / 8, r = r0 + threadIdx.x % 8;
    float v = 0.0f;
    for (int w = 0; w < kThreads / 32; ++w) v += red[w][threadIdx.x];  // fixed order
    if (i < m && r < rank) t[(size_t)i * rank + r] = v;
  }
}

// y[i, j] = (y[i, j] + (sum_r t[i, r] * B[r, j]) * scale) + bias[j]: the order of layers.rs:175-189.
__global__ void lora_add_kernel(float* __restrict__ y, const float* __restrict__ t, const float* __restrict__ b, const float* __restrict__ bias, uint32_t n,
                                uint32_t rank, float scale) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (j >= n) return;
  float d = 0.0f;
  for (uint32_t r = 0; r < rank; ++r) d = fmaf(t[(size_t)i * rank + r], b[(size_t)r * n + j], d);
  float v = y[(size_t)i * n + j] + d * scale;
  if (bias) v += bias[j];
  y[(size_t)i * n + j] = v;
}

}  // namespace

RUAI_API int ruai_matmul_q_grad_input(ruai_ctx* c, const float* g_dev, const ruai_qweight* w, float* dx_dev, uint32_t m) {
  if (!c || !g_dev || !w || !dx_dev) return ruai_fail(c, RUAI_ERR_ARG, "ruai_matmul_q_grad_input: NULL argument");
  if (w->layout == QL_DENSE) return ruai_fail(c, RUAI_ERR_UNSUPPORTED, "ruai_matmul_q_grad_input: the weight is not quantized");
  if (m == 0) return RUAI_OK;
  if (m > 65535u) return ruai_fail(c, RUAI_ERR_UNSUPPORTED, "ruai_matmul_q_grad_input: %u rows exceed 65535", m);
  DeviceGuard g(c->ordinal);
  if (w->layout == QL_CHUNK16) {
    if (m <= kGradFewRows) {
      const dim3 grid(w->chunks, m);
      if (w->bits == 4) grad_input_chunk_kernel<4><<<grid, kThreads, 0, c->stream>>>((const uint4*)w->data, w->scale, g_dev, w->k, w->n, dx_dev);
      else grad_input_chunk_kernel<8><<<grid, kThreads, 0, c->stream>>>((const uint4*)w->data, w->scale, g_dev, w->k, w->n, dx_dev);
      RUAI_CUDA(c, cudaGetLastError());
      return RUAI_OK;
    }
    const uint32_t row_tiles = (m + kGradTile - 1) / kGradTile, k_tiles = (w->k + kGradTile - 1) / kGradTile, steps = (w->n + kGradCols - 1) / kGradCols;
    // about four CTAs per SM, four steps at least for each
    uint32_t shares = 4u * (uint32_t)c->sm_count / (row_tiles * k_tiles);
    if (shares > steps / 4) shares = steps / 4;
    // Their sums lie in the scratch as every context has it from the start: a call neither allocates nor waits.  A graph would keep the
    // scratch's address, which a later call of another kind may change, so nothing is shared out in a capture.
    const size_t out_bytes = (size_t)m * w->k * sizeof(float);
    if (shares > kScratchBytes / out_bytes) shares = (uint32_t)(kScratchBytes / out_bytes);
    if (shares > 1) {
      cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
      RUAI_CUDA(c, cudaStreamIsCapturing(c->stream, &st));
      if (st != cudaStreamCaptureStatusNone) shares = 1;
    }
    if (shares < 1) shares = 1;
    const uint32_t cols = (steps + shares - 1) / shares * kGradCols;
    shares = (w->n + cols - 1) / cols;
    float* dst = dx_dev;
    if (shares > 1) {
      RUAI_TRY(ruai_ctx_reserve(c, shares * out_bytes, 0));
      dst = c->partial;
    }
    const dim3 grid(k_tiles, row_tiles, shares);
    if (w->bits == 4) grad_input_kernel<4><<<grid, kGradThreads, 0, c->stream>>>((const uint4*)w->data, w->scale, g_dev, m, w->k, w->n, w->chunks, cols, dst);
    else grad_input_kernel<8><<<grid, kGradThreads, 0, c->stream>>>((const uint4*)w->data, w->scale, g_dev, m, w->k, w->n, w->chunks, cols, dst);
    if (shares > 1) {
      RUAI_CUDA(c, cudaGetLastError());
      const size_t count = (size_t)m * w->k;
      sum_shares_kernel<<<(unsigned)((count + kThreads - 1) / kThreads), kThreads, 0, c->stream>>>(dst, count, shares, dx_dev);
    }
  } else {
    if (w->k / 2 > 65535u * 32768u) return ruai_fail(c, RUAI_ERR_UNSUPPORTED, "k too large");
    grad_input_ref4_kernel<<<dim3(w->k / 2, m), kThreads, 0, c->stream>>>((const int8_t*)w->data, w->scale, g_dev, w->k, w->n, w->group, dx_dev);
  }
  RUAI_CUDA(c, cudaGetLastError());
  return RUAI_OK;
}

RUAI_API int ruai_linear_lora_forward(ruai_ctx* c, const float* x_dev, const ruai_qweight* w, const float* lora_a_dev, const float* lora_b_dev,
                                      uint32_t rank, float scale, const float* bias_dev_or_null, float* out_dev, uint32_t m) {
  if (!c || !x_dev || !w || !lora_a_dev || !lora_b_dev || !out_dev) return ruai_fail(c, RUAI_ERR_ARG, "ruai_linear_lora_forward: NULL argument");
  if (rank == 0 || rank > 1024) return ruai_fail(c, RUAI_ERR_SHAPE, "LoRA rank %u must be in 1..1024", rank);
  if (m == 0) return RUAI_OK;
  if (m > 65535u) return ruai_fail(c, RUAI_ERR_UNSUPPORTED, "ruai_linear_lora_forward: %u rows exceed 65535", m);
  DeviceGuard g(c->ordinal);
  // the frozen base first (no bias: the reference adds it after the adapter), then the low-rank path into the scratch
  RUAI_TRY(ruai_matmul_q(c, RUAI_F32, x_dev, w, nullptr, out_dev, m));
  RUAI_TRY(ruai_ctx_reserve(c, (size_t)m * rank * sizeof(float), 0));
  float* t = c->partial;
  lora_xa_kernel<<<dim3((m + kXaRows - 1) / kXaRows, (rank + 7) / 8), kThreads, 0, c->stream>>>(x_dev, lora_a_dev, m, w->k, rank, t);
  RUAI_CUDA(c, cudaGetLastError());
  lora_add_kernel<<<dim3((w->n + 255) / 256, m), 256, 0, c->stream>>>(out_dev, t, lora_b_dev, bias_dev_or_null, w->n, rank, scale);
  RUAI_CUDA(c, cudaGetLastError());
  return RUAI_OK;
}
