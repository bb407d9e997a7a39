// The non-matmul kernels of one decode / prefill step: embedding gather, RMSNorm and
// LayerNorm, RoPE + KV-cache append, attention over the cache, greedy argmax.
//
// They replace the chains of generic elementwise launches the reference's CUDA
// backend issues for the same functions (binary_*/unary_*/reduce_rows_*/cat_copy_*/
// softmax_rows in src/nn/backend/cuda_kernels.cu, driven by src/nn/functional.rs) and
// the host round trips around them (rope tables rebuilt and uploaded every step,
// functional.rs:176-192; logits copied out for the host argmax, generation.rs:104).
// Positions and token ids are read from device memory so that a captured graph of
// the step can be replayed without host involvement.
#include <algorithm>
#include <cmath>

#include "decode_ops.cuh"
#include "pipeline.cuh"

namespace {

constexpr int kAttnWarps = 8;  // at the most

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  return v;
}

// Sum over the CTA (blockDim.x <= 1024, multiple of 32); every thread gets the result.
__device__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = 0.0f;
  for (int i = 0; i < nw; ++i) t += red[i];  // fixed order: deterministic
  return t;
}

// Embedding::forward (layers.rs:436-446); GPT-2 adds wpe[pos] (gpt2.rs:225-226).
// Row r = b*T + t; position = *len + t.
__global__ void embed_kernel(const int32_t* __restrict__ ids, const float* __restrict__ embed, const float* __restrict__ wpe,
                             const int32_t* __restrict__ len, uint32_t T, uint32_t d, uint32_t vocab, float* __restrict__ x,
                             int* __restrict__ err, float* __restrict__ sumsq) {
  __shared__ float red[32];
  grid_dependency_wait();
  grid_launch_dependents();
  const uint32_t r = blockIdx.x;
  int32_t id = ids[r];
  if (id < 0 || (uint32_t)id >= vocab) {  // the reference's index_select would panic; flag it and stay in bounds
    if (threadIdx.x == 0) atomicExch(err, 1);
    id = 0;
  }
  const float* e = embed + (size_t)id * d;
  const float* p = wpe ? wpe + (size_t)(*len + (r % T)) * d : nullptr;
  float ss = 0.0f;
#pragma unroll 8
  for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) {
    const float v = p ? e[i] + p[i] : e[i];
    x[(size_t)r * d + i] = v;
    ss = fmaf(v, v, ss);
  }
  if (sumsq) {  // one tile per row: the sum of squares the next RMSNorm needs
    ss = block_sum(ss, red);
    if (threadIdx.x == 0) sumsq[r] = ss;
  }
}

// F::rms_norm (functional.rs:151-165): x * (1/sqrt(sum(x^2) * (1/d) + eps)) * w.
__global__ void rms_norm_kernel(const float* __restrict__ x, const float* __restrict__ w, uint32_t d, float eps, float* __restrict__ y) {
  __shared__ float red[32];
  grid_dependency_wait();
  grid_launch_dependents();
  const float* xr = x + (size_t)blockIdx.x * d;
  float s = 0.0f;
  for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) s = fmaf(xr[i], xr[i], s);
  s = block_sum(s, red);
  const float rstd = 1.0f / sqrtf(s * (1.0f / (float)d) + eps);
  for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) y[(size_t)blockIdx.x * d + i] = xr[i] * rstd * w[i];
}

// F::layer_norm (functional.rs:137-146) over cpu.rs:855-876: two-pass mean, biased variance.
__global__ void layer_norm_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b, uint32_t d, float eps,
                                  float* __restrict__ y) {
  __shared__ float red[32];
  grid_dependency_wait();
  grid_launch_dependents();
  const float* xr = x + (size_t)blockIdx.x * d;
  float s = 0.0f;
  for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) s += xr[i];
  const float mean = block_sum(s, red) / (float)d;
  float v = 0.0f;
  for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) v = fmaf(xr[i] - mean, xr[i] - mean, v);
  const float rstd = 1.0f / sqrtf(block_sum(v, red) / (float)d + eps);
  for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) y[(size_t)blockIdx.x * d + i] = (xr[i] - mean) * rstd * w[i] + b[i];
}

// rope_cos_sin (functional.rs:176-192): angle = pos * inv_freq in f64, cos/sin rounded to f32.
// table[pos][i] = (cos, sin), i < hd/2.
__global__ void rope_table_kernel(const float* __restrict__ inv_freq, uint32_t half, uint32_t max_pos, float2* __restrict__ table) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)max_pos * half) return;
  const uint32_t pos = (uint32_t)(idx / half), i = (uint32_t)(idx % half);
  const double a = (double)pos * (double)inv_freq[i];
  double s, c;
  sincos(a, &s, &c);
  table[idx] = make_float2((float)c, (float)s);
}

// apply_rope (functional.rs:197-204) on q in place and on k while appending k, v to the
// cache (KvBuf::append, transformer.rs:27-53).  qkv row layout: [q heads | k heads | v heads].
// A CTA per token, a thread per pair (i, i + hd/2) of a head.
constexpr int kRopeThreads = 256;
__global__ void __launch_bounds__(kRopeThreads) rope_kv_kernel(float* __restrict__ qkv, uint32_t qkv_ld, uint32_t k_off, uint32_t v_off, const float2* __restrict__ table,
                               const int32_t* __restrict__ len, uint32_t T, uint32_t Hq, uint32_t KV, uint32_t hd, uint32_t cap,
                               float* __restrict__ kcache, float* __restrict__ vcache, int* __restrict__ status) {
  grid_dependency_wait();
  grid_launch_dependents();
  const uint32_t r = blockIdx.x, b = r / T, t = r % T, half = hd / 2;
  const uint32_t pos = (uint32_t)*len + t;
  float* row = qkv + (size_t)r * qkv_ld;
  const bool over = pos >= cap;  // never write past the cache (see attention_kernel)
  if (over && threadIdx.x == 0 && status) atomicCAS(status, 0, 5);
  const uint32_t begin = table ? 0u : Hq * half, end = (over ? Hq : Hq + KV) * half;
#pragma unroll 4
  for (uint32_t p = begin + threadIdx.x; p < end; p += kRopeThreads) {
    const uint32_t head = p / half, i = p % half;
    const bool key = head >= Hq;
    float* src = key ? row + k_off + (size_t)(head - Hq) * hd : row + (size_t)head * hd;
    const float x1 = src[i], x2 = src[i + half];
    const float2 cs = table ? table[(size_t)pos * half + i] : make_float2(1.0f, 0.0f);
    const size_t at = key ? (((size_t)b * KV + head - Hq) * cap + pos) * hd : 0;
    float* dst = key ? kcache + at : src;
    dst[i] = table ? x1 * cs.x + (-x2) * cs.y : x1;
    dst[i + half] = table ? x2 * cs.x + x1 * cs.y : x2;
    if (key) {
      const float* v = row + v_off + (size_t)(head - Hq) * hd;
      vcache[at + i] = v[i];
      vcache[at + i + half] = v[i + half];
    }
  }
}

// scaled_dot_product_attention over the cache (functional.rs:264-296, llama.rs:248-277):
// softmax(q k^T / sqrt(hd) + causal mask) v.  The `rep` query heads of one KV head are
// handled by one CTA so the cached rows are read once (the reference's [B, H_kv, rep*T, hd]
// view, llama.rs:264-268).
// With p.fuse (single new token per sequence) the kernel also does apply_rope
// (functional.rs:197-204) on q and on the new key and appends the new key / value to the
// cache (KvBuf::append, transformer.rs:27-53): the last key split owns the new position.
//
// Every warp works alone on keys of its own, 32 / LPK at a time, which it copies into its part of shared memory itself (in the fused
// step requested before the grid-dependency wait).  Scores: LPK lanes per key, a part of the head dimension each, against all REP
// query heads (key rows padded by four floats: no bank conflicts; the queries are broadcast); running softmax per head over the
// warp's lanes; values: a lane per four elements, all heads at once.  So a cached element is read from shared memory once per warp,
// and nothing but the warps' results meets at a barrier.  Keys are split over a cluster of gridDim.z CTAs as well; the first one
// merges the results, through distributed shared memory.
// Bound by its warps' latencies: a warp copies, waits, works (64 sequences of 256 keys, 4 key heads of 64 with 8 query heads each: 19 us alone
// and 25 in a step, 5 at the bandwidth; attn_chunks.cu, whose CTAs read every key and value once per head and meet at four barriers a chunk, 36
// and 52).  Where the keys of few items are many, or few query heads share a key, that one is the faster: ruai_attention_plan.
template <int REP, int LPK>  // lanes per key: 1, 2 or 4 for head dimensions up to 64, 128, 256, so that a warp's copy stays below 17 KB
__global__ void __launch_bounds__(kAttnWarps * 32) attention_kernel(const AttnParams p) {
  constexpr int kJ = LPK == 4 ? 2 : 1, kRepPad = REP == 3 ? 4 : REP, kKeys = 32 / LPK;
  extern __shared__ __align__(128) float sm[];
  __shared__ __align__(8) uint64_t bars[kAttnWarps];
  __shared__ float s_m[kAttnWarps][REP], s_l[kAttnWarps][REP];
  const uint32_t hd = p.hd, half = hd / 2, nq4 = hd / 4, kstride = hd + 4, warps = blockDim.x / 32, ns = gridDim.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t per_warp = max((uint32_t)kKeys * (kstride + hd), REP * hd);  // floats: keys, then values; at the end the warp's sums
  float* ks = sm + (size_t)warp * per_warp;
  float* vs = ks + kKeys * kstride;
  float* qs = sm + (size_t)warps * per_warp;                 // [REP][hd]
  float* knew = qs + REP * hd;                               // [hd], then the new value
  float* vnew = knew + hd;
  float* probs = vnew + hd + warp * kKeys * kRepPad;         // [kKeys][kRepPad] per warp
  float* cl = vnew + hd + warps * kKeys * kRepPad;           // the cluster's results: [ns][REP][hd + 4]
  const uint32_t bk = blockIdx.x, b = bk / p.KV, kvh = bk % p.KV, t = blockIdx.y, split = blockIdx.z;
  float* kbase = p.kcache + ((size_t)b * p.KV + kvh) * p.cap * hd;
  float* vbase = p.vcache + ((size_t)b * p.KV + kvh) * p.cap * hd;
  uint64_t* bar = &bars[warp];
  if (lane == 0) {
    pipe::mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  if (ns > 1) pipe::cluster_arrive();  // waited for ahead of the first store into another CTA
  uint32_t pos = 0, k0 = 0, k1 = 0;  // this warp's keys
  bool over = false;
  auto plan = [&]() {
    pos = (uint32_t)*p.len + t;  // causal_mask_offset, functional.rs:238-247
    // The host grows the cache before the step, so a position at or past the capacity means the device's position
    // word is not the host's: touch nothing of the cache, leave an error for the host (the step's output is void).
    over = pos >= p.cap;
    const uint32_t n = over ? 0u : p.fuse ? pos : pos + 1;
    const uint32_t shares = ns * warps, share = split * warps + warp;
    k0 = (uint32_t)((uint64_t)n * share / shares);
    k1 = (uint32_t)((uint64_t)n * (share + 1) / shares);
  };
  auto fetch = [&](uint32_t c0) {  // the whole warp: a lane per key
    const uint32_t nk = min((uint32_t)kKeys, k1 - c0);
    if (lane == 0) pipe::mbar_expect_tx(bar, nk * hd * 8u);
    __syncwarp();
    if ((uint32_t)lane < nk) pipe::bulk_load(ks + lane * kstride, kbase + (size_t)(c0 + lane) * hd, hd * 4u, bar);
    if (lane == 0) pipe::bulk_load(vs, vbase + (size_t)c0 * hd, nk * hd * 4u, bar);
  };
  // In the fused single-token step the cached rows were written by earlier steps, and the position by the
  // previous step's last kernel: both are safe to read while the predecessor (the q/k/v GEMV) still runs.
  if (p.fuse) {
    plan();
    if (k1 > k0) fetch(k0);
  }
  if (tid == 0) trace_min(p.trace, 0);
  grid_dependency_wait();
  if (tid == 0) trace_min(p.trace, 1);
  grid_launch_dependents();
  if (!p.fuse) {
    plan();
    if (k1 > k0) fetch(k0);
  }
  const bool owns_new = p.fuse && split == ns - 1;
  if (over && tid == 0 && p.status) atomicCAS(p.status, 0, 5);
  const float* row = p.q + (size_t)(b * p.T + t) * p.q_ld;
  const bool rot = p.fuse && p.table != nullptr;
  for (uint32_t i = tid; i < (REP + (owns_new ? 2 : 0)) * half; i += blockDim.x) {  // pairs (e, e + half) of the queries, the new key, the new value
    const uint32_t r = i / half, e = i % half;
    const float* src = row + (r < REP ? ((size_t)kvh * REP + r) * hd : r == REP ? p.k_off + (size_t)kvh * hd : p.v_off + (size_t)kvh * hd);
    float x1 = src[e], x2 = src[e + half];
    if (rot && r <= REP) {
      const float2 cs = p.table[(size_t)pos * half + e];
      const float y1 = x1 * cs.x + (-x2) * cs.y;
      x2 = x2 * cs.x + x1 * cs.y;
      x1 = y1;
    }
    float* dst = qs + r * hd;  // the new key and value lie behind the queries
    dst[e] = x1; dst[e + half] = x2;
    if (r >= REP && !over) {
      float* cache = (r == REP ? kbase : vbase) + (size_t)pos * hd;
      cache[e] = x1; cache[e + half] = x2;
    }
  }
  __syncthreads();
  // values: lanes of a row, rows side by side
  const uint32_t lanes = nq4 <= 8 ? 8 : nq4 <= 16 ? 16 : 32, groups = 32 / lanes, vg = lane / lanes, vc = lane % lanes;
  float m[REP], l[REP];  // l: this lane's part
  float4 o[kJ][REP];
#pragma unroll
  for (int r = 0; r < REP; ++r) {
    m[r] = -INFINITY; l[r] = 0.0f;
#pragma unroll
    for (int j = 0; j < kJ; ++j) o[j][r] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (owns_new && warp == 0) {  // the token's own key is the first one
#pragma unroll
    for (int r = 0; r < REP; ++r) {
      float a = 0.0f;
      for (uint32_t e = lane; e < hd; e += 32) a = fmaf(qs[r * hd + e], knew[e], a);
      m[r] = warp_sum(a) * p.scale;
      l[r] = lane == 0 ? 1.0f : 0.0f;
#pragma unroll
      for (int j = 0; j < kJ; ++j)
        if (vg == 0 && vc + 32u * j < nq4) o[j][r] = reinterpret_cast<const float4*>(vnew)[vc + 32u * j];
    }
  }
  uint32_t phase = 0;
  bool ok = true;
  const uint32_t key = lane % kKeys, share = nq4 / LPK;  // this lane's key, and of it `share` 16-byte columns (the last lanes: the rest)
  const uint32_t q_lo = (lane / kKeys) * share, q_hi = lane / kKeys == LPK - 1 ? nq4 : q_lo + share;
  for (uint32_t c0 = k0; c0 < k1; c0 += kKeys) {
    if (c0 != k0) {
      __syncwarp();  // the lanes are done with the last keys
      fetch(c0);
    }
    ok = __all_sync(0xFFFFFFFFu, pipe::mbar_wait(bar, phase & 1u));
    if (!ok) {
      (void)pipe::mbar_wait(bar, phase & 1u);  // whoever gives up: no copy in flight into shared memory that another CTA may get
      break;
    }
    ++phase;
    const uint32_t nk = min((uint32_t)kKeys, k1 - c0);
    const bool valid = key < nk;
    float a0[REP], a1[REP];
#pragma unroll
    for (int r = 0; r < REP; ++r) { a0[r] = 0.0f; a1[r] = 0.0f; }
    const float4* kr = reinterpret_cast<const float4*>(ks + (valid ? key : 0u) * kstride);
    const float4* q4 = reinterpret_cast<const float4*>(qs);
#pragma unroll 4
    for (uint32_t c = q_lo; c < q_hi; ++c) {
      const float4 kv = kr[c];
#pragma unroll
      for (int r = 0; r < REP; ++r) {
        const float4 qv = q4[r * nq4 + c];
        a0[r] = fmaf(qv.x, kv.x, a0[r]); a1[r] = fmaf(qv.y, kv.y, a1[r]); a0[r] = fmaf(qv.z, kv.z, a0[r]); a1[r] = fmaf(qv.w, kv.w, a1[r]);
      }
    }
#pragma unroll
    for (int r = 0; r < REP; ++r) {
      float a = a0[r] + a1[r];
#pragma unroll
      for (int off = kKeys; off < 32; off <<= 1) a += __shfl_xor_sync(0xFFFFFFFFu, a, off);
      const float s = valid ? a * p.scale : -INFINITY;
      const float m_new = fmaxf(m[r], warp_max(s)), m_use = m_new == -INFINITY ? 0.0f : m_new;  // keys with scores of -inf weigh nothing beside others
      const float pr = valid ? expf(s - m_use) : 0.0f, corr = m[r] == -INFINITY ? 0.0f : expf(m[r] - m_new);
      l[r] = fmaf(l[r], corr, lane < kKeys ? pr : 0.0f);
      m[r] = m_new;
#pragma unroll
      for (int j = 0; j < kJ; ++j) { o[j][r].x *= corr; o[j][r].y *= corr; o[j][r].z *= corr; o[j][r].w *= corr; }
      if (lane < kKeys) probs[lane * kRepPad + r] = pr;
    }
    __syncwarp();
#pragma unroll 2
    for (uint32_t k = vg; k < nk; k += groups) {
      float pr[kRepPad];
      if constexpr (kRepPad >= 4) {
#pragma unroll
        for (int r = 0; r < kRepPad; r += 4) *reinterpret_cast<float4*>(pr + r) = *reinterpret_cast<const float4*>(probs + k * kRepPad + r);
      } else {
#pragma unroll
        for (int r = 0; r < kRepPad; ++r) pr[r] = probs[k * kRepPad + r];
      }
#pragma unroll
      for (int j = 0; j < kJ; ++j) {
        if (vc + 32u * j < nq4) {
          const float4 v = reinterpret_cast<const float4*>(vs + (size_t)k * hd)[vc + 32u * j];
#pragma unroll
          for (int r = 0; r < REP; ++r) {
            o[j][r].x = fmaf(pr[r], v.x, o[j][r].x); o[j][r].y = fmaf(pr[r], v.y, o[j][r].y); o[j][r].z = fmaf(pr[r], v.z, o[j][r].z); o[j][r].w = fmaf(pr[r], v.w, o[j][r].w);
          }
        }
      }
    }
  }
  if (!ok && p.status && lane == 0) atomicCAS(p.status, 0, 3);
  // ---- this warp's result, over its lanes, into its part of shared memory: [REP][hd] ----
  __syncwarp();
#pragma unroll
  for (int r = 0; r < REP; ++r) {
    const float lt = warp_sum(l[r]);
    if (lane == 0) { s_m[warp][r] = m[r]; s_l[warp][r] = lt; }
#pragma unroll
    for (int j = 0; j < kJ; ++j) {
      for (uint32_t off = lanes; off < 32; off <<= 1) {
        o[j][r].x += __shfl_xor_sync(0xFFFFFFFFu, o[j][r].x, off); o[j][r].y += __shfl_xor_sync(0xFFFFFFFFu, o[j][r].y, off);
        o[j][r].z += __shfl_xor_sync(0xFFFFFFFFu, o[j][r].z, off); o[j][r].w += __shfl_xor_sync(0xFFFFFFFFu, o[j][r].w, off);
      }
      if (vg == 0 && vc + 32u * j < nq4) reinterpret_cast<float4*>(ks)[r * nq4 + vc + 32u * j] = o[j][r];
    }
  }
  __syncthreads();
  if (ns > 1) pipe::cluster_wait();
  // ---- the warps' results together; several CTAs: to the first one of the cluster ----
  float* out = p.out + (size_t)(b * p.T + t) * p.out_ld + (size_t)kvh * REP * hd;
  for (uint32_t i = tid; i < REP * nq4; i += blockDim.x) {
    const uint32_t r = i / nq4, c = i % nq4;
    float M = -INFINITY, L = 0.0f;
    for (uint32_t w = 0; w < warps; ++w) M = fmaxf(M, s_m[w][r]);
    float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t w = 0; w < warps; ++w) {
      const float f = s_m[w][r] == -INFINITY ? 0.0f : expf(s_m[w][r] - M);
      const float4 v = reinterpret_cast<const float4*>(sm + (size_t)w * per_warp)[i];
      L = fmaf(s_l[w][r], f, L);
      O.x = fmaf(v.x, f, O.x); O.y = fmaf(v.y, f, O.y); O.z = fmaf(v.z, f, O.z); O.w = fmaf(v.w, f, O.w);
    }
    if (ns == 1) {
      const float inv = 1.0f / L;
      reinterpret_cast<float4*>(out)[i] = make_float4(O.x * inv, O.y * inv, O.z * inv, O.w * inv);
    } else {
      float* dst = cl + ((size_t)split * REP + r) * (hd + 4);
      pipe::st_cluster_f4(dst + 4 * c, 0, O);
      if (c == 0) { pipe::st_cluster_f32(dst + hd, 0, M); pipe::st_cluster_f32(dst + hd + 1, 0, L); }
    }
  }
  if (ns > 1) {
    pipe::cluster_sync_all();
    if (split == 0) {
      for (uint32_t i = tid; i < REP * nq4; i += blockDim.x) {
        const uint32_t r = i / nq4, c = i % nq4;
        const float* src = cl + (size_t)r * (hd + 4);
        const uint32_t step = REP * (hd + 4);
        float M = -INFINITY, L = 0.0f;
        for (uint32_t s = 0; s < ns; ++s) M = fmaxf(M, src[s * step + hd]);
        float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t s = 0; s < ns; ++s) {
          const float ms = src[s * step + hd], f = ms == -INFINITY ? 0.0f : expf(ms - M);
          const float4 v = *reinterpret_cast<const float4*>(src + s * step + 4 * c);
          L = fmaf(src[s * step + hd + 1], f, L);
          O.x = fmaf(v.x, f, O.x); O.y = fmaf(v.y, f, O.y); O.z = fmaf(v.z, f, O.z); O.w = fmaf(v.w, f, O.w);
        }
        const float inv = 1.0f / L;
        reinterpret_cast<float4*>(out)[i] = make_float4(O.x * inv, O.y * inv, O.z * inv, O.w * inv);
      }
    }
  }
  if (tid == 0) trace_max(p.trace, 2);
}

// generation::argmax (generation.rs:6-8): the LAST index among equal maxima, in
// total_cmp order (sign-magnitude bits mapped to a signed integer order).
__device__ __forceinline__ int32_t total_order(float v) {
  int32_t i = __float_as_int(v);
  return i ^ (int32_t)(((uint32_t)(i >> 31)) >> 1);
}
__global__ void argmax_kernel(const float* __restrict__ logits, uint32_t ld, uint32_t n, int32_t* __restrict__ out, uint32_t out_offset) {
  __shared__ int32_t sv[32];
  __shared__ uint32_t si[32];
  grid_dependency_wait();
  grid_launch_dependents();
  const float* row = logits + (size_t)blockIdx.x * ld;
  int32_t bv = INT32_MIN;
  uint32_t bi = 0;
  bool any = false;
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    const int32_t v = total_order(row[i]);
    if (!any || v >= bv) { bv = v; bi = i; any = true; }  // ascending i per thread: >= keeps the last
  }
  auto better = [](int32_t v, uint32_t i, bool a, int32_t bv2, uint32_t bi2, bool b2) {
    if (!b2) return false;
    if (!a) return true;
    return bv2 > v || (bv2 == v && bi2 > i);
  };
  for (int o = 16; o > 0; o >>= 1) {
    const int32_t ov = __shfl_xor_sync(0xFFFFFFFFu, bv, o);
    const uint32_t oi = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
    const bool oa = __shfl_xor_sync(0xFFFFFFFFu, (int)any, o) != 0;
    if (better(bv, bi, any, ov, oi, oa)) { bv = ov; bi = oi; any = true; }
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) { sv[w] = any ? bv : INT32_MIN; si[w] = any ? bi : 0xFFFFFFFFu; }
  __syncthreads();
  if (threadIdx.x == 0) {
    int32_t v = INT32_MIN;
    uint32_t idx = 0;
    bool a = false;
    for (int i = 0; i < nw; ++i) {
      if (si[i] == 0xFFFFFFFFu) continue;
      if (!a || sv[i] > v || (sv[i] == v && si[i] > idx)) { v = sv[i]; idx = si[i]; a = true; }
    }
    out[blockIdx.x] = (int32_t)(idx + out_offset);
  }
}

__global__ void add_scalar_kernel(int32_t* p, int32_t v) {
  grid_dependency_wait();
  grid_launch_dependents();
  if (threadIdx.x == 0 && blockIdx.x == 0) *p += v;
}

// Copies rows (b*T + T-1) of x [B*T, d] to y [B, d].
__global__ void take_last_rows_kernel(const float* __restrict__ x, uint32_t T, uint32_t d, float* __restrict__ y) {
  grid_dependency_wait();
  grid_launch_dependents();
  const float* src = x + ((size_t)blockIdx.x * T + T - 1) * d;
  for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) y[(size_t)blockIdx.x * d + i] = src[i];
}

__global__ void take_rows_kernel(const float* __restrict__ x, const int32_t* __restrict__ rows, uint32_t d, float* __restrict__ y) {
  grid_dependency_wait();
  grid_launch_dependents();
  const float* src = x + (size_t)rows[blockIdx.x] * d;
  for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) y[(size_t)blockIdx.x * d + i] = src[i];
}

constexpr size_t kAttnSmemMax = 227 * 1024 - 1024;

uint32_t attn_keys(uint32_t hd) { return hd <= 64 ? 32 : hd <= 128 ? 16 : 8; }  // of a warp at a time
size_t attn_smem(uint32_t rep, uint32_t hd, uint32_t warps, uint32_t splits) {
  const size_t pad = rep == 3 ? 4 : rep, keys = attn_keys(hd);
  return ((size_t)warps * std::max(keys * (2 * hd + 4), (size_t)rep * hd) + (rep + 2) * (size_t)hd + warps * keys * pad +
          (splits > 1 ? (size_t)splits * rep * (hd + 4) : 0)) * sizeof(float);
}

template <int REP, int LPK>
cudaError_t launch_attn(ruai_ctx* c, const AttnParams& p, dim3 grid, uint32_t warps, size_t smem) {
  static bool attr_done[64] = {};
  if (!attr_done[c->ordinal & 63]) {
    cudaError_t e = cudaFuncSetAttribute(attention_kernel<REP, LPK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAttnSmemMax);
    if (e != cudaSuccess) return e;
    attr_done[c->ordinal & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(warps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (c->use_pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (grid.z > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1;
    attr[na].val.clusterDim.y = 1;
    attr[na++].val.clusterDim.z = grid.z;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  c->launches++;
  return cudaLaunchKernelEx(&cfg, attention_kernel<REP, LPK>, p);
}
template <int REP>
cudaError_t launch_attn(ruai_ctx* c, const AttnParams& p, dim3 grid, uint32_t warps, size_t smem) {
  const uint32_t keys = attn_keys(p.hd);
  return keys == 32 ? launch_attn<REP, 1>(c, p, grid, warps, smem) : keys == 16 ? launch_attn<REP, 2>(c, p, grid, warps, smem) : launch_attn<REP, 4>(c, p, grid, warps, smem);
}

}  // namespace

int ruai_embed(ruai_ctx* c, const int32_t* ids, const float* embed, const float* wpe, const int32_t* len, uint32_t rows, uint32_t T, uint32_t d,
               uint32_t vocab, float* x, int* err, float* sumsq) {
  RUAI_CUDA(c, ruai_launch(c, embed_kernel, dim3(rows), dim3(256), 0, true, ids, embed, wpe, len, T, d, vocab, x, err, sumsq));
  return RUAI_OK;
}

int ruai_rms_norm(ruai_ctx* c, const float* x, const float* w, uint32_t rows, uint32_t d, float eps, float* y) {
  RUAI_CUDA(c, ruai_launch(c, rms_norm_kernel, dim3(rows), dim3(d >= 2048 ? 512 : 256), 0, true, x, w, d, eps, y));
  return RUAI_OK;
}

int ruai_layer_norm(ruai_ctx* c, const float* x, const float* w, const float* b, uint32_t rows, uint32_t d, float eps, float* y) {
  RUAI_CUDA(c, ruai_launch(c, layer_norm_kernel, dim3(rows), dim3(256), 0, true, x, w, b, d, eps, y));
  return RUAI_OK;
}

int ruai_rope_table(ruai_ctx* c, const float* inv_freq, uint32_t half, uint32_t max_pos, float2* table) {
  const size_t total = (size_t)max_pos * half;
  rope_table_kernel<<<(unsigned)((total + 255) / 256), 256, 0, c->stream>>>(inv_freq, half, max_pos, table);
  RUAI_CUDA(c, cudaGetLastError());
  return RUAI_OK;
}

int ruai_rope_kv(ruai_ctx* c, float* qkv, uint32_t qkv_ld, uint32_t k_off, uint32_t v_off, const float2* table, const int32_t* len, uint32_t rows,
                 uint32_t T, uint32_t Hq, uint32_t KV, uint32_t hd, uint32_t cap, float* kcache, float* vcache) {
  RUAI_CUDA(c, ruai_launch(c, rope_kv_kernel, dim3(rows), dim3(kRopeThreads), 0, true, qkv, qkv_ld, k_off, v_off, table, len, T, Hq, KV, hd, cap,
                           kcache, vcache, c->status));
  return RUAI_OK;
}

namespace {
// The rounds that `ctas` take on `sms` SMs, per_sm at a time, and the CTAs that share an SM meanwhile.
struct Waves { double rounds, together; };
Waves waves(uint64_t ctas, uint64_t per_sm, double sms) {
  const double q = ctas / (sms * per_sm);
  return {q <= 1 ? 1.0 : q < 4 ? std::ceil(q) : q + 0.5, std::min((double)per_sm, std::max(1.0, std::ceil(ctas / sms)))};
}
double norm4(double a, double b, double c) { return std::sqrt(std::sqrt(a * a * a * a + b * b * b * b + c * c * c * c)); }

// What a launch takes in microseconds, in chunks and with warps that work alone.  A chunk's (a step's) time is the CTA's own, the SM's
// arithmetic or its share of the memory's rate, whichever is longest.  The constants are fitted to 2,300 launches: 13 head shapes (1 to 8 query heads per
// key head, 32 to 256 wide), 1 to 64 sequences of 32 to 32768 positions, 1 to 7 queries; two in three are within 10 %.
double chunks_us(const ruai_ctx* c, uint64_t items, uint32_t rep, uint32_t hd, uint32_t cap, uint32_t splits) {
  const uint64_t ctas = items * splits, sub = ctas > 2u * (uint64_t)c->sm_count ? 1 : 2, threads = 64u * rep * sub;
  const uint64_t per_sm = std::max<uint64_t>(1, std::min({2048 / threads, (uint64_t)(kAttnSmemMax / (ruai_attention_chunk_smem(rep, hd, (uint32_t)sub) + 1024)), 65536 / (80 * threads)}));
  const Waves w = waves(ctas, per_sm, c->sm_count);
  const uint32_t keys = (cap + splits - 1) / splits;
  const double h = hd / 64.0;
  const double chunk = norm4(0.81 + 0.049 * rep * h / sub + 0.2 * rep + 0.51 * h, w.together * 0.2 * (rep * h + 1.5), w.together * 0.54 * h * std::min(keys, 64u) / 64);
  return 0.18 * rep + w.rounds * ((keys + 63) / 64 * chunk + 1.8) + (splits > 1 ? 2.6 + 0.0085 * splits * rep * h : 0.0);
}
double warps_us(const ruai_ctx* c, uint64_t items, uint32_t rep, uint32_t hd, uint32_t cap, uint32_t warps, uint32_t splits) {
  const uint32_t registers = rep == 8 ? 144 : 64 + 8 * rep, shares = splits * warps * attn_keys(hd);
  const uint64_t per_sm = std::max<uint64_t>(1, std::min<uint64_t>(kAttnSmemMax / (attn_smem(rep, hd, warps, splits) + 1024), 65536 / (registers * 32 * warps)));
  // clusters lie within a group of SMs: of eight CTAs that fill an SM each there is room for 15, of four for 33
  const Waves w = waves(items * splits, per_sm, c->sm_count * (splits == 8 ? 120 / 148.0 : splits == 4 ? 132 / 148.0 : 1.0));
  const double h = hd / 64.0, f = attn_keys(hd) / 32.0, busy = w.together * warps;
  const double step = norm4(1.2 + 0.37 * rep + 1.5 * h * f, busy * 0.073 * (rep * h * f + 0.27 * h + 1.5), busy * 0.23 * h * f);
  // a last step of few keys is a short one
  const double full = cap / shares, part = (double)(cap % shares) / shares, steps = std::max(1.0, full + (part > 0 ? 0.35 + 0.65 * part : 0.0));
  return 0.18 * rep + w.rounds * (steps * step + 2.0) + (splits > 1 ? 0.86 + 0.074 * splits : 0.0);
}
}  // namespace

// The warps' numbers with the shortest launch, or chunks where that is not 13 % shorter by the formulas above (less 0.5 us, 1 with few query heads
// per key: behind a step's other launches warps that work alone gain that much on chunks).  Of 489 steps measured (1 to 64 sequences of 40 to 32768
// positions, six head shapes) none is more than 4 % slower than all in chunks, they are 5 % shorter on average, and 1 in 35 is more than 5 % slower than
// all on warps; so are, by up to 24 %, steps of one or two sequences whose cache has room for twice the positions that it holds.  Us of a launch, chunks | warps:
//   8 key heads of 128 with 4 query heads each: 1 sequence, 1024 positions 9.0 | 9.2, 8192 31 | 40, 32768 91 | 160; 16 sequences, 256 20 | 13,
//   1024 42 | 47, 4096 129 | 163;  4 of 64 with 8 each: 1 sequence, 1024 10.2 | 10.7, 32768 77 | 101; 64 sequences, 256 36 | 19, 1024 126 | 65;
//   3 of 64 with 3 each: 1 sequence, 8192 14 | 21; 64 sequences, 256 12.5 | 9.1, 4096 106 | 89;  12 of 64: 64 sequences, 1024 66 | 77
// Up to 64 positions chunks, one for all keys, whose arithmetic a CTA's warps share (4 of 64 with 8 each 6.7 | 8.3); but with one or two query heads
// per key a step is 0.4 to 1.3 us a layer shorter on warps, up to some 500 items (32 sequences of 16 heads: 1.9 longer).
AttnPlan ruai_attention_plan(const ruai_ctx* c, uint32_t B, uint32_t T, uint32_t KV, uint32_t rep, uint32_t hd, uint32_t cap) {
  AttnPlan plan;
  const uint64_t items = (uint64_t)B * KV * T;
  // chunks: one per CTA where the capacity allows it; with many (sequence, KV head) items there are CTAs enough without it
  const uint32_t by_len = (cap + 63) / 64;
  if (T > 1) plan.splits = 1;
  else if (items >= 512) plan.splits = std::max(1u, std::min(by_len, 2u));
  else plan.splits = std::max(1u, std::min(B >= 5 ? (by_len + 1) / 2 : by_len, 64u));
  if (cap <= 64) {
    if (rep <= 2 && items < 512) { plan.warps = 4; plan.splits = 1; }
    return plan;
  }
  double best = 0.87 * chunks_us(c, items, rep, hd, cap, plan.splits) + (rep < 4 ? 1.0 : 0.5);
  for (uint32_t w = 4; w <= (uint32_t)kAttnWarps; w *= 2)
    for (uint32_t s = 1; s <= 8; s *= 2) {
      if (attn_smem(rep, hd, w, s) > kAttnSmemMax) break;
      const double t = warps_us(c, items, rep, hd, cap, w, s);
      if (t < best) { best = t; plan.warps = w; plan.splits = s; }
    }
  return plan;
}

int ruai_attention(ruai_ctx* c, const AttnParams& p_in, uint32_t B, uint32_t rep, const AttnPlan& plan) {
  AttnParams p = p_in;
  p.trace = ruai_trace_slot(c);
  if (p.hd % 4 || p.hd > 256) return ruai_fail(c, RUAI_ERR_UNSUPPORTED, "head_dim %u must be a multiple of 4 and at most 256", p.hd);
  if (rep != 1 && rep != 2 && rep != 3 && rep != 4 && rep != 8) return ruai_fail(c, RUAI_ERR_UNSUPPORTED, "%u query heads per KV head (supported: 1, 2, 3, 4, 8)", rep);
  cudaError_t e;
  if (plan.warps == 0) {
    if (plan.splits > 1 && (!p.scratch || !p.counters)) return ruai_fail(c, RUAI_ERR_ARG, "attention in chunks: no memory for %u splits", plan.splits);
    e = ruai_attention_chunks(c, p, B, rep, plan.splits);
  } else {
    const size_t smem = attn_smem(rep, p.hd, plan.warps, plan.splits);
    const dim3 grid(B * p.KV, p.T, plan.splits);
    switch (rep) {
      case 1: e = launch_attn<1>(c, p, grid, plan.warps, smem); break;
      case 2: e = launch_attn<2>(c, p, grid, plan.warps, smem); break;
      case 3: e = launch_attn<3>(c, p, grid, plan.warps, smem); break;
      case 4: e = launch_attn<4>(c, p, grid, plan.warps, smem); break;
      default: e = launch_attn<8>(c, p, grid, plan.warps, smem); break;
    }
  }
  if (e != cudaSuccess) return ruai_fail(c, RUAI_ERR_CUDA, "attention launch: %s", cudaGetErrorString(e));
  return RUAI_OK;
}

int ruai_argmax(ruai_ctx* c, const float* logits, uint32_t ld, uint32_t rows, uint32_t n, int32_t* out, uint32_t out_offset) {
  RUAI_CUDA(c, ruai_launch(c, argmax_kernel, dim3(rows), dim3(1024), 0, true, logits, ld, n, out, out_offset));
  return RUAI_OK;
}

int ruai_add_scalar(ruai_ctx* c, int32_t* p, int32_t v) {
  RUAI_CUDA(c, ruai_launch(c, add_scalar_kernel, dim3(1), dim3(32), 0, true, p, v));
  return RUAI_OK;
}

int ruai_take_last_rows(ruai_ctx* c, const float* x, uint32_t B, uint32_t T, uint32_t d, float* y) {
  RUAI_CUDA(c, ruai_launch(c, take_last_rows_kernel, dim3(B), dim3(256), 0, true, x, T, d, y));
  return RUAI_OK;
}

int ruai_take_rows(ruai_ctx* c, const float* x, const int32_t* rows, uint32_t n, uint32_t d, float* y) {
  RUAI_CUDA(c, ruai_launch(c, take_rows_kernel, dim3(n), dim3(256), 0, true, x, rows, d, y));
  return RUAI_OK;
}
