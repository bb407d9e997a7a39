// Fused dequantize + GEMV on the integer dot-product units (dp4a) for a few rows of activations: the decode hot path.
//
// Arithmetic.  matmul_int4 / matmul_int8 (src/nn/backend/cpu.rs:1002-1067) are
//     int4: out[i,j] = sum_g scale[g,j] * sum_{l in g} x[i,l] * q[l,j],   int8: out[i,j] = scale[j] * sum_l x[i,l] * q[l,j].
// The activations of a block (int4: a scale group of 32; int8: up to 128 consecutive k) are written as block fixed point,
// x = f * 2^(e - F) with |f| <= 2^F, e from the block's largest magnitude, and f as balanced base-256 digits, each an int8
// (int4: F = 22, three digits; int8: F = 27, four), so that a dp4a multiplies four weights with one digit of four activations,
// exactly.  A block's integer is converted to f32 once and multiplied by its scales.  Stored int4 weights are u = q + 8
// (pack.cu): 8 * sum f is taken off the integer.  Roundings: x to 23 (28) bits of its block's largest magnitude, a block's integer (of up to
// 30 bits) to f32, and the f32 sums of blocks; blocks below 2^-104 (2^-99) keep a quantum of 2^-126.
//
// Organisation.  A CTA of sixteen warps owns TC columns at a time; every warp multiplies a range of k of its own with all of
// them, lane = column (TC below 32: 32 / TC chunks of k side by side), and the warps meet once per tile of columns, to add their
// sums up.  Weights go from memory to registers, kAhead loads per lane ahead of their use, the first ones before the
// grid-dependency wait (they do not depend on the predecessor kernel), and the next tile's behind the current tile's.  RMSNorm
// and LayerNorm of the input ride in the conversion to digits: every CTA reads all of x.
//
// What bounds it, in us of a launch in a chain of launches over weights that are not in the L2, and what the tcgen05 kernels
// (gemv_tc.cu, gemv_tc8.cu) take there.  Small weights: the chain's latency (x, its digits, one trip of weights, the sums):
// int4 576 x 576 2.3 | 3.3, 2048 x 2048 2.7 | 3.9; int8 2.2 | 4.0, 2.7 | 5.4; eight rows of 576 x 576 3.8 | 7.2, 3.9 | 8.0.  There is no
// cluster to launch and join, no tensor memory, no hand-over between warps.  Large ones: int4 the issue slots, 99 instructions of a warp per
// 32 chunks of 16 bytes (4096 x 28672 17.4 | 22.0, 4.2 TB/s); int8 HBM's latency with four loads of a lane in flight (4096 x 28672 25.7 | 31.1,
// 4.6 TB/s; 4096 x 128256 95 | 114, 5.5 TB/s).  Not won: long k with few columns, where the conversion of x in every
// CTA shows, and tiles that do not share out over the SMs (192 of int8 4096 x 6144): ruai_gemv_row_tc.
// Two CTAs of 64 registers per SM (row_kernel spills 8 to 28 bytes a thread, rows_kernel<4, 16> 72 to 76), not one with more and eight loads ahead: alone that is the faster launch (4096 x 28672 18.9 for
// 20.9 then), but a CTA that fills the register file keeps the next kernel's out until it ends, and with it the weights that this would
// request: steps were 10 % slower.
#include <algorithm>

#include "common.cuh"
#include "gemv_epilogue.cuh"
#include "pipeline.cuh"

namespace gemv_dot {

using namespace pipe;

constexpr int kWarps = 16, kThreads = kWarps * 32;
constexpr int kAhead = 4;                                            // weight loads of a lane in flight
constexpr int digits_of(int bits) { return bits == 4 ? 3 : 4; }
constexpr int rows_of(int bits) { return bits == 4 ? 32 : 16; }      // rows of W in a 16-byte chunk
constexpr int pass_chunks(int bits) { return 128 / rows_of(bits); }  // a warp converts 128 values at a time
constexpr int blocks_of(int bits) { return bits == 4 ? 4 : 1; }      // blocks of one exponent among them

struct Params {
  const uint4* w;
  const float* scale;
  const void* x;
  int x_dtype;
  uint32_t x_ld, m, k, n, chunks;
  uint32_t cpw;     // chunks of k per warp
  uint32_t passes;  // conversions of 128 values: per warp (row_kernel), per row (rows_kernel)
  uint32_t steps;   // chunks per lane and tile
  uint32_t iters;   // the same, rounded up to whole groups of loads (and, int8, blocks of an exponent)
  uint32_t tiles;   // of TC columns
  void* out;
  GemvEpilogue epi;
  GemvPrologue pro;
};

// Shared memory: digits, per block of one exponent (its scale, 8 * sum f as bits), the warps' sums [2][warp][row][column].
__host__ __device__ constexpr size_t digit_bytes(int bits, uint32_t passes) { return (size_t)passes * digits_of(bits) * 128; }
__host__ __device__ constexpr size_t meta_bytes(int bits, uint32_t passes) { return (size_t)passes * blocks_of(bits) * 8; }
constexpr size_t red_bytes(int mt, int tc) { return 2 * (size_t)kWarps * mt * tc * 4; }
constexpr size_t kSmemMax = 227 * 1024 - 4096;  // what a CTA can have, less the static part

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  return v;
}
template <int N>
__device__ __forceinline__ float tree(const float* t) {  // their sum, halves added up first: log2 N roundings in a row, not N
  if constexpr (N == 1) return t[0];
  else return tree<(N + 1) / 2>(t) + tree<N / 2>(t + (N + 1) / 2);
}

// Four values from `at` on, whose first k is kk; zeros from k_end on.
__device__ __forceinline__ float4 load4(const void* src, int dtype, size_t at, uint32_t kk, uint32_t k_end, bool vec) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (vec) {
    if (kk < k_end) v = ldg_f4(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(src) + at));
  } else {
    if (kk < k_end) v.x = load_as_f32(src, dtype, at);
    if (kk + 1 < k_end) v.y = load_as_f32(src, dtype, at + 1);
    if (kk + 2 < k_end) v.z = load_as_f32(src, dtype, at + 2);
    if (kk + 3 < k_end) v.w = load_as_f32(src, dtype, at + 3);
  }
  return v;
}
__device__ __forceinline__ bool aligned4(const Params& p) {
  return p.x_dtype == RUAI_F32 && (p.x_ld & 3u) == 0 && (p.k & 3u) == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15u) == 0 &&
         ((reinterpret_cast<uintptr_t>(p.pro.norm_w) | reinterpret_cast<uintptr_t>(p.pro.norm_b)) & 15u) == 0;
}

// The digits of a lane's four values, most significant first, and the (scale, 8 * sum f as bits) of the block that the lane is in: of
// 128 values of the warp, or, int4, of 32 of eight lanes.
template <int BITS>
__device__ __forceinline__ float2 to_digits(const float4& xv, uint32_t (&digit)[digits_of(BITS)]) {
  // magnitudes compared as integers: an infinity or a NaN comes out largest
  uint32_t mx = max(max(__float_as_uint(xv.x) & 0x7FFFFFFFu, __float_as_uint(xv.y) & 0x7FFFFFFFu), max(__float_as_uint(xv.z) & 0x7FFFFFFFu, __float_as_uint(xv.w) & 0x7FFFFFFFu));
  if (BITS == 4) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
  } else {
    mx = __reduce_max_sync(0xFFFFFFFFu, mx);
  }
  // mx < 2^e with e = biased exponent - 126; f = round(x * 2^(F - e)).  Not finite: the block's scale becomes NaN and with it this
  // row's sums, as f32 arithmetic would (cpu.rs:1002-1067)
  constexpr uint32_t F = BITS == 4 ? 22 : 27;
  const uint32_t eb = mx >> 23, ec = max(eb, F);
  const bool fin = eb < 255u;
  const float up = fin ? __uint_as_float((253u + F - ec) << 23) : 0.0f;
  const float scale = fin ? __uint_as_float((ec - F + 1u) << 23) : __int_as_float(0x7fc00000);
  // balanced digits are the bytes of f + 0x80..80, the lower ones with their top bit turned
  constexpr uint32_t kBias = BITS == 4 ? 0x8080u : 0x808080u;
  const int f0 = __float2int_rn(xv.x * up), f1 = __float2int_rn(xv.y * up), f2 = __float2int_rn(xv.z * up), f3 = __float2int_rn(xv.w * up);
  const uint32_t g0 = ((uint32_t)f0 + kBias) ^ kBias, g1 = ((uint32_t)f1 + kBias) ^ kBias, g2 = ((uint32_t)f2 + kBias) ^ kBias, g3 = ((uint32_t)f3 + kBias) ^ kBias;
  const uint32_t a01 = __byte_perm(g0, g1, 0x5140), a23 = __byte_perm(g2, g3, 0x5140);  // bytes 0 and 1 of two values each
  const uint32_t b01 = __byte_perm(g0, g1, 0x7362), b23 = __byte_perm(g2, g3, 0x7362);  // bytes 2 and 3
  constexpr int D = digits_of(BITS);
  digit[D - 1] = __byte_perm(a01, a23, 0x5410);
  digit[D - 2] = __byte_perm(a01, a23, 0x7632);
  digit[D - 3] = __byte_perm(b01, b23, 0x5410);
  if (BITS == 8) digit[0] = __byte_perm(b01, b23, 0x7632);
  int fs = 0;
  if (BITS == 4) {
    fs = (f0 + f1) + (f2 + f3);
    fs += __shfl_xor_sync(0xFFFFFFFFu, fs, 1);
    fs += __shfl_xor_sync(0xFFFFFFFFu, fs, 2);
    fs += __shfl_xor_sync(0xFFFFFFFFu, fs, 4);
  }
  return make_float2(scale, __int_as_float(8 * fs));
}

__device__ __forceinline__ int32_t dot16(const int (&w)[4], const unsigned char* digits, int32_t d) {
  const int4 x = *reinterpret_cast<const int4*>(digits);
  d = __dp4a(w[0], x.x, d); d = __dp4a(w[1], x.y, d); d = __dp4a(w[2], x.z, d);
  return __dp4a(w[3], x.w, d);
}
// A chunk of int4: its integer, from digits that lie `stride` bytes apart.
struct Nibbles {
  int lo[4], hi[4];
  __device__ __forceinline__ explicit Nibbles(const uint4& w)
      : lo{(int)(w.x & 0x0F0F0F0Fu), (int)(w.y & 0x0F0F0F0Fu), (int)(w.z & 0x0F0F0F0Fu), (int)(w.w & 0x0F0F0F0Fu)},
        hi{(int)((w.x >> 4) & 0x0F0F0F0Fu), (int)((w.y >> 4) & 0x0F0F0F0Fu), (int)((w.z >> 4) & 0x0F0F0F0Fu), (int)((w.w >> 4) & 0x0F0F0F0Fu)} {}
  __device__ __forceinline__ int32_t dot(const unsigned char* digits, int stride, int32_t eight_sum) const {
    int32_t d = 0;
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      d = t == 0 ? 0 : (int32_t)((uint32_t)d << 8) - (t == 2 ? eight_sum : 0);
      d = dot16(hi, digits + t * stride + 16, dot16(lo, digits + t * stride, d));
    }
    return d;
  }
};
// Int8: from the sums by digit, of which the upper and the lower two fit 32 bits together.
__device__ __forceinline__ float joined(const int32_t (&d)[4]) { return fmaf((float)(d[0] * 256 + d[1]), 65536.0f, (float)(d[2] * 256 + d[3])); }

// What the epilogue of a row will need of column j, requested ahead of the products.
struct Operands { float bias, resid, scale; };
template <int BITS>
__device__ __forceinline__ Operands operands(const Params& p, bool in, size_t out_row, uint32_t j) {
  const GemvEpilogue& e = p.epi;
  Operands o = {0.0f, 0.0f, 1.0f};
  if (in) {
    if (e.bias) o.bias = e.bias[j];
    if (BITS == 8) o.scale = p.scale[j];
    if (e.resid) o.resid = e.resid[out_row + (e.act == ACT_SWIGLU ? j >> 1 : j)];
  }
  return o;
}
struct Best { int32_t v = INT32_MIN, j = -1; };  // greedy pick: a lane's best column
// The sum v of column j in every lane of the column; lane `sub` 0 writes it.
template <int BITS>
__device__ __forceinline__ void finish(const Params& p, float v, const Operands& o, uint32_t row, size_t out_row, uint32_t tile, uint32_t j, bool active,
                                       int sub, Best& best) {
  const GemvEpilogue& e = p.epi;
  if (BITS == 8) v *= o.scale;
  v += o.bias;
  if (e.act == ACT_SWIGLU) {  // columns (2i, 2i+1) hold (gate_i, up_i): layers.rs:573-576
    const float other = __shfl_xor_sync(0xFFFFFFFFu, v, 1);
    if (sub == 0 && active && (j & 1u) == 0) store_from_f32(p.out, e.out_dtype, out_row + (j >> 1), o.resid + silu_ref(v) * other);
    return;
  }
  if (e.act == ACT_GELU) v = gelu_ref(v);
  if (e.resid) v = o.resid + v;
  if (sub == 0 && active) store_from_f32(p.out, e.out_dtype, out_row + j, v);
  if (e.sumsq) {  // of this tile's part of the stored row
    const float t = warp_sum(sub == 0 && active ? v * v : 0.0f);
    if ((threadIdx.x & 31) == 0) e.sumsq[(size_t)tile * p.m + row] = t;
  }
  if (e.argmax_out && active) {  // ties go to the larger column
    const int32_t bits = ordered_bits(v);
    if (bits >= best.v) { best.v = bits; best.j = (int32_t)j; }
  }
}
__device__ __forceinline__ void best_of_warp(int32_t& v, int32_t& j) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int32_t ov = __shfl_xor_sync(0xFFFFFFFFu, v, o), oj = __shfl_xor_sync(0xFFFFFFFFu, j, o);
    if (ov > v || (ov == v && oj > j)) { v = ov; j = oj; }
  }
}
// The CTAs' best columns (warp r holds row r's); the last CTA to finish picks the winners and advances the position.
__device__ __forceinline__ void pick(const Params& p, Best best) {
  const GemvEpilogue& e = p.epi;
  __shared__ unsigned s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < (int)p.m) {
    best_of_warp(best.v, best.j);
    if (lane == 0) e.argmax_slots[(size_t)blockIdx.x * p.m + warp] = make_int2(best.v, best.j);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(e.argmax_counter, 1u) == gridDim.x - 1 ? 1u : 0u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const volatile int* slots = (const volatile int*)e.argmax_slots;
  if (warp < (int)p.m) {
    int32_t v = INT32_MIN, j = -1;
    for (uint32_t t = lane; t < gridDim.x; t += 32) {
      const int tv = slots[2 * ((size_t)t * p.m + warp)], tj = slots[2 * ((size_t)t * p.m + warp) + 1];
      if (tv > v || (tv == v && tj > j)) { v = tv; j = tj; }
    }
    best_of_warp(v, j);
    if (lane == 0) e.argmax_out[warp] = j;
  }
  if (threadIdx.x == 0) {
    *e.argmax_counter = 0;
    if (e.len_ptr) *e.len_ptr += e.len_add;
  }
}

// One row.  A warp converts the activations of its own range of k itself, into its own part of shared memory, and starts with its
// products as soon as these have arrived: no CTA-wide wait ahead of them.  Digits [warp][pass][digit][128].
template <int BITS, int TC>
__global__ void __launch_bounds__(kThreads, 2) row_kernel(const Params p) {
  constexpr int kSubs = 32 / TC, kDigits = digits_of(BITS), kRows = rows_of(BITS), kPass = pass_chunks(BITS), kBlocks = blocks_of(BITS);
  constexpr int kBatch = 2;  // conversions whose activations are loaded together
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ float s_sum[kWarps], s_var[kWarps];
  unsigned char* dig = smem;
  float2* meta = reinterpret_cast<float2*>(smem + digit_bytes(BITS, kWarps * p.passes));
  float* red = reinterpret_cast<float*>(smem + digit_bytes(BITS, kWarps * p.passes) + meta_bytes(BITS, kWarps * p.passes));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int col = lane % TC, sub = lane / TC;
  const uint32_t c_begin = min(p.chunks, (uint32_t)warp * p.cpw), nch = min(p.chunks, c_begin + p.cpw) - c_begin;

  // ---- weights: iteration i of a tile is chunk c_begin + i * kSubs + sub; kAhead of them are in flight ----
  const uint32_t mine = nch > (uint32_t)sub ? (nch - sub + kSubs - 1) / kSubs : 0u;  // this lane's chunks
  const size_t step = (size_t)kSubs * p.n;
  const size_t first = (size_t)(c_begin + sub) * p.n + col;  // of column tile 0
  uint4 wq[kAhead];
  float sq[kAhead];
  auto load = [&](size_t at, bool in, uint4& w, float& s) {  // beyond the slice the old weights stay; int4: with a scale of zero, int8: the digits are zero
    if (in) w = ldg_stream_u4(p.w + at);
    if (BITS == 4) s = in ? ldg_stream_f32(p.scale + at) : 0.0f;
  };
  {
    const size_t at = first + (size_t)blockIdx.x * TC;
    const uint32_t limit = blockIdx.x * TC + col < p.n ? mine : 0u;
#pragma unroll
    for (int a = 0; a < kAhead; ++a) {
      wq[a] = make_uint4(0, 0, 0, 0);
      load(at + a * step, (uint32_t)a < limit, wq[a], sq[a]);
    }
  }

  const bool normed = p.pro.norm_w != nullptr, layer_norm = p.pro.norm_b != nullptr;
  const uint32_t k_begin = c_begin * kRows, k_end = min(p.k, (c_begin + nch) * kRows);
  if (normed && k_begin + 4 * lane < k_end) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p.pro.norm_w + k_begin + 4 * lane));
    if (layer_norm) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.pro.norm_b + k_begin + 4 * lane));
  }
  if (tid == 0) trace_min(p.pro.trace, 0);
  grid_dependency_wait();
  if (tid == 0) trace_min(p.pro.trace, 1);
  grid_launch_dependents();

  // ---- this warp's activations as digits ----
  const bool vec = aligned4(p);
  auto load_x = [&](uint32_t pass) {
    const uint32_t kk = k_begin + pass * 128 + 4 * lane;
    return load4(p.x, p.x_dtype, kk, kk, k_end, vec);
  };
  float mean = 0.0f, rstd = 1.0f, part = 0.0f;
  if (layer_norm) {  // mean and variance in two passes, as layer_norm_kernel
    for (uint32_t pass = 0; pass < p.passes; ++pass) {
      const float4 v = load_x(pass);
      part += (v.x + v.y) + (v.z + v.w);
    }
    part = warp_sum(part);
    if (lane == 0) s_sum[warp] = part;
    __syncthreads();
    mean = tree<kWarps>(s_sum) / (float)p.k;
    part = 0.0f;
    for (uint32_t pass = 0; pass < p.passes; ++pass) {
      const uint32_t left = k_end - min(k_end, k_begin + pass * 128 + 4 * lane);
      const float4 v = load_x(pass);
      const float a = left > 0 ? v.x - mean : 0.0f, b = left > 1 ? v.y - mean : 0.0f, c = left > 2 ? v.z - mean : 0.0f, d = left > 3 ? v.w - mean : 0.0f;
      part = fmaf(a, a, fmaf(b, b, fmaf(c, c, fmaf(d, d, part))));
    }
    part = warp_sum(part);
    if (lane == 0) s_var[warp] = part;
    __syncthreads();
    rstd = 1.0f / sqrtf(tree<kWarps>(s_var) / (float)p.k + p.pro.eps);
    part = 0.0f;
  }
  for (uint32_t p0 = 0; p0 < p.passes; p0 += kBatch) {
    float4 v[kBatch], nw[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const uint32_t kk = k_begin + (p0 + b) * 128 + 4 * lane;
      v[b] = load_x(p0 + b);
      nw[b] = normed ? load4(p.pro.norm_w, RUAI_F32, kk, kk, k_end, vec) : make_float4(1.f, 1.f, 1.f, 1.f);
    }
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const uint32_t pass = p0 + b;
      if (pass >= p.passes) break;
      float4 xv = v[b];
      if (layer_norm) {  // zero weights past the end of k make those values zero
        const uint32_t kk = k_begin + pass * 128 + 4 * lane;
        const float4 nb = load4(p.pro.norm_b, RUAI_F32, kk, kk, k_end, vec);
        xv.x = fmaf((xv.x - mean) * rstd, nw[b].x, nb.x); xv.y = fmaf((xv.y - mean) * rstd, nw[b].y, nb.y);
        xv.z = fmaf((xv.z - mean) * rstd, nw[b].z, nb.z); xv.w = fmaf((xv.w - mean) * rstd, nw[b].w, nb.w);
      } else if (normed) {  // RMSNorm: 1 / rms is one factor per row and multiplies the finished sums
        part = fmaf(xv.x, xv.x, fmaf(xv.y, xv.y, fmaf(xv.z, xv.z, fmaf(xv.w, xv.w, part))));
        xv.x *= nw[b].x; xv.y *= nw[b].y; xv.z *= nw[b].z; xv.w *= nw[b].w;
      }
      uint32_t digit[kDigits];
      const float2 mt = to_digits<BITS>(xv, digit);
      const uint32_t item = warp * p.passes + pass;
      uint32_t* dst = reinterpret_cast<uint32_t*>(dig + (size_t)item * (kDigits * 128)) + lane;
#pragma unroll
      for (int t = 0; t < kDigits; ++t) dst[t * 32] = digit[t];
      if (lane % (32 / kBlocks) == 0) meta[item * kBlocks + lane / (32 / kBlocks)] = mt;
    }
  }
  if (normed && !layer_norm) {
    part = warp_sum(part);
    if (lane == 0) s_sum[warp] = part;  // read behind the first tile's barrier
  }
  __syncwarp();

  // ---- tiles of columns ----
  Best best;
  uint32_t buf = 0;
  for (uint32_t tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, buf ^= 1u) {
    const uint32_t j = tile * TC + col;
    const bool active = j < p.n;
    const Operands ops = operands<BITS>(p, warp == 0 && active, 0, j);
    float acc = 0.0f;
    int32_t d8[4] = {0, 0, 0, 0};
    const uint32_t next = tile + gridDim.x;
    for (uint32_t i0 = 0; i0 < p.iters; i0 += kAhead) {
      // the loads kAhead further on: this tile's, or the next one's
      const bool wrap = i0 + kAhead >= p.iters;
      const uint32_t li = wrap ? 0u : i0 + kAhead, lt = wrap ? next : tile;
      const uint32_t limit = lt < p.tiles && lt * TC + col < p.n ? mine : 0u;
      const size_t at = first + (size_t)lt * TC + li * step;
      // kAhead * kSubs chunks of digits; whole passes but for int8 with kSubs = 1, half ones
      const uint32_t lc0 = i0 * kSubs + sub;
      const unsigned char* blk0 = dig + ((size_t)warp * p.passes + i0 * kSubs / kPass) * (kDigits * 128) + (i0 * kSubs % kPass + sub) * kRows;
      const float2* meta0 = meta + (size_t)warp * p.passes * kBlocks + (BITS == 4 ? lc0 : lc0 / kPass);
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {
        if (i0 + a < p.steps) {
          const unsigned char* blk = blk0 + (a * kSubs / kPass) * (kDigits * 128) + (a * kSubs % kPass) * kRows;
          const uint4 w = wq[a];
          if constexpr (BITS == 4) {
            const float2 mt = meta0[a * kSubs];
            acc = fmaf((float)Nibbles(w).dot(blk, 128, __float_as_int(mt.y)), sq[a] * mt.x, acc);
          } else {
            const int wi[4] = {(int)w.x, (int)w.y, (int)w.z, (int)w.w};
#pragma unroll
            for (int t = 0; t < 4; ++t) d8[t] = dot16(wi, blk + t * 128, d8[t]);
          }
        }
        if constexpr (BITS == 8) {
          // the end of a block of one exponent: kBlock chunks per lane, of which the first one exists
          constexpr int kBlock = kPass / kSubs;
          const bool ends = kAhead >= kBlock ? (a + 1) % kBlock == 0 : a + 1 == kAhead && (i0 + kAhead) % kBlock == 0;
          if (ends && i0 + a + 1 < p.steps + kBlock) {
            acc = fmaf(joined(d8), meta0[a * kSubs / kPass].x, acc);
            d8[0] = d8[1] = d8[2] = d8[3] = 0;
          }
        }
        load(at + a * step, li + a < limit, wq[a], sq[a]);
      }
    }
#pragma unroll
    for (int o = TC; o < 32; o <<= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
    if (sub == 0) red[((size_t)buf * kWarps + warp) * TC + col] = acc;
    __syncthreads();
    if (warp == 0) {
      constexpr int kMine = kWarps / kSubs;  // warps whose sums this lane adds up
      float t[kMine];
#pragma unroll
      for (int w = 0; w < kMine; ++w) t[w] = red[((size_t)buf * kWarps + sub * kMine + w) * TC + col];
      float v = tree<kMine>(t);
#pragma unroll
      for (int o = TC; o < 32; o <<= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
      if (normed && !layer_norm) v *= 1.0f / sqrtf(tree<kWarps>(s_sum) * (1.0f / (float)p.k) + p.pro.eps);
      finish<BITS>(p, v, ops, 0, 0, tile, j, active, sub, best);
    }
  }
  if (p.epi.argmax_out) pick(p, best);
  if (tid == 0) trace_max(p.pro.trace, 2);
}

// Up to sixteen rows of short k.  The warps share the conversions, of which there are more than warps' ranges of k would give.  Digits
// [row][chunk][digit][rows of the chunk]; sums of squares [row][pass].
template <int BITS, int MT, int TC>
__global__ void __launch_bounds__(kThreads, 1) rows_kernel(const Params p) {
  constexpr int kSubs = 32 / TC, kDigits = digits_of(BITS), kRows = rows_of(BITS), kBlocks = blocks_of(BITS);
  constexpr int kChunkBytes = kDigits * kRows, kPerBlock = BITS == 4 ? 1 : 8;  // chunks of a block of one exponent
  constexpr int kBatch = 4;  // conversions whose activations are loaded together
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ float2 s_norm[MT];  // LayerNorm: mean, 1 / deviation
  unsigned char* dig = smem;
  float2* meta = reinterpret_cast<float2*>(smem + digit_bytes(BITS, MT * p.passes));
  float* part = reinterpret_cast<float*>(smem + digit_bytes(BITS, MT * p.passes) + meta_bytes(BITS, MT * p.passes));
  float* red = part + MT * p.passes;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int col = lane % TC, sub = lane / TC;
  const uint32_t m0 = blockIdx.y * MT, rows = min((uint32_t)MT, p.m - m0);
  const uint32_t c_begin = min(p.chunks, (uint32_t)warp * p.cpw), nch = min(p.chunks, c_begin + p.cpw) - c_begin;

  // ---- the first weights ----
  const uint32_t mine = nch > (uint32_t)sub ? (nch - sub + kSubs - 1) / kSubs : 0u;  // this lane's chunks
  const size_t step = (size_t)kSubs * p.n;
  const size_t first = (size_t)(c_begin + sub) * p.n + col;  // of column tile 0
  uint4 wq[kAhead];
  float sq[kAhead];
  auto load = [&](size_t at, bool in, uint4& w, float& s) {  // beyond the slice the old weights stay; int4: with a scale of zero, int8: not multiplied
    if (in) w = ldg_stream_u4(p.w + at);
    if (BITS == 4) s = in ? ldg_stream_f32(p.scale + at) : 0.0f;
  };
  {
    const size_t at = first + (size_t)blockIdx.x * TC;
    const uint32_t limit = blockIdx.x * TC + col < p.n ? mine : 0u;
#pragma unroll
    for (int a = 0; a < kAhead; ++a) {
      wq[a] = make_uint4(0, 0, 0, 0);
      load(at + a * step, (uint32_t)a < limit, wq[a], sq[a]);
    }
  }
  const bool normed = p.pro.norm_w != nullptr, layer_norm = p.pro.norm_b != nullptr;
  if (normed)
    for (uint32_t i = tid * 32; i < p.k; i += kThreads * 32) {  // a line each
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p.pro.norm_w + i));
      if (layer_norm) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.pro.norm_b + i));
    }
  if (tid == 0) trace_min(p.pro.trace, 0);
  grid_dependency_wait();
  if (tid == 0) trace_min(p.pro.trace, 1);
  grid_launch_dependents();

  // ---- activations as digits: item = row * passes + pass, warp w takes every kWarps-th from w on ----
  const bool vec = aligned4(p);
  const uint32_t items = rows * p.passes;
  auto load_x = [&](uint32_t r, uint32_t kk) { return load4(p.x, p.x_dtype, (size_t)(m0 + r) * p.x_ld + kk, kk, p.k, vec); };
  if (layer_norm) {  // warp r: mean and variance of row r, in two passes, as layer_norm_kernel
    if (warp < (int)rows) {
      float t = 0.0f, u = 0.0f;
#pragma unroll 4
      for (uint32_t pass = 0; pass < p.passes; ++pass) {
        const float4 v = load_x(warp, pass * 128 + 4 * lane);
        t += (v.x + v.y) + (v.z + v.w);
      }
      const float mean = warp_sum(t) / (float)p.k;
#pragma unroll 4
      for (uint32_t pass = 0; pass < p.passes; ++pass) {
        const uint32_t kk = pass * 128 + 4 * lane, left = p.k - min(p.k, kk);
        const float4 v = load_x(warp, kk);
        const float a = left > 0 ? v.x - mean : 0.0f, b = left > 1 ? v.y - mean : 0.0f, c = left > 2 ? v.z - mean : 0.0f, d = left > 3 ? v.w - mean : 0.0f;
        u = fmaf(a, a, fmaf(b, b, fmaf(c, c, fmaf(d, d, u))));
      }
      u = warp_sum(u);
      if (lane == 0) s_norm[warp] = make_float2(mean, 1.0f / sqrtf(u / (float)p.k + p.pro.eps));
    }
    __syncthreads();
  }
  for (uint32_t i0 = warp; i0 < items; i0 += kBatch * kWarps) {
    float4 v[kBatch], nw[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const uint32_t item = i0 + b * kWarps, r = item / p.passes, kk = (item - r * p.passes) * 128 + 4 * lane;
      if (item < items) {
        v[b] = load_x(r, kk);
        if (normed) nw[b] = load4(p.pro.norm_w, RUAI_F32, kk, kk, p.k, vec);
      }
    }
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const uint32_t item = i0 + b * kWarps, r = item / p.passes, kk = (item - r * p.passes) * 128 + 4 * lane;
      if (item >= items) break;
      float4 xv = v[b];
      if (layer_norm) {  // weights of zero past k make those values zero
        const float mean = s_norm[r].x, rstd = s_norm[r].y;
        const float4 nb = load4(p.pro.norm_b, RUAI_F32, kk, kk, p.k, vec);
        xv.x = fmaf((xv.x - mean) * rstd, nw[b].x, nb.x); xv.y = fmaf((xv.y - mean) * rstd, nw[b].y, nb.y);
        xv.z = fmaf((xv.z - mean) * rstd, nw[b].z, nb.z); xv.w = fmaf((xv.w - mean) * rstd, nw[b].w, nb.w);
      } else if (normed) {  // RMSNorm: 1 / rms is one factor per row and multiplies the finished sums
        const float t = warp_sum(fmaf(xv.x, xv.x, fmaf(xv.y, xv.y, fmaf(xv.z, xv.z, xv.w * xv.w))));
        if (lane == 0) part[item] = t;
        xv.x *= nw[b].x; xv.y *= nw[b].y; xv.z *= nw[b].z; xv.w *= nw[b].w;
      }
      uint32_t digit[kDigits];
      const float2 mt = to_digits<BITS>(xv, digit);
      constexpr int kLanes = kRows / 4;  // lanes of a chunk
      uint32_t* dst = reinterpret_cast<uint32_t*>(dig + (size_t)item * (kDigits * 128) + (lane / kLanes) * kChunkBytes) + lane % kLanes;
#pragma unroll
      for (int t = 0; t < kDigits; ++t) dst[t * kLanes] = digit[t];
      if (lane % (32 / kBlocks) == 0) meta[item * kBlocks + lane / (32 / kBlocks)] = mt;
    }
  }
  __syncthreads();

  // ---- tiles of columns ----
  const uint32_t row_bytes = p.passes * (kDigits * 128), row_meta = p.passes * kBlocks;
  const size_t out_row = (size_t)(m0 + warp) * p.epi.out_ld;
  const uint32_t d_begin = c_begin + sub;  // this lane's first chunk; a range of k begins with a block
  Best best;
  uint32_t buf = 0;
  for (uint32_t tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, buf ^= 1u) {
    const uint32_t j = tile * TC + col;
    const bool active = j < p.n;
    const Operands ops = operands<BITS>(p, warp < (int)rows && active, out_row, j);
    float acc[MT];
    int32_t d8[MT][4];  // int8: sums by digit
#pragma unroll
    for (int r = 0; r < MT; ++r) {
      acc[r] = 0.0f;
      d8[r][0] = d8[r][1] = d8[r][2] = d8[r][3] = 0;
    }
    const uint32_t next = tile + gridDim.x;
    for (uint32_t i0 = 0; i0 < p.iters && nch; i0 += kAhead) {
      const bool wrap = i0 + kAhead >= p.iters;
      const uint32_t li = wrap ? 0u : i0 + kAhead, lt = wrap ? next : tile;
      const uint32_t limit = lt < p.tiles && lt * TC + col < p.n ? mine : 0u;
      const size_t at = first + (size_t)lt * TC + li * step;
      const unsigned char* dig0 = dig + (size_t)(d_begin + i0 * kSubs) * kChunkBytes;
      const float2* meta0 = meta + (d_begin + i0 * kSubs) / kPerBlock;
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {
        if (i0 + a < p.steps) {
          const uint4 w = wq[a];
          if constexpr (BITS == 4) {
            const Nibbles nib(w);
#pragma unroll
            for (int r = 0; r < MT; ++r) {
              const float2 mt = meta0[r * row_meta + a * kSubs];
              acc[r] = fmaf((float)nib.dot(dig0 + r * row_bytes + a * kSubs * kChunkBytes, kRows, __float_as_int(mt.y)), sq[a] * mt.x, acc[r]);
            }
          } else {
            const int wi[4] = {(int)w.x, (int)w.y, (int)w.z, (int)w.w};
#pragma unroll
            for (int r = 0; r < MT; ++r)
#pragma unroll
              for (int t = 0; t < 4; ++t) d8[r][t] = dot16(wi, dig0 + r * row_bytes + a * kSubs * kChunkBytes + t * kRows, d8[r][t]);
          }
        }
        if constexpr (BITS == 8) {
          constexpr int kBlock = kPerBlock / kSubs;
          const bool ends = kAhead >= kBlock ? (a + 1) % kBlock == 0 : a + 1 == kAhead && (i0 + kAhead) % kBlock == 0;
          if (ends && i0 + a + 1 < p.steps + kBlock) {
#pragma unroll
            for (int r = 0; r < MT; ++r) {
              acc[r] = fmaf(joined(d8[r]), meta0[r * row_meta + a * kSubs / kPerBlock].x, acc[r]);
              d8[r][0] = d8[r][1] = d8[r][2] = d8[r][3] = 0;
            }
          }
        }
        load(at + a * step, li + a < limit, wq[a], sq[a]);
      }
    }
#pragma unroll
    for (int r = 0; r < MT; ++r) {
#pragma unroll
      for (int o = TC; o < 32; o <<= 1) acc[r] += __shfl_xor_sync(0xFFFFFFFFu, acc[r], o);
      if (sub == 0) red[((size_t)buf * kWarps + warp) * MT * TC + r * TC + col] = acc[r];
    }
    __syncthreads();
    if (warp < (int)rows) {  // row m0 + warp
      constexpr int kMine = kWarps / kSubs;  // warps whose sums this lane adds up
      float t[kMine];
#pragma unroll
      for (int w = 0; w < kMine; ++w) t[w] = red[((size_t)buf * kWarps + sub * kMine + w) * MT * TC + warp * TC + col];
      float v = tree<kMine>(t);
#pragma unroll
      for (int o = TC; o < 32; o <<= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
      if (normed && !layer_norm) {  // a lane per pass: k of rows_kernel is below 32 passes
        const float ss = warp_sum(lane < (int)p.passes ? part[warp * p.passes + lane] : 0.0f);
        v *= 1.0f / sqrtf(ss * (1.0f / (float)p.k) + p.pro.eps);
      }
      finish<BITS>(p, v, ops, m0 + warp, out_row, tile, j, active, sub, best);
    }
  }
  if (p.epi.argmax_out) pick(p, best);
  if (tid == 0) trace_max(p.pro.trace, 2);
}

cudaError_t launch_kernel(ruai_ctx* c, void (*kernel)(Params), bool* done, const Params& p, dim3 grid, size_t smem) {
  if (!done[c->ordinal & 63]) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
    if (e != cudaSuccess) return e;
    done[c->ordinal & 63] = true;
  }
  return ruai_launch(c, kernel, grid, dim3(kThreads), smem, true, p);
}
template <int BITS, int MT, int TC>
cudaError_t launch_one(ruai_ctx* c, const Params& p, dim3 grid, size_t smem) {
  static bool done[64] = {};
  if constexpr (MT == 1) return launch_kernel(c, row_kernel<BITS, TC>, done, p, grid, smem);
  else return launch_kernel(c, rows_kernel<BITS, MT, TC>, done, p, grid, smem);
}
template <int BITS, int MT>
cudaError_t launch_tc(ruai_ctx* c, const Params& p, dim3 grid, size_t smem, uint32_t tc) {
  return tc == 32 ? launch_one<BITS, MT, 32>(c, p, grid, smem) : tc == 16 ? launch_one<BITS, MT, 16>(c, p, grid, smem) : launch_one<BITS, MT, 8>(c, p, grid, smem);
}
template <int BITS>
cudaError_t launch_mt(ruai_ctx* c, const Params& p, dim3 grid, size_t smem, int mt, uint32_t tc) {
  switch (mt) {
    case 1: return launch_tc<BITS, 1>(c, p, grid, smem, tc);
    case 2: return launch_tc<BITS, 2>(c, p, grid, smem, tc);
    case 4: return launch_tc<BITS, 4>(c, p, grid, smem, tc);
    case 8: return launch_tc<BITS, 8>(c, p, grid, smem, tc);
    default:
      if constexpr (BITS == 4) return launch_tc<BITS, 16>(c, p, grid, smem, tc);
      else return cudaErrorInvalidValue;
  }
}

struct Shape { uint32_t tc, cpw, passes, steps, iters, tiles, per_sm; int mt; size_t smem; };
Shape shape_of(const ruai_ctx* c, const ruai_qweight* w, uint32_t m) {
  Shape s;
  const int bits = (int)w->bits;
  const uint32_t sms = (uint32_t)c->sm_count, pass = (uint32_t)pass_chunks(bits);
  // Rows in one tile, but for sixteen where the columns leave half of the SMs idle.  Of the columns the narrowest tiles that an SM gets
  // one of at the most; 32 where that takes several rounds.  One row of long k: 16 up to two tiles per SM (int4 4096 x 4096 4.7 us, with 32
  // columns 4.9, int8 5.6, 6.3; with k of 2048 and 2560 columns the other way round for int4, 3.3 and 2.9).
  s.mt = m <= 1 ? 1 : m <= 2 ? 2 : m <= 4 ? 4 : m <= 8 || bits == 8 || w->n * 2 <= 16 * sms ? 8 : 16;
  const uint32_t wide = sms / ((m + s.mt - 1) / s.mt);
  s.tc = w->n <= 8 * wide ? 8 : w->n <= 16 * wide || (s.mt == 1 && w->k >= 4096 && w->n <= 32 * wide) ? 16 : 32;
  s.tiles = (w->n + s.tc - 1) / s.tc;
  const uint32_t subs = 32 / s.tc;
  // a warp's range of k; where the warps share the conversions it begins with a block of one exponent
  const uint32_t unit = s.mt == 1 ? (bits == 4 ? 1u : 2u) : bits == 4 ? subs : 8u;
  s.cpw = (w->chunks + kWarps * unit - 1) / (kWarps * unit) * unit;
  s.steps = (s.cpw + subs - 1) / subs;
  const uint32_t group = std::max<uint32_t>(kAhead, bits == 8 ? pass / subs : 1u);
  s.iters = (s.steps + group - 1) / group * group;
  // one row: per warp; several: of all chunks that a range holds, past the end of k too
  s.passes = ((s.mt == 1 ? s.steps * subs : (w->chunks + s.cpw - 1) / s.cpw * s.cpw) + pass - 1) / pass;
  const uint32_t all = s.mt == 1 ? kWarps * s.passes : s.mt * s.passes;
  s.smem = digit_bytes(bits, all) + meta_bytes(bits, all) + (s.mt == 1 ? 0 : (size_t)all * 4) + red_bytes(s.mt, s.tc);
  s.per_sm = s.mt == 1 && s.smem <= kSmemMax / 2 ? 2 : 1;
  return s;
}

// What one row of int8 takes, in microseconds: fitted to 213 shapes, k of 512 to 28672 and 512 to 32768 columns, in a chain of launches over weights that are
// not in the L2 (one standard deviation 6 %, as that of the tensor-core kernel's formula).
double row_us(const ruai_ctx* c, const ruai_qweight* w, const Shape& s) {
  const uint32_t sms = (uint32_t)c->sm_count, ctas = std::min(s.tiles, s.per_sm * sms);
  const double side = std::min<double>(s.per_sm, (s.tiles + sms - 1) / sms), rounds = (s.tiles + ctas - 1) / ctas;  // CTAs on an SM, tiles of a CTA
  return std::max(0.37 + 0.35 * s.passes * side + rounds * std::max(0.25 * s.steps + 1.2, 0.15 * s.steps * side) + 0.65 * (side - 1), 0.19e-6 * w->k * w->n);
}

}  // namespace gemv_dot

// One row of int8 by itself: the tensor-core kernel where its launch is the shorter one by the formulas, in one of five shapes: where the tiles of columns
// leave SMs with one more than others while that kernel's CTAs all find a place.  Us, here | there:  4096 x 4096 5.7 | 6.6, 4096 x 28672 25.7 | 31.1,
// 14336 x 2048 11.5 | 14.7;  4096 x 6144 8.3 | 7.5, 4096 x 12288 15.0 | 11.6, 11008 x 6144 20.7 | 14.8.  Over all shapes the choice takes 0.79 of that
// kernel's time and 0.97 of this one's; errors against 64 bits are equal (5.2e-8 to 9.0e-8 there, 6.5e-8 to 8.5e-8 here).
// Not in a decoder's step, where the norm rides along here and a change of kernels costs their overlap: steps of the 8B shape (4 layers) 357 us, with the
// choice 375.  Not int4: a few shapes are shorter on gemv_tc.cu (14336 x 4096 13.4 | 12.3, 28672 x 4096 24.7 | 21.9, 11008 x 3072 10.3 | 9.5), but its 21 bits
// err by 1.0e-6 to 2.0e-6 where the 23 here do by 2.6e-7 to 5.1e-7.
bool ruai_gemv_row_tc(const ruai_ctx* c, const ruai_qweight* w) {
  using namespace gemv_dot;
  if (w->layout != QL_CHUNK16 || w->bits != 8 || !ruai_gemv_tc8_eligible(w, 1)) return false;
  const Shape s = shape_of(c, w, 1);
  return s.smem > kSmemMax || row_us(c, w, s) > ruai_gemv_tc8_row_us(c, w);
}

// One row of int4 whose columns are a multiple of four, and of int8 with k up to 32768.  Others are served by f32 multiply-adds (gemv.cu, gemv_bulk.cu),
// which keep what a block of one exponent rounds away.  Several rows: as long as the dp4a of all of them cost less than the tensor cores' fixed parts, which is with short k
// (digits for all of k have to be made first) and few weights.  Us of a launch, here | gemv_tc.cu or gemv_tc8.cu:
//   int4, 2 rows: 576 x 576 2.5 | 3.8, 768 x 3072 2.8 | 4.4;  2048 x 2560 4.6 | 4.8, 3072 x 768 5.2 | 4.6, 5632 x 2048 8.2 | 6.9
//   int4, 4 rows: 576 x 576 3.2 | 5.0, 768 x 3072 3.7 | 5.5, 1536 x 576 4.0 | 5.2;  2048 x 2048 6.0 | 5.8, 3072 x 768 8.2 | 5.6
//   int4, 8 rows: 576 x 576 3.8 | 7.2, 768 x 3072 4.9 | 8.1, 1536 x 576 5.6 | 7.7;  2048 x 2048 9.2 | 8.9
//   int4, 16 rows: 576 x 576 3.8 | 7.5, 768 x 3072 8.4 | 9.0, 1536 x 576 5.7 | 8.0;  2048 x 2048 16.3 | 10.7
//   int8, 4 rows: 576 x 576 3.4 | 5.6, 768 x 2304 3.7 | 5.8;  768 x 3072 7.1 | 5.9
//   int8, 16 rows: 576 x 576 4.0 | 8.1, 768 x 2304 6.3 | 8.6;  768 x 3072 13.6 | 8.8
bool ruai_gemv_dot_takes(const ruai_ctx* c, const ruai_qweight* w, uint32_t m) {
  using namespace gemv_dot;
  if (!c->use_bulk || !c->use_tc || w->layout != QL_CHUNK16 || m == 0) return false;
  if (w->bits == 4 && (w->group != 32 || w->n % 4)) return false;
  if (w->bits == 8 && w->k > 32768) return false;
  if (m > 1 && (m > 16 || w->k > 1536 || (uint64_t)w->k * w->n > (5u << 19))) return false;
  if (m > 2 && w->bits == 8 && w->n > 16u * (uint32_t)c->sm_count) return false;
  return shape_of(c, w, m).smem <= kSmemMax;
}

uint32_t ruai_gemv_dot_tiles(const ruai_ctx* c, const ruai_qweight* w, uint32_t m) { return gemv_dot::shape_of(c, w, m).tiles; }

int ruai_gemv_dot_launch(ruai_ctx* c, const ruai_qweight* w, const void* x, int x_dtype, uint32_t x_ld, uint32_t m, void* out, const GemvEpilogue& epi_in,
                         const GemvPrologue& pro) {
  using namespace gemv_dot;
  GemvEpilogue epi = epi_in;
  if (epi.act == ACT_SWIGLU && (w->n & 1)) return ruai_fail(c, RUAI_ERR_SHAPE, "SwiGLU epilogue needs an even column count, got %u", w->n);
  if (epi.out_ld == 0) epi.out_ld = epi.act == ACT_SWIGLU ? w->n / 2 : w->n;
  if (epi.sumsq && epi.act == ACT_SWIGLU) return ruai_fail(c, RUAI_ERR_UNSUPPORTED, "sum of squares with the SwiGLU epilogue");
  if (epi.argmax_out && (m > kGemvDotPickRows || epi.act == ACT_SWIGLU)) return ruai_fail(c, RUAI_ERR_UNSUPPORTED, "fused argmax needs m <= %u", kGemvDotPickRows);
  const Shape s = shape_of(c, w, m);
  Params p;
  p.w = (const uint4*)w->data; p.scale = w->scale; p.x = x; p.x_dtype = x_dtype; p.x_ld = x_ld;
  p.m = m; p.k = w->k; p.n = w->n; p.chunks = w->chunks; p.cpw = s.cpw; p.passes = s.passes; p.steps = s.steps; p.iters = s.iters; p.tiles = s.tiles;
  p.out = out; p.epi = epi; p.pro = pro;
  p.pro.trace = ruai_trace_slot(c);
  // Tiles in turn over all CTAs that fit: an SM then has at most one tile more than another.  (The fewest CTAs with the same number each
  // left SMs with twice the tiles of others: int4 4096 x 28672 20.6 us for 17.4, 2048 x 11264 6.5 for 5.2.)
  const dim3 grid(std::min(s.tiles, s.per_sm * (uint32_t)c->sm_count), (m + s.mt - 1) / s.mt);
  const cudaError_t e = w->bits == 4 ? launch_mt<4>(c, p, grid, s.smem, s.mt, s.tc) : launch_mt<8>(c, p, grid, s.smem, s.mt, s.tc);
  if (e != cudaSuccess) return ruai_fail(c, RUAI_ERR_CUDA, "gemv launch failed: %s", cudaGetErrorString(e));
  return RUAI_OK;
}
