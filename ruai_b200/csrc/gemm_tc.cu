// Prefill / large-batch quantized GEMM on the tensor cores: out[m,n] = x[m,k] @ dequant(W)[k,n], m > 16.
//
// Replaces the reference's "dequantize the whole weight to f32, cast, cuBLAS" route for m > 16
// (src/nn/backend/cuda.rs:812-826) with one kernel that keeps the weight packed in HBM:
//   - the activations are stored once, by a small pre-kernel, as the tensor core's B operand: K-major with the 128-byte swizzle,
//     so that a stage of 64 k is one bulk copy.  f32 is scaled by a power of two per row and split into two fp16 pieces, 22
//     significant bits; fp16 is one piece as it is; so is bf16 for int4 (scaled to fp16 for int8).  What small elements keep is
//     set by fp16's quantum of 2^-24, by their distance from the row's largest element:
//       int4, x = hi + 2^-12 lo: 22 bits down to 2^-28, then a quantum of 2^-50 of the largest (17 bits at 2^-33);
//       int8, x = hi + lo: 22 bits down to 2^-16, then a quantum of 2^-38 (17 bits at 2^-21); bf16 exact down to 2^-31.
//     It shows only in a column whose weights for the large elements are all zero, since f32 sums have a quantum of 2^-24 of
//     theirs.  (Zeros are common in int4.  For int8 the same form costs 13 to 15 %: its sums cannot stay in tensor memory over
//     several stages then; 4096 x 4096 x 14336 835 -> 941 us, and 690 -> 764 with bf16 expanded weights);
//   - packed tiles of W (the chunk layout of pack.cu) come through a ring of bulk copies of their own and are expanded to fp16 or
//     bf16 (int4 and int8 values are exact) in tensor memory, the A operand;
//   - `tcgen05.mma kind::f16`, D[128 columns of W][rows of x], both pieces into the same f32 sums in tensor memory; int4: the lo
//     products first, the first hi product scales them by 2^-12 (exact);
//   - draining warps (thread = column of W) read the sums of every segment out and add them in f32 registers: int4: a segment
//     is a scale group of 32 k, times scale[g, j] (cpu.rs:1045-1063); int8: four stages, so that the tensor core's own
//     additions stay short, with the column scale at the end (cpu.rs:903-920).
// What bounds it: int8, the tensor pipe and the power limit (4096 x 4096 x 14336: 0.82 ms, 1.18 PFLOP/s counting both pieces, where
// cuBLAS sustains 1.40; 1.48 ms int4 and 1.45 int8 with unswizzled operands, which take twice as long); int4, the issue slots of the
// warps that expand and drain (1.23 to 1.25 ms: per scheduler and stage about 900 of the 1,037 clocks that its MMAs take).  A CTA of 256
// columns x 128 rows needs 16 MMAs of 64 clocks per stage.  256 columns, because every byte of x is then used twice: with 128 the
// copies of x alone ask the L2 for 64 bytes per clock and SM.  Three tile shapes and a split of k over a cluster cover the sizes that
// leave that tile's grid small (64 x 2048 x 2048 int8: 41 us before, 20 CTAs; 11 now).
// Every mbarrier wait is bounded.
#include "common.cuh"
#include "gemm_tile.cuh"
#include "gemv_epilogue.cuh"
#include "pipeline.cuh"

namespace gemm_tc {

using namespace pipe;

constexpr int kSegStages = 4;    // int8: stages per segment
constexpr int kLoShift = 12;     // int4: lo pieces are stored times 2^12.  Hi pieces below 2^15 leave out 2^3 at most: they stay below 2^15 too

// ---- activations -> fp16 pieces in B-operand layout --------------------------------------------------
// xs[row block of NT][stage][piece][row / 8][row % 8][8 chunks of 8 k, at chunk ^ (row % 8)]; the k of every four are stored in
// the order 0, 2, 1, 3, in which the packed weights unpack.  One CTA per row.  rowf[row]: what the row's sums are multiplied by.
struct SplitParams {
  const void* x;
  int x_dtype, pieces, vec;
  int raw;               // one piece, fp16 or bf16 as it is
  float lo_scale;
  uint32_t x_ld, m, k, stages, nt;
  const float* norm_w;   // RMSNorm folded in: x * norm_w
  const float* sumsq;    // [tiles][m] sums of squares of the row, or NULL: this kernel takes them (row_norm)
  uint32_t tiles;
  int row_norm;
  float eps;
  unsigned char* xs;
  float* rowf;
};

__device__ __forceinline__ void load8(const SplitParams& p, uint32_t row, uint32_t k0, float (&v)[8]) {
  const size_t at = (size_t)row * p.x_ld + k0;
  if (p.vec && k0 + 8u <= p.k) {
    if (p.x_dtype == RUAI_F32) {
      const float4 a = *reinterpret_cast<const float4*>((const float*)p.x + at), b = *reinterpret_cast<const float4*>((const float*)p.x + at + 4);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
      const uint4 a = *reinterpret_cast<const uint4*>((const uint16_t*)p.x + at);
      const uint32_t u[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (p.x_dtype == RUAI_BF16) {
          v[2 * i] = __uint_as_float(u[i] << 16); v[2 * i + 1] = __uint_as_float(u[i] & 0xFFFF0000u);
        } else {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u[i]));
          v[2 * i] = f.x; v[2 * i + 1] = f.y;
        }
      }
    }
  } else {
#pragma unroll
    for (uint32_t t = 0; t < 8; ++t) v[t] = k0 + t < p.k ? load_as_f32(p.x, p.x_dtype, at + t) : 0.0f;
  }
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {  // of values that are bf16
  return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
}
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

constexpr int kSplitThreads = 256;

__global__ void __launch_bounds__(kSplitThreads) xsplit_kernel(const SplitParams p) {
  __shared__ float red[2][kSplitThreads / 32];
  grid_dependency_wait();
  grid_launch_dependents();
  const uint32_t row = blockIdx.x, tid = threadIdx.x, chunks = p.stages * 8u;
  auto weigh = [&](uint32_t k0, float (&v)[8]) {
#pragma unroll
    for (uint32_t t = 0; t < 8; ++t)
      if (k0 + t < p.k) v[t] *= p.norm_w[k0 + t];
  };
  float f = 1.0f, back = 1.0f;
  if (!p.raw) {  // the row's largest magnitude (and its sum of squares)
    float mx = 0.0f, ss = 0.0f;
    for (uint32_t c = tid; c * 8u < p.k; c += kSplitThreads) {
      float v[8];
      load8(p, row, c * 8u, v);
      if (p.row_norm) {
#pragma unroll
        for (int t = 0; t < 8; ++t) ss = fmaf(v[t], v[t], ss);
      }
      if (p.norm_w) weigh(c * 8u, v);
#pragma unroll
      for (int t = 0; t < 8; ++t) mx = fmaxf(mx, fabsf(v[t]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
      ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
    }
    if ((tid & 31u) == 0) { red[0][tid >> 5] = mx; red[1][tid >> 5] = ss; }
    __syncthreads();
    mx = 0.0f; ss = 0.0f;
#pragma unroll
    for (int w = 0; w < kSplitThreads / 32; ++w) { mx = fmaxf(mx, red[0][w]); ss += red[1][w]; }
    // scaled by 2^e the largest magnitude lies in [2^14, 2^15): nothing overflows, and hi pieces are normal fp16 numbers down to
    // 2^-28 of it.  Zero and infinite rows stay as they are.
    const int ex = (int)((__float_as_uint(mx) >> 23) & 0xFFu) - 127;
    if (mx > 0.0f && ex < 128) {
      const int e = min(14 - ex, 126);
      f = __uint_as_float((uint32_t)(e + 127) << 23);
      back = __uint_as_float((uint32_t)(127 - e) << 23);
    }
    if (p.row_norm) back *= 1.0f / sqrtf(ss * (1.0f / (float)p.k) + p.eps);
    else if (p.norm_w && p.sumsq) {
      float t = 0.0f;
      for (uint32_t i = 0; i < p.tiles; ++i) t += p.sumsq[(size_t)i * p.m + row];
      back *= 1.0f / sqrtf(t * (1.0f / (float)p.k) + p.eps);
    }
  }
  if (tid == 0) p.rowf[row] = back;
  const uint32_t r = row % p.nt, piece = p.nt * 128u;
  const bool bf = p.raw && p.x_dtype == RUAI_BF16;
  unsigned char* base = p.xs + (size_t)(row / p.nt) * p.stages * p.pieces * piece + (r >> 3) * 1024u + (r & 7u) * 128u;
  for (uint32_t c = tid; c < chunks; c += kSplitThreads) {
    float v[8];
    load8(p, row, c * 8u, v);
    if (p.norm_w) weigh(c * 8u, v);
    float lo[8];
    uint32_t h[4];
#pragma unroll
    for (int t = 0; t < 8; ++t) v[t] *= f;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      h[2 * q] = bf ? pack_bf16(v[4 * q], v[4 * q + 2]) : pack_half2(v[4 * q], v[4 * q + 2]);
      h[2 * q + 1] = bf ? pack_bf16(v[4 * q + 1], v[4 * q + 3]) : pack_half2(v[4 * q + 1], v[4 * q + 3]);
    }
    unsigned char* dst = base + (size_t)(c >> 3) * p.pieces * piece + (((c & 7u) ^ (r & 7u)) << 4);
    *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
    if (p.pieces == 2) {
#pragma unroll
      for (int t = 0; t < 8; ++t) lo[t] = (v[t] - __half2float(__float2half_rn(v[t]))) * p.lo_scale;
      uint32_t l[4];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        l[2 * q] = pack_half2(lo[4 * q], lo[4 * q + 2]);
        l[2 * q + 1] = pack_half2(lo[4 * q + 1], lo[4 * q + 3]);
      }
      *reinterpret_cast<uint4*>(dst + piece) = make_uint4(l[0], l[1], l[2], l[3]);
    }
  }
}

// ---- the GEMM ------------------------------------------------------------------------------------------

struct Params {
  const uint4* w;
  const float* scale;
  const unsigned char* xs;
  const float* rowf;
  uint32_t m, n, chunks, groups;  // groups of 32 k
  uint32_t stages, stages_per_split, splits, row_blocks, tiles;
  int pieces;
  void* out;
  int* status;
  GemvEpilogue epi;
};

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr), "r"(v[0]),
      "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]),
      "r"(v[14]), "r"(v[15])
      : "memory");
}
// Two f32 multiply-adds in one instruction, each rounded like fmaf.
__device__ __forceinline__ void fma2(unsigned long long& acc, uint32_t d0, uint32_t d1, unsigned long long s) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(d0), "r"(d1));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(d), "l"(s));
}
__device__ __forceinline__ unsigned long long pair_of(float s) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "r"(__float_as_uint(s)));
  return r;
}
__device__ __forceinline__ float low_of(unsigned long long a) { return __uint_as_float((uint32_t)a); }
__device__ __forceinline__ float high_of(unsigned long long a) { return __uint_as_float((uint32_t)(a >> 32)); }

// Packed weights of one column -> fp16 pairs.  1024 + u has the bit pattern 0x6400 | u for u < 1024, so a mask and an OR make
// the number and one subtraction takes the offset out again, all exact.
// int4: a word holds rows 4w .. 4w+3 in its low nibbles and 16 + 4w .. in its high ones, as value + 8.
__device__ __forceinline__ uint32_t hsub2_bits(uint32_t a, uint32_t b) {
  const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t hfma2_bits(uint32_t a, uint32_t b, uint32_t c) {
  const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b), *reinterpret_cast<const __half2*>(&c));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ void expand_int4(const uint4& q, uint32_t (&o)[16]) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t t = w[i] >> 8;
    o[2 * i] = hsub2_bits((w[i] & 0x000F000Fu) | 0x64006400u, 0x64086408u);       // rows 4i, 4i + 2
    o[2 * i + 1] = hsub2_bits((t & 0x000F000Fu) | 0x64006400u, 0x64086408u);      // rows 4i + 1, 4i + 3
    o[8 + 2 * i] = hfma2_bits((w[i] & 0x00F000F0u) | 0x64006400u, 0x2C002C00u, 0xD480D480u);  // 1024 + 16 u: / 16, - 72
    o[8 + 2 * i + 1] = hfma2_bits((t & 0x00F000F0u) | 0x64006400u, 0x2C002C00u, 0xD480D480u);
  }
}
// The same to bf16: 128 + u has the bit pattern 0x4300 | u for u < 128.
__device__ __forceinline__ void expand_int4_bf16(const uint4& q, uint32_t (&o)[16]) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w}, offset = 0x43084308u;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const uint32_t u = ((w[i] >> (8 * (n & 1) + 4 * (n >> 1))) & 0x000F000Fu) | 0x43004300u;
      const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&u), *reinterpret_cast<const __nv_bfloat162*>(&offset));
      o[(n >> 1) * 8 + 2 * i + (n & 1)] = *reinterpret_cast<const uint32_t*>(&r);
    }
  }
}
__device__ __forceinline__ void expand_int8(const uint4& q, uint32_t* o) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // 1024 + 128 + value
    o[2 * i] = hsub2_bits((w[i] & 0x00FF00FFu) ^ 0x64806480u, 0x64806480u);
    o[2 * i + 1] = hsub2_bits(((w[i] >> 8) & 0x00FF00FFu) ^ 0x64806480u, 0x64806480u);
  }
}

// Row factor, column scale, bias, activation, residual and store of R consecutive rows of one column (a lane per column, the
// warp converged).  What is read is requested before the first store: the compiler cannot move loads over stores.
template <int R>
__device__ __forceinline__ void finish_rows(const Params& p, uint32_t end, float (&v)[R], const float (&rf)[R], uint32_t row, uint32_t j, bool active, float cs, float bias) {
  const GemvEpilogue& e = p.epi;
  const uint32_t nr = min((uint32_t)R, end - row);
#pragma unroll
  for (int t = 0; t < R; ++t) v[t] = v[t] * cs * rf[t] + bias;
  if (e.act == ACT_SWIGLU) {
    // columns (2i, 2i+1) hold (gate_i, up_i): the even lane finishes row t, the odd one row t + 1
    const uint32_t odd = j & 1u;
    float h[R / 2];
#pragma unroll
    for (int t = 0; t < R; t += 2) {
      const float other = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[t] : v[t + 1], 1);
      h[t / 2] = odd ? silu_ref(other) * v[t + 1] : silu_ref(v[t]) * other;
    }
    if (!active) return;
    const size_t o = (size_t)(row + odd) * e.out_ld + (j >> 1);
    if (e.resid) {
      float z[R / 2];
#pragma unroll
      for (int t = 0; t < R; t += 2) z[t / 2] = t + odd < nr ? e.resid[o + (size_t)t * e.out_ld] : 0.0f;
#pragma unroll
      for (int t = 0; t < R; t += 2) h[t / 2] += z[t / 2];
    }
#pragma unroll
    for (int t = 0; t < R; t += 2)
      if (t + odd < nr) store_from_f32(p.out, e.out_dtype, o + (size_t)t * e.out_ld, h[t / 2]);
    return;
  }
  if (!active) return;
  if (e.act == ACT_GELU) {
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = gelu_ref(v[t]);
  }
  const size_t o = (size_t)row * e.out_ld + j;
  if (e.resid) {
    float z[R];
#pragma unroll
    for (int t = 0; t < R; ++t) z[t] = (uint32_t)t < nr ? e.resid[o + (size_t)t * e.out_ld] : 0.0f;
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] += z[t];
  }
  if (e.out_dtype == RUAI_F32) {
    float* dst = (float*)p.out + o;
#pragma unroll
    for (int t = 0; t < R; ++t)
      if ((uint32_t)t < nr) dst[(size_t)t * e.out_ld] = v[t];
  } else {
#pragma unroll
    for (int t = 0; t < R; ++t)
      if ((uint32_t)t < nr) store_from_f32(p.out, e.out_dtype, o + (size_t)t * e.out_ld, v[t]);
  }
}

template <int BITS, int CB, int NT, bool BF>  // BF: both operands in bf16 (one piece)
__global__ void __launch_bounds__(Tile<BITS, CB, NT>::kThreads, 1) gemm_tc_kernel(const Params p) {
  using T = Tile<BITS, CB, NT>;
  constexpr uint32_t XS = T::kXSlots, WS = T::kWSlots, AB = T::kABufs;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t x_full[XS], x_empty[XS];   // x of a stage landed; the MMAs that read it completed
  __shared__ __align__(8) uint64_t w_full[WS], w_empty[WS];   // a packed stage (and its scales) landed; expanded (every expanding warp)
  __shared__ __align__(8) uint64_t a_ready[AB], a_free[AB];   // A operand of a stage written; the MMAs that read it completed
  // the sums of a unit (segment, column block) complete; read out (the column block's draining warps): of unit u at u % T::kUnitBars
  __shared__ __align__(8) uint64_t acc_full[T::kUnitBars], acc_free[T::kUnitBars];
  __shared__ __align__(8) uint64_t fin[2];
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort;
  // swizzled operands start on 1024-byte boundaries (the same offset in every CTA of a cluster: the window bases are alike)
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  if (tid == 0) {
    for (uint32_t s = 0; s < XS; ++s) { mbar_init(&x_full[s], 1); mbar_init(&x_empty[s], CB); }
    for (uint32_t s = 0; s < WS; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], T::kExpanders); }
    for (uint32_t s = 0; s < AB; ++s) { mbar_init(&a_ready[s], T::kExpanders); mbar_init(&a_free[s], CB); }
    for (uint32_t s = 0; s < T::kUnitBars; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_free[s], 4 * T::kDrains / CB); }
    mbar_init(&fin[0], 1); mbar_init(&fin[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_abort = 0;
  }
  __syncwarp();
  if (warp == 2) tmem_alloc(&s_tmem, T::kTmem);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = s_tmem;
  const uint32_t split = p.splits > 1 ? cluster_ctarank() : 0u;
  const uint32_t s0 = split * p.stages_per_split, s1 = min(p.stages, s0 + p.stages_per_split), nst = s1 - s0;  // splits are never empty
  const uint32_t tile0 = blockIdx.x / p.splits, stride = gridDim.x / p.splits;
  auto cols_of = [&](uint32_t t) { return (t / p.row_blocks) * (uint32_t)T::kCols; };  // row blocks fastest: a tile of W comes from HBM once
  auto rows_of = [&](uint32_t t) { return (t % p.row_blocks) * (uint32_t)NT; };

  // Stage `it` of this CTA: packed weights -> A operand, for one warp's columns of column block cb, groups u0 .. u1 of the stage.
  auto expand = [&](uint32_t it, uint32_t cb, uint32_t u0, uint32_t u1) -> bool {
    const uint32_t slot = it % WS, ab = it % AB, quarter = (uint32_t)warp & 3u;
    if (s_abort || !mbar_wait(&w_full[slot], (it / WS) & 1u)) return false;
    if (it >= AB && !mbar_wait(&a_free[ab], (it / AB - 1u) & 1u)) return false;
    const unsigned char* w = smem + T::off_w + slot * T::kWBytes + (cb * 128u + quarter * 32u + lane) * 16u;
    const uint32_t a = tmem + ((quarter * 32u) << 16) + T::kACol0 + (ab * CB + cb) * 32;
    tc_fence_after_sync();
    for (uint32_t u = u0; u < u1; ++u) {
      uint32_t o[16];
      if constexpr (BF) expand_int4_bf16(*reinterpret_cast<const uint4*>(w + u * T::kWChunk), o);
      else if constexpr (BITS == 4) expand_int4(*reinterpret_cast<const uint4*>(w + u * T::kWChunk), o);
      else {
        const uint4 q0 = *reinterpret_cast<const uint4*>(w + 2 * u * T::kWChunk), q1 = *reinterpret_cast<const uint4*>(w + (2 * u + 1) * T::kWChunk);
        expand_int8(q0, o);
        expand_int8(q1, o + 8);
      }
      tmem_st16(a + u * 16, o);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) { mbar_arrive(&a_ready[ab]); mbar_arrive(&w_empty[slot]); }
    return true;
  };

  if (warp < 4) {
    if (warp == 0 && elect_one()) {
      // ===== packed weights (and their scales).  They do not depend on the predecessor kernel. =====
      uint32_t it = 0;
      bool ok = true;
      for (uint32_t t = tile0; t < p.tiles && ok; t += stride) {
        const uint32_t j0 = cols_of(t), nc = min((uint32_t)T::kCols, p.n - j0);
        for (uint32_t s = s0; s < s1; ++s, ++it) {
          const uint32_t slot = it % WS;
          if (it >= WS && (s_abort || !mbar_wait(&w_empty[slot], (it / WS - 1u) & 1u))) { s_abort = 1; ok = false; break; }
          const uint32_t c0 = s * T::kChunks, chunks = min((uint32_t)T::kChunks, p.chunks - c0);
          unsigned char* dst = smem + T::off_w + slot * T::kWBytes;
          // int4: a chunk is a scale group.  That the scales' slot is free as well: see Tile::kScaleSlots.
          mbar_expect_tx(&w_full[slot], chunks * nc * (BITS == 4 ? 20u : 16u));
          for (uint32_t c = 0; c < chunks; ++c) {
            bulk_load(dst + c * T::kWChunk, p.w + (size_t)(c0 + c) * p.n + j0, nc * 16u, &w_full[slot]);
            if constexpr (BITS == 4)
              bulk_load(smem + T::off_scale + (it % T::kScaleSlots) * T::kScale + c * T::kCols * 4, p.scale + (size_t)(c0 + c) * p.n + j0, nc * 4u, &w_full[slot]);
          }
        }
      }
      if (s_abort)  // leave no copy in flight into shared memory that another CTA may get
        for (uint32_t i = it > WS ? it - WS : 0; i < it; ++i) (void)mbar_wait(&w_full[i % WS], (i / WS) & 1u);
    } else if (warp == 3 && elect_one()) {
      // ===== x =====
      grid_dependency_wait();
      grid_launch_dependents();
      uint32_t it = 0;
      bool ok = true;
      for (uint32_t t = tile0; t < p.tiles && ok; t += stride) {
        const uint32_t bytes = (uint32_t)p.pieces * T::kPiece;
        const unsigned char* src = p.xs + ((size_t)(t % p.row_blocks) * p.stages + s0) * bytes;
        for (uint32_t i = 0; i < nst; ++i, ++it) {
          const uint32_t slot = it % XS;
          if (it >= XS && (s_abort || !mbar_wait(&x_empty[slot], (it / XS - 1u) & 1u))) { s_abort = 1; ok = false; break; }
          mbar_expect_tx(&x_full[slot], bytes);
          bulk_load(smem + slot * T::kX, src + (size_t)i * bytes, bytes, &x_full[slot]);
        }
      }
      if (s_abort)
        for (uint32_t i = it > XS ? it - XS : 0; i < it; ++i) (void)mbar_wait(&x_full[i % XS], (i / XS) & 1u);
    } else if ((warp == 1 || warp == 2) && elect_one()) {
      // ===== MMAs.  A wait behind MMAs comes back only when those have left the issue queue (measured: 90 to 260 clocks in which
      // the tensor pipe has nothing to do), so two threads issue, each into its own sums: one per column block, or, with one
      // column block, every other stage each. =====
      constexpr uint32_t idesc = (1u << 4) | (BF ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(NT >> 3) << 17) | ((128u >> 4) << 24);  // fp16 x fp16 or bf16 x bf16 -> f32
      const uint64_t xd0 = umma_desc_sw128(smem_u32(smem));
      const uint32_t pieces = (uint32_t)p.pieces, h = (uint32_t)warp - 1u, cb = CB == 2 ? h : 0u;
      uint32_t it = 0, unit = BITS == 4 && CB == 1 ? 0u : h;
      bool ok = true;
      auto sums_free = [&](uint32_t u) { return u < 3 || mbar_wait(&acc_free[(u - 3) % T::kUnitBars], ((u - 3) / T::kUnitBars) & 1u); };
      for (uint32_t t = tile0; t < p.tiles && ok; t += stride) {
        for (uint32_t s = s0; s < s1 && ok; ++s, ++it) {
          const uint32_t ab = it % AB, slot = it % XS, ng = BITS == 4 ? min(2u, p.groups - 2u * s) : 1u, at = (s - s0) % kSegStages;
          const bool mine = CB == 2 || ((s - s0) & 1u) == h;
          if (BITS == 4 && !mine) { unit += ng; continue; }
          const bool last = at + 3 - CB >= kSegStages || s + 3 - CB >= s1;  // int8: of this thread's stages in the segment
          if (mine) {
            if (s_abort || !mbar_wait(&a_ready[ab], (it / AB) & 1u) || !mbar_wait(&x_full[slot], (it / XS) & 1u)) { ok = false; break; }
            const uint32_t a = tmem + T::kACol0 + (ab * CB + cb) * 32;
            const uint64_t xd = umma_desc_advance(xd0, slot * T::kX);
            if constexpr (BITS == 4) {
              for (uint32_t u = 0; u < ng; ++u, unit += CB) {
                if (!sums_free(unit)) { ok = false; break; }
                tc_fence_after_sync();
                const uint32_t d = tmem + (unit % 3) * NT, au = a + u * 16;
                const uint64_t xu = umma_desc_advance(xd, u * 64u);
                if (pieces == 2) {
                  umma_f16_ts(d, au, umma_desc_advance(xu, T::kPiece), idesc, 0u);
                  umma_f16_ts(d, au + 8, umma_desc_advance(xu, T::kPiece + 32u), idesc, 1u);
                  umma_f16_ts_after<kLoShift>(d, au, xu, idesc);
                } else {
                  umma_f16_ts(d, au, xu, idesc, 0u);
                }
                umma_f16_ts(d, au + 8, umma_desc_advance(xu, 32u), idesc, 1u);
                umma_commit(&acc_full[unit % T::kUnitBars]);
              }
            } else {
              const bool first = at < 3 - CB;
              if (first && !sums_free(unit)) { ok = false; break; }
              tc_fence_after_sync();
              const uint32_t d = tmem + (unit % 3) * NT;
              for (uint32_t pc = 0; pc < pieces; ++pc)
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q) umma_f16_ts(d, a + q * 8, umma_desc_advance(xd, pc * T::kPiece + q * 32u), idesc, !first || (pc | q) != 0 ? 1u : 0u);
              if (last) { umma_commit(&acc_full[unit % T::kUnitBars]); unit += 2; }
            }
            umma_commit(&x_empty[slot]);
            umma_commit(&a_free[ab]);
          } else if (h == 1 && at == 0 && s + 1 == s1) {  // int8, a segment of one stage: the other thread's sums are all there is
            if (!sums_free(unit)) { ok = false; break; }
            umma_commit(&acc_full[unit % T::kUnitBars]);
            unit += 2;
          }
        }
      }
      if (!ok) s_abort = 1;
      umma_commit(&fin[h]);  // nothing is left running when tensor memory is freed
      if (!mbar_wait(&fin[h], 0)) s_abort = 1;
    }
    __syncwarp();
    grid_dependency_wait();
  } else if (warp < T::kDrain0) {
    // ===== expanding warps (one column block) =====
    uint32_t it = 0;
    bool ok = true;
    for (uint32_t t = tile0; t < p.tiles && ok; t += stride)
      for (uint32_t s = s0; s < s1 && ok; ++s, ++it) ok = expand(it, 0, 0, 2);
    if (!ok) s_abort = 1;
    grid_dependency_wait();
  } else {
    // ===== draining warps: thread = column of one column block, 64 rows =====
    const uint32_t dw = (uint32_t)(warp - T::kDrain0), quarter = (uint32_t)warp & 3u, cb = (dw >> 2) & (CB - 1), half = dw / (4 * CB) * 64u;
    const uint32_t col = cb * 128u + quarter * 32u + lane, sums = tmem + ((quarter * 32u) << 16) + half;
    constexpr int kFinish = CB == 2 ? 8 : 16;  // rows finished together: what the registers beside the sums hold
    unsigned long long acc[32];
    uint32_t unit = cb;
    bool ok = true;
    // one unit's sums into the registers, times the scale of group u of a stage
    auto drain = [&](uint32_t scale_slot, uint32_t u, bool none) -> bool {
      const uint32_t set = unit % 3;
      if (s_abort || !mbar_wait(&acc_full[unit % T::kUnitBars], (unit / T::kUnitBars) & 1u)) return false;
      tc_fence_after_sync();
      float sv = 1.0f;
      if constexpr (BITS == 4)  // a column past the matrix reads what an earlier tile left: it is never stored
        sv = *reinterpret_cast<const float*>(smem + T::off_scale + scale_slot * T::kScale + (u * T::kCols + col) * 4u);
      const unsigned long long s2 = pair_of(sv);
      const uint32_t at = sums + set * NT;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t d[16];
        tmem_ld16(at + 16 * c, d);
        if (c == 3) {  // the buffer may be overwritten
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_free[unit % T::kUnitBars]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (!none) fma2(acc[8 * c + i], d[2 * i], d[2 * i + 1], s2);
      }
      unit += CB;
      return true;
    };
    // what stage s (number it of this CTA) completes
    auto drain_stage = [&](uint32_t it, uint32_t s) -> bool {
      if constexpr (BITS == 4) {
        const uint32_t ng = min(2u, p.groups - 2u * s);
#pragma unroll 1
        for (uint32_t u = 0; u < ng; ++u)
          if (!drain(it % T::kScaleSlots, u, false)) return false;
      } else if ((s - s0) % kSegStages == kSegStages - 1 || s + 1 == s1) {
        // one column block: both issuing threads' sums, of which the second has none in a segment of one stage
#pragma unroll 1
        for (uint32_t u = 0; u < 3 - CB; ++u)
          if (!drain(0, 0, u == 1 && (s - s0) % kSegStages == 0)) return false;
      }
      return true;
    };
    uint32_t it = 0;
    if constexpr (T::kBoth) ok = expand(0, cb, half / 64u, half / 64u + 1);
    grid_dependency_wait();
    for (uint32_t t = tile0; t < p.tiles && ok; t += stride) {
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[i] = 0ull;
#pragma unroll 1
      for (uint32_t s = s0; s < s1 && ok; ++s, ++it) {
        if constexpr (T::kBoth) {  // the next stage (the next tile's first) is ready before this one's sums are read
          if (s + 1 < s1 || t + stride < p.tiles) ok = expand(it + 1, cb, half / 64u, half / 64u + 1);
        }
        ok = ok && drain_stage(it, s);
      }
      if (!ok) break;
      if (p.splits > 1) break;  // one tile per cluster: see below
      const uint32_t j = cols_of(t) + col, row0 = rows_of(t) + half;
      const bool active = j < p.n;
      // everything the epilogue reads is requested ahead of its first store: loads between stores wait behind them (measured: 63,000
      // clocks for an epilogue that read the rows' factors in groups of eight)
      const float cs = BITS == 8 && active ? __ldg(p.scale + j) : 1.0f, bias = p.epi.bias && active ? __ldg(p.epi.bias + j) : 0.0f;
      const float rfl[2] = {row0 + lane < p.m ? __ldcg(p.rowf + row0 + lane) : 0.0f, row0 + 32u + lane < p.m ? __ldcg(p.rowf + row0 + 32u + lane) : 0.0f};
#pragma unroll
      for (int r = 0; r < 64; r += kFinish) {
        if (row0 + r >= p.m) break;
        float v[kFinish], rf[kFinish];
#pragma unroll
        for (int i = 0; i < kFinish; ++i) {
          v[i] = (i & 1) ? high_of(acc[(r + i) / 2]) : low_of(acc[(r + i) / 2]);
          rf[i] = __shfl_sync(0xFFFFFFFFu, rfl[r / 32], (r + i) % 32);
        }
        finish_rows<kFinish>(p, p.m, v, rf, row0 + r, j, active, cs, bias);
      }
    }
    if (!ok) s_abort = 1;
    if (p.splits > 1) {
      // k is split over the cluster: every CTA finishes its share of the rows, from the sums of all of them in a fixed order
      const uint32_t rows_per = (NT + p.splits - 1) / p.splits;
      float* red = reinterpret_cast<float*>(smem);  // [splits][rows_per][kCols]
      const uint32_t j = cols_of(tile0) + col, row0 = rows_of(tile0);
      const bool active = j < p.n;
      __syncwarp();
      cluster_sync_all();  // every CTA is through with its operands
      uint32_t owner = half / rows_per, at = half % rows_per;
#pragma unroll
      for (int r = 0; r < 64; ++r) {
        st_cluster_f32(red + ((size_t)split * rows_per + at) * T::kCols + col, owner, (r & 1) ? high_of(acc[r / 2]) : low_of(acc[r / 2]));
        if (++at == rows_per) { at = 0; ++owner; }
      }
      __syncwarp();
      cluster_sync_all();
      if (!s_abort) {
        const float cs = BITS == 8 && active ? __ldg(p.scale + j) : 1.0f, bias = p.epi.bias && active ? __ldg(p.epi.bias + j) : 0.0f;
        const uint32_t first = split * rows_per, last = min(first + rows_per, (uint32_t)NT);
        // eight rows at a time, in turn over the warpgroups of a column block
        for (uint32_t r = first + half / 8u; r < last; r += NT / 8u) {
          if (row0 + r >= p.m) break;
          float v[8], rf[8];
#pragma unroll
          for (uint32_t i = 0; i < 8; ++i) { v[i] = 0.0f; rf[i] = row0 + r + i < p.m ? __ldcg(p.rowf + row0 + r + i) : 0.0f; }
          for (uint32_t q = 0; q < p.splits; ++q) {
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i)
              if (r + i < last) v[i] += red[((size_t)q * rows_per + (r - first) + i) * T::kCols + col];
          }
          finish_rows<8>(p, min(p.m, row0 + last), v, rf, row0 + r, j, active, cs, bias);
        }
      }
    }
  }
  if (p.splits > 1 && warp < T::kDrain0) {  // the draining warps' two
    __syncwarp();
    cluster_sync_all();
    cluster_sync_all();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (s_abort && tid == 0) atomicExch(p.status, 3);
  if (warp == 2) tmem_dealloc(tmem, T::kTmem);
}

template <int BITS, int CB, int NT, bool BF>
cudaError_t launch(ruai_ctx* c, const Params& p) {
  using T = Tile<BITS, CB, NT>;
  static bool attr_done[64] = {};
  if (!attr_done[c->ordinal & 63]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel<BITS, CB, NT, BF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::kSmem);
    if (e != cudaSuccess) return e;
    attr_done[c->ordinal & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.splits > 1 ? p.tiles * p.splits : min(p.tiles, (uint32_t)c->sm_count));
  cfg.blockDim = dim3(T::kThreads);
  cfg.dynamicSmemBytes = T::kSmem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (c->use_pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (p.splits > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = p.splits;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  c->launches++;
  return cudaLaunchKernelEx(&cfg, gemm_tc_kernel<BITS, CB, NT, BF>, p);
}

struct Shape { uint32_t cb, nt, splits; };

template <int BITS, bool BF>
cudaError_t launch_tile(ruai_ctx* c, const Params& p, const Shape& sh) {
  return sh.cb == 2 ? launch<BITS, 2, 128, BF>(c, p) : sh.nt == 128 ? launch<BITS, 1, 128, BF>(c, p) : launch<BITS, 1, 64, BF>(c, p);
}

// The tile and the number of splits of k: a model of the launch in microseconds, fitted to launches of 37 to 2000 rows of the 1.1B and
// 8B shapes' Linears with every tile and 1 .. 8 splits.  Over 17 to 2000 rows of those and the 135M shape's (`python -m
// ruai_b200.sweep_splits`) the choice is within 5 % of the best tile and split at 115 of 132 sizes, the worst 1.19 times the best (a wrong
// one costs up to 2 x).
Shape choose(const ruai_ctx* c, uint32_t m, uint32_t n, uint32_t stages, int bits, int pieces) {
  struct Cand { uint32_t cb, nt; double stage4, stage8, split; };  // a stage of int4 and int8; what a split adds
  const Cand cand[3] = {{2, 128, 1.55, 1.0, 7.0}, {1, 128, 0.80, 0.55, 6.0}, {1, 64, 0.62, 0.45, 3.5}};
  Shape best = {1, 64, 1};
  double best_t = 1e300;
  for (const Cand& d : cand) {
    if (c->force_cols && (c->force_cols != d.cb * 128 || c->force_rows != d.nt)) continue;
    const uint32_t tiles = ((n + d.cb * 128 - 1) / (d.cb * 128)) * ((m + d.nt - 1) / d.nt);
    for (uint32_t s = 1; s <= 8; ++s) {
      const uint32_t per = (stages + s - 1) / s;
      if (s > 1 && (per < 2 || (s - 1) * per >= stages)) continue;
      // a cluster lies within one group of SMs: not every SM is reached (measured: sixteen clusters of 8 take two waves)
      const uint32_t sms = (uint32_t)c->sm_count, room = s == 1 ? sms : s >= 7 ? sms / 10u : sms * 15u / 16u / s;
      if (room == 0) continue;
      const double waves = (double)((tiles + room - 1) / room), stage = (bits == 4 ? d.stage4 : d.stage8) * (pieces == 2 ? 1.0 : 0.8);
      const double t = 4.0 + waves * (per * stage + 1.0 + (s > 1 ? d.split : 0.0));
      if (t < best_t) { best_t = t; best = {d.cb, d.nt, s}; }
    }
  }
  return best;
}

}  // namespace gemm_tc

bool ruai_gemm_tc_eligible(const ruai_qweight* w, uint32_t m) {
  return w->layout == QL_CHUNK16 && m > 16 && (w->bits == 8 || w->n % 4 == 0);
}

int ruai_gemm_tc_launch(ruai_ctx* c, const ruai_qweight* w, const void* x, int x_dtype, uint32_t x_ld, uint32_t m, void* out,
                        const GemvEpilogue& epi_in, const GemvPrologue& pro) {
  using namespace gemm_tc;
  GemvEpilogue epi = epi_in;
  if (epi.act == ACT_SWIGLU && (w->n & 1)) return ruai_fail(c, RUAI_ERR_SHAPE, "SwiGLU epilogue needs an even column count, got %u", w->n);
  if (epi.out_ld == 0) epi.out_ld = epi.act == ACT_SWIGLU ? w->n / 2 : w->n;
  if (epi.sumsq || epi.argmax_out) return ruai_fail(c, RUAI_ERR_UNSUPPORTED, "the prefill GEMM has no fused sum of squares / argmax");
  if ((m + 127u) / 128u > 65535u) return ruai_fail(c, RUAI_ERR_UNSUPPORTED, "m too large");
  const uint32_t groups = (w->k + 31) / 32, stages = (groups + 1) / 2;
  // fp16 and bf16 activations are one piece; not when a norm multiplies them
  const int pieces = x_dtype == RUAI_F32 || pro.norm_w ? 2 : 1;
  Shape sh = choose(c, m, w->n, stages, w->bits, pieces);
  if (c->force_splits >= 1 && c->force_splits <= 8) {
    sh.splits = c->force_splits;
    while (sh.splits > 1 && (sh.splits - 1) * ((stages + sh.splits - 1) / sh.splits) >= stages) --sh.splits;
  }
  const uint32_t row_blocks = (m + sh.nt - 1) / sh.nt, col_tiles = (w->n + sh.cb * 128 - 1) / (sh.cb * 128);
  // the split activations and the rows' factors live in the context's scratch
  const size_t xs_bytes = (size_t)row_blocks * stages * pieces * sh.nt * 128;
  RUAI_TRY(ruai_ctx_reserve(c, xs_bytes + (size_t)m * sizeof(float), 0));
  SplitParams sp;
  sp.x = x; sp.x_dtype = x_dtype; sp.pieces = pieces; sp.x_ld = x_ld; sp.m = m; sp.k = w->k; sp.stages = stages; sp.nt = sh.nt;
  sp.vec = ((uintptr_t)x & 15u) == 0 && x_ld % (x_dtype == RUAI_F32 ? 4u : 8u) == 0 ? 1 : 0;
  sp.norm_w = pro.norm_w; sp.sumsq = pro.sumsq; sp.tiles = pro.tiles; sp.row_norm = pro.norm_w && !pro.sumsq ? 1 : 0; sp.eps = pro.eps;
  sp.raw = pieces == 1 && (x_dtype == RUAI_F16 || w->bits == 4) ? 1 : 0;
  sp.lo_scale = w->bits == 4 ? (float)(1 << kLoShift) : 1.0f;
  sp.xs = reinterpret_cast<unsigned char*>(c->partial);
  sp.rowf = reinterpret_cast<float*>(sp.xs + xs_bytes);
  RUAI_CUDA(c, ruai_launch(c, xsplit_kernel, dim3(m), dim3(kSplitThreads), 0, true, sp));
  Params p;
  p.w = (const uint4*)w->data; p.scale = w->scale; p.xs = sp.xs; p.rowf = sp.rowf; p.m = m; p.n = w->n; p.chunks = w->chunks; p.groups = groups;
  p.stages = stages; p.splits = sh.splits; p.stages_per_split = (stages + sh.splits - 1) / sh.splits;
  p.row_blocks = row_blocks; p.tiles = row_blocks * col_tiles; p.pieces = pieces;
  p.out = out; p.status = c->status; p.epi = epi;
  const cudaError_t e = w->bits == 8 ? launch_tile<8, false>(c, p, sh) : sp.raw && x_dtype == RUAI_BF16 ? launch_tile<4, true>(c, p, sh) : launch_tile<4, false>(c, p, sh);
  if (e != cudaSuccess) return ruai_fail(c, RUAI_ERR_CUDA, "prefill GEMM launch failed: %s", cudaGetErrorString(e));
  return RUAI_OK;
}
