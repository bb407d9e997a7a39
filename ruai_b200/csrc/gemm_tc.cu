// Prefill / large-batch quantized GEMM on the tensor cores: out[m,n] = x[m,k] @ dequant(W)[k,n], m > 16.
//
// Replaces the reference's "dequantize the whole weight to f32, cast, cuBLAS" route for m > 16
// (src/nn/backend/cuda.rs:812-826) with one kernel that keeps the weight packed in HBM:
//   - the activations are scaled by a power of two per row and split once, by a small pre-kernel, into two fp16 pieces
//     x = hi + lo (22 significant bits; bf16 and fp16 activations are one piece, exactly) stored as the tensor core's B
//     operand: K-major with the 128-byte swizzle, so that a stage of 64 k is one bulk copy;
//   - packed tiles of W (the chunk layout of pack.cu) ride in the same ring of bulk copies; four warps expand them to fp16
//     (int4 and int8 values are exact) into the A operand, same swizzle;
//   - `tcgen05.mma kind::f16`, D[128 columns of W][rows of x], both pieces into the same f32 sums in tensor memory;
//   - draining warps (thread = column of W) read the sums of every segment out and add them in f32 registers: int4: a segment
//     is a scale group of 32 k, times scale[g, j] (cpu.rs:1045-1063); int8: four stages, so that the tensor core's own
//     additions stay short, with the column scale at the end (cpu.rs:903-920).
// What bounds it: the tensor pipe.  A CTA of 256 columns x 128 rows needs 16 MMAs of 64 clocks per stage (measured: one thread
// issues M 128, N 128, K 16 every 64 clocks, N 64 every 48 from swizzled shared memory; from the unswizzled layout that an
// earlier version used a stage took twice as long), while its four expanding and eight draining warps need about 900 issue slots
// per scheduler.  256 columns, because every B byte is then used twice: with 128 the copies of B alone ask the L2 for 64 bytes
// per clock and SM.  Three tile shapes and a split of k over a cluster cover the sizes that leave that tile's grid small.
// Every mbarrier wait is bounded.
#include "common.cuh"
#include "gemv_epilogue.cuh"
#include "pipeline.cuh"

namespace gemm_tc {

using namespace pipe;

constexpr int kSegStages = 4;    // int8: stages per segment

// ---- activations -> fp16 pieces in B-operand layout --------------------------------------------------
// xs[row block of NT][stage][piece][row / 8][row % 8][8 chunks of 8 k, at chunk ^ (row % 8)]; the k of every four are stored in
// the order 0, 2, 1, 3, in which the packed weights unpack.  One CTA per row.  rowf[row]: what the row's sums are multiplied by.
struct SplitParams {
  const void* x;
  int x_dtype, pieces, vec;
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
  if (p.x_dtype != RUAI_F16 || p.norm_w) {  // the row's largest magnitude (and its sum of squares)
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
    // scaled by 2^e the largest magnitude lies in [2^14, 2^15): both pieces of everything down to 2^-28 of it are normal fp16
    // numbers or exact, and nothing overflows.  Zero and infinite rows stay as they are.
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
      h[2 * q] = pack_half2(v[4 * q], v[4 * q + 2]);
      h[2 * q + 1] = pack_half2(v[4 * q + 1], v[4 * q + 3]);
    }
    unsigned char* dst = base + (size_t)(c >> 3) * p.pieces * piece + (((c & 7u) ^ (r & 7u)) << 4);
    *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
    if (p.pieces == 2) {
#pragma unroll
      for (int t = 0; t < 8; ++t) lo[t] = v[t] - __half2float(__float2half_rn(v[t]));
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

// CB column blocks of 128 x NT rows of x per CTA.  Warps: 0 copies, 1 issues MMAs, 4-7 expand, 8.. drain (four per column block).
template <int BITS, int CB, int NT>
struct Tile {
  static constexpr int kCols = CB * 128;
  static constexpr int kThreads = 256 + 128 * CB;
  static constexpr uint32_t kWChunk = kCols * 16;                        // one 16-byte chunk of every column
  static constexpr int kChunks = BITS == 4 ? 2 : 4;                      // chunks per stage
  static constexpr uint32_t kWBytes = kChunks * kWChunk;
  static constexpr uint32_t kPiece = NT * 128;                           // one piece of a stage
  static constexpr uint32_t kSlot = 2 * kPiece + kWBytes;
  static constexpr uint32_t kA = kCols * 128;                            // one stage of the A operand
  static constexpr int kFit = (int)((230400 - 1024 - 2 * kA) / kSlot);
  static constexpr int kSlots = kFit < 6 ? kFit : 6;
  static constexpr size_t kSmem = 1024 + 2 * (size_t)kA + (size_t)kSlots * kSlot;
  static constexpr uint32_t kTmem = 2 * CB * NT;                         // two sets of sums
  static_assert(kSlots >= 3, "ring too short");
};

__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {  // K-major, 128-byte swizzle, 1024 bytes between 8-row blocks
  return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b),
               "r"(idesc), "r"(accumulate)
               : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
// 16 consecutive 32-bit columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
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
__device__ __forceinline__ void expand_int8(const uint4& q, uint32_t (&o)[8]) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // 1024 + 128 + value
    o[2 * i] = hsub2_bits((w[i] & 0x00FF00FFu) ^ 0x64806480u, 0x64806480u);
    o[2 * i + 1] = hsub2_bits(((w[i] >> 8) & 0x00FF00FFu) ^ 0x64806480u, 0x64806480u);
  }
}

template <int R>
__device__ __forceinline__ void setmaxnreg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void setmaxnreg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }

// Row factor, column scale, bias, activation, residual and store of R consecutive rows of one column (a lane per column, the
// warp converged).  What is read is requested before the first store: the compiler cannot move loads over stores.
template <int R>
__device__ __forceinline__ void finish_rows(const Params& p, uint32_t end, float (&v)[R], uint32_t row, uint32_t j, bool active, float cs, float bias) {
  const GemvEpilogue& e = p.epi;
  const uint32_t nr = min((uint32_t)R, end - row);
  float rf[R];
#pragma unroll
  for (int t = 0; t < R; ++t) rf[t] = (uint32_t)t < nr ? __ldcg(p.rowf + row + t) : 0.0f;
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

template <int BITS, int CB, int NT>
__global__ void __launch_bounds__(Tile<BITS, CB, NT>::kThreads, 1) gemm_tc_kernel(const Params p) {
  using T = Tile<BITS, CB, NT>;
  constexpr uint32_t S = T::kSlots;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[S], empty[S];   // a slot's copies landed; the MMAs that read it completed
  __shared__ __align__(8) uint64_t a_ready[2];          // A operand of a stage written (4 expanding warps)
  __shared__ __align__(8) uint64_t acc_full[2], acc_free[2];  // a segment's sums complete; read out (4 CB warps)
  __shared__ __align__(8) uint64_t fin;
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort;
  // swizzled operands start on 1024-byte boundaries (the same offset in every CTA of a cluster: the window bases are alike)
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* abuf = smem;
  unsigned char* ring = smem + 2 * T::kA;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  if (tid == 0) {
    for (uint32_t s = 0; s < S; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&a_ready[s], 4); mbar_init(&acc_full[s], 1); mbar_init(&acc_free[s], 4 * CB); }
    mbar_init(&fin, 1);
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

  if (warp < 4) {
    if constexpr (NT == 128) setmaxnreg_dec<40>();
    if (warp == 0 && lane == 0) {
      // ===== copies.  Weights do not depend on the predecessor kernel: the first slots' are requested before the wait. =====
      const uint32_t bbytes = (uint32_t)p.pieces * T::kPiece;
      auto copy_w = [&](uint32_t t, uint32_t s, uint32_t slot) {
        const uint32_t j0 = cols_of(t), bytes = min((uint32_t)T::kCols, p.n - j0) * 16u, c0 = s * T::kChunks;
        const uint32_t nc = min((uint32_t)T::kChunks, p.chunks - c0);
        unsigned char* dst = ring + slot * T::kSlot + 2 * T::kPiece;
        mbar_expect_tx(&full[slot], nc * bytes + bbytes);
        for (uint32_t c = 0; c < nc; ++c) bulk_load(dst + c * T::kWChunk, p.w + (size_t)(c0 + c) * p.n + j0, bytes, &full[slot]);
      };
      auto copy_x = [&](uint32_t t, uint32_t s, uint32_t slot) {
        bulk_load(ring + slot * T::kSlot, p.xs + ((size_t)(t % p.row_blocks) * p.stages + s) * bbytes, bbytes, &full[slot]);
      };
      const uint32_t pre = min(nst, S);
      for (uint32_t i = 0; i < pre; ++i) copy_w(tile0, s0 + i, i);
      grid_dependency_wait();
      grid_launch_dependents();
      for (uint32_t i = 0; i < pre; ++i) copy_x(tile0, s0 + i, i);
      uint32_t it = pre;
      bool ok = true;
      for (uint32_t t = tile0; t < p.tiles && ok; t += stride) {
        for (uint32_t s = t == tile0 ? s0 + pre : s0; s < s1; ++s, ++it) {
          const uint32_t slot = it % S;
          if (it >= S && (s_abort || !mbar_wait(&empty[slot], (it / S - 1u) & 1u))) { s_abort = 1; ok = false; break; }
          copy_w(t, s, slot);
          copy_x(t, s, slot);
        }
      }
      if (s_abort)  // leave no copy in flight into shared memory that another CTA may get
        for (uint32_t i = it > S ? it - S : 0; i < it; ++i) (void)mbar_wait(&full[i % S], (i / S) & 1u);
    } else if (warp == 1 && elect_one()) {
      // ===== MMAs =====
      constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((128u >> 4) << 24);  // fp16 x fp16 -> f32
      uint32_t it = 0, seg = 0;
      bool ok = true;
      for (uint32_t t = tile0; t < p.tiles && ok; t += stride) {
        for (uint32_t s = s0; s < s1; ++s, ++it) {
          const uint32_t slot = it % S, ab = it & 1u;
          if (s_abort || !mbar_wait(&a_ready[ab], (it >> 1) & 1u) || !mbar_wait(&full[slot], (it / S) & 1u)) { ok = false; break; }
          const uint64_t ad = desc_sw128(smem_u32(abuf + ab * T::kA)), bd = desc_sw128(smem_u32(ring + slot * T::kSlot));
          if constexpr (BITS == 4) {
            const uint32_t ng = min(2u, p.groups - 2u * s);
            for (uint32_t u = 0; u < ng; ++u, ++seg) {
              const uint32_t set = seg & 1u;
              if (seg >= 2 && !mbar_wait(&acc_free[set], ((seg >> 1) - 1u) & 1u)) { ok = false; break; }
              tc_fence_after_sync();
#pragma unroll
              for (uint32_t cb = 0; cb < CB; ++cb)
                for (uint32_t pc = 0; pc < (uint32_t)p.pieces; ++pc)
#pragma unroll
                  for (uint32_t q = 0; q < 2; ++q)
                    mma_f16(tmem + (set * CB + cb) * NT, umma_desc_advance(ad, cb * 16384u + u * 64u + q * 32u),
                            umma_desc_advance(bd, pc * T::kPiece + u * 64u + q * 32u), idesc, (pc | q) != 0 ? 1u : 0u);
              umma_commit(&acc_full[set]);
            }
            if (!ok) break;
          } else {
            const uint32_t set = seg & 1u, at = (s - s0) % kSegStages;
            if (at == 0 && seg >= 2 && !mbar_wait(&acc_free[set], ((seg >> 1) - 1u) & 1u)) { ok = false; break; }
            tc_fence_after_sync();
#pragma unroll
            for (uint32_t cb = 0; cb < CB; ++cb)
              for (uint32_t pc = 0; pc < (uint32_t)p.pieces; ++pc)
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q)
                  mma_f16(tmem + (set * CB + cb) * NT, umma_desc_advance(ad, cb * 16384u + q * 32u),
                          umma_desc_advance(bd, pc * T::kPiece + q * 32u), idesc, (at | pc | q) != 0 ? 1u : 0u);
            if (at == kSegStages - 1 || s + 1 == s1) { umma_commit(&acc_full[set]); ++seg; }
          }
          umma_commit(&empty[slot]);
        }
      }
      if (!ok) s_abort = 1;
      umma_commit(&fin);  // nothing is left running when tensor memory is freed
      if (!mbar_wait(&fin, 0)) s_abort = 1;
    }
    __syncwarp();
    grid_dependency_wait();
  } else if (warp < 8) {
    if constexpr (NT == 128) setmaxnreg_dec<CB == 2 ? 72 : 152>();
    // ===== expanding warps: thread = column of each column block =====
    const uint32_t c = (uint32_t)tid - 128u, xr = c & 7u;
    uint32_t it = 0;
    bool ok = true;
    for (uint32_t t = tile0; t < p.tiles && ok; t += stride) {
      for (uint32_t s = s0; s < s1; ++s, ++it) {
        const uint32_t slot = it % S, ab = it & 1u;
        if (s_abort || !mbar_wait(&full[slot], (it / S) & 1u)) { ok = false; break; }
        // the A buffer was read last by the MMAs of stage it - 2, whose slot's barrier cannot have gone on: that takes this stage
        if (it >= 2 && !mbar_wait(&empty[(it - 2) % S], ((it - 2) / S) & 1u)) { ok = false; break; }
        const unsigned char* w = ring + slot * T::kSlot + 2 * T::kPiece + c * 16u;
        unsigned char* a = abuf + ab * T::kA + (c >> 3) * 1024u + xr * 128u;
#pragma unroll
        for (uint32_t cb = 0; cb < CB; ++cb) {
          uint4 q[T::kChunks];
#pragma unroll
          for (int u = 0; u < T::kChunks; ++u) q[u] = *reinterpret_cast<const uint4*>(w + u * T::kWChunk + cb * 2048u);
#pragma unroll
          for (int u = 0; u < T::kChunks; ++u) {
            if constexpr (BITS == 4) {
              uint32_t o[16];
              expand_int4(q[u], o);
#pragma unroll
              for (uint32_t i = 0; i < 4; ++i)
                *reinterpret_cast<uint4*>(a + cb * 16384u + (((4u * u + i) ^ xr) << 4)) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
            } else {
              uint32_t o[8];
              expand_int8(q[u], o);
#pragma unroll
              for (uint32_t i = 0; i < 2; ++i)
                *reinterpret_cast<uint4*>(a + cb * 16384u + (((2u * u + i) ^ xr) << 4)) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
            }
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_ready[ab]);
      }
    }
    if (!ok) s_abort = 1;
    grid_dependency_wait();
  } else {
    if constexpr (NT == 128) setmaxnreg_inc<CB == 2 ? 200 : 232>();
    // ===== draining warps: thread = column of one column block =====
    grid_dependency_wait();
    const uint32_t quarter = (uint32_t)warp & 3u, cb = (uint32_t)(warp - 8) >> 2, col = cb * 128u + quarter * 32u + lane;
    const uint32_t lane_base = (quarter * 32u) << 16;
    constexpr int kFinish = NT == 128 ? 8 : 16;  // rows finished together: what the registers beside the sums hold
    unsigned long long acc[NT / 2];
    uint32_t seg = 0;
    auto drain = [&](unsigned long long s2) -> bool {
      const uint32_t set = seg & 1u;
      if (s_abort || !mbar_wait(&acc_full[set], (seg >> 1) & 1u)) return false;
      tc_fence_after_sync();
      const uint32_t at = tmem + lane_base + (set * CB + cb) * NT;
#pragma unroll
      for (int c = 0; c < NT / 16; ++c) {
        uint32_t d[16];
        tmem_ld16(at + 16 * c, d);
        tmem_ld_wait();
        if (c == NT / 16 - 1) {  // the set may be overwritten
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_free[set]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) fma2(acc[8 * c + i], d[2 * i], d[2 * i + 1], s2);
      }
      ++seg;
      return true;
    };
    bool ok = true;
    for (uint32_t t = tile0; t < p.tiles && ok; t += stride) {
      const uint32_t j = cols_of(t) + col, row0 = rows_of(t);
      const bool active = j < p.n;
#pragma unroll
      for (int i = 0; i < NT / 2; ++i) acc[i] = 0ull;
      if constexpr (BITS == 4) {
        const uint32_t g0 = 2 * s0, g1 = min(p.groups, 2 * s1);
        float sc[4];  // the column's scales, four groups ahead
        auto scale_at = [&](uint32_t g) { return active && g < g1 ? __ldg(p.scale + (size_t)g * p.n + j) : 0.0f; };
#pragma unroll
        for (int q = 0; q < 4; ++q) sc[q] = scale_at(g0 + q);
        for (uint32_t g = g0; g < g1 && ok; g += 4) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (g + q >= g1) break;
            const unsigned long long s2 = pair_of(sc[q]);
            sc[q] = scale_at(g + q + 4);
            if (!drain(s2)) { ok = false; break; }
          }
        }
      } else {
        for (uint32_t s = 0; s < nst; s += kSegStages)
          if (!drain(pair_of(1.0f))) { ok = false; break; }
      }
      if (!ok) break;
      if (p.splits > 1) break;  // one tile per cluster: see below
      const float cs = BITS == 8 && active ? __ldg(p.scale + j) : 1.0f, bias = p.epi.bias && active ? __ldg(p.epi.bias + j) : 0.0f;
#pragma unroll
      for (int r = 0; r < NT; r += kFinish) {
        if (row0 + r >= p.m) break;
        float v[kFinish];
#pragma unroll
        for (int i = 0; i < kFinish / 2; ++i) { v[2 * i] = low_of(acc[r / 2 + i]); v[2 * i + 1] = high_of(acc[r / 2 + i]); }
        finish_rows<kFinish>(p, p.m, v, row0 + r, j, active, cs, bias);
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
      uint32_t owner = 0, at = 0;
#pragma unroll
      for (int r = 0; r < NT; ++r) {
        st_cluster_f32(red + ((size_t)split * rows_per + at) * T::kCols + col, owner, (r & 1) ? high_of(acc[r / 2]) : low_of(acc[r / 2]));
        if (++at == rows_per) { at = 0; ++owner; }
      }
      cluster_sync_all();
      if (!s_abort) {
        const float cs = BITS == 8 && active ? __ldg(p.scale + j) : 1.0f, bias = p.epi.bias && active ? __ldg(p.epi.bias + j) : 0.0f;
        const uint32_t first = split * rows_per, last = min(first + rows_per, (uint32_t)NT);
        for (uint32_t r = first; r < last; r += 8) {
          if (row0 + r >= p.m) break;
          float v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = 0.0f;
          for (uint32_t q = 0; q < p.splits; ++q) {
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i)
              if (r + i < last) v[i] += red[((size_t)q * rows_per + (r - first) + i) * T::kCols + col];
          }
          finish_rows<8>(p, min(p.m, row0 + last), v, row0 + r, j, active, cs, bias);
        }
      }
    }
  }
  if (p.splits > 1 && warp < 8) {  // the draining warps' two
    __syncwarp();
    cluster_sync_all();
    cluster_sync_all();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (s_abort && tid == 0) atomicExch(p.status, 3);
  if (warp == 2) tmem_dealloc(tmem, T::kTmem);
}

template <int BITS, int CB, int NT>
cudaError_t launch(ruai_ctx* c, const Params& p) {
  using T = Tile<BITS, CB, NT>;
  static bool attr_done[64] = {};
  if (!attr_done[c->ordinal & 63]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel<BITS, CB, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::kSmem);
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
  return cudaLaunchKernelEx(&cfg, gemm_tc_kernel<BITS, CB, NT>, p);
}

struct Shape { uint32_t cb, nt, splits; };

// The tile and the number of splits of k: a model of the launch in clocks.  A stage costs what its MMAs take (16 x 64 clocks,
// 8 x 64, 8 x 48) or, with one piece, what expanding and draining take; a wave of CTAs costs a fixed part and one for the
// epilogue; a split adds the exchange.
Shape choose(const ruai_ctx* c, uint32_t m, uint32_t n, uint32_t stages, int pieces) {
  struct Cand { uint32_t cb, nt; double stage2, stage1, epilogue; };
  const Cand cand[3] = {{2, 128, 1100, 750, 6000}, {1, 128, 620, 480, 5000}, {1, 64, 440, 360, 3000}};
  Shape best = {1, 64, 1};
  double best_t = 1e300;
  for (const Cand& d : cand) {
    const uint32_t tiles = ((n + d.cb * 128 - 1) / (d.cb * 128)) * ((m + d.nt - 1) / d.nt);
    for (uint32_t s = 1; s <= 8; ++s) {
      const uint32_t per = (stages + s - 1) / s;
      if (s > 1 && (per < 2 || (s - 1) * per >= stages)) continue;
      // clusters do not fill every SM: groups of SMs are not multiples of their size
      const uint32_t room = s > 1 ? (uint32_t)c->sm_count * 15u / 16u / s : (uint32_t)c->sm_count;
      if (room == 0) continue;
      const double waves = (double)((tiles + room - 1) / room);
      const double t = 4000.0 + waves * ((s > 1 ? 4000.0 : 0.0) + per * (pieces == 2 ? d.stage2 : d.stage1) + d.epilogue / s) + (s > 1 ? 2500.0 : 0.0);
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
  // fp16 and bf16 activations are one fp16 piece (bf16: after the row's scaling); not when a norm multiplies them
  const int pieces = x_dtype == RUAI_F32 || pro.norm_w ? 2 : 1;
  Shape sh = choose(c, m, w->n, stages, pieces);
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
  sp.xs = reinterpret_cast<unsigned char*>(c->partial);
  sp.rowf = reinterpret_cast<float*>(sp.xs + xs_bytes);
  RUAI_CUDA(c, ruai_launch(c, xsplit_kernel, dim3(m), dim3(kSplitThreads), 0, true, sp));
  Params p;
  p.w = (const uint4*)w->data; p.scale = w->scale; p.xs = sp.xs; p.rowf = sp.rowf; p.m = m; p.n = w->n; p.chunks = w->chunks; p.groups = groups;
  p.stages = stages; p.splits = sh.splits; p.stages_per_split = (stages + sh.splits - 1) / sh.splits;
  p.row_blocks = row_blocks; p.tiles = row_blocks * col_tiles; p.pieces = pieces;
  p.out = out; p.status = c->status; p.epi = epi;
  cudaError_t e;
  if (w->bits == 8)
    e = sh.cb == 2 ? launch<8, 2, 128>(c, p) : sh.nt == 128 ? launch<8, 1, 128>(c, p) : launch<8, 1, 64>(c, p);
  else
    e = sh.cb == 2 ? launch<4, 2, 128>(c, p) : sh.nt == 128 ? launch<4, 1, 128>(c, p) : launch<4, 1, 64>(c, p);
  if (e != cudaSuccess) return ruai_fail(c, RUAI_ERR_CUDA, "prefill GEMM launch failed: %s", cudaGetErrorString(e));
  return RUAI_OK;
}
