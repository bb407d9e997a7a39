// Causal attention over the KV cache for many query positions on the tensor cores (tcgen05): what attn_prefill.cu computes, with
// both products as matrix instructions at f32's precision.
//
// Precision.  Every f32 operand is scaled by a power of two (a query row's own; one per tile of 64 keys for the keys and one for the
// values; 2^14 for the probabilities) so that its largest magnitude lies below 2^15, and split into two fp16 pieces,
// x = hi + 2^-12 lo: 22 bits down to 2^-28 of the largest, then a quantum of 2^-50 of it.  A product takes three of the four products
// of pieces; the lo ones go first and the first hi one scales them by 2^-12 (exact).  The tensor core adds a tile's 64 keys (a
// score's head dimension) only: sums over tiles, the running softmax and its exponentials are f32 in registers.  A tile with an
// infinity or a NaN in it has a factor of NaN, and a CTA that meets one works its rows out again in f32, key by key: an infinite key may score
// -inf, and what a row does not see does not reach it, whereas 0 x inf is NaN in a product of tiles.  (In a query they make its row NaN either way.)
//
// The decoders built from a list of layers (p.pieces is 0) stay on attn_prefill.cu.  They round every layer's output to bf16, and
// sums in another order turn some of those roundings: their outputs would be others (2.3e-3 of a norm) without being nearer to 64 bits, and
// where a choice of experts follows, other experts.
//
// attn_split_kernel writes the pieces of keys and values once, in the form the tensor core reads (K-major, 128-byte swizzle; values
// transposed), so that a tile is one bulk copy for each of the query tiles that see it.
//
// attn_tc_kernel: a CTA owns 128 rows (queries x the query heads of a KV head).  One thread copies tiles, one issues
// the MMAs (scores of tile t + 1 ahead of the values of tile t), and 4 CS warps are the softmax: thread = row and a CS-th of the
// tile's keys, and of the output's columns.  Scores lie in tensor memory twice, probabilities (the A operand of the second product)
// and a tile's weighted values once; the latter are read out and added up in registers while the next tile's scores are made.
// Every mbarrier wait is bounded.
//
// Errors against 64 bits (norms over the output; heads of 16 to 192; f32 units | here): smaller nearly everywhere, as a row's sums are over tiles
// (heads of 128, normal queries, keys and values: 128 keys 2.7e-7 | 2.2e-7, 1030 keys 6.9e-7 | 3.4e-7; scores of 40 1.3e-6 | 6.1e-7).  Larger with few
// keys only: values around a common offset, 128 keys 1.4e-7 | 1.7e-7, 500 keys 2.4e-7 | 1.9e-7 (the tensor core's sums truncate); heads of 16 1.49e-7 | 1.55e-7.
//
// What bounds it: the softmax warps (scores read out, scaled, exponentials, split into pieces, and a tile's values read out and added up), whose
// waits for tensor memory leave half of the issue slots empty; the MMAs keep the tensor pipe busy for 35 % (for heads of 128 six products of 128 x 64 x
// 128 take 1540 clocks a tile at least, of some 6000).  attn_tc_kernel<4, 64> spills 100 bytes a thread.  2000 tokens of the 8B shape
// (32 heads of 128, 8 of keys): 180 to 200 us a layer and 23 for the split, where the f32 units took 1541.  Two warps per row and tile (CS = 2) where the values are at
// most 64 wide, else four: the registers that hold the output then leave room for the products' read-out.
#include <algorithm>

#include "common.cuh"
#include "decode_ops.cuh"
#include "pipeline.cuh"

namespace {

using namespace pipe;

constexpr int kKeys = 64;      // keys per tile
constexpr int kRows = 128;     // rows per CTA: the MMA's M
constexpr int kControl = 2;    // warps that do not own rows: copies, MMAs
constexpr int kLoShift = 12;
constexpr float kLoScale = 4096.0f;
constexpr uint32_t kSmemMax = 227 * 1024 - 1024 - 5120;  // what a CTA can have, less the alignment of operands and the static part

struct Pieces {
  unsigned char* k;   // [B * KV][tiles][piece][block of 64 elements][64 keys][128 bytes]
  unsigned char* v;   // [B * KV][tiles][piece][vdp][128 bytes: 64 keys]
  float* factor;      // [B * KV][tiles][2]: what a tile's scores and weighted values are multiplied by
  uint32_t tiles, blocks, vdp, kslots, vslots, tmem, rep, b0;
};

__device__ __forceinline__ uint32_t magnitude(float v) {  // of a finite number, as ordered bits; 0 for the others
  const uint32_t a = __float_as_uint(v) & 0x7FFFFFFFu;
  return a < 0x7F800000u ? a : 0u;
}
// The power of two that brings the largest magnitude (bits) into [2^14, 2^15), and its inverse.
__device__ __forceinline__ void scale_of(uint32_t largest, float& f, float& back) {
  const int ex = (int)(largest >> 23) - 127;
  const int e = largest ? min(14 - ex, 126) : 0;
  f = __uint_as_float((uint32_t)(e + 127) << 23);
  back = __uint_as_float((uint32_t)(127 - e) << 23);
}
__device__ __forceinline__ uint32_t half2_bits(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// Two numbers as packed hi and lo pieces.
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = half2_bits(a, b);
  const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  lo = half2_bits((a - h.x) * kLoScale, (b - h.y) * kLoScale);
}
__device__ __forceinline__ bool finite(const float4& v) {
  return isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w);
}

__device__ __forceinline__ uint32_t block_max(uint32_t v, uint32_t* red) {
  v = __reduce_max_sync(0xFFFFFFFFu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  for (uint32_t w = 0; w < blockDim.x / 32; ++w) v = max(v, red[w]);
  return v;
}

constexpr int kSplitThreads = 256;

// grid (tiles, sequences * KV): 64 keys and their values.
__global__ void __launch_bounds__(kSplitThreads) attn_split_kernel(const AttnParams p, const Pieces s) {
  extern __shared__ float vs[];  // [64][hd + 1]
  __shared__ uint32_t red[kSplitThreads / 32];
  grid_dependency_wait();
  grid_launch_dependents();
  const uint32_t tile = blockIdx.x, k0 = tile * kKeys, tid = threadIdx.x, n = (uint32_t)*p.len + p.T;
  if (k0 >= n || n > p.cap) return;  // beyond the cache: the attention kernel reports it
  const uint32_t nk = min((uint32_t)kKeys, n - k0), hd = p.hd;
  const uint32_t b = s.b0 + blockIdx.y / p.KV, kvh = blockIdx.y % p.KV;
  const size_t bk = (size_t)b * p.KV + kvh;
  const float* kbase = p.kcache + bk * p.cap * hd;
  const float* vbase = p.vcache + bk * p.cap * hd;
  auto key4 = [&](uint32_t k, uint32_t e) { return *reinterpret_cast<const float4*>(kbase + (size_t)(k0 + k) * hd + e); };  // of key k0 + k
  auto mag4 = [](const float4& v) { return max(max(magnitude(v.x), magnitude(v.y)), max(magnitude(v.z), magnitude(v.w))); };
  uint32_t km = 0, vm = 0;
  bool odd = false;
  for (uint32_t i = tid; i < nk * (hd / 4); i += kSplitThreads) {
    const float4 v = key4(i / (hd / 4), 4 * (i % (hd / 4)));
    km = max(km, mag4(v));
    odd = odd || !finite(v);
  }
  for (uint32_t i = tid; i < kKeys * (hd / 4); i += kSplitThreads) {
    const uint32_t k = i / (hd / 4), e = 4 * (i % (hd / 4));
    const float4 v = k < nk ? *reinterpret_cast<const float4*>(vbase + (size_t)(k0 + k) * hd + e) : make_float4(0.f, 0.f, 0.f, 0.f);
    float* d = vs + k * (hd + 1) + e;
    d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    vm = max(vm, mag4(v));
    odd = odd || !finite(v);
  }
  km = block_max(km, red);
  vm = block_max(vm, red);
  odd = __syncthreads_or(odd);
  float kf, kback, vf, vback;
  scale_of(km, kf, kback);
  scale_of(vm, vf, vback);
  const size_t at = (size_t)blockIdx.y * s.tiles + tile;
  if (tid == 0) {
    s.factor[2 * at] = odd ? __int_as_float(0x7fc00000) : kback * (p.scale * 1.44269504088896341f);  // scores in powers of two
    s.factor[2 * at + 1] = vback * (1.0f / 16384.0f);
  }
  const uint32_t piece = s.blocks * (kKeys * 128);
  unsigned char* kd = s.k + at * 2 * piece;
  for (uint32_t i = tid; i < kKeys * s.blocks * 8; i += kSplitThreads) {  // (key, chunk of eight elements)
    const uint32_t c = i % (s.blocks * 8), k = i / (s.blocks * 8);
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t e = 8 * c + 4 * h;
      const float4 v = k < nk && e < hd ? key4(k, e) : make_float4(0.f, 0.f, 0.f, 0.f);
      split2(v.x * kf, v.y * kf, hi[2 * h], lo[2 * h]);
      split2(v.z * kf, v.w * kf, hi[2 * h + 1], lo[2 * h + 1]);
    }
    unsigned char* dst = kd + (c >> 3) * (kKeys * 128) + k * 128 + (((c ^ k) & 7u) << 4);
    *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(dst + piece) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
  unsigned char* vdst = s.v + at * 2 * s.vdp * 128;
  for (uint32_t i = tid; i < s.vdp * 8; i += kSplitThreads) {  // (column of the values, chunk of eight keys)
    const uint32_t c = i & 7u, r = i >> 3;
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const float a = r < hd ? vs[(8 * c + 2 * h) * (hd + 1) + r] : 0.0f, d = r < hd ? vs[(8 * c + 2 * h + 1) * (hd + 1) + r] : 0.0f;
      split2(a * vf, d * vf, hi[h], lo[h]);
    }
    unsigned char* dst = vdst + r * 128 + (((c ^ r) & 7u) << 4);
    *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(dst + s.vdp * 128) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]),
               "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

__device__ __forceinline__ float exp2_of(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Two f32 operations in one instruction, each rounded like fmaf and a product.
__device__ __forceinline__ unsigned long long pair_of(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(__float_as_uint(a)), "r"(__float_as_uint(b)));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// The rows of a CTA again where its tiles hold infinities or NaN: a warp per row, a key at a time, in f32.
__device__ void rows_in_f32(const AttnParams& p, uint32_t b, uint32_t kvh, uint32_t rep, uint32_t past, uint32_t q0, uint32_t nq, uint32_t first, uint32_t step) {
  constexpr int kMost = 6;  // elements of a head per lane: heads above 192 are not taken
  const uint32_t lane = threadIdx.x & 31u, hd = p.hd;
  const float* kbase = p.kcache + ((size_t)b * p.KV + kvh) * p.cap * hd;
  const float* vbase = p.vcache + ((size_t)b * p.KV + kvh) * p.cap * hd;
  for (uint32_t r = first; r < nq * rep; r += step) {
    const size_t token = (size_t)b * p.T + q0 + r / rep;
    const uint32_t head = kvh * rep + r % rep;
    float q[kMost], o[kMost], m = -INFINITY, l = 0.0f;
#pragma unroll
    for (int j = 0; j < kMost; ++j) {
      const uint32_t e = lane + 32u * j;
      q[j] = e < hd ? p.q[token * p.q_ld + (size_t)head * hd + e] : 0.0f;
      o[j] = 0.0f;
    }
    for (uint32_t k = 0; k <= past + q0 + r / rep; ++k) {
      float a = 0.0f;
#pragma unroll
      for (int j = 0; j < kMost; ++j) {
        const uint32_t e = lane + 32u * j;
        if (e < hd) a = fmaf(q[j], kbase[(size_t)k * hd + e], a);
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xFFFFFFFFu, a, off);
      a *= p.scale;
      if (a == -INFINITY) continue;
      const float m_new = fmaxf(m, a), corr = m == -INFINITY ? 0.0f : expf(m - m_new), pr = expf(a - m_new);
      l = fmaf(l, corr, pr);
      m = m_new;
#pragma unroll
      for (int j = 0; j < kMost; ++j) {
        const uint32_t e = lane + 32u * j;
        if (e < hd) o[j] = fmaf(pr, vbase[(size_t)k * hd + e], o[j] * corr);
      }
    }
#pragma unroll
    for (int j = 0; j < kMost; ++j) {
      const uint32_t e = lane + 32u * j;
      if (e < hd) p.out[token * p.out_ld + (size_t)head * hd + e] = o[j] / l;
    }
  }
}

// Tensor memory: scores [2][64 columns], probabilities (hi 32 columns, lo 32), weighted values.
constexpr uint32_t kProbCol = 2 * kKeys, kValueCol = kProbCol + kKeys;

// CS: warps that share a row (keys of a tile, columns of the output).  OC: columns of the output per thread.
template <int CS, int OC>
__global__ void __launch_bounds__((kControl + 4 * CS) * 32, CS == 2 && OC == 32 ? 2 : 1) attn_tc_kernel(const AttnParams p, const Pieces s) {
  constexpr int kSoftWarps = 4 * CS, SC = kKeys / CS;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t q_ready, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], s_free[2], p_ready, o_full, fin;
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort;
  __shared__ float s_max[2][CS][kRows];  // a tile's row maxima by part; at the end the row sums
  __shared__ float s_qback[kRows];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // swizzled operands start on 1024-byte boundaries
  const uint32_t q_piece = s.blocks * (kRows * 128), k_piece = s.blocks * (kKeys * 128), k_slot = 2 * k_piece, v_piece = s.vdp * 128, v_slot = 2 * v_piece;
  const uint32_t off_k = 2 * q_piece, off_v = off_k + s.kslots * k_slot;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t hd = p.hd, rep = s.rep, qt = kRows / rep;  // queries per CTA
  const uint32_t bk = blockIdx.y, b = s.b0 + bk / p.KV, kvh = bk % p.KV;
  const uint32_t q0 = (gridDim.x - 1u - blockIdx.x) * qt;  // the tiles with the most keys first: they are the long ones
  const uint32_t head0 = kvh * rep;

  if (tid == 0) {
    mbar_init(&q_ready, kSoftWarps); mbar_init(&p_ready, kSoftWarps); mbar_init(&o_full, 1); mbar_init(&fin, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&s_free[i], kSoftWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_abort = 0;
  }
  __syncwarp();
  if (warp == 1) tmem_alloc(&s_tmem, s.tmem);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = s_tmem;
  grid_dependency_wait();
  grid_launch_dependents();
  const uint32_t past = (uint32_t)*p.len, nq = min(qt, p.T - q0);
  uint32_t kmax = past + q0 + nq;  // keys 0 .. kmax - 1 are seen by the tile's last query
  const bool over = past + p.T > p.cap;  // the device's position is not the host's: touch nothing beyond the cache, tell the host
  if (over) {
    kmax = 0;
    if (tid == 0 && p.status) atomicCAS(p.status, 0, 5);
  }
  const uint32_t ntiles = (kmax + kKeys - 1) / kKeys;

  if (warp < kControl) {
    if (warp == 0 && elect_one()) {
      // ===== copies =====
      const unsigned char* kbase = s.k + (size_t)bk * s.tiles * k_slot;
      const unsigned char* vbase = s.v + (size_t)bk * s.tiles * v_slot;
      // the keys of tile i, then the values of tile i - 1: keys are needed sooner and freed sooner
      uint32_t k = 0, v = 0;  // requested
      for (uint32_t i = 0; i <= ntiles && !s_abort && ntiles; ++i) {
        if (i < ntiles) {
          const uint32_t slot = i % s.kslots;
          if (i >= s.kslots && !mbar_wait(&k_empty[slot], (i / s.kslots - 1u) & 1u)) { s_abort = 1; break; }
          mbar_expect_tx(&k_full[slot], k_slot);
          bulk_load(smem + off_k + slot * k_slot, kbase + (size_t)i * k_slot, k_slot, &k_full[slot]);
          ++k;
        }
        if (i > 0) {
          const uint32_t slot = v % s.vslots;
          if (v >= s.vslots && !mbar_wait(&v_empty[slot], (v / s.vslots - 1u) & 1u)) { s_abort = 1; break; }
          mbar_expect_tx(&v_full[slot], v_slot);
          bulk_load(smem + off_v + slot * v_slot, vbase + (size_t)v * v_slot, v_slot, &v_full[slot]);
          ++v;
        }
      }
      // leave no copy in flight into shared memory that another CTA may get, whoever gives up
      for (uint32_t u = k > s.kslots ? k - s.kslots : 0; u < k; ++u) (void)mbar_wait(&k_full[u % s.kslots], (u / s.kslots) & 1u);
      for (uint32_t u = v > s.vslots ? v - s.vslots : 0; u < v; ++u) (void)mbar_wait(&v_full[u % s.vslots], (u / s.vslots) & 1u);
    } else if (warp == 1 && elect_one()) {
      // ===== MMAs: the scores of tile i, then the weighted values of tile i - 1 =====
      const uint32_t idesc_s = (1u << 4) | ((uint32_t)(kKeys >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
      const uint32_t idesc_v = (1u << 4) | ((s.vdp >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
      const uint64_t qd = umma_desc_sw128(smem_u32(smem)), kd = umma_desc_sw128(smem_u32(smem + off_k)), vd0 = umma_desc_sw128(smem_u32(smem + off_v));
      const uint32_t steps = (hd + 15) / 16;
      bool ok = ntiles == 0 || mbar_wait(&q_ready, 0);
      for (uint32_t i = 0; i <= ntiles && ok && ntiles; ++i) {
        if (i < ntiles) {
          const uint32_t ks = i % s.kslots, sb = i & 1u, d = tmem + sb * kKeys;
          if (s_abort || !mbar_wait(&k_full[ks], (i / s.kslots) & 1u) || (i >= 2 && !mbar_wait(&s_free[sb], (i / 2 - 1u) & 1u))) { ok = false; break; }
          tc_fence_after_sync();
          const uint64_t kt = umma_desc_advance(kd, ks * k_slot);
          auto at_q = [&](uint32_t e) { return umma_desc_advance(qd, (e >> 2) * (kRows * 128) + (e & 3u) * 32u); };
          auto at_k = [&](uint32_t e) { return umma_desc_advance(kt, (e >> 2) * (kKeys * 128) + (e & 3u) * 32u); };
          for (uint32_t e = 0; e < steps; ++e) {
            umma_f16_ss(d, at_q(e), umma_desc_advance(at_k(e), k_piece), idesc_s, e != 0 ? 1u : 0u);
            umma_f16_ss(d, umma_desc_advance(at_q(e), q_piece), at_k(e), idesc_s, 1u);
          }
          umma_f16_ss_after<kLoShift>(d, at_q(0), at_k(0), idesc_s);
          for (uint32_t e = 1; e < steps; ++e) umma_f16_ss(d, at_q(e), at_k(e), idesc_s, 1u);
          umma_commit(&k_empty[ks]);
          umma_commit(&s_full[sb]);
        }
        if (i > 0) {
          const uint32_t t = i - 1, vs = t % s.vslots, d = tmem + kValueCol, ph = tmem + kProbCol, pl = ph + kKeys / 2;
          if (s_abort || !mbar_wait(&v_full[vs], (t / s.vslots) & 1u) || !mbar_wait(&p_ready, t & 1u)) { ok = false; break; }
          tc_fence_after_sync();
          const uint64_t vt = umma_desc_advance(vd0, vs * v_slot);
#pragma unroll
          for (uint32_t e = 0; e < kKeys / 16; ++e) {
            umma_f16_ts(d, ph + e * 8, umma_desc_advance(vt, v_piece + e * 32u), idesc_v, e != 0 ? 1u : 0u);
            umma_f16_ts(d, pl + e * 8, umma_desc_advance(vt, e * 32u), idesc_v, 1u);
          }
          umma_f16_ts_after<kLoShift>(d, ph, vt, idesc_v);
#pragma unroll
          for (uint32_t e = 1; e < kKeys / 16; ++e) umma_f16_ts(d, ph + e * 8, umma_desc_advance(vt, e * 32u), idesc_v, 1u);
          umma_commit(&v_empty[vs]);
          umma_commit(&o_full);
        }
      }
      if (!ok) s_abort = 1;
      umma_commit(&fin);  // nothing is left running when tensor memory is freed
      if (!mbar_wait(&fin, 0)) s_abort = 1;
    }
    __syncwarp();
  } else {
    // ===== softmax: thread = row, part `cp` of a tile's keys and of the output's columns =====
    const uint32_t quarter = (uint32_t)warp & 3u, cp = (uint32_t)(warp - kControl) >> 2, row = quarter * 32u + lane;
    // queries as pieces: a warp's rows of shared memory, one row at a time, a lane per four elements
    for (uint32_t r = warp - kControl; r < (uint32_t)kRows; r += kSoftWarps) {
      const uint32_t qi = r / rep, h = r % rep;
      const bool in = r < qt * rep && qi < nq;
      const float* src = p.q + (size_t)(b * p.T + q0 + qi) * p.q_ld + (size_t)(head0 + h) * hd;
      float4 v[2];
      uint32_t mx = 0;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t e = 4 * (lane + 32 * j);
        v[j] = in && e < hd ? *reinterpret_cast<const float4*>(src + e) : make_float4(0.f, 0.f, 0.f, 0.f);
        mx = max(mx, max(max(magnitude(v[j].x), magnitude(v[j].y)), max(magnitude(v[j].z), magnitude(v[j].w))));
      }
      mx = __reduce_max_sync(0xFFFFFFFFu, mx);
      float f, back;
      scale_of(mx, f, back);
      if (lane == 0) s_qback[r] = back;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t e = 4 * (lane + 32 * j);
        if (e < s.blocks * 64) {
          uint2 hi, lo2;
          split2(v[j].x * f, v[j].y * f, hi.x, lo2.x);
          split2(v[j].z * f, v[j].w * f, hi.y, lo2.y);
          unsigned char* dst = smem + (e >> 6) * (kRows * 128) + r * 128 + ((((e & 63u) >> 3) ^ (r & 7u)) << 4) + (e & 4u) * 2u;
          *reinterpret_cast<uint2*>(dst) = hi;
          *reinterpret_cast<uint2*>(dst + q_piece) = lo2;
        }
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(&q_ready);
    asm volatile("bar.sync 8, %0;" ::"n"(kSoftWarps * 32) : "memory");  // the rows' factors

    const float qback = s_qback[row];
    const uint32_t qi = row / rep, h = row % rep;
    const uint32_t qpos = past + q0 + min(qi, nq - 1u);  // the last key this row's query sees (rows without a query: any)
    const uint32_t lanes = (quarter * 32u) << 16;
    float m_run = -INFINITY, l_run = 0.0f, corr_prev = 0.0f, vf_prev = 0.0f;
    bool odd = false;  // a tile's factor was NaN: the same for the whole CTA
    unsigned long long sums[OC / 2];  // pairs of columns
#pragma unroll
    for (int j = 0; j < OC / 2; ++j) sums[j] = 0ull;
    // A warp whose wait ran out walks on without waiting, so that a quarter's warps meet at every barrier below.
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) {  // the same answer for the whole warp
      if (ok) ok = __all_sync(0xFFFFFFFFu, !s_abort && mbar_wait(bar, parity));
      if (!ok) s_abort = 1;
      tc_fence_after_sync();
    };
    // the weighted values of tile t: out of tensor memory, onto the sums
    auto drain = [&](uint32_t t) {
      wait(&o_full, t & 1u);
      const bool same = __all_sync(0xFFFFFFFFu, corr_prev == 1.0f);  // no row's maximum has grown
      const unsigned long long v2 = pair_of(vf_prev, vf_prev), c2 = pair_of(corr_prev, corr_prev);
#pragma unroll
      for (int c = 0; c < OC; c += 16) {
        uint32_t d[16];
        tmem_ld16(tmem + lanes + kValueCol + cp * OC + c, d);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const unsigned long long add = pair_of(__uint_as_float(d[2 * j]), __uint_as_float(d[2 * j + 1]));
          sums[c / 2 + j] = fma2(add, v2, same ? sums[c / 2 + j] : mul2(sums[c / 2 + j], c2));
        }
      }
    };
    const float* factor = s.factor + (size_t)bk * s.tiles * 2;
    float2 fac = ntiles ? *reinterpret_cast<const float2*>(factor) : make_float2(0.f, 0.f);
    for (uint32_t i = 0; i < ntiles; ++i) {
      const uint32_t sb = i & 1u, key0 = i * kKeys + cp * SC;  // this thread's first key
      const float2 cur = fac;
      odd = odd || cur.x != cur.x;
      if (i + 1 < ntiles) fac = *reinterpret_cast<const float2*>(factor + 2 * (i + 1));
      wait(&s_full[sb], (i >> 1) & 1u);
      float sc[SC];
#pragma unroll
      for (int c = 0; c < SC; c += 16) {
        uint32_t d[16];
        tmem_ld16(tmem + lanes + sb * kKeys + cp * SC + c, d);
#pragma unroll
        for (int j = 0; j < 16; ++j) sc[c + j] = __uint_as_float(d[j]);
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_free[sb]);
      // which of the keys the row sees: bit j = key0 + j <= qpos
      const uint32_t all = SC == 32 ? 0xFFFFFFFFu : (1u << (SC & 31)) - 1u;
      const uint32_t seen = qpos < key0 ? 0u : qpos - key0 >= 31u ? all : ((2u << (qpos - key0)) - 1u) & all;
      const bool whole = __all_sync(0xFFFFFFFFu, seen == all);
      if (!whole) {
#pragma unroll
        for (int j = 0; j < SC; ++j) sc[j] = (seen >> j) & 1u ? sc[j] : -INFINITY;
      }
      const float f = qback * cur.x;
      float mx = sc[0];
#pragma unroll
      for (int j = 1; j < SC; ++j) mx = fmaxf(mx, sc[j]);
      mx = mx == -INFINITY ? mx : mx * f;  // (f may be 0)
      s_max[sb][cp][row] = mx;
      asm volatile("bar.sync %0, %1;" ::"r"(1 + quarter), "n"(CS * 32) : "memory");
#pragma unroll
      for (int c = 0; c < CS; ++c) mx = fmaxf(mx, s_max[sb][c][row]);
      const float m_new = fmaxf(m_run, mx), m_use = m_new == -INFINITY ? 0.0f : m_new;
      const float corr = m_run == -INFINITY ? 0.0f : exp2_of(m_run - m_new);
      float sum = 0.0f;
#pragma unroll
      for (int j = 0; j < SC; ++j) {
        const float e = exp2_of(fmaf(sc[j], f, -m_use));
        sc[j] = whole || ((seen >> j) & 1u) ? e : 0.0f;
        sum += sc[j];
      }
      l_run = fmaf(l_run, corr, sum);
      m_run = m_new;
      if (i > 0) drain(i - 1);  // also: the probabilities of tile i - 1 have been read
      corr_prev = corr;
      vf_prev = cur.y;
#pragma unroll
      for (int c = 0; c < SC; c += 16) {
        uint32_t hi[8], lo2[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) split2(sc[c + 2 * j] * 16384.0f, sc[c + 2 * j + 1] * 16384.0f, hi[j], lo2[j]);
        tmem_st8(tmem + lanes + kProbCol + (cp * SC + c) / 2, hi);
        tmem_st8(tmem + lanes + kProbCol + kKeys / 2 + (cp * SC + c) / 2, lo2);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready);
    }
    if (ntiles) drain(ntiles - 1);
    // the parts' row sums
    asm volatile("bar.sync %0, %1;" ::"r"(1 + quarter), "n"(CS * 32) : "memory");
    s_max[0][cp][row] = l_run;
    asm volatile("bar.sync %0, %1;" ::"r"(1 + quarter), "n"(CS * 32) : "memory");
    float l = 0.0f, o[OC];
#pragma unroll
    for (int c = 0; c < CS; ++c) l += s_max[0][c][row];
#pragma unroll
    for (int j = 0; j < OC; ++j) o[j] = __uint_as_float((uint32_t)(sums[j / 2] >> (32 * (j & 1))));
    if (odd) {
      if (!over && !s_abort) rows_in_f32(p, b, kvh, rep, past, q0, nq, (uint32_t)(warp - kControl), kSoftWarps);
    } else if (!over && !s_abort && row < qt * rep && qi < nq) {
      const size_t token = (size_t)b * p.T + q0 + qi;
      const uint32_t c0 = cp * OC;
      const float inv = 1.0f / l;
      float* dst = p.out + token * p.out_ld + (size_t)(head0 + h) * hd;
#pragma unroll
      for (int j = 0; j < OC; j += 4)
        if (c0 + j < hd) *reinterpret_cast<float4*>(dst + c0 + j) = make_float4(o[j] * inv, o[j + 1] * inv, o[j + 2] * inv, o[j + 3] * inv);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (s_abort && tid == 0 && p.status) atomicCAS(p.status, 0, 3);
  if (warp == 1) tmem_dealloc(tmem, s.tmem);
}

template <int CS, int OC>
cudaError_t launch_tc(ruai_ctx* c, const AttnParams& p, const Pieces& s, dim3 grid, uint32_t smem) {
  static bool done[64] = {};
  if (!done[c->ordinal & 63]) {
    cudaError_t e = cudaFuncSetAttribute(attn_tc_kernel<CS, OC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSmemMax + 1024));
    if (e != cudaSuccess) return e;
    done[c->ordinal & 63] = true;
  }
  return ruai_launch(c, attn_tc_kernel<CS, OC>, grid, dim3((kControl + 4 * CS) * 32), smem, true, p, s);
}

constexpr size_t kScratchMost = 256u << 20;  // a step's pieces at a time
// Fewer tokens leave most of the 128 rows and of the tensor core's time to nothing while the splitting costs a launch.  Us of a whole prompt, here |
// attn_prefill.cu: 64 tokens of the 8B shape's 2 layers 656 | 648, of the 135M shape's 10 718 | 687; 96 tokens 700 | 718, 768 | 796, of
// the 1.1B shape's 6 803 | 836, of GPT-2 1056 | 1126; 160 tokens 1080 | 1123, 833 | 937, 1105 | 1197, 1226 | 1410.
constexpr uint32_t kFromTokens = 96;

}  // namespace

// 1: launched; 0: this shape is not taken; < 0: error.  `p`: as ruai_attention_prefill has completed it.
int ruai_attention_prefill_tc(ruai_ctx* c, const AttnParams& p, uint32_t B, uint32_t rep) {
  if (!c->use_tc || !p.pieces || p.T < kFromTokens || rep > 64) return 0;
  if (p.maps != 1 || p.window || p.keep || p.vd != p.hd || p.vd_out != p.hd || p.out_dtype != RUAI_F32 || p.k_pos || p.sink || p.gate) return 0;
  Pieces s = {};
  s.rep = rep;
  s.blocks = (p.hd + 63) / 64;
  s.vdp = (p.hd + 15) / 16 * 16;
  s.tiles = (p.cap + kKeys - 1) / kKeys;
  s.tmem = s.vdp <= 64 ? 256 : 512;
  const uint32_t q = 2 * s.blocks * kRows * 128, ks = 2 * s.blocks * kKeys * 128, vs = 2 * s.vdp * 128;
  if (q + ks + vs > kSmemMax) return 0;
  s.kslots = q + 2 * ks + vs <= kSmemMax ? 2 : 1;
  s.vslots = q + s.kslots * ks + 2 * vs <= kSmemMax ? 2 : 1;
  const uint32_t smem = q + s.kslots * ks + s.vslots * vs + 1024;
  // sequences at a time: what their pieces take of the scratch
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t k1 = (size_t)p.KV * s.tiles * ks, v1 = (size_t)p.KV * s.tiles * vs, f1 = (size_t)p.KV * s.tiles * 2 * sizeof(float);
  const size_t one = k1 + v1 + f1 + 1024;
  if (one > kScratchMost) return 0;
  const uint32_t per = (uint32_t)std::min<size_t>(B, std::min<size_t>(kScratchMost / one, 65535u / p.KV));
  if (!per) return 0;
  const size_t held = c->partial_bytes;
  if ((size_t)per * one > held) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c->stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) return 0;  // nothing may be allocated
    if (ruai_ctx_reserve(c, (size_t)per * one, 0) != RUAI_OK) {  // no memory for the pieces: the kernel without them, the scratch as it was
      (void)cudaGetLastError();
      return ruai_ctx_reserve(c, held, 0) == RUAI_OK ? 0 : -1;
    }
  }
  unsigned char* at = reinterpret_cast<unsigned char*>(c->partial);
  s.k = at; at += up(per * k1);
  s.v = at; at += up(per * v1);
  s.factor = reinterpret_cast<float*>(at);
  static bool done[64] = {};
  cudaError_t e = cudaSuccess;
  if (!done[c->ordinal & 63]) {
    e = cudaFuncSetAttribute(attn_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kKeys * 257 * 4);
    done[c->ordinal & 63] = e == cudaSuccess;
  }
  const uint32_t qt = kRows / rep;
  for (uint32_t b0 = 0; b0 < B && e == cudaSuccess; b0 += per) {
    const uint32_t nb = std::min(per, B - b0);
    s.b0 = b0;
    e = ruai_launch(c, attn_split_kernel, dim3(s.tiles, nb * p.KV), dim3(kSplitThreads), (size_t)kKeys * (p.hd + 1) * 4, true, p, s);
    const dim3 grid((p.T + qt - 1) / qt, nb * p.KV);
    if (e == cudaSuccess) e = p.hd <= 64 ? launch_tc<2, 32>(c, p, s, grid, smem) : p.hd <= 128 ? launch_tc<4, 32>(c, p, s, grid, smem) : launch_tc<4, 64>(c, p, s, grid, smem);
  }
  if (e != cudaSuccess) { ruai_fail(c, RUAI_ERR_CUDA, "prefill attention launch: %s", cudaGetErrorString(e)); return -1; }
  return 1;
}
