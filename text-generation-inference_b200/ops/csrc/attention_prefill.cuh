// What the prefill attention kernels share: parameters, visible ranges, operand descriptors and the softmax of a group of scores.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "sm100.cuh"

namespace prefill {

using namespace sm100;

constexpr int kD = 128;            // value size of a head
constexpr int kRows = 128;         // query rows per CTA
constexpr int kKeys = 128;         // KV tokens per tile
constexpr int kPage = 16;          // tokens per page
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kSlab = kRows * 128;             // bytes of one [128 rows x 128 bytes] swizzled slab
constexpr int kTileBytes = 2 * kSlab;          // a 128 x 128 tile of 16-bit values: two slabs (32 KB)

struct PrefillParams {
  const __nv_bfloat16* q;       // [T, Hq, 128 or 192]
  const int* block_tables;      // [B, max_blocks]
  const int* cu_seqlens_q;      // [B + 1]
  const int* kv_lens;           // [B]
  const float* k_scale;         // [Hkv] or null (e4m3 pages)
  const float* v_scale;
  __nv_bfloat16* out;           // [T, Hq, 128]
  const int* horizon;           // optional [T]
  const __nv_bfloat16* gate;    // optional [T, ld_gate]: the output of head h is multiplied by the sigmoid of column h
  long long ld_gate;
  int max_blocks, Hq, Hkv, num_blocks;
  float scale, softcap;
  int window;
  int chunk;                    // > 0: a row sees only keys of its own chunk of `chunk` positions
  int keep;                     // first tokens that every row sees whatever its window
  const float* sink;            // [Hq] or null: score of one more key per head that has no value
  int* status;
};

// First KV position that the query at `pos` may see.
__device__ __forceinline__ int first_visible(const PrefillParams& p, int pos) {
  int lo = p.window > 0 ? pos - p.window + 1 : 0;
  if (p.chunk > 0 && pos > 0) lo = max(lo, pos - pos % p.chunk);
  return max(lo, 0);
}

__device__ __forceinline__ void report(int* status, int code) {
  if (status != nullptr) atomicCAS(status, 0, code);
}

// MN-major operand with the 128-byte swizzle (rows = K index, 128 bytes = 64 MN elements per row; groups of 8
// rows 1024 bytes apart; the next 64 MN elements `lbo` bytes further): the layout TMA leaves a [tokens x head]
// tile in.  Canonical form: cute/atom/mma_traits_sm100.hpp, make_umma_desc<Major::MN>.
__device__ __forceinline__ uint64_t make_desc_mn_sw128(uint32_t smem_addr, uint32_t lbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(lbo_bytes >> 4) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
// instruction descriptor: D fp32, A K-major, B K-major or MN-major, fmt 0 = f16, 1 = bf16
__device__ __forceinline__ constexpr uint32_t idesc16(uint32_t fmt, bool b_mn) {
  return (1u << 4) | (fmt << 7) | (fmt << 10) | (0u << 15) | ((b_mn ? 1u : 0u) << 16) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ uint32_t swz_chunk(int row, int chunk) { return static_cast<uint32_t>(row * 128 + ((chunk ^ (row & 7)) << 4)); }
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t (&r)[32]) {
  tmem_ld_32x32b_x32(addr, r);
  tmem_ld_wait(r);
}

// 2^x on the FMA pipe, for x <= 8 (the bf16 kernel's rows may outgrow their reference by 2^8, the e4m3 kernel's x are <= 0): the
// special-function unit does 16 ex2 per cycle and SM and is the busiest unit of a tile (16 K exponentials), so every POLY-th
// probability is computed this way instead, as in FlashAttention-4.  Round x to the nearest integer with the 1.5 * 2^23 trick,
// evaluate a cubic for 2^f on [-0.5, 0.5] (relative error 1.4e-4, well under the 16-bit rounding of P) and add the integer to the
// exponent field (the reduction of W. J. Cody and W. Waite, Software Manual for the Elementary Functions, 1980).
__device__ __forceinline__ float poly_exp2(float x) {
  x = fmaxf(x, -125.f);
  const float t = x + 12582912.f;
  const float f = x - (t - 12582912.f);
  float r = fmaf(0.05502927f, f, 0.24225698f);
  r = fmaf(r, f, 0.69325305f);
  r = fmaf(r, f, 0.99995134f);
  return __int_as_float(__float_as_int(r) + (__float_as_int(t) << 23));
}
__device__ __forceinline__ float fast_tanh(float y) {      // 1 - 2 / (1 + e^(2y)); saturates cleanly at +-1
  return 1.f - __fdividef(2.f, 1.f + fast_exp2(y * (2.f * kLog2e)));
}
// How a softmax thread reads its scores.  Key i of a 32-key group is visible when i - lo lies in [0, range]
// (one unsigned compare); with soft-capping a raw score x becomes cap_out * tanh(x * cap_in), already in log2 units,
// otherwise it is scaled by scale_log2 (> 0) — both after the maximum in the first pass, inside the FMA in the second.
struct ScoreArgs {
  float scale_log2, cap_in, cap_out;
  int lo;
  unsigned range;
};
template <bool MASK>
__device__ __forceinline__ float group_max(const uint32_t (&v)[32], float mx, const ScoreArgs& a) {
  float other = -INFINITY;
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    float x[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      x[e] = __uint_as_float(v[i + e]);
      if (MASK) x[e] = static_cast<unsigned>(i + e - a.lo) <= a.range ? x[e] : -INFINITY;
    }
    mx = fmaxf(fmaxf(mx, x[0]), x[1]);
    other = fmaxf(fmaxf(other, x[2]), x[3]);
  }
  return fmaxf(mx, other);
}
// Probabilities of a 32-key group as sixteen packed 16-bit pairs (fp16 next to fp16 V tiles, bf16 otherwise);
// returns their sum.  m is the row maximum in log2 units.
template <bool MASK, bool CAP, bool F16, int POLY>
__device__ __forceinline__ float group_prob(const uint32_t (&v)[32], uint32_t (&packed)[16], float m, const ScoreArgs& a) {
  float rs0 = 0.f, rs1 = 0.f;
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    float pr[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float x = __uint_as_float(v[i + e]);
      if (CAP) pr[e] = fast_exp2(a.cap_out * fast_tanh(x * a.cap_in) - m);
      else if ((i + e) % POLY == 1) pr[e] = poly_exp2(fmaf(x, a.scale_log2, -m));
      else pr[e] = fast_exp2(fmaf(x, a.scale_log2, -m));
      if (MASK) pr[e] = static_cast<unsigned>(i + e - a.lo) <= a.range ? pr[e] : 0.f;
    }
    rs0 += pr[0];
    rs1 += pr[1];
    if (F16) {
      const __half2 hh = __floats2half2_rn(pr[0], pr[1]);
      packed[i >> 1] = *reinterpret_cast<const uint32_t*>(&hh);
    } else {
      const __nv_bfloat162 bb = __floats2bfloat162_rn(pr[0], pr[1]);
      packed[i >> 1] = *reinterpret_cast<const uint32_t*>(&bb);
    }
  }
  return rs0 + rs1;
}

// Kernels by page type.  `k_pitch`, `v_pitch`: elements from a token's keys (values) to the next token's; dim: 128 or 192 query and
// key elements of a head.  Return the entry points' codes.
int launch_bf16(const PrefillParams& p, int dim, const void* k_cache, const void* v_cache, long long k_pitch, long long v_pitch, int B,
                int max_q, cudaStream_t stream);
int launch_e4m3(const PrefillParams& p, const void* k_cache, const void* v_cache, long long k_pitch, long long v_pitch, int B, int max_q,
                cudaStream_t stream);

}  // namespace prefill
