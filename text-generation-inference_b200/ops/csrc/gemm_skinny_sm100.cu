// GEMMs of a few tokens for sm_100a:   C[M, N] = X[M, K] * W[N, K]^T (+ bias),  M <= 32
//
//   bf16   X, W bf16
//   fp8    X, W e4m3 with block scales (X: 1x128 per token, stored K-block major; W: 128x128)
//   int4   X bf16, W packed 4-bit with a scale and a zero point per group of 128 (or a multiple) input features
//
// A decode step of a lightly loaded server reads every weight for a handful of rows: the weights' way from HBM is the
// bound, and what a launch spends outside of it (filling and draining, and combining partial tiles) is what can be lost.
// The tcgen05 kernels cover at least 128 weight rows per CTA, so a matrix of 4096 or 8192 rows has to be split along K
// over CTAs and put together through global memory; that and 128 KB partial tiles cost them 13 us per launch.  Here a
// CTA owns blocks of 16 weight rows and the WHOLE of K; its eight consumer warps take every eighth K unit each and
// are added up in shared memory at the end.  Nothing crosses CTAs, and a matrix of 4096 rows gives 256 blocks.
//
//   warp 8      one thread brings weights: a TMA box of 16 rows x 1024 bytes (eight pieces of 128 bytes per row, 128-byte
//               swizzle) per stage of 16 KB; int4: also the scales and zero points of its sixteen units
//   warp 9      one thread brings the tokens of eight units (int4: every other of sixteen) per slot, fp8: and their scales.
//               Tokens read by the consumers from global memory kept the load units so busy that the shared loads of the
//               weights queued behind them (32 tokens: 53 us for 28672 x 4096 bf16).
//   warps 0-7   warp w takes piece w of a stage: fragments of `mma.sync.m16n8k16` (weights are its 16 rows, tokens its 8
//               columns) by 16-byte shared loads.  Blocks of a walk over K share the token fragments.
// The order of K inside an MMA is free as long as A and B agree, so a lane takes 16 (32) consecutive bytes of its row as
// they lie.  At up to 32 tokens `mma.sync` keeps up with HBM (24 bytes per clock and SM): a unit of 16 rows x 64 features
// is 4 MMAs per 8 tokens, 8 clocks of the tensor pipe for 2 KB.
//
// fp8 values become fp16 (exact), the products of a 128-deep block accumulate in fp32 and are added to the total times
// both block scales.  4-bit values enter the MMA as 128 + q in bf16 (exact, one instruction per pair); the tokens' sum
// over the group, from MMAs with a matrix of ones that all blocks share, times 128 + z is taken off the group's sum before it
// is multiplied by the fp32 scale.
//
// Settled weights (gemm_skinny.h) are fetched from the moment the launch ahead lets this one be placed: up to 28 MB are in
// shared memory when its tokens are there.  Steps without it / with it, us: 8B for one sequence 1917 / 1762, for 19 2230 / 2175, 70B fp8
// for eight 1877 / 1827, 8B 4-bit for twelve 1835 / 1790.
//
// Waits are bounded (sm100.cuh): on expiry the status word is set and the launch ends with wrong results, never late.
#include <cuda_fp16.h>

#include <atomic>

#include "gemm_skinny.h"
#include "launch.cuh"
#include "sm100.cuh"
#include "tensor_map.cuh"

using namespace sm100;

namespace {

enum : int { kBf16 = 0, kFp8 = 1, kInt4 = 2 };
constexpr int kWarps = 8;                            // consumer warps
constexpr int kThreads = (kWarps + 2) * 32;
constexpr int kRows = 16;                            // weight rows of a block
constexpr int kBlocks = 4;                           // blocks that share a walk over K and its token fragments
constexpr int kTileBytes = kRows * 1024;
constexpr int kSmemMax = 227 * 1024;

template <int FMT, int NT>
struct Cfg {
  static constexpr int kUnitK = FMT == kBf16 ? 64 : 128;          // features of a unit
  static constexpr int kUnits = FMT == kInt4 ? 2 : 1;             // units in 128 bytes of a weight row
  static constexpr int kPieces = FMT == kInt4 ? 2 : 1;            // 128-byte pieces of a token in a unit
  // MMA chains of a unit with scales of its own.  4-bit: one whatever the tokens, so that a token's sums are the same in every
  // instance (two for up to 8 tokens: 28672 x 4096 29.3 us, one 28.9)
  static constexpr int kChains = FMT == kFp8 ? 2 : 1;
  static constexpr int kXRegs = FMT == kBf16 ? 8 : 16;            // B fragments of a unit, per 8 tokens
  static constexpr int kScaleBytes = FMT == kInt4 ? 16 * kRows * 2 : 0;               // of a stage, zero points as many
  static constexpr int kStageBytes = kTileBytes + (FMT == kInt4 ? 1024 : 0);
  static constexpr int kXBytes = kWarps * kPieces * NT * 8 * 128;
  static constexpr int kXScaleBytes = FMT == kFp8 ? kWarps * 8 * 4 : 0;
  static constexpr int kSlotBytes = (kXBytes + kXScaleBytes + 1023) / 1024 * 1024;
  static constexpr int kSlots = FMT == kInt4 ? (NT == 1 ? 3 : 2) : (NT == 1 ? 4 : NT == 2 ? 3 : 2);
  static constexpr int kRedFloats = kBlocks * kRows * NT * 8;     // of one warp; half of the warps write at a time
  static constexpr int kFixed = kSlots * kSlotBytes + kWarps / 2 * kRedFloats * 4 + 1024 + 512;
  static constexpr int kStages = (kSmemMax - kFixed) / kStageBytes < 12 ? (kSmemMax - kFixed) / kStageBytes : 12;
  static constexpr int kSmem = kFixed + kStages * kStageBytes;
  static_assert(FMT != kFp8 || NT == 1, "fp8 takes up to eight tokens");
  static_assert(kStages >= 6 && (2 * kStages + 2 * kSlots) * 8 <= 512, "carve-up of the shared memory");
};

struct Args {
  const float* wscale;            // fp8: [ceil(N / 128), K / 128]
  int has_zp;                     // int4: zero points are given (8 otherwise)
  int group_units;                // int4: units per group
  __nv_bfloat16* C;
  const __nv_bfloat16* bias;
  int M, N, K;
  int* status;
  uint32_t zero;                  // 0 (see `loaded_arrive`)
  int settled;                    // the weights are not written by the launch ahead of this one
};

__device__ __forceinline__ void report(int* status, int code) {
  if (status != nullptr) atomicCAS(status, 0, code);
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_fp16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// two e4m3 values (low / high half of v) as fp16x2
__device__ __forceinline__ uint32_t e4m3_lo(uint32_t v) {
  uint32_t r;
  asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, lo;\n\t}" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ uint32_t e4m3_hi(uint32_t v) {
  uint32_t r;
  asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, hi;\n\t}" : "=r"(r) : "r"(v));
  return r;
}
// nibbles 0 and 4 of v as 128 + q in bf16x2
__device__ __forceinline__ uint32_t nibbles(uint32_t v) {
  uint32_t p;
  asm("lop3.b32 %0, %1, 0x000f000f, 0x43004300, 0xea;" : "=r"(p) : "r"(v));
  return p;
}
template <int CH, int NT>
__device__ __forceinline__ void join(float (&part)[CH][NT][4]) {
#pragma unroll
  for (int h = 1; h < CH; ++h)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) part[0][j][e] += part[h][j][e];
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float2 lds_f2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float lds_half(uint32_t addr) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
  return __half2float(__ushort_as_half(v));
}
__device__ __forceinline__ void tma_load_3d_hint(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int32_t c0, int32_t c1,
                                                 int32_t c2, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%3, %4, %5}], [%2], %6;"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_load_5d_hint(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int32_t c0, int32_t c1,
                                                 int32_t c2, int32_t c3, int32_t c4, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%3, %4, %5, %6, %7}], [%2], %8;"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void consumer_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kWarps * 32) : "memory"); }

// Position in a ring of N slots.
template <int N>
struct Ring {
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next() {
    if (++slot == N) {
      slot = 0;
      phase ^= 1;
    }
  }
};

// A CTA's blocks in walks over K of at most MOST, as even as they come.
template <int MOST>
struct Walks {
  int b0, n, walks;
  __device__ __forceinline__ Walks(int N) {
    const int blocks = (N + kRows - 1) / kRows;
    b0 = static_cast<int>(static_cast<long long>(blocks) * blockIdx.x / gridDim.x);
    n = static_cast<int>(static_cast<long long>(blocks) * (blockIdx.x + 1) / gridDim.x) - b0;
    walks = (n + MOST - 1) / MOST;
  }
  __device__ __forceinline__ int first(int p) const { return b0 + n * p / walks; }
  __device__ __forceinline__ int count(int p) const { return n * (p + 1) / walks - n * p / walks; }
};

template <int FMT, int NT>
__global__ void __launch_bounds__(kThreads, 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                   const __grid_constant__ CUtensorMap tmS, const __grid_constant__ CUtensorMap tmZ,
                   const __grid_constant__ Args a) {
  using C = Cfg<FMT, NT>;
  constexpr int STAGES = C::kStages, SLOTS = C::kSlots, U = C::kUnits, XR = C::kXRegs, BL = kBlocks, CH = C::kChains;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* slots = smem + STAGES * C::kStageBytes;
  float2* red = reinterpret_cast<float2*>(slots + SLOTS * C::kSlotBytes);
  uint64_t* full = reinterpret_cast<uint64_t*>(red + kWarps / 2 * C::kRedFloats / 2);
  uint64_t* empty = full + STAGES;
  uint64_t* xfull = empty + STAGES;
  uint64_t* xempty = xfull + SLOTS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int units = a.K / C::kUnitK;
  const int chunks = (units + kWarps * U - 1) / (kWarps * U);       // stages per block
  const Walks<BL> walk(a.N);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kWarps);
    }
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(&xfull[s], 1);
      mbar_init(&xempty[s], kWarps);
    }
    fence_barrier_init();
  }
  __syncthreads();
  // Settled weights are on their way while the launch ahead (a norm, an activation, attention) still runs
  if (warp != kWarps || !a.settled) tgi::pdl_wait();

  if (warp == kWarps) {
    // ---------------- weights ----------------
    if (elect_one()) {
      prefetch_tensormap(&tmW);
      const uint64_t pol = policy_evict_first();
      const uint32_t bytes = kTileBytes + C::kScaleBytes * (a.has_zp ? 2 : 1);
      Ring<STAGES> r;
      r.phase = 1;                                // the ring starts empty: the first round's waits pass
      bool ok = true;
      int issued = 0;
      for (int p = 0; p < walk.walks && ok; ++p) {
        const int blk0 = walk.first(p), nb = walk.count(p);
        for (int c = 0; c < chunks && ok; ++c) {
          for (int t = 0; t < nb; ++t, ++issued, r.next()) {
            // the ring is full of settled weights: room comes when the launch ahead has ended, however long that takes
            if (a.settled && issued == STAGES) tgi::pdl_wait();
            ok = mbar_wait(&empty[r.slot], r.phase);
            if (!ok) {
              report(a.status, kErrProducerWait);
              break;
            }
            const uint32_t dst = smem_u32(smem + r.slot * C::kStageBytes);
            mbar_arrive_expect_tx(&full[r.slot], bytes);
            tma_load_3d_hint(dst, &tmW, &full[r.slot], 0, (blk0 + t) * kRows, c * kWarps, pol);
            if (FMT == kInt4) {
              const int g0 = c * kWarps * U / a.group_units;
              tma_load_2d_hint(smem + r.slot * C::kStageBytes + kTileBytes, &tmS, &full[r.slot], (blk0 + t) * kRows, g0, pol);
              if (a.has_zp)
                tma_load_2d_hint(smem + r.slot * C::kStageBytes + kTileBytes + C::kScaleBytes, &tmZ, &full[r.slot],
                                 (blk0 + t) * kRows, g0, pol);
            }
          }
        }
      }
      // no copy may land in shared memory after the CTA has gone
      for (int i = max(0, issued - STAGES); i < issued; ++i) mbar_wait(&full[i % STAGES], (i / STAGES) & 1, 1u << 12);
    }
  } else if (warp == kWarps + 1) {
    // ---------------- tokens ----------------
    if (elect_one()) {
      const uint64_t pol = policy_evict_last();
      const int steps = chunks * U;
      Ring<SLOTS> r;
      r.phase = 1;
      bool ok = true;
      int issued = 0;
      for (int p = 0; p < walk.walks && ok; ++p) {
        for (int i = 0; i < steps; ++i, ++issued, r.next()) {
          ok = mbar_wait(&xempty[r.slot], r.phase);
          if (!ok) {
            report(a.status, kErrProducerWait);
            break;
          }
          const uint32_t dst = smem_u32(slots + r.slot * C::kSlotBytes);
          mbar_arrive_expect_tx(&xfull[r.slot], C::kXBytes + C::kXScaleBytes);
          if (FMT == kInt4) tma_load_5d_hint(dst, &tmX, &xfull[r.slot], 0, 0, 0, i % U, i / U * kWarps, pol);
          else tma_load_3d_hint(dst, &tmX, &xfull[r.slot], 0, 0, i * kWarps, pol);
          if (FMT == kFp8) tma_load_2d_hint(slots + r.slot * C::kSlotBytes + C::kXBytes, &tmS, &xfull[r.slot], 0, i * kWarps, pol);
        }
      }
      for (int i = max(0, issued - SLOTS); i < issued; ++i) mbar_wait(&xfull[i % SLOTS], (i / SLOTS) & 1, 1u << 12);
    }
  } else {
    // ---------------- consumers ----------------
    const int g = lane >> 2, q = lane & 3;           // MMA row (and token) / quarter of the unit
    const uint32_t smem0 = smem_u32(smem), slots0 = smem_u32(slots);
    // byte offset of 16-byte piece 2 q (a lane's 32 bytes are two pieces, the second's offset differs in bit 4)
    const uint32_t off0 = static_cast<uint32_t>((((2 * q) ^ g) << 4) + g * 128);
    Ring<STAGES> r;
    Ring<SLOTS> xr;
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t phase) {
      if (!ok) return;
      ok = mbar_wait(bar, phase);
      if (!ok && lane == 0) report(a.status, kErrMmaWaitFull);
    };
    // Shared memory goes back to its producer when the loads from it have returned.  An arrival that only follows the loads in
    // the program was seen to overtake them (they had queued in the load units; the warp then read the next weights), so its
    // address depends on a register of every load.
    auto loaded_arrive = [&](uint64_t* bar, uint32_t loaded) {
      __syncwarp();
      if (lane == 0) mbar_arrive(bar + (loaded & a.zero));
    };

    for (int p = 0; p < walk.walks; ++p) {
      const int blk0 = walk.first(p), nb = walk.count(p);
      float acc[BL][NT][4];
#pragma unroll
      for (int t = 0; t < BL; ++t)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[t][j][e] = 0.f;

      for (int c = 0; c < chunks; ++c) {
        const Ring<STAGES> r0 = r;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          // ---- token fragments of this warp's unit, shared by the blocks ----
          float sw[BL];
          if (FMT == kFp8) {
            const int unit = c * kWarps + warp;
#pragma unroll
            for (int t = 0; t < BL; ++t)
              sw[t] = unit < units && t < nb ? __ldg(a.wscale + static_cast<size_t>(((blk0 + t) * kRows) >> 7) * units + unit) : 0.f;
          }
          wait(&xfull[xr.slot], xr.phase);
          const uint32_t xs = slots0 + xr.slot * C::kSlotBytes, xt = xs + warp * (C::kPieces * NT * 8 * 128);
          uint32_t b[NT][XR];
          float2 sx[NT];             // fp8: scales of tokens 8 j + 2 q and + 1;  int4: their sums over the unit
          uint32_t seen = 0;
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            if (FMT == kInt4) {
              // features 32 e + 8 q .. + 7 as pairs (0, 4) (1, 5) (2, 6) (3, 7), as the nibbles come
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const uint4 v = lds128(xt + (e >> 1) * (NT * 8 * 128) + (j * 8 + g) * 128 + ((((e & 1) * 4 + q) ^ g) << 4));
                b[j][4 * e] = __byte_perm(v.x, v.z, 0x5410);
                b[j][4 * e + 1] = __byte_perm(v.x, v.z, 0x7632);
                b[j][4 * e + 2] = __byte_perm(v.y, v.w, 0x5410);
                b[j][4 * e + 3] = __byte_perm(v.y, v.w, 0x7632);
                seen |= b[j][4 * e];
              }
            } else {
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                const uint4 v = lds128(xt + j * 1024 + (off0 ^ (i * 16)));
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
                seen |= v.x;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  if (FMT == kBf16) {
                    b[j][4 * i + e] = w[e];
                  } else {
                    b[j][(8 * i + 2 * e) % XR] = e4m3_lo(w[e]);
                    b[j][(8 * i + 2 * e + 1) % XR] = e4m3_hi(w[e]);
                  }
                }
              }
              if (FMT == kFp8) {
                sx[j] = lds_f2(xs + C::kXBytes + (warp * 8 + 2 * q) * 4);
                seen |= __float_as_uint(sx[j].x);
              }
            }
          }
          loaded_arrive(&xempty[xr.slot], seen);
          xr.next();
          if (FMT == kInt4) {
            float sums[NT][4];
#pragma unroll
            for (int j = 0; j < NT; ++j) {
#pragma unroll
              for (int e = 0; e < 4; ++e) sums[j][e] = 0.f;
#pragma unroll
              for (int e = 0; e < XR; e += 2)
                mma_bf16(sums[j], 0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u, b[j][e], b[j][e + 1]);
              sx[j] = make_float2(sums[j][0], sums[j][1]);
            }
          }

          // ---- the blocks ----
          r = r0;
#pragma unroll
          for (int t = 0; t < BL; ++t) {
            if (t >= nb) break;
            if (u == 0) wait(&full[r.slot], r.phase);
            const uint32_t stage = smem0 + r.slot * C::kStageBytes, tile = stage + warp * (kRows * 128);
            uint64_t* free = &empty[r.slot];
            r.next();
            if (FMT == kInt4) {
              uint32_t wl[4], wh[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const uint32_t off = static_cast<uint32_t>((((4 * u + e) ^ g) << 4) + q * 4 + g * 128);
                wl[e] = lds32(tile + off);
                wh[e] = lds32(tile + 1024 + off);
              }
              const int group = a.group_units == 1 ? warp * U + u
                                                   : (c * kWarps * U + warp * U + u) / a.group_units - c * kWarps * U / a.group_units;
              const uint32_t at = stage + kTileBytes + (group * kRows + g) * 2;
              const float s0 = lds_half(at), s1 = lds_half(at + 16);
              const float z0 = a.has_zp ? lds_half(at + C::kScaleBytes) : 8.f, z1 = a.has_zp ? lds_half(at + C::kScaleBytes + 16) : 8.f;
              if (u == U - 1)
                loaded_arrive(free, wl[0] | wl[1] | wl[2] | wl[3] | wh[0] | wh[1] | wh[2] | wh[3] |
                                        __float_as_uint(s0) | __float_as_uint(s1) | __float_as_uint(z0) | __float_as_uint(z1));
              float part[CH][NT][4];
#pragma unroll
              for (int h = 0; h < CH; ++h)
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                  for (int e = 0; e < 4; ++e) part[h][j][e] = 0.f;
#pragma unroll
              for (int e = 0; e < 4; ++e) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const uint32_t a0 = nibbles(wl[e] >> (8 * h)), a1 = nibbles(wh[e] >> (8 * h));
                  const uint32_t a2 = nibbles(wl[e] >> (8 * h + 4)), a3 = nibbles(wh[e] >> (8 * h + 4));
#pragma unroll
                  for (int j = 0; j < NT; ++j) mma_bf16(part[h % CH][j], a0, a1, a2, a3, b[j][4 * e + 2 * h], b[j][4 * e + 2 * h + 1]);
                }
              }
              join(part);
              const float n0 = -128.f - z0, n1 = -128.f - z1;
#pragma unroll
              for (int j = 0; j < NT; ++j) {
                acc[t][j][0] = fmaf(fmaf(n0, sx[j].x, part[0][j][0]), s0, acc[t][j][0]);
                acc[t][j][1] = fmaf(fmaf(n0, sx[j].y, part[0][j][1]), s0, acc[t][j][1]);
                acc[t][j][2] = fmaf(fmaf(n1, sx[j].x, part[0][j][2]), s1, acc[t][j][2]);
                acc[t][j][3] = fmaf(fmaf(n1, sx[j].y, part[0][j][3]), s1, acc[t][j][3]);
              }
            } else {
              uint4 lo[2], hi[2];
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                lo[i] = lds128(tile + (off0 ^ (i * 16)));
                hi[i] = lds128(tile + 1024 + (off0 ^ (i * 16)));
              }
              loaded_arrive(free, lo[0].x | lo[1].x | hi[0].x | hi[1].x);
              if (FMT == kBf16) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
#pragma unroll
                  for (int j = 0; j < NT; ++j)
                    mma_bf16(acc[t][j], lo[i].x, hi[i].x, lo[i].y, hi[i].y, b[j][4 * i], b[j][4 * i + 1]);
#pragma unroll
                  for (int j = 0; j < NT; ++j)
                    mma_bf16(acc[t][j], lo[i].z, hi[i].z, lo[i].w, hi[i].w, b[j][4 * i + 2], b[j][4 * i + 3]);
                }
              } else {
                float part[CH][NT][4];
#pragma unroll
                for (int h = 0; h < CH; ++h)
#pragma unroll
                  for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) part[h][j][e] = 0.f;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                  const uint32_t wl[4] = {lo[i].x, lo[i].y, lo[i].z, lo[i].w}, wh[4] = {hi[i].x, hi[i].y, hi[i].z, hi[i].w};
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    const uint32_t a0 = e4m3_lo(wl[e]), a1 = e4m3_lo(wh[e]), a2 = e4m3_hi(wl[e]), a3 = e4m3_hi(wh[e]);
#pragma unroll
                    for (int j = 0; j < NT; ++j)
                      mma_fp16(part[e % CH][j], a0, a1, a2, a3, b[j][(8 * i + 2 * e) % XR], b[j][(8 * i + 2 * e + 1) % XR]);
                  }
                }
                join(part);
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                  const float s0 = sx[j].x * sw[t], s1 = sx[j].y * sw[t];
                  acc[t][j][0] = fmaf(part[0][j][0], s0, acc[t][j][0]);
                  acc[t][j][1] = fmaf(part[0][j][1], s1, acc[t][j][1]);
                  acc[t][j][2] = fmaf(part[0][j][2], s0, acc[t][j][2]);
                  acc[t][j][3] = fmaf(part[0][j][3], s1, acc[t][j][3]);
                }
              }
            }
          }
        }
      }

      // ---- the eight warps' sums, in a fixed order: the upper four's, added to the lower four's, added up ----
      float2* mine = red + (warp & 3) * (C::kRedFloats / 2) + lane;
#pragma unroll
      for (int half = 1; half >= 0; --half) {
        if ((warp >> 2) == half) {
#pragma unroll
          for (int t = 0; t < BL; ++t) {
            if (t >= nb) break;
#pragma unroll
            for (int j = 0; j < NT; ++j) {
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                float2* at = mine + ((t * NT + j) * 2 + h) * 32;
                float2 v = make_float2(acc[t][j][2 * h], acc[t][j][2 * h + 1]);
                if (half == 0) {
                  v.x += at->x;
                  v.y += at->y;
                }
                *at = v;
              }
            }
          }
        }
        consumer_barrier();
      }
      for (int i = threadIdx.x; i < nb * NT * 64; i += kWarps * 32) {
        float2 sum = red[i];
#pragma unroll
        for (int w = 1; w < kWarps / 2; ++w) {
          const float2 v = red[w * (C::kRedFloats / 2) + i];
          sum.x += v.x;
          sum.y += v.y;
        }
        const int l = i & 31, half = (i >> 5) & 1, tj = i >> 6;
        const int n = (blk0 + tj / NT) * kRows + half * 8 + (l >> 2), m = (tj % NT) * 8 + 2 * (l & 3);
        if (n < a.N) {
          const float bias = a.bias != nullptr ? __bfloat162float(a.bias[n]) : 0.f;
          if (m < a.M) a.C[static_cast<size_t>(m) * a.N + n] = __float2bfloat16(sum.x + bias);
          if (m + 1 < a.M) a.C[static_cast<size_t>(m + 1) * a.N + n] = __float2bfloat16(sum.y + bias);
        }
      }
      if (p + 1 < walk.walks) consumer_barrier();
    }
  }
  __syncthreads();
}

int make_map(CUtensorMap* map, CUtensorMapDataType type, int rank, const void* base, const cuuint64_t* dims, const cuuint64_t* strides,
             const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
  tgi::EncodeTiledFn enc = tgi::get_encode();
  if (enc == nullptr) return -100;
  const cuuint32_t step[5] = {1, 1, 1, 1, 1};
  const CUresult r = enc(map, type, rank, const_cast<void*>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -static_cast<int>(r) - 1000;
}

// Rows as [pieces of 128 bytes][rows][128 bytes], so that one box holds eight pieces of some rows.
int make_row_map(CUtensorMap* map, bool bf16, const void* base, uint64_t rows, uint64_t row_bytes, uint64_t pitch, uint32_t box_rows) {
  const cuuint32_t inner = bf16 ? 64 : 128;
  const cuuint64_t dims[3] = {inner, rows, row_bytes / 128}, strides[2] = {pitch, 128};
  const cuuint32_t box[3] = {inner, box_rows, kWarps};
  return make_map(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box,
                  CU_TENSOR_MAP_SWIZZLE_128B);
}

// Operands as the entry points give them.
struct Operands {
  const void* X;
  long long x_pitch;              // bytes between tokens
  const void* W;
  const float* xs;                // fp8: xs[unit * xs_pitch + token]
  int xs_pitch;
  const void *scale, *zp;         // int4: fp16 [K / group, N]; zp may be null
};

template <int FMT, int NT>
int launch_nt(const Operands& o, const Args& a, int max_ctas, cudaStream_t stream) {
  using C = Cfg<FMT, NT>;
  CUtensorMap tmW, tmX, tmS, tmZ;
  const uint64_t w_row = FMT == kBf16 ? 2ull * a.K : FMT == kFp8 ? a.K : a.K / 2;
  int rc = make_row_map(&tmW, FMT == kBf16, o.W, a.N, w_row, w_row, kRows);
  if (rc) return rc;
  if (FMT == kInt4) {
    // tokens of every other unit: [pairs of units][unit of a pair][piece of a unit][tokens][128 bytes]
    const cuuint64_t dims[5] = {64, static_cast<cuuint64_t>(a.M), 2, 2, static_cast<cuuint64_t>(a.K / 256)};
    const cuuint64_t strides[4] = {static_cast<cuuint64_t>(o.x_pitch), 128, 256, 512};
    const cuuint32_t box[5] = {64, NT * 8, 2, 1, kWarps};
    rc = make_map(&tmX, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, o.X, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  } else {
    rc = make_row_map(&tmX, FMT == kBf16, o.X, a.M, FMT == kBf16 ? 2ull * a.K : a.K, o.x_pitch, NT * 8);
  }
  if (rc) return rc;
  tmS = tmZ = tmW;
  if (FMT == kFp8) {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(a.M), static_cast<cuuint64_t>(a.K / 128)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(o.xs_pitch) * 4};
    const cuuint32_t box[2] = {8, kWarps};
    rc = make_map(&tmS, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, o.xs, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc) return rc;
  }
  if (FMT == kInt4) {
    const cuuint64_t groups = (a.K / 128 + a.group_units - 1) / a.group_units;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(a.N), groups}, strides[1] = {static_cast<cuuint64_t>(a.N) * 2};
    const cuuint32_t box[2] = {kRows, 16};
    rc = make_map(&tmS, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, o.scale, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc == 0 && o.zp != nullptr)
      rc = make_map(&tmZ, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, o.zp, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc) return rc;
  }
  auto kern = gemm_skinny_kernel<FMT, NT>;
  static std::atomic<unsigned long long> attr_set{0};      // the shared-memory opt-in is per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -2;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(attr_set.load(std::memory_order_acquire) & bit)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem) != cudaSuccess) return -2;
    attr_set.fetch_or(bit, std::memory_order_release);
  }
  const int blocks = (a.N + kRows - 1) / kRows;
  const int grid = blocks < max_ctas ? blocks : max_ctas;
  if (grid < 1) return -4;
  const cudaError_t err = tgi::launch_after(a.settled || tgi::pdl_enabled(), kern, dim3(grid), dim3(kThreads), C::kSmem, stream, tmW, tmX,
                                            tmS, tmZ, a);
  return err == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -3;
}

template <int FMT>
int launch(const Operands& o, const Args& a, int max_ctas, cudaStream_t stream) {
  if constexpr (FMT == kBf16) {
    if (a.M > 24) return launch_nt<FMT, 4>(o, a, max_ctas, stream);
    if (a.M > 16) return launch_nt<FMT, 3>(o, a, max_ctas, stream);
  }
  if constexpr (FMT != kFp8) {
    if (a.M > 8) return launch_nt<FMT, 2>(o, a, max_ctas, stream);
  }
  return launch_nt<FMT, 1>(o, a, max_ctas, stream);
}

constexpr int kInt4Tokens = 16;      // of one launch: the fragments of 32 tokens and 128 features do not fit the registers

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

Args base_args(void* C, const void* bias, int M, int N, int K, int settled, int* status) {
  Args a{};
  a.C = static_cast<__nv_bfloat16*>(C);
  a.bias = static_cast<const __nv_bfloat16*>(bias);
  a.M = M;
  a.N = N;
  a.K = K;
  a.status = status;
  a.settled = settled;
  return a;
}

}  // namespace

namespace tgi {

// Up to 16 tokens always; up to 32 where the 256-row tiles of the tcgen05 kernel leave half of the CTAs without one of their own,
// so that it splits K.  Both measured on B200, us, here / tcgen05:
//   16 tokens  6144 x 4096 13.3 / 22.2   28672 x 4096 40.6 / 44     128256 x 4096 160 / 190
//   32 tokens  6144 x 4096 14.8 / 22.2    4096 x 14336 27.4 / 31.0   28672 x 4096 48.1 / 43.9
bool skinny_bf16_applies(const void* X, const void* W, int M, int N, int K, int ldx, int max_ctas) {
  if (K % 64 != 0 || ldx % 8 != 0 || !aligned16(X) || !aligned16(W)) return false;
  return M <= 16 || (M <= 32 && (N + 255) / 256 * 2 <= max_ctas);
}

int skinny_bf16(const void* X, int ldx, const void* W, void* C, const void* bias, int M, int N, int K, int max_ctas, int settled,
                int* status, cudaStream_t stream) {
  return launch<kBf16>(Operands{X, 2LL * ldx, W, nullptr, 0, nullptr, nullptr}, base_args(C, bias, M, N, K, settled, status), max_ctas,
                       stream);
}

// Up to 8 tokens (us, here / tcgen05: 57344 x 8192 79 / 114, 8192 x 28672 44 / 58, 10240 x 8192 22 / 32).  From 9 to 16 tokens it
// would still be the faster one (91 / 104, 48 / 51, 24 / 31).  The line lies at 8 because activations are quantised anew for every
// product, so that the last bit of a sum can become a sixteenth of a value: the tcgen05 kernel gives tokens from 9 to 128 the same
// sums in every batch, and with the line at 16 a short prompt that was sent alone and then four times at once got other greedy
// answers.  A prompt of up to 8 tokens (or such a rest of one) and a decode step of up to 8 sequences don't have that: among more
// tokens their sums have another order.  In bf16 and with 4-bit weights a token's sums are the same in all batches that come here and
// others in larger ones, but there a last bit stays one.
bool skinny_fp8_applies(const void* X, const float* xs_t, const void* W, int M, int K) {
  return M <= 8 && K % 128 == 0 && aligned16(X) && aligned16(xs_t) && aligned16(W);
}

int skinny_fp8(const void* X, const float* xs_t, int xs_pitch, const void* W, const float* wscale, void* C, const void* bias,
               int M, int N, int K, int max_ctas, int settled, int* status, cudaStream_t stream) {
  Args a = base_args(C, bias, M, N, K, settled, status);
  a.wscale = wscale;
  return launch<kFp8>(Operands{X, K, W, xs_t, xs_pitch, nullptr, nullptr}, a, max_ctas, stream);
}

// Up to 32 tokens in two launches: 28672 x 4096 38 us for 12 tokens and 74 for 32, 4096 x 14336 20 and 39, where the kernel that
// expands weights for tcgen05 takes 91 - 110 and 46 at any number of tokens up to 128.
bool skinny_int4_applies(const void* X, const void* W, const void* scale, const void* zp, int M, int N, int K, int group) {
  return M <= 2 * kInt4Tokens && K % 256 == 0 && group % 128 == 0 && N % 8 == 0 && aligned16(X) && aligned16(W) && aligned16(scale) && aligned16(zp);
}

int skinny_int4(const void* X, const void* W, const void* scale, const void* zp, int group, void* C, const void* bias, int M, int N,
                int K, int max_ctas, int settled, int* status, cudaStream_t stream) {
  for (int m0 = 0; m0 < M; m0 += kInt4Tokens) {
    Args a = base_args(static_cast<__nv_bfloat16*>(C) + static_cast<size_t>(m0) * N, bias,
                       M - m0 < kInt4Tokens ? M - m0 : kInt4Tokens, N, K, settled && m0 == 0, status);
    a.has_zp = zp != nullptr;
    a.group_units = group / 128;
    const int rc = launch<kInt4>(Operands{static_cast<const __nv_bfloat16*>(X) + static_cast<size_t>(m0) * K, 2LL * K, W, nullptr, 0,
                                          scale, zp}, a, max_ctas, stream);
    if (rc) return rc;
  }
  return 0;
}

}  // namespace tgi
