// Paged causal prefill attention on the 5th-generation tensor cores (sm_100a), bf16 pages of 16 tokens: head size 128 (or 192
// for queries and keys), ragged batches with a cached prefix (chunked prefill), GQA, sliding window with kept first tokens,
// soft-capping, per-row horizons and a gate per token and head.
//
// Replaces, in the reference, flashinfer `BatchPrefillWithPagedKVCache` / FA2 `varlen_fwd`
// (layers/attention/cuda.py:244-296, layers/attention/flashinfer.py:58-128).
//
// A CTA owns 128 query rows of one head and walks the KV range in tiles of 128 tokens.  Even and odd tiles are two chains, each
// with its own four softmax warps (a thread per row), running maximum and sum, and accumulators; they meet once at the end:
//   S  = Q K^T     tcgen05.mma, M 128 (rows) x N 128 (keys) x K 128 (head dim), one TMEM accumulator per chain
//   P  = softmax   TMEM -> registers, maximum, then probabilities as 16-bit values into a shared-memory tile in the swizzled
//                  operand layout.  Tiles that a row sees completely (below the diagonal, inside the window and the sequence)
//                  take a path without per-element masks
//   O += P V       tcgen05.mma, M 128 x N 128 (head dim) x K 128 (keys), accumulated in TMEM over the chain; V is taken as the
//                  MN-major operand, i.e. exactly as the page boxes land in shared memory (rows = tokens, 128 bytes = 64
//                  head elements).  A chain's reference maximum moves only when a row's maximum has outgrown it by 2^8 (P is
//                  then up to 256: the relative precision of its 16 bits is the same); its warps then rescale O in TMEM (rescaling only when the
//                  maximum has grown by a threshold: FlashAttention-4)
//   out            (O_even a_even + O_odd a_odd) / l with a = 2^(m_chain - m)
// What bounds it is the softmax's instructions (about six per score, 16 K scores a tile, against 512 cycles of MMA).  While a chain
// waits for its scores or for room for P the other one computes.  A single chain whose eight warps shared a tile, with the running
// output in registers, was a serial sequence of about 3400 cycles a tile.  32 heads, 8192 tokens on 20480 cached ones: 4712 -> 3180 us
// (700 -> 1037 TFLOP/s), 2048 on 8192 545 -> 381, 2048 on none 112 -> 94.5.
// K and V pages are fetched with TMA boxes of one page (16 tokens x 128 bytes) straight from the page pool, no
// per-lane address arithmetic.
// Queries and keys of 192 take a third 64-element slab each; V and P are then single-buffered (V of the next tile is wanted
// only after that tile's softmax, P is free again after the PV product, during the softmax's first pass).
// Every wait is bounded; a wait that runs out sets the status word, the CTA drains and frees its TMEM.
#include <atomic>

#include "attention_prefill.cuh"
#include "launch.cuh"
#include "tensor_map.cuh"

using namespace prefill;

namespace {

constexpr int kWarps = 12;                    // K producer, MMA, V producer, spare, 8 softmax
constexpr float kSlack = 8.f;                 // how far (log2) a row's maximum may outgrow the chain's reference
constexpr int kPolyEvery = 8;                 // see `poly_exp2`

// registers of a load that an earlier wait has covered: not to be read ahead of this point
__device__ __forceinline__ void tmem_ld_use(uint32_t (&r)[32]) {
#pragma unroll
  for (int i = 0; i < 32; i += 8)
    asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]), "+r"(r[i + 6]), "+r"(r[i + 7]));
}

// Shared memory (bytes):  Q 32 K | K 2 x 32 K | V 2 x 32 K | P 2 x 32 K | barriers;
// with KS = 3 slabs of queries and keys:  Q 48 K | K 2 x 48 K | V 32 K | P 32 K | barriers
template <int KS>
struct Layout {
  static constexpr int kStagesVP = KS == 2 ? 2 : 1;               // of V and of P
  static constexpr int kQ = 0;
  static constexpr int kK = KS * kSlab;
  static constexpr int kKTile = KS * kSlab;
  static constexpr int kV = kK + 2 * kKTile;
  static constexpr int kP = kV + kStagesVP * kTileBytes;
  static constexpr int kBars = kP + kStagesVP * kTileBytes;       // two P tiles: one per chain
  static constexpr int kStats = kBars + 256;                      // float2 [2][128]: maximum and sum of the chains' rows
  static constexpr int kAbort = kStats + 2 * 128 * 8;             // int: a softmax warp gave up
  // no slack for aligning the base: the kernel checks that the dynamic shared memory starts on a 1024-byte
  // boundary (it does when the kernel has no static shared memory) and reports an error otherwise
  static constexpr int kTotal = kAbort + 64;
  static_assert(kTotal <= 227 * 1024, "shared memory of a CTA");
  // stage and round of tile j
  static __device__ __forceinline__ int stage(int j) { return kStagesVP == 2 ? j & 1 : 0; }
  static __device__ __forceinline__ int round(int j) { return kStagesVP == 2 ? j >> 1 : j; }
};

template <int KS>
__global__ void __launch_bounds__(kWarps * 32, 1)
prefill_chains_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const PrefillParams p) {
  using L = Layout<KS>;
  static_assert(KS == 2 || KS == 3, "queries and keys of two or three slabs");
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if ((smem_u32(smem) & 1023u) != 0u) {       // uniform over the CTA, before anything is allocated
    if (threadIdx.x == 0) report(p.status, kErrProducerWait);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBars);
  uint64_t* k_full = bars;             // [2] TMA landed
  uint64_t* k_free = bars + 2;         // [2] MMA done with the stage
  uint64_t* v_full = bars + 4;        // [2]
  uint64_t* v_free = bars + 6;        // [2]
  uint64_t* s_full = bars + 12;       // [2] S accumulator of the chain written
  uint64_t* p_ready = bars + 14;      // [2] P tile of the chain written, its S accumulator read
  uint64_t* pv_done = bars + 16;      // [2] PV product of the chain added to its output, P tile free
  uint64_t* q_ready = bars + 18;      // Q tile staged
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 20);
  float2* s_stats = reinterpret_cast<float2*>(smem + L::kStats);
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + L::kAbort);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.z, h = blockIdx.y;
  const int qt = gridDim.x - 1 - blockIdx.x;       // long tiles (late rows) first: the grid drains on short ones
  const int q_begin = p.cu_seqlens_q[b], n = p.cu_seqlens_q[b + 1] - q_begin;
  const int Lkv = p.kv_lens[b];
  if (qt * kRows >= n || Lkv < n) return;            // uniform over the CTA, before anything is allocated; Lkv < n: left out
  const int kvh = h / (p.Hq / p.Hkv);
  const int row_base = qt * kRows;
  const int pos_first = Lkv - n + row_base;
  const int pos_last = min(Lkv - 1, pos_first + kRows - 1);
  const int t_lo = first_visible(p, pos_first) / kKeys * kKeys;
  const int t_hi = p.horizon != nullptr ? Lkv : pos_last + 1;
  // Kept first tokens come in tiles of their own ahead of the window's: a row whose window starts at `lo` reads keys
  // 0 .. min(keep, lo) - 1 of them and the window's tiles from `lo` on, so a tile has one range of visible keys per row.
  const int kept = (min(p.keep, first_visible(p, pos_last)) + kKeys - 1) / kKeys;
  const int ntiles = kept + (t_hi - t_lo + kKeys - 1) / kKeys;
  auto tile_start = [&](int j) { return j < kept ? j * kKeys : t_lo + (j - kept) * kKeys; };

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&k_free[i], 1);
      mbar_init(&v_free[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_ready[i], 4);
      mbar_init(&pv_done[i], 1);
    }
    mbar_init(q_ready, kWarps - 2);
    *s_abort = 0;
    fence_barrier_init();
    prefetch_tensormap(&tmK);
    prefetch_tensormap(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, 512);
    tmem_relinquish();
  }
  tgi::pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tS = tmem_base, tO = tmem_base + 256;      // 128 columns per chain each

  // ---------------- TMA producers: one box per page and 64-element half of the head ----------------
  // A thread's TMA copies issue one after the other (about 400 cycles each, measured), so a tile's boxes are
  // spread over lanes: lane l copies page l % 8, half (l / 8) % 2.  Lanes 0..7 read the tile's block ids with one
  // coalesced load; lane 0 does the waits and posts the expected byte count.  Warp 0 brings K and warp 2 brings
  // V, each on its own ring of two stages.
  auto produce = [&](bool do_k, bool do_v) {
    bool ok = true;
    for (int j = 0; j < ntiles && ok; ++j) {
      const int s = j & 1, vs = L::stage(j);
      const int t0 = tile_start(j);
      int blk = 0;
      if (lane < kKeys / kPage) {
        const int blk_i = (t0 >> 4) + lane;
        if (blk_i < p.max_blocks) blk = p.block_tables[static_cast<size_t>(b) * p.max_blocks + blk_i];
        blk = min(max(blk, 0), p.num_blocks - 1);        // pages past the sequence are masked later
      }
      blk = __shfl_sync(0xffffffffu, blk, lane & 7);
      if (lane == 0) {
        if (do_k) {
          if (j >= 2) ok = mbar_wait(&k_free[s], ((j >> 1) - 1) & 1);
          if (ok) mbar_arrive_expect_tx(&k_full[s], L::kKTile);
        }
        if (do_v && ok) {
          if (j >= L::kStagesVP) ok = mbar_wait(&v_free[vs], (L::round(j) - 1) & 1);
          if (ok) mbar_arrive_expect_tx(&v_full[vs], kTileBytes);
        }
        if (!ok) report(p.status, kErrProducerWait);
      }
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      const int pg = lane & 7;
      const int hf = lane >> 3;                              // 64-element slab
      if (do_k && hf < KS)
        tma_load_2d(smem + L::kK + s * L::kKTile + hf * kSlab + pg * (kPage * 128), &tmK, &k_full[s], kvh * (64 * KS) + hf * 64, blk * kPage);
      if (do_v && hf < 2)
        tma_load_2d(smem + L::kV + vs * kTileBytes + hf * kSlab + pg * (kPage * 128), &tmV, &v_full[vs], kvh * kD + hf * 64, blk * kPage);
      __syncwarp();
    }
  };
  if (warp != 0 && warp != 2) {
    // ---- Q tile -> shared, swizzled operand layout (slabs of 64 head elements).  The two
    // producer warps are already fetching K and V meanwhile; the MMA issuer waits for q_ready. ----
    const int st = (warp == 1 ? 0 : warp - 2) * 32 + lane;
    for (int c = st; c < kRows * 8 * KS; c += (kWarps - 2) * 32) {
      const int row = c / (8 * KS), ch = c % (8 * KS);
      uint4 v = make_uint4(0, 0, 0, 0);
      if (row_base + row < n)
        v = *reinterpret_cast<const uint4*>(p.q + (static_cast<size_t>(q_begin + row_base + row) * p.Hq + h) * (64 * KS) + ch * 8);
      *reinterpret_cast<uint4*>(smem + L::kQ + (ch >> 3) * kSlab + swz_chunk(row, ch & 7)) = v;
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(q_ready);
  }
  if (warp == 0) {
    produce(true, false);
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      constexpr uint32_t id_qk = idesc16(1u, false);
      constexpr uint32_t id_pv = idesc16(1u, true);
      const uint32_t q_addr = smem_u32(smem + L::kQ);
      const uint32_t p_base = smem_u32(smem + L::kP);
      bool ok = true;
      auto issue_qk = [&](int j) {
        const int s = j & 1;
        uint32_t k_addr;
        if (!mbar_wait(&k_full[s], (j >> 1) & 1)) { report(p.status, kErrMmaWaitFull); return false; }
        k_addr = smem_u32(smem + L::kK + s * L::kKTile);
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 4 * KS; ++k) { // 16 head elements (32 bytes) per MMA; 4 per slab
          const uint64_t da = make_desc_sw128(q_addr + (k >> 2) * kSlab) + ((k & 3) * 32 >> 4);
          const uint64_t db = make_desc_sw128(k_addr + (k >> 2) * kSlab) + ((k & 3) * 32 >> 4);
          mma_f16(tS + s * 128, da, db, id_qk, k > 0 ? 1u : 0u);
        }
        tc_commit(&s_full[s]);
        tc_commit(&k_free[s]);
        return true;
      };
      auto issue_pv = [&](int j) {
        const int s = j & 1, vs = L::stage(j);
        uint32_t v_addr;
        if (!mbar_wait(&v_full[vs], L::round(j) & 1)) { report(p.status, kErrMmaWaitFull); return false; }
        v_addr = smem_u32(smem + L::kV + vs * kTileBytes);
        const uint32_t p_addr = p_base + vs * kTileBytes;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 8; ++k) {      // 16 keys per MMA: 32 bytes along a P row, two 8-row groups of V
          const uint64_t da = make_desc_sw128(p_addr + (k >> 2) * kSlab) + ((k & 3) * 32 >> 4);
          const uint64_t db = make_desc_mn_sw128(v_addr + k * 2048, kSlab);
          mma_f16(tO + s * 128, da, db, id_pv, j >= 2 || k > 0 ? 1u : 0u);
        }
        tc_commit(&pv_done[s]);
        tc_commit(&v_free[vs]);
        return true;
      };
      ok = mbar_wait(q_ready, 0);
      if (!ok) report(p.status, kErrMmaWaitFull);
      ok = ok && issue_qk(0);
      if (ok && ntiles > 1) ok = issue_qk(1);
      for (int j = 0; j < ntiles && ok; ++j) {
        // the chain's scores have been read and its P is written: scores of its next tile first, they are waited for
        ok = mbar_wait(&p_ready[j & 1], (j >> 1) & 1);
        if (!ok) { report(p.status, kErrMmaWaitAccum); break; }
        tc_fence_after();
        if (j + 2 < ntiles) ok = issue_qk(j + 2);
        if (ok) ok = issue_pv(j);
      }
    }
  } else if (warp == 2) {
    produce(false, true);
  } else if (warp == 3) {
    // spare
  } else {
    // ---------------- softmax: a thread per query row, four warps per chain ----------------
    const int quarter = warp & 3;
    const int ch = (warp - 4) >> 2;              // chain: tiles ch, ch + 2, ...
    const int r = quarter * 32 + lane;
    const int pos = pos_first + r;
    int hz = pos;
    if (p.horizon != nullptr && row_base + r < n) hz = max(pos, min(p.horizon[q_begin + row_base + r], Lkv - 1));
    const float scale_log2 = p.scale * kLog2e;
    const uint32_t quarter_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t s_addr = tS + quarter_addr + ch * 128, o_addr = tO + quarter_addr + ch * 128;
    uint8_t* p_tile = smem + L::kP + (L::kStagesVP == 2 ? ch : 0) * kTileBytes;
    const bool cap = p.softcap > 0.f;
    ScoreArgs sa;
    sa.scale_log2 = scale_log2;
    sa.cap_in = cap ? p.scale / p.softcap : 0.f;
    sa.cap_out = p.softcap * kLog2e;
    // visible keys of this row in a tile of its window
    const int win_max = min(hz, Lkv - 1), win_min = first_visible(p, pos);
    float m = -INFINITY, l = 0.f;                // reference maximum and sum of the chain's row
    bool ok = true;                              // the same in all lanes of a warp
    auto wait = [&](uint64_t* bar, int round) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar, round & 1));
      if (!ok && lane == 0) report(p.status, kErrEpilogueWait);
      return ok;
    };
    for (int j = ch; j < ntiles; j += 2) {
      const int t0 = tile_start(j);
      const int t_min = j < kept ? 0 : win_min, t_max = j < kept ? min(p.keep, win_min) - 1 : win_max;
      if (!wait(&s_full[ch], j >> 1)) break;
      tc_fence_after();
      // a warp whose rows all see the whole tile (below the diagonal / horizon, inside the window and the sequence) takes the
      // code without masks; the choice is per warp so that no path diverges
      const bool plain = __all_sync(0xffffffffu, t0 >= t_min && t0 + kKeys - 1 <= t_max);
      sa.range = t_max >= t_min ? static_cast<unsigned>(t_max - t_min) : 0u;
      const int lo0 = t_max >= t_min ? t_min - t0 : (1 << 30);
      // pass 1: maximum of the (masked) scores; those of a plain tile stay in registers for pass 2
      float mx = -INFINITY;
      uint32_t v[4][32];
      tmem_ld_32x32b_x32(s_addr, v[0]);
      if (plain) {
#pragma unroll
        for (int c = 1; c < 4; ++c) tmem_ld_32x32b_x32(s_addr + c * 32, v[c]);
        tmem_ld_wait(v[0]);
        mx = group_max<false>(v[0], mx, sa);
#pragma unroll
        for (int c = 1; c < 4; ++c) {
          tmem_ld_use(v[c]);
          mx = group_max<false>(v[c], mx, sa);
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < 4; c += 2) {
          tmem_ld_wait(v[0]);
          tmem_ld_32x32b_x32(s_addr + (c + 1) * 32, v[1]);
          sa.lo = lo0 - c * 32;
          mx = group_max<true>(v[0], mx, sa);
          tmem_ld_wait(v[1]);
          if (c == 0) tmem_ld_32x32b_x32(s_addr + 64, v[0]);
          sa.lo = lo0 - c * 32 - 32;
          mx = group_max<true>(v[1], mx, sa);
        }
      }
      // the cap is monotonic: the maximum of the raw scores is capped
      if (!cap) mx *= scale_log2;     // scale_log2 > 0
      else if (mx > -INFINITY) mx = sa.cap_out * fast_tanh(mx * sa.cap_in);
      // room for P (and O at rest): the chain's last PV product is done, with one P tile also the other chain's
      if (L::kStagesVP == 1 ? (j >= 1 && !wait(&pv_done[ch ^ 1], (j - 1) >> 1)) : (j >= 2 && !wait(&pv_done[ch], (j >> 1) - 1))) break;
      const bool grown = mx > m + kSlack;         // also the first visible key of a row
      if (__any_sync(0xffffffffu, grown)) {
        const float alpha = grown ? fast_exp2(m - mx) : 1.f;
        if (grown) m = mx;
        l *= alpha;
        if (j >= 2) {
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 128; c += 16) {
            uint32_t o[16];
            tmem_ld_32x32b_x16(o_addr + c, o);
            tmem_ld_wait(o);
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x32b_x16(o_addr + c, o);
          }
          tmem_st_wait();
        }
      }
      // pass 2: probabilities as 16-bit values into the P operand tile, row sum.  A row without a visible key so far has
      // m = -inf: every key of it is masked, so the value never reaches P.
      auto store = [&](int c, const uint32_t(&packed)[16]) {
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4)       // four 16-byte chunks (8 keys each) of the 32-key group c
          *reinterpret_cast<uint4*>(p_tile + (c >> 1) * kSlab + swz_chunk(r, (c & 1) * 4 + q4)) =
              make_uint4(packed[4 * q4], packed[4 * q4 + 1], packed[4 * q4 + 2], packed[4 * q4 + 3]);
      };
      uint32_t packed[16];
      if (plain && !cap) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          l += group_prob<false, false, false, kPolyEvery>(v[c], packed, m, sa);
          store(c, packed);
        }
      } else {
#pragma unroll 1
        for (int c = 3; c >= 0; --c) {
          tmem_ld32(s_addr + c * 32, v[0]);
          sa.lo = lo0 - c * 32;
          if (!cap) l += group_prob<true, false, false, kPolyEvery>(v[0], packed, m, sa);
          else if (plain) l += group_prob<false, true, false, kPolyEvery>(v[0], packed, m, sa);
          else l += group_prob<true, true, false, kPolyEvery>(v[0], packed, m, sa);
          store(c, packed);
        }
      }
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[ch]);
    }
    // ---- the two chains together: this thread's row, columns 64 ch .. 64 ch + 63 ----
    const int tiles = (ntiles + 1 - ch) >> 1;      // of this chain
    if (ok && tiles > 0) wait(&pv_done[ch], tiles - 1);
    if (!ok) *s_abort = 1;
    s_stats[ch * 128 + r] = make_float2(m, l);
    asm volatile("bar.sync 2, 256;" ::: "memory");
    if (*s_abort == 0) {
      tc_fence_after();
      const float2 st0 = s_stats[r], st1 = s_stats[128 + r];
      const float mm = fmaxf(st0.x, st1.x);
      const float a0 = st0.x == -INFINITY ? 0.f : fast_exp2(st0.x - mm), a1 = st1.x == -INFINITY ? 0.f : fast_exp2(st1.x - mm);
      float ll = st0.y * a0 + st1.y * a1;
      if (p.sink != nullptr) ll += exp2f(fmaf(p.sink[h], kLog2e, -mm));
      float inv = ll > 0.f ? 1.f / ll : 0.f;
      if (p.gate != nullptr && row_base + r < n)
        inv *= __fdividef(1.f, 1.f + __expf(-__bfloat162float(p.gate[static_cast<long long>(q_begin + row_base + r) * p.ld_gate + h])));
      const float w0 = a0 * inv, w1 = a1 * inv;
      __nv_bfloat16* dst = p.out + (static_cast<size_t>(q_begin + row_base + r) * p.Hq + h) * kD + ch * 64;
#pragma unroll
      for (int c = 0; c < 64; c += 16) {
        uint32_t o0[16], o1[16];
        tmem_ld_32x32b_x16(tO + quarter_addr + ch * 64 + c, o0);
        if (ntiles > 1) tmem_ld_32x32b_x16(tO + quarter_addr + 128 + ch * 64 + c, o1);
        tmem_ld_wait(o0);
        if (ntiles > 1) tmem_ld_wait(o1);
        float f[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          f[i] = __uint_as_float(o0[i]) * w0;
          if (ntiles > 1) f[i] = fmaf(__uint_as_float(o1[i]), w1, f[i]);
        }
        if (row_base + r < n) {
#pragma unroll
          for (int i = 0; i < 16; i += 8) {
            __nv_bfloat162 w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = __floats2bfloat162_rn(f[i + 2 * e], f[i + 2 * e + 1]);
            *reinterpret_cast<uint4*>(dst + c + i) = *reinterpret_cast<uint4*>(w);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

template <int KS>
int launch_prefill(const PrefillParams& p, const void* k_cache, const void* v_cache, long long k_pitch, long long v_pitch, int B,
                   int max_q, cudaStream_t stream) {
  using L = Layout<KS>;
  CUtensorMap tmK, tmV;
  const uint64_t rows = static_cast<uint64_t>(p.num_blocks) * kPage;
  const uint64_t k_cols = static_cast<uint64_t>(p.Hkv) * 64 * KS, v_cols = static_cast<uint64_t>(p.Hkv) * kD;
  int rc;
  rc = tgi::make_map_2d(&tmK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, k_cache, rows, k_cols, k_pitch * 2, kPage, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  rc = tgi::make_map_2d(&tmV, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, v_cache, rows, v_cols, v_pitch * 2, kPage, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  auto kern = prefill_chains_kernel<KS>;
  static std::atomic<unsigned long long> attr_set{0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -2;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(attr_set.load(std::memory_order_acquire) & bit)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal) != cudaSuccess) return -2;
    attr_set.fetch_or(bit, std::memory_order_release);
  }
  const dim3 grid((max_q + kRows - 1) / kRows, p.Hq, B);
  const cudaError_t err = tgi::launch(kern, grid, dim3(kWarps * 32), static_cast<size_t>(L::kTotal), stream, tmK, tmV, p);
  return err == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace

int prefill::launch_bf16(const PrefillParams& p, int dim, const void* k_cache, const void* v_cache, long long k_pitch, long long v_pitch,
                         int B, int max_q, cudaStream_t stream) {
  return dim == 192 ? launch_prefill<3>(p, k_cache, v_cache, k_pitch, v_pitch, B, max_q, stream)
                    : launch_prefill<2>(p, k_cache, v_cache, k_pitch, v_pitch, B, max_q, stream);
}
