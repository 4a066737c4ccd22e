// Fused sampler: repetition penalty, temperature, top-k, top-p, typical-p, Gumbel-max sampling (or argmax) and the
// log-probability of the chosen token, one CTA per row.  Replaces the reference's chain of logits warpers and its
// `probs / Exp(1)` multinomial with a CPU generator per request (utils/tokens.py:346-399,
// utils/logits_process.py:25-358, 151-218): no sort, no [B, V] probability matrix, no host round trip.
//
//   x_j = logit_j / T, the logits of ids in the row's history first divided (negative ones: multiplied) by the penalty
//   top-k: keep x_j unless k entries are larger;  top-p: keep x_j unless the mass of strictly larger entries
//   already reaches p (same sets as the sort-based torch filters).
//   sample: argmax_j (x_j + g_j) over the kept set, g_j = -log(-log u_j), u_j from Philox4x32-10
//   keyed by the request's seed with counter (j, step): reproducible for a given seed.
//   logprob = x_c - logsumexp over the kept set.
//
// What bounds it is reading the logits once from DRAM (256 rows x 128256 bf16: 66 MB, 10 us).  A row is read for its maximum and,
// from L2, once more: one that nothing cuts for its mass and the choice (four noises from one Philox block), one that top-k or
// top-p cut for its mass (top-p alone) and to collect the entries within kReach of the maximum; as a rule they decide
// both cuts (top-k: there are at least k of them; top-p: their mass reaches p of the whole), and thresholds, noise and
// sums are then a matter of a few hundred entries in shared memory.  Rows for which they do not (flat distributions
// under a p near 1, more than kList entries that close) and typical-p take thresholds from histograms over the whole row.
// Measured, 256 rows x 128256 bf16, temperature 0.7, top-p 0.9, repetition penalty over 350 to 1050 ids: 60 us where the lists
// decide all rows, 177 where one row in the batch is left to the histograms.  A radix select over every row (bytes of the float as
// bins: most atomics met on a few of them, and one thread walked 255 bins per byte) took 686 us after 47 us for a penalised fp32 copy
// of the logits.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "launch.cuh"
#include "sampling.cuh"

namespace {

using tgi_sampling::gumbel_noise;
using tgi_sampling::order_bits;
using tgi_sampling::philox4x32;

// A row of logits as the sampler sees it.  Penalised entries are met once each, apart from the others: a 16-byte load that
// holds some (the ids of a 1000-token history are in most warps' loads) leaves them out, and their scores, computed with
// one division each when the row is set up, follow from a list.
template <typename T>
struct Row {
  const T* p;
  int V;
  float inv_t;
  const uint32_t* marks;       // a bit per id: penalised (null: none)
  const float* pen_x;          // scores of the penalised entries and their indices, n_pen of them in any order
  const int* pen_i;
  int n_pen;
  static constexpr int VEC = 16 / sizeof(T);

  __device__ __forceinline__ int vectors() const { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 ? V / VEC : 0; }
  __device__ __forceinline__ void unpack(const uint4& raw, int v, float (&x)[VEC]) const {
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int j = 0; j < VEC; ++j) x[j] = static_cast<float>(e[j]) * inv_t;
    if (marks == nullptr) return;
    const uint32_t bits = marks[(v * VEC) >> 5] >> ((v * VEC) & 31);
    if ((bits & ((1u << VEC) - 1u)) == 0u) return;
#pragma unroll
    for (int j = 0; j < VEC; ++j)
      if ((bits >> j) & 1u) x[j] = -INFINITY;
  }
  // fv(first index, scores) for runs of VEC entries (16-byte loads, four in flight per thread), f1(index, score) for
  // the others; -inf may stand in for an entry that is met elsewhere
  template <typename FV, typename F1>
  __device__ __forceinline__ void scan(FV&& fv, F1&& f1) const {
    const int nvec = vectors(), step = blockDim.x;
    const uint4* src = reinterpret_cast<const uint4*>(p);
    for (int v = threadIdx.x; v < nvec; v += 4 * step) {
      uint4 raw[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (v + u * step < nvec) raw[u] = __ldg(src + v + u * step);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (v + u * step < nvec) {
          float x[VEC];
          unpack(raw[u], v + u * step, x);
          fv((v + u * step) * VEC, x);
        }
      }
    }
    for (int i = nvec * VEC + threadIdx.x; i < V; i += step)
      if (marks == nullptr || ((marks[i >> 5] >> (i & 31)) & 1u) == 0u) f1(i, static_cast<float>(p[i]) * inv_t);
    for (int j = threadIdx.x; j < n_pen; j += step) f1(pen_i[j], pen_x[j]);
  }
  template <typename F>
  __device__ __forceinline__ void each(F&& f) const {
    scan([&](int i, const float(&x)[VEC]) {
#pragma unroll
      for (int j = 0; j < VEC; ++j) f(i + j, x[j]);
    }, f);
  }
};

__device__ __forceinline__ unsigned long long block_sum(unsigned long long v, unsigned long long* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  unsigned long long t = 0ull;
  for (int w = 0; w < (blockDim.x >> 5); ++w) t += red[w];
  return t;
}

constexpr int kHistCopies = 16;          // of a 256-bin histogram: one per warp or pair of warps
constexpr int kBins = 1024, kBinCopies = 4;      // the same memory as bins of 1/32 below the maximum
constexpr float kBinScale = 32.f;
// History that is listed: with it and 160k bits of marks a row takes 108 KB, two rows to an SM.  The caller turns to a penalised
// copy of the scores for longer ones; dividing where an entry is read instead took 3247 us for typical-p over 256 rows x 128256 with
// 4096 ids and 454 for top-k, the copy and the sampler 1170 and 201.
constexpr int kPenalised = 3072;
constexpr float kFixedOne = 1099511627776.f;   // 2^40
constexpr float kReach = 8.f;            // entries below the maximum by more than this are not listed
constexpr int kList = 4096;              // listed entries

// Weights are summed as 2^-40 fixed point in 64-bit integers, every one of them: the sums do not depend on the order in which atomics
// land or penalised ids were listed, nor on the number of threads or the row's alignment.  The same row always yields the same
// thresholds and the same log-probability, whatever batch it is in.
__device__ __forceinline__ unsigned long long mass_of(float x, float m) {
  return static_cast<unsigned long long>(__expf(x - m) * kFixedOne);
}

// Smallest t in [0, 2^bits) such that  sum of w(x) over the entries with key(x) > t  is below `lim`  (w = 1 or
// exp(x - m)), for the entries that `each` visits and whose `key(x, k)` is true.  Radix select, most significant byte
// first: one pass per byte builds a 256-bin histogram of the weights of the entries that match the bytes found so far,
// and a walk down the bins (by one warp, eight bins a lane) finds the byte of t: the lowest bin whose entries can still
// be left out.
template <bool MASS, int COPIES, typename E, typename K>
__device__ uint32_t find_threshold(E&& each, K&& key, int bits, float m, unsigned long long lim, unsigned long long* hist,
                                   unsigned long long* tot) {
  const int copy = (threadIdx.x >> 5) % COPIES;
  uint32_t prefix = 0u;
  unsigned long long above = 0ull;         // weight of the entries whose leading bytes exceed the prefix
  unsigned int* hist32 = reinterpret_cast<unsigned int*>(hist);      // counts fit 32 bits: the cheaper atomic
  for (int shift = bits; shift > 0;) {
    const int hi = shift;
    shift = shift > 8 ? shift - 8 : 0;
    __syncthreads();
    for (int i = threadIdx.x; i < COPIES * 256; i += blockDim.x) hist[i] = 0ull;
    __syncthreads();
    const uint32_t hi_mask = hi >= 32 ? 0u : (0xffffffffu << hi);
    each([&](int, float x) {
      uint32_t k;
      if (key(x, k) && (k & hi_mask) == prefix) {
        if (MASS) {
          const unsigned long long w = mass_of(x, m);
          if (w != 0ull) atomicAdd(&hist[copy * 256 + ((k >> shift) & 255u)], w);
        } else {
          atomicAdd(&hist32[copy * 256 + ((k >> shift) & 255u)], 1u);
        }
      }
    });
    __syncthreads();
    for (int b = threadIdx.x; b < 256; b += blockDim.x) {
      unsigned long long t = 0ull;
#pragma unroll
      for (int c = 0; c < COPIES; ++c)
        t += MASS ? hist[c * 256 + b] : static_cast<unsigned long long>(hist32[c * 256 + b]);
      tot[b] = t;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      // lane l holds the bins 255 - 8 l .. 248 - 8 l; `before` is the weight above them
      const int top = 255 - 8 * static_cast<int>(threadIdx.x);
      unsigned long long own = 0ull;
      for (int j = 0; j < 8; ++j) own += tot[top - j];
      unsigned long long incl = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
        if (static_cast<int>(threadIdx.x) >= o) incl += y;
      }
      const unsigned int reach = __ballot_sync(0xffffffffu, above + incl >= lim);
      const int at = reach != 0u ? __ffs(reach) - 1 : 31;      // none: the walk ends in bin 0
      if (static_cast<int>(threadIdx.x) == at) {
        unsigned long long run = above + incl - own;
        int v = top;
        while (v > top - 7 && run + tot[v] < lim) run += tot[v--];
        tot[256] = run;
        tot[257] = static_cast<unsigned long long>(v);
      }
    }
    __syncthreads();
    above = tot[256];
    prefix |= static_cast<uint32_t>(tot[257]) << shift;
  }
  __syncthreads();
  return prefix;
}

// The same threshold for a whole row, as order_bits, in two passes over it: a histogram over 1024 bins of 1/32 below
// the maximum (bytes of the float would put most entries of a row into a handful of bins, and atomics on one address
// take turns), then the entries of the one bin that holds the threshold, which are listed and decided by a radix
// select.  A bin with more entries than the list holds, of more than one value, sends the row to a radix select over all
// of it.  Entries below `floor_bits` are left out; 0: nothing is cut.
template <bool MASS, typename T>
__device__ uint32_t row_threshold(const Row<T>& row, uint32_t floor_bits, float m, unsigned long long lim, unsigned long long* hist,
                                  unsigned long long* tot, float* list_x, int* list_i, int* s_n, uint32_t* s_lo_hi) {
  const int copy = (threadIdx.x >> 5) % kBinCopies;
  unsigned int* hist32 = reinterpret_cast<unsigned int*>(hist);
  auto bin_of = [&](float x) { return static_cast<int>(fminf((m - x) * kBinScale, static_cast<float>(kBins - 1))); };
  __syncthreads();
  for (int i = threadIdx.x; i < kBinCopies * kBins; i += blockDim.x) hist[i] = 0ull;
  __syncthreads();
  row.each([&](int, float x) {
    if (x == -INFINITY || order_bits(x) < floor_bits) return;
    if (MASS) {
      const unsigned long long w = mass_of(x, m);
      if (w != 0ull) atomicAdd(&hist[copy * kBins + bin_of(x)], w);
    } else {
      atomicAdd(&hist32[copy * kBins + bin_of(x)], 1u);
    }
  });
  __syncthreads();
  if (threadIdx.x == 0) {
    *s_n = 0;
    s_lo_hi[0] = 0xffffffffu;
    s_lo_hi[1] = 0u;
  }
  if (threadIdx.x < 32) {
    // 32 bins a lane, nearest the maximum first: the first bin with which the sum reaches the limit
    auto sum_of = [&](int b) {
      unsigned long long t = 0ull;
#pragma unroll
      for (int c = 0; c < kBinCopies; ++c)
        t += MASS ? hist[c * kBins + b] : static_cast<unsigned long long>(hist32[c * kBins + b]);
      return t;
    };
    const int first = threadIdx.x * (kBins / 32);
    unsigned long long own = 0ull;
    for (int j = 0; j < kBins / 32; ++j) own += sum_of(first + j);
    unsigned long long incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
      if (static_cast<int>(threadIdx.x) >= o) incl += y;
    }
    const unsigned int reach = __ballot_sync(0xffffffffu, incl >= lim);
    if (reach == 0u) {
      if (threadIdx.x == 0) tot[257] = kBins;
    } else if (static_cast<int>(threadIdx.x) == __ffs(reach) - 1) {
      unsigned long long run = incl - own;
      int b = first;
      for (unsigned long long t; b < first + kBins / 32 - 1 && run + (t = sum_of(b)) < lim; ++b) run += t;
      tot[256] = run;
      tot[257] = static_cast<unsigned long long>(b);
    }
  }
  __syncthreads();
  const int bin = static_cast<int>(tot[257]);
  const unsigned long long before = tot[256];
  if (bin == kBins) return 0u;
  row.each([&](int i, float x) {
    if (x == -INFINITY || order_bits(x) < floor_bits || bin_of(x) != bin) return;
    const uint32_t o = order_bits(x);
    if (o < s_lo_hi[0]) atomicMin(&s_lo_hi[0], o);
    if (o > s_lo_hi[1]) atomicMax(&s_lo_hi[1], o);
    const int at = atomicAdd(s_n, 1);
    if (at < kList) {
      list_x[at] = x;
      list_i[at] = i;
    }
  });
  __syncthreads();
  const int n = *s_n;
  const uint32_t lo = s_lo_hi[0], hi = s_lo_hi[1];
  if (lo >= hi) return min(lo, order_bits(m));
  auto all = [&](float x, uint32_t& key) {
    key = order_bits(x);
    return key >= floor_bits;
  };
  if (n <= kList) {
    auto listed = [&](auto&& f) {
      for (int j = threadIdx.x; j < n; j += blockDim.x) f(list_i[j], list_x[j]);
    };
    return find_threshold<MASS, 1>(listed, all, 32, m, lim - before, hist, tot);
  }
  return find_threshold<MASS, kHistCopies>([&](auto&& f) { row.each([&](int i, float x) { if (x != -INFINITY) f(i, x); }); }, all, 32,
                                           m, lim, hist, tot);
}

// The image for rows that may hold NaN: below every number that is not negative.  The bits of a NaN depend on the instructions that the
// compiler makes of a product or a division, so order_bits would differ from pass to pass.
__device__ __forceinline__ uint32_t key_bits(float x) { return x == x ? order_bits(x) : 0x7fffffffu; }

// Mass of the entries of a row from `keep_from` on; `none`: some of them has no mass (NaN, or an infinite maximum).
template <typename T>
__device__ unsigned long long kept_mass(const Row<T>& row, float m, uint32_t keep_from, unsigned long long* red, bool& none) {
  unsigned long long w = 0ull;
  bool odd = false;
  row.each([&](int, float x) {
    if (key_bits(x) < keep_from) return;
    const float e = __expf(x - m);
    if (e == e) w += static_cast<unsigned long long>(e * kFixedOne);
    else odd = true;
  });
  none = __syncthreads_or(odd);
  return block_sum(w, red);
}

// Typical-p (utils/logits_process.py:389-448): over the entries the earlier filters kept, with p_j their
// renormalised probabilities and H their entropy, keep the entries with the smallest |-log p_j - H| whose mass
// reaches `mass`.  Returns the largest kept deviation as float bits (deviations are >= 0, so their bit patterns
// order like the values); found by bisection, no sort.
template <typename T>
__device__ uint32_t typical_threshold(const Row<T>& row, float m, uint32_t keep_from, float mass, unsigned long long* red,
                                      float* log_z_out, float* entropy_out) {
  // H = log z + sum of exp(x - m) (m - x) / z, the sum in the same fixed point (no term above 1 / e)
  unsigned long long w = 0ull, s = 0ull;
  bool odd = false;
  row.each([&](int, float x) {
    if (key_bits(x) < keep_from || x == -INFINITY) return;
    const float e = __expf(x - m);
    if (e == e) {
      w += static_cast<unsigned long long>(e * kFixedOne);
      s += static_cast<unsigned long long>(e * (m - x) * kFixedOne);
    } else {
      odd = true;
    }
  });
  odd = __syncthreads_or(odd);
  w = block_sum(w, red);
  s = block_sum(s, red);
  const float z = odd ? __uint_as_float(0x7fc00000u) : static_cast<float>(w) / kFixedOne;
  const float log_z = __logf(z), H = log_z + static_cast<float>(s) / kFixedOne / z;
  *log_z_out = log_z;
  *entropy_out = H;
  if (odd) return 0x7f800000u;
  const unsigned long long lim = static_cast<unsigned long long>(fmaxf(mass * z, 0.f) * kFixedOne);
  uint32_t lo = 0u, hi = 0x7f800000u;       // predicate "mass of deviations <= t reaches `lim`": true at +inf
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    unsigned long long acc = 0ull;
    row.each([&](int, float x) {
      if (key_bits(x) >= keep_from && x != -INFINITY) {
        const float lp = x - m - log_z;
        if (__float_as_uint(fabsf(-lp - H)) <= mid) acc += mass_of(x, m);
      }
    });
    if (block_sum(acc, red) >= lim) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

// The entry with the largest key so far; of equal keys the one with the smallest index.
struct Best {
  float key = -INFINITY, x = 0.f;
  int i = 0x7fffffff;
  __device__ __forceinline__ void take(float k2, float x2, int i2) {
    if (k2 > key || (k2 == key && i2 < i)) {
      key = k2;
      x = x2;
      i = i2;
    }
  }
};

// `hist`, `list_x`, `list_i`, `marks` share the dynamic shared memory; see sample_bytes().
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
sample_kernel(const T* __restrict__ scores, long long row_stride, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p, const float* __restrict__ typical_p,
              const unsigned char* __restrict__ do_sample, const long long* __restrict__ seeds,
              const int* __restrict__ steps, const long long* __restrict__ history, int L, const float* __restrict__ rep,
              long long* __restrict__ ids, float* __restrict__ logprob, int V) {
  tgi::pdl_wait();      // inputs come from earlier kernels of the stream
  extern __shared__ __align__(16) unsigned char dyn[];
  unsigned long long* hist = reinterpret_cast<unsigned long long*>(dyn);          // [kHistCopies * 256]
  unsigned long long* tot = hist + kHistCopies * 256;                            // [258]
  float* list_x = reinterpret_cast<float*>(tot + 258);                           // [kList]
  int* list_i = reinterpret_cast<int*>(list_x + kList);                          // [kList]
  float* pen_x = reinterpret_cast<float*>(list_i + kList);                       // [kPenalised], with rep only
  int* pen_i = reinterpret_cast<int*>(pen_x + kPenalised);                       // [kPenalised]
  uint32_t* marks = reinterpret_cast<uint32_t*>(pen_i + kPenalised);             // [V / 32, rounded up]
  __shared__ float red[32], s_x[32];
  __shared__ int s_i[32], s_n;
  __shared__ uint32_t s_lo_hi[2];
  __shared__ unsigned long long red64[32];
  const int b = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kWarps = THREADS / 32;
  const float temp = temperature != nullptr ? temperature[b] : 1.f;
  Row<T> row{scores + static_cast<size_t>(b) * row_stride, V, 1.f / (temp > 0.f ? temp : 1.f), nullptr, pen_x, pen_i, 0};
  if (rep != nullptr && rep[b] != 1.f) {
    const float rp = rep[b];
    row.marks = marks;
    for (int w = threadIdx.x; w < (V + 31) / 32; w += THREADS) marks[w] = 0u;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    const long long* h = history + static_cast<size_t>(b) * L;
    for (int l = threadIdx.x; l < L; l += THREADS) {
      const long long t = h[l];
      if (t < 0 || t >= V) continue;
      const uint32_t bit = 1u << (t & 31);
      if (atomicOr(&marks[t >> 5], bit) & bit) continue;         // met before
      const int at = atomicAdd(&s_n, 1);                         // below L <= kPenalised
      const float x = static_cast<float>(row.p[t]);
      pen_x[at] = (x < 0.f ? x * rp : x / rp) * row.inv_t;
      pen_i[at] = static_cast<int>(t);
    }
    __syncthreads();
    row.n_pen = s_n;
    __syncthreads();
  }
  const int k = top_k != nullptr ? top_k[b] : 0;
  const float p = top_p != nullptr ? top_p[b] : 1.f;
  const float typ = typical_p != nullptr ? typical_p[b] : 1.f;
  const bool sample = do_sample != nullptr && do_sample[b] != 0;
  const uint64_t seed = seeds != nullptr ? static_cast<uint64_t>(seeds[b]) : 0ull;
  const uint32_t step = steps != nullptr ? static_cast<uint32_t>(steps[b]) : 0u;
  const bool cut_k = k > 0 && k < V, cut_p = p < 1.f, cut_typ = typ < 1.f;

  // ---- first pass: maximum ----
  float m = -INFINITY;
  bool odd = false;               // a NaN somewhere
  row.each([&](int, float x) {
    m = fmaxf(m, x);
    odd |= x != x;
  });
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) red[warp] = m;
  if (threadIdx.x == 0) s_n = 0;
  odd = __syncthreads_or(odd);
  m = red[0];
  for (int w = 1; w < kWarps; ++w) m = fmaxf(m, red[w]);
  __syncthreads();
  Best best;

  // the choice among `best` of all threads, and its log-probability
  auto finish = [&](float z_kept) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float k2 = __shfl_xor_sync(0xffffffffu, best.key, o), x2 = __shfl_xor_sync(0xffffffffu, best.x, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, best.i, o);
      best.take(k2, x2, i2);
    }
    __syncthreads();
    if (lane == 0) {
      red[warp] = best.key;
      s_i[warp] = best.i;
      s_x[warp] = best.x;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < kWarps; ++w) best.take(red[w], s_x[w], s_i[w]);
      ids[b] = best.i == 0x7fffffff ? 0 : best.i;
      logprob[b] = best.x - m - __logf(z_kept);
    }
  };
  if (!cut_k && !cut_p && !cut_typ) {
    // ---- second pass over a row that nothing cuts: its mass and the choice ----
    unsigned long long w = 0ull;
    row.scan([&](int i, const float(&x)[Row<T>::VEC]) {
#pragma unroll
      for (int j = 0; j < Row<T>::VEC; ++j)
        if (x[j] > -INFINITY) w += mass_of(x[j], m);
      if (sample) {
#pragma unroll
        for (int q = 0; q < Row<T>::VEC; q += 4) {
          // one Philox block holds the noise of four entries (the same numbers as gumbel_noise entry by entry)
          const uint4 r = philox4x32(static_cast<uint32_t>(i + q) >> 2, step, static_cast<uint32_t>(seed),
                                     static_cast<uint32_t>(seed >> 32));
          const uint32_t bits[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (x[q + j] == -INFINITY) continue;
            best.take(x[q + j] + tgi_sampling::gumbel_of(bits[j]), x[q + j], i + q + j);
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < Row<T>::VEC; ++j)
          if (x[j] != -INFINITY) best.take(x[j], x[j], i + j);
      }
    }, [&](int i, float x) {
      if (x > -INFINITY) w += mass_of(x, m);
      if (x != -INFINITY) best.take(sample ? x + gumbel_noise(static_cast<uint32_t>(i), step, seed) : x, x, i);
    });
    w = block_sum(w, red64);
    finish(odd ? __uint_as_float(0x7fc00000u) : static_cast<float>(w) / kFixedOne);
    return;
  }

  unsigned long long all = 0ull;          // mass of the row, where the second pass took it
  if (!cut_typ && !odd && m > -INFINITY && m < INFINITY) {
    // ---- second pass: the entries within kReach of the maximum, for top-p without top-k the mass of the row ----
    // compared as order_bits, as the keys below are: these put -0 under +0
    const uint32_t base = order_bits(m - kReach);
    auto put = [&](int i, float x) {
      if (order_bits(x) >= base) {
        const int at = atomicAdd(&s_n, 1);
        if (at < kList) {
          list_x[at] = x;
          list_i[at] = i;
        }
      }
    };
    if (cut_k) {
      row.each(put);
      __syncthreads();
    } else {
      row.each([&](int i, float x) {
        all += mass_of(x, m);
        put(i, x);
      });
      all = block_sum(all, red64);
    }
    const int n = s_n;
    const int bits = 32 - __clz(order_bits(m) - base);
    auto listed = [&](auto&& f) {
      for (int j = threadIdx.x; j < n; j += THREADS) f(list_i[j], list_x[j]);
    };
    bool decided = n <= kList && (!cut_k || n >= k);
    uint32_t from = 0u;                    // keep listed entries whose order_bits - base >= from
    if (decided && cut_k) {
      from = find_threshold<false, 1>(listed, [&](float x, uint32_t& key) { key = order_bits(x) - base; return true; }, bits, m,
                                      static_cast<unsigned long long>(k), hist, tot);
      from = min(from, order_bits(m) - base);
    }
    if (decided && cut_p) {
      unsigned long long w = 0ull;
      listed([&](int, float x) {
        if (order_bits(x) - base >= from) w += mass_of(x, m);
      });
      const unsigned long long have = block_sum(w, red64);
      const float z_all = static_cast<float>(cut_k ? have : all) / kFixedOne;
      const unsigned long long lim = static_cast<unsigned long long>(fmaxf(p * z_all, 0.f) * kFixedOne);
      // entries outside the list are left out if those above them reach the limit already
      decided = cut_k || have >= lim;
      if (decided) {
        const uint32_t t = find_threshold<true, 1>(listed, [&](float x, uint32_t& key) {
          key = order_bits(x) - base;
          return key >= from;
        }, bits, m, lim, hist, tot);
        from = max(from, min(t, order_bits(m) - base));
      }
    }
    if (decided) {
      unsigned long long w = 0ull;
      listed([&](int i, float x) {
        if (order_bits(x) - base < from) return;
        w += mass_of(x, m);
        best.take(sample ? x + gumbel_noise(static_cast<uint32_t>(i), step, seed) : x, x, i);
      });
      finish(static_cast<float>(block_sum(w, red64)) / kFixedOne);
      return;
    }
  }

  // ---- general way: thresholds from the whole row ----
  uint32_t keep_from = 0u;                      // keep entries whose order_bits >= keep_from
  if (odd || !(m > -INFINITY && m < INFINITY)) {
    // distances from the maximum say nothing: radix select over the row
    auto each = [&](auto&& f) { row.each(f); };
    auto key = [&](float x, uint32_t& out) {
      out = key_bits(x);
      return out >= keep_from;
    };
    if (cut_k)
      keep_from = min(find_threshold<false, kHistCopies>(each, key, 32, m, static_cast<unsigned long long>(k), hist, tot), order_bits(m));
    if (cut_p) {
      bool none;
      const float zk = static_cast<float>(kept_mass(row, m, keep_from, red64, none)) / kFixedOne;
      const unsigned long long lim = none ? 0ull : static_cast<unsigned long long>(fmaxf(p * zk, 0.f) * kFixedOne);
      keep_from = max(keep_from, min(find_threshold<true, kHistCopies>(each, key, 32, m, lim, hist, tot), order_bits(m)));
    }
  } else {
    if (cut_k)
      keep_from = min(row_threshold<false, T>(row, 0u, m, static_cast<unsigned long long>(k), hist, tot, list_x, list_i, &s_n, s_lo_hi),
                      order_bits(m));
    if (cut_p) {
      bool none;
      const float zk = static_cast<float>(cut_k || cut_typ ? kept_mass(row, m, keep_from, red64, none) : all) / kFixedOne;
      const uint32_t t = row_threshold<true, T>(row, keep_from, m, static_cast<unsigned long long>(fmaxf(p * zk, 0.f) * kFixedOne), hist,
                                                tot, list_x, list_i, &s_n, s_lo_hi);
      keep_from = max(keep_from, min(t, order_bits(m)));
    }
  }
  uint32_t typ_bits = 0xffffffffu;
  float typ_log_z = 0.f, typ_h = 0.f;
  if (cut_typ) typ_bits = typical_threshold<T>(row, m, keep_from, typ, red64, &typ_log_z, &typ_h);
  unsigned long long w = 0ull;
  bool none = false;
  row.each([&](int i, float x) {
    if (key_bits(x) < keep_from || x == -INFINITY) return;
    if (cut_typ && __float_as_uint(fabsf(-(x - m - typ_log_z) - typ_h)) > typ_bits) return;
    const float e = __expf(x - m);
    if (e == e) w += static_cast<unsigned long long>(e * kFixedOne);
    else none = true;
    best.take(sample ? x + gumbel_noise(static_cast<uint32_t>(i), step, seed) : x, x, i);
  });
  none = __syncthreads_or(none);
  w = block_sum(w, red64);
  finish(none ? __uint_as_float(0x7fc00000u) : static_cast<float>(w) / kFixedOne);
}

size_t sample_bytes(int V, bool rep) {
  return (kHistCopies * 256 + 258) * sizeof(unsigned long long) + kList * 8 +
         (rep ? kPenalised * 8 + (static_cast<size_t>(V) + 31) / 32 * 4 : 0);
}

template <typename T, int THREADS>
int launch_sample(const void* scores, long long row_stride, const float* temperature, const int* top_k, const float* top_p,
                  const float* typical_p, const unsigned char* do_sample, const long long* seeds, const int* steps,
                  const long long* history, int L, const float* rep, long long* ids, float* logprob, int B, int V,
                  cudaStream_t stream) {
  auto kern = sample_kernel<T, THREADS>;
  const size_t smem = sample_bytes(V, rep != nullptr);
  if (smem > 200 * 1024 || (rep != nullptr && L > kPenalised)) return -10;
  static std::atomic<unsigned long long> attr_set{0};      // per device: the opt-in to the largest size that is launched
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -2;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(attr_set.load(std::memory_order_acquire) & bit)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess) return -2;
    attr_set.fetch_or(bit, std::memory_order_release);
  }
  tgi::launch(kern, dim3(B), dim3(THREADS), smem, stream, static_cast<const T*>(scores), row_stride, temperature, top_k, top_p,
              typical_p, do_sample, seeds, steps, history, L, rep, ids, logprob, V);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace

extern "C" {

// Fused repetition penalty / temperature / top-k / top-p / sampling; any of temperature, top_k, top_p, do_sample, seeds, steps
// may be null (stage off).  `rep` [B] (null: none) with `history` int64 [B, L], L <= 3072.  `is_fp32` selects the element type of
// `scores`.  As many rows as the device has SMs run on 1024 threads each, more on 512, two rows to an SM; results are the same.
int tgi_sample(const void* scores, long long row_stride, int is_fp32, const float* temperature, const int* top_k,
               const float* top_p, const float* typical_p, const unsigned char* do_sample, const long long* seeds,
               const int* steps, const long long* history, int L, const float* rep, long long* ids, float* logprob, int B, int V,
               cudaStream_t stream) {
  if (B <= 0) return 0;
  if (V <= 0) return -10;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -2;
  if (is_fp32)
    return B <= sms ? launch_sample<float, 1024>(scores, row_stride, temperature, top_k, top_p, typical_p, do_sample, seeds, steps,
                                                 history, L, rep, ids, logprob, B, V, stream)
                    : launch_sample<float, 512>(scores, row_stride, temperature, top_k, top_p, typical_p, do_sample, seeds, steps,
                                                history, L, rep, ids, logprob, B, V, stream);
  return B <= sms ? launch_sample<__nv_bfloat16, 1024>(scores, row_stride, temperature, top_k, top_p, typical_p, do_sample, seeds,
                                                       steps, history, L, rep, ids, logprob, B, V, stream)
                  : launch_sample<__nv_bfloat16, 512>(scores, row_stride, temperature, top_k, top_p, typical_p, do_sample, seeds,
                                                      steps, history, L, rep, ids, logprob, B, V, stream);
}

}  // extern "C"
