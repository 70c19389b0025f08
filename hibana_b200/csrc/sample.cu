// Sampling and speculative verify-and-accept kernels for sm_100a.
//
//  * argmax over bf16 / fp32 logits rows (greedy), optional grammar bitmask.
//  * temperature / top-k / top-p sampling, one CTA per row, counter-based RNG keyed by (seed, offset) so a
//    request's draws do not depend on batch composition.
//  * exact greedy acceptance of a drafted block (longest matching prefix + the target's own token), with stop
//    ids and a token budget, producing device-resident counts.
//  * rank / logit gap of a drafted token in its verify row (relaxed acceptance).
//
// Reference counterparts: hibana/engine/sampler.py:87-123, hibana/engine/accept.py:18-56,
// hibana/kernels/relaxed_rank.py:13, hibana/kernels/sampled_verify.py:17, hibana/engine/accept_graphs.py.
#include "hb_api.h"
#include "hb_common.cuh"

namespace hb {
namespace {

template <typename T>
__device__ __forceinline__ float ldf(const T* p, long long i);
template <>
__device__ __forceinline__ float ldf<float>(const float* p, long long i) { return p[i]; }
template <>
__device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p, long long i) {
  return __bfloat162float(p[i]);
}

__device__ __forceinline__ bool mask_ok(const int* mask, int i) {
  return mask == nullptr || ((mask[i >> 5] >> (i & 31)) & 1);
}

// Lowest index wins ties (same as torch.argmax on CPU for exact ties).
template <typename T>
__global__ void __launch_bounds__(256)
argmax_kernel(const T* __restrict__ logits, long long ld, int vocab, const int* __restrict__ bitmask, int mask_words,
              long long* __restrict__ out, float* __restrict__ out_val) {
  grid_dep_wait(logits, bitmask);
  grid_dep_launch();
  __shared__ float sv[8];
  __shared__ int si[8];
  const int row = blockIdx.x;
  const T* lr = logits + row * ld;
  const int* mask = bitmask ? bitmask + static_cast<long long>(row) * mask_words : nullptr;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
    if (!mask_ok(mask, i)) continue;
    const float v = ldf<T>(lr, i);
    if (v > best || (v == best && i < bi)) {
      best = v;
      bi = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) {
      best = ov;
      bi = oi;
    }
  }
  if ((threadIdx.x & 31) == 0) {
    sv[threadIdx.x >> 5] = best;
    si[threadIdx.x >> 5] = bi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w)
      if (sv[w] > best || (sv[w] == best && si[w] < bi)) {
        best = sv[w];
        bi = si[w];
      }
    out[row] = bi == 0x7fffffff ? 0 : bi;
    if (out_val) out_val[row] = best;
  }
}

// Two-stage argmax for wide vocabularies: `nch` CTAs per row each scan a slice, then one warp per row combines.
template <typename T>
__global__ void __launch_bounds__(256)
argmax_partial_kernel(const T* __restrict__ logits, long long ld, int vocab, const int* __restrict__ bitmask,
                      int mask_words, int nch, float* __restrict__ pv, int* __restrict__ pi) {
  grid_dep_wait(logits, bitmask);
  grid_dep_launch();
  __shared__ float sv[8];
  __shared__ int si[8];
  const int row = blockIdx.x, ch = blockIdx.y;
  const T* lr = logits + row * ld;
  const int* mask = bitmask ? bitmask + static_cast<long long>(row) * mask_words : nullptr;
  const int per = (vocab + nch - 1) / nch;
  const int lo = ch * per, hi = min(vocab, lo + per);
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    if (!mask_ok(mask, i)) continue;
    const float v = ldf<T>(lr, i);
    if (v > best || (v == best && i < bi)) {
      best = v;
      bi = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) {
      best = ov;
      bi = oi;
    }
  }
  if ((threadIdx.x & 31) == 0) {
    sv[threadIdx.x >> 5] = best;
    si[threadIdx.x >> 5] = bi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w)
      if (sv[w] > best || (sv[w] == best && si[w] < bi)) {
        best = sv[w];
        bi = si[w];
      }
    pv[row * nch + ch] = best;
    pi[row * nch + ch] = bi;
  }
}

// One warp per row. Rows whose temperature is > 0 are left to the sampling kernel.
__global__ void argmax_final_kernel(const float* __restrict__ pv, const int* __restrict__ pi, int nch, int rows,
                                    const float* __restrict__ temperature, long long* __restrict__ out,
                                    float* __restrict__ out_val) {
  grid_dep_wait(pv, pi, temperature);
  grid_dep_launch();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  if (temperature != nullptr && temperature[row] > 0.f) return;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int c = lane; c < nch; c += 32) {
    const float v = pv[row * nch + c];
    const int i = pi[row * nch + c];
    if (v > best || (v == best && i < bi)) {
      best = v;
      bi = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) {
      best = ov;
      bi = oi;
    }
  }
  if (lane == 0) {
    out[row] = bi == 0x7fffffff ? 0 : bi;
    if (out_val) out_val[row] = best;
  }
}

// splitmix64-based counter RNG -> uniform in [0, 1).
__device__ __forceinline__ float uniform01(unsigned long long seed, unsigned long long offset) {
  unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (offset + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return static_cast<float>(z >> 40) * (1.0f / 16777216.0f);
}

// ---- full-vocabulary sampling (top-k off or above SAMPLE_K): softmax over every allowed token, nucleus by an exact
// threshold search, inverse-CDF draw in index order. Same law as engine/rejection.py `distribution`.
__device__ __forceinline__ unsigned order_key(float v) {   // order-preserving map float -> uint32
  const unsigned b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_value(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
// A row's kernels run 1024 threads: a pass over the vocabulary is a chain of L2 loads per thread, so its length is what counts.
// The mass above a key and the sums of the draw keep one fixed order of additions whatever the thread count: SUM_T strided
// accumulators, a tree over each warp, then the warps one after the other. The masses that the nucleus search compares with p_lim * kept
// are whole numbers, which have no order (search_key).
constexpr int LAW_T = 1024, LAW_WARPS = LAW_T / 32, SUM_T = 256;
__device__ __forceinline__ float sum_in_order(float v, float* red) {   // v counts on the first SUM_T threads; whole CTA
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int w = 0; w < SUM_T / 32; ++w) t += red[w];
  return t;
}
__device__ __forceinline__ int block_sum_i(int v, int* red) {
  v = __reduce_add_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  return __reduce_add_sync(0xffffffffu, red[threadIdx.x & 31]);
}

// A row as order keys, 0 for what is out of the law (masked, NaN, -inf: finite and +inf values have keys above 0x007fffff). Rows that
// fit are brought into shared memory once (STAGED), others are read and converted at each pass. ONE_ZERO: -0.0 has the key of 0.0.
template <typename T, bool STAGED, bool ONE_ZERO = false>
struct RowKeys {
  const T* lr;
  const int* mask;
  const unsigned* staged;
  // keys of i, i + step, ... (0 from `end` on), all loads in flight before the first is used
  template <bool RAW, int U>
  __device__ __forceinline__ void load(unsigned (&k)[U], int i, int step, int end) const {
    if (STAGED && !RAW) {
#pragma unroll
      for (int u = 0; u < U; ++u) k[u] = i + u * step < end ? staged[i + u * step] : 0u;
    } else {
      float v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = ldf<T>(lr, min(i + u * step, end - 1));
      if (mask != nullptr) {
        int m[U];
#pragma unroll
        for (int u = 0; u < U; ++u) m[u] = mask[min(i + u * step, end - 1) >> 5];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (!((m[u] >> ((i + u * step) & 31)) & 1)) v[u] = -INFINITY;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) k[u] = i + u * step < end && v[u] > -INFINITY ? order_key(v[u]) : 0u;
    }
    if (ONE_ZERO)
#pragma unroll
      for (int u = 0; u < U; ++u) k[u] = k[u] == 0x7fffffffu ? 0x80000000u : k[u];
  }
  __device__ __forceinline__ unsigned operator()(int i) const {
    unsigned k[1];
    load<false>(k, i, 1, i + 1);
    return k[0];
  }
};

// f(key, index) over begin, begin + step, ... < end in order, U loads at once (0 past the end).
template <int U = 8, typename R, typename F>
__device__ __forceinline__ void scan(const R& row, int begin, int end, int step, F f) {
  for (int i = begin; i < end; i += U * step) {
    unsigned k[U];
    row.template load<false>(k, i, step, end);
#pragma unroll
    for (int u = 0; u < U; ++u) f(k[u], i + u * step);
  }
}

// The largest key of a row (at least that of -inf); a staged row is in shared memory afterwards. Whole CTA.
template <typename R>
__device__ unsigned stage_row(const R& row, bool keep, unsigned* keys, int vocab, unsigned* red) {
  unsigned mk = order_key(-INFINITY);
  for (int i = threadIdx.x; i < vocab; i += 16 * LAW_T) {
    unsigned k[16];
    row.template load<true>(k, i, LAW_T, vocab);
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      if (keep && i + u * LAW_T < vocab) keys[i + u * LAW_T] = k[u];
      mk = max(mk, k[u]);
    }
  }
  mk = __reduce_max_sync(0xffffffffu, mk);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mk;
  __syncthreads();
  return __reduce_max_sync(0xffffffffu, red[threadIdx.x & 31]);
}

// Largest key x above `lo` that a token has and for which holds(f(x)), where f(x) is the sum of whole(k) over the tokens of keys
// k >= x above `lo`; `lo` if there is none. holds() stays true as its argument grows, no token is above hi = the key of `top`.
// Weights are whole numbers (at most 2^FIX each, 1 with ONES), so f has one value however it is added up, and every step asks
// holds() about that value: a bucket that reaches the goal has a token that does. (With fp32 sums in the second step one draw in
// about a million found none.)
// One pass adds the weights up in BUCKETS of 1/16 `width` below `top` (a nucleus ends within some temperatures of the maximum); the
// first bucket whose end holds has the answer. Its tokens are listed and each finds its own f; the largest key that holds is it. More than
// RANKED of them (ties, long rows, the last bucket) are narrowed first: buckets again, of keys, 256 to a pass. At 18992 tokens that is one
// pass and the list where narrowing 32 bits by 16 took eight passes. Whole CTA.
constexpr int BUCKETS = 256, RANKED = 1024;
constexpr int FIX = 41, FIX_PART = 14, SLAB = 1 << 18;    // a sum is kept in three parts: 2^14 * 2^18 tokens fill 32 bits
constexpr int LIST_PART = 21;                             // a listed weight in two: 2^21 * 2^10 tokens
struct SearchScratch {
  union {
    struct {
      unsigned bucket[3][BUCKETS];
      unsigned long long sum[BUCKETS];
    };
    uint4 list[RANKED];      // key, weight in two parts
  };
  unsigned long long before;
  int count[LAW_WARPS];
  unsigned best, low;
  int at;
};
__device__ __forceinline__ unsigned long long fixed(float w) { return __float2ull_rn(w * static_cast<float>(1ull << FIX)); }
__device__ __forceinline__ float from_fixed(unsigned long long s) {
  return static_cast<float>(static_cast<double>(s) * (1.0 / static_cast<double>(1ull << FIX)));
}

template <bool ONES, typename R, typename W, typename H>
__device__ unsigned search_key(const R& row, int vocab, unsigned lo, unsigned hi, float top, float width, W whole, H holds,
                               SearchScratch& sc) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (!(lo < hi)) return lo;
  if (holds(0ull)) return hi;
  unsigned long long beyond = 0;           // f of the keys above the range that is left
  // The first bucket of the keys that are `in` whose end holds (BUCKETS: none); `beyond` is then the sum in front of it. bucket(k) rises
  // as the key falls.
  auto reached = [&](auto in, auto bucket) {
    __syncthreads();
    if (tid < BUCKETS) sc.sum[tid] = 0ull;
    if (tid == 0) sc.at = BUCKETS;
    for (int from = 0; from < vocab; from += SLAB) {
      if (tid < 3 * BUCKETS) sc.bucket[0][tid] = 0u;
      __syncthreads();
      scan(row, from + tid, min(vocab - from, SLAB) + from, LAW_T, [&](unsigned k, int) {
        if (in(k)) {
          const int b = bucket(k);
          const unsigned long long w = whole(k);
          constexpr unsigned PART = (1u << FIX_PART) - 1u;
          atomicAdd(&sc.bucket[0][b], static_cast<unsigned>(w) & PART);
          if (!ONES) {
            atomicAdd(&sc.bucket[1][b], static_cast<unsigned>(w >> FIX_PART) & PART);
            atomicAdd(&sc.bucket[2][b], static_cast<unsigned>(w >> (2 * FIX_PART)));
          }
        }
      });
      __syncthreads();
      if (tid < BUCKETS)
        sc.sum[tid] += sc.bucket[0][tid] + (static_cast<unsigned long long>(sc.bucket[1][tid]) << FIX_PART) +
                       (static_cast<unsigned long long>(sc.bucket[2][tid]) << (2 * FIX_PART));
      __syncthreads();
    }
    if (tid < 32) {          // each lane owns BUCKETS / 32 in a row
      constexpr int OWN = BUCKETS / 32;
      unsigned long long own[OWN], upto = 0;
#pragma unroll
      for (int j = 0; j < OWN; ++j) own[j] = upto += sc.sum[tid * OWN + j];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      const unsigned long long front = beyond + upto - own[OWN - 1];
      const unsigned there = __ballot_sync(0xffffffffu, holds(beyond + upto));
      if (there && lane == __ffs(there) - 1)
#pragma unroll
        for (int j = OWN - 1; j >= 0; --j)
          if (holds(front + own[j])) {
            sc.at = tid * OWN + j;
            sc.before = front + (j == 0 ? 0ull : own[j - 1]);
          }
    }
    __syncthreads();
    if (sc.at < BUCKETS) beyond = sc.before;
    return sc.at;
  };
  // Lists the tokens that are `in`; if they are few the answer is found (true).
  auto ranked = [&](auto in, unsigned& answer) {
    int mine = 0;
    scan(row, tid, vocab, LAW_T, [&](unsigned k, int) { mine += in(k); });
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    if (lane == 31) sc.count[warp] = upto;
    if (tid == 0) sc.best = 0u;
    __syncthreads();
    const int c = sc.count[lane];
    const int total = __reduce_add_sync(0xffffffffu, c);
    if (total > RANKED) return false;
    int at = __reduce_add_sync(0xffffffffu, lane < warp ? c : 0) + upto - mine;
    if (mine != 0)
      scan(row, tid, vocab, LAW_T, [&](unsigned k, int) {
        if (in(k)) {
          const unsigned long long w = whole(k);
          sc.list[at++] = make_uint4(k, static_cast<unsigned>(w) & ((1u << LIST_PART) - 1u), static_cast<unsigned>(w >> LIST_PART), 0u);
        }
      });
    __syncthreads();
    if (tid < total) {
      const unsigned k = sc.list[tid].x;
      unsigned f0 = 0u, f1 = 0u;
#pragma unroll 8
      for (int i = 0; i < total; ++i) {
        const uint4 e = sc.list[i];
        f0 += e.x >= k ? e.y : 0u;
        f1 += e.x >= k ? e.z : 0u;
      }
      if (holds(beyond + f0 + (static_cast<unsigned long long>(f1) << LIST_PART))) atomicMax(&sc.best, k);
    }
    __syncthreads();
    answer = sc.best;
    return true;
  };
  const float per = 16.f / width;
  auto bucket = [&](unsigned k) {           // by roundings that keep the order
    return static_cast<int>(fminf((top - key_value(k)) * per, static_cast<float>(BUCKETS - 1)));
  };
  const int at = reached([&](unsigned k) { return k > lo; }, bucket);
  if (at == BUCKETS) return lo;
  auto in = [&](unsigned k) { return k > lo && bucket(k) == at; };
  unsigned answer;
  if (ranked(in, answer)) return answer;
  unsigned kmin = 0xffffffffu, kmax = 0u;
  scan(row, tid, vocab, LAW_T, [&](unsigned k, int) {
    if (in(k)) {
      kmin = min(kmin, k);
      kmax = max(kmax, k);
    }
  });
  if (tid == 0) sc.low = 0xffffffffu;
  __syncthreads();
  kmin = __reduce_min_sync(0xffffffffu, kmin);
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  if (lane == 0) {
    atomicMin(&sc.low, kmin);
    atomicMax(&sc.best, kmax);
  }
  __syncthreads();
  kmin = sc.low;
  kmax = sc.best;
  while (kmin < kmax) {
    const int shift = max(0, 24 - __clz(kmax - kmin));
    auto left = [&](unsigned k) { return k >= kmin && k <= kmax; };
    kmax -= static_cast<unsigned>(reached(left, [&](unsigned k) { return static_cast<int>((kmax - k) >> shift); })) << shift;
    kmin = kmax - min(kmax - kmin, (1u << shift) - 1u);
    if (ranked(left, answer)) return answer;
  }
  return kmax;
}

// The 32 values of a warp added to `acc` one after the other; `after` = the running sum behind this lane's own. Every lane gets the end.
__device__ __forceinline__ float sum_lanes(float acc, float w, int lane, float& after) {
#pragma unroll
  for (int src = 0; src < 32; ++src) {
    acc += __shfl_sync(0xffffffffu, w, src);
    if (lane == src) after = acc;
  }
  return acc;
}

// The sampling law of one row as engine/rejection.py `distribution` defines it: softmax(logits / temp) over the
// allowed tokens, cut to the first `k_lim` tokens in (value desc, index asc) order (0 = no cut), then to the
// smallest prefix of that order whose mass reaches p_lim. Draws one token by inverse CDF in index order from the
// law with token `exclude` removed (-1: nothing removed; the residual of a point-mass draft in speculative
// sampling) and reports the probability of token `probe` under the law. LAW_T threads, whole CTA. Bound by the chain of its passes
// over the row, so the row is staged where it fits. With a nucleus cut, us at 11 rows, a pass over the row for every 4
// bits of the cut / now: 18992 tokens 85 / 31, 31040 113 / 43, 52224 167 / 68, 151936 (not staged) 479 / 287; cut off
// 26 / 17, 36 / 22, 53 / 31, 163 / 116 (0 of 23040 draws differed).
template <typename T, bool STAGED>
__device__ void law_row(const T* lr, int vocab, const int* mask, float temp, int k_lim, float p_lim, float u01, int exclude,
                        int probe, long long* out, float* out_prob, float* out_probe, SearchScratch& sc) {
  constexpr int CHUNKS = 256;              // contiguous pieces of the row for the draw
  extern __shared__ unsigned row_keys[];   // STAGED: vocab of them
  __shared__ unsigned redu[LAW_WARPS];
  __shared__ float red[LAW_WARPS];
  __shared__ int redi[LAW_WARPS];
  __shared__ float cweight[CHUNKS];
  __shared__ int ceq[CHUNKS];              // threshold tokens in front of a chunk
  __shared__ int ceq_warp[CHUNKS / 32];
  const int tid = threadIdx.x;
  const float inv_t = 1.f / temp;
  const RowKeys<T, STAGED> row{lr, mask, row_keys};
  const unsigned mk = stage_row(row, STAGED, row_keys, vocab, redu);
  const float mx = key_value(mk);
  // ---- top-k cut: tk_key = value of the k-th token, need_k = how many of the tokens equal to it are inside
  unsigned tk_key = 0;
  int need_k = 0x7fffffff;
  bool cut_k = k_lim > 0 && k_lim < vocab;
  if (cut_k) {
    tk_key = search_key<true>(row, vocab, 0u, mk, mx, temp, [](unsigned) { return 1ull; },
                              [&](unsigned long long n) { return n >= k_lim; }, sc);
    cut_k = tk_key != 0u;                  // fewer live tokens than that: all of them are inside
  }
  if (cut_k) {
    int above = 0;
    scan(row, tid, vocab, LAW_T, [&](unsigned k, int) { above += k > tk_key; });
    need_k = k_lim - block_sum_i(above, redi);
  }
  // mass above a key and number of tokens equal to it
  float m_above = 0.f;
  int n_eq = 0;
  auto mass_above = [&](unsigned key) {
    m_above = 0.f;
    n_eq = 0;
    if (tid < SUM_T)
      scan(row, tid, vocab, SUM_T, [&](unsigned k, int) {
        const float w = __expf((key_value(max(k, 0x00800000u)) - mx) * inv_t);    // (no branch around it)
        m_above += k > key ? w : 0.f;
        n_eq += k == key && k != 0u;
      });
    m_above = sum_in_order(m_above, red);
    n_eq = block_sum_i(n_eq, redi);
  };
  mass_above(tk_key);
  unsigned t_key = tk_key;
  int need_eq = min(need_k, n_eq);
  float w_t = cut_k ? __expf((key_value(tk_key) - mx) * inv_t) : 0.f;
  float kept = m_above + (cut_k ? need_eq * w_t : 0.f);
  // ---- nucleus inside the cut: the smallest prefix, in the same order, whose mass reaches p_lim * kept
  if (p_lim < 1.f) {
    const float want = p_lim * kept;
    // mass(key >= tk_key) = kept >= want, and every token above tk_key is inside the cut
    unsigned lo = search_key<false>(row, vocab, tk_key, mk, mx, temp,
                                    [&](unsigned k) { return fixed(__expf((key_value(k) - mx) * inv_t)); },
                                    [&](unsigned long long m) { return from_fixed(m) >= want; }, sc);
    if (lo == 0u) {        // the whole numbers' mass is a rounding short of p_lim * kept (p_lim next to 1): all tokens are inside
      lo = 0xffffffffu;
      scan(row, tid, vocab, LAW_T, [&](unsigned k, int) { lo = min(lo, k - 1u); });      // (0, no token's, becomes the largest)
      lo = __reduce_min_sync(0xffffffffu, lo);
      if (tid % 32 == 0) redu[tid / 32] = lo;
      __syncthreads();
      lo = __reduce_min_sync(0xffffffffu, redu[tid % 32]) + 1u;
    }
    if (lo != tk_key || !cut_k) {
      t_key = lo;
      mass_above(t_key);
      w_t = __expf((key_value(t_key) - mx) * inv_t);
      need_eq = n_eq;
    }
    int need = w_t > 0.f ? static_cast<int>(ceilf((want - m_above) / w_t)) : 1;
    need_eq = max(1, min(need, need_eq));
    kept = m_above + need_eq * w_t;
  }
  // ---- membership and weight of the probed / excluded token (its rank among equals decides at the threshold)
  float w_probe = 0.f, w_ex = 0.f;
  for (int pass = 0; pass < 2; ++pass) {
    const int tok = pass == 0 ? probe : exclude;
    if (tok < 0 || tok >= vocab) continue;
    if (pass == 1 && exclude == probe) {
      w_ex = w_probe;
      continue;
    }
    const unsigned k = row(tok);
    float w = 0.f;
    if (k > t_key) w = __expf((key_value(k) - mx) * inv_t);
    else if (k == t_key && k != 0u) {
      int before = 0;
      scan(row, tid, tok, LAW_T, [&](unsigned k2, int) { before += k2 == t_key; });
      before = block_sum_i(before, redi);
      if (before < need_eq) w = w_t;
    }
    if (pass == 0) w_probe = w;
    else w_ex = w;
  }
  if (out_probe != nullptr && tid == 0) *out_probe = w_probe / kept;
  if (!(kept - w_ex > kept * 1e-6f)) {      // nothing left beside the excluded token: the law itself is drawn from
    exclude = -1;
    w_ex = 0.f;
  }
  const float kept_draw = kept - w_ex;
  // ---- draw: mass and number of threshold tokens per chunk, the chunk the draw falls into, then the token in it; all sums in
  // index order
  const int per = (vocab + CHUNKS - 1) / CHUNKS;
  const int ex_chunk = exclude >= 0 ? exclude / per : -1;
  float mine = 0.f;
  int my_eq = 0, eq_before = 0;
  if (tid < CHUNKS) {
    scan(row, tid * per, min(vocab, (tid + 1) * per), 1, [&](unsigned k, int) {
      const float w = __expf((key_value(max(k, 0x00800000u)) - mx) * inv_t);
      mine += k > t_key ? w : 0.f;
      my_eq += k == t_key && k != 0u;
    });
    eq_before = my_eq;                      // running count over the chunks: whole numbers, any order
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, eq_before, o);
      if ((tid & 31) >= o) eq_before += v;
    }
    if ((tid & 31) == 31) ceq_warp[tid >> 5] = eq_before;
    eq_before -= my_eq;
  }
  __syncthreads();
  if (tid < CHUNKS) {
    for (int w = 0; w < (tid >> 5); ++w) eq_before += ceq_warp[w];
    const int take = max(0, min(my_eq, need_eq - eq_before));
    float w = mine + take * w_t;
    if (tid == ex_chunk) w = fmaxf(w - w_ex, 0.f);
    cweight[tid] = w;
    ceq[tid] = eq_before;
  }
  __syncthreads();
  const float u = u01 * kept_draw;
  if (tid < 32) {        // one warp adds 32 chunks, then 32 tokens of the chunk, at a time and in order
    float acc = 0.f, base = -1.f, after = 0.f;
    int pick = -1, last = 0;
    for (int t = 0; t < CHUNKS && pick < 0; t += 32) {
      const float w = cweight[t + tid], before = acc;
      acc = sum_lanes(acc, w, tid, after);
      const unsigned kept_mask = __ballot_sync(0xffffffffu, w > 0.f), hit = __ballot_sync(0xffffffffu, u < after);
      if (kept_mask) last = t + 31 - __clz(kept_mask);
      if (hit) {
        const int at = __ffs(hit) - 1;
        pick = t + at;
        base = at == 0 ? before : __shfl_sync(0xffffffffu, after, at - 1);
      }
    }
    if (pick < 0) pick = last;             // rounding: u landed past the last kept token (base stays -1)
    acc = base;
    int eq_seen = ceq[pick], chosen = -1, last_kept = -1;
    float w_chosen = 0.f, w_last = 0.f;
    const int hi_i = min(vocab, (pick + 1) * per);
    for (int i0 = pick * per; i0 < hi_i && chosen < 0; i0 += 32) {
      const int i = i0 + tid;
      const unsigned k = i < hi_i ? row(i) : 0u;
      const unsigned equal = __ballot_sync(0xffffffffu, k == t_key && k != 0u);
      float w = 0.f;
      if (k > t_key) w = __expf((key_value(k) - mx) * inv_t);
      else if (k == t_key && k != 0u && eq_seen + __popc(equal & ((1u << tid) - 1u)) < need_eq) w = w_t;
      if (i == exclude || !(w > 0.f)) w = 0.f;
      eq_seen += __popc(equal);
      acc = sum_lanes(acc, w, tid, after);                 // (a dropped token's zero changes nothing)
      const unsigned kept_mask = __ballot_sync(0xffffffffu, w > 0.f);
      const unsigned hit = __ballot_sync(0xffffffffu, w > 0.f && base >= 0.f && u < after);
      if (kept_mask == 0u) continue;
      const int at = hit ? __ffs(hit) - 1 : 31 - __clz(kept_mask);
      last_kept = i0 + at;
      w_last = __shfl_sync(0xffffffffu, w, at);
      if (hit) {
        chosen = last_kept;
        w_chosen = w_last;
      }
    }
    if (chosen < 0) {
      chosen = last_kept < 0 ? 0 : last_kept;
      w_chosen = w_last;
    }
    if (tid == 0) {
      *out = chosen;
      if (out_prob) *out_prob = w_chosen / kept_draw;
    }
  }
  __syncthreads();
}

constexpr int SAMPLE_K = 64;  // candidates kept per row for 1 <= top-k <= 64 (top-p is applied inside them)

// The k first tokens of a row in (value desc, index asc) order, 0.0 and -0.0 equal: value and index to cv, ci. False, and nothing
// written, when the row has fewer. Whole CTA.
template <typename T, bool STAGED>
__device__ bool list_candidates(const T* lr, int vocab, const int* mask, int k, float temp, float* cv, int* ci,
                                SearchScratch& sc) {
  extern __shared__ unsigned row_keys[];
  __shared__ unsigned redu[LAW_WARPS], gk[SAMPLE_K];
  __shared__ int gi[SAMPLE_K], ei[SAMPLE_K], n_above, n_equal;
  const int tid = threadIdx.x;
  const RowKeys<T, STAGED, true> row{lr, mask, row_keys};
  const unsigned mk = stage_row(row, STAGED, row_keys, vocab, redu);
  const unsigned tk = search_key<true>(row, vocab, 0u, mk, key_value(mk), temp, [](unsigned) { return 1ull; },
                                       [&](unsigned long long n) { return n >= k; }, sc);
  if (tk <= 0x007fffffu) return false;
  if (tid == 0) n_above = n_equal = 0;
  __syncthreads();
  scan(row, tid, vocab, LAW_T, [&](unsigned x, int i) {
    if (x > tk) {
      const int at = atomicAdd(&n_above, 1);               // fewer than k of them
      gk[at] = x;
      gi[at] = i;
    } else if (x == tk) {
      const int at = atomicAdd(&n_equal, 1);
      if (at < SAMPLE_K) ei[at] = i;
    }
  });
  __syncthreads();
  const int above = n_above, equal = n_equal;
  if (tid < above) {
    int rank = 0;
    for (int j = 0; j < above; ++j) rank += gk[j] > gk[tid] || (gk[j] == gk[tid] && gi[j] < gi[tid]);
    cv[rank] = key_value(gk[tid]);
    ci[rank] = gi[tid];
  }
  if (equal <= SAMPLE_K) {
    if (tid < equal) {
      int rank = above;
      for (int j = 0; j < equal; ++j) rank += ei[j] < ei[tid];
      if (rank < k) {
        cv[rank] = key_value(tk);
        ci[rank] = ei[tid];
      }
    }
  } else {                                                 // many: in index order, a warp at a time
    if (tid < 32)
      for (int i0 = 0, got = above; i0 < vocab && got < k; i0 += 32) {
        const bool is = i0 + tid < vocab && row(i0 + tid) == tk;
        const unsigned m = __ballot_sync(0xffffffffu, is);
        const int rank = got + __popc(m & ((1u << tid) - 1u));
        if (is && rank < k) {
          cv[rank] = key_value(tk);
          ci[rank] = i0 + tid;
        }
        got += __popc(m);
      }
  }
  __syncthreads();
  return true;
}

// One CTA per row. Lists the k <= SAMPLE_K largest logits, then softmax / top-p / inverse-CDF draw on the candidates; k off or
// above: the law of the whole row. temperature <= 0 means greedy.
template <typename T, bool STAGED>
__global__ void __launch_bounds__(LAW_T)
sample_kernel(const T* __restrict__ logits, long long ld, int vocab, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p,
              const unsigned long long* __restrict__ seeds, const unsigned long long* __restrict__ offsets,
              const int* __restrict__ bitmask, int mask_words, long long* __restrict__ out,
              float* __restrict__ out_prob, int skip_greedy) {
  grid_dep_wait(logits, temperature, top_k, top_p, seeds, offsets, bitmask);
  grid_dep_launch();
  __shared__ float cv[SAMPLE_K];
  __shared__ int ci[SAMPLE_K];
  __shared__ float wv[LAW_WARPS];
  __shared__ int wi[LAW_WARPS];
  __shared__ float s_prev_v;
  __shared__ int s_prev_i;
  __shared__ SearchScratch sc;
  const int row = blockIdx.x;
  const T* lr = logits + row * ld;
  const int* mask = bitmask ? bitmask + static_cast<long long>(row) * mask_words : nullptr;
  const float temp = temperature ? temperature[row] : 0.f;
  if (skip_greedy && temp <= 0.f) return;   // the two-stage argmax owns greedy rows
  int k = top_k ? top_k[row] : 0;
  if (temp > 0.f && (k <= 0 || k > SAMPLE_K)) {
    // top-k off (the API default) or wider than the candidate list: the law is the softmax over the whole
    // vocabulary (then top-p), not over the SAMPLE_K largest logits
    law_row<T, STAGED>(lr, vocab, mask, temp, k > SAMPLE_K ? k : 0, top_p ? top_p[row] : 1.f,
                       uniform01(seeds ? seeds[row] : 0ull, offsets ? offsets[row] : 0ull), -1, -1, out + row,
                       out_prob ? out_prob + row : nullptr, nullptr, sc);
    return;
  }
  if (temp <= 0.f) k = 1;
  // From four candidates on by the key of the k-th one (a search and a list against k passes over the row; 50 of
  // 18992 169 -> 30 us, of 151936 1772 -> 133). Fewer live tokens than candidates: the passes.
  const bool listed = k > 3 && list_candidates<T, STAGED>(lr, vocab, mask, k, temp, cv, ci, sc);
  if (threadIdx.x == 0) {
    s_prev_v = INFINITY;
    s_prev_i = -1;
  }
  __syncthreads();
  // Selection by successive maxima in (value desc, index asc) order: exact and deterministic.
  for (int c = listed ? k : 0; c < k; ++c) {
    const float pv = s_prev_v;
    const int pi = s_prev_i;
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
      if (!mask_ok(mask, i)) continue;
      const float v = ldf<T>(lr, i);
      const bool after_prev = v < pv || (v == pv && i > pi);
      if (after_prev && (v > best || (v == best && i < bi))) {
        best = v;
        bi = i;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) {
        best = ov;
        bi = oi;
      }
    }
    if ((threadIdx.x & 31) == 0) {
      wv[threadIdx.x >> 5] = best;
      wi[threadIdx.x >> 5] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < LAW_WARPS; ++w)
        if (wv[w] > best || (wv[w] == best && wi[w] < bi)) {
          best = wv[w];
          bi = wi[w];
        }
      cv[c] = best;
      ci[c] = bi == 0x7fffffff ? 0 : bi;
      s_prev_v = best;
      s_prev_i = bi;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    if (k == 1) {
      out[row] = ci[0];
      if (out_prob) out_prob[row] = 1.f;
      return;
    }
    const float inv_t = 1.f / temp;
    const float m = cv[0];
    float sum = 0.f;
    for (int c = 0; c < k; ++c) {
      cv[c] = (cv[c] == -INFINITY) ? 0.f : __expf((cv[c] - m) * inv_t);
      sum += cv[c];
    }
    const float p_lim = top_p ? top_p[row] : 1.f;
    int keep = k;
    if (p_lim < 1.f) {
      float acc = 0.f;
      for (int c = 0; c < k; ++c) {
        acc += cv[c] / sum;
        if (acc >= p_lim) {
          keep = c + 1;
          break;
        }
      }
    }
    float ksum = 0.f;
    for (int c = 0; c < keep; ++c) ksum += cv[c];
    const float u = uniform01(seeds ? seeds[row] : 0ull, offsets ? offsets[row] : 0ull) * ksum;
    float acc = 0.f;
    int pick = keep - 1;
    for (int c = 0; c < keep; ++c) {
      acc += cv[c];
      if (u < acc) {
        pick = c;
        break;
      }
    }
    out[row] = ci[pick];
    if (out_prob) out_prob[row] = cv[pick] / ksum;
  }
}

// Walk of a block drafter's candidate lattice, one warp per request, lane = candidate (width <= 32). Step j scores
// candidate w as scores[b][j][previous choice][w]; the greedy walk takes the best (lowest index on ties), the
// sampled walk draws from softmax(row / T) by inverse CDF with the caller's uniform. Writes the chosen tokens and
// candidate indices, the probability of every candidate at every step (the draft law on its support, what
// speculative sampling divides by) and the unit-temperature probability of the chosen one (acceptance estimate).
__global__ void lattice_walk_kernel(const long long* __restrict__ cand, const float* __restrict__ scores,
                                    const float* __restrict__ temperature, const float* __restrict__ uniforms,
                                    int batch, int k, int width, long long* __restrict__ tokens,
                                    int* __restrict__ chosen, float* __restrict__ probs, float* __restrict__ estimate) {
  const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (b >= batch) return;
  const float temp = temperature ? temperature[b] : 0.f;
  const bool sampled = temp > 0.f && uniforms != nullptr;
  int prev = 0;
  for (int j = 0; j < k; ++j) {
    const long long base = (static_cast<long long>(b) * k + j) * width;
    const float x = lane < width ? scores[(base + prev) * width + lane] : -INFINITY;
    const float mx = warp_max(x);
    const float e1 = lane < width ? __expf(x - mx) : 0.f;              // unit temperature: the estimate
    const float z1 = warp_sum(e1);
    float p = e1 / z1;
    int pick;
    if (sampled) {
      const float et = lane < width ? __expf((x - mx) / temp) : 0.f;
      p = et / warp_sum(et);
      float cdf = p;                                                   // inclusive scan over the lanes
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, cdf, o);
        if (lane >= o) cdf += up;
      }
      const unsigned below = __ballot_sync(0xffffffffu, lane < width && cdf < uniforms[static_cast<long long>(b) * k + j]);
      pick = min(__popc(below), width - 1);
    } else {
      const unsigned best = __ballot_sync(0xffffffffu, lane < width && x == mx);
      pick = __ffs(best) - 1;
    }
    if (probs != nullptr && lane < width) probs[base + lane] = p;
    const float p1 = __shfl_sync(0xffffffffu, e1 / z1, pick);
    if (lane == 0) {
      tokens[static_cast<long long>(b) * k + j] = cand[base + pick];
      chosen[static_cast<long long>(b) * k + j] = pick;
      if (estimate != nullptr) estimate[static_cast<long long>(b) * k + j] = p1;
    }
    prev = pick;
  }
}

// Speculative rejection sampling against point-mass drafts, one CTA per verified row. Request b owns logits rows
// [b * (k + 1), (b + 1) * (k + 1)); row j < k sees draft d = drafts[b][j]: with p the row's law (law_row) the draft
// stands when u * 1 < p[d] (or, for a relaxed request, u < e^soft * p[d]); otherwise the row's token is a draw from
// max(p - onehot(d), 0) renormalised. Row k draws the bonus token from p. The kernel writes, per row, the token the
// target "says" there: d where the draft stands, the draw where it does not; the exact-prefix accept kernel below
// then yields the emitted tokens, so sampled and greedy rounds share one accept path (greedy requests, temp <= 0,
// fall out of the same rule: their law is the one-hot argmax). Uniforms are counter draws at (seed, 2 * (draws + j)
// + 1) for the test and + 2 for the draw.
template <typename T, bool STAGED>
__global__ void __launch_bounds__(LAW_T)
spec_targets_kernel(const T* __restrict__ logits, long long ld, int vocab, int k, const long long* __restrict__ drafts,
                    const float* __restrict__ temperature, const int* __restrict__ top_k,
                    const float* __restrict__ top_p, const unsigned long long* __restrict__ seeds,
                    const unsigned long long* __restrict__ draws, const float* __restrict__ soft,
                    const int* __restrict__ bitmask, int mask_words, const long long* __restrict__ greedy_pick,
                    long long* __restrict__ target, float* __restrict__ p_draft) {
  __shared__ long long s_tok;
  __shared__ float s_probe;
  __shared__ SearchScratch sc;
  const int row = blockIdx.x, b = row / (k + 1), j = row - b * (k + 1);
  const T* lr = logits + row * ld;
  const int* mask = bitmask ? bitmask + static_cast<long long>(row) * mask_words : nullptr;
  float temp = temperature ? temperature[b] : 0.f;
  int k_lim = top_k ? top_k[b] : 0;
  float p_lim = top_p ? top_p[b] : 1.f;
  if (temp <= 0.f && greedy_pick != nullptr) {      // the caller already has this row's argmax
    if (threadIdx.x == 0) {
      target[row] = greedy_pick[row];
      if (p_draft) p_draft[row] = j < k && greedy_pick[row] == drafts[static_cast<long long>(b) * k + j] ? 1.f : 0.f;
    }
    return;
  }
  if (temp <= 0.f) {
    temp = 1.f;
    k_lim = 1;
    p_lim = 1.f;
  }
  const unsigned long long seed = seeds ? seeds[b] : 0ull, base = draws ? draws[b] : 0ull;
  const int d = j < k ? static_cast<int>(drafts[static_cast<long long>(b) * k + j]) : -1;
  law_row<T, STAGED>(lr, vocab, mask, temp, k_lim, p_lim, uniform01(seed, 2 * (base + j) + 2), d, d, &s_tok, nullptr,
                     &s_probe, sc);
  if (threadIdx.x == 0) {
    long long tok = s_tok;
    if (j < k) {
      const float u = uniform01(seed, 2 * (base + j) + 1), pd = s_probe;
      const float sf = soft ? soft[b] : 0.f;
      if (u < pd || (sf > 0.f && u < __expf(sf) * pd)) tok = d;
      if (p_draft) p_draft[row] = pd;
    } else if (p_draft) {
      p_draft[row] = 1.f;
    }
    target[row] = tok;
  }
}

// Exact greedy acceptance. Row layout: request b owns rows [b*(k+1), (b+1)*(k+1)); row j holds the target's
// argmax after consuming [pending, draft_1..draft_j]. Accept drafts while draft[j] == target[j-1]; emit the
// accepted drafts plus the target token of the first mismatch (or the bonus token). Emission stops at a stop id
// (inclusive) or when `budget[b]` tokens are out. Writes emitted[b, 0..count) and count[b].
__global__ void accept_greedy_kernel(const long long* __restrict__ target, const long long* __restrict__ drafts,
                                     const long long* __restrict__ stop_ids, int n_stop,
                                     const int* __restrict__ budget, const int* __restrict__ depth, int k_max, int batch,
                                     long long* __restrict__ emitted, int* __restrict__ count,
                                     int* __restrict__ accepted) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  const int k = depth ? min(depth[b], k_max) : k_max;
  const long long* t = target + static_cast<long long>(b) * (k_max + 1);
  const long long* d = drafts + static_cast<long long>(b) * k_max;
  long long* e = emitted + static_cast<long long>(b) * (k_max + 1);
  const int lim = budget ? budget[b] : k + 1;
  int n = 0, acc = 0;
  bool stopped = false;
  for (int j = 0; j <= k && n < lim && !stopped; ++j) {
    const long long tok = t[j];
    e[n++] = tok;
    for (int s = 0; s < n_stop; ++s)
      if (stop_ids[static_cast<long long>(b) * n_stop + s] == tok) stopped = true;
    if (j < k && d[j] == tok) ++acc;
    else break;
  }
  count[b] = n;
  if (accepted) accepted[b] = acc;
}

// Rank (number of strictly larger logits) and gap to the row maximum of token ids[row].
template <typename T>
__global__ void __launch_bounds__(256)
rank_gap_kernel(const T* __restrict__ logits, long long ld, int vocab, const long long* __restrict__ ids,
                int* __restrict__ rank, float* __restrict__ gap) {
  __shared__ float smax[8];
  __shared__ int scnt[8];
  const int row = blockIdx.x;
  const T* lr = logits + row * ld;
  const float mine = ldf<T>(lr, ids[row]);
  float mx = -INFINITY;
  int cnt = 0;
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
    const float v = ldf<T>(lr, i);
    mx = fmaxf(mx, v);
    cnt += v > mine;
  }
  mx = warp_max(mx);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  if ((threadIdx.x & 31) == 0) {
    smax[threadIdx.x >> 5] = mx;
    scnt[threadIdx.x >> 5] = cnt;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      mx = fmaxf(mx, smax[w]);
      cnt += scnt[w];
    }
    rank[row] = cnt;
    gap[row] = mx - mine;
  }
}

// Rows of up to 52224 tokens (204 KB of keys beside 20 KB of scratch) are staged.
inline size_t staged_bytes(int vocab) { return vocab <= 52224 ? static_cast<size_t>(vocab) * sizeof(unsigned) : 0; }
template <typename K>
bool row_kernel(K kern, size_t smem) {
  return smem <= 32 * 1024 ||
         cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) == cudaSuccess;
}

}  // namespace
}  // namespace hb

using namespace hb;

extern "C" {

int hb_argmax(const void* logits, long long ld, int rows, int vocab, int is_f32, const void* bitmask, int mask_words,
              void* out, void* out_val, void* stream) {
  if (rows <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (is_f32)
    launch_dep(argmax_kernel<float>, dim3(rows), dim3(256), 0, st, static_cast<const float*>(logits), ld, vocab,
               static_cast<const int*>(bitmask), mask_words,
               static_cast<long long*>(out), static_cast<float*>(out_val));
  else
    launch_dep(argmax_kernel<__nv_bfloat16>, dim3(rows), dim3(256), 0, st, static_cast<const __nv_bfloat16*>(logits), ld, vocab,
               static_cast<const int*>(bitmask), mask_words,
               static_cast<long long*>(out), static_cast<float*>(out_val));
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int hb_sample(const void* logits, long long ld, int rows, int vocab, int is_f32, const void* temperature,
              const void* top_k, const void* top_p, const void* seeds, const void* offsets, const void* bitmask,
              int mask_words, void* out, void* out_prob, int skip_greedy, void* stream) {
  if (rows <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
#define HB_SAMPLE_ARGS                                                                                     \
  ld, vocab, static_cast<const float*>(temperature), static_cast<const int*>(top_k),                       \
      static_cast<const float*>(top_p), static_cast<const unsigned long long*>(seeds),                     \
      static_cast<const unsigned long long*>(offsets), static_cast<const int*>(bitmask), mask_words,       \
      static_cast<long long*>(out), static_cast<float*>(out_prob), skip_greedy
  const size_t smem = staged_bytes(vocab);
  auto go = [&](auto kern, auto* p) {
    return row_kernel(kern, smem) &&
           launch_dep(kern, dim3(rows), dim3(LAW_T), smem, st, p, HB_SAMPLE_ARGS) == cudaSuccess;
  };
  const float* lf = static_cast<const float*>(logits);
  const __nv_bfloat16* lb = static_cast<const __nv_bfloat16*>(logits);
  const bool ok = smem ? (is_f32 ? go(sample_kernel<float, true>, lf) : go(sample_kernel<__nv_bfloat16, true>, lb))
                       : (is_f32 ? go(sample_kernel<float, false>, lf) : go(sample_kernel<__nv_bfloat16, false>, lb));
#undef HB_SAMPLE_ARGS
  return cudaGetLastError() == cudaSuccess && ok ? 0 : 2;
}

int hb_lattice_walk(const void* cand, const void* scores, const void* temperature, const void* uniforms, int batch,
                    int k, int width, void* tokens, void* chosen, void* probs, void* estimate, void* stream) {
  if (batch <= 0 || k <= 0) return 0;
  if (width < 1 || width > 32) return 1;
  lattice_walk_kernel<<<(batch + 3) / 4, 128, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const long long*>(cand), static_cast<const float*>(scores), static_cast<const float*>(temperature),
      static_cast<const float*>(uniforms), batch, k, width, static_cast<long long*>(tokens),
      static_cast<int*>(chosen), static_cast<float*>(probs), static_cast<float*>(estimate));
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int hb_spec_targets(const void* logits, long long ld, int batch, int k, int vocab, int is_f32, const void* drafts,
                    const void* temperature, const void* top_k, const void* top_p, const void* seeds,
                    const void* draws, const void* soft, const void* bitmask, int mask_words,
                    const void* greedy_pick, void* target, void* p_draft, void* stream) {
  if (batch <= 0) return 0;
  if (k < 0 || vocab <= 0) return 1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int rows = batch * (k + 1);
#define HB_SPEC_ARGS                                                                                          \
  ld, vocab, k, static_cast<const long long*>(drafts), static_cast<const float*>(temperature),                \
      static_cast<const int*>(top_k), static_cast<const float*>(top_p),                                       \
      static_cast<const unsigned long long*>(seeds), static_cast<const unsigned long long*>(draws),           \
      static_cast<const float*>(soft), static_cast<const int*>(bitmask), mask_words,                          \
      static_cast<const long long*>(greedy_pick), static_cast<long long*>(target), static_cast<float*>(p_draft)
  const size_t smem = staged_bytes(vocab);
  auto go = [&](auto kern, auto* p) {
    if (!row_kernel(kern, smem)) return false;
    kern<<<rows, LAW_T, smem, st>>>(p, HB_SPEC_ARGS);
    return true;
  };
  const float* lf = static_cast<const float*>(logits);
  const __nv_bfloat16* lb = static_cast<const __nv_bfloat16*>(logits);
  const bool ok = smem ? (is_f32 ? go(spec_targets_kernel<float, true>, lf) : go(spec_targets_kernel<__nv_bfloat16, true>, lb))
                       : (is_f32 ? go(spec_targets_kernel<float, false>, lf) : go(spec_targets_kernel<__nv_bfloat16, false>, lb));
#undef HB_SPEC_ARGS
  return cudaGetLastError() == cudaSuccess && ok ? 0 : 2;
}

int hb_accept_greedy(const void* target, const void* drafts, const void* stop_ids, int n_stop, const void* budget,
                     const void* depth, int k_max, int batch, void* emitted, void* count, void* accepted,
                     void* stream) {
  if (batch <= 0) return 0;
  accept_greedy_kernel<<<(batch + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const long long*>(target), static_cast<const long long*>(drafts),
      static_cast<const long long*>(stop_ids), n_stop, static_cast<const int*>(budget),
      static_cast<const int*>(depth), k_max, batch, static_cast<long long*>(emitted), static_cast<int*>(count),
      static_cast<int*>(accepted));
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int hb_rank_gap(const void* logits, long long ld, int rows, int vocab, int is_f32, const void* ids, void* rank,
                void* gap, void* stream) {
  if (rows <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (is_f32)
    rank_gap_kernel<float><<<rows, 256, 0, st>>>(static_cast<const float*>(logits), ld, vocab,
                                                 static_cast<const long long*>(ids), static_cast<int*>(rank),
                                                 static_cast<float*>(gap));
  else
    rank_gap_kernel<__nv_bfloat16><<<rows, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(logits), ld, vocab,
                                                         static_cast<const long long*>(ids),
                                                         static_cast<int*>(rank), static_cast<float*>(gap));
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

// Two-stage greedy argmax. scratch_v / scratch_i hold rows * nch partials. With `temperature` given, rows whose
// temperature is > 0 are skipped (their token comes from hb_sample with skip_greedy).
int hb_argmax2(const void* logits, long long ld, int rows, int vocab, int is_f32, const void* bitmask, int mask_words,
               int nch, void* scratch_v, void* scratch_i, const void* temperature, void* out, void* out_val,
               void* stream) {
  if (rows <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const dim3 grid(rows, nch);
  if (is_f32)
    launch_dep(argmax_partial_kernel<float>, grid, dim3(256), 0, st, static_cast<const float*>(logits), ld, vocab,
               static_cast<const int*>(bitmask), mask_words, nch,
               static_cast<float*>(scratch_v), static_cast<int*>(scratch_i));
  else
    launch_dep(argmax_partial_kernel<__nv_bfloat16>, grid, dim3(256), 0, st,
               static_cast<const __nv_bfloat16*>(logits), ld, vocab, static_cast<const int*>(bitmask), mask_words, nch,
               static_cast<float*>(scratch_v), static_cast<int*>(scratch_i));
  launch_dep(argmax_final_kernel, dim3((rows + 3) / 4), dim3(128), 0, st, static_cast<const float*>(scratch_v),
             static_cast<const int*>(scratch_i), nch, rows,
             static_cast<const float*>(temperature),
             static_cast<long long*>(out), static_cast<float*>(out_val));
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // extern "C"
