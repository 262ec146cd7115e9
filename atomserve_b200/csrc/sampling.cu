// Sampling on the device: a cluster of up to eight blocks per row of float32 logits [B, V].
//
// The rules are the reference sampler's (atomserve/sampler.py:82-129): top-k on the raw
// logits (0 or >= V keeps all; temperature 0 is the single best), divide by the temperature,
// softmax over the kept, top-p drops a token once the probability mass ranked above it has
// reached top_p (the best always stays), then an exponential race: argmax of p_i / E_i with
// E_i ~ Exp(1) picks token i with probability p_i / sum(p). The presence penalty is a
// separate scatter that runs first (atomserve/sampler.py:144-168).
//
// The reference sorts (torch.topk, or its 1024-thread Metal kernel, atomserve/kernels.py:336-435).
// Here a whole row is never sorted: the k-th largest logit is found by a radix select on order-preserving
// integer keys (digits of 11, 11 and 10 bits, counting histograms in shared memory), and the top-p cut
// by the same walk over histograms of probability mass, kept as 64-bit fixed point so that
// the sums do not depend on the order of the atomic additions. Ties at a cut are broken towards
// the lower token id, by a further select over the ids. When top-k leaves at most 1024
// candidates they are gathered into one block's shared memory and ranked there.
//
// The walk over masses begins with equal steps below the largest logit instead of a digit of the key (`step_key`): a key's
// leading digit is its exponent and two bits, so that half a row falls into some sixteen bins and its atomics wait for
// one another, while 2,048 equal steps spread it; and what shares the deciding step is so few (a row of 151,936 has under
// 200 to a step) that it is gathered and ranked in place of two more passes. Rows with a NaN or an infinity on top, and
// those with more in one step than the buffer holds, take the digits. 48 rows of 151,936 normal logits, top-p 0.95 alone, us:
// deviation 3 at temperature 0.6 and 0.8 86 -> 64 and 107 -> 80, deviation 1 at 1 132 -> 106, after a top-k of 2,000
// 140 -> 112; all logits within 0.01 of each other 131 -> 102. Slower: where hundreds of logits are equal at the cut the
// histogram of steps is one pass more (deviation 1 in whole quarters: 202 -> 228; digits within the deciding step alone
// took 240), and rows that end in a top-k of 20 by 2 % (40.1 -> 41.0; without their smallest logit 40.7, and the others slower).
//
// What bounds it: a row of 151,936 logits is 600 KB, and with one block a row every one of
// seven passes over it moved at the rate of one SM. Here each block of the cluster brings its share of the row
// into shared memory once (76 KB, two blocks an SM) and all passes read it there; what is left is the
// chain of passes with two cluster barriers each. Measured, 1 / 48 rows of 151,936: temperature 0.6, top-k 20, top-p
// 0.95 122 / 124 -> 17 / 41 us; top-p 0.95 alone at 0.6 371 / 480 -> 24 / 64 us (the steps included); argmax 8.8 / 8.8 -> 3.8 / 6.5 us. An eighth and not a quarter, because rows in flight on the
// device are the same (74 KB x 2 against 148 KB x 1 an SM) while a pass takes half as long.
//
// Random numbers are Philox-4x32-10 keyed by the row's seed; the counter is (token id, the
// row's draw counter). A seeded request passes its own seed and counts its own draws, so what
// it draws does not depend on its neighbours in the batch (atomserve/sampler.py:123-127).
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kMostBlocks = 8;                   // blocks a row: 8, 4, 2 or 1 (the kernels' C)
constexpr int kBins = 2048;                      // an 11-bit digit
constexpr int kSegment = 256;                    // bins that are searched together
constexpr int kSegments = kBins / kSegment;      // a block of C forms the totals of kSegments / C of them
constexpr int kCompact = 1024;
constexpr int kSplitSlice = 65535;               // most elements whose masses two 32-bit words can add up (see Scratch)

__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);  // ascending with the float order
}

struct Philox {
  static __device__ __forceinline__ void round(uint32_t (&c)[4], uint32_t k0, uint32_t k1) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
    const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
    c[0] = n0; c[1] = lo1; c[2] = n2; c[3] = lo0;
  }
  static __device__ __forceinline__ uint32_t draw(uint64_t seed, uint64_t counter, uint32_t index) {
    uint32_t c[4] = {index, (uint32_t)counter, (uint32_t)(counter >> 32), 0x5a17u};
    uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
    for (int i = 0; i < 10; ++i) {
      round(c, k0, k1);
      k0 += 0x9E3779B9u;
      k1 += 0xBB67AE85u;
    }
    return c[0];
  }
};

// A block's share of a row: `n` values from token `first` on, in shared memory where they fit, else in place.
struct Slice {
  const float* val;
  int first, n;
};

struct Best {
  float score;
  int token;
  __device__ __forceinline__ void take(float s, int t) {
    if (s > score || (s == score && t < token)) { score = s; token = t; }
  }
};

template <int C>
struct Scratch {
  static constexpr int kOwn = kSegments / C;
  // A digit's histogram. Counts: word[0]. Masses, at most 2^32 each: the low 16 bits of each are added up in
  // word[0] and the rest in word[1] (both native 32-bit atomics; 64-bit ones in shared memory are loops), which
  // holds for up to kSplitSlice elements; otherwise, and where a mass may be out of that range (a row with an
  // infinity on top or a NaN), 64-bit words.
  union {
    unsigned int word[2][kBins];
    unsigned long long wide[kBins];
    struct {  // the candidates in order, once the selects are over in every block
      uint32_t key[kCompact];
      int id[kCompact];
    } sorted;
  } hist;
  unsigned long long total[kOwn * kSegment];  // over the cluster, of this block's segments of the bins
  unsigned long long segment_sum[kOwn];
  unsigned long long warp_part[kOwn > 2 ? kOwn * kSegment / 32 : kWarps];  // a sum being formed over the block
  int odd;                               // this block's slice holds a NaN
  Best best[2], warp_best[kWarps];  // [0]: the largest logit, [1]: the winner of the race
  float low, warp_low[kWarps];           // the smallest logit
  unsigned long long found[4];
  int cand_n;
  __align__(16) uint32_t cand_key[kCompact];
  __align__(16) int cand_id[kCompact];
};

constexpr int kMaxSmem = 227 * 1024;
// Floats of a row that a block of C can hold in shared memory.
template <int C>
constexpr int kMaxSlice = (kMaxSmem - (int)sizeof(Scratch<C>)) / 16 * 4 < 48 * 1024 ? (kMaxSmem - (int)sizeof(Scratch<C>)) / 16 * 4 : 48 * 1024;

__device__ __forceinline__ float key_value(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}

// Calls f(token, value) for every element of the slice; 16-byte reads, four elements a thread at a time.
template <typename F>
__device__ __forceinline__ void for_each_value(const Slice& row, F f) {
  int done = 0;
  if (((uintptr_t)row.val & 15) == 0) {
    const float4* v4 = reinterpret_cast<const float4*>(row.val);
    const int n4 = row.n >> 2;
#pragma unroll 2
    for (int i = threadIdx.x; i < n4; i += kThreads) {
      const float4 x = v4[i];
      const int t = row.first + 4 * i;
      f(t, x.x);
      f(t + 1, x.y);
      f(t + 2, x.z);
      f(t + 3, x.w);
    }
    done = n4 << 2;
  }
  for (int i = done + threadIdx.x; i < row.n; i += kThreads) f(row.first + i, row.val[i]);
}

// `p` of block `c` of the cluster.
template <int C, typename T>
__device__ __forceinline__ T* peer(T* p, int c) {
  if constexpr (C == 1) return p;
  else return cg::this_cluster().map_shared_rank(p, c);
}
template <int C>
__device__ __forceinline__ void row_sync() {
  if constexpr (C == 1) __syncthreads();
  else cg::this_cluster().sync();
}
template <int C>
__device__ __forceinline__ int row_rank() {
  if constexpr (C == 1) return 0;
  else return (int)cg::this_cluster().block_rank();
}

// The best over the block, then over the cluster: every thread of every block gets it. `slot`: which of the
// scratch's two (each is used once a kernel, so no barrier keeps a second use from a slow reader).
// Likewise the smallest of `low`, where it is given.
template <int C>
__device__ Best cluster_best(Scratch<C>& s, Best b, int slot, float* low = nullptr) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float os = __shfl_xor_sync(0xffffffffu, b.score, o);
    const int ot = __shfl_xor_sync(0xffffffffu, b.token, o);
    b.take(os, ot);
  }
  if (low)
    for (int o = 16; o > 0; o >>= 1) *low = fminf(*low, __shfl_xor_sync(0xffffffffu, *low, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    s.warp_best[threadIdx.x >> 5] = b;
    if (low) s.warp_low[threadIdx.x >> 5] = *low;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kWarps; ++w) b.take(s.warp_best[w].score, s.warp_best[w].token);
    s.best[slot] = b;
  }
  if (low && threadIdx.x == 32) {
    for (int w = 0; w < kWarps; ++w) *low = fminf(*low, s.warp_low[w]);
    s.low = *low;
  }
  row_sync<C>();
  b = s.best[slot];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const Best o = *peer<C>(&s.best[slot], c);
    b.take(o.score, o.token);
    if (low) *low = fminf(*low, *peer<C>(&s.low, c));
  }
  return b;
}

// Descending radix select over 32-bit keys of the cluster's row. `item(token, value, key)` says whether an
// element takes part, and its key; `weight(value)` is its non-negative integer weight, worked out only for elements
// that a digit's histogram counts. `target_of(total)` gives the target once the first histogram has told the total
// weight (which so needs no pass of its own). Finds the largest key c such that the
// weight of all taking-part elements with key > c is < target <= that weight plus the weight
// of key == c. Returns c, and in `above` the weight strictly above c, in `equal` that of key == c. (With weight 1
// and target k this is the k-th largest key.) If the total weight is below target, returns 0 with
// `above` = total: everything is kept.
//
// `digits` 1 or 2 stops after that many: the result then has its low bits clear and names a range of keys,
// `above` and `equal` counting what lies above and inside it.
//
// kUnit: every weight is 1 (a count). `wide`: weights added up in 64-bit words (see Scratch).
template <bool kUnit, int C, typename Item, typename Weight, typename Target>
__device__ uint32_t cluster_select(const Slice& row, Scratch<C>& s, Target target_of,
                                   unsigned long long* above, unsigned long long* equal, bool wide, int digits, Item item,
                                   Weight weight) {
  uint32_t prefix = 0, mask = 0;
  unsigned long long acc = 0, target = 0;
  constexpr int kOwn = Scratch<C>::kOwn;
  const int rank = row_rank<C>(), lane = threadIdx.x & 31;
  for (int digit = 0; digit < digits; ++digit) {
    const int shift = digit == 0 ? 21 : (digit == 1 ? 10 : 0);
    const uint32_t bins = digit == 2 ? 1024u : 2048u;
    for (int i = threadIdx.x; i < kBins; i += kThreads) s.hist.wide[i] = 0ull;
    __syncthreads();
    for_each_value(row, [&](int token, float v) {
      uint32_t key = 0;
      if (!item(token, v, key) || (key & mask) != prefix) return;
      const uint32_t bin = (key >> shift) & (bins - 1u);
      if (kUnit) {
        atomicAdd(&s.hist.word[0][bin], 1u);
        return;
      }
      const unsigned long long w = weight(v);
      if (wide) {
        if (w) atomicAdd(&s.hist.wide[bin], w);
      } else {
        const unsigned int lo = (unsigned int)w & 0xffffu, hi = (unsigned int)(w >> 16);
        if (lo) atomicAdd(&s.hist.word[0][bin], lo);
        if (hi) atomicAdd(&s.hist.word[1][bin], hi);
      }
    });
    row_sync<C>();
    // this block's segments of the bins, over the cluster (a warp's 32 bins lie in one of them)
    for (int i = threadIdx.x; i < kOwn * kSegment; i += kThreads) {
      const int bin = rank * kOwn * kSegment + i;
      unsigned long long t = 0;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const Scratch<C>* o = peer<C>(&s, c);
        if (kUnit) t += o->hist.word[0][bin];
        else if (wide) t += o->hist.wide[bin];
        else t += (unsigned long long)o->hist.word[0][bin] + ((unsigned long long)o->hist.word[1][bin] << 16);
      }
      s.total[i] = t;
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) s.warp_part[i >> 5] = t;
    }
    __syncthreads();
    if (threadIdx.x < kOwn) {
      unsigned long long t = 0;
      for (int w = 0; w < kSegment / 32; ++w) t += s.warp_part[threadIdx.x * (kSegment / 32) + w];
      s.segment_sum[threadIdx.x] = t;
    }
    row_sync<C>();
    if (threadIdx.x < 32) {
      // the segment, from the top, in which the weight so far reaches the target, then the bin within it: lane l
      // walks eight of its bins downwards, after a scan over the lanes has told it the weight above them
      unsigned long long sums[kSegments], a = acc;
#pragma unroll
      for (int c = 0; c < kSegments; ++c) sums[c] = *peer<C>(&s.segment_sum[c % kOwn], c / kOwn);
      if (digit == 0) {
        unsigned long long total = 0;
#pragma unroll
        for (int c = 0; c < kSegments; ++c) total += sums[c];
        target = target_of(total);
        if (lane == 0) s.found[3] = target;
      }
      int segment = -1;
#pragma unroll
      for (int c = kSegments - 1; c >= 0; --c)
        if (segment < 0) {
          if (a + sums[c] >= target) segment = c;
          else a += sums[c];
        }
      if (segment < 0) {  // the whole set weighs less than the target
        if (lane == 0) {
          s.found[0] = a;
          s.found[1] = ~0ull;
          s.found[2] = 0ull;
        }
      } else {
        const unsigned long long* totals = peer<C>(&s.total[segment % kOwn * kSegment], segment / kOwn);
        constexpr int kEach = kSegment / 32;
        unsigned long long mine[kEach], lane_sum = 0;
#pragma unroll
        for (int j = 0; j < kEach; ++j) {
          mine[j] = totals[kSegment - 1 - (kEach * lane + j)];
          lane_sum += mine[j];
        }
        unsigned long long upto = lane_sum;  // inclusive scan over the lanes
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned long long t = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= o) upto += t;
        }
        a += upto - lane_sum;
        int at = -1;
        unsigned long long in_bin = 0;
#pragma unroll
        for (int j = 0; j < kEach; ++j)
          if (at < 0) {
            if (a + mine[j] >= target) { at = j; in_bin = mine[j]; }
            else a += mine[j];
          }
        const unsigned hit = __ballot_sync(0xffffffffu, at >= 0);
        if (hit != 0u && lane == __ffs(hit) - 1) {
          s.found[0] = a;
          s.found[1] = (unsigned long long)(segment * kSegment + kSegment - 1 - (kEach * lane + at));
          s.found[2] = in_bin;
        }
      }
    }
    __syncthreads();
    acc = s.found[0];
    *equal = s.found[2];
    target = s.found[3];
    const unsigned long long bin = s.found[1];
    __syncthreads();
    if (bin == ~0ull) {  // the whole set weighs less than target
      *above = acc;
      return 0u;
    }
    prefix |= (uint32_t)bin << shift;
    mask |= (bins - 1u) << shift;
  }
  *above = acc;
  return prefix;
}

// A count as the target, whatever the total.
struct Count {
  unsigned long long n;
  __device__ __forceinline__ unsigned long long operator()(unsigned long long) const { return n; }
};
struct One {
  __device__ __forceinline__ unsigned long long operator()(float) const { return 1ull; }
};

// The cut of one stage: keep key > cut_key, and of key == cut_key the tokens with id <= cut_id.
struct Cut {
  uint32_t key;
  int id;
  __device__ __forceinline__ bool keeps(uint32_t k, int token) const {
    return k > key || (k == key && token <= id);
  }
};

// After a select that found `key` with `need` more units wanted among the ties: the id below
// which ties are kept. Unit weights (top-k) keep exactly `need` ties.
template <int C, typename Item>
__device__ Cut cut_with_ties(const Slice& row, Scratch<C>& s, uint32_t key, unsigned long long need,
                             unsigned long long equal, unsigned long long unit, Item item) {
  Cut cut{key, 0x7fffffff};
  if (key == 0u || unit == 0ull) return cut;
  // how many ties are wanted: the smallest t with t * unit >= need
  const unsigned long long want = (need + unit - 1) / unit;
  if (want * unit >= equal) return cut;  // all of them: no pass over the ids
  unsigned long long dummy, dummy2;
  const uint32_t idk = cluster_select<true>(row, s, Count{want}, &dummy, &dummy2, false, 3,
                                            [&](int token, float v, uint32_t& k2) {
    uint32_t k;
    if (!item(token, v, k) || k != key) return false;
    k2 = ~(uint32_t)token;  // descending on ~id is ascending on id
    return true;
  }, One{});
  if (idk != 0u) cut.id = (int)~idk;
  return cut;
}

// Probability mass of one token as 64-bit fixed point: exp((v - max) / T) * 2^32 (a scaling by a power of two is
// exact in float32 too).
__device__ __forceinline__ unsigned long long mass_of(float v, float vmax, float inv_t) {
  return __float2ull_rz(expf((v - vmax) * inv_t) * 4294967296.f);  // the exponential is in [0, 1]
}

// What a kept token scores in the exponential race.
__device__ __forceinline__ float race_score(float v, float vmax, float inv_t, uint64_t seed, uint64_t counter, int token) {
  const float w = expf((v - vmax) * inv_t);
  const uint32_t bits = Philox::draw(seed, counter, (uint32_t)token);
  const float u = ((float)(bits >> 8) + 0.5f) * (1.f / 16777216.f);  // (0, 1)
  const float e = fmaxf(-logf(u), 1e-10f);
  return w / e;
}

// top-p's target: the mass at which the walk from the largest key down stops (the best token always stays).
__device__ __forceinline__ unsigned long long mass_target(float p, unsigned long long total) {
  unsigned long long target = (unsigned long long)ceil((double)p * (double)total);
  if (target < 1ull) target = 1ull;
  return target > total ? total : target;
}

// The step below the largest logit, out of kBins of 1 / per_step each, in which v lies, as a key whose first digit it is,
// the highest on top (finite vmax, v not a NaN). Falls with v: it selects as v's own key does, but for ties within a step.
__device__ __forceinline__ uint32_t step_key(float v, float vmax, float per_step) {
  const float step = fminf((vmax - v) * per_step, (float)(kBins - 1));
  return (uint32_t)(kBins - 1 - (int)step) << 21;
}

// Orders the block's n candidates (at most kCompact) by descending key, then ascending id: each is ranked by counting
// those before it.
template <int C>
__device__ void rank_candidates(Scratch<C>& s, int n) {
  for (int i = threadIdx.x; i < n; i += kThreads) {
    const uint32_t key = s.cand_key[i];
    const int id = s.cand_id[i];
    int before = 0, j = 0;
    for (; j + 4 <= n; j += 4) {
      const uint4 kk = *reinterpret_cast<const uint4*>(&s.cand_key[j]);
      const int4 ii = *reinterpret_cast<const int4*>(&s.cand_id[j]);
      before += (kk.x > key || (kk.x == key && ii.x < id)) + (kk.y > key || (kk.y == key && ii.y < id)) +
                (kk.z > key || (kk.z == key && ii.z < id)) + (kk.w > key || (kk.w == key && ii.w < id));
    }
    for (; j < n; ++j) before += s.cand_key[j] > key || (s.cand_key[j] == key && s.cand_id[j] < id);
    s.hist.sorted.key[before] = key;
    s.hist.sorted.id[before] = id;
  }
  __syncthreads();
}

// The masses of two neighbouring places of the ordered candidates, this thread's, and what lies before them; `keep` places
// count. Returns the mass of all.
template <int C>
__device__ unsigned long long candidate_masses(Scratch<C>& s, int keep, float vmax, float inv_t, unsigned long long (&m)[2],
                                               unsigned long long* before) {
  static_assert(kCompact == 2 * kThreads, "two places a thread");
  const int at = 2 * threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  m[0] = m[1] = 0ull;
#pragma unroll
  for (int u = 0; u < 2; ++u)
    if (at + u < keep) {
      const float v = key_value(s.hist.sorted.key[at + u]);
      m[u] = v == v ? mass_of(v, vmax, inv_t) : 0ull;  // a NaN takes a place among the k and has no mass
    }
  unsigned long long upto = m[0] + m[1];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += t;
  }
  if (lane == 31) s.warp_part[warp] = upto;
  __syncthreads();
  unsigned long long total = 0;
  *before = upto - m[0] - m[1];
  for (int w = 0; w < kWarps; ++w) {
    if (w < warp) *before += s.warp_part[w];
    total += s.warp_part[w];
  }
  return total;
}

// top-p's cut, among the candidates of the step that decides it: the one with which the mass, `above` before the first
// of them, reaches `target`.
template <int C>
__device__ void cut_among_candidates(Scratch<C>& s, unsigned long long above, unsigned long long target, float vmax, float inv_t) {
  const int n = s.cand_n;
  rank_candidates(s, n);
  unsigned long long m[2], before;
  candidate_masses(s, n, vmax, inv_t, m, &before);
  before += above;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    if (before < target && before + m[u] >= target) {
      s.found[0] = s.hist.sorted.key[2 * threadIdx.x + u];
      s.found[1] = (unsigned long long)s.hist.sorted.id[2 * threadIdx.x + u];
    }
    before += m[u];
  }
}

// The end of a row whose top-k left candidates (at most kCompact, the k best among them) in this block's scratch:
// each is ranked by counting those before it, the k best fall into their places, masses are added up along
// them, and the kept ones race. A token is kept while the mass before it is below top-p's target: the cut that the
// selects above find, ties (equal keys, equal masses) by ascending id included.
template <int C>
__device__ int finish_candidates(Scratch<C>& s, int k, float p, float vmax, float inv_t, uint64_t seed, uint64_t counter, int best) {
  const int n = min(s.cand_n, kCompact), keep = min(k, n);
  rank_candidates(s, n);
  const int at = 2 * threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long m[2], before;
  const unsigned long long total = candidate_masses(s, keep, vmax, inv_t, m, &before);
  const bool cuts = p < 1.f;
  const unsigned long long target = cuts ? mass_target(p, total) : 0ull;
  Best mine{-1.f, 0x7fffffff};
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    if (at + u < keep && (!cuts || before < target)) {
      const int token = s.hist.sorted.id[at + u];
      mine.take(race_score(key_value(s.hist.sorted.key[at + u]), vmax, inv_t, seed, counter, token), token);
    }
    before += m[u];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float os = __shfl_xor_sync(0xffffffffu, mine.score, o);
    const int ot = __shfl_xor_sync(0xffffffffu, mine.token, o);
    mine.take(os, ot);
  }
  __syncthreads();
  if (lane == 0) s.warp_best[warp] = mine;
  __syncthreads();
  for (int w = 0; w < kWarps; ++w) mine.take(s.warp_best[w].score, s.warp_best[w].token);
  return mine.token == 0x7fffffff ? best : mine.token;
}

// This block's share of the cluster's row, brought into shared memory where it fits, and the best of it.
template <int C>
__device__ Slice take_slice(const float* logits, int V, float* room, int room_floats, Best* best, bool* nan, float* low = nullptr) {
  const int each = ((V + C - 1) / C + 3) & ~3;
  const int first = min(V, row_rank<C>() * each), n = min(each, V - first);
  const float* from = logits + first;
  const bool keep = n <= room_floats;
  *best = Best{-INFINITY, 0x7fffffff};
  if (low) *low = INFINITY;
  *nan = false;  // whether this thread met one
  int done = 0;
  if (((uintptr_t)from & 15) == 0) {
    const float4* v4 = reinterpret_cast<const float4*>(from);
    const int n4 = n >> 2;
    for (int i = threadIdx.x; i < n4; i += 4 * kThreads) {  // four loads in flight
      float4 x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + u * kThreads < n4) x[u] = v4[i + u * kThreads];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = i + u * kThreads;
        if (j >= n4) break;
        if (keep) reinterpret_cast<float4*>(room)[j] = x[u];
        const int t = first + 4 * j;
        *nan |= x[u].x != x[u].x || x[u].y != x[u].y || x[u].z != x[u].z || x[u].w != x[u].w;
        best->take(x[u].x, t);
        best->take(x[u].y, t + 1);
        best->take(x[u].z, t + 2);
        best->take(x[u].w, t + 3);
        if (low) *low = fminf(*low, fminf(fminf(x[u].x, x[u].y), fminf(x[u].z, x[u].w)));
      }
    }
    done = n4 << 2;
  }
  for (int i = done + threadIdx.x; i < n; i += 8 * kThreads) {  // eight loads in flight
    float x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (i + u * kThreads < n) x[u] = from[i + u * kThreads];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = i + u * kThreads;
      if (j >= n) break;
      if (keep) room[j] = x[u];
      *nan |= x[u] != x[u];
      best->take(x[u], first + j);
      if (low) *low = fminf(*low, x[u]);
    }
  }
  __syncthreads();
  return Slice{keep ? room : from, first, n};
}

template <int C>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(kThreads, 2)
sample_rows_kernel(int* __restrict__ out, const float* __restrict__ logits, int V,
                   const float* __restrict__ temperature, const int* __restrict__ top_k,
                   const float* __restrict__ top_p, const unsigned long long* __restrict__ seed,
                   const unsigned long long* __restrict__ counter, int room_floats) {
  asb::pdl_wait();  // the stream's previous kernel has completed (programmatic dependent launch)
  asb::pdl_launch_dependents();
  __shared__ Scratch<C> s;
  extern __shared__ __align__(16) float room[];
  const int b = blockIdx.x / C;
  const bool leads = row_rank<C>() == 0;
  const float temp = temperature[b];

  if (threadIdx.x == 0) s.cand_n = 0;
  Best top;
  bool odd;
  float vmin;
  const Slice row = take_slice<C>(logits + (size_t)b * V, V, room, room_floats, &top, &odd, &vmin);
  s.odd = 0;
  __syncthreads();
  if (odd) s.odd = 1;
  top = cluster_best(s, top, 0, &vmin);
  const float vmax = top.score;
  const int best = top.token == 0x7fffffff ? 0 : top.token;  // a row of NaN or -inf only
  if (!(temp > 0.f)) {  // greedy: the single best, lowest id among equals
    if (leads && threadIdx.x == 0) out[b] = best;
    row_sync<C>();  // nobody leaves while a neighbour may still read its best
    return;
  }
  const float inv_t = 1.f / temp;
  const uint64_t sd = seed[b], ctr = counter[b];
  const float p = top_p[b];
  // masses are added up in 64-bit words where a slice has more elements than two 32-bit words can hold, or where a
  // mass may lie outside [0, 2^32]
  bool wide = V > C * (kSplitSlice - 3) || isinf(vmax);
#pragma unroll
  for (int c = 0; c < C; ++c) wide |= *peer<C>(&s.odd, c) != 0;

  // top-k
  const int k = top_k[b];
  Cut kcut{0u, 0x7fffffff};
  if (k > 0 && k < V) {
    auto any = [&](int token, float v, uint32_t& key) {
      key = order_key(v);
      return true;
    };
    const Count kth{(unsigned long long)k};
    unsigned long long above, equal;
    uint32_t from = 0u;  // candidates: keys from here on
    bool few = false;
    if (k <= kCompact) {
      // The high digits of the k-th largest key: if everything from that range of keys upwards fits the
      // candidate buffer (it holds at least k), the ranking of the candidates finishes the selection.
      // Only keys within four eighths of the exponent range's steps below the largest (a factor of 16 or so below
      // the best logit when it is positive) are counted here, which spares the atomics of nearly the whole
      // row; if fewer than k lie there, the result is 0 and the full selection below runs.
      const uint32_t top_bin = order_key(vmax) >> 24;
      const uint32_t floor_key = top_bin >= 3u ? (top_bin - 3u) << 24 : 0u;
      for (int digits = 1; digits <= 2 && !few; ++digits) {
        from = cluster_select<true>(row, s, kth, &above, &equal, false, digits, [&](int token, float v, uint32_t& key) {
          key = order_key(v);
          return key >= floor_key;
        }, One{});
        if (from == 0u) break;
        few = above + equal <= (unsigned long long)kCompact;
      }
    }
    if (!few) {
      const uint32_t key = cluster_select<true>(row, s, kth, &above, &equal, false, 3, any, One{});
      kcut = cut_with_ties(row, s, key, (unsigned long long)k - above, equal, 1ull, any);
    }
    if (k <= kCompact) {
      // to the first block, which ends the row alone (the order they arrive in does not matter)
      Scratch<C>* lead = peer<C>(&s, 0);
      for_each_value(row, [&](int token, float v) {
        const uint32_t key = order_key(v);
        if (few ? key >= from : kcut.keeps(key, token)) {
          const int at = atomicAdd(&lead->cand_n, 1);
          if (at < kCompact) { lead->cand_key[at] = key; lead->cand_id[at] = token; }
        }
      });
      row_sync<C>();
      if (!leads) return;  // (and the first block reads nothing of its neighbours from here on)
      const int token = finish_candidates(s, k, p, vmax, inv_t, sd, ctr, best);
      if (threadIdx.x == 0) out[b] = token;
      return;
    }
  }

  // the top-p cut
  Cut pcut{0u, 0x7fffffff};
  if (p < 1.f) {
    auto kept = [&](int token, float v, uint32_t& key) {
      key = order_key(v);
      return kcut.keeps(key, token);
    };
    auto mass = [&](float v) { return mass_of(v, vmax, inv_t); };
    auto reach = [&](unsigned long long total) { return mass_target(p, total); };
    // keep a token while the mass ranked above it is < p * total: find the first key whose
    // cumulative mass (itself included) exceeds p * total, ties by ascending id
    unsigned long long above, equal;
    bool found = false;
    if (!wide && inv_t < 1e30f && temp < 1e30f) {
      // steps down to the smallest logit, or to where a mass is 0: exp(-23) * 2^32 is below 1
      const float per_step = (float)(kBins - 1) / fmaxf(fminf(23.f * temp, vmax - vmin), 1e-30f);
      const uint32_t at = cluster_select<false>(row, s, reach, &above, &equal, false, 1, [&](int token, float v, uint32_t& key) {
        key = step_key(v, vmax, per_step);
        return kcut.keeps(order_key(v), token);
      }, mass);
      // (how many share the step, by its mass and the largest that one of them can have)
      const float most = expf(-(float)(kBins - 1 - (int)(at >> 21)) / per_step * inv_t) * 4294967296.f;
      found = (float)equal <= (float)kCompact * fmaxf(most, 1.f);
      const unsigned long long target = s.found[3];
      Scratch<C>* lead = peer<C>(&s, 0);
      if (found) {
        for_each_value(row, [&](int token, float v) {
          const uint32_t key = order_key(v);
          if (step_key(v, vmax, per_step) != at || !kcut.keeps(key, token)) return;
          const int place = atomicAdd(&lead->cand_n, 1);
          if (place < kCompact) { lead->cand_key[place] = key; lead->cand_id[place] = token; }
        });
        row_sync<C>();
        found = lead->cand_n <= kCompact;
        if (found) {
          if (leads) cut_among_candidates(s, above, target, vmax, inv_t);
          row_sync<C>();
          pcut = Cut{(uint32_t)lead->found[0], (int)lead->found[1]};
        }
        row_sync<C>();  // (all have read the first block's words before anything writes them again)
      }
    }
    if (!found) {
      const uint32_t key = cluster_select<false>(row, s, reach, &above, &equal, wide, 3, kept, mass);
      const unsigned long long target = s.found[3];
      // mass of one tied token (all ties share the key, hence the value)
      pcut = cut_with_ties(row, s, key, target - above, equal, mass_of(key_value(key), vmax, inv_t), kept);
    }
  }

  // exponential race among the kept
  Best winner{-1.f, 0x7fffffff};
  for_each_value(row, [&](int token, float v) {
    const uint32_t key = order_key(v);
    if (!kcut.keeps(key, token) || !pcut.keeps(key, token)) return;
    winner.take(race_score(v, vmax, inv_t, sd, ctr, token), token);
  });
  winner = cluster_best(s, winner, 1);
  if (leads && threadIdx.x == 0) out[b] = winner.token == 0x7fffffff ? best : winner.token;
  row_sync<C>();  // nobody leaves while a neighbour may still read its best
}

template <int C>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(kThreads, 2)
argmax_rows_kernel(int* __restrict__ out, const float* __restrict__ logits, int V) {
  asb::pdl_wait();  // the stream's previous kernel has completed (programmatic dependent launch)
  asb::pdl_launch_dependents();
  __shared__ Best slots[1 + kWarps];  // this block's best, and its warps'
  const int b = blockIdx.x / C;
  Best top;
  bool nan;
  take_slice<C>(logits + (size_t)b * V, V, nullptr, -1, &top, &nan);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float os = __shfl_xor_sync(0xffffffffu, top.score, o);
    const int ot = __shfl_xor_sync(0xffffffffu, top.token, o);
    top.take(os, ot);
  }
  if ((threadIdx.x & 31) == 0) slots[1 + (threadIdx.x >> 5)] = top;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kWarps; ++w) top.take(slots[1 + w].score, slots[1 + w].token);
    slots[0] = top;
  }
  row_sync<C>();
  if (row_rank<C>() == 0 && threadIdx.x == 0) {
    for (int c = 1; c < C; ++c) {
      const Best o = *peer<C>(&slots[0], c);
      top.take(o.score, o.token);
    }
    out[b] = top.token == 0x7fffffff ? 0 : top.token;  // a row of NaN or -inf only
  }
  row_sync<C>();  // nobody leaves while the first block reads its best
}

__global__ void presence_penalty_kernel(float* __restrict__ logits, const int* __restrict__ rows,
                                        const int* __restrict__ tokens,
                                        const float* __restrict__ amounts, int n, int V) {
  asb::pdl_wait();  // the stream's previous kernel has completed (programmatic dependent launch)
  asb::pdl_launch_dependents();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && tokens[i] >= 0 && tokens[i] < V) logits[(size_t)rows[i] * V + tokens[i]] -= amounts[i];
}

// Floats of a row that a block of C has.
int slice_floats(int V, int C) { return ((V + C - 1) / C + 3) & ~3; }

// Blocks a row, starting from what a row of this length is worth: what it takes per element against what the barriers
// of a cluster cost (top-p alone, one row of 4,000: 20.3 us in eight blocks, 13.6 in one; of 32,000: 24.4, 44.4). Half as
// many while all rows' blocks are more than run well at once (clusters of eight leave SMs out early) and, where rows are
// held in shared memory, while two blocks of the longer slice share an SM. 256 rows, top-p alone, eight blocks and those
// taken here: of 500 216 -> 13 us, of 32,000 260 -> 93, of 64,000 297 -> 193; 48 rows of 32,000 62 -> 33, of 151,936
// eight as before (108; in four 116).
int blocks_a_row(int B, int V, int one_below, int four_below, bool held) {
  constexpr int kTwoAnSM = 18 * 1024;  // floats
  int C = V <= one_below ? 1 : (V <= four_below ? 4 : 8);
  const int most8 = held ? 74 : 148;
  while (C > 1) {
    if ((long long)B * C <= (C == 8 ? most8 : (C == 4 ? 256 : 296))) break;
    if (held && slice_floats(V, C / 2) > kTwoAnSM) break;
    C /= 2;
  }
  return C;
}
int sample_blocks(int B, int V) { return blocks_a_row(B, V, 7000, 30000, true); }
// The same for the largest logit alone, which every block reads in place (256 rows of 32,000: 12.7 us in eight, 4.9 in
// one; of 151,936: 39 and 31).
int argmax_blocks(int B, int V) { return blocks_a_row(B, V, 16000, 16000, false); }

template <int C>
int launch_argmax(int* out, const float* logits, int B, int V, cudaStream_t stream) {
  asb::launch(argmax_rows_kernel<C>, C * B, kThreads, 0, stream, out, logits, V);
  return asb::check_launch("argmax_rows");
}

template <int C>
int launch_sample(int* out, const float* logits, int B, int V, const float* temperature, const int* top_k, const float* top_p,
                  const unsigned long long* seed, const unsigned long long* counter, cudaStream_t stream) {
  // a slice too long for shared memory is read in place in every pass
  const int each = slice_floats(V, C), room = each <= kMaxSlice<C> ? each : 0;
  cudaError_t e = cudaFuncSetAttribute(sample_rows_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(room * sizeof(float)));
  if (e != cudaSuccess) return asb::fail("sample_rows: shared memory of %d floats: %s", room, cudaGetErrorString(e));
  asb::launch(sample_rows_kernel<C>, C * B, kThreads, room * sizeof(float), stream, out, logits, V, temperature, top_k, top_p,
              seed, counter, room);
  return asb::check_launch("sample_rows");
}

}  // namespace

extern "C" int asb_argmax_rows(int* out, const float* logits, int B, int V, cudaStream_t stream) {
  if (B == 0) return 0;
  if (B > 0x7fffffff / kMostBlocks) return asb::fail("argmax_rows: %d rows", B);
  switch (argmax_blocks(B, V)) {
    case 1: return launch_argmax<1>(out, logits, B, V, stream);
    case 2: return launch_argmax<2>(out, logits, B, V, stream);
    case 4: return launch_argmax<4>(out, logits, B, V, stream);
    default: return launch_argmax<8>(out, logits, B, V, stream);
  }
}

// Each (row, token) pair must appear once: the penalty is subtracted once per distinct token.
extern "C" int asb_presence_penalty(float* logits, const int* rows, const int* tokens,
                                    const float* amounts, int n, int V, cudaStream_t stream) {
  if (n == 0) return 0;
  asb::launch(presence_penalty_kernel, (n + 255) / 256, 256, 0, stream, logits, rows, tokens, amounts, n, V);
  return asb::check_launch("presence_penalty");
}

extern "C" int asb_sample_rows(int* out, const float* logits, int B, int V,
                               const float* temperature, const int* top_k, const float* top_p,
                               const unsigned long long* seed, const unsigned long long* counter,
                               cudaStream_t stream) {
  if (B == 0) return 0;
  if (V < 1) return asb::fail("sample_rows: vocabulary %d", V);
  if (B > 0x7fffffff / kMostBlocks) return asb::fail("sample_rows: %d rows", B);
  switch (sample_blocks(B, V)) {
    case 1: return launch_sample<1>(out, logits, B, V, temperature, top_k, top_p, seed, counter, stream);
    case 2: return launch_sample<2>(out, logits, B, V, temperature, top_k, top_p, seed, counter, stream);
    case 4: return launch_sample<4>(out, logits, B, V, temperature, top_k, top_p, seed, counter, stream);
    default: return launch_sample<8>(out, logits, B, V, temperature, top_k, top_p, seed, counter, stream);
  }
}
