// Sampling on the device: one to eight blocks per row of float logits, token id out.
//
// The pipeline is the reference's (vllm-oxide, crates/vllm-oxide/src/sampler.rs:207-261):
// greedy short-circuit (temperature 0 or top_k 1) -> logits * (1/T) -> top-k (ties at the
// threshold are kept, sampler.rs:349-364) -> top-p over the survivors -> Gumbel-max
// argmax(x + g), g = -log(-log(u)).  Argmax ties go to the lowest index (sampler.rs:293-305).
// Two things are this engine's own:
//   * the uniform numbers come from a counter-based generator keyed per row (the caller
//     derives the key from seed, request and step), so a request's tokens do not depend on
//     what shares its batch (the reference draws all rows from one generator, sampler.rs:265-287);
//   * top-p keeps every token whose logit is >= the logit of the boundary token, the first
//     one in descending order at which the cumulative probability reaches p (the reference
//     keeps a prefix of its sort, which is the same set unless equal logits straddle the
//     boundary).  Probability mass is summed as 40-bit fixed point integers, so the set does
//     not depend on the order of summation.
#include <initializer_list>

#include "cluster.cuh"

namespace vob {

constexpr int SAMPLE_THREADS = 1024;
constexpr int SAMPLE_TOP_K = SAMPLE_THREADS / 16 * 15;      // the most that top-k gathers by the threads' maxima
constexpr int SAMPLE_CANDIDATES = 4096;    // tokens that top-p may still keep after one look at the row, held in shared memory

__device__ __forceinline__ uint32_t ordered_key(float x) {
  const uint32_t b = __float_as_uint(x + 0.f);      // -0 becomes +0: equal values get equal keys
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// The value that a key was made of (a zero without its sign).
__device__ __forceinline__ float value_of(uint32_t key) { return __uint_as_float((key & 0x80000000u) ? key & 0x7fffffffu : ~key); }

__device__ __forceinline__ unsigned long long pack_candidate(float value, int index) {
  return ((unsigned long long)ordered_key(value) << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)index);
}

__device__ __forceinline__ unsigned long long block_max_u64(unsigned long long v, unsigned long long* scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, v, o);
    v = other > v ? other : v;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  unsigned long long r = 0;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) r = scratch[i] > r ? scratch[i] : r;
  return r;
}

// uniform in (0,1), 24 bits, from (row key, token index)
__device__ __forceinline__ float counter_uniform(unsigned long long key, uint32_t index) {
  unsigned long long z = key + ((unsigned long long)index + 1ull) * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z = z ^ (z >> 31);
  return ((float)(uint32_t)(z >> 40) + 0.5f) * (1.0f / 16777216.0f);
}

// A histogram update of a whole warp at once: lanes that hit the same bin are found with match.any, their values
// summed with a warp reduction, and one lane per bin adds the sum.  The logits of a row crowd into a few bins (the
// first digit of a key is the sign and most of the exponent), and a 64-bit addition to shared memory is a
// compare-and-swap loop, so this takes top-p from 2.1 ms to 0.5 ms a batch (32-bit counts are quicker left alone).
// Every lane of the warp must call.
// values below 2^41: the low 20 bits and the rest are summed apart (32 lanes of 21 bits fit 32 bits)
__device__ __forceinline__ void warp_hist_mass(unsigned long long* hist, int bin, unsigned long long v, bool active) {
  const unsigned act = __ballot_sync(0xffffffffu, active);
  if (!active) return;
  const unsigned grp = __match_any_sync(act, bin);
  const unsigned lo = __reduce_add_sync(grp, (unsigned)(v & 0xFFFFFull));
  const unsigned hi = __reduce_add_sync(grp, (unsigned)(v >> 20));
  if ((int)(threadIdx.x & 31) == __ffs(grp) - 1) atomicAdd(&hist[bin], ((unsigned long long)hi << 20) + lo);
}

__device__ __forceinline__ unsigned long long fixed_mass(float x, float maxv) {
  return (unsigned long long)(expf(x - maxv) * 1099511627776.0f);  // 2^40
}

// f(value, index) for a thread's share of part `part` of `parts` of a row: four values a load, four loads in flight, where the row starts
// on a 16-byte boundary, the rest one by one.
template <typename F>
__device__ __forceinline__ void each_logit(const float* l, int V, int part, int parts, F f) {
  const float4* l4 = reinterpret_cast<const float4*>(l);
  const int v4 = (uintptr_t)l % 16 == 0 ? V / 4 : 0, rest = V - 4 * v4;
  const int end4 = (int)((long)v4 * (part + 1) / parts), end = 4 * v4 + (int)((long)rest * (part + 1) / parts);
  int i = (int)((long)v4 * part / parts) + threadIdx.x;
  for (; i + 3 * SAMPLE_THREADS < end4; i += 4 * SAMPLE_THREADS) {
    float4 x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = l4[i + k * SAMPLE_THREADS];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int at = 4 * (i + k * SAMPLE_THREADS);
      f(x[k].x, at); f(x[k].y, at + 1); f(x[k].z, at + 2); f(x[k].w, at + 3);
    }
  }
  for (; i < end4; i += SAMPLE_THREADS) {
    const float4 x = l4[i];
    f(x.x, 4 * i); f(x.y, 4 * i + 1); f(x.z, 4 * i + 2); f(x.w, 4 * i + 3);
  }
  for (i = 4 * v4 + (int)((long)rest * part / parts) + threadIdx.x; i < end; i += SAMPLE_THREADS) f(l[i], i);
}

// The same with every thread at every step: f(value, index, whether there is one).
template <typename F>
__device__ __forceinline__ void each_logit_together(const float* l, int V, int part, int parts, F f) {
  const float4* l4 = reinterpret_cast<const float4*>(l);
  const int v4 = (uintptr_t)l % 16 == 0 ? V / 4 : 0, rest = V - 4 * v4;
  const int end4 = (int)((long)v4 * (part + 1) / parts), end = 4 * v4 + (int)((long)rest * (part + 1) / parts);
  for (int i0 = (int)((long)v4 * part / parts); i0 < end4; i0 += 2 * SAMPLE_THREADS) {
    float4 x[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = i0 + k * SAMPLE_THREADS + threadIdx.x;
      x[k] = i < end4 ? l4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = i0 + k * SAMPLE_THREADS + threadIdx.x;
      const bool in = i < end4;
      f(x[k].x, 4 * i, in); f(x[k].y, 4 * i + 1, in); f(x[k].z, 4 * i + 2, in); f(x[k].w, 4 * i + 3, in);
    }
  }
  for (int i0 = 4 * v4 + (int)((long)rest * part / parts); i0 < end; i0 += SAMPLE_THREADS) {
    const int i = i0 + threadIdx.x;
    f(i < end ? l[i] : 0.f, i, i < end);
  }
}

// The same variable of shared memory in block `rank` of the cluster.
template <typename N>
__device__ __forceinline__ const volatile N* in_block(const N* mine, int rank) {
  unsigned long long a;
  asm("mapa.u64 %0, %1, %2;\n" : "=l"(a) : "l"(mine), "r"(rank));
  return reinterpret_cast<const volatile N*>(a);
}

__device__ __forceinline__ uint32_t block_max_u32(uint32_t v, unsigned long long* scratch) { return (uint32_t)block_max_u64(v, scratch); }

// Sum over a block; every thread gets it (integers: any order gives the same).
__device__ __forceinline__ unsigned long long block_sum_u64(unsigned long long v, unsigned long long* scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned long long total = 0;
  for (int i = 0; i < SAMPLE_THREADS / 32; ++i) total += scratch[i];
  return total;
}

// The bin in which the sum from the highest bin down reaches `need` (bin 0 if it does not), and the sum above it.  One warp, eight
// bins a lane: a single thread would walk 256 bins of shared memory one latency after the other, eight times a row.
template <typename N>
__device__ __forceinline__ void find_bin(const N* bins, N need, int& bin, N& above) {
  const int lane = threadIdx.x & 31;
  N mine = 0;
#pragma unroll
  for (int b = 0; b < 8; ++b) mine += bins[255 - 8 * lane - b];
  N upto = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const N v = __shfl_up_sync(0xffffffffu, upto, d);
    if (lane >= d) upto += v;
  }
  const unsigned reached = __ballot_sync(0xffffffffu, upto >= need);
  const int at = reached ? __ffs(reached) - 1 : 31;
  N cum = __shfl_sync(0xffffffffu, upto - mine, at);
  int b = 255 - 8 * at;
  for (int k = 0; k < 8 && b > 0; ++k) {
    if (cum + bins[b] >= need) break;
    cum += bins[b];
    --b;
  }
  bin = b;
  above = cum;
}

// A row is looked over by the blocks of a cluster, each its part: they find the maximum, what top-p's masses add up to, and the
// tokens that may still be drawn.  The first block then has all of those (it fetches the others' from their shared memory) and
// goes on alone.  Rows of whom top-k asks for more than SAMPLE_SHARED_K, and what is left to be searched as a whole, are the first block's
// from the start: the blocks' lists together would not fit, and such rows are rare.  (48 rows of 151,936, top-k 50, top-p 0.9: two blocks a
// row 44 us, one 53; of 16 flat rows with top-p alone: eight 258, one 717; of one: 98 and 559.  Timed one by one.)
constexpr int SAMPLE_SHARED_K = 256;
// Up to this many gathered tokens every thread compares its token with all: thresholds are then a look at a list that lies in shared
// memory and one reduction, where the digits of a key take four histograms with their barriers.
constexpr int SAMPLE_FEW = 512;

// MANY rows, more than there are SMs, a block each: two blocks share an SM, with 32 registers a thread.  (Top-k 50 and top-p 0.9, 149 rows of
// 151,936 tokens 66 us, 82 in two rounds; 229: 78 and 86; 229 of 32,768: 39 and 45.)
template <bool MANY>
__global__ void __launch_bounds__(SAMPLE_THREADS, MANY ? 2 : 1)
sample_kernel(const float* logits, long ld, int V, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p,
              const unsigned long long* __restrict__ keys, int* __restrict__ out, int blocks) {
  __shared__ unsigned long long scratch[32];
  __shared__ unsigned int hist[256];
  __shared__ unsigned long long mass[2][256], all_mass[256];      // (by turns: the other blocks read one while the next is made)
  __shared__ unsigned int s_prefix, s_remaining_k;
  __shared__ unsigned long long s_remaining_mass;
  __shared__ unsigned int s_ncand, s_short, s_gather;
  __shared__ unsigned long long s_told[5];          // what a block tells the others: a maximum, masses, gathered masses, how many, a draw
  __shared__ unsigned int s_bound;
  extern __shared__ unsigned long long cand_raw[];              // SAMPLE_CANDIDATES x (mass, key, index)
  unsigned long long* cand_mass = cand_raw;
  uint32_t* cand_key = reinterpret_cast<uint32_t*>(cand_raw + SAMPLE_CANDIDATES);
  uint32_t* cand_idx = cand_key + SAMPLE_CANDIDATES;
  const int row = blockIdx.x / blocks, rank = blockIdx.x % blocks, tid = threadIdx.x;
  pdl_wait();
  const float* l = logits + (size_t)row * ld;
  const float temp = temperature[row];
  const int k = top_k[row];
  const float p = top_p[row];
  const unsigned long long key_row = keys[row];
  const bool top_p_on = p > 0.f && p < 1.f;
  // (the same for every block of the row, and so is every meeting below)
  const int parts = k >= 1 && k < V && k > SAMPLE_SHARED_K && temp > 0.f ? 1 : blocks;
  if (rank >= parts) return;
  // what the blocks have told becomes every block's; a block's shared memory is read until the last meeting
  auto meet = [&]() { if (parts > 1) cluster_sync_all(); };
  auto most_of_all = [&](unsigned long long best) {
    best = block_max_u64(best, scratch);
    if (parts == 1) return best;
    if (tid == 0) s_told[0] = best;
    meet();
    for (int r = 0; r < parts; ++r) {
      const unsigned long long other = *in_block(&s_told[0], r);
      best = other > best ? other : best;
    }
    return best;
  };

  if (temp <= 0.f || k == 1) {  // greedy
    unsigned long long best = 0;
    each_logit(l, V, rank, parts, [&](float x, int i) {
      const unsigned long long c = pack_candidate(x, i);
      best = c > best ? c : best;
    });
    best = most_of_all(best);
    if (tid == 0 && rank == 0) out[row] = (int)(0xFFFFFFFFu - (uint32_t)(best & 0xFFFFFFFFull));
    meet();
    return;
  }
  const float inv_t = 1.0f / temp;

  // ---- top-k: key of the k-th largest scaled logit (0 keeps everything)
  // A token among the k largest is at least as large as the k-th largest of the threads' own maxima (k of them are tokens).  So
  // the first look at the row only takes maxima, the second gathers the tokens from that bound on into shared memory, and
  // everything after (the digits of the exact threshold, the maximum, top-p, the draw) runs over them alone: some
  // -1024 ln(1 - k / 1024) tokens of a long row, 51 for k = 50, 2,839 for 960.  The largest of the blocks' bounds is one for the whole
  // row.  (48 rows of 151,936 with top-k 50 and top-p 0.9, a block each: 35 us; 139 by the histogram alone, which is bound by atomics to a
  // handful of bins.)
  // More than SAMPLE_TOP_K asked for, or more than half of the threads' maxima equal to the bound (a masked vocabulary with fewer
  // than k tokens left: every masked token is at the bound): the first digit (sign and most of the exponent) is found by a histogram
  // over the row, and the tokens whose first digit is at least that of the k-th largest are gathered if they are few.
  uint32_t thr = 0;
  bool gathered = false;
  if (k >= 1 && k < V) {
    if (k <= SAMPLE_TOP_K) {
      uint32_t most = 0;
      each_logit(l, V, rank, parts, [&](float x, int) { most = max(most, ordered_key(x * inv_t)); });
      uint32_t bound = 0;
      for (int bit = 31; bit >= 0; --bit) {
        const uint32_t higher = bound | (1u << bit);
        if (__syncthreads_count(most >= higher) >= k) bound = higher;
      }
      // (a bound of 0: fewer threads than that have a token, and the row is short)
      const bool few = __syncthreads_count(most == bound) <= SAMPLE_THREADS / 2 && bound != 0;
      // (a part of a row where many are at the bound, such as a masked one, gathers what is above it: the bound of the others decides)
      if (!few) ++bound;
      if (tid == 0) { s_ncand = few || parts > 1 ? 0u : (unsigned)SAMPLE_CANDIDATES + 1; s_bound = bound; }
      __syncthreads();
      if (few || parts > 1) {
        each_logit(l, V, rank, parts, [&](float x, int i) {
          const uint32_t key = ordered_key(x * inv_t);
          if (key >= bound) {
            const unsigned pos = atomicAdd(&s_ncand, 1u);
            if (pos < (unsigned)SAMPLE_CANDIDATES) { cand_key[pos] = key; cand_idx[pos] = (uint32_t)i; }
          }
        });
      }
      __syncthreads();
      gathered = s_ncand <= (unsigned)SAMPLE_CANDIDATES;
      if (parts > 1) {
        meet();
        if (rank == 0) {
          // a lane asks a block how it went, then some warps a block fetch its tokens: one behind the other these are a chain of latencies
          // (8 rows of 32,768, top-k 50: 31 us and 35)
          const int lane = tid & 31, r = (tid >> 5) % parts;
          const unsigned has = lane < parts ? *in_block(&s_ncand, lane) : 0u, from = lane < parts ? *in_block(&s_bound, lane) : 0u;
          bound = __reduce_max_sync(0xffffffffu, from);
          gathered = __all_sync(0xffffffffu, has <= (unsigned)SAMPLE_CANDIDATES);
          const unsigned n = gathered && r > 0 ? __shfl_sync(0xffffffffu, has, r) : 0u;
          __syncthreads();      // (this block's own count grows from here on)
          if (n > 0) {
            const volatile uint32_t* key = in_block(cand_key, r);
            const volatile uint32_t* idx = in_block(cand_idx, r);
            for (unsigned c = (tid >> 5) / parts * 32 + lane; c < n; c += SAMPLE_THREADS / parts) {
              const uint32_t x = key[c];
              if (x < bound) continue;
              const unsigned pos = atomicAdd(&s_ncand, 1u);
              if (pos < (unsigned)SAMPLE_CANDIDATES) { cand_key[pos] = x; cand_idx[pos] = idx[c]; }
            }
          }
          __syncthreads();
          gathered = gathered && s_ncand <= (unsigned)SAMPLE_CANDIDATES;
          // every token from the largest bound on is there: if they are k, the k largest are among them
          unsigned long long have = 0;
          for (unsigned c = tid; gathered && c < s_ncand; c += SAMPLE_THREADS) have += cand_key[c] >= bound;
          gathered = block_sum_u64(have, scratch) >= (unsigned long long)k && gathered;
        }
        meet();
        if (rank > 0) return;
      }
    }
    __syncthreads();
    const bool few_left = gathered && s_ncand <= (unsigned)SAMPLE_FEW;
    if (few_left) {
      // the largest key that at least k tokens reach
      const unsigned n = s_ncand;
      const uint32_t mine = (unsigned)tid < n ? cand_key[tid] : 0u;
      unsigned reach = 0;
      if ((unsigned)tid < n)
        for (unsigned c = 0; c < n; ++c) reach += cand_key[c] >= mine;
      thr = block_max_u32((unsigned)tid < n && reach >= (unsigned)k ? mine : 0u, scratch);
    } else {
      if (tid == 0) { s_prefix = 0; s_remaining_k = (unsigned)k; s_gather = 0; }
      for (int pass = 0; pass < 4; ++pass) {
        const int shift = 24 - 8 * pass;
        if (tid < 256) hist[tid] = 0;
        __syncthreads();
        const uint32_t prefix = s_prefix;
        const uint32_t mask = pass == 0 ? 0u : (0xFFFFFFFFu << (shift + 8));
        if (gathered) {
          const unsigned ncand = s_ncand;
          for (unsigned c = tid; c < ncand; c += SAMPLE_THREADS) {
            const uint32_t key = cand_key[c];
            if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1u);
          }
        } else {
          each_logit(l, V, 0, 1, [&](float x, int) {
            const uint32_t key = ordered_key(x * inv_t);
            if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1u);
          });
        }
        __syncthreads();
        if (tid < 32) {
          const unsigned need = s_remaining_k;
          int b;
          unsigned cum;
          find_bin(hist, need, b, cum);
          if (tid == 0) {
            s_remaining_k = need - cum;
            s_prefix = prefix | ((uint32_t)b << shift);
            if (pass == 0 && !gathered && cum + hist[b] <= (unsigned)SAMPLE_CANDIDATES) { s_gather = 1; s_ncand = 0; }
          }
        }
        __syncthreads();
        if (pass == 0 && s_gather) {
          const uint32_t first = s_prefix >> 24;
          each_logit(l, V, 0, 1, [&](float x, int i) {
            const uint32_t key = ordered_key(x * inv_t);
            if ((key >> 24) >= first) {
              const unsigned pos = atomicAdd(&s_ncand, 1u);
              cand_key[pos] = key; cand_idx[pos] = (uint32_t)i;
            }
          });
          gathered = true;
          __syncthreads();
        }
      }
      thr = s_prefix;
    }
  }

  // the blocks that are still here share the row: all of them without a top-k, else the first alone
  const int of = k >= 1 && k < V ? 1 : parts;
  // ---- maximum of the scaled logits (always a survivor)
  unsigned long long best = 0;
  if (gathered) {
    const unsigned ncand = s_ncand;
    for (unsigned c = tid; c < ncand; c += SAMPLE_THREADS) {
      const unsigned long long cnd = ((unsigned long long)cand_key[c] << 32) | (unsigned long long)(0xFFFFFFFFu - cand_idx[c]);
      best = cnd > best ? cnd : best;
    }
  } else {
    each_logit(l, V, rank, of, [&](float x, int i) {
      const unsigned long long c = pack_candidate(x * inv_t, i);
      best = c > best ? c : best;
    });
  }
  best = of > 1 ? most_of_all(best) : block_max_u64(best, scratch);
  const float maxv = value_of((uint32_t)(best >> 32));

  // ---- top-p over the survivors
  if (top_p_on) {
    unsigned long long z = 0;
    if (gathered) {
      const unsigned ncand = s_ncand;
      for (unsigned c = tid; c < ncand; c += SAMPLE_THREADS) {
        const unsigned long long m = cand_key[c] >= thr ? fixed_mass(value_of(cand_key[c]), maxv) : 0ull;
        cand_mass[c] = m;
        z += m;
      }
    } else {
      each_logit(l, V, rank, of, [&](float raw, int) {
        const float x = raw * inv_t;
        if (ordered_key(x) >= thr) z += fixed_mass(x, maxv);
      });
    }
    unsigned long long total = block_sum_u64(z, scratch);
    if (of > 1) {
      if (tid == 0) s_told[1] = total;
      meet();
      total = 0;
      for (int r = 0; r < of; ++r) total += *in_block(&s_told[1], r);
    }
    if (tid == 0) {
      unsigned long long target = (unsigned long long)((double)p * (double)total);
      if (target < 1) target = 1;
      s_remaining_mass = target;
      s_prefix = 0;
    }
    __syncthreads();
    // The short way.  A token whose mass is below (1 - p) * total / V cannot lie above the boundary unless it IS the
    // boundary token (all tokens after it together weigh less than (1 - p) * total), so the tokens at or above that
    // mass are gathered into shared memory in one pass; if they fit and together reach the target, the boundary is
    // among them and the search (and later the draw) runs over them alone: a language model's distribution leaves
    // a few hundred.  Otherwise (a flat distribution) the row is searched as a whole, four more passes.
    if (tid == 0) { s_short = gathered ? 1u : 0u; if (!gathered) s_ncand = 0; }
    __syncthreads();
    if (!gathered) {
      const unsigned long long floor_mass = (unsigned long long)((1.0 - (double)p) * (double)total / (double)V);
      if (floor_mass >= 1) {
        each_logit(l, V, rank, of, [&](float raw, int i) {
          const float x = raw * inv_t;
          const uint32_t key = ordered_key(x);
          if (key < thr) return;
          const unsigned long long m = fixed_mass(x, maxv);
          if (m < floor_mass) return;
          const unsigned pos = atomicAdd(&s_ncand, 1u);
          if (pos < (unsigned)SAMPLE_CANDIDATES) { cand_mass[pos] = m; cand_key[pos] = key; cand_idx[pos] = (uint32_t)i; }
        });
      } else if (tid == 0) {
        s_ncand = SAMPLE_CANDIDATES + 1;
      }
    }
    __syncthreads();
    if (!gathered) {
      unsigned n = s_ncand;
      unsigned long long have = 0;
      if (n <= (unsigned)SAMPLE_CANDIDATES)
        for (unsigned i = tid; i < n; i += SAMPLE_THREADS) have += cand_mass[i];
      have = block_sum_u64(have, scratch);
      if (of > 1) {
        if (tid == 0) { s_told[2] = have; s_told[3] = n; }
        meet();
        have = n = 0;
        for (int r = 0; r < of; ++r) {
          have += *in_block(&s_told[2], r);
          n += (unsigned)min(*in_block(&s_told[3], r), (unsigned long long)SAMPLE_CANDIDATES + 1);
        }
      }
      const bool enough = n <= (unsigned)SAMPLE_CANDIDATES && have >= s_remaining_mass;
      if (tid == 0) s_short = enough ? 1u : 0u;
      if (enough && of > 1) {
        // the others' gathered tokens become the first block's
        if (rank == 0) {
          for (int r = 1; r < of; ++r) {
            const unsigned more = (unsigned)*in_block(&s_told[3], r);
            const volatile unsigned long long* m = in_block(cand_mass, r);
            const volatile uint32_t* key = in_block(cand_key, r);
            const volatile uint32_t* idx = in_block(cand_idx, r);
            for (unsigned c = tid; c < more; c += SAMPLE_THREADS) {
              const unsigned pos = atomicAdd(&s_ncand, 1u);
              cand_mass[pos] = m[c]; cand_key[pos] = key[c]; cand_idx[pos] = idx[c];
            }
          }
        }
        meet();
        if (rank > 0) return;
      }
      __syncthreads();
    }
    const unsigned ncand = s_ncand;
    const bool short_way = s_short != 0;
    if (short_way && ncand <= (unsigned)SAMPLE_FEW) {
      // the largest key down to which the masses reach the target
      const uint32_t mine = (unsigned)tid < ncand ? cand_key[tid] : 0u;
      unsigned long long reach = 0;
      if ((unsigned)tid < ncand)
        for (unsigned c = 0; c < ncand; ++c) reach += cand_key[c] >= mine ? cand_mass[c] : 0ull;
      const uint32_t at = block_max_u32((unsigned)tid < ncand && reach >= s_remaining_mass ? mine : 0u, scratch);
      if (tid == 0) s_prefix = at;
      __syncthreads();
    } else
    for (int pass = 0; pass < 4; ++pass) {
      const int shift = 24 - 8 * pass;
      unsigned long long* bins = mass[pass & 1];
      if (tid < 256) bins[tid] = 0;
      __syncthreads();
      const uint32_t prefix = s_prefix;
      const uint32_t mask = pass == 0 ? 0u : (0xFFFFFFFFu << (shift + 8));
      if (short_way) {
        for (unsigned i = tid; i < ncand; i += SAMPLE_THREADS) {
          const uint32_t key = cand_key[i];
          if ((key & mask) == prefix) atomicAdd(&bins[(key >> shift) & 255u], cand_mass[i]);
        }
      } else {
        each_logit_together(l, V, rank, of, [&](float raw, int, bool there) {
          const float x = there ? raw * inv_t : 0.f;
          const uint32_t key = ordered_key(x);
          const bool in = there && key >= thr && (key & mask) == prefix;
          warp_hist_mass(bins, (int)((key >> shift) & 255u), in ? fixed_mass(x, maxv) : 0ull, in);
        });
      }
      __syncthreads();
      if (of > 1 && !short_way) {
        meet();
        if (tid < 256) {
          unsigned long long sum = 0;
          for (int r = 0; r < of; ++r) sum += *in_block(&bins[tid], r);
          all_mass[tid] = sum;
        }
        bins = all_mass;
        __syncthreads();
      }
      if (tid < 32) {
        const unsigned long long need = s_remaining_mass;
        int b;
        unsigned long long cum;
        find_bin(bins, need, b, cum);
        if (tid == 0) {
          s_remaining_mass = need - cum;
          s_prefix = prefix | ((uint32_t)b << shift);
        }
      }
      __syncthreads();
    }
    const uint32_t thr_p = s_prefix;
    thr = thr_p > thr ? thr_p : thr;
  }

  // ---- Gumbel-max over the survivors (gathered ones are the first block's)
  const int drawing = top_p_on && s_short != 0 ? 1 : of;
  best = 0;
  if (gathered || (top_p_on && s_short != 0)) {
    // the survivors are among the gathered tokens
    const unsigned ncand = s_ncand;
    for (unsigned c = tid; c < ncand; c += SAMPLE_THREADS) {
      if (cand_key[c] < thr) continue;
      const int i = (int)cand_idx[c];
      const float x = value_of(cand_key[c]);
      const float u = counter_uniform(key_row, (uint32_t)i);
      const float g = -logf(-logf(u));
      const unsigned long long cnd = pack_candidate(x + g, i);
      best = cnd > best ? cnd : best;
    }
  } else
  each_logit(l, V, rank, drawing, [&](float raw, int i) {
    const float x = raw * inv_t;
    if (ordered_key(x) < thr) return;
    const float u = counter_uniform(key_row, (uint32_t)i);
    const float g = -logf(-logf(u));
    const unsigned long long c = pack_candidate(x + g, i);
    best = c > best ? c : best;
  });
  if (drawing > 1) {
    // (another variable than the maximum's: a block may still read that one)
    best = block_max_u64(best, scratch);
    if (tid == 0) s_told[4] = best;
    meet();
    for (int r = 0; r < drawing; ++r) {
      const unsigned long long other = *in_block(&s_told[4], r);
      best = other > best ? other : best;
    }
    meet();
    if (rank > 0) return;
  } else {
    best = block_max_u64(best, scratch);
  }
  if (tid == 0) out[row] = (int)(0xFFFFFFFFu - (uint32_t)(best & 0xFFFFFFFFull));
}

// Penalties before everything else (sampler.rs:320-345): for each distinct token seen so far,
// logit /= repetition (when != 0), logit -= presence, logit -= frequency * count.
__global__ void penalties_kernel(float* logits, long ld, int V, const int* __restrict__ row_of, const int* __restrict__ token,
                                 const int* __restrict__ count, const float* __restrict__ presence,
                                 const float* __restrict__ frequency, const float* __restrict__ repetition, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = row_of[i], tk = token[i];
  if (tk < 0 || tk >= V) return;
  float v = logits[(size_t)r * ld + tk];
  if (repetition[r] != 0.f) v /= repetition[r];
  v -= presence[r];
  if (frequency[r] != 0.f) v -= frequency[r] * (float)count[i];
  logits[(size_t)r * ld + tk] = v;
}

}  // namespace vob

using namespace vob;

VOB_API int vob_sample(const float* logits, long ld, int R, int V, const float* temperature, const int* top_k,
                       const float* top_p, const unsigned long long* keys, int* out, cudaStream_t stream) {
  if (R <= 0) return 0;
  if (V <= 0) return VOB_BAD_ARGUMENT;
  const int smem = SAMPLE_CANDIDATES * 16;
  static bool configured = false;
  static int rows_of[4] = {};      // rows that 1, 2, 4, 8 blocks each work on at once
  if (!configured) {
    for (auto kernel : {sample_kernel<false>, sample_kernel<true>}) {
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e != cudaSuccess) return (int)e;
    }
    for (int i = 1; i < 4; ++i) rows_of[i] = resident_clusters(sample_kernel<false>, SAMPLE_THREADS, smem, 1u << i);
    configured = true;
  }
  // Blocks a row: as many (8, 4, 2) as leave no row for a second round, of at least four thousand tokens each, else one.  Clusters lie inside a GPC,
  // so those of 8 are 15 and not 18, those of 4 33 and not 37 (151,936 tokens, top-k 50: 16 rows by eight blocks 53 us, by four 33; 34 rows by four
  // 47, by two 35; with top-p alone 252 and 209, 399 and 356).
  int i = 3;
  while (i > 0 && (R > rows_of[i] || V >> i < 4 * SAMPLE_THREADS)) --i;
  const int blocks = 1 << i;
  if (blocks == 1)
    return launch_kernel(R > sm_count() ? sample_kernel<true> : sample_kernel<false>, dim3((unsigned)R), SAMPLE_THREADS, smem, stream, logits, ld, V,
                         temperature, top_k, top_p, keys, out, blocks);
  return launch_kernel_cluster(sample_kernel<false>, dim3((unsigned)(R * blocks)), SAMPLE_THREADS, smem, stream, (unsigned)blocks, logits, ld, V,
                               temperature, top_k, top_p, keys, out, blocks);
}

// (row, token, count) triples: one per distinct token of a row's history; a triple must appear once.
VOB_API int vob_apply_penalties(float* logits, long ld, int V, const int* row_of, const int* token, const int* count,
                                const float* presence, const float* frequency, const float* repetition, int n,
                                cudaStream_t stream) {
  if (n <= 0) return 0;
  penalties_kernel<<<(n + 255) / 256, 256, 0, stream>>>(logits, ld, V, row_of, token, count, presence, frequency,
                                                        repetition, n);
  return launch_status();
}
