// The gated delta rule: a matrix state per head that forgets by a decay and is corrected toward each new value.
//
// Per head, with S [dim, vdim] float, carried from token to token in the request's state slot (stored [vdim][dim]):
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q          (the read-out sees the token's own write)
// q and k are unit vectors (x / sqrt(sum x^2 + 1e-6)), q also times dim^(-1/2); beta = sigmoid(b);
// g = exp(-exp(A_log) * softplus(a + dt_bias)): one number a head, or (`channel_decay`) one a head and key channel, which
// multiplies that row of S (a and dt_bias are then [heads, dim]).  q, k and v come out of short causal convolutions over time (one filter a
// channel, `taps` taps, the last one the current token's) followed by SiLU; the last taps - 1 inputs of every channel are
// part of the request's state, behind S in the same slot.  Query/key head h / (heads / kv_heads) serves value head h.
//
// Four kernels (short_conv_step is the first two in one, for steps of short portions):
//   short_conv_silu    out[t, c] = f(sum_j w[c, j] x[t - (taps-1) + j, c]), inputs before the portion's start from the slot;
//                      f is SiLU or (`act` 0) the identity.  With `bias_in` the filter's inputs are x + bias_in (zeros stay
//                      zeros before the sequence's start; the slot keeps the sums), with `bias_out` a number a channel is
//                      added behind the filter; the output is float or (TO) of the model's type
//   short_conv_state   the slot's taps - 1 inputs after this portion (run after the first: it overwrites what that one reads)
//   delta_scan         the recurrence.  A column of S lives in the registers of LANES threads (ROWS rows each, rows
//                      interleaved so that a warp's loads of the state fill whole sectors); a block takes the columns
//                      c0.. of one (request, head) and walks the request's tokens in order, while half of its warps
//                      prepare the next tokens in shared memory (unit vectors, decay and beta are made there, in float).
//   delta_out_norm     o / sqrt(mean(o^2) + eps) * w * SiLU(gate) (or * sigmoid(gate)), per head over vdim; w may be one gain for
//                      all heads or a gain an element of every head.  With a normaliser (`nq`, `gates`: see recurrent.cu,
//                      exponential gates) o is first divided by max(|nq|, floor) + 1e-6
// Everything but the inputs' type T is float on both paths.  The chain of operations of an output depends only on the
// request's tokens and the state it starts from, not on the cut, the batch or the slot.
#include "common.cuh"

namespace vob {

constexpr int DELTA_MAX_TAPS = 9;

__device__ __forceinline__ float silu_f(float x) { return x / (1.f + expf(-x)); }

constexpr int CONV_TOKENS = 8;    // tokens a thread walks in a large step: the filter's window slides through registers

// CONV_TOKENS tokens of one portion from token t_first (place j of the portion) on, for filters of up to MAX taps.
template <int MAX, typename T, typename TO>
__device__ __forceinline__ void conv_tokens(const T* x, long x_stride, const float* st, const float (&wt)[DELTA_MAX_TAPS], float b_in, float b_out,
                                            TO* out, int t_first, int j, int c, int C, int taps, int act) {
  float in[MAX - 1 + CONV_TOKENS];      // in[s]: input t_first - (MAX - 1) + s
#pragma unroll
  for (int s = 0; s < MAX - 1; ++s) {
    const int back = MAX - 1 - s;        // tokens before the thread's first
    in[s] = back > taps - 1 ? 0.f : (j >= back ? to_f<T>(x[(size_t)(t_first - back) * x_stride + c]) + b_in : st[(size_t)(taps - 1 + j - back) * C + c]);
  }
#pragma unroll
  for (int k = 0; k < CONV_TOKENS; ++k) in[MAX - 1 + k] = to_f<T>(x[(size_t)(t_first + k) * x_stride + c]) + b_in;
  float wr[MAX];                          // the filter, newest tap last, zeros in front
#pragma unroll
  for (int s = 0; s < MAX; ++s) {
    wr[s] = MAX == 4 ? wt[s] : 0.f;
    const int tap = s - (MAX - taps);
#pragma unroll
    for (int q = 0; q < MAX; ++q)
      if (MAX != 4 && q == tap) wr[s] = wt[q];
  }
#pragma unroll
  for (int k = 0; k < CONV_TOKENS; ++k) {
    float acc = b_out;
#pragma unroll
    for (int s = 0; s < MAX; ++s)
      if (MAX == 4 || s >= MAX - taps) acc = fmaf(wr[s], in[k + s], acc);          // oldest input first
    out[(size_t)(t_first + k) * C + c] = from_f<TO>(act ? silu_f(acc) : acc);
  }
}

// A thread's `walk` tokens of channel c one by one, over any portions.
template <typename T, typename TO>
__device__ __forceinline__ void conv_walk(const T* x, long x_stride, const float* state, long state_stride, long conv_off, const int* __restrict__ token_req,
                                          const int* __restrict__ cu_q, const int* __restrict__ state_slots, const float (&wt)[DELTA_MAX_TAPS],
                                          float w_now, float b_in, float b_out, TO* out, int t_first, int num_tokens, int walk, int c, int C, int taps,
                                          long num_slots, int act, int* err) {
  float win[DELTA_MAX_TAPS - 1];      // win[s]: the input taps - 1 - s tokens back
  bool have = false;
  for (int tt = 0; tt < walk; ++tt) {
    const int t = t_first + tt;
    if (t >= num_tokens) break;
    const int req = token_req[t];
    if (req < 0) { have = false; continue; }
    const int j = t - cu_q[req];
    if (!have || j == 0) {            // the window is filled anew at the start of the thread's tokens and of a portion
      const int slot = state_slots[req];
      if (slot < 0 || slot >= num_slots) {
        atomicOr(err, VOB_ERR_SLOT);
        have = false;
        continue;
      }
      const float* st = state + (size_t)slot * state_stride + conv_off;
#pragma unroll
      for (int s = 0; s < DELTA_MAX_TAPS - 1; ++s) {
        if (s < taps - 1) {
          const int rel = j - (taps - 1) + s;      // place within the portion; before its start the slot has the input
          win[s] = rel >= 0 ? to_f<T>(x[(size_t)(t - (taps - 1) + s) * x_stride + c]) + b_in : st[(size_t)(taps - 1 + rel) * C + c];
        }
      }
      have = true;
    }
    const float cur = to_f<T>(x[(size_t)t * x_stride + c]) + b_in;
    float acc = b_out;
#pragma unroll
    for (int s = 0; s < DELTA_MAX_TAPS - 1; ++s)
      if (s < taps - 1) acc = fmaf(wt[s], win[s], acc);          // oldest input first
    acc = fmaf(w_now, cur, acc);
    out[(size_t)t * C + c] = from_f<TO>(act ? silu_f(acc) : acc);
#pragma unroll
    for (int s = 0; s < DELTA_MAX_TAPS - 1; ++s) {
      if (s < taps - 2) win[s] = win[s + 1 < DELTA_MAX_TAPS - 1 ? s + 1 : s];
      else if (s == taps - 2) win[s] = cur;
    }
  }
}

// FOUR: filters of four taps in large steps, without the selections that a filter of any length needs (an instance of its own: both ways in
// one take registers from every filter, 3 to 12 % of their time).
template <typename T, typename TO, bool FOUR>
__global__ void __launch_bounds__(128)
short_conv_silu_kernel(const T* x, long x_stride, const float* __restrict__ w, const float* __restrict__ bias_in,
                       const float* __restrict__ bias_out, const float* state, long state_stride,
                       long conv_off, const int* __restrict__ token_req, const int* __restrict__ cu_q,
                       const int* __restrict__ state_slots, TO* out, int num_tokens, int walk, int C, int taps, long num_slots,
                       int act, int* err) {
  pdl_launch_dependents();
  const int t_first = blockIdx.x * walk;
  const int c = blockIdx.y * 128 + threadIdx.x;
  float wt[DELTA_MAX_TAPS];
#pragma unroll
  for (int s = 0; s < DELTA_MAX_TAPS; ++s) wt[s] = (c < C && s < taps) ? w[(size_t)c * taps + s] : 0.f;
  const float w_now = c < C ? w[(size_t)c * taps + taps - 1] : 0.f;      // the current token's tap
  const float b_in = bias_in && c < C ? bias_in[c] : 0.f, b_out = bias_out && c < C ? bias_out[c] : 0.f;
  pdl_wait();
  if (c >= C) return;
  // the usual case of a large step, all of the thread's tokens in one portion: every input is asked for before the first is used
  if (walk == CONV_TOKENS && t_first + CONV_TOKENS <= num_tokens) {
    const int req = token_req[t_first];
    if (req >= 0 && req == token_req[t_first + CONV_TOKENS - 1]) {
      const int j = t_first - cu_q[req];
      const int slot = state_slots[req];
      if (slot < 0 || slot >= num_slots) {
        atomicOr(err, VOB_ERR_SLOT);
        return;
      }
      const float* st = state + (size_t)slot * state_stride + conv_off;
      conv_tokens<FOUR ? 4 : DELTA_MAX_TAPS, T, TO>(x, x_stride, st, wt, b_in, b_out, out, t_first, j, c, C, taps, act);
      return;
    }
  }
  conv_walk<T, TO>(x, x_stride, state, state_stride, conv_off, token_req, cu_q, state_slots, wt, w_now, b_in, b_out, out, t_first, num_tokens, walk, c, C,
                   taps, num_slots, act, err);
}

// Filters of four taps in large steps, two neighbouring channels a thread (an even number of channels, rows on two elements' boundaries):
// the kernel is bound by memory, and 2-byte accesses leave it half of that.  (3,165 tokens of 4,096 channels into float: 30 us; 44 by a channel a
// thread.)
template <typename T, typename TO>
__global__ void __launch_bounds__(128)
short_conv_pairs_kernel(const T* x, long x_stride, const float* __restrict__ w, const float* __restrict__ bias_in,
                        const float* __restrict__ bias_out, const float* state, long state_stride, long conv_off,
                        const int* __restrict__ token_req, const int* __restrict__ cu_q, const int* __restrict__ state_slots, TO* out,
                        int num_tokens, int C, long num_slots, int act, int* err) {
  using P = Pair2<T>;
  pdl_launch_dependents();
  const int t_first = blockIdx.x * CONV_TOKENS;
  const int c = 2 * (blockIdx.y * 128 + threadIdx.x);
  if (c >= C) return;
  float wt[2][4], b_in[2], b_out[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
#pragma unroll
    for (int s = 0; s < 4; ++s) wt[e][s] = w[(size_t)(c + e) * 4 + s];
    b_in[e] = bias_in ? bias_in[c + e] : 0.f;
    b_out[e] = bias_out ? bias_out[c + e] : 0.f;
  }
  const int req = token_req[t_first];
  const bool one = t_first + CONV_TOKENS <= num_tokens && req >= 0 && req == token_req[min(t_first + CONV_TOKENS, num_tokens) - 1];
  const int j = one ? t_first - cu_q[req] : 0, slot = one ? state_slots[req] : 0;
  int place[CONV_TOKENS], slot_of[CONV_TOKENS];      // of several portions: a token's place in its own (-1: none) and its slot
  if (!one) {
#pragma unroll
    for (int k = 0; k < CONV_TOKENS; ++k) {
      const int r = t_first + k < num_tokens ? token_req[t_first + k] : -1;
      place[k] = r >= 0 ? t_first + k - cu_q[r] : -1;
      slot_of[k] = r >= 0 ? state_slots[r] : 0;
    }
  }
  pdl_wait();
  if (!one) {
    // portions' edges, and every block of a step of short ones: all rows are asked for at once here too, a token then takes its inputs before
    // its portion's start from its slot
    typename P::Raw rows[3 + CONV_TOKENS];
#pragma unroll
    for (int s = 0; s < 3 + CONV_TOKENS; ++s)
      if (s < 3 ? place[0] >= 3 - s : place[s - 3 < 0 ? 0 : s - 3] >= 0)
        rows[s] = *reinterpret_cast<const typename P::Raw*>(x + (size_t)(t_first - 3 + s) * x_stride + c);
    float o[CONV_TOKENS][2];
    bool bad = false;
#pragma unroll
    for (int k = 0; k < CONV_TOKENS; ++k) {
      if (place[k] < 0) continue;
      if (slot_of[k] < 0 || slot_of[k] >= num_slots) {
        bad = true;
        place[k] = -1;
        continue;
      }
      const float* st = state + (size_t)slot_of[k] * state_stride + conv_off;
      o[k][0] = b_out[0];
      o[k][1] = b_out[1];
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        float v[2];
        if (place[k] >= 3 - s) {
          const float2 r = P::get(rows[k + s]);
          v[0] = r.x + b_in[0];
          v[1] = r.y + b_in[1];
        } else {
          v[0] = st[(size_t)(place[k] + s) * C + c];
          v[1] = st[(size_t)(place[k] + s) * C + c + 1];
        }
        o[k][0] = fmaf(wt[0][s], v[0], o[k][0]);
        o[k][1] = fmaf(wt[1][s], v[1], o[k][1]);
      }
    }
#pragma unroll
    for (int k = 0; k < CONV_TOKENS; ++k)
      if (place[k] >= 0) Pair2<TO>::put(out + (size_t)(t_first + k) * C + c, act ? silu_f(o[k][0]) : o[k][0], act ? silu_f(o[k][1]) : o[k][1]);
    if (bad) atomicOr(err, VOB_ERR_SLOT);
    return;
  }
  if (slot < 0 || slot >= num_slots) {
    atomicOr(err, VOB_ERR_SLOT);
    return;
  }
  const float* st = state + (size_t)slot * state_stride + conv_off;
  typename P::Raw raw[3 + CONV_TOKENS];      // inputs t_first - 3, ...
#pragma unroll
  for (int s = 0; s < 3 + CONV_TOKENS; ++s)
    if (s >= 3 || j >= 3 - s) raw[s] = *reinterpret_cast<const typename P::Raw*>(x + (size_t)(t_first - 3 + s) * x_stride + c);
  float in[2][3 + CONV_TOKENS];
#pragma unroll
  for (int s = 0; s < 3 + CONV_TOKENS; ++s) {
    if (s >= 3 || j >= 3 - s) {
      const float2 v = P::get(raw[s]);
      in[0][s] = v.x + b_in[0];
      in[1][s] = v.y + b_in[1];
    } else {
#pragma unroll
      for (int e = 0; e < 2; ++e) in[e][s] = st[(size_t)(j + s) * C + c + e];      // (the slot's entry of the input 3 - s tokens back)
    }
  }
#pragma unroll
  for (int k = 0; k < CONV_TOKENS; ++k) {
    float o[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float acc = b_out[e];
#pragma unroll
      for (int s = 0; s < 4; ++s) acc = fmaf(wt[e][s], in[e][k + s], acc);          // oldest input first
      o[e] = act ? silu_f(acc) : acc;
    }
    Pair2<TO>::put(out + (size_t)(t_first + k) * C + c, o[0], o[1]);
  }
}

template <typename T>
__global__ void __launch_bounds__(128)
short_conv_state_kernel(const T* x, long x_stride, const float* __restrict__ bias_in, float* state, long state_stride, long conv_off,
                        const int* __restrict__ cu_q, const int* __restrict__ state_slots, int C, int taps, long num_slots) {
  pdl_launch_dependents();
  const int b = blockIdx.y;
  const int c = blockIdx.x * 128 + threadIdx.x;
  const int t0 = cu_q[b], n = cu_q[b + 1] - t0;
  const int slot = state_slots[b];
  pdl_wait();
  if (n <= 0 || slot < 0 || slot >= num_slots || c >= C) return;
  const float b_in = bias_in ? bias_in[c] : 0.f;
  float* st = state + (size_t)slot * state_stride + conv_off;
  float nv[DELTA_MAX_TAPS - 1];
#pragma unroll
  for (int s = 0; s < DELTA_MAX_TAPS - 1; ++s) {
    if (s < taps - 1) {
      const int rel = n - (taps - 1) + s;     // place within the portion of the input that entry s holds afterwards
      nv[s] = rel >= 0 ? to_f<T>(x[(size_t)(t0 + rel) * x_stride + c]) + b_in : st[(size_t)(s + n) * C + c];
    }
  }
#pragma unroll
  for (int s = 0; s < DELTA_MAX_TAPS - 1; ++s)
    if (s < taps - 1) st[(size_t)s * C + c] = nv[s];
}

// Both of the above in one launch for steps whose portions are short (decoding): a thread owns one channel of one request,
// takes its window from the slot, walks the request's few tokens and leaves the window in the slot.  The same sums in the
// same order as the two kernels.
template <typename T, typename TO>
__global__ void __launch_bounds__(128)
short_conv_step_kernel(const T* x, long x_stride, const float* __restrict__ w, const float* __restrict__ bias_in,
                       const float* __restrict__ bias_out, float* state, long state_stride, long conv_off,
                       const int* __restrict__ cu_q, const int* __restrict__ state_slots, TO* out, int C, int taps,
                       long num_slots, int act, int* err) {
  pdl_launch_dependents();
  const int b = blockIdx.y;
  const int c = blockIdx.x * 128 + threadIdx.x;
  const int t0 = cu_q[b], n = cu_q[b + 1] - t0;
  const int slot = state_slots[b];
  float wt[DELTA_MAX_TAPS];
#pragma unroll
  for (int s = 0; s < DELTA_MAX_TAPS; ++s) wt[s] = (c < C && s < taps) ? w[(size_t)c * taps + s] : 0.f;
  const float w_now = c < C ? w[(size_t)c * taps + taps - 1] : 0.f;
  const float b_in = bias_in && c < C ? bias_in[c] : 0.f, b_out = bias_out && c < C ? bias_out[c] : 0.f;
  pdl_wait();
  if (n <= 0) return;
  if (slot < 0 || slot >= num_slots) {
    if (threadIdx.x == 0) atomicOr(err, VOB_ERR_SLOT);
    return;
  }
  if (c >= C) return;
  float* st = state + (size_t)slot * state_stride + conv_off;
  float win[DELTA_MAX_TAPS - 1];
#pragma unroll
  for (int s = 0; s < DELTA_MAX_TAPS - 1; ++s) win[s] = s < taps - 1 ? st[(size_t)s * C + c] : 0.f;
  for (int i = 0; i < n; ++i) {
    const float cur = to_f<T>(x[(size_t)(t0 + i) * x_stride + c]) + b_in;
    float acc = b_out;
#pragma unroll
    for (int s = 0; s < DELTA_MAX_TAPS - 1; ++s)
      if (s < taps - 1) acc = fmaf(wt[s], win[s], acc);
    acc = fmaf(w_now, cur, acc);
    out[(size_t)(t0 + i) * C + c] = from_f<TO>(act ? silu_f(acc) : acc);
#pragma unroll
    for (int s = 0; s < DELTA_MAX_TAPS - 1; ++s) {
      if (s < taps - 2) win[s] = win[s + 1 < DELTA_MAX_TAPS - 1 ? s + 1 : s];
      else if (s == taps - 2) win[s] = cur;
    }
  }
#pragma unroll
  for (int s = 0; s < DELTA_MAX_TAPS - 1; ++s)
    if (s < taps - 1) st[(size_t)s * C + c] = win[s];
}

// ---------------------------------------------------------------- the recurrence
constexpr int DS_COMPUTE = 128;   // threads that hold the state
constexpr int DS_LOADERS = 128;   // threads that prepare the next tokens meanwhile
constexpr int DS_THREADS = DS_COMPUTE + DS_LOADERS;

// The request of grid layer z, the longest portion first (up to 32 requests; else in the order of the batch): blocks start in the
// order of the grid, and a long portion that starts late ends late.  Every lane of the warp must call.
__device__ __forceinline__ int longest_first(const int* __restrict__ cu_q) {
  const int B = gridDim.z, lane = threadIdx.x & 31;
  if (B == 1 || B > 32) return blockIdx.z;
  const int mine = lane < B ? cu_q[lane + 1] - cu_q[lane] : -1;
  if (__reduce_max_sync(0xffffffffu, mine) == __reduce_min_sync(0xffffffffu, lane < B ? mine : INT_MAX)) return blockIdx.z;      // decoding
  int rank = 0;
  for (int j = 0; j < B; ++j) {
    const int other = __shfl_sync(0xffffffffu, mine, j);
    rank += other > mine || (other == mine && j < lane);
  }
  return __ffs(__ballot_sync(0xffffffffu, lane < B && rank == (int)blockIdx.z)) - 1;
}

// qkv: float [tokens, 2 * kvh * dim + heads * vdim] (q heads, k heads, v heads: the convolutions' output);
// ab: rows of ab_stride elements of T, beta's pre-activation of head h at b_off + h, the decay's at a_off + h.
// A column of the state is held by LANES neighbouring threads, ROWS rows each (LANES * ROWS >= dim); 128 such threads
// walk the tokens, CH at a time from one of two buffers in shared memory, while four more warps fill the other buffer:
// unit vectors (laid out so that a thread finds its rows side by side), decay, beta and the block's slice of the values.
// The two groups meet on named barriers: "full" when a buffer is ready, "empty" when its tokens have been walked.
// AHEAD: a token's rows are asked for while the token before is worked on; without it a thread takes a quarter fewer registers and
// three blocks share an SM, which is what many requests of one or few tokens wait for (their states come from memory).  With it two do,
// also where the decay is one a row (left to itself the compiler takes 170 registers there, which is one block: a second
// round from 149 blocks on.  One portion of 2,048 tokens, 32 heads of 128 x 128: 838 us, 1,438 with one; 333, 1,055 and 1,777, 16 heads:
// 713 and 991; the loop before the read-outs went beside the exchange: 827 and 808).
template <typename T, int LANES, int ROWS, bool CHD, bool AHEAD>
__global__ void __launch_bounds__(DS_THREADS, ROWS != 16 ? 1 : (AHEAD ? 2 : 3))
delta_scan_kernel(const float* qkv, const T* ab, long ab_stride, int b_off, int a_off, const float* __restrict__ A_log,
                  const float* __restrict__ dt_bias, float* state, long state_stride, const int* __restrict__ cu_q,
                  const int* __restrict__ state_slots, float* raw, int heads, int kvh, int dim, int vdim, long num_slots,
                  int* err) {
  constexpr int COLS = DS_COMPUTE / LANES;
  constexpr int RS = ROWS + 4;                 // a thread's rows in shared memory, 16 bytes apart from the next thread's:
  constexpr int KW = LANES * RS;               // the 16-byte reads of a column's LANES threads then fall into different banks
  constexpr int CH = ROWS > 16 ? 8 : 16;       // tokens a buffer holds
  constexpr int BUF = CH * ((CHD ? 3 : 2) * KW + COLS + 2);     // CHD: a decay for every row of the head beside k and q
  extern __shared__ __align__(16) float ds_smem[];
  pdl_launch_dependents();
  const int h = blockIdx.y, c0 = blockIdx.x * COLS;
  const int tid = threadIdx.x, lane = tid & 31;
  const int b = AHEAD ? longest_first(cu_q) : blockIdx.z;
  const int t0 = cu_q[b], t1 = cu_q[b + 1];
  const int slot = state_slots[b];
  const float neg_rate = -expf(A_log[h]), bias = CHD ? 0.f : dt_bias[h];
  pdl_wait();
  if (t1 <= t0) return;
  if (slot < 0 || slot >= num_slots) {
    if (tid == 0) atomicOr(err, VOB_ERR_SLOT);
    return;
  }
  const int kh = h / (heads / kvh);
  const int C = 2 * kvh * dim + heads * vdim;
  const int chunks = (t1 - t0 + CH - 1) / CH;
  if (tid >= DS_COMPUTE) {
    // ------------------------------------------------ loaders
    const int lw = (tid - DS_COMPUTE) >> 5;
    const float qscale = 1.f / sqrtf((float)dim);
    for (int c = 0; c < chunks; ++c) {
      float* ks = ds_smem + (c & 1) * BUF;
      float* qs = ks + CH * KW;
      float* vs = qs + CH * KW;
      float* gs = vs + CH * COLS;
      float* bs = gs + CH;
      float* gv = bs + CH;                                    // CHD: [CH][KW], laid out as ks
      if (c >= 2) named_sync(3 + (c & 1), DS_THREADS);        // the walkers have left this buffer
      const int base = t0 + c * CH, n = min(CH, t1 - base);
      // a warp takes tokens lw, lw + 4, ...: all their loads are issued before the first sum is taken
      constexpr int NV = (LANES * ROWS + 31) / 32, TPW = CH / (DS_LOADERS / 32);
      float qv[TPW][NV], kv[TPW][NV], av[CHD ? TPW : 1][CHD ? NV : 1];
#pragma unroll
      for (int tt = 0; tt < TPW; ++tt) {
        const int i = lw + tt * (DS_LOADERS / 32);
        const float* qrow = qkv + (size_t)(base + min(i, n - 1)) * C + (size_t)kh * dim;
        const float* krow = qrow + (size_t)kvh * dim;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const int d = lane + 32 * j;
          const bool ok = i < n && d < dim;
          qv[tt][j] = ok ? qrow[d] : 0.f;
          kv[tt][j] = ok ? krow[d] : 0.f;
          if constexpr (CHD)      // the decay's pre-activation of (head h, key channel d), with its bias
            av[tt][j] = ok ? to_f<T>(ab[(size_t)(base + i) * ab_stride + a_off + (size_t)h * dim + d]) + dt_bias[(size_t)h * dim + d]
                           : 0.f;
        }
      }
      if (lane < TPW && lw + lane * (DS_LOADERS / 32) < n) {
        const int i = lw + lane * (DS_LOADERS / 32);
        const T* abrow = ab + (size_t)(base + i) * ab_stride;
        const float bv = to_f<T>(abrow[b_off + h]);
        bs[i] = 1.f / (1.f + expf(-bv));
        if (!CHD) {
          const float a1 = to_f<T>(abrow[a_off + h]) + bias;
          const float sp = a1 > 20.f ? a1 : log1pf(expf(a1));
          gs[i] = expf(neg_rate * sp);
        }
      }
      // The sums of squares of all tokens side by side (one after the other they are a chain of forty exchanges); then one lane a sum
      // takes its root and quotient.  With a token or two a request only those that there are, below.
      float sums[2 * TPW];
#pragma unroll
      for (int tt = 0; tt < TPW; ++tt) {
        sums[2 * tt] = sums[2 * tt + 1] = 0.f;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          sums[2 * tt] = fmaf(qv[tt][j], qv[tt][j], sums[2 * tt]);
          sums[2 * tt + 1] = fmaf(kv[tt][j], kv[tt][j], sums[2 * tt + 1]);
        }
      }
      float unit = 0.f;
      if (AHEAD) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int r = 0; r < 2 * TPW; ++r) sums[r] += __shfl_xor_sync(0xffffffffu, sums[r], o);
        float sum = sums[0];
#pragma unroll
        for (int r = 1; r < 2 * TPW; ++r) sum = lane % (2 * TPW) == r ? sums[r] : sum;
        unit = (lane & 1 ? 1.f : qscale) / sqrtf(sum + 1e-6f);
      }
#pragma unroll
      for (int tt = 0; tt < TPW; ++tt) {
        const int i = lw + tt * (DS_LOADERS / 32);
        if (!AHEAD && i >= n) continue;
        const float iq = AHEAD ? __shfl_sync(0xffffffffu, unit, 2 * tt) : qscale / sqrtf(warp_sum(sums[2 * tt]) + 1e-6f);
        const float ik = AHEAD ? __shfl_sync(0xffffffffu, unit, 2 * tt + 1) : 1.f / sqrtf(warp_sum(sums[2 * tt + 1]) + 1e-6f);
        if (i >= n) continue;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const int d = lane + 32 * j;                       // head row d lies at shared index (d % LANES) * RS + d / LANES
          if (d < LANES * ROWS) {
            const int idx = (d % LANES) * RS + d / LANES;
            qs[i * KW + idx] = qv[tt][j] * iq;               // rows past dim were read as zeros
            ks[i * KW + idx] = kv[tt][j] * ik;
            if constexpr (CHD) {
              const float a1 = av[tt][j];
              gv[i * KW + idx] = expf(neg_rate * (a1 > 20.f ? a1 : log1pf(expf(a1))));
            }
          }
        }
      }
      for (int i = tid - DS_COMPUTE; i < n * COLS; i += DS_LOADERS) {
        const int tk = i / COLS, cc = i % COLS;
        vs[tk * COLS + cc] = c0 + cc < vdim ? qkv[(size_t)(base + tk) * C + (size_t)2 * kvh * dim + (size_t)h * vdim + c0 + cc] : 0.f;
      }
      __threadfence_block();
      named_arrive(1 + (c & 1), DS_THREADS);
    }
    return;
  }
  // -------------------------------------------------- walkers
  const int colb = tid / LANES, seg = tid % LANES;
  const int col = c0 + colb;
  const bool live = col < vdim;
  // this thread's rows of its column: seg, seg + LANES, ... (row r of the thread is row seg + LANES * r of the head), two to a
  // 64-bit register: a multiply-add instruction serves both.
  f32x2 S[ROWS / 2];
  // (the slot keeps a head's matrix column by column, [vdim][dim]: the LANES threads of a column then read neighbours)
  float* mine = state + (size_t)slot * state_stride + ((size_t)h * vdim + col) * dim;
#pragma unroll
  for (int r = 0; r < ROWS; r += 2) {
    const int row = seg + LANES * r;
    S[r / 2] = pack2((live && row < dim) ? mine[row] : 0.f, (live && row + LANES < dim) ? mine[row + LANES] : 0.f);
  }
  float* dst = raw + ((size_t)t0 * heads + h) * vdim + col;
  const long dst_step = (long)heads * vdim;
  const bool writes = seg == 0 && live;
  auto load_rows = [&](const float* rows, int i, f32x2 (&x)[ROWS / 2]) {
    const ulonglong2* x2 = reinterpret_cast<const ulonglong2*>(rows + i * KW + seg * RS);
#pragma unroll
    for (int r = 0; r < ROWS / 4; ++r) {
      const ulonglong2 y = x2[r];
      x[2 * r] = y.x;
      x[2 * r + 1] = y.y;
    }
  };
  auto fold = [](const f32x2 (&a)[2]) {          // four partial sums of a thread
    const float2 a01 = unpack2(a[0]), a23 = unpack2(a[1]);
    return (a01.x + a01.y) + (a23.x + a23.y);
  };
  if constexpr (AHEAD) {
    // A token is a chain: the decay, the dot product with k, its exchange between the column's lanes, the update.  Everything else runs
    // beside that exchange: the read-out of the token before (from the registers that the decay has not replaced), the loads
    // of the next token's rows, and the read-outs' own exchanges, a level a token (o_[e]: a share with e levels done).  Nothing in a
    // token branches: a branch keeps the compiler from putting these between the exchange's steps (448 us instead of 340).  One
    // portion of 2,048 tokens, 16 heads of 128 x 128: 340 us, 379 with the read-out in the chain; portions of 333, 1,055 and 1,777: 446 us,
    // 516 so and in the order of the batch.  The same sums in the same order.
    constexpr int LEVELS = LANES >= 8 ? 3 : (LANES >= 4 ? 2 : (LANES >= 2 ? 1 : 0));
    f32x2 k[ROWS / 2], q[ROWS / 2];
#pragma unroll
    for (int r = 0; r < ROWS / 2; ++r) q[r] = 0ull;
    float o_[LEVELS + 1];
#pragma unroll
    for (int e = 0; e <= LEVELS; ++e) o_[e] = 0.f;
    int at = -(LEVELS + 2);                      // the token whose read-out the next pass completes
    // the tokens' read-outs move on by a level; `share`: this thread's share of the newest
    auto pass_read_outs = [&](float share) {
      float in[LEVELS + 1];
#pragma unroll
      for (int e = 0; e < LEVELS; ++e) in[e] = __shfl_xor_sync(0xffffffffu, o_[e], 1 << e);
      const float done = o_[LEVELS];
#pragma unroll
      for (int e = LEVELS; e > 0; --e) o_[e] = o_[e - 1] + in[e - 1];
      o_[0] = share;
      asm volatile("{\n.reg .pred p;\nsetp.ge.s32 p, %0, 0;\n@p st.global.f32 [%1], %2;\n}\n" ::"r"(writes ? at : -1),
                   "l"(dst + (long)at * dst_step), "f"(done));
      ++at;
    };
    for (int c = 0; c < chunks; ++c) {
      const float* ks = ds_smem + (c & 1) * BUF;
      const float* qs = ks + CH * KW;
      const float* vs = qs + CH * KW;
      const float* gs = vs + CH * COLS;
      const float* bs = gs + CH;
      const float* gv = bs + CH;
      const int n = min(CH, t1 - t0 - c * CH);
      named_sync(1 + (c & 1), DS_THREADS);
      f32x2 gr[CHD ? ROWS / 2 : 1];
      float g = 1.f;
      load_rows(ks, 0, k);
      if constexpr (CHD) load_rows(gv, 0, gr);
      else g = gs[0];
      float beta = bs[0], v = vs[colb];
#pragma unroll 2
      for (int i = 0; i < n; ++i) {
        if constexpr (!CHD) gr[0] = pack2(g, g);
        f32x2 D[ROWS / 2], a[2] = {0ull, 0ull}, y[2] = {0ull, 0ull};
#pragma unroll
        for (int r = 0; r < ROWS / 2; ++r) {
          D[r] = mul2(S[r], gr[CHD ? r : 0]);
          a[r & 1] = fma2(D[r], k[r], a[r & 1]);
        }
        float dot = fold(a);
        const float first = LANES > 1 ? __shfl_xor_sync(0xffffffffu, dot, 1) : 0.f;
#pragma unroll
        for (int r = 0; r < ROWS / 2; ++r) y[r & 1] = fma2(S[r], q[r], y[r & 1]);
        load_rows(qs, i, q);
        // (the last token of a buffer reads its own row again: what follows it comes with the next buffer)
        const int next = min(i + 1, n - 1);
        f32x2 k_next[ROWS / 2];
        load_rows(ks, next, k_next);
        if constexpr (CHD) load_rows(gv, next, gr);
        else g = gs[next];
        const float beta_next = bs[next], v_next = vs[next * COLS + colb];
        if (LANES > 1) dot += first;
        pass_read_outs(fold(y));
#pragma unroll
        for (int o = 2; o < LANES; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        const float u = beta * (v - dot);
        const f32x2 u2 = pack2(u, u);
#pragma unroll
        for (int r = 0; r < ROWS / 2; ++r) {
          S[r] = fma2(k[r], u2, D[r]);
          k[r] = k_next[r];
        }
        beta = beta_next;
        v = v_next;
      }
      if (c + 2 < chunks) named_arrive(3 + (c & 1), DS_THREADS);
    }
    f32x2 y[2] = {0ull, 0ull};
#pragma unroll
    for (int r = 0; r < ROWS / 2; ++r) y[r & 1] = fma2(S[r], q[r], y[r & 1]);
    pass_read_outs(fold(y));
#pragma unroll
    for (int e = 0; e <= LEVELS; ++e) pass_read_outs(0.f);
  } else {
    for (int c = 0; c < chunks; ++c) {
      const float* ks = ds_smem + (c & 1) * BUF;
      const float* qs = ks + CH * KW;
      const float* vs = qs + CH * KW;
      const float* gs = vs + CH * COLS;
      const float* bs = gs + CH;
      const float* gv = bs + CH;
      const int n = min(CH, t1 - t0 - c * CH);
      named_sync(1 + (c & 1), DS_THREADS);
#pragma unroll 1
      for (int i = 0; i < n; ++i) {
        f32x2 k[ROWS / 2], q[ROWS / 2], gr[CHD ? ROWS / 2 : 1];
        load_rows(ks, i, k);
        if constexpr (CHD) load_rows(gv, i, gr);
        else gr[0] = pack2(gs[i], gs[i]);
        f32x2 a[2] = {0ull, 0ull}, y[2] = {0ull, 0ull};
#pragma unroll
        for (int r = 0; r < ROWS / 2; ++r) {
          S[r] = mul2(S[r], gr[CHD ? r : 0]);
          a[r & 1] = fma2(S[r], k[r], a[r & 1]);
        }
        load_rows(qs, i, q);
        float dot = fold(a);
#pragma unroll
        for (int o = 1; o < LANES; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        const float u = bs[i] * (vs[i * COLS + colb] - dot);
        const f32x2 u2 = pack2(u, u);
#pragma unroll
        for (int r = 0; r < ROWS / 2; ++r) {
          S[r] = fma2(k[r], u2, S[r]);
          y[r & 1] = fma2(S[r], q[r], y[r & 1]);
        }
        float o_ = fold(y);
#pragma unroll
        for (int o = 1; o < LANES; o <<= 1) o_ += __shfl_xor_sync(0xffffffffu, o_, o);
        if (writes) *dst = o_;
        dst += dst_step;
      }
      if (c + 2 < chunks) named_arrive(3 + (c & 1), DS_THREADS);
    }
  }
#pragma unroll
  for (int r = 0; r < ROWS; r += 2) {
    const float2 x = unpack2(S[r / 2]);
    const int row = seg + LANES * r;
    if (live && row < dim) mine[row] = x.x;
    if (live && row + LANES < dim) mine[row + LANES] = x.y;
  }
}

// What a head's outputs of a token are multiplied by before their norm: 1, or one over its normaliser.
__device__ __forceinline__ float head_unit(const float* nq, const float4* gates, size_t at) {
  return nq ? 1.f / (fmaxf(fabsf(nq[at]), gates[at].z) + 1e-6f) : 1.f;
}

// out[t, h, :] = raw[t, h, :] / sqrt(mean(raw[t, h, :]^2) + eps) * w * SiLU(gate[t, h, :]); one warp a (token, head).
template <typename T>
__global__ void __launch_bounds__(128)
delta_out_norm_kernel(const float* raw, const T* gate, long gate_stride, const float* __restrict__ w, int w_head, const float* nq,
                      const float4* gates, T* out, int heads, int vdim, float eps, int total, int gate_sigmoid, int wide) {
  pdl_launch_dependents();
  pdl_wait();
  const int idx = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (idx >= total) return;
  const int t = idx / heads, h = idx % heads;
  const float* o = raw + ((size_t)t * heads + h) * vdim;
  const float unit = head_unit(nq, gates, (size_t)idx);
  if (wide) {
    // heads of up to 512 elements that start on 16-byte boundaries: a lane holds its elements, four an access
    const float* gain = w + (size_t)h * w_head;
    const T* grow = gate + (size_t)t * gate_stride + (size_t)h * vdim;
    T* orow = out + ((size_t)t * heads + h) * vdim;
    float x[4][4], g[4][4], ss = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int d = (k * 32 + lane) * 4;
      if (d < vdim) {
        load4(o + d, x[k]);
        load4(grow + d, g[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if ((k * 32 + lane) * 4 < vdim) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          x[k][i] *= unit;
          ss = fmaf(x[k][i], x[k][i], ss);
        }
      }
    const float inv = 1.f / sqrtf(warp_sum(ss) / (float)vdim + eps);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int d = (k * 32 + lane) * 4;
      if (d < vdim) {
        float wv[4], y[4];
        load4(gain + d, wv);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // behind a 16-bit output the hardware's exponential and division (far below its rounding)
          const float e = sizeof(T) == 2 ? __fdividef(1.f, 1.f + __expf(-g[k][i])) : 1.f / (1.f + expf(-g[k][i]));
          y[i] = x[k][i] * inv * wv[i] * (gate_sigmoid ? e : g[k][i] * e);
        }
        store4(orow + d, y);
      }
    }
    return;
  }
  float ss = 0.f;
  for (int d = lane; d < vdim; d += 32) { const float x = o[d] * unit; ss = fmaf(x, x, ss); }
  ss = warp_sum(ss);
  const float inv = 1.f / sqrtf(ss / (float)vdim + eps);
  const float* gain = w + (size_t)h * w_head;
  const T* grow = gate + (size_t)t * gate_stride + (size_t)h * vdim;
  T* orow = out + ((size_t)t * heads + h) * vdim;
  for (int d = lane; d < vdim; d += 32) {
    const float gv = to_f<T>(grow[d]);
    orow[d] = from_f<T>(o[d] * unit * inv * gain[d] * (gate_sigmoid ? 1.f / (1.f + expf(-gv)) : silu_f(gv)));
  }
}

// The same for wide rows (all heads normed as one): a block takes a row.
template <typename T>
__global__ void __launch_bounds__(256)
delta_out_norm_wide_kernel(const float* raw, const T* gate, long gate_stride, const float* __restrict__ w, int w_head,
                           const float* nq, const float4* gates, T* out, int heads, int vdim, float eps, int gate_sigmoid) {
  __shared__ float scratch[32];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x / heads, h = blockIdx.x % heads;
  const float* o = raw + ((size_t)t * heads + h) * vdim;
  const T* grow = gate + (size_t)t * gate_stride + (size_t)h * vdim;
  T* orow = out + ((size_t)t * heads + h) * vdim;
  const float unit = head_unit(nq, gates, (size_t)blockIdx.x);
  const float* gain = w + (size_t)h * w_head;
  float ss = 0.f;
  for (int d = threadIdx.x; d < vdim; d += 256) { const float x = o[d] * unit; ss = fmaf(x, x, ss); }
  const float inv = 1.f / sqrtf(block_sum<256>(ss, scratch) / (float)vdim + eps);
  for (int d = threadIdx.x; d < vdim; d += 256) {
    const float gv = to_f<T>(grow[d]);
    orow[d] = from_f<T>(o[d] * unit * inv * gain[d] * (gate_sigmoid ? 1.f / (1.f + expf(-gv)) : silu_f(gv)));
  }
}

}  // namespace vob

using namespace vob;

// x: rows of x_stride elements of `dtype`, the C channels first; w float [C, taps]; bias_in, bias_out float [C] or null; state
// float [num_slots, state_stride] with the convolutions' part ((taps - 1) x C) at conv_off; out [T, C] float, or of `dtype`
// without `out_float`.
VOB_API int vob_short_conv_silu(const void* x, long x_stride, const float* w, const float* bias_in, const float* bias_out,
                                const float* state, long state_stride, long conv_off, const int* token_req, const int* cu_q,
                                const int* state_slots, void* out, int T, int C, int taps, long num_slots, int act, int out_float,
                                int dtype, int* err, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (C <= 0 || taps < 1 || taps > DELTA_MAX_TAPS) return VOB_UNSUPPORTED;
  const int walk = T >= 32 * CONV_TOKENS ? CONV_TOKENS : 1;      // few tokens (decoding): one each, nothing to slide
  dim3 grid((T + walk - 1) / walk, (C + 127) / 128);
  if (grid.y > 65535) return VOB_UNSUPPORTED;
  const size_t in_size = dtype == VOB_F32 ? 4 : 2, out_size = dtype == VOB_F32 || out_float ? 4 : 2;
  const bool pairs = taps == 4 && walk > 1 && C % 2 == 0 && x_stride % 2 == 0 && (uintptr_t)x % (2 * in_size) == 0 && (uintptr_t)out % (2 * out_size) == 0;
#define VOB_SC(TT, TO)                                                                                                           \
  if (pairs)                                                                                                                     \
    return launch_kernel(short_conv_pairs_kernel<TT, TO>, dim3(grid.x, (C + 255) / 256), 128, 0, stream, (const TT*)x, x_stride, w, bias_in, \
                         bias_out, state, state_stride, conv_off, token_req, cu_q, state_slots, (TO*)out, T, C, num_slots, act, err); \
  if (taps == 4 && walk > 1)                                                                                                     \
    return launch_kernel(short_conv_silu_kernel<TT, TO, true>, grid, 128, 0, stream, (const TT*)x, x_stride, w, bias_in, bias_out, \
                         state, state_stride, conv_off, token_req, cu_q, state_slots, (TO*)out, T, walk, C, taps, num_slots, act, err); \
  return launch_kernel(short_conv_silu_kernel<TT, TO, false>, grid, 128, 0, stream, (const TT*)x, x_stride, w, bias_in, bias_out, \
                       state, state_stride, conv_off, token_req, cu_q, state_slots, (TO*)out, T, walk, C, taps, num_slots, act, err)
  if (dtype == VOB_F32) { VOB_SC(float, float); }
  if (dtype == VOB_BF16) {
    if (out_float) { VOB_SC(__nv_bfloat16, float); }
    VOB_SC(__nv_bfloat16, __nv_bfloat16);
  }
#undef VOB_SC
  return VOB_BAD_ARGUMENT;
}

VOB_API int vob_short_conv_state(const void* x, long x_stride, const float* bias_in, float* state, long state_stride, long conv_off,
                                 const int* cu_q, const int* state_slots, int B, int C, int taps, long num_slots, int dtype,
                                 cudaStream_t stream) {
  if (B <= 0 || taps <= 1) return 0;
  if (C <= 0 || taps > DELTA_MAX_TAPS) return VOB_UNSUPPORTED;
  dim3 grid((C + 127) / 128, B);
  if (dtype == VOB_F32)
    return launch_kernel(short_conv_state_kernel<float>, grid, 128, 0, stream, (const float*)x, x_stride, bias_in, state, state_stride,
                         conv_off, cu_q, state_slots, C, taps, num_slots);
  if (dtype == VOB_BF16)
    return launch_kernel(short_conv_state_kernel<__nv_bfloat16>, grid, 128, 0, stream, (const __nv_bfloat16*)x, x_stride, bias_in,
                         state, state_stride, conv_off, cu_q, state_slots, C, taps, num_slots);
  return VOB_BAD_ARGUMENT;
}

VOB_API int vob_short_conv_step(const void* x, long x_stride, const float* w, const float* bias_in, const float* bias_out, float* state,
                                long state_stride, long conv_off, const int* cu_q, const int* state_slots, void* out, int B, int C,
                                int taps, long num_slots, int act, int out_float, int dtype, int* err, cudaStream_t stream) {
  if (B <= 0) return 0;
  if (C <= 0 || taps < 1 || taps > DELTA_MAX_TAPS || B > 65535) return VOB_UNSUPPORTED;
  dim3 grid((C + 127) / 128, B);
#define VOB_SC(TT, TO)                                                                                                           \
  return launch_kernel(short_conv_step_kernel<TT, TO>, grid, 128, 0, stream, (const TT*)x, x_stride, w, bias_in, bias_out, state, \
                       state_stride, conv_off, cu_q, state_slots, (TO*)out, C, taps, num_slots, act, err)
  if (dtype == VOB_F32) { VOB_SC(float, float); }
  if (dtype == VOB_BF16) {
    if (out_float) { VOB_SC(__nv_bfloat16, float); }
    VOB_SC(__nv_bfloat16, __nv_bfloat16);
  }
#undef VOB_SC
  return VOB_BAD_ARGUMENT;
}

template <typename T>
static int launch_delta_scan(const float* qkv, const void* ab, long ab_stride, int b_off, int a_off, const float* A_log,
                             const float* dt_bias, float* state, long state_stride, const int* cu_q, const int* state_slots,
                             float* raw, long T_all, int B, int heads, int kvh, int dim, int vdim, long num_slots, int channel_decay,
                             int* err, cudaStream_t stream) {
  // rows a thread keeps, and threads a column: the fewest threads whose rows cover the head
  const int rows = dim <= 128 ? 16 : 32;
  const int lanes = dim <= rows ? 1 : (dim <= 2 * rows ? 2 : (dim <= 4 * rows ? 4 : 8));
  // Without AHEAD where more blocks than two an SM have up to eight tokens a request on average (decoding): 64 requests of one token, 16
  // heads of 128 x 128: 59 us, 75 with; of four: 83 and 95; 16 of sixteen: 47 and 44.  (Where fewer blocks have one token each it is the slower
  // one, two requests, 16 heads, a decay a row, one launch behind the other: 5.1 us, 4.3 with.)
  const long blocks = (long)((vdim + DS_COMPUTE / lanes - 1) / (DS_COMPUTE / lanes)) * heads * B;
  const bool ahead = blocks <= 2 * sm_count() || T_all > 8 * (long)B;
#define VOB_DS_LAUNCH(L, R, D, A)                                                                                          \
  do {                                                                                                                     \
    constexpr int cols = DS_COMPUTE / L, ch = R > 16 ? 8 : 16;                                                             \
    dim3 grid((vdim + cols - 1) / cols, heads, B);                                                                         \
    constexpr size_t smem = (size_t)2 * ch * ((D ? 3 : 2) * L * (R + 4) + cols + 2) * sizeof(float);                       \
    if (smem > 48 * 1024)                                                                                                  \
      cudaFuncSetAttribute(delta_scan_kernel<T, L, R, D, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);      \
    return launch_kernel(delta_scan_kernel<T, L, R, D, A>, grid, DS_THREADS, smem, stream, qkv, (const T*)ab, ab_stride,   \
                         b_off, a_off, A_log, dt_bias, state, state_stride, cu_q, state_slots, raw, heads, kvh, dim, vdim, \
                         num_slots, err);                                                                                  \
  } while (0)
#define VOB_DS(L, R)                                                                                                       \
  if (lanes == L && rows == R) {                                                                                           \
    if (channel_decay && ahead) VOB_DS_LAUNCH(L, R, true, true);                                                           \
    if (channel_decay) VOB_DS_LAUNCH(L, R, true, false);                                                                   \
    if (ahead) VOB_DS_LAUNCH(L, R, false, true);                                                                           \
    VOB_DS_LAUNCH(L, R, false, false);                                                                                     \
  }
  VOB_DS(1, 16) VOB_DS(2, 16) VOB_DS(4, 16) VOB_DS(8, 16) VOB_DS(8, 32)
#undef VOB_DS
#undef VOB_DS_LAUNCH
  return VOB_UNSUPPORTED;
}

VOB_API int vob_delta_scan(const float* qkv, const void* ab, long ab_stride, int b_off, int a_off, const float* A_log,
                           const float* dt_bias, float* state, long state_stride, const int* cu_q, const int* state_slots,
                           float* raw, int num_tokens, int B, int heads, int kvh, int dim, int vdim, long num_slots, int channel_decay,
                           int dtype, int* err, cudaStream_t stream) {
  if (B <= 0) return 0;
  if (heads <= 0 || kvh <= 0 || heads % kvh || dim <= 0 || dim > 256 || vdim <= 0 || B > 65535) return VOB_UNSUPPORTED;
  if (dtype == VOB_F32)
    return launch_delta_scan<float>(qkv, ab, ab_stride, b_off, a_off, A_log, dt_bias, state, state_stride, cu_q, state_slots, raw,
                                    num_tokens, B, heads, kvh, dim, vdim, num_slots, channel_decay, err, stream);
  if (dtype == VOB_BF16)
    return launch_delta_scan<__nv_bfloat16>(qkv, ab, ab_stride, b_off, a_off, A_log, dt_bias, state, state_stride, cu_q,
                                            state_slots, raw, num_tokens, B, heads, kvh, dim, vdim, num_slots, channel_decay, err, stream);
  return VOB_BAD_ARGUMENT;
}

// w float [vdim], or [heads * vdim] with w_head = vdim (else 0); nq float [T, heads] and gates float [T, heads, 4], or null.
VOB_API int vob_delta_out_norm(const float* raw, const void* gate, long gate_stride, const float* w, int w_head, const float* nq,
                               const float* gates_, void* out, int T, int heads, int vdim, float eps, int gate_sigmoid, int dtype,
                               cudaStream_t stream) {
  if (T <= 0) return 0;
  const float4* gates = (const float4*)gates_;
  if (nq && (!gates || ((uintptr_t)gates & 15))) return VOB_BAD_ARGUMENT;
  const int total = T * heads;
  if (vdim > 512) {
    if (dtype == VOB_F32)
      return launch_kernel(delta_out_norm_wide_kernel<float>, dim3(total), 256, 0, stream, raw, (const float*)gate, gate_stride, w,
                           w_head, nq, gates, (float*)out, heads, vdim, eps, gate_sigmoid);
    if (dtype == VOB_BF16)
      return launch_kernel(delta_out_norm_wide_kernel<__nv_bfloat16>, dim3(total), 256, 0, stream, raw, (const __nv_bfloat16*)gate,
                           gate_stride, w, w_head, nq, gates, (__nv_bfloat16*)out, heads, vdim, eps, gate_sigmoid);
    return VOB_BAD_ARGUMENT;
  }
  const int wide = vdim % 4 == 0 && gate_stride % 4 == 0 && (((uintptr_t)raw | (uintptr_t)gate | (uintptr_t)w | (uintptr_t)out) & 15) == 0;
  dim3 grid((total + 3) / 4);
  if (dtype == VOB_F32)
    return launch_kernel(delta_out_norm_kernel<float>, grid, 128, 0, stream, raw, (const float*)gate, gate_stride, w,
                         w_head, nq, gates, (float*)out, heads, vdim, eps, total, gate_sigmoid, wide);
  if (dtype == VOB_BF16)
    return launch_kernel(delta_out_norm_kernel<__nv_bfloat16>, grid, 128, 0, stream, raw, (const __nv_bfloat16*)gate,
                         gate_stride, w, w_head, nq, gates, (__nv_bfloat16*)out, heads, vdim, eps, total, gate_sigmoid, wide);
  return VOB_BAD_ARGUMENT;
}
