// Matrix states with one decay a head and token, 16 tokens at a time on the tensor cores.
//
// Per head a state S [dk, dv] goes S_i = g_i S_{i-1} + put_i k_i v_i^T, o_i = S_i^T q_i.  Over a chunk of 16 tokens, with
// b_i = g_0 .. g_i and D_ij = g_{j+1} .. g_i,
//     o_i = b_i S^T q_i + sum_{j <= i} D_ij put_j (q_i . k_j) v_j,      S' = b_15 S + sum_j D_15,j put_j k_j v_j^T,
// so a token costs a sixteenth of a few contractions, where a walk by multiply-adds touches all of S for every token.  Decays are
// products, never quotients: nothing overflows.
//
// A block takes 32 columns of one head of one request, and what bounds it is the chain from chunk to chunk, so its warps share a
// chunk's work.  Eight computing warps hold S^T in registers, a warp 16 columns and a quarter of the rows, as accumulators of
// mma.m16n8k16: two neighbouring accumulators lie like an A operand, so S never passes through memory.  The four warps of 16
// columns add their shares of S^T q through shared memory, once a chunk; two of them finish 8 tokens each.  Eight loader warps
// prepare the next chunk meanwhile in the other of two buffers, its rows and D put (q . k), and one warp the decays and the normaliser.
//
// Bits.  Everything is held in float, and no result is further from the recurrence in 64 bits than the walk's:
//   * a float enters a product as three bfloat16 slices that add up to it, x = hi + mid + lo.  A product of two slices has 16
//     bits, so the tensor cores' sums, which cut off instead of rounding, are exact for hi hi while the terms lie within some
//     8 bits of each other; the other pairs of slices (down to 2^-25) are summed apart, where what is cut off is 2^-8 of that;
//   * what goes into the state, and the scores, are cut on a grid (hi: multiples of 2^-7 of the largest that is summed): numbers
//     far below that one then leave nothing to cut off;
//   * products of decays carry their rounding errors along (hi + lo), and b_15 multiplies S as such a pair: over a long text
//     nothing drifts.
// Values that are infinite, NaN or not below 2^36 would mix in such sums.  A chunk that holds one is walked token by token in the same
// registers, with the walk's own operations, and so is a share of S with one: a token never reaches another column or an earlier token.
#pragma once
#include "common.cuh"

namespace vob {

constexpr int CS_C = 16, CS_COLS = 32;                 // tokens of a chunk, columns of a block
constexpr int CS_COMPUTE = 256, CS_LOADERS = 256, CS_DECAYS = 32, CS_THREADS = CS_COMPUTE + CS_LOADERS + CS_DECAYS;
constexpr int CS_VS = CS_COLS + 4, CS_TS = CS_C + 4;   // rows in shared memory: a fragment's reads fall into different banks
constexpr float CS_MOST = 68719476736.f;               // 2^36: values that are not below go by multiply-adds (q k v of 2^108 still adds up)
// named barriers: a buffer is full (everyone), a buffer is empty (computing warps and loaders; computing warps and decays), a chunk's
// rows and decays are there (loaders, decays), the shares of 16 columns are there (their computing warps)
enum { CS_FULL = 1, CS_EMPTY = 3, CS_ROWS = 5, CS_SHARES = 6, CS_EMPTY_DECAYS = 8 };

// Offsets (32-bit words) in a buffer, for heads of up to KP rows.  EXACT: q and k are bfloat16 numbers, one slice, else three.
template <int KP, bool EXACT> struct ChunkLayout {
  static constexpr int SLICES = EXACT ? 1 : 3, KS = KP / 2 + 4, SLICE = CS_C * KS;      // a slice: [token][row], two rows a word
  static constexpr int Q = 0, K = Q + SLICES * SLICE, V = K + SLICES * SLICE;            // v: floats
  static constexpr int A = V + CS_C * CS_VS;           // scores D_ij put_j (q_i . k_j), zeros above the diagonal: two halves of the sum over the rows
  static constexpr int D = A + 2 * CS_C * CS_TS;       // D_ij put_j, times the read-out's scale
  static constexpr int PRE = D + CS_C;                 // b_i, times the read-out's scale: column 16 of the rows of D
  static constexpr int END = D + CS_C * CS_TS;         // D_15,j put_j, behind them what is missing from each
  static constexpr int KEEP = END + 2 * CS_C, PUT = KEEP + CS_C;
  static constexpr int ODD = PUT + CS_C;               // a loader warp's word: it has seen a value that is not below CS_MOST
  static constexpr int ALL = ODD + CS_LOADERS / 32;    // b_15, and what is missing from it
  static constexpr int FLOATS = ALL + 4;
  // behind the two buffers: the shares of S^T q, by the chunk's parity, 16 columns, 8 tokens and quarter of the rows
  static constexpr int SHARES = 2 * FLOATS, SHARE = 4 * 32;
  static constexpr int TOTAL = SHARES + 2 * 2 * 2 * 4 * SHARE;
  static_assert(KS % 4 == 0 && FLOATS % 4 == 0 && ODD % 4 == 0 && END % 4 == 0 && D % 4 == 0, "rows and vectors start on 16 bytes");
};

__device__ __forceinline__ void cs_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Four 8 x 8 matrices of 16-bit elements; lane l names row l % 8 of matrix l / 8.
__device__ __forceinline__ void cs_ldmatrix(uint32_t (&r)[4], const float* row) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(row)));
}
__device__ __forceinline__ void cs_ldmatrix_trans(uint32_t (&r)[4], const float* row) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(row)));
}
// The larger magnitude, NaN if one is NaN.
__device__ __forceinline__ float cs_larger(float x, float y) {
  float m;
  asm("max.NaN.f32 %0, %1, %2;\n" : "=f"(m) : "f"(fabsf(x)), "f"(fabsf(y)));
  return m;
}
// Two bfloat16 numbers in a word, the first in the low half.
__device__ __forceinline__ uint32_t cs_pack(float x, float y) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float2 cs_unpack(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
// (x, y) = hi + mid + lo, exactly: 24 bits are 8 + 8 + 8.
__device__ __forceinline__ void cs_slices(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = cs_pack(x, y);
  const float2 h = cs_unpack(hi);
  x -= h.x;
  y -= h.y;
  mid = cs_pack(x, y);
  const float2 m = cs_unpack(mid);
  lo = cs_pack(x - m.x, y - m.y);
}
// The same for values of any size, cut off instead of rounded: an infinity or NaN is hi alone.
__device__ __forceinline__ uint32_t cs_top(float x) { return __float_as_uint(x != x ? __uint_as_float(0x7fff0000u) : x) & 0xffff0000u; }
__device__ __forceinline__ void cs_slices_any(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const uint32_t hx = cs_top(x), hy = cs_top(y);
  const float rx = isfinite(x) ? x - __uint_as_float(hx) : 0.f, ry = isfinite(y) ? y - __uint_as_float(hy) : 0.f;
  const uint32_t mx = cs_top(rx), my = cs_top(ry);
  hi = hx >> 16 | hy;
  mid = mx >> 16 | my;
  lo = cs_top(rx - __uint_as_float(mx)) >> 16 | cs_top(ry - __uint_as_float(my));
}
// (x + rx, y + ry) as slices of which hi lies on the grid of 2^-7 of the power of two in `most` (the largest |x| of those that are summed).
__device__ __forceinline__ void cs_grid_slices(float x, float y, float rx, float ry, float most, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const float shift = __uint_as_float(__float_as_uint(most) & 0x7f800000u) * 98304.f;       // 1.5 * 2^23 steps of 2^-7
  const float hx = (x + shift) - shift, hy = (y + shift) - shift;
  x = (x - hx) + rx;
  y = (y - hy) + ry;
  hi = cs_pack(hx, hy);
  mid = cs_pack(x, y);
  const float2 m = cs_unpack(mid);
  lo = cs_pack(x - m.x, y - m.y);
}
__device__ __forceinline__ float cs_most_of_four(float x) {        // over the lanes of a row of a fragment
  x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
  return fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
}
// Slices of A times slices of B: hi hi into d, all others that matter into x.  A_EXACT, B_EXACT: that operand is its hi slice.  GRID: one
// of the two lies on a grid, its mid slice is up to 2^-8 of its largest, and mid lo counts too.
template <bool A_EXACT, bool B_EXACT, bool GRID>
__device__ __forceinline__ void cs_products(float (&d)[4], float (&x)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2]) {
  cs_mma(d, a[0], b[0][0], b[0][1]);
  if (!A_EXACT) cs_mma(x, a[1], b[0][0], b[0][1]);
  if (!B_EXACT) cs_mma(x, a[0], b[1][0], b[1][1]);
  if (!A_EXACT) cs_mma(x, a[2], b[0][0], b[0][1]);
  if (!B_EXACT) cs_mma(x, a[0], b[2][0], b[2][1]);
  if (!A_EXACT && !B_EXACT) {
    cs_mma(x, a[1], b[1][0], b[1][1]);
    if (GRID) {
      cs_mma(x, a[2], b[1][0], b[1][1]);
      cs_mma(x, a[1], b[2][0], b[2][1]);
    }
  }
}

// A SOURCE gives, for token t of the step and head h: q_raw, k_raw (row d) and v_raw (column c) as stored, act (what becomes of
// them), gate_raw and gates (g and put).  EXACT: q, k and v are bfloat16 numbers.  NORMALISER: a further column whose v is 1, read
// out into nq [tokens, heads], its state behind all heads' matrices, [heads, dk].
template <class SRC, int KP>
__global__ void __launch_bounds__(CS_THREADS, 1)
chunk_scan_kernel(const SRC src, float* state, long state_stride, const int* __restrict__ cu_q, const int* __restrict__ state_slots,
                  float* raw, int heads, int dk, int dv, long num_slots, int* err) {
  constexpr bool EXACT = SRC::EXACT;
  using LO = ChunkLayout<KP, EXACT>;
  constexpr int KS = LO::KS, SLICES = LO::SLICES, HK = KP / 4, NT = HK / 8, NV = KP / 32;
  static_assert(EXACT || !SRC::NORMALISER, "the normaliser's walk reads rows that lie as they are");
  extern __shared__ float4 sm4[];
  float* sm = reinterpret_cast<float*>(sm4);
  pdl_launch_dependents();
  // (requests from the last to the first: prompts commonly stand behind the requests that decode, and the longest should start early)
  const int h = blockIdx.y, b = gridDim.z - 1 - blockIdx.z, c0 = blockIdx.x * CS_COLS;
  const int t0 = cu_q[b], t1 = cu_q[b + 1], slot = state_slots[b];
  const int chunks = (t1 - t0 + CS_C - 1) / CS_C;
  const typename SRC::Fixed fx = src.fixed(h);
  const float scale = src.out_scale();
  pdl_wait();
  if (t1 <= t0) return;
  if (slot < 0 || slot >= num_slots) {
    if (threadIdx.x == 0) atomicOr(err, VOB_ERR_SLOT);
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  float* mine = state + (size_t)slot * state_stride + (size_t)h * dk * dv + c0;                       // [dk] rows dv apart
  float* norm = state + (size_t)slot * state_stride + (size_t)heads * dk * dv + (size_t)h * dk;       // [dk]
  const bool norm_here = SRC::NORMALISER && blockIdx.x == 0;
  if (t1 - t0 == 1) {
    // ------------------------------------------------ a single token (a request that decodes beside portions): one pass over the state
    constexpr int WARPS = CS_THREADS / 32;
    float* qs = sm;                                     // [KP], behind it k, then partial sums [WARPS][32]
    for (int i = threadIdx.x; i < 2 * KP; i += CS_THREADS) {
      const int d = i % KP;
      qs[i] = d < dk ? src.act(to_f(i < KP ? src.q_raw((size_t)t0, h, d) : src.k_raw((size_t)t0, h, d))) : 0.f;
    }
    const float2 gt = src.gates(src.gate_raw((size_t)t0, h), fx);
    const float v = c0 + lane < dv ? src.act(to_f(src.v_raw((size_t)t0, h, c0 + lane))) : 0.f;
    __syncthreads();
    float o = 0.f;
    if (c0 + lane < dv) {
#pragma unroll 8
      for (int row = warp; row < dk; row += WARPS) {
        const float S = fmaf(gt.x, mine[(size_t)row * dv + lane], qs[KP + row] * gt.y * v);
        mine[(size_t)row * dv + lane] = S;
        o = fmaf(S, qs[row], o);
      }
    }
    float* part = sm + 2 * KP;
    part[warp * 32 + lane] = o;
    if constexpr (SRC::NORMALISER) {
      if (norm_here && warp == WARPS - 1) {
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const int d = lane + 32 * j;
          if (d < dk) {
            const float x = fmaf(gt.x, norm[d], qs[KP + d] * gt.y);
            norm[d] = x;
            s = fmaf(x, qs[d], s);
          }
        }
        s = warp_sum(s);
        if (lane == 0) src.nq[(size_t)t0 * heads + h] = s * scale;
      }
    }
    __syncthreads();
    if (warp == 0 && c0 + lane < dv) {
      o = 0.f;
#pragma unroll
      for (int k = 0; k < WARPS; ++k) o += part[k * 32 + lane];
      raw[((size_t)t0 * heads + h) * dv + c0 + lane] = o * scale;
    }
    return;
  }
  if (threadIdx.x >= CS_COMPUTE + CS_LOADERS) {
    // ------------------------------------------------ decays and normaliser
    auto gates_of = [&](const typename SRC::GateRaw& r, int c) {
      return lane < min(CS_C, t1 - t0 - c * CS_C) ? src.gates(r, fx) : make_float2(1.f, 0.f);
    };
    float2 gt = gates_of(src.gate_raw((size_t)min(t0 + lane, t1 - 1), h), 0);
    constexpr int NE = KP / 32;                         // a lane holds elements 2 * lane, 2 * lane + 1 of every 64 of the normaliser
    float n4[NE];
    auto element = [&](int e) { return 64 * (e / 2) + 2 * lane + (e & 1); };
    if constexpr (SRC::NORMALISER) {
#pragma unroll
      for (int e = 0; e < NE; ++e) n4[e] = norm_here && element(e) < dk ? norm[element(e)] : 0.f;
    }
    for (int c = 0; c < chunks; ++c) {
      float* bf = sm + (c & 1) * LO::FLOATS;
      const typename SRC::GateRaw next = src.gate_raw((size_t)min(t0 + (c + 1) * CS_C + lane, t1 - 1), h);
      if (c >= 2) named_sync(CS_EMPTY_DECAYS + (c & 1), CS_COMPUTE + CS_DECAYS);
      // lane j < 16: D_ij down its column; lane 16: the products b_i; both with their rounding errors beside them
      float run = 1.f, rest = 0.f;
      const float factor = lane == CS_C ? scale : gt.y * scale;
#pragma unroll
      for (int i = 0; i < CS_C; ++i) {
        const float keep = __shfl_sync(0xffffffffu, gt.x, i), mine_too = lane < i || lane == CS_C ? keep : 1.f;
        const float next_run = run * mine_too;
        rest = fmaf(rest, mine_too, fmaf(run, mine_too, -next_run));
        run = next_run;
        if (lane <= CS_C) bf[LO::D + i * CS_TS + lane] = fmaf(run, factor, rest * factor);
      }
      if (lane < CS_C) {
        const float end = run * gt.y;
        bf[LO::END + lane] = end;
        bf[LO::END + CS_C + lane] = fmaf(rest, gt.y, fmaf(run, gt.y, -end));
        bf[LO::KEEP + lane] = gt.x;
        bf[LO::PUT + lane] = gt.y;
      }
      if (lane == CS_C) {
        const float all = run + rest;
        bf[LO::ALL] = all;
        bf[LO::ALL + 1] = rest - (all - run);
      }
      __threadfence_block();
      named_sync(CS_ROWS, CS_LOADERS + CS_DECAYS);      // (waited for, not only told: two chunks' arrivals must not meet)
      named_arrive(CS_FULL + (c & 1), CS_THREADS);
      // (the normaliser's reads of this buffer end before the next chunk's rows are told, and the loaders come back to it after that)
      if constexpr (SRC::NORMALISER) {
        if (norm_here) {
          float dots[CS_C];
#pragma unroll
          for (int i = 0; i < CS_C; ++i) {
            const float keep = __shfl_sync(0xffffffffu, gt.x, i), put = __shfl_sync(0xffffffffu, gt.y, i);
            float q[NE], k[NE];
#pragma unroll
            for (int e = 0; e < NE; e += 2) {
              const float2 q2 = cs_unpack(__float_as_uint(bf[LO::Q + i * KS + 32 * (e / 2) + lane]));
              const float2 k2 = cs_unpack(__float_as_uint(bf[LO::K + i * KS + 32 * (e / 2) + lane]));
              q[e] = q2.x; q[e + 1] = q2.y; k[e] = k2.x; k[e + 1] = k2.y;
            }
            dots[i] = 0.f;
#pragma unroll
            for (int e = 0; e < NE; ++e) {
              n4[e] = fmaf(keep, n4[e], k[e] * put);
              dots[i] = fmaf(n4[e], q[e], dots[i]);
            }
          }
          // sixteen sums over the lanes: every exchange halves the tokens a lane still sums
#pragma unroll
          for (int w = CS_C / 2; w > 0; w >>= 1) {
            const bool upper = lane & w;
#pragma unroll
            for (int i = 0; i < CS_C / 2; ++i)
              if (i < w) {
                const float give = upper ? dots[i] : dots[i + w], keep = upper ? dots[i + w] : dots[i];
                dots[i] = keep + __shfl_xor_sync(0xffffffffu, give, w);
              }
          }
          dots[0] += __shfl_xor_sync(0xffffffffu, dots[0], CS_C);
          // (lane bits 8, 4, 2, 1 chose the token's halves in that order)
          const int tok = lane & (CS_C - 1);
          if (lane < CS_C && t0 + c * CS_C + tok < t1) src.nq[(size_t)(t0 + c * CS_C + tok) * heads + h] = dots[0] * scale;
        }
      }
      if (c + 1 < chunks) gt = gates_of(next, c + 1);
    }
    if constexpr (SRC::NORMALISER) {
#pragma unroll
      for (int e = 0; e < NE; ++e)
        if (norm_here && element(e) < dk) norm[element(e)] = n4[e];
    }
    return;
  }
  if (threadIdx.x >= CS_COMPUTE) {
    // ------------------------------------------------ loaders
    const int lw = (threadIdx.x - CS_COMPUTE) >> 5;
    constexpr int STEP = CS_LOADERS / 32, TPW = CS_C / STEP;       // a warp takes tokens lw, lw + STEP, ...
    // (as stored and from clamped places: a load that is used at once, or that a branch guards, waits for memory by itself)
    typename SRC::Raw qv[TPW][NV], kv[TPW][NV], vv[TPW];
    auto fetch = [&](int c) {
      const int base = t0 + c * CS_C, n = min(CS_C, t1 - base);
#pragma unroll
      for (int tt = 0; tt < TPW; ++tt) {
        const size_t at = (size_t)(base + min(lw + STEP * tt, n - 1));
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const int d = min(2 * lane + 64 * (j >> 1) + (j & 1), dk - 1);      // neighbouring rows share a word
          qv[tt][j] = src.q_raw(at, h, d);
          kv[tt][j] = src.k_raw(at, h, d);
        }
        vv[tt] = src.v_raw(at, h, min(c0 + lane, dv - 1));
      }
    };
    fetch(0);
    const bool v_live = c0 + lane < dv;
    for (int c = 0; c < chunks; ++c) {
      float* bf = sm + (c & 1) * LO::FLOATS;
      const int n = min(CS_C, t1 - t0 - c * CS_C);
      if (c >= 2) named_sync(CS_EMPTY + (c & 1), CS_COMPUTE + CS_LOADERS);
      bool odd = false;
#pragma unroll
      for (int tt = 0; tt < TPW; ++tt) {
        const int i = lw + STEP * tt;
        uint32_t* qd = reinterpret_cast<uint32_t*>(bf) + LO::Q + i * KS + lane;
        uint32_t* kd = reinterpret_cast<uint32_t*>(bf) + LO::K + i * KS + lane;
        float x[2 * NV], most = 0.f;                       // q's and k's rows, two by two
#pragma unroll
        for (int e = 0; e < 2 * NV; ++e) {
          const int j = (e >> 2) * 2 + (e & 1);
          x[e] = i < n && 2 * lane + 32 * (j & ~1) + (j & 1) < dk ? src.act(to_f(e & 2 ? kv[tt][j] : qv[tt][j])) : 0.f;
          most = cs_larger(most, x[e]);
        }
        const bool usual = most < CS_MOST;
#pragma unroll
        for (int e = 0; e < 2 * NV; e += 2) {
          uint32_t s[3];
          if (EXACT) s[0] = cs_pack(x[e], x[e + 1]);
          else if (usual) cs_slices(x[e], x[e + 1], s[0], s[1], s[2]);
          else cs_slices_any(x[e], x[e + 1], s[0], s[1], s[2]);
#pragma unroll
          for (int p = 0; p < SLICES; ++p) (e & 2 ? kd : qd)[p * LO::SLICE + 32 * (e >> 2)] = s[p];
        }
        const float v = i < n && v_live ? src.act(to_f(vv[tt])) : 0.f;
        odd |= !(cs_larger(most, v) < CS_MOST);
        bf[LO::V + i * CS_VS + lane] = v;
      }
      odd = __any_sync(0xffffffffu, odd);
      if (lane == 0) bf[LO::ODD + lw] = __int_as_float(odd ? 1 : 0);
      if (c + 1 < chunks) fetch(c + 1);
      named_sync(CS_ROWS, CS_LOADERS + CS_DECAYS);
      // scores: a warp of the first four takes 8 of the chunk's k and half of the rows
      if (lw < 4) {
        const int nt = lw >> 1, kh = lw & 1;
        constexpr int NK = KP / 32;                       // steps of 16 rows
        float acc[NK][4] = {}, small[4] = {};
        const float* qr = bf + LO::Q + ((lane & 7) + ((lane >> 3) & 1) * 8) * KS + kh * (KP / 4) + (lane >> 4) * 4;
        const float* kr = bf + LO::K + (nt * 8 + (lane & 7)) * KS + kh * (KP / 4) + (lane >> 3) * 4;
#pragma unroll
        for (int ks = 0; ks < NK; ks += 2) {
          uint32_t b4[3][4];
#pragma unroll
          for (int p = 0; p < SLICES; ++p) cs_ldmatrix(b4[p], kr + p * LO::SLICE + ks * 8);
#pragma unroll
          for (int two = 0; two < 2; ++two) {
            uint32_t a[3][4], b[3][2];
#pragma unroll
            for (int p = 0; p < SLICES; ++p) {
              cs_ldmatrix(a[p], qr + p * LO::SLICE + (ks + two) * 8);
              b[p][0] = b4[p][2 * two];
              b[p][1] = b4[p][2 * two + 1];
            }
            cs_products<EXACT, EXACT, false>(acc[ks + two], small, a, b);
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = g + (e >> 1) * 8, j = nt * 8 + 2 * t + (e & 1);
          float dot = acc[0][e] + acc[1][e];
          if constexpr (NK == 4) dot += acc[2][e] + acc[3][e];
          if (!EXACT) dot += small[e];
          bf[LO::A + (kh * CS_C + i) * CS_TS + j] = j <= i ? dot * bf[LO::D + i * CS_TS + j] : 0.f;
        }
      }
      __threadfence_block();
      named_arrive(CS_FULL + (c & 1), CS_THREADS);
    }
    return;
  }
  // -------------------------------------------------- computing warps: S^T, 16 columns x a quarter of the rows
  const int ct = warp >> 2, part = warp & 3, d0 = part * HK;
  const int col = ct * 16 + g;                            // this thread's columns: col, col + 8
  float S[NT][4];
#pragma unroll
  for (int k = 0; k < NT; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = d0 + k * 8 + 2 * t + (e & 1), j = col + (e >> 1) * 8;
      S[k][e] = row < dk && c0 + j < dv ? mine[(size_t)row * dv + j] : 0.f;
    }
  auto odd_share = [&]() {                              // (the same for the warp)
    float most[4] = {};
#pragma unroll
    for (int k = 0; k < NT; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) most[e] = cs_larger(most[e], S[k][e]);
    return __any_sync(0xffffffffu, !(cs_larger(cs_larger(most[0], most[1]), cs_larger(most[2], most[3])) < CS_MOST)) != 0;
  };
  bool share_is_odd = odd_share();
  for (int c = 0; c < chunks; ++c) {
    const float* bf = sm + (c & 1) * LO::FLOATS;
    const int base = t0 + c * CS_C, n = min(CS_C, t1 - base);
    float* shares = sm + LO::SHARES + ((c & 1) * 2 + ct) * (2 * 4 * LO::SHARE) + lane;
    // the chunk's tokens one after the other by multiply-adds, as the walk: S updated by them, S^T q of this warp's rows read out, or both
    auto walk = [&](bool update, bool read) {
      auto element = [&](int at, int i, int row) {
        float x = 0.f;
#pragma unroll
        for (int p = SLICES - 1; p >= 0; --p) {
          const float2 two = cs_unpack(__float_as_uint(bf[at + p * LO::SLICE + i * KS + (row >> 1)]));
          x += row & 1 ? two.y : two.x;
        }
        return x;
      };
#pragma unroll 1
      for (int i = 0; i < n; ++i) {
        const float keep = bf[LO::KEEP + i], put = bf[LO::PUT + i], v[2] = {bf[LO::V + i * CS_VS + col], bf[LO::V + i * CS_VS + col + 8]};
        float o[2] = {0.f, 0.f};
#pragma unroll
        for (int k = 0; k < NT; ++k)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int row = d0 + k * 8 + 2 * t + (e & 1);
            if (row >= dk) continue;
            if (update) S[k][e] = fmaf(keep, S[k][e], element(LO::K, i, row) * put * v[e >> 1]);
            if (read) o[e >> 1] = fmaf(S[k][e], element(LO::Q, i, row), o[e >> 1]);
          }
        if (!read) continue;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          o[half] += __shfl_xor_sync(0xffffffffu, o[half], 1);
          o[half] += __shfl_xor_sync(0xffffffffu, o[half], 2);
          if (t == (i & 7) >> 1) shares[((i >> 3) * 4 + part) * LO::SHARE + ((i & 1) + 2 * half) * 32] = o[half];
        }
      }
    };
    named_sync(CS_FULL + (c & 1), CS_THREADS);
    const uint4 odd0 = *reinterpret_cast<const uint4*>(bf + LO::ODD), odd1 = *reinterpret_cast<const uint4*>(bf + LO::ODD + 4);
    const bool odd = (odd0.x | odd0.y | odd0.z | odd0.w | odd1.x | odd1.y | odd1.z | odd1.w) != 0;      // (the same for the block)
    // v^T as an A operand: tokens 2t, 2t + 1 of columns col and col + 8, then tokens 2t + 8, 2t + 9
    const float* vs = bf + LO::V + col;
    float U[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int e = 0; e < 2; ++e) U[r][e] = vs[(2 * t + e + (r >> 1) * 8) * CS_VS + (r & 1) * 8];
    if (odd || share_is_odd) {
      walk(odd, true);
    } else {
      // S^T q over this warp's rows: [16 columns] x [16 tokens]
      float O[2][NT / 2][4] = {}, Ox[2][4] = {};
      const float* qr = bf + LO::Q + ((lane & 7) + (lane >> 4) * 8) * KS + d0 / 2 + ((lane >> 3) & 1) * 4;
#pragma unroll
      for (int ks = 0; ks < NT / 2; ++ks) {
        uint32_t a[3][4], b4[3][4];
#pragma unroll
        for (int r = 0; r < 4; ++r) cs_slices(S[2 * ks + (r >> 1)][2 * (r & 1)], S[2 * ks + (r >> 1)][2 * (r & 1) + 1], a[0][r], a[1][r], a[2][r]);
#pragma unroll
        for (int p = 0; p < SLICES; ++p) cs_ldmatrix(b4[p], qr + p * LO::SLICE + ks * 8);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          uint32_t b[3][2];
#pragma unroll
          for (int p = 0; p < SLICES; ++p) {
            b[p][0] = b4[p][2 * m];
            b[p][1] = b4[p][2 * m + 1];
          }
          cs_products<false, EXACT, false>(O[m][ks], Ox[m], a, b);
        }
      }
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float o = O[m][0][e] + Ox[m][e];
          if (NT == 4) o += O[m][NT / 2 - 1][e];
          shares[(m * 4 + part) * LO::SHARE + e * 32] = o;
        }
    }
    // S = b_15 S + sum_j D_15,j put_j k_j v_j^T
    if (!odd && share_is_odd) {
      walk(true, false);
    } else if (!odd) {
      uint32_t u[3][4];
      {
        const float* end = bf + LO::END + 2 * t;
        const float2 e[2] = {*reinterpret_cast<const float2*>(end), *reinterpret_cast<const float2*>(end + 8)};
        const float2 r[2] = {*reinterpret_cast<const float2*>(end + CS_C), *reinterpret_cast<const float2*>(end + CS_C + 8)};
        float w[4][2], rest[4][2], most[2];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          w[k][0] = U[k][0] * e[k >> 1].x;
          w[k][1] = U[k][1] * e[k >> 1].y;
          rest[k][0] = fmaf(U[k][0], r[k >> 1].x, fmaf(U[k][0], e[k >> 1].x, -w[k][0]));
          rest[k][1] = fmaf(U[k][1], r[k >> 1].y, fmaf(U[k][1], e[k >> 1].y, -w[k][1]));
        }
#pragma unroll
        for (int half = 0; half < 2; ++half)
          most[half] = cs_most_of_four(fmaxf(fmaxf(fabsf(w[half][0]), fabsf(w[half][1])), fmaxf(fabsf(w[half + 2][0]), fabsf(w[half + 2][1]))));
#pragma unroll
        for (int k = 0; k < 4; ++k) cs_grid_slices(w[k][0], w[k][1], rest[k][0], rest[k][1], most[k & 1], u[0][k], u[1][k], u[2][k]);
      }
      const float all = bf[LO::ALL], all_rest = bf[LO::ALL + 1];
      const float* kr = bf + LO::K + ((lane & 7) + ((lane >> 3) & 1) * 8) * KS + d0 / 2 + (lane >> 4) * 4;
#pragma unroll
      for (int k = 0; k < NT; k += 2) {
        uint32_t b4[3][4];
#pragma unroll
        for (int p = 0; p < SLICES; ++p) cs_ldmatrix_trans(b4[p], kr + p * LO::SLICE + k * 4);
#pragma unroll
        for (int two = 0; two < 2; ++two) {
          uint32_t b[3][2];
#pragma unroll
          for (int p = 0; p < SLICES; ++p) {
            b[p][0] = b4[p][2 * two];
            b[p][1] = b4[p][2 * two + 1];
          }
          float acc[4] = {}, x[4] = {};
          cs_products<false, EXACT, true>(acc, x, u, b);
#pragma unroll
          for (int e = 0; e < 4; ++e) S[k + two][e] = acc[e] + fmaf(all, S[k + two][e], fmaf(all_rest, S[k + two][e], x[e]));
        }
      }
    }
    share_is_odd = odd_share();
    // o = b S^T q + sum_j A_ij v_j: warps 0 and 1 of the four finish tokens 8 part + 2t, + 1, the others only hand their shares in
    if (part >= 2) {
      __threadfence_block();
      named_arrive(CS_SHARES + ct, 128);
    } else {
      named_sync(CS_SHARES + ct, 128);
      float acc[4] = {}, x[4] = {};
      if (!odd) {
        uint32_t a[3][4], b[3][2];
        float w[2][2];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          if (EXACT) a[0][r] = cs_pack(U[r][0], U[r][1]);
          else cs_slices(U[r][0], U[r][1], a[0][r], a[1][r], a[2][r]);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float* at = bf + LO::A + (part * 8 + g) * CS_TS + r * 8 + 2 * t;
          const float2 a0 = *reinterpret_cast<const float2*>(at), a1 = *reinterpret_cast<const float2*>(at + CS_C * CS_TS);
          w[r][0] = a0.x + a1.x;
          w[r][1] = a0.y + a1.y;
        }
        const float most = cs_most_of_four(fmaxf(fmaxf(fabsf(w[0][0]), fabsf(w[0][1])), fmaxf(fabsf(w[1][0]), fabsf(w[1][1]))));
#pragma unroll
        for (int r = 0; r < 2; ++r) cs_grid_slices(w[r][0], w[r][1], 0.f, 0.f, most, b[0][r], b[1][r], b[2][r]);
        cs_products<EXACT, false, true>(acc, x, a, b);
      }
      const float* sh = shares + part * 4 * LO::SHARE;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int tok = part * 8 + 2 * t + (e & 1), j = col + (e >> 1) * 8;
        const float o = (sh[e * 32] + sh[LO::SHARE + e * 32]) + (sh[2 * LO::SHARE + e * 32] + sh[3 * LO::SHARE + e * 32]);
        const float y = odd ? o * scale : fmaf(bf[LO::PRE + tok * CS_TS], o, acc[e] + x[e]);
        if (tok < n && c0 + j < dv) raw[((size_t)(base + tok) * heads + h) * dv + c0 + j] = y;
      }
    }
    if (c + 2 < chunks) {
      named_arrive(CS_EMPTY + (c & 1), CS_COMPUTE + CS_LOADERS);
      named_arrive(CS_EMPTY_DECAYS + (c & 1), CS_COMPUTE + CS_DECAYS);
    }
  }
#pragma unroll
  for (int k = 0; k < NT; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = d0 + k * 8 + 2 * t + (e & 1), j = col + (e >> 1) * 8;
      if (row < dk && c0 + j < dv) mine[(size_t)row * dv + j] = S[k][e];
    }
}

inline bool chunk_scan_takes(int dk, int dv, int heads, int B) { return dk > 0 && dk <= 128 && dv > 0 && heads > 0 && heads <= 65535 && B <= 65535; }

template <class SRC, int KP>
int launch_chunk_scan(const SRC& src, float* state, long state_stride, const int* cu_q, const int* state_slots, float* raw, int B,
                      int heads, int dk, int dv, long num_slots, int* err, cudaStream_t stream) {
  constexpr int smem = ChunkLayout<KP, SRC::EXACT>::TOTAL * (int)sizeof(float);
  static_assert(ChunkLayout<KP, SRC::EXACT>::TOTAL >= 2 * KP + CS_THREADS, "a single token's sums fit");
  cudaError_t e = cudaFuncSetAttribute(chunk_scan_kernel<SRC, KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  return launch_kernel(chunk_scan_kernel<SRC, KP>, dim3((dv + CS_COLS - 1) / CS_COLS, heads, B), dim3(CS_THREADS), smem, stream,
                       src, state, state_stride, cu_q, state_slots, raw, heads, dk, dv, num_slots, err);
}

template <class SRC>
int run_chunk_scan(const SRC& src, float* state, long state_stride, const int* cu_q, const int* state_slots, float* raw, int B,
                   int heads, int dk, int dv, long num_slots, int* err, cudaStream_t stream) {
  if (!chunk_scan_takes(dk, dv, heads, B)) return VOB_UNSUPPORTED;
  if (dk <= 64) return launch_chunk_scan<SRC, 64>(src, state, state_stride, cu_q, state_slots, raw, B, heads, dk, dv, num_slots, err, stream);
  return launch_chunk_scan<SRC, 128>(src, state, state_stride, cu_q, state_slots, raw, B, heads, dk, dv, num_slots, err, stream);
}

}  // namespace vob
