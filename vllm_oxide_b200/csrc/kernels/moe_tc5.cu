// The experts' products of a mixture of experts for steps of many tokens, in bfloat16 on the fifth-generation tensor
// cores: tcgen05.mma over pairs of SMs with the accumulators in tensor memory.  The same kernel makes the logits of many rows (one
// "expert", no padding).
//
// The step's (token, choice) pairs lie sorted by expert (moe.cu: moe_align), every expert's rows padded to a tile of 128,
// so a row tile belongs to one expert: C[rows of the tile] = f(A[rows] W_e^T) with W stacked [experts * N, K].  The weights are the
// operand of 256 rows: a work item is 256 rows of W_e against the rows of two row tiles of one expert, or of one where the step has
// none to join (tiles 2 i and 2 i + 1 are joined, so one at an odd place whose right neighbour is the same expert's stays alone) or too
// few items for it to pay.  A cluster of two blocks, one per SM, shares an item (cta_group::2): each brings 128 rows of W
// and half of the item's rows, and holds the 128 x 256 accumulators of its rows of W; the tensor cores read the other half of the
// rows from the neighbour's shared memory.  What bounds the product is bringing operands in: an SM brings 32 KB per
// 128 x 256 x 64 products, where blocks of their own with 128 x 128 accumulators brought 32 KB per 128 x 128 x 64.
// B200, 16,004 pairs of 16 experts, 4096 -> 2 x 3072 -> 4096: 689 + 347 us here, 1.17 PFLOP/s; 1,009 + 543 by such blocks.  A sum
// runs along K in order, whatever its item is shared with.
// The blocks are persistent; a warp of each lists the step's items first (which exist is only known on the device), row tile major,
// so that clusters side by side share an expert's matrix in L2.
//   warp 0      producer: per 64 columns of K one TMA copy of the W tile [128 x 64] and one or two of the rows [64 x 64]
//               (128-byte swizzle) into a ring of stages; the bytes of both blocks count on the first block's barrier;
//   warp 1      allocates tensor memory (two accumulators); in the first block it issues the MMAs of the pair: four tcgen05.mma
//               (K = 16 each) per stage; tcgen05.commit hands a stage back to both producers and, after an item's last, the
//               accumulators to both epilogues;
//   warps 2-5   epilogue: tcgen05.ld brings the accumulator to registers (a thread owns one output feature for all rows of
//               the item), applies f (identity into float, the squared relu into bfloat16, or, rows of W in (gate, up)
//               pairs, SiLU(gate) * up into bfloat16 feature / 2: the up value comes from the neighbouring lane; a row's weight,
//               where the weights multiply the experts' inputs, multiplies both) and stores
//               the rows that name a token; the next item's MMAs run meanwhile into the other accumulator.
// Nothing is copied before the wait for the kernels ahead.  Every wait on an mbarrier is bounded; on a timeout the block sets an
// error bit, stops issuing work, and still frees its tensor memory before it returns; the blocks of a cluster leave together.
#define VOB_TIMEOUT_WHERE 0x2000
#include "cluster.cuh"
#include "tcgen05.cuh"

namespace vob {

constexpr int MT_ROWS = 128;      // rows of W a block brings per item (half of the MMA's M)
constexpr int MT_NT = 128;        // rows of a row tile
constexpr int MT_BOX = 64;        // rows of a copy of the sorted rows
constexpr int MT_KC = 64;         // columns of K per stage: one 128-byte swizzle atom
constexpr int MT_THREADS = 192;
constexpr int MT_EPI_WARPS = 4;
constexpr int MT_A_BYTES = MT_ROWS * 128;
constexpr int MT_STAGE_BYTES = MT_A_BYTES + 2 * MT_BOX * 128;
constexpr int MT_S = 6;
constexpr int MT_NUM_BARRIERS = 2 * MT_S + 4;
constexpr int MT_MAX_TILES = 8192;                          // row tiles of a launch: their items are listed in shared memory
constexpr int MT_SMEM = 1024 + MT_S * MT_STAGE_BYTES + MT_NUM_BARRIERS * 8 + 16;      // and two bytes a row tile

enum { MT_EPI_RELU2_BF16 = 0, MT_EPI_F32 = 1, MT_EPI_SILU_PAIRS_BF16 = 2, MT_EPI_F32_OF_BF16 = 3 };

// tmW: W [experts * N, K] as 2-D map with box [128 rows, 64 columns]; tmX: the sorted rows [rows, K], box [64 rows, 64 columns].
// tile_expert: one entry per 64 rows (the sorting kernel's granularity), or null: one expert; row_token: one per row, -1 for
// padding, or null: the first `rows` rows.
template <int EPI>
__global__ void __launch_bounds__(MT_THREADS, 1)
moe_tc5_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, void* out, long ldo,
               const int* row_token, const float* row_weight, const int* tile_expert, int first_tile, int row_tiles, int rows, int N,
               int K, float glu_limit, float pair_cost, int* err) {
  constexpr int S = MT_S, STAGE_BYTES = MT_STAGE_BYTES;
  constexpr int ACC_COLS = 2 * MT_NT, TMEM_COLS = 2 * ACC_COLS;
  extern __shared__ __align__(1024) char smem_raw[];
  char* stages = reinterpret_cast<char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(stages + S * STAGE_BYTES);      // used in the first block only
  uint64_t* empty = full + S;
  uint64_t* acc_full = empty + S;       // [2] MMA -> epilogue
  uint64_t* acc_empty = acc_full + 2;   // [2] both epilogues -> MMA (the first block's)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* num_units = reinterpret_cast<int*>(tmem_slot + 2);
  uint16_t* units = reinterpret_cast<uint16_t*>(tmem_slot + 4);                // row tile * 2 + (with its neighbour)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  const int k_iters = (K + MT_KC - 1) / MT_KC;
  const int n_tiles = (N + 2 * MT_ROWS - 1) / (2 * MT_ROWS);
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 2 * MT_EPI_WARPS); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    tma_prefetch_map(&tmW);
    tma_prefetch_map(&tmX);
  }
  if (warp == 1) t5_alloc_pair(tmem_slot, TMEM_COLS);
  pdl_launch_dependents();
  pdl_wait();                       // which items exist, and the rows themselves, come from the kernels ahead
  auto expert_of = [&](int tile) { return tile >= row_tiles ? -1 : (tile_expert ? tile_expert[(first_tile + tile) * (MT_NT / 64)] : 0); };
  if (warp == 2) {
    // An item of two tiles takes as long as `pair_cost` items of one, so it pays where it saves rounds of items enough: the rounds
    // at the items' mean, the last one at a pair's.
    int live = 0, joined = 0;
    for (int mt = 2 * lane; mt < row_tiles; mt += 64) {
      const int e0 = expert_of(mt), e1 = expert_of(mt + 1);
      live += (e0 >= 0) + (e1 >= 0);
      joined += e0 >= 0 && e1 == e0;
    }
    live = __reduce_add_sync(0xffffffffu, live);
    joined = __reduce_add_sync(0xffffffffu, joined);
    const unsigned clusters = gridDim.x / 2;
    const unsigned rounds = ((unsigned)live * n_tiles + clusters - 1) / clusters, rounds_joined = ((unsigned)(live - joined) * n_tiles + clusters - 1) / clusters;
    const float mean = 1.f + (pair_cost - 1.f) * (float)joined / (float)max(live - joined, 1);
    const bool join = joined > 0 && (float)(rounds_joined - 1) * mean + pair_cost <= (float)rounds;
    int count = 0;
    for (int p0 = 0; 2 * p0 < row_tiles; p0 += 32) {
      const int mt = 2 * (p0 + lane);
      const int e0 = expert_of(mt), e1 = expert_of(mt + 1);
      const bool both = join && e1 == e0;
      const int mine = (e0 >= 0) + (e1 >= 0 && !both);
      int upto = mine;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= d) upto += v;
      }
      int at = count + upto - mine;
      if (e0 >= 0) units[at++] = (uint16_t)(mt * 2 + both);
      if (e1 >= 0 && !both) units[at] = (uint16_t)((mt + 1) * 2);
      count += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (lane == 0) *num_units = count;
  }
  t5_fence_before();
  __syncthreads();
  cluster_sync_all();               // the barriers of both blocks exist, and both have their tensor memory
  t5_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const long total = (long)*num_units * n_tiles;
  const long first_item = blockIdx.x / 2, item_step = gridDim.x / 2;

  if (warp == 0) {
    // ------------------------------------------------ producer (one thread)
    if (lane == 0) {
      long p_it = 0;
      bool ok = true;
      for (long item = first_item; item < total && ok; item += item_step) {
        const int unit = units[item / n_tiles], nt = (int)(item % n_tiles);
        const int mt = unit >> 1, half = (unit & 1) ? 2 : 1;       // copies of 64 rows that are this block's share
        const int w_row = expert_of(mt) * N + (nt * 2 + rank) * MT_ROWS;
        const int x_row = (first_tile + mt) * MT_NT + rank * half * MT_BOX;
        for (int kb = 0; kb < k_iters; ++kb, ++p_it) {
          const int s = (int)(p_it % S);
          if (p_it >= S) {
            ok = mbar_wait(&empty[s], (unsigned)(((p_it / S) - 1) & 1), abort_flag, err);
            if (!ok) break;
          }
          if (rank == 0) mbar_expect_tx(&full[s], (unsigned)(2 * (MT_A_BYTES + half * MT_BOX * 128)));
          const uint32_t bar = map_to_rank(smem_addr(&full[s]), 0);
          char* st = stages + s * STAGE_BYTES;
          tma_load_2d_pair(st, &tmW, kb * MT_KC, w_row, bar);
          tma_load_2d_pair(st + MT_A_BYTES, &tmX, kb * MT_KC, x_row, bar);
          if (half == 2) tma_load_2d_pair(st + MT_A_BYTES + MT_BOX * 128, &tmX, kb * MT_KC, x_row + MT_BOX, bar);
        }
      }
      // copies in flight must land before the blocks exit: the first block sees both blocks' bytes, and they leave together
      if (rank == 0) {
        const long first = p_it > S ? p_it - S : 0;
        for (long j = first; j < p_it; ++j) {
          bool done = false;
          for (unsigned i = 0; i < MBAR_SPIN_LIMIT && !done; ++i) done = mbar_try_wait(&full[j % S], (unsigned)((j / S) & 1));
          if (!done) atomicOr(err, VOB_ERR_TIMEOUT_BITS);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer of the pair (one thread of the first block)
    if (lane == 0 && rank == 0) {
      long it = 0;
      int lt = 0;
      bool ok = true;
      for (long item = first_item; item < total && ok; item += item_step, ++lt) {
        const uint32_t idesc = t5_instr_desc(2 * MT_ROWS, (units[item / n_tiles] & 1) ? 2 * MT_NT : MT_NT);
        const int a = lt & 1;
        if (lt >= 2) {   // both epilogues must have drained this accumulator (two items ago)
          ok = mbar_wait_cluster(&acc_empty[a], (unsigned)(((lt >> 1) - 1) & 1), abort_flag, err);
          if (!ok) break;
          t5_fence_after();
        }
        const uint32_t d_tmem = tmem_base + (uint32_t)(a * ACC_COLS);
        for (int kb = 0; kb < k_iters; ++kb, ++it) {
          const int s = (int)(it % S);
          ok = mbar_wait(&full[s], (unsigned)((it / S) & 1), abort_flag, err);
          if (!ok) break;
          t5_fence_after();
          const char* st = stages + s * STAGE_BYTES;
#pragma unroll
          for (int k = 0; k < MT_KC / 16; ++k)      // 16 columns = 32 bytes further into the swizzle atom
            t5_mma_pair(d_tmem, t5_smem_desc(st + k * 32), t5_smem_desc(st + MT_A_BYTES + k * 32), idesc, (kb | k) ? 1u : 0u);
          t5_commit_pair(&empty[s]);                 // the stage is free in both blocks once these MMAs have read it
        }
        if (ok) t5_commit_pair(&acc_full[a]);        // the accumulators are complete once they have all finished
      }
    }
  } else {
    // ------------------------------------------------ epilogue: warp w reads tensor-memory lanes 32*(w%4) .. +31
    const int q = warp & 3;
    const int row = q * 32 + lane;                                // this thread's row of the block's W tile
    const uint32_t drained = map_to_rank(smem_addr(acc_empty), 0);
    int lt = 0;
    for (long item = first_item; item < total; item += item_step, ++lt) {
      const int unit = units[item / n_tiles], nt = (int)(item % n_tiles);
      const int m0 = (first_tile + (unit >> 1)) * MT_NT, cols = (unit & 1) ? 2 * MT_NT : MT_NT;
      const int a = lt & 1;
      bool ok = mbar_wait(&acc_full[a], (unsigned)((lt >> 1) & 1), abort_flag, err);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      t5_fence_after();
      const long n = (long)(nt * 2 + rank) * MT_ROWS + row;       // one output feature
#pragma unroll 1
      for (int c0 = 0; c0 < cols; c0 += 32) {
        float v[32];
        __syncwarp();
        t5_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * ACC_COLS + c0), v);
        // lane j's entry belongs to column c0 + j
        const int tok = row_token ? row_token[m0 + c0 + lane] : (m0 + c0 + lane < rows ? 0 : -1);
        const float rw = EPI == MT_EPI_SILU_PAIRS_BF16 && row_weight && tok >= 0 ? row_weight[m0 + c0 + lane] : 1.f;
        const unsigned live = __ballot_sync(0xffffffffu, tok >= 0);
        if (live == 0u) continue;
        if (EPI == MT_EPI_SILU_PAIRS_BF16) {
          // Two lanes hold a (gate, up) pair of features.  They finish two token columns at a time, the even lane column
          // j and the odd lane column j + 1, so every lane takes one exponential for two columns and one exchange
          // serves both.
          const bool odd = lane & 1;
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            if (!((live >> j) & 3u)) continue;                    // the same for every lane of the warp
            const float got = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
            const float wt = row_weight ? __shfl_sync(0xffffffffu, rw, odd ? j + 1 : j) : 1.f;
            const float gate = (odd ? got : v[j]) * wt, up = (odd ? v[j + 1] : got) * wt;
            if (((live >> (odd ? j + 1 : j)) & 1u) && (n | 1) < N) {
              const long m = (long)m0 + c0 + j + (odd ? 1 : 0);
              reinterpret_cast<__nv_bfloat16*>(out)[m * ldo + (n >> 1)] =
                  __float2bfloat16_rn(glu_limit > 0.f
                                          ? __fdividef(fminf(gate, glu_limit), 1.f + __expf(-1.702f * fminf(gate, glu_limit))) *
                                                (fminf(fmaxf(up, -glu_limit), glu_limit) + 1.f)
                                          : __fdividef(gate, 1.f + __expf(-gate)) * up);
            }
          }
          continue;
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          if (!((live >> j) & 1u) || n >= N) continue;
          const long m = (long)m0 + c0 + j;
          if (EPI == MT_EPI_F32) {
            reinterpret_cast<float*>(out)[m * ldo + n] = v[j];
          } else if (EPI == MT_EPI_F32_OF_BF16) {
            reinterpret_cast<float*>(out)[m * ldo + n] = __bfloat162float(__float2bfloat16_rn(v[j]));
          } else {
            const float r = fmaxf(v[j], 0.f);
            reinterpret_cast<__nv_bfloat16*>(out)[m * ldo + n] = __float2bfloat16_rn(r * r);
          }
        }
      }
      t5_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(drained + (uint32_t)(a * 8));
    }
  }
  // every path ends here: the blocks of the pair leave together, and the tensor memory goes back before they do
  t5_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    t5_fence_after();
    t5_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// xs[row] = x[row_token[row]] (rows that name no token are left as they are); D a multiple of 8, 16-byte aligned rows.
__global__ void __launch_bounds__(128)
moe_gather_rows_kernel(const __nv_bfloat16* x, long ldx, __nv_bfloat16* xs, const int* row_token, int D) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x;
  const int tok = row_token[row];
  if (tok < 0) return;
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)tok * ldx);
  uint4* dst = reinterpret_cast<uint4*>(xs + (size_t)row * D);
  for (int i = threadIdx.x; i < D / 8; i += 128) dst[i] = src[i];
}

}  // namespace vob

using namespace vob;

VOB_API int vob_moe_tc5_row_tile() { return MT_NT; }

// How many pairs of blocks the device runs at once (a pair sits on neighbouring SMs).
template <typename KERNEL>
static int mt_resident_clusters(KERNEL kernel) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(sm_count() / 2 * 2)); cfg.blockDim = dim3(MT_THREADS); cfg.dynamicSmemBytes = MT_SMEM + 2 * MT_MAX_TILES;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
  return n;
}

// Rows of the box of the sorted rows' tensor map.
VOB_API int vob_moe_tc5_row_box() { return MT_BOX; }

// Whether logits of `rows` rows go by this kernel rather than by the library's product and the pass that turns its bfloat16 into float.
// That pass costs the same for every width while this kernel's product is the slower one (1.1 to 1.2 PFLOP/s against 1.3 to 1.5), more so where the
// last round of items leaves pairs of SMs idle: the wider the matrix, the fuller the rounds must be.  Measured on B200, the library's
// time over this kernel's, at widths of 1,024 / 2,048 / 4,096 / 5,120 / 8,192: 1,024 rows of a vocabulary of 32,768 (97 % full): 2.1, 2.1, 1.4,
// 1.3, 1.0; 384 rows (65 %): 1.4, 1.2, 0.97, 0.94, 0.8; 256 rows of 151,936 (89 %): 2.1, 1.8, 1.4, 1.4, 1.3; 384 (71 %): 1.6, 1.3, 1.03, 0.98,
// 0.9; 1,024 rows of 4,096 (86 %): 1.4, 1.3, 1.2, 1.2, 1.05; 1,357 (59 %): 1.2, 1.04, 0.9, 0.9, 0.8; 256 (22 %): 1.0, 0.8, 0.6, 0.6, 0.5.
VOB_API int vob_logits_by_tc5(int rows, int N, int K) {
  if (rows <= 0 || N <= 0 || K <= 0 || K > 5120) return 0;
  const long pairs = sm_count() / 2, tiles = (rows + MT_NT - 1) / MT_NT, cols = (N + 2 * MT_ROWS - 1) / (2 * MT_ROWS);
  const long rounds = ((tiles / 2 + tiles % 2) * cols + pairs - 1) / pairs;
  const double full = 0.5 * (double)(tiles * cols) / (double)(rounds * pairs);      // (an odd last row tile is half an item's work)
  return full >= (K <= 2048 ? 0.55 : (K <= 4096 ? 0.7 : 0.84)) ? 1 : 0;
}

// map_w: tensor map of W [experts * N, K] with box 128 rows; map_x: tensor map of the sorted rows [max_rows, K] with box
// vob_moe_tc5_row_box() rows (vob_tensor_map_bf16_2d).  out [max_rows, ldo]: bfloat16 with the squared relu (epilogue 0), float (1),
// bfloat16 SiLU(gate) * up over rows of W in (gate, up) pairs (2: N / 2 columns; with glu_limit > 0 the clamped form
// min(gate, limit) * sigmoid(1.702 min(gate, limit)) * (clamp(up, -limit, limit) + 1)), or float rounded to bfloat16 first (3).
// row_weight [max_rows] (epilogue 2) or null: a factor on every row's gate and up.  tile_expert and row_token null: one expert,
// every row counts (max_rows is then any number).
VOB_API int vob_moe_gemm_tc5(const void* map_w, const void* map_x, void* out, long ldo, const int* row_token,
                             const float* row_weight, const int* tile_expert, int max_rows, int N, int K, int epilogue, float glu_limit, int* err,
                             cudaStream_t stream) {
  if (max_rows <= 0 || N <= 0) return 0;
  if (!map_w || !map_x || K <= 0 || K % 8 || (row_weight && epilogue != MT_EPI_SILU_PAIRS_BF16) || !row_token != !tile_expert ||
      (row_token && max_rows % MT_NT))
    return VOB_BAD_ARGUMENT;
  const int all_tiles = (max_rows + MT_NT - 1) / MT_NT;
  // What an item of two row tiles costs in items of one: less than the sum, for the rows of W are brought in once; the activation's
  // epilogue, which hides behind the next item's products, is twice as long and shows at small K.  Measured on B200 over 8, 16 and 64
  // experts and 64 to 4,001 tokens, in us with two tiles an item, with one, and by the rule: SiLU of 3,072 x 2,048, 16 experts, 1,000 tokens of 4
  // choices: 98, 94, 94; 4,001: 228, 279, 228; of 512 x 1,024, 8 experts, 2,048 of 2: 35, 27, 27; of 6,144 x 4,096, 16 experts, 1,000 of 4:
  // 280, 296, 280; no activation, 4,096 x 3,072, 4,001 of 4: 334, 494, 334; 2,048 x 768, 8 experts, 1,000 of 2: 29, 23, 23.
  float pair_cost = 1.2f;
  if (epilogue == MT_EPI_SILU_PAIRS_BF16) pair_cost = 0.8f + 2048.f / (float)K;
  pair_cost = pair_cost < 1.2f ? 1.2f : (pair_cost > 2.f ? 2.f : pair_cost);
#define VOB_MT(EPI)                                                                                                        \
  do {                                                                                                                     \
    static int resident = 0;                                                                                               \
    if (resident < 1) {                                                                                                    \
      cudaError_t e = cudaFuncSetAttribute(moe_tc5_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,               \
                                           MT_SMEM + 2 * MT_MAX_TILES);                                                    \
      if (e != cudaSuccess) return (int)e;                                                                                 \
      resident = mt_resident_clusters(moe_tc5_kernel<EPI>);                                                                \
      if (resident < 1) return VOB_UNSUPPORTED;                                                                            \
    }                                                                                                                      \
    for (int first = 0; first < all_tiles; first += MT_MAX_TILES) {                                                        \
      const int tiles = all_tiles - first < MT_MAX_TILES ? all_tiles - first : MT_MAX_TILES;                               \
      const long most = (long)tiles * ((N + 2 * MT_ROWS - 1) / (2 * MT_ROWS));                                             \
      const int pairs = (int)(most < resident ? most : resident);                                                          \
      const int code = launch_kernel_cluster(moe_tc5_kernel<EPI>, dim3(2 * pairs), MT_THREADS,                             \
                                             MT_SMEM + (2 * tiles + 15) / 16 * 16, stream, 2u, *(const CUtensorMap*)map_w, \
                                             *(const CUtensorMap*)map_x, out, ldo, row_token, row_weight, tile_expert,     \
                                             first, tiles, max_rows, N, K, glu_limit, pair_cost, err);                                \
      if (code != 0) return code;                                                                                          \
    }                                                                                                                      \
    return 0;                                                                                                              \
  } while (0)
  if (epilogue == MT_EPI_RELU2_BF16) VOB_MT(MT_EPI_RELU2_BF16);
  if (epilogue == MT_EPI_F32) VOB_MT(MT_EPI_F32);
  if (epilogue == MT_EPI_SILU_PAIRS_BF16 && N % 2 == 0) VOB_MT(MT_EPI_SILU_PAIRS_BF16);
  if (epilogue == MT_EPI_F32_OF_BF16) VOB_MT(MT_EPI_F32_OF_BF16);
#undef VOB_MT
  return VOB_BAD_ARGUMENT;
}

VOB_API int vob_moe_gather_rows(const void* x, long ldx, void* xs, const int* row_token, int max_rows, int D, cudaStream_t stream) {
  if (max_rows <= 0) return 0;
  if (D % 8 || ((uintptr_t)x | (uintptr_t)xs) % 16 || (ldx * 2) % 16) return VOB_UNSUPPORTED;
  return launch_kernel(moe_gather_rows_kernel, dim3(max_rows), 128, 0, stream, (const __nv_bfloat16*)x, ldx, (__nv_bfloat16*)xs,
                       row_token, D);
}
