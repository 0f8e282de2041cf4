// The routed experts' products on the tensor cores (bfloat16): tcgen05.mma with the accumulator in
// tensor memory, operands by TMA, as the dense product kernel (gemm_tc.cu) does it, for rows that are
// grouped by expert ON THE DEVICE.
//
// Rows of all (token, choice) pairs lie ordered by expert in one matrix; offsets[e] .. offsets[e + 1]
// is expert e's range, known to the device only.  So the launch covers the most row tiles any routing
// can produce, and every CTA finds its (expert, first row) from the offsets; a CTA beyond the last
// tile returns.  One tensor map covers all rows and one the stacked weights of all experts
// [E * rows_per_expert, K]: a tile of token rows may start at any row (TMA's alignment rule is about
// the innermost coordinate only) and may run into the next expert's rows or weights; what it computes
// for those is not stored.
//
// The weight is the M side of the MMA (128 weight rows per tile, one accumulator lane each), the
// token rows the N side (BN per tile), as in gemm_tc.cu.  Three epilogues:
//   plain   out[row, n] = acc            (32-bit; the experts' down projections)
//   unit    act[row, n] = function(acc)  (bfloat16; the first product of experts without a gate)
//   GLU     act[row, f] = g' sigmoid(alpha g') (u' + up_add), g' = min(g, limit), u' = clamp(u, +-limit),
//           for weights whose rows alternate in blocks of 64 between gate and up of the same 64 features
//           (lanes 0-63 of a tile hold g, lanes 64-127 u).
#include <stdlib.h>

#include <mutex>
#include <unordered_map>

#include "hybrid.cuh"
#include "sm100.cuh"

namespace {

using namespace sm100;

constexpr int BM = 128, BK = 64, UMMA_K = 16;
// (stages: as many as leave room for two blocks an SM; narrow tiles with four leave room for three, which launches of more blocks than two an SM
// need: us with six and with four, 32 experts, 128 rows of 512 x 2 x 2,048 33.5 and 27.9, 32 rows of 2,048 x 2 x 1,024 37.8 and 32.6; 8 rows of these 12.9 and
// 14.4)
template <int BN> constexpr int stages_of() { return BN <= 64 ? 4 : 3; }
constexpr int FEW_STAGES = 6;
constexpr int W_TILE_BYTES = BM * BK * 2;
constexpr int STATUS_TIMEOUT = 24;

struct GroupedParams {
  const int* offsets;
  int E, rows_per_expert, n_valid;   // weight rows per expert in the stacked matrix; rows that exist per expert
  int mode;                          // 0 GLU, 1 plain, 2 a function of the sums
  int fn;                            // (mode 2) the function's number
  void* out; long long ldo;
  int total_kb;
  float alpha, limit, up_add;
  int* status;
};

__device__ __forceinline__ void epilogue_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

template <int BN, int STAGES>
__global__ void __launch_bounds__(192)
moe_experts_tc_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                      const GroupedParams p) {
  constexpr int X_TILE_BYTES = BN * BK * 2, STAGE_BYTES = W_TILE_BYTES + X_TILE_BYTES;
  constexpr int TMEM_COLS = BN < 32 ? 32 : BN;
  pdl_trigger();
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], tmem_full_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nkb = p.total_kb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&tmem_full_bar, 1);
    abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
  pdl_wait();                                   // the offsets and the rows come from the kernels before

  // this CTA's expert and rows: every warp asks for the ranges of 32 experts at a time (one by one they were a chain of loads)
  int e = -1, r0 = 0, r1 = 0;
  for (int e0 = 0, before = 0; e0 < p.E && e < 0; e0 += 32) {
    const int mine = e0 + lane, lo = mine < p.E ? p.offsets[mine] : 0, hi = mine < p.E ? p.offsets[mine + 1] : 0;
    const int n_tiles = (hi - lo + BN - 1) / BN;
    int upto = n_tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, before + upto > (int)blockIdx.y);
    if (hit) {
      const int src = __ffs(hit) - 1;
      e = e0 + src;
      r0 = __shfl_sync(0xffffffffu, lo, src) + BN * ((int)blockIdx.y - before - __shfl_sync(0xffffffffu, upto - n_tiles, src));
      r1 = __shfl_sync(0xffffffffu, hi, src);
    }
    before += __shfl_sync(0xffffffffu, upto, 31);
  }
  if (e < 0) return;                            // (before any tensor-memory allocation)
  const int n0 = e * p.rows_per_expert + blockIdx.x * BM;     // row of the stacked weights
  if (warp == 1) {
    tmem_alloc(&tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      for (int i = 0; i < nkb; ++i) {
        const int s = i % STAGES;
        if (i >= STAGES) {
          const uint32_t ph = (i / STAGES) & 1;
          if (!mbar_wait(&empty_bar[s], ph ^ 1)) {
            abort_flag = 1;
            atomicExch(p.status, STATUS_TIMEOUT);
            break;
          }
          if (abort_flag) break;
        }
        uint8_t* st = tiles + (size_t)s * STAGE_BYTES;
        mbar_arrive_expect_tx(&full_bar[s], STAGE_BYTES);
        tma_load_2d(st, &tmap_w, i * BK, n0, &full_bar[s]);
        tma_load_2d(st + W_TILE_BYTES, &tmap_x, i * BK, r0, &full_bar[s]);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = idesc_bf16_f32(BM, BN);
      for (int i = 0; i < nkb; ++i) {
        const int s = i % STAGES;
        const uint32_t ph = (i / STAGES) & 1;
        if (!mbar_wait(&full_bar[s], ph)) {
          abort_flag = 1;
          atomicExch(p.status, STATUS_TIMEOUT + 1);
          break;
        }
        if (abort_flag) break;
        tc_fence_after();
        uint8_t* st = tiles + (size_t)s * STAGE_BYTES;
        const uint64_t da = smem_desc_sw128(st);
        const uint64_t db = smem_desc_sw128(st + W_TILE_BYTES);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_bf16(tmem_base, da + 2 * k, db + 2 * k, idesc, (uint32_t)((i | k) != 0));
        umma_commit(&empty_bar[s]);
      }
      umma_commit(&tmem_full_bar);
    }
    __syncwarp();
  } else {
    // ---- epilogue warps (threads 64..191) ----
    const bool ok = mbar_wait(&tmem_full_bar, 0);
    if (!ok) {
      abort_flag = 1;
      if (lane == 0) atomicExch(p.status, STATUS_TIMEOUT + 2);
    }
    tc_fence_after();
    epilogue_barrier();
    const bool good = !abort_flag;
    const int q = warp & 3;                      // tensor-memory lanes 32q .. 32q + 31
    const int row = 32 * q + lane;               // weight row within the tile
    const int cols = min(BN, r1 - r0);           // token rows of this tile that belong to the expert
    if (good && p.mode == 1) {
      const int n = blockIdx.x * BM + row;       // output feature
      float* out = (float*)p.out;
#pragma unroll 1
      for (int c0 = 0; c0 < cols; c0 += 16) {
        float v[16];
        tmem_ld_16(tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)c0, v);
        if (n < p.n_valid) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c0 + j < cols) out[(size_t)(r0 + c0 + j) * p.ldo + n] = v[j];
        }
      }
    } else if (good && p.mode == 2) {
      const int n = blockIdx.x * BM + row;
      bf16* out = (bf16*)p.out;
#pragma unroll 1
      for (int c0 = 0; c0 < cols; c0 += 16) {
        float v[16];
        tmem_ld_16(tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)c0, v);
        if (n < p.n_valid) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c0 + j < cols) out[(size_t)(r0 + c0 + j) * p.ldo + n] = __float2bfloat16_rn(hy_act(v[j], p.fn));
        }
      }
    } else if (good) {
      // u of one 16-column chunk through shared memory (the pipeline's first stage is free once the
      // accumulator is complete); the threads of lanes 0-63 hold g and finish the unit
      float (*ubuf)[17] = reinterpret_cast<float (*)[17]>(tiles);
      bf16* act = (bf16*)p.out;
      const int f = blockIdx.x * 64 + (row & 63);        // feature
#pragma unroll 1
      for (int c0 = 0; c0 < cols; c0 += 16) {
        float v[16];
        tmem_ld_16(tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)c0, v);
        if (row >= 64) {
#pragma unroll
          for (int j = 0; j < 16; ++j) ubuf[row - 64][j] = v[j];
        }
        epilogue_barrier();
        if (row < 64 && f < p.n_valid) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c0 + j < cols)
              act[(size_t)(r0 + c0 + j) * p.ldo + f] =
                  __float2bfloat16_rn(hy_clamped_glu(v[j], ubuf[row][j], p.alpha, p.limit, p.up_add));
        }
        if (c0 + 16 < cols) epilogue_barrier();          // ubuf is rewritten by the next chunk
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) {
    // give copies that are still in flight time to land before the shared memory is released
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// ---------------------------------------------------------------- CTA pairs (many rows an expert)
// Two CTAs of a cluster compute 256 weight rows x up to 256 token rows with tcgen05.mma.cta_group::2, as the dense
// product's pair kernel does (gemm_tc.cu): each stages 128 weight rows and half of the token rows a k-block, the leader
// issues for both, six stages, the accumulator twice in tensor memory so that a tile's epilogue (two groups of four warps,
// every other 32 token rows each) runs beside the next tile's products.  Persistent: the pairs walk the (expert, 256 weight
// rows, token tile) tiles, the token tiles of the same weights next to each other.
// An expert's rows are cut evenly into ceil(rows / 256) tiles of a multiple of 32 rows: the width is the instruction's N and
// known on the device only, so the token rows arrive in boxes of 16 (whole 8-row groups of the 128-byte swizzle).
// Bound by what the tiles read from L2: one CTA of 128 x 128 reads 32 KB a k-block for 128 x 128 multiply-adds; here it is
// 32 KB for 128 x 256, and experts of 257 rows take two tiles of 160 and not three of 128: 2,695 tokens, four of 32 experts of
// 2,048 x 2 x 1,024 each, 121 -> 79 us a launch.
constexpr int PAIR_STAGES = 6, PAIR_GROUPS = 2, PAIR_THREADS = 64 + PAIR_GROUPS * 128, PAIR_ROWS = 256, PAIR_BOX = 16;
constexpr int PAIR_STAGE_BYTES = W_TILE_BYTES + PAIR_ROWS / 2 * BK * 2;
constexpr int PAIR_STAGING_BYTES = 16 * 1024;                      // of a group: 32 token rows of 64 (g, u) in 32-bit
constexpr int PAIR_SMEM = PAIR_STAGES * PAIR_STAGE_BYTES + PAIR_GROUPS * PAIR_STAGING_BYTES + 1024;
// With few tiles the narrowest width at which the pairs take them in one round is used (a launch waits for one tile then, and a
// tile's epilogue is as long as it is wide).
//
// Which launches the pairs take, by rows an expert on average and `tiles`, the experts' weight tiles of 256 rows.  Time on the
// pairs over one CTA a tile, 4 to 128 experts of 256 x 128 to 2,048 x 1,024, even and uneven rows:
//   GLU       0.5 to 1 from 32 rows; with 75 to 148 tiles (a second round that is half empty) 0.9 to 1.2 below 64 rows: not taken.  A few
//             uneven launches of about one round remain at 1.04 to 1.17.
//   function  0.3 to 1 from 32 rows
//   plain     the other kernel's epilogue is as short, so only launches that fill the pairs gain: 0.65 to 1.0 from 128 tiles and 16,384 rows x
//             weight tiles, or 30,720 at K of 1,024 and more; below that 1.1 to 1.5, and at K of 256 1.2 to 2.2 at any size
constexpr int PAIR_MIN_ROWS = 32;
bool takes_pairs(int mode, int pairs, int E, int weight_tiles, int K) {
  // GIBBS_B200_MOE_PAIR_ROWS: from so many rows an expert, whatever the rest (for comparison runs)
  static const int forced = [] { const char* e = getenv("GIBBS_B200_MOE_PAIR_ROWS"); return e ? atoi(e) : 0; }();
  if (forced > 0) return (long long)pairs >= (long long)forced * E;
  if ((long long)pairs < (long long)PAIR_MIN_ROWS * E) return false;
  const long long tiles = (long long)weight_tiles * E, work = (long long)weight_tiles * pairs;
  if (mode == 0) return tiles <= 74 || tiles > 148 || (long long)pairs >= 64ll * E;
  if (mode == 1) return (K >= 512 && tiles >= 128 && work >= 16384) || (K >= 1024 && work >= 30720);
  return true;
}
constexpr int PAIR_MAX_EXPERTS = 128;                              // (by what shared memory is left)

// Barrier of one group of epilogue warps; true for all of its threads when any of them brought true.
__device__ __forceinline__ bool group_any(int group, bool v) {
  int r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %2, 0;\n\tbar.red.or.pred q, %1, 128, p;\n\tselp.b32 %0, 1, 0, q;\n\t}\n"
               : "=r"(r) : "r"(1 + group), "r"((int)v) : "memory");
  return r != 0;
}
__device__ __forceinline__ void group_barrier(int group) { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); }

// A function of 32 finished sums: one switch for all of them.
__device__ __forceinline__ void pair_act(float (&v)[32], int fn) {
  switch (fn) {
#define PAIR_ACT(kind)                                 \
    case kind:                                         \
      _Pragma("unroll") for (int j = 0; j < 32; ++j) v[j] = hy_act(v[j], kind); \
      break
    PAIR_ACT(ACT_GELU_ERF);
    PAIR_ACT(ACT_GELU_TANH);
    PAIR_ACT(ACT_SILU);
    PAIR_ACT(ACT_RELU);
    PAIR_ACT(ACT_RELU2);
#undef PAIR_ACT
    default: break;
  }
}

__global__ void __launch_bounds__(PAIR_THREADS)
moe_experts_tc_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                           const GroupedParams p) {
  pdl_trigger();
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[PAIR_STAGES], empty_bar[PAIR_STAGES], tmem_full_bar[2], tmem_empty_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  __shared__ int row_at[PAIR_MAX_EXPERTS + 1], tile_at[PAIR_MAX_EXPERTS + 1];    // first row, first token tile of every expert
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();                          // 0: leader
  const int nkb = p.total_kb, E = p.E;

  if (threadIdx.x == 0) {
    for (int s = 0; s < PAIR_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);                                   // the leader's producer arrives; both CTAs' loads add bytes
      mbar_init(&empty_bar[s], 1);                                  // one multicast commit
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full_bar[a], 1);                              // one multicast commit
      mbar_init(&tmem_empty_bar[a], 2 * PAIR_GROUPS);               // the epilogue groups of both CTAs (the leader's copy is used)
    }
    abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_slot, 512);
    tmem_relinquish_pair();
  }
  pdl_wait();                                                       // the offsets and the rows come from the kernels before
  const int weight_tiles = (p.rows_per_expert + 2 * BM - 1) / (2 * BM);
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  if (warp == 2) {
    constexpr int PER_LANE = PAIR_MAX_EXPERTS / 32;
    int lo[PER_LANE], rows[PER_LANE];
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int e = lane + 32 * i;
      lo[i] = e < E ? p.offsets[e] : 0;
      rows[i] = e < E ? p.offsets[e + 1] - lo[i] : 0;
    }
    // the narrowest tiles that the pairs take in one round, whole ones where there are more
    int cap = 32;
    for (; cap < PAIR_ROWS; cap *= 2) {
      int n = 0;
#pragma unroll
      for (int i = 0; i < PER_LANE; ++i) n += (rows[i] + cap - 1) / cap;
      if (__reduce_add_sync(0xffffffffu, n) * weight_tiles <= n_pairs) break;
    }
    int before = 0;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int e = lane + 32 * i, mine = (rows[i] + cap - 1) / cap;
      int upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      if (e < E) {
        row_at[e] = lo[i];
        tile_at[e] = before + upto - mine;
        if (e + 1 == E) {
          row_at[E] = lo[i] + rows[i];
          tile_at[E] = before + upto;
        }
      }
      before += __shfl_sync(0xffffffffu, upto, 31);
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                               // both CTAs' barriers are initialised before anyone signals them
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  const int n_tiles = tile_at[E] * weight_tiles;

  struct Tile { int e, wt, r0, width, rows; };                      // expert, weight tile, first token row, N, rows that are the expert's
  auto tile_of = [&](int t) {
    // the expert whose tiles hold t: the last one with tile_at[e] * weight_tiles <= t
    int lo = 0, hi = E;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tile_at[mid] * weight_tiles <= t) lo = mid; else hi = mid;
    }
    const int mine = tile_at[lo + 1] - tile_at[lo], rows = row_at[lo + 1] - row_at[lo];
    const int rem = t - tile_at[lo] * weight_tiles;
    Tile r;
    r.e = lo;
    r.wt = rem / mine;
    const int rt = rem - r.wt * mine;
    r.width = ((rows + mine - 1) / mine + 31) & ~31;
    r.r0 = row_at[lo] + rt * r.width;
    r.rows = max(0, min(r.width, row_at[lo + 1] - r.r0));
    return r;
  };

  if (warp == 0) {
    if (elect_one()) {
      int it = 0;
      for (int t = pair; t < n_tiles && !abort_flag; t += n_pairs) {
        const Tile tl = tile_of(t);
        const int n0 = tl.e * p.rows_per_expert + tl.wt * 2 * BM + (int)rank * BM;     // this CTA's rows of the stacked weights
        const int half = tl.width / 2, m0 = tl.r0 + (int)rank * half;                  // this CTA's half of the token rows
        for (int i = 0; i < nkb; ++i, ++it) {
          const int s = it % PAIR_STAGES;
          const uint32_t ph = (it / PAIR_STAGES) & 1;
          if (!mbar_wait(&empty_bar[s], ph ^ 1)) {
            abort_flag = 1;
            atomicExch(p.status, STATUS_TIMEOUT);
            break;
          }
          if (abort_flag) break;
          uint8_t* st = tiles + (size_t)s * PAIR_STAGE_BYTES;
          if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], 2 * (W_TILE_BYTES + half * BK * 2));
          tma_load_2d_pair(st, &tmap_w, i * BK, n0, &full_bar[s]);
          for (int b = 0; b < half; b += PAIR_BOX)
            tma_load_2d_pair(st + W_TILE_BYTES + b * BK * 2, &tmap_x, i * BK, m0 + b, &full_bar[s]);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      int it = 0, tile_i = 0;
      for (int t = pair; t < n_tiles && !abort_flag; t += n_pairs, ++tile_i) {
        const uint32_t idesc = idesc_bf16_f32(2 * BM, tile_of(t).width);
        const int a = tile_i & 1;
        if (!mbar_wait(&tmem_empty_bar[a], ((tile_i >> 1) & 1) ^ 1)) {
          abort_flag = 1;
          atomicExch(p.status, STATUS_TIMEOUT + 1);
          break;
        }
        tc_fence_after();
        const uint32_t acc = tmem_base + (uint32_t)(a * PAIR_ROWS);
        for (int i = 0; i < nkb; ++i, ++it) {
          const int s = it % PAIR_STAGES;
          const uint32_t ph = (it / PAIR_STAGES) & 1;
          if (!mbar_wait(&full_bar[s], ph)) {
            abort_flag = 1;
            atomicExch(p.status, STATUS_TIMEOUT + 2);
            break;
          }
          if (abort_flag) break;
          tc_fence_after();
          uint8_t* st = tiles + (size_t)s * PAIR_STAGE_BYTES;
          const uint64_t da = smem_desc_sw128(st);
          const uint64_t db = smem_desc_sw128(st + W_TILE_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16_pair(acc, da + 2 * k, db + 2 * k, idesc, (uint32_t)((i | k) != 0));
          umma_commit_pair(&empty_bar[s]);
        }
        umma_commit_pair(&tmem_full_bar[a]);
      }
    }
    __syncwarp();
  } else {
    // ---- epilogue ----
    const int eg = (warp - 2) >> 2, et = threadIdx.x - 64 - 128 * eg;          // group, thread of the group
    const int q = warp & 3, row = 32 * q + lane;                               // lane of the accumulator = weight row of this CTA's 128
    uint8_t* staging = tiles + (size_t)PAIR_STAGES * PAIR_STAGE_BYTES + (size_t)eg * PAIR_STAGING_BYTES;
    const bool pieces = ((uintptr_t)p.out & 3) == 0 && p.ldo % 2 == 0 && p.n_valid % 2 == 0;      // (mode 2) stores of two values
    int tile_i = 0;
    for (int t = pair; t < n_tiles; t += n_pairs, ++tile_i) {
      const Tile tl = tile_of(t);
      const int a = tile_i & 1;
      const bool ok = mbar_wait(&tmem_full_bar[a], (tile_i >> 1) & 1);
      if (!ok) {
        abort_flag = 1;
        if (lane == 0) atomicExch(p.status, STATUS_TIMEOUT + 3);
      }
      tc_fence_after();
      if (group_any(eg, abort_flag != 0)) break;
      const uint32_t acc = tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(a * PAIR_ROWS);
      const int w0 = tl.wt * 2 * BM + (int)rank * BM;                          // first weight row of this CTA within the expert
      bool arrived = false;
      for (int h0 = eg * 32; h0 < tl.width; h0 += 32 * PAIR_GROUPS) {
        const int hc = max(0, min(32, tl.rows - h0));
        float v[32];
        tmem_ld_32(acc + (uint32_t)h0, v);
        if (h0 + 32 * PAIR_GROUPS >= tl.width) {                               // this group's last piece: the accumulator is read
          tc_fence_before();
          group_barrier(eg);
          if (et == 0) mbar_arrive_leader(&tmem_empty_bar[a]);
          arrived = true;
        }
        if (p.mode == 0) {
          // g (rows 0-63) and u (rows 64-127) meet in shared memory; all threads share the 32 x 64 activations, four a step
          float* gs = reinterpret_cast<float*>(staging);                       // [32][64]
          float* us = gs + 32 * 64;                                            // [32][64]
          float* mine = row < 64 ? gs + row : us + (row - 64);
#pragma unroll
          for (int j = 0; j < 32; ++j) mine[j * 64] = v[j];
          group_barrier(eg);
          if ((w0 >> 1) < p.n_valid) {                                         // (n_valid is a multiple of 64)
            bf16* dst = (bf16*)p.out + (size_t)(tl.r0 + h0) * p.ldo + (w0 >> 1);
            for (int idx = et; idx < hc * 16; idx += 128) {
              const int mm = idx >> 4, f = (idx & 15) * 4;
              const float4 g4 = *reinterpret_cast<const float4*>(gs + mm * 64 + f);
              const float4 u4 = *reinterpret_cast<const float4*>(us + mm * 64 + f);
              __nv_bfloat162 x, y;
              x.x = __float2bfloat16_rn(hy_clamped_glu(g4.x, u4.x, p.alpha, p.limit, p.up_add));
              x.y = __float2bfloat16_rn(hy_clamped_glu(g4.y, u4.y, p.alpha, p.limit, p.up_add));
              y.x = __float2bfloat16_rn(hy_clamped_glu(g4.z, u4.z, p.alpha, p.limit, p.up_add));
              y.y = __float2bfloat16_rn(hy_clamped_glu(g4.w, u4.w, p.alpha, p.limit, p.up_add));
              uint2 packed;
              packed.x = *reinterpret_cast<uint32_t*>(&x);
              packed.y = *reinterpret_cast<uint32_t*>(&y);
              *reinterpret_cast<uint2*>(dst + (size_t)mm * p.ldo + f) = packed;
            }
          }
          group_barrier(eg);                                                   // (the pieces are rewritten by the next 32 rows)
        } else if (p.mode == 1) {
          if (w0 + row < p.n_valid) {
            float* dst = (float*)p.out + (size_t)(tl.r0 + h0) * p.ldo + w0 + row;      // a warp's store: 128 bytes of one token's row
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < hc) dst[(size_t)j * p.ldo] = v[j];
          }
        } else {
          pair_act(v, p.fn);
          if (pieces) {
            // neighbouring lanes (weight rows n, n + 1) swap every other token's value: a store of a warp is two whole sectors of two
            // tokens' rows
            const bool odd = lane & 1;
            bf16* dst = (bf16*)p.out + (size_t)(tl.r0 + h0 + odd) * p.ldo + w0 + (row & ~1);
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              const float other = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
              const __nv_bfloat162 two = odd ? __floats2bfloat162_rn(other, v[j + 1]) : __floats2bfloat162_rn(v[j], other);
              if (j + odd < hc && w0 + row < p.n_valid) *reinterpret_cast<__nv_bfloat162*>(dst + (size_t)j * p.ldo) = two;
            }
          } else if (w0 + row < p.n_valid) {
            bf16* dst = (bf16*)p.out + (size_t)(tl.r0 + h0) * p.ldo + w0 + row;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < hc) dst[(size_t)j * p.ldo] = __float2bfloat16_rn(v[j]);
          }
        }
      }
      if (!arrived && et == 0) mbar_arrive_leader(&tmem_empty_bar[a]);         // (a tile of 32 rows has none for the second group)
    }
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
  __syncthreads();
  cluster_sync_all();                                               // nobody leaves while its partner may still use its memory
  if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// ---------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  });
  return fn;
}

// A [rows, K] bfloat16 matrix with row stride ld (elements), read in boxes of box_rows x 64, 128-byte swizzle.
bool make_tmap(CUtensorMap* map, const void* base, long long rows, long long K, long long ld, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct WKey {
  const void* p; long long rows, k;
  bool operator==(const WKey& o) const { return p == o.p && rows == o.rows && k == o.k; }
};
struct WKeyHash {
  size_t operator()(const WKey& k) const {
    return std::hash<const void*>()(k.p) ^ (std::hash<long long>()(k.rows) * 31) ^ (std::hash<long long>()(k.k) * 131);
  }
};
std::mutex g_wmap_mutex;
std::unordered_map<WKey, CUtensorMap, WKeyHash> g_wmaps;   // weights do not move: their maps are made once

template <int BN, int STAGES = stages_of<BN>()>
int launch(const CUtensorMap& tw, const CUtensorMap& tx, const GroupedParams& p, int weight_tiles, int row_tiles,
           cudaStream_t stream) {
  constexpr int SMEM = STAGES * (W_TILE_BYTES + BN * BK * 2) + 1024;
  static bool raised = false;
  if (!raised) {
    GB_CUDA((cudaFuncSetAttribute(moe_experts_tc_kernel<BN, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM)));
    raised = true;
  }
  gb_launch(moe_experts_tc_kernel<BN, STAGES>, dim3(weight_tiles, row_tiles), dim3(192), SMEM, stream, tw, tx, p);
  GB_CHECK_LAUNCH("moe_experts_tc");
  return 1;
}

int launch_pairs(const CUtensorMap& tw, const CUtensorMap& tx, const GroupedParams& p, long long most_tiles, cudaStream_t stream) {
  static bool raised = false;
  if (!raised) {
    GB_CUDA(cudaFuncSetAttribute(moe_experts_tc_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PAIR_SMEM));
    raised = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (unsigned)(most_tiles < 74 ? most_tiles : 74));
  cfg.blockDim = dim3(PAIR_THREADS);
  cfg.dynamicSmemBytes = PAIR_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = gb_pdl_enabled() ? 2 : 1;
  GB_CUDA(cudaLaunchKernelEx(&cfg, moe_experts_tc_pair_kernel, tw, tx, p));
  GB_CHECK_LAUNCH("moe_experts_tc (pairs)");
  return 1;
}

}  // namespace

// Whether gb_op_moe_experts_tc takes these sizes (mode 0: GLU, the weights' gate and up rows alternating
// in blocks of 64; mode 1: plain; mode 2: a function of the sums).  K: features in; ld: row strides of the rows and of the weights.
GB_API int gb_moe_experts_tc_supported(int mode, int n_out, int K, long long ld_rows, long long ld_w) {
  if (K % 8 || ld_rows % 8 || ld_w % 8) return 0;
  if (mode == 0 && n_out % 64) return 0;
  return 1;
}

// a0 input rows (bf16), a1 their stride, a2 rows the matrix has room for, a3 weights [E, rows per expert, K]
// (bf16, contiguous), a4 unused, a5 offsets [E + 1], a6 experts, a7 out, a8 its row stride, a9 tokens, a10 features out
// (GLU: ff), a11 features in (K), a12 mode (0: GLU, out bf16 [rows, ff]; 1: plain, out f32; 2: a function of the sums, out
// bf16), a13 top, a14 (mode 2) the function's number; f0 alpha, f1 limit, f2 what is added to u
GB_OP(gb_op_moe_experts_tc) {
  const int pairs = (int)(a[9] * a[13]), E = (int)a[6], n_out = (int)a[10], K = (int)a[11], mode = (int)a[12];
  if (pairs <= 0) return 0;
  if (!gb_moe_experts_tc_supported(mode, n_out, K, a[1], K) || (a[0] & 15) || (a[3] & 15))
    GB_FAIL(GB_ERR_ARG, "moe_experts_tc: sizes or alignment the tensor-core kernel does not take");
  const int rows_per_expert = mode == 0 ? 2 * n_out : n_out;
  CUtensorMap tw, tx;
  {
    std::lock_guard<std::mutex> lock(g_wmap_mutex);
    const WKey key{op_ptr<const void>(a[3]), (long long)E * rows_per_expert, K};
    auto it = g_wmaps.find(key);
    if (it == g_wmaps.end()) {
      if (!make_tmap(&tw, key.p, key.rows, K, K, BM)) GB_FAIL(GB_ERR_CUDA, "moe_experts_tc: cuTensorMapEncodeTiled failed (W)");
      g_wmaps.emplace(key, tw);
    } else {
      tw = it->second;
    }
  }
  // few rows an expert (decoding): narrow token tiles
  // (and wide ones where an expert has many: a tile's weights are read from L2 once for twice the tokens)
  const int BN = pairs <= 16 * E ? 16 : pairs < 192 * E ? 64 : 128;
  const bool on_pairs = E <= PAIR_MAX_EXPERTS && takes_pairs(mode, pairs, E, gb_div_up(rows_per_expert, 2 * BM), K) &&
                        (mode != 0 || (a[8] % 4 == 0 && (a[7] & 7) == 0));
  if (!make_tmap(&tx, op_ptr<const void>(a[0]), a[2], K, a[1], on_pairs ? PAIR_BOX : BN))
    GB_FAIL(GB_ERR_CUDA, "moe_experts_tc: cuTensorMapEncodeTiled failed (rows)");
  GroupedParams p;
  p.offsets = op_ptr<const int>(a[5]);
  p.E = E; p.rows_per_expert = rows_per_expert; p.n_valid = n_out; p.mode = mode; p.fn = (int)a[14];
  if (mode < 0 || mode > 2 || (mode == 2 && (p.fn < 0 || p.fn > ACT_NONE))) GB_FAIL(GB_ERR_ARG, "moe_experts_tc: mode %d, function %d", mode, p.fn);
  p.out = op_ptr<void>(a[7]); p.ldo = a[8];
  p.total_kb = gb_div_up(K, BK);
  p.alpha = (float)f[0]; p.limit = (float)f[1]; p.up_add = (float)f[2];
  p.status = ctx->status;
  if (on_pairs)                                                     // (rows / 32 + E: at most this many token tiles over all experts)
    return launch_pairs(tw, tx, p, (long long)gb_div_up(rows_per_expert, 2 * BM) * (pairs / 32 + E), ctx->stream);
  const int weight_tiles = gb_div_up(rows_per_expert, BM);
  const int row_tiles = gb_div_up(pairs, BN) + E;          // at most this many over all experts
  // (blocks that find rows, at most: whole tiles and a partly filled one for every expert that has any)
  const bool few = (long long)weight_tiles * (pairs / BN + (pairs < E ? pairs : E)) <= 2 * 148;
  return BN == 16   ? (few ? launch<16, FEW_STAGES>(tw, tx, p, weight_tiles, row_tiles, ctx->stream)
                           : launch<16>(tw, tx, p, weight_tiles, row_tiles, ctx->stream))
         : BN == 64 ? launch<64>(tw, tx, p, weight_tiles, row_tiles, ctx->stream)
                    : launch<128>(tw, tx, p, weight_tiles, row_tiles, ctx->stream);
}

// Forget the tensor maps of weights (a model was unloaded).
GB_API void gb_moe_experts_tc_forget() {
  std::lock_guard<std::mutex> lock(g_wmap_mutex);
  g_wmaps.clear();
}
