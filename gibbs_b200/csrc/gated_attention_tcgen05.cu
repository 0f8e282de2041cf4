// The attention of gated_attention_tc.cuh for prompt portions on the 5th generation tensor cores: keys of 64 entries, values
// of 64 or 128, sliding window or blocks, soft cap, sink, output gate, maps, and the form with sigmoids in the softmax's place.
//
// A CTA takes one (kv head, map, tile of consecutive tokens of one request); its 128 rows are (token, query head of the
// group) pairs.  It walks the visible keys in tiles of 64 positions:
//
//   producer warp   TMA: Q once (a box of 64 columns x group heads x tokens); then K_j, V_j, K_j+1, ... page by page through
//                   the block table into a ring of three buffers
//   MMA warp        S = Q K_j^T (tensor memory columns 0..63); when the softmax warps have written P_j: O += P_j V_j
//   softmax warps   thread = row: S from tensor memory, scale, soft cap, mask, running maximum and sum in 32-bit; the
//                   weights as TWO bfloat16 terms (p = hi + lo, O += hi V + lo V), which keep 16 bits of every weight.  O
//                   in tensor memory is rescaled only when the maximum has grown by more than 8 (a factor of 256).
//
// Three CTAs fit on an SM at values of 64 (73 KB of shared memory, 128 tensor-memory columns, 112 registers a thread), two at
// 128: while one is in its softmax the others' products run.  2,695 tokens, 32 / 8 heads of 64, soft cap, window of 1,024: 187 us a
// layer on the mma.sync kernel, 123 here; with sigmoids 128 and 55.  Bound by the special functions of the softmax warps (three a
// score under a soft cap, 16 a cycle and SM) and by the chain of a key tile.
//
// The arithmetic of a weight (scores times log2(e), the hardware's 2^x and 1/x) is that of gated_attention_tc.cuh.
// A weight of zero does not keep what is not finite out of a product, so the values of positions that no row of the tile
// sees (the rest of the last page, pages the window has passed) are zeroed in shared memory before they are multiplied.  Of the
// others a row may meet one that only another row sees: a row whose result is not finite is worked out again by itself, over its own
// keys.  (Looking at the values of every key tile that not all rows see whole cost 5 to 8 % of a launch.)
// Every wait is bounded; a wait that runs out sets *status and the CTA drains and returns.
#include <mutex>

#include "gated_attention_tcgen05.cuh"
#include "hybrid.cuh"
#include "sm100.cuh"

namespace {

using namespace sm100;

constexpr int GT_ROWS = 128, GT_KEYS = 64, GT_RING = 3, GT_DK = 64;
// LONG: every GT_FOLD key tiles O moves from tensor memory to a sum beside it.  The tensor core truncates its sums, so one over a long context
// is off by the more the longer it is, here as on mma.sync (relative error of values of one sign, 64-entry heads: 4,096 keys 1.4e-5, 8,192
// 3.8e-5 on both, 32,768 2.0e-4; with LONG 1.5e-5 at all of these).  A kernel of its own, because the code for it costs the others 2 to
// 5 % of a launch.
constexpr int GT_FOLD = 64;
constexpr int GT_TIMEOUT = 40;
enum { GT_BAD_PAGE_READ = 2 };

struct GtParams {
  const int* block_table; int bt_stride, page_size, n_pages;
  const int* tok_req; const int* tok_pos; const int* q_start;
  const float* gate; long long ld_gate;
  bf16* out; float* out_f32; long long ldo;
  int N, R, H, G, tpt, maps, window, blocked, sink;
  float scale, softcap;
  const float* sink_scores;
  const float* score_bias; float factor;
  const bf16 *q, *k_pages, *v_pages;     // (for rows that are worked out again)
  int* status;
};

template <int DV> struct GtCfg {
  static constexpr int Q_BYTES = GT_ROWS * GT_DK * 2;
  static constexpr int P_BYTES = GT_ROWS * GT_KEYS * 2;                         // of one term
  static constexpr int K_BYTES = GT_KEYS * GT_DK * 2, V_BYTES = GT_KEYS * DV * 2, KV_BYTES = V_BYTES > K_BYTES ? V_BYTES : K_BYTES;
  static constexpr int SMEM_BYTES = Q_BYTES + 2 * P_BYTES + GT_RING * KV_BYTES + 1024;
  static constexpr int TMEM_COLS = GT_KEYS + DV <= 128 ? 128 : 256;
  static constexpr int REGS = DV <= 64 ? 112 : 168;                             // three CTAs an SM, or two (by shared memory)
};

__device__ __forceinline__ float gt_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float gt_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// total[0 .. DV - 1] = total * 2^(total[DV] - m) + O * corr, total[DV] = m; the first time without what was there.
template <int DV, bool SIG>
__device__ __noinline__ void gt_fold(float* total, bool more, float corr, float m, uint32_t tmem_row) {
  const float f = !more ? 0.f : SIG ? 1.f : total[DV] == -INFINITY ? 0.f : gt_ex2(total[DV] - m);
#pragma unroll 1
  for (int c0 = 0; c0 < DV; c0 += 16) {
    float o[16];
    tmem_ld_16(tmem_row + (uint32_t)c0, o);
#pragma unroll
    for (int i = 0; i < 16; ++i) total[c0 + i] = more ? fmaf(total[c0 + i], f, o[i] * corr) : o[i] * corr;
  }
  total[DV] = m;
}

// One row (a token's query head) again, by itself and over the keys first .. last that it sees, in 32-bit: sum[0 .. DV - 1] its weighted
// sum, m and l its maximum and its sum of weights.  For rows whose result is not finite, which another row's value may have done.
template <int DV, bool CAPPED, bool SIG>
__device__ __noinline__ void gt_row(float* sum, float& m, float& l, const GtParams& p, const int* bt, int g, int mp, const bf16* q, int first,
                                    int last, float c_in, float c_mul, float c_add, float bias) {
  m = -INFINITY;
  l = 0.f;
  for (int d = 0; d < DV; ++d) sum[d] = 0.f;
  for (int key = max(first, 0); key <= last; ++key) {
    int page = bt[key / p.page_size];
    if (page < 0 || page >= p.n_pages) page = 0;                // (as its tile was brought)
    const size_t at = ((size_t)page * p.G + g) * p.page_size + key % p.page_size;
    const __nv_bfloat162* k = reinterpret_cast<const __nv_bfloat162*>(p.k_pages + (at * p.maps + mp) * GT_DK);
    const __nv_bfloat162* v = reinterpret_cast<const __nv_bfloat162*>(p.v_pages + at * DV);
    float s0 = 0.f, s1 = 0.f;
    for (int d = 0; d < GT_DK / 2; ++d) {
      const float2 x = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(q)[d]), y = __bfloat1622float2(k[d]);
      s0 = fmaf(x.x, y.x, s0);
      s1 = fmaf(x.y, y.y, s1);
    }
    float s = (s0 + s1) * c_in;
    if (CAPPED) s = fmaf(c_mul, gt_rcp(gt_ex2(s) + 1.f), c_add);
    float w;
    if (SIG) {
      w = gt_rcp(1.f + gt_ex2(-(s + bias)));
    } else {
      if (s > m) {
        const float c = m == -INFINITY ? 0.f : gt_ex2(m - s);
        l *= c;
        for (int d = 0; d < DV; ++d) sum[d] *= c;
        m = s;
      }
      w = gt_ex2(s - (m == -INFINITY ? 0.f : m));
      l += w;
    }
    for (int d = 0; d < DV / 2; ++d) {
      const float2 y = __bfloat1622float2(v[d]);
      sum[2 * d] = fmaf(w, y.x, sum[2 * d]);
      sum[2 * d + 1] = fmaf(w, y.y, sum[2 * d + 1]);
    }
  }
}

template <int DV, bool CAPPED, bool SIG, bool LONG>
__global__ void __launch_bounds__(192) __maxnreg__((GtCfg<DV>::REGS))
sink_attention_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                              const __grid_constant__ CUtensorMap map_v, const __grid_constant__ GtParams p) {
  pdl_trigger();
  using C = GtCfg<DV>;
  constexpr int VSUB = DV / 64;                                 // 64-column sub-tiles of a V tile
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t q_full, kv_full[GT_RING], kv_empty[GT_RING], s_full, s_free, p_full, o_full;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sq = base;                                           // [128 rows][128 B]
  uint8_t* sp = sq + C::Q_BYTES;                                // [2 terms][128 rows][128 B]
  uint8_t* skv = sp + 2 * C::P_BYTES;                           // [RING]: K [64 keys][128 B] or V [VSUB][64 keys][128 B]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = p.H / p.G, tpt = p.tpt;
  const int g = blockIdx.x / p.maps, mp = blockIdx.x - g * p.maps;      // kv head and map

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    for (int s = 0; s < GT_RING; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1);
    }
    mbar_init(&s_full, 1);
    mbar_init(&s_free, 4);                                      // one arrival per softmax warp
    mbar_init(&p_full, 4);
    mbar_init(&o_full, 1);
    abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
  }
  // which request's which tile, from the last to the first (a prompt's last tiles see the most keys: they start first); every warp
  // looks at 32 requests at a time
  int t0 = -1, n_tok = 0;
  for (int r0 = 0, before = 0; r0 < p.R && t0 < 0; r0 += 32) {
    const int r = p.R - 1 - r0 - lane;
    const int qs = r >= 0 ? p.q_start[r] : 0, qe = r < 0 ? 0 : r + 1 < p.R ? p.q_start[r + 1] : p.N;
    const int nt = (qe - qs + tpt - 1) / tpt;
    int upto = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, before + upto > (int)blockIdx.y);
    if (hit) {
      // (its first tile is the request's last)
      const int src = __ffs(hit) - 1, from_end = before + __shfl_sync(0xffffffffu, upto, src) - (int)blockIdx.y;
      t0 = __shfl_sync(0xffffffffu, qs, src) + (from_end - 1) * tpt;
      n_tok = min(tpt, __shfl_sync(0xffffffffu, qe, src) - t0);
    }
    before += __shfl_sync(0xffffffffu, upto, 31);
  }
  if (t0 < 0) return;
  const int pos0 = p.tok_pos[t0];
  const int* bt = p.block_table + (size_t)p.tok_req[t0] * p.bt_stride;
  const int hi_all = pos0 + n_tok;                              // keys lo_all <= k < hi_all may be seen
  // the first position that position p sees (with `blocked` its own block of `window` positions, counted from 0)
  auto first_seen = [&](int pos) { return p.window <= 0 ? 0 : p.blocked ? pos / p.window * p.window : pos - p.window + 1; };
  const int lo_all = max(0, first_seen(pos0));
  const int t_lo = lo_all / GT_KEYS, t_hi = (hi_all + GT_KEYS - 1) / GT_KEYS, n_tiles = t_hi - t_lo;

  if (warp == 1) {
    tmem_alloc(&tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  // Lane i of the producer brings page slot i of every tile; slots outside the visible range bring the first visible page
  // again (their keys are masked and their values zeroed).
  const int pages_per_tile = GT_KEYS / p.page_size;
  constexpr int OUTSIDE = -0x7fffffff;
  auto lookup = [&](int t) {
    if (lane >= pages_per_tile) return OUTSIDE;
    const int j0 = t * GT_KEYS + lane * p.page_size;
    return (j0 < hi_all && j0 + p.page_size > lo_all) ? bt[j0 / p.page_size] : OUTSIDE;
  };
  int first_page = 0, page_cur = OUTSIDE;
  if (warp == 0) {
    first_page = bt[lo_all / p.page_size];
    page_cur = lookup(t_lo);
    gb_pin(first_page);
    gb_pin(page_cur);
  }
  if (group * tpt < GT_ROWS) {
    // a group that does not divide 128: the tile's last rows have no (token, head), zeros keep them numbers
    const int spare = GT_ROWS - group * tpt;
    for (int i = threadIdx.x; i < spare * 8; i += blockDim.x)
      *reinterpret_cast<uint4*>(sq + (size_t)(group * tpt + i / 8) * 128 + (i & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_s = tmem_slot, tmem_o = tmem_slot + GT_KEYS;

  if (warp == 0) {
    // ---- producer ----
    pdl_wait();                                                 // q and the pages are written by the kernels before
    if (lane == 0) {
      mbar_arrive_expect_tx(&q_full, (uint32_t)(group * tpt * 128));
      tma_load_3d(sq, &map_q, mp * GT_DK, g * group, t0, &q_full);
    }
    int it = 0;
    for (int t = t_lo; t < t_hi && !abort_flag; ++t) {
      const int page_next = t + 1 < t_hi ? lookup(t + 1) : OUTSIDE;
      int page = page_cur == OUTSIDE ? first_page : page_cur;
      if (page < 0 || page >= p.n_pages) {
        if (lane < pages_per_tile) atomicExch(p.status, GT_BAD_PAGE_READ);
        page = 0;
      }
      const int row = (page * p.G + g) * p.page_size;
      for (int kv = 0; kv < 2; ++kv, ++it) {                    // K_t, then V_t
        const int s = it % GT_RING;
        bool ok = true;
        if (lane == 0) {
          ok = mbar_wait(&kv_empty[s], ((it / GT_RING) & 1) ^ 1);
          if (!ok) {
            abort_flag = 1;
            atomicExch(p.status, GT_TIMEOUT);
          } else {
            mbar_arrive_expect_tx(&kv_full[s], kv == 0 ? C::K_BYTES : C::V_BYTES);
          }
        }
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        if (!ok) break;
        uint8_t* dst = skv + (size_t)s * C::KV_BYTES + (size_t)lane * p.page_size * 128;
        if (lane < pages_per_tile) {
          if (kv == 0) {
            tma_load_2d(dst, &map_k, mp * GT_DK, row, &kv_full[s]);
          } else {
            for (int sub = 0; sub < VSUB; ++sub)
              tma_load_2d(dst + (size_t)sub * GT_KEYS * 128, &map_v, sub * 64, row, &kv_full[s]);
          }
        }
      }
      page_cur = page_next;
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---- MMA issuer: S_0, then for every tile S_{j+1} before O += P_j V_j; ring items are K_j = 2j and V_j = 2j + 1 ----
    if (elect_one()) {
      constexpr uint32_t idesc_s = idesc_bf16_f32(GT_ROWS, GT_KEYS);
      constexpr uint32_t idesc_o = idesc_bf16_f32_b_mn(GT_ROWS, DV);
      bool ok = mbar_wait(&q_full, 0);
      auto issue_s = [&](int j) {
        const int item = 2 * j, s = item % GT_RING;
        if (!mbar_wait(&kv_full[s], (item / GT_RING) & 1)) return false;
        tc_fence_after();
        const uint64_t da = smem_desc_sw128(sq), db = smem_desc_sw128(skv + (size_t)s * C::KV_BYTES);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16(tmem_s, da + 2 * k, db + 2 * k, idesc_s, (uint32_t)(k != 0));
        umma_commit(&kv_empty[s]);
        umma_commit(&s_full);
        return true;
      };
      if (ok) ok = issue_s(0);
      for (int j = 0; j < n_tiles && ok && !abort_flag; ++j) {
        if (j + 1 < n_tiles) {
          ok = mbar_wait(&s_free, j & 1);
          if (!ok) break;
          tc_fence_after();
          ok = issue_s(j + 1);
          if (!ok) break;
        }
        const int item = 2 * j + 1, s = item % GT_RING;
        ok = mbar_wait(&p_full, j & 1) && mbar_wait(&kv_full[s], (item / GT_RING) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint8_t* vt = skv + (size_t)s * C::KV_BYTES;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          // 16 keys = two 8-row groups of 1024 bytes further in V; a second 64-column block of DV lies one sub-tile
          // further, which the descriptor's leading offset says
          uint64_t db = smem_desc_sw128(vt + (size_t)k * 16 * 128);
          if (VSUB > 1) db = (db & ~((uint64_t)0x3FFF << 16)) | ((uint64_t)((GT_KEYS * 128) >> 4) << 16);
#pragma unroll
          for (int term = 0; term < 2; ++term)
            umma_bf16(tmem_o, smem_desc_sw128(sp + (size_t)term * C::P_BYTES) + 2 * k, db, idesc_o, (uint32_t)(((LONG ? j % GT_FOLD : j) | k | term) != 0));
        }
        umma_commit(&kv_empty[s]);
        umma_commit(&o_full);
      }
      if (!ok) {
        abort_flag = 1;
        atomicExch(p.status, GT_TIMEOUT + 1);
      }
    }
    __syncwarp();
  } else {
    // ---- softmax warps: thread = row ----
    const int q4 = warp & 3, row = 32 * q4 + lane;
    const int tl = row / group, hh = row - tl * group;
    const bool rvalid = tl < n_tok;
    const int rpos = pos0 + tl, rfirst = first_seen(rpos), last_first = first_seen(pos0 + tpt - 1);
    const uint32_t lane_off = (uint32_t)(32 * q4) << 16;
    constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;
    const float c_in = CAPPED ? p.scale * 2.f * LOG2E / p.softcap : p.scale * LOG2E;
    const float c_mul = -2.f * p.softcap * LOG2E, c_add = p.softcap * LOG2E;
    const float bias = SIG && p.score_bias && rvalid ? p.score_bias[g * group + hh] * LOG2E : 0.f;
    float m_used = -INFINITY, l_run = 0.f;
    // In local memory: with LONG, O of the tiles in front and the maximum it is relative to; a row that is worked out again.
    float total[DV + 1];
    bool alive = true;
    for (int j = 0; j < n_tiles; ++j) {
      if (!__all_sync(0xffffffffu, mbar_wait(&s_full, j & 1) && !abort_flag)) {
        abort_flag = 1;
        if (lane == 0) atomicExch(p.status, GT_TIMEOUT + 2);
        alive = false;
        break;
      }
      tc_fence_after();
      // which of the tile's columns this row may see: lo_c <= column <= hi_c; most tiles need no mask
      const int col0 = (t_lo + j) * GT_KEYS;
      const int hi_c = rvalid ? rpos - col0 : -1;
      const int lo_c = rfirst - col0;
      const bool full = col0 + GT_KEYS - 1 <= pos0 && col0 >= last_first;
      float v[GT_KEYS];
#pragma unroll
      for (int c = 0; c < GT_KEYS; c += 32) tmem_ld_32_issue(tmem_s + lane_off + (uint32_t)c, v + c);
      tmem_ld_wait_n<GT_KEYS>(v);
      // the row is in registers: the next tile's first product may overwrite S
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_free);
#pragma unroll
      for (int i = 0; i < GT_KEYS; ++i) {
        v[i] *= c_in;
        if (CAPPED) v[i] = fmaf(c_mul, gt_rcp(gt_ex2(v[i]) + 1.f), c_add);
      }
      if (!full) {
#pragma unroll
        for (int i = 0; i < GT_KEYS; ++i) v[i] = (i >= lo_c && i <= hi_c) ? v[i] : -INFINITY;
      }
      float corr = 1.f;
      bool grow = false;
      if (SIG) {
        // 1 / (1 + 2^-v): 0 for a key that is not seen (2^inf = inf, 1 / inf = 0)
#pragma unroll
        for (int i = 0; i < GT_KEYS; ++i) v[i] = gt_rcp(1.f + gt_ex2(-(v[i] + bias)));
      } else {
        float mx[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
        for (int i = 4; i < GT_KEYS; ++i) mx[i & 3] = fmaxf(mx[i & 3], v[i]);
        const float m_tile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        // the maximum in use follows only when it would otherwise fall behind by more than 2^8
        grow = m_tile > m_used + 8.f || (m_used == -INFINITY && m_tile > -INFINITY);
        if (grow) {
          corr = m_used == -INFINITY ? 0.f : gt_ex2(m_used - m_tile);
          m_used = m_tile;
          l_run *= corr;
        }
        const float ref = m_used == -INFINITY ? 0.f : m_used;
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < GT_KEYS; ++i) {
          v[i] = gt_ex2(v[i] - ref);
          sum[i & 3] += v[i];
        }
        l_run += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      }
      // P and O of the tile before are still being read by its second product until o_full
      if (j > 0 && !__all_sync(0xffffffffu, mbar_wait(&o_full, (j - 1) & 1))) {
        abort_flag = 1;
        if (lane == 0) atomicExch(p.status, GT_TIMEOUT + 3);
        alive = false;
        break;
      }
      tc_fence_after();
      const bool fold = LONG && j > 0 && j % GT_FOLD == 0;
      if (!SIG && j > 0 && !fold && __any_sync(0xffffffffu, grow)) {
#pragma unroll 1
        for (int c0 = 0; c0 < DV; c0 += 16) {
          float o[16];
          tmem_ld_16(tmem_o + lane_off + (uint32_t)c0, o);
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] *= corr;
          tmem_st_16(tmem_o + lane_off + (uint32_t)c0, o);
        }
      }
      // eight keys (16 bytes) of each term at a time into the swizzled tiles
#pragma unroll
      for (int chunk = 0; chunk < GT_KEYS / 8; ++chunk) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float x = v[8 * chunk + 2 * e], y = v[8 * chunk + 2 * e + 1];
          const __nv_bfloat162 h2 = __floats2bfloat162_rn(x, y);
          const float2 hf = __bfloat1622float2(h2);
          const __nv_bfloat162 l2 = __floats2bfloat162_rn(x - hf.x, y - hf.y);
          hi[e] = *reinterpret_cast<const uint32_t*>(&h2);
          lo[e] = *reinterpret_cast<const uint32_t*>(&l2);
        }
        uint8_t* dst = sp + (size_t)row * 128 + ((chunk ^ (row & 7)) << 4);
        *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(dst + C::P_BYTES) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
      if (fold) {
        gt_fold<DV, SIG>(total, j > GT_FOLD, corr, m_used, tmem_o + lane_off);
        tc_fence_before();                                      // (the next product starts a new sum in O)
      }
      if (col0 + GT_KEYS > hi_all || col0 < lo_all) {
        // values of positions that nobody here sees: zeros
        const int item = 2 * j + 1, s = item % GT_RING;
        if (!__all_sync(0xffffffffu, mbar_wait(&kv_full[s], (item / GT_RING) & 1))) {
          abort_flag = 1;
          if (lane == 0) atomicExch(p.status, GT_TIMEOUT + 4);
          alive = false;
          break;
        }
        const int key = col0 + (row & 63);
        if (key >= hi_all || key < lo_all) {
          // (rows 0-63 of the tile take the first half of a key's 128 bytes, rows 64-127 the second)
#pragma unroll
          for (int sub = 0; sub < VSUB; ++sub) {
            uint4* dst = reinterpret_cast<uint4*>(skv + (size_t)s * C::KV_BYTES + ((size_t)sub * GT_KEYS + (row & 63)) * 128) + 4 * (row >> 6);
#pragma unroll
            for (int e = 0; e < 4; ++e) dst[e] = make_uint4(0u, 0u, 0u, 0u);
          }
        }
      }
      fence_proxy_async();                                      // P is read by the tensor core (async proxy)
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full);
    }
    if (alive && !__all_sync(0xffffffffu, mbar_wait(&o_full, (n_tiles - 1) & 1))) {
      abort_flag = 1;
      if (lane == 0) atomicExch(p.status, GT_TIMEOUT + 5);
      alive = false;
    }
    tc_fence_after();
    if (alive) {
      pdl_wait();                                               // (long over; the gate's logits come from a kernel before)
      const int h = (g * group + hh) * p.maps + mp, t = t0 + tl;
      auto scale_of = [&](float m2, float l) {
        if (SIG) return p.factor;
        const float m = m2 * LN2;                               // natural units (-inf stays)
        const float z = p.sink_scores && rvalid ? p.sink_scores[g * group + hh] : 0.f;
        const float M = p.sink ? fmaxf(m, z) : m;
        const float e = expf(m - M);
        return e * (1.0f / fmaf(e, l, p.sink ? expf(z - M) : 0.f));
      };
      const float* gt = p.gate ? p.gate + (size_t)t * p.ld_gate + (size_t)h * DV : nullptr;
      const size_t at = (size_t)t * p.ldo + (size_t)h * DV;
      auto store = [&](int c0, float (&o)[16], float f) {
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] *= gt ? f * hy_sigmoid(gt[c0 + i]) : f;
        if (p.out_f32) {
#pragma unroll
          for (int i = 0; i < 16; i += 2) *reinterpret_cast<float2*>(p.out_f32 + at + c0 + i) = make_float2(o[i], o[i + 1]);
        } else {
#pragma unroll
          for (int i = 0; i < 16; i += 2) *reinterpret_cast<__nv_bfloat162*>(p.out + at + c0 + i) = __floats2bfloat162_rn(o[i], o[i + 1]);
        }
      };
      const float f = scale_of(m_used, l_run);
      const bool folded = LONG && n_tiles > GT_FOLD;
      const float f_total = !folded ? 0.f : SIG ? 1.f : total[DV] == -INFINITY ? 0.f : gt_ex2(total[DV] - m_used);
      float check = 0.f;                                        // (x * 0 is a zero or not a number)
#pragma unroll 1
      for (int c0 = 0; c0 < DV; c0 += 16) {
        float o[16];
        tmem_ld_16(tmem_o + lane_off + (uint32_t)c0, o);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (folded) o[i] = fmaf(total[c0 + i], f_total, o[i]);
          check = fmaf(o[i], 0.f, check);
        }
        if (rvalid) store(c0, o, f);
      }
      if (rvalid && !(check == 0.f)) {
        float m, l;
        gt_row<DV, CAPPED, SIG>(total, m, l, p, bt, g, mp, p.q + ((size_t)t * p.H * p.maps + h) * GT_DK, rfirst, rpos, c_in, c_mul, c_add, bias);
        const float fr = scale_of(m, l);
#pragma unroll 1
        for (int c0 = 0; c0 < DV; c0 += 16) {
          float o[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = total[c0 + i];
          store(c0, o, fr);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);           // copies still in flight land before the memory goes
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_slot, C::TMEM_COLS);
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

bool encode(CUtensorMap* map, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes,
            const cuuint32_t* box) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), dims, strides_bytes, box,
            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The rows of a page pool, `width` entries each, in boxes of 64 columns x a page's rows.
bool pages_map(CUtensorMap* map, const void* pages, long long rows, int width, int page_size) {
  cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)width * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)page_size};
  return encode(map, pages, 2, dims, strides, box);
}

template <int DV, bool CAPPED, bool SIG, bool LONG>
int launch_gt(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const GtParams& p, dim3 grid, cudaStream_t stream) {
  static bool raised = false;
  if (!raised) {
    GB_CUDA((cudaFuncSetAttribute(sink_attention_tcgen05_kernel<DV, CAPPED, SIG, LONG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  GtCfg<DV>::SMEM_BYTES)));
    raised = true;
  }
  gb_launch(sink_attention_tcgen05_kernel<DV, CAPPED, SIG, LONG>, grid, dim3(192), GtCfg<DV>::SMEM_BYTES, stream, mq, mk, mv, p);
  GB_CHECK_LAUNCH("sink_attention_tcgen05");
  return 1;
}

}  // namespace

bool gb_gated_tcgen05_takes(const GatedTcgen05Launch& a) {
  return a.dim == GT_DK && (a.vdim == 64 || a.vdim == 128) && a.page_size >= 8 && a.page_size <= GT_KEYS && GT_KEYS % a.page_size == 0 &&
         a.H / a.G <= GT_ROWS / 2 && (long long)a.n_pages * a.G * a.page_size < (1ll << 31) &&
         gb_div_up(a.n, GT_ROWS / (a.H / a.G)) + a.R <= 65535;
}

int gb_gated_tcgen05_launch(const GatedTcgen05Launch& a, cudaStream_t stream) {
  const int group = a.H / a.G, tpt = GT_ROWS / group;
  CUtensorMap mq, mk, mv;
  {
    // q as [token][head][maps * dim]: a box of 64 columns x the group's heads x the tile's tokens lands as rows (token, head)
    cuuint64_t dims[3] = {(cuuint64_t)a.maps * GT_DK, (cuuint64_t)a.H, (cuuint64_t)a.n};
    cuuint64_t strides[2] = {(cuuint64_t)a.maps * GT_DK * 2, (cuuint64_t)a.H * a.maps * GT_DK * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)group, (cuuint32_t)tpt};
    if (!encode(&mq, a.q, 3, dims, strides, box)) GB_FAIL(GB_ERR_CUDA, "sink_attention_tcgen05: cuTensorMapEncodeTiled failed (q)");
  }
  const long long page_rows = (long long)a.n_pages * a.G * a.page_size;
  if (!pages_map(&mk, a.k_pages, page_rows, a.maps * GT_DK, a.page_size) || !pages_map(&mv, a.v_pages, page_rows, a.vdim, a.page_size))
    GB_FAIL(GB_ERR_CUDA, "sink_attention_tcgen05: cuTensorMapEncodeTiled failed (pages)");
  GtParams p;
  p.block_table = a.block_table; p.bt_stride = a.bt_stride; p.page_size = a.page_size; p.n_pages = a.n_pages;
  p.tok_req = a.tok_req; p.tok_pos = a.tok_pos; p.q_start = a.q_start; p.gate = a.gate; p.ld_gate = a.ld_gate;
  p.out = a.out; p.out_f32 = a.out_f32; p.ldo = a.ldo; p.N = a.n; p.R = a.R; p.H = a.H; p.G = a.G; p.tpt = tpt; p.maps = a.maps;
  p.window = a.window; p.blocked = a.blocked; p.sink = a.sink; p.scale = a.scale; p.softcap = a.softcap; p.sink_scores = a.sink_scores;
  p.score_bias = a.score_bias; p.factor = a.factor; p.q = a.q; p.k_pages = a.k_pages; p.v_pages = a.v_pages; p.status = a.status;
  // (every request may end with a partly filled tile)
  const dim3 grid(a.G * a.maps, gb_div_up(a.n, tpt) + a.R);
  const bool capped = a.softcap > 0.f;
  const bool is_long = a.longest > GT_FOLD * GT_KEYS;
#define GT_AS(DV, CAPPED, SIG) \
  (is_long ? launch_gt<DV, CAPPED, SIG, true>(mq, mk, mv, p, grid, stream) : launch_gt<DV, CAPPED, SIG, false>(mq, mk, mv, p, grid, stream))
#define GT(DV) (a.sigmoid ? (capped ? GT_AS(DV, true, true) : GT_AS(DV, false, true)) : (capped ? GT_AS(DV, true, false) : GT_AS(DV, false, false)))
  return a.vdim == 64 ? GT(64) : GT(128);
#undef GT
#undef GT_AS
}
