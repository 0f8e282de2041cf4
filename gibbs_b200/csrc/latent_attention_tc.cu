// Attention over a latent cache on tensor cores, in the absorbed form, for steps that carry portions of prompts.
//
// Every head's keys AND values are the same cached rows [c_j | k_rot,j] (kv_rank + rot_dim entries, bfloat16; the
// rotated part may be absent): with q'_h = [W_uk,h^T q_h | rot(q_rot,h)] the score is q'_h . [c_j | k_rot,j] and the
// head's output is sum_j p_j c_j: the first product reads whole rows, the second their first kv_rank entries.  So the rows of a tile are (token, head) pairs of one
// request, all of which read the same key rows, and one tile of cached rows in shared memory is the second operand of
// both products: S = Q' C^T (rows of C as they lie) and O += P C (the same rows, transposed on the way to the
// registers).
//
//  CTA: 64 rows = TPT consecutive tokens of one request x all heads (TPT = 64 / heads, rounded down), 4 warps of 16
//  rows; where the latent is wider than 256, a second group of 4 warps takes the other half of O's columns and
//  computes the same S (O of 16 x 256 is 128 registers a thread).  Key tiles of 64 rows arrive by cp.async through
//  the block table into two buffers.  mma.sync.m16n8k16, bfloat16 operands, 32-bit accumulators; the softmax (base
//  2, running maximum and sum per row) is 32-bit, and its weights enter the second product as TWO bfloat16 terms
//  (p = hi + lo), so 16 bits of every weight count.  A learned sink per head joins the denominator at the end; an
//  optional gate multiplies the result.  With `splits` 2 (a step of few tiles: one long prompt) the key tiles of
//  every row tile are cut in two halves for two CTAs, which leave (maximum, sum, weighted sum) per row for the merge
//  kernel of latent_attention.cu, and the row tiles with the most keys are launched first.  Causal, no window: what has one runs
//  on the second kernel below, as do steps of single tokens; 32-bit pages run on the generic kernel.  Rows in shared memory lie `stride` entries apart: the row's length rounded up
//  to 16, plus 8 (an odd number of 16-byte pieces, so that ldmatrix meets no bank twice).
#include "hybrid.cuh"

namespace {

enum { LTC_BAD_PAGE_READ = 2 };
#ifndef LTC_SPLIT_KEYS
#define LTC_SPLIT_KEYS 1
#endif
constexpr int LTC_ROWS = 64, LTC_KEYS = 64;

__device__ __forceinline__ void ltc_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void ltc_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}
__device__ __forceinline__ void ltc_ldmatrix(unsigned (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ltc_ldmatrix_t(unsigned (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ltc_mma(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned ltc_pack(float x, float y) {
  __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<unsigned*>(&v);
}
// (hi, lo) of two weights: hi the nearest bfloat16, lo the nearest bfloat16 of what is left
__device__ __forceinline__ void ltc_split(float x, float y, unsigned& hi, unsigned& lo) {
  const bf16 hx = __float2bfloat16_rn(x), hy = __float2bfloat16_rn(y);
  __nv_bfloat162 h;
  h.x = hx;
  h.y = hy;
  hi = *reinterpret_cast<unsigned*>(&h);
  lo = ltc_pack(x - __bfloat162float(hx), y - __bfloat162float(hy));
}

struct LtcParams {
  const float* qp;          // [tokens][heads][dk]
  const bf16* pages;        // [n_pages][page_size][dk]
  const int* block_table;
  int bt_stride, page_size, n_pages;
  const int* tok_req;
  const int* tok_pos;
  const int* q_start;      // first row per request; a request's rows end where the next one's begin
  int n, R;
  const float* gate;
  long long ld_gate;
  float* out;
  long long ldo;
  int H, r, tpt;
  int dk, stride;           // entries of a cached row (r + rotated part); entries between rows in shared memory
  int splits;               // 1, or 2: blockIdx.z takes one half of a row tile's key tiles and writes partial results
  float* ws;                // [tokens * heads][splits][r + 2] partial results (splits > 1)
  float scale_log2;
  const float* sink;
  int* status;
};

// A thread's part of two finished rows: columns wn * OC + 8 j + 2 t4 and the one behind.
template <int OC>
__device__ __forceinline__ void ltc_store(const LtcParams& p, const float (&o)[OC / 8][4], float m_a, float m_b, float l_a, float l_b, int row_a,
                                          int row_b, int rows_live, int tl_a, int tl_b, int h_a, int h_b, int t_first, int wn, int t4) {
  const int H = p.H, r = p.r;
  constexpr float LOG2E = 1.4426950408889634f;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int row = half ? row_b : row_a;
    if (row >= rows_live) continue;
    const int tl = half ? tl_b : tl_a, h = half ? h_b : h_a;
    const float m = half ? m_b : m_a, l = half ? l_b : l_a;
    const size_t t = (size_t)t_first + tl;
    if (p.splits > 1) {
      // this half's partial result: maximum (natural units), sum of weights, weighted sum, for the merge kernel
      float* w = p.ws + ((t * H + h) * p.splits + blockIdx.z) * (size_t)(r + 2);
      if (wn == 0 && t4 == 0) {
        w[0] = m * 0.6931471805599453f;                    // (-inf stays -inf: a half without keys)
        w[1] = l;
      }
#pragma unroll
      for (int j = 0; j < OC / 8; ++j) {
        const int col = wn * OC + 8 * j + 2 * t4;
        if (col < r) {
          w[2 + col] = o[j][2 * half];
          w[2 + col + 1] = o[j][2 * half + 1];
        }
      }
      continue;
    }
    float f = 1.f / l;
    if (p.sink) {
      // a learned score without a key or a value: only the denominator knows it
      const float s2 = p.sink[h] * LOG2E, top = fmaxf(m, s2), e = exp2f(m - top);
      f = e / (exp2f(s2 - top) + e * l);
    }
    if (p.gate) f *= hy_sigmoid(p.gate[t * p.ld_gate + h]);
    float* dst = p.out + t * p.ldo + (size_t)h * r + wn * OC + 2 * t4;
#pragma unroll
    for (int j = 0; j < OC / 8; ++j) {
      if (wn * OC + 8 * j < r)
        *reinterpret_cast<float2*>(dst + 8 * j) = make_float2(o[j][2 * half] * f, o[j][2 * half + 1] * f);
    }
  }
}

template <int RP>
__global__ void __launch_bounds__(RP > 256 ? 256 : 128, 1) latent_attention_tc_kernel(const LtcParams p) {
  constexpr int NSPLIT = RP > 256 ? 2 : 1, OC = RP / NSPLIT, THREADS = 128 * NSPLIT;
  const int STRIDE = p.stride, dk = p.dk;
  extern __shared__ __align__(16) unsigned char ltc_smem[];
  bf16* Qs = reinterpret_cast<bf16*>(ltc_smem);           // [64][STRIDE]
  bf16* Cs = Qs + LTC_ROWS * STRIDE;                       // [2][64][STRIDE]
  pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = warp & 3, wn = warp >> 2;
  const int g = lane >> 2, t4 = lane & 3;
  const int req = blockIdx.y;
  const int first = p.q_start[req], len = (req + 1 < p.R ? p.q_start[req + 1] : p.n) - first;
  // (the row tiles with the most keys go first: where the grid is more than a wave, the short ones fill the end)
  const int tok0 = (int)(gridDim.x - 1 - blockIdx.x) * p.tpt;
  if (tok0 >= len) return;
  const int ntok = min(p.tpt, len - tok0), H = p.H, r = p.r;
  const int rows_live = ntok * H;
  const int t_first = first + tok0;
  const int pos0 = p.tok_pos[t_first];
  const int kmax = pos0 + ntok - 1;
  const int* table = p.block_table + (size_t)p.tok_req[t_first] * p.bt_stride;
  // zeros where nothing is copied: rows beyond the live ones, columns dk .. stride
  for (int i = threadIdx.x; i < 3 * LTC_ROWS * STRIDE / 8; i += THREADS)
    reinterpret_cast<uint4*>(ltc_smem)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();

  const int pieces = dk >> 3;                              // 16-byte pieces of a cached row
  auto stage = [&](int kt, int b) {
    bf16* dst = Cs + (size_t)b * LTC_KEYS * STRIDE;
    for (int j = warp; j < LTC_KEYS; j += THREADS / 32) {
      const int key = min(kt * LTC_KEYS + j, kmax);         // (rows behind the last visible key are masked)
      int page = table[key / p.page_size];
      if (page < 0 || page >= p.n_pages) {
        if (lane == 0) atomicExch(p.status, LTC_BAD_PAGE_READ);
        continue;                                          // (the row keeps what it had: zeros or an older row)
      }
      const bf16* src = p.pages + ((size_t)page * p.page_size + key % p.page_size) * dk;
      for (int c = lane; c < pieces; c += 32) gb_cp_async_16(dst + j * STRIDE + 8 * c, src + 8 * c);
    }
    ltc_commit();
  };
  const int tiles = kmax / LTC_KEYS + 1;
  const int half_tiles = (tiles + 1) >> 1;
  const int kt_begin = p.splits > 1 ? (int)blockIdx.z * half_tiles : 0;
  const int kt_end = p.splits > 1 ? min(tiles, kt_begin + half_tiles) : tiles;
  pdl_wait();
  if (kt_begin < kt_end) stage(kt_begin, 0);
  {
    // this tile's queries: rows_live consecutive rows of dk floats, rounded to bfloat16
    const float* src = p.qp + (size_t)t_first * H * dk;
    const int quads = dk >> 2;
    for (int row = warp; row < rows_live; row += THREADS / 32)
      for (int c = lane; c < quads; c += 32) {
        const float4 v = *reinterpret_cast<const float4*>(src + (size_t)row * dk + 4 * c);
        uint2 w;
        w.x = ltc_pack(v.x, v.y);
        w.y = ltc_pack(v.z, v.w);
        *reinterpret_cast<uint2*>(Qs + row * STRIDE + 4 * c) = w;
      }
  }
  // this thread's two rows: wm * 16 + g and + 8
  const int row_a = wm * 16 + g, row_b = row_a + 8;
  const int tl_a = row_a / H, tl_b = row_b / H;
  const int h_a = row_a - tl_a * H, h_b = row_b - tl_b * H;
  const int pos_a = pos0 + tl_a, pos_b = pos0 + tl_b;
  const bool warp_live = wm * 16 < rows_live;

  float o[OC / 8][4];
#pragma unroll
  for (int j = 0; j < OC / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  float m_a = -INFINITY, m_b = -INFINITY, l_a = 0.f, l_b = 0.f;
  const int ksteps = (dk + 15) >> 4;                       // k-steps of the first product that hold anything
  const int npairs = min(OC / 16, max(0, (r - wn * OC + 15) >> 4));   // pairs of 8 output columns likewise

  if (kt_begin >= kt_end) __syncthreads();                 // (the queries and zeros are written; no key tile follows)
  for (int kt = kt_begin; kt < kt_end; ++kt) {
    const int b = (kt - kt_begin) & 1;
    if (kt + 1 < kt_end) {
      stage(kt + 1, b ^ 1);
      ltc_wait<1>();
    } else {
      ltc_wait<0>();
    }
    __syncthreads();
    if (warp_live) {
      const bf16* C = Cs + (size_t)b * LTC_KEYS * STRIDE;
      float s[8][4];
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
      const bf16* qa = Qs + (wm * 16 + (lane & 15)) * STRIDE + (lane >> 4) * 8;
      const bf16* cb = C + ((lane & 7) + (lane >> 4) * 8) * STRIDE + ((lane >> 3) & 1) * 8;
#pragma unroll 2
      for (int ks = 0; ks < ksteps; ++ks) {
        unsigned a[4];
        ltc_ldmatrix(a, qa + ks * 16);
#pragma unroll
        for (int np = 0; np < 4; ++np) {
          unsigned bb[4];
          ltc_ldmatrix(bb, cb + np * 16 * STRIDE + ks * 16);
          ltc_mma(s[2 * np], a, bb[0], bb[1]);
          ltc_mma(s[2 * np + 1], a, bb[2], bb[3]);
        }
      }
      // scores in base 2, the causal mask, the running maximum
      const int key0 = kt * LTC_KEYS + 2 * t4;
      float mx_a = -INFINITY, mx_b = -INFINITY;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int k = key0 + 8 * j;
        s[j][0] = k <= pos_a ? s[j][0] * p.scale_log2 : -INFINITY;
        s[j][1] = k + 1 <= pos_a ? s[j][1] * p.scale_log2 : -INFINITY;
        s[j][2] = k <= pos_b ? s[j][2] * p.scale_log2 : -INFINITY;
        s[j][3] = k + 1 <= pos_b ? s[j][3] * p.scale_log2 : -INFINITY;
        mx_a = fmaxf(mx_a, fmaxf(s[j][0], s[j][1]));
        mx_b = fmaxf(mx_b, fmaxf(s[j][2], s[j][3]));
      }
      mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 1));
      mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 2));
      mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 1));
      mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 2));
      const float mn_a = fmaxf(m_a, mx_a), mn_b = fmaxf(m_b, mx_b);
      // (a row of a later token may see no key of this tile's first rows only if the tile lies behind it, and
      // such tiles are not visited by a CTA whose last token is that far; key 0 is visible to every row, so after
      // the first tile the maxima are finite.  A dead row of a partly filled tile has a clamped position.)
      const float ref_a = mn_a == -INFINITY ? 0.f : mn_a, ref_b = mn_b == -INFINITY ? 0.f : mn_b;
      const float corr_a = exp2f(m_a - ref_a), corr_b = exp2f(m_b - ref_b);
      m_a = mn_a;
      m_b = mn_b;
      float sum_a = 0.f, sum_b = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        s[j][0] = exp2f(s[j][0] - ref_a);
        s[j][1] = exp2f(s[j][1] - ref_a);
        s[j][2] = exp2f(s[j][2] - ref_b);
        s[j][3] = exp2f(s[j][3] - ref_b);
        sum_a += s[j][0] + s[j][1];
        sum_b += s[j][2] + s[j][3];
      }
      l_a = l_a * corr_a + sum_a;                          // (this lane's share; the quad is added at the end)
      l_b = l_b * corr_b + sum_b;
#pragma unroll
      for (int j = 0; j < OC / 8; ++j) {
        o[j][0] *= corr_a;
        o[j][1] *= corr_a;
        o[j][2] *= corr_b;
        o[j][3] *= corr_b;
      }
      // O += P C, the weights as hi + lo
      const bf16* ct = C + ((lane & 7) + ((lane >> 3) & 1) * 8) * STRIDE + wn * OC + (lane >> 4) * 8;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        unsigned hi[4], lo[4];
        ltc_split(s[2 * kk][0], s[2 * kk][1], hi[0], lo[0]);
        ltc_split(s[2 * kk][2], s[2 * kk][3], hi[1], lo[1]);
        ltc_split(s[2 * kk + 1][0], s[2 * kk + 1][1], hi[2], lo[2]);
        ltc_split(s[2 * kk + 1][2], s[2 * kk + 1][3], hi[3], lo[3]);
#pragma unroll
        for (int np = 0; np < OC / 16; ++np) {
          if (np < npairs) {
            unsigned bb[4];
            ltc_ldmatrix_t(bb, ct + kk * 16 * STRIDE + np * 16);
            ltc_mma(o[2 * np], hi, bb[0], bb[1]);
            ltc_mma(o[2 * np], lo, bb[0], bb[1]);
            ltc_mma(o[2 * np + 1], hi, bb[2], bb[3]);
            ltc_mma(o[2 * np + 1], lo, bb[2], bb[3]);
          }
        }
      }
    }
    __syncthreads();                                       // before the tile after next lands in this buffer
  }
  if (!warp_live) return;
  l_a += __shfl_xor_sync(0xffffffffu, l_a, 1);
  l_a += __shfl_xor_sync(0xffffffffu, l_a, 2);
  l_b += __shfl_xor_sync(0xffffffffu, l_b, 1);
  l_b += __shfl_xor_sync(0xffffffffu, l_b, 2);
  ltc_store<OC>(p, o, m_a, m_b, l_a, l_b, row_a, row_b, rows_live, tl_a, tl_b, h_a, h_b, t_first, wn, t4);
}

// The same for latents wider than 256 whose rows leave room for the weights in shared memory: 16 warps, four groups of 16 rows x
// four slices.  For S a slice is 16 of a key tile's 64 keys (every score once, where the kernel above works every score out in
// both groups of warps), for O a quarter of the latent's columns; maxima and the weights' two terms go through shared memory
// between the four warps of a row group, which meet at a barrier of their own.  Bound by waiting, as below: portions of 1,801 and
// 894 tokens, 16 heads, latent of 512, 475 us a launch and 583 with the kernel above.
constexpr int LTW_SLICES = 4, LTW_THREADS = 128 * LTW_SLICES, LTW_OC = 128, LTW_PLD = 72;

size_t ltw_smem(int stride) {
  return sizeof(bf16) * (3 * LTC_ROWS * (size_t)stride + 2 * LTC_ROWS * LTW_PLD) + sizeof(float) * 2 * LTW_SLICES * LTC_ROWS;
}

__global__ void __launch_bounds__(LTW_THREADS, 1) latent_attention_tc_wide_kernel(const LtcParams p) {
  constexpr int OC = LTW_OC;
  const int STRIDE = p.stride, dk = p.dk;
  extern __shared__ __align__(16) unsigned char ltc_smem[];
  bf16* Qs = reinterpret_cast<bf16*>(ltc_smem);            // [64][STRIDE]
  bf16* Cs = Qs + LTC_ROWS * STRIDE;                       // [2][64][STRIDE]
  bf16* Ps = Cs + 2 * LTC_KEYS * STRIDE;                   // [2 terms][64][LTW_PLD]
  float* top = reinterpret_cast<float*>(Ps + 2 * LTC_ROWS * LTW_PLD);    // [slice][64] maxima over a tile, then [slice][64] sums
  pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = warp & 3, wn = warp >> 2;
  const int g = lane >> 2, t4 = lane & 3;
  const int req = blockIdx.y;
  const int first = p.q_start[req], len = (req + 1 < p.R ? p.q_start[req + 1] : p.n) - first;
  const int tok0 = (int)(gridDim.x - 1 - blockIdx.x) * p.tpt;
  if (tok0 >= len) return;
  const int ntok = min(p.tpt, len - tok0), H = p.H, r = p.r;
  const int rows_live = ntok * H;
  const int t_first = first + tok0;
  const int pos0 = p.tok_pos[t_first];
  const int kmax = pos0 + ntok - 1;
  const int* table = p.block_table + (size_t)p.tok_req[t_first] * p.bt_stride;
  // zeros where nothing is copied: rows beyond the live ones, columns dk .. stride
  for (int i = threadIdx.x; i < 3 * LTC_ROWS * STRIDE / 8; i += LTW_THREADS)
    reinterpret_cast<uint4*>(ltc_smem)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();

  const int pieces = dk >> 3;                              // 16-byte pieces of a cached row
  auto stage = [&](int kt, int b) {
    bf16* dst = Cs + (size_t)b * LTC_KEYS * STRIDE;
    for (int j = warp; j < LTC_KEYS; j += LTW_THREADS / 32) {
      const int key = min(kt * LTC_KEYS + j, kmax);        // (rows behind the last visible key are masked)
      const int page = table[key / p.page_size];
      if (page < 0 || page >= p.n_pages) {
        if (lane == 0) atomicExch(p.status, LTC_BAD_PAGE_READ);
        continue;                                          // (the row keeps what it had: zeros or an older row)
      }
      const bf16* src = p.pages + ((size_t)page * p.page_size + key % p.page_size) * dk;
      for (int c = lane; c < pieces; c += 32) gb_cp_async_16(dst + j * STRIDE + 8 * c, src + 8 * c);
    }
    ltc_commit();
  };
  const int tiles = kmax / LTC_KEYS + 1;
  const int half_tiles = (tiles + 1) >> 1;
  const int kt_begin = p.splits > 1 ? (int)blockIdx.z * half_tiles : 0;
  const int kt_end = p.splits > 1 ? min(tiles, kt_begin + half_tiles) : tiles;
  pdl_wait();
  if (kt_begin < kt_end) stage(kt_begin, 0);
  {
    // this tile's queries: rows_live consecutive rows of dk floats, rounded to bfloat16
    const float* src = p.qp + (size_t)t_first * H * dk;
    const int quads = dk >> 2;
    for (int row = warp; row < rows_live; row += LTW_THREADS / 32)
      for (int c = lane; c < quads; c += 32) {
        const float4 v = *reinterpret_cast<const float4*>(src + (size_t)row * dk + 4 * c);
        uint2 w;
        w.x = ltc_pack(v.x, v.y);
        w.y = ltc_pack(v.z, v.w);
        *reinterpret_cast<uint2*>(Qs + row * STRIDE + 4 * c) = w;
      }
  }
  // this thread's two rows: wm * 16 + g and + 8
  const int row_a = wm * 16 + g, row_b = row_a + 8;
  const int tl_a = row_a / H, tl_b = row_b / H;
  const int h_a = row_a - tl_a * H, h_b = row_b - tl_b * H;
  const int pos_a = pos0 + tl_a, pos_b = pos0 + tl_b;
  const bool warp_live = wm * 16 < rows_live;              // (the same for the four warps of a row group)
  auto group_barrier = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + wm) : "memory"); };

  float o[OC / 8][4];
#pragma unroll
  for (int j = 0; j < OC / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  float m_a = -INFINITY, m_b = -INFINITY, l_a = 0.f, l_b = 0.f;
  const int ksteps = (dk + 15) >> 4;                       // k-steps of the first product that hold anything
  const int npairs = min(OC / 16, max(0, (r - wn * OC + 15) >> 4));   // pairs of 8 output columns likewise

  if (kt_begin >= kt_end) __syncthreads();                 // (the queries and zeros are written; no key tile follows)
  for (int kt = kt_begin; kt < kt_end; ++kt) {
    const int b = (kt - kt_begin) & 1;
    if (kt + 1 < kt_end) {
      stage(kt + 1, b ^ 1);
      ltc_wait<1>();
    } else {
      ltc_wait<0>();
    }
    __syncthreads();
    if (warp_live) {
      const bf16* C = Cs + (size_t)b * LTC_KEYS * STRIDE;
      float s[2][4], s2[2][4];                             // even and odd k-steps: two chains
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
        s2[j][0] = s2[j][1] = s2[j][2] = s2[j][3] = 0.f;
      }
      const bf16* qa = Qs + (wm * 16 + (lane & 15)) * STRIDE + (lane >> 4) * 8;
      const bf16* cb = C + (wn * 16 + (lane & 7) + (lane >> 4) * 8) * STRIDE + ((lane >> 3) & 1) * 8;
#pragma unroll 2
      for (int ks = 0; ks + 1 < ksteps; ks += 2) {
        unsigned a[2][4], bb[2][4];
        ltc_ldmatrix(a[0], qa + ks * 16);
        ltc_ldmatrix(bb[0], cb + ks * 16);
        ltc_ldmatrix(a[1], qa + ks * 16 + 16);
        ltc_ldmatrix(bb[1], cb + ks * 16 + 16);
        ltc_mma(s[0], a[0], bb[0][0], bb[0][1]);
        ltc_mma(s[1], a[0], bb[0][2], bb[0][3]);
        ltc_mma(s2[0], a[1], bb[1][0], bb[1][1]);
        ltc_mma(s2[1], a[1], bb[1][2], bb[1][3]);
      }
      if (ksteps & 1) {
        unsigned a[4], bb[4];
        ltc_ldmatrix(a, qa + (ksteps - 1) * 16);
        ltc_ldmatrix(bb, cb + (ksteps - 1) * 16);
        ltc_mma(s[0], a, bb[0], bb[1]);
        ltc_mma(s[1], a, bb[2], bb[3]);
      }
      // scores in base 2, the causal mask, the maximum over this slice's keys
      const int key0 = kt * LTC_KEYS + wn * 16 + 2 * t4;
      float mx_a = -INFINITY, mx_b = -INFINITY;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int k = key0 + 8 * j;
        s[j][0] = k <= pos_a ? (s[j][0] + s2[j][0]) * p.scale_log2 : -INFINITY;
        s[j][1] = k + 1 <= pos_a ? (s[j][1] + s2[j][1]) * p.scale_log2 : -INFINITY;
        s[j][2] = k <= pos_b ? (s[j][2] + s2[j][2]) * p.scale_log2 : -INFINITY;
        s[j][3] = k + 1 <= pos_b ? (s[j][3] + s2[j][3]) * p.scale_log2 : -INFINITY;
        mx_a = fmaxf(mx_a, fmaxf(s[j][0], s[j][1]));
        mx_b = fmaxf(mx_b, fmaxf(s[j][2], s[j][3]));
      }
      mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 1));
      mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 2));
      mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 1));
      mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 2));
      if (t4 == 0) {
        top[wn * LTC_ROWS + row_a] = mx_a;
        top[wn * LTC_ROWS + row_b] = mx_b;
      }
      group_barrier();
      float mn_a = m_a, mn_b = m_b;
#pragma unroll
      for (int w = 0; w < LTW_SLICES; ++w) {
        mn_a = fmaxf(mn_a, top[w * LTC_ROWS + row_a]);
        mn_b = fmaxf(mn_b, top[w * LTC_ROWS + row_b]);
      }
      const float ref_a = mn_a == -INFINITY ? 0.f : mn_a, ref_b = mn_b == -INFINITY ? 0.f : mn_b;
      const float corr_a = exp2f(m_a - ref_a), corr_b = exp2f(m_b - ref_b);
      m_a = mn_a;
      m_b = mn_b;
      float sum_a = 0.f, sum_b = 0.f;
      unsigned* pw = reinterpret_cast<unsigned*>(Ps + wn * 16 + 2 * t4);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        s[j][0] = exp2f(s[j][0] - ref_a);
        s[j][1] = exp2f(s[j][1] - ref_a);
        s[j][2] = exp2f(s[j][2] - ref_b);
        s[j][3] = exp2f(s[j][3] - ref_b);
        sum_a += s[j][0] + s[j][1];
        sum_b += s[j][2] + s[j][3];
        unsigned hi, lo;
        ltc_split(s[j][0], s[j][1], hi, lo);
        pw[(row_a * LTW_PLD + 8 * j) / 2] = hi;
        pw[((LTC_ROWS + row_a) * LTW_PLD + 8 * j) / 2] = lo;
        ltc_split(s[j][2], s[j][3], hi, lo);
        pw[(row_b * LTW_PLD + 8 * j) / 2] = hi;
        pw[((LTC_ROWS + row_b) * LTW_PLD + 8 * j) / 2] = lo;
      }
      l_a = l_a * corr_a + sum_a;                          // (this lane's share of this slice's keys; added up at the end)
      l_b = l_b * corr_b + sum_b;
#pragma unroll
      for (int j = 0; j < OC / 8; ++j) {
        o[j][0] *= corr_a;
        o[j][1] *= corr_a;
        o[j][2] *= corr_b;
        o[j][3] *= corr_b;
      }
      group_barrier();
      // O += P C, the weights as hi + lo
      const bf16* ct = C + ((lane & 7) + ((lane >> 3) & 1) * 8) * STRIDE + wn * OC + (lane >> 4) * 8;
      const bf16* pa = Ps + (wm * 16 + (lane & 15)) * LTW_PLD + (lane >> 4) * 8;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        unsigned hi[4], lo[4];
        ltc_ldmatrix(hi, pa + kk * 16);
        ltc_ldmatrix(lo, pa + LTC_ROWS * LTW_PLD + kk * 16);
#pragma unroll
        for (int np = 0; np < OC / 16; ++np) {
          if (np < npairs) {
            unsigned bb[4];
            ltc_ldmatrix_t(bb, ct + kk * 16 * STRIDE + np * 16);
            ltc_mma(o[2 * np], hi, bb[0], bb[1]);
            ltc_mma(o[2 * np + 1], hi, bb[2], bb[3]);
            ltc_mma(o[2 * np], lo, bb[0], bb[1]);
            ltc_mma(o[2 * np + 1], lo, bb[2], bb[3]);
          }
        }
      }
    }
    __syncthreads();                                       // before the tile after next lands in this buffer
  }
  if (!warp_live) return;
  l_a += __shfl_xor_sync(0xffffffffu, l_a, 1);
  l_a += __shfl_xor_sync(0xffffffffu, l_a, 2);
  l_b += __shfl_xor_sync(0xffffffffu, l_b, 1);
  l_b += __shfl_xor_sync(0xffffffffu, l_b, 2);
  float* share = top + LTW_SLICES * LTC_ROWS;
  if (t4 == 0) {
    share[wn * LTC_ROWS + row_a] = l_a;
    share[wn * LTC_ROWS + row_b] = l_b;
  }
  group_barrier();
  l_a = l_b = 0.f;
#pragma unroll
  for (int w = 0; w < LTW_SLICES; ++w) {
    l_a += share[w * LTC_ROWS + row_a];
    l_b += share[w * LTC_ROWS + row_b];
  }
  ltc_store<OC>(p, o, m_a, m_b, l_a, l_b, row_a, row_b, rows_live, tl_a, tl_b, h_a, h_b, t_first, wn, t4);
}

template <int RP> int ltc_launch(const LtcParams& p, int tiles, int R, cudaStream_t stream) {
  constexpr int NSPLIT = RP > 256 ? 2 : 1;
  const size_t smem = sizeof(bf16) * 3 * LTC_ROWS * (size_t)p.stride;
  static size_t allowed = 48 * 1024;       // raised once per size, before any stream capture replays the launch
  if (smem > allowed) {
    if (cudaFuncSetAttribute(latent_attention_tc_kernel<RP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
      return -1;
    allowed = smem;
  }
  gb_launch(latent_attention_tc_kernel<RP>, dim3(tiles, R, p.splits), dim3(128 * NSPLIT), smem, stream, p);
  return 0;
}

// The same for windows and for steps of single tokens, with the queries and the softmax weights kept whole: each is
// cut into THREE bfloat16 terms (truncated, so 8 + 8 + 8 bits hold all 24), the cached rows are bfloat16 as they lie,
// every product of two terms is exact and the sums are 32-bit, as on the generic kernel.  The tensor cores truncate
// where they add, so the first terms' products, which carry the sum, are added there 16 at a time, each time from zero,
// and from there on in rounded 32-bit additions; the second and third terms' (2^-8 and 2^-16 of them) have a sum of
// their own, which joins last.  Exponentials are expf: the weights carry 32 bits.  Error against 64 bits over the generic
// kernel's, 12 sizes from 1 head of 32 entries to 64 of 512 + 64, steps of 1 to 300 tokens: 0.77 in the mean, 1.07 at most
// (two rows of one head; with the terms in one chain and scores in base 2 it was 0.93, and up to 1.54 for small latents).
//
//  CTA: 32 consecutive (token, head) rows of one request, whatever the number of heads; 16 warps = 2 groups of 16 rows x
//  8 slices.  Key tiles of 32 rows by cp.async into two buffers.  For S a slice is an eighth of the row's entries: a
//  warp takes 16 rows x 32 keys over its eighth (the queries' three terms would otherwise be read from shared memory
//  by every warp: 3 x 37 KB a tile), the eight partial scores are added in shared memory, sixteen threads a row keep the
//  maximum and the sum in 32-bit and leave the weights' three terms there.  For O a slice is an eighth of the latent's
//  columns.  Key tiles lie at multiples of 32, so a row's sums are grouped by its position alone, whatever the rows
//  beside it.  With `splits`, blockIdx.y takes a chunk of keys, a multiple of `chunk` from position 0, and leaves (maximum,
//  sum, weighted sum) per row for the merge kernel.
//  Bound by waiting: a step of 32 rows x 32 keys takes about 9,600 cycles at 512 + 64 entries.  Its 408 products on each of the SM's
//  four schedulers need 3,300 (independent mma.sync.m16n8k16 issue one in 8.0 cycles a scheduler, with 4 to 16 warps; one behind
//  another in 20), its operand reads from shared memory 2,700; scores, softmax and weighted sum follow one another, with barriers
//  between.  Sixteen warps and the tiles with the most keys first: portions of 1,801 and 894 tokens, 16 heads, 1,067 -> 957 us; two
//  single tokens 12.6 -> 9.5.
constexpr int LTX_ROWS = 32, LTX_KEYS = 32, LTX_SLICES = 8, LTX_WARPS = 2 * LTX_SLICES, LTX_SLD = 32, LTX_PLD = 40;

struct LtxParams {
  const float* qp;          // [tokens * heads][dk]
  const bf16* pages;        // [n_pages][page_size][dk]
  const int* block_table;
  int bt_stride, page_size, n_pages;
  const int* tok_req;
  const int* tok_pos;
  const int* q_start;
  int n, R, H, r, dk, stride, window, splits, chunk;
  const float* gate;
  long long ld_gate;
  float* out;
  long long ldo;
  float* ws;                // [tokens * heads][splits][r + 2] partial results (splits > 1)
  float scale;
  const float* sink;
  int* status;
};

size_t ltx_smem(int stride) {
  return sizeof(bf16) * (3 * LTX_ROWS + 2 * LTX_KEYS) * (size_t)stride + sizeof(float) * LTX_SLICES * LTX_ROWS * LTX_SLD +
         sizeof(bf16) * 3 * LTX_ROWS * LTX_PLD + sizeof(float) * 3 * LTX_ROWS + 2 * sizeof(int);
}

// x = t0 + t1 + t2, each a bfloat16 (the upper half of a 32-bit number)
__device__ __forceinline__ void ltx_split(float x, unsigned short (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const unsigned u = __float_as_uint(x) & 0xffff0000u;
    t[i] = (unsigned short)(u >> 16);
    x -= __uint_as_float(u);
  }
}

// The score of a row and a key of the tile without tensor cores, for what is not finite: the terms of an infinite number
// are no numbers, and an infinite entry is lost on a term that is 0.
__device__ __noinline__ float ltx_score(const bf16* Qs, const bf16* C, int row, int key, int stride, int dk) {
  float s = 0.f;
  for (int d = 0; d < dk; ++d) {
    float q = 0.f;
    for (int t = 0; t < 3; ++t) q += __bfloat162float(Qs[((size_t)t * LTX_ROWS + row) * stride + d]);
    s = fmaf(q, __bfloat162float(C[key * stride + d]), s);
  }
  return s;
}

template <int OC>                                          // columns of the latent a warp takes
__global__ void __launch_bounds__(32 * LTX_WARPS, 1) latent_attention_split_kernel(const LtxParams p) {
  extern __shared__ __align__(16) unsigned char ltc_smem[];
  const int STRIDE = p.stride, dk = p.dk, H = p.H, r = p.r;
  bf16* Qs = reinterpret_cast<bf16*>(ltc_smem);            // [3][32][STRIDE]
  bf16* Cs = Qs + 3 * LTX_ROWS * STRIDE;                   // [2][32][STRIDE]
  float* Sp = reinterpret_cast<float*>(Cs + 2 * LTX_KEYS * STRIDE);      // [8][32][LTX_SLD]
  bf16* Pt = reinterpret_cast<bf16*>(Sp + LTX_SLICES * LTX_ROWS * LTX_SLD);       // [3][32][LTX_PLD]
  float* corr = reinterpret_cast<float*>(Pt + 3 * LTX_ROWS * LTX_PLD);   // [3][32]
  volatile int* odd = reinterpret_cast<int*>(corr + 3 * LTX_ROWS);       // [2]: whether a tile holds what is not finite
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wr = warp & 1, wk = warp >> 1, g = lane >> 2, t4 = lane & 3;
  // which request's which tile: requests have ceil(rows / 32) tiles each, one after the other; taken from the last to the first
  // (a prompt's last tiles see the most keys: they start first)
  const int order = (int)(gridDim.x - 1 - blockIdx.x);
  int req = -1, tile = 0, first = 0, len = 0, before = 0;
  for (int r0 = 0; r0 < p.R && req < 0; r0 += 32) {
    const int mine = r0 + lane;
    const int b = mine < p.R ? p.q_start[mine] : 0, e = mine + 1 < p.R ? p.q_start[mine + 1] : p.n;
    const int tiles = mine < p.R ? (int)(((long long)(e - b) * H + LTX_ROWS - 1) / LTX_ROWS) : 0;
    int upto = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, before + upto > order);
    if (hit) {
      const int src = __ffs(hit) - 1;
      req = r0 + src;
      first = __shfl_sync(0xffffffffu, b, src);
      len = __shfl_sync(0xffffffffu, e - b, src);
      tile = order - before - __shfl_sync(0xffffffffu, upto - tiles, src);
    }
    before += __shfl_sync(0xffffffffu, upto, 31);
  }
  if (req < 0) return;
  const int row0 = tile * LTX_ROWS;                        // (rows of the request)
  const int rows_live = min(LTX_ROWS, len * H - row0);
  const int pos_req = p.tok_pos[first];                    // the request's tokens have consecutive positions
  const int pos0 = pos_req + row0 / H, kmax = pos_req + (row0 + rows_live - 1) / H;
  const int* table = p.block_table + (size_t)p.tok_req[first] * p.bt_stride;
  const int base = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;
  // (key tiles lie at multiples of 32 and chunks at multiples of `chunk`, whatever row the tile begins with; the last chunk
  // takes what is left)
  const int origin = p.splits > 1 ? base / p.chunk * p.chunk + (int)blockIdx.y * p.chunk : 0;
  const int k_begin = max(origin, base / LTX_KEYS * LTX_KEYS);
  const int k_end = (int)blockIdx.y + 1 < p.splits ? min(kmax, origin + p.chunk - 1) : kmax;      // (the last key)
  if (k_begin > k_end) {                                   // (splits > 1) no row sees a key of this chunk: the merge skips it
    pdl_wait();
    if (tid < rows_live) {
      float* w = p.ws + (((size_t)first * H + row0 + tid) * p.splits + blockIdx.y) * (size_t)(r + 2);
      w[0] = -INFINITY;
      w[1] = 0.f;
    }
    return;
  }
  // zeros where nothing is copied: columns dk .. stride
  const int pad = (STRIDE - dk) >> 3;
  for (int i = tid; i < (3 * LTX_ROWS + 2 * LTX_KEYS) * pad; i += 32 * LTX_WARPS)
    *reinterpret_cast<uint4*>(Qs + (size_t)(i / pad) * STRIDE + dk + 8 * (i % pad)) = make_uint4(0u, 0u, 0u, 0u);

  const int pieces = dk >> 3;                              // 16-byte pieces of a cached row
  auto stage = [&](int k0, int b) {
    bf16* dst = Cs + (size_t)b * LTX_KEYS * STRIDE;
#pragma unroll
    for (int u = 0; u < LTX_KEYS / LTX_WARPS; ++u) {
      const int j = warp + LTX_WARPS * u, key = min(max(k0 + j, base), k_end);    // (rows in front of the first key and behind the last are masked)
      const int page = table[key / p.page_size];
      const bool bad = page < 0 || page >= p.n_pages;
      if (bad && lane == 0) atomicExch(p.status, LTC_BAD_PAGE_READ);
      const bf16* src = p.pages + ((size_t)(bad ? 0 : page) * p.page_size + key % p.page_size) * dk;
      for (int c = lane; c < pieces; c += 32) {
        if (bad) *reinterpret_cast<uint4*>(dst + j * STRIDE + 8 * c) = make_uint4(0u, 0u, 0u, 0u);
        else gb_cp_async_16(dst + j * STRIDE + 8 * c, src + 8 * c);
      }
    }
    ltc_commit();
  };
  pdl_wait();
  stage(k_begin, 0);
  {
    // (a warp asks for two rows at once: up to ten trips to L2 side by side)
    const float* src = p.qp + ((size_t)first * H + row0) * dk;
    constexpr int QL = 5;                                  // quads a lane takes of a row: 32 * 5 >= 576 / 4
    const int quads = dk >> 2;
#pragma unroll
    for (int rr = 0; rr < LTX_ROWS / LTX_WARPS; rr += 2) {
      float4 v[2][QL];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int row = warp + LTX_WARPS * (rr + u);
#pragma unroll
        for (int i = 0; i < QL; ++i)
          v[u][i] = row < rows_live && lane + 32 * i < quads
                        ? ldcg_now(reinterpret_cast<const float4*>(src + (size_t)row * dk) + lane + 32 * i)
                        : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int row = warp + LTX_WARPS * (rr + u);
#pragma unroll
        for (int i = 0; i < QL; ++i) {
          if (lane + 32 * i >= quads) break;
          unsigned short a[3], b[3], d[3], e[3];
          ltx_split(v[u][i].x, a);
          ltx_split(v[u][i].y, b);
          ltx_split(v[u][i].z, d);
          ltx_split(v[u][i].w, e);
#pragma unroll
          for (int t = 0; t < 3; ++t)
            *reinterpret_cast<uint2*>(Qs + ((size_t)t * LTX_ROWS + row) * STRIDE + 4 * (lane + 32 * i)) =
                make_uint2(a[t] | (unsigned)b[t] << 16, d[t] | (unsigned)e[t] << 16);
        }
      }
    }
  }
  if (tid < 2) odd[tid] = 0;
  // the softmax's view: sixteen threads a row, two keys each
  const int srow = tid >> 4, scol = (tid & 15) * 2;
  const int spos = pos_req + (row0 + srow) / H, slo = p.window > 0 ? spos - p.window + 1 : 0;
  float m = -INFINITY, l = 0.f;
  float o[OC / 8][4];
#pragma unroll
  for (int j = 0; j < OC / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  const int ksteps = (dk + 15) >> 4;
  const int ks_begin = ksteps * wk / LTX_SLICES, ks_end = ksteps * (wk + 1) / LTX_SLICES;
  const int npairs = min(OC / 16, max(0, (r - wk * OC + 15) >> 4));       // pairs of 8 output columns that hold anything
  const bool warp_live = wr * 16 < rows_live;

  int b = 0;
  for (int k0 = k_begin; k0 <= k_end; k0 += LTX_KEYS, b ^= 1) {
    ltc_wait<0>();
    __syncthreads();                                       // this tile is there, the one before it has been used
    if (k0 + LTX_KEYS <= k_end) stage(k0 + LTX_KEYS, b ^ 1);
    const bf16* C = Cs + (size_t)b * LTX_KEYS * STRIDE;
    if (warp_live) {
      float s[4][4], s_low[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
        s_low[j][0] = s_low[j][1] = s_low[j][2] = s_low[j][3] = 0.f;
      }
      const bf16* qa = Qs + (wr * 16 + (lane & 15)) * STRIDE + (lane >> 4) * 8;
      const bf16* cb = C + ((lane & 7) + (lane >> 4) * 8) * STRIDE + ((lane >> 3) & 1) * 8;
#pragma unroll 1
      for (int ks = ks_begin; ks < ks_end; ++ks) {
        unsigned bb[2][4], a[3][4];
        ltc_ldmatrix(bb[0], cb + ks * 16);
        ltc_ldmatrix(bb[1], cb + 16 * STRIDE + ks * 16);
#pragma unroll
        for (int t = 0; t < 3; ++t) ltc_ldmatrix(a[t], qa + (size_t)t * LTX_ROWS * STRIDE + ks * 16);
#pragma unroll
        for (int np = 0; np < 2; ++np) {
          float low[2][4], top[2][4];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            low[j][0] = low[j][1] = low[j][2] = low[j][3] = 0.f;
            top[j][0] = top[j][1] = top[j][2] = top[j][3] = 0.f;
          }
#pragma unroll
          for (int t = 2; t >= 0; --t) {
            ltc_mma(t == 0 ? top[0] : low[0], a[t], bb[np][0], bb[np][1]);
            ltc_mma(t == 0 ? top[1] : low[1], a[t], bb[np][2], bb[np][3]);
          }
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              s[2 * np + j][e] += top[j][e];
              s_low[2 * np + j][e] += low[j][e];
            }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[j][e] += s_low[j][e];
      // (a row's pieces of eight keys lie in an order that its number gives, so that a half warp meets no bank twice)
      float* dst = Sp + (wk * LTX_ROWS + wr * 16 + g) * LTX_SLD + 2 * t4;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        *reinterpret_cast<float2*>(dst + 8 * (j ^ (g & 3))) = make_float2(s[j][0], s[j][1]);
        *reinterpret_cast<float2*>(dst + 8 * LTX_SLD + 8 * (j ^ (g & 3))) = make_float2(s[j][2], s[j][3]);
      }
    }
    __syncthreads();
    {
      float s[2] = {0.f, 0.f};
#pragma unroll
      for (int w = 0; w < LTX_SLICES; ++w) {
        const float2 v = *reinterpret_cast<const float2*>(Sp + (w * LTX_ROWS + srow) * LTX_SLD + (scol ^ 8 * (srow & 3)));
        s[0] += v.x;
        s[1] += v.y;
      }
      float mx = -INFINITY;
      if (srow < rows_live && !(fabsf(s[0]) + fabsf(s[1]) < INFINITY)) {
        odd[b] = 1;                                        // (a query or a cached row is not finite, or a sum)
        s[0] = ltx_score(Qs, C, srow, scol, STRIDE, dk);
        s[1] = ltx_score(Qs, C, srow, scol + 1, STRIDE, dk);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int k = k0 + scol + e;
        s[e] = (srow < rows_live && k <= min(spos, k_end) && k >= slo) ? s[e] * p.scale : -INFINITY;
        mx = fmaxf(mx, s[e]);
      }
#pragma unroll
      for (int x = 1; x < 16; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
      const float mn = fmaxf(m, mx), ref = mn == -INFINITY ? 0.f : mn;    // (a row may see no key of this tile)
      const float c = expf(m - ref);
      m = mn;
      unsigned short t[2][3];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        s[e] = expf(s[e] - ref);
        ltx_split(s[e], t[e]);
      }
      l = l * c + (s[0] + s[1]);                           // (this thread's share; the row is added at the end)
#pragma unroll
      for (int i = 0; i < 3; ++i)
        *reinterpret_cast<unsigned*>(Pt + (i * LTX_ROWS + srow) * LTX_PLD + scol) = t[0][i] | (unsigned)t[1][i] << 16;
      if ((tid & 15) == 0) corr[srow] = c;
    }
    // A weight of 0 does not keep what is not finite out of a product, so a tile that holds any such thing takes only the keys
    // each row sees.
    __syncthreads();
    if (tid == 0) odd[b ^ 1] = 0;                          // (the next tile's; this one's is read behind this barrier only)
    if (odd[b] && warp_live) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int row = wr * 16 + g + 8 * half, pos = pos_req + (row0 + row) / H;
        const float c = corr[row];
#pragma unroll
        for (int j = 0; j < OC / 8; ++j) {
          o[j][2 * half] *= c;
          o[j][2 * half + 1] *= c;
        }
        for (int k = 0; k < LTX_KEYS; ++k) {
          if (k0 + k > min(pos, k_end) || (p.window > 0 && k0 + k <= pos - p.window)) continue;
          const bf16* w = Pt + row * LTX_PLD + k;
          const float weight = __bfloat162float(w[0]) + __bfloat162float(w[LTX_ROWS * LTX_PLD]) + __bfloat162float(w[2 * LTX_ROWS * LTX_PLD]);
          const bf16* v = C + k * STRIDE + wk * OC + 2 * t4;
#pragma unroll
          for (int j = 0; j < OC / 8; ++j)
            if (j < 2 * npairs) {
              o[j][2 * half] = fmaf(weight, __bfloat162float(v[8 * j]), o[j][2 * half]);
              o[j][2 * half + 1] = fmaf(weight, __bfloat162float(v[8 * j + 1]), o[j][2 * half + 1]);
            }
        }
      }
    } else if (warp_live) {
      const float c_a = corr[wr * 16 + g], c_b = corr[wr * 16 + g + 8];
      const bf16* ct = C + ((lane & 7) + ((lane >> 3) & 1) * 8) * STRIDE + wk * OC + (lane >> 4) * 8;
      const bf16* pa = Pt + (wr * 16 + (lane & 15)) * LTX_PLD + (lane >> 4) * 8;
      unsigned a[2][3][4];
#pragma unroll
      for (int kk = 0; kk < 2; ++kk)
#pragma unroll
        for (int t = 0; t < 3; ++t) ltc_ldmatrix(a[kk][t], pa + t * LTX_ROWS * LTX_PLD + kk * 16);
#pragma unroll
      for (int np = 0; np < OC / 16; ++np) {
        if (np < npairs) {
          float low[2][4], top[2][2][4];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            low[j][0] = low[j][1] = low[j][2] = low[j][3] = 0.f;
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) top[kk][j][0] = top[kk][j][1] = top[kk][j][2] = top[kk][j][3] = 0.f;
          }
          unsigned bb[2][4];
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) ltc_ldmatrix_t(bb[kk], ct + kk * 16 * STRIDE + np * 16);
#pragma unroll
          for (int t = 2; t >= 0; --t)
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
              ltc_mma(t == 0 ? top[kk][0] : low[0], a[kk][t], bb[kk][0], bb[kk][1]);
              ltc_mma(t == 0 ? top[kk][1] : low[1], a[kk][t], bb[kk][2], bb[kk][3]);
            }
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              o[2 * np + j][e] = fmaf(o[2 * np + j][e], e < 2 ? c_a : c_b, top[0][j][e] + top[1][j][e] + low[j][e]);
        }
      }
    }
  }
#pragma unroll
  for (int x = 1; x < 16; x <<= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
  const size_t flat0 = (size_t)first * H + row0;           // this tile's first (token, head) row of the step
  if (p.splits > 1) {
    if ((tid & 15) == 0 && srow < rows_live) {
      float* w = p.ws + ((flat0 + srow) * p.splits + blockIdx.y) * (size_t)(r + 2);
      w[0] = m;                                            // (-inf: a chunk without keys)
      w[1] = l;
    }
  } else if ((tid & 15) == 0 && srow < rows_live) {
    const size_t flat = flat0 + srow, t = flat / H;
    const int h = (int)(flat - t * H);
    // (by the merge kernel's arithmetic, so that one chunk and several of which one holds keys give the same bits)
    const float top = p.sink ? fmaxf(m, p.sink[h]) : m, e = expf(m - top);
    const float open = p.gate ? hy_sigmoid(p.gate[t * p.ld_gate + h]) : 1.f;
    corr[LTX_ROWS + srow] = e;
    corr[2 * LTX_ROWS + srow] = open / __fadd_rn(p.sink ? expf(p.sink[h] - top) : 0.f, __fmul_rn(e, l));
  }
  __syncthreads();
  if (!warp_live) return;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int row = wr * 16 + g + 8 * half;
    if (row >= rows_live) continue;
    const size_t flat = flat0 + row;
    float* dst;
    float e = 1.f, inv = 1.f;
    if (p.splits > 1) {
      dst = p.ws + (flat * p.splits + blockIdx.y) * (size_t)(r + 2) + 2;
    } else {
      dst = p.out + (flat / H) * p.ldo + (flat % H) * (size_t)r;
      e = corr[LTX_ROWS + row];
      inv = corr[2 * LTX_ROWS + row];
    }
    dst += wk * OC + 2 * t4;
#pragma unroll
    for (int j = 0; j < OC / 8; ++j)
      if (wk * OC + 8 * j < r)
        *reinterpret_cast<float2*>(dst + 8 * j) =
            make_float2(__fmul_rn(__fmul_rn(e, o[j][2 * half]), inv), __fmul_rn(__fmul_rn(e, o[j][2 * half + 1]), inv));
  }
}

template <int OC> cudaError_t ltx_launch(const LtxParams& p, cudaStream_t stream) {
  const size_t smem = ltx_smem(p.stride);
  const cudaError_t e = cudaFuncSetAttribute(latent_attention_split_kernel<OC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  // (every request's last tile may be partly filled: at most R tiles beside the whole ones)
  const unsigned tiles = (unsigned)((long long)p.n * p.H / LTX_ROWS + p.R);
  return gb_launch(latent_attention_split_kernel<OC>, dim3(tiles, p.splits), dim3(32 * LTX_WARPS), smem, stream, p);
}

// out[t, h, :] = x[t, h, :] W[h]^T on tensor cores, for the two per-head products around the attention (W_uk^T on the
// queries, W_uv on the weighted latents) when a step has rows enough.  A CTA takes 64 rows x 64 outputs of one head
// in steps of 32 inputs; x is 32-bit and rounded to bfloat16 on its way into shared memory, as the framework's other
// products round their inputs; the next step's operands are on their way in registers while this step's multiply.
constexpr int HLT_STRIDE = 40;     // bfloat16 entries a row of a 64 x 32 tile takes (80 bytes: ldmatrix without conflicts)

template <typename TO>
__global__ void __launch_bounds__(128) head_linear_tc_kernel(const float* x, long long ldx, long long xh,
                                                             const bf16* __restrict__ W, TO* out, long long ldo,
                                                             long long oh, int n, int O, int I, const float* gate,
                                                             long long ld_gate) {
  __shared__ __align__(16) bf16 As[64 * HLT_STRIDE];
  __shared__ __align__(16) bf16 Bs[64 * HLT_STRIDE];
  pdl_trigger();
  const int lane = threadIdx.x & 31, wm = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int h = blockIdx.z, r0 = blockIdx.y * 64, c0 = blockIdx.x * 64;
  const float* xb = x + (size_t)h * xh;
  const bf16* wb = W + (size_t)h * O * I;
  float acc[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  float4 ra[4];
  uint4 rb[2];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int idx = threadIdx.x + 128 * u, row = idx >> 3, c = k0 + 4 * (idx & 7);
      ra[u] = (r0 + row < n && c < I) ? *reinterpret_cast<const float4*>(xb + (size_t)(r0 + row) * ldx + c)
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int idx = threadIdx.x + 128 * u, row = idx >> 2, c = k0 + 8 * (idx & 3);
      rb[u] = (c0 + row < O && c < I) ? *reinterpret_cast<const uint4*>(wb + (size_t)(c0 + row) * I + c)
                                      : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  auto put = [&]() {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int idx = threadIdx.x + 128 * u, row = idx >> 3, c = 4 * (idx & 7);
      uint2 w;
      w.x = ltc_pack(ra[u].x, ra[u].y);
      w.y = ltc_pack(ra[u].z, ra[u].w);
      *reinterpret_cast<uint2*>(As + row * HLT_STRIDE + c) = w;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int idx = threadIdx.x + 128 * u, row = idx >> 2, c = 8 * (idx & 3);
      *reinterpret_cast<uint4*>(Bs + row * HLT_STRIDE + c) = rb[u];
    }
  };
  pdl_wait();
  fetch(0);
  for (int k0 = 0; k0 < I; k0 += 32) {
    __syncthreads();                                       // the last step's tiles have been used
    put();
    __syncthreads();
    if (k0 + 32 < I) fetch(k0 + 32);
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      unsigned a[4];
      ltc_ldmatrix(a, As + (wm * 16 + (lane & 15)) * HLT_STRIDE + ks * 16 + (lane >> 4) * 8);
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        unsigned bb[4];
        ltc_ldmatrix(bb, Bs + (np * 16 + (lane & 7) + (lane >> 4) * 8) * HLT_STRIDE + ks * 16 + ((lane >> 3) & 1) * 8);
        ltc_mma(acc[2 * np], a, bb[0], bb[1]);
        ltc_mma(acc[2 * np + 1], a, bb[2], bb[3]);
      }
    }
  }
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int row = r0 + wm * 16 + g + 8 * half;
    if (row >= n) continue;
    TO* dst = out + (size_t)row * ldo + (size_t)h * oh;
    // (a gate logit per output element, laid out like the outputs of a row)
    const float* gt = gate ? gate + (size_t)row * ld_gate + (size_t)h * oh : nullptr;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int col = c0 + 8 * j + 2 * t4;
      if (col < O) dst[col] = from_f32<TO>(gt ? acc[j][2 * half] * hy_sigmoid(gt[col]) : acc[j][2 * half]);
      if (col + 1 < O) dst[col + 1] = from_f32<TO>(gt ? acc[j][2 * half + 1] * hy_sigmoid(gt[col + 1]) : acc[j][2 * half + 1]);
    }
  }
}

}  // namespace

// Whether the per-head product runs on tensor cores: bfloat16 weights whose rows can be read in 16-byte pieces, 32-bit
// inputs readable four at a time, and at least a tile of rows.
bool gb_head_linear_tc_takes(int n, int I, long long ldx, long long xh, const void* x, const void* W) {
  return n >= 64 && I % 8 == 0 && ldx % 4 == 0 && xh % 4 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)W & 15) == 0;
}

void gb_head_linear_tc_launch(const float* x, long long ldx, long long xh, const bf16* W, void* out, bool out_bf16,
                              long long ldo, long long oh, int n, int H, int O, int I, const float* gate,
                              long long ld_gate, cudaStream_t stream) {
  const dim3 grid(gb_div_up(O, 64), gb_div_up(n, 64), H), block(128);
  if (out_bf16)
    gb_launch(head_linear_tc_kernel<bf16>, grid, block, 0, stream, x, ldx, xh, W, static_cast<bf16*>(out), ldo, oh, n, O, I,
              gate, ld_gate);
  else
    gb_launch(head_linear_tc_kernel<float>, grid, block, 0, stream, x, ldx, xh, W, static_cast<float*>(out), ldo, oh, n, O, I,
              gate, ld_gate);
}

// Whether the tensor-core kernel takes a launch: bfloat16 pages whose rows can be copied in 16-byte pieces (a latent
// and a rotated part of multiples of 8 entries, together at most 576, which is what three tiles of 64 rows leave room
// for in shared memory), no window, at most 64 heads, and a step that carries portions (eight tokens a request on
// average).
bool gb_latent_attention_tc_takes(int n, int R, int H, int r, int dr, int window, bool pages_bf16, const void* pages,
                                  const void* qp, const void* out, long long ldo) {
  return pages_bf16 && dr >= 0 && dr % 8 == 0 && r + dr <= 576 && window == 0 && H >= 1 && H <= LTC_ROWS && r % 8 == 0 && r >= 8 && r <= 512 && R >= 1 &&
         n >= 8 * R && (long long)n * H >= 256 && ((uintptr_t)pages & 15) == 0 && ((uintptr_t)qp & 15) == 0 &&
         ((uintptr_t)out & 7) == 0 && ldo % 2 == 0;
}

// Returns the number of partial results a row has after the launch (1: `out` is final; 2: the caller merges the
// workspace's partial results), or -1 when the kernel's shared memory could not be had.  The key tiles are split in
// two when the launch has few CTAs (a long prompt of one or two requests) and the workspace has the rows.
int gb_latent_attention_tc_launch(const float* qp, const bf16* pages, const int* block_table, int bt_stride, int page_size,
                                  int n_pages, const int* tok_req, const int* tok_pos, const int* q_start,
                                  const float* gate, long long ld_gate, float* out, long long ldo, int n, int R, int H, int r,
                                  int dr, float scale, const float* sink, float* ws, long long ws_rows, int* status,
                                  cudaStream_t stream) {
  LtcParams p;
  p.ws = ws;
  p.dk = r + dr;
  p.stride = 16 * ((p.dk + 15) / 16) + 8;
  p.qp = qp; p.pages = pages; p.block_table = block_table; p.bt_stride = bt_stride; p.page_size = page_size;
  p.n_pages = n_pages; p.tok_req = tok_req; p.tok_pos = tok_pos; p.q_start = q_start; p.n = n; p.R = R; p.gate = gate;
  p.ld_gate = ld_gate; p.out = out; p.ldo = ldo; p.H = H; p.r = r; p.tpt = LTC_ROWS / H;
  p.scale_log2 = scale * 1.4426950408889634f; p.sink = sink; p.status = status;
  const int tiles = gb_div_up(n, p.tpt);                   // (no request has more tokens than the step)
  // (which way a launch goes depends on its numbers of tokens, requests and heads only)
  // two halves where the row tiles alone do not fill the GPU's resident CTAs (two an SM by registers, fewer where three
  // tiles of rows need more than half of an SM's shared memory)
  const size_t smem = sizeof(bf16) * 3 * LTC_ROWS * (size_t)p.stride;
  const int resident = 148 * (smem <= 113 * 1024 ? 2 : 1);
  p.splits = (LTC_SPLIT_KEYS && ws != nullptr && (long long)tiles * R <= resident && n >= 512 * R && 2LL * n * H <= ws_rows) ? 2 : 1;
  int rc;
  if (r <= 64) rc = ltc_launch<64>(p, tiles, R, stream);
  else if (r <= 128) rc = ltc_launch<128>(p, tiles, R, stream);
  else if (r <= 256) rc = ltc_launch<256>(p, tiles, R, stream);
  else if (ltw_smem(p.stride) <= 227 * 1024) {
    static bool raised = false;                            // (before any stream capture replays the launch)
    if (!raised) {
      if (cudaFuncSetAttribute(latent_attention_tc_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) return -1;
      raised = true;
    }
    gb_launch(latent_attention_tc_wide_kernel, dim3(tiles, R, p.splits), dim3(LTW_THREADS), ltw_smem(p.stride), stream, p);
    rc = 0;
  }
  else rc = ltc_launch<512>(p, tiles, R, stream);
  return rc < 0 ? rc : p.splits;
}

// Whether the second kernel takes a launch the first does not: bfloat16 pages whose rows can be copied in 16-byte
// pieces, a latent of at most 512 entries and a row of at most 576.
bool gb_latent_attention_split_takes(int n, int R, int H, int r, int dr, bool pages_bf16, const void* pages, const void* qp,
                                     const void* out, long long ldo) {
  return pages_bf16 && dr >= 0 && dr % 8 == 0 && r + dr <= 576 && H >= 1 && r % 8 == 0 && r >= 8 && r <= 512 && R >= 1 &&
         (long long)n * H <= (1 << 30) && ((uintptr_t)pages & 15) == 0 && ((uintptr_t)qp & 15) == 0 &&
         ((uintptr_t)out & 7) == 0 && ldo % 2 == 0;
}

// `splits` chunks of `chunk` keys (a multiple of the key tile), from the one that holds a row tile's first visible key on; the
// last takes all that follow.
cudaError_t gb_latent_attention_split_launch(const float* qp, const bf16* pages, const int* block_table, int bt_stride,
                                             int page_size, int n_pages, const int* tok_req, const int* tok_pos,
                                             const int* q_start, const float* gate, long long ld_gate, float* out,
                                             long long ldo, int n, int R, int H, int r, int dr, float scale, int window,
                                             const float* sink, float* ws, int splits, int chunk, int* status,
                                             cudaStream_t stream) {
  LtxParams p;
  p.qp = qp; p.pages = pages; p.block_table = block_table; p.bt_stride = bt_stride; p.page_size = page_size;
  p.n_pages = n_pages; p.tok_req = tok_req; p.tok_pos = tok_pos; p.q_start = q_start; p.n = n; p.R = R; p.H = H; p.r = r;
  p.dk = r + dr; p.stride = 16 * ((p.dk + 15) / 16) + 8; p.window = window; p.splits = splits; p.chunk = chunk;
  p.gate = gate; p.ld_gate = ld_gate; p.out = out; p.ldo = ldo; p.ws = ws; p.scale = scale;
  p.sink = sink; p.status = status;
  if (r <= 128) return ltx_launch<16>(p, stream);
  if (r <= 256) return ltx_launch<32>(p, stream);
  return ltx_launch<64>(p, stream);
}
