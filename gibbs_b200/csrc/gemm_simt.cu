// out[m, n] (+)= sum_k A[m, k] * W[n, k] (+ bias[n]) with 32-bit FMA on the CUDA
// cores: the matrix product of the true 32-bit path, and of any operand pair
// the tensor-core kernel does not take (a weight kept in 32-bit beside 16-bit
// activations, sizes it refuses).  No tensor-core mode of any kind is used.
//
// The order of every sum depends on K alone.  K is cut into at most eight segments of equal length
// (simt_segment(K)); inside a segment two accumulators walk its even and its odd k upwards and are
// added at its end, and the segments' sums are added in ascending order.  The kernels below (one
// for a few rows, which spreads the segments over threads, one for a few rows of a short K, one with tiles of rows x columns,
// which spreads them over the CTAs of a cluster) therefore give the same bits however the rows are cut, and
// find parallel work in a narrow weight.  Against 64 bits the sums are off by 0.27 of what one
// accumulator over all of K is (K = 1536: 1.9e-7 against 7.0e-7).  A general kernel (one accumulator over all of K) takes what cannot be read in pieces of
// four elements.
// (MisterTK/gibbs Linear: src/graph/cpu.rs:249-274, 2338-2417; its blocked
// 32-bit product: src/model/nn.rs:383-529.)
#include "common.cuh"

namespace {

constexpr int SEGS = 8;       // at most this many segments of K (one CTA of a cluster each in the tile kernel)
constexpr int SK = 32;        // a segment is a multiple of this long

inline int simt_segment(int K) { return gb_div_up(gb_div_up(K, SEGS), SK) * SK; }

// Two 32-bit accumulators, of the even and of the odd k: a pair of neighbouring elements is one operand of
// fma.rn.f32x2 as it comes from memory (one instruction for two fused multiply-adds, each rounded as fmaf's).
typedef unsigned long long f32x2;
__device__ __forceinline__ void fma2(f32x2& acc, f32x2 a, f32x2 w) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(w));
}
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float sum2(f32x2 v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return lo + hi;
}

// Four consecutive elements in shared memory as 32-bit values, in two pairs.
__device__ __forceinline__ ulonglong2 lds4(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ ulonglong2 lds4(const bf16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&u.x);
  const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
  return make_ulonglong2(pack2(__low2float(lo), __high2float(lo)), pack2(__low2float(hi), __high2float(hi)));
}

// Four consecutive elements on their way to shared memory; zeros where `live` is false (the source
// address is then not read, wherever it points).
__device__ __forceinline__ void copy4(float* dst, const float* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
               ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy4(bf16* dst, const bf16* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;"
               ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(live ? 8 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

__device__ __forceinline__ void store_out(void* out, int out_dtype, int accumulate, size_t o, float v) {
  if (out_dtype == GB_F32) {
    float* of = (float*)out;
    of[o] = accumulate ? of[o] + v : v;
  } else {
    ((bf16*)out)[o] = __float2bfloat16_rn(v);
  }
}

// ---- a few rows (decode): bound by the weight's stream from HBM.  A block takes 8 x CG x CPT columns; a
// thread walks one segment for CPT columns and MT of the RG x MT rows, so a weight of N rows is spread
// over N / (8 CG CPT) blocks and a chain of additions is K / 16 long.  Rows of weight and activations pass
// through a ring of ST stages of 32 k per segment, copied 16 bytes (8 for bfloat16) a thread; the
// weight's first stages are on their way before the kernel in front has finished where no such kernel writes it (`ahead`).  Rows are padded
// to 36 elements, which leaves the 16-byte reads of eight columns without bank conflicts.
// Measured (weights not in L2, us; one accumulator over all of K, no ring before -> now): 2 rows
// 1536 x 4608 51 -> 9, 1536 x 1536 25 -> 3.8, 1536 x 13824 119 -> 19 (4.4 TB/s), 6912 x 1536 94 -> 14,
// 1536 x 65536 417 -> 71 (5.6 TB/s); 8 rows 52 -> 11, 25 -> 7, 120 -> 24, 95 -> 25, 421 -> 83.
constexpr int RPAD = SK + 4;

template <typename TA, typename TW, int RG, int CG, int MT, int CPT, int ST>
struct RowsRing {
  static constexpr int A_SEG = RG * MT * RPAD + 4;                       // (the 4 keep the segments' reads apart)
  static constexpr int W_STAGE = SEGS * 8 * CG * CPT * RPAD;
  static constexpr int A_STAGE = SEGS * A_SEG;
  static constexpr int STAGE = W_STAGE * (int)sizeof(TW) + A_STAGE * (int)sizeof(TA);
  static_assert(SEGS * RG * MT * 8 * CG * CPT * 4 <= STAGE, "the segments' sums take the ring's place");
};

template <typename TA, typename TW, int RG, int CG, int MT, int CPT, int ST>
__global__ void __launch_bounds__(64 * RG * CG)
gemm_simt_rows_kernel(const TA* A, long long lda, const TW* __restrict__ W, long long ldw,
                      const float* __restrict__ bias, void* __restrict__ out, long long ldo, int out_dtype,
                      int accumulate, int M, int N, int K, int L, int ahead) {
  using Ring = RowsRing<TA, TW, RG, CG, MT, CPT, ST>;
  constexpr int NB = 8 * CG * CPT, MR = RG * MT, T = 64 * RG * CG;
  extern __shared__ __align__(16) unsigned char smem[];
  pdl_trigger();
  const int tid = threadIdx.x;
  const int n0 = blockIdx.x * NB;
  const int segs = (K + L - 1) / L, steps = L / SK;
  TW* ws = reinterpret_cast<TW*>(smem);
  TA* as = reinterpret_cast<TA*>(smem + ST * Ring::W_STAGE * sizeof(TW));
  // what this thread copies: four k (at lk) of every T/8-th row of both tiles; the weight's rows are
  // (segment, column) pairs, the activations' (segment, row) pairs
  constexpr int RC = T / 8;                            // 8, 16 or 32 rows at once
  constexpr int WN = SEGS * NB / RC, AN = (SEGS * MR + RC - 1) / RC;
  const int lr = tid >> 3, lk = (tid & 7) * 4;
  auto copy_w = [&](int step) {
    TW* dst = ws + (step % ST) * Ring::W_STAGE + lr * RPAD + lk;
    const int k = step * SK + lk;
#pragma unroll
    for (int i = 0; i < WN; ++i) {
      const int r = lr + RC * i, s = r / NB, n = n0 + r % NB;
      const int gk = s * L + k;
      if (s < segs) copy4(dst + RC * i * RPAD, W + (size_t)n * ldw + gk, n < N && gk < K);      // (the sums of others are not read)
    }
  };
  auto copy_a = [&](int step) {
    TA* dst = as + (step % ST) * Ring::A_STAGE + lk;
    const int k = step * SK + lk;
#pragma unroll
    for (int i = 0; i < AN; ++i) {
      const int r = lr + RC * i, s = r / MR, m = r % MR;
      const int gk = s * L + k;
      if (s >= segs) break;
      copy4(dst + s * Ring::A_SEG + m * RPAD, A + (size_t)m * lda + gk, m < M && gk < K);
    }
  };
  if (!ahead) pdl_wait();
#pragma unroll
  for (int i = 0; i < ST - 1; ++i)
    if (i < steps) copy_w(i);
  if (ahead) pdl_wait();
#pragma unroll
  for (int i = 0; i < ST - 1; ++i) {
    if (i < steps) copy_a(i);
    copies_commit();
  }
  // this thread's row group, segment and columns col + 8 CG j
  const int rg = tid / (64 * CG), seg = (tid >> 3) & 7, col = (tid & 7) + 8 * (tid / 64 % CG);
  f32x2 acc[MT][CPT];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int j = 0; j < CPT; ++j) acc[m][j] = 0;
  for (int step = 0; step < steps; ++step) {
    copies_wait<ST - 2>();
    __syncthreads();                                   // the stage has arrived, the one before it has been used
    if (step + ST - 1 < steps) {
      copy_w(step + ST - 1);
      copy_a(step + ST - 1);
    }
    copies_commit();
    const TW* w = ws + (step % ST) * Ring::W_STAGE + (seg * NB + col) * RPAD;
    const TA* a = as + (step % ST) * Ring::A_STAGE + seg * Ring::A_SEG + rg * MT * RPAD;
#pragma unroll
    for (int k = 0; k < SK; k += 4) {
      ulonglong2 wv[CPT];
#pragma unroll
      for (int j = 0; j < CPT; ++j) wv[j] = lds4(w + j * 8 * CG * RPAD + k);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const ulonglong2 av = lds4(a + m * RPAD + k);
#pragma unroll
        for (int j = 0; j < CPT; ++j) {
          fma2(acc[m][j], av.x, wv[j].x);
          fma2(acc[m][j], av.y, wv[j].y);
        }
      }
    }
  }
  copies_wait<0>();
  __syncthreads();                                     // the ring is free: the segments' sums go there
  float* red = reinterpret_cast<float*>(smem);         // [segment][row][column]
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int j = 0; j < CPT; ++j) red[(seg * MR + rg * MT + m) * NB + j * 8 * CG + col] = sum2(acc[m][j]);
  __syncthreads();
  for (int i = tid; i < MR * NB; i += T) {
    const int m = i / NB, n = n0 + i % NB;
    if (m >= M || n >= N) continue;
    float v = 0.f;
    for (int s = 0; s < segs; ++s) v += red[s * MR * NB + i];
    if (bias) v += bias[n];
    store_out(out, out_dtype, accumulate, (size_t)m * ldo + n, v);
  }
}

// ---- a few rows of up to four segments of 32: a block takes 16 columns and up to 16 rows, an output a thread, so little that the
// next kernel's blocks find room beside it; the sums in the same order as above.  Measured (us; the kernel above -> this one): 16
// rows 64 x 2048 3.2 -> 2.0, 8 rows 3.0 -> 2.1, 16 rows 128 x 2048 3.3 -> 3.1, 96 x 1000 2.8 -> 2.5.
// Four consecutive elements as 32-bit values, through L2 (the compiler must not take them for invariant: see common.cuh).
__device__ __forceinline__ float4 load4(const float* p) { return ldcg_now(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 load4(const bf16* p) {
  uint2 u;
  asm volatile("ld.global.cg.v2.u32 {%0, %1}, [%2];" : "=r"(u.x), "=r"(u.y) : "l"(p));
  const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&u.x);
  const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
  return make_float4(__low2float(lo), __high2float(lo), __low2float(hi), __high2float(hi));
}

template <typename TA, typename TW>
__global__ void __launch_bounds__(256)
gemm_simt_short_kernel(const TA* A, long long lda, const TW* __restrict__ W, long long ldw, const float* __restrict__ bias,
                       void* __restrict__ out, long long ldo, int out_dtype, int accumulate, int M, int N, int K, int ahead) {
  constexpr int KB = 2 * SK;
  __shared__ float As[16][KB + 1], Ws[16][KB + 1];
  pdl_trigger();
  const int tid = threadIdx.x, tn = tid & 15, tm = tid >> 4;       // this thread's output: row tm, column n0 + tn
  const int n0 = blockIdx.x * 16, lr = tid >> 4, lk = (tid & 15) * 4;      // what it fetches: four k of row lr of both
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!ahead) pdl_wait();
  float4 fw = n0 + lr < N && lk < K ? load4(W + (size_t)(n0 + lr) * ldw + lk) : none;
  if (ahead) pdl_wait();
  float4 fa = lr < M && lk < K ? load4(A + (size_t)lr * lda + lk) : none;
  float v = 0.f;
  for (int k0 = 0; k0 < K; k0 += KB) {
    As[lr][lk] = fa.x; As[lr][lk + 1] = fa.y; As[lr][lk + 2] = fa.z; As[lr][lk + 3] = fa.w;
    Ws[lr][lk] = fw.x; Ws[lr][lk + 1] = fw.y; Ws[lr][lk + 2] = fw.z; Ws[lr][lk + 3] = fw.w;
    __syncthreads();
    const int gk = k0 + KB + lk;
    if (k0 + KB < K) {
      fa = lr < M && gk < K ? load4(A + (size_t)lr * lda + gk) : none;
      fw = n0 + lr < N && gk < K ? load4(W + (size_t)(n0 + lr) * ldw + gk) : none;
    }
#pragma unroll
    for (int s = 0; s < KB; s += SK) {
      float even = 0.f, odd = 0.f;
#pragma unroll
      for (int k = 0; k < SK; k += 2) {
        even = fmaf(As[tm][s + k], Ws[tn][s + k], even);
        odd = fmaf(As[tm][s + k + 1], Ws[tn][s + k + 1], odd);
      }
      if (k0 + s < K) v += even + odd;
    }
    __syncthreads();
  }
  if (tm < M && n0 + tn < N) {
    if (bias) v += bias[n0 + tn];
    store_out(out, out_dtype, accumulate, (size_t)tm * ldo + n0 + tn, v);
  }
}

// ---- more rows: bound by the FMA pipe (and near it, by the reads of shared memory that feed it).  Tiles
// of 32 rows x 64 columns, one warp, 8 x 8 outputs a thread.  The CTAs of a cluster take a segment of K
// each and add their tiles through distributed shared memory, so that a narrow product of a short prompt
// still fills the chip and no workspace or second launch is needed; one warp a CTA waits for nobody else's
// copies.  A quarter of a warp reads one row of activations and eight of weights (pad 4: no conflicts).
// Measured (225 rows, us; 128 x 128 tiles over the whole of K before -> now): 1536 x 4608 213 -> 97,
// 1536 x 1536 197 -> 43, 1536 x 13824 307 -> 262 (36 TFLOP/s of the 72 an FMA loop reaches), 6912 x 1536
// 887 -> 169; 1600 rows: 587 -> 528, 301 -> 186, 1490 -> 1523, 1334 -> 769; 60 rows (the general kernel
// before) 1536 x 1536 310 -> 22.  From about 900 rows on a wide weight is slower than on those 128 x 128 tiles, whose
// single accumulator an output left room for 16 warps an SM (1024 rows 1536 x 4608 302 -> 344, 1536 x 13824 902 -> 978; 2134
// rows 128 x 2048 29 -> 37).  Tiles of 64 x 64, 64 x 128 and 128 x 128 by copies: 2 to 10% slower; of 128 x 64 and 128 x 128
// with K k by k in shared memory, 16 and 8 warps an SM, 1600 rows 1536 x 13824: 1984 and 1978; stages of
// 16 k 10% (twice the cache lines a copy touches), more CTAs an SM by fewer registers 40% (spills).
constexpr int BM = 32, BNT = 64;                       // a tile
constexpr int TK = SK, TPAD = TK + 4, TST = 2;         // a ring of two stages of 32 k

template <typename TA, typename TW>
struct TileSmem {
  static constexpr int RING = TST * TPAD * (BM * (int)sizeof(TA) + BNT * (int)sizeof(TW));
  static constexpr int LD = BNT + 8;               // (eight columns of four rows are stored at once)
  static constexpr int SUMS = BM * LD * 4;
  static constexpr int BYTES = RING > SUMS ? RING : SUMS;      // (the sums take the ring's place)
};

template <typename TA, typename TW, bool WHOLE>
__global__ void __launch_bounds__(BM * BNT / 64, 8)
gemm_simt_tile_kernel(const TA* A, long long lda, const TW* __restrict__ W, long long ldw,
                      const float* __restrict__ bias, void* __restrict__ out, long long ldo, int out_dtype,
                      int accumulate, int M, int N, int K, int L, int segs, int ahead) {
  constexpr int T = BM * BNT / 64, TX = BNT / 8, TY = BM / 8, RT = T * 4 / TK;     // RT rows of a tile are copied at once
  static_assert(BM % RT == 0 && BNT % RT == 0, "");
  extern __shared__ __align__(16) unsigned char smem[];
  TA* as = reinterpret_cast<TA*>(smem);
  TW* ws = reinterpret_cast<TW*>(smem + TST * TPAD * BM * sizeof(TA));
  pdl_trigger();
  const int tid = threadIdx.x;
  const int seg = blockIdx.x % segs;                                       // (= the CTA's rank in its cluster)
  const int n0 = (blockIdx.x / segs) * BNT, m0 = blockIdx.y * BM;
  const int k_lo = seg * L, k_hi = WHOLE ? K : min(K, k_lo + L);
  const int steps = (k_hi - k_lo + TK - 1) / TK;
  const int lr = tid / (TK / 4), lk = tid % (TK / 4) * 4;
  auto copy_w = [&](int step) {
    TW* dst = ws + (step % TST) * TPAD * BNT + lr * TPAD + lk;
    const int k = k_lo + step * TK + lk;
    const int rows = k < k_hi ? N - n0 - lr : 0;
    const TW* src = W + (size_t)(n0 + lr) * ldw + k;
#pragma unroll
    for (int i = 0; i < BNT / RT; ++i, src += RT * ldw) copy4(dst + RT * i * TPAD, src, RT * i < rows);
  };
  auto copy_a = [&](int step) {
    TA* dst = as + (step % TST) * TPAD * BM + lr * TPAD + lk;
    const int k = k_lo + step * TK + lk;
    const int rows = k < k_hi ? M - m0 - lr : 0;
    const TA* src = A + (size_t)(m0 + lr) * lda + k;
#pragma unroll
    for (int i = 0; i < BM / RT; ++i, src += RT * lda) copy4(dst + RT * i * TPAD, src, RT * i < rows);
  };
  if (!ahead) pdl_wait();
#pragma unroll
  for (int i = 0; i < TST - 1; ++i)
    if (i < steps) copy_w(i);
  if (ahead) pdl_wait();
#pragma unroll
  for (int i = 0; i < TST - 1; ++i) {
    if (i < steps) copy_a(i);
    copies_commit();
  }
  constexpr int LD = TileSmem<TA, TW>::LD;
  float* sums = reinterpret_cast<float*>(smem);        // [BM][LD]
  const int tx = tid % TX, ty = tid / TX;              // outputs: rows ty + TY i, columns tx + TX j
  f32x2 acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0;
  float done[WHOLE ? 8 : 1][WHOLE ? 8 : 1];            // (a CTA for all segments: the sums of those before; in registers, so that as many CTAs stay on an SM)
  for (int step = 0; step < steps; ++step) {
    copies_wait<TST - 2>();
    __syncthreads();
    if (step + TST - 1 < steps) {
      copy_w(step + TST - 1);
      copy_a(step + TST - 1);
    }
    copies_commit();
    const TA* a = as + ((step % TST) * BM + ty) * TPAD;
    const TW* w = ws + ((step % TST) * BNT + tx) * TPAD;
#pragma unroll
    for (int k = 0; k < TK; k += 4) {
      ulonglong2 av[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) av[i] = lds4(a + i * TY * TPAD + k);
      ulonglong2 next = lds4(w + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const ulonglong2 wv = next;                    // (the next column's four are asked for ahead of this one's products)
        if (j < 7) next = lds4(w + (j + 1) * TX * TPAD + k);
#pragma unroll
        for (int i = 0; i < 8; ++i) fma2(acc[i][j], av[i].x, wv.x);
#pragma unroll
        for (int i = 0; i < 8; ++i) fma2(acc[i][j], av[i].y, wv.y);
      }
    }
    if (WHOLE && ((step + 1) % (L / TK) == 0 || step + 1 == steps)) {
      const bool first = step < L / TK;
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float& d = done[WHOLE ? i : 0][WHOLE ? j : 0];
          d = (first ? 0.f : d) + sum2(acc[i][j]);
          acc[i][j] = 0;
        }
    }
  }
  copies_wait<0>();
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      sums[(ty + TY * i) * LD + tx + TX * j] = WHOLE ? done[WHOLE ? i : 0][WHOLE ? j : 0] : sum2(acc[i][j]);
  // every CTA adds and stores its share of the tile, four columns a thread
  if constexpr (WHOLE) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  constexpr int QUADS = BM * BNT / 4;
  const int share = (QUADS + segs - 1) / segs;
  const int q_end = min(QUADS, (seg + 1) * share);
  const unsigned base = (unsigned)__cvta_generic_to_shared(sums);
  const bool vec = out_dtype == GB_F32 && ldo % 4 == 0 && ((uintptr_t)out & 15) == 0;
  for (int q = seg * share + tid; q < q_end; q += T) {
    const int gm = m0 + q / (BNT / 4), gn = n0 + (q % (BNT / 4)) * 4;
    if (gm >= M || gn >= N) continue;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if constexpr (WHOLE) {
      const float4 x = *reinterpret_cast<const float4*>(sums + q / (BNT / 4) * LD + q % (BNT / 4) * 4);
      v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
    float4 p[SEGS];
#pragma unroll
    for (int s = 0; s < SEGS; ++s) {
      if (s >= segs) break;
      unsigned at;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(base + 4u * (q / (BNT / 4) * LD + q % (BNT / 4) * 4)), "r"(s));
      asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(p[s].x), "=f"(p[s].y), "=f"(p[s].z), "=f"(p[s].w) : "r"(at) : "memory");
    }
#pragma unroll
    for (int s = 0; s < SEGS; ++s) {
      if (s >= segs) break;
      v[0] += p[s].x; v[1] += p[s].y; v[2] += p[s].z; v[3] += p[s].w;
    }
    }
    if (bias) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (gn + e < N) v[e] += bias[gn + e];
    }
    const size_t o = (size_t)gm * ldo + gn;
    if (vec && gn + 3 < N) {
      float4* of = reinterpret_cast<float4*>((float*)out + o);
      if (accumulate) {
        const float4 x = *of;
        v[0] = x.x + v[0]; v[1] = x.y + v[1]; v[2] = x.z + v[2]; v[3] = x.w + v[3];
      }
      *of = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (gn + e < N) store_out(out, out_dtype, accumulate, o + e, v[e]);
    }
  }
  // (a CTA's shared memory stays until its peers have read it)
  if constexpr (!WHOLE) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// ---- the general kernel: any sizes and strides, one accumulator over all of K

constexpr int BN = 64;
constexpr int BK = 16;

template <typename TA, typename TW, int TM>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TA* A, long long lda, const TW* __restrict__ W, long long ldw,
                 const float* __restrict__ bias, void* __restrict__ out, long long ldo, int out_dtype,
                 int accumulate, int M, int N, int K) {
  pdl_trigger();
  pdl_wait();
  constexpr int BM = 16 * TM;
  __shared__ float As[BK][BM + 1];
  __shared__ float Ws[BK][BN + 1];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;

  float acc[TM][4];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    for (int idx = tid; idx < BM * BK; idx += 256) {
      const int m = idx / BK, k = idx % BK;
      const int gm = m0 + m, gk = k0 + k;
      As[k][m] = (gm < M && gk < K) ? to_f32(A[(size_t)gm * lda + gk]) : 0.f;
    }
    for (int idx = tid; idx < BN * BK; idx += 256) {
      const int n = idx / BK, k = idx % BK;
      const int gn = n0 + n, gk = k0 + k;
      Ws[k][n] = (gn < N && gk < K) ? to_f32(W[(size_t)gn * ldw + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[TM], w[4];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[k][ty * TM + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = Ws[k][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }

#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty * TM + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[gn];
      store_out(out, out_dtype, accumulate, (size_t)gm * ldo + gn, v);
    }
  }
}

template <typename TA, typename TW, int RG, int CG, int MT, int CPT, int ST>
cudaError_t launch_rows(const TA* A, long long lda, const TW* W, long long ldw, const float* bias, void* out, long long ldo,
                        int out_dtype, int accumulate, int ahead, int M, int N, int K, cudaStream_t stream) {
  auto kernel = gemm_simt_rows_kernel<TA, TW, RG, CG, MT, CPT, ST>;
  constexpr int stage = RowsRing<TA, TW, RG, CG, MT, CPT, ST>::STAGE;
  const int smem = ST * stage;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ST * stage);
  if (e != cudaSuccess) return e;
  return gb_launch(kernel, dim3(gb_div_up(N, 8 * CG * CPT)), dim3(64 * RG * CG), smem, stream, A, lda, W, ldw, bias, out, ldo, out_dtype,
                   accumulate, M, N, K, simt_segment(K), ahead);
}

template <typename TA, typename TW>
cudaError_t launch_tile(const TA* A, long long lda, const TW* W, long long ldw, const float* bias, void* out, long long ldo,
                        int out_dtype, int accumulate, int ahead, int M, int N, int K, cudaStream_t stream) {
  using Smem = TileSmem<TA, TW>;
  static_assert(Smem::BYTES <= 48 * 1024, "no more shared memory than every launch may have");
  const int L = simt_segment(K);
  const long long tiles = (long long)gb_div_up(M, BM) * gb_div_up(N, BNT);
  // Whether one CTA takes all segments of a tile: short ones are over before the CTA of each has started and ended (us of a CTA a
  // segment and of one for all: 2134 rows 128 x 2048 50 and 37, 64 x 2048 29 and 21, 1600 rows 39 and 29), and where there are
  // many rounds of tiles there is nothing to spread (1600 rows 1536 x 13824 1553 and 1524, 225 rows 1536 x 65536 1182 and 1133; but
  // 1024 rows 1536 x 1536, 1.3 rounds of the eight an SM holds, 125 and 180, 1600 rows 1536 x 4608, 3 rounds, 528 and 571).
  const bool whole = L < 128 ? tiles >= 4 * 148 : tiles >= 5 * 8 * 148;
  const int segs = whole ? 1 : gb_div_up(K, L);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)gb_div_up(N, BNT) * segs, gb_div_up(M, BM));
  cfg.blockDim = dim3(BM * BNT / 64);
  cfg.dynamicSmemBytes = Smem::BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[gb_pdl_enabled() ? 1 : 0].id = cudaLaunchAttributeClusterDimension;
  attr[gb_pdl_enabled() ? 1 : 0].val.clusterDim.x = segs;
  attr[gb_pdl_enabled() ? 1 : 0].val.clusterDim.y = 1;
  attr[gb_pdl_enabled() ? 1 : 0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (gb_pdl_enabled() ? 1 : 0) + (whole ? 0 : 1);
  auto kernel = whole ? gemm_simt_tile_kernel<TA, TW, true> : gemm_simt_tile_kernel<TA, TW, false>;
  return cudaLaunchKernelEx(&cfg, kernel, A, lda, W, ldw, bias, out, ldo, out_dtype, accumulate, M, N, K, L, segs, ahead);
}

template <typename TA, typename TW>
cudaError_t launch(const void* a, long long lda, const void* w, long long ldw, const float* bias, void* out, long long ldo,
                   int out_dtype, int accumulate, int ahead, int M, int N, int K, cudaStream_t stream) {
  const TA* A = (const TA*)a;
  const TW* W = (const TW*)w;
  // (K up to 2^30: the last segment's end is worked out in 32 bits)
  const bool rows4 = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A % (4 * sizeof(TA))) == 0 &&
                     ((uintptr_t)W % (4 * sizeof(TW))) == 0 && K <= (1 << 30);
#define GB_ARGS A, lda, W, ldw, bias, out, ldo, out_dtype, accumulate, ahead, M, N, K, stream
  if (rows4 && M <= 16) {
    // Every block reads the same activations, all of them at about the same k, so those few lines of L2
    // bound the stream: 32 columns a block where the weight has enough rows for the chip (two rows,
    // 1536 x 65536: 71 us against 97 with 8 columns), 8 and a deeper ring where it is narrow, unless the ring would not turn (up
    // to four rows, 128 x 2048: 2.1 us against 2.4).
    const bool wide = N >= 16 * 148 || (M <= 4 && simt_segment(K) <= 2 * SK && N >= 6 * 148);
    if (K <= 4 * SK && (M > 8 || (M > 2 && K <= 2 * SK)))
      return gb_launch(gemm_simt_short_kernel<TA, TW>, dim3(gb_div_up(N, 16)), dim3(256), 0, stream, A, lda, W, ldw, bias, out, ldo,
                       out_dtype, accumulate, M, N, K, ahead);
    if (M == 1) return wide ? launch_rows<TA, TW, 1, 2, 1, 2, 2>(GB_ARGS) : launch_rows<TA, TW, 1, 1, 1, 1, 6>(GB_ARGS);
    if (M == 2) return wide ? launch_rows<TA, TW, 1, 2, 2, 2, 2>(GB_ARGS) : launch_rows<TA, TW, 1, 1, 2, 1, 6>(GB_ARGS);
    if (M <= 4) return wide ? launch_rows<TA, TW, 1, 2, 4, 2, 2>(GB_ARGS) : launch_rows<TA, TW, 1, 1, 4, 1, 6>(GB_ARGS);
    if (M <= 8) return wide ? launch_rows<TA, TW, 2, 2, 4, 2, 2>(GB_ARGS) : launch_rows<TA, TW, 2, 1, 4, 1, 4>(GB_ARGS);
    return wide ? launch_rows<TA, TW, 4, 2, 4, 2, 2>(GB_ARGS) : launch_rows<TA, TW, 4, 1, 4, 1, 4>(GB_ARGS);
  }
  if (rows4 && gb_div_up(N, BNT) <= 2147483647LL / SEGS) {
    return launch_tile<TA, TW>(GB_ARGS);
  }
#undef GB_ARGS
  if (M <= 16) {
    dim3 grid(gb_div_up(N, BN), gb_div_up(M, 16));
    return gb_launch(gemm_simt_kernel<TA, TW, 1>, dim3(grid), dim3(256), 0, stream, A, lda, W, ldw, bias, out, ldo, out_dtype,
                     accumulate, M, N, K);
  }
  dim3 grid(gb_div_up(N, BN), gb_div_up(M, 64));
  return gb_launch(gemm_simt_kernel<TA, TW, 4>, dim3(grid), dim3(256), 0, stream, A, lda, W, ldw, bias, out, ldo, out_dtype,
                   accumulate, M, N, K);
}

}  // namespace

// A: [M, K] with row stride lda; W: [N, K] with row stride ldw; out: [M, N]
// with row stride ldo (strides in elements).  `mode` bits 0 to 29, if any is set: adds into a 32-bit output; bit 30: W and the
// bias are a model's, which no kernel in front on the stream writes, so that W is asked for before those kernels have finished.
GB_API int gb_linear_simt(const void* A, int a_dtype, long long lda, const void* W, int w_dtype, long long ldw,
                          const float* bias, void* out, int out_dtype, long long ldo, int mode, int M, int N, int K,
                          cudaStream_t stream) {
  const int accumulate = (mode & ~(1 << 30)) != 0, ahead = (mode >> 30) & 1;
  if (M <= 0 || N <= 0) return GB_OK;
  if (K <= 0) GB_FAIL(GB_ERR_ARG, "gb_linear_simt: K = %d", K);
  if (accumulate && out_dtype != GB_F32)
    GB_FAIL(GB_ERR_ARG, "gb_linear_simt: accumulation needs a 32-bit output");
  if (out_dtype != GB_F32 && out_dtype != GB_BF16) GB_FAIL(GB_ERR_ARG, "gb_linear_simt: output dtype %d", out_dtype);
  if (gb_div_up(M, 16) > 65535 || gb_div_up(N, 16) > 2147483647LL)
    GB_FAIL(GB_ERR_ARG, "gb_linear_simt: M = %d or N = %d is too large", M, N);
  cudaError_t e;
  if (a_dtype == GB_F32 && w_dtype == GB_F32)
    e = launch<float, float>(A, lda, W, ldw, bias, out, ldo, out_dtype, accumulate, ahead, M, N, K, stream);
  else if (a_dtype == GB_BF16 && w_dtype == GB_BF16)
    e = launch<bf16, bf16>(A, lda, W, ldw, bias, out, ldo, out_dtype, accumulate, ahead, M, N, K, stream);
  else if (a_dtype == GB_BF16 && w_dtype == GB_F32)
    e = launch<bf16, float>(A, lda, W, ldw, bias, out, ldo, out_dtype, accumulate, ahead, M, N, K, stream);
  else if (a_dtype == GB_F32 && w_dtype == GB_BF16)
    e = launch<float, bf16>(A, lda, W, ldw, bias, out, ldo, out_dtype, accumulate, ahead, M, N, K, stream);
  else
    GB_FAIL(GB_ERR_ARG, "gb_linear_simt: operand dtypes %d, %d", a_dtype, w_dtype);
  if (e != cudaSuccess) GB_FAIL(GB_ERR_CUDA, "gb_linear_simt: %s", cudaGetErrorString(e));
  GB_CHECK_LAUNCH("gb_linear_simt");
  return GB_OK;
}
