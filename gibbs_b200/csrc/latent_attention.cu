// Attention over a compressed ("latent") key/value cache, in the absorbed form.
//
// A token's cache row is [c | k_rot]: the RMS-normed latent c (kv_rank values), from which every head's
// unrotated keys W_uk c and values W_uv c derive, and one rotated key part shared by all heads.  With
//   q'_h = [W_uk,h^T q_plain,h | rot(q_rot,h)]
// the score of head h against a cached row is q'_h . [c | k_rot], and the head's output is
// W_uv,h (sum_j p_j c_j): nothing but the cache rows is read per key, for prompts and decoding alike.
//
//  gb_op_latent_prep       RMS norm of the latent and rotation of the shared key part, written into the
//                          token's page; rotation of the queries' rotated parts into q'
//  gb_op_head_linear       out[t, h, :] = x[t, h, :] W[h]^T for every head (absorbing W_uk, applying W_uv)
//  gb_op_latent_attention  softmax(scale * q' . rows) over the last `window` rows (all when 0), times the
//                          rows' latent part, times sigmoid(gate[t, h]) where there is a gate; with a sink,
//                          exp(sink[h]) is added to the softmax's denominator; scores and weights in 32-bit
//
// Rotation: the first `rot_dims` entries of a rotated part turn in adjacent pairs (2i, 2i+1) by
// pos * inv_freq[i] (angle in 32-bit); the rest passes unchanged.
// Pages: [n_pages, page_size, kv_rank + rot_dim]; a page id outside the pool is never dereferenced: the
// access is skipped and *status is set.
#include "hybrid.cuh"

namespace {

enum { STATUS_BAD_PAGE_WRITE = 1, STATUS_BAD_PAGE_READ = 2 };

// one block per token: warp 0 writes the cache row, the others rotate the heads' queries
template <typename TC, int ROT, int LAT>                   // rotated pairs and latent entries a lane holds
__global__ void latent_prep_kernel(const float* fused, long long ld, int dkv_col, const float* queries, long long ldq,
                                   const float* __restrict__ gain,
                                   const float* __restrict__ inv_freq, int rot_dims, const int* tok_req,
                                   const int* tok_pos, const int* block_table, int bt_stride, int page_size, TC* pages,
                                   int n_pages, int H, int dn, int dr, int r, float* qp, float eps, int* status) {
  pdl_trigger();
  const int t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int pos = tok_pos[t];
  const int half = rot_dims >> 1;
  // The angles, the page and the gains are known before the kernel in front has finished (pinned, see gb_pin); behind the wait
  // all of a row's values are asked for before the first is used.
  constexpr int HEADS = 3;                                 // heads a warp takes at a time
  const bool rot_here = half <= 32 * ROT, lat_here = r <= 32 * LAT;
  float c[ROT], s[ROT], g[LAT];
#pragma unroll
  for (int i = 0; i < ROT; ++i) {
    const int j = lane + 32 * i;
    c[i] = s[i] = 0.f;
    if (rot_here && 32 * i < half) {                       // (the same in a whole warp: what no lane needs is not worked out)
      const float ang = j < half ? (float)pos * inv_freq[j] : 0.f;
      c[i] = cosf(ang);
      s[i] = sinf(ang);
    }
    gb_pin(c[i]);
    gb_pin(s[i]);
  }
  int page = 0;
  if (warp == 0) {
    page = block_table[(size_t)tok_req[t] * bt_stride + pos / page_size];
#pragma unroll
    for (int i = 0; i < LAT; ++i) {
      g[i] = lat_here && lane + 32 * i < r ? gain[lane + 32 * i] : 0.f;
      gb_pin(g[i]);
    }
  }
  gb_pin(page);
  pdl_wait();
  const float* row = fused + (size_t)t * ld;
  if (warp == 0) {
    if (page < 0 || page >= n_pages) {
      if (lane == 0) atomicExch(status, STATUS_BAD_PAGE_WRITE);
    } else {
      TC* dst = pages + ((size_t)page * page_size + pos % page_size) * (r + dr);
      const float* lat = row + dkv_col;
      const float* kr = lat + r;
      float u[ROT], v[ROT];
#pragma unroll
      for (int i = 0; i < ROT; ++i) {
        const int j = lane + 32 * i;
        u[i] = rot_here && j < half ? ldcg_now(kr + 2 * j) : 0.f;
        v[i] = rot_here && j < half ? ldcg_now(kr + 2 * j + 1) : 0.f;
      }
      float ss = 0.f;
      if (lat_here) {
        float x[LAT];
#pragma unroll
        for (int i = 0; i < LAT; ++i) {
          x[i] = 0.f;
          if (32 * i < r && lane + 32 * i < r) x[i] = ldcg_now(lat + lane + 32 * i);
        }
#pragma unroll
        for (int i = 0; i < LAT; ++i)
          if (lane + 32 * i < r) ss += x[i] * x[i];
        const float rstd = 1.0f / sqrtf(warp_sum(ss) / (float)r + eps);
#pragma unroll
        for (int i = 0; i < LAT; ++i)
          if (lane + 32 * i < r) dst[lane + 32 * i] = from_f32<TC>(x[i] * rstd * g[i]);
      } else {
        for (int d = lane; d < r; d += 32) ss += lat[d] * lat[d];
        const float rstd = 1.0f / sqrtf(warp_sum(ss) / (float)r + eps);
        for (int d = lane; d < r; d += 32) dst[d] = from_f32<TC>(lat[d] * rstd * gain[d]);
      }
#pragma unroll
      for (int i = 0; i < ROT; ++i) {
        const int j = lane + 32 * i;
        if (rot_here && j < half) {
          dst[r + 2 * j] = from_f32<TC>(u[i] * c[i] - v[i] * s[i]);
          dst[r + 2 * j + 1] = from_f32<TC>(v[i] * c[i] + u[i] * s[i]);
        }
      }
      if (!rot_here)
        for (int j = lane; j < half; j += 32) {
          const float ang = (float)pos * inv_freq[j], cj = cosf(ang), sj = sinf(ang);
          const float uj = kr[2 * j], vj = kr[2 * j + 1];
          dst[r + 2 * j] = from_f32<TC>(uj * cj - vj * sj);
          dst[r + 2 * j + 1] = from_f32<TC>(vj * cj + uj * sj);
        }
      for (int d = 2 * half + lane; d < dr; d += 32) dst[r + d] = from_f32<TC>(kr[d]);
    }
  }
  const int w0 = warps > 1 ? 1 : 0, step = warps > 1 ? warps - 1 : 1;
  if (warps > 1 && warp == 0) return;
  const float* q0 = queries + (size_t)t * ldq + dn;        // a head's rotated part lies dn behind its first entry
  float* o0 = qp + (size_t)t * H * (r + dr) + r;
  if (dr == 0) return;
  for (int h0 = warp - w0; h0 < H; h0 += HEADS * step) {
    float u[HEADS][ROT], v[HEADS][ROT];
#pragma unroll
    for (int k = 0; k < HEADS; ++k)
#pragma unroll
      for (int i = 0; i < ROT; ++i) {
        const int h = h0 + k * step, j = lane + 32 * i;
        const bool in = rot_here && h < H && j < half;
        u[k][i] = in ? ldcg_now(q0 + (size_t)h * (dn + dr) + 2 * j) : 0.f;
        v[k][i] = in ? ldcg_now(q0 + (size_t)h * (dn + dr) + 2 * j + 1) : 0.f;
      }
#pragma unroll
    for (int k = 0; k < HEADS; ++k) {
      const int h = h0 + k * step;
      if (h >= H) break;
      const float* q = q0 + (size_t)h * (dn + dr);
      float* o = o0 + (size_t)h * (r + dr);
#pragma unroll
      for (int i = 0; i < ROT; ++i) {
        const int j = lane + 32 * i;
        if (rot_here && j < half) {
          o[2 * j] = u[k][i] * c[i] - v[k][i] * s[i];
          o[2 * j + 1] = v[k][i] * c[i] + u[k][i] * s[i];
        }
      }
      if (!rot_here)
        for (int j = lane; j < half; j += 32) {
          const float ang = (float)pos * inv_freq[j], cj = cosf(ang), sj = sinf(ang);
          const float uj = q[2 * j], vj = q[2 * j + 1];
          o[2 * j] = uj * cj - vj * sj;
          o[2 * j + 1] = vj * cj + uj * sj;
        }
      for (int d = 2 * half + lane; d < dr; d += 32) o[d] = q[d];
    }
  }
}

template <typename TW, typename TO>
__global__ void head_linear_kernel(const float* x, long long ldx, long long xh, const TW* __restrict__ W, TO* out,
                                   long long ldo, long long oh, int n, int O, int I, const float* gate, long long ld_gate) {
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.z, r0 = blockIdx.y * 64, c0 = blockIdx.x * 64;
  const float* xb = x + (size_t)h * xh;
  const TW* wb = W + (size_t)h * O * I;
  float acc[4][4];
  int ty, tx;
  hy_tile_64x64<float, TW>(
      [&](int i) -> const float* { return r0 + i < n ? xb + (size_t)(r0 + i) * ldx : nullptr; },
      [&](int j) -> const TW* { return c0 + j < O ? wb + (size_t)(c0 + j) * I : nullptr; }, I, acc, ty, tx);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int row = r0 + ty * 4 + r;
    if (row >= n) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int col = c0 + tx * 4 + c;
      if (col < O) {
        const float gt = gate ? hy_sigmoid(gate[(size_t)row * ld_gate + (size_t)h * oh + col]) : 1.f;
        out[(size_t)row * ldo + (size_t)h * oh + col] = from_f32<TO>(gate ? acc[r][c] * gt : acc[r][c]);
      }
    }
  }
}

// A few rows (decoding): one block per (8 outputs, head), the head's inputs of all rows in shared memory,
// one warp per output with the lanes over the inputs.
constexpr int HL_SMALL_ROWS = 16;

template <typename TW, typename TO>
__global__ void head_linear_small_kernel(const float* x, long long ldx, long long xh, const TW* __restrict__ W, TO* out,
                                         long long ldo, long long oh, int n, int O, int I, const float* gate,
                                         long long ld_gate) {
  extern __shared__ float xs[];                          // [n][I]
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < n * I; i += blockDim.x) {
    const int t = i / I;
    xs[i] = x[(size_t)t * ldx + (size_t)h * xh + (i - t * I)];
  }
  __syncthreads();
  {
    const int o = blockIdx.x * (blockDim.x >> 5) + warp;
    if (o >= O) return;
    const TW* w = W + ((size_t)h * O + o) * I;
    float acc[HL_SMALL_ROWS];
#pragma unroll
    for (int t = 0; t < HL_SMALL_ROWS; ++t) acc[t] = 0.f;
    for (int i = lane; i < I; i += 32) {
      const float wv = to_f32(w[i]);
#pragma unroll
      for (int t = 0; t < HL_SMALL_ROWS; ++t)
        if (t < n) acc[t] = fmaf(xs[t * I + i], wv, acc[t]);
    }
#pragma unroll
    for (int t = 0; t < HL_SMALL_ROWS; ++t) {
      if (t < n) {
        const float v = warp_sum(acc[t]);
        if (lane == 0) {
          const float gt = gate ? hy_sigmoid(gate[(size_t)t * ld_gate + (size_t)h * oh + o]) : 1.f;
          out[(size_t)t * ldo + (size_t)h * oh + o] = from_f32<TO>(gate ? v * gt : v);
        }
      }
    }
  }
}

// The same where the weight's rows are whole 16-byte pieces, at most PIECES (1, 2 or 4) a lane: a warp takes HLF_OUT outputs of
// a head, its weights are in registers before the kernel in front has finished, and the inputs of 8 / PIECES rows at a
// time are read once for all of them.  A lane adds its even and its odd inputs in two chains (one of all of a piece was 1.05 to 1.2
// times as far off as the kernel above).  Bound by the trip to L2 for the inputs, one for every 8 / PIECES rows.
// Measured (us, the kernel above -> this one; weights of 8 launches, not all in L2): 16 heads 512 -> 128, 2 rows 12.0 -> 2.6, 16 rows
// 24.6 -> 8.4 (12.0 with two rows at a time whatever the pieces); 128 -> 512, 2 rows 7.0 -> 4.6, 16 rows 16.0 -> 10.4 (20.1); 8
// heads 64 -> 64, 16 rows 5.4 -> 4.9 (8.1).
constexpr int HLF_OUT = 4, HLF_PIECES = 4;

// Eight bfloat16 or four 32-bit weights.
__device__ __forceinline__ void hlf_unpack(const uint4& u, float (&v)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = __bfloat1622float2(h[e]);
    v[2 * e] = f.x;
    v[2 * e + 1] = f.y;
  }
}
__device__ __forceinline__ void hlf_unpack(const uint4& u, float (&v)[4]) {
  v[0] = __uint_as_float(u.x);
  v[1] = __uint_as_float(u.y);
  v[2] = __uint_as_float(u.z);
  v[3] = __uint_as_float(u.w);
}

template <typename TW, typename TO, int PIECES>
__global__ void __launch_bounds__(128)
head_linear_few_kernel(const float* x, long long ldx, long long xh, const TW* __restrict__ W, TO* out, long long ldo,
                       long long oh, int n, int O, int I, const float* gate, long long ld_gate) {
  constexpr int E = 16 / (int)sizeof(TW), ROWS = 8 / PIECES;
  pdl_trigger();
  const int h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int o0 = (blockIdx.x * 4 + warp) * HLF_OUT;
  if (o0 >= O) return;                                     // (whole warps; nothing below meets the block)
  uint4 w[HLF_OUT][PIECES];
#pragma unroll
  for (int j = 0; j < HLF_OUT; ++j)
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
      const int c = E * (lane + 32 * i);
      w[j][i] = o0 + j < O && c < I ? *reinterpret_cast<const uint4*>(W + ((size_t)h * O + o0 + j) * I + c) : make_uint4(0u, 0u, 0u, 0u);
      asm volatile("" : "+r"(w[j][i].x), "+r"(w[j][i].y), "+r"(w[j][i].z), "+r"(w[j][i].w));      // (stays here, see gb_pin)
    }
  pdl_wait();
  for (int t0 = 0; t0 < n; t0 += ROWS) {
    const int live = n - t0;                               // (the first two rows are worked out whether there or not)
    float acc[ROWS][HLF_OUT], odd[ROWS][HLF_OUT];
    float4 xv[ROWS][PIECES][E / 4];
#pragma unroll
    for (int u = 0; u < ROWS; ++u)
#pragma unroll
      for (int i = 0; i < PIECES; ++i) {
        const int c = E * (lane + 32 * i);
#pragma unroll
        for (int e = 0; e < E / 4; ++e)
          xv[u][i][e] = t0 + u < n && c < I ? ldcg_now(reinterpret_cast<const float4*>(x + (size_t)(t0 + u) * ldx + (size_t)h * xh + c + 4 * e))
                                            : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
    for (int u = 0; u < ROWS; ++u)
#pragma unroll
      for (int j = 0; j < HLF_OUT; ++j) acc[u][j] = odd[u][j] = 0.f;
#pragma unroll
    for (int i = 0; i < PIECES; ++i)
#pragma unroll
      for (int j = 0; j < HLF_OUT; ++j) {
        float wv[E];
        hlf_unpack(w[j][i], wv);
#pragma unroll
        for (int u = 0; u < ROWS; ++u) {
          if (u >= 2 && u >= live) break;
#pragma unroll
          for (int e = 0; e < E / 4; ++e) {
            acc[u][j] = fmaf(xv[u][i][e].x, wv[4 * e], acc[u][j]);
            odd[u][j] = fmaf(xv[u][i][e].y, wv[4 * e + 1], odd[u][j]);
            acc[u][j] = fmaf(xv[u][i][e].z, wv[4 * e + 2], acc[u][j]);
            odd[u][j] = fmaf(xv[u][i][e].w, wv[4 * e + 3], odd[u][j]);
          }
        }
      }
#pragma unroll
    for (int u = 0; u < ROWS; ++u)
#pragma unroll
      for (int j = 0; j < HLF_OUT; ++j) acc[u][j] += odd[u][j];
#pragma unroll
    for (int u = 0; u < ROWS; u += 2) {
      if (u >= 2 && u >= live) break;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1)
#pragma unroll
        for (int j = 0; j < 2 * HLF_OUT; ++j)
          acc[u + j / HLF_OUT][j % HLF_OUT] += __shfl_xor_sync(0xffffffffu, acc[u + j / HLF_OUT][j % HLF_OUT], s);
    }
    // lane (u, j) stores its output
#pragma unroll
    for (int u = 0; u < ROWS; ++u)
#pragma unroll
      for (int j = 0; j < HLF_OUT; ++j)
        if (lane == u * HLF_OUT + j && t0 + u < n && o0 + j < O) {
          const size_t t = t0 + u, o = (size_t)h * oh + o0 + j;
          const float g = gate ? acc[u][j] * hy_sigmoid(gate[t * ld_gate + o]) : acc[u][j];
          out[t * ldo + o] = from_f32<TO>(g);
        }
  }
}

// A cache row into shared memory as 32-bit values, 16 bytes at a time; `sub` of eight threads share the row.
__device__ __forceinline__ void load_row_vec(const bf16* src, float* dst, int Dk, int sub) {
  // (up to four pieces are requested before any is stored: a store to shared memory in between would make
  // every load wait for the one before it)
  for (int d0 = sub * 8; d0 < Dk; d0 += 256) {
    uint4 raw[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (d0 + 64 * u < Dk) raw[u] = *reinterpret_cast<const uint4*>(src + d0 + 64 * u);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int d = d0 + 64 * u;
      if (d < Dk) {
        const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw[u]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f2 = __bfloat1622float2(h2[e]);
          dst[d + 2 * e] = f2.x;
          dst[d + 2 * e + 1] = f2.y;
        }
      }
    }
  }
}
__device__ __forceinline__ void load_row_vec(const float* src, float* dst, int Dk, int sub) {
  for (int d = sub * 4; d < Dk; d += 32) {
    const float4 v = *reinterpret_cast<const float4*>(src + d);
    dst[d] = v.x; dst[d + 1] = v.y; dst[d + 2] = v.z; dst[d + 3] = v.w;
  }
}

// One block per (token, group of up to LA_HB heads, chunk of keys); a warp looks after LA_HW heads, whose
// queries it holds in registers, the lanes over the dimensions of a cache row.  Key rows arrive in tiles
// of LA_KT in shared memory (32-bit), shared by the block's heads.  Per key a warp reads the row ONCE
// (conflict-free, consecutive lanes consecutive values): the same registers give the scores of its heads
// (a product summed over the lanes) and then enter the weighted sums; the softmax is kept per key (the
// sums are rescaled only when a score exceeds the running maximum, a branch the whole warp takes together).
// (Measured against a variant that takes a tile's scores first, lane j keeping key j's, and then the
// weighted sums in a second pass over the tile: 17.9 against 26.0 ms for four layers of a 2,048-token
// prompt at 16 heads, latent 512 + 64, window 1,024.)
// Exponentials of the softmax: the accurate one where the cache is 32-bit; where the cache rows are bfloat16
// (2^-9 relative) the hardware's 2^x, whose error of a few 2^-23 relative is far below what the rows carry.
template <typename TC> __device__ __forceinline__ float la_exp(float x) { return expf(x); }
template <> __device__ __forceinline__ float la_exp<bf16>(float x) { return __expf(x); }

constexpr int LA_HW = 2, LA_WARPS = 8, LA_HB = LA_HW * LA_WARPS, LA_KT = 32, LA_RR = 4;   // rotated part: up to 128

template <typename TC, int RL>
__global__ void __launch_bounds__(32 * LA_WARPS, 2)      // (two blocks an SM: at most 128 registers a thread)
latent_attention_kernel(const float* qp, const TC* pages, const int* block_table, int bt_stride, int page_size,
                        int n_pages, const int* tok_req, const int* tok_pos, const float* gate, long long ld_gate,
                        float* out, long long ldo, int H, int r, int dr, float scale, int window, int splits, int chunk,
                        float* ws, const float* __restrict__ sink, int* status) {
  extern __shared__ __align__(16) float ks[];      // [LA_KT][Dk]
  pdl_trigger();
  const int Dk = r + dr;
  const int t = blockIdx.x, h0 = blockIdx.y * LA_HB;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int hw = h0 + warp * LA_HW;                // this warp's first head
  const int pos = tok_pos[t];
  const int* table = block_table + (size_t)tok_req[t] * bt_stride;
  const int lo = window > 0 ? max(0, pos - window + 1) : 0;
  // rows of pages can be read in 16-byte pieces when their length allows (pages are 16-byte aligned)
  const bool vec = (Dk * (int)sizeof(TC)) % 16 == 0 && (((uintptr_t)pages) & 15) == 0;
  // this block's share of the visible keys lo .. pos: chunk number blockIdx.z, counted from lo
  const int k_begin = splits > 1 ? lo + (int)blockIdx.z * chunk : lo;
  const int k_end = splits > 1 ? min(pos, k_begin + chunk - 1) : pos;
  pdl_wait();
  float ql[LA_HW][RL], qr[LA_HW][LA_RR], acc[LA_HW][RL], m[LA_HW], l[LA_HW];
#pragma unroll
  for (int hh = 0; hh < LA_HW; ++hh) {
    const bool live = hw + hh < H;
    const float* src = qp + ((size_t)t * H + (live ? hw + hh : 0)) * Dk;
#pragma unroll
    for (int i = 0; i < RL; ++i) {
      const int d = lane + 32 * i;
      ql[hh][i] = (live && d < r) ? src[d] : 0.f;
      acc[hh][i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < LA_RR; ++i) {
      const int d = lane + 32 * i;
      qr[hh][i] = (live && d < dr) ? src[r + d] : 0.f;
    }
    m[hh] = -INFINITY;
    l[hh] = 0.f;
  }
  for (int k0 = k_begin; k0 <= k_end; k0 += LA_KT) {
    __syncthreads();                       // the last tile has been used
    {
      // eight threads share a key row; its page is looked up once
      const int sub = threadIdx.x & 7;
      for (int j = threadIdx.x >> 3; j < LA_KT; j += blockDim.x >> 3) {
      const int kp = k0 + j;
      const TC* src = nullptr;
      if (kp <= k_end) {
        const int page = table[kp / page_size];
        if (page < 0 || page >= n_pages) {
          if (sub == 0) atomicExch(status, STATUS_BAD_PAGE_READ);
        } else {
          src = pages + ((size_t)page * page_size + kp % page_size) * Dk;
        }
      }
      float* dst = ks + j * Dk;
      if (src == nullptr) {
        for (int d = sub; d < Dk; d += 8) dst[d] = 0.f;
      } else if (vec) {
        load_row_vec(src, dst, Dk, sub);
      } else {
        for (int d = sub; d < Dk; d += 8) dst[d] = to_f32(src[d]);
      }
      }
    }
    __syncthreads();
    if (hw >= H) continue;
    const int n_keys = min(LA_KT, k_end - k0 + 1);
    // Keys are taken KG at a time: their rows are read and their scores' partial products and warp sums are worked
    // out side by side (independent chains that hide one another's latencies: a step of a few tokens is bound by
    // them), then the softmax takes the keys one after the other.  Every number is computed by the same operations
    // in the same order as with one key at a time.
    constexpr int KG = RL <= 8 ? 4 : 1;                     // (latents beyond 256 entries fill the registers: one key at a time)
    for (int j0 = 0; j0 < n_keys; j0 += KG) {
      float kl[KG][RL], kr[KG][LA_RR], sc[KG][LA_HW];
#pragma unroll
      for (int u = 0; u < KG; ++u) {
        const float* row = ks + min(j0 + u, n_keys - 1) * Dk;      // (a key beyond the tile's last: read again, not used)
#pragma unroll
        for (int i = 0; i < RL; ++i) {
          const int d = lane + 32 * i;
          kl[u][i] = d < r ? row[d] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < LA_RR; ++i) {
          const int d = lane + 32 * i;
          kr[u][i] = d < dr ? row[r + d] : 0.f;
        }
      }
#pragma unroll
      for (int u = 0; u < KG; ++u) {
#pragma unroll
        for (int hh = 0; hh < LA_HW; ++hh) {
          float p0 = 0.f, p1 = 0.f;                          // two chains; added in a fixed order
#pragma unroll
          for (int i = 0; i < RL; ++i) {
            if (i & 1) p1 = fmaf(ql[hh][i], kl[u][i], p1);
            else p0 = fmaf(ql[hh][i], kl[u][i], p0);
          }
#pragma unroll
          for (int i = 0; i < LA_RR; ++i) {
            if (i & 1) p1 = fmaf(qr[hh][i], kr[u][i], p1);
            else p0 = fmaf(qr[hh][i], kr[u][i], p0);
          }
          sc[u][hh] = p0 + p1;
        }
      }
      // the warp sums of all scores, step by step (every lane gets the same sums)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int u = 0; u < KG; ++u) {
#pragma unroll
          for (int hh = 0; hh < LA_HW; ++hh) sc[u][hh] += __shfl_xor_sync(0xffffffffu, sc[u][hh], o);
        }
      }
#pragma unroll
      for (int u = 0; u < KG; ++u) {
        if (j0 + u >= n_keys) break;                         // (the whole warp together)
#pragma unroll
        for (int hh = 0; hh < LA_HW; ++hh) {
          const float s1 = sc[u][hh] * scale;
          if (s1 > m[hh]) {                                  // (the whole warp together)
            const float corr = la_exp<TC>(m[hh] - s1);       // 0 for the first key: m = -inf
            l[hh] *= corr;
#pragma unroll
            for (int i = 0; i < RL; ++i) acc[hh][i] *= corr;
            m[hh] = s1;
          }
          const float p = la_exp<TC>(s1 - m[hh]);
          l[hh] += p;
#pragma unroll
          for (int i = 0; i < RL; ++i) acc[hh][i] = fmaf(p, kl[u][i], acc[hh][i]);
        }
      }
    }
  }
#pragma unroll
  for (int hh = 0; hh < LA_HW; ++hh) {
    const int h = hw + hh;
    if (h >= H) continue;
    if (splits > 1) {
      // partial result of this chunk: running maximum, sum of weights, weighted sum (not yet divided)
      float* w = ws + (((size_t)t * H + h) * splits + blockIdx.z) * (r + 2);
      if (lane == 0) { w[0] = m[hh]; w[1] = l[hh]; }
#pragma unroll
      for (int i = 0; i < RL; ++i) {
        const int d = lane + 32 * i;
        if (d < r) w[2 + d] = acc[hh][i];
      }
      continue;
    }
    const float g = gate ? hy_sigmoid(gate[(size_t)t * ld_gate + h]) : 1.f;
    float inv = g / l[hh], e = 1.f;
    if (sink) {
      // a learned score without a key or a value: it only joins the denominator (by the merge kernel's
      // arithmetic, so that one chunk and several of which one holds keys give the same bits)
      const float top = fmaxf(m[hh], sink[h]);
      e = expf(m[hh] - top);
      inv = g / __fadd_rn(expf(sink[h] - top), __fmul_rn(e, l[hh]));
    }
    float* o = out + (size_t)t * ldo + (size_t)h * r;
#pragma unroll
    for (int i = 0; i < RL; ++i) {
      const int d = lane + 32 * i;
      if (d < r) o[d] = __fmul_rn(e, acc[hh][i]) * inv;
    }
  }
}

// One block per (token, head): the chunks' partial results, merged in chunk order.  The chunks' weights
// exp(m_s - M) are worked out once into shared memory; then every thread has its columns and asks for
// sixteen chunks' values at a time.  Bound by the trips to L2 (weights, then sums).  Measured, 2 tokens x 16 heads,
// 32 chunks of 512: 6 us in a decode step, 37 to 40 with a warp per (token, head) that took one chunk after the other.
constexpr int LM_CHUNKS = 96;                              // (the cuts give 64 at most, and with a window up to three more)

__global__ void latent_attention_merge_kernel(const float* ws, int splits, const float* gate, long long ld_gate,
                                              float* out, long long ldo, int H, int r, const float* __restrict__ sink) {
  __shared__ float es[LM_CHUNKS];
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long idx = blockIdx.x;
  const int t = (int)(idx / H), h = (int)(idx - (long long)t * H);
  const size_t ld = (size_t)r + 2;
  const float* w = ws + (size_t)idx * splits * ld;
  // (every warp takes the maxima and denominators for itself: lane s has chunks s, s + 32 and s + 64)
  float m[LM_CHUNKS / 32], l[LM_CHUNKS / 32], M = -INFINITY;
#pragma unroll
  for (int i = 0; i < LM_CHUNKS / 32; ++i) {
    const int s = lane + 32 * i;
    m[i] = s < splits ? w[s * ld] : -INFINITY;
    l[i] = s < splits ? w[s * ld + 1] : 0.f;
    M = fmaxf(M, m[i]);
  }
  M = warp_max(M);
  if (sink) M = fmaxf(M, sink[h]);
  float L = sink ? expf(sink[h] - M) : 0.f;
#pragma unroll
  for (int i = 0; i < LM_CHUNKS / 32; ++i) {
    const float e = m[i] > -INFINITY ? expf(m[i] - M) : 0.f, el = e * l[i];
    for (int s = 32 * i; s < splits && s < 32 * i + 32; ++s) L += __shfl_sync(0xffffffffu, el, s & 31);      // in chunk order
    if (threadIdx.x < 32) es[lane + 32 * i] = e;
  }
  __syncthreads();
  const float g = gate ? hy_sigmoid(gate[(size_t)t * ld_gate + h]) : 1.f;
  const float inv = g / L;
  float* dst = out + (size_t)t * ldo + (size_t)h * r;
  for (int d = threadIdx.x; d < r; d += blockDim.x) {
    float a = 0.f;
    for (int s0 = 0; s0 < splits; s0 += 16) {
      float v[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) v[u] = s0 + u < splits && es[s0 + u] != 0.f ? ldcg_now(w + (s0 + u) * ld + 2 + d) : 0.f;
#pragma unroll
      for (int u = 0; u < 16; ++u)
        if (s0 + u < splits && es[s0 + u] != 0.f) a = fmaf(es[s0 + u], v[u], a);      // (a chunk without keys left no sum)
    }
    dst[d] = a * inv;
  }
}

// The same with a warp per (token, head), four to a block, for the few chunks of many rows (a prompt cut in two): the additions
// in the same order, so the same bits.  Blocks of their own for rows of two chunks are mostly prologue.
__global__ void __launch_bounds__(128)
latent_attention_merge_rows_kernel(const float* ws, int splits, const float* gate, long long ld_gate, float* out, long long ldo,
                                   long long rows, int H, int r, const float* __restrict__ sink) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long idx = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (idx >= rows) return;
  const int t = (int)(idx / H), h = (int)(idx - (long long)t * H);
  const size_t ld = (size_t)r + 2;
  const float* w = ws + (size_t)idx * splits * ld;
  const float m = lane < splits ? w[lane * ld] : -INFINITY, l = lane < splits ? w[lane * ld + 1] : 0.f;
  float M = warp_max(m);
  if (sink) M = fmaxf(M, sink[h]);
  const float e = m > -INFINITY ? expf(m - M) : 0.f, el = e * l;
  float L = sink ? expf(sink[h] - M) : 0.f;
  for (int s = 0; s < splits; ++s) L += __shfl_sync(0xffffffffu, el, s);
  const float g = gate ? hy_sigmoid(gate[(size_t)t * ld_gate + h]) : 1.f;
  const float inv = g / L;
  float* dst = out + (size_t)t * ldo + (size_t)h * r;
  for (int d0 = 0; d0 < r; d0 += 128) {                    // four columns a lane at a time
    float a[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) a[v] = 0.f;
    for (int s = 0; s < splits; ++s) {
      const float es = __shfl_sync(0xffffffffu, e, s);
      if (es == 0.f) continue;                             // (the whole warp together)
      const float* ws_s = w + s * ld + 2;
      float x[4];
#pragma unroll
      for (int v = 0; v < 4; ++v) x[v] = d0 + lane + 32 * v < r ? ldcg_now(ws_s + d0 + lane + 32 * v) : 0.f;
#pragma unroll
      for (int v = 0; v < 4; ++v) a[v] = fmaf(es, x[v], a[v]);
    }
#pragma unroll
    for (int v = 0; v < 4; ++v)
      if (d0 + lane + 32 * v < r) dst[d0 + lane + 32 * v] = a[v] * inv;
  }
}

}  // namespace

bool gb_head_linear_tc_takes(int n, int I, long long ldx, long long xh, const void* x, const void* W);
void gb_head_linear_tc_launch(const float* x, long long ldx, long long xh, const bf16* W, void* out, bool out_bf16,
                              long long ldo, long long oh, int n, int H, int O, int I, const float* gate, long long ld_gate,
                              cudaStream_t stream);
bool gb_latent_attention_tc_takes(int n, int R, int H, int r, int dr, int window, bool pages_bf16, const void* pages,
                                  const void* qp, const void* out, long long ldo);
int gb_latent_attention_tc_launch(const float* qp, const bf16* pages, const int* block_table, int bt_stride, int page_size,
                                  int n_pages, const int* tok_req, const int* tok_pos, const int* q_start,
                                  const float* gate, long long ld_gate, float* out, long long ldo, int n, int R, int H, int r,
                                  int dr, float scale, const float* sink, float* ws, long long ws_rows, int* status,
                                  cudaStream_t stream);

bool gb_latent_attention_split_takes(int n, int R, int H, int r, int dr, bool pages_bf16, const void* pages, const void* qp,
                                     const void* out, long long ldo);
cudaError_t gb_latent_attention_split_launch(const float* qp, const bf16* pages, const int* block_table, int bt_stride,
                                             int page_size, int n_pages, const int* tok_req, const int* tok_pos,
                                             const int* q_start, const float* gate, long long ld_gate, float* out,
                                             long long ldo, int n, int R, int H, int r, int dr, float scale, int window,
                                             const float* sink, float* ws, int splits, int chunk, int* status,
                                             cudaStream_t stream);

// The second of a launch's two kernels where the keys were cut: 2 (kernels launched), or a failure's code.
static int launch_merge(const float* ws, int splits, const float* gate, long long ld_gate, float* out, long long ldo, int n,
                        int H, int r, const float* sink, cudaStream_t stream) {
  if (splits > LM_CHUNKS) GB_FAIL(GB_ERR_ARG, "latent_attention_merge: %d chunks", splits);
  // (us of a block and of a warp a row: 2 chunks of 512, 256 rows 3.1 and 3.1, 1024 8.8 and 3.4, 8192 63 and 7.4; 8 chunks, 512 rows
  // 6.3 and 7.6, 1024 10.6 and 7.7; 4 chunks of 64, 512 rows 2.8 and 2.5)
  if (splits <= 8 && (long long)n * H >= 128 * splits)
    gb_launch(latent_attention_merge_rows_kernel, dim3(gb_div_up((long long)n * H, 4)), dim3(128), 0, stream, ws, splits, gate,
              ld_gate, out, ldo, (long long)n * H, H, r, sink);
  else
    gb_launch(latent_attention_merge_kernel, dim3((unsigned)((long long)n * H)), dim3(r <= 128 ? 128 : r <= 256 ? 256 : 512), 0,
            stream, ws, splits, gate, ld_gate, out, ldo, H, r, sink);
  GB_CHECK_LAUNCH("latent_attention_merge");
  return 2;
}

// How the visible keys of a launch are cut into chunks of whole key tiles: (chunks, keys per chunk).
// Few tokens (decoding) get many chunks, so that the GPU is occupied; a launch with enough (token, head
// group) blocks of its own gets one.  With a window the chunk depends on the launch's sizes only, not on
// the contexts' lengths; chunks lie at fixed distances from the first visible key, so a chunk's partial
// result does not depend on how many chunks there are.
GB_API int gb_latent_attention_chunks(int n, int H, int window, int max_ctx, int* chunk_out) {
  const int blocks = n * gb_div_up(H, LA_HB);
  int wanted = 592 / (blocks > 0 ? blocks : 1);
  if (wanted > 64) wanted = 64;
  const int span = window > 0 ? window : (max_ctx > 0 ? max_ctx : 1);
  if (wanted <= 1 || span <= 32) { *chunk_out = span; return 1; }
  int chunk;
  if (window > 0) {
    chunk = 32 * gb_div_up(gb_div_up(span, wanted), 32);
    if (chunk < 32) chunk = 32;
  } else {
    chunk = 2 * LA_KT;
    while (gb_div_up(span, chunk) > wanted) chunk *= 2;
  }
  *chunk_out = chunk;
  return gb_div_up(span, chunk);
}
// The same for the kernel with whole weights on tensor cores, which has one CTA an SM and row tiles of 32 rows: about two rounds
// of CTAs.  It takes the rows of several tokens together, so its chunks lie at multiples of their length: a row tile's keys
// (its tokens' positions and the window in front of the first) may begin and end inside one; none lies behind the longest
// context.
static int split_chunks(int n, int H, int window, int max_ctx, int* chunk_out) {
  const long long tiles = (long long)n * gb_div_up(H, 32);
  const int wanted = tiles <= 4 ? 64 : (int)(296 / tiles), longest = max_ctx > 0 ? max_ctx : 1;
  if (wanted <= 1 || (window > 0 ? window : longest) <= 32) { *chunk_out = 32; return 1; }
  int chunk, splits;
  if (window > 0) {
    chunk = 32 * gb_div_up(gb_div_up((long long)window + 31, wanted), 32);
    splits = gb_div_up((long long)window + gb_div_up(31, H) + chunk - 1, chunk);
    if (max_ctx > 0 && splits > gb_div_up(longest, chunk)) splits = gb_div_up(longest, chunk);
  } else {
    chunk = 64;
    while (gb_div_up(longest, chunk) > wanted) chunk *= 2;
    splits = gb_div_up(longest, chunk);
  }
  *chunk_out = chunk;
  return splits;
}
// Whether that kernel pays where the generic one could run: its CTA prepares 32 rows however few a token brings, and has an SM to
// itself.  Measured (us, generic and whole weights on tensor cores): contexts of 2 and 7 keys 3.3 to 5.7 and 4.9 to 10.8; of 15, up to
// 288 entries, 5.1 to 7.0 and 5.3 to 7.9, 256 tokens of 512 + 64 17 and 22; single tokens of up to 8 heads and 160 entries, 16
// tokens at 1024 keys 16 to 19 and 17 to 21, 64 at 256 12 to 18 and 18 to 23, at 64 14 and 8 to 9, 128 at 1024 70 to 95 and 77 to 97,
// 64 with a window of 128 11 to 13 and 14 to 15 (16 heads of 160: 16 and 18); 8 heads of 288 entries, 64 tokens with a window of 256 23 and 27, at 1024 keys without one 70 and 73, 32 tokens 40 and 38.
static bool split_pays(int n, int R, int H, int dk, int window, int max_ctx) {
  const int longest = max_ctx > 0 ? max_ctx : 1, span = window > 0 && window < longest ? window : longest;
  if (span <= 8 || (span <= 16 && (dk <= 288 || n >= 192))) return false;
  const bool near = window > 0 && window <= 256;
  return !(n == R && n >= 16 && (dk <= 160 || (dk <= 288 && near)) && (H <= 8 || (dk <= 160 && window > 0 && window <= 128)) &&
           (long long)n * span >= (near ? 8192 : 16384));
}
// Rows of (latent size + 2) floats a launch's partial results may need, whatever its sizes.
// (also: two partial results a row for a prompt of up to 2,048 tokens and 16 heads on the tensor-core kernel)
GB_API int gb_latent_attention_workspace_rows() { return 65536 > LA_HB * 2 * (592 + 592) ? 65536 : LA_HB * 2 * (592 + 592); }

// a0 fused rows [q heads (plain | rotated) | ... ] (f32), a1 their stride, a2 column of [latent | rotated key],
// a3 gain of the latent's norm [r], a4 inv_freq [rot_dims / 2], a5 rot_dims, a6 token -> request, a7 token ->
// position, a8 block table, a9 its entries per request, a10 page size, a11 pages, a12 number of pages, a13 their dtype,
// a14 tokens, a15 heads, a16 plain query size, a17 rotated size, a18 latent size, a19 q' [tokens, heads, r + rot]
// (f32), a20 the queries [tokens, heads * (plain + rotated)] (f32) when they are no part of the fused rows (they came
// through a product of their own), else 0, a21 their row stride; f0 eps
GB_OP(gb_op_latent_prep) {
  const int n = (int)a[14], H = (int)a[15];
  if (n <= 0) return 0;
  if (a[5] % 2 || a[5] > a[17]) GB_FAIL(GB_ERR_ARG, "latent_prep: %lld rotated dimensions of %lld", a[5], a[17]);
  const int warps = H + 1 < 8 ? H + 1 : 8;
#define PREP(TC, ROT, LAT)                                                                                                 \
  gb_launch(latent_prep_kernel<TC, ROT, LAT>, dim3(n), dim3(32 * warps), 0, ctx->stream, op_ptr<const float>(a[0]), a[1], (int)a[2], \
            a[20] ? op_ptr<const float>(a[20]) : op_ptr<const float>(a[0]), a[20] ? a[21] : a[1], op_ptr<const float>(a[3]), \
            op_ptr<const float>(a[4]), (int)a[5], op_ptr<const int>(a[6]),                   \
            op_ptr<const int>(a[7]), op_ptr<const int>(a[8]), (int)a[9], (int)a[10], op_ptr<TC>(a[11]), (int)a[12], H,  \
            (int)a[16], (int)a[17], (int)a[18], op_ptr<float>(a[19]), (float)f[0], ctx->status)
#define PREP_LAT(TC, ROT)                                                                                   \
  do {                                                                                                      \
    if (a[18] <= 128) PREP(TC, ROT, 4); else if (a[18] <= 256) PREP(TC, ROT, 8); else PREP(TC, ROT, 16);   \
  } while (0)
#define PREP_ROT(TC)                                            \
  do {                                                          \
    if (a[5] <= 64) PREP_LAT(TC, 1); else PREP_LAT(TC, 2);      \
  } while (0)
  if (a[13] == GB_BF16) PREP_ROT(bf16); else PREP_ROT(float);
#undef PREP_ROT
#undef PREP_LAT
#undef PREP
  GB_CHECK_LAUNCH("latent_prep");
  return 1;
}

// a0 x (f32), a1 its row stride, a2 elements between heads in a row, a3 W [H, O, I], a4 its dtype, a5 out, a6 its
// dtype, a7 its row stride, a8 elements between heads in a row, a9 rows, a10 heads, a11 O, a12 I, a13 gate logits
// (f32, one per output element, laid out like a row of out) or 0: the outputs are multiplied by their sigmoid, a14
// their row stride; flags bit 0: the generic kernels whatever the sizes
GB_OP(gb_op_head_linear) {
  const int n = (int)a[9], H = (int)a[10], O = (int)a[11], I = (int)a[12];
  if (n <= 0) return 0;
  if (a[4] == GB_BF16 && !(flags & 1) &&
      gb_head_linear_tc_takes(n, I, a[1], a[2], op_ptr<const void>(a[0]), op_ptr<const void>(a[3]))) {
    gb_head_linear_tc_launch(op_ptr<const float>(a[0]), a[1], a[2], op_ptr<const bf16>(a[3]), op_ptr<void>(a[5]),
                             a[6] == GB_BF16, a[7], a[8], n, H, O, I, op_ptr<const float>(a[13]), a[14], ctx->stream);
    GB_CHECK_LAUNCH("head_linear (tensor cores)");
    return 1;
  }
  // a few rows whose weights come in whole 16-byte pieces (both sides measured at the kernel)
  if (n <= HL_SMALL_ROWS && I % (a[4] == GB_BF16 ? 8 : 4) == 0 && I <= 32 * HLF_PIECES * (a[4] == GB_BF16 ? 8 : 4) &&
      a[1] % 4 == 0 && a[2] % 4 == 0 && ((a[0] | a[3]) & 15) == 0) {
#define HLF(TW, TO)                                                                                                       \
    gb_launch(I <= 512 / (int)sizeof(TW)    ? head_linear_few_kernel<TW, TO, 1>                                           \
              : I <= 1024 / (int)sizeof(TW) ? head_linear_few_kernel<TW, TO, 2> : head_linear_few_kernel<TW, TO, 4>,      \
              dim3(gb_div_up(O, 4 * HLF_OUT), H), dim3(128), 0, ctx->stream,                                              \
              op_ptr<const float>(a[0]), a[1], a[2], op_ptr<const TW>(a[3]), op_ptr<TO>(a[5]), a[7], a[8], n, O, I,       \
              op_ptr<const float>(a[13]), a[14])
    if (a[4] == GB_BF16) { if (a[6] == GB_BF16) { HLF(bf16, bf16); } else { HLF(bf16, float); } }
    else { if (a[6] == GB_BF16) { HLF(float, bf16); } else { HLF(float, float); } }
#undef HLF
    GB_CHECK_LAUNCH("head_linear (few rows)");
    return 1;
  }
  const bool small = n <= HL_SMALL_ROWS && (size_t)n * I * sizeof(float) <= 48 * 1024;
  const dim3 grid = small ? dim3(gb_div_up(O, 8), H) : dim3(gb_div_up(O, 64), gb_div_up(n, 64), H);
  const dim3 block(256);
  const size_t smem = small ? (size_t)n * I * sizeof(float) : 0;
#define HL(TW, TO)                                                                                                  \
  if (small)                                                                                                        \
    gb_launch(head_linear_small_kernel<TW, TO>, grid, block, smem, ctx->stream, op_ptr<const float>(a[0]), a[1], a[2], \
              op_ptr<const TW>(a[3]), op_ptr<TO>(a[5]), a[7], a[8], n, O, I, op_ptr<const float>(a[13]), a[14]);     \
  else                                                                                                              \
    gb_launch(head_linear_kernel<TW, TO>, grid, block, 0, ctx->stream, op_ptr<const float>(a[0]), a[1], a[2],       \
              op_ptr<const TW>(a[3]), op_ptr<TO>(a[5]), a[7], a[8], n, O, I, op_ptr<const float>(a[13]), a[14])
  if (a[4] == GB_BF16) { if (a[6] == GB_BF16) { HL(bf16, bf16); } else { HL(bf16, float); } }
  else { if (a[6] == GB_BF16) { HL(float, bf16); } else { HL(float, float); } }
#undef HL
  GB_CHECK_LAUNCH("head_linear");
  return 1;
}

// a0 q' [tokens, heads, r + rot] (f32), a1 pages, a2 their dtype, a3 block table, a4 its entries per request, a5 page
// size, a6 number of pages, a7 token -> request, a8 token -> position, a9 gate logits (f32, [t, h] at a row stride) or
// 0, a10 that stride, a11 out [tokens, heads * r] (f32), a12 its row stride, a13 tokens, a14 heads, a15 latent size,
// a16 rotated size, a17 window (0: every earlier position), a18 longest context of the step (an upper bound will do),
// a19 workspace for partial results, gb_latent_attention_workspace_rows() rows of (latent size + 2) floats, a20 a
// learned sink score per head (f32 [heads]) whose exponential joins the softmax's denominator, or 0; a21 requests of
// the step, a22 first row per request (requests' rows follow one another in the order of the requests; a22 = 0: the
// generic kernel whatever the step); f0 scale
GB_OP(gb_op_latent_attention) {
  const int n = (int)a[13], H = (int)a[14], r = (int)a[15], dr = (int)a[16];
  if (n <= 0) return 0;
  // a step that carries portions of prompts, bfloat16 pages: the tensor-core kernel (latent_attention_tc.cu)
  if (a[22] &&
      gb_latent_attention_tc_takes(n, (int)a[21], H, r, dr, (int)a[17], a[2] == GB_BF16, op_ptr<const void>(a[1]),
                                   op_ptr<const void>(a[0]), op_ptr<const void>(a[11]), a[12])) {
    const int parts = gb_latent_attention_tc_launch(
        op_ptr<const float>(a[0]), op_ptr<const bf16>(a[1]), op_ptr<const int>(a[3]), (int)a[4], (int)a[5], (int)a[6],
        op_ptr<const int>(a[7]), op_ptr<const int>(a[8]), op_ptr<const int>(a[22]), op_ptr<const float>(a[9]), a[10],
        op_ptr<float>(a[11]), a[12], n, (int)a[21], H, r, dr, (float)f[0], op_ptr<const float>(a[20]), op_ptr<float>(a[19]),
        gb_latent_attention_workspace_rows(), ctx->status, ctx->stream);
    if (parts >= 1) {
      GB_CHECK_LAUNCH("latent_attention (tensor cores)");
      if (parts == 1) return 1;
      return launch_merge(op_ptr<const float>(a[19]), parts, op_ptr<const float>(a[9]), a[10], op_ptr<float>(a[11]), a[12], n,
                          H, r, op_ptr<const float>(a[20]), ctx->stream);
    }
  }
  if (r > 512) GB_FAIL(GB_ERR_ARG, "latent_attention: latent size %d (at most 512)", r);
  const int Dk = r + dr;
  if (dr > 32 * LA_RR) GB_FAIL(GB_ERR_ARG, "latent_attention: rotated size %d (at most %d)", dr, 32 * LA_RR);
  const size_t smem = sizeof(float) * (size_t)LA_KT * Dk;
  int chunk = 0;
  int splits = gb_latent_attention_chunks(n, H, (int)a[17], (int)a[18], &chunk);
  float* ws = op_ptr<float>(a[19]);
  if (ws == nullptr || (long long)n * H * splits > gb_latent_attention_workspace_rows()) splits = 1;
  // bfloat16 pages, a window or single tokens: tensor cores with whole queries and weights (latent_attention_tc.cu).
  // Measured at 16 heads, 512 + 64 entries, window 1024 (with the merge): portions of 1801 and 333 tokens 0.77 ms against 3.66 on
  // the kernel below, two single tokens at 1801 and 900 keys 16 us against 60.
  if (a[22] && gb_latent_attention_split_takes(n, (int)a[21], H, r, dr, a[2] == GB_BF16, op_ptr<const void>(a[1]),
                                               op_ptr<const void>(a[0]), op_ptr<const void>(a[11]), a[12]) &&
      split_pays(n, (int)a[21], H, r + dr, (int)a[17], (int)a[18])) {
    splits = split_chunks(n, H, (int)a[17], (int)a[18], &chunk);
    if (ws == nullptr || (long long)n * H * splits > gb_latent_attention_workspace_rows()) splits = 1;
    const cudaError_t e = gb_latent_attention_split_launch(
        op_ptr<const float>(a[0]), op_ptr<const bf16>(a[1]), op_ptr<const int>(a[3]), (int)a[4], (int)a[5], (int)a[6],
        op_ptr<const int>(a[7]), op_ptr<const int>(a[8]), op_ptr<const int>(a[22]), op_ptr<const float>(a[9]), a[10],
        op_ptr<float>(a[11]), a[12], n, (int)a[21], H, r, dr, (float)f[0], (int)a[17], op_ptr<const float>(a[20]), ws, splits,
        chunk, ctx->status, ctx->stream);
    if (e != cudaSuccess) GB_FAIL(GB_ERR_CUDA, "latent_attention: %s", cudaGetErrorString(e));
    GB_CHECK_LAUNCH("latent_attention (tensor cores, whole weights)");
    if (splits == 1) return 1;
    return launch_merge(ws, splits, op_ptr<const float>(a[9]), a[10], op_ptr<float>(a[11]), a[12], n, H, r,
                        op_ptr<const float>(a[20]), ctx->stream);
  }
  // (fewer heads than a block has room for: fewer warps, so that none idles through the key tiles)
  const int warps = H >= LA_HB ? LA_WARPS : (gb_div_up(H, LA_HW) < 2 ? 2 : gb_div_up(H, LA_HW));
  const dim3 grid(n, gb_div_up(H, LA_HB), splits), block(32 * warps);
#define LA(TC, RL)                                                                                                   \
  do {                                                                                                               \
    static size_t allowed = 48 * 1024;     /* raised once per size, before any stream capture replays the launch */ \
    if (smem > allowed) {                                                                                            \
      GB_CUDA(cudaFuncSetAttribute(latent_attention_kernel<TC, RL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
      allowed = smem;                                                                                                \
    }                                                                                                                \
    gb_launch(latent_attention_kernel<TC, RL>, grid, block, smem, ctx->stream, op_ptr<const float>(a[0]),             \
              op_ptr<const TC>(a[1]), op_ptr<const int>(a[3]), (int)a[4], (int)a[5], (int)a[6], op_ptr<const int>(a[7]), \
              op_ptr<const int>(a[8]), op_ptr<const float>(a[9]), a[10], op_ptr<float>(a[11]), a[12], H, r, dr,       \
              (float)f[0], (int)a[17], splits, chunk, ws, op_ptr<const float>(a[20]), ctx->status);                                              \
  } while (0)
#define LA_RL(TC)                                                                                                    \
  do {                                                                                                               \
    if (r <= 32) LA(TC, 1); else if (r <= 64) LA(TC, 2); else if (r <= 128) LA(TC, 4);                              \
    else if (r <= 256) LA(TC, 8); else LA(TC, 16);                                                                   \
  } while (0)
  if (a[2] == GB_BF16) LA_RL(bf16); else LA_RL(float);
#undef LA_RL
#undef LA
  GB_CHECK_LAUNCH("latent_attention");
  if (splits == 1) return 1;
  return launch_merge(ws, splits, op_ptr<const float>(a[9]), a[10], op_ptr<float>(a[11]), a[12], n, H, r,
                      op_ptr<const float>(a[20]), ctx->stream);
}
