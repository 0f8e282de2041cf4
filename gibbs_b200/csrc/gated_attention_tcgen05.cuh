// The launch of gated_attention_tcgen05.cu, for gated_attention_tc.cuh.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

struct GatedTcgen05Launch {
  const __nv_bfloat16* q;          // [tokens][heads * maps * dim]
  const __nv_bfloat16 *k_pages, *v_pages;
  const int* block_table; int bt_stride, page_size, n_pages;
  const int *tok_req, *tok_pos, *q_start;
  const float* gate; long long ld_gate;
  __nv_bfloat16* out; float* out_f32; long long ldo;      // one of the two
  int n, R, H, G, dim, vdim, maps, window, blocked, sink;
  float scale, softcap;
  const float* sink_scores;
  bool sigmoid;                    // weights sigmoid(score + score_bias[head]), the output times `factor`
  const float* score_bias; float factor;
  int longest;                     // positions that a tile walks at most
  int* status;
};

// Whether the kernel takes the launch's sizes (the alignment that gated_attention_tc.cuh asks for holds).
bool gb_gated_tcgen05_takes(const GatedTcgen05Launch& a);
// Launches it; returns the number of kernels launched, or a negative error code.
int gb_gated_tcgen05_launch(const GatedTcgen05Launch& a, cudaStream_t stream);
