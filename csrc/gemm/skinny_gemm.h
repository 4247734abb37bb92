// Products of few tokens (decode steps): see skinny_gemm.cu.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "comm_desc.h"

namespace fi {

// Whether skinny_gemm is the better kernel for T tokens and N outputs (gated: of two weight rows each).  16-bit weights: products
// with a fused RMSNorm of few staged tokens (a TinyLlama step of one token: 1.200 ms without, 1.183 with the gated one alone, 1.181
// with q|k|v alone).  The others are faster alone too, but not in a step, where their predecessors' rings hide the start of
// dense_gemm.cu's stream (o 1.264 ms, down 1.246, logits of 151936 rows at three tokens 160 us slower).
bool skinny_takes(bool int4, bool norm, int T, int N, int K, bool gated);
// us of an int4 product of 9 to 16 tokens in the faster one of this kernel and awq_gemm.cu.
float int4_few_us(int T, int N, int K, bool gated);

struct SkinnyParams {
  const void* x;            // [T, K] rows of pitch ldx, 16-bit
  const int* x_rows;        // grouped: row of x of sorted route r is x_rows[r] / x_div (null: r itself)
  int x_div;
  const void* w;            // dense: [rows, K] of pitch ldw, 16-bit; int4: [rows, K / 8] words
  const void* scales;       // int4: [K / group, rows_total]
  const uint8_t* zeros;     // int4: the same shape, or null (zero point 8)
  int group, rows_total;
  void* C;
  const void* bias;
  const void* residual;
  int T, N, K, ldx, ldw, ldc;
  int act, dual_rows, out_fp32, is_fp16, int4;
  float act_limit, rms_eps;
  const float* rope_cs;     // rotary embedding and cache write behind a merged q|k|v product (FiRope)
  const int* rope_pos;
  const int* rope_slots;
  void* k_cache;
  void* v_cache;
  int rope_nh, rope_nkv, rope_hd, rope_bs;
  const int* tile_expert;   // grouped mode: FiGrouped
  const int* tile_row0;
  const int* tile_rows;
  const int* n_tiles;
  int expert_rows, max_tiles, tile_tokens;     // tile_tokens: rows per tile the table was built for (8 or 16)
};

// Returns 0, a positive CUDA error or a negative argument error.
int skinny_gemm(const SkinnyParams& p, cudaStream_t stream);

}  // namespace fi
