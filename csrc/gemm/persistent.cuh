// What the persistent kernels of products share: their parameters, the order of their tiles and the way a finished accumulator
// leaves tensor memory.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "../common/ptx.cuh"

namespace fi {

constexpr int kTileRows = 128;   // weight rows per tile (UMMA M)

struct PersistentParams {
  void* C;
  const void* bias;
  const void* residual;
  int T, N, K, ldc;
  int dual_rows, act, is_fp16, out_fp32;
  float act_limit;     // act 4
  int second_off;   // weight rows between the two A tiles of a CTA: dual_rows (gated) or 128 (grouped plain form, 256-row tile)
  int rows_per_tile;   // output rows (of N) one tile covers: 128, or 256 in the grouped plain form
  int n_tiles_n, n_tiles;
  int n_group;         // weight tiles that are worked on together over all token tiles (grouped mode: all of them)
  int* status;
  // grouped mode (tile_expert != null): n_tiles is the grid's upper bound, the true number of token tiles is *tiles
  const int* tile_expert;
  const int* tile_row0;
  const int* tile_rows;
  const int* tiles;
  int expert_rows;     // weight rows per expert
};

template <int ACT>
__device__ __forceinline__ float act_f(float g) {
  if constexpr (ACT == 1) return g / (1.f + __expf(-g));
  if constexpr (ACT == 2) {
    const float inner = 0.7978845608028654f * (g + 0.044715f * g * g * g);
    return g / (1.f + __expf(-2.f * inner));
  }
  if constexpr (ACT == 3) return fmaxf(g, 0.f);
  if constexpr (ACT == 5) { g = fmaxf(g, 0.f); return g * g; }
  if constexpr (ACT == 6) return 1.f - 2.f / (1.f + __expf(2.f * g));
  return g;
}
// Gated form of one channel: act(g) * u; 4: bounds on both halves (g from above only), g sigmoid(1.702 g) * (u + 1).
template <int ACT>
__device__ __forceinline__ float gated_f(float g, float u, float limit) {
  if constexpr (ACT == 4) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.f + __expf(-1.702f * g)) * (u + 1.f);
  }
  return act_f<ACT>(g) * u;
}
// Several channels at a time: the activation is chosen once and not for each of them.
template <int ACT, int M>
__device__ __forceinline__ void act_as(uint32_t (&r)[M], const uint32_t (&u)[M], bool gated, float bias_g, float bias_u, float limit) {
#pragma unroll
  for (int j = 0; j < M; ++j) {
    const float v = __uint_as_float(r[j]);
    r[j] = __float_as_uint(gated ? gated_f<ACT>(v + bias_g, __uint_as_float(u[j]) + bias_u, limit) : act_f<ACT>(v) + bias_g);
  }
}
template <int M>
__device__ __forceinline__ void act_all(uint32_t (&r)[M], const uint32_t (&u)[M], bool gated, float bias_g, float bias_u, int act, float limit) {
  switch (act) {
    case 1: return act_as<1>(r, u, gated, bias_g, bias_u, limit);
    case 2: return act_as<2>(r, u, gated, bias_g, bias_u, limit);
    case 3: return act_as<3>(r, u, gated, bias_g, bias_u, limit);
    case 4: return act_as<4>(r, u, gated, bias_g, bias_u, limit);
    case 5: return act_as<5>(r, u, gated, bias_g, bias_u, limit);
    case 6: return act_as<6>(r, u, gated, bias_g, bias_u, limit);
    default: return act_as<0>(r, u, gated, bias_g, bias_u, limit);
  }
}
__device__ __forceinline__ float ld16(const void* p, size_t i, int is_fp16) {
  if (is_fp16) return __half2float(reinterpret_cast<const __half*>(p)[i]);
  return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
}

// a / b of non-negative numbers.  The estimate is within one below 2^22 (two units in its last place are half a unit there); the
// exact division takes 0.2 us of a tile's start, twice (gated 2 x 4096 x 256 at 4096 tokens: 69.2 us, so 65.8).
__device__ __forceinline__ int quotient(int a, int b) {
  if (a >= (1 << 22)) return a / b;
  const int q = static_cast<int>(__fdividef(static_cast<float>(a), static_cast<float>(b)));
  const int r = a - q * b;
  return r < 0 ? q - 1 : r >= b ? q + 1 : q;
}

// Weight tile and token tile of a place in the order of work.  The tiles in flight at a time form a block of n_group weight tiles
// by as many token tiles as there are CTAs for, so that what they share stays in L2 and matrices larger than L2 leave HBM once.
// us with 2, 8, 16, 32 and all weight tiles in a group (one B200): gated 2 x 12288 x 4096 (201 MB) at 2048 tokens 321, 298, 312, 330, 407;
// 2 x 8192 x 2816 (92 MB) 133, 135, 135, 145, 168; plain 12288 x 4096 (101 MB) 160, 161, 160, 166, 204; below about 50 MB all the same.
__device__ __forceinline__ void tile_at(const PersistentParams& p, int tile, int n_token_tiles, int* n, int* tt) {
  const int per = p.n_group * n_token_tiles;
  const int g = quotient(tile, per), at = tile - g * per;
  const int width = min(p.n_group, p.n_tiles_n - g * p.n_group);      // the last group may be narrower
  *tt = quotient(at, width);
  *n = g * p.n_group + (at - *tt * width);
}

constexpr int kPatchPitch = 36;                        // floats between the tokens of a patch: 16-byte reads of eight lanes meet no bank twice
constexpr int kPatchFloats = 16 * kPatchPitch;
constexpr int kPairPitch = 20;                         // the same for 32 tokens x 16 rows (drain_gate_up), the second sixteen 16 floats on
constexpr int kPairPatchFloats = 32 * kPairPitch + 16;
static_assert(kPairPatchFloats >= kPatchFloats, "a patch of CTA pairs serves both forms");

// Eight outputs of one token: bias is in, residual (raw: eight 16-bit values) is added, the result rounded once and stored.
__device__ __forceinline__ void store8(const PersistentParams& p, size_t off, const float4& a0, const float4& a1, const uint4& raw) {
  if (p.out_fp32) {               // 32-bit output (no residual in this form)
    float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(p.C) + off);
    dst[0] = a0;
    dst[1] = a1;
    return;
  }
  const float v[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
  const uint32_t rw[4] = {raw.x, raw.y, raw.z, raw.w};
  uint32_t ow[4];
  if (p.is_fp16) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 rr = __half22float2(*reinterpret_cast<const __half2*>(&rw[e]));
      const __half2 o = __floats2half2_rn(v[2 * e] + rr.x, v[2 * e + 1] + rr.y);
      ow[e] = *reinterpret_cast<const uint32_t*>(&o);
    }
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const __nv_bfloat162 o = __floats2bfloat162_rn(v[2 * e] + __uint_as_float(rw[e] << 16),
                                                     v[2 * e + 1] + __uint_as_float(rw[e] & 0xffff0000u));
      ow[e] = *reinterpret_cast<const uint32_t*>(&o);
    }
  }
  *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.C) + off) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
}

// One warp's part of a finished tile: the 32 weight rows of TMEM quarter q, tokens [c_begin, c_end) of the tile whose first token is
// t0 (rows from t_end on are not stored).  taddr: the accumulator (gated: gate rows, BN columns later the up rows; otherwise with
// DUAL the rows 128 further on); patch: kPatchFloats of this warp.
// Each thread owns one weight row (a TMEM lane) but the output is token-major: 16 tokens x 32 rows at a time go through the patch
// as fp32 and come back as 8-row vectors, so residual and store are 16-byte accesses.  Bound by the instructions of one warp: the
// activation is chosen once per batch (asked for each value anew a batch of 16 x 32 took 1.1 to 1.9 us).
template <int BN, bool DUAL>
__device__ __forceinline__ void drain_tile(const PersistentParams& p, uint32_t taddr, float* patch, int n0, int t0, int t_end, int c_begin,
                                           int c_end, int q, int lane) {
  const bool gated = DUAL && p.dual_rows > 0;
  c_end = min(c_end, t_end - t0);
  const int vc = lane & 3;                // which 8-row chunk of the warp's 32 rows this lane finishes
  const int vj = lane >> 2;               // tokens vj and vj + 8 of the batch
  // gated: one output row per thread (gate and up combined); plain wide tile: two rows, 128 apart
  const int halves = (DUAL && !gated) ? 2 : 1;
  for (int hh = 0; hh < halves; ++hh) {
    const int row = n0 + hh * kTileRows + q * 32 + lane;       // this thread's weight row
    if (row - lane >= p.N) break;
    float bias_g = 0.f, bias_u = 0.f;
    if (p.bias != nullptr && row < p.N) {
      bias_g = ld16(p.bias, row, p.is_fp16);
      if (gated) bias_u = ld16(p.bias, p.dual_rows + row, p.is_fp16);
    }
    const int nv = n0 + hh * kTileRows + q * 32 + vc * 8;      // first of the 8 rows this lane stores
    const bool nv_ok = nv < p.N;
    const bool with_res = p.residual != nullptr;
    // the residual values of a batch are requested one batch ahead, so their latency hides behind
    // the TMEM read and the transposition of the batch in front
    auto load_res = [&](int c0, uint4 (&dst)[2]) {
#pragma unroll
      for (int rep = 0; rep < 2; ++rep) {
        const int c = c0 + vj + rep * 8;
        dst[rep] = make_uint4(0, 0, 0, 0);
        if (nv_ok && c < c_end)
          dst[rep] = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.residual) +
                                                     static_cast<size_t>(t0 + c) * p.ldc + nv);
      }
    };
    uint4 res[2], res_next[2];
    res[0] = res[1] = res_next[0] = res_next[1] = make_uint4(0, 0, 0, 0);
    if (with_res) load_res(c_begin, res);
#pragma unroll 1
    for (int c0 = c_begin; c0 < c_end; c0 += 16) {
      uint32_t r[16], u[16];
      tmem_ld_x16(taddr + hh * BN + c0, r);
      if (gated) tmem_ld_x16(taddr + BN + c0, u);
      if (with_res) load_res(c0 + 16, res_next);
      tmem_ld_wait();
      act_all(r, u, gated, bias_g, bias_u, p.act, p.act_limit);
#pragma unroll
      for (int j = 0; j < 16; ++j) patch[j * kPatchPitch + lane] = __uint_as_float(r[j]);
      __syncwarp();
#pragma unroll
      for (int rep = 0; rep < 2; ++rep) {
        const int j = vj + rep * 8;
        if (nv_ok && c0 + j < c_end) {
          const float4 a0 = *reinterpret_cast<const float4*>(patch + j * kPatchPitch + vc * 8);
          const float4 a1 = *reinterpret_cast<const float4*>(patch + j * kPatchPitch + vc * 8 + 4);
          store8(p, static_cast<size_t>(t0 + c0 + j) * p.ldc + nv, a0, a1, res[rep]);
        }
      }
      __syncwarp();
      res[0] = res_next[0];
      res[1] = res_next[1];
    }
  }
}

// The same for a gated tile whose weight rows lie as eight gate rows, their eight up rows, and so on (make_tmap_gate_up_16bit_sw128): the
// warp finishes 16 outputs from n on.  32 tokens at a time; lanes of gate rows take the first sixteen of them and lanes of up rows the
// others, so that either sends its partner (lane ^ 8) what that one lacks and no lane computes in vain.
__device__ __forceinline__ void drain_gate_up(const PersistentParams& p, uint32_t taddr, float* patch, int n, int t0, int t_end, int c_begin,
                                              int c_end, int lane) {
  if (n >= p.N) return;
  c_end = min(c_end, t_end - t0);
  const bool up = (lane & 8) != 0;
  const int o = (lane >> 4) * 8 + (lane & 7);             // this lane's output of the 16
  float bias_g = 0.f, bias_u = 0.f;
  if (p.bias != nullptr && n + o < p.N) {
    bias_g = ld16(p.bias, n + o, p.is_fp16);
    bias_u = ld16(p.bias, p.dual_rows + n + o, p.is_fp16);
  }
  float* const mine = patch + (up ? 16 * kPairPitch + 16 : 0) + o;
  const float* const token = patch + lane * kPairPitch + (lane >= 16 ? 16 : 0);
#pragma unroll 1
  for (int c0 = c_begin; c0 < c_end; c0 += 32) {
    uint32_t r[32], g[16], u[16];
    tmem_ld_x32(taddr + c0, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? r[j] : r[16 + j], 8);
      g[j] = up ? got : r[j];
      u[j] = up ? r[16 + j] : got;
    }
    act_all(g, u, true, bias_g, bias_u, p.act, p.act_limit);
#pragma unroll
    for (int j = 0; j < 16; ++j) mine[j * kPairPitch] = __uint_as_float(g[j]);
    __syncwarp();
    if (c0 + lane < c_end) {
      const size_t off = static_cast<size_t>(t0 + c0 + lane) * p.ldc + n;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (n + h * 8 >= p.N) break;
        uint4 raw = make_uint4(0, 0, 0, 0);
        if (p.residual != nullptr) raw = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.residual) + off + h * 8);
        store8(p, off + h * 8, *reinterpret_cast<const float4*>(token + h * 8), *reinterpret_cast<const float4*>(token + h * 8 + 4), raw);
      }
    }
    __syncwarp();
  }
}

// dense_gemm_pair.cu: the product with CTA pairs, `tokens` of 128, 192 or 256 per tile.  0, or an error as in fi_dense_gemm_persistent.
int dense_gemm_pair(const void* X, const void* W, PersistentParams p, int ldx, int ldw, int tokens, cudaStream_t stream);

}  // namespace fi
