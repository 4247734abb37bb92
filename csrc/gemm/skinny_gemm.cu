// C[T, N] = X[T, K] W[N, K]^T for decode steps (T <= 16), W in 16 bits or packed int4, sm_100a.
//
// What bounds such a product is the stream of weights and, for the matrices of one layer (a few MB), the chain of
// latencies around it: start, first bytes, reduction, store.  The tensor-memory kernels (dense_gemm.cu, awq_gemm.cu) pay
// for a shared-memory ring of up to 160 KB, which keeps the next kernel of the stream from moving in beside them, and for
// two trips through shared memory.  Here weights go from global memory straight into the registers that
// mma.m16n8k16 takes as operand A:
//
//   * a tile is 16 weight rows; KS of a CTA's eight warps split its K in chunks (64 values of a 16-bit row, 128 of an int4
//     row: the four lanes of a quad read 64 contiguous bytes) that they take in turn, the 8 / KS groups of warps work on
//     tiles of their own, and a CTA stays for as many tiles as the chip has too few CTAs for.  Partial sums of a group meet in
//     shared memory, two buffers in turn, one barrier of the group per tile
//   * every warp keeps a ring of DW chunks in registers that runs on from tile to tile
//   * the tokens are staged in shared memory once (in segments of K where they do not fit), in an order that the
//     16-byte reads of eight lanes meet without bank conflicts
//   * lane (g, t) of a warp holds 8 (or 32) consecutive k of rows g and g + off; the k order inside a chunk is permuted
//     the same way for both operands, so no value ever changes lanes
//   * the second eight rows of a tile stand `off` rows behind the first: 8 (plain), the up half of a gated pair, or half a
//     head (rotary), so every epilogue finds its pairs in one thread
//   * the first chunks are requested before the wait for the preceding kernel, the other lines of the first tile are asked
//     into L2
//   * int4: the nibbles become 16-bit integers q - z (exact).  Where a scale covers a whole chunk (groups of 128 and multiples)
//     it multiplies the chunk's fp32 sums instead of the weights, otherwise the weights, as in awq_gemm.cu
//   * sums of squares for the fused RMSNorm come from the same token registers, as the diagonal of X X^T
//
// Grouped mode (mixture of experts): blockIdx.y names a tile of a device-built table (expert, first sorted row, rows).
//
// Measured (one B200, us per launch in a captured chain with cold weights; before: dense_gemm.cu / awq_gemm.cu; the stream of
// the weights alone at 6.65 TB/s):
//   16-bit with RMSNorm, one token, N x K: 2560 x 2048   6.6 -> 4.7 (1.6)    2 x 5632 x 2048   14.4 -> 9.9 (6.9)
//   int4 group 128, three tokens:  6144 x 4096  20.6 -> 8.2 (1.9)    2 x 12288 x 4096  48.4 -> 20.5 (7.6)   4096 x 12288   29.5 -> 14.0 (3.8)
//   int4 group 32, 16 tokens:      8192 x 2816  17.0 -> 11.8 (1.7)   2 x 2112 x 2816   13.3 -> 8.2 (0.9)
// The int4 forms are bound by the issue of 3.6 (layers) to 5.4 (experts' down products) instructions per weight (56 to 62 % of the
// slots, ALU 45 to 51 %), the 16-bit forms of large matrices by memory, small ones by the latencies of one CTA's life.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>

#include "../common/launch.cuh"
#include "epilogue.cuh"
#include "skinny_gemm.h"

namespace fi {
namespace {

constexpr int kWarps = 8;
constexpr int kSkinnyThreads = 32 * kWarps;
constexpr int kRedPitch = 20;      // floats between the 16 rows of neighbouring tokens: a quad's stores hit different banks

template <typename T> struct Num;
template <> struct Num<__nv_bfloat16> {
  using v2 = __nv_bfloat162;
  static constexpr uint32_t kMagic2 = 0x43004300u;    // 128 in both halves: (q | magic) = 128 + q
  static __device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
  static __device__ __forceinline__ float scale(uint16_t s) { return __uint_as_float(static_cast<uint32_t>(s) << 16); }
};
template <> struct Num<__half> {
  using v2 = __half2;
  static constexpr uint32_t kMagic2 = 0x64006400u;    // 1024 in both halves
  static __device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
  static __device__ __forceinline__ float scale(uint16_t s) { return __half2float(__ushort_as_half(s)); }
};

__device__ __forceinline__ uint4 ld_weight(const uint8_t* p) {      // never written while a kernel runs, read once
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t word(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// (w & 0x000F000F) | magic in one instruction
__device__ __forceinline__ uint32_t nibbles(uint32_t w, uint32_t magic) {
  uint32_t r;
  asm("lop3.b32 %0, %1, 0x000F000F, %2, 0xEA;" : "=r"(r) : "r"(w), "r"(magic));
  return r;
}

// First weight row of a tile and the distance of its second eight rows.
__device__ __forceinline__ void tile_rows_of(const SkinnyParams& p, int tile, int* r0, int* off) {
  if (p.dual_rows > 0) {
    *r0 = tile * 8;
    *off = p.dual_rows;
  } else if (p.rope_cs != nullptr) {
    const int half = p.rope_hd >> 1, pr = tile * 8;
    *r0 = (pr / half) * p.rope_hd + pr % half;
    *off = half;
  } else {
    *r0 = tile * 16;
    *off = 8;
  }
}

// Sums over the KS warps of a group and the epilogue of its tiles.  red: [KS][MT][8 NT tokens][kRedPitch], ss: [KS][8 NT].
template <typename T, int KS, int MT, int NT>
__device__ __forceinline__ void finish(const SkinnyParams& p, const float* red, const float* ss, int first_tile, int n_tiles, int out_row0,
                                       int tokens, int tid) {
  constexpr int TOK = NT * 8;
  const int n_out = p.dual_rows > 0 ? p.dual_rows : p.N;
  for (int item = tid; item < n_tiles * tokens * 4; item += KS * 32) {
    const int q = item & 3, tk = (item >> 2) % tokens, i = (item >> 2) / tokens;
    float v[4] = {0.f, 0.f, 0.f, 0.f};        // rows 2q, 2q + 1 of the first eight and of the second
#pragma unroll
    for (int w = 0; w < KS; ++w) {
      const float* src = red + ((w * MT + i) * TOK + tk) * kRedPitch + 2 * q;
      const float2 a = *reinterpret_cast<const float2*>(src), b = *reinterpret_cast<const float2*>(src + 8);
      v[0] += a.x; v[1] += a.y; v[2] += b.x; v[3] += b.y;
    }
    if (p.rms_eps > 0.f) {
      float sum = 0.f;
#pragma unroll
      for (int w = 0; w < KS; ++w) sum += ss[w * TOK + tk];
      const float r = rsqrtf(sum / static_cast<float>(p.K) + p.rms_eps);
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] *= r;
    }
    int r0, off;
    tile_rows_of(p, first_tile + i, &r0, &off);
    const int lo = r0 + 2 * q, hi = lo + off;
    const int t = out_row0 + tk;
    if (p.dual_rows > 0) {
      if (lo >= n_out) continue;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float bg = 0.f, bu = 0.f;
        if (p.bias != nullptr && lo + j < n_out) {
          bg = ld16_as_float(p.bias, lo + j, p.is_fp16);
          bu = ld16_as_float(p.bias, p.dual_rows + lo + j, p.is_fp16);
        }
        v[j] = apply_gated(v[j] + bg, v[2 + j] + bu, p.act, p.act_limit);
      }
    } else {
      if (lo >= p.N) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = (j < 2 ? lo : hi) + (j & 1);
        v[j] = apply_act(v[j], p.act);
        if (p.bias != nullptr && n < p.N) v[j] += ld16_as_float(p.bias, n, p.is_fp16);
      }
    }
    if (p.rope_cs != nullptr) {
      const int hd = p.rope_hd, half = hd >> 1;
      const int q_end = p.rope_nh * hd, k_end = q_end + p.rope_nkv * hd;
      const int sec = lo < q_end ? 0 : (lo < k_end ? 1 : 2);
      const int d = lo & (hd - 1);
      if (sec != 2) {
        const float* cs = p.rope_cs + static_cast<size_t>(p.rope_pos[t]) * hd + d;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float c = cs[j], s = cs[half + j], a = v[j], b = v[2 + j];
          v[j] = a * c - b * s;
          v[2 + j] = b * c + a * s;
        }
      }
      if (sec != 0) {
        const int slot = p.rope_slots[t];
        if (slot >= 0) {
          const int blk = slot / p.rope_bs, at = slot - blk * p.rope_bs;
          const int hn = lo - (sec == 1 ? q_end : k_end);
          T* cache = reinterpret_cast<T*>(sec == 1 ? p.k_cache : p.v_cache) +
                     ((static_cast<size_t>(blk) * p.rope_nkv + hn / hd) * p.rope_bs + at) * hd + d;
          cache[0] = T(v[0]); cache[1] = T(v[1]);
          cache[half] = T(v[2]); cache[half + 1] = T(v[3]);
        }
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int n = h == 0 ? lo : hi;
      if (h == 1 && p.dual_rows > 0) break;
      const size_t at = static_cast<size_t>(t) * p.ldc + n;
      float y[2] = {v[h * 2], v[h * 2 + 1]};
      const bool pair = n + 1 < n_out;       // n and the row pitch are even: pairs are aligned
      if (n >= n_out) continue;
      if (p.residual != nullptr) {
        for (int j = 0; j < (pair ? 2 : 1); ++j)
          y[j] += p.out_fp32 ? reinterpret_cast<const float*>(p.residual)[at + j] : ld16_as_float(p.residual, at + j, p.is_fp16);
      }
      if (p.out_fp32) {
        float* c = reinterpret_cast<float*>(p.C) + at;
        if (pair) *reinterpret_cast<float2*>(c) = make_float2(y[0], y[1]);
        else *c = y[0];
      } else {
        T* c = reinterpret_cast<T*>(p.C) + at;
        if (pair) {
          alignas(4) const T two[2] = {T(y[0]), T(y[1])};
          *reinterpret_cast<uint32_t*>(c) = *reinterpret_cast<const uint32_t*>(two);
        } else {
          *c = T(y[0]);
        }
      }
    }
  }
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
template <int KS>
__device__ __forceinline__ void group_sync(int group) {
  if constexpr (KS == 1) __syncwarp();
  else if constexpr (KS == kWarps) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(KS * 32) : "memory");
}

// 16-byte words of one token row in shared memory: whole chunks, and a remainder that puts the rows of neighbouring lanes on other banks.
__host__ __device__ constexpr int row_units(bool int4, int k) { return int4 ? (k + 127) / 128 * 16 + 1 : (k + 63) / 64 * 8 + 4; }

template <typename T, bool INT4, bool POST, bool RMS, int KS, int MT, int NT, int DW>
__global__ void __launch_bounds__(kSkinnyThreads, MT * NT <= 2 ? 2 : 1) skinny_kernel(const SkinnyParams p, int tiles, int seg_chunks) {
  using N = Num<T>;
  constexpr int TOK = NT * 8;
  constexpr int CH = INT4 ? 128 : 64;          // k per chunk
  constexpr int WV = INT4 ? 1 : 2;             // 16-byte words of a weight row per lane and chunk
  constexpr int XV = INT4 ? 4 : 2;             // 16-byte words of a token row per lane and chunk
  constexpr int GP = kWarps / KS;              // groups of warps with tiles of their own
  constexpr int kBuf = kWarps * MT * TOK * kRedPitch;
  extern __shared__ __align__(16) uint8_t smem[];
  float* red = reinterpret_cast<float*>(smem);                       // [2][kWarps][MT][TOK][kRedPitch]
  float* ssum = red + 2 * kBuf;                                      // [kWarps][TOK]
  uint8_t* xs = reinterpret_cast<uint8_t*>(ssum + kWarps * TOK);     // [tokens][row_units] 16-byte words

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int group = warp / KS, kw = warp % KS;
  pdl_launch_dependents();
  const bool grouped = p.tile_expert != nullptr;
  int tokens = p.T, row0 = 0, w_row0 = 0;
  if (grouped) pdl_wait();      // the table comes from the kernel in front
  if (grouped) {
    if (static_cast<int>(blockIdx.y) >= *p.n_tiles) return;
    tokens = p.tile_rows[blockIdx.y];
    row0 = p.tile_row0[blockIdx.y];
    w_row0 = p.tile_expert[blockIdx.y] * p.expert_rows;
  }
  const int rows_here = p.dual_rows > 0 ? 2 * p.dual_rows : p.N;     // weight rows of this product
  const int chunks = (p.K + CH - 1) / CH;
  const int per_tile = (chunks + KS * DW - 1) / (KS * DW) * DW;      // ring entries of a warp per tile, the last ones may be empty
  const int step = gridDim.x * GP;                                   // in units of MT tiles
  const int units = (tiles + MT - 1) / MT;
  const int first = blockIdx.x * GP + group;
  const int rounds = (units - static_cast<int>(blockIdx.x) * GP + step - 1) / step;     // of the CTA (its first group has most)

  // ---- ring of weight chunks: the load side runs DW entries ahead of the sums
  uint4 wb[DW][MT][2][WV];
  // int4: scales and zero points as they were loaded; a warp issues in order, so nothing may touch them before their chunk is due
  uint32_t sb[DW][MT][2], zb[DW][MT][2];
  const uint16_t* scales = reinterpret_cast<const uint16_t*>(p.scales);
  const int gshift = INT4 && (p.group & (p.group - 1)) == 0 ? 31 - __clz(p.group) : -1;
  const uint8_t* const w_base = reinterpret_cast<const uint8_t*>(p.w);
  const uint32_t row_words = INT4 ? static_cast<uint32_t>(p.K) >> 5 : static_cast<uint32_t>(p.ldw) >> 3;     // 16-byte words
  uint32_t woff[MT][2], srow[MT][2];            // of the load side's tile: first 16-byte word and number of this lane's rows
  int l_unit = first, l_entry = 0, l_k = kw * CH + (INT4 ? 32 : 8) * t;      // this lane's first k of the chunk
  auto set_rows = [&]() {
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      int r0, off;
      tile_rows_of(p, l_unit * MT + i, &r0, &off);
      // rows past the end are read from the last one and never stored
      srow[i][0] = w_row0 + min(r0 + g, rows_here - 1);
      srow[i][1] = w_row0 + min(r0 + g + off, rows_here - 1);
#pragma unroll
      for (int h = 0; h < 2; ++h) woff[i][h] = srow[i][h] * row_words;
    }
  };
  set_rows();
  auto load_next = [&](int d) {
    const bool on = l_unit < units && l_k < p.K;
    const uint32_t kg = INT4 ? static_cast<uint32_t>(gshift >= 0 ? l_k >> gshift : l_k / p.group) * static_cast<uint32_t>(p.rows_total) : 0u;
    const uint32_t kw16 = static_cast<uint32_t>(l_k) >> (INT4 ? 5 : 3);
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint8_t* src = w_base + static_cast<size_t>(woff[i][h] + kw16) * 16;
#pragma unroll
        for (int v = 0; v < WV; ++v) {
          wb[d][i][h][v] = make_uint4(0, 0, 0, 0);
          if (on && (v == 0 || l_k + 32 < p.K)) wb[d][i][h][v] = ld_weight(src + v * 64);
        }
        if constexpr (INT4) {
          sb[d][i][h] = 0u;
          zb[d][i][h] = 8u;
          if (on) {
            const uint32_t at = kg + srow[i][h];
            asm volatile("ld.global.nc.u16 %0, [%1];" : "=r"(sb[d][i][h]) : "l"(scales + at));
            if (p.zeros != nullptr) asm volatile("ld.global.nc.u8 %0, [%1];" : "=r"(zb[d][i][h]) : "l"(p.zeros + at));
          }
        }
      }
    l_k += KS * CH;
    if (++l_entry == per_tile) {
      l_entry = 0;
      l_k -= per_tile * KS * CH;
      l_unit += step;
      if (l_unit < units) set_rows();
    }
  };
  if (!grouped && first < units) {
    for (int e = DW; e < per_tile; ++e) {        // lanes 0 and 1 of a quad: the line of either row of each tile
      const int k = (kw + KS * e) * CH;
#pragma unroll
      for (int i = 0; i < MT; ++i)
        if (t < 2 && k < p.K) prefetch_l2(w_base + static_cast<size_t>((t == 0 ? woff[i][0] : woff[i][1]) + (k >> (INT4 ? 5 : 3))) * 16);
    }
  }
#pragma unroll
  for (int d = 0; d < DW; ++d) load_next(d);
  if (!grouped) pdl_wait();

  // ---- tokens
  const int segs = (chunks + seg_chunks - 1) / seg_chunks;
  const int pitch = row_units(INT4, min(chunks, seg_chunks) * CH) * 16;
  auto stage = [&](int seg) {
    const int u0 = seg * seg_chunks * (CH / 8), u_end = min(chunks - seg * seg_chunks, seg_chunks) * (CH / 8), u_k = p.K / 8 - u0;
    // CTAs begin at different places: all of them read the same lines
    const int turn0 = static_cast<int>(blockIdx.x) % tokens;
    for (int j = 0; j < tokens; ++j) {
      const int r = j + turn0 < tokens ? j + turn0 : j + turn0 - tokens;
      const int row = p.x_rows != nullptr ? p.x_rows[row0 + r] / p.x_div : row0 + r;
      const uint8_t* src = reinterpret_cast<const uint8_t*>(p.x) + (static_cast<size_t>(row) * p.ldx + u0 * 8) * 2;
      for (int u = threadIdx.x; u < u_end; u += kSkinnyThreads) {
        uint8_t* dst = xs + r * pitch + (INT4 ? u ^ ((u >> 2) & 2) : u) * 16;       // the upper half of a 256-byte chunk is turned by two words
        if (u < u_k) cp_async16(smem_u32(dst), src + u * 16);
        else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
      }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  };
  const uint8_t* xrow[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n)      // columns past the last token repeat it and are never stored
    xrow[n] = xs + min(n * 8 + g, tokens - 1) * pitch + (INT4 ? t * 64 : t * 16);
  const int turn = INT4 ? (t >> 1) * 2 : 0;

  for (int round = 0; round < rounds; ++round) {
    const int unit = first + round * step;
    float acc[MT][NT][4], sq[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sq[n][j] = 0.f;
#pragma unroll
        for (int i = 0; i < MT; ++i) acc[i][n][j] = 0.f;
      }
    for (int seg = 0; seg < segs; ++seg) {
      if (segs > 1 || round == 0) {
        if (segs > 1 && (seg > 0 || round > 0)) __syncthreads();       // everyone is done with the segment in front
        stage(seg);
        __syncthreads();
      }
      const int e0 = seg * (seg_chunks / KS), e1 = min(per_tile, e0 + seg_chunks / KS);
      for (int eb = e0; eb < e1; eb += DW) {
#pragma unroll
        for (int d = 0; d < DW; ++d) {
          const int c = kw + KS * (eb + d);
          if (unit < units && c < chunks) {
            const int xo = (c - seg * seg_chunks) * (CH * 2);
            float part[POST ? MT : 1][POST ? NT : 1][4];
            if constexpr (POST) {
#pragma unroll
              for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                  for (int j = 0; j < 4; ++j) part[i][n][j] = 0.f;
            }
#pragma unroll
            for (int v = 0; v < XV; ++v) {
              uint4 xb[NT];
#pragma unroll
              for (int n = 0; n < NT; ++n)
                xb[n] = *reinterpret_cast<const uint4*>(xrow[n] + xo + (INT4 ? (v ^ turn) * 16 : v * 64));
              if constexpr (RMS) {
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                  N::mma(sq[n], xb[n].x, xb[n].x, xb[n].y, xb[n].y, xb[n].x, xb[n].y);
                  N::mma(sq[n], xb[n].z, xb[n].z, xb[n].w, xb[n].w, xb[n].z, xb[n].w);
                }
              }
#pragma unroll
              for (int i = 0; i < MT; ++i) {
                uint32_t a[2][4];                     // [first or second eight rows][pair of k]
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  if constexpr (INT4) {
                    const uint32_t w = word(wb[d][i][h][0], v);
                    const uint32_t z2 = N::kMagic2 + zb[d][i][h] * 0x00010001u;
                    const uint32_t s2 = sb[d][i][h] * 0x00010001u;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                      const uint32_t m = nibbles(w >> (4 * e), N::kMagic2);
                      typename N::v2 y = __hsub2(*reinterpret_cast<const typename N::v2*>(&m), *reinterpret_cast<const typename N::v2*>(&z2));
                      if constexpr (!POST) y = __hmul2(y, *reinterpret_cast<const typename N::v2*>(&s2));
                      a[h][e] = *reinterpret_cast<uint32_t*>(&y);
                    }
                  } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) a[h][e] = word(wb[d][i][h][WV > 1 ? v : 0], e);
                  }
                }
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                  float (&dst)[4] = POST ? part[POST ? i : 0][POST ? n : 0] : acc[i][n];
                  N::mma(dst, a[0][0], a[1][0], a[0][1], a[1][1], xb[n].x, xb[n].y);
                  N::mma(dst, a[0][2], a[1][2], a[0][3], a[1][3], xb[n].z, xb[n].w);
                }
              }
            }
            if constexpr (POST) {
#pragma unroll
              for (int i = 0; i < MT; ++i) {
                // the scale of a whole chunk; lane 0 of the quad holds its first k, which always exists
                const uint32_t l = __shfl_sync(0xffffffffu, sb[d][i][0], lane & 28), h = __shfl_sync(0xffffffffu, sb[d][i][1], lane & 28);
                const float s0 = N::scale(static_cast<uint16_t>(l)), s1 = N::scale(static_cast<uint16_t>(h));
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                  acc[i][n][0] = fmaf(s0, part[i][n][0], acc[i][n][0]);
                  acc[i][n][1] = fmaf(s0, part[i][n][1], acc[i][n][1]);
                  acc[i][n][2] = fmaf(s1, part[i][n][2], acc[i][n][2]);
                  acc[i][n][3] = fmaf(s1, part[i][n][3], acc[i][n][3]);
                }
              }
            }
          }
          load_next(d);
        }
      }
    }
    // ---- the group's sums meet; a buffer is written again only after the next tile's barrier
    float* buf = red + (round & 1) * kBuf + group * KS * MT * TOK * kRedPitch;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        float* dst = buf + ((kw * MT + i) * TOK + n * 8 + 2 * t) * kRedPitch + g;
        dst[0] = acc[i][n][0];
        dst[kRedPitch] = acc[i][n][1];
        dst[8] = acc[i][n][2];
        dst[kRedPitch + 8] = acc[i][n][3];
      }
    if constexpr (RMS) {
      if (round == 0) {      // the same for every tile
#pragma unroll
        for (int n = 0; n < NT; ++n)
          if ((g >> 1) == t) ssum[warp * TOK + n * 8 + g] = (g & 1) ? sq[n][1] : sq[n][0];       // entry (g, g) of X X^T
      }
    }
    group_sync<KS>(group);
    if (unit < units)
      finish<T, KS, MT, NT>(p, buf, ssum + group * KS * TOK, unit * MT, min(MT, tiles - unit * MT), row0, tokens, threadIdx.x - group * KS * 32);
  }
}

inline int sm_count() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 148;
  }();
  return n;
}

// What a launch needs by its sizes: tokens in one piece up to kMostBytes of shared memory, beyond in segments of K that every round
// stages again; kernels of few accumulators run two CTAs per SM where their tokens leave room.
struct Shape { int seg, segs, smem, per_sm, blocks; };

template <bool INT4, int KS, int MT, int NT, int DW>
Shape shape_of(int tokens, int K, int tiles) {
  constexpr int CH = INT4 ? 128 : 64, kMostBytes = 200 * 1024;
  constexpr int fixed = (2 * kWarps * MT * NT * 8 * kRedPitch + kWarps * NT * 8) * 4;
  const int chunks = (K + CH - 1) / CH;
  int seg = (chunks + KS * DW - 1) / (KS * DW) * (KS * DW);
  while (seg > KS * DW && fixed + tokens * row_units(INT4, (seg < chunks ? seg : chunks) * CH) * 16 > kMostBytes) seg -= KS * DW;
  Shape s;
  s.seg = seg;
  s.segs = (chunks + seg - 1) / seg;
  s.smem = fixed + tokens * row_units(INT4, (seg < chunks ? seg : chunks) * CH) * 16;
  s.per_sm = MT * NT <= 2 && s.smem <= 113 * 1024 ? 2 : 1;
  s.blocks = ((tiles + MT - 1) / MT + kWarps / KS - 1) / (kWarps / KS);
  return s;
}

template <typename T, bool INT4, bool POST, bool RMS, int KS, int MT, int NT, int DW>
int launch(const SkinnyParams& p, int tiles, cudaStream_t s) {
  auto kern = skinny_kernel<T, INT4, POST, RMS, KS, MT, NT, DW>;
  const bool grouped = p.tile_expert != nullptr;
  const Shape f = shape_of<INT4, KS, MT, NT, DW>(grouped ? p.tile_tokens : p.T, p.K, tiles);
  if (f.smem > 227 * 1024) return -31;
  cudaError_t e = ensure_dynamic_smem(kern, f.smem > 48 * 1024 ? f.smem : 48 * 1024);
  if (e != cudaSuccess) return static_cast<int>(e);
  int gx = f.blocks;
  if (grouped) {        // about four CTAs per place over the experts that can occur
    const int want = (4 * f.per_sm * sm_count() + p.max_tiles - 1) / p.max_tiles;
    if (gx > want) gx = want;
  } else if (gx > f.per_sm * sm_count()) {
    gx = f.per_sm * sm_count();
  }
  return static_cast<int>(launch_kernel(kern, dim3(gx, grouped ? p.max_tiles : 1, 1), dim3(kSkinnyThreads), f.smem, s, 0, p, tiles, f.seg));
}

// Which split of the warps.  Measured on one B200, us per launch in a captured chain, weights cold (512 tiles: N = 8192):
//   plain products split every tile's K over all eight warps; fewer warps per tile lengthen the chain of a warp and were
//   slower at every size tried (int4 N = K = 4096, one token: 5.7 against 7.5 with four warps, 11.2 with two).
//   Two tiles per warp share the reads of the tokens but halve the CTAs.  For up to 8 tokens one tile per warp needs a second round
//   of CTAs past 296 tiles: two tiles pay from there on (one / two, K = 4096, one token: 0.87 of the time at 288 tiles, 1.13 at 320, 1.07 at 512;
//   K = 2816 0.89, 1.16, 1.12), with K of 8192 and more less or not at all (0.74, 0.92, 1.00), with K up to 1024 everywhere.  For 9 to
//   16 tokens, whose accumulators leave one CTA per SM either way, two tiles are 0 to 45 % faster at nearly every size (K = 704 to
//   12288, 192 to 1536 tiles), up to 10 % slower at 128 tiles.
//   Experts of up to 8 rows: about as many warps per tile as there are warps on the chip for the tiles of the experts that occur when
//   routes fall evenly.  Fewer lengthen the chain of a warp, the more the longer K is; more cost rounds of CTAs with their table reads,
//   tokens and sums (us with one warp for two tiles / one / two / four / eight for one): 240 tiles of K = 5120 - / 22 / 15 / 10 / 9, 512 of 4096
//   27 / 18 / 13 / 11 / 14, 684 of 2816 21 / 15 / 13 / 16 / 18, 1365 of 704 9.8 / 9.5 / 12 / 15 / 21, 3600 of 768 12 / 16 / 21 / 27 / 37.
//   The line between one and two warps is where a decode step crosses (1365 tiles of 704 in a step of one token: two warps 1 % faster).
//   The layer's products, two warps always / by this: 128 experts of 2816 x 704, 8 per token, 1 / 2 / 4 / 6 tokens 30 / 43 / 64 / 77 -> 30 / 40 /
//   58 / 64; 60 of 2048 x 1408 at 32 routes 65 -> 52; 256 of 2048 x 1024 at 32 routes 63 -> 44; 8 of 4096 x 2048 at 2 routes 28 -> 22.
//   Experts of 9 to 16 rows have many tiles: two warps per tile (128 experts of 2816 x 704, 32 tokens: 153; four warps 202).
template <typename T, bool POST>
int int4_by_size(const SkinnyParams& p, cudaStream_t s) {
  const int tiles = p.dual_rows > 0 ? (p.dual_rows + 7) / 8 : (p.N + 15) / 16;
  if (p.tile_expert != nullptr) {
    if (p.tile_tokens > 8) return launch<T, true, POST, false, 2, 1, 2, 4>(p, tiles, s);
    const float experts = static_cast<float>(p.rows_total / p.expert_rows);
    const float n = tiles * fminf(static_cast<float>(p.max_tiles), experts * (1.f - expf(-p.T / experts)));
    const float warps = 2.f * kWarps * sm_count();
    if (8.f * n <= warps) return launch<T, true, POST, false, 8, 1, 1, 2>(p, tiles, s);
    if (4.f * n <= warps) return launch<T, true, POST, false, 4, 1, 1, 4>(p, tiles, s);
    if (2.f * n <= fmaxf(1.25f * warps, (POST ? 0.6f : 0.875f) * p.K)) return launch<T, true, POST, false, 2, 1, 1, 4>(p, tiles, s);
    if (n <= fmaxf(warps, 1.25f * p.K)) return launch<T, true, POST, false, 1, 1, 1, 4>(p, tiles, s);
    return launch<T, true, POST, false, 1, 2, 1, 2>(p, tiles, s);
  }
  if (p.T > 8) return launch<T, true, POST, false, 8, 2, 2, 2>(p, tiles, s);
  return tiles >= 320 ? launch<T, true, POST, false, 8, 2, 1, 2>(p, tiles, s) : launch<T, true, POST, false, 8, 1, 1, 4>(p, tiles, s);
}

// Int4 layers of up to 16 tokens: against awq_gemm.cu, which splits K over clusters and stages the tokens with the weights.
// Up to 8 tokens in one piece this kernel is 1.2 to 3 times as fast at every size tried but the shortest K under the most rows (K =
// 256, 12288 rows: 5.8 / 6.3 us).  More tokens, and pieces, cost what follows: estimates in us of both, fitted to 1660 products
// of 9 to 16 tokens (K = 256 to 16384, 64 to 12288 outputs).  Over 3100 products of 1 to 16 tokens choosing by them takes 0.2 % longer
// than the better kernel each time and 0.67 of awq_gemm.cu's time; 33 are more than 3 % longer than there (at most 17 %), with
// this kernel always 259 (up to 1.7 times).  us there / here: 1024 x 12288 15 / 18 at 9 tokens, 15 / 22 at 16; 4096 x 12288 29 / 25
// at 16; gated 2 x 8192 x 12288 71 / 91 at 16.
struct Int4Estimate { float here, there; bool settled; };      // settled: this kernel, whatever the estimates say
Int4Estimate int4_estimate(int T, int N, int K, bool gated) {
  const int tiles = gated ? (N + 7) / 8 : (N + 15) / 16;
  const Shape f = T > 8 ? shape_of<true, 8, 2, 2, 2>(T, K, tiles) : tiles >= 320 ? shape_of<true, 8, 2, 1, 2>(T, K, tiles)
                                                                             : shape_of<true, 8, 1, 1, 4>(T, K, tiles);
  const int rounds = (f.blocks + f.per_sm * sm_count() - 1) / (f.per_sm * sm_count());
  const float tk = static_cast<float>(T) * K;
  const float piece = f.segs == 1 ? 0.f : T > 8 ? 5.8e-5f : 2.4e-5f;        // of a token's value, staged again in each round
  const float here = 1.63f + (f.segs == 1 ? 6.8e-6f * tk : 0.f) + rounds * (1.86f + f.per_sm * K * (5.2e-4f + 1.22e-5f * T) + piece * tk);
  const int rows = (N + 127) / 128, most = (gated ? 1 : 2) * sm_count() * 19 / 20;      // clusters leave some SMs over
  int split = (107 + rows - 1) / rows;
  if (split > 8) split = 8;
  if (split > K / 128) split = K / 128 > 0 ? K / 128 : 1;
  while (split > 1 && rows * split > most) --split;
  const float k = static_cast<float>(K) / split;
  const float there = gated ? 8.3f + 0.0084f * k + rows * (1.67e-5f * K + 0.0011f) : 4.36f + 0.0061f * k + rows * (2.7e-5f * K + 0.0011f);
  return {here, there, T <= 8 && f.segs == 1};
}
bool int4_pays(int T, int N, int K, bool gated) {
  const Int4Estimate e = int4_estimate(T, N, K, gated);
  return e.settled || e.here <= e.there;
}

// 16-bit products with a fused norm: against dense_gemm.cu, whose rings stream long rows better (us there / here, one token: 6144 x
// 8192 22 / 24, 256 x 12288 7.6 / 10.5, gated 2 x 2560 x 12288 30 / 34) and which has no rounds of CTAs to fill (K = 256: 10240 rows 4.2 /
// 6.4; a third round that is nearly empty: 10240 x 2560 at 6 tokens 13.5 / 14.8).  Up to the lines below: 2560 x 2048 7.0 / 5.2, 6144 x
// 4096 14.4 / 13.6, gated 2 x 5632 x 2048 15.3 / 11.0, 2 x 704 x 4096 8.8 / 5.5.  Over 832 products of 1 to 8 tokens (K = 256 to 19968,
// 64 to 32000 outputs) 0.84 of the time there, 0.4 % over the better one each time; 4 are more than 3 % longer (at most 4 %).
bool norm_pays(int T, int N, int K, bool gated) {
  const int tiles = gated ? (N + 7) / 8 : (N + 15) / 16, round = 2 * sm_count();
  if (K < 512) return gated ? tiles <= 512 : tiles <= 160 && T <= 5;
  if (gated) return K <= 6144 || (K <= 8192 && tiles <= round);
  if (K > 4096) return K <= 6144 && tiles >= 64 && tiles <= round;
  return T <= 2 || tiles <= 2 * round || (tiles + round - 1) / round * round <= 1.3f * tiles;
}

template <typename T>
int by_kind(const SkinnyParams& p, cudaStream_t s) {
  if (p.int4) return p.group % 128 == 0 ? int4_by_size<T, true>(p, s) : int4_by_size<T, false>(p, s);
  return launch<T, false, false, true, 8, 1, 1, 4>(p, p.dual_rows > 0 ? (p.dual_rows + 7) / 8 : (p.N + 15) / 16, s);
}

}  // namespace

float int4_few_us(int T, int N, int K, bool gated) {
  const Int4Estimate e = int4_estimate(T, N, K, gated);
  return e.here < e.there ? e.here : e.there;
}

bool skinny_takes(bool int4, bool norm, int T, int N, int K, bool gated) {
  if (static_cast<double>(N) * K * (gated ? 2 : 1) >= 3.e10) return false;      // rows are counted in 32 bits (skinny_gemm)
  if (int4) return !norm && T > 0 && T <= 16 && int4_pays(T, N, K, gated);
  return norm && T > 0 && T <= 8 && static_cast<long>(T) * K <= 20000 && norm_pays(T, N, K, gated);
}

int skinny_gemm(const SkinnyParams& p, cudaStream_t stream) {
  if (p.T <= 0 || p.N <= 0) return 0;
  const bool norm = p.rms_eps > 0.f;
  if (p.tile_expert == nullptr && !skinny_takes(p.int4 != 0, norm, p.T, p.N, p.K, p.dual_rows > 0)) return -30;
  if (p.int4 ? norm : p.tile_expert != nullptr) return -30;
  // rows are counted in 16-byte words of 32 bits, scales in elements of 32 bits
  const uint64_t rows = p.int4 ? p.rows_total : p.dual_rows > 0 ? 2ull * p.dual_rows : p.N;
  if (rows * (p.int4 ? p.K / 32 : p.ldw / 8) >= (1ull << 32) || (p.int4 && rows * (p.K / p.group + 1) >= (1ull << 32))) return -32;
  return p.is_fp16 ? by_kind<__half>(p, stream) : by_kind<__nv_bfloat16>(p, stream);
}

}  // namespace fi

// skinny_takes, for whoever wants to know the route of a product.
extern "C" int fi_skinny_takes(int int4, int norm, int T, int N, int K, int gated) {
  return fi::skinny_takes(int4 != 0, norm != 0, T, N, K, gated != 0) ? 1 : 0;
}

// Routed int4 experts of few rows each: the rows of X that the sorted routes name (x_rows[r] / x_div; null: row r itself)
// meet the weights of their expert; C [n_rows, ldc] in the order of the routes.  g: table of tiles of `bn` (8 or 16) rows.
extern "C" int fi_awq_gemm_grouped_rows(const void* X, const int* x_rows, int x_div, const void* qw, const void* scales,
                                        const void* zeros, void* C, int n_rows, int N, int K, int group, int ldx, int ldc, int act,
                                        int dual_rows, int dtype, int bn, const FiGrouped* g, void* stream) {
  if (n_rows <= 0 || N <= 0 || K <= 0 || g->max_tiles <= 0) return 0;
  if ((K % 64) != 0 || (ldc % 8) != 0 || (ldx % 8) != 0 || (reinterpret_cast<uintptr_t>(C) & 15) != 0 ||
      (reinterpret_cast<uintptr_t>(X) & 15) != 0 || (reinterpret_cast<uintptr_t>(qw) & 15) != 0)
    return -10;
  if (group != 32 && group != 64 && group != 128 && !(group > 128 && group % 64 == 0)) return -13;
  if (dual_rows > 0 && N != dual_rows) return -11;
  if ((bn != 8 && bn != 16) || g->max_tiles > 65535 || (x_rows != nullptr && x_div <= 0)) return -25;
  fi::SkinnyParams p = {};
  p.x = X; p.x_rows = x_rows; p.x_div = x_div; p.w = qw; p.scales = scales; p.zeros = reinterpret_cast<const uint8_t*>(zeros);
  p.group = group; p.rows_total = g->num_experts * g->expert_rows; p.C = C; p.T = n_rows; p.N = N; p.K = K;
  p.ldx = ldx; p.ldc = ldc; p.act = act; p.dual_rows = dual_rows; p.is_fp16 = dtype == 1; p.int4 = 1;
  p.tile_expert = g->tile_expert; p.tile_row0 = g->tile_row0; p.tile_rows = g->tile_rows; p.n_tiles = g->n_tiles;
  p.expert_rows = g->expert_rows; p.max_tiles = g->max_tiles; p.tile_tokens = bn;
  return fi::skinny_gemm(p, reinterpret_cast<cudaStream_t>(stream));
}
