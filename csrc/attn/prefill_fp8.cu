// Chunked-prefill attention with heads of 256 channels on an e4m3 KV cache, tcgen05.
//
// The general kernel (paged_attention.cu) expands keys and values into shared memory between its barriers, 32 of them at a time for 64 query
// rows: two prompts of 384 tokens, 16 heads on 8, took it 81 us.  Here a CTA owns 128 query rows of one head and walks tiles of 64 keys:
//
//   warp 0     TMA: the query tile once, raw e4m3 keys and values page by page
//   warp 1     UMMA: S = Q K^T (128 x 64, two buffers in tensor memory), O += P V (128 x 256 in tensor memory, P too)
//   warps 2-5  softmax, one thread per query row, as in prefill_tc.cu: O is rescaled when a row of the warp has a new maximum
//   warps 6-13 expand a tile of keys, then one of values, into the swizzled 16-bit tiles that the products read (exact: e4m3 has
//              four significant bits); two tiles of each, so that they work one tile ahead
//
// Bound by what is serial in a tile, about 3700 cycles: 20 products into the same two accumulators one after the other (1500), the row's
// softmax with a full-precision soft cap, the rescaling of 256 columns of O.  Two prompts of 384 tokens, 16 heads on 8, soft cap 50: 19.5 us
// (general kernel 74.5), 32 tokens after 2000: 65 us (309).  Four expanding warps instead of eight: 21.8 and 80 us, eight are enough to
// stay off the chain.  The row sums add the weights as they were rounded: the error against 64 bits is then that of the general kernel
// (1.937e-3 against 1.944e-3; with unrounded weights 1.954e-3, the maximum being exact less often with 64 keys than with 32).
// Every wait is bounded; a wait that runs out sets the status word and the CTA leaves through the common teardown.
// The reference: vllm/attention/ops/triton_prefix_prefill.py in the reference tree.
#include <math_constants.h>

#include "../common/launch.cuh"
#include "../common/ptx.cuh"
#include "../common/tensormap.h"

namespace {
using namespace fi;

constexpr int kHd = 256, kRows = 128, kKeys = 64;
constexpr int kExpanders = 8;                                       // warps
constexpr int kThreads = 32 * (6 + kExpanders);
constexpr int kQAtom = kRows * 128, kKvAtom = kKeys * 128;          // 64 channels of a tile
constexpr int kQBytes = 4 * kQAtom, kKvBytes = 4 * kKvAtom, kRawBytes = kKeys * kHd;
constexpr int kHead = 1024;
constexpr int kSmem = kHead + kQBytes + 4 * kKvBytes + 2 * kRawBytes;
static_assert(kSmem <= 227 * 1024, "shared memory of one SM");
constexpr uint32_t kPCol = 128, kOCol = 256;                        // tensor memory: S 0..63 and 64..127, P, O
constexpr float kLog2e = 1.4426950408889634f;

struct Params {
  void* out;                 // [T, nh * 256]
  const int* block_tables;   // [B, max_blocks]
  const int* seq_lens;       // [B]
  const int* cu_q;           // [B + 1]
  int* status;
  int max_blocks, block_size, nh, nkv, window;
  float scale, softcap, v_scale;      // scale: of the raw products (softmax scale x scale of the keys)
  int is_fp16;
};

__device__ __forceinline__ uint32_t pack2(float a, float b, int is_fp16) {
  if (is_fp16) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack2(uint32_t w, int is_fp16) {
  if (is_fp16) return __half22float2(*reinterpret_cast<const __half2*>(&w));
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
// Two e4m3 values in the 16-bit type of the products.
__device__ __forceinline__ uint32_t expand2(uint32_t pair, int is_fp16) {
  uint32_t h;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h) : "h"(static_cast<uint16_t>(pair)));
  if (is_fp16) return h;
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  return pack2(f.x, f.y, 0);
}

__global__ void __launch_bounds__(kThreads, 1)
prefill_fp8_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                   const __grid_constant__ CUtensorMap v_map, const Params p) {
  pdl_wait();          // before all 512 TMEM columns are taken: see prefill_tc.cu
  if (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != 0) return;
  const int b = blockIdx.z, head = blockIdx.x;
  const int q_begin = p.cu_q[b], q_len = p.cu_q[b + 1] - q_begin;
  // the tiles with the longest KV range are scheduled first
  const int qt0 = (static_cast<int>(gridDim.y) - 1 - static_cast<int>(blockIdx.y)) * kRows;
  if (qt0 >= q_len) return;
  const int seq_len = p.seq_lens[b], pos0 = seq_len - q_len;
  const int rows = min(kRows, q_len - qt0), first_pos = pos0 + qt0, last_pos = first_pos + rows - 1;
  const int kv_lo = p.window > 0 ? max(0, first_pos - p.window + 1) : 0;
  const int tile_begin = kv_lo / kKeys;
  const int n_tiles = last_pos / kKeys + 1 - tile_begin;
  const int kvh = head / (p.nh / p.nkv);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) set_status(p.status, kStatusBadArg);
    return;
  }
  uint8_t* sQ = smem_raw + kHead;
  uint8_t* sK = sQ + kQBytes;                // [2]
  uint8_t* sV = sK + 2 * kKvBytes;           // [2]
  uint8_t* rawK = sV + 2 * kKvBytes;
  uint8_t* rawV = rawK + kRawBytes;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem_raw);
  uint64_t* raw_full = q_full + 1;           // [2]: keys, values
  uint64_t* raw_empty = raw_full + 2;        // [2]
  uint64_t* k_full = raw_empty + 2;          // [2] stages, and so on
  uint64_t* k_empty = k_full + 2;
  uint64_t* v_full = k_empty + 2;
  uint64_t* v_empty = v_full + 2;
  uint64_t* s_full = v_empty + 2;
  uint64_t* s_free = s_full + 2;
  uint64_t* p_full = s_free + 2;             // one of each: nobody can complete it again before all who wait have passed
  uint64_t* pv_done = p_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 1);
  volatile int* aborted = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int box_rows = min(p.block_size, kKeys), n_boxes = kKeys / box_rows;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&raw_full[i], n_boxes);      // every producer lane announces its own box
      mbar_init(&raw_empty[i], kExpanders);
      mbar_init(&k_full[i], kExpanders);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], kExpanders);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&s_free[i], 4);
    }
    mbar_init(p_full, 4);
    mbar_init(pv_done, 1);
    *aborted = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer: lane l < n_boxes keys, the next n_boxes lanes values
    if (lane == 0) {
      tma_prefetch_desc(&q_map);
      mbar_expect_tx(q_full, kQBytes);
#pragma unroll
      for (int a = 0; a < 4; ++a) tma_load_2d(sQ + a * kQAtom, &q_map, q_full, head * kHd + a * 64, q_begin + qt0);
    }
    if (lane < 2 * n_boxes) {
      const int which = lane >= n_boxes ? 1 : 0, pg = lane % n_boxes;
      const uint32_t box_bytes = static_cast<uint32_t>(box_rows) * kHd;
      const CUtensorMap* map = which ? &v_map : &k_map;
      uint8_t* dst = (which ? rawV : rawK) + pg * box_bytes;
      tma_prefetch_desc(map);
      const int* bt = p.block_tables + static_cast<long>(b) * p.max_blocks;
      auto row_of = [&](int j) -> int {
        const int tok = (tile_begin + j) * kKeys + pg * box_rows;
        const int blk = tok < seq_len ? bt[tok / p.block_size] : 0;     // past the end: the null block
        return (blk * p.nkv + kvh) * p.block_size + tok % p.block_size;
      };
      int row_next = row_of(0), issued = 0;
      for (int j = 0; j < n_tiles; ++j) {
        const int row = row_next;
        if (j + 1 < n_tiles) row_next = row_of(j + 1);   // the page id of the next tile is in flight during the wait
        if (!mbar_wait(&raw_empty[which], (j & 1) ^ 1)) {
          set_status(p.status, kStatusTimeoutEmpty);
          *aborted = 1;
          break;
        }
        mbar_expect_tx(&raw_full[which], box_bytes);
        tma_load_2d(dst, map, &raw_full[which], 0, row);
        issued = j + 1;
      }
      // own copies in flight must have landed before the CTA may leave
      if (issued > 0 && !mbar_wait(&raw_full[which], (issued - 1) & 1)) set_status(p.status, kStatusTimeoutFull);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ UMMA issuer
    if (elect_one()) {
      const uint32_t fmt = p.is_fp16 ? 0 : 1;
      const uint32_t idesc_qk = umma_idesc_f16(fmt, kRows, kKeys);
      const uint32_t idesc_pv = umma_idesc_f16(fmt, kRows, kHd) | kUmmaBMnMajor;
      bool ok = mbar_wait(q_full, 0);
      auto scores = [&](int j) -> bool {
        const int st = j & 1;
        if (!mbar_wait(&k_full[st], (j >> 1) & 1)) return false;
        if (j >= 2 && !mbar_wait(&s_free[st], ((j >> 1) - 1) & 1)) return false;
        tc_fence_after();
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const uint64_t dq = umma_desc_sw128_kmajor(smem_u32(sQ + a * kQAtom));
          const uint64_t dk = umma_desc_sw128_kmajor(smem_u32(sK + st * kKvBytes + a * kKvAtom));
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_f16(tmem_base + st * kKeys, dq + 2 * k, dk + 2 * k, idesc_qk, (a | k) != 0 ? 1u : 0u);
        }
        umma_commit(&s_full[st]);
        umma_commit(&k_empty[st]);
        return true;
      };
      ok = ok && scores(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles) ok = scores(j + 1);
        const int st = j & 1;
        ok = ok && mbar_wait(&v_full[st], (j >> 1) & 1) && mbar_wait(p_full, j & 1);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < kKeys / 16; ++k) {
          const uint64_t dv = umma_desc_sw128_mnmajor(smem_u32(sV + st * kKvBytes + k * 2048), kKvAtom);
          umma_f16_a_tmem(tmem_base + kOCol, tmem_base + kPCol + k * 8, dv, idesc_pv, (k | j) != 0 ? 1u : 0u);
        }
        umma_commit(pv_done);
        umma_commit(&v_empty[st]);
      }
      if (!ok) {
        set_status(p.status, kStatusTimeoutFull);
        *aborted = 1;
      }
    }
  } else if (warp >= 6) {
    // ------------------------------------------------------------------ expansion: kShare keys of a tile per warp
    constexpr int kShare = kKeys / kExpanders;
    const int r0 = (warp - 6) * kShare;
    bool ok = true;
    auto expand = [&](int j, int which) -> bool {
      const int st = j & 1;
      uint64_t* full = which ? v_full : k_full;
      if (!mbar_wait(&raw_full[which], j & 1) || !mbar_wait(&(which ? v_empty : k_empty)[st], ((j >> 1) & 1) ^ 1)) return false;
      const uint8_t* raw = which ? rawV : rawK;
      uint8_t* tile = (which ? sV : sK) + st * kKvBytes;
      // a row per pass: a lane's eight channels are one 16-byte chunk of the tile, no two lanes of a phase meet in a bank
      uint8_t* atom = tile + (lane >> 3) * kKvAtom;
#pragma unroll
      for (int i = 0; i < kShare; ++i) {
        const int r = r0 + i;
        uint2 w = *reinterpret_cast<const uint2*>(raw + r * kHd + lane * 8);
        if ((tile_begin + j) * kKeys + r >= seq_len) w = make_uint2(0, 0);            // whatever lies behind the last key
        *reinterpret_cast<uint4*>(atom + sw128_offset(r, lane & 7)) =
            make_uint4(expand2(w.x & 0xffffu, p.is_fp16), expand2(w.x >> 16, p.is_fp16), expand2(w.y & 0xffffu, p.is_fp16),
                       expand2(w.y >> 16, p.is_fp16));
      }
      fence_proxy_async_smem();      // plain writes -> visible to the tensor core
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&full[st]);
        mbar_arrive(&raw_empty[which]);
      }
      return true;
    };
    for (int j = 0; j < n_tiles && ok; ++j) ok = expand(j, 0) && expand(j, 1);
    if (!ok) {
      set_status(p.status, kStatusTimeoutFull);
      *aborted = 1;
    }
  } else {
    // ------------------------------------------------------------------ softmax + output rows
    const int quad = warp & 3, row = quad * 32 + lane, qpos = first_pos + row;
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const bool capped = p.softcap > 0.f;
    const float to_log2 = (capped ? 1.f : p.scale) * kLog2e;
    float m = -CUDART_INF_F, l = 0.f;                // maximum (log2), denominator
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      const int st = j & 1;
      ok = mbar_wait(&s_full[st], (j >> 1) & 1);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      tc_fence_after();
      uint32_t sr[kKeys];                            // this row's scores: read once, kept in registers
      tmem_ld_x32(t_lane + st * kKeys, sr);
      tmem_ld_x32(t_lane + st * kKeys + 32, sr + 32);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_free[st]);
      const int k0 = (tile_begin + j) * kKeys;
      if (capped) {
#pragma unroll
        for (int e = 0; e < kKeys; ++e) sr[e] = __float_as_uint(p.softcap * tanhf(__uint_as_float(sr[e]) * p.scale / p.softcap));
      }
      // keys of this tile the row may see: [vis_lo, vis_hi); only tiles on an edge look at them
      if ((k0 + kKeys - 1 > first_pos) || (p.window > 0 && k0 <= last_pos - p.window)) {
        const int vis_hi = qpos - k0 + 1;
        const int vis_lo = p.window > 0 ? qpos - p.window + 1 - k0 : 0;
#pragma unroll
        for (int e = 0; e < kKeys; ++e)
          if (e < vis_lo || e >= vis_hi) sr[e] = 0xff800000u;   // -inf: probability 0
      }
      float mt4[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
      for (int e = 0; e < kKeys; ++e) mt4[e & 3] = fmaxf(mt4[e & 3], __uint_as_float(sr[e]));
      const float mt = fmaxf(fmaxf(mt4[0], mt4[1]), fmaxf(mt4[2], mt4[3])) * to_log2;   // the factor is positive
      const float m_old = m;
      m = fmaxf(m, mt);
      const float alpha = m == -CUDART_INF_F ? 1.f : fast_exp2(m_old - m);
      const float m_use = m == -CUDART_INF_F ? 0.f : m;
      float rs0 = 0.f, rs1 = 0.f;                    // of the rounded weights: their errors then cancel in part
#pragma unroll
      for (int e = 0; e < kKeys; e += 2) {
        const float p0 = fast_exp2(fmaf(__uint_as_float(sr[e]), to_log2, -m_use));
        const float p1 = fast_exp2(fmaf(__uint_as_float(sr[e + 1]), to_log2, -m_use));
        sr[e >> 1] = pack2(p0, p1, p.is_fp16);
        const float2 f = unpack2(sr[e >> 1], p.is_fp16);
        rs0 += f.x;
        rs1 += f.y;
      }
      l = l * alpha + (rs0 + rs1);
      if (j > 0) {                                   // P of the tile in front has been read, its product is in O
        ok = mbar_wait(pv_done, (j - 1) & 1);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        tc_fence_after();
        if (__any_sync(0xffffffffu, m > m_old)) {
#pragma unroll 1
          for (int c = 0; c < kHd; c += 32) {
            uint32_t r[32];
            tmem_ld_x32(t_lane + kOCol + c, r);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * alpha);
            tmem_st_x32(t_lane + kOCol + c, r);
          }
        }
      }
      tmem_st_x32(t_lane + kPCol, sr);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    ok = ok && mbar_wait(pv_done, (n_tiles - 1) & 1);
    if (__all_sync(0xffffffffu, ok)) {
      tc_fence_after();
      const float inv = l > 0.f ? p.v_scale / l : 0.f;
      uint16_t* dst = reinterpret_cast<uint16_t*>(p.out) + (static_cast<long>(q_begin + qt0 + row) * p.nh + head) * kHd;
#pragma unroll 1
      for (int c = 0; c < kHd; c += 32) {
        uint32_t o[32];
        tmem_ld_x32(t_lane + kOCol + c, o);
        tmem_ld_wait();
        if (row >= rows) continue;
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) w[e] = pack2(__uint_as_float(o[i + 2 * e]) * inv, __uint_as_float(o[i + 2 * e + 1]) * inv, p.is_fp16);
          *reinterpret_cast<uint4*>(dst + c + i) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
    if (!ok) {
      set_status(p.status, kStatusTimeoutAccum);
      *aborted = 1;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace

// As fi_paged_prefill_tc for caches of e4m3 values with one scale per tensor and heads of 256 channels: caches [num_blocks, nkv, block_size,
// 256], pages of 16, 32 or a multiple of 64 tokens.  Returns -12 when the arguments are outside what this kernel covers.
extern "C" int fi_paged_prefill_fp8(const void* q, long q_stride, const void* k_cache, const void* v_cache, void* out,
                                    const int* block_tables, const int* seq_lens, const int* cu_q, int B, int T_total, int max_q_len, int nh,
                                    int nkv, int hd, long num_blocks, int max_blocks, int block_size, int window, float sm_scale,
                                    float softcap, float k_scale, float v_scale, int dtype, int* status, void* stream) {
  if (B <= 0 || max_q_len <= 0 || T_total <= 0) return 0;
  if (nkv <= 0 || nh <= 0 || nh % nkv != 0) return -10;
  if (hd != kHd || (dtype != 0 && dtype != 1)) return -12;
  if (!(sm_scale * k_scale > 0.f)) return -12;      // the largest raw product is taken for the largest score
  if (block_size != 16 && block_size != 32 && block_size % 64 != 0) return -12;
  if ((reinterpret_cast<uintptr_t>(q) & 15) != 0 || (q_stride * 2) % 16 != 0 || (reinterpret_cast<uintptr_t>(out) & 15) != 0) return -12;
  CUtensorMap qm, km, vm;
  const uint64_t kv_rows = static_cast<uint64_t>(num_blocks) * nkv * block_size;
  const uint32_t box = block_size < kKeys ? block_size : kKeys;
  if (make_tmap_2d_16bit_sw128(&qm, q, T_total, static_cast<uint64_t>(nh) * hd, q_stride, kRows) != 0 ||
      make_tmap_plain(&km, k_cache, kv_rows, hd, 1, kHd, box) != 0 || make_tmap_plain(&vm, v_cache, kv_rows, hd, 1, kHd, box) != 0)
    return -12;
  Params p = {};
  p.out = out; p.block_tables = block_tables; p.seq_lens = seq_lens; p.cu_q = cu_q; p.status = status;
  p.max_blocks = max_blocks; p.block_size = block_size; p.nh = nh; p.nkv = nkv; p.window = window;
  p.scale = sm_scale * k_scale; p.softcap = softcap; p.v_scale = v_scale; p.is_fp16 = dtype == 1;
  cudaError_t ce = ensure_dynamic_smem(prefill_fp8_kernel, kSmem);
  if (ce != cudaSuccess) return static_cast<int>(ce);
  ce = launch_kernel(prefill_fp8_kernel, dim3(nh, (max_q_len + kRows - 1) / kRows, B), dim3(kThreads), kSmem, reinterpret_cast<cudaStream_t>(stream), 0,
                     qm, km, vm, p);
  return static_cast<int>(ce != cudaSuccess ? ce : cudaGetLastError());
}
