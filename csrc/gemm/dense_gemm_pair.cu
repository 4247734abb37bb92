// Persistent dense GEMM with CTA pairs, sm_100a: the products of dense_gemm_persistent.cu whose sizes fill tiles of 256 weight rows.
//
// What bounds a product of many tokens is what an SM gets from L2: 64 bytes per cycle.  A tile of 128 rows x 256 tokens needs 48 KB per
// k-block of 64, 768 cycles for 512 cycles of tensor pipe.  Two CTAs that share one tcgen05.mma (cta_group::2, 256 rows) need 32 KB each: either
// loads its 128 weight rows and half of the tokens, and the tensor cores read the other half from the neighbour.
//
// The second bound is the accumulator: a product that adds to the accumulator of the one in front waits some 40 cycles for it (256 x 256 x 16: 173
// cycles, and 70 for each of two halves of 128 tokens that take turns).  So a tile has two accumulators, one per half of its
// tokens, and tensor memory holds the two of this tile and those of the next one (the epilogue of a tile runs under the next).
//
// Gated products: a CTA's 128 rows are eight gate rows, their eight up rows and so on (one four-dimensional TMA box), so that a pair's
// tile is 128 outputs x 256 tokens and both halves of an output meet in one warp.
//
// Roles (320 threads) as in dense_gemm_persistent.cu: warp 0 TMA, warp 1 MMA issuer (rank 0) and TMEM owner, warps 2..9 epilogue.  Barriers: `full` lives in
// rank 0, both CTAs' loads report to it; `empty` and acc_full are arrived at in both CTAs by the commit; acc_empty lives in rank 0.
// Every wait is bounded.
#include "../common/launch.cuh"
#include "../common/tensormap.h"
#include "persistent.cuh"

namespace fi {
namespace {

constexpr int kBk = 64;
constexpr int kPairEpilogueWarps = 8;
constexpr int kPairGemmThreads = 64 + 32 * kPairEpilogueWarps;

template <int BN> struct PairLayout {
  static constexpr int kA = kTileRows * 128;
  static constexpr int kHalf = BN / 4 * 128;               // this CTA's tokens of one half of the tile
  static constexpr int kStage = kA + 2 * kHalf;
  static constexpr int kStages = BN == 256 ? 6 : BN == 192 ? 7 : 8;
  static constexpr int kBytes = kStages * kStage + (2 * kStages + 4) * 8 + 16 + kPairEpilogueWarps * kPairPatchFloats * 4 + 1024;
  static_assert(kStage % 1024 == 0 && kHalf % 1024 == 0 && kBytes <= 227 * 1024, "swizzled tiles, shared memory of one SM");
};

template <int BN, bool GATED>
__global__ void __launch_bounds__(kPairGemmThreads, 1)
dense_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const PersistentParams p) {
  using L = PairLayout<BN>;
  constexpr int STAGES = L::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * L::kStage);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;        // [2]
  uint64_t* acc_empty = acc_full + 2;         // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* aborted = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* patches = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(tmem_slot) + 16);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 2 * kPairEpilogueWarps); }
    *aborted = 0;
    mbar_fence_init();
  }
  // All 512 columns: the kernel in front must not find them taken by a CTA that waits for it, so the wait comes first and the
  // kernels behind may start only when the columns are held here.
  pdl_wait();
  if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync();                              // the neighbour's barriers exist
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();

  const int kb_total = (p.K + kBk - 1) / kBk;
  const int n_token_tiles = p.n_tiles / p.n_tiles_n;
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tmap_w);
      tma_prefetch_desc(&tmap_x);
      int s = 0;
      uint32_t ph = 1;
      for (int tile = first; tile < p.n_tiles && !*aborted; tile += step) {
        int nt, tt;
        tile_at(p, tile, n_token_tiles, &nt, &tt);
        const int n0 = nt * p.rows_per_tile + static_cast<int>(rank) * (p.rows_per_tile / 2);
        const int t0 = tt * BN + static_cast<int>(rank) * (BN / 4);
        for (int kb = 0; kb < kb_total; ++kb) {
          if (!mbar_wait(&empty[s], ph)) {
            set_status(p.status, kStatusTimeoutEmpty);
            *aborted = 1;
            break;
          }
          uint8_t* a = smem + s * L::kStage;
          if (rank == 0) mbar_expect_tx(&full[s], 2 * L::kStage);
          const uint32_t bar = cluster_addr(&full[s], 0);
          if constexpr (GATED) tma_load_4d_pair(a, &tmap_w, bar, kb * kBk, 0, 0, n0 / 8);
          else tma_load_2d_pair(a, &tmap_w, bar, kb * kBk, n0);
          tma_load_2d_pair(a + L::kA, &tmap_x, bar, kb * kBk, t0);
          tma_load_2d_pair(a + L::kA + L::kHalf, &tmap_x, bar, kb * kBk, t0 + BN / 2);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (rank 0)
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = umma_idesc_f16(p.is_fp16 ? 0 : 1, 2 * kTileRows, BN / 2);
      int s = 0, local = 0;
      uint32_t ph = 0;
      for (int tile = first; tile < p.n_tiles && !*aborted; tile += step, ++local) {
        const int b = local & 1;
        if (!mbar_wait(&acc_empty[b], ((static_cast<uint32_t>(local) >> 1) & 1u) ^ 1u)) {     // both epilogues have drained it
          set_status(p.status, kStatusTimeoutAccum);
          *aborted = 1;
          break;
        }
        tc_fence_after();
        const uint32_t acc = tmem_base + static_cast<uint32_t>(b * 256);
        bool ok = true;
        for (int kb = 0; kb < kb_total; ++kb) {
          if (!mbar_wait(&full[s], ph)) {
            set_status(p.status, kStatusTimeoutFull);
            *aborted = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t at = smem_u32(smem + s * L::kStage);
          const uint64_t da = umma_desc_sw128_kmajor(at), d0 = umma_desc_sw128_kmajor(at + L::kA);
          const uint64_t d1 = umma_desc_sw128_kmajor(at + L::kA + L::kHalf);
#pragma unroll
          for (int k = 0; k < kBk / 16; ++k) {
            const uint32_t more = (kb | k) != 0 ? 1u : 0u;
            umma_f16_pair<true>(acc, da + 2 * k, d0 + 2 * k, idesc, more);
            umma_f16_pair<false>(acc + BN / 2, da + 2 * k, d1 + 2 * k, idesc, more);
          }
          umma_commit_pair(&empty[s]);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (!ok) break;
        umma_commit_pair(&acc_full[b]);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue warps, each half of the tile's tokens
    const int q = warp & 3, c_begin = ((warp - 2) >> 2) * (BN / 2), c_end = c_begin + BN / 2;
    float* patch = patches + (warp - 2) * kPairPatchFloats;
    int local = 0;
    for (int tile = first; tile < p.n_tiles; tile += step, ++local) {
      const int b = local & 1;
      if (*aborted || !mbar_wait(&acc_full[b], (static_cast<uint32_t>(local) >> 1) & 1u)) {
        if (!*aborted) { set_status(p.status, kStatusTimeoutAccum); *aborted = 1; }
        break;
      }
      tc_fence_after();
      int nt, tt;
      tile_at(p, tile, n_token_tiles, &nt, &tt);
      const int n0 = nt * p.rows_per_tile + static_cast<int>(rank) * (p.rows_per_tile / 2);
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(b * 256);
      if constexpr (GATED) drain_gate_up(p, taddr, patch, n0 + q * 16, tt * BN, p.T, c_begin, c_end, lane);
      else drain_tile<BN, false>(p, taddr, patch, n0, tt * BN, p.T, c_begin, c_end, q, lane);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[b], 0));
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                              // nobody reads this CTA's shared memory or arrives at its barriers any more
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

template <int BN, bool GATED>
int launch(const CUtensorMap& tw, const CUtensorMap& tx, const PersistentParams& p, int sms, cudaStream_t stream) {
  auto kern = dense_gemm_pair_kernel<BN, GATED>;
  const cudaError_t e = ensure_dynamic_smem(kern, PairLayout<BN>::kBytes);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int pairs = p.n_tiles < sms / 2 ? p.n_tiles : sms / 2;
  return static_cast<int>(launch_kernel_cluster(kern, dim3(2 * pairs), dim3(kPairGemmThreads), PairLayout<BN>::kBytes, stream, dim3(2, 1, 1), tw,
                                                tx, p));
}

inline int sm_count() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 1 ? v : 148;
  }();
  return n;
}

}  // namespace

int dense_gemm_pair(const void* X, const void* W, PersistentParams p, int ldx, int ldw, int tokens, cudaStream_t stream) {
  const bool gated = p.dual_rows > 0;
  CUtensorMap tw, tx;
  int r = gated ? make_tmap_gate_up_16bit_sw128(&tw, W, p.dual_rows, p.K, ldw) : make_tmap_2d_16bit_sw128(&tw, W, p.N, p.K, ldw, kTileRows);
  if (r != 0) return r * 100 - 1;
  r = make_tmap_2d_16bit_sw128(&tx, X, p.T, p.K, ldx, tokens / 4);
  if (r != 0) return r * 100 - 2;
  p.rows_per_tile = gated ? kTileRows : 2 * kTileRows;      // outputs of a pair's tile
  p.n_tiles_n = (p.N + p.rows_per_tile - 1) / p.rows_per_tile;
  p.n_tiles = p.n_tiles_n * ((p.T + tokens - 1) / tokens);
  p.n_group = 8;           // about as many weight rows as tokens in the block of tiles in flight (tile_at)
  if (p.n_group > p.n_tiles_n) p.n_group = p.n_tiles_n;
  const int sms = sm_count();
  switch (tokens) {
    case 256: return gated ? launch<256, true>(tw, tx, p, sms, stream) : launch<256, false>(tw, tx, p, sms, stream);
    case 192: return gated ? launch<192, true>(tw, tx, p, sms, stream) : launch<192, false>(tw, tx, p, sms, stream);
    case 128: return gated ? launch<128, true>(tw, tx, p, sms, stream) : launch<128, false>(tw, tx, p, sms, stream);
    default: return -14;
  }
}

}  // namespace fi

// The same with a tile chosen by the caller: measurements and tests.
extern "C" int fi_dense_gemm_pair(const void* X, const void* W, void* C, const void* bias, const void* residual, int T, int N, int K,
                                  int ldx, int ldw, int ldc, int act, float act_limit, int dual_rows, int out_fp32, int dtype, int tokens,
                                  int* status, void* stream) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  if ((K % 8) != 0 || (ldx % 8) != 0 || (ldw % 8) != 0 || (N % 8) != 0 || (ldc % 8) != 0 ||
      (reinterpret_cast<uintptr_t>(C) & 15) != 0 || (residual != nullptr && (reinterpret_cast<uintptr_t>(residual) & 15) != 0))
    return -10;
  if (dual_rows > 0 && N != dual_rows) return -11;
  if (act == 4 && (dual_rows <= 0 || !(act_limit > 0.f))) return -12;
  if (out_fp32 && residual != nullptr) return -13;
  fi::PersistentParams p = {};
  p.C = C; p.bias = bias; p.residual = residual;
  p.T = T; p.N = N; p.K = K; p.ldc = ldc;
  p.dual_rows = dual_rows; p.act = act; p.act_limit = act_limit; p.is_fp16 = dtype == 1; p.out_fp32 = out_fp32; p.status = status;
  return fi::dense_gemm_pair(X, W, p, ldx, ldw, tokens, reinterpret_cast<cudaStream_t>(stream));
}
