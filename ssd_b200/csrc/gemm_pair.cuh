// gemm_pair.cuh — tcgen05 GEMM of calls with many rows (prompt portions): C[M, N] = X[M, K] · W[N, K]^T, bf16 operands, fp32
// accumulation in TMEM.  Two CTAs of a cluster work on one tile of 256 weight rows x up to 256 tokens (cta_group::2).
//
// What bounds it and why this shape.  A k-block of 64 takes the tensor core 512 clocks for 256 tokens.  One CTA with 128 weight rows
// and 256 tokens must bring 48 KB into shared memory in that time; the pair shares the tile, each CTA holds 128 weight rows and half
// of the tokens: 32 KB per k-block and SM.  The pairs are persistent (74 of them on 148 SMs): accumulators of 2 x 256 TMEM columns let
// the epilogue of a tile run under the products of the next one, and the load ring runs on across tiles, where a CTA per tile
// (gemm_ws_kernel) pays its set-up, its first loads and its stores in the open.  Tiles are walked token chunks first, so that the tiles
// in flight share the weight rows through L2.  Measured, cold L2, us (TFLOP/s), gemm_ws_kernel -> this one: 2048 x 4096 x 2048
// 47.1 (729) -> 37.9 (907); 2048 x 10272 x 2048 111.6 (772) -> 77.8 (1107); 2048 x 4096 x 14336 192 (1249) -> 186 (1290);
// gated 2048 x 2 6144 x 2048 165 (625) -> 106 (968); gated 2048 x 2 14336 x 4096 555 (867) -> 369 (1305).  What is left: the last
// wave (128 tiles on 74 pairs) and the L2 latency that six stages of 32 KB cover at about 1300 TFLOP/s.
//   warp 0     loads: 6 stages of {128 weight rows, up to 128 token rows} x 64 k, 128B-swizzled; both CTAs' bytes count on the
//              leader's full barrier
//   warp 1     leader only: tcgen05.mma.cta_group::2 M = 256, N = the tile's tokens rounded up to 64; commits free the stage in both CTAs
//   warps 2-5  epilogue of this CTA's 128 weight rows: fp32 or bf16 store, or act(gate) * up in bf16.  For the latter the weight rows of a tile
//              alternate in runs of 16 gate and 16 up rows, so that gate and up of an output column sit 16 lanes apart in one warp
// Grouped mode (mixture of experts): a device-side list of row tiles, each of one expert, as in gemm_ws_kernel.
// The order of the sums over K is that of gemm_ws_kernel without split-K: the results are the same bits.
#pragma once
#include <cuda.h>
#include "gemm.cuh"

namespace ssdk {

constexpr int kPairStages = 6, kPairTokens = 256, kPairStageBytes = 2 * 16384, kPairThreads = 192;
constexpr int kPairSmem = kPairStages * kPairStageBytes + 1024;
// A load instruction costs the load unit some 40 clocks whatever its size: with 4 KB boxes (eight and more per stage) the kernel ran
// at 1129 TFLOP/s instead of 1335 (2048 x 4096 x 14336), the gated form at 799 instead of 1320.  A stage is one load of 128 weight
// rows (a five-dimensional box picks the gated form's runs of 16) and one of the tile's token half: 128 rows, or 32-row boxes for up to 64.
constexpr int kPairXBox = 128, kPairXSmall = 32, kPairGluRun = 16;

// activations of the gated form; SILU_ROUNDED rounds gate and up to bf16 first (the dense decoders' linear layers return bf16)
enum { GLU_SILU = 0, GLU_GELU = 1, GLU_SILU_ROUNDED = 2 };

struct GemmPairParams {
  void* out;          // EPI_PARTIAL: fp32 [M, ldo]; EPI_GLU, EPI_BF16: bf16 [M, ldo]
  int M, N, ldo;      // N: output columns (EPI_GLU: of the product act(gate) * up; the up rows start N rows behind the gate rows)
  int num_kb;         // K / 64
  int w_tiles;        // tiles along the weight rows: 256 columns (EPI_PARTIAL) or 128 (EPI_GLU) of the output
  int chunks;         // row chunks of kPairTokens tokens (dense)
  int act;            // EPI_GLU: GLU_*
  // dense: products of the same shape side by side (heads): product b reads X's columns from b x_step, the weight rows from b N, and
  // writes out + b out_step
  int batch, x_step, out_step;
  // W_COLS (dense): the weights are [heads][K][w_head] (w_head a multiple of 64): output column n is column n % w_head of head n / w_head
  int w_head;
  // grouped mode: see GemmParams
  const int* g_tile_expert;
  const int* g_tile_row0;
  const int* g_tile_rows;
  const int* g_n_tiles;
  int g_expert_rows;
  unsigned* timeout;  // host-mapped word: set when a wait runs out (the results are then invalid)
};

// ---- cluster and cta_group::2 forms ----
SSDK_DEVINL uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
SSDK_DEVINL void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of `smem` in the CTA of rank `rank`
SSDK_DEVINL uint32_t map_shared(const void* smem, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(smem)), "r"(rank));
  return r;
}
SSDK_DEVINL void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// bounded wait; false: it ran out
SSDK_DEVINL bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, unsigned* timeout) {
  const long long t0 = clock64();
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - t0 > 4000000000LL) {   // ~2 s
      if (timeout) *(volatile unsigned*)timeout = 1u;
      return false;
    }
  }
}
SSDK_DEVINL void tma_load_2d_pair(void* smem_dst, const void* tmap, uint32_t bar_addr, int c0, int c1, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar_addr), "r"(c0), "r"(c1), "l"(policy)
      : "memory");
}
// gated weights as {k, row of a run, gate / up, run, expert}: 64 k x 16 rows x both x 4 runs from run `run` of expert `ex`
SSDK_DEVINL void tma_load_5d_pair(void* smem_dst, const void* tmap, uint32_t bar_addr, int k, int run, int ex) {
  asm volatile(
      "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar_addr), "r"(k), "r"(0), "r"(run), "r"(ex)
      : "memory");
}
SSDK_DEVINL void umma_bf16_ss_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier at this offset in both CTAs once the products issued so far are done
SSDK_DEVINL void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3)
               : "memory");
}
// all 512 TMEM columns of both CTAs (a whole warp in each)
SSDK_DEVINL void tmem_alloc_pair(uint32_t* smem_dst) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(512) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
SSDK_DEVINL void tmem_dealloc_pair(uint32_t taddr) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(512) : "memory");
}

// Operand that is contiguous along M or N, 128-byte swizzle: atoms of 64 elements x 8 k; the next 8 k follow 1024 B on (SBO), the next 64
// elements `next64` bytes on (LBO)
SSDK_DEVINL uint64_t make_umma_desc_mn128(const void* smem_tile, uint32_t next64) {
  const uint32_t addr = smem_u32(smem_tile);
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)((next64 >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)(1024u >> 4) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)2u << 61;
  return d;
}

// W_COLS: weights whose output columns are contiguous and not their k (two boxes of 64 columns x 64 k per stage)
template <int EPI, bool W_COLS = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmXs,
                 const GemmPairParams p) {
  extern __shared__ uint8_t pair_smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kPairStages];    // the leader's are used: both CTAs' bytes of a stage
  __shared__ __align__(8) uint64_t empty_bar[kPairStages];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  uint8_t* smem = pair_smem_raw + ((1024u - (smem_u32(pair_smem_raw) & 1023u)) & 1023u);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = (int)blockIdx.x >> 1, n_pairs = (int)gridDim.x >> 1;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmXs);
    for (int s = 0; s < kPairStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 8); }   // four epilogue warps in each CTA
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc_pair(&tmem_slot);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // both CTAs' barriers are set up before a load or a commit of the other one reaches them
  tc_fence_after();
  const uint32_t tmem_d = tmem_slot;

  pdl_launch_dependents();
  pdl_wait();

  const bool grouped = p.g_tile_expert != nullptr;
  const int row_tiles = grouped ? *p.g_n_tiles : p.chunks;
  const int per = row_tiles * p.w_tiles, tiles = grouped ? per : per * p.batch;
  // tile t: row chunk (the inner index), weight rows, product of the batch
  struct Tile { int m0, rows, n, col, ex, b; };   // first token, valid tokens, multiplied tokens, this CTA's first output column, expert, product
  auto tile_of = [&](int t) {
    Tile r;
    r.b = grouped ? 0 : t / per;
    t -= r.b * per;
    const int wt = t / row_tiles, c = t - wt * row_tiles;
    r.ex = 0;
    if (grouped) {
      r.m0 = p.g_tile_row0[c]; r.rows = min(kPairTokens, p.g_tile_rows[c]); r.ex = p.g_tile_expert[c];
    } else {
      r.m0 = c * kPairTokens; r.rows = min(kPairTokens, p.M - r.m0);
    }
    r.n = (r.rows + 63) & ~63;
    r.col = EPI == EPI_GLU ? wt * 128 + (int)rank * 64 : wt * 256 + (int)rank * 128;
    return r;
  };

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      bool ok = true;
      for (int t = pair; t < tiles && ok; t += n_pairs) {
        const Tile tl = tile_of(t);
        const int half = tl.n >> 1, x0 = tl.m0 + (int)rank * half;
        const bool big = half > 64;
        const int w_row = tl.ex * p.g_expert_rows + tl.b * p.N + tl.col, kx = tl.b * p.x_step;
        const uint32_t bytes = 2u * (16384u + (big ? (uint32_t)kPairXBox : (uint32_t)half) * 128u);
        for (int kb = 0; kb < p.num_kb; ++kb, ++it) {
          const int s = it % kPairStages;
          if (!(ok = mbar_wait_cluster(&empty_bar[s], ((uint32_t)(it / kPairStages) & 1u) ^ 1u, p.timeout))) break;
          uint8_t* a_s = smem + s * kPairStageBytes;
          uint8_t* b_s = a_s + 16384;
          if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], bytes);
          const uint32_t bar = map_shared(&full_bar[s], 0);
          const int k = kb * kBlockK;
          if (EPI == EPI_GLU) tma_load_5d_pair(a_s, &tmW, bar, k, tl.col / kPairGluRun, tl.ex);
          else if (W_COLS)
            for (int b = 0; b < 2; ++b) {
              const int n = tl.col + b * 64, head = n / p.w_head;
              tma_load_2d_pair(a_s + b * 8192, &tmW, bar, n - head * p.w_head, head * p.num_kb * kBlockK + k, kEvictNormal);
            }
          else tma_load_2d_pair(a_s, &tmW, bar, k, w_row, kEvictNormal);
          if (big) tma_load_2d_pair(b_s, &tmX, bar, kx + k, x0, kEvictNormal);
          else
            for (int b = 0; b < half; b += kPairXSmall) tma_load_2d_pair(b_s + b * 128, &tmXs, bar, kx + k, x0 + b, kEvictNormal);
        }
      }
      // the last commits of the leader reach this CTA's barriers before it leaves
      for (int i = 0; i < kPairStages && ok; ++i, ++it)
        ok = mbar_wait_cluster(&empty_bar[it % kPairStages], ((uint32_t)(it / kPairStages) & 1u) ^ 1u, p.timeout);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      int it = 0, nt = 0;
      bool ok = true;
      for (int t = pair; t < tiles && ok; t += n_pairs, ++nt) {
        const Tile tl = tile_of(t);
        const uint32_t idesc = make_umma_idesc_bf16(256, tl.n) | (W_COLS ? 1u << 15 : 0u), acc = tmem_d + (uint32_t)(nt & 1) * 256u;
        if (!(ok = mbar_wait_cluster(&acc_empty[nt & 1], ((uint32_t)(nt >> 1) & 1u) ^ 1u, p.timeout))) break;
        tc_fence_after();
        for (int kb = 0; kb < p.num_kb; ++kb, ++it) {
          const int s = it % kPairStages;
          if (!(ok = mbar_wait_cluster(&full_bar[s], (uint32_t)(it / kPairStages) & 1u, p.timeout))) break;
          tc_fence_after();
          uint8_t* a_s = smem + s * kPairStageBytes;
          const uint64_t adesc = W_COLS ? make_umma_desc_mn128(a_s, 8192) : make_umma_desc_k128(a_s), bdesc = make_umma_desc_k128(a_s + 16384);
#pragma unroll
          for (int k = 0; k < kBlockK / 16; ++k)   // 16 k: 32 B of a row, 16 rows of 128 B of W_COLS
            umma_bf16_ss_pair(acc, adesc + (uint64_t)((W_COLS ? 128 : 2) * k), bdesc + (uint64_t)(2 * k), idesc, (uint32_t)((kb | k) != 0));
          umma_commit_pair(&empty_bar[s]);
        }
        if (ok) umma_commit_pair(&acc_full[nt & 1]);
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3;   // the quarter of the TMEM lanes that this warp reads
    int nt = 0;
    for (int t = pair; t < tiles; t += n_pairs, ++nt) {
      const Tile tl = tile_of(t);
      const int b = nt & 1;
      if (!mbar_wait_cluster(&acc_full[b], (uint32_t)(nt >> 1) & 1u, p.timeout)) break;
      tc_fence_after();
      const uint32_t src = tmem_d + ((uint32_t)(q * 32) << 16) + (uint32_t)b * 256u;
      for (int m0 = 0; m0 < tl.rows; m0 += 32) {
        uint32_t r[32];
        tmem_ld_32x32b_x16(src + m0, r);
        tmem_ld_32x32b_x16(src + m0 + 16, r + 16);
        tmem_ld_wait();
        const int left = tl.rows - m0;
        if (EPI == EPI_GLU) {
          // lanes 0 .. 15 hold gate, 16 .. 31 up of columns q * 16 .. of this CTA: of two tokens the low half computes the first,
          // the high half the second
          const bool lo = lane < 16;
          const int n = tl.col + q * 16 + (lane & 15);
          __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)(tl.m0 + m0 + (lo ? 0 : 1)) * p.ldo + n;
#pragma unroll
          for (int m = 0; m < 32; m += 2) {
            const float keep = __uint_as_float(lo ? r[m] : r[m + 1]);
            const float got = __shfl_xor_sync(0xffffffffu, __uint_as_float(lo ? r[m + 1] : r[m]), 16);
            float g = lo ? keep : got, u = lo ? got : keep;
            if (p.act == GLU_SILU_ROUNDED) { g = bf16_round(g); u = bf16_round(u); }
            const float a = p.act == GLU_GELU ? 0.5f * g * (1.0f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) : __fdividef(g, 1.0f + __expf(-g));
            if (n < p.N && m + (lo ? 0 : 1) < left) out[(size_t)m * p.ldo] = f2bf(a * u);
          }
        } else if (EPI == EPI_BF16) {
          const int n = tl.col + q * 32 + lane;
          if (n < p.N) {
            __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)tl.b * p.out_step + (size_t)(tl.m0 + m0) * p.ldo + n;
#pragma unroll
            for (int m = 0; m < 32; ++m)
              if (m < left) out[(size_t)m * p.ldo] = f2bf(__uint_as_float(r[m]));
          }
        } else {
          const int n = tl.col + q * 32 + lane;
          if (n < p.N) {
            float* out = reinterpret_cast<float*>(p.out) + (size_t)tl.b * p.out_step + (size_t)(tl.m0 + m0) * p.ldo + n;
            if (left >= 32) {
#pragma unroll
              for (int m = 0; m < 32; ++m) out[(size_t)m * p.ldo] = __uint_as_float(r[m]);
            } else {
#pragma unroll
              for (int m = 0; m < 32; ++m)
                if (m < left) out[(size_t)m * p.ldo] = __uint_as_float(r[m]);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_shared(&acc_empty[b], 0));
    }
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // neither CTA leaves while the other one may still arrive on its barriers or read its shared memory
  if (warp == 1) tmem_dealloc_pair(tmem_d);
}

}  // namespace ssdk
