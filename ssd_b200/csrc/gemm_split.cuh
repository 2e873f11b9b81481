// gemm_split.cuh — fp32 GEMM of the exact mode on the tensor cores: C[M, N] = X[M, K] · W[N, K]^T with fp32 operands and results at the
// accuracy of a chain of fp32 FMAs.
//
// Every operand is the sum of three bf16 pieces, x = h + m + l (8 significant bits each, what is left over is below 2^-27 of x), and
// a product is taken as hh + (hm + mh + mm + hl + lh): six tcgen05.mma of kind::f16 whose products are exact; the terms that are left out
// are below 2^-26.  The tensor core truncates when it adds to its fp32 accumulator: measured against 64 bits (random signs) 2.2e-7 of
// the result over 256 steps of k but 2.1e-6 over 2048, where a chain of FMAs is off by 1.0e-7 and 3.8e-7.  So the hh sums leave TMEM every
// 256 k and are added up in registers (fp32, round to nearest); the five small terms, 2^-8 of the result, stay in an accumulator of
// their own up to the end.  Relative error of 1000 x 4096 x 2048 against 64 bits: 2.4e-7, the FMA form 7.9e-7.
//
// Where pieces do not do: an operand that is infinite or above bf16's largest number (3.39e38) has an infinite first piece, so that its
// products are infinite or NaN, and pieces below bf16's normal range (2^-126) may be lost, which is below 2^-24 of a result from 2^-70
// on (as long as K times the largest other operand is below 2^30).  Results that are not finite, and results below 2^-70 that are not zero, are
// therefore taken again as the FMA chain over k that linear_kernel walks (see split_again).  What still differs: a result below 2^-126 may be zero.
//
// What bounds it: the tensor core takes about 85 clocks for an instruction and one more for four tokens, so that a k-block of 64 (24 products) is 2040 clocks
// and 6 a token; measured, with what the stages do not cover, 3100 and 7.5 (960 x 4096 x 2048 with chunks of 96, 128, 160, 192 tokens: 3800, 4090, 4410, 4520).
// Chunks of up to 192 tokens therefore (of 128, in three stages: 1000 x 3072 x 2048 137 us, 82 here).  The FMA form that it took over from (linear_kernel,
// 64 x 64 tiles) was bound by its shared-memory operands: 1000 x 4096 x 2048 539 us (31 TFLOP/s), 2000 x 8192 x 2048 2092.  With few rows the kernel streams
// the weights (8 x 8192 x 2048 148 us in the FMA form), which is why the tokens of a tile go down to 32.  Pairs of CTAs and the persistent walk as in
// gemm_pair.cuh; the weights are read as fp32 and split on their way into shared memory (6 bytes in memory for every 4 would cost more
// than the conversion), the rows of X, read by every tile, are split beforehand.  Two stages of 84 KB.  The large sums (hh) and the five small ones have an accumulator
// of 192 columns each; the small terms of a k-block go first, so that the large sums of the segment before leave tensor memory under them.
//   warp 0       loads: the three pieces of this CTA's token half (up to 96 rows x 64 k each, in boxes of 32 rows)
//   warp 1       leader only: the products
//   warps 4-7    sums: thread = output column, up to 192 tokens in registers (232 of them)
//   warps 8-15   weights: 128 rows x 64 k of fp32, the next k-block's loads in flight while this one is split and stored (128B swizzle)
#pragma once
#include "gemm_pair.cuh"

namespace ssdk {

constexpr int kSplitTokens = 192, kSplitStages = 2, kSplitThreads = 512, kSplitSegment = 4;   // segment: k-blocks between two drains
constexpr int kSplitXBox = 32, kSplitSeeTiles = 128;
constexpr int kSplitWPlane = 128 * 128, kSplitXPlane = kSplitTokens / 2 * 128, kSplitStageBytes = 3 * (kSplitWPlane + kSplitXPlane);
constexpr int kSplitSmem = kSplitStages * kSplitStageBytes + 1024;

struct GemmSplitParams {
  const float* W;     // [N, ldw]
  float* out;         // [splits][M, ldc]
  int M, N, K, ldw, ldc;
  int num_kb, kb_per_split, splits;
  int w_tiles, chunks, tokens;   // tiles of 256 columns; dense: chunks of `tokens` rows (a multiple of 32, at most kSplitTokens)
  int batch;                  // dense: products of the same shape, their weights and results w_stride and c_stride floats apart, X's rows in turn
  int plane_rows;             // rows of one piece of X (the map holds three of them)
  const float* X;             // the rows themselves, for results that are taken again: row r of matrix b is row x_rows[r] (or r) from X + b x_stride
  const int* x_rows;
  long long x_stride;
  int ldx;
  long long w_stride, c_stride;   // grouped: w_stride between two experts
  const int* g_tile_expert;   // grouped mode: see GemmParams (tiles of up to kSplitTokens rows)
  const int* g_tile_row0;
  const int* g_tile_rows;
  const int* g_n_tiles;
  // Attention (dense, splits 1): row r of a matrix has to do with columns (see_k: steps of k) below see + r / see_heads only.  Tiles beyond are left
  // out, or k ends there (X holds what lies between a row's own end and that of its chunk's last row; chunks then go from the longest to the
  // shortest, there and back over the pairs).  see_heads 0: all of it
  int see, see_heads, see_k;
  unsigned* timeout;
};

// two floats -> their three bf16 pieces, packed
SSDK_DEVINL void split3(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
  const __nv_bfloat162 hh = __floats2bfloat162_rn(a, b);
  const float2 hf = __bfloat1622float2(hh);
  const float a1 = a - hf.x, b1 = b - hf.y;
  const __nv_bfloat162 mm = __floats2bfloat162_rn(a1, b1);
  const float2 mf = __bfloat1622float2(mm);
  const __nv_bfloat162 ll = __floats2bfloat162_rn(a1 - mf.x, b1 - mf.y);
  h = *reinterpret_cast<const uint32_t*>(&hh);
  m = *reinterpret_cast<const uint32_t*>(&mm);
  l = *reinterpret_cast<const uint32_t*>(&ll);
}

// rows of X as three pieces: dst [3][batch * M, K] (bf16).  grid (ceil(M / blockDim.y), batch): row r of matrix b (`stride` floats apart) is row rows[r]
// of src if there is a list; rows from *n_rows on are left out.  Narrow rows share a block: 25152 rows of 64 columns 25 -> 4 us
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ src, int ld, long long stride, const int* __restrict__ rows,
                                                         const int* __restrict__ n_rows, __nv_bfloat16* __restrict__ dst, int M, int K) {
  pdl_launch_dependents();
  pdl_wait();
  const int r = blockIdx.x * blockDim.y + threadIdx.y;
  if (r >= M || (n_rows && r >= *n_rows)) return;
  const float4* s = reinterpret_cast<const float4*>(src + blockIdx.y * stride + (size_t)(rows ? rows[r] : r) * ld);
  const size_t plane = (size_t)M * gridDim.y * K;
  __nv_bfloat16* d = dst + ((size_t)blockIdx.y * M + r) * K;
  for (int c = threadIdx.x; c < K / 4; c += blockDim.x) {
    const float4 v = s[c];
    uint2 h, m, l;
    split3(v.x, v.y, h.x, m.x, l.x);
    split3(v.z, v.w, h.y, m.y, l.y);
    reinterpret_cast<uint2*>(d)[c] = h;
    reinterpret_cast<uint2*>(d + plane)[c] = m;
    reinterpret_cast<uint2*>(d + 2 * plane)[c] = l;
  }
}

// a result that the pieces cannot vouch for: infinite, NaN, or below 2^-70 and not zero
SSDK_DEVINL bool split_again(float v) {
  constexpr uint32_t lo = (127u - 70u) << 24, hi = 255u << 24;
  const uint32_t u = __float_as_uint(v) << 1;
  return u != 0u && u - lo >= hi - lo;
}

// registers of a warpgroup: 56 + 232 + 2 x 112 = 4 x 128, what the block is launched with
template <int R>
SSDK_DEVINL void regs_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
SSDK_DEVINL void regs_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kSplitThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmX, const GemmSplitParams p) {
  extern __shared__ uint8_t split_smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kSplitStages];   // the leader's are used: the loads' bytes and eight weight warps of both CTAs
  __shared__ __align__(8) uint64_t empty_bar[kSplitStages];
  __shared__ __align__(8) uint64_t main_full, main_empty, rest_full, rest_empty;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_again;   // some result of this CTA's is to be taken again
  __shared__ int s_seen[kSplitSeeTiles + 1];   // tiles in front of a column tile's, where some are left out
  uint8_t* smem = split_smem_raw + ((1024u - (smem_u32(split_smem_raw) & 1023u)) & 1023u);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = (int)blockIdx.x >> 1, n_pairs = (int)gridDim.x >> 1;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmX);
    for (int s = 0; s < kSplitStages; ++s) { mbar_init(&full_bar[s], 17); mbar_init(&empty_bar[s], 1); }
    mbar_init(&main_full, 1); mbar_init(&main_empty, 8); mbar_init(&rest_full, 1); mbar_init(&rest_empty, 8);   // four sum warps in each CTA
    fence_mbar_init();
    s_again = 0;
    if (p.see_heads && !p.see_k) {   // column tile w: the chunks from that of the first row which sees column 256 w
      s_seen[0] = 0;
      for (int w = 0; w < p.w_tiles; ++w) s_seen[w + 1] = s_seen[w] + max(0, p.chunks - max(0, w * 256 - p.see + 1) * p.see_heads / p.tokens);
    }
  }
  if (warp == 1) tmem_alloc_pair(&tmem_slot);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_main = tmem_slot, tmem_rest = tmem_slot + 256u;

  pdl_launch_dependents();
  pdl_wait();

  const bool grouped = p.g_tile_expert != nullptr;
  const int row_tiles = grouped ? *p.g_n_tiles : p.chunks;
  const bool see_k = p.see_heads && p.see_k, see_cols = p.see_heads && !p.see_k;
  const int per = see_cols ? s_seen[p.w_tiles] : row_tiles * p.splits * p.w_tiles, tiles = grouped ? per : per * p.batch;
  // this pair's i-th tile
  auto tile_at = [&](int i) { return i * n_pairs + (see_k && (i & 1) ? n_pairs - 1 - pair : pair); };
  struct Tile { int m0, rows, n, col, kb0, kb1, split, b; long long w0; };
  auto tile_of = [&](int t) {   // row chunk (innermost), k range, 256 columns, matrix of the batch
    Tile r;
    int c, wt;
    r.split = 0;
    if (see_k) {
      r.b = t % p.batch;
      t /= p.batch;
      wt = t % p.w_tiles; c = p.chunks - 1 - t / p.w_tiles;
    } else {
      r.b = grouped ? 0 : t / per;
      t -= r.b * per;
      if (see_cols) {
        for (wt = 0; s_seen[wt + 1] <= t; ++wt);
        c = p.chunks - (s_seen[wt + 1] - t);
      } else {
        const int u = t / row_tiles;
        c = t - u * row_tiles; wt = u / p.splits;
        r.split = u - wt * p.splits;
      }
    }
    if (grouped) {
      r.m0 = p.g_tile_row0[c]; r.rows = min(kSplitTokens, p.g_tile_rows[c]); r.w0 = p.g_tile_expert[c] * p.w_stride;
    } else {
      r.m0 = c * p.tokens; r.rows = min(p.tokens, p.M - r.m0); r.w0 = r.b * p.w_stride;
    }
    r.n = (r.rows + 31) & ~31;
    r.col = wt * 256 + (int)rank * 128;
    r.kb0 = r.split * p.kb_per_split;
    r.kb1 = min(p.num_kb, r.kb0 + p.kb_per_split);
    if (see_k) r.kb1 = min(r.kb1, (p.see + (r.m0 + r.rows - 1) / p.see_heads + kBlockK - 1) / kBlockK);
    return r;
  };

  if (warp < 4) {
    regs_down<56>();
    if (warp == 0 && lane == 0) {
      int it = 0;
      bool ok = true;
      for (int i = 0, t; (t = tile_at(i)) < tiles && ok; ++i) {
        const Tile tl = tile_of(t);
        const int half = tl.n >> 1, x0 = tl.b * p.M + tl.m0 + (int)rank * half, boxes = (half + kSplitXBox - 1) / kSplitXBox;
        for (int kb = tl.kb0; kb < tl.kb1; ++kb, ++it) {
          const int s = it % kSplitStages;
          if (!(ok = mbar_wait_cluster(&empty_bar[s], ((uint32_t)(it / kSplitStages) & 1u) ^ 1u, p.timeout))) break;
          uint8_t* b_s = smem + s * kSplitStageBytes + 3 * kSplitWPlane;
          if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], 2u * 3u * (uint32_t)boxes * kSplitXBox * 128u);
          const uint32_t bar = map_shared(&full_bar[s], 0);
          for (int i = 0; i < boxes; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j)
              tma_load_2d_pair(b_s + j * kSplitXPlane + i * kSplitXBox * 128, &tmX, bar, kb * kBlockK, j * p.plane_rows + x0 + i * kSplitXBox, kEvictNormal);
        }
      }
      for (int i = 0; i < kSplitStages && ok; ++i, ++it)   // the last commits reach this CTA before it leaves
        ok = mbar_wait_cluster(&empty_bar[it % kSplitStages], ((uint32_t)(it / kSplitStages) & 1u) ^ 1u, p.timeout);
    } else if (warp == 1 && lane == 0 && rank == 0) {
      int it = 0, nt = 0, sg = 0;
      bool ok = true;
      for (int t; (t = tile_at(nt)) < tiles && ok; ++nt) {
        const Tile tl = tile_of(t);
        const uint32_t idesc = make_umma_idesc_bf16(256, tl.n);
        if (!(ok = mbar_wait_cluster(&rest_empty, ((uint32_t)nt & 1u) ^ 1u, p.timeout))) break;
        for (int kb = tl.kb0; kb < tl.kb1; ++kb, ++it) {
          const int in_seg = (kb - tl.kb0) % kSplitSegment, s = it % kSplitStages;
          if (!(ok = mbar_wait_cluster(&full_bar[s], (uint32_t)(it / kSplitStages) & 1u, p.timeout))) break;
          tc_fence_after();
          uint8_t* a_s = smem + s * kSplitStageBytes;
          uint64_t wd[3], xd[3];
#pragma unroll
          for (int j = 0; j < 3; ++j) { wd[j] = make_umma_desc_k128(a_s + j * kSplitWPlane); xd[j] = make_umma_desc_k128(a_s + 3 * kSplitWPlane + j * kSplitXPlane); }
          // the small terms first: the sums of the segment before are fetched from their accumulator meanwhile
#pragma unroll
          for (int k = 0; k < kBlockK / 16; ++k) {
            const uint64_t o = (uint64_t)(2 * k);
            umma_bf16_ss_pair(tmem_rest, wd[0] + o, xd[1] + o, idesc, (uint32_t)(((kb - tl.kb0) | k) != 0));
            umma_bf16_ss_pair(tmem_rest, wd[1] + o, xd[0] + o, idesc, 1u);
            umma_bf16_ss_pair(tmem_rest, wd[1] + o, xd[1] + o, idesc, 1u);
            umma_bf16_ss_pair(tmem_rest, wd[0] + o, xd[2] + o, idesc, 1u);
            umma_bf16_ss_pair(tmem_rest, wd[2] + o, xd[0] + o, idesc, 1u);
          }
          if (in_seg == 0) {
            if (!(ok = mbar_wait_cluster(&main_empty, ((uint32_t)sg & 1u) ^ 1u, p.timeout))) break;
            tc_fence_after();
          }
#pragma unroll
          for (int k = 0; k < kBlockK / 16; ++k)
            umma_bf16_ss_pair(tmem_main, wd[0] + (uint64_t)(2 * k), xd[0] + (uint64_t)(2 * k), idesc, (uint32_t)((in_seg | k) != 0));
          umma_commit_pair(&empty_bar[s]);
          if (in_seg == kSplitSegment - 1 || kb + 1 == tl.kb1) { umma_commit_pair(&main_full); ++sg; }
        }
        if (ok) umma_commit_pair(&rest_full);
      }
    }
    __syncwarp();
  } else if (warp < 8) {
    regs_up<232>();
    const int q = warp & 3;
    int nt = 0, sg = 0;
    bool ok = true;
    for (int t; (t = tile_at(nt)) < tiles && ok; ++nt) {
      const Tile tl = tile_of(t);
      float acc[kSplitTokens];
#pragma unroll
      for (int m = 0; m < kSplitTokens; ++m) acc[m] = 0.f;
      auto add = [&](uint32_t src) {
        src += (uint32_t)(q * 32) << 16;
#pragma unroll
        for (int c = 0; c < kSplitTokens / 16; ++c) {
          if (c * 16 < tl.n) {
            uint32_t r[16];
            tmem_ld_32x32b_x16(src + c * 16, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[c * 16 + i] += __uint_as_float(r[i]);
          }
        }
        tc_fence_before();
        __syncwarp();
      };
      const int segs = (tl.kb1 - tl.kb0 + kSplitSegment - 1) / kSplitSegment;
      for (int g = 0; g < segs; ++g, ++sg) {
        if (!(ok = mbar_wait_cluster(&main_full, (uint32_t)sg & 1u, p.timeout))) break;
        tc_fence_after();
        add(tmem_main);
        if (lane == 0) mbar_arrive_cluster(map_shared(&main_empty, 0));
      }
      if (!ok || !(ok = mbar_wait_cluster(&rest_full, (uint32_t)nt & 1u, p.timeout))) break;
      tc_fence_after();
      add(tmem_rest);
      if (lane == 0) mbar_arrive_cluster(map_shared(&rest_empty, 0));
      const int n = tl.col + q * 32 + lane;
      if (n < p.N) {
        float* out = p.out + tl.b * p.c_stride + ((size_t)tl.split * p.M + tl.m0) * p.ldc + n;
        bool again = false;
#pragma unroll
        for (int c = 0; c < kSplitTokens; c += 16) {
          if (c >= tl.rows) break;   // (few rows fetch no more instructions than they need: with those of 192 rows a decoding step took 4 us more per product: kefurax s, 3 layers, 2 sequences 657 us, 473 so)
#pragma unroll
          for (int m = c; m < c + 16; ++m)
            if (m < tl.rows) { out[(size_t)m * p.ldc] = acc[m]; again |= split_again(acc[m]); }
        }
        if (again) s_again = 1;
      }
    }
    __syncwarp();
  } else {
    regs_down<112>();
    // lane: row lane / 8 of four, eight floats from column 8 (lane % 8) of the k-block; four steps cover the warp's 16 rows
    const int r0 = (warp - 8) * 16 + (lane >> 3), piece = lane & 7;
    const float* src[4];   // this thread's four weight rows of the tile whose loads are asked for
    auto rows_of = [&](const Tile& tl) {   // (rows behind the matrix: the last one's, whose results nobody takes)
#pragma unroll
      for (int i = 0; i < 4; ++i) src[i] = p.W + tl.w0 + (long long)min(tl.col + r0 + i * 4, p.N - 1) * p.ldw + piece * 8;
    };
    float4 v[8];
    auto load = [&](int kb, int i) {
      const bool in = kb * kBlockK + piece * 8 < p.K;
      const float4* at = reinterpret_cast<const float4*>(src[i] + kb * kBlockK);
      v[2 * i] = in ? __ldg(at) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[2 * i + 1] = in ? __ldg(at + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    int it = 0, step = 0, t = tile_at(0), kb = 0;
    Tile tl = {};
    if (t < tiles) {
      tl = tile_of(t);
      kb = tl.kb0;
      rows_of(tl);
#pragma unroll
      for (int i = 0; i < 4; ++i) load(kb, i);
    }
    bool ok = true;
    while (t < tiles && ok) {
      int t2 = t, kb2 = kb + 1;   // the k-block after this one
      if (kb2 >= tl.kb1) {
        t2 = tile_at(++step);
        if (t2 < tiles) { tl = tile_of(t2); kb2 = tl.kb0; rows_of(tl); }
      }
      const int s = it % kSplitStages;
      if (!(ok = mbar_wait_cluster(&empty_bar[s], ((uint32_t)(it / kSplitStages) & 1u) ^ 1u, p.timeout))) break;
      uint8_t* a_s = smem + s * kSplitStageBytes;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = r0 + i * 4;
        uint4 h, m, l;
        split3(v[2 * i].x, v[2 * i].y, h.x, m.x, l.x);
        split3(v[2 * i].z, v[2 * i].w, h.y, m.y, l.y);
        split3(v[2 * i + 1].x, v[2 * i + 1].y, h.z, m.z, l.z);
        split3(v[2 * i + 1].z, v[2 * i + 1].w, h.w, m.w, l.w);
        if (t2 < tiles) load(kb2, i);
        uint8_t* dst = a_s + row * 128 + ((piece ^ (row & 7)) << 4);
        *reinterpret_cast<uint4*>(dst) = h;
        *reinterpret_cast<uint4*>(dst + kSplitWPlane) = m;
        *reinterpret_cast<uint4*>(dst + 2 * kSplitWPlane) = l;
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_shared(&full_bar[s], 0));
      ++it; t = t2; kb = kb2;
    }
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (s_again) {   // (nothing waits for this CTA any more but its partner's exit)
    for (int j = 0, t; (t = tile_at(j)) < tiles; ++j) {
      const Tile tl = tile_of(t);
      for (int i = threadIdx.x; i < tl.rows * 128; i += kSplitThreads) {
        const int r = tl.m0 + (i >> 7), n = tl.col + (i & 127);
        if (n >= p.N) continue;
        float* out = p.out + tl.b * p.c_stride + ((size_t)tl.split * p.M + r) * p.ldc + n;
        if (!split_again(*out)) continue;
        const float* x = p.X + tl.b * p.x_stride + (size_t)(p.x_rows ? p.x_rows[r] : r) * p.ldx;
        const float* w = p.W + tl.w0 + (long long)n * p.ldw;
        const int k1 = min(p.K, tl.kb1 * kBlockK);
        float s = 0.f;
        for (int k = tl.kb0 * kBlockK; k < k1; k += 4) {
          const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
          s = fmaf(a.x, b.x, s); s = fmaf(a.y, b.y, s); s = fmaf(a.z, b.z, s); s = fmaf(a.w, b.w, s);
        }
        *out = s;
      }
    }
  }
  cluster_sync_all();
  if (warp == 1) tmem_dealloc_pair(tmem_slot);
}

}  // namespace ssdk
