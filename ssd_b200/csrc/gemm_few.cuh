// gemm_few.cuh — Y[M, N] = X[M, K] · W[N, K]^T for a handful of rows (a decoding step): the weights go from memory straight into the
// operand registers of mma.sync, no shared memory, no barriers and no split-K partials in front of the products.
//
// What bounds it: with M <= 8 every weight is used M times, so the call is a stream of W; in a decoding step of a small model it is a
// chain of such calls of a few microseconds each, bound by what a call has to do after the kernel in front of it is done.  The tile form
// (gemm_ws_kernel) sets up barriers, tensor memory and a TMA ring, splits K over CTAs to fill the machine and leaves the sum to a kernel of its own.
// Here a CTA owns 16 weight rows over all of K, its warps take a share of K each:
//   * m16n8k16 with the weight rows as the 16 (gate and up rows of 8 columns for the gated form) and the tokens as the 8.  The order of k
//     inside a product is free as long as both operands agree, so a thread's 16-byte load of 8 consecutive k of its row IS its part of two
//     A fragments, and the same 8 k of a token its part of the B fragments.
//   * A warp has four units of 64 k in flight (64 bytes a thread each); the first four, which do not depend on the kernel in front, are asked for
//     before the wait for it, the next tile's while the last ones of this tile are multiplied.
//   * The warps' sums meet in shared memory in a fixed order, in fp32 (round to nearest throughout).
//   * The kernel behind starts when this one's CTAs leave: let in earlier (a trigger in front of the wait, or behind it) its CTAs, and those of the
//     kernels behind it, take up room; a step with the 0.6B draft then took 6.34 and 6.39 ms instead of 5.87.
// us alone with cold weights, gemm_ws_kernel with its sum -> this one, M = 4: 1024 x 1024 5.7 -> 3.1, 4096 x 1024 7.0 -> 4.0, 2048 x 2048 7.0 -> 4.1,
// 4096 x 4096 10.7 -> 8.1 (4.2 TB/s), 16384 x 2048 17.1 -> 14.0, gated 2 x 3072 x 1024 8.5 -> 4.8; calls of one token through 4 layers of size s 285 -> 214.
#pragma once
#include "attention.cuh"   // mma_bf16_16816

namespace ssdk {

constexpr int kFewUnit = 64, kFewDepth = 4, kFewWarps = 8, kFewRows = 16, kFewTokens = 8;
enum { FEW_F32 = 0, FEW_BF16 = 1, FEW_SILU = 2, FEW_GLU = 3 };

struct GemmFewParams {
  const __nv_bfloat16* W;   // [N, ldw] (gated: 2 N rows, the up row of column n is row n + N)
  const __nv_bfloat16* X;   // [M, ldx]
  void* out;                // [M, ldo]: fp32 or bf16
  int M, N, K, ldw, ldx, ldo;
  int gelu;                 // FEW_GLU: gelu_tanh instead of silu
  const __nv_bfloat16* ahead[2];   // weights of products behind this one, asked for into L2: ahead_lines of 128 bytes each
  int ahead_lines[2];
  int x_step, out_step;     // products side by side (heads): product b reads X's columns from b x_step, the weight rows from b N, and writes out + b out_step
};

template <int EPI>
__global__ void __launch_bounds__(kFewWarps * 32, 2) gemm_few_kernel(const GemmFewParams p) {
  constexpr bool GATED = EPI == FEW_SILU || EPI == FEW_GLU;
  constexpr int COLS = GATED ? kFewRows / 2 : kFewRows, D = kFewDepth;
  __shared__ float red[2][kFewWarps][4 * 33];   // [value of the fragment][lane]: writes and reads without bank conflicts
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int tiles = (p.N + COLS - 1) / COLS;
  const int units = p.K / kFewUnit, u0 = warp * units / nw, u1 = (warp + 1) * units / nw;
  const __nv_bfloat16 *W = p.W + (size_t)blockIdx.y * p.N * p.ldw, *X = p.X + (size_t)blockIdx.y * p.x_step;
  const bool keep_x = u1 - u0 <= D;   // this warp's part of X stays in its registers

  const __nv_bfloat16 *wa, *wb;       // this thread's two weight rows of a tile
  auto rows_of = [&](int tile) {
    const int r = min(tile * COLS + g, p.N - 1);   // (columns behind N are multiplied and dropped)
    wa = W + (size_t)r * p.ldw + t * 8;
    wb = W + (size_t)(GATED ? r + p.N : min(tile * COLS + g + 8, p.N - 1)) * p.ldw + t * 8;
  };
  uint4 w[D][4], x[D][2];
  auto load_w = [&](uint4* v, int u) {
    v[0] = ld_nc_v4_evict_first(wa + u * kFewUnit);
    v[1] = ld_nc_v4_evict_first(wb + u * kFewUnit);
    v[2] = ld_nc_v4_evict_first(wa + u * kFewUnit + 32);
    v[3] = ld_nc_v4_evict_first(wb + u * kFewUnit + 32);
  };
  auto load_x = [&](uint4* v, int u) {
    const uint4* src = reinterpret_cast<const uint4*>(X + (size_t)g * p.ldx + u * kFewUnit + t * 8);
    v[0] = g < p.M ? src[0] : make_uint4(0u, 0u, 0u, 0u);
    v[1] = g < p.M ? src[4] : make_uint4(0u, 0u, 0u, 0u);
  };

  int tile = blockIdx.x;
  rows_of(tile);
#pragma unroll
  for (int j = 0; j < D; ++j)
    if (u0 + j < u1) load_w(w[j], u0 + j);
  // Never taken (a stride is positive): without a branch here the compiler moves the requests above behind the wait, and the step above takes 6.70 ms instead of 5.87, so that
  // a timing of that step shows whether another compiler still needs it.  (Plain loads that name memory as clobbered stay in front of the wait by themselves, but spill:
  // one token through four layers of a 1B model 363 us instead of 355)
  if (p.ldx < 0) pdl_launch_dependents();
  pdl_wait();
  if (threadIdx.x == 0) trace_mark(TR_GEMM);
#pragma unroll
  for (int a = 0; a < 2; ++a)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < p.ahead_lines[a]; i += gridDim.x * blockDim.x) prefetch_l2(p.ahead[a] + (size_t)i * 64);
#pragma unroll
  for (int j = 0; j < D; ++j)
    if (u0 + j < u1) load_x(x[j], u0 + j);

  for (int buf = 0; tile < tiles; buf ^= 1) {
    const int next = tile + gridDim.x;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int u = u0; u < u1; u += D) {
      const bool last = u + D >= u1;
      if (last && next < tiles) rows_of(next);   // (all that is left to load is the next tile's)
#pragma unroll
      for (int j = 0; j < D; ++j) {
        if (u + j < u1) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint4 a = w[j][2 * h], b = w[j][2 * h + 1];
            const uint32_t f0[4] = {a.x, b.x, a.y, b.y}, f1[4] = {a.z, b.z, a.w, b.w};
            mma_bf16_16816(acc, f0, x[j][h].x, x[j][h].y);
            mma_bf16_16816(acc, f1, x[j][h].z, x[j][h].w);
          }
        }
        const int v = last ? u0 + j : u + D + j;
        if (v < u1 && (!last || next < tiles)) {
          load_w(w[j], v);
          if (!keep_x) load_x(x[j], v);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) red[buf][warp][c * 33 + lane] = acc[c];
    __syncthreads();   // (the other buffer is written next: whoever still reads this one is a barrier behind)
    for (int i = threadIdx.x; i < COLS * kFewTokens; i += blockDim.x) {
      const int col = i % COLS, m = i / COLS, n = tile * COLS + col;
      if (m >= p.M || n >= p.N) continue;
      const float* src = &red[buf][0][(m & 1) * 33 + (col & 7) * 4 + (m >> 1)];   // fragment value: 2 (row / 8) + token & 1
      const int up = 2 * 33;
      float s = 0.f, s2 = 0.f;
      if (GATED) {
        for (int q = 0; q < nw; ++q) { s += src[q * 132]; s2 += src[q * 132 + up]; }
      } else {
        if (col >= 8) src += up;
        for (int q = 0; q < nw; ++q) s += src[q * 132];
      }
      const size_t at = (size_t)m * p.ldo + (size_t)blockIdx.y * p.out_step + n;
      if (EPI == FEW_F32) {
        reinterpret_cast<float*>(p.out)[at] = s;
      } else if (EPI == FEW_BF16) {
        reinterpret_cast<__nv_bfloat16*>(p.out)[at] = f2bf(s);
      } else if (EPI == FEW_SILU) {   // the dense decoders' linear layers return bf16
        const float a = bf16_round(s), b = bf16_round(s2);
        reinterpret_cast<__nv_bfloat16*>(p.out)[at] = f2bf((a / (1.0f + __expf(-a))) * b);
      } else {
        const float a = p.gelu ? 0.5f * s * (1.0f + tanhf(0.7978845608028654f * (s + 0.044715f * s * s * s))) : s / (1.0f + expf(-s));
        reinterpret_cast<__nv_bfloat16*>(p.out)[at] = f2bf(a * s2);
      }
    }
    tile = next;
  }
}

}  // namespace ssdk
