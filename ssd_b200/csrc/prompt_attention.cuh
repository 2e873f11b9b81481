// prompt_attention.cuh — causal attention of a prompt pass over the paged KV cache on tcgen05.
//
// A CTA owns one kv head and a tile of 128 rows: 128 / G query tokens x the G query heads that share the kv head, so a key is loaded once
// for all of them.  Chunks of 64 keys stream through two stages by TMA (a chunk lies in one page).  Per chunk:
//   S = Q K^T      128 x 64, both operands K-major in shared memory, fp32 in TMEM (two buffers: the next chunk's is computed under the softmax)
//   P = exp2(S - m) one row per thread, no shuffles; rounded to bf16 and stored over the S it came from
//   O += P V       P from TMEM, V as it lies in the cache (MN-major operand), fp32 in TMEM
// m is raised, and O and the sum rescaled, only when a row's maximum has grown by more than kPromptSlack (base 2): P then stays below
// 2^kPromptSlack, where bf16 and fp32 are as fine relative to a value as below 1.  But a row's largest weight is no longer exactly 1, and is rounded like all others;
// paged_attn_kernel follows the maximum of every token slice and rounds none of those.  The calls that this kernel takes over from it therefore give P
// as two bf16 pieces, 16 significant bits, which both meet V.  Relative error of a 70B layer's attention against 64 bits, 8 x 7 rows of contexts of 4500
// to 8000 / 4 x 8 of 1880 to 3000 / 2 x 8 of 220 to 300: 0.00275, 0.00268, 0.00252 in paged_attn_kernel, 0.00289, 0.00286, 0.00264 with one piece, 0.00237,
// 0.00237, 0.0023 with two.  The softmax hardly notices; what costs is a second product per chunk (the first: 60 -> 67 us, 109 in paged_attn_kernel).  Calls of up to 64 rows
// and long tables load their queries twice: rows 64 .. 127 are the same rows again, give the low pieces and add up in accumulator lanes of their own, so that one product
// takes both, and the warps that would idle do the work (62 us).
// Warps: 0 loads, 1 issues the products, 2-5 softmax and output.  Two CTAs per SM (97 KB, 256 TMEM columns each), so that one's products
// run under the other's exponentials, which bound the kernel.
// 2003 tokens, 32 heads of 128 over 8: 205 us on mma.sync tiles of 64 rows (paged_attn_kernel), 47 us here = 700 TFLOP/s of the masked work;
// 8B widths, 4 layers: 4779 -> 4143 us a prompt.  Tensor pipe active 30 % of the time, issue slots 41 %.
#pragma once
#include "gemm_pair.cuh"

namespace ssdk {

constexpr int kPromptRows = 128, kPromptKeys = 64, kPromptStages = 2, kPromptThreads = 192;
constexpr float kPromptSlack = 8.f;
constexpr int prompt_attn_smem(int HD) { return kPromptRows * HD * 2 + kPromptStages * 2 * kPromptKeys * HD * 2 + 1024; }

struct PromptAttnParams {
  const int32_t* block_tables;   // [B, max_blocks]
  const int32_t* context_lens;   // [B], includes the Q new tokens
  __nv_bfloat16* out;            // [B*Q, H, hd]
  int Q, H, KV, g_shift;         // H / KV = 1 << g_shift <= 16
  int block_size, max_blocks;    // block_size a multiple of kPromptKeys
  int n_slots;                   // token slots of the cache: a chunk without a page is loaded from behind them (zeros)
  float scale_log2;              // > 0
  unsigned* timeout;             // (rows whose waits ran out are NaN)
  // SPLIT: the keys of a sequence in n_split ranges of whole chunks, as paged_attn_kernel cuts them; what a range gives goes to
  // part_o [B*Q*H, n_split, hd] and part_lse [B*Q*H, n_split] (fp32, see attn_combine_kernel)
  int n_split;
  float* part_o;
  float* part_lse;
};

// a whole warp's bounded wait: all of it goes on, or none
SSDK_DEVINL bool warp_wait(uint64_t* bar, uint32_t parity, unsigned* timeout) {
  return __all_sync(0xffffffffu, mbar_wait_cluster(bar, parity, timeout));
}
SSDK_DEVINL void tma_load_3d(void* smem_dst, const void* tmap, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// A from TMEM (a lane per row, two bf16 of K per column), B from shared memory
SSDK_DEVINL void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
SSDK_DEVINL void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
SSDK_DEVINL void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// largest of a row's 64 scores
SSDK_DEVINL float row_max(const uint32_t (&u)[64]) {
  float m[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) m[c] = max3(__uint_as_float(u[c]), __uint_as_float(u[c + 4]), __uint_as_float(u[c + 8]));
#pragma unroll
  for (int c = 12; c < 60; c += 8)
#pragma unroll
    for (int e = 0; e < 4; ++e) m[e] = max3(m[e], __uint_as_float(u[c + e]), __uint_as_float(u[c + 4 + e]));
  return fmaxf(max3(m[0], m[1], __uint_as_float(u[60])), max3(m[2], m[3], max3(__uint_as_float(u[61]), __uint_as_float(u[62]), __uint_as_float(u[63]))));
}
// Weights of a product with V: one bf16 piece; two, side by side in the columns of their scores; two, in rows of their own
enum { kPromptOne = 0, kPromptTwo = 1, kPromptTwin = 2 };

// 2^(score * scale - ms) of a row, and their sum (of the unrounded ones) back.  HIGH: rounded to bf16 in the first 32 words; LOW: what that leaves, rounded, in the
// others (without HIGH in the first).  Products and sums two at a time; a probability below 2^-126 is zero (the row's largest is at least 2^-kPromptSlack).
template <bool HIGH, bool LOW>
SSDK_DEVINL float row_exp(uint32_t (&u)[64], float scale, float ms) {
  const uint64_t sc = pack2(scale, scale), off = pack2(-ms, -ms), minus = pack2(-1.f, -1.f);
  uint64_t sum[2] = {0, 0};
  uint32_t low[32];
#pragma unroll
  for (int c = 0; c < 64; c += 2) {
    float a, e;
    unpack2(fma2(pack2(__uint_as_float(u[c]), __uint_as_float(u[c + 1])), sc, off), &a, &e);
    a = ex2_ftz(a); e = ex2_ftz(e);
    sum[(c >> 1) & 1] = add2(sum[(c >> 1) & 1], pack2(a, e));
    const uint32_t h = pack_bf16x2(a, e);
    if (HIGH) u[c >> 1] = h;
    if (LOW) {   // (exact differences)
      float x, y;
      unpack2(fma2(pack2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u)), minus, pack2(a, e)), &x, &y);
      (HIGH ? low : u)[c >> 1] = pack_bf16x2(x, y);
    }
  }
  if (HIGH && LOW) {
#pragma unroll
    for (int c = 0; c < 32; ++c) u[32 + c] = low[c];
  }
  float s0, s1, s2, s3;
  unpack2(sum[0], &s0, &s1);
  unpack2(sum[1], &s2, &s3);
  return (s0 + s1) + (s2 + s3);
}

// grid (kv heads, q tiles, sequences x ranges).  P: kPromptTwin takes tiles of up to 64 rows (their map's boxes hold as many)
template <int HD, bool SPLIT, int P>
__global__ void __launch_bounds__(kPromptThreads, 2)
prompt_attn_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                   const PromptAttnParams p) {
  constexpr int HALVES = HD / 64;                    // 64-column boxes of a row
  constexpr int kQHalf = kPromptRows * 128, kKHalf = kPromptKeys * 128, kTile = HALVES * kKHalf;
  extern __shared__ uint8_t prompt_smem_raw[];
  __shared__ __align__(8) uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], pv_done[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_failed;   // TWIN: a wait of the low pieces' warps ran out
  uint8_t* smem = prompt_smem_raw + ((1024u - (smem_u32(prompt_smem_raw) & 1023u)) & 1023u);
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + HALVES * kQHalf;
  uint8_t* sV = sK + kPromptStages * kTile;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = blockIdx.x, qt = (int)gridDim.y - 1 - (int)blockIdx.y;   // (the tiles that see most keys first)
  const int b = SPLIT ? (int)blockIdx.z / p.n_split : (int)blockIdx.z, split = SPLIT ? (int)blockIdx.z - b * p.n_split : 0;
  constexpr bool TWIN = P == kPromptTwin;
  constexpr int ROWS = TWIN ? kPromptRows / 2 : kPromptRows;
  const int G = 1 << p.g_shift, TQ = ROWS >> p.g_shift;
  const int tok0 = qt * TQ, tq = min(TQ, p.Q - tok0);
  const int half = ((tq << p.g_shift) + 31) & ~31;                       // rows of the warps that have some
  const int live = TWIN ? 2 * half : SPLIT ? half : kPromptRows;         // threads that hand P over

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    mbar_init(&q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1);
      mbar_init(&s_full[s], 1); mbar_init(&p_full[s], live); mbar_init(&pv_done[s], 1);
    }
    fence_mbar_init();
    s_failed = 0;
  }
  if (warp == 1) { tmem_alloc(&tmem_slot, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot, tmem_o = tmem + 128;   // S / P buffers at columns 0 and 64, O behind them

  pdl_launch_dependents();
  pdl_wait();

  const int ctx0 = p.context_lens[b] - p.Q;
  const int kv_max = ctx0 + tok0 + tq;               // exclusive upper bound of the keys the tile sees
  int n = (kv_max + kPromptKeys - 1) / kPromptKeys, first = 0;   // chunks of this CTA, and the first key of the first one
  if (SPLIT) {   // (a range without chunks leaves no partial: the merge reads those that have some)
    const int per = (n + p.n_split - 1) / p.n_split;
    first = split * per * kPromptKeys;
    n = max(0, min(per, n - split * per));
  }
  // Every pair of barriers is used in turn, chunk i on barrier i & 1; parity(i) is that use's.  A wait by parity is only right while the barrier
  // is in that use or the one behind it.  pv_done: whoever waits for chunk j has seen s_full of chunk j + 1 or later (or issued its
  // scores), which was committed behind the product of chunk j - 1, and the product of chunk j + 2 needs the P that this thread (or this
  // warp's rows) has not handed over yet.  (One barrier for all chunks could run a phase ahead of a softmax warp that is held up between
  // handing P over and asking: the wait then never ended.)
  auto parity = [](int i) { return (uint32_t)(i >> 1) & 1u; };

  if (warp == 0) {
    if (lane == 0 && n > 0) {
      mbar_arrive_expect_tx(&q_full, HALVES * kQHalf);
      for (int h = 0; h < HALVES; ++h)
        for (int r = 0; r < kPromptRows; r += ROWS) tma_load_3d(sQ + h * kQHalf + r * 128, &tmQ, &q_full, h * 64, kvh << p.g_shift, b * p.Q + tok0);
      const int32_t* bt = p.block_tables + (size_t)b * p.max_blocks;
      int i = 0;
      for (; i < n; ++i) {
        const int s = i & 1, base = first + i * kPromptKeys;
        const int blk = bt[base / p.block_size];
        const int slot = blk >= 0 ? blk * p.block_size + base % p.block_size : p.n_slots;
        if (!mbar_wait_cluster(&k_empty[s], parity(i) ^ 1u, p.timeout)) break;
        mbar_arrive_expect_tx(&k_full[s], kTile);
        for (int h = 0; h < HALVES; ++h) tma_load_3d(sK + s * kTile + h * kKHalf, &tmK, &k_full[s], h * 64, kvh, slot);
        if (!mbar_wait_cluster(&v_empty[s], parity(i) ^ 1u, p.timeout)) { mbar_wait_cluster(&k_full[s], parity(i), p.timeout); break; }
        mbar_arrive_expect_tx(&v_full[s], kTile);
        for (int h = 0; h < HALVES; ++h) tma_load_3d(sV + s * kTile + h * kKHalf, &tmV, &v_full[s], h * 64, kvh, slot);
      }
      // nothing is in flight into this CTA's memory when it leaves, also after a wait ran out
      mbar_wait_cluster(&q_full, 0, p.timeout);
      for (int j = max(0, i - 2); j < i; ++j) {
        mbar_wait_cluster(&k_full[j & 1], parity(j), p.timeout);
        mbar_wait_cluster(&v_full[j & 1], parity(j), p.timeout);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_umma_idesc_bf16(kPromptRows, kPromptKeys);
      constexpr uint32_t idesc_o = make_umma_idesc_bf16(kPromptRows, HD) | (1u << 16);   // V: b_major = MN
      auto scores = [&](int i) {
        if (!mbar_wait_cluster(&k_full[i & 1], parity(i), p.timeout)) return false;
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < HALVES; ++h) {
          const uint64_t qd = make_umma_desc_k128(sQ + h * kQHalf), kd = make_umma_desc_k128(sK + (i & 1) * kTile + h * kKHalf);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_ss(tmem + (i & 1) * 64, qd + 2 * k, kd + 2 * k, idesc_s, (uint32_t)((h | k) != 0));
        }
        umma_commit(&k_empty[i & 1]);
        umma_commit(&s_full[i & 1]);
        return true;
      };
      bool ok = n > 0 && mbar_wait_cluster(&q_full, 0, p.timeout) && scores(0);
      for (int i = 0; i < n && ok; ++i) {
        // the scores of chunk i + 1 go over the P that the product of chunk i - 1 reads: products of different shapes and accumulators
        // have no order of their own
        if (i > 0 && !(ok = mbar_wait_cluster(&pv_done[(i - 1) & 1], parity(i - 1), p.timeout))) break;
        if (i + 1 < n && !(ok = scores(i + 1))) break;
        if (!(ok = mbar_wait_cluster(&p_full[i & 1], parity(i), p.timeout) && mbar_wait_cluster(&v_full[i & 1], parity(i), p.timeout))) break;
        tc_fence_after();
        const uint64_t vd = make_umma_desc_mn128(sV + (i & 1) * kTile, kKHalf);
#pragma unroll
        for (int k = 0; k < kPromptKeys / 16; ++k)   // 16 keys: 2048 B of V, 8 columns of P
          umma_bf16_ts(tmem_o, tmem + (i & 1) * 64 + 8 * k, vd + 128 * k, idesc_o, (uint32_t)((i | k) != 0));
        if (P == kPromptTwo) {
#pragma unroll
          for (int k = 0; k < kPromptKeys / 16; ++k) umma_bf16_ts(tmem_o, tmem + (i & 1) * 64 + 32 + 8 * k, vd + 128 * k, idesc_o, 1u);
        }
        umma_commit(&v_empty[i & 1]);
        umma_commit(&pv_done[i & 1]);
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3, r = TWIN ? (q & 1) * 32 + lane : q * 32 + lane, tok = r >> p.g_shift;
    const bool low = TWIN && q >= 2;   // (the whole warp) the same row as two warps before, its low pieces
    const uint32_t lanes = (uint32_t)(q * 32) << 16;
    const int lim = min(ctx0 + tok0 + tok + 1, kv_max);   // keys this row sees (rows behind the tile's tokens: some, dropped)
    float m = -INFINITY, l = 0.f;
    const bool in = !(SPLIT || TWIN) || (r & ~31) < half;   // (a warp without rows: what the products make of its lanes, nobody reads)
    bool ok = in;
    for (int i = 0; i < n && in; ++i) {
      const int base = first + i * kPromptKeys;
      const uint32_t sp = tmem + lanes + (uint32_t)(i & 1) * 64u;
      if (!(ok = warp_wait(&s_full[i & 1], parity(i), p.timeout))) break;
      tc_fence_after();
      uint32_t u[64];
#pragma unroll
      for (int c = 0; c < 64; c += 16) tmem_ld_32x32b_x16(sp + c, u + c);
      tmem_ld_wait();
      if (base + kPromptKeys > lim) {
#pragma unroll
        for (int c = 0; c < 64; ++c)
          if (base + c >= lim) u[c] = 0xff800000u;   // -inf
      }
      const float mx = row_max(u) * p.scale_log2;
      const bool grow = mx > m + kPromptSlack;
      if (__any_sync(0xffffffffu, grow)) {
        const float f = grow ? exp2f(m - mx) : 1.f;   // (m = -inf: 0)
        if (grow) m = mx;
        l *= f;
        if (i > 0) {
          if (!(ok = warp_wait(&pv_done[(i - 1) & 1], parity(i - 1), p.timeout))) break;
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < HD; c += 16) {
            uint32_t o[16];
            tmem_ld_32x32b_x16(tmem_o + lanes + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
            tmem_st_32x32b_x16(tmem_o + lanes + c, o);
          }
        }
      }
      const float ms = m == -INFINITY ? 0.f : m;
      l += low ? row_exp<false, true>(u, p.scale_log2, ms) : row_exp<true, P == kPromptTwo>(u, p.scale_log2, ms);
#pragma unroll
      for (int c = 0; c < (P == kPromptTwo ? 64 : 32); c += 16) tmem_st_32x32b_x16(sp + c, u + c);
      tmem_st_wait();
      if (base + kPromptKeys > kv_max) {   // the last chunk: slots behind the tile's keys hold anything, and 0 x NaN is NaN
        if (!(ok = warp_wait(&v_full[i & 1], parity(i), p.timeout))) break;
        const int from = kv_max - base, pieces = (kPromptKeys - from) * 8;   // 16-byte pieces per half (a row's stay in its 128 bytes)
        for (int h = 0; h < HALVES; ++h)
          for (int j = low ? half + r : r; j < pieces; j += live)
            *reinterpret_cast<uint4*>(sV + (i & 1) * kTile + h * kKHalf + from * 128 + j * 16) = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async_smem();
      }
      tc_fence_before();
      mbar_arrive(&p_full[i & 1]);
    }
    if (ok && n > 0) ok = warp_wait(&pv_done[(n - 1) & 1], parity(n - 1), p.timeout);
    tc_fence_after();
    constexpr int LDO = HD + 4;
    float* o2 = reinterpret_cast<float*>(sK) + (size_t)(r & (ROWS - 1)) * LDO;   // (the stages: every product has read them)
    if (TWIN && n > 0 && in) {   // what the low pieces gave goes to the warps of the high ones
      if (low && !ok) s_failed = 1;
      if (low && ok) {
        for (int c = 0; c < HD; c += 16) {
          uint32_t o[16];
          tmem_ld_32x32b_x16(tmem_o + lanes + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; j += 4) *reinterpret_cast<uint4*>(o2 + c + j) = make_uint4(o[j], o[j + 1], o[j + 2], o[j + 3]);
        }
      }
      asm volatile("bar.sync 1, %0;" ::"r"(live) : "memory");
      ok = ok && !*(volatile int*)&s_failed;
    }
    auto sums = [&](int c, float (&f)[16]) {   // 16 columns of this row
      uint32_t o[16];
      tmem_ld_32x32b_x16(tmem_o + lanes + c, o);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) f[j] = __uint_as_float(o[j]);
      if (TWIN && n > 0) {
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          const float4 x = *reinterpret_cast<const float4*>(o2 + c + j);
          f[j] += x.x; f[j + 1] += x.y; f[j + 2] += x.z; f[j + 3] += x.w;
        }
      }
    };
    const float inv = !ok ? __int_as_float(0x7fffffff) : l > 0.f ? 1.f / l : 0.f;   // NaN: a wait ran out
    const bool mine = in && !low && tok < tq;
    const size_t row = (size_t)(b * p.Q + tok0 + tok) * p.H + (kvh << p.g_shift) + (r & (G - 1));
    if (SPLIT) {
      if (n > 0 && in && !low) {
        float* dst = p.part_o + (row * p.n_split + split) * HD;
#pragma unroll 2
        for (int c = 0; c < HD; c += 16) {
          float f[16];
          sums(c, f);
          if (mine) {
#pragma unroll
            for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(dst + c + j) = make_float4(f[j] * inv, f[j + 1] * inv, f[j + 2] * inv, f[j + 3] * inv);
          }
        }
        if (mine) p.part_lse[row * p.n_split + split] = l > 0.f ? m + log2f(l) : -INFINITY;
      }
    } else if (!low) {
      __nv_bfloat16* dst = p.out + row * HD;
#pragma unroll 2
      for (int c = 0; c < HD; c += 16) {
        float f[16];
        sums(c, f);
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = n <= 0 ? 0u : pack_bf16x2(f[2 * j] * inv, f[2 * j + 1] * inv);
        if (mine) {
          *reinterpret_cast<uint4*>(dst + c) = make_uint4(w[0], w[1], w[2], w[3]);
          *reinterpret_cast<uint4*>(dst + c + 8) = make_uint4(w[4], w[5], w[6], w[7]);
        }
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem, 256);
}

}  // namespace ssdk
