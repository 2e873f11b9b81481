// gqa_prompt.cuh — prompt portions of grouped-query attention over the layered models' page pool on tcgen05 (bf16 storage): windows, kept first
// keys, sinks, output gates, and the two maps of differential attention.
//
// The pipeline is prompt_attn_kernel's: a CTA owns 128 (map, query, head) rows of one key/value head, chunks of 64 keys (of one page) stream through two
// stages by TMA, S = Q K^T and O += P V on the tensor core with S, P and O in TMEM, one row of the softmax per thread, O rescaled only when a row's
// maximum has grown by more than kPromptSlack.  What is different:
//   * the chunks that a mask leaves: those of the kept keys, then from the one that holds the tile's first visible key on; a chunk that every key
//     of is visible to a row costs that row no comparisons;
//   * two maps (DK = 128, keys of 64): rows 0 .. 63 are the first map's queries in columns 0 .. 63 of the operand, rows 64 .. 127 the second's in
//     columns 64 .. 127, zeros elsewhere.  One product against the two maps' keys, side by side in the page row, then gives both, and both meet one
//     copy of the values; the maps are joined through shared memory and leave as normed heads.
// What bounds it: the exponentials (one row of 64 per thread and chunk) under the products of the other CTA of the SM.
#pragma once
#include "gqa_attention.cuh"
#include "prompt_attention.cuh"

namespace ssdk {

constexpr int gqa_prompt_smem(int DK, int VD) { return kPromptRows * DK * 2 + kPromptStages * kPromptKeys * (DK + VD) * 2 + 1024; }

struct GqaPromptArgs {
  void* y;            // [M, H V] bf16 (two maps: [M, H / 2 V])
  const float* gate;  // pre-activations of a sigmoid gate, gate[m * ld_gate + h V + v], or nullptr
  int ld_gate;
  int G, D, g_shift;  // keys (of all maps) per token and their size, H / G = 1 << g_shift <= 16
  float scale_log2, sink;
  const void* sinks;  // [H] bf16 learned sink logits (they replace the constant), or nullptr
  KeyMask mask;
  DiffArgs diff;      // MAPS = 2
  int key_rot, query_rot, query_ld;   // LATENT: columns of the rotated parts (of a head's keys, which all heads share, and of a query) and of a query row
  unsigned* timeout;
};

// LATENT: latent attention over whole prompts with keys and values of every head made first (one query per key head, G heads): DK - 64 columns of keys and
// queries in [M, G (DK - 64)] each, 64 rotated ones that all heads' keys share, values [M, G VD]; rows by their place in the call, no pages.
// Prompts of 1000, 831 and 664 tokens, 16 heads of 128 over latents of 512: gathers, score products, softmax and P C one sequence after the other 245 us, with the
// absorption and the value projection 298; 125 in this form (keys and values 30, rows 6, attention 90).  The whole call 852 -> 707 us.
struct GqaLatentMaps {
  CUtensorMap q_rot, k_rot, v;
};

// grid (row tiles of the longest portion, G / MAPS, n_seqs)
template <int DK, int VD, int MAPS, bool LATENT>
__global__ void __launch_bounds__(kPromptThreads, 2)
gqa_prompt_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV, const __grid_constant__ GqaLatentMaps lm, const GqaPromptArgs p,
                  const Ragged rg) {
  constexpr int HK = DK / 64, HV = VD / 64, R = kPromptRows / MAPS;   // 64-column boxes of keys and values, rows of a map
  // Weights as two bf16 pieces (see prompt_attention.cuh): the tiles that this form took over from keep the largest weights of their slices unrounded.  vegilix m,
  // prompts of 2001 and 2 x 700 tokens against 64 bits: 0.00338, 0.00328 with one piece, 0.00324, 0.00313 with two; 518 -> 523 us.  Latent attention: the absorbed form that
  // whole prompts took before rounds its weights once as well
  constexpr bool FINE = !LATENT;
  constexpr int kQHalf = kPromptRows * 128, kHalf = kPromptKeys * 128;
  static_assert(MAPS == 1 || (DK == 128 && !LATENT), "two maps of 64");
  extern __shared__ uint8_t prompt_smem_raw[];
  __shared__ __align__(8) uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], pv_done[2];
  __shared__ uint32_t tmem_slot;
  uint8_t* smem = prompt_smem_raw + ((1024u - (smem_u32(prompt_smem_raw) & 1023u)) & 1023u);
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + HK * kQHalf;
  uint8_t* sV = sK + kPromptStages * HK * kHalf;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // (in front of the trigger: a product that this kernel lets start early finds its tensor memory taken, and not the other way round)
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmKV);
    if (LATENT) { tma_prefetch_desc(&lm.q_rot); tma_prefetch_desc(&lm.k_rot); tma_prefetch_desc(&lm.v); }
    mbar_init(&q_full, MAPS == 1 ? 1 : 1 + kPromptRows);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&k_full[b], 1); mbar_init(&k_empty[b], 1); mbar_init(&v_full[b], 1); mbar_init(&v_empty[b], 1);
      mbar_init(&s_full[b], 1); mbar_init(&p_full[b], kPromptRows); mbar_init(&pv_done[b], 1);
    }
    fence_mbar_init();
  }
  if (warp == 1) { tmem_alloc(&tmem_slot, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot, tmem_o = tmem + 128;   // S / P buffers at columns 0 and 64, O behind them

  pdl_launch_dependents();
  pdl_wait();
  const int gv = blockIdx.y, s = blockIdx.z, r0 = rg.cu[s], p0 = rg.pos0[s], shift = p.g_shift;
  const int rows = (rg.cu[s + 1] - r0) << shift, row0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * R;   // (the tiles that see most keys first)
  if (rows < 2 << shift || row0 >= rows) {   // (the whole CTA)
    if (warp == 1) tmem_dealloc(tmem, 256);
    return;
  }

  // keys that the tile's rows see together: those below `keep`, and first .. k_end - 1
  const int first = p.mask.first(p0 + (row0 >> shift)), keep = p.mask.kept(first), k_end = p0 + ((min(rows, row0 + R) - 1) >> shift) + 1;
  const int fc = first / kPromptKeys, kc = min((keep + kPromptKeys - 1) / kPromptKeys, fc), n = kc + (k_end + kPromptKeys - 1) / kPromptKeys - fc;
  auto base_of = [&](int i) { return (i < kc ? i : fc + i - kc) * kPromptKeys; };
  auto parity = [](int i) { return (uint32_t)(i >> 1) & 1u; };   // (see prompt_attn_kernel)

  if (warp == 0) {
    if (lane == 0) {
      mbar_arrive_expect_tx(&q_full, MAPS == 1 ? HK * kQHalf : kQHalf);
      const int q_row = ((gv * MAPS * rg.M + r0) << shift) + row0;
      if (LATENT) {
        const int row = r0 + row0;
        for (int h = 0; h < HK - 1; ++h) tma_load_2d(sQ + h * kQHalf, &tmQ, &q_full, gv * (DK - 64) + h * 64, row, kEvictNormal);
        tma_load_2d(sQ + (HK - 1) * kQHalf, &lm.q_rot, &q_full, gv * p.query_ld + p.query_rot, row, kEvictNormal);
      } else if (MAPS == 1) {
        for (int h = 0; h < HK; ++h) tma_load_2d(sQ + h * kQHalf, &tmQ, &q_full, h * 64, q_row, kEvictNormal);
      } else {
        tma_load_2d(sQ, &tmQ, &q_full, 0, q_row, kEvictNormal);
        tma_load_2d(sQ + kQHalf + R * 128, &tmQ, &q_full, 0, q_row + (rg.M << shift), kEvictNormal);
      }
      const int k_col = gv * (LATENT ? DK - 64 : DK), v_col = (LATENT ? 0 : p.G * p.D) + gv * VD;
      const int* table = rg.tables + (size_t)s * rg.max_blocks;
      int i = 0;
      for (; i < n; ++i) {
        const int b = i & 1, base = base_of(i), slot = LATENT ? r0 + base : table[base / rg.block_size] * rg.block_size + base % rg.block_size;
        if (!mbar_wait_cluster(&k_empty[b], parity(i) ^ 1u, p.timeout)) break;
        mbar_arrive_expect_tx(&k_full[b], HK * kHalf);
        for (int h = 0; h < HK; ++h) {
          if (LATENT && h == HK - 1) tma_load_2d(sK + (b * HK + h) * kHalf, &lm.k_rot, &k_full[b], p.key_rot, slot, kEvictNormal);
          else tma_load_2d(sK + (b * HK + h) * kHalf, &tmKV, &k_full[b], k_col + h * 64, slot, kEvictNormal);
        }
        if (!mbar_wait_cluster(&v_empty[b], parity(i) ^ 1u, p.timeout)) { mbar_wait_cluster(&k_full[b], parity(i), p.timeout); break; }
        mbar_arrive_expect_tx(&v_full[b], HV * kHalf);
        for (int h = 0; h < HV; ++h) tma_load_2d(sV + (b * HV + h) * kHalf, LATENT ? &lm.v : &tmKV, &v_full[b], v_col + h * 64, slot, kEvictNormal);
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
      constexpr uint32_t idesc_o = make_umma_idesc_bf16(kPromptRows, VD) | (1u << 16);   // V: b_major = MN
      auto scores = [&](int i) {
        if (!mbar_wait_cluster(&k_full[i & 1], parity(i), p.timeout)) return false;
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < HK; ++h) {
          const uint64_t qd = make_umma_desc_k128(sQ + h * kQHalf), kd = make_umma_desc_k128(sK + ((i & 1) * HK + h) * kHalf);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_ss(tmem + (i & 1) * 64, qd + 2 * k, kd + 2 * k, idesc_s, (uint32_t)((h | k) != 0));
        }
        umma_commit(&k_empty[i & 1]);
        umma_commit(&s_full[i & 1]);
        return true;
      };
      bool ok = mbar_wait_cluster(&q_full, 0, p.timeout) && scores(0);
      for (int i = 0; i < n && ok; ++i) {
        // (the scores of chunk i + 1 go over the P that the product of chunk i - 1 reads)
        if (i > 0 && !(ok = mbar_wait_cluster(&pv_done[(i - 1) & 1], parity(i - 1), p.timeout))) break;
        if (i + 1 < n && !(ok = scores(i + 1))) break;
        if (!(ok = mbar_wait_cluster(&p_full[i & 1], parity(i), p.timeout) && mbar_wait_cluster(&v_full[i & 1], parity(i), p.timeout))) break;
        tc_fence_after();
        const uint64_t vd = make_umma_desc_mn128(sV + (i & 1) * HV * kHalf, kHalf);
#pragma unroll
        for (int k = 0; k < kPromptKeys / 16; ++k)   // 16 keys: 2048 B of V, 8 columns of P
          umma_bf16_ts(tmem_o, tmem + (i & 1) * 64 + 8 * k, vd + 128 * k, idesc_o, (uint32_t)((i | k) != 0));
        if (FINE) {
#pragma unroll
          for (int k = 0; k < kPromptKeys / 16; ++k) umma_bf16_ts(tmem_o, tmem + (i & 1) * 64 + 32 + 8 * k, vd + 128 * k, idesc_o, 1u);
        }
        umma_commit(&v_empty[i & 1]);
        umma_commit(&pv_done[i & 1]);
      }
    }
    __syncwarp();
  } else {
    typedef __nv_bfloat16 T;
    const int q = warp & 3, r = q * 32 + lane, map = r / R, row = row0 + r % R, tok = row >> shift;   // (row: behind the portion, dropped)
    const uint32_t lanes = (uint32_t)(q * 32) << 16;
    if (MAPS == 2) {   // the blocks of the operand that hold no queries
      for (int j = r; j < 2 * R * 8; j += kPromptRows) {
        const int h = j / (R * 8), at = j % (R * 8);
        *reinterpret_cast<uint4*>(sQ + h * kQHalf + (1 - h) * R * 128 + at * 16) = make_uint4(0u, 0u, 0u, 0u);
      }
      fence_proxy_async_smem();
      mbar_arrive(&q_full);
    }
    const int hi = min(p0 + tok, k_end - 1), lo = p.mask.first(hi);   // the row sees keys lo .. hi and those below the mask's `keep`
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int i = 0; i < n; ++i) {
      const int base = base_of(i);
      const uint32_t sp = tmem + lanes + (uint32_t)(i & 1) * 64u;
      if (!(ok = warp_wait(&s_full[i & 1], parity(i), p.timeout))) break;
      tc_fence_after();
      uint32_t u[64];
#pragma unroll
      for (int c = 0; c < 64; c += 16) tmem_ld_32x32b_x16(sp + c, u + c);
      tmem_ld_wait();
      if (base + kPromptKeys - 1 > hi || (base < lo && base + kPromptKeys > p.mask.keep)) {
#pragma unroll
        for (int c = 0; c < 64; ++c)
          if (base + c > hi || (base + c < lo && base + c >= p.mask.keep)) u[c] = 0xff800000u;   // -inf
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
          for (int c = 0; c < VD; c += 16) {
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
      l += row_exp<true, FINE>(u, p.scale_log2, ms);
#pragma unroll
      for (int c = 0; c < (FINE ? 64 : 32); c += 16) tmem_st_32x32b_x16(sp + c, u + c);
      tmem_st_wait();
      // values that no row of the tile sees may be anything, and 0 x NaN is NaN: those between the kept keys and the first one, those behind the last
      const int gap0 = min(max(keep - base, 0), kPromptKeys), gap1 = min(max(first - base, gap0), kPromptKeys), end = min(k_end - base, kPromptKeys);
      if (gap1 > gap0 || end < kPromptKeys) {
        if (!(ok = warp_wait(&v_full[i & 1], parity(i), p.timeout))) break;
        for (int j = r; j < kPromptKeys * 8; j += kPromptRows) {   // 16-byte pieces per half (a row's stay in its 128 bytes)
          const int key = j >> 3;
          if ((key >= gap0 && key < gap1) || key >= end)
            for (int h = 0; h < HV; ++h) *reinterpret_cast<uint4*>(sV + ((i & 1) * HV + h) * kHalf + j * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_proxy_async_smem();
      }
      tc_fence_before();
      mbar_arrive(&p_full[i & 1]);
    }
    if (ok) ok = warp_wait(&pv_done[(n - 1) & 1], parity(n - 1), p.timeout);
    tc_fence_after();
    if (MAPS == 1) {
      const int head = (gv << shift) + (row & ((1 << shift) - 1)), at = r0 + tok;
      if (ok) {
        if (p.sinks) l += exp2f(ld_f<T>((const T*)p.sinks + head) * 1.4426950408889634f - m);
        else if (p.sink > 0.f) l += p.sink * exp2f(-m);
        const float inv = 1.0f / l;
        const bool mine = row < rows;
        T* dst = (T*)p.y + ((size_t)at * p.G << shift) * VD + (size_t)head * VD;
        const float* gz = p.gate + (size_t)at * p.ld_gate + (size_t)head * VD;
        for (int c = 0; c < VD; c += 16) {
          uint32_t o[16];
          tmem_ld_32x32b_x16(tmem_o + lanes + c, o);
          tmem_ld_wait();
          if (!mine) continue;
          float f[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) f[j] = __uint_as_float(o[j]) * inv;
          if (p.gate) {
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
              const float4 g = *reinterpret_cast<const float4*>(gz + c + j);
              f[j] *= sigmoid_f(g.x); f[j + 1] *= sigmoid_f(g.y); f[j + 2] *= sigmoid_f(g.z); f[j + 3] *= sigmoid_f(g.w);
            }
          }
          *reinterpret_cast<uint4*>(dst + c) = pack_bf16x8(f);
          *reinterpret_cast<uint4*>(dst + c + 8) = pack_bf16x8(f + 8);
        }
      }
    } else {
      // the second map's rows, times lambda, go through shared memory (the stages: every product has read them); the first map's finish the heads
      constexpr int LDO = VD + 4;
      float* o2 = reinterpret_cast<float*>(sK) + (size_t)(r % R) * LDO;
      const float lam = diff_lambda<T>(p.diff), inv = 1.0f / l;
      if (map == 1 && ok) {
        const float f = inv * lam;
        for (int c = 0; c < VD; c += 16) {
          uint32_t o[16];
          tmem_ld_32x32b_x16(tmem_o + lanes + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            *reinterpret_cast<float4*>(o2 + c + j) = make_float4(__uint_as_float(o[j]) * f, __uint_as_float(o[j + 1]) * f, __uint_as_float(o[j + 2]) * f, __uint_as_float(o[j + 3]) * f);
        }
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (map == 0 && ok) {
        const bool mine = row < rows;
        T* dst = (T*)p.y + ((size_t)(r0 + tok) * (p.G / 2) << shift) * VD + (size_t)((gv << shift) + (row & ((1 << shift) - 1))) * VD;
        float ss = 0.f, f = 0.f;
        for (int pass = 0; pass < 2; ++pass) {
          for (int c = 0; c < VD; c += 16) {
            uint32_t o[16];
            tmem_ld_32x32b_x16(tmem_o + lanes + c, o);
            tmem_ld_wait();
            float x[16];
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
              const float4 b = *reinterpret_cast<const float4*>(o2 + c + j);
              x[j] = fmaf(__uint_as_float(o[j]), inv, -b.x); x[j + 1] = fmaf(__uint_as_float(o[j + 1]), inv, -b.y);
              x[j + 2] = fmaf(__uint_as_float(o[j + 2]), inv, -b.z); x[j + 3] = fmaf(__uint_as_float(o[j + 3]), inv, -b.w);
            }
            if (pass == 0) {
#pragma unroll
              for (int j = 0; j < 16; ++j) ss = fmaf(x[j], x[j], ss);
            } else if (mine) {
#pragma unroll
              for (int j = 0; j < 16; ++j) x[j] *= f;
              *reinterpret_cast<uint4*>(dst + c) = pack_bf16x8(x);
              *reinterpret_cast<uint4*>(dst + c + 8) = pack_bf16x8(x + 8);
            }
          }
          f = (1.0f - p.diff.diff) / sqrtf(ss / (float)VD + p.diff.eps);
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
