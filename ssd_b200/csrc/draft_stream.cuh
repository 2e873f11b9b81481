// draft_stream.cuh — the whole speculate phase of a sync-SD step (SpeculatorSync.speculate, engine/speculator_sync.py:25-69:
// K+1 single-token draft forwards + K samplings) as ONE persistent kernel, for up to eight sequences.
//
// What bounds it: at one token per sequence every weight is used once per sequence, so a forward is a stream of the weights (1B draft: 2.47 GB,
// 0.377 ms at copy bandwidth; 0.6B: 1.06 GB) and, with long contexts, of the keys.  What keeps it from that is the chain of five dependent stages per layer: every
// row of the next matrix needs the whole previous vector, from all CTAs.  Two things shorten it:
//   * The weights do not depend on the activations, so every CTA (one per SM) streams ITS rows of every matrix, in program order and without
//     ever waiting for a stage, through a ring of shared-memory slots (bulk copies, one per row; a PRODUCER warp asks for them as the consumers
//     give slots back).  While the CTAs wait for one another the ring (148 x 200 KB = 30 MB on chip, 4.5 us of the memory) fills with the next stages' weights.
//   * The stages meet WITHOUT a barrier: a result leaves as one 32-bit word {tag, bf16}, whose reader polls the very words it needs until they carry the
//     tag of this layer and forward.  No fence, no arrival counter, no load of the vector behind the wait: one trip through L2 instead of four.
//
// Program order per forward (the five dependent stages of the reference's decoder layer, models/llama3.py:185-199):
//   A  [residual add + input RMSNorm, by every CTA for itself] -> q|k|v rows
//   B  q/k head norm + RoPE + KV store + attention for (sequence, kv head, split) units; splits exchange partial results and merge a part of the heads each
//   C  o-proj rows
//   D  [residual add + post-attention RMSNorm, every CTA] -> gate|up row pairs + SiLU*mul
//   E  down-proj rows
// then final norm -> lm_head rows -> in-kernel sampling (greedy argmax over the bf16 logits, lowest index wins, or the
// Philox exponential race of layers/sampler.py:27-34 — the SAME scores sample_kernel computes, so the tokens are identical)
// -> the next forward starts inside the same launch.  The last forward of a step only writes KV (speculator_sync.py:52-56).
// Rounding points are the reference's: every linear output, the residual, the norm output, q/k
// after RoPE and the attention output are rounded to bf16; accumulation is fp32, in the tensor cores for chains of two products of 16 columns (more than
// four sequences: four), which fp32 adds bring together.  Of logits of
// 2048 columns 7.2e-5 (one sequence), 8.7e-5 (three), 8.6e-5 (eight) are not the rounded exact sum; chains of fp32 FMA that one warp per row ran before left 7.8e-5, the kernel-by-kernel
// form, which batches took before, 8.7e-4 .. 9.1e-4.
//
// Products: a CTA owns a run of consecutive rows of every matrix (N / #CTAs, to one row), walked in tiles of 8 rows x up to 2048 columns = one slot.
// mma.sync m16n8k16; the eight warps take an eighth of the columns each and meet in shared memory once per group of tiles.  The order of k inside a product is free as long
// as both operands agree, so a 16-byte read of 8 consecutive k of a row IS a thread's part of two fragments, and the same 8 k of a token its part of the other operand's.
//
// Measured, us a forward of the 1B draft (16 layers, context 203): with device-wide barriers between the stages and one warp per row on CUDA cores 738 (40.8 a layer, 18.6 of them weights at
// copy bandwidth); tags 705; all reads of a slot in front of its products, which then go in four chains 665; one rolled copy of the code for all stages, which stays in the instruction
// caches 622; two steps of k per product and missing words asked for again together 552; no
// first piece asked for alone in front of gate|up's words 532; a key's place looked up once for a warp 506 (context 135).  Of the 27.8 us of a layer: attention 4.9 (one CTA per key head fetches
// the keys), the four other exchanges with their norms 1.7 to 2.1 each (the CTA whose weights come last is waited for in them), rows 15.6 (18.6 is the memory's rate; what the ring holds is ahead);
// the head 72.  (The code has to stay small: a slot's steps written out for every count, or the attention twice, cost more than 4 % though it is not run.)  Contexts of 60 to 8000 tokens and other batches: use_draft_stream (engine.cu).
//
// Tags.  tag = forward * L + layer + 1; the words are zeroed at kernel start (a device-wide barrier follows), so no word of another launch is taken for this one's.
// A word is overwritten only after everybody has read it: with at least one row of every matrix on every CTA (d, ffn, q|k|v and vocabulary >= #CTAs, checked by
// the host), a CTA's words of a stage are written after it has read ALL words of the stage in front, so whoever holds all of stage s knows that every CTA is done
// reading stage s - 1, and the next use of a vector lies five stages behind.
#pragma once
#include "common.cuh"
#include "sampling.cuh"

namespace ssdk {

constexpr int kDsConsumers = 256;                 // threads 0..255: 8 consumer warps
constexpr int kDsWarps = kDsConsumers / 32;
constexpr int kDsThreads = kDsConsumers + 128;    // + a warpgroup whose first warp is the producer
// registers: the block is meant to be launched with 384 x 168; the producer's warpgroup gives most of its own to the consumers (heads of 128: keys and values in flight)
constexpr int kDsRegsLaunch = 168, kDsRegsProducer = 40, kDsRegsConsumer = 232;
// whether a kernel that was built with that many registers can be launched: a split above what the block has would wait for ever
__host__ inline constexpr bool ds_registers_fit(int regs) {
  return regs >= kDsRegsProducer && regs <= kDsRegsConsumer && kDsConsumers * kDsRegsConsumer + 128 * kDsRegsProducer <= kDsThreads * regs;
}
static_assert(ds_registers_fit(kDsRegsLaunch), "register split");
constexpr int kDsMaxLayers = 32;
constexpr int kDsMaxBatch = 8;
constexpr int kDsSplits = 16;         // most ranges of a sequence's keys in stage B
constexpr int kDsUnitKeys = 256;      // keys of a unit that ONE round of loads covers (8 warps x 32)
constexpr int kDsTile = 8;            // weight rows of a tile
constexpr int kDsMaxChunk = 2048;     // columns of a slot
constexpr int kDsMaxChunks = 4;       // slots per tile (K <= 8192)
constexpr int kDsPad = 64;            // bytes behind a row in a slot: rows of a quarter-warp on different banks
constexpr int kDsSlotBytes = 33 * 1024;   // room for a slot of kDsMaxChunk columns
constexpr int kDsMaxSlots = 12;
constexpr int kDsStage = 33 * 1024;   // vectors up to this many bytes are laid out for the fragments in shared memory
constexpr int kDsBtSmem = 32;         // page-table entries of a sequence staged in shared memory at kernel start (the table is launch-constant)

#ifdef SSDK_HOST_EMU
inline long long ds_wait_cycles = 4000000000000LL;   // (tests set it)
#else
constexpr long long ds_wait_cycles = 4000000000LL;   // of clock64: about two seconds
#endif

struct DsLayer {
  const __nv_bfloat16 *qkv, *o, *gate_up, *down, *in_norm, *post_norm, *q_norm, *k_norm;
};

struct DsParams {
  int d, L, H, KV, ffn, vocab, qk_norm;
  float eps, scale_log2;
  const __nv_bfloat16 *embed, *final_norm, *lm_head;
  const float* rope;  // [max_pos, hd]: cos | sin
  __nv_bfloat16 *k_cache, *v_cache;
  long long cache_layer_stride;  // elements between layers
  int block_size, max_blocks;
  int64_t* tok_buf;              // sequence b at tok_buf + b * tok_ld: [n_fwd (+1)]: [0] = first input token; the kernel writes [f + 1]
  int n_fwd;                     // forwards in this launch
  int skip_last_head;            // 1: the last forward runs without lm_head / sampling (it only writes KV)
  int logits_only;               // 1: nobody reads tokens (one forward, whose logits another kernel samples)
  const int32_t* ctx0;           // [batch]: tokens in the cache before the first forward
  const int32_t* block_table;    // [batch][max_blocks]
  __nv_bfloat16* logits;         // row of sequence b and forward f at logits + b * logits_seq_ld + f * logits_ld (may be null: no logits kept)
  long long logits_ld;
  const float* temp;             // draft temperatures [batch] (device)
  const uint64_t* dyn;           // optional device {seed, step}: call_id = step * 16 + f
  uint64_t seed, call_base;      // used when dyn == nullptr: call_id = call_base + f
  ArgMax* samp_partial;          // [batch][#CTAs]
  unsigned* bar_state;           // one 64-bit arrival counter (8-byte aligned), only ever grows; zero before the first launch
  int n_slots;                   // ring depth
  int batch;                     // sequences (0: one)
  int tok_ld;
  long long logits_seq_ld;
  int max_chunk;                 // most columns of a slot (0: kDsMaxChunk)
  int slot_bytes;                // ring stride (0: that of kDsMaxChunk columns)
  uint32_t* words;               // ds_words() words: exchange of the stages
  unsigned* timeout;             // set when a bounded wait runs out
#ifdef SSDK_HOST_EMU
  // a test's second form, without `words`: the vectors as plain bf16, stages meet at the device-wide barrier (one sequence)
  __nv_bfloat16 *vec_qkv, *vec_attn, *vec_o, *vec_act, *vec_down, *resid0, *resid1;
  float* attn_part;              // [H][kDsSplits][hd + 2]: o | m | l
  unsigned* attn_ticket;
#endif
  DsLayer layers[kDsMaxLayers];
};

// consumer-only block barrier (the producer warp runs on its own)
SSDK_DEVINL void ds_sync() {
#ifdef SSDK_HOST_EMU
  ::emu::named_barrier(1, kDsConsumers);
#else
  asm volatile("bar.sync 1, 256;" ::: "memory");
#endif
}

// The thread's number, anew for every stage: what is worked out from it cannot be moved in front of the loop over layers, where the compiler would keep
// the addresses of all stages alive at once.
SSDK_DEVINL int ds_tid() {
  int t = (int)threadIdx.x;
#ifndef SSDK_HOST_EMU
  asm volatile("" : "+r"(t));
#endif
  return t;
}

// ---------------------------------------------------------------------------------------------
// waits: all have a limit.  One that runs out sets the launch's word (the host's next look at it is an error of the call) and the CTA goes on without what it waited for: its results are
// garbage that stays in bounds, under the tags that other CTAs wait for, and it arrives at every barrier, so that the launch ends and leaves the next one a whole count.
// `dead`: words and barriers, which other CTAs bring; every later wait of the CTA for one returns at once, while its weights, which it fetches itself, are waited for as ever.
// `broken`: slots of the ring; neither side waits for them any more, and the producer asks for nothing more and waits, again with a limit, for what is in flight.
// ---------------------------------------------------------------------------------------------
struct DsWait {
  volatile int* dead;   // shared by the CTA
  unsigned* timeout;
  SSDK_DEVINL bool give_up(long long t0) const {
    if (*dead) return true;
    if (clock64() - t0 < ds_wait_cycles) return false;
    *dead = 1;
    if (timeout) *reinterpret_cast<volatile unsigned*>(timeout) = 1u;
    return true;
  }
};
SSDK_DEVINL bool ds_ring_wait(uint64_t* bar, uint32_t parity, const DsWait& broken) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity))
    if (broken.give_up(t0)) return false;
  return true;
}

// ---------------------------------------------------------------------------------------------
// device-wide barrier of the consumers (kernel start, and once per forward behind the sampling, where it also orders the new keys and values): ONE 64-bit arrival
// counter that only ever grows.  Barrier number n of a launch is complete when the counter reaches base + n * #CTAs, where base = the counter rounded down to a multiple
// of #CTAs at kernel start (every launch performs whole barriers, and the first barrier of a launch cannot complete before this CTA has arrived, so every CTA computes the
// same base).  Arrival = one release-add without a return value; waiting = relaxed polling loads + one acquire fence at the end.
// ---------------------------------------------------------------------------------------------
struct DsGridBar {
  unsigned long long* counter;
  unsigned long long target;
  __device__ void init() {
    if (threadIdx.x == 0) {
      const unsigned long long c = ld_relaxed_gpu_u64(counter);
      target = c - c % (unsigned long long)gridDim.x;
    }
  }
  __device__ void sync(const DsWait& w) {
    ds_sync();  // every consumer thread's writes are ordered before thread 0's release
    if (threadIdx.x == 0) {
      target += (unsigned long long)gridDim.x;
      red_add_release_gpu_u64(counter, 1ull);
      const long long t0 = clock64();
      while (ld_relaxed_gpu_u64(counter) < target)
        if (w.give_up(t0)) break;
      fence_acq_rel_gpu();
    }
    ds_sync();
  }
};

SSDK_DEVINL uint4 ds_ldcg16(const void* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }
SSDK_DEVINL float ds_bits_f(uint32_t low16) { return __bfloat162float(__ushort_as_bfloat16((unsigned short)low16)); }
SSDK_DEVINL uint32_t ds_f_bits(float x) {
  const __nv_bfloat16 b = f2bf(x);
  return (uint32_t)*reinterpret_cast<const unsigned short*>(&b);
}

// timeline marks of the second forward of a launch (CTA 0, thread 0; only when ssdk_debug_trace is on): ids 64 + point
SSDK_DEVINL void ds_mark(int f, int point) {
  if (f == 1 && threadIdx.x == 0) trace_mark(64 + point);
}

// ---------------------------------------------------------------------------------------------
// matrix geometry
// ---------------------------------------------------------------------------------------------
enum { DS_QKV = 0, DS_O = 1, DS_GU = 2, DS_DOWN = 3, DS_HEAD = 4 };
struct DsGeom {
  int K;       // row length
  int rows;    // output rows (gate|up: pairs)
  int chunks;  // slots of a tile
  int ck;      // columns of a slot: K / chunks, a multiple of 256
  int r0, r1;  // this CTA's rows
};
__host__ SSDK_DEVINL bool ds_geometry(int K, int rows, int max_chunk, DsGeom* g) {
  g->K = K; g->rows = rows;
  for (g->chunks = 1; g->chunks <= kDsMaxChunks; ++g->chunks) {
    g->ck = K / g->chunks;
    if (K % g->chunks == 0 && g->ck % 256 == 0 && g->ck <= max_chunk) return K > 0;
  }
  return false;
}
__host__ SSDK_DEVINL int ds_slot_bytes(int max_chunk) { return kDsTile * (2 * max_chunk + kDsPad); }
// exchange words of a launch: q|k|v, attention, o, act, down of every sequence, then the attention's partial results (two words each)
__host__ SSDK_DEVINL long long ds_vec_words(int batch, int d, int H, int KV, int hd, int ffn) {
  return (long long)batch * ((H + 2 * KV) * hd + H * hd + 2 * d + ffn);
}
__host__ SSDK_DEVINL int ds_max_splits(int batch, int KV, int ctas) {   // units that the CTAs hold at once
  const int n = ctas / (batch * KV);
  return n < 1 ? 1 : (n < kDsSplits ? n : kDsSplits);
}
__host__ SSDK_DEVINL long long ds_words(int batch, int d, int H, int KV, int hd, int ffn, int ctas) {
  return ds_vec_words(batch, d, H, KV, hd, ffn) + 2ll * batch * H * ds_max_splits(batch, KV, ctas) * (hd + 2);
}
// bytes behind the ring and the tile sums: normed rows, a vector laid out for the fragments, or the attention's scratch (never two of them at once)
__host__ SSDK_DEVINL size_t ds_stage_bytes(int batch, int K) { return (size_t)kDsWarps * batch * (K / kDsWarps * 2 + kDsPad); }
__host__ SSDK_DEVINL size_t ds_attn_bytes(int G, int hd) {
  return (size_t)G * (2 * hd + kDsPad) + 4 * hd + (size_t)kDsWarps * G * (hd + 2) * 4;
}
__host__ SSDK_DEVINL bool ds_staged(int MT, int batch, int K) { return MT <= 4 && ds_stage_bytes(batch, K) <= (size_t)kDsStage; }
__host__ SSDK_DEVINL constexpr int ds_group(int MT) { return MT == 1 ? 16 : 32 / MT; }   // tiles whose sums meet at once: 256 threads, one per row and token (one token: half of them)
__host__ SSDK_DEVINL size_t ds_part_bytes(int MT) { return (size_t)ds_group(MT) * kDsWarps * MT * 8 * 4; }

SSDK_DEVINL bool ds_has_head(const DsParams& p, int f) { return !(p.skip_last_head && f == p.n_fwd - 1); }
SSDK_DEVINL void ds_own_rows(DsGeom* g) {
  g->r0 = (int)((long long)g->rows * blockIdx.x / gridDim.x);
  g->r1 = (int)((long long)g->rows * (blockIdx.x + 1) / gridDim.x);
}

// the producer warp: walks the tiles of this CTA and refills slots as the consumers release them, a bulk copy per row.  (Tiles
// behind the ring asked for into L2 as well were measured three times and do not pay: by the copy engine 8B + 1B 8.53 / 8.63 vs 8.34 / 8.48 ms per step; by prefetches of the
// producer's lanes while the ring is full, paced to the memory's rate, 551 -> 563 us a forward.)
struct DsProducer {
  uint8_t* ring;
  uint64_t *full, *empty;
  unsigned n_slots, slot_bytes, slot, phase;
  DsWait broken;
  unsigned used;   // slots that have been asked for at least once
};
template <int MT>
SSDK_DEVINL bool ds_feed(DsProducer& r, const DsGeom& g, const __nv_bfloat16* w, bool pair) {
  constexpr int group = ds_group(MT);
  const int lane = threadIdx.x & 31, sub = pair ? 2 : 1, r1 = g.r1;
  for (int t0 = g.r0; t0 < r1; t0 += kDsTile * group / sub)   // the order of ds_consume: groups, chunks, tiles
    for (int c = 0; c < g.chunks; ++c)
      for (int i = 0; i < group; ++i) {
        const int t = t0 + i / sub * kDsTile, n = min(kDsTile, r1 - t);
        if (n <= 0) break;
        int ok = 1;   // (consumers that have given up say so before they give a slot back: a slot whose last copy may be in flight is not asked for again)
        if (lane == 0) {
          ok = ds_ring_wait(&r.empty[r.slot], r.phase ^ 1u, r.broken) && !*r.broken.dead;  // a fresh barrier passes the first round at once
          if (ok) mbar_arrive_expect_tx(&r.full[r.slot], (unsigned)(n * g.ck * 2));
        }
        if (!__shfl_sync(0xffffffffu, ok, 0)) return false;
        if (lane < n)
          bulk_load_g2s(r.ring + (size_t)r.slot * r.slot_bytes + (size_t)lane * (g.ck * 2 + kDsPad),
                        w + ((size_t)(i % sub ? g.rows : 0) + t + lane) * g.K + (size_t)c * g.ck, (unsigned)g.ck * 2u, &r.full[r.slot]);
        if (++r.slot == r.n_slots) { r.slot = 0; r.phase ^= 1u; r.used = r.n_slots; }
        r.used = max(r.used, r.slot);
      }
  return true;
}
template <int MT>
SSDK_DEVINL void ds_producer(const DsParams& p, const DsGeom* geom, DsProducer& r) {
  bool ok = true;
  for (int f = 0; ok && f < p.n_fwd; ++f) {
    for (int l = 0; ok && l < p.L; ++l) {
      const DsLayer& lw = p.layers[l];
      ok = ds_feed<MT>(r, geom[DS_QKV], lw.qkv, false) && ds_feed<MT>(r, geom[DS_O], lw.o, false) && ds_feed<MT>(r, geom[DS_GU], lw.gate_up, true) &&
           ds_feed<MT>(r, geom[DS_DOWN], lw.down, false);
    }
    if (ok && ds_has_head(p, f)) ok = ds_feed<MT>(r, geom[DS_HEAD], p.lm_head, false);
  }
  // no copy is in flight when the CTA leaves: the last one into every slot
  for (unsigned s = threadIdx.x & 31; s < r.used; s += 32) {
    const uint32_t parity = s < r.slot ? r.phase : r.phase ^ 1u;
    const long long t0 = clock64();
    while (!mbar_try_wait(&r.full[s], parity))
      if (clock64() - t0 > ds_wait_cycles) break;
  }
}

// ---------------------------------------------------------------------------------------------
// the exchange
// ---------------------------------------------------------------------------------------------
struct DsVec {                // one stage's results: [batch][n]
  uint32_t* words;
  int n;
#ifdef SSDK_HOST_EMU
  __nv_bfloat16* plain;       // without words
#endif
};
SSDK_DEVINL void ds_put(const DsVec& v, int b, int i, uint32_t tag, float x) {
#ifdef SSDK_HOST_EMU
  if (!v.words) { v.plain[(size_t)b * v.n + i] = f2bf(x); return; }
#endif
  st_relaxed_gpu_u32(v.words + (size_t)b * v.n + i, (tag << 16) | ds_f_bits(x));
}
SSDK_DEVINL bool ds_tagged(const uint4& w, uint32_t tag) {
  return (w.x >> 16) == tag && (w.y >> 16) == tag && (w.z >> 16) == tag && (w.w >> 16) == tag;
}
SSDK_DEVINL uint2 ds_pack4(const uint4& w) { return make_uint2(__byte_perm(w.x, w.y, 0x5410), __byte_perm(w.z, w.w, 0x5410)); }
// four consecutive words of sequence b, at i; one (the tag is the one that is waited for: host emulation without words)
SSDK_DEVINL uint32_t ds_ask_one(const DsVec& v, size_t at, uint32_t tag) {
#ifdef SSDK_HOST_EMU
  if (!v.words) return tag << 16 | ds_f_bits(bf2f(v.plain[at]));
#endif
  return ld_relaxed_gpu_u32(v.words + at);
}
SSDK_DEVINL uint4 ds_ask(const DsVec& v, int b, int i, uint32_t tag) {
#ifdef SSDK_HOST_EMU
  if (!v.words) {
    const size_t at = (size_t)b * v.n + i;
    return make_uint4(ds_ask_one(v, at, tag), ds_ask_one(v, at + 1, tag), ds_ask_one(v, at + 2, tag), ds_ask_one(v, at + 3, tag));
  }
#endif
  return ld_relaxed_gpu_v4(v.words + (size_t)b * v.n + i);
}
// waits until every piece of r carries the tag: all that are missing are asked for again at once (one after another costs a trip to L2 each: 5 us per norm of four tokens)
template <int N, class Ask>
SSDK_DEVINL void ds_have(uint4 (&r)[N], uint32_t tag, const DsWait& wait, Ask ask) {
  const long long t0 = clock64();
  for (;;) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < N; ++i) ok = ok && ds_tagged(r[i], tag);
    if (ok || wait.give_up(t0)) return;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (!ds_tagged(r[i], tag)) r[i] = ask(i);
  }
}
// a single piece, for as long as nothing is there yet: 148 CTAs that ask for everything over and over take L2's time from the weights
SSDK_DEVINL void ds_wait_first(const DsVec& v, int b, int i, uint32_t tag, const DsWait& wait) {
  uint4 r[1] = {ds_ask(v, b, i, tag)};
  ds_have(r, tag, wait, [&](int) { return ds_ask(v, b, i, tag); });
}

// ---------------------------------------------------------------------------------------------
// consumers: products
// ---------------------------------------------------------------------------------------------
struct DsRing {
  const uint8_t* base;
  uint64_t *full, *empty;
  unsigned n_slots, slot_bytes, slot, phase;
  DsWait broken;
};
// x of a chunk, this thread's fragments, steps of 32 columns of the warp's ck / 8.  Five tokens and more: step j, columns 32 j + 8 (lane & 3) .. + 8 of token lane / 4.
// Up to four: steps 2 j (lanes 0 .. 15) and 2 j + 1 (16 .. 31) of token (lane / 4) & 3.
template <int MT>
struct DsX {
  static constexpr int kHalf = MT <= 4 ? 2 : 1;
  uint4 v[8 / kHalf];
};
// N steps of a slot: all reads first, then the products in chains of their own (one or two chains, each read behind a test of its step: 0.8 us for a slot of 2048 columns).
// Up to four tokens a product takes two steps: the weights are the 16 rows, eight rows at one step above the same eight at the next, the tokens of both steps the eight columns, and
// the quarters of the result that belong together are those of the same step.  Otherwise the tokens are the rows (eight of the sixteen), the weights the columns.
template <int MT, int N>
SSDK_DEVINL void ds_steps(const uint8_t* w, const uint4* x, float (&c)[4][4]) {
  uint4 b[N];
#pragma unroll
  for (int j = 0; j < N; ++j) b[j] = *reinterpret_cast<const uint4*>(w + j * 64);
  if constexpr (MT <= 4) {
#pragma unroll
    for (int j = 0; j < N / 2; ++j) {
      const uint32_t a0[4] = {b[2 * j].x, b[2 * j + 1].x, b[2 * j].y, b[2 * j + 1].y}, a1[4] = {b[2 * j].z, b[2 * j + 1].z, b[2 * j].w, b[2 * j + 1].w};
      mma_bf16_16816(c[2 * j & 3], a0, x[j].x, x[j].y);
      mma_bf16_16816(c[(2 * j + 1) & 3], a1, x[j].z, x[j].w);
    }
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const uint32_t a0[4] = {x[j].x, 0u, x[j].y, 0u}, a1[4] = {x[j].z, 0u, x[j].w, 0u};
      mma_bf16_16816(c[2 * j & 3], a0, b[j].x, b[j].y);
      mma_bf16_16816(c[(2 * j + 1) & 3], a1, b[j].z, b[j].w);
    }
  }
}
// one slot: 8 rows x a chunk, into (c > 0: onto) the tile's sums [token][row]
template <int MT>
SSDK_DEVINL void ds_slot(DsRing& ring, int steps, int at, int lane, const DsX<MT>& x, int M, float* sums, bool onto) {
  constexpr int H = DsX<MT>::kHalf;
  float c[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) c[i][e] = 0.f;
  ds_ring_wait(&ring.full[ring.slot], ring.phase, ring.broken);   // (given up: whatever lies there)
  const uint8_t* w = ring.base + (unsigned)(ring.slot * ring.slot_bytes + at);
  if (steps == 8) {
    ds_steps<MT, 8>(w, x.v, c);
  } else if (steps == 4) {
    ds_steps<MT, 4>(w, x.v, c);
  } else {
#pragma unroll
    for (int j = 0; j < 8 / H; ++j) {
      if (H * j + H <= steps) {
        ds_steps<MT, H>(w + H * j * 64, x.v + j, c);
      } else if (H == 2 && 2 * j < steps) {   // an odd number of steps: the second half of the last product is zero
        const uint4 b = *reinterpret_cast<const uint4*>(w + 2 * j * 64);
        const uint32_t a0[4] = {b.x, 0u, b.y, 0u}, a1[4] = {b.z, 0u, b.w, 0u};
        mma_bf16_16816(c[0], a0, x.v[j].x, x.v[j].y);
        mma_bf16_16816(c[1], a1, x.v[j].z, x.v[j].w);
      }
    }
  }
  __syncwarp();
  if (lane == 0) mbar_arrive(&ring.empty[ring.slot]);   // one arrive per consumer warp, after its last read
  if (++ring.slot == ring.n_slots) { ring.slot = 0; ring.phase ^= 1u; }
  float s[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) s[e] = (c[0][e] + c[1][e]) + (c[2][e] + c[3][e]);
  const int q = lane & 3;
  float v0, v1;
  int t0, row, step;   // sums of tokens t0 (v0) and, `step` floats on, of the next token or row
  bool mine0, mine1;
  if (H == 2) {   // row lane / 4; tokens 2q, 2q + 1 of the even steps (q < 2), 2q - 4, 2q - 3 of the odd ones
    v0 = q < 2 ? s[0] : s[2];
    v1 = q < 2 ? s[1] : s[3];
    v0 += __shfl_xor_sync(0xffffffffu, v0, 2);
    v1 += __shfl_xor_sync(0xffffffffu, v1, 2);
    t0 = 2 * q; row = lane >> 2; step = 8;
    mine0 = t0 < min(M, 4); mine1 = t0 + 1 < min(M, 4);
  } else {        // token lane / 4; rows 2q, 2q + 1
    v0 = s[0]; v1 = s[1];
    t0 = lane >> 2; row = 2 * q; step = 1;
    mine0 = mine1 = t0 < M;
  }
  float* to = sums + t0 * 8 + row;
  if (mine0) to[0] = onto ? to[0] + v0 : v0;
  if (mine1) to[step] = onto ? to[step] + v1 : v1;
}

// sampling state of the lm_head stage (a thread always sees the same sequence)
struct DsSample {
  float T;
  uint64_t seed, call_id;
  uint32_t row;
  __nv_bfloat16* logits;   // of the sequence, or null
  ArgMax best;
};
SSDK_DEVINL float ds_score(const DsSample& s, float logit, int idx) {
  if (s.T == 0.f) return logit;
  // scores = softmax(l/T) / (E + 1e-10) in the log domain, the very expression of sample_kernel (sampling.cuh)
  const uint4 rnd = philox_draw((uint32_t)(idx >> 2), s.row, s.call_id, TAG_SAMPLE, s.seed);
  const float e = u32_to_exp1(u4_word(rnd, idx & 3)) + 1e-10f;
  return logit * (1.f / s.T) - __logf(e);
}

enum { DS_ROWS = 0, DS_GATED = 1, DS_LOGITS = 2 };
// this CTA's rows of a matrix.  The warps' sums of a group of tiles meet in `part` [group][kDsWarps][8 MT], summed in warp order; thread t has
// tile t / (8 MT), token (t / 8) % MT, row t % 8.
//   DS_ROWS   out[token][row] = bf16(W[row] . x)
//   DS_GATED  act[i] = bf16(silu(bf16 g_i) * bf16 u_i)   (layers/activation.py:11-14 on the bf16-rounded linear output), tiles 2i gate, 2i + 1 up
//   DS_LOGITS logits, and the thread's running best score
// The tiles of a group go chunk after chunk, so that only one chunk of x has to be at hand: load(c, x) brings it.
// One copy of this serves all stages, with its loops rolled: written out per stage the kernel's code does not stay in the instruction caches, and a slot takes 610 cycles where
// the same instructions take 340 (clock64 around them here, and in a loop by themselves).
template <int MT, class Load>
SSDK_DEVINL void ds_consume(DsRing& ring, const DsGeom& g, int mode, int M, float* part, const DsVec& out, uint32_t tag, Load load, DsSample& smp) {
  constexpr int group = ds_group(MT);
  const int per = mode == DS_GATED ? 2 : 1, rows = kDsTile * group / per;
  const int tid = ds_tid(), warp = tid >> 5, lane = tid & 31, r1 = g.r1, steps = g.ck >> 8;
  const int at = (lane >> 2) * (g.ck * 2 + kDsPad) + warp * (g.ck >> 2) + (lane & 3) * 16;   // this thread's part of a slot
  DsX<MT> x;
  if (g.chunks == 1) load(0, x);
  for (int t0 = g.r0; t0 < r1; t0 += rows) {
    const int n = min(group, (r1 - t0 + kDsTile - 1) / kDsTile * per);   // tiles of the group
    if (t0 > g.r0) ds_sync();   // (the sums in front have been read; a stage's first ones: there is a barrier in every stage's operands)
    float* mine = part + warp * (8 * MT);
    for (int c = 0; c < g.chunks; ++c) {
      if (g.chunks > 1) load(c, x);
#pragma unroll 1
      for (int i = 0; i < n; ++i) ds_slot<MT>(ring, steps, at, lane, x, M, mine + i * kDsWarps * (8 * MT), c > 0);
    }
    ds_sync();
    const int tile = tid / (8 * MT), tok = (tid >> 3) & (MT - 1), row = t0 + tile * kDsTile + (tid & 7);
    if (tile * per < n && tok < M && row < r1) {
      const float* src = part + tile * per * kDsWarps * (8 * MT) + (tid & (8 * MT - 1));
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < kDsWarps; ++w) s += src[w * 8 * MT];
      if (mode == DS_GATED) {
        float u = 0.f;
#pragma unroll
        for (int w = 0; w < kDsWarps; ++w) u += src[(kDsWarps + w) * 8 * MT];
        s = bf16_round(s);
        u = bf16_round(u);
        s = (s / (1.0f + __expf(-s))) * u;
      }
      if (mode == DS_LOGITS) {
        const __nv_bfloat16 o = f2bf(s);
        if (smp.logits) smp.logits[row] = o;
        smp.best = argmax_better(smp.best, ArgMax{ds_score(smp, bf2f(o), row), row});
      } else {
        ds_put(out, tok, row, tag, s);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// consumers: operands of a stage
// ---------------------------------------------------------------------------------------------
// xs[m] = bf16r( r * rsqrt(mean r^2 + eps) * w ),  r = a (+ resid) in fp32;  resid = bf16(r), which every CTA keeps for itself (thread t only touches elements 8 t .. 8 t + 8).
// a: a stage's results, or (src == nullptr) rows of the embedding, which are their own residual.
template <int MT>
SSDK_DEVINL void ds_norm(const DsVec* src, const __nv_bfloat16* embed, int vocab, const int* tok, uint8_t* resid, const __nv_bfloat16* w, float eps, int d, int M, uint32_t tag,
                         const DsWait& wait, uint8_t* xs, float* red) {
  const int tid = ds_tid(), i0 = tid * 8, warp = tid >> 5, lane = tid & 31;
  const bool on = i0 < d;
  uint4 wv = make_uint4(0u, 0u, 0u, 0u);
  if (on) wv = *reinterpret_cast<const uint4*>(w + i0);
  float x[MT][8];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int j = 0; j < 8; ++j) x[m][j] = 0.f;
  if (src) {
    if (on) {
      uint4 v[2 * MT];   // (tokens that the batch has not ask for the first one's; every register of a stage is written in full: one that is written here and there
                         // stays alive from layer to layer, and all stages' together spill, 1250 us a forward)
      auto ask = [&](int i) { return ds_ask(*src, (i >> 1) < M ? i >> 1 : 0, i0 + 4 * (i & 1), tag); };
#pragma unroll
      for (int i = 0; i < 2 * MT; ++i) v[i] = ask(i);
      ds_have(v, tag, wait, ask);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        if (m < M) {
          unpack_bf16x8(*reinterpret_cast<const uint4*>(resid + ((size_t)m * d + i0) * 2), x[m]);
          const uint4 lo = v[2 * m], hi = v[2 * m + 1];
          x[m][0] += ds_bits_f(lo.x); x[m][1] += ds_bits_f(lo.y); x[m][2] += ds_bits_f(lo.z); x[m][3] += ds_bits_f(lo.w);
          x[m][4] += ds_bits_f(hi.x); x[m][5] += ds_bits_f(hi.y); x[m][6] += ds_bits_f(hi.z); x[m][7] += ds_bits_f(hi.w);
        }
      }
    }
  } else {
#pragma unroll
    for (int m = 0; m < MT; ++m)
      if (m < M && on && (unsigned)tok[m] < (unsigned)vocab) unpack_bf16x8(*reinterpret_cast<const uint4*>(embed + (size_t)tok[m] * d + i0), x[m]);
  }
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    if (m < M) {
      float ss = 0.f;
      if (on) {
        *reinterpret_cast<uint4*>(resid + ((size_t)m * d + i0) * 2) = pack_bf16x8(x[m]);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += x[m][j] * x[m][j];
      }
      ss = warp_sum(ss);
      if (lane == 0) red[warp * MT + m] = ss;
    }
  }
  ds_sync();
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    if (m < M && on) {
      float ss = 0.f;
#pragma unroll
      for (int q = 0; q < kDsWarps; ++q) ss += red[q * MT + m];
      const float rstd = rsqrtf(ss / (float)d + eps);
      float wf[8];
      unpack_bf16x8(wv, wf);
#pragma unroll
      for (int j = 0; j < 8; ++j) x[m][j] = x[m][j] * rstd * wf[j];
      *reinterpret_cast<uint4*>(xs + (size_t)m * (2 * d + kDsPad) + i0 * 2) = pack_bf16x8(x[m]);
    }
  }
  ds_sync();
}
// A stage's results as they are, up to four tokens: a warp asks for its columns with all its lanes (all requests in flight at once) and lays them out
// in shared memory of its own.  patient: asks for one piece until there is something.  Behind the attention, where most CTAs wait while a few fetch keys (asking for everything takes 8 %
// of a 0.6B forward); behind gate|up the CTAs arrive together, and one token's first piece would cost a trip to L2 more than it saves (8B + 1B, k = 6, two target layers: 4428 -> 4167 us).
template <int MT>
SSDK_DEVINL const uint8_t* ds_stage_vec(const DsVec& v, const DsGeom& g, int M, uint32_t tag, const DsWait& wait, uint8_t* stage, bool patient) {
  const int tid = ds_tid(), warp = tid >> 5, lane = tid & 31;
  const int part = g.ck >> 3, pitch = g.K / kDsWarps * 2 + kDsPad;   // this warp's columns of a chunk; bytes of a token
  uint8_t* mine = stage + (size_t)warp * M * pitch;
  constexpr int N = MT == 1 ? 8 : 16;   // requests in flight
  const int halves = part > 128 ? 2 : 1, n = M * g.chunks * halves;   // pieces of 128 words: half, chunk, token
  const int last = (part - 1) & ~3;   // (lanes behind the last column ask for it)
  if (MT > 1 || patient) ds_wait_first(v, 0, warp * part + min(4 * lane, last), tag, wait);
  for (int e = 0; e < n; e += N) {
    auto where = [&](int i, int& b, int& c, int& col) {
      const int u = min(e + i, n - 1);   // (n <= 4 x 4 x 2)
      b = u / (g.chunks * halves);
      const int r = u - b * g.chunks * halves;
      c = r / halves;
      col = 4 * lane + 128 * (r - c * halves);
    };
    auto ask = [&](int i) {
      int b, c, col;
      where(i, b, c, col);
      return ds_ask(v, b, c * g.ck + warp * part + min(col, last), tag);
    };
    uint4 r[N];
#pragma unroll
    for (int i = 0; i < N; ++i) r[i] = ask(i);
    ds_have(r, tag, wait, ask);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      int b, c, col;
      where(i, b, c, col);
      if (e + i < n && col < part) *reinterpret_cast<uint2*>(mine + (size_t)b * pitch + (c * part + col) * 2) = ds_pack4(r[i]);
    }
  }
  __syncwarp();
  ds_sync();
  return mine;
}
// More tokens: every thread asks for its own words of a chunk.
template <int MT>
SSDK_DEVINL int ds_x_token(int lane) { return MT <= 4 ? (lane >> 2) & 3 : lane >> 2; }
template <int MT>
SSDK_DEVINL int ds_x_step(int lane, int j) { return MT <= 4 ? 2 * j + (lane >> 4) : j; }
template <int MT>
SSDK_DEVINL void ds_frag_vec(const DsVec& v, const DsGeom& g, int c, int M, uint32_t tag, const DsWait& wait, DsX<MT>& x) {
  constexpr int J = 8 / DsX<MT>::kHalf;
  const int tid = ds_tid(), warp = tid >> 5, lane = tid & 31, m = ds_x_token<MT>(lane);
  const int steps = g.ck >> 8, at = c * g.ck + warp * (g.ck >> 3) + 8 * (lane & 3);
  uint4 r[2 * J];
  auto ask = [&](int i) {   // (whoever has no token or step asks for another's)
    const int j = ds_x_step<MT>(lane, i >> 1);
    return ds_ask(v, m < M ? m : 0, at + 32 * (j < steps ? j : 0) + 4 * (i & 1), tag);
  };
#pragma unroll
  for (int i = 0; i < 2 * J; ++i) r[i] = ask(i);
  ds_have(r, tag, wait, ask);
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const uint2 lo = ds_pack4(r[2 * j]), hi = ds_pack4(r[2 * j + 1]);
    x.v[j] = ds_x_step<MT>(lane, j) < steps && m < M ? make_uint4(lo.x, lo.y, hi.x, hi.y) : make_uint4(0u, 0u, 0u, 0u);
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------------------------
// stage B unit: sequence b, kv head h, split s.  Rebuilds the rotated q rows of the head group and the new token's k / v from the
// q|k|v words, stores k / v into the page slot (split 0 only) and runs its token range: warp w takes 32 keys at a time, scores on mma.sync (q as A, keys as B), online
// softmax in registers, weights in three bf16 pieces (all of their bits) times the values as the other operand.  A thread's 16-byte loads ARE its fragments: eight
// dims of one key; of a value row, eight dims of which each product takes two.  The cached keys and values do not depend on this layer's stages, so they are asked for before
// the wait for q|k|v; the next 32 keys' are asked for as soon as their registers are free.
// (A lane per head dim with a five-shuffle sum per key and head, partials, a ticket and a merge by the last split: 4.8 us per layer at contexts of 135.)
// ---------------------------------------------------------------------------------------------
SSDK_DEVINL int ds_num_splits(int ctx, int most) { return min(most, (ctx + kDsUnitKeys - 1) / kDsUnitKeys); }

struct DsPages {
  const int32_t* table;   // of the sequence
  const int* staged;      // its copy in shared memory, or null
  int block_size, shift;  // (shift < 0: not a power of two)
  SSDK_DEVINL int page(int t) const {   // negative: the table names none
    const int i = shift >= 0 ? t >> shift : t / block_size;
    return staged ? staged[i] : table[i];
  }
  SSDK_DEVINL size_t slot(int t, int page) const { return (size_t)page * block_size + (shift >= 0 ? t & (block_size - 1) : t % block_size); }
};
// Keys tb .. tb + 32 of a warp.  Every lane looks one of them up and the loads take its row from there.  Keys behind the range and the new one (pos) are zero; whoever has none reads an
// earlier key, so that no load waits for a branch (1.2 us to get sixteen loads under way with one).  Tokens without a page count as zeros, as in paged_attn_kernel: they are read from
// ds_no_page (a flag or a bit per key next to the loads in flight spills: with heads of 128 212 bytes -> 536 and more).
__device__ uint4 ds_no_page[16];
constexpr uint32_t kDsNoSlot = 0xffffffffu;   // (a cache of that many rows is larger than the memory)
SSDK_DEVINL uint32_t ds_slots(const DsPages& pg, int lane, int tb, int t1, int pos) {
  const int t = min(tb + lane, max(min(t1, pos) - 1, 0));   // (at most the last key that is in the cache; none: the new one's slot, not used)
  const int page = pg.page(t);
  return page < 0 ? kDsNoSlot : (uint32_t)pg.slot(t, page);
}
SSDK_DEVINL const __nv_bfloat16* ds_key_row(const __nv_bfloat16* base, uint32_t slots, int key, int ld) {
  const uint32_t slot = __shfl_sync(0xffffffffu, slots, key);
  return slot == kDsNoSlot ? reinterpret_cast<const __nv_bfloat16*>(ds_no_page) : base + (size_t)slot * ld;
}
SSDK_DEVINL uint4 ds_keep(const uint4& v, bool on) { return make_uint4(on ? v.x : 0u, on ? v.y : 0u, on ? v.z : 0u, on ? v.w : 0u); }
// keys tb + 8 j + lane / 4, dims 32 k + 8 (lane & 3) .. + 8
template <int HD>
SSDK_DEVINL void ds_load_k(const __nv_bfloat16* base, uint32_t slots, int ld, int lane, uint4 (&k)[4][HD / 32]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __nv_bfloat16* s = ds_key_row(base, slots, 8 * j + (lane >> 2), ld) + 8 * (lane & 3);
#pragma unroll
    for (int i = 0; i < HD / 32; ++i) k[j][i] = ds_ldcg16(s + 32 * i);
  }
}
// value rows tb + 16 kk + {2q, 2q + 1, 2q + 8, 2q + 9} (q = lane & 3), dims 64 i + 8 (lane / 4) .. + 8
template <int HD>
SSDK_DEVINL void ds_load_v(const __nv_bfloat16* base, uint32_t slots, int ld, int lane, uint4 (&v)[2][4][HD / 64]) {
#pragma unroll
  for (int kk = 0; kk < 2; ++kk)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat16* s = ds_key_row(base, slots, 16 * kk + 2 * (lane & 3) + (j & 1) + 8 * (j >> 1), ld) + 8 * (lane >> 2);
#pragma unroll
      for (int i = 0; i < HD / 64; ++i) v[kk][j][i] = ds_ldcg16(s + 64 * i);
    }
}
// Two weights in three bf16 pieces each, whose sum is the weight in all of its 24 bits (what is left of it has 16 bits, then 8)
SSDK_DEVINL void ds_pieces(float p0, float p1, uint32_t (&w)[3]) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    w[q] = pack_bf16x2(p0, p1);
    p0 -= ds_bits_f(w[q] & 0xffffu);
    p1 -= ds_bits_f(w[q] >> 16);
  }
}
SSDK_DEVINL uint32_t ds_word(const uint4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }

struct DsPartial {            // partial results of the splits: per sequence, head and split hd sums, maximum, sum of weights
  unsigned long long* words;  // {fp32, tag}
  int most;                   // splits that there is room for
#ifdef SSDK_HOST_EMU
  float* plain;               // without words
#endif
};
SSDK_DEVINL void ds_put_part(const DsPartial& q, size_t i, uint32_t tag, float x) {
#ifdef SSDK_HOST_EMU
  if (!q.words) { q.plain[i] = x; return; }
#endif
  st_relaxed_gpu_u64(q.words + i, ((unsigned long long)tag << 32) | *reinterpret_cast<const uint32_t*>(&x));
}
SSDK_DEVINL unsigned long long ds_ask_part(const DsPartial& q, size_t i, uint32_t tag) {
#ifdef SSDK_HOST_EMU
  if (!q.words) return ((unsigned long long)tag << 32) | *reinterpret_cast<const uint32_t*>(q.plain + i);
#endif
  return ld_relaxed_gpu_u64(q.words + i);
}
SSDK_DEVINL float ds_part_value(unsigned long long w) {
  const uint32_t u = (uint32_t)w;
  return *reinterpret_cast<const float*>(&u);
}

template <int HD>
SSDK_DEVINL void ds_attention_unit(const DsParams& p, int layer, int b, int h, int s, int ns, int ctx, uint32_t tag, const DsVec& qkv, const DsVec& attn, const DsPartial& part,
                                   const DsPages& pg, const DsWait& wait, uint8_t* sm) {
  constexpr int HALF = HD / 2, PT = HALF / 32, KB = HD / 32, LDR = HD + 2, LDQ = 2 * HD + kDsPad;
  const int tid = ds_tid(), warp = tid >> 5, lane = tid & 31, quad = lane & 3;
  const int G = p.H / p.KV, pos = ctx - 1, ld = p.KV * HD;
  uint8_t* sq = sm;                                          // [G] rotated q rows, bf16
  __nv_bfloat16* sk = reinterpret_cast<__nv_bfloat16*>(sq + (size_t)G * LDQ);   // [HD] new k
  __nv_bfloat16* sv = sk + HD;                               // [HD] new v
  float* sred = reinterpret_cast<float*>(sv + HD);           // [kDsWarps][G][HD + 2] per-warp partials

  // ---- token range of this split; the first keys and values ----
  const int per = ((ctx + ns - 1) / ns + 31) & ~31;
  const int t0 = s * per, t1 = min(ctx, t0 + per);   // (the last ranges may be empty: their maximum is -inf)
  __nv_bfloat16* kbase = p.k_cache + (size_t)layer * p.cache_layer_stride + (size_t)h * HD;
  __nv_bfloat16* vbase = p.v_cache + (size_t)layer * p.cache_layer_stride + (size_t)h * HD;
  uint4 kf[4][KB], vf[2][4][HD / 64];
  int tb = t0 + warp * 32;
  uint32_t slots = ds_slots(pg, lane, tb, t1, pos);
  ds_load_k<HD>(kbase, slots, ld, lane, kf);
  ds_load_v<HD>(vbase, slots, ld, lane, vf);

  const int new_page = pg.page(pos);   // (in front of the wait)

  // ---- q rows, k, v: one warp per row, rotate-half pairs (i, i + HALF) ----
  const float* cs = p.rope + (size_t)pos * HD;
  for (int row = warp; row < G + 2; row += kDsWarps) {
    const int kind = row < G ? 0 : (row == G ? 1 : 2);
    const int col0 = (kind == 0 ? (h * G + row) : (kind == 1 ? p.H + h : p.H + p.KV + h)) * HD;
    float x1[PT], x2[PT], c[PT], sn[PT], n1[PT], n2[PT];
    const __nv_bfloat16* nw = p.qk_norm && kind < 2 ? (kind == 0 ? p.layers[layer].q_norm : p.layers[layer].k_norm) : nullptr;
#pragma unroll
    for (int t = 0; t < PT; ++t) {   // (what does not depend on this layer, in front of the wait)
      const int i = lane + 32 * t;
      c[t] = cs[i]; sn[t] = cs[HALF + i];
      n1[t] = nw ? bf2f(nw[i]) : 1.f; n2[t] = nw ? bf2f(nw[HALF + i]) : 1.f;
    }
    const size_t src = (size_t)b * qkv.n + col0 + lane;
    const long long w0 = clock64();
    bool ok;
    do {
      ok = true;
#pragma unroll
      for (int t = 0; t < PT; ++t) {
        const uint32_t u1 = ds_ask_one(qkv, src + 32 * t, tag), u2 = ds_ask_one(qkv, src + HALF + 32 * t, tag);
        ok = ok && (u1 >> 16) == tag && (u2 >> 16) == tag;
        x1[t] = ds_bits_f(u1 & 0xffffu); x2[t] = ds_bits_f(u2 & 0xffffu);
      }
    } while (!ok && !wait.give_up(w0));
    __syncwarp();
    if (nw) {
      float ss = 0.f;
#pragma unroll
      for (int t = 0; t < PT; ++t) ss += x1[t] * x1[t] + x2[t] * x2[t];
      ss = warp_sum(ss);
      const float rstd = rsqrtf(ss / (float)HD + p.eps);
#pragma unroll
      for (int t = 0; t < PT; ++t) { x1[t] = bf16_round(x1[t] * rstd * n1[t]); x2[t] = bf16_round(x2[t] * rstd * n2[t]); }
    }
    if (kind > 0 && new_page < 0) {   // a new token without a page counts like any other
#pragma unroll
      for (int t = 0; t < PT; ++t) x1[t] = x2[t] = 0.f;
    }
    if (kind == 2) {
#pragma unroll
      for (int t = 0; t < PT; ++t) { sv[lane + 32 * t] = f2bf(x1[t]); sv[HALF + lane + 32 * t] = f2bf(x2[t]); }
      continue;
    }
    __nv_bfloat16* dst = kind == 0 ? reinterpret_cast<__nv_bfloat16*>(sq + (size_t)row * LDQ) : sk;
#pragma unroll
    for (int t = 0; t < PT; ++t) {
      const int i = lane + 32 * t;
      dst[i] = f2bf(x1[t] * c[t] - x2[t] * sn[t]);
      dst[HALF + i] = f2bf(x2[t] * c[t] + x1[t] * sn[t]);
    }
  }
  ds_sync();

  // ---- KV store of the new token (one unit per kv head) ----
  if (s == 0 && tid < HD / 4 && new_page >= 0) {
    const int e = tid % (HD / 8) * 8;
    const bool val = tid >= HD / 8;
    *reinterpret_cast<uint4*>((val ? vbase : kbase) + pg.slot(pos, new_page) * ld + e) = *reinterpret_cast<const uint4*>((val ? sv : sk) + e);
  }

  uint4 qf[KB];
#pragma unroll
  for (int i = 0; i < KB; ++i)
    qf[i] = (lane >> 2) < G ? *reinterpret_cast<const uint4*>(sq + (size_t)(lane >> 2) * LDQ + 64 * i + 16 * quad) : make_uint4(0u, 0u, 0u, 0u);
  float o[HD / 16][4], m = -INFINITY, l = 0.f;   // o: dims 8 (lane / 4) + 2 (jd % 4) + {0, 0, 1, 1} (+ 64), heads 2 quad + {0, 1, 0, 1}; m, l: head lane / 4
#pragma unroll
  for (int j = 0; j < HD / 16; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  for (; tb < t1; tb += kDsUnitKeys) {
    const bool more = tb + kDsUnitKeys < t1;
    if (tb + 32 > min(t1, pos)) {   // the new token comes from shared memory, never from the cache; behind it and behind the range there is nothing
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = tb + 8 * j + (lane >> 2);
#pragma unroll
        for (int i = 0; i < KB; ++i) kf[j][i] = t == pos ? *reinterpret_cast<const uint4*>(sk + 32 * i + 8 * quad) : ds_keep(kf[j][i], t < min(t1, pos));
      }
#pragma unroll
      for (int kk = 0; kk < 2; ++kk)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int t = tb + 16 * kk + 2 * quad + (j & 1) + 8 * (j >> 1);
#pragma unroll
          for (int i = 0; i < HD / 64; ++i) vf[kk][j][i] = t == pos ? *reinterpret_cast<const uint4*>(sv + 64 * i + 8 * (lane >> 2)) : ds_keep(vf[kk][j][i], t < min(t1, pos));
        }
    }
    float sc[4][4];   // [j][0, 1]: head lane / 4, keys tb + 8 j + 2 quad + {0, 1}
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      sc[j][0] = sc[j][1] = sc[j][2] = sc[j][3] = 0.f;
#pragma unroll
      for (int i = 0; i < KB; ++i) {
        const uint32_t a0[4] = {qf[i].x, 0u, qf[i].y, 0u}, a1[4] = {qf[i].z, 0u, qf[i].w, 0u};
        mma_bf16_16816(sc[j], a0, kf[j][i].x, kf[j][i].y);
        mma_bf16_16816(sc[j], a1, kf[j][i].z, kf[j][i].w);
      }
    }
    if (more) {
      slots = ds_slots(pg, lane, tb + kDsUnitKeys, t1, pos);
      ds_load_k<HD>(kbase, slots, ld, lane, kf);
    }
    float mn = m;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        sc[j][e] = tb + 8 * j + 2 * quad + e < t1 ? sc[j][e] * p.scale_log2 : -INFINITY;
        mn = fmaxf(mn, sc[j][e]);
      }
    mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
    mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2));
    const float base = mn == -INFINITY ? 0.f : mn;   // (every key of a head at -inf)
    const float corr = exp2f(m - base);              // m = -inf -> 0
    m = mn;
    l *= corr;
    const float corr0 = __shfl_sync(0xffffffffu, corr, 8 * quad), corr1 = __shfl_sync(0xffffffffu, corr, 8 * quad + 4);
#pragma unroll
    for (int j = 0; j < HD / 16; ++j) { o[j][0] *= corr0; o[j][1] *= corr1; o[j][2] *= corr0; o[j][3] *= corr1; }
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      uint32_t w[2][3];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float p0 = exp2f(sc[2 * kk + e][0] - base), p1 = exp2f(sc[2 * kk + e][1] - base);
        l += p0 + p1;
        ds_pieces(p0, p1, w[e]);
      }
#pragma unroll
      for (int i = 0; i < HD / 64; ++i)
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          const uint32_t u0 = ds_word(vf[kk][0][i], d), u1 = ds_word(vf[kk][1][i], d), u2 = ds_word(vf[kk][2][i], d), u3 = ds_word(vf[kk][3][i], d);
          const uint32_t a[4] = {__byte_perm(u0, u1, 0x5410), __byte_perm(u0, u1, 0x7632), __byte_perm(u2, u3, 0x5410), __byte_perm(u2, u3, 0x7632)};
#pragma unroll
          for (int q = 0; q < 3; ++q) mma_bf16_16816(o[4 * i + d], a, w[0][q], w[1][q]);
        }
    }
    if (more) ds_load_v<HD>(vbase, slots, ld, lane, vf);
  }
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  // ---- merge the warps through shared memory, one thread per (head, dim) ----
  float* mine = sred + (size_t)warp * G * LDR;
#pragma unroll
  for (int j = 0; j < HD / 16; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (2 * quad + (e & 1) < G) mine[(size_t)(2 * quad + (e & 1)) * LDR + 64 * (j >> 2) + 8 * (lane >> 2) + 2 * (j & 3) + (e >> 1)] = o[j][e];
  if (quad == 0 && (lane >> 2) < G) {
    mine[(size_t)(lane >> 2) * LDR + HD] = m;
    mine[(size_t)(lane >> 2) * LDR + HD + 1] = l;
  }
  ds_sync();
  for (int idx = tid; idx < G * HD; idx += kDsConsumers) {
    const int g = idx / HD, dim = idx % HD;
    float mx = -INFINITY;
#pragma unroll
    for (int w = 0; w < kDsWarps; ++w) mx = fmaxf(mx, sred[((size_t)w * G + g) * LDR + HD]);
    float sum = 0.f, ll = 0.f;
    if (mx != -INFINITY) {
#pragma unroll
      for (int w = 0; w < kDsWarps; ++w) {
        const float* r = sred + ((size_t)w * G + g) * LDR;
        const float wt = exp2f(r[HD] - mx);
        sum += r[dim] * wt;
        ll += r[HD + 1] * wt;
      }
    }
    if (ns == 1) {  // the only split: this is the attention output
      ds_put(attn, b, (h * G + g) * HD + dim, tag, ll > 0.f ? sum / ll : 0.f);
    } else {
      const size_t at = (((size_t)b * p.H + h * G + g) * part.most + s) * LDR;
      ds_put_part(part, at + dim, tag, sum);  // un-normalised: sum_t 2^(s_t - mx) v_t
      if (dim == 0) {
        ds_put_part(part, at + HD, tag, mx);
        ds_put_part(part, at + HD + 1, tag, ll);
      }
    }
  }
  ds_sync();  // the scratch is written again by what comes next
}
// split s of ns merges its part of the head group's outputs
template <int HD>
SSDK_DEVINL void ds_attention_merge(const DsParams& p, int b, int h, int s, int ns, uint32_t tag, const DsVec& attn, const DsPartial& part, const DsWait& wait) {
  constexpr int LDR = HD + 2;
  const int G = p.H / p.KV, per = (G * HD + ns - 1) / ns;
  for (int idx = s * per + ds_tid(); idx < min(G * HD, (s + 1) * per); idx += kDsConsumers) {
    const int g = idx / HD, dim = idx % HD;
    const size_t at = ((size_t)b * p.H + h * G + g) * part.most * LDR;
    float mx = -INFINITY, o = 0.f, l = 0.f;
    for (int q0 = 0; q0 < ns; q0 += 4) {   // (four splits' requests in flight)
      unsigned long long w[12];   // (sums, maximum, sum of weights of each; splits that the context has not: the last one's again)
      auto ask = [&](int i) { return ds_ask_part(part, at + (size_t)min(q0 + (i & 3), ns - 1) * LDR + (i < 4 ? HD : (i < 8 ? HD + 1 : dim)), tag); };
#pragma unroll
      for (int i = 0; i < 12; ++i) w[i] = ask(i);
      const long long c0 = clock64();
      for (;;) {
        bool ok = true;
#pragma unroll
        for (int i = 0; i < 12; ++i) ok = ok && (uint32_t)(w[i] >> 32) == tag;
        if (ok || wait.give_up(c0)) break;
#pragma unroll
        for (int i = 0; i < 12; ++i)
          if ((uint32_t)(w[i] >> 32) != tag) w[i] = ask(i);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (q0 + i < ns) {
          const float mq = ds_part_value(w[i]), mn = fmaxf(mx, mq), base = mn == -INFINITY ? 0.f : mn;
          const float e0 = exp2f(mx - base), e1 = exp2f(mq - base);
          o = o * e0 + ds_part_value(w[8 + i]) * e1;
          l = l * e0 + ds_part_value(w[4 + i]) * e1;
          mx = mn;
        }
      }
    }
    ds_put(attn, b, (h * G + g) * HD + dim, tag, l > 0.f ? o / l : 0.f);
  }
}

// ---------------------------------------------------------------------------------------------
// the stages.  What they share is in shared memory.  `st`: ring slot | ring phase << 8.
// ---------------------------------------------------------------------------------------------
struct DsShared {
  DsParams p;
  DsGeom geom[5];
  DsVec vec[5];             // results of the stages: q|k|v, attention, o, act, down
  DsPartial part;
  int M, shift, staged, dead, broken;
  unsigned slot_bytes;
  uint8_t *sums, *resid, *scratch;
  int tok[kDsMaxBatch];
  int bt[kDsMaxBatch * kDsBtSmem];
  float red[kDsWarps * kDsMaxBatch];
  ArgMax best[kDsWarps * 4];
  uint64_t full[kDsMaxSlots], empty[kDsMaxSlots];
};
enum { DS_VQKV = 0, DS_VATTN = 1, DS_VO = 2, DS_VACT = 3, DS_VDOWN = 4 };
#ifdef SSDK_HOST_EMU
SSDK_DEVINL DsShared& ds_shared() { return *::emu::static_smem<DsShared>(1, 1 << 20); }
#else
__shared__ DsShared ds_shared_mem;
SSDK_DEVINL DsShared& ds_shared() { return ds_shared_mem; }
#endif
// stage `kind` (DS_QKV = A, DS_O = C, DS_GU = D, DS_DOWN = E, DS_HEAD) of layer l, forward f: operands, then this CTA's rows
template <int MT>
SSDK_DEVINL unsigned ds_stage(int kind, int l, int f, uint32_t tag, unsigned st) {
  SSDK_DYN_SMEM(uint8_t, ds_smem);
  DsShared& S = ds_shared();
  const DsWait wait{&S.dead, S.p.timeout};
  const DsGeom g = S.geom[kind];
  const int M = S.M;
  // in: A, head <- E; C <- B; D <- C; E <- D
  const DsVec src = S.vec[kind == DS_O ? DS_VATTN : (kind == DS_GU ? DS_VO : (kind == DS_DOWN ? DS_VACT : DS_VDOWN))];
  const DsVec out = S.vec[kind == DS_O ? DS_VO : (kind == DS_GU ? DS_VACT : (kind == DS_DOWN ? DS_VDOWN : DS_VQKV))];
  const uint8_t* xrow = nullptr;   // the warp's columns of the first token in shared memory: chunk c at + c ck / 4, step j at + 64 j
  int pitch = 0;                   // bytes of a token
  bool direct = false;
  const int tid = ds_tid(), lane = tid & 31;
  if (kind == DS_O || kind == DS_DOWN) {
    if constexpr (MT <= 4) {
      if (MT == 1 || ds_staged(MT, M, g.K)) { xrow = ds_stage_vec<MT>(src, g, M, tag, wait, S.scratch, kind == DS_O); pitch = g.K / kDsWarps * 2 + kDsPad; }   // (one token always fits)
      else direct = true;
    } else {
      direct = true;
    }
  } else {
    const __nv_bfloat16* w = kind == DS_QKV ? S.p.layers[l].in_norm : (kind == DS_GU ? S.p.layers[l].post_norm : S.p.final_norm);
    const bool embed = kind == DS_QKV && l == 0;   // first layer: hidden = norm(embed), residual = embed (models/llama3.py:192-193)
    ds_norm<MT>(embed ? nullptr : &src, S.p.embed, S.p.vocab, S.tok, S.resid, w, S.p.eps, S.p.d, M, kind == DS_QKV ? tag - 1u : tag, wait, S.scratch, S.red);
    xrow = S.scratch + (tid >> 5) * (g.ck >> 2);   // (one chunk)
    pitch = 2 * g.K + kDsPad;
  }
  ds_mark(f, 2 * kind);
  if (direct) ds_sync();   // (in front of the sums: see ds_consume)
  const int m = ds_x_token<MT>(lane), steps = m < M ? g.ck >> 8 : 0;
  xrow += m * pitch + (lane & 3) * 16;
  auto load = [&](int c, DsX<MT>& x) {
    if (MT > 1 && direct) {
      ds_frag_vec<MT>(src, g, c, M, tag, wait, x);
      return;
    }
#pragma unroll
    for (int j = 0; j < 8 / DsX<MT>::kHalf; ++j) {
      const int step = ds_x_step<MT>(lane, j);
      x.v[j] = step < steps ? *reinterpret_cast<const uint4*>(xrow + c * (g.ck >> 2) + step * 64) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  const int tok = (tid >> 3) & (MT - 1);   // the sequence of this thread's sums
  DsSample smp;
  smp.T = 0.f; smp.seed = smp.call_id = 0; smp.row = (uint32_t)tok; smp.logits = nullptr; smp.best = ArgMax{-INFINITY, 0x7fffffff};
  if (kind == DS_HEAD) {
    smp.T = S.p.temp && tok < M ? S.p.temp[tok] : 0.f;
    smp.seed = S.p.dyn ? S.p.dyn[0] : S.p.seed;
    smp.call_id = (S.p.dyn ? S.p.dyn[1] * 16ull : S.p.call_base) + (uint64_t)f;
    if (S.p.logits) smp.logits = S.p.logits + (size_t)f * S.p.logits_ld + (size_t)tok * S.p.logits_seq_ld;
  }
  DsRing ring{ds_smem, S.full, S.empty, (unsigned)S.p.n_slots, S.slot_bytes, st & 0xffu, st >> 8, DsWait{&S.broken, S.p.timeout}};
  ds_consume<MT>(ring, g, kind == DS_GU ? DS_GATED : (kind == DS_HEAD ? DS_LOGITS : DS_ROWS), M, reinterpret_cast<float*>(S.sums), out, tag, load, smp);
  ds_mark(f, 2 * kind + 1);
  if (kind == DS_HEAD && !S.p.logits_only) {   // eight threads of a warp per sequence -> per-CTA best
    ArgMax a = smp.best;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      ArgMax c;
      c.v = __shfl_xor_sync(0xffffffffu, a.v, o);
      c.i = __shfl_xor_sync(0xffffffffu, a.i, o);
      a = argmax_better(a, c);
    }
    if ((tid & 7) == 0) S.best[tid >> 3] = a;   // [tile in the group][sequence]
    ds_sync();
    if (tid < M) {
      ArgMax c = S.best[tid];
      for (int t = 1; t < 32 / MT; ++t) c = argmax_better(c, S.best[MT * t + tid]);
      S.p.samp_partial[(size_t)tid * gridDim.x + blockIdx.x] = c;
    }
  }
  return ring.slot | ring.phase << 8;
}
// B: units of this CTA (pass 0), their merges (pass 1: behind all units of a CTA, since a merge waits for units of other CTAs)
template <int HD>
SSDK_DEVINL void ds_stage_attention(int l, int f, uint32_t tag, int pass) {
  DsShared& S = ds_shared();
  const DsWait wait{&S.dead, S.p.timeout};
  const int M = S.M, KV = S.p.KV;
  for (int u = blockIdx.x; u < M * KV * S.part.most; u += gridDim.x) {
    const int s = u / (M * KV), b = u / KV % M, h = u % KV;
    const int ctx = S.p.ctx0[b] + f + 1, ns = ds_num_splits(ctx, S.part.most);  // tokens visible to this forward, the new one included
    if (s >= ns) continue;
    const DsPages pg{S.p.block_table + (size_t)b * S.p.max_blocks, S.staged ? S.bt + b * kDsBtSmem : nullptr, S.p.block_size, S.shift};
    if (pass == 0) ds_attention_unit<HD>(S.p, l, b, h, s, ns, ctx, tag, S.vec[DS_VQKV], S.vec[DS_VATTN], S.part, pg, wait, S.scratch);
    else if (ns > 1) ds_attention_merge<HD>(S.p, b, h, s, ns, tag, S.vec[DS_VATTN], S.part, wait);
  }
}

// MT: most sequences of the instance (1, 4 or 8)
template <int HD, int MT>
__global__ void __launch_bounds__(kDsThreads, 1) draft_stream_kernel(const __grid_constant__ DsParams p) {
  SSDK_DYN_SMEM(uint8_t, ds_smem);
  DsShared& S = ds_shared();
  const int M = p.batch > 0 ? p.batch : 1;
  const int max_chunk = p.max_chunk > 0 ? p.max_chunk : kDsMaxChunk;
  const unsigned slot_bytes = p.slot_bytes > 0 ? (unsigned)p.slot_bytes : (unsigned)ds_slot_bytes(kDsMaxChunk);
  for (int i = threadIdx.x; i < (int)(sizeof(DsParams) / 4); i += kDsThreads) reinterpret_cast<uint32_t*>(&S.p)[i] = reinterpret_cast<const uint32_t*>(&p)[i];
  const bool staged = p.max_blocks <= kDsBtSmem;
  if (staged)
    for (int i = threadIdx.x; i < M * p.max_blocks; i += kDsThreads) S.bt[i / p.max_blocks * kDsBtSmem + i % p.max_blocks] = p.block_table[i];
  if ((int)threadIdx.x < M) {
    const int64_t t = p.tok_buf[(size_t)threadIdx.x * p.tok_ld];
    S.tok[threadIdx.x] = t >= 0 && t < p.vocab ? (int)t : -1;   // (ids outside the vocabulary: zero rows)
  }
  if (threadIdx.x == 0) {
    trace_mark(TR_MISC);
    ds_geometry(p.d, (p.H + 2 * p.KV) * HD, max_chunk, &S.geom[DS_QKV]);
    ds_geometry(p.H * HD, p.d, max_chunk, &S.geom[DS_O]);
    ds_geometry(p.d, p.ffn, max_chunk, &S.geom[DS_GU]);
    ds_geometry(p.ffn, p.d, max_chunk, &S.geom[DS_DOWN]);
    ds_geometry(p.d, p.vocab, max_chunk, &S.geom[DS_HEAD]);
    for (int i = 0; i < 5; ++i) ds_own_rows(&S.geom[i]);
    // dynamic shared memory: [ring][sums of the tiles][residual rows][normed rows / fragments / attention scratch]
    S.M = M; S.dead = S.broken = 0; S.staged = staged; S.slot_bytes = slot_bytes;
    S.sums = ds_smem + (size_t)p.n_slots * slot_bytes;
    S.resid = S.sums + ds_part_bytes(MT);
    S.scratch = S.resid + (size_t)M * p.d * 2;
    S.shift = -1;
    for (int i = 0; i < 20; ++i)
      if (p.block_size == (1 << i)) S.shift = i;
    const int rows[5] = {(p.H + 2 * p.KV) * HD, p.H * HD, p.d, p.ffn, p.d};   // DS_VQKV ..
    uint32_t* words = p.words;
    for (int i = 0; i < 5; ++i) {
      S.vec[i].words = words;
      S.vec[i].n = rows[i];
      words += (size_t)M * rows[i];
    }
    S.part.words = reinterpret_cast<unsigned long long*>(words);
    S.part.most = ds_max_splits(M, p.KV, (int)gridDim.x);
#ifdef SSDK_HOST_EMU
    if (!p.words) {
      __nv_bfloat16* const plain[5] = {p.vec_qkv, p.vec_attn, p.vec_o, p.vec_act, p.vec_down};
      for (int i = 0; i < 5; ++i) { S.vec[i].words = nullptr; S.vec[i].plain = plain[i]; }
      S.part.words = nullptr; S.part.plain = p.attn_part; S.part.most = kDsSplits;
    }
#endif
    for (int s = 0; s < p.n_slots; ++s) {
      mbar_init(&S.full[s], 1);           // the producer's arrive.expect_tx + the copies' transaction bytes
      mbar_init(&S.empty[s], kDsWarps);   // one arrive per consumer warp
    }
    fence_mbar_init();
  }
  __syncthreads();  // the only block-wide barrier: mbarriers and the shared state exist before anybody uses them

  if (threadIdx.x >= kDsConsumers) {
    reg_dec<kDsRegsProducer>();
    if (threadIdx.x >= kDsConsumers + 32) return;
    // ===================== producer warp: the weight stream never waits for a stage =====================
    DsProducer r{ds_smem, S.full, S.empty, (unsigned)p.n_slots, slot_bytes, 0u, 0u, DsWait{&S.broken, p.timeout}, 0u};
    ds_producer<MT>(p, S.geom, r);
    return;
  }

  // ===================== consumer warps =====================
  reg_inc<kDsRegsConsumer>();
  const DsWait wait{&S.dead, p.timeout};
  DsGridBar bar;
  bar.counter = reinterpret_cast<unsigned long long*>(p.bar_state);
  bar.target = 0;
  bar.init();
#ifdef SSDK_HOST_EMU
  if (p.words)
#endif
  {
    const long long n = ds_words(M, p.d, p.H, p.KV, HD, p.ffn, (int)gridDim.x) / 4;   // (vectors of whole 8 words, partial results of whole four)
    for (long long i = (long long)blockIdx.x * kDsConsumers + threadIdx.x; i < n; i += (long long)gridDim.x * kDsConsumers)
      reinterpret_cast<uint4*>(p.words)[i] = make_uint4(0u, 0u, 0u, 0u);
  }
#ifdef SSDK_HOST_EMU
  auto meet = [&] { if (!p.words) bar.sync(wait); };   // (the product exchanges by tags alone)
#else
  auto meet = [] {};
#endif
  unsigned st = 0u;
  uint32_t tag = 0u;
  bar.sync(wait);

  for (int f = 0; f < p.n_fwd; ++f) {
    if (threadIdx.x == 0 && f > 0) trace_mark(TR_MISC);
    const int stages = 4 * p.L + (ds_has_head(p, f) ? 1 : 0);
#pragma unroll 1
    for (int i = 0; i < stages; ++i) {   // layer i / 4: q|k|v, attention and o, gate|up, down; last the head (final add + norm, models/llama3.py:198)
      const int l = i >> 2, kind = l < p.L ? i & 3 : DS_HEAD;
      if (kind == DS_QKV) ++tag;
      if (kind == DS_O) {
        ds_stage_attention<HD>(l, f, tag, 0);
        meet();
        ds_stage_attention<HD>(l, f, tag, 1);
        ds_mark(f, 10);
        meet();
      }
      st = ds_stage<MT>(kind, l, f, tag, st);
      if (kind != DS_HEAD) meet();
    }
    if (!ds_has_head(p, f) || p.logits_only) break;
    bar.sync(wait);
    if ((int)(threadIdx.x >> 5) < M) {   // device-wide reduction: every CTA learns the tokens
      const int b = threadIdx.x >> 5;
      ArgMax a{-INFINITY, 0x7fffffff};
      for (int i = threadIdx.x & 31; i < (int)gridDim.x; i += 32) {
        ArgMax q;
        q.v = __ldcg(&p.samp_partial[(size_t)b * gridDim.x + i].v);
        q.i = __ldcg(&p.samp_partial[(size_t)b * gridDim.x + i].i);
        a = argmax_better(a, q);
      }
      a = warp_argmax(a);
      if ((threadIdx.x & 31) == 0) {
        const int t = min(max(a.i, 0), p.vocab - 1);   // (logits that are all NaN have no best; behind a wait that ran out there may be anything)
        S.tok[b] = t;
        if (blockIdx.x == 0) p.tok_buf[(size_t)b * p.tok_ld + f + 1] = t;
      }
    }
    ds_sync();
  }
}

}  // namespace ssdk
