// Runs the SOURCE of csrc/draft_stream.cuh on host threads (cuda_emu.h) with the exchange that the product uses (tagged words instead of barriers), for a
// batch of sequences.  TEST INFRASTRUCTURE.
//   run_draft_words <input blob> <output blob>
//   run_draft_words <input blob> <output blob> words|copies <n>   in the first of two launches the last CTA's words, or copies of weights, are lost from the n-th on
//   run_draft_words registers        the launches that the kernel's register split is for
//   run_draft_words pieces           the attention's weights against the sum of their pieces
// blob layout: see tests/test_draft_words_emu_cpu.py (the writer).
#include "cuda_emu.h"
#define SSDK_HOST_EMU 1
#include "../../ssd_b200/csrc/draft_stream.cuh"

#include <fstream>
#include <iostream>
#include <string>

using bf16 = __nv_bfloat16;

struct Reader {
  std::ifstream f;
  explicit Reader(const char* p) : f(p, std::ios::binary) {}
  template <typename T>
  std::vector<T> vec(size_t n) {
    std::vector<T> v(n);
    f.read(reinterpret_cast<char*>(v.data()), (std::streamsize)(n * sizeof(T)));
    if (!f) {
      std::cerr << "short read\n";
      std::exit(2);
    }
    return v;
  }
  int i32() { return vec<int32_t>(1)[0]; }
};

static int check_pieces() {
  uint32_t x = 12345u;
  for (int i = 0; i < 1000000; ++i) {
    float p[2];
    for (float& v : p) {
      x = x * 1664525u + 1013904223u;
      v = std::exp2((float)-(int)(x >> 25)) * (1.0f + (float)(x & 0x7fffffu) * 0x1p-23f);   // all mantissas, 2^-127 .. 2
      if (v > 1.0f) v *= 0.5f;
    }
    uint32_t w[3];
    ssdk::ds_pieces(p[0], p[1], w);
    for (int h = 0; h < 2; ++h) {
      double sum = 0;
      for (uint32_t q : w) sum += (double)ssdk::ds_bits_f(h ? q >> 16 : q & 0xffffu);
      if (std::abs(sum - (double)p[h]) > 0x1p-133) {   // (below that a bf16 has no bits)
        std::cerr << "weight " << p[h] << " is " << sum << "\n";
        return 1;
      }
    }
  }
  return 0;
}

int main(int argc, char** argv) {
  if (argc == 2 && std::string(argv[1]) == "pieces") return check_pieces();
  if (argc == 2 && std::string(argv[1]) == "registers") {   // the numbers of registers that a build may have, up to what a thread can have
    for (int regs = 0; regs <= 255; ++regs)
      if (ssdk::ds_registers_fit(regs)) std::cout << regs << "\n";
    return 0;
  }
  if (argc != 3 && argc != 5) return 2;
  const bool lose = argc == 5;
  Reader r(argv[1]);
  const int B = r.i32(), d = r.i32(), L = r.i32(), H = r.i32(), KV = r.i32(), hd = r.i32(), ffn = r.i32(), vocab = r.i32();
  const int qk_norm = r.i32(), block_size = r.i32(), max_blocks = r.i32(), nslots = r.i32(), n_fwd = r.i32(), grid = r.i32(), max_pos = r.i32(), ring = r.i32(), max_chunk = r.i32();
  const float eps = r.vec<float>(1)[0];
  auto temps = r.vec<float>(B);
  auto rng = r.vec<uint64_t>(2);
  auto first = r.vec<int64_t>(B);
  auto ctx = r.vec<int32_t>(B);
  auto table = r.vec<int32_t>((size_t)B * max_blocks);
  auto embed = r.vec<bf16>((size_t)vocab * d), final_norm = r.vec<bf16>(d), lm_head = r.vec<bf16>((size_t)vocab * d);
  auto rope = r.vec<float>((size_t)max_pos * hd);
  struct LW { std::vector<bf16> w[8]; };
  std::vector<LW> lw(L);
  for (auto& w : lw) {
    const size_t n[8] = {(size_t)(H + 2 * KV) * hd * d, (size_t)d * H * hd, (size_t)2 * ffn * d, (size_t)d * ffn, (size_t)d, (size_t)d, (size_t)hd, (size_t)hd};
    for (int i = 0; i < 8; ++i) w.w[i] = r.vec<bf16>(n[i]);
  }
  const size_t cache_layer = (size_t)nslots * KV * hd;
  auto kc = r.vec<bf16>(cache_layer * L), vc = r.vec<bf16>(cache_layer * L);

  std::vector<bf16> logits((size_t)B * n_fwd * vocab);
  std::vector<ssdk::ArgMax> partial((size_t)B * grid);
  std::vector<int64_t> tok((size_t)B * (n_fwd + 1), -1);
  const long long nw = ssdk::ds_words(B, d, H, KV, hd, ffn, grid);
  std::vector<uint32_t> store((size_t)nw + 16, 0xffffffffu);   // (whatever another launch left there)
  uint32_t* words = store.data();
  while ((uintptr_t)words & 31) ++words;
  alignas(8) unsigned sync[2] = {0};
  const int MT = B == 1 ? 1 : (B <= 4 ? 4 : 8);
  size_t scratch = std::max((size_t)B * (2 * d + ssdk::kDsPad), ssdk::ds_attn_bytes(H / KV, hd));
  for (int K : {H * hd, ffn})
    if (ssdk::ds_staged(MT, B, K)) scratch = std::max(scratch, ssdk::ds_stage_bytes(B, K));
  const size_t smem = (size_t)ring * ssdk::ds_slot_bytes(max_chunk) + ssdk::ds_part_bytes(MT) + (size_t)B * d * 2 + scratch + 64;

  ssdk::DsParams p;
  std::memset(&p, 0, sizeof(p));
  p.d = d; p.L = L; p.H = H; p.KV = KV; p.ffn = ffn; p.vocab = vocab; p.qk_norm = qk_norm; p.eps = eps;
  p.scale_log2 = (1.0f / std::sqrt((float)hd)) * 1.4426950408889634f;
  p.embed = embed.data(); p.final_norm = final_norm.data(); p.lm_head = lm_head.data(); p.rope = rope.data();
  p.k_cache = kc.data(); p.v_cache = vc.data(); p.cache_layer_stride = (long long)cache_layer;
  p.block_size = block_size; p.max_blocks = max_blocks;
  p.tok_buf = tok.data(); p.tok_ld = n_fwd + 1; p.n_fwd = n_fwd; p.skip_last_head = 1;
  p.ctx0 = ctx.data(); p.block_table = table.data();
  p.logits = logits.data(); p.logits_ld = vocab; p.logits_seq_ld = (long long)n_fwd * vocab;
  p.temp = temps.data(); p.seed = rng[0]; p.call_base = rng[1];
  p.samp_partial = partial.data(); p.bar_state = sync;
  p.n_slots = ring; p.batch = B; p.max_chunk = max_chunk; p.slot_bytes = ssdk::ds_slot_bytes(max_chunk); p.words = words;
  for (int l = 0; l < L; ++l)
    p.layers[l] = ssdk::DsLayer{lw[l].w[0].data(), lw[l].w[1].data(), lw[l].w[2].data(), lw[l].w[3].data(), lw[l].w[4].data(), lw[l].w[5].data(), lw[l].w[6].data(), lw[l].w[7].data()};
  unsigned gave_up = 0;
  p.timeout = &gave_up;
  for (int rep = 0; rep < 2; ++rep) {   // a second launch finds the words and tags of the first
    if (lose) {
      ssdk::ds_wait_cycles = rep == 0 ? 1000000000LL : 4000000000000LL;   // half a second
      (std::string(argv[3]) == "words" ? emu::lost_words : emu::lost_copies) = rep == 0 ? std::atoi(argv[4]) : -1;
    }
    for (int b = 0; b < B; ++b) {
      std::fill(tok.begin() + (size_t)b * (n_fwd + 1), tok.begin() + (size_t)(b + 1) * (n_fwd + 1), -1);
      tok[(size_t)b * (n_fwd + 1)] = first[b];
    }
#define RUN(HD, T) emu::launch(ssdk::draft_stream_kernel<HD, T>, p, grid, ssdk::kDsThreads, smem)
    if (hd == 64) { if (MT == 1) RUN(64, 1); else if (MT == 4) RUN(64, 4); else RUN(64, 8); }
    else { if (MT == 1) RUN(128, 1); else if (MT == 4) RUN(128, 4); else RUN(128, 8); }
    unsigned long long arrivals;
    std::memcpy(&arrivals, sync, 8);
    if (arrivals % (unsigned long long)grid != 0) {
      std::cerr << "barrier arrival counter is not a whole number of barriers\n";
      return 3;
    }
    if (gave_up != (lose && rep == 0 ? 1u : 0u)) {
      std::cerr << (gave_up ? "a wait ran out\n" : "no wait ran out\n");
      return 3;
    }
    gave_up = 0;
    for (int b = 0; b < B; ++b)
      for (int f = 1; f < n_fwd; ++f)
        if (tok[(size_t)b * (n_fwd + 1) + f] < 0 || tok[(size_t)b * (n_fwd + 1) + f] >= vocab) {
          std::cerr << "token out of range\n";
          return 3;
        }
  }
  std::ofstream o(argv[2], std::ios::binary);
  o.write(reinterpret_cast<const char*>(logits.data()), (std::streamsize)(logits.size() * 2));
  o.write(reinterpret_cast<const char*>(kc.data()), (std::streamsize)(kc.size() * 2));
  o.write(reinterpret_cast<const char*>(vc.data()), (std::streamsize)(vc.size() * 2));
  o.write(reinterpret_cast<const char*>(tok.data()), (std::streamsize)(tok.size() * 8));
  return 0;
}
