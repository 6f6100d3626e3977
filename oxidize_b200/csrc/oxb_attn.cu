// liboxb, paged attention entry points.
#include "common.cuh"
#include "attention.cuh"
#include "attention_prefill.cuh"
using namespace oxb;

// ----------------------------------------------------------------------------- attention
// Sizes of the split-KV scratch for a launch shape (floats).
OXB_API int oxb_attn_ws_floats(int B, int nkv, int max_mtiles, int n_cta_splits, int hd, size_t* o_floats,
                               size_t* ml_floats) {
  const size_t tasks = (size_t)B * nkv * max_mtiles * n_cta_splits;
  *o_floats = n_cta_splits > 1 ? tasks * 16 * hd : 0;
  *ml_floats = n_cta_splits > 1 ? tasks * 16 * 2 : 0;
  return 0;
}

template <int HD, int MODE, int NR>
static int attn_launch_rows(const AttnArgs& a, const AttnSkip& skip, int B, int G, cudaStream_t stream) {
  constexpr int smem = AttPage<HD, MODE>::SMEM;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(paged_attention_kernel<HD, MODE, NR>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  dim3 grid(a.max_mtiles * a.n_cta_splits, a.nkv, B);
  // (The KV splits of a row tile stay independent CTAs and the last one to finish merges: inside a thread-block
  // cluster every CTA would wait for the slowest split.)
  if (a.n_cta_splits > 1 && (a.ws_o == nullptr || a.ws_ml == nullptr || a.counters == nullptr)) return (int)cudaErrorInvalidValue;
  oxb_launch(paged_attention_kernel<HD, MODE, NR>, grid, dim3(ATT_WARPS * 32), (size_t)smem, stream, a, G, skip);
  OXB_CHECK_LAUNCH();
  return 0;
}

template <int HD, int MODE = 0>
static int attn_launch(const AttnArgs& a, const AttnSkip& skip, int B, int G, int max_query_len, cudaStream_t stream) {
  if constexpr (HD == 64 || HD == 128) {
    if (max_query_len * G <= 8) return attn_launch_rows<HD, MODE, 1>(a, skip, B, G, stream);
  }
  return attn_launch_rows<HD, MODE, 2>(a, skip, B, G, stream);
}

// skip (host, skip_words words, or null): bit b of it leaves sequence b alone, whose rows are another kernel's (max_query_len: of the
// others).
OXB_API int oxb_paged_attention(const void* q, void* out, const void* kv_data, const float* kv_scales,
                                const int* block_tables, const int* seq_lens, const int* query_start, int B,
                                int max_blocks, int nq, int nkv, int hd, int kv_mode, int max_query_len,
                                int n_cta_splits, int window, float scale, float softcap, const float* sink, int ld_out,
                                float out_scale, float* ws_o, float* ws_ml, int* counters, int num_blocks,
                                const void* gate, int ld_gate, int gate_per_value, const uint32_t* skip_bits, int skip_words,
                                cudaStream_t stream) {
  if (B <= 0) return 0;
  if (nq % nkv != 0 || (gate != nullptr && gate_per_value && (ld_gate % 2 != 0 || (reinterpret_cast<uintptr_t>(gate) & 3) != 0)))
    return (int)cudaErrorInvalidValue;
  AttnSkip skip;
  skip.any = skip_bits != nullptr && skip_words > 0;
  if (skip.any && (skip_words > ATT_SKIP_WORDS || B > 32 * skip_words)) return (int)cudaErrorInvalidValue;
  for (int i = 0; i < ATT_SKIP_WORDS; ++i) skip.bits[i] = skip.any && i < skip_words ? skip_bits[i] : 0;
  const int G = nq / nkv;
  AttnArgs a;
  a.q = reinterpret_cast<const __nv_bfloat16*>(q);
  a.out = reinterpret_cast<__nv_bfloat16*>(out);
  a.kv_data = kv_data;
  a.kv_scales = kv_scales;
  a.block_tables = block_tables;
  a.seq_lens = seq_lens;
  a.query_start = query_start;
  a.max_blocks = max_blocks;
  a.nq = nq;
  a.nkv = nkv;
  a.kv_mode = kv_mode;
  a.n_cta_splits = n_cta_splits < 1 ? 1 : n_cta_splits;
  a.max_mtiles = (max_query_len * G + 15) / 16;
  a.window = window;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.cap_log2 = softcap > 0.f ? softcap * 1.4426950408889634f : 0.f;
  a.cap_arg = softcap > 0.f ? scale / softcap : 0.f;
  a.sink = sink;
  a.ld_out = ld_out;
  a.out_scale = out_scale;
  a.gate = HeadGate{gate, ld_gate, gate_per_value};
  a.ws_o = ws_o;
  a.ws_ml = ws_ml;
  a.counters = counters;
  a.num_blocks = num_blocks;
  a.trace = g_oxb_attn_trace;
  if (kv_mode == 2 && hd == 128) return attn_launch<128, 2>(a, skip, B, G, max_query_len, stream);
  if (kv_mode == 2 && hd == 64) return attn_launch<64, 2>(a, skip, B, G, max_query_len, stream);
  if (kv_mode == 3 && hd == 128) return attn_launch<128, 3>(a, skip, B, G, max_query_len, stream);
  if (kv_mode == 3 && hd == 64) return attn_launch<64, 3>(a, skip, B, G, max_query_len, stream);
  if (hd == 128) return attn_launch<128>(a, skip, B, G, max_query_len, stream);
  if (hd == 64) return attn_launch<64>(a, skip, B, G, max_query_len, stream);
  if (kv_mode != 0) return (int)cudaErrorInvalidValue;
  if (hd == 32) return attn_launch<32>(a, skip, B, G, max_query_len, stream);
  if (hd == 96) return attn_launch<96>(a, skip, B, G, max_query_len, stream);
  if (hd == 192) return attn_launch<192>(a, skip, B, G, max_query_len, stream);
  if (hd == 256) return attn_launch<256>(a, skip, B, G, max_query_len, stream);
  return (int)cudaErrorInvalidValue;
}

// ----------------------------------------------------------------------------- long portions
template <int HD>
static int prefill_convert(int mode, const void* kv_data, const float* kv_scales, const int* block_tables, const int* seq_lens,
                           const int* query_start, int max_blocks, int num_blocks, int nkv, int window, const AttnPrefillSeqs& ls,
                           __nv_bfloat16* pages, cudaStream_t stream) {
  const uint8_t* src = reinterpret_cast<const uint8_t*>(kv_data);
  const dim3 grid(ls.first_page[ls.n] - ls.first_page[0], nkv), block(256);
  auto go = [&](auto kernel) {
    return oxb_launch(kernel, grid, block, 0, stream, src, kv_scales, query_start, seq_lens, block_tables, max_blocks, num_blocks, nkv,
                      window, ls, pages);
  };
  const cudaError_t e = mode == 1 ? go(prefill_pages_kernel<HD, 1>) : mode == 2 ? go(prefill_pages_kernel<HD, 2>) : go(prefill_pages_kernel<HD, 3>);
  if (e != cudaSuccess) return (int)e;
  OXB_CHECK_LAUNCH();
  return 0;
}

template <int HD>
static int prefill_launch(const void* q, const void* pages, const AttnPrefillArgs& a, const AttnPrefillSeqs& ls, int T, int nq,
                          cudaStream_t stream) {
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
  if (!configured[dev]) {
    const cudaError_t e =
        cudaFuncSetAttribute(paged_prefill_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, attn_prefill_smem<HD>());
    if (e != cudaSuccess) return (int)e;
    configured[dev] = true;
  }
  CUtensorMap tq, tkv;
  const uint64_t qs[3] = {(uint64_t)HD, (uint64_t)nq, (uint64_t)T}, qb[2] = {(uint64_t)HD * 2, (uint64_t)nq * HD * 2};
  const uint32_t box[3] = {64, (uint32_t)a.gp, (uint32_t)(AP_M / a.gp)};
  int e = oxb_make_tmap_3d(&tq, q, qs, qb, box);
  if (e) return e;
  e = oxb_make_tmap_2d(&tkv, pages, (uint64_t)a.num_blocks * a.nkv * 2 * ATT_PAGE, HD, (uint64_t)HD * 2, ATT_PAGE, 64, 2);
  if (e) return e;
  const dim3 grid(ls.first_item[ls.n], nq / a.gp);
  const cudaError_t le = oxb_launch(paged_prefill_kernel<HD>, grid, dim3(AP_THREADS), (size_t)attn_prefill_smem<HD>(), stream, tq, tkv, a, ls);
  if (le != cudaSuccess) return (int)le;
  OXB_CHECK_LAUNCH();
  return 0;
}

// 1 when oxb_paged_prefill covers heads of this width and these counts
OXB_API int oxb_paged_prefill_supported(int hd, int nq, int nkv) {
  return (hd == 64 || hd == 128) && nkv > 0 && nq % nkv == 0 && nq <= 65535;
}

// Attention of some sequences of a step (the others are left alone), arguments as oxb_paged_attention: `count` of them, with their
// index, rows and context length (host arrays; the last two bound the launches, the kernels go by the device's).  scale > 0.
// kv_mode > 0: `pages` [cap_pages, nkv, 2, 16, hd] bf16 receives the pages that their rows see, decoded.
OXB_API int oxb_paged_prefill(const void* q, void* out, const void* kv_data, const float* kv_scales, const int* block_tables,
                              const int* seq_lens, const int* query_start, int T, int max_blocks, int nq, int nkv, int hd,
                              int kv_mode, const int* seqs, const int* rows, const int* ctx, int count, int window, float scale,
                              const float* sink, int ld_out, float out_scale, int num_blocks, const void* gate, int ld_gate,
                              int gate_per_value, void* pages, int cap_pages, cudaStream_t stream) {
  if (count <= 0 || T <= 0) return 0;
  if (!oxb_paged_prefill_supported(hd, nq, nkv) || kv_mode < 0 || kv_mode > 3 || ld_out % 2 != 0 || !(scale > 0.f) ||
      (kv_mode > 0 && pages == nullptr) ||
      (gate != nullptr && gate_per_value && (ld_gate % 2 != 0 || (reinterpret_cast<uintptr_t>(gate) & 3) != 0)))
    return (int)cudaErrorInvalidValue;
  AttnPrefillArgs a;
  a.query_start = query_start;
  a.seq_lens = seq_lens;
  a.block_tables = kv_mode > 0 ? nullptr : block_tables;
  a.sink = sink;
  a.out = reinterpret_cast<__nv_bfloat16*>(out);
  a.max_blocks = max_blocks;
  a.num_blocks = kv_mode > 0 ? cap_pages : num_blocks;
  a.nkv = nkv;
  a.G = nq / nkv;
  a.gp = 1;
  while (a.gp < AP_M && a.G % (2 * a.gp) == 0) a.gp *= 2;  // the largest power of two that divides the group
  a.window = window;
  a.ld_out = ld_out;
  a.out_scale = out_scale;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.gate = HeadGate{gate, ld_gate, gate_per_value};
  const int tok_per_cta = 2 * AP_M / a.gp;
  __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(pages);
  const void* src = kv_mode > 0 ? pages : kv_data;
  int page = 0;  // of the buffer
  for (int at = 0; at < count; at += AP_SEQS) {
    AttnPrefillSeqs ls;
    ls.n = count - at < AP_SEQS ? count - at : AP_SEQS;
    int item = 0;
    for (int i = 0; i <= AP_SEQS; ++i) {  // (entries past the last sequence repeat the ends)
      ls.first_item[i] = item;
      ls.first_page[i] = page;
      if (i == AP_SEQS) break;
      ls.seq[i] = 0;
      if (i >= ls.n) continue;
      const int n = rows[at + i], c = ctx[at + i];
      if (n <= 0 || c < n) return (int)cudaErrorInvalidValue;
      ls.seq[i] = seqs[at + i];
      item += (n + tok_per_cta - 1) / tok_per_cta;
      if (kv_mode > 0) page += (c + ATT_PAGE - 1) / ATT_PAGE - prefill_first_page(n, c, window);
    }
    if (kv_mode > 0) {
      if (page > cap_pages) return (int)cudaErrorInvalidValue;
      const int e = hd == 128 ? prefill_convert<128>(kv_mode, kv_data, kv_scales, block_tables, seq_lens, query_start, max_blocks, num_blocks,
                                                     nkv, window, ls, dst, stream)
                              : prefill_convert<64>(kv_mode, kv_data, kv_scales, block_tables, seq_lens, query_start, max_blocks, num_blocks,
                                                    nkv, window, ls, dst, stream);
      if (e) return e;
    }
    const int e = hd == 128 ? prefill_launch<128>(q, src, a, ls, T, nq, stream) : prefill_launch<64>(q, src, a, ls, T, nq, stream);
    if (e) return e;
  }
  return 0;
}
