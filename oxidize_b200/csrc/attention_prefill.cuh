// Paged grouped-query attention for long portions of prompts: flash attention on tcgen05 over the cache's own pages.
//
// paged_attention_kernel gives a warp 16 query rows, so every 16 rows read the whole context from the L2 again and the
// products run as mma.sync: at 2048 rows over a context of 14000 it reached 0.14 PFLOP/s (3690 us, 32 query heads of width
// 128, 8 key heads; here 647 us, 0.78 PFLOP/s).  Here a CTA owns 256 rows: a row is a (token, query head) pair and the rows of `gp`
// heads that share a key head lie together, so that a short portion still fills the tile and what a causal mask wastes is a few
// tokens.  They are two tiles of 128 rows: S = Q K^T (N = 64 keys) goes to tensor memory, a warpgroup per tile does the softmax with
// one thread per row and writes P back to tensor memory as the A operand of O += P V (V read MN-major).  The tiles alternate on the
// tensor core, so one's softmax runs under the other's products, and S is double-buffered, so a tile's softmax never waits for its
// own.
//
// P goes in as two bf16 numbers, its rounding and the remainder.  One alone was no more exact than the kernel above (in fact 3 to
// 10 % less against 64 bits, as that one keeps a running maximum per 16 keys and the largest probabilities are exactly 1); with the
// remainder the error is that of the bf16 output alone, and the running maximum can lag, which saves most rescales of O.  Per 64
// keys and 256 rows that is 1790 cycles of products (768 of them S: an MMA of 64 columns takes 48) against about 1000 of exponentials.
//
// A page of 16 rows of one head is a contiguous 16-row box of the cache seen as a matrix of rows, which is what TMA loads;
// sixteen rows are two of the 128-byte swizzle's eight-row groups, so four boxes make the tile that the tensor core reads.
// f16 and quantized pages are converted to bf16 pages first (prefill_pages_kernel), each once per layer.
#pragma once
#include "attention.cuh"

namespace oxb {

constexpr int AP_KEYS = 64, AP_M = 128, AP_STAGES = 4, AP_PAGES = AP_KEYS / ATT_PAGE;
constexpr int AP_QCHUNK = AP_M * 128, AP_KCHUNK = AP_KEYS * 128;  // bytes of a 64-value column chunk
constexpr float AP_LAZY = 8.f;  // log2 of the factor by which scores may exceed the running maximum
constexpr int AP_WARP_TMA = 8, AP_WARP_MMA = 9, AP_THREADS = 320;

struct AttnPrefillArgs {
  const int* query_start;   // [B + 1]
  const int* seq_lens;      // [B]
  const int* block_tables;  // [.., max_blocks], or null: pages converted by prefill_pages_kernel
  const float* sink;        // [nq] or null
  __nv_bfloat16* out;       // [T, nq * HD], rows ld_out apart
  int max_blocks, num_blocks, nkv, G, gp, window, ld_out;
  float out_scale, scale_log2;
  HeadGate gate;
};

// The sequences of a launch, as the host knows them: a step's others cost it nothing.  (A grid of the longest portion's tiles times
// all sequences is mostly CTAs without work where a portion runs among decoding sequences: one of 4096 tokens of context and 63 of
// those, 32 key heads, q8, had 524288 CTAs convert 8192 pages.)
constexpr int AP_SEQS = 64;
struct AttnPrefillSeqs {
  int n;
  int seq[AP_SEQS];             // index in the step
  int first_item[AP_SEQS + 1];  // of its row tiles in the launch
  int first_page[AP_SEQS + 1];  // of its converted pages in the buffer
};

// Where a value lies in ascending starts[0 .. n] (starts[0] <= v < starts[n])
__device__ __forceinline__ int prefill_find(const int (&starts)[AP_SEQS + 1], int n, int v) {
  int i = 0;
  while (i + 1 < n && starts[i + 1] <= v) ++i;
  return i;
}
// First page that any row of a sequence sees
__host__ __device__ __forceinline__ int prefill_first_page(int rows, int ctx, int window) {
  const int key = ctx - rows - window + 1;
  return window > 0 && key > 0 ? key / ATT_PAGE : 0;
}

// f16 / q8 / q4 pages of the launch's sequences as bf16 pages, a CTA for every page and head: out [pages, nkv, K | V, 16, HD].
template <int HD, int MODE>
static __global__ void __launch_bounds__(256)
prefill_pages_kernel(const uint8_t* __restrict__ cache, const float* __restrict__ scales, const int* __restrict__ query_start,
                     const int* __restrict__ seq_lens, const int* __restrict__ block_tables, int max_blocks, int num_blocks, int nkv,
                     int window, const __grid_constant__ AttnPrefillSeqs ls, __nv_bfloat16* __restrict__ out) {
  pdl_launch_dependents();
  pdl_wait();
  const int dst_page = ls.first_page[0] + blockIdx.x, at = prefill_find(ls.first_page, ls.n, dst_page), b = ls.seq[at];
  const int len = seq_lens[b];
  const int page = prefill_first_page(query_start[b + 1] - query_start[b], len, window) + dst_page - ls.first_page[at];
  if (page * ATT_PAGE >= len || page >= max_blocks) return;
  int blk = block_tables[(size_t)b * max_blocks + page];
  if ((unsigned)blk >= (unsigned)num_blocks) {
    if (threadIdx.x == 0) oxb_report(OXB_BAD_BLOCK_ID, blk);
    blk = 0;
  }
  const int rows = 2 * ATT_PAGE;  // of this head
  const size_t row0 = ((size_t)blk * nkv + blockIdx.y) * rows;
  __nv_bfloat16* o = out + ((size_t)dst_page * nkv + blockIdx.y) * rows * HD;
  for (int c = threadIdx.x; c < rows * (HD / 8); c += 256) {  // 8 values
    const int row = c / (HD / 8), col = (c % (HD / 8)) * 8;
    float v[8];
    if constexpr (MODE == 1) {
      const uint4 raw = *reinterpret_cast<const uint4*>(cache + ((row0 + row) * HD + col) * 2);
      const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
        v[2 * j] = f.x;
        v[2 * j + 1] = f.y;
      }
    } else {
      const float s = scales[(row0 + row) * (HD / 32) + (col >> 5)];
      if constexpr (MODE == 2) {
        const uint2 w = *reinterpret_cast<const uint2*>(cache + (row0 + row) * HD + col);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[j] = ((float)((w.x >> (8 * j)) & 0xFF) - 127.f) * s;
          v[4 + j] = ((float)((w.y >> (8 * j)) & 0xFF) - 127.f) * s;
        }
      } else {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(cache + (row0 + row) * (HD / 2) + (col >> 1));
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = ((float)((w >> (4 * j)) & 0xF) - 7.f) * s;
      }
    }
    *reinterpret_cast<uint4*>(o + (size_t)row * HD + col) =
        make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
  }
}

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* d, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(d)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

template <int HD>
constexpr int attn_prefill_smem() {
  return 2 * (HD / 64) * AP_QCHUNK + 2 * AP_STAGES * (HD / 64) * AP_KCHUNK + 1024;
}

template <int HD>
__global__ void __launch_bounds__(AP_THREADS, 1)
paged_prefill_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV, const AttnPrefillArgs a,
                     const __grid_constant__ AttnPrefillSeqs ls) {
  constexpr int CH = HD / 64;
  extern __shared__ uint8_t ap_raw[];
  __shared__ uint64_t q_full, k_full[AP_STAGES], k_empty[AP_STAGES], v_full[AP_STAGES], v_empty[AP_STAGES], s_full[2][2],
      p_full[2][2], pv_done[2];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int at = prefill_find(ls.first_item, ls.n, blockIdx.x), b = ls.seq[at], h0 = blockIdx.y * a.gp;  // first query head of this CTA
  const int kvh = h0 / a.G;
  const int q0 = a.query_start[b], qlen = a.query_start[b + 1] - q0;
  const int tok_per = AP_M / a.gp;  // tokens of a tile
  // (the last rows have the longest way to go: they start first)
  const int m0 = (ls.first_item[at + 1] - 1 - (int)blockIdx.x) * 2 * tok_per;
  const int seq_len = a.seq_lens[b];
  if (m0 >= qlen || seq_len < qlen) {
    pdl_wait();
    return;
  }
  const int pos0 = seq_len - qlen + m0;                          // position of the first row
  const int hi = min(pos0 + 2 * tok_per, seq_len) - 1;           // last key of the last row
  const int lo = (a.window > 0 ? max(0, pos0 - a.window + 1) : 0) & ~(AP_KEYS - 1);
  const int tiles = (hi - lo) / AP_KEYS + 1;

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ap_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* s_q = smem;                                    // [2 tiles][CH][128 rows][128 bytes]
  uint8_t* s_k = s_q + 2 * CH * AP_QCHUNK;                // [AP_STAGES][CH][64 keys][128 bytes]
  uint8_t* s_v = s_k + AP_STAGES * CH * AP_KCHUNK;

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    for (int i = 0; i < AP_STAGES; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      for (int j = 0; j < 2; ++j) {
        mbar_init(&s_full[i][j], 1);
        mbar_init(&p_full[i][j], 128);
      }
      mbar_init(&pv_done[i], 1);
    }
    abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == AP_WARP_MMA) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();  // (only now: a CTA of the next kernel must not take the tensor memory that this one still waits for)
  // tensor-memory columns of tile t: S of every other step at 128 t and 128 t + 64, P in its place, O at 256 + 128 t
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
  pdl_wait();

  if (warp == AP_WARP_TMA) {
    const bool leader = elect_one();
    if (leader) {
      mbar_expect_tx(&q_full, 2 * CH * AP_QCHUNK);
      for (int t = 0; t < 2; ++t)
        for (int c = 0; c < CH; ++c)
          tma_load_3d(s_q + (t * CH + c) * AP_QCHUNK, &tmQ, &q_full, c * 64, h0, q0 + m0 + t * tok_per);
    }
    // lane = (page of the tile, column chunk); pages before the first one that a row sees, which a window may have given back
    // and whose table entries mean nothing, and past the last one repeat those (their keys are masked)
    const int pg = lane % AP_PAGES, ch = lane / AP_PAGES;
    const int last_page = (seq_len - 1) / ATT_PAGE, first_page = lo / ATT_PAGE;
    const int first_seen = a.window > 0 ? max(0, pos0 - a.window + 1) / ATT_PAGE : 0;
    const int base = ls.first_page[at] - prefill_first_page(qlen, seq_len, a.window);  // (converted pages)
    auto block_of = [&](int i) {  // cache block of this lane's page in tile i
      const int p = min(max(first_page + i * AP_PAGES + pg, first_seen), last_page);
      return a.block_tables == nullptr ? base + p : a.block_tables[(size_t)b * a.max_blocks + p];
    };
    int next = block_of(0);
    bool ok = true;
    int s = 0;
    uint32_t ph = 1;  // parity of the use of stage s before this one
    for (int i = 0; i < tiles && ok; ++i) {
      int blk = next;
      if (i + 1 < tiles) next = block_of(i + 1);
      if ((unsigned)blk >= (unsigned)a.num_blocks) {  // never follow a bad block id: record it, read page 0
        oxb_report(OXB_BAD_BLOCK_ID, blk);
        blk = 0;
      }
      const int row = (blk * a.nkv + kvh) * 2 * ATT_PAGE;
      if (i >= AP_STAGES) ok = mbar_wait_bounded(&k_empty[s], ph, &abort_flag, OXB_TIMEOUT_TMA_EMPTY, blockIdx.x);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (leader) mbar_expect_tx(&k_full[s], CH * AP_KCHUNK);
      __syncwarp();
      if (ch < CH) tma_load_2d(s_k + (s * CH + ch) * AP_KCHUNK + pg * ATT_PAGE * 128, &tmKV, &k_full[s], ch * 64, row);
      if (i >= AP_STAGES) ok = mbar_wait_bounded(&v_empty[s], ph, &abort_flag, OXB_TIMEOUT_TMA_EMPTY, blockIdx.x);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (leader) mbar_expect_tx(&v_full[s], CH * AP_KCHUNK);
      __syncwarp();
      if (ch < CH) tma_load_2d(s_v + (s * CH + ch) * AP_KCHUNK + pg * ATT_PAGE * 128, &tmKV, &v_full[s], ch * 64, row + ATT_PAGE);
      __syncwarp();
      if (++s == AP_STAGES) {
        s = 0;
        ph ^= 1;
      }
    }
  } else if (warp == AP_WARP_MMA) {
    const bool leader = elect_one();
    constexpr uint32_t idesc_s = umma_idesc_bf16(AP_M, AP_KEYS);
    constexpr uint32_t idesc_o = umma_idesc_bf16(AP_M, HD) | UMMA_B_MN_MAJOR;
    const uint32_t qa = smem_u32(s_q), ka = smem_u32(s_k), va = smem_u32(s_v);
    auto first = [&](int i, int s, int t) {  // S of tile t against keys i, which are in stage s
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const uint32_t qd = umma_desc_lo(qa + (t * CH + c) * AP_QCHUNK), kd = umma_desc_lo(ka + (s * CH + c) * AP_KCHUNK);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16_if<UMMA_DESC_HI_SW128, UMMA_DESC_HI_SW128, idesc_s>(leader, tmem + 128 * t + 64 * (i & 1), qd + 2 * k, kd + 2 * k,
                                                                        k > 0 || c > 0);
      }
      umma_commit_if(leader, &s_full[t][i & 1]);
      if (t == 1) umma_commit_if(leader, &k_empty[s]);
    };
    bool ok = mbar_wait_bounded(&q_full, 0, &abort_flag, OXB_TIMEOUT_TMA_FULL, blockIdx.x) &&
              mbar_wait_bounded(&k_full[0], 0, &abort_flag, OXB_TIMEOUT_TMA_FULL, blockIdx.x);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    if (ok) {
      first(0, 0, 0);
      first(0, 0, 1);
    }
    int s = 0;
    uint32_t ph = 0;
    for (int i = 0; i < tiles && ok; ++i) {
      // The next keys' scores are under way before this step's probabilities are waited for, so the softmax of a tile never
      // waits for its own products.  Their place held P of the step before, which PV of that step, issued earlier, reads first.
      const int s1 = s + 1 == AP_STAGES ? 0 : s + 1;
      const uint32_t ph1 = s1 == 0 ? ph ^ 1 : ph;
      if (i + 1 < tiles) {
        ok = mbar_wait_bounded(&k_full[s1], ph1, &abort_flag, OXB_TIMEOUT_TMA_FULL, blockIdx.x);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        first(i + 1, s1, 0);
        first(i + 1, s1, 1);
      }
      ok = mbar_wait_bounded(&v_full[s], ph, &abort_flag, OXB_TIMEOUT_TMA_FULL, blockIdx.x);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        ok = mbar_wait_bounded(&p_full[t][i & 1], (i >> 1) & 1, &abort_flag, OXB_TIMEOUT_ACCUM, blockIdx.x) && ok;
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t vd = umma_desc_lo(va + s * CH * AP_KCHUNK, AP_KCHUNK);
#pragma unroll
        for (int k = 0; k < 2 * AP_KEYS / 16; ++k)  // 16 keys: 8 columns of P (then of its remainders), 2 KB of the value tile
          umma_bf16_ts_if(leader, tmem + 256 + 128 * t, tmem + 128 * t + 64 * (i & 1) + 8 * k, vd + k % (AP_KEYS / 16) * (2048 >> 4),
                          UMMA_DESC_HI_SW128, idesc_o, i > 0 || k > 0);
        umma_commit_if(leader, &pv_done[t]);
        if (t == 1) umma_commit_if(leader, &v_empty[s]);
      }
      s = s1;
      ph = ph1;
    }
    __syncwarp();
  } else {
    // ---------------- softmax: warpgroup t = tile, thread = row
    const int t = warp >> 2, row = threadIdx.x & 127;
    const int tok = m0 + t * tok_per + row / a.gp, head = h0 + row % a.gp;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_cols = tmem + lanes + 128 * t, o_col = tmem + lanes + 256 + 128 * t;
    const int pos = seq_len - qlen + min(tok, qlen - 1);  // rows past the end repeat the last token; never stored
    const int first_key = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    const int w_lo = __reduce_max_sync(0xffffffffu, first_key), w_hi = __reduce_min_sync(0xffffffffu, pos);  // keys every row sees
    const float sink = a.sink != nullptr ? a.sink[head] * 1.4426950408889634f : -INFINITY;
    float m = sink, l = 0.f;
    for (int i = 0; i < tiles; ++i) {
      // (no early exit on a failed wait: every thread arrives at every barrier, later waits return at once)
      const uint32_t s_col = s_cols + 64 * (i & 1);
      mbar_wait_bounded(&s_full[t][i & 1], (i >> 1) & 1, &abort_flag, OXB_TIMEOUT_ACCUM, blockIdx.x);
      __syncwarp();
      tc_fence_after();
      float s[AP_KEYS];
#pragma unroll
      for (int c = 0; c < AP_KEYS / 16; ++c) tmem_ld16(s_col + 16 * c, reinterpret_cast<uint32_t*>(s) + 16 * c);
      tmem_ld_wait();
      const int key0 = lo + i * AP_KEYS;
      if (key0 < w_lo || key0 + AP_KEYS - 1 > w_hi) {
        const int ka = first_key - key0, kb = pos - key0;
#pragma unroll
        for (int j = 0; j < AP_KEYS; ++j)
          if (j < ka || j > kb) s[j] = -INFINITY;
      }
      float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int j = 4; j < AP_KEYS; ++j) mx[j & 3] = fmaxf(mx[j & 3], s[j]);
      const float tm = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * a.scale_log2;
      // the running maximum moves with the first keys and then only when a score exceeds it by more than 2^8
      const bool move = tm > m + (l == 0.f ? 0.f : AP_LAZY);
      const float m_new = move ? tm : m;
      const float f = move ? exp2f(m - m_new) : 1.f;  // 0 when nothing was accumulated
      m = m_new;
      l *= f;
      const float base = m == -INFINITY ? 0.f : m;
      uint32_t pk[AP_KEYS / 2], pl[AP_KEYS / 2];
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < AP_KEYS; j += 2) {
        const float p0 = exp2f(fmaf(s[j], a.scale_log2, -base)), p1 = exp2f(fmaf(s[j + 1], a.scale_log2, -base));
        sum[j & 2] += p0;
        sum[(j & 2) + 1] += p1;
        const uint32_t hi = pack_bf16x2(p0, p1);
        pk[j >> 1] = hi;
        pl[j >> 1] = pack_bf16x2(p0 - __uint_as_float(hi << 16), p1 - __uint_as_float(hi & 0xFFFF0000u));
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      tmem_st16(s_col, pk);
      tmem_st16(s_col + 16, pk + 16);
      tmem_st16(s_col + 32, pl);
      tmem_st16(s_col + 48, pl + 16);
      // O is complete up to the step before.  (Waited for in every step, moved or not: the barrier's one-bit phase cannot tell
      // steps apart that were passed over.)
      if (i > 0) mbar_wait_bounded(&pv_done[t], (i - 1) & 1, &abort_flag, OXB_TIMEOUT_ACCUM, blockIdx.x);
      __syncwarp();
      tc_fence_after();
      if (i > 0 && __any_sync(0xffffffffu, move)) {
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t o[32];
          tmem_ld16(o_col + 32 * c, o);
          tmem_ld16(o_col + 32 * c + 16, o + 16);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
          tmem_st16(o_col + 32 * c, o);
          tmem_st16(o_col + 32 * c + 16, o + 16);
        }
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&p_full[t][i & 1]);
    }
    mbar_wait_bounded(&pv_done[t], (tiles - 1) & 1, &abort_flag, OXB_TIMEOUT_ACCUM, blockIdx.x);
    __syncwarp();
    tc_fence_after();
    if (sink > -INFINITY) l += exp2f(sink - m);  // the sink's share of the denominator, once
    float inv = l > 0.f ? a.out_scale / l : 0.f;
    const int tok_in = min(tok, qlen - 1);
    if (a.gate.rows != nullptr && !a.gate.per_value)
      inv *= head_gate_of(__bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.gate.rows)[(size_t)(q0 + tok_in) * a.gate.ld + head]));
    __nv_bfloat16* o_row = a.out + (size_t)(q0 + tok) * a.ld_out + head * HD;
#pragma unroll 1
    for (int c = 0; c < HD / 16; ++c) {
      uint32_t o[16];
      tmem_ld16(o_col + 16 * c, o);
      tmem_ld_wait();
      if (tok < qlen) {
        if (a.gate.rows != nullptr && a.gate.per_value) {
          const __nv_bfloat16* gates =
              reinterpret_cast<const __nv_bfloat16*>(a.gate.rows) + (size_t)(q0 + tok) * a.gate.ld + head * HD + 16 * c;
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float2 z = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(gates + j));
            o[j] = __float_as_uint(__uint_as_float(o[j]) * head_gate_of(z.x));
            o[j + 1] = __float_as_uint(__uint_as_float(o[j + 1]) * head_gate_of(z.y));
          }
        }
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = pack_bf16x2(__uint_as_float(o[2 * e]) * inv, __uint_as_float(o[2 * e + 1]) * inv);
        if (a.ld_out % 8 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0) {
          *reinterpret_cast<uint4*>(o_row + 16 * c) = make_uint4(w[0], w[1], w[2], w[3]);
          *reinterpret_cast<uint4*>(o_row + 16 * c + 8) = make_uint4(w[4], w[5], w[6], w[7]);
        } else {  // (rows on 4-byte boundaries, as paged_attention_kernel writes them)
#pragma unroll
          for (int e = 0; e < 8; ++e) *reinterpret_cast<uint32_t*>(o_row + 16 * c + 2 * e) = w[e];
        }
      }
    }
  }
  if (abort_flag) {
    // a wait gave up: give copies that may still be in flight time to land before the CTA exits
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == AP_WARP_MMA) tmem_dealloc(tmem, 512);
}

}  // namespace oxb
