// Paged-KV inference kernels for sm_100a.
//
// KV cache layout (both K and V, per layer):  [num_blocks, block_size, kv_heads, head_dim]  (token-major inside a block,
// 16-byte vectors along head_dim; one (block, head) tile is a strided 2-D box, i.e. directly TMA-addressable).
//
//   cb_kv_cache_write        : scatter this step's K,V rows [tokens, kv_heads, D] into their paged slots (prefill: all
//                              prompt tokens via cu_seqlens; decode: one token per sequence), optional fp8(e5m2) cast
//   cb_paged_decode_attention: split-KV flash-decoding: grid (seq, group of <= 8 kv heads, split); one WARP serves a
//                              kv head (its whole GQA group, so K/V are read once per group) and the warps of a CTA
//                              stream adjacent head slices of the same token rows; fp32 online softmax; second pass
//                              merges splits
//   cb_gather_cos_sin        : per-token cos/sin rows from the [max_pos, D/2] caches
//   cb_convert_fp8           : fp16/bf16/fp32 <-> fp8 e5m2 storage
//
// Capability parity: reference inference_ops_cuda (extensions/csrc/kernel/cuda/{flash_decoding_attention,
// decode_kv_cache_memcpy,context_kv_cache_memcpy,fused_rotary_emb_and_cache,get_cos_and_sin,convert_fp8}_kernel.cu,
// N12-N19) and the Triton twins (kernel/triton/{flash_decoding,kvcache_copy,no_pad_rotary_embedding}.py).
// Decode attention is HBM-bound (every K/V byte is read once): the design goal is full-sector 16-byte loads, many of them
// in flight per SM, and enough CTAs (seqs x kv_heads x splits >= 2 waves of 2 x 148) rather than tensor cores.
#include "common.cuh"

namespace {

constexpr int DEC_THREADS = 256;   // at most 8 (kv head, query-head set) units per CTA
constexpr int MAX_GROUP = 8;   // q heads per kv head handled by one CTA

template <typename T> CB_DEVICE float kv_to_f32(T v) { return to_f32<T>(v); }

// 16-byte asynchronous global -> shared copy; src_bytes < 16 zero-fills the rest (0 = pure zero fill)
CB_DEVICE void cp_async_16(void* smem_dst, const void* gmem_src, uint32_t src_bytes) {
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem_src), "r"(src_bytes) : "memory");
}
CB_DEVICE float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
CB_DEVICE void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> CB_DEVICE void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ---- how a decode step's sequences are cut (cb_decode_num_splits)
// Warps of a CTA, one for each kv head.  Four heads of 128, so that two CTAs fit an SM and one's beginning and end lie under the other's
// loads; all heads of 64 up to eight, four where there are more.  Device time, us, eight / four warps: 64 x 2048 tokens of 32 / 8 heads of 128
// 78.0 / 76.4, 128 x 1024 85.3 / 82.5, 128 x 1024 of 12 heads of 64 62.3 / 56.6, 48 x 2700 of 24 / 8 heads of 64 40.6 / 41.0.  Six heads of 128 in one CTA: 8 x
// 500 9.9 instead of 10.8, but 8 x 2000 18.0 instead of 16.9.
constexpr int DEC_MMA_WARPS = 4;
// Few sequences are cut into as many partitions as run at once, equal ones of each sequence's own length: a second round of CTAs, and twice as
// many partial results to add up, cost more than they balance, and what a table has room for is often several times what is in it.
// Two rounds of what the table holds / one of the length, tables just wide enough, us: 16 x 1024 tokens of 32 / 8 heads of 128 22.6 / 18.2, 16 x 8000
// 86 / 79, 2 x 16000 38.0 / 29.6, 10 x 8000 60.0 / 54.9, 28 x 4000 75.0 / 69.8, 6 x 12000 of 16 / 2 heads of 64 29.1 / 22.4, 60 x 2000 of 16 / 2 heads of 128
// 37.8 / 31.2, 5 x 8000 of 12 heads 50.5 / 43.9; tables of 8192 tokens of which 500 to 1000 are in use, 16 sequences 40.8 / 17, 28 64 / 21.  Four heads gain
// where tables are wide or lengths equal (6 x 8000 34 / 27); 32 to 64 sequences of uneven lengths in tables just wide enough lose 7 to 11 %.
// How many that is at most: decode_most_splits.  Where a round is fewer than DEC_ROUND_SPLITS partitions - lengths differ by more than one - two rounds
// (one / two: 40 x 3000 79.8 / 73.0, 32 x 4000 79.8 / 76.0), unless three or four are of DEC_SHORT / 4 to DEC_SHORT tokens, whose beginnings count for more
// (32 x 1000 26.4 / 28.7, 24 x 1000 of 12 heads 24.7 / 28.1, 64 x 500 of four 16.5 / 19.2, 128 x 1000 of two 25.8 / 29.0; 64 x 2000 of four, parts of 500, 44.6 /
// 45.1).  Where two rounds are as few, and for more than four heads of 64, by what the table holds (64 x 2048 76.9, own 80.3; 30 x 4000 of 24 / 8 heads of 64
// 38.6, own 43.4).
constexpr int DEC_PART_MIN = 64, DEC_ROUND_SPLITS = 5, DEC_MOST_SPLITS = 64, DEC_SHORT_SPLITS = 3, DEC_SHORT = 384;
constexpr int DEC_WIDE = 48;           // partitions from which decode_reduce_wide_kernel adds them up
static inline int decode_warps(int kv_heads, int head_dim) {
  const int most = head_dim == 128 || kv_heads > 8 ? DEC_MMA_WARPS : 8;
  return kv_heads < most ? kv_heads : most;
}
struct DecodeCut {
  const int* seq_lens;
  int capacity, part_len, window;      // tokens that a table has room for
  unsigned per;                        // 2^32 / part_len, rounded up, where that divides what a table has room for; or 0
};
// tokens of a partition: part_len, or, where that is negative, an equal share of the sequence's own, of -part_len at least
CB_DEVICE int decode_partition(int cached, int splits, int part_len) {
  return part_len > 0 ? part_len : max(-part_len, ((cached + splits - 1) / splits + 15) & ~15);
}
// Of a window (`window_start`: its first token, or 0) the tokens in sight are shared out, from here on; they are all that is read then.  By whole
// lengths 16 sequences of 32768 tokens with a window of 4096 had work for two of nine partitions: 254 us, cut by what the table holds 140, so 48.
CB_DEVICE int decode_first(int window_start, int part_len) { return part_len < 0 ? window_start & ~15 : 0; }
// partitions of a sequence up to the last that has tokens
CB_DEVICE int decode_used(const DecodeCut& c, int seq, int splits) {
  if (c.per) return min(splits, (int)__umulhi(max(0, min(c.seq_lens[seq], c.capacity)) + c.part_len - 1, c.per));   // (a division: + .2 us)
  const int len = c.seq_lens[seq], first = c.window > 0 ? decode_first(max(0, len - c.window), c.part_len) : 0;
  const int cached = min(len, c.capacity) - first, part = decode_partition(cached, splits, c.part_len);
  return max(0, min(splits, (cached + part - 1) / part));
}
// tokens that partitions of a sequence's own length can have to share out, with what is before a window on its first 16
static inline int decode_in_sight(int capacity, int window) { return window > 0 && window < capacity - 15 ? window + 15 : capacity; }

// At most: DEC_MOST_SPLITS, or half as many as there are SMs for a sequence alone, unless few heads walk long.  A warp takes 16 tokens of 128 in
// 1.0 us, the sum a partition in .07, so one sequence of T tokens is balanced at sqrt(.88 T) partitions (heads of 64: .5 T); no more than two
// rounds of CTAs of eight heads, nor than most of one round of these - with every place taken they are slower (2 x 16000 tokens of four heads, 100 / 148
// partitions, 24.5 / 30.2; of eight heads, 64 / 74, 29.7 / 33.5).  us with the usual number / so: 1 x 16000 of one head 24.3 / 21.2, 1 x 128000
// 118.7 / 52.8, 2 x 16000 of two heads 25.6 / 22.7, 3 x 16000 of four 28.8 / 26.4, 1 x 16000 of eight 27.0 / 24.3, 1 x 128000 137 / 101.
// Partitions of DEC_PART_MIN tokens where half again as many are enough for that: their weights need no rest (1 x 6000 of one head 14.5 / 14.0).
// Parts are of whole pairs of tiles, of 64 by fours (4 x 16000 of two heads, parts of 192 / 224 / 256 19.9 / 21.8 / 19.7).
static inline int decode_most_splits(int num_seqs, int kv_heads, int head_dim, int one_round, int tokens) {
  const int sms = cb_num_sms(), usual = num_seqs == 1 ? sms / 2 : DEC_MOST_SPLITS, least = (tokens + DEC_PART_MIN - 1) / DEC_PART_MIN;
  const int rounds = 2 * sms / (num_seqs * ((kv_heads + 7) / 8)), room = one_round * (num_seqs == 1 ? 15 : 18) / 20, most = rounds < room ? rounds : room;
  const bool wide = head_dim == 128;
  if (wide && least <= most && 2 * least <= 3 * usual) return least;
  int many = (int)sqrtf((wide ? .875f : .5f) * tokens);
  if (many > most) many = most;
  if (many <= usual) return usual;
  const int part = wide ? (tokens / many + 16) / 32 * 32 : (tokens / many + 63) / 64 * 64;
  many = (tokens + part - 1) / part;
  return many < usual ? usual : many < most ? many : most;
}

template <typename T, typename TC>
__global__ void __launch_bounds__(256) kv_cache_write_kernel(const T* __restrict__ k, const T* __restrict__ v,
                                                             TC* __restrict__ k_cache, TC* __restrict__ v_cache,
                                                             const int* __restrict__ block_tables,
                                                             const int* __restrict__ token_seq,   // [tokens] seq id
                                                             const int* __restrict__ token_pos,   // [tokens] position
                                                             int tokens, int kv_heads, int D, int block_size,
                                                             int max_blocks_per_seq, int64_t k_stride,
                                                             int64_t v_stride) {
  const int t = blockIdx.x;
  if (t >= tokens) return;
  const int seq = token_seq[t], pos = token_pos[t];
  const int blk = block_tables[seq * max_blocks_per_seq + pos / block_size];
  const int slot = pos % block_size;
  const int64_t dst = ((int64_t)blk * block_size + slot) * kv_heads * D;
  const int n = kv_heads * D;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    k_cache[dst + i] = (TC)k[(int64_t)t * k_stride + i];
    v_cache[dst + i] = (TC)v[(int64_t)t * v_stride + i];
  }
}

// 16-byte vectorised variants (the hot ones): one thread moves one 16-byte vector, grid = all vectors of the step, so a
// prefill of thousands of tokens is a single HBM-rate streaming kernel instead of one small CTA per token.
template <typename T>
__global__ void __launch_bounds__(256) kv_cache_write_vec_kernel(const T* __restrict__ k, const T* __restrict__ v,
                                                                 T* __restrict__ k_cache, T* __restrict__ v_cache,
                                                                 const int* __restrict__ block_tables,
                                                                 const int* __restrict__ token_seq,
                                                                 const int* __restrict__ token_pos, int tokens,
                                                                 int vec_per_tok, int block_size, int max_blocks_per_seq,
                                                                 int64_t k_stride, int64_t v_stride) {
  // vec_per_tok = kv_heads * D / 8 (16-bit elements); work items = tokens * 2 (K, V) * vec_per_tok
  cb_early_start();
  const int64_t total = (int64_t)tokens * 2 * vec_per_tok;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (int64_t)gridDim.x * blockDim.x) {
    const int t = (int)(w / (2 * vec_per_tok));
    const int r = (int)(w - (int64_t)t * 2 * vec_per_tok);
    const bool is_v = r >= vec_per_tok;
    const int i = is_v ? r - vec_per_tok : r;
    const int seq = __ldg(token_seq + t), pos = __ldg(token_pos + t);
    const int blk = __ldg(block_tables + seq * max_blocks_per_seq + pos / block_size);
    const int64_t dst = ((int64_t)blk * block_size + pos % block_size) * vec_per_tok + i;       // in 16-byte units
    const uint4 val = is_v ? __ldg(reinterpret_cast<const uint4*>(v + (int64_t)t * v_stride) + i)
                           : __ldg(reinterpret_cast<const uint4*>(k + (int64_t)t * k_stride) + i);
    reinterpret_cast<uint4*>(is_v ? v_cache : k_cache)[dst] = val;
  }
}

// One CTA: sequence `seq`, kv head `kvh`, KV partition `split`.  q: [num_seqs, Hq, D].
// partial outputs: o_part [num_seqs, Hq, splits, D] fp32, ml_part [num_seqs, Hq, splits, 2] (max, sumexp)
//
// Work mapping (the kernel is HBM-bound: every K/V byte is read once, so the job is to keep many full-sector loads in
// flight per SM and to spend few instructions per byte):
//   * a K or V row of one (token, kv head) is D contiguous elements; LPT = D/16 adjacent lanes cover one row with two
//     16-byte loads each, so a warp reads 32/LPT whole rows per pass (fully used 32-byte sectors, 128-byte lines);
//   * the rows travel through a per-warp cp.async ring in shared memory (DEC_STAGES stages of DEC_U passes = 4 KB each):
//     3 stages = 12 KB per warp, ~96 KB per SM stay in flight while one stage is consumed - enough to cover the HBM
//     latency at full bandwidth, independent of the register budget (the first two versions kept the rows in
//     registers: 8 warps / SM at 255 registers, 43 % issue-active, 2.4 TB/s under ncu - load and FMA phases of a warp
//     alternated, then only 32 KB per SM in flight); no block-wide barrier in the main loop;
//   * the query rows live in registers (GH = 4 query heads per warp, the lane's 16 dims of each); a GQA group wider
//     than 4 takes two warps of the CTA (the second read of a K/V row by the sibling warp is an L1/L2 hit);
//   * every lane group keeps its OWN online-softmax state (m, l, o) for the tokens it sees - no cross-lane traffic in
//     the loop except the log2(LPT) shuffles that finish a dot product; the 32/LPT states of a warp are merged once at
//     the end and written as this (head set, partition)'s partial result - no shared-memory reduction, no barrier.
constexpr int DEC_U = 2;    // passes of the warp per pipeline stage
constexpr int DEC_STAGES = 4;   // shared-memory ring depth per warp (DEC_STAGES - 1 stages in flight)
constexpr int DEC_GH = 4;   // query heads per warp

template <typename T, typename TC, int D>
__global__ void __launch_bounds__(DEC_THREADS, 1) paged_decode_kernel(
    const T* __restrict__ q, const TC* __restrict__ k_cache, const TC* __restrict__ v_cache,
    const int* __restrict__ block_tables, const int* __restrict__ seq_lens, float* __restrict__ o_part,
    float* __restrict__ ml_part, int Hq, int Hkv, int block_size, int max_blocks_per_seq, int splits, int part_len,
    float scale, const float* __restrict__ alibi_slopes, int64_t q_stride, int window) {
  static_assert(sizeof(TC) == 2, "the paged cache is read as 16-byte vectors of 16-bit elements");
  constexpr int EPL = 16;                       // elements of a row owned by a lane
  constexpr int LPT = D / EPL;                  // lanes per token row: 4 / 8 / 16
  constexpr int TPW = 32 / LPT;                 // token rows per warp pass
  constexpr int GH = DEC_GH, U = DEC_U;
  constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;
  // CTA = (sequence, group of kv heads, KV partition); warp = one (kv head, set of <= 4 query heads) unit walking ALL
  // tokens of the partition.  The warps of a CTA read ADJACENT 256-byte head slices of the same token rows at the same
  // time, so the CTA streams contiguous [tokens x heads x D] spans of the cache (with one CTA per kv head the 2 KB
  // stride between a head's rows cost ~60 % of the DRAM bandwidth: 2.4 TB/s whatever the number of bytes in flight).
  const int seq = blockIdx.x, split = blockIdx.z;
  const int G = Hq / Hkv;
  const int nsets = (G + GH - 1) / GH;          // sets of <= 4 query heads per kv head
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit = blockIdx.y * (blockDim.x >> 5) + warp;
  const int kvh = unit / nsets, set = unit - kvh * nsets;
  if (kvh >= Hkv) return;                       // (no block-wide barrier anywhere in this kernel)
  const int len = seq_lens[seq];
  // sliding-window attention (Mistral): only the last `window` cached tokens are visible - partitions that lie before
  // the window start contribute nothing (m = -inf, l = 0) and are skipped by the merge
  const int window_start = window > 0 ? max(0, len - window) : 0;
  const int cached = min(len, max_blocks_per_seq * block_size);                                 // (no pages beyond the table's row)
  const int first = decode_first(window_start, part_len);
  const int part = decode_partition(cached - first, splits, part_len);
  const int t0 = max(first + split * part, window_start);
  const int t1 = min(cached, first + split * part + part);
  const int g0 = set * GH;
  const int ng = min(GH, G - g0);
  const int grp = lane / LPT, sub = lane - grp * LPT;

  float qr[GH][EPL];
#pragma unroll
  for (int g = 0; g < GH; ++g) {
    const T* qp = q + (int64_t)seq * q_stride + (int64_t)(kvh * G + g0 + (g < ng ? g : 0)) * D + sub * EPL;
#pragma unroll
    for (int e = 0; e < EPL; ++e) qr[g][e] = g < ng ? to_f32<T>(qp[e]) * (scale * LOG2E) : 0.f;   // scores in the exp2 domain
  }
  float slope[GH];
#pragma unroll
  for (int g = 0; g < GH; ++g) slope[g] = (alibi_slopes && g < ng) ? alibi_slopes[kvh * G + g0 + g] * LOG2E : 0.f;
  const bool has_alibi = alibi_slopes != nullptr;
  float m[GH], l[GH], o[GH][EPL];
#pragma unroll
  for (int g = 0; g < GH; ++g) {
    m[g] = -INFINITY; l[g] = 0.f;
#pragma unroll
    for (int e = 0; e < EPL; ++e) o[g][e] = 0.f;
  }
  const int* bt = block_tables + seq * max_blocks_per_seq;
  const int bs_shift = (block_size & (block_size - 1)) == 0 ? 31 - __clz(block_size) : -1;   // power-of-two blocks: no division
  // K/V travel through a per-warp ring of DEC_STAGES shared-memory stages filled with cp.async (16 bytes per lane and
  // vector; a stage = U passes of the warp = U * TPW token rows, K and V): the bytes in flight are bounded by shared
  // memory, not by registers, so DEC_STAGES - 1 stages (6 KB) per warp stay outstanding while one is consumed.  Every
  // lane reads back exactly the vectors it requested itself (slot = [stage][k|v][pass][half][lane]), so no barrier is
  // needed beyond cp.async.wait_group, and the 16-byte slots of a warp are consecutive (conflict-free LDS.128).
  extern __shared__ __align__(16) unsigned char dec_smem[];
  constexpr int NST = DEC_STAGES;
  constexpr int STAGE_VECS = 2 * U * 2 * 32;                      // uint4 slots per stage: (K|V) x pass x half x lane
  uint4* ring = reinterpret_cast<uint4*>(dec_smem) + (size_t)warp * NST * STAGE_VECS;
  auto issue_stage = [&](int base, int stage) {
    uint4* st = ring + stage * STAGE_VECS;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = base + u * TPW + grp;
      const bool ok = t < t1;
      const int tt = ok ? t : t0;                                 // any valid row: src-size 0 zero-fills instead
      const int blk = bt[bs_shift >= 0 ? (tt >> bs_shift) : (tt / block_size)];
      const int slot = bs_shift >= 0 ? (tt & (block_size - 1)) : (tt % block_size);
      const int64_t row = (((int64_t)blk * block_size + slot) * Hkv + kvh) * D + sub * EPL;
      const uint32_t nbytes = ok ? 16u : 0u;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        cp_async_16(st + ((0 * U + u) * 2 + h) * 32 + lane, k_cache + row + h * 8, nbytes);
        cp_async_16(st + ((1 * U + u) * 2 + h) * 32 + lane, v_cache + row + h * 8, nbytes);
      }
    }
  };
  auto consume = [&](int base, int stage) {
    const uint4* st = ring + stage * STAGE_VECS;
    float sc[U][GH];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      Vec16<TC> k0, k1;
      k0.raw = st[((0 * U + u) * 2 + 0) * 32 + lane];
      k1.raw = st[((0 * U + u) * 2 + 1) * 32 + lane];
      const int t = base + u * TPW + grp;
#pragma unroll
      for (int g = 0; g < GH; ++g) {
        float acc = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) acc += qr[g][e] * k0.get(e);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc += qr[g][8 + e] * k1.get(e);
#pragma unroll
        for (int off = LPT / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
        if (has_alibi) acc += slope[g] * (float)(t - (len - 1));
        sc[u][g] = (t < t1) ? acc : -INFINITY;
      }
    }
    float pr[U][GH];
#pragma unroll
    for (int g = 0; g < GH; ++g) {
      float nm = m[g];
#pragma unroll
      for (int u = 0; u < U; ++u) nm = fmaxf(nm, sc[u][g]);
      if (__any_sync(0xffffffffu, nm > m[g])) {                   // the running max moved for some row group: rescale
        const float corr = (nm == -INFINITY) ? 1.f : ex2_approx(m[g] - nm);
        l[g] *= corr;
#pragma unroll
        for (int e = 0; e < EPL; ++e) o[g][e] *= corr;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        pr[u][g] = (sc[u][g] == -INFINITY) ? 0.f : ex2_approx(sc[u][g] - nm);
        l[g] += pr[u][g];
      }
      m[g] = nm;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      Vec16<TC> v0, v1;
      v0.raw = st[((1 * U + u) * 2 + 0) * 32 + lane];
      v1.raw = st[((1 * U + u) * 2 + 1) * 32 + lane];
#pragma unroll
      for (int g = 0; g < GH; ++g) {
#pragma unroll
        for (int e = 0; e < 8; ++e) o[g][e] += pr[u][g] * v0.get(e);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[g][8 + e] += pr[u][g] * v1.get(e);
      }
    }
  };
  {
    const int step = TPW * U;
    const int first = t0;
    // prologue: NST - 1 stages in flight (empty groups keep the group count uniform at the tail)
#pragma unroll
    for (int s = 0; s < NST - 1; ++s) {
      if (first + s * step < t1) issue_stage(first + s * step, s);
      cp_async_commit();
    }
    int it = 0;
    for (int base = first; base < t1; base += step, ++it) {
      const int ahead = base + (NST - 1) * step;
      if (ahead < t1) issue_stage(ahead, (it + NST - 1) % NST);
      cp_async_commit();
      cp_async_wait<NST - 1>();                                   // the group of stage `it` has landed
      consume(base, it % NST);
    }
    cp_async_wait<0>();
  }
  // merge the TPW lane-group states of the warp (butterfly over the group index)
#pragma unroll
  for (int off = LPT; off < 32; off <<= 1) {
#pragma unroll
    for (int g = 0; g < GH; ++g) {
      const float mo = __shfl_xor_sync(0xffffffffu, m[g], off);
      const float lo = __shfl_xor_sync(0xffffffffu, l[g], off);
      const float nm = fmaxf(m[g], mo);
      const float c1 = (m[g] == -INFINITY) ? 0.f : ex2_approx(m[g] - nm);
      const float c2 = (mo == -INFINITY) ? 0.f : ex2_approx(mo - nm);
      l[g] = l[g] * c1 + lo * c2;
#pragma unroll
      for (int e = 0; e < EPL; ++e) o[g][e] = o[g][e] * c1 + __shfl_xor_sync(0xffffffffu, o[g][e], off) * c2;
      m[g] = nm;
    }
  }
  // every lane group now holds the merged state; group 0 writes this unit's partial result
  if (grp == 0) {
#pragma unroll
    for (int g = 0; g < GH; ++g) {
      if (g < ng) {
        const int64_t oi = (((int64_t)seq * Hq + kvh * G + g0 + g) * splits + split);
        float4* dst = reinterpret_cast<float4*>(o_part + oi * D + sub * EPL);
#pragma unroll
        for (int e = 0; e < EPL; e += 4) dst[e >> 2] = make_float4(o[g][e], o[g][e + 1], o[g][e + 2], o[g][e + 3]);
        if (sub == 0) { ml_part[oi * 2] = m[g] * LN2; ml_part[oi * 2 + 1] = l[g]; }   // max back in natural-log units
      }
    }
  }
}

// ----------------------------------------------------------------------------------------------------------------
// Tensor-core formulation of the same split-KV decode step (the default; `CB200_DECODE=simt` selects the kernel above).
//
// The CUDA-core kernel above executes ~89 warp-instructions per (token, kv head) - two FMAs per cached element and q
// head - which is as much issue time as the HBM transfer takes (ncu: 93 M warp-instructions, 45 % issue-active,
// 2.2-2.4 TB/s).  Here the GQA group of a kv head (<= 8 q heads, padded to the 16 rows of an MMA) is the M dimension of
// `mma.sync.m16n8k16`:  S[heads x 16 tokens] = Q K^T  and  O[heads x D] += P V  per 16-token tile, i.e. 32 MMAs instead of
// ~4000 FMAs per tile and lane.
//   * warp = (sequence, kv head, partition) unit, as above; Q fragments (A operand) live in registers;
//   * a tile of 16 token rows of K and of V (16 x D 16-bit values each) is fetched with cp.async into a per-warp ring
//     (DEC_MMA_STAGES deep); a row's 16-byte chunks are stored XOR-swizzled by (token mod 8), so the ldmatrix reads - K
//     plain (B operand of Q K^T), V transposed (B operand of P V) - are bank-conflict free;
//   * softmax state per head row is replicated over the four lanes of a quad; the probabilities go straight from the
//     accumulator layout of S to the A-operand layout of P V (no shared-memory round trip); the output accumulator is
//     rescaled only when a row max moved;
//   * partial results use the same (o_part, ml_part) format, so the reduce kernel is shared.
constexpr int DEC_MMA_TOKENS = 16;
constexpr int DEC_MMA_STAGES = 3;

CB_DEVICE void ldmatrix_x4(uint32_t (&r)[4], const void* smem_row) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem_row);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
CB_DEVICE void ldmatrix_x4_trans(uint32_t (&r)[4], const void* smem_row) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem_row);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
template <typename T> CB_DEVICE void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <> CB_DEVICE void mma_16816<__nv_bfloat16>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <> CB_DEVICE void mma_16816<__half>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <typename T> CB_DEVICE uint32_t pack2(float lo, float hi);
template <> CB_DEVICE uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <> CB_DEVICE uint32_t pack2<__half>(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

template <typename T> CB_DEVICE float2 unpack2(uint32_t v);
template <> CB_DEVICE float2 unpack2<__nv_bfloat16>(uint32_t v) { return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&v)); }
template <> CB_DEVICE float2 unpack2<__half>(uint32_t v) { return __half22float2(*reinterpret_cast<__half2*>(&v)); }

// REST: the rows of P V that have no heads take what the rounding of the weights to 16 bits left.  The largest weight of a partition is exact, and
// sequences that are cut into fewer partitions than of DEC_PART_MIN tokens have fewer exact ones: error against 64 bits, 16 sequences of up to 1024 tokens
// in bf16, 2.03e-3 in short partitions, 2.06e-3 in long ones, 1.66e-3 with the rest; one of 16000 in fp16 2.55e-4, 2.70e-4 and 2.10e-4.  For calls
// that are cut by their own lengths where the table has room for more than DEC_PART_MIN tokens a partition, or in a window; the others' are no longer
// than they ever were, and 64 sequences of 2048 tokens, cut by their table, would take 79 us with it instead of 77.
template <typename T, int D, bool REST>
__global__ void __launch_bounds__(DEC_THREADS, 1) paged_decode_mma_kernel(
    const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
    const int* __restrict__ block_tables, const int* __restrict__ seq_lens, float* __restrict__ o_part,
    float* __restrict__ ml_part, int Hq, int Hkv, int block_size, int max_blocks_per_seq, int splits, int part_len,
    float scale, const float* __restrict__ alibi_slopes, int64_t q_stride, int window) {
  constexpr int NT = DEC_MMA_TOKENS, NST = DEC_MMA_STAGES;
  constexpr int KS = D / 16;                    // k-steps of Q K^T
  constexpr int NO = D / 8;                     // 8-wide column tiles of the output
  constexpr int CPR = D / 8;                    // 16-byte chunks per token row
  constexpr int ROW_BYTES = D * 2;
  constexpr int TILE_BYTES = NT * ROW_BYTES;    // one operand (K or V) of one stage
  constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;
  const int seq = blockIdx.x, split = blockIdx.z;
  const int G = Hq / Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = blockIdx.y * (blockDim.x >> 5) + warp;
  if (kvh >= Hkv) return;                       // (no block-wide barrier in this kernel)
  cb_early_start();
  const int len = seq_lens[seq];
  const int window_start = window > 0 ? max(0, len - window) : 0;
  const int cached = min(len, max_blocks_per_seq * block_size);                                 // (no pages beyond the table's row)
  const int first = REST ? decode_first(window_start, part_len) : 0;           // (in every call: one sequence of 4097 tokens 14.4 us, 14.0 so)
  const int part = decode_partition(cached - first, splits, part_len);
  const int t0 = max(first + split * part, window_start);
  const int t1 = min(cached, first + split * part + part);
  const int row = lane >> 2, quad = lane & 3;   // accumulator layout: head row, column pair inside an 8-wide tile
  const bool row_ok = row < G;                  // rows G..15 of the MMA are padding
  const float scale2 = scale * LOG2E;           // scores in the exp2 domain
  const float slope2 = (alibi_slopes != nullptr && row_ok) ? alibi_slopes[kvh * G + row] * LOG2E : 0.f;
  const bool has_alibi = alibi_slopes != nullptr;

  // ---- Q fragments: A operand [16 heads x 16 d] per k-step; a1 / a3 are head rows 8..15 = zero (G <= 8)
  uint32_t qa[KS][4];
  {
    const T* qrow = q + (int64_t)seq * q_stride + (int64_t)(kvh * G + (row_ok ? row : 0)) * D;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      const uint32_t lo = *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + quad * 2);
      const uint32_t hi = *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 8 + quad * 2);
      qa[ks][0] = row_ok ? lo : 0u; qa[ks][1] = 0u; qa[ks][2] = row_ok ? hi : 0u; qa[ks][3] = 0u;
    }
  }
  float o[NO][4];
#pragma unroll
  for (int j = 0; j < NO; ++j) { o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f; }
  float m_run = -INFINITY, l_run = 0.f;         // per head row, replicated over the quad (l: this lane's share)

  extern __shared__ __align__(128) unsigned char dec_smem[];
  unsigned char* ring = dec_smem + (size_t)warp * NST * 2 * TILE_BYTES;
  const int* bt = block_tables + seq * max_blocks_per_seq;
  const int bs_shift = (block_size & (block_size - 1)) == 0 ? 31 - __clz(block_size) : -1;
  auto issue_stage = [&](int base, int stage) {
    unsigned char* kt = ring + (size_t)stage * 2 * TILE_BYTES;
    unsigned char* vt = kt + TILE_BYTES;
#pragma unroll
    for (int i = 0; i < NT * CPR / 32; ++i) {
      const int cid = lane + 32 * i;
      const int tr = cid / CPR, c = cid - tr * CPR;          // token row inside the tile, 16-byte chunk inside the row
      const int t = base + tr;
      const bool ok = t < t1;
      const int tt = ok ? t : t0;
      const int blk = bt[bs_shift >= 0 ? (tt >> bs_shift) : (tt / block_size)];
      const int slot = bs_shift >= 0 ? (tt & (block_size - 1)) : (tt % block_size);
      const int64_t src = (((int64_t)blk * block_size + slot) * Hkv + kvh) * D + c * 8;
      const int dst = tr * ROW_BYTES + ((c ^ (tr & 7)) << 4);
      const uint32_t nbytes = ok ? 16u : 0u;
      cp_async_16(kt + dst, k_cache + src, nbytes);
      cp_async_16(vt + dst, v_cache + src, nbytes);
    }
  };
  auto consume = [&](int base, int stage) {
    const unsigned char* kt = ring + (size_t)stage * 2 * TILE_BYTES;
    const unsigned char* vt = kt + TILE_BYTES;
    // ---- S = Q K^T for 16 tokens (two 8-token column tiles)
    float sacc[2][4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      sacc[nt][0] = sacc[nt][1] = sacc[nt][2] = sacc[nt][3] = 0.f;
      const int tr = nt * 8 + (lane & 7);                    // token row whose address this lane supplies
#pragma unroll
      for (int ks = 0; ks < KS; ks += 2) {
        // matrices: (ks, d 0..7), (ks, d 8..15), (ks + 1, d 0..7), (ks + 1, d 8..15)
        const int c = 2 * ks + (lane >> 3);
        uint32_t b[4];
        ldmatrix_x4(b, kt + tr * ROW_BYTES + ((c ^ (tr & 7)) << 4));
        mma_16816<T>(sacc[nt], qa[ks], b[0], b[1]);
        mma_16816<T>(sacc[nt], qa[ks + 1], b[2], b[3]);
      }
    }
    // ---- online softmax of head row `row` (this lane: tokens nt * 8 + quad * 2 + {0, 1})
    float sv[4];
    float mx = -INFINITY;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = base + nt * 8 + quad * 2 + e;
        float x = sacc[nt][e] * scale2;
        if (has_alibi) x = fmaf(slope2, (float)(t - (len - 1)), x);
        x = (t < t1) ? x : -INFINITY;
        sv[nt * 2 + e] = x;
        mx = fmaxf(mx, x);
      }
    }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float m_new = fmaxf(m_run, mx);
    if (__any_sync(0xffffffffu, m_new > m_run)) {
      const float corr = (m_new == -INFINITY) ? 1.f : ex2_approx(m_run - m_new);
      l_run *= corr;
#pragma unroll
      for (int j = 0; j < NO; ++j) {
        o[j][0] *= corr; o[j][1] *= corr;
        if (REST) { o[j][2] *= corr; o[j][3] *= corr; }
      }
    }
    m_run = m_new;
    float pv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      pv[i] = (sv[i] == -INFINITY) ? 0.f : ex2_approx(sv[i] - m_new);
      l_run += pv[i];
    }
    // P as A operand [16 heads x 16 tokens]: a0 = tokens 0..7 of this row, a2 = tokens 8..15; rows 8..15 are zero or REST
    uint32_t pa[4];
    pa[0] = row_ok ? pack2<T>(pv[0], pv[1]) : 0u; pa[1] = 0u;
    pa[2] = row_ok ? pack2<T>(pv[2], pv[3]) : 0u; pa[3] = 0u;
    if (REST) {
      const float2 a = unpack2<T>(pa[0]), b = unpack2<T>(pa[2]);
      pa[1] = row_ok ? pack2<T>(pv[0] - a.x, pv[1] - a.y) : 0u;
      pa[3] = row_ok ? pack2<T>(pv[2] - b.x, pv[3] - b.y) : 0u;
    }
    // ---- O += P V: V^T fragments through ldmatrix.trans
    {
      const int tr = (lane & 7) + ((lane >> 3) & 1) * 8;     // matrices: (tok 0..7, j), (tok 8..15, j), (0..7, j+1), (8..15, j+1)
#pragma unroll
      for (int j = 0; j < NO; j += 2) {
        const int c = j + (lane >> 4);
        uint32_t b[4];
        ldmatrix_x4_trans(b, vt + tr * ROW_BYTES + ((c ^ (tr & 7)) << 4));
        mma_16816<T>(o[j], pa, b[0], b[1]);
        mma_16816<T>(o[j + 1], pa, b[2], b[3]);
      }
    }
  };
  {
#pragma unroll
    for (int s = 0; s < NST - 1; ++s) {
      if (t0 + s * NT < t1) issue_stage(t0 + s * NT, s);
      cp_async_commit();
    }
    int it = 0;
    for (int base = t0; base < t1; base += NT, ++it) {
      const int ahead = base + (NST - 1) * NT;
      if (ahead < t1) issue_stage(ahead, (it + NST - 1) % NST);
      cp_async_commit();
      cp_async_wait<NST - 1>();
      __syncwarp();                                          // the tile was written by all lanes of the warp
      consume(base, it % NST);
      __syncwarp();                                          // all lanes done reading before the stage is refilled
    }
    cp_async_wait<0>();
  }
  // ---- this unit's partial result (row sum over the quad first).  (Of a partition behind the sequence's end nobody asks for one where there are
  // many; looked at before the queries are loaded it cost every call .5 us.)
  if (splits >= DEC_WIDE && first + split * part >= cached) return;
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
  if (row_ok) {
    const int64_t oi = (((int64_t)seq * Hq + kvh * G + row) * splits + split);
    float* dst = o_part + oi * D + quad * 2;
#pragma unroll
    for (int j = 0; j < NO; ++j) {
      if (REST) {                               // (an infinite value stays what it is: its remainder's sign would make a NaN of it)
        if (isfinite(o[j][0])) o[j][0] += o[j][2];
        if (isfinite(o[j][1])) o[j][1] += o[j][3];
      }
      *reinterpret_cast<float2*>(dst + j * 8) = make_float2(o[j][0], o[j][1]);
    }
    if (quad == 0) { ml_part[oi * 2] = m_run * LN2; ml_part[oi * 2 + 1] = l_run; }
  }
}

template <typename T, int D>
__global__ void __launch_bounds__(128) decode_reduce_kernel(const float* __restrict__ o_part,
                                                            const float* __restrict__ ml_part, T* __restrict__ out,
                                                            int Hq, int splits, int64_t out_stride) {
  cb_early_start();
  const int seq = blockIdx.x, h = blockIdx.y;
  const int64_t base = ((int64_t)seq * Hq + h) * splits;
  float gm = -INFINITY;
  for (int s = 0; s < splits; ++s) gm = fmaxf(gm, ml_part[(base + s) * 2]);
  float ls = 0.f;
  bool nan = false;                             // scores that are all NaN in a partition: its sum is NaN, its maximum -inf
  for (int s = 0; s < splits; ++s) {
    const float mm = ml_part[(base + s) * 2];
    ls += (mm == -INFINITY) ? 0.f : ml_part[(base + s) * 2 + 1] * __expf(mm - gm);
    nan |= isnan(ml_part[(base + s) * 2 + 1]);
  }
  const float inv = nan ? NAN : ls > 0.f ? 1.f / ls : 0.f;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    float acc = 0.f;
    for (int s = 0; s < splits; ++s) {
      const float mm = ml_part[(base + s) * 2];
      if (mm != -INFINITY) acc += o_part[(base + s) * D + d] * __expf(mm - gm);
    }
    out[(int64_t)seq * out_stride + (int64_t)h * D + d] = from_f32<T>(acc * inv);
  }
}

// The same for DEC_WIDE partitions and more, which means few long sequences: the weights are worked out side by side and DEC_AHEAD
// partial results are on their way to a thread at a time, where the kernel above waits for each in turn (65 partitions of one
// sequence of 4097 tokens: the call on the device 16.2 us, 13.9 so).  With fewer of them it is no faster (16 x 2048 tokens, 64 / 8 heads, 19
// partitions 30 us, 33 so) and with many sequences slower (1024 of 64 tokens 78 us, 89 so).
// Sums in the same order with the same roundings.
constexpr int DEC_AHEAD = 16, DEC_WIDE_THREADS = 128;
template <typename T, int D>
__global__ void __launch_bounds__(DEC_WIDE_THREADS) decode_reduce_wide_kernel(const float* __restrict__ o_part,
                                                                              const float* __restrict__ ml_part,
                                                                              T* __restrict__ out, int Hq, int all_splits,
                                                                              int64_t out_stride, DecodeCut cut) {
  constexpr int COLS = (D + DEC_WIDE_THREADS - 1) / DEC_WIDE_THREADS;
  __shared__ float max_s[DEC_WIDE_THREADS / 32];
  __shared__ float w_s[DEC_WIDE_THREADS], l_s[DEC_WIDE_THREADS];      // weight (-1: a partition without tokens), sum
  const int seq = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int64_t base = ((int64_t)seq * Hq + h) * all_splits;
  const float2* ml = reinterpret_cast<const float2*>(ml_part) + base;
  cb_early_start();
  const int splits = decode_used(cut, seq, all_splits);
  float gm = -INFINITY;
  for (int s = tid; s < all_splits; s += DEC_WIDE_THREADS) {     // (asked for beside the length)
    const float x = ml[s].x;
    if (s < splits) gm = fmaxf(gm, x);
  }
  gm = warp_max(gm);
  if ((tid & 31) == 0) max_s[tid >> 5] = gm;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < DEC_WIDE_THREADS / 32; ++w) gm = fmaxf(gm, max_s[w]);
  float ls = 0.f, acc[COLS];
  bool nan = false;                             // as above
#pragma unroll
  for (int c = 0; c < COLS; ++c) acc[c] = 0.f;
  for (int s0 = 0; s0 < splits; s0 += DEC_WIDE_THREADS) {
    const int n = min(DEC_WIDE_THREADS, splits - s0);
    if (s0 > 0) __syncthreads();
    if (tid < n) {
      const float2 x = ml[s0 + tid];
      w_s[tid] = x.x == -INFINITY ? -1.f : __expf(x.x - gm);
      l_s[tid] = x.y;
    }
    __syncthreads();
    for (int s = 0; s < n; ++s) {
      if (w_s[s] >= 0.f) ls = __fadd_rn(ls, __fmul_rn(l_s[s], w_s[s]));
      nan |= isnan(l_s[s]);
    }
    for (int s = 0; s < n; s += DEC_AHEAD) {
      float o[DEC_AHEAD][COLS];
#pragma unroll
      for (int u = 0; u < DEC_AHEAD; ++u)
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
          const int d = tid + c * DEC_WIDE_THREADS;
          if (s + u < n && d < D) o[u][c] = o_part[(base + s0 + s + u) * D + d];
        }
#pragma unroll
      for (int u = 0; u < DEC_AHEAD; ++u)
        if (s + u < n && w_s[s + u] >= 0.f) {
#pragma unroll
          for (int c = 0; c < COLS; ++c) acc[c] = fmaf(o[u][c], w_s[s + u], acc[c]);
        }
    }
  }
  const float inv = nan ? NAN : ls > 0.f ? 1.f / ls : 0.f;
#pragma unroll
  for (int c = 0; c < COLS; ++c) {
    const int d = tid + c * DEC_WIDE_THREADS;
    if (d < D) out[(int64_t)seq * out_stride + (int64_t)h * D + d] = from_f32<T>(acc[c] * inv);
  }
}

template <typename T, int D>
int launch_decode_reduce(const float* o_part, const float* ml_part, T* out, int num_seqs, int Hq, int splits, int64_t out_stride,
                         const DecodeCut& cut, cudaStream_t s) {
  const dim3 grid(num_seqs, Hq);
  return splits < DEC_WIDE ? cb_launch_early(decode_reduce_kernel<T, D>, grid, 128, 0, s, o_part, ml_part, out, Hq, splits, out_stride)
                           : cb_launch_early(decode_reduce_wide_kernel<T, D>, grid, DEC_WIDE_THREADS, 0, s, o_part, ml_part, out, Hq, splits,
                                             out_stride, cut);
}

__global__ void gather_cos_sin_kernel(const float* __restrict__ cos_c, const float* __restrict__ sin_c,
                                      const int* __restrict__ pos, float* __restrict__ cos_o,
                                      float* __restrict__ sin_o, int tokens, int half) {
  const int t = blockIdx.x;
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    cos_o[(int64_t)t * half + i] = cos_c[(int64_t)pos[t] * half + i];
    sin_o[(int64_t)t * half + i] = sin_c[(int64_t)pos[t] * half + i];
  }
}

template <typename TI, typename TO>
__global__ void convert_kernel(const TI* __restrict__ in, TO* __restrict__ out, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (TO)(float)in[i];
}

}  // namespace

extern "C" {

// k, v: [tokens, kv_heads, D] (row strides in elements).  cache dtype == input dtype (fp8 path: cb_convert_fp8 first).
int cb_kv_cache_write(const void* k, const void* v, void* k_cache, void* v_cache, const int* block_tables,
                      const int* token_seq, const int* token_pos, int tokens, int kv_heads, int D, int block_size,
                      int max_blocks_per_seq, int64_t k_stride, int64_t v_stride, int dtype, cudaStream_t s) {
  if (tokens == 0) return 0;
  const int n = kv_heads * D;
  if (n % 8 == 0 && k_stride % 8 == 0 && v_stride % 8 == 0 && ((uintptr_t)k % 16) == 0 && ((uintptr_t)v % 16) == 0 &&
      ((uintptr_t)k_cache % 16) == 0 && ((uintptr_t)v_cache % 16) == 0) {
    const int64_t total = (int64_t)tokens * 2 * (n / 8);
    const int grid = (int)((total + 255) / 256 < 16 * cb_num_sms() ? (total + 255) / 256 : 16 * cb_num_sms());
    CB_DISPATCH_HALF(dtype, T, {
      return cb_launch_early(kv_cache_write_vec_kernel<T>, grid, 256, 0, s, (const T*)k, (const T*)v, (T*)k_cache, (T*)v_cache,
                             block_tables, token_seq, token_pos, tokens, n / 8, block_size, max_blocks_per_seq, k_stride, v_stride);
    });
    return CB_LAUNCH_CHECK();
  }
  CB_DISPATCH_HALF(dtype, T, {
    kv_cache_write_kernel<T, T><<<tokens, 256, 0, s>>>((const T*)k, (const T*)v, (T*)k_cache, (T*)v_cache, block_tables,
                                                      token_seq, token_pos, tokens, kv_heads, D, block_size,
                                                      max_blocks_per_seq, k_stride, v_stride);
  });
  return CB_LAUNCH_CHECK();
}

// partitions of every sequence, and the `part_len` that goes with them (decode_partition).  window: of the attention, 0 for none.  What a
// sequence's result is depends on the call's sizes and on its own length, not on the others' lengths.
int cb_decode_num_splits(int num_seqs, int kv_heads, int head_dim, int max_len, int window, int* part_len_out) {
  *part_len_out = DEC_PART_MIN;
  if (num_seqs <= 0 || kv_heads <= 0) return 1;
  const int sms = cb_num_sms();
  const int warps = decode_warps(kv_heads, head_dim);
  // CTAs of an SM: as many as fit, of eight warps in all for heads of 128 (three heads, two or three CTAs: 32 x 2000 23 and 29, 64 x 500 15 and 19)
  const int fit = 227 * 1024 / (warps * DEC_MMA_STAGES * 2 * DEC_MMA_TOKENS * head_dim * 2), some = (head_dim == 128 ? 8 : 16) / warps;
  const int per_sm = fit < some ? fit : some < 8 ? some : 8;
  const int ctas = num_seqs * ((kv_heads + warps - 1) / warps), one_round = per_sm * sms / ctas, two_rounds = 2 * per_sm * sms / ctas;
  if ((head_dim == 128 || kv_heads <= 4) && head_dim <= 128 && (one_round >= DEC_ROUND_SPLITS || two_rounds > DEC_ROUND_SPLITS)) {
    *part_len_out = -DEC_PART_MIN;
    const int tokens = decode_in_sight(max_len, window), most = (tokens + DEC_PART_MIN - 1) / DEC_PART_MIN;
    const bool short_parts = one_round >= DEC_SHORT_SPLITS && tokens <= DEC_SHORT * one_round && tokens > DEC_SHORT / 4 * one_round;
    const int own = one_round >= DEC_ROUND_SPLITS || short_parts ? one_round : two_rounds;
    const int cap = decode_most_splits(num_seqs, kv_heads, head_dim, one_round, tokens);
    int splits = own < cap ? own : cap;
    if (most <= cap && most <= own + own / 4) splits = most;          // (a few more than fit, whose weights need no rest)
    if (splits < most) return splits;
    if (window <= 0) *part_len_out = DEC_PART_MIN;                    // what every length's own share comes to then
    return most < 1 ? 1 : most;
  }
  // two rounds of CTAs of eight kv heads, partitions of at least DEC_PART_MIN of the tokens that a table has room for
  const int most = (max_len + DEC_PART_MIN - 1) / DEC_PART_MIN;
  const int ctas_per_split = num_seqs * ((kv_heads + 7) / 8);
  int splits = (2 * sms + ctas_per_split - 1) / ctas_per_split;
  if (splits > most) splits = most;
  if (splits < 1) splits = 1;
  int part = (max_len + splits - 1) / splits;
  part = ((part + 31) / 32) * 32;
  splits = (max_len + part - 1) / part;
  if (splits < 1) splits = 1;
  *part_len_out = part;
  return splits;
}

// q: [num_seqs, Hq, D]; out same; caches [nb, bs, Hkv, D]; o_part fp32 [num_seqs, Hq, splits, D]; ml_part [.., 2]
int cb_paged_decode_attention(const void* q, const void* k_cache, const void* v_cache, const int* block_tables,
                              const int* seq_lens, void* out, float* o_part, float* ml_part, int num_seqs, int Hq,
                              int Hkv, int D, int block_size, int max_blocks_per_seq, int splits, int part_len,
                              float scale, const float* alibi_slopes, int64_t q_stride, int64_t out_stride, int dtype,
                              int window, cudaStream_t s) {
  if (num_seqs == 0) return 0;
  if (Hq % Hkv != 0 || Hq / Hkv > MAX_GROUP) return (int)cudaErrorInvalidValue;
  const int G = Hq / Hkv;
  const int units = Hkv * ((G + DEC_GH - 1) / DEC_GH);             // (kv head, query-head set) pairs = warps needed
  const int warps = units < DEC_THREADS / 32 ? units : DEC_THREADS / 32;
  dim3 grid(num_seqs, (units + warps - 1) / warps, splits);
  const int dec_smem = warps * DEC_STAGES * (2 * DEC_U * 2 * 32) * 16;                    // per-warp cp.async rings
  constexpr int dec_smem_max = (DEC_THREADS / 32) * DEC_STAGES * (2 * DEC_U * 2 * 32) * 16;
  // default: the tensor-core formulation (mma.sync over the GQA group) where it applies (head_dim 64 / 128, groups of
  // <= 8 q heads); CB200_DECODE=simt forces the CUDA-core kernel (also used for head_dim 256)
  const char* impl_env = getenv("CB200_DECODE");
  const bool use_mma = !(impl_env != nullptr && impl_env[0] == 's') && G <= 8 && (D == 128 || D == 64);
  const int mma_warps = decode_warps(Hkv, D);
  const int capacity = max_blocks_per_seq * block_size;
  const bool divides = part_len > 0 && (int64_t)(capacity + part_len) * part_len < (1ll << 32);
  const DecodeCut cut{seq_lens, capacity, part_len, window, divides ? (unsigned)(((1ull << 32) + part_len - 1) / part_len) : 0u};
  dim3 mma_grid(num_seqs, (Hkv + mma_warps - 1) / mma_warps, splits);
#define LAUNCH_DEC_MMA(T, DD)                                                                                       \
  {                                                                                                                  \
    constexpr int per_warp = DEC_MMA_STAGES * 2 * DEC_MMA_TOKENS * DD * 2;                                           \
    static CbDeviceAttr attr;                                                                                        \
    static CbDeviceAttr attr_rest;                                                                                   \
    const bool rest = part_len < 0;                                                                                  \
    auto kern = rest ? paged_decode_mma_kernel<T, DD, true> : paged_decode_mma_kernel<T, DD, false>;                 \
    if (const int e = cb_allow_smem(rest ? attr_rest : attr, kern, (DEC_THREADS / 32) * per_warp)) return e;         \
    if (const int e = cb_launch_early(kern, mma_grid, mma_warps * 32, mma_warps * per_warp, s, \
        (const T*)q, (const T*)k_cache, (const T*)v_cache, block_tables, seq_lens, o_part, ml_part, Hq, Hkv,        \
        block_size, max_blocks_per_seq, splits, part_len, scale, alibi_slopes, q_stride, window)) return e;         \
    if (const int e = launch_decode_reduce<T, DD>(o_part, ml_part, (T*)out, num_seqs, Hq, splits, out_stride, cut, s)) return e; \
  }
#define LAUNCH_DEC(T, DD)                                                                                           \
  {                                                                                                                  \
    static CbDeviceAttr attr;                                                                                        \
    if (const int e = cb_allow_smem(attr, paged_decode_kernel<T, T, DD>, dec_smem_max)) return e;                    \
  }                                                                                                                  \
  paged_decode_kernel<T, T, DD><<<grid, warps * 32, dec_smem, s>>>((const T*)q, (const T*)k_cache, (const T*)v_cache, \
      block_tables, seq_lens, o_part, ml_part, Hq, Hkv, block_size, max_blocks_per_seq, splits, part_len, scale,     \
      alibi_slopes, q_stride, window);                                                                               \
  if (const int e = launch_decode_reduce<T, DD>(o_part, ml_part, (T*)out, num_seqs, Hq, splits, out_stride, cut, s)) return e
  CB_DISPATCH_HALF(dtype, T, {
    if (use_mma && D == 128) { LAUNCH_DEC_MMA(T, 128); }
    else if (use_mma && D == 64) { LAUNCH_DEC_MMA(T, 64); }
    else if (D == 128) { LAUNCH_DEC(T, 128); }
    else if (D == 64) { LAUNCH_DEC(T, 64); }
    else if (D == 256) { LAUNCH_DEC(T, 256); }
    else return (int)cudaErrorInvalidValue;
  });
#undef LAUNCH_DEC
#undef LAUNCH_DEC_MMA
  return CB_LAUNCH_CHECK();
}

int cb_gather_cos_sin(const float* cos_c, const float* sin_c, const int* pos, float* cos_o, float* sin_o, int tokens,
                      int half, cudaStream_t s) {
  if (tokens == 0) return 0;
  gather_cos_sin_kernel<<<tokens, 128, 0, s>>>(cos_c, sin_c, pos, cos_o, sin_o, tokens, half);
  return CB_LAUNCH_CHECK();
}

// direction 0: (fp16|bf16|fp32) -> e5m2 ; 1: e5m2 -> (fp16|bf16|fp32)
int cb_convert_fp8(const void* in, void* out, int64_t n, int dtype, int direction, cudaStream_t s) {
  if (n == 0) return 0;
  const int grid = (int)((n + 255) / 256 > 4096 ? 4096 : (n + 255) / 256);
  if (direction == 0) {
    if (dtype == CB_BF16) convert_kernel<__nv_bfloat16, __nv_fp8_e5m2><<<grid, 256, 0, s>>>((const __nv_bfloat16*)in, (__nv_fp8_e5m2*)out, n);
    else if (dtype == CB_F16) convert_kernel<__half, __nv_fp8_e5m2><<<grid, 256, 0, s>>>((const __half*)in, (__nv_fp8_e5m2*)out, n);
    else convert_kernel<float, __nv_fp8_e5m2><<<grid, 256, 0, s>>>((const float*)in, (__nv_fp8_e5m2*)out, n);
  } else {
    if (dtype == CB_BF16) convert_kernel<__nv_fp8_e5m2, __nv_bfloat16><<<grid, 256, 0, s>>>((const __nv_fp8_e5m2*)in, (__nv_bfloat16*)out, n);
    else if (dtype == CB_F16) convert_kernel<__nv_fp8_e5m2, __half><<<grid, 256, 0, s>>>((const __nv_fp8_e5m2*)in, (__half*)out, n);
    else convert_kernel<__nv_fp8_e5m2, float><<<grid, 256, 0, s>>>((const __nv_fp8_e5m2*)in, (float*)out, n);
  }
  return CB_LAUNCH_CHECK();
}

}  // extern "C"
