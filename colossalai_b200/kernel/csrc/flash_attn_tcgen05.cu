// Flash attention forward for sm_100a on the 5th-generation tensor cores.
//
//   O = softmax(scale * Q K^T + causal mask) V,   LSE = log sum exp     (GQA: Hq = g * Hkv, head_dim 64 or 128)
//
// Persistent CTAs, one per SM, walk a list of work units, the longest first.  A unit = TWO 128-row query tiles over the same
// key tiles: two query heads of one kv head where the group is even (the same keys are visible to both), else two
// neighbouring query tiles of one head.  A step is 64 keys: half of a key tile, for each of the two query tiles.  Sixteen warps:
//   warp 0       TMA producer: both Q tiles of a unit, then K_0, V_0, K_1, V_1, ... (128 keys each) through one ring
//   warp 1       MMA issuer: S_t = Q_t K_j^T and O_t += P_t V_j with tcgen05.mma, accumulators in TMEM
//   warp 3       finds the units of a packed batch from its device-resident boundaries, two units ahead
//   warps 4..7   softmax of tile 0, warps 8..11 of tile 1: thread r owns query row r - tcgen05.ld of its S row, running max /
//                sum in the exp2 domain, P_t written back to TMEM as the 16-bit A operand of the second product
//   warps 12..15 output: the rows of a finished unit, divided by their sums
// Bound: the softmax - 128 exponentials per row and key tile at 16 a clock and SM take as long as the products of D = 128.
// Two tiles, so that one tile's softmax runs under the other's products (one tile per CTA and the mask as predicated code:
// 4096 tokens, 32 / 8 heads of 128, causal 239 us = 575 TFLOP/s).  P through TMEM, because a product with both operands in
// shared memory reads 8 KB per 64-clock MMA, all that shared memory delivers.  Persistent, because a unit of a short sequence
// walks a handful of key tiles and a CTA of its own spent a third of its life on launch, allocation and its first loads.
// Half steps, because S_t, P_t and O_t of D = 128 fill the tensor memory: with one S_t per tile the next Q K^T waited for the
// softmax and P V of this one, and the softmax for it; with two halves one is multiplied while the other is exponentiated (and
// 64 scores of a row in registers instead of 128 leave room for the output warps).  The issuing warp converged and its
// descriptors in uniform registers: one thread in a branch took 80 clocks a product, which was the bound of this kernel once the
// steps were halved.  2 x 4096 tokens, 32 / 8 heads of 128, causal: whole steps 309 us, half steps 450, with the converged
// issuer 289, with output warps of their own 256, and 263 with the first reference from both halves of a key tile; five documents of
// 8192 tokens together 181 -> 156; sixteen of 16384, heads of 64, 223 -> 191.  Two threads per row (16 softmax warps) were 5 - 10 %
// slower than one.  The two tiles' exponentials in turn (`take_turn`): sixteen prompts of 16384 tokens, heads of 64, 188 -> 171 us, two
// of 8192 920 -> 765; heads of 128, one call after the other, 2 x 4096 tokens 321 -> 281, five documents of 8192 163 -> 153; short walks take them
// together (launch_flash_fwd).  Taken back since: a quarter or an eighth of the exponentials as polynomials of degree 5 (765 -> 840), the next step's scores
// fetched under the exponentials (997), turns only in units of 8 steps and more (heads of 128: 281 -> 304).
// TMEM map (512 columns): [0,128) S_0, [128,256) S_1, then O_0, O_1, D wide each; P_t of a half overwrites the first 32 columns of
// that half of S_t once its scores are in registers.
// Shared memory at D = 128: 2 x Q 32 KB + 4 ring slots of 32 KB (at D = 64 2 x 16 KB + 8 x 16 KB) + 4 x 32 rows of the output +
// mbarriers.
//
// Reference being replaced: flash-attn 2 `flash_attn_func` / `_flash_attn_varlen_forward` (mma.sync kernels) used by
// `colossalai/shardformer/layer/attn.py:356-372,720-755`.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "common.cuh"
#include "sm100.cuh"

namespace {
using namespace sm100;

constexpr int BLOCK_Q = 128;
constexpr int BLOCK_KV = 128;
constexpr int HALF_KV = 64;            // keys of a step: a score tile is taken in two halves
constexpr int UMMA_K = 16;
constexpr int SOFTMAX_WARP0 = 4;
constexpr int OUTPUT_WARP0 = SOFTMAX_WARP0 + 8;
constexpr int NUM_THREADS = (OUTPUT_WARP0 + 4) * 32;
constexpr int UNIT_RING = 2;

// Waits give up after a bounded number of polls (each of which the hardware may suspend), far beyond any wait of a kernel
// that works.  The CTA then waits, bounded again, for its copies and products in flight, writes the status word, frees its
// tensor memory and leaves; the next launch from the host returns cudaErrorLaunchTimeout instead of launching.
constexpr int WAIT_LIMIT = 1 << 22;

SM100_DEVICE bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int limit = WAIT_LIMIT) {
  if (mbar_try_wait(bar, parity)) return true;
  for (int i = 0; i < limit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 63) == 63 && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
// one thread: the rows of a CTA that gave up are not valid.  (Without a fence: the host looks after the kernel has ended, and a
// system-wide fence anywhere in the backward kernel made all of its reductions slower, 467 -> 525 us.)
SM100_DEVICE void report_abort(int* status) { *reinterpret_cast<volatile int*>(status) = 1; }

// Every role of the backward is done: the producer and the issuer wait for the others, which only say so, and see whether one gave
// up.  Inside the roles, because code behind their last common barrier cost the kernel 2 % (461 and 473 us; the forward
// kernels lose by the second barrier instead, 169 and 175 us, and have it behind).
template <int THREADS> SM100_DEVICE void roles_done_wait() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); }
template <int THREADS> SM100_DEVICE void roles_done() { asm volatile("bar.arrive 1, %0;" ::"n"(THREADS) : "memory"); }

// The status word: pinned host memory, so that the host reads it without a call (null: there is none to be had).  One per
// process, whatever the device.
int* flash_status() {
  static int* const word = [] {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;       // a first launch may be under capture
    cudaThreadExchangeStreamCaptureMode(&mode);
    void* p = nullptr;
    if (cudaHostAlloc(&p, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
      (void)cudaGetLastError();
      p = nullptr;
    } else {
      *static_cast<int*>(p) = 0;
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    return static_cast<int*>(p);
  }();
  return word;
}
// what an earlier launch reported, once: every launcher asks before it launches
int flash_earlier() {
  int* const word = flash_status();
  if (word == nullptr) return (int)cudaErrorMemoryAllocation;
  return __atomic_load_n(word, __ATOMIC_RELAXED) && __atomic_exchange_n(word, 0, __ATOMIC_ACQ_REL) ? (int)cudaErrorLaunchTimeout : 0;
}

// the wait alone, on a barrier at which nothing arrives
__global__ void flash_wait_probe_kernel(int limit, int* status) {
  __shared__ uint64_t bar;
  __shared__ int gave_up;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    gave_up = 0;
    fence_barrier_init();
    if (!wait_or_abort(&bar, 0, &gave_up, limit) && gave_up) report_abort(status);
  }
}

template <int D> struct FaCfg {
  static constexpr int Q_BYTES = BLOCK_Q * D * 2;
  static constexpr int SLOT_BYTES = BLOCK_KV * D * 2;      // one K or V tile
  static constexpr int SLOTS = D == 128 ? 4 : 8;
  static constexpr int BOX_BYTES = 32 * D * 2;             // an output warp's 32 rows on their way out
  static constexpr int ROW_BYTES = 2 * BLOCK_Q * 8;        // a row's reference maximum and sum
  static constexpr int BAR_BYTES = 512;
  static constexpr int SMEM_BYTES = 2 * Q_BYTES + SLOTS * SLOT_BYTES + 4 * BOX_BYTES + ROW_BYTES + BAR_BYTES;
  static constexpr int TMEM_COLS = 512;
  static constexpr int O_COL = 256;
};

struct FaParams {
  // packed / variable-length batches: cu_seqlens[b] .. cu_seqlens[b + 1] are the token rows of sequence b (self
  // attention, the same boundaries for queries and keys); null = `batch` equal-length sequences
  const int* cu_seqlens;
  int batch, seqlen_q, seqlen_k;     // equal-length sequences, token-major tensors [batch * seqlen, heads * D]
  int hq, hkv;
  int causal;
  int pair_heads;                    // a unit's tiles: 1 = one query tile of two heads, 0 = two query tiles of one head
  int head_units;                    // hq / 2 or hq
  int seq_units;                     // equal lengths: units of one sequence and head
  float scale_log2;                  // softmax scale * log2(e)
  void* out;                         // [batch * seqlen_q, hq * D]
  float* lse;                        // [batch * seqlen_q, hq] natural-log LSE
  // ring / blockwise attention: the online-softmax state of every query row lives in (o_state, lse) between launches.
  // has_prev: start from that state (m = lse, l = 1, acc = o_state) instead of (-inf, 0, 0); the result - the merge of
  // the previous partial result with this launch's keys - is written back in fp32.  No separate rescale / merge pass.
  float* o_state;                    // [rows, hq * D] fp32, or null (plain attention: `out` in the input dtype)
  int has_prev;
  int* status;                       // raised when a wait ran out
  uint32_t idesc_qk, idesc_pv;
  // EXTRA variant of the kernel only (inference prefill of sliding-window / ALiBi models):
  int window;                        // > 0: query q sees keys (q - window, q]; key tiles left of every window are skipped
  const float* alibi;                // [hq] slopes (score += slope * (key - query)), or null
};

SM100_DEVICE float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// two fp32 operations in one instruction
SM100_DEVICE uint64_t pack_f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
SM100_DEVICE void unpack_f32x2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
SM100_DEVICE uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
SM100_DEVICE uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
SM100_DEVICE uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
template <bool BF16> SM100_DEVICE uint32_t pack_16(float a, float b) {
  if (BF16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// Packed batches: units of `per` rows in descending order of their index inside the sequence (the unit with index i walks the
// key tiles of i + 1 units), over all sequences: count(i) = units with an index >= i.  One warp, every lane gets the result.  The
// boundaries of the first 32 sequences stay in registers, a lane a sequence: a search is a dozen counts one after the other, and
// read from memory for each of them it took longer than a short unit (packed_batch).
struct PackedBatch {
  const int* cu;
  int batch, per, start, len;       // of this lane's sequence (0: none)
  int units, longest;               // units of this lane's sequence, of the longest one
};
SM100_DEVICE int packed_units(const PackedBatch& s, int b) { return (__ldg(s.cu + b + 1) - __ldg(s.cu + b) + s.per - 1) / s.per; }
SM100_DEVICE PackedBatch packed_batch(const int* cu, int batch, int per) {
  const int lane = threadIdx.x & 31;
  PackedBatch s;
  s.cu = cu; s.batch = batch; s.per = per;
  s.start = lane < batch ? __ldg(cu + lane) : 0;
  s.len = lane < batch ? __ldg(cu + lane + 1) - s.start : 0;
  s.units = (s.len + per - 1) / per;
  int longest = s.units;
  for (int b = lane + 32; b < batch; b += 32) longest = max(longest, packed_units(s, b));
  s.longest = __reduce_max_sync(0xffffffffu, longest);
  return s;
}
SM100_DEVICE int packed_count(const PackedBatch& s, int i) {
  int c = max(0, s.units - i);
  for (int b = (threadIdx.x & 31) + 32; b < s.batch; b += 32) c += max(0, packed_units(s, b) - i);
  return __reduce_add_sync(0xffffffffu, c);
}
SM100_DEVICE void packed_unit(const PackedBatch& s, int r, int& unit, int& start, int& len) {
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = s.longest;                                     // largest index lo with count(lo) > r
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (packed_count(s, mid) > r) lo = mid; else hi = mid;
  }
  int nth = r - packed_count(s, lo + 1);                          // the nth sequence that has a unit `lo`
  unit = lo; start = 0; len = 0;
  for (int b0 = 0; b0 < s.batch; b0 += 32) {
    const int b = b0 + lane;
    const int s0 = b0 == 0 ? s.start : b < s.batch ? __ldg(s.cu + b) : 0;
    const int n = b0 == 0 ? s.len : b < s.batch ? __ldg(s.cu + b + 1) - s0 : 0;
    const unsigned m = __ballot_sync(0xffffffffu, (n + s.per - 1) / s.per > lo);
    if (nth < __popc(m)) {
      const int pick = (int)__fns(m, 0, nth + 1);
      start = __shfl_sync(0xffffffffu, s0, pick);
      len = __shfl_sync(0xffffffffu, n, pick);
      return;
    }
    nth -= __popc(m);
  }
}

// the same value in every lane, in a way that the compiler sees
template <typename V> SM100_DEVICE V uniform(V v) { return __shfl_sync(0xffffffffu, v, 0); }

struct FaUnit {
  int live, index, q_start, k_start, len_q, len_k, head0;
};

// TURNS: the exponentials of a unit's two tiles in turn (`take_turn`)
template <int D, bool EXTRA, bool BF16, bool TURNS>
__global__ void __launch_bounds__(NUM_THREADS, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                 const __grid_constant__ CUtensorMap tmap_v, const FaParams p) {
  using C = FaCfg<D>;
  constexpr int SLOTS = C::SLOTS;
  extern __shared__ __align__(1024) uint8_t smem[];          // (the swizzle's patterns repeat every 1024 bytes)
  uint8_t* smem_q = smem;                                    // two tiles
  uint8_t* smem_kv = smem + 2 * C::Q_BYTES;
  uint8_t* smem_box = smem_kv + SLOTS * C::SLOT_BYTES;       // [4 warps]
  float2* smem_row = reinterpret_cast<float2*>(smem_box + 4 * C::BOX_BYTES);   // [2 tiles][BLOCK_Q]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_row + 2 * BLOCK_Q);
  uint64_t* q_full = bars;                 // [1]
  uint64_t* q_empty = bars + 1;            // [1]  the unit's last Q K^T retired
  uint64_t* full = bars + 2;               // [SLOTS]
  uint64_t* empty = full + SLOTS;          // [SLOTS]
  uint64_t* s_full = empty + SLOTS;        // [2][2]  a half of S_t is in tensor memory
  uint64_t* p_full = s_full + 4;           // [2][2]  4 softmax warps have written P_t over it
  uint64_t* o_full = p_full + 4;           // [2][2]  the product that read P_t there has retired
  uint64_t* o_empty = o_full + 4;          // [2]  4 output warps have read O_t
  uint64_t* row_full = o_empty + 2;        // [2]  4 softmax warps are through with a unit: maxima and sums of its rows
  uint64_t* row_empty = row_full + 2;      // [2]  4 output warps have read them
  uint64_t* turn = row_empty + 2;          // [2][4]  a warp of that tile may exponentiate
  uint64_t* u_full = turn + 8;             // [UNIT_RING]
  uint64_t* u_empty = u_full + UNIT_RING;  // [UNIT_RING]  14 warps have read the unit
  FaUnit* units = reinterpret_cast<FaUnit*>(u_empty + UNIT_RING);
  uint64_t* drained = reinterpret_cast<uint64_t*>(units + UNIT_RING);   // [1]  a CTA that gives up: its products have retired
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(drained + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  volatile int* copies = abort_flag + 1;   // [2]  key / value tiles and query tiles that the producer asked for

  const int warp = uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const bool resume = p.o_state != nullptr && p.has_prev != 0;   // block mode: continue from the stored state

  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tmap_q);
    prefetch_tensormap(&tmap_k);
    prefetch_tensormap(&tmap_v);
  }
  if (warp == 1 && lane == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int i = 0; i < SLOTS; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&o_full[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&o_empty[i], 4);
      mbar_init(&row_full[i], 4);
      mbar_init(&row_empty[i], 4);
    }
    for (int i = 0; i < 8; ++i) mbar_init(&turn[i], 1);
    for (int i = 0; i < UNIT_RING; ++i) {
      mbar_init(&u_full[i], 1);
      mbar_init(&u_empty[i], 14);
    }
    mbar_init(drained, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 2) tmem_alloc<C::TMEM_COLS>(tmem_ptr_smem);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;

  // ---- a unit as every role sees it
  FaUnit un;
  int ui = 0;                               // units taken so far
  auto next_unit = [&]() -> bool {          // whole warps
    const int e = ui % UNIT_RING;
    if (!__all_sync(0xffffffffu, wait_or_abort(&u_full[e], (uint32_t)((ui / UNIT_RING) & 1), abort_flag))) return false;
    un = units[e];
    __syncwarp();
    if (lane == 0) mbar_arrive(&u_empty[e]);
    ++ui;
    return un.live != 0;
  };
  auto tile_of = [&](int t) { return p.pair_heads ? un.index : 2 * un.index + t; };
  auto head_of = [&](int t) { return p.pair_heads ? un.head0 + t : un.head0; };
  // causal with seqlen_q == seqlen_k: key tiles 0..q_tile; otherwise all of them.  Sliding window: the lowest key any row of
  // the first tile can see is (tile_of(0) * BLOCK_Q - window + 1)
  auto first_key_tile = [&]() { return (EXTRA && p.window > 0) ? max(0, tile_of(0) * BLOCK_Q - p.window + 1) / BLOCK_KV : 0; };
  auto steps_of = [&](int t) {              // steps of 64 keys that tile t walks (0: the tile lies behind the sequence's end)
    if (tile_of(t) * BLOCK_Q >= un.len_q) return 0;
    const int all = (un.len_k + HALF_KV - 1) / HALF_KV;
    return (p.causal ? min(2 * tile_of(t) + 2, all) : all) - 2 * first_key_tile();
  };

  if (warp == 3) {
    // ================================================================ unit list
    const int per = p.pair_heads ? BLOCK_Q : 2 * BLOCK_Q;      // query rows of a unit
    PackedBatch packed{};
    if (p.cu_seqlens != nullptr) packed = packed_batch(p.cu_seqlens, p.batch, per);
    const int ranks = p.cu_seqlens != nullptr ? packed_count(packed, 0) : p.seq_units * p.batch;
    const int total = ranks * p.head_units;
    bool ok = true;
    for (int i = 0; ok; ++i) {
      // CTA c takes the list's entries c, 2 G - 1 - c, 2 G + c, ...: the longest first, and no CTA always the longer of a round
      const int u = i * (int)gridDim.x + ((i & 1) ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x);
      FaUnit x;
      x.live = i * (int)gridDim.x < total;
      x.index = 0; x.q_start = x.k_start = x.len_q = x.len_k = x.head0 = 0;      // (a unit without rows: not this CTA's turn)
      if (u < total) {
        const int rank = u / p.head_units;
        x.head0 = (u - rank * p.head_units) * (p.pair_heads ? 2 : 1);
        if (p.cu_seqlens != nullptr) {
          packed_unit(packed, rank, x.index, x.q_start, x.len_q);
          x.k_start = x.q_start; x.len_k = x.len_q;
        } else {
          const int b = rank % p.batch;
          x.index = p.causal ? p.seq_units - 1 - rank / p.batch : rank / p.batch;
          x.q_start = b * p.seqlen_q; x.k_start = b * p.seqlen_k; x.len_q = p.seqlen_q; x.len_k = p.seqlen_k;
        }
      }
      const int e = i % UNIT_RING;
      ok = __all_sync(0xffffffffu, wait_or_abort(&u_empty[e], (uint32_t)(((i / UNIT_RING) & 1) ^ 1), abort_flag));
      if (lane == 0 && ok) {
        units[e] = x;
        mbar_arrive(&u_full[e]);
      }
      __syncwarp();
      if (!x.live) break;
    }
  } else if (warp == 0) {
    // ================================================================ TMA producer
    int issued = 0, nq = 0;
    while (next_unit()) {
      const int n0 = steps_of(0), n1 = steps_of(1), tiles = (max(n0, n1) + 1) / 2;
      if (tiles == 0) continue;
      bool ok = true;
      if (lane == 0) {
        ok = wait_or_abort(q_empty, (uint32_t)((nq & 1) ^ 1), abort_flag);
        if (ok) {
          mbar_arrive_expect_tx(q_full, (n1 > 0 ? 2 : 1) * C::Q_BYTES);
          for (int t = 0; t < (n1 > 0 ? 2 : 1); ++t)
#pragma unroll
            for (int h = 0; h < D / 64; ++h)                   // boxes [128 rows, 64 d] -> K-major swizzled sub-tiles
              tma_load_2d(&tmap_q, q_full, smem_q + t * C::Q_BYTES + h * (BLOCK_Q * 128), head_of(t) * D + h * 64,
                          un.q_start + tile_of(t) * BLOCK_Q);
          ++nq;
          const int kv_head = un.head0 / (p.hq / p.hkv), k_tile0 = first_key_tile();
          for (int i = 0; i < 2 * tiles && ok; ++i) {          // K_j (K-major B of Q K^T), V_j (MN-major B of P V)
            const int slot = issued % SLOTS;
            ok = wait_or_abort(&empty[slot], (uint32_t)(((issued / SLOTS) & 1) ^ 1), abort_flag);
            if (!ok) break;
            mbar_arrive_expect_tx(&full[slot], C::SLOT_BYTES);
            const int row = un.k_start + (k_tile0 + (i >> 1)) * BLOCK_KV;
#pragma unroll
            for (int h = 0; h < D / 64; ++h)
              tma_load_2d((i & 1) ? &tmap_v : &tmap_k, &full[slot], smem_kv + slot * C::SLOT_BYTES + h * (BLOCK_KV * 128),
                          kv_head * D + h * 64, row);
            ++issued;
          }
        }
      }
      if (!__all_sync(0xffffffffu, ok)) break;
    }
    if (lane == 0) { copies[0] = issued; copies[1] = nq; }
    __syncwarp();
  } else if (warp == 1) {
    // ================================================================ MMA issuer
    const uint64_t dq = make_smem_desc_sw128(smem_u32(smem_q), 16, 1024);                 // K-major, K = D
    const uint64_t dk0 = make_smem_desc_sw128(smem_u32(smem_kv), 16, 1024);               // K-major
    const uint64_t dv0 = make_smem_desc_sw128(smem_u32(smem_kv), BLOCK_KV * 128, 1024);   // MN-major: [keys, D] row-major
    const uint32_t leader = elect_one();
    int nq = 0, slot = 0;                    // units with work so far; next slot of the ring
    int uses[2] = {0, 0};                    // per tile: units it had work in
    uint32_t phase = 0, turn = 0;            // bit 2 t + half: parity of the next P_t in that half; parity of the ring's next slot
    auto warp_wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag)) != 0; };
    while (next_unit()) {
      const int n0 = uniform(steps_of(0)), n1 = uniform(steps_of(1)), steps = max(n0, n1), tiles = (steps + 1) / 2;
      if (steps == 0) continue;
      auto take = [&](int& at) {             // the next tile of the ring: K_0, V_0, K_1, V_1, ...
        at = slot;
        const bool here = warp_wait(&full[slot], turn);
        if (++slot == SLOTS) { slot = 0; turn ^= 1; }
        return here;
      };
      int ks = 0, vs = 0;                    // slots of the key tile and the value tile in use
      // half h of S_t <- Q_t times the 64 keys of a step.  What was there has been read: P_t came from it, and the product
      // that reads P_t was issued before (products of one thread run in order).
      auto qk = [&](int t, int h) {
        tc_fence_after();
        const uint32_t a = desc_lo(dq) + t * (C::Q_BYTES >> 4), b = desc_lo(dk0) + ks * (C::SLOT_BYTES >> 4) + h * (HALF_KV * 128 >> 4);
#pragma unroll
        for (int k = 0; k < D / UMMA_K; ++k) {
          const uint32_t off = ((k >> 2) * (128 * 128) + (k & 3) * (UMMA_K * 2)) >> 4;
          umma_f16_ss_warp(leader, tmem_base + t * BLOCK_KV + h * HALF_KV, a + off, desc_hi(dq), b + off, desc_hi(dk0), p.idesc_qk,
                           k > 0 ? 1u : 0u);
        }
        umma_commit_warp(leader, &s_full[2 * t + h]);
      };
      auto pv = [&](int t, int h, bool first) -> bool {
        const int i = 2 * t + h;
        if (!warp_wait(&p_full[i], (phase >> i) & 1)) return false;      // O_t rescaled if it had to be
        phase ^= 1u << i;
        // O accumulates in TMEM over all steps (the first MMA of a unit overwrites, unless the accumulator was
        // pre-loaded with the state of earlier launches); P: 16 keys = 8 columns
        const bool fresh = first && !resume;
        if (fresh && !warp_wait(&o_empty[t], (uint32_t)((uses[t] & 1) ^ 1))) return false;
        tc_fence_after();
        const uint32_t b = desc_lo(dv0) + vs * (C::SLOT_BYTES >> 4) + h * (HALF_KV * 128 >> 4);
#pragma unroll
        for (int k = 0; k < HALF_KV / UMMA_K; ++k)
          umma_f16_ts_warp(leader, tmem_base + C::O_COL + t * D, tmem_base + t * BLOCK_KV + h * HALF_KV + k * 8,
                           b + (k * (UMMA_K * 128) >> 4), desc_hi(dv0), p.idesc_pv, (fresh && k == 0) ? 0u : 1u);
        umma_commit_warp(leader, &o_full[i]);
        return true;
      };
      bool ok = warp_wait(q_full, (uint32_t)(nq & 1)) && take(ks);
      if (!ok) break;
      if (n0 > 0) qk(0, 0);
      if (n1 > 0) qk(1, 0);
      if (n0 > 1) qk(0, 1);
      if (n1 > 1) qk(1, 1);
      umma_commit_warp(leader, &empty[ks]);
      if (tiles == 1) umma_commit_warp(leader, q_empty);       // the unit's last Q K^T has been issued
      for (int j = 0; j < tiles && ok; ++j) {
        ok = take(vs) && (j + 1 == tiles || take(ks));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int s = 2 * j + h;
          if (ok && s < n0) {
            ok = pv(0, h, s == 0);
            if (ok && s + 2 < n0) qk(0, h);
          }
          if (ok && s < n1) {
            ok = pv(1, h, s == 0);
            if (ok && s + 2 < n1) qk(1, h);
          }
        }
        if (!ok) break;
        umma_commit_warp(leader, &empty[vs]);
        if (j + 1 < tiles) umma_commit_warp(leader, &empty[ks]);
        if (j + 2 == tiles) umma_commit_warp(leader, q_empty);
      }
      if (!ok) break;
      ++nq;
      uses[0] += n0 > 0; uses[1] += n1 > 0;
    }
    __syncwarp();
  } else if (warp >= OUTPUT_WARP0) {
    // ================================================================ output
    // What a unit ends with - its last P V, the division, the way out - runs beside the softmax of the next one.  A warp takes 32
    // rows of either tile, and through shared memory, so that a store writes whole lines: a lane's own row at a time, every 16
    // bytes in another line, held up the softmax warps for 8700 clocks per unit of D = 128 (70000 for one of 2112 keys).
    const int quarter = warp & 3;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    uint8_t* box = smem_box + quarter * C::BOX_BYTES;
    constexpr int CHUNKS = D / 8;                          // 16-byte pieces of a row
    uint32_t phase = 0, units_of = 0;                      // bit 2 t + h: parity of the next P V of half h;  bit t: of the next unit
    bool ok = true;
    auto warp_wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag)) != 0; };
    while (ok && next_unit()) {
#pragma unroll 1
      for (int t = 0; t < 2 && ok; ++t) {
        const int n = steps_of(t);
        if (n == 0) continue;
        // the softmax warps are through: S of the last step has come, so the P V before the last of either half has retired
        ok = warp_wait(&row_full[t], (units_of >> t) & 1);
        if (!ok) break;
        units_of ^= 1u << t;
        const int last = 2 * t + ((n - 1) & 1);
        phase ^= (uint32_t)(((n + 1) / 2) & 1) << (2 * t) | (uint32_t)((n / 2) & 1) << (2 * t + 1);
        const int r = quarter * 32 + lane;
        const float2 ml = smem_row[t * BLOCK_Q + r];
        __syncwarp();
        if (lane == 0) mbar_arrive(&row_empty[t]);
        ok = warp_wait(&o_full[last], ((phase >> last) & 1) ^ 1);
        if (!ok) break;
        tc_fence_after();
        const int head = head_of(t), row0 = tile_of(t) * BLOCK_Q + quarter * 32, live = un.len_q - row0;   // rows of this warp
        const size_t token0 = (size_t)un.q_start + row0, ld = (size_t)p.hq * D;
        const float inv_l = ml.y > 0.f ? 1.f / ml.y : 0.f;
#pragma unroll
        for (int c = 0; c < D; c += 32) {
          uint32_t w[32];
          tmem_ld_32x32b_x32(tmem_base + lane_addr + C::O_COL + t * D + c, w);
          tmem_ld_wait();
          if (c + 32 == D) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&o_empty[t]);       // O_t may be overwritten by the next unit
          }
          if (p.o_state != nullptr) {
            if (lane < live) {
              float4* dst = reinterpret_cast<float4*>(p.o_state + (token0 + lane) * ld + (size_t)head * D + c);
#pragma unroll
              for (int i = 0; i < 8; ++i)
                dst[i] = make_float4(__uint_as_float(w[4 * i]) * inv_l, __uint_as_float(w[4 * i + 1]) * inv_l,
                                     __uint_as_float(w[4 * i + 2]) * inv_l, __uint_as_float(w[4 * i + 3]) * inv_l);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint32_t h[4];
#pragma unroll
              for (int e = 0; e < 4; ++e)
                h[e] = pack_16<BF16>(__uint_as_float(w[8 * i + 2 * e]) * inv_l, __uint_as_float(w[8 * i + 2 * e + 1]) * inv_l);
              *reinterpret_cast<uint4*>(box + (lane * CHUNKS + ((c / 8 + i) ^ (lane & 7))) * 16) = make_uint4(h[0], h[1], h[2], h[3]);
            }
          }
        }
        if (p.o_state == nullptr) {
          __syncwarp();
          uint8_t* out = reinterpret_cast<uint8_t*>(p.out) + (token0 * ld + (size_t)head * D) * 2;
#pragma unroll
          for (int i = 0; i < CHUNKS; ++i) {
            const int at = i * 32 + lane, row = at / CHUNKS, chunk = at % CHUNKS;
            const uint4 x = *reinterpret_cast<const uint4*>(box + (row * CHUNKS + (chunk ^ (row & 7))) * 16);
            if (row < live) *reinterpret_cast<uint4*>(out + row * (ld * 2) + chunk * 16) = x;
          }
          __syncwarp();
        }
        if (p.lse && lane < live)
          p.lse[(token0 + lane) * p.hq + head] = ml.y > 0.f ? (ml.x + log2f(ml.y)) * 0.6931471805599453f : -INFINITY;
      }
    }
  } else if (warp >= SOFTMAX_WARP0) {
    // ================================================================ softmax
    // Thread = query row.  The output accumulator lives in TMEM for the whole walk (P_j V_j accumulates onto it in the
    // tensor core); the exponentials are taken against a LAGGING row max: the accumulator is only rescaled when the
    // true max has grown by more than 2^TAU since the last rescale (exact: numerator and denominator use the same
    // reference, which is what the log-sum-exp is reported against).
    constexpr float TAU = 8.f;
    const int t = (warp - SOFTMAX_WARP0) >> 2;           // this warp's query tile
    const int quarter = warp & 3;                        // TMEM lane quarter this warp may access
    const int r = quarter * 32 + lane;                   // query row inside the tile
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint32_t o_addr = tmem_base + lane_addr + C::O_COL + t * D;
    const uint32_t s_addr = tmem_base + lane_addr + t * BLOCK_KV;
    uint32_t phase = 0, units_of = 0;                    // bit h: parity of the next S_t in half h; units of this tile so far
    // The two tiles' warps of a quarter share a scheduler and exponentiate in turn, tile 0 first: at once each took twice as long, while
    // nothing ran under the maxima, loads and waits of both.  They have as many turns in a unit as the longer tile has steps.
    uint32_t turns = t ^ 1;                              // parity of the next turn
    uint64_t* const mine = &turn[4 * t + quarter];
    uint64_t* const theirs = &turn[4 * (t ^ 1) + quarter];
    auto take_turn = [&]() -> bool {
      if (!TURNS) return true;
      const bool here = __all_sync(0xffffffffu, wait_or_abort(mine, turns & 1, abort_flag)) != 0;
      turns ^= 1;
      return here;
    };
    auto pass_turn = [&]() {
      if (!TURNS) return;
      __syncwarp();
      if (lane == 0) mbar_arrive(theirs);
    };
    bool ok = true;
    while (ok && next_unit()) {
      const int n_steps = steps_of(t), turns_of_unit = TURNS ? max(n_steps, steps_of(t ^ 1)) : n_steps;
      if (n_steps == 0) {
        for (int j = 0; j < turns_of_unit && ok; ++j) { ok = take_turn(); pass_turn(); }
        continue;
      }
      const int q_tile = tile_of(t), head = head_of(t), len_k = un.len_k;
      const int kv_first = first_key_tile();
      const int q_pos = q_tile * BLOCK_Q + r;              // position inside the sequence
      const size_t row = (size_t)un.q_start + q_pos;       // row in the token-major Q / O
      float m_run = -INFINITY;                             // reference max of the exponentials (exp2 domain)
      float l_run = 0.f;
      float m_ahead = -INFINITY;                           // maximum of scores that a later step takes
      if (resume) {
        ok = __all_sync(0xffffffffu, wait_or_abort(&o_empty[t], (units_of & 1) ^ 1, abort_flag));
        if (!ok) break;
        tc_fence_after();
        // resume from the merged result of the key blocks processed by earlier launches (normalised output + LSE):
        // every row stores its previous output (or zeros) into the TMEM accumulator, P_0 V_0 accumulates onto it
        float lse_prev = -INFINITY;
        if (q_pos < un.len_q) lse_prev = p.lse[row * p.hq + head];
        const bool live = lse_prev > -INFINITY;
        if (live) { m_run = lse_prev * 1.4426950408889634f; l_run = 1.f; }
        const float4* src = reinterpret_cast<const float4*>(p.o_state + row * ((size_t)p.hq * D) + (size_t)head * D);
#pragma unroll
        for (int c = 0; c < D; c += 16) {
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 t4 = live ? src[(c >> 2) + i] : make_float4(0.f, 0.f, 0.f, 0.f);
            w[4 * i] = __float_as_uint(t4.x); w[4 * i + 1] = __float_as_uint(t4.y);
            w[4 * i + 2] = __float_as_uint(t4.z); w[4 * i + 3] = __float_as_uint(t4.w);
          }
          tmem_st_32x32b_x16(o_addr + c, w);
        }
        tmem_st_wait();
      }
      const float slope2 = (EXTRA && p.alibi != nullptr) ? p.alibi[head] * 1.4426950408889634f : 0.f;
      (void)slope2;
      // P V of step j, the last one in its half: the one before in that half retired before S of step j came
      auto product_done = [&](int j) -> bool {
        const int h = j & 1;
        return __all_sync(0xffffffffu, wait_or_abort(&o_full[2 * t + h], ((phase >> h) & 1) ^ 1, abort_flag)) != 0;
      };
      // plain variant: the softmax scale (> 0) is folded into the exponent's FMA, the max is taken on the raw scores;
      // EXTRA variant: scale and ALiBi bias are applied here and the exponent uses a unit multiplier
      const float ex_mul = EXTRA ? 1.f : p.scale_log2;
      auto visible = [&](uint32_t (&v)[HALF_KV], int k_base, auto masked_tag) {
        constexpr bool MASKED = decltype(masked_tag)::value;
        if (EXTRA || MASKED) {
          const int k_lim = p.causal ? min(q_pos, len_k - 1) : len_k - 1;                        // last visible key of this row
          const int k_low = (EXTRA && p.window > 0) ? q_pos - p.window + 1 : 0;                  // first visible key
#pragma unroll
          for (int i = 0; i < HALF_KV; ++i) {
            float sc = __uint_as_float(v[i]);
            if (EXTRA) sc = fmaf(slope2, (float)(k_base + i - q_pos), sc * p.scale_log2);
            if (MASKED && ((k_base + i) > k_lim || (EXTRA && (k_base + i) < k_low))) sc = -INFINITY;
            v[i] = __float_as_uint(sc);
          }
        }
      };
      // (four independent partial maxima / sums: a single running value would be a 64-long dependent chain)
      auto largest = [&](const uint32_t (&v)[HALF_KV]) {
        float mt[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < HALF_KV; i += 8)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            mt[e] = fmaxf(fmaxf(mt[e], __uint_as_float(v[i + e])), __uint_as_float(v[i + e + 4]));
        return fmaxf(fmaxf(mt[0], mt[1]), fmaxf(mt[2], mt[3])) * ex_mul;
      };
      auto load = [&](uint32_t (&v)[HALF_KV], int j) {
#pragma unroll
        for (int c = 0; c < HALF_KV; c += 32)
          tmem_ld_32x32b_x32(s_addr + (j & 1) * HALF_KV + c, *reinterpret_cast<uint32_t(*)[32]>(&v[c]));
        tmem_ld_wait();
      };
      // the largest score of step j, in the exp2 domain
      auto row_max = [&](int j, auto masked_tag) {
        uint32_t v[HALF_KV];
        load(v, j);
        visible(v, kv_first * BLOCK_KV + j * HALF_KV, masked_tag);
        return largest(v);
      };
      // one step of 64 keys; two copies of the code, because a branch around the mask alone is turned into predicated
      // comparisons and selections that every step executes
      auto step = [&](int j, auto masked_tag) -> bool {
        const uint32_t half_addr = s_addr + (j & 1) * HALF_KV;
        uint32_t v[HALF_KV];
        load(v, j);
        visible(v, kv_first * BLOCK_KV + j * HALF_KV, masked_tag);
        const float m_tile = fmaxf(largest(v), m_ahead);
        m_ahead = -INFINITY;
        // ---- lagging max / rare rescale of the TMEM accumulator
        const float m_new = fmaxf(m_run, m_tile);
        if (j == 0 && !resume) {
          m_run = m_new;                                       // nothing accumulated yet
        } else {
          const bool need = (m_new - m_run) > TAU;             // (-inf) - (-inf) = NaN -> false
          if (__any_sync(0xffffffffu, need)) {
            if (j > 0) {
              if (!product_done(j - 1)) return false;
              tc_fence_after();
            }
            const float alpha = need ? fast_exp2(m_run - m_new) : 1.f;
#pragma unroll 1
            for (int c = 0; c < D; c += 16) {
              uint32_t w[16];
              tmem_ld_32x32b_x16(o_addr + c, w);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(__uint_as_float(w[i]) * alpha);
              tmem_st_32x32b_x16(o_addr + c, w);
            }
            tmem_st_wait();
            l_run *= alpha;
            if (need) m_run = m_new;
          }
        }
        const float m_use = (m_run == -INFINITY) ? 0.f : m_run;     // keeps the exponent finite on a fully masked row
        // ---- p = exp2(s - m), row sum, 16-bit P over the scores it came from
        const uint64_t mul2 = pack_f32x2(ex_mul, ex_mul), sub2 = pack_f32x2(-m_use, -m_use);
        uint64_t lt[2] = {0ull, 0ull};
        if (!take_turn()) return false;
#pragma unroll
        for (int c = 0; c < HALF_KV; c += 32) {
          uint32_t packed[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            if (c + i == 48) pass_turn();                          // (32 to 56 are the same, 64 is 5 % slower)
            float p0, p1;
            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[c + i]), __uint_as_float(v[c + i + 1])), mul2, sub2), p0, p1);
            p0 = fast_exp2(p0);
            p1 = fast_exp2(p1);
            lt[(i >> 1) & 1] = add_f32x2(lt[(i >> 1) & 1], pack_f32x2(p0, p1));
            packed[i >> 1] = pack_16<BF16>(p0, p1);
          }
          tmem_st_32x32b_x16(half_addr + (c >> 1), packed);
        }
        float l0, l1, l2, l3;
        unpack_f32x2(lt[0], l0, l1);
        unpack_f32x2(lt[1], l2, l3);
        l_run += (l0 + l1) + (l2 + l3);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[2 * t + (j & 1)]);  // P is in tensor memory, the accumulator is consistent
        return true;
      };
      // a step needs the mask if its last key is behind what this warp's first row sees, or behind the end of the sequence
      const int k_all = p.causal ? min(q_tile * BLOCK_Q + quarter * 32, len_k - 1) : len_k - 1;
      auto needs_mask = [&](int j) { return kv_first * BLOCK_KV + j * HALF_KV + HALF_KV - 1 > k_all || (EXTRA && p.window > 0); };
      // The first reference is the maximum of the whole first key tile: against that of its first half, a row whose largest score is
      // in the second rounds its largest weight, which is exactly one otherwise (16 x 1024 tokens, heads of 64: error 2.051e-3, 2.035e-3
      // so, for 189 and 194.5 us; both halves of a tile in one product 193.5, but 2 x 8192 tokens 944 instead of 926).
      if (n_steps > 1) {
        ok = __all_sync(0xffffffffu, wait_or_abort(&s_full[2 * t + 1], (phase >> 1) & 1, abort_flag));
        if (!ok) break;
        tc_fence_after();
        m_ahead = needs_mask(1) ? row_max(1, std::true_type{}) : row_max(1, std::false_type{});
      }
      for (int j = 0; j < n_steps && ok; ++j) {
        const int h = j & 1;
        ok = __all_sync(0xffffffffu, wait_or_abort(&s_full[2 * t + h], (phase >> h) & 1, abort_flag));
        if (!ok) break;
        phase ^= 1u << h;
        tc_fence_after();
        ok = needs_mask(j) ? step(j, std::true_type{}) : step(j, std::false_type{});
      }
      for (int j = n_steps; j < turns_of_unit && ok; ++j) { ok = take_turn(); pass_turn(); }
      if (!ok) break;
      // ---- the row's maximum and sum go to the output warps
      ok = __all_sync(0xffffffffu, wait_or_abort(&row_empty[t], (units_of & 1) ^ 1, abort_flag));
      if (!ok) break;
      ++units_of;
      smem_row[t * BLOCK_Q + r] = make_float2(m_run, l_run);
      __syncwarp();
      if (lane == 0) mbar_arrive(&row_full[t]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {                         // (nothing writes it any more: uniform) leave nothing in flight behind
    int none = 0;
    if (warp == 0 && lane == 0) {
      const int issued = copies[0], nq = copies[1];
      if (nq > 0) wait_or_abort(q_full, (uint32_t)((nq - 1) & 1), &none);
      for (int i = max(0, issued - SLOTS); i < issued; ++i) {
        none = 0;
        wait_or_abort(&full[i % SLOTS], (uint32_t)((i / SLOTS) & 1), &none);
      }
    }
    if (warp == 1 && elect_one()) {          // the thread that issued the products
      umma_commit(drained);
      wait_or_abort(drained, 0, &none);
    }
    __syncthreads();
    if (threadIdx.x == 0) report_abort(p.status);
  }
  if (warp == 2) tmem_dealloc<C::TMEM_COLS>(tmem_base);
}

// One query tile per CTA, for calls whose tiles all find an SM at once: six warps (producer, issuer, four softmax warps of one
// thread per row), two score buffers so that Q K^T of the next key tile runs under the softmax of this one, P through shared
// memory.  With a single tile to walk the two-tile kernel has nothing to put under it - at heads of 128 its next Q K^T even
// waits for P V - and the walk of a CTA is the call: 32 / 8 heads of 128, 256 / 512 tokens 15.7 / 21.3
// us in the two-tile kernel, 8.8 / 13.1 here; 12 heads, 1024 tokens 29.5 and 20.5; 32 heads, 1024 tokens (256 tiles) 31 in both.
constexpr int TILE_THREADS = 192, TILE_KV_STAGES = 2;
template <int D> struct FaTileCfg {
  static constexpr int Q_BYTES = BLOCK_Q * D * 2;
  static constexpr int K_BYTES = BLOCK_KV * D * 2;
  static constexpr int V_BYTES = BLOCK_KV * D * 2;
  static constexpr int P_BYTES = BLOCK_Q * BLOCK_KV * 2;
  static constexpr int KV_STAGE_BYTES = K_BYTES + V_BYTES;
  static constexpr int SMEM_BYTES = Q_BYTES + TILE_KV_STAGES * KV_STAGE_BYTES + 2 * P_BYTES + 1024 /*align*/ + 256 /*barriers*/;
  static constexpr int TMEM_COLS = 512;
  static constexpr int O_COL = 256;
};

template <int D, bool EXTRA, bool BF16>
__global__ void __launch_bounds__(TILE_THREADS, 1)
flash_fwd_tile_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                 const __grid_constant__ CUtensorMap tmap_v, const FaParams p) {
  using C = FaTileCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_q = smem;
  uint8_t* smem_kv = smem + C::Q_BYTES;
  uint8_t* smem_p = smem_kv + TILE_KV_STAGES * C::KV_STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_p + 2 * C::P_BYTES);
  uint64_t* q_full = bars;                 // [1]
  uint64_t* kv_full = bars + 1;            // [2]
  uint64_t* kv_empty = bars + 3;           // [2]
  uint64_t* s_full = bars + 5;             // [2]
  uint64_t* s_empty = bars + 7;            // [2]  4 softmax warps
  uint64_t* p_full = bars + 9;             // [1]  4 softmax warps
  uint64_t* o_full = bars + 10;            // [1]
  uint64_t* o_empty = bars + 11;           // [1]  4 softmax warps
  uint64_t* drained = bars + 12;           // [1]  a CTA that gives up: its products have retired
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 13);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  volatile int* copies = abort_flag + 1;   // [1]  key / value tiles that the producer asked for

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int head = blockIdx.y;
  const int kv_head = head / (p.hq / p.hkv);
  int q_tile, seq_row0, len_q, len_k;
  if (p.cu_seqlens != nullptr) {
    // packed batch: blockIdx.x enumerates (sequence, query tile) pairs in order; surplus CTAs (the grid is sized for
    // the worst case without knowing the lengths on the host) leave at once
    int t = (int)blockIdx.x, bsel = -1, start = 0, len = 0;
    for (int bb = 0; bb < p.batch; ++bb) {
      start = p.cu_seqlens[bb];
      len = p.cu_seqlens[bb + 1] - start;
      const int nt = (len + BLOCK_Q - 1) / BLOCK_Q;
      if (t < nt) { bsel = bb; break; }
      t -= nt;
    }
    if (bsel < 0) return;                      // uniform across the CTA: nothing has been allocated yet
    q_tile = t; seq_row0 = start; len_q = len; len_k = len;
  } else {
    // heaviest (longest causal) query tiles first
    const int q_tiles = (p.seqlen_q + BLOCK_Q - 1) / BLOCK_Q;
    q_tile = p.causal ? (q_tiles - 1 - (int)blockIdx.x) : (int)blockIdx.x;
    seq_row0 = -1; len_q = p.seqlen_q; len_k = p.seqlen_k;
  }
  const int b = blockIdx.z;
  const int q_row0 = (seq_row0 >= 0 ? seq_row0 : b * p.seqlen_q) + q_tile * BLOCK_Q;   // row in the token-major Q / O
  const int kv_row0 = seq_row0 >= 0 ? seq_row0 : b * p.seqlen_k;
  const int kv_tiles_all = (len_k + BLOCK_KV - 1) / BLOCK_KV;
  // causal with seqlen_q == seqlen_k: key tiles 0..q_tile; otherwise all of them
  const int kv_last = p.causal ? min(q_tile + 1, kv_tiles_all) : kv_tiles_all;   // one past the last visible key tile
  // sliding window: the lowest key any row of this query tile can see is (q_tile * BLOCK_Q - window + 1)
  const int kv_first = (EXTRA && p.window > 0) ? max(0, q_tile * BLOCK_Q - p.window + 1) / BLOCK_KV : 0;
  const int kv_tiles = kv_last - kv_first;         // tiles walked; loop index j <-> key tile kv_first + j
  const bool ragged_k = (len_k % BLOCK_KV) != 0;   // the last key tile runs past the end of the sequence
  const bool resume = p.o_state != nullptr && p.has_prev != 0;   // block mode: continue from the stored state

  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tmap_q);
    prefetch_tensormap(&tmap_k);
    prefetch_tensormap(&tmap_v);
  }
  if (warp == 1 && lane == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&s_empty[i], 4);
    }
    mbar_init(p_full, 4);
    mbar_init(o_full, 1);
    mbar_init(o_empty, 4);
    mbar_init(drained, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 2) tmem_alloc<C::TMEM_COLS>(tmem_ptr_smem);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  auto warp_wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag)) != 0; };

  if (warp == 0) {
    // ================================================================ TMA producer
    if (lane == 0) {
      mbar_arrive_expect_tx(q_full, C::Q_BYTES);
#pragma unroll
      for (int h = 0; h < D / 64; ++h)                     // boxes [128 rows, 64 d] -> K-major swizzled sub-tiles
        tma_load_2d(&tmap_q, q_full, smem_q + h * (BLOCK_Q * 128), head * D + h * 64, q_row0);
    }
    if (lane == 0) {
      int j = 0;
      for (; j < kv_tiles; ++j) {
        const int stage = j % TILE_KV_STAGES;
        if (!wait_or_abort(&kv_empty[stage], (uint32_t)(((j / TILE_KV_STAGES) & 1) ^ 1), abort_flag)) break;
        uint8_t* sk = smem_kv + stage * C::KV_STAGE_BYTES;
        uint8_t* sv = sk + C::K_BYTES;
        mbar_arrive_expect_tx(&kv_full[stage], C::KV_STAGE_BYTES);
        const int row = kv_row0 + (kv_first + j) * BLOCK_KV;
#pragma unroll
        for (int h = 0; h < D / 64; ++h) {
          tma_load_2d(&tmap_k, &kv_full[stage], sk + h * (BLOCK_KV * 128), kv_head * D + h * 64, row);   // K-major B
          tma_load_2d(&tmap_v, &kv_full[stage], sv + h * (BLOCK_KV * 128), kv_head * D + h * 64, row);   // MN-major B
        }
      }
      *copies = j;
    }
    __syncwarp();
  } else if (warp == 1) {
    // ================================================================ MMA issuer
    const uint32_t sq = smem_u32(smem_q);
    const uint32_t sp = smem_u32(smem_p);
    const uint64_t dq = make_smem_desc_sw128(sq, 16, 1024);                       // K-major, K = D
    const uint64_t dp = make_smem_desc_sw128(sp, 16, 1024);                       // K-major, K = keys
    if (lane == 0) {
      auto issue_qk = [&](int j) -> bool {
        const int stage = j % TILE_KV_STAGES;
        const int sb = j & 1;
        if (!wait_or_abort(&kv_full[stage], (uint32_t)((j / TILE_KV_STAGES) & 1), abort_flag)) return false;
        if (!wait_or_abort(&s_empty[sb], (uint32_t)(((j >> 1) & 1) ^ 1), abort_flag)) return false;
        tc_fence_after();
        const uint64_t dk = make_smem_desc_sw128(smem_u32(smem_kv + stage * C::KV_STAGE_BYTES), 16, 1024);
#pragma unroll
        for (int k = 0; k < D / UMMA_K; ++k) {
          const uint32_t off = (k >> 2) * (128 * 128) + (k & 3) * (UMMA_K * 2);
          umma_f16_ss(tmem_base + sb * BLOCK_KV, advance_desc(dq, off), advance_desc(dk, off), p.idesc_qk, k > 0 ? 1u : 0u);
        }
        umma_commit(&s_full[sb]);
        return true;
      };
      bool ok = wait_or_abort(q_full, 0, abort_flag) && issue_qk(0);
      for (int j = 0; j < kv_tiles && ok; ++j) {
        if (j + 1 < kv_tiles) ok = issue_qk(j + 1);         // tensor pipe works on the next scores during softmax(j)
        const int stage = j % TILE_KV_STAGES;
        ok = ok && wait_or_abort(p_full, (uint32_t)(j & 1), abort_flag);   // P_j is in shared memory, O rescaled if it had to be
        if (!ok) break;
        tc_fence_after();
        const uint32_t sv = smem_u32(smem_kv + stage * C::KV_STAGE_BYTES + C::K_BYTES);
        const uint64_t dv = make_smem_desc_sw128(sv, BLOCK_KV * 128, 1024);          // MN-major: [keys, D] row-major
        const uint64_t dpj = advance_desc(dp, (uint32_t)(j & 1) * C::P_BYTES);
        // O accumulates in TMEM over all key tiles (the first MMA of the first tile overwrites, unless the accumulator was
        // pre-loaded with the state of earlier launches)
        const bool fresh = (j == 0) && !resume;
#pragma unroll
        for (int k = 0; k < BLOCK_KV / UMMA_K; ++k) {
          const uint32_t ao = (k >> 2) * (128 * 128) + (k & 3) * (UMMA_K * 2);
          umma_f16_ss(tmem_base + C::O_COL, advance_desc(dpj, ao), advance_desc(dv, k * (UMMA_K * 128)), p.idesc_pv,
                      (fresh && k == 0) ? 0u : 1u);
        }
        umma_commit(o_full);
        umma_commit(&kv_empty[stage]);                      // K_j and V_j are consumed once P_j V_j has retired
      }
    }
    __syncwarp();
  } else {
    // ================================================================ softmax + output (warps 2..5)
    // Thread = query row.  The output accumulator lives in TMEM for the whole walk (P_j V_j accumulates onto it in the
    // tensor core); the exponentials are taken against a LAGGING row max: the accumulator is only rescaled when the
    // true max has grown by more than 2^TAU since the last rescale (exact: numerator and denominator use the same
    // reference, which is what the log-sum-exp is reported against).  Per key tile a thread therefore reads its 128
    // scores ONCE (four tcgen05.ld in flight, one wait), releases the score buffer at once, and touches the
    // accumulator only on the rare rescale.
    constexpr float TAU = 8.f;
    const int quarter = warp & 3;                        // TMEM lane quarter this warp may access
    const int r = quarter * 32 + lane;                   // query row inside the tile
    const int q_pos = q_tile * BLOCK_Q + r;              // position inside the sequence
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint32_t o_addr = tmem_base + lane_addr + C::O_COL;
    float m_run = -INFINITY;                             // reference max of the exponentials (exp2 domain)
    float l_run = 0.f;
    if (resume) {
      // resume from the merged result of the key blocks processed by earlier launches (normalised output + LSE):
      // every row stores its previous output (or zeros) into the TMEM accumulator, P_0 V_0 accumulates onto it
      const size_t row_ = (size_t)q_row0 + r;
      float lse_prev = -INFINITY;
      if (q_pos < len_q) lse_prev = p.lse[row_ * p.hq + head];
      const bool live = lse_prev > -INFINITY;
      if (live) { m_run = lse_prev * 1.4426950408889634f; l_run = 1.f; }
      const float4* src = reinterpret_cast<const float4*>(p.o_state + row_ * ((size_t)p.hq * D) + (size_t)head * D);
#pragma unroll
      for (int c = 0; c < D; c += 16) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 t4 = live ? src[(c >> 2) + i] : make_float4(0.f, 0.f, 0.f, 0.f);
          w[4 * i] = __float_as_uint(t4.x); w[4 * i + 1] = __float_as_uint(t4.y);
          w[4 * i + 2] = __float_as_uint(t4.z); w[4 * i + 3] = __float_as_uint(t4.w);
        }
        tmem_st_32x32b_x16(o_addr + c, w);
      }
      tmem_st_wait();
    }
    const float slope2 = (EXTRA && p.alibi != nullptr) ? p.alibi[head] * 1.4426950408889634f : 0.f;
    (void)slope2;
    bool ok = true;                                      // this thread's waits so far
    int j = 0;
    for (; j < kv_tiles; ++j) {
      const int sb = j & 1;
      ok = ok && wait_or_abort(&s_full[sb], (uint32_t)((j >> 1) & 1), abort_flag);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      const uint32_t s_addr = tmem_base + lane_addr + sb * BLOCK_KV;
      const int kt = kv_first + j;                                       // key tile of this step
      const bool diag = p.causal && (kt == q_tile);
      const bool tail_k = ragged_k && (kt == kv_tiles_all - 1);
      const bool masked = diag || tail_k || (EXTRA && p.window > 0);
      const int k_lim = diag ? min(q_pos, len_k - 1) : (len_k - 1);      // last visible key position of this row
      const int k_low = (EXTRA && p.window > 0) ? q_pos - p.window + 1 : 0;   // first visible key position
      const int k_base = kt * BLOCK_KV;
      // ---- the whole score row into registers
      uint32_t v[BLOCK_KV];
#pragma unroll
      for (int c = 0; c < BLOCK_KV; c += 32) tmem_ld_32x32b_x32(s_addr + c, *reinterpret_cast<uint32_t(*)[32]>(&v[c]));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_empty[sb]);          // S buffer may be overwritten by Q K_{j+2}^T
      // plain variant: the softmax scale (> 0) is folded into the exponent's FMA, the max is taken on the raw scores;
      // EXTRA variant: scale and ALiBi bias are applied here and the exponent uses a unit multiplier
      // (four independent partial maxima / sums: a single running value would be a 128-long dependent chain)
      float mt[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < BLOCK_KV; ++i) {
        float sc = __uint_as_float(v[i]);
        if (EXTRA) sc = fmaf(slope2, (float)(k_base + i - q_pos), sc * p.scale_log2);
        if (masked && ((k_base + i) > k_lim || (EXTRA && (k_base + i) < k_low))) sc = -INFINITY;
        v[i] = __float_as_uint(sc);
        mt[i & 3] = fmaxf(mt[i & 3], sc);
      }
      float m_tile = fmaxf(fmaxf(mt[0], mt[1]), fmaxf(mt[2], mt[3]));
      const float ex_mul = EXTRA ? 1.f : p.scale_log2;
      m_tile *= ex_mul;
      // ---- lagging max / rare rescale of the TMEM accumulator
      const float m_new = fmaxf(m_run, m_tile);
      if (j == 0 && !resume) {
        m_run = m_new;                                   // nothing accumulated yet
      } else {
        const bool need = (m_new - m_run) > TAU;         // (-inf) - (-inf) = NaN -> false
        if (__any_sync(0xffffffffu, need)) {
          if (j > 0) {                                   // P_{j-1} V_{j-1} has retired: the accumulator is stable
            if (!warp_wait(o_full, (uint32_t)((j - 1) & 1))) break;
            tc_fence_after();
          }
          const float alpha = need ? fast_exp2(m_run - m_new) : 1.f;
#pragma unroll 1
          for (int c = 0; c < D; c += 32) {
            uint32_t t[32];
            tmem_ld_32x32b_x32(o_addr + c, t);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) t[i] = __float_as_uint(__uint_as_float(t[i]) * alpha);
            tmem_st_32x32b_x16(o_addr + c, *reinterpret_cast<uint32_t(*)[16]>(&t[0]));
            tmem_st_32x32b_x16(o_addr + c + 16, *reinterpret_cast<uint32_t(*)[16]>(&t[16]));
          }
          tmem_st_wait();
          l_run *= alpha;
          if (need) m_run = m_new;
        }
      }
      const float m_use = (m_run == -INFINITY) ? 0.f : m_run;     // keeps the exponent finite on a fully masked row
      // ---- p = exp2(s - m), row sum, 16-bit P into the swizzled K-major tile of buffer j & 1
      // (that buffer was last read by P_{j-2} V_{j-2}, which retired before Q K_j^T - issued after it - completed)
      uint8_t* p_row = smem_p + (j & 1) * C::P_BYTES + r * 128;
      float lt[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < BLOCK_KV; c += 32) {
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float p0 = fast_exp2(fmaf(__uint_as_float(v[c + i]), ex_mul, -m_use));
          const float p1 = fast_exp2(fmaf(__uint_as_float(v[c + i + 1]), ex_mul, -m_use));
          lt[(i >> 1) & 3] += p0 + p1;
          packed[i >> 1] = pack_16<BF16>(p0, p1);
        }
        // 32 keys = 64 bytes = four 16-byte chunks of this row inside sub-tile (c / 64)
        uint8_t* sub = p_row + (c >> 6) * (BLOCK_Q * 128);
        const int chunk0 = (c & 32) ? 4 : 0;
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          const int chunk = (chunk0 + q4) ^ (r & 7);     // SWIZZLE_128B: 16-byte chunk index XOR (row mod 8)
          *reinterpret_cast<uint4*>(sub + chunk * 16) =
              make_uint4(packed[q4 * 4], packed[q4 * 4 + 1], packed[q4 * 4 + 2], packed[q4 * 4 + 3]);
        }
      }
      const float l_tile = (lt[0] + lt[1]) + (lt[2] + lt[3]);
      l_run += l_tile;
      // keep in step with the accumulator barrier: observe "P_{j-1} V_{j-1} retired" once per tile.  It completed long
      // ago in the common case (no stall), but a parity wait is only unambiguous while the waiter is at most ONE phase
      // behind - the epilogue's wait for the last tile would otherwise pass on the phase before the previous one
      // (seen on hardware with two-tile launches: output read before the last two P V had landed).
      if (j > 0) ok = wait_or_abort(o_full, (uint32_t)((j - 1) & 1), abort_flag);
      tc_fence_before();
      fence_proxy_async();                               // generic-proxy smem writes -> visible to the tensor core
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);                // P_j is in shared memory, the accumulator is consistent
    }
    // ---- epilogue: the last P V has retired; normalise and store this thread's row
    ok = __all_sync(0xffffffffu, ok && j == kv_tiles && wait_or_abort(o_full, (uint32_t)((kv_tiles - 1) & 1), abort_flag));
    tc_fence_after();
    const float inv_l = l_run > 0.f ? 1.f / l_run : 0.f;
    const size_t row = (size_t)q_row0 + r;
    const bool row_ok = q_pos < len_q;                   // rows past the end of a (packed) sequence are never stored
#pragma unroll 1
    for (int c = 0; c < D && ok; c += 32) {
      uint32_t t[32];
      __syncwarp();
      tmem_ld_32x32b_x32(o_addr + c, t);                 // executed by every lane (warp-collective), stores predicated
      tmem_ld_wait();
      if (!row_ok) {
        // a row past the end of its (packed) sequence: computed on garbage, never stored
      } else if (p.o_state != nullptr) {
        float4* dst = reinterpret_cast<float4*>(p.o_state + row * ((size_t)p.hq * D) + (size_t)head * D + c);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          dst[i] = make_float4(__uint_as_float(t[4 * i]) * inv_l, __uint_as_float(t[4 * i + 1]) * inv_l,
                               __uint_as_float(t[4 * i + 2]) * inv_l, __uint_as_float(t[4 * i + 3]) * inv_l);
      } else {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i)
          w[i] = pack_16<BF16>(__uint_as_float(t[2 * i]) * inv_l, __uint_as_float(t[2 * i + 1]) * inv_l);
        uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p.out) +
                                              (row * ((size_t)p.hq * D) + (size_t)head * D + c) * 2);
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
      }
    }
    if (ok && p.lse && row_ok)
      p.lse[row * p.hq + head] = l_run > 0.f ? (m_run + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {                         // (nothing writes it any more: uniform) leave nothing in flight behind
    int none = 0;
    if (warp == 0 && lane == 0) {
      wait_or_abort(q_full, 0, &none);
      for (int i = max(0, *copies - TILE_KV_STAGES); i < *copies; ++i) {
        none = 0;
        wait_or_abort(&kv_full[i % TILE_KV_STAGES], (uint32_t)((i / TILE_KV_STAGES) & 1), &none);
      }
    }
    if (warp == 1 && lane == 0) {            // the thread that issued the products
      umma_commit(drained);
      wait_or_abort(drained, 0, &none);
    }
    __syncthreads();
    if (threadIdx.x == 0) report_abort(p.status);
  }
  if (warp == 2) tmem_dealloc<C::TMEM_COLS>(tmem_base);
}

template <int D, bool EXTRA, bool BF16>
int launch_flash_fwd_tile_kernel(dim3 grid, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaParams& p,
                                 cudaStream_t stream) {
  using C = FaTileCfg<D>;
  static CbDeviceAttr attr;
  if (const int e = cb_allow_smem(attr, flash_fwd_tile_kernel<D, EXTRA, BF16>, C::SMEM_BYTES)) return e;
  flash_fwd_tile_kernel<D, EXTRA, BF16><<<grid, TILE_THREADS, C::SMEM_BYTES, stream>>>(tq, tk, tv, p);
  return (int)cudaGetLastError();
}

template <int D, bool EXTRA, bool BF16>
int launch_flash_fwd_kernel(dim3 grid, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaParams& p,
                            bool turns, cudaStream_t stream) {
  using C = FaCfg<D>;
  static CbDeviceAttr attr[2];
  auto kern = turns ? flash_fwd_kernel<D, EXTRA, BF16, true> : flash_fwd_kernel<D, EXTRA, BF16, false>;
  if (const int e = cb_allow_smem(attr[turns], kern, C::SMEM_BYTES)) return e;
  kern<<<grid, NUM_THREADS, C::SMEM_BYTES, stream>>>(tq, tk, tv, p);
  return (int)cudaGetLastError();
}

template <int D>
int launch_flash_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int batch, int seqlen_q,
                     int seqlen_k, int hq, int hkv, int causal, float scale, int dtype, cudaStream_t stream,
                     const int* cu_seqlens = nullptr, long long total_tokens = 0, float* o_state = nullptr,
                     int has_prev = 0, int window = 0, const float* alibi = nullptr) {
  const bool bf16 = dtype == CB_BF16;
  CUtensorMap tq, tk, tv;
  const uint64_t rows_q = cu_seqlens ? (uint64_t)total_tokens : (uint64_t)batch * seqlen_q;
  const uint64_t rows_k = cu_seqlens ? (uint64_t)total_tokens : (uint64_t)batch * seqlen_k;
  int r = make_tmap_2d_16b(&tq, q, rows_q, (uint64_t)hq * D, (uint64_t)hq * D, BLOCK_Q, 64, bf16);
  if (r) return 1000 + r;
  r = make_tmap_2d_16b(&tk, k, rows_k, (uint64_t)hkv * D, (uint64_t)hkv * D, BLOCK_KV, 64, bf16);
  if (r) return 2000 + r;
  r = make_tmap_2d_16b(&tv, v, rows_k, (uint64_t)hkv * D, (uint64_t)hkv * D, BLOCK_KV, 64, bf16);
  if (r) return 3000 + r;
  FaParams p;
  p.cu_seqlens = cu_seqlens;
  p.o_state = o_state; p.has_prev = has_prev;
  p.batch = batch; p.seqlen_q = seqlen_q; p.seqlen_k = seqlen_k; p.hq = hq; p.hkv = hkv; p.causal = causal;
  p.pair_heads = (hq / hkv) % 2 == 0;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.out = out; p.lse = lse; p.status = flash_status();
  p.window = window; p.alibi = alibi;
  p.idesc_qk = make_idesc_f16(BLOCK_Q, BLOCK_KV, bf16 ? 1 : 0, 0, 0);      // S[128 x 128] = Q (K-major) x K (K-major)
  p.idesc_pv = make_idesc_f16(BLOCK_Q, D, bf16 ? 1 : 0, 0, 1);              // O[128 x D]  = P (K-major) x V (MN-major)
  // Few tiles: one each.  Packed batches have between max(total / BLOCK_Q, batch) and total / BLOCK_Q + batch of them per head.  The
  // walks of causal tiles differ in length, so half as many again still fit beside the longest, unless many short sequences
  // fill the SMs evenly (12 heads of 128: one causal sequence of 2048 tokens, 192 tiles, 44 us here and 47 by twos; without the
  // mask 64 and 49; 4 x 512 tokens 20 and 18).
  const long long blocks = (cu_seqlens ? total_tokens + BLOCK_Q - 1 : (long long)seqlen_q + BLOCK_Q - 1) / BLOCK_Q;
  const long long tiles = cu_seqlens ? total_tokens / BLOCK_Q + batch : blocks;
  const long long few = (cu_seqlens ? (blocks > batch ? blocks : batch) : blocks * batch) * hq;
  if (few <= cb_num_sms() || (causal && (cu_seqlens || batch == 1) && few <= cb_num_sms() * 3 / 2)) {
    const dim3 grid((unsigned)tiles, hq, cu_seqlens ? 1 : batch);
    if (window > 0 || alibi != nullptr)
      return bf16 ? launch_flash_fwd_tile_kernel<D, true, true>(grid, tq, tk, tv, p, stream)
                  : launch_flash_fwd_tile_kernel<D, true, false>(grid, tq, tk, tv, p, stream);
    return bf16 ? launch_flash_fwd_tile_kernel<D, false, true>(grid, tq, tk, tv, p, stream)
                : launch_flash_fwd_tile_kernel<D, false, false>(grid, tq, tk, tv, p, stream);
  }
  // units of `per` query rows; packed: at most total / per + batch of them exist per head
  const int per = p.pair_heads ? BLOCK_Q : 2 * BLOCK_Q;
  p.head_units = p.pair_heads ? hq / 2 : hq;
  p.seq_units = cu_seqlens ? 0 : (seqlen_q + per - 1) / per;
  p.idesc_qk = make_idesc_f16(BLOCK_Q, HALF_KV, bf16 ? 1 : 0, 0, 0);
  const long long most = (cu_seqlens ? total_tokens / per + batch : (long long)p.seq_units * batch) * p.head_units;
  if (most > (1ll << 30)) return (int)cudaErrorInvalidValue;
  // In turn the tile that is ahead waits for the other: in short walks, and where the two tiles of a causal unit walk differently, for nothing.  Together / in
  // turn, us: heads of 64, units of two tiles of a head, 32 x 256 tokens of 40 / 8 heads 67 / 73, 16 x 384 65 / 70, 20 x 492 98 / 102, 10 x 768 the same,
  // 8 x 1000 7 % faster in turn; units of two heads 40 x 200 of 64 / 8 heads 118 / 121, 8 x 200 3 % faster in turn, 20 x 492 2 %, 8 x 1000 8 %.  Heads of
  // 128: 64 x 128 of 40 / 8 112 / 117, 16 x 384 77 / 78, 3 x 768 1 % faster in turn, 4 x 2000 of 32 / 8 5 %.  A template: as a branch between the
  // exponentials either form took what the slower one does, and long walks up to 12 % more.
  const long long walk = cu_seqlens ? total_tokens / (batch > 0 ? batch : 1) : seqlen_k;
  const bool turns = walk >= 704 || ((p.pair_heads || !causal) && (walk >= 320 || most <= 5 * cb_num_sms()));
  const dim3 grid((unsigned)(most < cb_num_sms() ? most : cb_num_sms()));
  if (window > 0 || alibi != nullptr)
    return bf16 ? launch_flash_fwd_kernel<D, true, true>(grid, tq, tk, tv, p, turns, stream)
                : launch_flash_fwd_kernel<D, true, false>(grid, tq, tk, tv, p, turns, stream);
  return bf16 ? launch_flash_fwd_kernel<D, false, true>(grid, tq, tk, tv, p, turns, stream)
              : launch_flash_fwd_kernel<D, false, false>(grid, tq, tk, tv, p, turns, stream);
}


// =====================================================================================================================
// Flash attention BACKWARD on tcgen05 / TMEM.
//
//   P = exp(scale * Q K^T - LSE),  dP = dO V^T,  dS = P o (dP - delta),  delta = rowsum(dO o O)
//   dV = P^T dO,   dK = scale * dS^T Q,   dQ = scale * dS K
//
// One CTA owns ONE key tile (128 keys) of ONE kv head and walks over every query tile (64 rows) of every query head of
// its GQA group that can see it.  dK / dV therefore accumulate in TMEM across the whole walk - over the query tiles AND
// over the query heads of the group - and are written exactly once (no atomics, no KV expansion); dQ leaves the CTA as
// fp32 `red.global.add` into an accumulator that a cast kernel turns into bf16/fp16 afterwards.
//
// Everything is computed TRANSPOSED so that every MMA has M = 128 (full TMEM lanes) and the softmax threads own KEY
// rows:   S^T = K Q^T and dP^T = V dO^T are [128 keys x 64 q] accumulators; thread k of the softmax warps reads key row k,
// forms P^T and dS^T, and stores them as bf16 [keys x q] K-major swizzled tiles.  Those two tiles feed
//   dV  += P^T  (A, K-major)  x dO (B, MN-major: the SAME smem bytes that were the K-major B of dP^T = V dO^T)
//   dK  += dS^T (A, K-major)  x Q  (B, MN-major: the same bytes as the B of S^T = K Q^T)
//   dQ^T = K^T  (A, MN-major view of the resident K tile) x dS (B, MN-major view of the dS^T tile)      [128 d x 64 q]
// i.e. five tensor-core GEMMs per (key tile, query tile) pair out of four smem operands, no transposition pass.
//
// Warps (16): 0 TMA producer (K, V once; Q_i / dO_i through a 3-stage ring), 1 MMA issuer (converged, as in the forward), 2..3 row
// statistics (log-sum-exp and delta of the query rows, three tiles ahead), 4..11 softmax (two threads per key row, 32 queries
// each), 12..15 dQ drain (thread = head-dim lane; 128-byte coalesced fp32 reductions per query row).
// The issuer runs S^T / dP^T of tile i+1 BEFORE the three accumulation GEMMs of tile i, so the tensor pipe works while
// the softmax warps are busy (same trick as the forward kernel); P^T / dS^T are double-buffered, so the softmax of tile i+1
// does not wait for those GEMMs either.
// Bound: 1280 clocks of MMA per (key tile, query tile), of which products with N = 64 take half as long again for reading their
// operands from shared memory.  4096 x 32 / 8 heads x 128 causal, two sequences, this kernel alone: 936 us; with the converged
// issuer (32 products a tile at about 80 clocks each were its bound) 780, with two dQ^T accumulators - the drain of one no longer
// holds up the issue of what the next tile needs - and without the waits that an earlier one implies 759.
// TMEM (512 columns): [0,64) S^T, [64,128) dP^T, [128,192) and [192,256) dQ^T, [256,384) dV, [384,512) dK.
// Shared memory: K 32 KB + V 32 KB + 3 x (Q 16 KB + dO 16 KB) + 2 x (P^T 16 KB + dS^T 16 KB) + statistics = 226 KB (D = 128).
constexpr int BWD_BLOCK_KV = 128;
constexpr int BWD_BLOCK_Q = 64;
constexpr int BWD_THREADS = 512;
constexpr int BWD_QSTAGES = 3;
constexpr int BWD_STAT_WARP0 = 2, BWD_SOFTMAX_WARP0 = 4, BWD_SOFTMAX_WARPS = 8, BWD_DRAIN_WARP0 = 12;

template <int D> struct FaBwdCfg {
  static constexpr int K_BYTES = BWD_BLOCK_KV * D * 2;
  static constexpr int V_BYTES = BWD_BLOCK_KV * D * 2;
  static constexpr int Q_BYTES = BWD_BLOCK_Q * D * 2;
  static constexpr int DO_BYTES = BWD_BLOCK_Q * D * 2;
  static constexpr int QDO_STAGE_BYTES = Q_BYTES + DO_BYTES;
  static constexpr int PT_BYTES = BWD_BLOCK_KV * BWD_BLOCK_Q * 2;
  static constexpr int STAT_BYTES = 2 * BWD_BLOCK_Q * 4;                // -lse * log2(e), -delta of a query tile
  static constexpr int SMEM_BYTES = K_BYTES + V_BYTES + BWD_QSTAGES * QDO_STAGE_BYTES + 4 * PT_BYTES +
                                    BWD_QSTAGES * STAT_BYTES + 1024 /*align*/ + 256 /*barriers*/;
  static constexpr int TMEM_COLS = 512;
  static constexpr int COL_ST = 0, COL_DPT = 64, COL_DQT = 128, COL_DV = 256, COL_DK = 384;
};

struct FaBwdParams {
  const int* cu_seqlens;             // packed batch boundaries (see FaParams) or null
  int batch, seqlen;                 // equal-length sequences, seqlen_q == seqlen_k (self attention)
  int hq, hkv;
  int causal;
  float scale, scale_log2;
  const float* lse;                  // [batch * seqlen, hq] natural log
  const float* delta;                // [batch * seqlen, hq] rowsum(dO o O)
  float* dq_acc;                     // [batch * seqlen, hq * D] fp32, zero-initialised
  void* dk;                          // [batch * seqlen, hkv * D]
  void* dv;
  // ring attention: dK / dV of this key block are ADDED (fp32 vector reductions) into accumulators that may live in
  // the block owner's memory (peer-mapped symmetric buffer: the reduction crosses NVLink) instead of being stored
  float* dk_acc;                     // [rows, hkv * D] fp32 or null
  float* dv_acc;
  int* status;                       // raised when a wait ran out
  uint32_t idesc_st, idesc_dv, idesc_dqt;
};

// the (query head, query tile) pairs that a key tile walks, tiles fastest
struct QueryWalk {
  int first, end, tile, head;
  SM100_DEVICE QueryWalk(int first_tile, int tiles, int first_head) : first(first_tile), end(tiles), tile(first_tile), head(first_head) {}
  SM100_DEVICE void next() {
    if (++tile == end) { tile = first; ++head; }
  }
};

template <int D, bool BF16>
__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                 const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                 const FaBwdParams p) {
  using C = FaBwdCfg<D>;
  static_assert(D == 128, "head_dim 128");
  constexpr int ST = BWD_QSTAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_k = smem;
  uint8_t* smem_v = smem_k + C::K_BYTES;
  uint8_t* smem_qdo = smem_v + C::V_BYTES;
  uint8_t* smem_pt = smem_qdo + ST * C::QDO_STAGE_BYTES;                  // [2]
  uint8_t* smem_dst = smem_pt + 2 * C::PT_BYTES;                          // [2]
  float* smem_stat = reinterpret_cast<float*>(smem_dst + 2 * C::PT_BYTES);   // [ST][2][64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_stat + ST * 2 * BWD_BLOCK_Q);
  uint64_t* kv_full = bars;                // [1]
  uint64_t* qdo_full = bars + 1;           // [ST]
  uint64_t* qdo_empty = qdo_full + ST;     // [ST]
  uint64_t* stat_full = qdo_empty + ST;    // [ST]  2 statistics warps
  uint64_t* stat_empty = stat_full + ST;   // [ST]  softmax warps
  uint64_t* sp_full = stat_empty + ST;     // [1]  S^T and dP^T are in TMEM
  uint64_t* sp_empty = sp_full + 1;        // [1]  the softmax warps have read them
  uint64_t* pds_full = sp_empty + 1;       // [2]  the softmax warps wrote P^T / dS^T to smem
  uint64_t* dq_full = pds_full + 2;       // [2]  dQ^T is in TMEM
  uint64_t* dq_empty = dq_full + 2;        // [2]  4 drain warps have read it
  uint64_t* acc_full = dq_empty + 2;       // [1]  final dK / dV complete
  uint64_t* drained = acc_full + 1;        // [1]  a CTA that gives up: its products have retired
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(drained + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  int* work = reinterpret_cast<int*>(tmem_ptr_smem + 2);

  const int warp = uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  // key tiles that see the most queries first; heads vary fastest (both in grid.x: a packed batch may have more key tiles than
  // grid.y holds)
  const int unit_of_head = blockIdx.x / p.hkv, kv_head = blockIdx.x - unit_of_head * p.hkv;
  const int group = p.hq / p.hkv;
  int kv_tile, seq_row0, len;
  if (p.cu_seqlens != nullptr) {
    if (warp == 0) {
      int unit = -1, start = 0, n = 0;
      const PackedBatch packed = packed_batch(p.cu_seqlens, p.batch, BWD_BLOCK_KV);
      if (unit_of_head < packed_count(packed, 0)) packed_unit(packed, unit_of_head, unit, start, n);
      if (lane == 0) { work[0] = unit; work[1] = start; work[2] = n; }
    }
    __syncthreads();
    if (work[0] < 0) return;                 // uniform across the CTA: nothing has been allocated yet
    seq_row0 = uniform(work[1]); len = uniform(work[2]);
    kv_tile = (len + BWD_BLOCK_KV - 1) / BWD_BLOCK_KV - 1 - uniform(work[0]);
  } else {
    kv_tile = unit_of_head; seq_row0 = (int)blockIdx.y * p.seqlen; len = p.seqlen;
  }
  const int q_tiles = (len + BWD_BLOCK_Q - 1) / BWD_BLOCK_Q;
  // causal: query tile i (rows 64 i ..) sees key tile j (keys 128 j ..) iff 64 i + 63 >= 128 j  <=>  i >= 2 j
  const int i_start = p.causal ? 2 * kv_tile : 0;
  const int n_i = max(q_tiles - i_start, 0);
  const int n_iter = n_i * group;                                  // (query head of the group, query tile) pairs
  const int kv_row0 = seq_row0 + kv_tile * BWD_BLOCK_KV;
  const bool ragged = (len % BWD_BLOCK_KV) != 0;                    // partial last key tile and / or query tile

  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tmap_q);
    prefetch_tensormap(&tmap_k);
    prefetch_tensormap(&tmap_v);
    prefetch_tensormap(&tmap_do);
  }
  if (warp == 1 && lane == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < ST; ++i) {
      mbar_init(&qdo_full[i], 1);
      mbar_init(&qdo_empty[i], 1);
      mbar_init(&stat_full[i], 2);
      mbar_init(&stat_empty[i], BWD_SOFTMAX_WARPS);
    }
    mbar_init(sp_full, 1);
    mbar_init(sp_empty, BWD_SOFTMAX_WARPS);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&pds_full[i], BWD_SOFTMAX_WARPS);
      mbar_init(&dq_full[i], 1);
      mbar_init(&dq_empty[i], 4);
    }
    mbar_init(acc_full, 1);
    mbar_init(drained, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 2) tmem_alloc<C::TMEM_COLS>(tmem_ptr_smem);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  auto ring_parity = [](int it) { return (uint32_t)((it / ST) & 1); };
  auto warp_wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag)) != 0; };

  if (warp == 0) {
    // ================================================================ TMA producer
    int it = 0;
    if (lane == 0) {
      mbar_arrive_expect_tx(kv_full, C::K_BYTES + C::V_BYTES);
#pragma unroll
      for (int h = 0; h < D / 64; ++h) {
        tma_load_2d(&tmap_k, kv_full, smem_k + h * (BWD_BLOCK_KV * 128), kv_head * D + h * 64, kv_row0);
        tma_load_2d(&tmap_v, kv_full, smem_v + h * (BWD_BLOCK_KV * 128), kv_head * D + h * 64, kv_row0);
      }
      QueryWalk at(i_start, q_tiles, kv_head * group);
      for (; it < n_iter; ++it, at.next()) {
        const int stage = it % ST, hq = at.head;
        const int q_row0 = seq_row0 + at.tile * BWD_BLOCK_Q;
        if (!wait_or_abort(&qdo_empty[stage], ring_parity(it) ^ 1, abort_flag)) break;
        uint8_t* sq = smem_qdo + stage * C::QDO_STAGE_BYTES;
        uint8_t* sdo = sq + C::Q_BYTES;
        mbar_arrive_expect_tx(&qdo_full[stage], C::QDO_STAGE_BYTES);
#pragma unroll
        for (int h = 0; h < D / 64; ++h) {               // boxes [64 rows, 64 d]
          tma_load_2d(&tmap_q, &qdo_full[stage], sq + h * (BWD_BLOCK_Q * 128), hq * D + h * 64, q_row0);
          tma_load_2d(&tmap_do, &qdo_full[stage], sdo + h * (BWD_BLOCK_Q * 128), hq * D + h * 64, q_row0);
        }
      }
    }
    __syncwarp();
    roles_done_wait<BWD_THREADS>();
    if (lane == 0 && (*abort_flag || n_iter == 0)) {     // leave no copy in flight behind (without queries nothing waits for K, V)
      int none = 0;
      wait_or_abort(kv_full, 0, &none);
      for (int i = max(0, it - ST); i < it; ++i) {
        none = 0;
        wait_or_abort(&qdo_full[i % ST], ring_parity(i), &none);
      }
      if (*abort_flag) report_abort(p.status);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ================================================================ MMA issuer
    const uint32_t leader = elect_one();
    if (n_iter > 0) {
      const uint32_t sk = smem_u32(smem_k), sv = smem_u32(smem_v);
      const uint64_t dk_kmaj = make_smem_desc_sw128(sk, 16, 1024);                        // A of S^T: [keys x d] K-major
      const uint64_t dv_kmaj = make_smem_desc_sw128(sv, 16, 1024);                        // A of dP^T
      const uint64_t dk_mnmaj = make_smem_desc_sw128(sk, BWD_BLOCK_KV * 128, 1024);       // A of dQ^T: K^T, M = d contiguous
      // of stage / buffer 0; B operands of the accumulations are MN-major views of the Q / dO tiles: rows = q (the reduction
      // dim), N = d contiguous, 64-element N chunks are BWD_BLOCK_Q * 128 bytes apart
      const uint32_t sq = smem_u32(smem_qdo), spt = smem_u32(smem_pt), sdst = smem_u32(smem_dst);
      const uint64_t dq_b = make_smem_desc_sw128(sq, 16, 1024), ddo_b = make_smem_desc_sw128(sq + C::Q_BYTES, 16, 1024);
      const uint64_t dq_mn = make_smem_desc_sw128(sq, BWD_BLOCK_Q * 128, 1024);
      const uint64_t ddo_mn = make_smem_desc_sw128(sq + C::Q_BYTES, BWD_BLOCK_Q * 128, 1024);
      const uint64_t d_pt = make_smem_desc_sw128(spt, 16, 1024);                          // A of dV: [keys x q] K-major
      const uint64_t d_dst = make_smem_desc_sw128(sdst, 16, 1024);                        // A of dK
      const uint64_t d_ds_mn = make_smem_desc_sw128(sdst, BWD_BLOCK_KV * 128, 1024);      // B of dQ^T (N = q)
      // one product: COUNT instructions of 16 along the reduction; a_off / b_off: bytes of the stage or buffer in use
      auto product = [&](uint32_t col, uint64_t da, uint32_t a_off, auto a_step, uint64_t db, uint32_t b_off, auto b_step, auto count,
                         uint32_t idesc, uint32_t acc) {
#pragma unroll
        for (int k = 0; k < decltype(count)::value; ++k)
          umma_f16_ss_warp(leader, tmem_base + col, desc_lo(da) + ((a_off + a_step(k)) >> 4), desc_hi(da),
                           desc_lo(db) + ((b_off + b_step(k)) >> 4), desc_hi(db), idesc, k > 0 ? 1u : acc);
      };
      auto kmaj_kv = [](int k) { return (uint32_t)((k >> 2) * (BWD_BLOCK_KV * 128) + (k & 3) * (UMMA_K * 2)); };
      auto kmaj_q = [](int k) { return (uint32_t)((k >> 2) * (BWD_BLOCK_Q * 128) + (k & 3) * (UMMA_K * 2)); };
      auto mnmaj = [](int k) { return (uint32_t)(k * (UMMA_K * 128)); };
      using OverD = std::integral_constant<int, D / UMMA_K>;
      using OverQ = std::integral_constant<int, BWD_BLOCK_Q / UMMA_K>;
      using OverKV = std::integral_constant<int, BWD_BLOCK_KV / UMMA_K>;
      int ahead = 0;                                           // stage of the next S^T / dP^T
      auto issue_sp = [&](int it) -> bool {
        if (!warp_wait(&qdo_full[ahead], ring_parity(it))) return false;
        if (!warp_wait(sp_empty, (uint32_t)((it & 1) ^ 1))) return false;   // softmax of it-1 has read S^T / dP^T
        tc_fence_after();
        const uint32_t off = ahead * C::QDO_STAGE_BYTES;
        product(C::COL_ST, dk_kmaj, 0, kmaj_kv, dq_b, off, kmaj_q, OverD{}, p.idesc_st, 0u);
        product(C::COL_DPT, dv_kmaj, 0, kmaj_kv, ddo_b, off, kmaj_q, OverD{}, p.idesc_st, 0u);
        umma_commit_warp(leader, sp_full);
        if (++ahead == ST) ahead = 0;
        return true;
      };
      bool ok = warp_wait(kv_full, 0) && issue_sp(0);
      for (int it = 0, stage = 0; it < n_iter && ok; ++it) {
        if (it + 1 < n_iter) ok = issue_sp(it + 1);            // tensor pipe stays busy during softmax(it)
        const int buf = it & 1;
        ok = ok && warp_wait(&pds_full[buf], (uint32_t)((it >> 1) & 1));
        if (!ok) break;
        tc_fence_after();
        const uint32_t off = stage * C::QDO_STAGE_BYTES, pds = buf * C::PT_BYTES;
        const uint32_t acc = it > 0 ? 1u : 0u;
        // dV += P^T dO and dK += dS^T Q (reductions over the 64 query rows)
        product(C::COL_DV, d_pt, pds, kmaj_q, ddo_mn, off, mnmaj, OverQ{}, p.idesc_dv, acc);
        product(C::COL_DK, d_dst, pds, kmaj_q, dq_mn, off, mnmaj, OverQ{}, p.idesc_dv, acc);
        umma_commit_warp(leader, &qdo_empty[stage]);           // Q_i / dO_i consumed
        ok = warp_wait(&dq_empty[buf], (uint32_t)(((it >> 1) & 1) ^ 1));    // dQ^T of iteration it-2 has been read
        if (!ok) break;
        tc_fence_after();
        // dQ^T = K^T dS (reduction over the 128 keys)
        product(C::COL_DQT + buf * BWD_BLOCK_Q, dk_mnmaj, 0, mnmaj, d_ds_mn, pds, mnmaj, OverKV{}, p.idesc_dqt, 0u);
        umma_commit_warp(leader, &dq_full[buf]);
        if (it == n_iter - 1) umma_commit_warp(leader, acc_full);
        if (++stage == ST) stage = 0;
      }
    }
    __syncwarp();
    roles_done_wait<BWD_THREADS>();
    if (leader && *abort_flag) {                             // nor a product
      int none = 0;
      umma_commit(drained);
      wait_or_abort(drained, 0, &none);
    }
    __syncwarp();
  } else if (warp < BWD_SOFTMAX_WARP0) {
    // ================================================================ statistics of the query rows (one row per thread)
    const int qr = (warp - BWD_STAT_WARP0) * 32 + lane;
    QueryWalk walk(i_start, q_tiles, kv_head * group);
    for (int it = 0; it < n_iter; ++it, walk.next()) {
      const int stage = it % ST, hq = walk.head;
      const int q_pos = walk.tile * BWD_BLOCK_Q + qr;
      // rows past the end of the sequence read as 0 (their P / dS are forced to 0 by the softmax warps)
      const size_t at = (size_t)(seq_row0 + q_pos) * p.hq + hq;
      const float l = q_pos < len ? __ldg(p.lse + at) : 0.f, d = q_pos < len ? __ldg(p.delta + at) : 0.f;
      if (!warp_wait(&stat_empty[stage], ring_parity(it) ^ 1)) break;
      smem_stat[stage * 2 * BWD_BLOCK_Q + qr] = -l * 1.4426950408889634f;
      smem_stat[stage * 2 * BWD_BLOCK_Q + BWD_BLOCK_Q + qr] = -d;
      __syncwarp();
      if (lane == 0) mbar_arrive(&stat_full[stage]);
    }
    roles_done<BWD_THREADS>();
  } else if (warp < BWD_DRAIN_WARP0) {
    // ================================================================ softmax warps: two threads per key row
    constexpr int COLS = BWD_BLOCK_Q / (BWD_SOFTMAX_WARPS / 4);
    const int quarter = warp & 3;
    const int part = (warp - BWD_SOFTMAX_WARP0) >> 2;        // this thread's 32 queries of the tile
    const int r = quarter * 32 + lane;                       // key row inside the tile
    const int key_pos = kv_tile * BWD_BLOCK_KV + r;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const bool key_live = key_pos < len;
    const int q_lo = p.causal ? key_pos : 0;                 // this key is visible to query positions [q_lo, len)
    bool ok = true;
    // two copies of the code: a mask only inside a branch becomes predicated code that every tile executes
    auto tile = [&](int it, int q_base, auto masked_tag) -> bool {
      constexpr bool MASKED = decltype(masked_tag)::value;
      const int stage = it % ST, buf = it & 1;
      if (!warp_wait(sp_full, (uint32_t)(it & 1))) return false;
      tc_fence_after();
      uint32_t sv[COLS], dpv[COLS];
      tmem_ld_32x32b_x32(tmem_base + lane_addr + C::COL_ST + part * COLS, sv);
      tmem_ld_32x32b_x32(tmem_base + lane_addr + C::COL_DPT + part * COLS, dpv);
      const bool stats = warp_wait(&stat_full[stage], ring_parity(it));
      tmem_ld_wait();
      if (!stats) return false;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(sp_empty);                  // S^T / dP^T may be overwritten by iteration it+1
      const ulonglong2* nlse = reinterpret_cast<const ulonglong2*>(smem_stat + stage * 2 * BWD_BLOCK_Q + part * COLS);
      const ulonglong2* ndel = reinterpret_cast<const ulonglong2*>(smem_stat + stage * 2 * BWD_BLOCK_Q + BWD_BLOCK_Q + part * COLS);
      const uint64_t mul2 = pack_f32x2(p.scale_log2, p.scale_log2);
      uint32_t p_packed[COLS / 2], ds_packed[COLS / 2];
#pragma unroll
      for (int c = 0; c < COLS; c += 4) {
        const ulonglong2 l4 = nlse[c / 4], d4 = ndel[c / 4];
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          const uint64_t x = fma_f32x2(pack_f32x2(__uint_as_float(sv[c + e]), __uint_as_float(sv[c + e + 1])), mul2, e ? l4.y : l4.x);
          const uint64_t y = add_f32x2(pack_f32x2(__uint_as_float(dpv[c + e]), __uint_as_float(dpv[c + e + 1])), e ? d4.y : d4.x);
          float p0, p1, d0, d1;
          unpack_f32x2(x, p0, p1);
          p0 = fast_exp2(p0);
          p1 = fast_exp2(p1);
          unpack_f32x2(mul_f32x2(y, pack_f32x2(p0, p1)), d0, d1);
          if (MASKED) {
            const int q0 = q_base + part * COLS + c + e;
            if (!(key_live && q0 >= q_lo && q0 < len)) p0 = d0 = 0.f;
            if (!(key_live && q0 + 1 >= q_lo && q0 + 1 < len)) p1 = d1 = 0.f;
          }
          p_packed[(c + e) >> 1] = pack_16<BF16>(p0, p1);
          ds_packed[(c + e) >> 1] = pack_16<BF16>(d0, d1);
        }
      }
      // the products of iteration it - 2, which read this buffer, have retired: they were issued before S^T of this one
      uint8_t* pt_row = smem_pt + buf * C::PT_BYTES + r * 128;
      uint8_t* dst_row = smem_dst + buf * C::PT_BYTES + r * 128;
#pragma unroll
      for (int i = 0; i < COLS / 8; ++i) {                   // 64 q = 128 bytes = 8 chunks of 16 B, SWIZZLE_128B
        const int pos = ((part * (COLS / 8) + i) ^ (r & 7)) * 16;
        *reinterpret_cast<uint4*>(pt_row + pos) =
            make_uint4(p_packed[i * 4], p_packed[i * 4 + 1], p_packed[i * 4 + 2], p_packed[i * 4 + 3]);
        *reinterpret_cast<uint4*>(dst_row + pos) =
            make_uint4(ds_packed[i * 4], ds_packed[i * 4 + 1], ds_packed[i * 4 + 2], ds_packed[i * 4 + 3]);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&pds_full[buf]);
        mbar_arrive(&stat_empty[stage]);
      }
      return true;
    };
    QueryWalk at(i_start, q_tiles, kv_head * group);
    for (int it = 0; it < n_iter && ok; ++it, at.next()) {
      const int q_tile = at.tile;
      const bool masked = (p.causal && (q_tile <= 2 * kv_tile + 1)) ||
                          (ragged && (kv_tile == (len - 1) / BWD_BLOCK_KV || q_tile == q_tiles - 1));
      ok = masked ? tile(it, q_tile * BWD_BLOCK_Q, std::true_type{}) : tile(it, q_tile * BWD_BLOCK_Q, std::false_type{});
    }
    // ---- epilogue: this key's row of dV (first half of the warps) or of scale * dK (second)
    if (ok && n_iter > 0) ok = warp_wait(acc_full, 0);
    if (ok) {
      tc_fence_after();
      const size_t row = (size_t)kv_row0 + r;
      const size_t ld = (size_t)p.hkv * D;
      const uint32_t col0 = part == 0 ? C::COL_DV : C::COL_DK;
      const float mul = part == 0 ? 1.f : p.scale;
      float* acc_row = p.dk_acc != nullptr ? (part == 0 ? p.dv_acc : p.dk_acc) + (row * ld + (size_t)kv_head * D) : nullptr;
      uint8_t* base = reinterpret_cast<uint8_t*>(part == 0 ? p.dv : p.dk) + (row * ld + (size_t)kv_head * D) * 2;
      // NOTE: tcgen05.ld is warp-collective (.sync.aligned): every lane runs the loads, only the STORES are predicated on
      // the key being inside the sequence (a ragged last tile leaves some lanes of a warp without a row)
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        uint32_t v[32];
        __syncwarp();
        tmem_ld_32x32b_x32(tmem_base + lane_addr + col0 + c, v);
        tmem_ld_wait();
        if (!key_live) continue;
        if (acc_row != nullptr) {
          if (n_iter > 0) {
#pragma unroll
            for (int i = 0; i < 32; i += 4)
              asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                           :: "l"(acc_row + c + i), "f"(__uint_as_float(v[i]) * mul), "f"(__uint_as_float(v[i + 1]) * mul),
                              "f"(__uint_as_float(v[i + 2]) * mul), "f"(__uint_as_float(v[i + 3]) * mul) : "memory");
          }
          continue;
        }
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i)
          w[i] = n_iter > 0 ? pack_16<BF16>(__uint_as_float(v[2 * i]) * mul, __uint_as_float(v[2 * i + 1]) * mul) : 0u;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(base + (c + i * 8) * 2) = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
      }
    }
    __syncwarp();
    roles_done<BWD_THREADS>();
  } else {
    // ================================================================ dQ drain warps: thread = head-dim lane
    const int quarter = warp & 3;
    const int dlane = quarter * 32 + lane;                   // d index (row of dQ^T)
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const size_t row_stride = (size_t)p.hq * D;
    QueryWalk at(i_start, q_tiles, kv_head * group);
    for (int it = 0; it < n_iter; ++it, at.next()) {
      const int q_row0 = seq_row0 + at.tile * BWD_BLOCK_Q, hq = at.head, buf = it & 1;
      const int q_live = min(len - at.tile * BWD_BLOCK_Q, BWD_BLOCK_Q);    // rows of this tile that belong to the sequence
      if (!warp_wait(&dq_full[buf], (uint32_t)((it >> 1) & 1))) break;
      tc_fence_after();
      float* dst = p.dq_acc + ((size_t)q_row0 * p.hq + hq) * D + dlane;
#pragma unroll
      for (int c = 0; c < BWD_BLOCK_Q; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(tmem_base + lane_addr + C::COL_DQT + buf * BWD_BLOCK_Q + c, v);
        tmem_ld_wait();
        if (c + 32 == BWD_BLOCK_Q) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&dq_empty[buf]);        // dQ^T may be overwritten while the reductions are on their way
        }
        if (q_live == BWD_BLOCK_Q) {
#pragma unroll
          for (int i = 0; i < 32; ++i)                       // one 128-byte coalesced fp32 reduction per warp and row
            atomicAdd(dst + (size_t)(c + i) * row_stride, __uint_as_float(v[i]) * p.scale);
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c + i < q_live) atomicAdd(dst + (size_t)(c + i) * row_stride, __uint_as_float(v[i]) * p.scale);
        }
      }
    }
    __syncwarp();
    roles_done<BWD_THREADS>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc<C::TMEM_COLS>(tmem_base);
}

// delta[t, h] = sum_d dO[t, h, d] * O[t, h, d], and zeros for the fp32 dQ accumulator of the same rows.  D / 8 lanes per (token,
// head) row, a row after the other in memory: a warp takes 32 * 8 / D rows at once, each thread BWD_DELTA_ROWS of them in
// flight (one warp per row of 128 left half its lanes idle: 42 us for 262144 rows, and a memset of 23 us beside it; now 40 us
// for both).  D is a power of two.
constexpr int BWD_DELTA_ROWS = 4;
template <typename T>
__global__ void __launch_bounds__(256) flash_bwd_delta_kernel(const T* __restrict__ out, const T* __restrict__ dout,
                                                              float* __restrict__ delta, float* __restrict__ zero, long long rows,
                                                              int D) {
  const int per = D / 8;                                     // lanes of a row
  const long long step = (long long)gridDim.x * blockDim.x;
  const long long total = rows * per;
  const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  Vec16<T> a[BWD_DELTA_ROWS], b2[BWD_DELTA_ROWS];
#pragma unroll
  for (int u = 0; u < BWD_DELTA_ROWS; ++u) {
    const long long i = i0 + u * step;
    if (i < total) { a[u].load_nc(out + i * 8); b2[u].load_nc(dout + i * 8); }
  }
#pragma unroll
  for (int u = 0; u < BWD_DELTA_ROWS; ++u) {
    const long long i = i0 + u * step;
    float acc = 0.f;
    if (i < total) {
#pragma unroll
      for (int e = 0; e < 8; ++e) acc += a[u].get(e) * b2[u].get(e);
      if (zero != nullptr) {
        float4* z = reinterpret_cast<float4*>(zero + i * 8);
        z[0] = z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    for (int o = per >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (i < total && (threadIdx.x & (per - 1)) == 0) delta[i / per] = acc;
  }
}

template <typename T>
int launch_flash_bwd_delta(const void* out, const void* dout, float* delta, float* zero, long long rows, int D, cudaStream_t stream) {
  if (D != 64 && D != 128) return (int)cudaErrorInvalidValue;
  const long long threads = (rows * (D / 8) + BWD_DELTA_ROWS - 1) / BWD_DELTA_ROWS;
  flash_bwd_delta_kernel<T><<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>((const T*)out, (const T*)dout, delta, zero, rows, D);
  return (int)cudaGetLastError();
}

template <typename T>
__global__ void flash_bwd_cast_dq_kernel(const float* __restrict__ acc, T* __restrict__ dq, long long n) {
  const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  const float4 a = *reinterpret_cast<const float4*>(acc + i);
  const float4 b2 = *reinterpret_cast<const float4*>(acc + i + 4);
  Vec16<T> o;
  o.set(0, a.x); o.set(1, a.y); o.set(2, a.z); o.set(3, a.w);
  o.set(4, b2.x); o.set(5, b2.y); o.set(6, b2.z); o.set(7, b2.w);
  o.store(dq + i);
}

template <int D>
int launch_flash_bwd(const void* q, const void* k, const void* v, const void* dout, const float* lse, const float* delta,
                     float* dq_acc, void* dk, void* dv, int batch, int seqlen, int hq, int hkv, int causal, float scale,
                     int dtype, cudaStream_t stream, const int* cu_seqlens = nullptr, long long total_tokens = 0,
                     float* dk_acc = nullptr, float* dv_acc = nullptr) {
  using C = FaBwdCfg<D>;
  const bool bf16 = dtype == CB_BF16;
  CUtensorMap tq, tk, tv, tdo;
  const uint64_t T = cu_seqlens ? (uint64_t)total_tokens : (uint64_t)batch * seqlen;
  int r = make_tmap_2d_16b(&tq, q, T, (uint64_t)hq * D, (uint64_t)hq * D, BWD_BLOCK_Q, 64, bf16);
  if (r) return 1000 + r;
  r = make_tmap_2d_16b(&tdo, dout, T, (uint64_t)hq * D, (uint64_t)hq * D, BWD_BLOCK_Q, 64, bf16);
  if (r) return 4000 + r;
  r = make_tmap_2d_16b(&tk, k, T, (uint64_t)hkv * D, (uint64_t)hkv * D, BWD_BLOCK_KV, 64, bf16);
  if (r) return 2000 + r;
  r = make_tmap_2d_16b(&tv, v, T, (uint64_t)hkv * D, (uint64_t)hkv * D, BWD_BLOCK_KV, 64, bf16);
  if (r) return 3000 + r;
  FaBwdParams p;
  p.cu_seqlens = cu_seqlens;
  p.batch = batch; p.seqlen = seqlen; p.hq = hq; p.hkv = hkv; p.causal = causal;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.lse = lse; p.delta = delta; p.dq_acc = dq_acc; p.dk = dk; p.dv = dv; p.status = flash_status();
  p.dk_acc = dk_acc; p.dv_acc = dv_acc;
  const int f = bf16 ? 1 : 0;
  p.idesc_st = make_idesc_f16(BWD_BLOCK_KV, BWD_BLOCK_Q, f, 0, 0);     // [128 keys x 64 q]  = K-major x K-major
  p.idesc_dv = make_idesc_f16(BWD_BLOCK_KV, D, f, 0, 1);                // [128 keys x D]     = K-major x MN-major
  p.idesc_dqt = make_idesc_f16(D, BWD_BLOCK_Q, f, 1, 1);                // [D x 64 q]         = MN-major x MN-major
  auto kern = bf16 ? flash_bwd_kernel<D, true> : flash_bwd_kernel<D, false>;
  static CbDeviceAttr attr[2];
  if (const int e = cb_allow_smem(attr[f], kern, C::SMEM_BYTES)) return e;
  const long long units = (cu_seqlens ? total_tokens / BWD_BLOCK_KV + batch : ((long long)seqlen + BWD_BLOCK_KV - 1) / BWD_BLOCK_KV) * hkv;
  const dim3 grid((unsigned)units, cu_seqlens ? 1 : batch);
  if (units > 0x7fffffffll || grid.y > 65535) return (int)cudaErrorInvalidValue;
  kern<<<grid, BWD_THREADS, C::SMEM_BYTES, stream>>>(tq, tk, tv, tdo, p);
  return (int)cudaGetLastError();
}

}  // namespace

extern "C" {

// cudaErrorLaunchTimeout, once, if a wait of a launch that has run since the last call of any function here ran out
int cb_flash_attn_status() { return flash_earlier(); }

// A wait that runs out after `limit` polls and reports it, with no copy or product in flight.
int cb_flash_attn_wait_probe(int limit, cudaStream_t stream) {
  if (flash_status() == nullptr) return (int)cudaErrorMemoryAllocation;
  flash_wait_probe_kernel<<<1, 32, 0, stream>>>(limit, flash_status());
  return (int)cudaGetLastError();
}

// q [batch * seqlen_q, hq, D], k / v [batch * seqlen_k, hkv, D] contiguous token-major; out like q; lse [batch *
// seqlen_q, hq] fp32 (may be null).  Requirements: D in {64, 128}, seqlen_q and seqlen_k multiples of 128,
// causal => seqlen_q == seqlen_k, hq % hkv == 0, 16-byte aligned bases.
int cb_flash_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int batch, int seqlen_q,
                      int seqlen_k, int hq, int hkv, int head_dim, int causal, float scale, int dtype,
                      cudaStream_t stream) {
  if (batch <= 0 || seqlen_q <= 0) return 0;
  if (hq % hkv || (causal && seqlen_q != seqlen_k)) return (int)cudaErrorInvalidValue;
  // sequence lengths need not be multiples of the tile: partial tiles are masked (keys) / not stored (queries)
  if (dtype != CB_BF16 && dtype != CB_F16) return (int)cudaErrorInvalidValue;
  if (const int e = flash_earlier()) return e;
  if (head_dim == 128)
    return launch_flash_fwd<128>(q, k, v, out, lse, batch, seqlen_q, seqlen_k, hq, hkv, causal, scale, dtype, stream);
  if (head_dim == 64)
    return launch_flash_fwd<64>(q, k, v, out, lse, batch, seqlen_q, seqlen_k, hq, hkv, causal, scale, dtype, stream);
  return (int)cudaErrorInvalidValue;
}

// Packed (variable-length) self attention: q / k / v [total_tokens, heads, D]; cu_seqlens int32[batch + 1] ON THE DEVICE
// (never read by the host: the grid is sized for the worst case and surplus CTAs exit).  Reference counterpart:
// `flash_attn_varlen_kvpacked_func` behind `extensions/pybind/flash_attention/flash_attention_dao_cuda.py:37-96`.
int cb_flash_attn_varlen_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int* cu_seqlens,
                             int batch, long long total_tokens, int hq, int hkv, int head_dim, int causal, float scale,
                             int dtype, cudaStream_t stream) {
  if (batch <= 0 || total_tokens <= 0) return 0;
  if (hq % hkv || (dtype != CB_BF16 && dtype != CB_F16) || cu_seqlens == nullptr) return (int)cudaErrorInvalidValue;
  if (const int e = flash_earlier()) return e;
  if (head_dim == 128)
    return launch_flash_fwd<128>(q, k, v, out, lse, batch, 0, 0, hq, hkv, causal, scale, dtype, stream, cu_seqlens, total_tokens);
  if (head_dim == 64)
    return launch_flash_fwd<64>(q, k, v, out, lse, batch, 0, 0, hq, hkv, causal, scale, dtype, stream, cu_seqlens, total_tokens);
  return (int)cudaErrorInvalidValue;
}

// Packed causal forward for inference prefill with a sliding window (Mistral: query q sees keys (q - window, q]) and /
// or ALiBi slopes ([hq] fp32: score += slope * (key - query); BLOOM, Baichuan-13B).  Forward only.
int cb_flash_attn_varlen_fwd_ex(const void* q, const void* k, const void* v, void* out, float* lse,
                                const int* cu_seqlens, int batch, long long total_tokens, int hq, int hkv, int head_dim,
                                float scale, int window, const float* alibi_slopes, int dtype, cudaStream_t stream) {
  if (batch <= 0 || total_tokens <= 0) return 0;
  if (hq % hkv || (dtype != CB_BF16 && dtype != CB_F16) || cu_seqlens == nullptr || window < 0)
    return (int)cudaErrorInvalidValue;
  if (const int e = flash_earlier()) return e;
  if (head_dim == 128)
    return launch_flash_fwd<128>(q, k, v, out, lse, batch, 0, 0, hq, hkv, 1, scale, dtype, stream, cu_seqlens,
                                 total_tokens, nullptr, 0, window, alibi_slopes);
  if (head_dim == 64)
    return launch_flash_fwd<64>(q, k, v, out, lse, batch, 0, 0, hq, hkv, 1, scale, dtype, stream, cu_seqlens,
                                total_tokens, nullptr, 0, window, alibi_slopes);
  return (int)cudaErrorInvalidValue;
}

// Backward of cb_flash_attn_fwd for self attention (seqlen_q == seqlen_k).  q / out / dout / dq [T, hq, D], k / v / dk /
// dv [T, hkv, D], lse [T, hq] fp32 from the forward.  Workspaces: delta [T, hq] fp32 and dq_acc [T, hq, D] fp32 (this
// function zeroes dq_acc).  Requirements as the forward; head_dim 128 (64 also instantiated).
int cb_flash_attn_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout, const float* lse,
                      void* dq, void* dk, void* dv, float* delta, float* dq_acc, int batch, int seqlen, int hq, int hkv,
                      int head_dim, int causal, float scale, int dtype, const int* cu_seqlens, long long total_tokens,
                      cudaStream_t stream) {
  // cu_seqlens != null: packed batch of `total_tokens` rows (seqlen ignored); else `batch` sequences of `seqlen`
  if (batch <= 0 || (cu_seqlens ? total_tokens <= 0 : seqlen <= 0)) return 0;
  // head_dim 64 would make dQ^T an M = 64 MMA (different TMEM lane layout): not wired up yet
  if (hq % hkv || head_dim != 128) return (int)cudaErrorInvalidValue;
  if (dtype != CB_BF16 && dtype != CB_F16) return (int)cudaErrorInvalidValue;
  if (const int e = flash_earlier()) return e;
  const long long rows = (cu_seqlens ? total_tokens : (long long)batch * seqlen) * hq;
  const long long n = rows * head_dim;
  const int re = dtype == CB_BF16 ? launch_flash_bwd_delta<__nv_bfloat16>(out, dout, delta, dq_acc, rows, head_dim, stream)
                                  : launch_flash_bwd_delta<__half>(out, dout, delta, dq_acc, rows, head_dim, stream);
  if (re) return re;
  int rc = launch_flash_bwd<128>(q, k, v, dout, lse, delta, dq_acc, dk, dv, batch, seqlen, hq, hkv, causal, scale, dtype,
                                 stream, cu_seqlens, total_tokens);
  if (rc) return rc;
  const unsigned blocks = (unsigned)((n / 8 + 255) / 256);
  if (dtype == CB_BF16) flash_bwd_cast_dq_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(dq_acc, (__nv_bfloat16*)dq, n);
  else flash_bwd_cast_dq_kernel<__half><<<blocks, 256, 0, stream>>>(dq_acc, (__half*)dq, n);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------------------------------
// Blockwise entry points for fused ring (context-parallel) attention.  One launch = the queries of this rank against ONE
// key/value block that may live in a PEER's memory (k / v are then peer-mapped symmetric-buffer addresses: the TMA
// loads of the main loop pull the tiles over NVLink, GQA heads only, no staging copy).
//   forward : the online-softmax state (o_state fp32, lse) is carried from launch to launch inside the kernel
//             (`has_prev`), which replaces the reference's per-hop `_rescale_out_lse` pass (`layer/attn.py:376-403`);
//   backward: dQ accumulates in the local fp32 `dq_acc` (not zeroed here), dK / dV are reduced straight into the block
//             owner's fp32 accumulators (`dk_acc` / `dv_acc`, peer pointers) - the reference circulates fp32 dKV
//             buffers around the ring instead (`layer/attn.py:1066-1163`).  `delta` = rowsum(dO o O) is an input.
int cb_flash_attn_block_fwd(const void* q, const void* k, const void* v, float* o_state, float* lse, int rows, int hq,
                            int hkv, int head_dim, int causal, int has_prev, float scale, int dtype, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (hq % hkv || (dtype != CB_BF16 && dtype != CB_F16) || o_state == nullptr || lse == nullptr)
    return (int)cudaErrorInvalidValue;
  if (const int e = flash_earlier()) return e;
  if (head_dim == 128)
    return launch_flash_fwd<128>(q, k, v, nullptr, lse, 1, rows, rows, hq, hkv, causal, scale, dtype, stream, nullptr, 0,
                                 o_state, has_prev);
  if (head_dim == 64)
    return launch_flash_fwd<64>(q, k, v, nullptr, lse, 1, rows, rows, hq, hkv, causal, scale, dtype, stream, nullptr, 0,
                                o_state, has_prev);
  return (int)cudaErrorInvalidValue;
}

int cb_flash_attn_block_bwd(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                            const float* delta, float* dq_acc, float* dk_acc, float* dv_acc, int rows, int hq, int hkv,
                            int head_dim, int causal, float scale, int dtype, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (hq % hkv || head_dim != 128 || (dtype != CB_BF16 && dtype != CB_F16) || !dq_acc || !dk_acc || !dv_acc)
    return (int)cudaErrorInvalidValue;
  if (const int e = flash_earlier()) return e;
  return launch_flash_bwd<128>(q, k, v, dout, lse, delta, dq_acc, nullptr, nullptr, 1, rows, hq, hkv, causal, scale, dtype,
                               stream, nullptr, 0, dk_acc, dv_acc);
}

// delta[t, h] = sum_d dO o O for `rows` (token, head) rows of width head_dim
int cb_flash_attn_delta(const void* out, const void* dout, float* delta, long long rows, int head_dim, int dtype,
                        cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (dtype == CB_BF16) return launch_flash_bwd_delta<__nv_bfloat16>(out, dout, delta, nullptr, rows, head_dim, stream);
  if (dtype == CB_F16) return launch_flash_bwd_delta<__half>(out, dout, delta, nullptr, rows, head_dim, stream);
  return (int)cudaErrorInvalidValue;
}

}  // extern "C"
