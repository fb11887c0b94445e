// y = x w^T (+ residual) for a few token rows on sm_100a: the projections of a decode step.  And its embedding lookup.
//
//   x [M, K] 16-bit, M <= 32; w [N, K] (torch.nn.Linear's layout); y [M, N]; residual [M, N], added before the rounding
//   gated unit: w [2 N, K], gate rows before up rows; y = act(x gate^T) (x up^T), both rounded to 16 bits first, as a projection and
//   the unit behind it would leave them
//
// Bound: HBM - every weight is read once and meets a handful of rows.  The product is computed transposed, 128 rows of w being the
// M of tcgen05.mma and the tokens, padded to 16 or 32, its N, so that the tensor pipe needs an eighth of the time the loads
// take.  A CTA streams its k-blocks through a TMA ring of STAGES x 16 KB of w; two CTAs fit on an SM and keep about 180 KB
// in flight, more than the 70 KB that 6.5 TB/s times a loaded latency of 1.5 us come to.  Where a matrix has fewer 128-row tiles than
// SMs, the reduction is split over the CTAs of a cluster: each leaves its fp32 sums in shared memory, and every one adds a part of
// the tile's rows over the cluster in ascending order of k - no workspace, no counters, and the same bits whatever M is.
// Launched while the kernel before it still runs: what that one does not write - the first blocks of w - is fetched into L2
// meanwhile (a prefetch delivers nothing: the copies themselves follow the wait).
// 16 rows, bf16, us back to back in a graph, cuBLAS and this: 4096 x 4096 9.4 and 8.6, 6144 x 4096 12.1 and 11.5, 28672 x 4096 40.4 and
// 39.2, 4096 x 14336 22.9 and 20.4, 32000 x 4096 45.5 and 43.0, 2048 x 8192 13.0 and 8.8, 1536 x 1024 3.6 and 3.7; 32 rows 9.9 / 8.9,
// 12.4 / 12.0, 41.6 / 39.8, 27.3 / 21.3, 45.8 / 44.3, 13.1 / 9.5, 3.7 / 4.0.  Three stages and four CTAs on an SM were slower for deep
// matrices (4096 x 14336 22.4).  A decode step of four layers of 4096 x 14336, 16 sequences: 530 us with cuBLAS, 509.
// There is no lower bound on the matrix: alone cuBLAS is ahead by 0.1 - 0.3 us at 1536 x 1024, but in a step the early launches are
// worth more.  Two layers of 1024 x 2816, 5 sequences, with cuBLAS for the projections 103 us, with this 87; four of them, one
// sequence 198 and 141.
#include "activations.cuh"
#include "checked_id.h"
#include "common.cuh"
#include "sm100.cuh"

using namespace sm100;

namespace {

constexpr int UMMA_K = 16;
constexpr int TILE = 128;              // rows of w; of a gated unit half of them gate, half up
constexpr int HALF = TILE / 2;
constexpr int BK = 64;
constexpr int ROWS_THREADS = 192;      // producer, issuer, four epilogue warps
constexpr int W_BYTES = TILE * BK * 2;
constexpr int MAX_SPLITS = 8;          // CTAs of a cluster
constexpr int WAIT_LIMIT = 1 << 22;

template <int NT> struct RowsCfg {
  static constexpr int STAGES = NT == 16 ? 6 : 5;
  static constexpr int X_BYTES = NT * BK * 2;
  static constexpr int SMEM = STAGES * (W_BYTES + X_BYTES) + 256;
};

struct RowsParams {
  int M, N, k_blocks, per_split;       // N: columns of y; k-blocks in all / of one CTA of the cluster
  int packed;                          // rows of y are 8-byte aligned
  int64_t ldy, ldr;
  void* y;
  const void* residual;
  uint32_t idesc;
};

// gives up after a bounded number of polls: the CTA then writes NaN
SM100_DEVICE bool wait_bounded(uint64_t* bar, uint32_t parity) {
  for (int i = 0; i < WAIT_LIMIT; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
SM100_DEVICE void prefetch_l2_2d(const CUtensorMap* map, int32_t c0, int32_t c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1)
               : "memory");
}
SM100_DEVICE float4 load_cluster_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// ACT: of a gated unit, as in activations.cuh, or PLAIN.  Its tile is HALF gate rows and the HALF up rows that belong to them, in two boxes,
// so that a CTA has both sides of a product of the unit.  (The unit in a launch of its own cost a decode step 2 us a layer; elementwise.cu.)
constexpr int PLAIN = -1;
template <typename T, int NT, int ACT>
__global__ void __launch_bounds__(ROWS_THREADS, 2)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const RowsParams p) {
  using C = RowsCfg<NT>;
  constexpr int STAGES = C::STAGES;
  constexpr bool GATED = ACT != PLAIN;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* smem_w = smem;
  uint8_t* smem_x = smem + STAGES * W_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_x + STAGES * C::X_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_ptr + 1);
  float* part = reinterpret_cast<float*>(smem);              // [NT][TILE] sums, over the ring when it is done

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const int splits = gridDim.y, split = blockIdx.y;          // a cluster is one tile's splits
  const int n0 = blockIdx.x * (GATED ? HALF : TILE);         // first column of y
  const int kb0 = split * p.per_split, kbs = max(0, min(p.k_blocks - kb0, p.per_split));

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tmap_w);
    prefetch_tensormap(&tmap_x);
    for (int i = 0; i < min(kbs, STAGES); ++i) {
      prefetch_l2_2d(&tmap_w, (kb0 + i) * BK, n0);
      if (GATED) prefetch_l2_2d(&tmap_w, (kb0 + i) * BK, p.N + n0);
    }
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(acc_full, 1);
    *gave_up = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc<32>(tmem_ptr);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;
  asm volatile("griddepcontrol.wait;" ::: "memory");

  bool ok = true;
  if (warp == 0) {
    // ================================================================ TMA producer
    if (lane == 0) {
      int stage = 0, issued = 0;
      uint32_t phase = 0;
      for (int i = 0; i < kbs && ok; ++i) {
        ok = wait_bounded(&empty[stage], phase ^ 1);
        if (!ok) break;
        mbar_arrive_expect_tx(&full[stage], W_BYTES + C::X_BYTES);
        tma_load_2d(&tmap_w, &full[stage], smem_w + stage * W_BYTES, (kb0 + i) * BK, n0);
        if (GATED) tma_load_2d(&tmap_w, &full[stage], smem_w + stage * W_BYTES + W_BYTES / 2, (kb0 + i) * BK, p.N + n0);
        tma_load_2d(&tmap_x, &full[stage], smem_x + stage * C::X_BYTES, (kb0 + i) * BK, 0);
        ++issued;
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok)                                               // nothing may land after the CTA has left
        for (int i = max(0, issued - STAGES); i < issued; ++i) wait_bounded(&full[i % STAGES], (uint32_t)((i / STAGES) & 1));
    }
    __syncwarp();
  } else if (warp == 1) {
    // ================================================================ MMA issuer, converged
    const uint32_t leader = elect_one();
    const uint64_t dw = make_smem_desc_sw128(smem_u32(smem_w), 16, 1024), dx = make_smem_desc_sw128(smem_u32(smem_x), 16, 1024);
    int stage = 0;
    uint32_t phase = 0;
    for (int i = 0; i < kbs && ok; ++i) {
      ok = __all_sync(0xffffffffu, wait_bounded(&full[stage], phase)) != 0;
      if (!ok) break;
      tc_fence_after();
      const uint32_t a = desc_lo(dw) + stage * (W_BYTES >> 4), b = desc_lo(dx) + stage * (C::X_BYTES >> 4);
#pragma unroll
      for (int k = 0; k < BK / UMMA_K; ++k)
        umma_f16_ss_warp(leader, tmem, a + (k * UMMA_K * 2 >> 4), desc_hi(dw), b + (k * UMMA_K * 2 >> 4), desc_hi(dx), p.idesc,
                         (i > 0 || k > 0) ? 1u : 0u);
      umma_commit_warp(leader, &empty[stage]);
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    if (leader && !ok) *gave_up = 1;
    __syncwarp();
    umma_commit_warp(leader, acc_full);                      // (also where it gave up: nobody leaves before its products)
    wait_bounded(acc_full, 0);
  } else {
    // ================================================================ epilogue: lane = row of w
    const int quarter = warp & 3, r = quarter * 32 + lane;
    ok = __all_sync(0xffffffffu, wait_bounded(acc_full, 0)) != 0 && !*gave_up;
    tc_fence_after();
    uint32_t v[NT];
    if (NT == 32) tmem_ld_32x32b_x32(tmem + ((uint32_t)(quarter * 32) << 16), *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
    else tmem_ld_32x32b_x16(tmem + ((uint32_t)(quarter * 32) << 16), *reinterpret_cast<uint32_t(*)[16]>(&v[0]));
    tmem_ld_wait();
    if (kbs == 0 || !ok) {
#pragma unroll
      for (int t = 0; t < NT; ++t) v[t] = ok ? 0u : 0x7fffffffu;
    }
    if (!GATED && splits == 1) {
      const int n = n0 + r;
      if (n < p.N) {
        T* y = reinterpret_cast<T*>(p.y) + n;
        const T* res = reinterpret_cast<const T*>(p.residual) + n;
#pragma unroll
        for (int t = 0; t < NT; ++t)
          if (t < p.M)
            y[t * p.ldy] = from_f32<T>(__uint_as_float(v[t]) + (p.residual != nullptr ? to_f32<T>(res[t * p.ldr]) : 0.f));
      }
    } else {
#pragma unroll
      for (int t = 0; t < NT; ++t) part[t * TILE + r] = __uint_as_float(v[t]);
      if (splits == 1) asm volatile("bar.sync 1, 128;" ::: "memory");        // the epilogue's own warps
    }
  }
  if (GATED || splits > 1) {
    if (splits > 1) cluster_sync();
    if (warp >= 2) {
      // four rows of w at a time, of one token; every CTA has its share of neighbours.  All parts of a sum are asked for before
      // the first is added: one after the other the sums of 32 tokens took 3 us.
      constexpr int COLS = GATED ? HALF : TILE;
      const int groups = COLS / 4 * p.M, share = (groups + splits - 1) / splits;
      for (int e = split * share + threadIdx.x - 64; e < min(groups, (split + 1) * share); e += 128) {
        const int t = e / (COLS / 4), r = e % (COLS / 4) * 4, n = n0 + r;
        const uint32_t at = smem_u32(part + t * TILE + r);
        float4 v[MAX_SPLITS];
        auto ask = [&](uint32_t from) {
#pragma unroll
          for (int s = 0; s < MAX_SPLITS; ++s)
            if (s < splits) v[s] = load_cluster_v4(map_to_cta(from, s));
        };
        auto add_up = [&](float (&sum)[4]) {
          sum[0] = v[0].x; sum[1] = v[0].y; sum[2] = v[0].z; sum[3] = v[0].w;
#pragma unroll
          for (int s = 1; s < MAX_SPLITS; ++s)
            if (s < splits) { sum[0] += v[s].x; sum[1] += v[s].y; sum[2] += v[s].z; sum[3] += v[s].w; }
        };
        float sum[4];
        ask(at);
        add_up(sum);
        if (GATED) {
          float up[4];
          ask(at + HALF * 4);
          add_up(up);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            sum[i] = act_f<GATED ? ACT : 0>(to_f32<T>(from_f32<T>(sum[i]))) * to_f32<T>(from_f32<T>(up[i]));
        }
        T* y = reinterpret_cast<T*>(p.y) + t * p.ldy + n;
        const T* res = reinterpret_cast<const T*>(p.residual) + t * p.ldr + n;
        union { uint2 raw; T v[4]; } o;
#pragma unroll
        for (int i = 0; i < 4; ++i) o.v[i] = from_f32<T>(sum[i] + (p.residual != nullptr && n + i < p.N ? to_f32<T>(res[i]) : 0.f));
        if (p.packed && n + 4 <= p.N) {
          *reinterpret_cast<uint2*>(y) = o.raw;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (n + i < p.N) y[i] = o.v[i];
        }
      }
    }
    if (splits > 1) cluster_sync();                                          // nobody leaves while its sums are read
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc<32>(tmem);
}

// out[i] = table[ids[i]]: a block per id, 16 bytes a thread and step
__global__ void __launch_bounds__(256) embed_rows_kernel(const int64_t* __restrict__ ids, const uint4* __restrict__ table, uint4* __restrict__ out,
                                                         int64_t entries, int vecs) {
  cb_early_start();
  const uint4* src = table + cb_checked_id(ids[blockIdx.x], entries) * vecs;
  uint4* dst = out + (int64_t)blockIdx.x * vecs;
  for (int i = threadIdx.x; i < vecs; i += 256) dst[i] = src[i];
}

template <typename T, int NT, int ACT>
int launch_rows(const CUtensorMap& tw, const CUtensorMap& tx, const RowsParams& p, int tiles, int splits, cudaStream_t stream) {
  static CbDeviceAttr attr;
  if (const int e = cb_allow_smem(attr, gemm_rows_kernel<T, NT, ACT>, RowsCfg<NT>::SMEM)) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles, splits);
  cfg.blockDim = dim3(ROWS_THREADS);
  cfg.dynamicSmemBytes = RowsCfg<NT>::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 1;
  at[1].val.clusterDim.y = splits;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cb_launch_error(cudaLaunchKernelEx(&cfg, gemm_rows_kernel<T, NT, ACT>, tw, tx, p));
}

// N columns of y, w_rows of w
template <int ACT>
int rows_product(const void* x, const void* w, void* y, const void* residual, int M, int N, int w_rows, int K, int64_t ldx, int64_t ldy,
                 int64_t ldr, int dtype, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (M > 32 || K <= 0 || (K & 7) || (ldx & 7) || (dtype != CB_BF16 && dtype != CB_F16)) return (int)cudaErrorInvalidValue;
  const bool bf16 = dtype == CB_BF16;
  const int nt = M <= 16 ? 16 : 32, columns = ACT == PLAIN ? TILE : HALF;
  CUtensorMap tw, tx;
  int r = make_tmap_2d_16b(&tw, w, w_rows, K, K, columns, BK, bf16);
  if (r) return 1000 + r;
  r = make_tmap_2d_16b(&tx, x, M, K, ldx, nt, BK, bf16);
  if (r) return 2000 + r;
  RowsParams p{};
  p.M = M; p.N = N; p.ldy = ldy; p.ldr = ldr; p.y = y; p.residual = residual;
  p.packed = ldy % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 7) == 0;
  p.k_blocks = (K + BK - 1) / BK;
  p.idesc = make_idesc_f16(TILE, nt, bf16 ? 1 : 0, 0, 0);
  // as many CTAs as run at once, two on an SM, none of fewer than four k-blocks.  A second round of a few costs a round, and
  // clusters of other sizes than powers of two find their SMs late: 6144 x 4096 in 384 CTAs of 8 splits 15.5 us, in 288 of 6 14.9,
  // in 192 of 4 11.5.
  const int tiles = (N + columns - 1) / columns;
  int splits = 1;
  while (splits < MAX_SPLITS && tiles * splits <= cb_num_sms() && p.k_blocks >= splits * 8) splits *= 2;
  p.per_split = (p.k_blocks + splits - 1) / splits;
  if (nt == 16)
    return bf16 ? launch_rows<__nv_bfloat16, 16, ACT>(tw, tx, p, tiles, splits, stream) : launch_rows<__half, 16, ACT>(tw, tx, p, tiles, splits, stream);
  return bf16 ? launch_rows<__nv_bfloat16, 32, ACT>(tw, tx, p, tiles, splits, stream) : launch_rows<__half, 32, ACT>(tw, tx, p, tiles, splits, stream);
}

}  // namespace

extern "C" {

// x [M, K] (row stride ldx), w [N, K] contiguous, y [M, N] (row stride ldy), residual [M, N] (row stride ldr) or null.  M <= 32;
// K, ldx multiples of 8 and x, w 16-byte aligned (TMA).
int cb_gemm_rows(const void* x, const void* w, void* y, const void* residual, int M, int N, int K, int64_t ldx, int64_t ldy, int64_t ldr,
                 int dtype, cudaStream_t stream) {
  return rows_product<PLAIN>(x, w, y, residual, M, N, N, K, ldx, ldy, ldr, dtype, stream);
}

// The gated unit behind a projection: w [2 N, K], y [M, N]; act: 0 silu, 1 gelu (tanh), 2 gelu (erf)
int cb_gemm_rows_gated(const void* x, const void* w, void* y, int M, int N, int K, int64_t ldx, int64_t ldy, int act, int dtype,
                       cudaStream_t stream) {
  if (N > 0x3fffffff) return (int)cudaErrorInvalidValue;
  if (act == 0) return rows_product<0>(x, w, y, nullptr, M, N, 2 * N, K, ldx, ldy, 0, dtype, stream);
  if (act == 1) return rows_product<1>(x, w, y, nullptr, M, N, 2 * N, K, ldx, ldy, 0, dtype, stream);
  if (act == 2) return rows_product<2>(x, w, y, nullptr, M, N, 2 * N, K, ldx, ldy, 0, dtype, stream);
  return (int)cudaErrorInvalidValue;
}

// table [entries, row_bytes], out [n, row_bytes]; row_bytes a multiple of 16, both 16-byte aligned
int cb_embed_rows(const int64_t* ids, const void* table, void* out, int64_t n, int64_t entries, int64_t row_bytes, cudaStream_t stream) {
  if (n == 0) return 0;
  if ((row_bytes & 15) || n > 0x7fffffffll || row_bytes / 16 > 0x7fffffffll) return (int)cudaErrorInvalidValue;
  return cb_launch_early(embed_rows_kernel, dim3((unsigned)n), dim3(256), 0, stream, ids, (const uint4*)table, (uint4*)out, entries,
                         (int)(row_bytes / 16));
}

}  // extern "C"
