// Grouped (per-expert) tcgen05 GEMM for sm_100a: the three GEMMs of a mixture-of-experts MLP over token rows that are
// grouped by expert, with the group boundaries read ON THE DEVICE (no host sync, no per-expert launches).
//
//   MODE_NT  (forward)  Y[rows of e, N]  = X[rows of e, K] x W[e][N, K]^T         variable M per group
//   MODE_NN  (dgrad)    dX[rows of e, N] = dY[rows of e, K] x W[e][K, N]           variable M per group
//   MODE_TN  (wgrad)    dW[e][M, N]     (+)= dY[rows of e, M]^T x X[rows of e, N]  variable K (= rows) per group
//
// `offs[e]` is the exclusive end row of group e (cumulative counts, int32, device memory).  One persistent launch of CTA
// pairs (cta_group::2); every role warp walks the same tile list:
//   * variable-M modes compute the transpose: a tile is 256 output columns (the M of the instruction, rows or columns of the
//     weight) x up to 256 token rows (its N, any multiple of 16), so that a group's rows are cut into equal tiles with less than 16
//     rows of padding each and an expert with a handful of rows costs a handful.  With the rows as M, in tiles of 256, 64 experts
//     of 128-row multiples around 384 rows did a third more products than their rows, and the tensor pipe was 80 - 87 % busy with
//     them (two layers of 64 experts, 24576 rows, 2048 x 2816 and 1408 x 2048: forward 403 us, input gradients 412; now 336 and
//     360, bound by the loads: a tile of 196 rows wants 70 bytes a clock and SM).  The list is built from `offs` at kernel start.
//     Row tiles are taken in bands (tile_order.h; one expert of 16384 rows, 4096 x 4096, 416 - 448 us without, 351 so; of 65536
//     1600 - 1850 and 1340 - 1360).
//     A tile's last rows may be the next group's (or TMA zero fill) and are not stored;
//   * variable-K mode: every group owns (M / 256) x (N / 256) tiles whose reduction runs over the group's token rows; the
//     row range of a group must start and end on a multiple of 16, the reduction of one instruction - the dispatch lays groups out
//     that way (`moe/grouped_gemm.py` pads with zero rows otherwise) - so that no instruction mixes two experts.  Only as many
//     of them are issued, and as many rows loaded (in boxes of 32), as the group has.
//
// Replaces the reference's python loop over local experts (`shardformer/modeling/mixtral.py:177-191`) and the
// library's `torch._grouped_mm`.
#include <stdlib.h>

#include "activations.cuh"
#include "common.cuh"
#include "sm100.cuh"
#include "tile_order.h"

using namespace sm100;

namespace {

constexpr int UMMA_K = 16;
constexpr int UNGATED = -1;            // of the variable-M modes' ACT: a product alone
// epilogue warps behind the producer and the issuer: a product's own work hides behind four; a gated unit's does not
// (64 experts of 25088 rows as below: input gradient 178 us with four, 170 with eight; 8 of 8256, 1024 -> 2 x 512: 22.6 and 20.6, forward 24.7 and 22.6)
constexpr int rows_warps(int act) { return act == UNGATED ? 4 : 8; }
constexpr int WGRAD_THREADS = 320;     // .., eight
constexpr int BOX_ROWS = 32;           // token rows of the smaller TMA box: a request takes as long to issue as one of 64 rows
constexpr int ROWS_BOX = 64;           // of the larger one, variable-M modes (weight gradients: a k-block, as many)
constexpr int PAIR_M = 256;
constexpr int PAIR_N = 256;
constexpr int MAX_GROUPS = 512;
enum { MODE_NT = 0, MODE_NN = 1, MODE_TN = 2 };
// K-blocks and stages.  A tile of few rows is bound by its loads and takes them in small pieces (two layers of 64 experts, 2048 x 2816 and 1408 x
// 2048: K-blocks of 128 forward 347 us, input gradients 367; of 64 337 and 361).  A weight gradient gives a stage for second boxes of
// its epilogue (blocks of 96 and three stages: 498, 482 so).
constexpr int BK = 64;
template <int MODE> struct Block {
  static constexpr int STAGES = MODE == MODE_TN ? 5 : 6;
  static constexpr int A_BYTES = 128 * BK * 2, B_BYTES = 128 * BK * 2;
};
template <int MODE> constexpr int stage_ring() { return Block<MODE>::STAGES * (Block<MODE>::A_BYTES + Block<MODE>::B_BYTES); }
constexpr int BOXES = 2;               // of an epilogue warp of weight gradients
// behind the stages: the staging of the epilogue (weight gradients: BOXES of 32 x 64 per epilogue warp; variable-M modes: 32 rows x
// 32 columns per warp), the barriers, the groups' boundaries and the tile list of the variable-M modes
constexpr int BOX_BYTES = 32 * 128;
constexpr int ROW_BOX_BYTES = 32 * 64;
template <int MODE> constexpr int smem_bytes(int warps = 8) {
  return stage_ring<MODE>() + 256 + (MAX_GROUPS + 1) * 4 +
         (MODE == MODE_TN ? warps * BOXES * BOX_BYTES : warps * ROW_BOX_BYTES + (MAX_GROUPS + 1) * 4);
}

SM100_DEVICE void tma_store_3d(const CUtensorMap* map, const void* smem_src, int32_t c0, int32_t c1, int32_t c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               :: "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}

struct GroupedParams {
  const int* offs;          // [E] cumulative row ends
  int E;
  int total_rows;           // rows of the grouped operand(s) (buffer size; >= offs[E-1])
  int M, N, K;              // NT / NN: N = output columns, K = reduction; TN: M x N = per-expert output, K unused
  int ldc;
  long long c_group_stride; // TN: elements between the outputs of consecutive experts
  int w_group_rows;         // NT: N rows per expert in the [E * N, K] view of W; NN: K rows per expert in [E * K, N]
  int out_dtype;
  int accumulate;
  int tma_store;            // TN: 16-bit results that overwrite leave through shared memory and TMA
  uint32_t idesc;           // variable-M: without N, which is the tile's number of rows
  void* C;
  // gated forward: N = I columns of the unit's result, w [E, 2 I, K]; C [rows, 2 I] gate | up, unit [rows, I] = act(gate) up.
  // gated input gradient: N = I, what a row's product is is the unit's gradient; gate_up [rows, 2 I] from the forward, C [rows, 2 I] its gradient
  void* unit;
  const void* gate_up;
};

struct Tile {
  int group, m_blk, n_blk;
  int row0, row_end;        // variable-M: rows of the tile that exist;  TN: k range [row0, row_end)
  int n;                    // variable-M: rows of the tile, a multiple of 16
};

// bounds[e] .. bounds[e + 1]: the rows of group e; tile_start[e]: number of row tiles of groups < e (variable-M modes).  Both
// in shared memory, and every role looks its tiles up one ahead: read from memory where a tile begins they were 1300 of the 6300
// clocks that a tile of a weight gradient took.  `cur` is the last group found: tiles are visited in increasing order by every
// role.  `blocks`: 256-column blocks of the output.
template <int MODE>
SM100_DEVICE Tile find_tile(int t, int num_tiles, const GroupedParams& p, const int* bounds, const int* tile_start, int blocks, int& cur) {
  Tile r{};
  if (t >= num_tiles) return r;
  if (MODE == MODE_TN) {
    const int m_blocks = (p.M + PAIR_M - 1) / PAIR_M, per_group = m_blocks * blocks;
    while (t >= (cur + 1) * per_group) ++cur;
    r.group = cur;
    cb_tile_order(t - cur * per_group, m_blocks, blocks, r.m_blk, r.n_blk);
    r.row0 = bounds[cur];
    r.row_end = bounds[cur + 1];
    return r;
  }
  while (cur + 1 < p.E && t >= tile_start[cur + 1] * blocks) ++cur;
  r.group = cur;
  const int g0 = bounds[cur], end = bounds[cur + 1];
  const int local = t - tile_start[cur] * blocks, row_tiles = tile_start[cur + 1] - tile_start[cur];
  int row_tile;
  cb_tile_order(local, row_tiles, blocks, row_tile, r.m_blk);
  const int per = ((end - g0 + row_tiles - 1) / row_tiles + 15) & ~15;    // <= 256, and row_tiles - 1 of them are less than all
  r.row0 = g0 + row_tile * per;
  r.row_end = min(end, r.row0 + per);
  r.n = (r.row_end - r.row0 + 15) & ~15;
  return r;
}

template <typename T16>
SM100_DEVICE void store_row(T16* __restrict__ dst, const uint32_t (&acc)[32], int n_valid, bool accumulate) {
  if (n_valid >= 32) {
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      Vec16<T16> o;
      if (accumulate) o.load(dst + j);
#pragma unroll
      for (int i = 0; i < 8; ++i) o.set(i, __uint_as_float(acc[j + i]) + (accumulate ? o.get(i) : 0.f));
      o.store(dst + j);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < n_valid) dst[j] = from_f32<T16>(__uint_as_float(acc[j]) + (accumulate ? to_f32<T16>(dst[j]) : 0.f));
  }
}
SM100_DEVICE void store_row(float* __restrict__ dst, const uint32_t (&acc)[32], int n_valid, bool accumulate) {
#pragma unroll
  for (int j = 0; j < 32; ++j)
    if (j < n_valid) dst[j] = __uint_as_float(acc[j]) + (accumulate ? dst[j] : 0.f);
}

// The variable-M modes.  A = the weight (NT: rows of W[e], K-major; NN: columns of W[e], MN-major), B = the token rows (K-major).
// ACT: the gated unit of activations.cuh that lies between two layers of an expert, or UNGATED.  Forward: a CTA's 128 rows of the weight are 64 of the gate and the
// 64 of up that belong to them, so that both factors meet in its epilogue, which writes the unit's result beside them.  Input gradient: the
// epilogue has the unit's gradient in its boxes and turns it into that of gate and up.  The roundings are those of launches of their own, which read
// again what was just written, at the memory's rate.  64 experts of 25088 rows, 2048 -> 2 x 1408 -> 2048: forward 281 -> 255 us (the product alone
// 239), input gradient 191 -> 170 (137 alone); 16 experts of 16512, 2048 -> 2 x 1024: 120 -> 110 and 83 -> 73.  What is left of the unit are the bytes
// that it has to move, past products that the SMs' reads bound already.
template <int MODE, typename T, int ACT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(64 + 32 * rows_warps(ACT), 1)
grouped_rows_2cta_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                         const __grid_constant__ CUtensorMap tmap_x32, const GroupedParams p) {
  constexpr int WARPS = rows_warps(ACT);
  constexpr bool A_MN = MODE == MODE_NN, GATED = ACT != UNGATED;
  constexpr int BLOCK_COLS = GATED && MODE == MODE_NT ? PAIR_M / 2 : PAIR_M;             // columns of N that a pair has
  constexpr int STAGES = Block<MODE>::STAGES, A_BYTES = Block<MODE>::A_BYTES, B_BYTES = Block<MODE>::B_BYTES;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + STAGES * A_BYTES;
  uint8_t* smem_box = smem + stage_ring<MODE>();                                                // [epilogue warps]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_box + WARPS * ROW_BOX_BYTES);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tmem_full = bars + 2 * STAGES;
  uint64_t* tmem_empty = bars + 2 * STAGES + 2;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  int* bounds = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(bars) + 256);         // [E + 1]
  int* tile_start = bounds + MAX_GROUPS + 1;                                            // [E + 1]

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();
  const bool leader_cta = cta_rank == 0;
  const int num_pairs = gridDim.x >> 1;
  const int pair_id = blockIdx.x >> 1;
  const int blocks = (p.N + BLOCK_COLS - 1) / BLOCK_COLS;

  // ---- tile list: per-group row-tile counts -> exclusive prefix (every CTA builds its own copy), a warp
  if (warp == 3) {
    int before = 0;
    for (int e0 = 0; e0 < p.E; e0 += 32) {
      const int e = e0 + lane;
      const int rows = e < p.E ? p.offs[e] - (e == 0 ? 0 : p.offs[e - 1]) : 0;
      int sum = (rows + PAIR_N - 1) / PAIR_N;
      const int own = sum;
#pragma unroll
      for (int d = 1; d < 32; d *= 2) {
        const int x = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += x;
      }
      if (e < p.E) {
        tile_start[e] = before + sum - own;
        bounds[e + 1] = p.offs[e];
      }
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) {
      tile_start[p.E] = before;
      bounds[0] = 0;
    }
  }
  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tmap_w);
    prefetch_tensormap(&tmap_x);
    prefetch_tensormap(&tmap_x32);
  }
  if (warp == 1 && lane == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 2 * WARPS);
    }
    fence_barrier_init();
  }
  cluster_sync();
  if (warp == 2) tmem_alloc_2cta<512>(tmem_ptr_smem);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  const int num_tiles = tile_start[p.E] * blocks;
  const int k_blocks = (p.K + BK - 1) / BK;

  if (warp == 0) {
    // ================================================================ TMA producer (both CTAs)
    int stage = 0, cur = 0;
    uint32_t phase = 0;
    Tile ahead = find_tile<MODE>(pair_id, num_tiles, p, bounds, tile_start, blocks, cur);
    for (int t = pair_id; t < num_tiles; t += num_pairs) {
      const Tile tl = ahead;
      ahead = find_tile<MODE>(t + num_pairs, num_tiles, p, bounds, tile_start, blocks, cur);
      const int a_m0 = tl.m_blk * PAIR_M + (int)cta_rank * 128;
      const int x_row0 = tl.row0 + (int)cta_rank * (tl.n / 2);
      const int boxes = (tl.n / 2 + BOX_ROWS - 1) / BOX_ROWS;              // <= 4: a CTA loads its half of the rows
      const uint32_t bytes = 2 * (A_BYTES + boxes * (BOX_ROWS * BK * 2));
      for (int kb = 0; kb < k_blocks; ++kb) {
        mbar_wait(&empty_bar[stage], phase ^ 1);
        if (lane == 0) {
          if (leader_cta) mbar_arrive_expect_tx(&full_bar[stage], bytes);
          const uint32_t fb = map_to_cta(smem_u32(&full_bar[stage]), 0);
          uint8_t* sa = smem_a + stage * A_BYTES;
          uint8_t* sb = smem_b + stage * B_BYTES;
          const int k0 = kb * BK;
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
              tma_load_2d_2sm(&tmap_w, fb, sa + j * (BK * 128), a_m0 + j * 64, tl.group * p.w_group_rows + k0);
          } else if (GATED) {
            const int gate = tl.group * p.w_group_rows + tl.m_blk * BLOCK_COLS + (int)cta_rank * 64;
            tma_load_2d_2sm(&tmap_w, fb, sa, k0, gate);
            tma_load_2d_2sm(&tmap_w, fb, sa + 64 * 128, k0, gate + p.N);
          } else {
            tma_load_2d_2sm(&tmap_w, fb, sa, k0, tl.group * p.w_group_rows + a_m0);
          }
          for (int i = 0; i < boxes; i += 2)
            tma_load_2d_2sm(i + 1 < boxes ? &tmap_x : &tmap_x32, fb, sb + i * (BOX_ROWS * 128), k0, x_row0 + i * BOX_ROWS);
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ================================================================ MMA issuer (leader CTA)
    if (leader_cta) {
      const uint32_t leader = elect_one();
      const uint64_t da0 = A_MN ? make_smem_desc_sw128(smem_u32(smem_a), BK * 128, 1024) : make_smem_desc_sw128(smem_u32(smem_a), 16, 1024);
      const uint64_t db0 = make_smem_desc_sw128(smem_u32(smem_b), 16, 1024);
      int stage = 0, cur = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      Tile ahead = find_tile<MODE>(pair_id, num_tiles, p, bounds, tile_start, blocks, cur);
      for (int t = pair_id; t < num_tiles; t += num_pairs) {
        const uint32_t idesc = p.idesc | (uint32_t)(ahead.n >> 3) << 17;
        mbar_wait(&tmem_empty[acc], acc_phase ^ 1);
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * PAIR_N;
        for (int kb = 0; kb < k_blocks; ++kb) {
          mbar_wait(&full_bar[stage], phase);
          tc_fence_after();
          const uint32_t a = desc_lo(da0) + stage * (A_BYTES >> 4), b = desc_lo(db0) + stage * (B_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint32_t kmaj = k * (UMMA_K * 2) >> 4;
            umma_f16_ss_2cta_warp(leader, tmem_d, a + (A_MN ? k * (UMMA_K * 128) >> 4 : kmaj), desc_hi(da0), b + kmaj, desc_hi(db0), idesc,
                                  (kb > 0 || k > 0) ? 1u : 0u);
          }
          if (leader) {
            umma_commit_2cta(&empty_bar[stage], 3);
            if (kb == k_blocks - 1) umma_commit_2cta(&tmem_full[acc], 3);
          }
          __syncwarp();
          if (kb == 0) ahead = find_tile<MODE>(t + num_pairs, num_tiles, p, bounds, tile_start, blocks, cur);   // under the products
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (k_blocks == 0) ahead = find_tile<MODE>(t + num_pairs, num_tiles, p, bounds, tile_start, blocks, cur);
        if (k_blocks == 0 && leader) umma_commit_2cta(&tmem_full[acc], 3);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else {
    // ================================================================ epilogue (warps 2..5, gated 2..9, both CTAs): lane = output column
    const int quarter = warp & 3, turn = (warp - 2) >> 2;                  // gated: 32 rows of each 64 a warp
    uint8_t* box = smem_box + (turn * 4 + quarter) * ROW_BOX_BYTES;        // [32 token rows][32 columns]
    const auto drained = [&](int a) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (leader_cta) mbar_arrive(&tmem_empty[a]);
        else mbar_arrive_cluster(map_to_cta(smem_u32(&tmem_empty[a]), 0));
      }
    };
    int acc = 0, cur = 0;
    uint32_t acc_phase = 0;
    Tile ahead = find_tile<MODE>(pair_id, num_tiles, p, bounds, tile_start, blocks, cur);
    for (int t = pair_id; t < num_tiles; t += num_pairs) {
      const Tile tl = ahead;
      ahead = find_tile<MODE>(t + num_pairs, num_tiles, p, bounds, tile_start, blocks, cur);
      // gated forward: two warps have the gate and two the up of the CTA's 64 columns
      const int col = GATED && MODE == MODE_NT ? tl.m_blk * BLOCK_COLS + (int)cta_rank * 64 + (quarter & 1) * 32 + (lane & 3) * 8
                                               : tl.m_blk * PAIR_M + (int)cta_rank * 128 + quarter * 32 + (lane & 3) * 8;
      const size_t row = (size_t)(tl.row0 + (lane >> 2));
      T* out = reinterpret_cast<T*>(p.C) + row * p.ldc + col + (GATED && MODE == MODE_NT && quarter >= 2 ? p.N : 0);
      const int rows = col < p.N ? tl.row_end - tl.row0 - (lane >> 2) : 0;     // N % 8 == 0: a lane's columns exist or do not
      mbar_wait(&tmem_full[acc], acc_phase);
      tc_fence_after();
      const uint32_t taddr = tmem_base + acc * PAIR_N + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
      for (int c = turn * 32; c < tl.n; c += WARPS * 8) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(taddr + c, v);
        Vec16<T> gate[4], up[4];                                           // gated input gradient: asked for ahead, read once
        if constexpr (GATED && MODE == MODE_NN) {
          const T* gu = reinterpret_cast<const T*>(p.gate_up) + row * p.ldc + col;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (c + i * 8 < rows) {
              gate[i].raw = __ldcs(reinterpret_cast<const uint4*>(gu + (size_t)(c + i * 8) * p.ldc));
              up[i].raw = __ldcs(reinterpret_cast<const uint4*>(gu + (size_t)(c + i * 8) * p.ldc + p.N));
            }
        }
        tmem_ld_wait();
        if (c + WARPS * 8 >= tl.n) drained(acc);
        T* mine = reinterpret_cast<T*>(box) + lane;
#pragma unroll
        for (int i = 0; i < 32; ++i) mine[i * 32] = from_f32<T>(k_blocks > 0 ? __uint_as_float(v[i]) : 0.f);
        if constexpr (GATED && MODE == MODE_NT) asm volatile("bar.sync %0, 128;" ::"r"(1 + turn) : "memory");
        else __syncwarp();
        const uint8_t* piece = box + lane * 16;
#pragma unroll
        for (int i = 0; i < 4; ++i) {                                      // 16 bytes of eight rows at a time
          if (c + i * 8 >= rows) break;
          T* dst = out + (size_t)(c + i * 8) * p.ldc;
          Vec16<T> x;
          x.load(reinterpret_cast<const T*>(piece + i * 512));
          if constexpr (GATED && MODE == MODE_NN) {
            Vec16<T> dg, du;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float gf = gate[i].get(e), uf = up[i].get(e), df = x.get(e);
              dg.set(e, df * uf * act_grad_f<GATED ? ACT : 0>(gf));
              du.set(e, df * act_f<GATED ? ACT : 0>(gf));
            }
            dg.store(dst);
            du.store(dst + p.N);
          } else {
            x.store(dst);
          }
          if constexpr (GATED && MODE == MODE_NT) {                        // the unit: half of the rows each
            if ((i >= 2) == (quarter >= 2)) {
              const uint8_t* pair = smem_box + (turn * 4 + (quarter & 1)) * ROW_BOX_BYTES + lane * 16 + i * 512;
              Vec16<T> g, u, o;
              g.load(reinterpret_cast<const T*>(pair));
              u.load(reinterpret_cast<const T*>(pair + 2 * ROW_BOX_BYTES));
#pragma unroll
              for (int e = 0; e < 8; ++e) o.set(e, act_f<GATED ? ACT : 0>(g.get(e)) * u.get(e));
              o.store(reinterpret_cast<T*>(p.unit) + (row + c + i * 8) * p.N + col);
            }
          }
        }
        __syncwarp();
        if constexpr (GATED && MODE == MODE_NT) asm volatile("bar.sync %0, 128;" ::"r"(1 + turn) : "memory");
      }
      if (turn * 32 >= tl.n) drained(acc);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  }
  tc_fence_before();
  cluster_sync();
  if (warp == 2) tmem_dealloc_2cta<512>(tmem_base);
}

// The variable-K mode.
template <typename OUT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(WGRAD_THREADS, 1)
grouped_wgrad_2cta_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                          const __grid_constant__ CUtensorMap tmap_a32, const __grid_constant__ CUtensorMap tmap_b32,
                          const __grid_constant__ CUtensorMap tmap_c, const GroupedParams p) {
  using B = Block<MODE_TN>;
  constexpr int STAGES = B::STAGES, A_BYTES = B::A_BYTES, B_BYTES = B::B_BYTES;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + STAGES * A_BYTES;
  uint8_t* smem_box = smem + stage_ring<MODE_TN>();                                                // [8 warps], 1024-byte aligned
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_box + 8 * BOXES * BOX_BYTES);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tmem_full = bars + 2 * STAGES;
  uint64_t* tmem_empty = bars + 2 * STAGES + 2;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  int* bounds = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(bars) + 256);         // [E + 1]

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();
  const bool leader = cta_rank == 0;
  const int num_pairs = gridDim.x >> 1;
  const int pair_id = blockIdx.x >> 1;
  const int n_blocks = (p.N + PAIR_N - 1) / PAIR_N;
  const int num_tiles = p.E * ((p.M + PAIR_M - 1) / PAIR_M) * n_blocks;

  for (int e = threadIdx.x; e <= p.E; e += WGRAD_THREADS) bounds[e] = e == 0 ? 0 : p.offs[e - 1];
  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_b);
  }
  if (warp == 1 && lane == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 16);
    }
    fence_barrier_init();
  }
  cluster_sync();
  if (warp == 2) tmem_alloc_2cta<512>(tmem_ptr_smem);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;

  if (warp == 0) {
    // ================================================================ TMA producer (both CTAs)
    int stage = 0, cur = 0;
    uint32_t phase = 0;
    Tile ahead = find_tile<MODE_TN>(pair_id, num_tiles, p, bounds, nullptr, n_blocks, cur);
    for (int t = pair_id; t < num_tiles; t += num_pairs) {
      const Tile tl = ahead;
      ahead = find_tile<MODE_TN>(t + num_pairs, num_tiles, p, bounds, nullptr, n_blocks, cur);
      const int k_rows = tl.row_end - tl.row0;
      const int a_m0 = tl.m_blk * PAIR_M + (int)cta_rank * 128;      // columns m of dY, n of X (MN-major, rows = tokens)
      const int b_n0 = tl.n_blk * PAIR_N + (int)cta_rank * 128;
      for (int k = 0; k < k_rows; k += BK) {
        mbar_wait(&empty_bar[stage], phase ^ 1);
        if (lane == 0) {
          const int boxes = (min(k_rows - k, BK) + BOX_ROWS - 1) / BOX_ROWS;
          if (leader) mbar_arrive_expect_tx(&full_bar[stage], 2 * boxes * (4 * BOX_ROWS * 128));
          const uint32_t fb = map_to_cta(smem_u32(&full_bar[stage]), 0);
          uint8_t* sa = smem_a + stage * A_BYTES;
          uint8_t* sb = smem_b + stage * B_BYTES;
          if (boxes == BK / BOX_ROWS) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              tma_load_2d_2sm(&tmap_a, fb, sa + j * (BK * 128), a_m0 + j * 64, tl.row0 + k);
              tma_load_2d_2sm(&tmap_b, fb, sb + j * (BK * 128), b_n0 + j * 64, tl.row0 + k);
            }
          } else {
            for (int i = 0; i < boxes; ++i)
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                const int at = j * (BK * 128) + i * (BOX_ROWS * 128), row = tl.row0 + k + i * BOX_ROWS;
                tma_load_2d_2sm(&tmap_a32, fb, sa + at, a_m0 + j * 64, row);
                tma_load_2d_2sm(&tmap_b32, fb, sb + at, b_n0 + j * 64, row);
              }
          }
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ================================================================ MMA issuer (leader CTA)
    if (leader) {
      const uint32_t one = elect_one();
      const uint64_t da0 = make_smem_desc_sw128(smem_u32(smem_a), BK * 128, 1024), db0 = make_smem_desc_sw128(smem_u32(smem_b), BK * 128, 1024);
      int stage = 0, cur = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      Tile ahead = find_tile<MODE_TN>(pair_id, num_tiles, p, bounds, nullptr, n_blocks, cur);
      for (int t = pair_id; t < num_tiles; t += num_pairs) {
        const int k_rows = __shfl_sync(0xffffffffu, ahead.row_end - ahead.row0, 0);
        mbar_wait(&tmem_empty[acc], acc_phase ^ 1);
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * PAIR_N;
        for (int k0 = 0; k0 < k_rows; k0 += BK) {
          mbar_wait(&full_bar[stage], phase);
          tc_fence_after();
          const uint32_t a = desc_lo(da0) + stage * (A_BYTES >> 4), b = desc_lo(db0) + stage * (B_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)                // as many as the group has rows
            if (k0 + k * UMMA_K < k_rows)
              umma_f16_ss_2cta_warp(one, tmem_d, a + (k * (UMMA_K * 128) >> 4), desc_hi(da0), b + (k * (UMMA_K * 128) >> 4), desc_hi(db0), p.idesc,
                                    (k0 > 0 || k > 0) ? 1u : 0u);
          if (one) {
            umma_commit_2cta(&empty_bar[stage], 3);
            if (k0 + BK >= k_rows) umma_commit_2cta(&tmem_full[acc], 3);
          }
          __syncwarp();
          if (k0 == 0) ahead = find_tile<MODE_TN>(t + num_pairs, num_tiles, p, bounds, nullptr, n_blocks, cur);   // under the products
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (k_rows <= 0) ahead = find_tile<MODE_TN>(t + num_pairs, num_tiles, p, bounds, nullptr, n_blocks, cur);
        if (k_rows <= 0 && lane == 0) umma_commit_2cta(&tmem_full[acc], 3);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else {
    // ================================================================ epilogue (warps 2..9, both CTAs)
    const int quarter = warp & 3, half = (warp - 2) >> 2;                    // 32 rows x 128 columns of the CTA's 128 x 256
    constexpr int COLS = PAIR_N / 2;
    uint8_t* const boxes = smem_box + (warp - 2) * BOXES * BOX_BYTES;
    int acc = 0, cur = 0;
    uint32_t acc_phase = 0;
    Tile ahead = find_tile<MODE_TN>(pair_id, num_tiles, p, bounds, nullptr, n_blocks, cur);
    auto release = [&]() {                               // the accumulator's columns of this warp are in registers
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (leader) mbar_arrive(&tmem_empty[acc]);
        else mbar_arrive_cluster(map_to_cta(smem_u32(&tmem_empty[acc]), 0));
      }
    };
    for (int t = pair_id; t < num_tiles; t += num_pairs) {
      const Tile tl = ahead;
      ahead = find_tile<MODE_TN>(t + num_pairs, num_tiles, p, bounds, nullptr, n_blocks, cur);
      const int m0 = tl.m_blk * PAIR_M + (int)cta_rank * 128 + quarter * 32, n0 = tl.n_blk * PAIR_N + half * COLS;
      const bool empty_k = tl.row_end <= tl.row0;        // an expert without tokens: its gradient is zero
      mbar_wait(&tmem_full[acc], acc_phase);
      tc_fence_after();
      const uint32_t taddr = tmem_base + acc * PAIR_N + half * COLS + ((uint32_t)(quarter * 32) << 16);
      if (p.tma_store) {
        if constexpr (sizeof(OUT) == 2) {
          // A weight gradient's reduction is an expert's few hundred rows, so the store of a tile costs as much as its product:
          // sixteen bytes per lane to 32 rows at a time (4096 clocks a tile) bound this mode (two GEMMs of 64 experts x 2048 x
          // 2816 / 1408, 384 rows each: 672 us).  The 32 x 64 box of a warp goes through shared memory in the 128-byte swizzle
          // and leaves as one TMA store, clipped at the expert's edges, the next box read while one is packed (501).  Four warps
          // took 5000 clocks for a tile whose product takes 3100: eight of them and fewer rows of padding, 465.  Two boxes a warp,
          // so that one is packed while the other leaves, and a converged issuer: one call after the other 507 -> 482, 64 experts with 28 rows each 291 ->
          // 277.  Of that 282 are the 1.1 GB that are written, at the 3.9 TB/s that HBM takes from writes alone.  The tiles of three to sixteen experts in
          // turn, so that large and small reductions meet, were no faster (3: 493, 16: 543).
          uint32_t v[2][64];
          tmem_ld_32x32b_x32(taddr, *reinterpret_cast<uint32_t(*)[32]>(&v[0][0]));
          tmem_ld_32x32b_x32(taddr + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[0][32]));
#pragma unroll
          for (int b = 0; b < COLS / 64; ++b) {
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 64; ++i) asm volatile("" : "+r"(v[b & 1][i]));                  // nothing reads them earlier
            if (b + 1 < COLS / 64) {
              tmem_ld_32x32b_x32(taddr + (b + 1) * 64, *reinterpret_cast<uint32_t(*)[32]>(&v[(b + 1) & 1][0]));
              tmem_ld_32x32b_x32(taddr + (b + 1) * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[(b + 1) & 1][32]));
            } else {
              release();
            }
            uint8_t* box = boxes + (b % BOXES) * BOX_BYTES;
            if (lane == 0) tma_store_wait_read<BOXES - 1>();   // the store that last read this box has read it
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              Vec16<OUT> w;
#pragma unroll
              for (int i = 0; i < 8; ++i) w.set(i, empty_k ? 0.f : __uint_as_float(v[b & 1][8 * j + i]));
              w.store(reinterpret_cast<OUT*>(box + lane * 128 + ((j ^ (lane & 7)) << 4)));
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
              if (m0 < p.M && n0 + b * 64 < p.N) tma_store_3d(&tmap_c, box, n0 + b * 64, m0, tl.group);
              tma_store_commit();
            }
          }
        }
      } else {
        const int row = m0 + lane;
        OUT* out = reinterpret_cast<OUT*>(p.C) + (size_t)tl.group * (size_t)p.c_group_stride + (size_t)row * p.ldc + n0;
#pragma unroll 1
        for (int c = 0; c < COLS; c += 32) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(taddr + c, v);
          tmem_ld_wait();
          if (empty_k) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
          }
          if (row < p.M && n0 + c < p.N) store_row(out + c, v, p.N - (n0 + c), p.accumulate);
        }
        release();
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    if (p.tma_store && lane == 0) tma_store_wait<0>();
  }
  tc_fence_before();
  cluster_sync();
  if (warp == 2) tmem_dealloc_2cta<512>(tmem_base);
}

// the number of tiles is only known on the device: full persistent grids
template <int MODE, typename T, int ACT = UNGATED>
int launch_rows(const CUtensorMap& tw, const CUtensorMap& tx, const CUtensorMap& tx32, const GroupedParams& p, cudaStream_t stream) {
  static CbDeviceAttr attr;
  constexpr int warps = rows_warps(ACT), smem = smem_bytes<MODE>(warps);
  if (const int e = cb_allow_smem(attr, grouped_rows_2cta_kernel<MODE, T, ACT>, smem)) return e;
  grouped_rows_2cta_kernel<MODE, T, ACT><<<cb_num_sms() / 2 * 2, 64 + 32 * warps, smem, stream>>>(tw, tx, tx32, p);
  return (int)cudaGetLastError();
}

template <int MODE>
int launch_gated(const CUtensorMap& tw, const CUtensorMap& tx, const CUtensorMap& tx32, const GroupedParams& p, bool bf16, int act, cudaStream_t stream) {
  if (act < 0 || act > 2) return (int)cudaErrorInvalidValue;
  if (bf16) return act == 0   ? launch_rows<MODE, __nv_bfloat16, 0>(tw, tx, tx32, p, stream)
                   : act == 1 ? launch_rows<MODE, __nv_bfloat16, 1>(tw, tx, tx32, p, stream) : launch_rows<MODE, __nv_bfloat16, 2>(tw, tx, tx32, p, stream);
  return act == 0   ? launch_rows<MODE, __half, 0>(tw, tx, tx32, p, stream)
         : act == 1 ? launch_rows<MODE, __half, 1>(tw, tx, tx32, p, stream) : launch_rows<MODE, __half, 2>(tw, tx, tx32, p, stream);
}

template <typename OUT>
int launch_wgrad(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& ta32, const CUtensorMap& tb32, const CUtensorMap& tc,
                 const GroupedParams& p, cudaStream_t stream) {
  static CbDeviceAttr attr;
  if (const int e = cb_allow_smem(attr, grouped_wgrad_2cta_kernel<OUT>, smem_bytes<MODE_TN>())) return e;
  grouped_wgrad_2cta_kernel<OUT><<<cb_num_sms() / 2 * 2, WGRAD_THREADS, smem_bytes<MODE_TN>(), stream>>>(ta, tb, ta32, tb32, tc, p);
  return (int)cudaGetLastError();
}

}  // namespace

extern "C" {

// Variable-M grouped GEMM.  x [total_rows, K] (rows grouped by expert, `offs` = cumulative row ends on the device);
// transpose_b != 0: w [E, N, K] and y = x w[e]^T (forward);  transpose_b == 0: w [E, K, N] and y = x w[e] (dgrad with
// the forward weight [E, K(out), N(in)]).  y [total_rows, N].  Requirements: contiguous w, K % 8 == 0, N % 8 == 0,
// 16-byte aligned pointers, E <= 512; transpose_b == 0 additionally needs K % 128 == 0 (a k-block must not straddle
// two experts' weights: blocks of 64 rows would allow K % 64, which no caller has asked for and no test has run).
int cb_grouped_gemm(const void* x, const void* w, void* y, const int* offs, int E, int total_rows, int N, int K, int ldx,
                    int ldy, int transpose_b, int dtype, cudaStream_t stream) {
  if (E <= 0 || total_rows <= 0 || N <= 0) return 0;
  if (E > MAX_GROUPS || (dtype != CB_BF16 && dtype != CB_F16) || (K & 7) || (N & 7)) return (int)cudaErrorInvalidValue;
  if (!transpose_b && (K % 128)) return (int)cudaErrorInvalidValue;
  const bool bf16 = dtype == CB_BF16;
  CUtensorMap tx, tx32, tw;
  int r = make_tmap_2d_16b(&tx, x, total_rows, K, ldx, ROWS_BOX, 64, bf16);
  if (!r) r = make_tmap_2d_16b(&tx32, x, total_rows, K, ldx, BOX_ROWS, 64, bf16);
  if (r) return 1000 + r;
  GroupedParams p{};
  p.offs = offs; p.E = E; p.total_rows = total_rows; p.N = N; p.K = K; p.ldc = ldy; p.out_dtype = dtype; p.C = y;
  p.idesc = make_idesc_f16(PAIR_M, 0, bf16 ? 1 : 0, transpose_b ? 0 : 1, 0);
  if (transpose_b) {
    r = make_tmap_2d_16b(&tw, w, (uint64_t)E * N, K, K, 128, 64, bf16);
    if (r) return 2000 + r;
    p.w_group_rows = N;
    return bf16 ? launch_rows<MODE_NT, __nv_bfloat16>(tw, tx, tx32, p, stream) : launch_rows<MODE_NT, __half>(tw, tx, tx32, p, stream);
  }
  r = make_tmap_2d_16b(&tw, w, (uint64_t)E * K, N, N, BK, 64, bf16);
  if (r) return 2000 + r;
  p.w_group_rows = K;
  return bf16 ? launch_rows<MODE_NN, __nv_bfloat16>(tw, tx, tx32, p, stream) : launch_rows<MODE_NN, __half>(tw, tx, tx32, p, stream);
}

// The forward of a gated layer: w [E, 2 I, K] gate | up, gate_up [total_rows, 2 I] = x w[e]^T, unit [total_rows, I] = act(gate) up; act 0 silu,
// 1 gelu (tanh), 2 gelu (erf).  K, I multiples of 8.
int cb_grouped_gemm_gated(const void* x, const void* w, void* gate_up, void* unit, const int* offs, int E, int total_rows, int I, int K, int ldx,
                          int act, int dtype, cudaStream_t stream) {
  if (E <= 0 || total_rows <= 0 || I <= 0) return 0;
  if (E > MAX_GROUPS || (dtype != CB_BF16 && dtype != CB_F16) || (K & 7) || (I & 7) || I > 0x3fffffff) return (int)cudaErrorInvalidValue;
  const bool bf16 = dtype == CB_BF16;
  CUtensorMap tx, tx32, tw;
  int r = make_tmap_2d_16b(&tx, x, total_rows, K, ldx, ROWS_BOX, 64, bf16);
  if (!r) r = make_tmap_2d_16b(&tx32, x, total_rows, K, ldx, BOX_ROWS, 64, bf16);
  if (r) return 1000 + r;
  r = make_tmap_2d_16b(&tw, w, (uint64_t)E * 2 * I, K, K, 64, 64, bf16);
  if (r) return 2000 + r;
  GroupedParams p{};
  p.offs = offs; p.E = E; p.total_rows = total_rows; p.N = I; p.K = K; p.ldc = 2 * I; p.out_dtype = dtype; p.C = gate_up; p.unit = unit;
  p.idesc = make_idesc_f16(PAIR_M, 0, bf16 ? 1 : 0, 0, 0);
  p.w_group_rows = 2 * I;
  return launch_gated<MODE_NT>(tw, tx, tx32, p, bf16, act, stream);
}

// The input gradient of the layer behind it, on through the unit: w [E, K, I], dy [total_rows, K]; d_gate_up [total_rows, 2 I] from dy w[e] and gate_up.
// K a multiple of 128, I of 8.
int cb_grouped_gemm_gated_bwd(const void* dy, const void* w, const void* gate_up, void* d_gate_up, const int* offs, int E, int total_rows, int I,
                              int K, int lddy, int act, int dtype, cudaStream_t stream) {
  if (E <= 0 || total_rows <= 0 || I <= 0) return 0;
  if (E > MAX_GROUPS || (dtype != CB_BF16 && dtype != CB_F16) || (K % 128) || (I & 7) || I > 0x3fffffff) return (int)cudaErrorInvalidValue;
  const bool bf16 = dtype == CB_BF16;
  CUtensorMap tx, tx32, tw;
  int r = make_tmap_2d_16b(&tx, dy, total_rows, K, lddy, ROWS_BOX, 64, bf16);
  if (!r) r = make_tmap_2d_16b(&tx32, dy, total_rows, K, lddy, BOX_ROWS, 64, bf16);
  if (r) return 1000 + r;
  r = make_tmap_2d_16b(&tw, w, (uint64_t)E * K, I, I, BK, 64, bf16);
  if (r) return 2000 + r;
  GroupedParams p{};
  p.offs = offs; p.E = E; p.total_rows = total_rows; p.N = I; p.K = K; p.ldc = 2 * I; p.out_dtype = dtype; p.C = d_gate_up; p.gate_up = gate_up;
  p.idesc = make_idesc_f16(PAIR_M, 0, bf16 ? 1 : 0, 1, 0);
  p.w_group_rows = K;
  return launch_gated<MODE_NN>(tw, tx, tx32, p, bf16, act, stream);
}

// Variable-K grouped GEMM (weight gradients): dw[e] [M, N] (+)= dy[rows of e, M]^T x[rows of e, N].  Every group's row
// range must start and end on a multiple of 16.  out_dtype: bf16 / fp16 / fp32.
int cb_grouped_gemm_wgrad(const void* dy, const void* x, void* dw, const int* offs, int E, int total_rows, int M, int N,
                          int lddy, int ldx, int in_dtype, int out_dtype, int accumulate, cudaStream_t stream) {
  if (E <= 0 || M <= 0 || N <= 0) return 0;
  if (E > MAX_GROUPS || (in_dtype != CB_BF16 && in_dtype != CB_F16) || (M & 7) || (N & 7)) return (int)cudaErrorInvalidValue;
  const bool bf16 = in_dtype == CB_BF16;
  CUtensorMap ta, tb, ta32, tb32;
  int r = make_tmap_2d_16b(&ta, dy, total_rows, M, lddy, BK, 64, bf16);
  if (!r) r = make_tmap_2d_16b(&ta32, dy, total_rows, M, lddy, BOX_ROWS, 64, bf16);
  if (r) return 1000 + r;
  r = make_tmap_2d_16b(&tb, x, total_rows, N, ldx, BK, 64, bf16);
  if (!r) r = make_tmap_2d_16b(&tb32, x, total_rows, N, ldx, BOX_ROWS, 64, bf16);
  if (r) return 2000 + r;
  GroupedParams p{};
  p.offs = offs; p.E = E; p.total_rows = total_rows; p.M = M; p.N = N; p.K = 0; p.ldc = N;
  p.c_group_stride = (long long)M * N; p.out_dtype = out_dtype; p.accumulate = accumulate; p.C = dw;
  p.idesc = make_idesc_f16(PAIR_M, PAIR_N, bf16 ? 1 : 0, 1, 1);
  CUtensorMap tc = ta;
  p.tma_store = out_dtype != CB_F32 && !accumulate && (reinterpret_cast<uintptr_t>(dw) & 15) == 0;
  if (p.tma_store) {
    r = make_tmap_3d_16b(&tc, dw, N, M, E, N, (uint64_t)M * N, 64, 32, 1, out_dtype == CB_BF16);
    if (r) return 3000 + r;
  }
  if (out_dtype == CB_F32) return launch_wgrad<float>(ta, tb, ta32, tb32, tc, p, stream);
  return out_dtype == CB_BF16 ? launch_wgrad<__nv_bfloat16>(ta, tb, ta32, tb32, tc, p, stream)
                              : launch_wgrad<__half>(ta, tb, ta32, tb32, tc, p, stream);
}

}  // extern "C"
