// Fused (vocab-parallel) cross-entropy building blocks for sm_100a.
// One CTA per token row.  Forward reads the logits once: running max and sum of exponentials against it, and the target's
// logit (vocab-parallel callers rescale the sums to the all-reduced max); a one-block kernel turns the rows into the loss.
// Backward reads once and writes the gradient once.  Replaces the eager torch composition in the reference's DistCrossEntropy
// (colossalai/shardformer/layer/loss.py:25-127) which materialises exp(logits) and a one-hot mask.
// Bound: HBM.  4096 rows of 128256 bf16: max and sum in passes of their own took 174 + 180 us, the one pass 172 us; the
// gradient (read + write) runs at 6.3 TB/s.
#include <type_traits>

#include "common.cuh"

constexpr int CE_UNROLL = 4;           // 16-byte vectors a thread has in flight
// Threads of a row: enough for CE_UNROLL vectors each, 32 to 512 (131072 rows of 1024 / 8192 bf16:
// 512 threads 739 / 1234 us, 32 / 256 of them 71 / 556).  A constant of the kernel:
// with a stride read from the launch 4096 rows of 128256 took 196 us instead of 172.
template <typename F> int ce_by_width(int vecs, const F& launch) {
  if (vecs <= 32 * CE_UNROLL) return launch(std::integral_constant<int, 32>());
  if (vecs <= 64 * CE_UNROLL) return launch(std::integral_constant<int, 64>());
  if (vecs <= 128 * CE_UNROLL) return launch(std::integral_constant<int, 128>());
  if (vecs <= 256 * CE_UNROLL) return launch(std::integral_constant<int, 256>());
  return launch(std::integral_constant<int, 512>());
}

// stats: [3, rows] fp32 = max over the row, sum of exp(x - max), the target's logit (0 if it is not in this shard)
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS) ce_row_stats_kernel(const T* __restrict__ x, const int64_t* __restrict__ target,
                                                               float* __restrict__ stats, int rows, int V, int Vv,
                                                               int64_t vocab_start, int64_t ignore_index) {
  constexpr int VEC = Vec16<T>::N;
  __shared__ float red[64];
  const int r = blockIdx.x;
  const T* row = x + (size_t)r * V;
  float m = -INFINITY, s = 0.f;
  constexpr int STEP = THREADS * VEC;
  auto take = [&](int c0, auto whole_tag) {      // (a row's end is a copy of the code: no comparison per element elsewhere)
    constexpr bool WHOLE = decltype(whole_tag)::value;
    Vec16<T> v[CE_UNROLL];
#pragma unroll
    for (int u = 0; u < CE_UNROLL; ++u)
      if (WHOLE || c0 + u * STEP < Vv) v[u].load_nc(row + c0 + u * STEP);
    float mc = -INFINITY;
#pragma unroll
    for (int u = 0; u < CE_UNROLL; ++u)
#pragma unroll
      for (int i = 0; i < VEC; ++i)
        if (WHOLE || c0 + u * STEP + i < Vv) mc = fmaxf(mc, v[u].get(i));
    if (mc > m) {                                // (a row of -inf so far keeps s = 0: exp(-inf - -inf) is not taken)
      s *= __expf(m - mc);
      m = mc;
    }
    const float ref = m == -INFINITY ? 0.f : m;
#pragma unroll
    for (int u = 0; u < CE_UNROLL; ++u)
#pragma unroll
      for (int i = 0; i < VEC; ++i)
        if (WHOLE || c0 + u * STEP + i < Vv) s += __expf(v[u].get(i) - ref);
  };
  int c0 = threadIdx.x * VEC;
  for (; c0 + (CE_UNROLL - 1) * STEP + VEC <= Vv; c0 += CE_UNROLL * STEP) take(c0, std::true_type{});
  for (; c0 < Vv; c0 += CE_UNROLL * STEP) take(c0, std::false_type{});
  const float mr = block_max(m, red);
  float t[1] = {s * (m == -INFINITY ? 1.f : __expf(m - mr))};          // m = -inf: s is 0, or NaN from a NaN logit
  block_sum<1>(t, red + 32);
  if (threadIdx.x == 0) {
    stats[r] = mr;
    stats[rows + r] = t[0];
    const int64_t tg = target[r], local = tg - vocab_start;
    stats[2 * rows + r] = (tg != ignore_index && local >= 0 && local < Vv) ? to_f32<T>(row[local]) : 0.f;
  }
}

// loss = sum over rows with a label of log(sumexp) + max - target logit, divided by their number (at least 1) when `mean`.
// One block up to CE_LOSS_ROWS rows; more rows are dealt out to up to CE_LOSS_BLOCKS blocks, whose sums a second launch adds up in
// their order (131072 rows: one block
// 130 us, now 3.6 and 2.4 to add them up; 16384 rows 17 us, 3.4 and 1.8).
constexpr int CE_LOSS_ROWS = 4096, CE_LOSS_BLOCKS = 128;
struct CePart {
  double sum;
  unsigned count;
};
// sums over the block, always in the same order; in thread 0
CB_DEVICE void ce_block_sum(double& sum, unsigned& count, double* sums, unsigned* counts) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  count = __reduce_add_sync(0xffffffffu, count);
  if (lane == 0) { sums[warp] = sum; counts[warp] = count; }
  __syncthreads();
  if (warp != 0) return;
  const bool live = lane < (int)blockDim.x / 32;
  sum = live ? sums[lane] : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  count = __reduce_add_sync(0xffffffffu, live ? counts[lane] : 0u);
}
CB_DEVICE void ce_loss_finish(double sum, unsigned count, int mean, float* loss, int64_t* n_valid) {
  *n_valid = count;
  *loss = (float)(mean ? sum / max(count, 1u) : sum);
}

__global__ void __launch_bounds__(1024) ce_loss_kernel(const float* __restrict__ stats, const int64_t* __restrict__ target,
                                                       float* __restrict__ loss, int64_t* __restrict__ n_valid,
                                                       CePart* __restrict__ parts, int rows, int64_t ignore_index, int mean) {
  __shared__ double sums[32];
  __shared__ unsigned counts[32];
  double acc = 0.0;
  unsigned count = 0;                  // whole numbers: an fp32 count is exact up to 2^24 rows only
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += (int64_t)gridDim.x * blockDim.x)
    if (target[r] != ignore_index) {
      acc += log((double)stats[rows + r]) + stats[r] - stats[2 * (int64_t)rows + r];               // (logf is approximate here)
      ++count;
    }
  ce_block_sum(acc, count, sums, counts);
  if (threadIdx.x == 0) {
    if (gridDim.x > 1) parts[blockIdx.x] = CePart{acc, count};
    else ce_loss_finish(acc, count, mean, loss, n_valid);
  }
}

__global__ void __launch_bounds__(CE_LOSS_BLOCKS) ce_loss_join_kernel(const CePart* __restrict__ parts, int n, float* __restrict__ loss,
                                                                      int64_t* __restrict__ n_valid, int mean) {
  __shared__ double sums[32];
  __shared__ unsigned counts[32];
  CePart a = {0.0, 0u};
  if ((int)threadIdx.x < n) a = parts[threadIdx.x];
  ce_block_sum(a.sum, a.count, sums, counts);
  if (threadIdx.x == 0) ce_loss_finish(a.sum, a.count, mean, loss, n_valid);
}

template <typename T>
__global__ void __launch_bounds__(512) ce_softmax_grad_kernel(const T* __restrict__ x,
                                                              const int64_t* __restrict__ target,
                                                              const float* __restrict__ gmax,
                                                              const float* __restrict__ sumexp,
                                                              const float* __restrict__ row_scale,
                                                              const float* __restrict__ scale,
                                                              const int64_t* __restrict__ n_valid, T* __restrict__ g,
                                                              int V, int Vv, int64_t vocab_start,
                                                              int64_t ignore_index) {
  constexpr int VEC = Vec16<T>::N;
  const int r = gridDim.x - 1 - blockIdx.x;                    // from the end: what the forward read last is in L2 yet (533 -> 526 us)
  const T* row = x + (size_t)r * V;
  T* grow = g + (size_t)r * V;
  const int64_t t = target[r];
  const bool ignored = (t == ignore_index);
  // a factor per row, or one for all divided by the number of labels
  const float f = row_scale != nullptr ? row_scale[r] : (n_valid != nullptr ? *scale / (float)max(*n_valid, (int64_t)1) : *scale);
  const float m = gmax[r], inv = ignored ? 0.f : f / sumexp[r];
  const float sc = ignored ? 0.f : f;
  const int64_t local = t - vocab_start;
  // Without a label every gradient is an exponential times zero: zero, unless one is not finite, which the maximum and the sum show
  // (a sum that is zero: a row of -inf).  The logits are not read again then; 4096 x 128256 bf16, a third of them: 532 -> 478 us.
  if (ignored && fabsf(m) < INFINITY && sumexp[r] > 0.f && sumexp[r] < INFINITY) {
    Vec16<T> o;
    o.raw = make_uint4(0u, 0u, 0u, 0u);
    for (int c = threadIdx.x * VEC; c < V; c += blockDim.x * VEC) o.store_na(grow + c);
    return;
  }
  constexpr int STEP = 512 * VEC;
  // 4096 x 128256 bf16, all with labels: one vector at a time 560 us (with the forward), four 528; fp32, one and two: 64 x 32000 19.1 and 17.8, 300 x 128256
  // 98 and 87, 2000 x 102400 397 and 390 (one, as the compiler unrolled it in a plain loop, 18.1, 97.7 and 399)
  constexpr int UNROLL = sizeof(T) == 4 ? 2 : CE_UNROLL;
  auto part = [&](int c0, auto whole_tag) {      // (a copy of the code for a row's end, as above)
    constexpr bool WHOLE = decltype(whole_tag)::value;
    Vec16<T> v[UNROLL], o;
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      if (WHOLE || c0 + u * STEP < V) v[u].load_nc(row + c0 + u * STEP);
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int c = c0 + u * STEP;
      if (!WHOLE && c >= V) break;
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        float p = (WHOLE || c + i < Vv) ? __expf(v[u].get(i) - m) * inv : 0.f;
        if ((int64_t)(c + i) == local) p -= sc;
        o.set(i, p);
      }
      o.store_na(grow + c);
    }
  };
  int c0 = threadIdx.x * VEC;
  for (; c0 + (UNROLL - 1) * STEP + VEC <= Vv; c0 += UNROLL * STEP) part(c0, std::true_type{});
  for (; c0 < V; c0 += UNROLL * STEP) part(c0, std::false_type{});
}

extern "C" {

int cb_ce_row_stats(const void* x, const int64_t* target, float* stats, int rows, int V, int Vv, int64_t vocab_start,
                    int64_t ignore_index, int dtype, cudaStream_t s) {
  if (rows == 0) return 0;
  CB_DISPATCH_FLOAT(dtype, T, {
    return ce_by_width(V / Vec16<T>::N, [&](auto threads) {
      ce_row_stats_kernel<T, decltype(threads)::value>
          <<<rows, decltype(threads)::value, 0, s>>>((const T*)x, target, stats, rows, V, Vv, vocab_start, ignore_index);
      return CB_LAUNCH_CHECK();
    });
  });
  return CB_LAUNCH_CHECK();
}

// blocks of cb_ce_loss: its scratch `parts` is 16 bytes for each of them (none for one)
int cb_ce_loss_blocks(int rows) {
  if (rows <= CE_LOSS_ROWS) return 1;
  const int blocks = rows / 1024 + (rows % 1024 != 0);
  return blocks < CE_LOSS_BLOCKS ? blocks : CE_LOSS_BLOCKS;
}

int cb_ce_loss(const float* stats, const int64_t* target, float* loss, int64_t* n_valid, void* parts, int rows,
               int64_t ignore_index, int mean, cudaStream_t s) {
  static_assert(sizeof(CePart) == 16, "");
  const int blocks = cb_ce_loss_blocks(rows);
  if (blocks > 1 && parts == nullptr) return (int)cudaErrorInvalidValue;
  ce_loss_kernel<<<blocks, 1024, 0, s>>>(stats, target, loss, n_valid, (CePart*)parts, rows, ignore_index, mean);
  if (blocks > 1) ce_loss_join_kernel<<<1, CE_LOSS_BLOCKS, 0, s>>>((const CePart*)parts, blocks, loss, n_valid, mean);
  return CB_LAUNCH_CHECK();
}

// row_scale: fp32 [T], or null and then scale fp32 [1] and n_valid int64 [1] (null: 1)
int cb_ce_softmax_grad(const void* x, const int64_t* target, const float* gmax, const float* sumexp,
                       const float* row_scale, const float* scale, const int64_t* n_valid, void* g, int T_, int V, int Vv,
                       int64_t vocab_start, int64_t ignore_index, int dtype, cudaStream_t s) {
  if (T_ == 0) return 0;
  CB_DISPATCH_FLOAT(dtype, T, {
    ce_softmax_grad_kernel<T><<<T_, 512, 0, s>>>((const T*)x, target, gmax, sumexp, row_scale, scale, n_valid, (T*)g, V, Vv,
                                                vocab_start, ignore_index);
  });
  return CB_LAUNCH_CHECK();
}

}  // extern "C"
