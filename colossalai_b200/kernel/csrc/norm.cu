// Fused RMSNorm / LayerNorm forward + backward for sm_100a (memory-bound: 16-byte vector I/O, row in registers,
// fp32 statistics, one pass over HBM per tensor).
//
// Capability parity: reference apex FusedRMSNorm/FusedLayerNorm usage (shardformer/layer/normalization.py:27-135),
// extensions/csrc/kernel/cuda/layer_norm_kernel.cu (N8) and rms_layernorm_kernel.cu (N17: residual-add fusion).
// Design here is new: a single kernel handles (optional) residual-add + norm and emits rstd for backward;
// backward is a persistent grid that keeps dgamma/dbeta partials in registers and a tiny second pass reduces them.
#include "common.cuh"

constexpr int MAX_ITERS_LIMIT = 4;

// A block takes ROWS neighbouring rows, loaded and summed together: two wide ones in calls that fill the SMs several times over (8192 x 4096
// bf16 with a residual 43.7 -> 42.9 us, 3001 x 5120 21.7 -> 20.8, 5000 x 4096 fp32 54.5 -> 52.3; 8192 x 2048 22.3 and 22.4), else one.  With a
// residual, blocks of 512 threads and 32-bit rows fill the SMs later (two / one: 1200 x 4096 bf16 7.3 / 6.8 us, 1300 7 % slower, 1800 2 % faster; 1200 x
// 4096 fp32 6 % slower, 2100 1.5 %, 3200 1 % faster, 8192 82.6 / 86.8), and 32-bit rows of less than 768 threads gain nothing (2048 wide 2 to 11 %
// slower).  Bound: HBM, two rows in and two out.
constexpr int NORM_ROWS = 2;
template <typename T, bool HAS_RES, int MAX_ITERS, int ROWS>
__global__ void __launch_bounds__(1024) rmsnorm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ res_in,
                                                           const T* __restrict__ w, T* __restrict__ y,
                                                           T* __restrict__ res_out, float* __restrict__ rstd_out,
                                                           int rows, int H, float eps) {
  constexpr int VEC = Vec16<T>::N;
  __shared__ float red[64];
  static_assert(ROWS <= 2, "red holds two sums of 32 warps");
  cb_early_start();
  const int row0 = blockIdx.x * ROWS;
  Vec16<T> hv[ROWS][MAX_ITERS], rv[ROWS][MAX_ITERS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int it = 0; it < MAX_ITERS; ++it) {
      const int col = (it * blockDim.x + threadIdx.x) * VEC;
      if (col < H && (ROWS == 1 || row0 + r < rows)) {
        hv[r][it].load_nc(x + (size_t)(row0 + r) * H + col);
        if (HAS_RES) rv[r][it].load_nc(res_in + (size_t)(row0 + r) * H + col);
      }
    }
  float ss[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    ss[r] = 0.f;
#pragma unroll
    for (int it = 0; it < MAX_ITERS; ++it) {
      const int col = (it * blockDim.x + threadIdx.x) * VEC;
      if (col < H && (ROWS == 1 || row0 + r < rows)) {
        Vec16<T>& v = hv[r][it];
        if (HAS_RES) {
#pragma unroll
          for (int i = 0; i < VEC; ++i) v.set(i, v.get(i) + rv[r][it].get(i));
          v.store(res_out + (size_t)(row0 + r) * H + col);
        }
#pragma unroll
        for (int i = 0; i < VEC; ++i) { float f = v.get(i); ss[r] += f * f; }
      }
    }
  }
  block_sum<ROWS>(ss, red);
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    if (ROWS > 1 && row0 + r >= rows) break;
    const float rstd = rsqrtf(ss[r] / (float)H + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row0 + r] = rstd;
#pragma unroll
    for (int it = 0; it < MAX_ITERS; ++it) {
      const int col = (it * blockDim.x + threadIdx.x) * VEC;
      if (col < H) {
        Vec16<T> wv, o;
        wv.load(w + col);
#pragma unroll
        for (int i = 0; i < VEC; ++i) o.set(i, hv[r][it].get(i) * rstd * wv.get(i));
        o.store_na(y + (size_t)(row0 + r) * H + col);
      }
    }
  }
}

// dx = rstd * (w*dy - xhat * mean(w*dy*xhat)) (+ dres);   dw_partial[cta] = sum_rows dy * xhat
// Bound: HBM (three rows in, one out).  A block's rows follow one another through a reduction, so the next row is loaded before
// the current one's sum is taken; without that 8192 x 4096 bf16 took 64.8 us (4.1 TB/s), with it 54.9, and 44 since the launch
// bounds ask for no more than one block of 1024 threads per SM, which leaves the compiler the registers to do it with.
template <typename T, bool HAS_DRES, int MAX_ITERS>
__global__ void __launch_bounds__(1024, MAX_ITERS == 1 && !HAS_DRES && sizeof(T) == 4 ? 2 : 1) rmsnorm_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ h,
                                                           const T* __restrict__ w, const float* __restrict__ rstd,
                                                           const T* __restrict__ dres, T* __restrict__ dx,
                                                           float* __restrict__ dw_partial, int rows, int H) {
  constexpr int VEC = Vec16<T>::N;
  // Wider rows fill the registers of a 1024-thread block as they are; 32-bit rows without a second gradient need so few that two
  // blocks of 1024 threads fit an SM, which the next row's registers would make one (16384 x 4096: 135 us without, 204 with).
  constexpr bool AHEAD = MAX_ITERS == 1 && (HAS_DRES || VEC == 8);
  cb_early_start();
  __shared__ float red[64];
  struct Row { Vec16<T> dy[MAX_ITERS], h[MAX_ITERS], dr[MAX_ITERS]; float rs; };
  auto fetch = [&](Row& v, int row) {
    const size_t base = (size_t)row * H;
    v.rs = rstd[row];
#pragma unroll
    for (int it = 0; it < MAX_ITERS; ++it) {
      const int col = (it * blockDim.x + threadIdx.x) * VEC;
      if (col < H) {
        v.dy[it].load_nc(dy + base + col);
        v.h[it].load_nc(h + base + col);
        if (HAS_DRES && AHEAD) v.dr[it].load_nc(dres + base + col);
      }
    }
  };
  float dw_acc[MAX_ITERS][VEC];
  Vec16<T> wv[MAX_ITERS];
#pragma unroll
  for (int it = 0; it < MAX_ITERS; ++it) {
    const int col = (it * blockDim.x + threadIdx.x) * VEC;
    if (col < H) wv[it].load(w + col);
#pragma unroll
    for (int i = 0; i < VEC; ++i) dw_acc[it][i] = 0.f;
  }
  Row cur, nxt;
  if (AHEAD && (int)blockIdx.x < rows) fetch(cur, blockIdx.x);
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t base = (size_t)row * H;
    if (!AHEAD) fetch(cur, row);
    else if (row + (int)gridDim.x < rows) fetch(nxt, row + gridDim.x);
    float c[1] = {0.f};
#pragma unroll
    for (int it = 0; it < MAX_ITERS; ++it) {
      const int col = (it * blockDim.x + threadIdx.x) * VEC;
      if (col < H) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          const float xhat = cur.h[it].get(i) * cur.rs, g = cur.dy[it].get(i);
          c[0] += g * wv[it].get(i) * xhat;
          dw_acc[it][i] += g * xhat;
        }
      }
    }
    block_sum<1>(c, red);
    const float c1 = c[0] / (float)H;
#pragma unroll
    for (int it = 0; it < MAX_ITERS; ++it) {
      const int col = (it * blockDim.x + threadIdx.x) * VEC;
      if (col < H) {
        Vec16<T> o;
        if (HAS_DRES && !AHEAD) cur.dr[it].load_nc(dres + base + col);
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          const float xhat = cur.h[it].get(i) * cur.rs;
          float v = (cur.dy[it].get(i) * wv[it].get(i) - xhat * c1) * cur.rs;
          if (HAS_DRES) v += cur.dr[it].get(i);
          o.set(i, v);
        }
        o.store_na(dx + base + col);
      }
    }
    if (AHEAD) cur = nxt;
  }
  float* out = dw_partial + (size_t)blockIdx.x * H;
#pragma unroll
  for (int it = 0; it < MAX_ITERS; ++it) {
    const int col = (it * blockDim.x + threadIdx.x) * VEC;
    if (col < H) {
#pragma unroll
      for (int i = 0; i < VEC; i += 4)
        *reinterpret_cast<float4*>(out + col + i) = make_float4(dw_acc[it][i], dw_acc[it][i + 1], dw_acc[it][i + 2], dw_acc[it][i + 3]);
    }
  }
}

// out[c] = sum_p partial[p][c].  A block takes 32 columns, each of its 32 warps every 32nd partial row (128 bytes of it): one
// thread per column was 16 blocks of serial loads for H = 4096, 13.7 us for 296 rows; now 2.9.
template <typename T>
__global__ void __launch_bounds__(1024) reduce_partials_kernel(const float* __restrict__ partial, T* __restrict__ out, int P, int H,
                                                               int accumulate) {
  __shared__ float s[32][33];
  cb_early_start();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float v = 0.f;
  if (c < H) {
#pragma unroll 8
    for (int p = warp; p < P; p += 32) v += partial[(size_t)p * H + c];
  }
  s[warp][lane] = v;
  __syncthreads();
  const float t = warp_sum(s[lane][warp]);                 // this warp's column of the 32
  const int cw = blockIdx.x * 32 + warp;
  if (lane == 0 && cw < H) out[cw] = from_f32<T>(accumulate ? t + to_f32<T>(out[cw]) : t);
}

// ------------------------------------------------------------------------------------------- LayerNorm
template <typename T, int MAX_ITERS>
__global__ void __launch_bounds__(1024) layernorm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ w,
                                                             const T* __restrict__ b, T* __restrict__ y,
                                                             float* __restrict__ mean_out, float* __restrict__ rstd_out,
                                                             int rows, int H, float eps) {
  constexpr int VEC = Vec16<T>::N;
  __shared__ float red[64];
  const int row = blockIdx.x;
  const size_t base = (size_t)row * H;
  Vec16<T> xv[MAX_ITERS];
  float s[1] = {0.f};
#pragma unroll
  for (int it = 0; it < MAX_ITERS; ++it) {
    const int col = (it * blockDim.x + threadIdx.x) * VEC;
    if (col < H) {
      xv[it].load_nc(x + base + col);
#pragma unroll
      for (int i = 0; i < VEC; ++i) s[0] += xv[it].get(i);
    }
  }
  block_sum<1>(s, red);
  const float mean = s[0] / (float)H;
  float v[1] = {0.f};
#pragma unroll
  for (int it = 0; it < MAX_ITERS; ++it) {
    const int col = (it * blockDim.x + threadIdx.x) * VEC;
    if (col < H) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) { float d = xv[it].get(i) - mean; v[0] += d * d; }
    }
  }
  block_sum<1>(v, red);
  const float rstd = rsqrtf(v[0] / (float)H + eps);
  if (threadIdx.x == 0) {
    if (mean_out) mean_out[row] = mean;
    if (rstd_out) rstd_out[row] = rstd;
  }
#pragma unroll
  for (int it = 0; it < MAX_ITERS; ++it) {
    const int col = (it * blockDim.x + threadIdx.x) * VEC;
    if (col < H) {
      Vec16<T> wv, bv, o;
      wv.load(w + col);
      if (b) bv.load(b + col);
#pragma unroll
      for (int i = 0; i < VEC; ++i) o.set(i, (xv[it].get(i) - mean) * rstd * wv.get(i) + (b ? bv.get(i) : 0.f));
      o.store_na(y + base + col);
    }
  }
}

template <typename T, int MAX_ITERS>
__global__ void __launch_bounds__(1024) layernorm_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                             const T* __restrict__ w, const float* __restrict__ mean,
                                                             const float* __restrict__ rstd, T* __restrict__ dx,
                                                             float* __restrict__ dw_partial,
                                                             float* __restrict__ db_partial, int rows, int H) {
  constexpr int VEC = Vec16<T>::N;
  __shared__ float red[64];
  float dw_acc[MAX_ITERS][VEC], db_acc[MAX_ITERS][VEC];
  Vec16<T> wv[MAX_ITERS];
#pragma unroll
  for (int it = 0; it < MAX_ITERS; ++it) {
    const int col = (it * blockDim.x + threadIdx.x) * VEC;
    if (col < H) wv[it].load(w + col);
#pragma unroll
    for (int i = 0; i < VEC; ++i) { dw_acc[it][i] = 0.f; db_acc[it][i] = 0.f; }
  }
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t base = (size_t)row * H;
    const float mu = mean[row], rs = rstd[row];
    Vec16<T> dyv[MAX_ITERS], xv[MAX_ITERS];
    float c[2] = {0.f, 0.f};
#pragma unroll
    for (int it = 0; it < MAX_ITERS; ++it) {
      const int col = (it * blockDim.x + threadIdx.x) * VEC;
      if (col < H) {
        dyv[it].load_nc(dy + base + col);
        xv[it].load_nc(x + base + col);
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          const float xhat = (xv[it].get(i) - mu) * rs, g = dyv[it].get(i), wg = g * wv[it].get(i);
          c[0] += wg;
          c[1] += wg * xhat;
          dw_acc[it][i] += g * xhat;
          db_acc[it][i] += g;
        }
      }
    }
    block_sum<2>(c, red);
    const float c0 = c[0] / (float)H, c1 = c[1] / (float)H;
#pragma unroll
    for (int it = 0; it < MAX_ITERS; ++it) {
      const int col = (it * blockDim.x + threadIdx.x) * VEC;
      if (col < H) {
        Vec16<T> o;
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          const float xhat = (xv[it].get(i) - mu) * rs;
          o.set(i, (dyv[it].get(i) * wv[it].get(i) - c0 - xhat * c1) * rs);
        }
        o.store_na(dx + base + col);
      }
    }
  }
#pragma unroll
  for (int it = 0; it < MAX_ITERS; ++it) {
    const int col = (it * blockDim.x + threadIdx.x) * VEC;
    if (col < H) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        dw_partial[(size_t)blockIdx.x * H + col + i] = dw_acc[it][i];
        db_partial[(size_t)blockIdx.x * H + col + i] = db_acc[it][i];
      }
    }
  }
}

static inline int pick_block(int H, int vec) {
  int threads = ((H / vec + 31) / 32) * 32;
  if (threads > 1024) threads = 1024;
  if (threads < 32) threads = 32;
  return threads;
}
static inline int pick_iters(int H, int vec, int block) {
  int it = (H / vec + block - 1) / block;
  return it <= 1 ? 1 : (it <= 2 ? 2 : 4);
}
#define CB_DISPATCH_ITERS(iters, IT, ...)            \
  if (iters == 1) { constexpr int IT = 1; __VA_ARGS__; }    \
  else if (iters == 2) { constexpr int IT = 2; __VA_ARGS__; } \
  else { constexpr int IT = 4; __VA_ARGS__; }

extern "C" {

// Max hidden size supported by the register-resident path.
int cb_norm_max_hidden(int dtype) { return 1024 * MAX_ITERS_LIMIT * (dtype == CB_F32 ? 4 : 8); }

// Blocks of the backward kernels = rows of their partial sums: what fits an SM at 1024 threads, so that narrow rows keep as
// many bytes in flight as wide ones (two blocks of H / 8 threads per SM whatever H is: 1024 wide rows at 1.5 TB/s).
int cb_norm_bwd_grid(int rows, int H, int dtype) {
  const int block = pick_block(H, dtype == CB_F32 ? 4 : 8);
  const int per_sm = block >= 512 ? 2 : 1024 / block;
  const int g = cb_num_sms() * per_sm;
  return rows < g ? rows : g;
}

int cb_rmsnorm_fwd(const void* x, const void* res_in, const void* w, void* y, void* res_out, float* rstd, int rows,
                   int H, float eps, int dtype, cudaStream_t stream) {
  if (rows == 0) return 0;
  CB_DISPATCH_FLOAT(dtype, T, {
    const int block = pick_block(H, Vec16<T>::N);
    const int iters = pick_iters(H, Vec16<T>::N, block);
    CB_DISPATCH_ITERS(iters, IT, {
      constexpr int R = IT == 1 ? NORM_ROWS : 1;
      const bool wide_sums = res_in && sizeof(T) == 4;
      const int least = wide_sums ? 16 : res_in && block == 512 ? 12 : 8;
      const bool several = block >= (wide_sums ? 768 : 512) && rows >= least * cb_num_sms();
      auto kernel = several ? (res_in ? rmsnorm_fwd_kernel<T, true, IT, R> : rmsnorm_fwd_kernel<T, false, IT, R>)
                            : (res_in ? rmsnorm_fwd_kernel<T, true, IT, 1> : rmsnorm_fwd_kernel<T, false, IT, 1>);
      return cb_launch_early(kernel, several ? (rows + R - 1) / R : rows, block, 0, stream, (const T*)x, (const T*)res_in, (const T*)w, (T*)y,
                             res_in ? (T*)res_out : nullptr, rstd, rows, H, eps);
    });
  });
  return CB_LAUNCH_CHECK();
}

// dw_partial: fp32 [cb_norm_bwd_grid(rows, H, dtype), H] scratch.  dw: T[H]; accumulate!=0 adds into dw.  Both launches begin while what is
// before them ends: 8192 x 4096 with the forward 90.8 -> 87.0 us.
int cb_rmsnorm_bwd(const void* dy, const void* h, const void* w, const float* rstd, const void* dres, void* dx,
                   float* dw_partial, void* dw, int accumulate, int rows, int H, int dtype, cudaStream_t stream) {
  if (rows == 0) return 0;
  const int grid = cb_norm_bwd_grid(rows, H, dtype);
  CB_DISPATCH_FLOAT(dtype, T, {
    const int block = pick_block(H, Vec16<T>::N);
    const int iters = pick_iters(H, Vec16<T>::N, block);
    CB_DISPATCH_ITERS(iters, IT, {
      const int e = dres ? cb_launch_early(rmsnorm_bwd_kernel<T, true, IT>, grid, block, 0, stream, (const T*)dy, (const T*)h, (const T*)w, rstd,
                                           (const T*)dres, (T*)dx, dw_partial, rows, H)
                         : cb_launch_early(rmsnorm_bwd_kernel<T, false, IT>, grid, block, 0, stream, (const T*)dy, (const T*)h, (const T*)w, rstd,
                                           (const T*)nullptr, (T*)dx, dw_partial, rows, H);
      if (e) return e;
    });
    return cb_launch_early(reduce_partials_kernel<T>, (H + 31) / 32, 1024, 0, stream, dw_partial, (T*)dw, grid, H, accumulate);
  });
  return CB_LAUNCH_CHECK();
}

int cb_layernorm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd, int rows, int H,
                     float eps, int dtype, cudaStream_t stream) {
  if (rows == 0) return 0;
  CB_DISPATCH_FLOAT(dtype, T, {
    const int block = pick_block(H, Vec16<T>::N);
    const int iters = pick_iters(H, Vec16<T>::N, block);
    CB_DISPATCH_ITERS(iters, IT, {
      layernorm_fwd_kernel<T, IT><<<rows, block, 0, stream>>>((const T*)x, (const T*)w, (const T*)b, (T*)y, mean,
                                                             rstd, rows, H, eps);
    });
  });
  return CB_LAUNCH_CHECK();
}

int cb_layernorm_bwd(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, void* dx,
                     float* dw_partial, float* db_partial, void* dw, void* db, int accumulate, int rows, int H,
                     int dtype, cudaStream_t stream) {
  if (rows == 0) return 0;
  const int grid = cb_norm_bwd_grid(rows, H, dtype);
  CB_DISPATCH_FLOAT(dtype, T, {
    const int block = pick_block(H, Vec16<T>::N);
    const int iters = pick_iters(H, Vec16<T>::N, block);
    CB_DISPATCH_ITERS(iters, IT, {
      layernorm_bwd_kernel<T, IT><<<grid, block, 0, stream>>>((const T*)dy, (const T*)x, (const T*)w, mean, rstd,
                                                             (T*)dx, dw_partial, db_partial, rows, H);
    });
    reduce_partials_kernel<T><<<(H + 31) / 32, 1024, 0, stream>>>(dw_partial, (T*)dw, grid, H, accumulate);
    if (db) reduce_partials_kernel<T><<<(H + 31) / 32, 1024, 0, stream>>>(db_partial, (T*)db, grid, H, accumulate);
  });
  return CB_LAUNCH_CHECK();
}

}  // extern "C"
