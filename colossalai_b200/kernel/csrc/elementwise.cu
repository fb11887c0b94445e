// Fused elementwise kernels for sm_100a: SwiGLU / GeGLU fwd+bwd on a packed [rows, 2*I] gate|up buffer,
// RoPE of the q and k head ranges of packed QKV rows in one pass (fwd and bwd),
// bias+GELU fwd/bwd, bias+dropout+residual add, scale+inf/nan check.
//
// Capability parity: reference silu_and_mul (extensions/csrc/kernel/cuda/activation_kernel.cu, N16),
// rotary_embedding (fused_rotary_emb_and_cache_kernel.cu, N15), Triton LlamaActCombine
// (kernel/triton/llama_act_combine_kernel.py), TorchScript bias_gelu / bias_dropout_add (kernel/jit/*.py),
// multi_tensor_scale (N7).  All are pure HBM-bandwidth kernels: 16-byte vector I/O, grid-stride, fp32 math.
#include "activations.cuh"
#include "common.cuh"

// Gated unit, forward and backward.  A block takes an equal part of one row, GLU_ITEMS vectors per thread, so that a thread has
// all its loads in flight before its first store and no index needs a 64-bit division; at most 256 threads, and no more than
// the part needs (176 vectors of a 1408 wide expert, 28700 rows: 256 threads 50 us forward, 80 backward; 96 threads 42, 62).
// Bound: HBM.  8192 x 14336 bf16: one vector per thread of a grid-stride loop 118 us forward (6.0 TB/s) and 189 us backward
// (6.2); now 102 (6.9) and 169 (7.0).
// row_limit (device scalar, optional): only the first *row_limit rows hold data - expert-parallel receive buffers are sized
// for the worst case and the number of rows that actually arrived is only known on the device.
// Rows of at most GLU_NARROW vectors share a block: 100000 x 64 bf16: a block per row 53 us in either direction, together 6.4
// and 8.5; 28700 x 1408, 176 vectors, a block per row as above
constexpr int GLU_THREADS = 256;
constexpr int GLU_ITEMS = 2;
constexpr int GLU_NARROW = 128;

struct GluPart {                      // what a thread works on: its row, first column and the threads of the row's part
  int64_t row;
  int c0, lanes;
};
template <int VEC, bool NARROW> CB_DEVICE bool glu_part(GluPart& p, int64_t rows, int blocks_per_row, int rows_per_block, int I,
                                                        const int64_t* row_limit) {
  if (NARROW) {
    p.lanes = (I / VEC + GLU_ITEMS - 1) / GLU_ITEMS;
    const int r = threadIdx.x / p.lanes;
    p.row = (int64_t)blockIdx.x * rows_per_block + r;
    p.c0 = (threadIdx.x - r * p.lanes) * VEC;
    if (r >= rows_per_block || p.row >= rows) return false;
  } else {
    const unsigned r = blockIdx.x / (unsigned)blocks_per_row;
    p.lanes = blockDim.x;
    p.row = r;
    p.c0 = ((blockIdx.x - r * blocks_per_row) * blockDim.x * GLU_ITEMS + threadIdx.x) * VEC;
  }
  return row_limit == nullptr || p.row < *row_limit;
}

template <typename T, int ACT, bool NARROW>
__global__ void __launch_bounds__(GLU_THREADS) glu_fwd_kernel(const T* __restrict__ gu, T* __restrict__ out, int64_t rows,
                                                              int blocks_per_row, int rows_per_block, int I,
                                                              const int64_t* __restrict__ row_limit) {
  constexpr int VEC = Vec16<T>::N;
  cb_early_start();
  GluPart p;
  if (!glu_part<VEC, NARROW>(p, rows, blocks_per_row, rows_per_block, I, row_limit)) return;
  const T* gr = gu + p.row * 2 * I;
  T* o_r = out + p.row * I;
  Vec16<T> g[GLU_ITEMS], u[GLU_ITEMS], o;
#pragma unroll
  for (int k = 0; k < GLU_ITEMS; ++k) {
    const int c = p.c0 + k * p.lanes * VEC;
    if (c < I) { g[k].load_nc(gr + c); u[k].load_nc(gr + I + c); }
  }
#pragma unroll
  for (int k = 0; k < GLU_ITEMS; ++k) {
    const int c = p.c0 + k * p.lanes * VEC;
    if (c < I) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) o.set(i, act_f<ACT>(g[k].get(i)) * u[k].get(i));
      o.store_na(o_r + c);
    }
  }
}

template <typename T, int ACT, bool NARROW>
__global__ void __launch_bounds__(GLU_THREADS) glu_bwd_kernel(const T* __restrict__ dout, const T* __restrict__ gu,
                                                              T* __restrict__ dgu, int64_t rows, int blocks_per_row,
                                                              int rows_per_block, int I, const int64_t* __restrict__ row_limit) {
  constexpr int VEC = Vec16<T>::N;
  GluPart p;
  if (!glu_part<VEC, NARROW>(p, rows, blocks_per_row, rows_per_block, I, row_limit)) return;
  const T* gr = gu + p.row * 2 * I;
  const T* dr = dout + p.row * I;
  T* or_ = dgu + p.row * 2 * I;
  Vec16<T> g[GLU_ITEMS], u[GLU_ITEMS], d[GLU_ITEMS], dg, du;
#pragma unroll
  for (int k = 0; k < GLU_ITEMS; ++k) {
    const int c = p.c0 + k * p.lanes * VEC;
    if (c < I) { g[k].load_nc(gr + c); u[k].load_nc(gr + I + c); d[k].load_nc(dr + c); }
  }
#pragma unroll
  for (int k = 0; k < GLU_ITEMS; ++k) {
    const int c = p.c0 + k * p.lanes * VEC;
    if (c < I) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        const float gf = g[k].get(i), uf = u[k].get(i), df = d[k].get(i);
        dg.set(i, df * uf * act_grad_f<ACT>(gf));
        du.set(i, df * act_f<ACT>(gf));
      }
      dg.store_na(or_ + c);
      du.store_na(or_ + I + c);
    }
  }
}

// RoPE on heads [0, n_rot_heads) of every token row, `dst` row = rotated heads | the rest of the row as it is: row r of src
// starts at r * src_stride elements, of dst at r * width.  Head h starts at h * D; its first rot_dim elements turn.
// cos/sin: fp32 caches [max_pos, rot_dim / 2]; pos: int64 [T].  sign = +1 forward, -1 backward (the inverse rotation).
//
// Bound: HBM, every row is read once and written once.  Rotating in place behind a copy of the rows moved them 1.8 times
// (8192 rows of 6144 bf16: 34.5 us for the copy and 25.5 us for the rotation; now 35.1 us).  A block takes one token, so its cos /
// sin rows come from L1 after the first head; an item is two 16-byte vectors - a pair of rotated ones or two that pass
// through - so that no thread's share differs from another's.  Rows of at most ROPE_NARROW items share a block of ROPE_BLOCK
// threads, one item each: 300000 rows of 48 bf16 forward and
// backward: a block each 313 us, together 38.  A form of its own: with the stride and the row worked out at run time 8192 rows of 6144
// took 40 us a direction instead of 35.  Wide rows of 16 bits in calls of
// several rounds of blocks: ROPE_ITEMS items a thread, all their loads before the first store (8192 rows of 6144: one item, in as many more
// threads, 34.5 us, two 33.0, three 32.7, four 33.2).  In one round of blocks a block more is worth more than what one has on its way, and the narrower
// the row the longer: three / one, us, 384 items 1000 tokens 5.84 / 5.18, 2500 1.5 % slower, 4000 16.9 / 17.6, 12000 44.7 / 49.0; 288 items 3000
// tokens 3 % slower, 4000 3 % faster; 144 items 4000 8.06 / 7.06, 8000 13.8 / 13.7, 30000 4 % faster; 160 items of which 144 are rotated, so that a warp
// has both kinds, 8000 6 % slower, 20000 3 %; 640 items, which a block does not hold one each, 600 4 % faster, 4000 28.3 / 30.7 (fewer: 512 threads).  32 bits: 2 %
// slower up to 384 items at any number of tokens, at 768 1 % faster.
constexpr int ROPE_NARROW = 64, ROPE_BLOCK = 256, ROPE_ITEMS = 3;
// Where a step's keys and values go beside dst (PAGES): rows of kv_width elements of pages of `page` tokens, found through the page tables.
// A decode step then has a launch a layer less; with the gated unit's too (gemm_rows_tcgen05.cu) 16 sequences, 4 layers of 4096 x 14336,
// take 498 us instead of 513, 5 sequences, 2 layers of 1024 x 2816, 81 instead of 85.
template <typename T, bool PAGES> struct RopePages {
  T *k, *v;
  const int *tables, *token_seq, *token_pos;
  int page, table_width, kv_width;     // tokens of a page, entries of a table, elements of a token's keys
  int k_at;                            // first element of the keys in a row; the values follow them
};
template <typename T> struct RopePages<T, false> {};
enum { ROPE_SHARED, ROPE_ONE, ROPE_SEVERAL };             // narrow rows that share a block; of a row with its own, items of a thread
template <typename T, bool VEC_TABLE, int FORM, bool PAGES>
__global__ void __launch_bounds__(FORM == ROPE_SHARED ? ROPE_BLOCK : 512) rope_kernel(const T* __restrict__ src, T* __restrict__ dst,
                                                   const int64_t* __restrict__ pos, const float* __restrict__ cos_c,
                                                   const float* __restrict__ sin_c, int64_t tokens, int per_block,
                                                   int64_t src_stride, int width, int n_rot_heads, int D, int rot_dim,
                                                   float sign, int interleaved, RopePages<T, PAGES> pages) {
  constexpr bool NARROW = FORM == ROPE_SHARED;
  constexpr int VEC = Vec16<T>::N, UN = FORM == ROPE_SEVERAL ? ROPE_ITEMS : 1;
  cb_early_start();
  const int half = rot_dim / 2;
  const int vec_per_head = half / VEC;                       // rotated items of a head
  const int n_rot = n_rot_heads * vec_per_head;
  const int copy_per_head = (D - rot_dim) / VEC;             // vectors of a rotated head that pass through
  const int n_head_copy = n_rot_heads * copy_per_head;
  const int n_copy = n_head_copy + (width - n_rot_heads * D) / VEC;
  const int items = n_rot + (n_copy + 1) / 2;
  const int row = NARROW ? threadIdx.x / items : 0;
  const int64_t t = NARROW ? (int64_t)blockIdx.x * per_block + row : (int64_t)blockIdx.x;
  if (NARROW && (row >= per_block || t >= tokens)) return;
  const T* in = src + t * src_stride;
  T* out = dst + t * width;
  const int64_t p = pos[t];
  int64_t slot = 0;                                          // first element of the token's rows in the pages
  if constexpr (PAGES) {
    const int at = pages.token_pos[t], page = pages.tables[pages.token_seq[t] * pages.table_width + at / pages.page];
    slot = ((int64_t)page * pages.page + at % pages.page) * pages.kv_width;
  }
  auto put = [&](const Vec16<T>& x, int o) {
    x.store_na(out + o);
    if constexpr (PAGES) {
      if (o >= pages.k_at)
        x.store(o < pages.k_at + pages.kv_width ? pages.k + slot + (o - pages.k_at) : pages.v + slot + (o - pages.k_at - pages.kv_width));
    }
  };
  auto copy_at = [&](int c) {
    return c < n_head_copy ? (c / copy_per_head) * D + rot_dim + (c % copy_per_head) * VEC : n_rot_heads * D + (c - n_head_copy) * VEC;
  };
  const int step = NARROW ? items : blockDim.x;
  for (int j0 = threadIdx.x - row * items; j0 < items; j0 += UN * step) {
    Vec16<T> a[UN], b[UN];
    int o0[UN], o1[UN];
#pragma unroll
    for (int k = 0; k < UN; ++k) {
      const int j = j0 + k * step;
      if (j >= items) break;
      if (j >= n_rot) {
        const int c0 = 2 * (j - n_rot);
        o0[k] = copy_at(c0);
        o1[k] = c0 + 1 < n_copy ? copy_at(c0 + 1) : o0[k];
      } else {
        const int h = j / vec_per_head, v = j - h * vec_per_head;
        o0[k] = h * D + (interleaved ? 2 * v * VEC : v * VEC);
        o1[k] = interleaved ? o0[k] + VEC : o0[k] + half;
      }
      a[k].load_nc(in + o0[k]);
      b[k].load_nc(in + o1[k]);
    }
#pragma unroll
    for (int k = 0; k < UN; ++k) {
      const int j = j0 + k * step;
      if (j >= items) break;
      if (j >= n_rot) {
        put(a[k], o0[k]);
        if (o1[k] != o0[k]) put(b[k], o1[k]);
        continue;
      }
      const int v = j % vec_per_head;
      float c[VEC], s[VEC];
      const float* cp = cos_c + p * half + v * VEC;
      const float* sp = sin_c + p * half + v * VEC;
      if (VEC_TABLE) {
#pragma unroll
        for (int i = 0; i < VEC; i += 4) {
          const float4 c4 = __ldg(reinterpret_cast<const float4*>(cp + i)), s4 = __ldg(reinterpret_cast<const float4*>(sp + i));
          c[i] = c4.x; c[i + 1] = c4.y; c[i + 2] = c4.z; c[i + 3] = c4.w;
          s[i] = s4.x; s[i + 1] = s4.y; s[i + 2] = s4.z; s[i + 3] = s4.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < VEC; ++i) { c[i] = __ldg(cp + i); s[i] = __ldg(sp + i); }
      }
      if (!interleaved) {
        Vec16<T> u, w;
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          const float x = a[k].get(i), y = b[k].get(i), sn = s[i] * sign;
          u.set(i, x * c[i] - y * sn);
          w.set(i, y * c[i] + x * sn);
        }
        put(u, o0[k]);
        put(w, o1[k]);
      } else {
        // GPT-J / ChatGLM style: pairs are adjacent elements (2i, 2i + 1); the item's 2 VEC elements hold VEC pairs
#pragma unroll
        for (int i = 0; i < VEC; i += 2) {
          const float ca = c[i / 2], sa = s[i / 2] * sign, cb = c[VEC / 2 + i / 2], sb = s[VEC / 2 + i / 2] * sign;
          const float x = a[k].get(i), y = a[k].get(i + 1), z = b[k].get(i), w = b[k].get(i + 1);
          a[k].set(i, x * ca - y * sa);
          a[k].set(i + 1, y * ca + x * sa);
          b[k].set(i, z * cb - w * sb);
          b[k].set(i + 1, w * cb + z * sb);
        }
        put(a[k], o0[k]);
        put(b[k], o1[k]);
      }
    }
  }
}

template <typename T, int ACT>
__global__ void __launch_bounds__(256) bias_act_fwd_kernel(const T* __restrict__ x, const T* __restrict__ bias,
                                                           T* __restrict__ y, int64_t rows, int H) {
  constexpr int VEC = Vec16<T>::N;
  const int64_t vpr = H / VEC, total = rows * vpr;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(idx % vpr) * VEC;
    Vec16<T> xv, bv, o;
    xv.load_nc(x + idx * VEC);
    if (bias) bv.load(bias + c);
#pragma unroll
    for (int i = 0; i < VEC; ++i) o.set(i, act_f<ACT>(xv.get(i) + (bias ? bv.get(i) : 0.f)));
    o.store_na(y + idx * VEC);
  }
}

template <typename T, int ACT>
__global__ void __launch_bounds__(256) bias_act_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                           const T* __restrict__ bias, T* __restrict__ dx,
                                                           int64_t rows, int H) {
  constexpr int VEC = Vec16<T>::N;
  const int64_t vpr = H / VEC, total = rows * vpr;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(idx % vpr) * VEC;
    Vec16<T> xv, bv, dv, o;
    xv.load_nc(x + idx * VEC);
    dv.load_nc(dy + idx * VEC);
    if (bias) bv.load(bias + c);
#pragma unroll
    for (int i = 0; i < VEC; ++i) o.set(i, dv.get(i) * act_grad_f<ACT>(xv.get(i) + (bias ? bv.get(i) : 0.f)));
    o.store_na(dx + idx * VEC);
  }
}

// out = in * scale ; sets *flag = 1 if any element is inf/nan (loss-scale unscale + overflow check)
template <typename TI, typename TO>
__global__ void __launch_bounds__(256) scale_check_kernel(const TI* __restrict__ in, TO* __restrict__ out,
                                                          int64_t n, float scale, int* __restrict__ flag) {
  bool bad = false;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float v = to_f32<TI>(in[i]);
    if (!isfinite(v)) bad = true;
    out[i] = from_f32<TO>(v * scale);
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) *flag = 1;
}

template <typename T, bool PAGES>
static int launch_rope(const T* src, T* dst, const int64_t* pos, const float* cos_c, const float* sin_c, int64_t tokens, int64_t src_stride,
                       int width, int n_rot_heads, int D, int rot_dim, float sign, int interleaved, const RopePages<T, PAGES>& pages,
                       cudaStream_t s) {
  if (tokens == 0) return 0;
  const bool vec_table = (((uintptr_t)cos_c | (uintptr_t)sin_c) & 15) == 0;
  // (the same count as in the kernel: rotated pairs, and vectors that pass through two by two)
  const int rotated = n_rot_heads * (rot_dim / 2 / Vec16<T>::N), items = rotated + (width / Vec16<T>::N - 2 * rotated + 1) / 2;
  const int per_block = items > 0 && items <= ROPE_NARROW ? ROPE_BLOCK / items : 1;
  const int third = ((items + ROPE_ITEMS - 1) / ROPE_ITEMS + 31) / 32 * 32;
  const int rounds = items > 512 ? 0 : third >= 96 ? 2560 : rotated % 32 == 0 ? 4096 : 8192;
  const bool several = (sizeof(T) == 2 || items > 512) && tokens >= 4 * cb_num_sms() && tokens * third >= (int64_t)rounds * cb_num_sms();
  const int share = several ? third : (items + 31) / 32 * 32;
  const int block = per_block > 1 ? ROPE_BLOCK : share >= 512 ? 512 : share;
  const unsigned grid = (unsigned)((tokens + per_block - 1) / per_block);
  auto kern = per_block > 1 ? (vec_table ? rope_kernel<T, true, ROPE_SHARED, PAGES> : rope_kernel<T, false, ROPE_SHARED, PAGES>)
              : block < items ? (vec_table ? rope_kernel<T, true, ROPE_SEVERAL, PAGES> : rope_kernel<T, false, ROPE_SEVERAL, PAGES>)
                              : (vec_table ? rope_kernel<T, true, ROPE_ONE, PAGES> : rope_kernel<T, false, ROPE_ONE, PAGES>);
  return cb_launch_early(kern, grid, block, 0, s, src, dst, pos, cos_c, sin_c, tokens, per_block, src_stride, width, n_rot_heads, D,
                         rot_dim, sign, interleaved, pages);
}

static inline int ew_grid(int64_t items, int block) {
  int64_t g = (items + block - 1) / block;
  const int64_t cap = (int64_t)cb_num_sms() * 16;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

extern "C" {

#define GLU_LAUNCH(LAUNCH, KERNEL, ...)                                                                                 \
  CB_DISPATCH_FLOAT(dtype, T, {                                                                                         \
    const int vecs = I / Vec16<T>::N, per = GLU_THREADS * GLU_ITEMS, bpr = (vecs + per - 1) / per;                      \
    const int rpb = vecs <= GLU_NARROW ? GLU_THREADS / ((vecs + GLU_ITEMS - 1) / GLU_ITEMS) : 1;                        \
    const int64_t blocks = rpb > 1 ? (rows + rpb - 1) / rpb : rows * bpr;                                               \
    if (blocks > 0x7fffffffll) return (int)cudaErrorInvalidValue;                                                       \
    const int part = (vecs + bpr - 1) / bpr;                                                                            \
    const int block = rpb > 1 ? GLU_THREADS : ((part + GLU_ITEMS - 1) / GLU_ITEMS + 31) / 32 * 32;                      \
    auto kern = rpb > 1 ? (act == 0 ? KERNEL<T, 0, true> : act == 1 ? KERNEL<T, 1, true> : KERNEL<T, 2, true>)            \
                        : (act == 0 ? KERNEL<T, 0, false> : act == 1 ? KERNEL<T, 1, false> : KERNEL<T, 2, false>);        \
    LAUNCH((unsigned)blocks, block, __VA_ARGS__, rows, bpr, rpb, I, row_limit);                                          \
  })

int cb_glu_fwd_bounded(const void* gu, void* out, int64_t rows, int I, int act, int dtype, const int64_t* row_limit, cudaStream_t s) {
  if (rows == 0 || I == 0) return 0;
#define EARLY(GRID, BLOCK, ...) if (const int e = cb_launch_early(kern, GRID, BLOCK, 0, s, __VA_ARGS__)) return e
  GLU_LAUNCH(EARLY, glu_fwd_kernel, (const T*)gu, (T*)out);
#undef EARLY
  return CB_LAUNCH_CHECK();
}

int cb_glu_bwd_bounded(const void* dout, const void* gu, void* dgu, int64_t rows, int I, int act, int dtype,
                       const int64_t* row_limit, cudaStream_t s) {
  if (rows == 0 || I == 0) return 0;
#define PLAIN(GRID, BLOCK, ...) kern<<<GRID, BLOCK, 0, s>>>(__VA_ARGS__)
  GLU_LAUNCH(PLAIN, glu_bwd_kernel, (const T*)dout, (const T*)gu, (T*)dgu);
  return CB_LAUNCH_CHECK();
}
#undef PLAIN
#undef GLU_LAUNCH

int cb_glu_fwd(const void* gu, void* out, int64_t rows, int I, int act, int dtype, cudaStream_t s) {
  return cb_glu_fwd_bounded(gu, out, rows, I, act, dtype, nullptr, s);
}

int cb_glu_bwd(const void* dout, const void* gu, void* dgu, int64_t rows, int I, int act, int dtype, cudaStream_t s) {
  return cb_glu_bwd_bounded(dout, gu, dgu, rows, I, act, dtype, nullptr, s);
}

// src rows and dst rows 16-byte aligned (src_stride, width, D and rot_dim / 2 multiples of a vector's elements)
int cb_rope(const void* src, void* dst, const int64_t* pos, const float* cos_c, const float* sin_c, int64_t tokens,
            int64_t src_stride, int width, int n_rot_heads, int D, int rot_dim, float sign, int interleaved, int dtype,
            cudaStream_t s) {
  CB_DISPATCH_FLOAT(dtype, T, {
    return (launch_rope<T, false>((const T*)src, (T*)dst, pos, cos_c, sin_c, tokens, src_stride, width, n_rot_heads, D, rot_dim, sign,
                                  interleaved, RopePages<T, false>{}, s));
  });
  return CB_LAUNCH_CHECK();
}

// The same of rows q | k | v with kv_heads heads of keys and of values each (n_rot_heads: q and k), 16-bit, forward; keys and values
// also go to their pages: token t to (tables[token_seq[t]][token_pos[t] / page], token_pos[t] % page).  Pages 16-byte aligned.
int cb_rope_pages(const void* src, void* dst, const int64_t* pos, const float* cos_c, const float* sin_c, int64_t tokens,
                  int64_t src_stride, int width, int n_rot_heads, int kv_heads, int D, int rot_dim, int interleaved, int dtype,
                  void* k_pages, void* v_pages, const int* tables, const int* token_seq, const int* token_pos, int page, int table_width,
                  cudaStream_t s) {
  if (width != (n_rot_heads + kv_heads) * D) return (int)cudaErrorInvalidValue;
  CB_DISPATCH_HALF(dtype, T, {
    const RopePages<T, true> pages{(T*)k_pages, (T*)v_pages, tables, token_seq, token_pos, page, table_width, kv_heads * D,
                             (n_rot_heads - kv_heads) * D};
    return (launch_rope<T, true>((const T*)src, (T*)dst, pos, cos_c, sin_c, tokens, src_stride, width, n_rot_heads, D, rot_dim, 1.f,
                                 interleaved, pages, s));
  });
  return CB_LAUNCH_CHECK();
}

int cb_bias_act_fwd(const void* x, const void* bias, void* y, int64_t rows, int H, int act, int dtype,
                    cudaStream_t s) {
  if (rows == 0) return 0;
  CB_DISPATCH_FLOAT(dtype, T, {
    const int g = ew_grid(rows * (H / Vec16<T>::N), 256);
    if (act == 0) bias_act_fwd_kernel<T, 0><<<g, 256, 0, s>>>((const T*)x, (const T*)bias, (T*)y, rows, H);
    else if (act == 1) bias_act_fwd_kernel<T, 1><<<g, 256, 0, s>>>((const T*)x, (const T*)bias, (T*)y, rows, H);
    else if (act == 3) bias_act_fwd_kernel<T, 3><<<g, 256, 0, s>>>((const T*)x, (const T*)bias, (T*)y, rows, H);
    else bias_act_fwd_kernel<T, 2><<<g, 256, 0, s>>>((const T*)x, (const T*)bias, (T*)y, rows, H);
  });
  return CB_LAUNCH_CHECK();
}

int cb_bias_act_bwd(const void* dy, const void* x, const void* bias, void* dx, int64_t rows, int H, int act,
                    int dtype, cudaStream_t s) {
  if (rows == 0) return 0;
  CB_DISPATCH_FLOAT(dtype, T, {
    const int g = ew_grid(rows * (H / Vec16<T>::N), 256);
    if (act == 0) bias_act_bwd_kernel<T, 0><<<g, 256, 0, s>>>((const T*)dy, (const T*)x, (const T*)bias, (T*)dx, rows, H);
    else if (act == 1) bias_act_bwd_kernel<T, 1><<<g, 256, 0, s>>>((const T*)dy, (const T*)x, (const T*)bias, (T*)dx, rows, H);
    else if (act == 3) bias_act_bwd_kernel<T, 3><<<g, 256, 0, s>>>((const T*)dy, (const T*)x, (const T*)bias, (T*)dx, rows, H);
    else bias_act_bwd_kernel<T, 2><<<g, 256, 0, s>>>((const T*)dy, (const T*)x, (const T*)bias, (T*)dx, rows, H);
  });
  return CB_LAUNCH_CHECK();
}

// in dtype -> out dtype with scale; flag (int32 device) set to 1 on inf/nan
int cb_scale_check(const void* in, void* out, int64_t n, float scale, int* flag, int in_dtype, int out_dtype,
                   cudaStream_t s) {
  if (n == 0) return 0;
  const int g = ew_grid(n, 256);
#define SC(TI, TO) scale_check_kernel<TI, TO><<<g, 256, 0, s>>>((const TI*)in, (TO*)out, n, scale, flag)
  if (in_dtype == CB_F32 && out_dtype == CB_F32) SC(float, float);
  else if (in_dtype == CB_BF16 && out_dtype == CB_F32) SC(__nv_bfloat16, float);
  else if (in_dtype == CB_F16 && out_dtype == CB_F32) SC(__half, float);
  else if (in_dtype == CB_F32 && out_dtype == CB_BF16) SC(float, __nv_bfloat16);
  else if (in_dtype == CB_F32 && out_dtype == CB_F16) SC(float, __half);
  else if (in_dtype == CB_BF16 && out_dtype == CB_BF16) SC(__nv_bfloat16, __nv_bfloat16);
  else if (in_dtype == CB_F16 && out_dtype == CB_F16) SC(__half, __half);
  else return (int)cudaErrorInvalidValue;
#undef SC
  return CB_LAUNCH_CHECK();
}

}  // extern "C"
