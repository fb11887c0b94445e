// Host side of the small hot operators in native code: allocation, autograd and launch without the interpreter.
//
// A python autograd function costs 30 us for a forward and 155 us for a forward + backward of a norm whose kernels take 2 and
// 5 us (measured on the host of a B200: stream lookup 3.3 us, argument conversion and launch 9.6 us, three allocations, the
// hand-over of the interpreter to the autograd thread 47 us); every serving call and every training call on a few hundred
// rows was bound by that.  The same functions as C++ autograd functions: norm of 16 rows 35.8 -> 13.7 us a call
// (with the python checks in front), forward + backward of a few rows 143 -> 86 us, most of which is autograd itself.
// The kernels stay behind their C launchers (`bind` takes their addresses); tensors that something watches - tracing,
// functorch, forward-mode, dispatch modes, subclasses - never come here (`ops/_dispatch.py:plain_call`).
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <atomic>
#include <cmath>
#include <map>
#include <string>

using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = c10::optional<Tensor>;

namespace {

int code_of(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return 0;
    case at::kHalf: return 1;
    case at::kBFloat16: return 2;
    default: TORCH_CHECK(false, "unsupported dtype ", t.scalar_type());
  }
}
const void* ptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
void* mut(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
template <typename T> T* mut_as(const Tensor& t) { return reinterpret_cast<T*>(mut(t)); }
template <typename T> const T* as(const Tensor& t) { return reinterpret_cast<const T*>(ptr(t)); }
cudaStream_t stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
// 16-byte loads: a contiguous tensor at an odd offset of its storage is copied
Tensor packed(const Tensor& t) {
  Tensor c = t.contiguous();
  return reinterpret_cast<uintptr_t>(c.const_data_ptr()) % 16 == 0 ? c : c.clone(at::MemoryFormat::Contiguous);
}

// ---- launchers
struct Launchers {
  int (*rmsnorm_fwd)(const void*, const void*, const void*, void*, void*, float*, int, int, float, int, cudaStream_t);
  int (*rmsnorm_bwd)(const void*, const void*, const void*, const float*, const void*, void*, float*, void*, int, int, int, int,
                     cudaStream_t);
  int (*norm_bwd_grid)(int, int, int);
  int (*glu_fwd)(const void*, void*, int64_t, int, int, int, const int64_t*, cudaStream_t);
  int (*glu_bwd)(const void*, const void*, void*, int64_t, int, int, int, const int64_t*, cudaStream_t);
  int (*rope)(const void*, void*, const int64_t*, const float*, const float*, int64_t, int64_t, int, int, int, int, float, int, int,
              cudaStream_t);
  int (*rope_pages)(const void*, void*, const int64_t*, const float*, const float*, int64_t, int64_t, int, int, int, int, int, int, int, void*,
                    void*, const int*, const int*, const int*, int, int, cudaStream_t);
  int (*row_stats)(const void*, const int64_t*, float*, int, int, int, int64_t, int64_t, int, cudaStream_t);
  int (*ce_loss_blocks)(int);
  int (*ce_loss)(const float*, const int64_t*, float*, int64_t*, void*, int, int64_t, int, cudaStream_t);
  int (*softmax_grad)(const void*, const int64_t*, const float*, const float*, const float*, const float*, const int64_t*, void*,
                      int, int, int, int64_t, int64_t, int, cudaStream_t);
  int (*flash_varlen_fwd)(const void*, const void*, const void*, void*, float*, const int*, int, long long, int, int, int, int,
                          float, int, cudaStream_t);
  int (*flash_bwd)(const void*, const void*, const void*, const void*, const void*, const float*, void*, void*, void*, float*,
                   float*, int, int, int, int, int, int, float, int, const int*, long long, cudaStream_t);
  int (*gemm_rows)(const void*, const void*, void*, const void*, int, int, int, int64_t, int64_t, int64_t, int, cudaStream_t);
  int (*gemm_rows_gated)(const void*, const void*, void*, int, int, int, int64_t, int64_t, int, int, cudaStream_t);
  int (*embed_rows)(const int64_t*, const void*, void*, int64_t, int64_t, int64_t, cudaStream_t);
  int (*decode_splits)(int, int, int, int, int, int*);
  int (*decode)(const void*, const void*, const void*, const int*, const int*, void*, float*, float*, int, int, int, int, int, int,
                int, int, float, const float*, int64_t, int64_t, int, int, cudaStream_t);
  int (*moe_sort)(const int64_t*, int64_t, int, int, int, int*, int*, int*, int64_t*, int*, int64_t*, cudaStream_t);
  int (*moe_take)(const void*, const int*, void*, int, int, int, cudaStream_t);
  int (*moe_sum)(const void*, const int*, const float*, void*, int, int, int, int, cudaStream_t);
  int (*moe_sum_bwd)(const void*, const void*, const int*, const float*, void*, float*, int, int, int, int, cudaStream_t);
  int (*grouped)(const void*, const void*, void*, const int*, int, int, int, int, int, int, int, int, cudaStream_t);
  int (*gated)(const void*, const void*, void*, void*, const int*, int, int, int, int, int, int, int, cudaStream_t);
  int (*gated_bwd)(const void*, const void*, const void*, void*, const int*, int, int, int, int, int, int, int, cudaStream_t);
  int (*grouped_wgrad)(const void*, const void*, void*, const int*, int, int, int, int, int, int, int, int, int, cudaStream_t);
} L;

// launches by name since the last `counts`
struct Count {
  const char* name;
  std::atomic<long long> n{0};
};
Count n_norm_fwd{"rmsnorm_fwd"}, n_norm_bwd{"rmsnorm_bwd"}, n_glu_fwd{"glu_fwd"}, n_glu_bwd{"glu_bwd"}, n_rope{"rope"},
    n_stats{"ce_row_stats"}, n_loss{"ce_loss"}, n_grad{"ce_softmax_grad"}, n_flash_fwd{"flash_attn_varlen_fwd"},
    n_flash_bwd{"flash_attn_bwd"}, n_decode{"paged_decode_attention"}, n_rows{"gemm_rows"}, n_embed{"embed_rows"},
    n_sort{"moe_sort"}, n_take{"moe_take_rows"}, n_sum{"moe_sum_rows"}, n_sum_bwd{"moe_sum_rows_bwd"}, n_grouped{"grouped_gemm"},
    n_wgrad{"grouped_gemm_wgrad"};
Count* const COUNTS[] = {&n_norm_fwd, &n_norm_bwd, &n_glu_fwd, &n_glu_bwd, &n_rope, &n_stats, &n_loss, &n_grad, &n_flash_fwd, &n_flash_bwd,
                         &n_decode, &n_rows, &n_embed, &n_sort, &n_take, &n_sum, &n_sum_bwd, &n_grouped, &n_wgrad};

void launched(int rc, Count& c, int n = 1) {
  TORCH_CHECK(rc != cudaErrorLaunchTimeout, c.name, ": a wait inside an earlier attention kernel ran out; what it wrote is not valid (CUDA error ",
              rc, ")");
  TORCH_CHECK(rc == 0, c.name, ": native launcher returned CUDA error ", rc);
  c.n.fetch_add(n, std::memory_order_relaxed);
}

// ------------------------------------------------------------------------------------------------ RMS norm
struct RmsNorm : torch::autograd::Function<RmsNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, double eps, const OptTensor& residual) {
    const c10::cuda::CUDAGuard guard(x.device());
    const bool has_res = residual.has_value() && residual->defined();
    const Tensor x2 = x.contiguous(), r2 = has_res ? residual->contiguous() : Tensor();
    const int H = (int)x2.size(-1), rows = H ? (int)(x2.numel() / H) : 0;
    Tensor y = at::empty_like(x2), h = has_res ? at::empty_like(x2) : x2;
    Tensor rstd = at::empty({rows}, x.options().dtype(at::kFloat));
    launched(L.rmsnorm_fwd(ptr(x2), ptr(r2), ptr(weight), mut(y), has_res ? mut(h) : nullptr, mut_as<float>(rstd), rows, H, (float)eps,
                           code_of(x), stream_of(x)),
             n_norm_fwd);
    ctx->save_for_backward({h, weight, rstd});
    ctx->saved_data["has_res"] = has_res;
    ctx->set_materialize_grads(false);
    return has_res ? variable_list{y, h} : variable_list{y};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &h = saved[0], &weight = saved[1], &rstd = saved[2];
    const bool has_res = ctx->saved_data["has_res"].toBool();
    if (!grads[0].defined() && (!has_res || !grads[1].defined())) return {Tensor(), Tensor(), Tensor(), Tensor()};
    const c10::cuda::CUDAGuard guard(h.device());
    const int H = (int)h.size(-1), rows = H ? (int)(h.numel() / H) : 0;
    const Tensor dy = grads[0].defined() ? grads[0].contiguous() : at::zeros_like(h);
    const Tensor dres = has_res && grads[1].defined() ? grads[1].contiguous() : Tensor();
    Tensor dx = at::empty_like(h), dw = rows ? at::empty_like(weight) : at::zeros_like(weight);
    Tensor partial = at::empty({(int64_t)L.norm_bwd_grid(rows, H, code_of(h)) * H}, rstd.options());
    launched(L.rmsnorm_bwd(ptr(dy), ptr(h), ptr(weight), as<float>(rstd), ptr(dres), mut(dx), mut_as<float>(partial), mut(dw), 0, rows, H,
                           code_of(h), stream_of(h)),
             n_norm_bwd, 2);
    return {dx, dw, Tensor(), has_res ? dx : Tensor()};
  }
};

// ------------------------------------------------------------------------------------------------ gated unit
// valid: int64 [1] on the device, rows to compute, or none
struct Glu : torch::autograd::Function<Glu> {
  static Tensor forward(AutogradContext* ctx, const Tensor& gate_up, int64_t act, const OptTensor& valid) {
    const c10::cuda::CUDAGuard guard(gate_up.device());
    const Tensor gu = gate_up.contiguous();
    const int64_t I = gu.size(-1) / 2, rows = I ? gu.numel() / (2 * I) : 0;
    std::vector<int64_t> shape = gu.sizes().vec();
    shape.back() = I;
    Tensor out = at::empty(shape, gu.options());
    launched(L.glu_fwd(ptr(gu), mut(out), rows, (int)I, (int)act, code_of(gu), valid.has_value() ? as<int64_t>(*valid) : nullptr,
                       stream_of(gu)),
             n_glu_fwd);
    ctx->save_for_backward({gu, valid.has_value() ? *valid : Tensor()});
    ctx->saved_data["act"] = act;
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &gu = saved[0], &valid = saved[1];
    const c10::cuda::CUDAGuard guard(gu.device());
    const int64_t I = gu.size(-1) / 2, rows = I ? gu.numel() / (2 * I) : 0;
    const Tensor d = grads[0].contiguous();
    Tensor dgu = at::empty_like(gu);
    launched(L.glu_bwd(ptr(d), ptr(gu), mut(dgu), rows, (int)I, (int)ctx->saved_data["act"].toInt(), code_of(gu),
                       as<int64_t>(valid), stream_of(gu)),
             n_glu_bwd);
    return {dgu, Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------------------ rotary positions
// a contiguous tensor of x's shape whose rows are x's with the first heads turned; rows that are strided as wholes are read
// where they lie
Tensor rotated(const Tensor& x, const Tensor& pos, const Tensor& cos, const Tensor& sin, int64_t heads, int64_t D, int64_t rot,
               float sign, bool interleaved) {
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t vec = 16 / x.element_size();
  const bool as_is = x.dim() == 2 && x.stride(1) == 1 && x.stride(0) % vec == 0 &&
                     reinterpret_cast<uintptr_t>(x.const_data_ptr()) % 16 == 0;
  const Tensor rows = as_is ? x : packed(x);
  const int64_t T = rows.size(0), width = T ? rows.numel() / T : 0;
  Tensor out = at::empty(x.sizes(), x.options());
  launched(L.rope(ptr(rows), mut(out), as<int64_t>(pos), as<float>(cos), as<float>(sin), T, T ? rows.stride(0) : 0, (int)width,
                  (int)heads, (int)D, (int)rot, sign, interleaved, code_of(x), stream_of(x)),
           n_rope);
  return out;
}

struct Rope : torch::autograd::Function<Rope> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const Tensor& pos, const Tensor& cos, const Tensor& sin,
                        int64_t heads, int64_t D, int64_t rot, bool interleaved) {
    ctx->save_for_backward({pos, cos, sin});
    ctx->saved_data["args"] = std::vector<int64_t>{heads, D, rot, (int64_t)interleaved};
    return rotated(qkv, pos, cos, sin, heads, D, rot, 1.f, interleaved);
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const std::vector<int64_t> a = ctx->saved_data["args"].toIntVector();
    return {rotated(grads[0], s[0], s[1], s[2], a[0], a[1], a[2], -1.f, a[3] != 0), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(),
            Tensor(), Tensor()};
  }
};

// a decode step's rows q | k | v [T, (Hq + 2 Hkv) D], rotated, their keys and values also in the pages [pages, page, Hkv, D] (16-byte
// aligned) that tables int32 [sequences, width] name; rows that are strided as wholes are read where they lie
Tensor rope_pages(const Tensor& x, const Tensor& pos, const Tensor& cos, const Tensor& sin, int64_t Hq, int64_t rot, bool interleaved,
                  const Tensor& k_pages, const Tensor& v_pages, const Tensor& tables, const Tensor& token_seq, const Tensor& token_pos) {
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t Hkv = k_pages.size(2), D = k_pages.size(3), T = x.size(0), width = x.size(1), vec = 16 / x.element_size();
  const Tensor rows = x.stride(1) == 1 && x.stride(0) % vec == 0 && reinterpret_cast<uintptr_t>(x.const_data_ptr()) % 16 == 0 ? x : packed(x);
  Tensor out = at::empty(x.sizes(), x.options());
  launched(L.rope_pages(ptr(rows), mut(out), as<int64_t>(pos), as<float>(cos), as<float>(sin), T, rows.stride(0), (int)width, (int)(Hq + Hkv),
                        (int)Hkv, (int)D, (int)rot, interleaved, code_of(x), mut(k_pages), mut(v_pages), as<int>(tables), as<int>(token_seq),
                        as<int>(token_pos), (int)k_pages.size(1), (int)tables.size(1), stream_of(x)),
           n_rope);
  return out;
}

// ------------------------------------------------------------------------------------------------ cross entropy
// one vocabulary shard: logits [T, V] contiguous, target int64 [T] contiguous
struct CrossEntropy : torch::autograd::Function<CrossEntropy> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& target, int64_t ignore, int64_t start, int64_t valid,
                        bool mean) {
    const c10::cuda::CUDAGuard guard(logits.device());
    const int rows = (int)logits.size(0), V = (int)logits.size(1);
    Tensor stats = at::empty({3, rows}, logits.options().dtype(at::kFloat));
    Tensor loss = at::empty({}, stats.options()), n_valid = at::empty({}, target.options());
    const cudaStream_t s = stream_of(logits);
    launched(L.row_stats(ptr(logits), as<int64_t>(target), mut_as<float>(stats), rows, V, (int)valid, start, ignore, code_of(logits), s),
             n_stats);
    const int blocks = L.ce_loss_blocks(rows);
    const Tensor parts = blocks > 1 ? at::empty({2 * blocks}, stats.options().dtype(at::kDouble)) : Tensor();
    launched(L.ce_loss(as<float>(stats), as<int64_t>(target), mut_as<float>(loss), mut_as<int64_t>(n_valid), mut(parts), rows, ignore,
                       mean, s),
             n_loss, 1 + (blocks > 1));
    ctx->save_for_backward({logits, target, stats, n_valid});
    ctx->saved_data["args"] = std::vector<int64_t>{ignore, start, valid, (int64_t)mean};
    return loss;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &logits = saved[0], &target = saved[1], &stats = saved[2], &n_valid = saved[3];
    const std::vector<int64_t> a = ctx->saved_data["args"].toIntVector();
    const c10::cuda::CUDAGuard guard(logits.device());
    const int rows = (int)logits.size(0), V = (int)logits.size(1);
    const Tensor scale = grads[0].to(at::kFloat).contiguous();
    Tensor g = at::empty_like(logits);
    launched(L.softmax_grad(ptr(logits), as<int64_t>(target), as<float>(stats), as<float>(stats) + rows, nullptr, as<float>(scale),
                            a[3] ? as<int64_t>(n_valid) : nullptr, mut(g), rows, V, (int)a[2], a[1], a[0], code_of(logits),
                            stream_of(logits)),
             n_grad);
    return {g, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------------------ packed attention
// q [T, Hq, D], k / v [T, Hkv, D] contiguous and 16-byte aligned, cu int32 [B + 1] contiguous on the device
struct PackedAttention : torch::autograd::Function<PackedAttention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu, bool causal,
                        double scale) {
    const c10::cuda::CUDAGuard guard(q.device());
    const int64_t T = q.size(0), Hq = q.size(1), D = q.size(2);
    Tensor out = at::empty_like(q), lse = at::empty({T, Hq}, q.options().dtype(at::kFloat));
    launched(L.flash_varlen_fwd(ptr(q), ptr(k), ptr(v), mut(out), mut_as<float>(lse), as<int>(cu), (int)cu.numel() - 1, T, (int)Hq,
                                (int)k.size(1), (int)D, causal, (float)scale, code_of(q), stream_of(q)),
             n_flash_fwd);
    ctx->save_for_backward({q, k, v, out, lse});
    ctx->saved_data["cu"] = cu;              // a program may refill a buffer of boundaries: kept without a version check
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &q = s[0], &k = s[1], &v = s[2], &out = s[3], &lse = s[4];
    const Tensor cu = ctx->saved_data["cu"].toTensor();
    const c10::cuda::CUDAGuard guard(q.device());
    const int64_t T = q.size(0), Hq = q.size(1), D = q.size(2);
    const Tensor dout = packed(grads[0]);
    Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
    Tensor delta = at::empty({T, Hq}, lse.options()), acc = at::empty({T, Hq, D}, lse.options());
    launched(L.flash_bwd(ptr(q), ptr(k), ptr(v), ptr(out), ptr(dout), as<float>(lse), mut(dq), mut(dk), mut(dv), mut_as<float>(delta),
                         mut_as<float>(acc), (int)cu.numel() - 1, 0, (int)Hq, (int)k.size(1), (int)D,
                         ctx->saved_data["causal"].toBool(), (float)ctx->saved_data["scale"].toDouble(), code_of(q), as<int>(cu), T,
                         stream_of(q)),
             n_flash_bwd);
    return {dq, dk, dv, Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------------------ paged decode
// q [n, Hq, D]; caches [pages, page, Hkv, D]; tables int32 [n, width], lens int32 [n]; workspaces: fp32 buffers the caller
// keeps (used when they are large enough), else allocated here
Tensor paged_decode(const Tensor& q, const Tensor& kc, const Tensor& vc, const Tensor& tables, const Tensor& lens, double scale,
                    const OptTensor& slopes, int64_t window, const OptTensor& ws_out, const OptTensor& ws_ml) {
  const c10::cuda::CUDAGuard guard(q.device());
  const int64_t n = q.size(0), Hq = q.size(1), D = q.size(2), page = kc.size(1), Hkv = kc.size(2), width = tables.size(1);
  int part = 0;
  const int64_t splits = L.decode_splits((int)n, (int)Hkv, (int)D, (int)(width * page), (int)window, &part);
  const int64_t rows = n * splits * Hq;
  Tensor o = ws_out.has_value() && ws_out->numel() >= rows * D ? *ws_out : Tensor();
  Tensor ml = ws_ml.has_value() && ws_ml->numel() >= rows * 2 ? *ws_ml : Tensor();
  if (!o.defined() || !ml.defined()) {
    o = at::empty({rows * D}, q.options().dtype(at::kFloat));
    ml = at::empty({rows * 2}, q.options().dtype(at::kFloat));
  }
  const Tensor qc = q.stride(2) == 1 && q.stride(1) == D ? q : q.contiguous();
  Tensor out = at::empty(q.sizes(), q.options());
  const float* sl = slopes.has_value() ? as<float>(*slopes) : nullptr;
  launched(L.decode(ptr(qc), ptr(kc), ptr(vc), as<int>(tables), as<int>(lens), mut(out), mut_as<float>(o), mut_as<float>(ml), (int)n,
                    (int)Hq, (int)Hkv, (int)D, (int)page, (int)width, (int)splits, part, (float)scale, sl, qc.stride(0), out.stride(0),
                    code_of(q), (int)window, stream_of(q)),
           n_decode, 2);
  return out;
}

// ------------------------------------------------------------------------------------------------ a step's projections and lookup
// x [M, K], w [N, K], residual [M, N] or none; the caller has checked types, strides and alignment
Tensor linear_rows(const Tensor& x, const Tensor& w, const OptTensor& residual) {
  const c10::cuda::CUDAGuard guard(x.device());
  const int M = (int)x.size(0), K = (int)x.size(1), N = (int)w.size(0);
  const bool add = residual.has_value() && residual->defined();
  Tensor y = at::empty({M, N}, x.options());
  launched(L.gemm_rows(ptr(x), ptr(w), mut(y), add ? ptr(*residual) : nullptr, M, N, K, x.stride(0), N, add ? residual->stride(0) : 0,
                       code_of(x), stream_of(x)),
           n_rows);
  return y;
}
// x [M, K], w [2 N, K] -> act(x gate^T) (x up^T) [M, N]
Tensor gated_rows(const Tensor& x, const Tensor& w, int64_t act) {
  const c10::cuda::CUDAGuard guard(x.device());
  const int M = (int)x.size(0), K = (int)x.size(1), N = (int)(w.size(0) / 2);
  Tensor y = at::empty({M, N}, x.options());
  launched(L.gemm_rows_gated(ptr(x), ptr(w), mut(y), M, N, K, x.stride(0), N, (int)act, code_of(x), stream_of(x)), n_rows);
  return y;
}
// ids [n] int64, table [entries, H]
Tensor embed_rows(const Tensor& ids, const Tensor& table) {
  const c10::cuda::CUDAGuard guard(ids.device());
  Tensor out = at::empty({ids.size(0), table.size(1)}, table.options());
  launched(L.embed_rows(as<int64_t>(ids), ptr(table), mut(out), ids.size(0), table.size(0), table.size(1) * table.element_size(),
                        stream_of(ids)),
           n_embed);
  return out;
}

// ------------------------------------------------------------------------------------------------ local experts
// The operators of a mixture-of-experts layer (`ops/moe.py`, `moe/grouped_gemm.py`).  As python functions a forward and backward of 64
// tokens took 518 us, nearly all of it here on the host, and a layer of 24576 rows still waited 120 us for it at its two ends.

// topk_idx [T, k] -> slot, src, padded counts, ends, total, as `ops/moe.py:sort_choices` describes them
std::vector<Tensor> sort_choices(const Tensor& topk_idx, int64_t E, int64_t align) {
  const c10::cuda::CUDAGuard guard(topk_idx.device());
  const Tensor idx = topk_idx.reshape({-1}).to(at::kLong).contiguous();
  const int64_t n = idx.numel(), bound = (n + E * (align - 1) + align - 1) / align * align;
  const Tensor work = at::empty({2 * E + n + bound}, idx.options().dtype(at::kInt)), wide = at::empty({E + 1}, idx.options());
  const Tensor counts = work.narrow(0, 0, E), ends = work.narrow(0, E, E), slot = work.narrow(0, 2 * E, n),
               src = work.narrow(0, 2 * E + n, bound), padded = wide.narrow(0, 0, E), total = wide.narrow(0, E, 1);
  launched(L.moe_sort(as<int64_t>(idx), n, (int)E, (int)align, (int)bound, mut_as<int>(counts), mut_as<int>(slot), mut_as<int>(src),
                      mut_as<int64_t>(padded), mut_as<int>(ends), mut_as<int64_t>(total), stream_of(idx)),
           n_sort, 2);
  return {slot, src, padded, ends, total};
}

Tensor sum_rows(const Tensor& rows, const Tensor& slot, const Tensor& w, int64_t T, int64_t k) {
  Tensor out = at::empty({T, rows.size(1)}, rows.options());
  launched(L.moe_sum(ptr(rows), as<int>(slot), as<float>(w), mut(out), (int)T, (int)k, (int)rows.size(1), code_of(rows), stream_of(rows)),
           n_sum);
  return out;
}
// [T, k, H]: every choice's row (zeros for a choice of no expert), differentiable
Tensor pick_rows(const Tensor& rows, const Tensor& slot, int64_t T, int64_t k) {
  const Tensor picked = rows.index_select(0, slot.clamp_min(0).to(at::kLong));
  return at::where(slot.ge(0).unsqueeze(-1), picked, at::zeros_like(picked)).view({T, k, -1});
}

// x [T, H] -> rows [bound, H] grouped by expert; a gradient that is to be differentiated again is made of torch operations
struct TakeRows : torch::autograd::Function<TakeRows> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& slot, const Tensor& src, int64_t k) {
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor xa = packed(x);
    Tensor rows = at::empty({src.numel(), xa.size(1)}, xa.options());
    launched(L.moe_take(ptr(xa), as<int>(src), mut(rows), (int)src.numel(), (int)k, (int)(xa.size(1) * xa.element_size()), stream_of(xa)),
             n_take);
    ctx->save_for_backward({slot});
    ctx->saved_data["shape"] = std::vector<int64_t>{xa.size(0), k};
    return rows;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor slot = ctx->get_saved_variables()[0], &d = grads[0];
    const std::vector<int64_t> s = ctx->saved_data["shape"].toIntVector();
    const c10::cuda::CUDAGuard guard(d.device());
    const Tensor dx = at::GradMode::is_enabled() ? pick_rows(d, slot, s[0], s[1]).to(at::kFloat).sum(1).to(d.scalar_type())
                                                 : sum_rows(packed(d), slot, Tensor(), s[0], s[1]);
    return {dx, Tensor(), Tensor(), Tensor()};
  }
};

// rows [bound, H], weights [T, k] -> out [T, H] = sum_j weights[t, j] rows[slot[t, j]]
struct CombineRows : torch::autograd::Function<CombineRows> {
  static Tensor forward(AutogradContext* ctx, const Tensor& rows, const Tensor& weights, const Tensor& slot, const Tensor& src) {
    const c10::cuda::CUDAGuard guard(rows.device());
    ctx->save_for_backward({rows, weights, slot, src});
    return sum_rows(packed(rows), slot, weights.to(at::kFloat).contiguous(), weights.size(0), weights.size(1));
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &rows = s[0], &weights = s[1], &slot = s[2], &src = s[3];
    const c10::cuda::CUDAGuard guard(rows.device());
    const int64_t T = weights.size(0), k = weights.size(1);
    if (at::GradMode::is_enabled()) {
      const Tensor live = src.ge(0).unsqueeze(-1), choice = src.clamp_min(0).to(at::kLong), dout = grads[0].to(at::kFloat);
      const Tensor g = dout.index_select(0, choice.floor_divide(k));
      const Tensor w = weights.to(at::kFloat).reshape({-1}).index_select(0, choice).unsqueeze(-1);
      const Tensor dw = (pick_rows(rows, slot, T, k).to(at::kFloat) * dout.unsqueeze(1)).sum(-1);
      return {at::where(live, w * g, at::zeros_like(g)).to(rows.scalar_type()), dw.to(weights.scalar_type()), Tensor(), Tensor()};
    }
    const Tensor g = packed(grads[0]), r = packed(rows), w = weights.to(at::kFloat).contiguous();
    Tensor drows = at::empty_like(r), dw = at::zeros_like(w);
    launched(L.moe_sum_bwd(ptr(g), ptr(r), as<int>(src), as<float>(w), mut(drows), mut_as<float>(dw), (int)src.numel(), (int)k,
                           (int)r.size(1), code_of(r), stream_of(r)),
             n_sum_bwd);
    return {drows, dw.to(weights.scalar_type()), Tensor(), Tensor()};
  }
};

// The same product in torch operations, zeros behind the last expert's rows: what gradients that are to be differentiated again are made of
Tensor product_by_expert(const Tensor& x, const Tensor& w, const Tensor& ends) {
  const Tensor host = ends.cpu();
  variable_list parts;
  int64_t from = 0;
  for (int64_t e = 0; e < w.size(0); ++e) {
    const int64_t to = host.const_data_ptr<int>()[e];
    parts.push_back(at::matmul(x.slice(0, from, to), w.select(0, e).t()));
    from = to;
  }
  parts.push_back(at::zeros({x.size(0) - from, w.size(1)}, x.options()));
  return at::cat(parts, 0);
}
// gradients, with a graph of their own, of y for the inputs that want one; `tensors`: as many inputs as forward has tensors
variable_list grads_with_graph(AutogradContext* ctx, const Tensor& y, const Tensor& dy, const variable_list& tensors) {
  variable_list wanted, out(tensors.size());
  for (size_t i = 0; i < tensors.size(); ++i)
    if (ctx->needs_input_grad(i)) wanted.push_back(tensors[i]);
  const variable_list got = torch::autograd::grad({y}, wanted, {dy}, c10::nullopt, true);
  for (size_t i = 0, n = 0; i < tensors.size(); ++i)
    if (ctx->needs_input_grad(i)) out[i] = got[n++];
  return out;
}

// y[rows of e] = x[rows of e] w[e]^T; w [E, N, K] contiguous, N a multiple of 128 (the input gradient's blocks), ends int32 [E]: where
// each expert's rows end, multiples of 16.  The caller has checked types and sizes.
struct GroupedLinear : torch::autograd::Function<GroupedLinear> {
  static Tensor product(const Tensor& x, const Tensor& w, const Tensor& ends, bool transposed) {
    const int64_t N = w.size(transposed ? 1 : 2);
    Tensor y = at::empty({x.size(0), N}, x.options());
    launched(L.grouped(ptr(x), ptr(w), mut(y), as<int>(ends), (int)w.size(0), (int)x.size(0), (int)N, (int)x.size(1), (int)x.stride(0),
                       (int)N, transposed, code_of(x), stream_of(x)),
             n_grouped);
    return y;
  }

  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Tensor& ends) {
    const c10::cuda::CUDAGuard guard(x.device());
    ctx->save_for_backward({x, w, ends});
    return product(x.contiguous(), w, ends, true);
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &w = s[1], &ends = s[2], dy = grads[0].contiguous();
    const c10::cuda::CUDAGuard guard(w.device());
    if (at::GradMode::is_enabled()) {
      const variable_list d = grads_with_graph(ctx, product_by_expert(s[0], w, ends), grads[0], {s[0], w});
      return {d[0], d[1], Tensor()};
    }
    Tensor dx, dw;
    if (ctx->needs_input_grad(0)) dx = product(dy, w, ends, false);
    if (ctx->needs_input_grad(1)) dw = weight_grad(dy, s[0].contiguous(), w, ends);
    return {dx, dw, Tensor()};
  }

  static Tensor weight_grad(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& ends) {
    Tensor dw = at::empty({w.size(0), dy.size(1), x.size(1)}, w.options());
    launched(L.grouped_wgrad(ptr(dy), ptr(x), mut(dw), as<int>(ends), (int)w.size(0), (int)x.size(0), (int)dy.size(1), (int)x.size(1),
                             (int)dy.stride(0), (int)x.stride(0), code_of(x), code_of(w), 0, stream_of(x)),
             n_wgrad);
    return dw;
  }
};

// Both layers of gated experts: x w_up[e]^T, the unit, its result times w_down[e]^T; w_up [E, 2 I, H], w_down [E, H', I], H' a multiple of 128, I of 64
struct GatedExperts : torch::autograd::Function<GatedExperts> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w_up, const Tensor& w_down, const Tensor& ends, int64_t act) {
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor xc = x.contiguous();
    const int64_t R = xc.size(0), I = w_up.size(1) / 2;
    Tensor gu = at::empty({R, 2 * I}, x.options()), unit = at::empty({R, I}, x.options());
    launched(L.gated(ptr(xc), ptr(w_up), mut(gu), mut(unit), as<int>(ends), (int)w_up.size(0), (int)R, (int)I, (int)xc.size(1), (int)xc.stride(0),
                     (int)act, code_of(x), stream_of(x)),
             n_grouped);
    ctx->save_for_backward({x, w_up, w_down, ends, gu, unit});
    ctx->saved_data["act"] = act;
    return GroupedLinear::product(unit, w_down, ends, true);
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &w_up = s[1], &w_down = s[2], &ends = s[3], &gu = s[4], &unit = s[5], dy = grads[0].contiguous();
    const c10::cuda::CUDAGuard guard(gu.device());
    if (at::GradMode::is_enabled()) {
      const int64_t act = ctx->saved_data["act"].toInt();
      const variable_list h = product_by_expert(s[0], w_up, ends).to(at::kFloat).chunk(2, 1);
      const Tensor a = (act == 0 ? at::silu(h[0]) : at::gelu(h[0], act == 1 ? "tanh" : "none")) * h[1];
      const variable_list d = grads_with_graph(ctx, product_by_expert(a.to(unit.scalar_type()), w_down, ends), grads[0], {s[0], w_up, w_down});
      return {d[0], d[1], d[2], Tensor(), Tensor()};
    }
    Tensor dx, d_up, d_down, dgu;
    if (ctx->needs_input_grad(0) || ctx->needs_input_grad(1)) {
      dgu = at::empty_like(gu);
      launched(L.gated_bwd(ptr(dy), ptr(w_down), ptr(gu), mut(dgu), as<int>(ends), (int)w_down.size(0), (int)gu.size(0), (int)unit.size(1),
                           (int)dy.size(1), (int)dy.stride(0), (int)ctx->saved_data["act"].toInt(), code_of(gu), stream_of(gu)),
               n_grouped);
    }
    if (ctx->needs_input_grad(2)) d_down = GroupedLinear::weight_grad(dy, unit, w_down, ends);
    if (ctx->needs_input_grad(0)) dx = GroupedLinear::product(dgu, w_up, ends, false);
    if (ctx->needs_input_grad(1)) d_up = GroupedLinear::weight_grad(dgu, s[0].contiguous(), w_up, ends);
    return {dx, d_up, d_down, Tensor(), Tensor()};
  }
};

template <typename F> void take(const std::map<std::string, uint64_t>& table, const char* name, F& slot) {
  const auto it = table.find(name);
  TORCH_CHECK(it != table.end() && it->second != 0, "launcher ", name, " is missing");
  slot = reinterpret_cast<F>(it->second);
}

void bind(const std::map<std::string, uint64_t>& t) {
  take(t, "cb_rmsnorm_fwd", L.rmsnorm_fwd);
  take(t, "cb_rmsnorm_bwd", L.rmsnorm_bwd);
  take(t, "cb_norm_bwd_grid", L.norm_bwd_grid);
  take(t, "cb_glu_fwd_bounded", L.glu_fwd);
  take(t, "cb_glu_bwd_bounded", L.glu_bwd);
  take(t, "cb_rope", L.rope);
  take(t, "cb_rope_pages", L.rope_pages);
  take(t, "cb_ce_row_stats", L.row_stats);
  take(t, "cb_ce_loss_blocks", L.ce_loss_blocks);
  take(t, "cb_ce_loss", L.ce_loss);
  take(t, "cb_ce_softmax_grad", L.softmax_grad);
  take(t, "cb_flash_attn_varlen_fwd", L.flash_varlen_fwd);
  take(t, "cb_flash_attn_bwd", L.flash_bwd);
  take(t, "cb_gemm_rows", L.gemm_rows);
  take(t, "cb_gemm_rows_gated", L.gemm_rows_gated);
  take(t, "cb_embed_rows", L.embed_rows);
  take(t, "cb_decode_num_splits", L.decode_splits);
  take(t, "cb_paged_decode_attention", L.decode);
  take(t, "cb_moe_sort", L.moe_sort);
  take(t, "cb_moe_take_rows", L.moe_take);
  take(t, "cb_moe_sum_rows", L.moe_sum);
  take(t, "cb_moe_sum_rows_bwd", L.moe_sum_bwd);
  take(t, "cb_grouped_gemm", L.grouped);
  take(t, "cb_grouped_gemm_wgrad", L.grouped_wgrad);
  take(t, "cb_grouped_gemm_gated", L.gated);
  take(t, "cb_grouped_gemm_gated_bwd", L.gated_bwd);
}

std::map<std::string, long long> counts(bool clear) {
  std::map<std::string, long long> r;
  for (Count* c : COUNTS) {
    const long long n = clear ? c->n.exchange(0) : c->n.load();
    if (n) r[c->name] = n;
  }
  return r;
}

}  // namespace

PYBIND11_MODULE(cb200_host, m) {
  using release = py::call_guard<py::gil_scoped_release>;
  m.def("bind", &bind);
  m.def("counts", &counts);
  m.def("rms_norm", [](const Tensor& x, const Tensor& w, double eps) { return RmsNorm::apply(x, w, eps, OptTensor())[0]; }, release());
  m.def("rms_norm_residual",
        [](const Tensor& x, const Tensor& w, double eps, const Tensor& r) {
          const variable_list o = RmsNorm::apply(x, w, eps, OptTensor(r));
          return std::make_tuple(o[0], o[1]);
        },
        release());
  m.def("glu", [](const Tensor& gu, int64_t act) { return Glu::apply(gu, act, OptTensor()); }, release());
  m.def("glu_of_rows", [](const Tensor& gu, int64_t act, const Tensor& valid) { return Glu::apply(gu, act, OptTensor(valid)); }, release());
  m.def("rope",
        [](const Tensor& x, const Tensor& pos, const Tensor& cos, const Tensor& sin, int64_t heads, int64_t D, int64_t rot,
           bool interleaved) { return Rope::apply(x, pos, cos, sin, heads, D, rot, interleaved); },
        release());
  m.def("rope_pages", &rope_pages, release());
  m.def("cross_entropy",
        [](const Tensor& x, const Tensor& t, int64_t ignore, int64_t start, int64_t valid, bool mean) {
          return CrossEntropy::apply(x, t, ignore, start, valid, mean);
        },
        release());
  m.def("packed_attention",
        [](const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu, bool causal, double scale) {
          return PackedAttention::apply(q, k, v, cu, causal, scale);
        },
        release());
  m.def("paged_decode", &paged_decode, release());
  m.def("linear_rows", &linear_rows, release());
  m.def("gated_rows", &gated_rows, release());
  m.def("embed_rows", &embed_rows, release());
  m.def("sort_choices", &sort_choices, release());
  m.def("take_rows", [](const Tensor& x, const Tensor& slot, const Tensor& src, int64_t k) { return TakeRows::apply(x, slot, src, k); },
        release());
  m.def("combine_rows",
        [](const Tensor& rows, const Tensor& weights, const Tensor& slot, const Tensor& src) {
          return CombineRows::apply(rows, weights, slot, src);
        },
        release());
  m.def("gated_experts",
        [](const Tensor& x, const Tensor& w_up, const Tensor& w_down, const Tensor& ends, int64_t act) {
          return GatedExperts::apply(x, w_up, w_down, ends, act);
        },
        release());
  m.def("grouped_linear", [](const Tensor& x, const Tensor& w, const Tensor& ends) { return GroupedLinear::apply(x, w, ends); }, release());
}
