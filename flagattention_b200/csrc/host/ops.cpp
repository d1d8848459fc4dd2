// The operators' usual calls, from the Python call to the launches, without Python in between: checks, allocations,
// argument structs and the autograd nodes.  A small call is bound by its host work (a decode step of one layer spent
// 27 us of it for 8 us of kernels, a training step 150 us for 22), most of that in Python's autograd.Function, argument
// packing and ctypes.
//
// Every function returns None for a call that it does not take: other dtypes, devices, options, transforms (functorch,
// forward mode, tracing, dispatch modes), and everything that is an error.  The caller then goes through the Python form
// of the same operator, which words the errors and holds the general path.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/Context.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <atomic>
#include <climits>
#include <cmath>
#include <cstdio>
#include <stdexcept>

#include "flagattn_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

void check(int status, const char *what) {
  if (status == FA_OK) return;
  char text[256];
  std::snprintf(text, sizeof(text), "%s failed: %s (status %d)", what, fa_status_string(status), status);
  throw std::runtime_error(text);
}

// 0 auto, 1 one_pass, 2 two_kernel: what flash.set_backward_mode() selected
std::atomic<int> g_backward_mode{0};
bool one_pass() {
  const int mode = g_backward_mode.load(std::memory_order_relaxed);
  return mode == 0 ? !at::globalContext().deterministicAlgorithms() : mode == 1;
}

// ---- which tensors and which surroundings are taken ----------------------------------------------------------------
// an ordinary CUDA tensor on the current device: no subclass, wrapper, fake, lazy conjugate or forward-mode tangent
bool plain(const Tensor &t, int device) {
  static const c10::DispatchKeySet usual({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA,
                                          c10::DispatchKey::AutocastCUDA, c10::DispatchKey::ADInplaceOrView});
  return t.defined() && !(t.key_set().raw_repr() & ~usual.raw_repr()) && t.is_cuda() && t.get_device() == device && t.has_storage() &&
         t.layout() == at::kStrided && !t._fw_grad(0).defined();
}
bool usual_surroundings() {
  static const c10::DispatchKeySet modes(
      {c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::PythonDispatcher,
       c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::FuncTorchDynamicLayerBackMode,
       c10::DispatchKey::FuncTorchVmapMode, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
       c10::DispatchKey::Functionalize});
  return !c10::impl::tls_local_dispatch_key_set().included_.has_any(modes) &&
         c10::impl::TorchDispatchModeTLS::stack_len() == 0 && !torch::jit::tracer::isTracing();
}
bool dtype_code(const Tensor &t, int32_t *code) {
  if (t.scalar_type() == at::kHalf) *code = FA_F16;
  else if (t.scalar_type() == at::kBFloat16) *code = FA_BF16;
  else return false;
  return true;
}
bool aligned16(const Tensor &t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }
// the kernels' layout rule: unit inner stride, 16-byte aligned rows (_C.kernel_ready() keeps such a tensor as it is)
bool kernel_ready(const Tensor &t) {
  if (t.dim() != 4 || !aligned16(t)) return false;
  if (t.is_contiguous() && t.size(3) % 8 == 0) return true;
  if (t.stride(3) != 1) return false;
  for (int i = 0; i < 3; ++i)
    if (t.size(i) > 1 && t.stride(i) % 8 != 0) return false;
  return true;
}
bool fits(const Tensor &t) {
  if (t.numel() == 0) return false;
  for (int64_t n : t.sizes())
    if (n > INT_MAX) return false;
  return true;
}
fa_tensor4 tensor4(const Tensor &t) {
  return {t.data_ptr(), t.size(0) > 1 ? t.stride(0) : 0, t.size(1) > 1 ? t.stride(1) : 0, t.size(2) > 1 ? t.stride(2) : 0};
}
void *stream_of(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
int sm_count() { return at::cuda::getCurrentDeviceProperties()->multiProcessorCount; }
Tensor new_like(const Tensor &t) { return at::empty(t.sizes(), t.options(), at::MemoryFormat::Contiguous); }
Tensor ready(const Tensor &t) { return kernel_ready(t) ? t : t.contiguous(); }

fa_flash_shape shape_of(const Tensor &q, const Tensor &k, bool causal, double scale) {
  fa_flash_shape s{};
  dtype_code(q, &s.dtype);
  s.B = (int32_t)q.size(0), s.H = (int32_t)q.size(1), s.Hk = (int32_t)k.size(1);
  s.M = (int32_t)q.size(2), s.N = (int32_t)k.size(2), s.D = (int32_t)q.size(3);
  s.causal = causal, s.sm_scale = (float)scale;
  return s;
}

// ---- flash_attention -----------------------------------------------------------------------------------------------
// the split-KV kernels: split_kv._splitkv_forward()
std::pair<Tensor, Tensor> splitkv_forward(const Tensor &q, const Tensor &k, const Tensor &v, bool causal, double scale,
                                          int64_t splits) {
  const int64_t B = q.size(0), H = q.size(1), M = q.size(2), D = q.size(3), N = k.size(2), tile = 64;
  const int64_t per_split = ((N + tile - 1) / tile + splits - 1) / splits * tile;
  splits = (N + per_split - 1) / per_split;   // (none empty)
  const auto f32 = q.options().dtype(at::kFloat);
  const int64_t rows = B * H * splits * M;
  Tensor parts = at::empty({rows * (D + 1)}, f32), o = new_like(q), lse = at::empty({B, H, M}, f32);
  float *o_part = parts.data_ptr<float>(), *l_part = o_part + rows * D;   // (B, H, splits, M, D) and (B, H, splits, M)
  const fa_flash_shape s = shape_of(q, k, causal, scale);
  const fa_tensor4 tq = tensor4(q), tk = tensor4(k), tv = tensor4(v), to = tensor4(o);
  void *stream = stream_of(q);
  check(fa_splitkv_fwd(&s, &tq, &tk, &tv, (int32_t)splits, (int32_t)per_split, o_part, l_part, stream), "fa_splitkv_fwd");
  check(fa_splitkv_combine(&s, (int32_t)splits, o_part, l_part, &to, lse.data_ptr<float>(), stream), "fa_splitkv_combine");
  return {o, lse};
}

// `few_rows`: the form for calls that split their keys; undefined tensors for a layout that it does not take
std::pair<Tensor, Tensor> flash_forward(const Tensor &q, const Tensor &k, const Tensor &v, bool causal, double scale,
                                        bool few_rows) {
  Tensor o = new_like(q), lse = at::empty({q.size(0), q.size(1), q.size(2)}, q.options().dtype(at::kFloat));
  const fa_flash_shape s = shape_of(q, k, causal, scale);
  const fa_tensor4 tq = tensor4(q), tk = tensor4(k), tv = tensor4(v), to = tensor4(o);
  if (few_rows) {
    const int st = fa_flash_fwd_few_rows(&s, &tq, &tk, &tv, &to, lse.data_ptr<float>(), stream_of(q));
    if (st == FA_ERR_UNSUPPORTED) return {};
    check(st, "fa_flash_fwd_few_rows");
  } else {
    check(fa_flash_fwd(&s, &tq, &tk, &tv, &to, lse.data_ptr<float>(), stream_of(q)), "fa_flash_fwd");
  }
  return {o, lse};
}

// dq, dk, dv: the counterpart of flash._backward()
variable_list flash_backward(const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &o, const Tensor &lse,
                             const Tensor &grad, bool causal, double scale) {
  const c10::cuda::CUDAGuard guard(q.device());
  const Tensor d_o = ready(grad);
  Tensor dk = new_like(k), dv = new_like(v), dq = new_like(q);
  const fa_flash_shape s = shape_of(q, k, causal, scale);
  const fa_tensor4 tq = tensor4(q), tk = tensor4(k), tv = tensor4(v), to = tensor4(o), tdo = tensor4(d_o),
                   tdq = tensor4(dq), tdk = tensor4(dk), tdv = tensor4(dv);
  void *stream = stream_of(q);
  const float *l = lse.data_ptr<float>();
  if (one_pass()) {
    int64_t bytes = fa_flash_bwd_workspace_bytes(&s);
    if (bytes > 0) {
      const auto u8 = q.options().dtype(at::kByte);
      Tensor ws;
      try {
        ws = at::empty({bytes}, u8);
      } catch (const c10::OutOfMemoryError &) {   // without room for shared walks, if that is less
        const int64_t least = fa_flash_bwd_least_workspace_bytes(&s);
        if (least >= bytes) throw;
        ws = at::empty({bytes = least}, u8);
      }
      const int st = fa_flash_bwd(&s, &tq, &tk, &tv, &to, &tdo, l, &tdq, &tdk, &tdv, ws.data_ptr(), bytes, stream);
      if (st != FA_ERR_UNSUPPORTED) {   // a layout the one-pass kernel cannot map goes to the pair below
        check(st, "fa_flash_bwd");
        return {dq, dk, dv};
      }
    }
  }
  Tensor delta = at::empty(lse.sizes(), lse.options());
  float *d = delta.data_ptr<float>();
  check(fa_flash_bwd_delta(&s, &to, &tdo, d, stream), "fa_flash_bwd_delta");
  check(fa_flash_bwd_dkdv(&s, &tq, &tk, &tv, &tdo, l, d, &tdk, &tdv, stream), "fa_flash_bwd_dkdv");
  check(fa_flash_bwd_dq(&s, &tq, &tk, &tv, &tdo, l, d, &tdq, stream), "fa_flash_bwd_dq");
  return {dq, dk, dv};
}

struct FlashAttention : torch::autograd::Function<FlashAttention> {
  // q, k, v (or their copies in the kernels' layout), o and lse: made by the caller, who may find that the call is not
  // for this form
  struct Computed {
    Tensor q, k, v, o, lse;
  };
  static Tensor forward(AutogradContext *ctx, const Tensor &, const Tensor &, const Tensor &, bool causal, double scale,
                        const Computed *c) {
    ctx->save_for_backward({c->q, c->k, c->v, c->o, c->lse});
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return c->o;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const auto t = ctx->get_saved_variables();
    variable_list g = flash_backward(t[0], t[1], t[2], t[3], t[4], grads[0], ctx->saved_data["causal"].toBool(),
                                     ctx->saved_data["scale"].toDouble());
    g.resize(6);
    return g;
  }
};

// paged.coarsen_partition()
int64_t coarsen_partition(int64_t size, int64_t pairs, int64_t context, int64_t sms, int64_t most) {
  while (size < most && (double)(pairs * ((context + 2 * size - 1) / (2 * size))) >= 0.8 * (double)sms) size *= 2;
  return size;
}

// flash._decode_covered()
bool decode_covered(const Tensor &q, const Tensor &k, const Tensor &v, bool causal) {
  const int64_t M = q.size(2), N = k.size(2);
  if (M < 1 || N % 16 != 0 || N == 0 || q.size(1) / k.size(1) * M > 64) return false;
  if (causal && M > 1 && N < M) return false;   // rows that see no key at all
  if (k.strides() != v.strides() || k.stride(3) != 1 || !aligned16(k) || !aligned16(v)) return false;
  const int64_t sl = k.stride(2);
  return sl > 0 && sl % 8 == 0 && k.stride(1) % 8 == 0 && k.stride(0) % (16 * sl) == 0;
}

// flash._decode_forward() for one query a head
Tensor decode_forward(const Tensor &q, const Tensor &k, const Tensor &v, double scale) {
  const int64_t B = q.size(0), H = q.size(1), D = q.size(3), Hk = k.size(1), N = k.size(2);
  const int64_t sb = k.stride(0), sl = k.stride(2);
  int64_t partition = coarsen_partition(256, B * Hk, N, sm_count(), 4096);
  if (N <= partition) partition = 0;
  Tensor rows, o = new_like(q), ws;
  int64_t row_stride = q.stride(1), seq_stride = q.stride(0);
  if (row_stride % 8 || seq_stride % 8) rows = q.contiguous(), row_stride = D, seq_stride = H * D;   // of a size of one
  fa_paged_args a{};
  dtype_code(q, &a.dtype);
  a.num_seqs = (int32_t)B, a.num_q_heads = (int32_t)H, a.num_kv_heads = (int32_t)Hk, a.head_size = (int32_t)D;
  a.block_size = 16, a.max_context_len = (int32_t)N, a.block_table_is_i64 = FA_BLOCK_TABLE_IN_PLACE;
  a.partition_size = (int32_t)partition, a.attn_scale = (float)scale;
  a.query = (rows.defined() ? rows : q).data_ptr(), a.q_stride_s = seq_stride, a.q_stride_h = row_stride;
  a.key_cache = k.data_ptr(), a.value_cache = v.data_ptr();
  a.kv_stride_b = 16 * sl, a.kv_stride_h = Hk > 1 ? k.stride(1) : 0, a.kv_stride_t = sl;
  a.bt_stride_s = sb / (16 * sl);
  a.out = o.data_ptr(), a.o_stride_s = H * D, a.o_stride_h = D;
  if (partition) {
    const int64_t n = B * H, P = (N + partition - 1) / partition, stats = (n * P + 63) / 64 * 64;
    ws = at::empty({n * P * D + 2 * stats}, q.options().dtype(at::kFloat));
    a.part_out = ws.data_ptr<float>();
    a.part_max = a.part_out + n * P * D;
    a.part_sum = a.part_max + stats;
  }
  void *stream = stream_of(q);
  check(fa_paged_decode(&a, stream), "fa_paged_decode");
  if (partition) check(fa_paged_reduce(&a, stream), "fa_paged_reduce");
  return o;
}

bool head_dim_built(int64_t D) { return D == 16 || D == 32 || D == 64 || D == 128; }

// o, or an undefined tensor.  `rest`: the calls that the usual form leaves, since their views need a copy or their few
// queries are for the split-KV kernels.  `few`: set, with no o, for a step of 2 to 16 queries a head that the decode kernels
// take: flash._decode_forward() launches those.  (Refused calls pay for both forms: a view or a split call took 58 us where the Python
// form alone takes 38 and this one 12.)
Tensor flash(const Tensor &q_in, const Tensor &k_in, const Tensor &v_in, bool causal, bool default_scale, double scale,
             bool rest, bool *few) {
  *few = false;
  if (!q_in.is_cuda() || !usual_surroundings()) return {};
  const int device = c10::cuda::current_device();
  if (!plain(q_in, device) || !plain(k_in, device) || !plain(v_in, device)) return {};
  if (q_in.dim() != 4 || k_in.dim() != 4 || k_in.sizes() != v_in.sizes() || !fits(q_in) || !fits(k_in)) return {};
  int32_t code;
  if (!dtype_code(q_in, &code) || q_in.scalar_type() != k_in.scalar_type() || q_in.scalar_type() != v_in.scalar_type())
    return {};
  const int64_t B = q_in.size(0), H = q_in.size(1), M = q_in.size(2), D = q_in.size(3), Hk = k_in.size(1), N = k_in.size(2);
  if (!head_dim_built(D) || k_in.size(3) != D || k_in.size(0) != B || H % Hk != 0) return {};
  Tensor copies[3];
  const bool copy = !kernel_ready(q_in) || !kernel_ready(k_in) || !kernel_ready(v_in);
  if (copy) {
    if (!rest) return {};
    at::AutoGradMode no_graph(false);
    copies[0] = ready(q_in), copies[1] = ready(k_in), copies[2] = ready(v_in);
    for (const Tensor &t : copies)
      if (!kernel_ready(t)) return {};
  }
  const Tensor &q = copy ? copies[0] : q_in, &k = copy ? copies[1] : k_in, &v = copy ? copies[2] : v_in;
  if (default_scale) scale = 1.0 / std::sqrt((double)D);
  const bool grads = q_in.requires_grad() || k_in.requires_grad() || v_in.requires_grad();
  const int64_t splits =
      fa_num_splits_heuristic((int32_t)B, (int32_t)H, (int32_t)M, (int32_t)N, 16, 128, sm_count(), 128);
  if (M <= 16 && !grads && (M == 1 || splits > 1) && decode_covered(q, k, v, causal)) {
    *few = M > 1;
    return *few ? Tensor() : decode_forward(q, k, v, scale);
  }
  bool clusters = false;
  if (splits > 1) {
    const fa_flash_shape s = shape_of(q, k, causal, scale);
    clusters = fa_flash_few_rows_pays(&s, sm_count());
  }
  std::pair<Tensor, Tensor> out;
  {
    at::AutoGradMode no_graph(false);
    if (splits <= 1 || clusters) out = flash_forward(q, k, v, causal, scale, splits > 1);
    if (!out.first.defined() && (rest || M >= 32)) out = splitkv_forward(q, k, v, causal, scale, splits);
  }
  if (!out.first.defined() || !grads || !at::GradMode::is_enabled()) return out.first;
  const FlashAttention::Computed c{q, k, v, out.first, out.second};
  return FlashAttention::apply(q_in, k_in, v_in, causal, scale, &c);
}

// ---- piecewise_attention -------------------------------------------------------------------------------------------
std::pair<Tensor, Tensor> piecewise_forward(const Tensor &q1, const Tensor &k1, const Tensor &q2, const Tensor &k2,
                                            const Tensor &v, int64_t w, bool causal, double scale) {
  Tensor o = new_like(q1), lse = at::empty({q1.size(0), q1.size(1), q1.size(2)}, q1.options().dtype(at::kFloat));
  const fa_flash_shape s = shape_of(q1, k1, causal, scale);
  const fa_tensor4 tq1 = tensor4(q1), tk1 = tensor4(k1), tq2 = tensor4(q2), tk2 = tensor4(k2), tv = tensor4(v),
                   to = tensor4(o);
  check(fa_piecewise_fwd(&s, (int32_t)w, &tq1, &tk1, &tq2, &tk2, &tv, &to, lse.data_ptr<float>(), stream_of(q1)),
        "fa_piecewise_fwd");
  return {o, lse};
}

struct PiecewiseAttention : torch::autograd::Function<PiecewiseAttention> {
  // x: q1, k1, q2, k2, v, or their copies in the kernels' layout
  static Tensor forward(AutogradContext *ctx, const Tensor &, const Tensor &, const Tensor &, const Tensor &, const Tensor &,
                        int64_t w, bool causal, double scale, const Tensor *x) {
    auto out = piecewise_forward(x[0], x[1], x[2], x[3], x[4], w, causal, scale);
    ctx->save_for_backward({x[0], x[1], x[2], x[3], x[4], out.first, out.second});
    ctx->saved_data["w"] = w;
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return out.first;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const auto t = ctx->get_saved_variables();
    const Tensor &q1 = t[0], &k1 = t[1], &q2 = t[2], &k2 = t[3], &v = t[4], &o = t[5], &lse = t[6];
    const int32_t w = (int32_t)ctx->saved_data["w"].toInt();
    const c10::cuda::CUDAGuard guard(q1.device());
    const Tensor d_o = ready(grads[0]);
    Tensor delta = at::empty(lse.sizes(), lse.options());
    Tensor dk1 = new_like(k1), dk2 = new_like(k2), dv = new_like(v), dq1 = new_like(q1), dq2 = new_like(q2);
    const fa_flash_shape s =
        shape_of(q1, k1, ctx->saved_data["causal"].toBool(), ctx->saved_data["scale"].toDouble());
    const fa_tensor4 tq1 = tensor4(q1), tk1 = tensor4(k1), tq2 = tensor4(q2), tk2 = tensor4(k2), tv = tensor4(v),
                     to = tensor4(o), tdo = tensor4(d_o), tdq1 = tensor4(dq1), tdq2 = tensor4(dq2), tdk1 = tensor4(dk1),
                     tdk2 = tensor4(dk2), tdv = tensor4(dv);
    void *stream = stream_of(q1);
    const float *l = lse.data_ptr<float>();
    float *d = delta.data_ptr<float>();
    const variable_list out{dq1, dk1, dq2, dk2, dv, Tensor(), Tensor(), Tensor(), Tensor()};
    check(fa_flash_bwd_delta(&s, &to, &tdo, d, stream), "fa_flash_bwd_delta");
    if (one_pass()) {
      const int64_t bytes = fa_piecewise_bwd_fused_workspace_bytes(&s);
      if (bytes > 0) {
        Tensor ws = at::empty({bytes}, q1.options().dtype(at::kByte));
        const int st = fa_piecewise_bwd_fused(&s, w, &tq1, &tk1, &tq2, &tk2, &tv, &tdo, l, d, &tdq1, &tdq2, &tdk1, &tdk2,
                                              &tdv, ws.data_ptr(), bytes, stream);
        if (st != FA_ERR_UNSUPPORTED) {
          check(st, "fa_piecewise_bwd_fused");
          return out;
        }
      }
    }
    check(fa_piecewise_bwd_dkdv(&s, w, &tq1, &tk1, &tq2, &tk2, &tv, &tdo, l, d, &tdk1, &tdk2, &tdv, stream),
          "fa_piecewise_bwd_dkdv");
    check(fa_piecewise_bwd_dq(&s, w, &tq1, &tk1, &tq2, &tk2, &tv, &tdo, l, d, &tdq1, &tdq2, stream), "fa_piecewise_bwd_dq");
    return out;
  }
};

Tensor piecewise(const Tensor &q1, const Tensor &k1, const Tensor &q2, const Tensor &k2, const Tensor &v, int64_t w,
                 bool causal, bool default_scale, double scale) {
  if (!q1.is_cuda() || !usual_surroundings()) return {};
  const int device = c10::cuda::current_device();
  int32_t code;
  bool grads = false;
  for (const Tensor *t : {&q1, &k1, &q2, &k2, &v}) {
    if (!plain(*t, device) || t->dim() != 4 || !fits(*t) || t->scalar_type() != q1.scalar_type()) return {};
    grads = grads || t->requires_grad();
  }
  if (!dtype_code(q1, &code) || w < INT_MIN || w > INT_MAX) return {};
  if (q1.sizes() != q2.sizes() || k1.sizes() != k2.sizes() || k1.sizes() != v.sizes()) return {};
  if (!head_dim_built(q1.size(3)) || k1.size(3) != q1.size(3) || k1.size(1) != q1.size(1) || k1.size(0) != q1.size(0))
    return {};
  if (default_scale) scale = 1.0 / std::sqrt((double)q1.size(3));
  Tensor x[5];
  {
    at::AutoGradMode no_graph(false);
    int i = 0;
    for (const Tensor *t : {&q1, &k1, &q2, &k2, &v}) {
      x[i] = ready(*t);
      if (!kernel_ready(x[i++])) return {};
    }
  }
  if (!grads || !at::GradMode::is_enabled()) return piecewise_forward(x[0], x[1], x[2], x[3], x[4], w, causal, scale).first;
  return PiecewiseAttention::apply(q1, k1, q2, k2, v, w, causal, scale, static_cast<const Tensor *>(x));
}

// ---- rotary_pair (no positions) ------------------------------------------------------------------------------------
struct RotaryPair : torch::autograd::Function<RotaryPair> {
  static variable_list forward(AutogradContext *ctx, const Tensor &x, const Tensor &cos1, const Tensor &sin1,
                               const Tensor &cos2, const Tensor &sin2, bool interleaved) {
    Tensor out1 = at::empty_like(x), out2 = at::empty_like(x);
    const fa_tensor4 tx = tensor4(x), t1 = tensor4(out1), t2 = tensor4(out2);
    int32_t code = 0;
    dtype_code(x, &code);
    check(fa_rotary_pair_fwd(code, (int32_t)x.size(0), (int32_t)x.size(1), (int32_t)x.size(2), (int32_t)x.size(3),
                             interleaved, &tx, cos1.data_ptr<float>(), sin1.data_ptr<float>(), cos2.data_ptr<float>(),
                             sin2.data_ptr<float>(), cos1.stride(0), (int32_t)cos1.size(0), nullptr, 0, &t1, &t2,
                             stream_of(x)),
          "fa_rotary_pair_fwd");
    ctx->save_for_backward({cos1, sin1, cos2, sin2});
    ctx->saved_data["interleaved"] = interleaved;
    return {out1, out2};
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const auto t = ctx->get_saved_variables();
    const c10::cuda::CUDAGuard guard(t[0].device());
    const Tensor g1 = ready(grads[0]), g2 = ready(grads[1]);
    Tensor dx = at::empty_like(g1);
    const fa_tensor4 t1 = tensor4(g1), t2 = tensor4(g2), tdx = tensor4(dx);
    int32_t code = 0;
    dtype_code(g1, &code);
    check(fa_rotary_pair_bwd(code, (int32_t)g1.size(0), (int32_t)g1.size(1), (int32_t)g1.size(2), (int32_t)g1.size(3),
                             ctx->saved_data["interleaved"].toBool(), &t1, &t2, t[0].data_ptr<float>(),
                             t[1].data_ptr<float>(), t[2].data_ptr<float>(), t[3].data_ptr<float>(), t[0].stride(0),
                             (int32_t)t[0].size(0), nullptr, 0, &tdx, stream_of(g1)),
          "fa_rotary_pair_bwd");
    return {dx, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

variable_list rotary_pair(const Tensor &x, const Tensor &cos1, const Tensor &sin1, const Tensor &cos2, const Tensor &sin2,
                          bool interleaved) {
  if (!x.is_cuda() || !usual_surroundings()) return {};
  const int device = c10::cuda::current_device();
  int32_t code;
  if (!plain(x, device) || !kernel_ready(x) || !fits(x) || !dtype_code(x, &code)) return {};
  const int64_t D = x.size(3);
  if (D % 16 != 0 || D > 512) return {};
  for (const Tensor *t : {&cos1, &sin1, &cos2, &sin2})
    if (!plain(*t, device) || t->scalar_type() != at::kFloat || t->dim() != 2 || !fits(*t) ||
        t->size(0) != cos1.size(0) || t->size(1) < D / 2 || t->stride(1) != 1 || t->stride(0) != cos1.stride(0) ||
        t->stride(0) % 4 != 0 || !aligned16(*t) || t->requires_grad())
      return {};
  return RotaryPair::apply(x, cos1, sin1, cos2, sin2, interleaved);
}

// ---- paged_attention, reshape_and_cache ------------------------------------------------------------------------------
// what both ask of a pair of caches [blocks, kv heads, block, head] beside the query's or the new tokens' dtype
bool caches_ready(const Tensor &kc, const Tensor &vc, const Tensor &like, int device) {
  if (!plain(kc, device) || !plain(vc, device) || kc.dim() != 4 || kc.sizes() != vc.sizes() ||
      kc.strides() != vc.strides() || !fits(kc) || kc.scalar_type() != like.scalar_type() ||
      vc.scalar_type() != like.scalar_type() || kc.stride(3) != 1)
    return false;
  return kc.stride(0) % 8 == 0 && kc.stride(1) % 8 == 0 && kc.stride(2) % 8 == 0;
}

// 32 or 64 bit integers
bool integers(const Tensor &t) { return t.scalar_type() == at::kInt || t.scalar_type() == at::kLong; }
// unit inner stride, 16-byte aligned rows
bool rows_ready(const Tensor &t) {
  return t.stride(2) == 1 && aligned16(t) && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0;
}

Tensor paged(const Tensor &query, const Tensor &kc, const Tensor &vc, const Tensor &lens, const Tensor &table,
             double scale, int64_t most, int64_t partition, const uintptr_t (&parts)[3], const int64_t (&sizing)[4]) {
  if (!query.is_cuda() || !usual_surroundings()) return {};
  const int device = c10::cuda::current_device();
  int32_t code;
  if (!plain(query, device) || query.dim() != 3 || !fits(query) || !dtype_code(query, &code) ||
      !caches_ready(kc, vc, query, device))
    return {};
  const int64_t seqs = query.size(0), H = query.size(1), D = query.size(2), Hk = kc.size(1), block = kc.size(2);
  if (kc.size(3) != D || H % Hk != 0 || (H != Hk && block < 16)) return {};
  if (D != 16 && D != 32 && D != 64 && D != 128 && D != 256) return {};
  if (!plain(lens, device) || !integers(lens) || !plain(table, device) || table.dim() != 2 || !integers(table)) return {};
  const bool table_ready = table.stride(1) == 1 || table.size(1) <= 1;
  if (!rows_ready(query) || lens.scalar_type() != at::kInt || !lens.is_contiguous() || !table_ready) {
    if (!rows_ready(query) && query.is_contiguous()) return {};   // off the alignment
    at::AutoGradMode no_graph(false);
    return paged(rows_ready(query) ? query : query.contiguous(), kc, vc, lens.to(at::kInt).contiguous(),
                 table_ready ? table : table.contiguous(), scale, most, partition, parts, sizing);
  }
  if (most > INT_MAX || (partition && (partition < block || partition % block || partition % 16))) return {};
  Tensor out = new_like(query);
  fa_paged_args a{};
  a.dtype = code;
  a.num_seqs = (int32_t)seqs, a.num_q_heads = (int32_t)H, a.num_kv_heads = (int32_t)Hk, a.head_size = (int32_t)D;
  a.block_size = (int32_t)block, a.max_context_len = (int32_t)most;
  a.block_table_is_i64 = table.scalar_type() == at::kLong, a.partition_size = (int32_t)partition;
  a.attn_scale = (float)scale;
  a.query = query.data_ptr(), a.q_stride_s = query.stride(0), a.q_stride_h = query.stride(1);
  a.key_cache = kc.data_ptr(), a.value_cache = vc.data_ptr();
  a.kv_stride_b = kc.stride(0), a.kv_stride_h = kc.stride(1), a.kv_stride_t = kc.stride(2);
  a.context_lens = lens.data_ptr<int32_t>(), a.block_tables = table.data_ptr(), a.bt_stride_s = table.stride(0);
  a.out = out.data_ptr(), a.o_stride_s = out.stride(0), a.o_stride_h = out.stride(1);
  a.part_out = reinterpret_cast<float *>(parts[0]), a.part_max = reinterpret_cast<float *>(parts[1]);
  a.part_sum = reinterpret_cast<float *>(parts[2]);
  void *stream = stream_of(query);
  if (partition && sizing[0]) {
    check(fa_paged_attention(&a, (int32_t)sizing[0], (int32_t)sizing[1], (int32_t)sizing[2], (int32_t)sizing[3], stream),
          "fa_paged_attention");
  } else {
    check(fa_paged_decode(&a, stream), "fa_paged_decode");
    if (partition) check(fa_paged_reduce(&a, stream), "fa_paged_reduce");
  }
  return out;
}

bool append(const Tensor &key, const Tensor &value, const Tensor &kc, const Tensor &vc, const Tensor &slots) {
  if (!key.is_cuda() || !usual_surroundings()) return false;
  const int device = c10::cuda::current_device();
  int32_t code;
  if (!plain(key, device) || !plain(value, device) || key.dim() != 3 || !fits(key) ||
      !dtype_code(key, &code) || value.scalar_type() != key.scalar_type() || !caches_ready(kc, vc, key, device))
    return false;
  if (value.sizes() != key.sizes() || kc.size(1) != key.size(1) || kc.size(3) != key.size(2)) return false;
  if (!plain(slots, device) || !integers(slots) || slots.numel() != key.size(0)) return false;
  if (slots.scalar_type() != at::kLong || !slots.is_contiguous())
    return append(key, value, kc, vc, slots.to(at::kLong).contiguous());
  if (value.strides() != key.strides() || !rows_ready(key) || !rows_ready(value)) {
    if (key.is_contiguous() && value.is_contiguous()) return false;   // off the alignment
    at::AutoGradMode no_graph(false);
    return append(key.contiguous(), value.contiguous(), kc, vc, slots);
  }
  check(fa_paged_cache_append(code, (int32_t)key.size(0), (int32_t)key.size(1), (int32_t)key.size(2), (int32_t)kc.size(2),
                              key.data_ptr(), value.data_ptr(), key.stride(0), key.stride(1), kc.data_ptr(),
                              vc.data_ptr(), kc.stride(0), kc.stride(1), kc.stride(2), slots.data_ptr<int64_t>(),
                              stream_of(key)),
        "fa_paged_cache_append");
  return true;
}

// ---- Python ----------------------------------------------------------------------------------------------------------
// Arguments that are not what the fast form takes (a missing tensor, a float where a count is due) are not errors here:
// the Python form says what is wrong with them.
bool tensors(PyObject *const *args, int n, const Tensor **out) {
  for (int i = 0; i < n; ++i) {
    if (!THPVariable_CheckExact(args[i]) && Py_TYPE(args[i]) != (PyTypeObject *)ParameterClass) return false;
    out[i] = &THPVariable_Unpack(args[i]);
  }
  return true;
}
bool integer(PyObject *o, int64_t *out) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  *out = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}
// a float, an int, or None for the default
bool scale_of(PyObject *o, bool *is_default, double *out) {
  *is_default = o == Py_None;
  if (*is_default) return true;
  if (PyFloat_CheckExact(o)) {
    *out = PyFloat_AS_DOUBLE(o);
    return true;
  }
  int64_t i;
  if (!integer(o, &i)) return false;
  *out = (double)i;
  return true;
}
bool truth(PyObject *o, bool *out) {
  if (!PyBool_Check(o)) return false;
  *out = o == Py_True;
  return true;
}
PyObject *wrap_or_none(const Tensor &t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}

template <bool REST>
PyObject *py_flash(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *t[3];
  bool causal, is_default;
  double scale = 0;
  if (n != 5 || !tensors(args, 3, t) || !truth(args[3], &causal) || !scale_of(args[4], &is_default, &scale)) Py_RETURN_NONE;
  Tensor o;
  bool few;
  {
    pybind11::gil_scoped_release release;
    o = flash(*t[0], *t[1], *t[2], causal, is_default, scale, REST, &few);
  }
  if (few) Py_RETURN_FALSE;
  return wrap_or_none(o);
  END_HANDLE_TH_ERRORS
}

PyObject *py_piecewise(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *t[5];
  bool causal, is_default;
  int64_t w;
  double scale = 0;
  if (n != 8 || !tensors(args, 5, t) || !integer(args[5], &w) || !truth(args[6], &causal) ||
      !scale_of(args[7], &is_default, &scale))
    Py_RETURN_NONE;
  Tensor o;
  {
    pybind11::gil_scoped_release release;
    o = piecewise(*t[0], *t[1], *t[2], *t[3], *t[4], w, causal, is_default, scale);
  }
  return wrap_or_none(o);
  END_HANDLE_TH_ERRORS
}

PyObject *py_rotary_pair(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *t[5];
  bool interleaved;
  if (n != 6 || !tensors(args, 5, t) || !truth(args[5], &interleaved)) Py_RETURN_NONE;
  variable_list out;
  {
    pybind11::gil_scoped_release release;
    out = rotary_pair(*t[0], *t[1], *t[2], *t[3], *t[4], interleaved);
  }
  if (out.empty()) Py_RETURN_NONE;
  PyObject *pair = PyTuple_New(2);
  if (!pair) return nullptr;
  PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(out[0]));
  PyTuple_SET_ITEM(pair, 1, THPVariable_Wrap(out[1]));
  return pair;
  END_HANDLE_TH_ERRORS
}

// (query, key_cache, value_cache, context_lens, block_tables, scale, max_context_len, partition, part_out, part_max,
// part_sum, finest, coarsest, ctas, parts): the last four 0 for partitions of `partition` tokens throughout
PyObject *py_paged(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *t[5];
  bool is_default;
  double scale = 0;
  int64_t x[9];
  if (n != 15 || !tensors(args, 5, t) || !scale_of(args[5], &is_default, &scale) || is_default) Py_RETURN_NONE;
  for (int i = 0; i < 9; ++i)
    if (!integer(args[6 + i], &x[i])) Py_RETURN_NONE;
  Tensor o;
  {
    pybind11::gil_scoped_release release;
    o = paged(*t[0], *t[1], *t[2], *t[3], *t[4], scale, x[0], x[1],
              {(uintptr_t)x[2], (uintptr_t)x[3], (uintptr_t)x[4]}, {x[5], x[6], x[7], x[8]});
  }
  return wrap_or_none(o);
  END_HANDLE_TH_ERRORS
}

PyObject *py_append(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *t[5];
  if (n != 5 || !tensors(args, 5, t)) Py_RETURN_FALSE;
  bool done;
  {
    pybind11::gil_scoped_release release;
    done = append(*t[0], *t[1], *t[2], *t[3], *t[4]);
  }
  return PyBool_FromLong(done);
  END_HANDLE_TH_ERRORS
}

PyObject *py_backward_mode(PyObject *, PyObject *mode) {
  const long m = PyLong_AsLong(mode);
  if (m == -1 && PyErr_Occurred()) return nullptr;
  g_backward_mode.store((int)m, std::memory_order_relaxed);
  Py_RETURN_NONE;
}

PyObject *py_coarsen(PyObject *, PyObject *const *args, Py_ssize_t n) {
  int64_t x[5];
  for (int i = 0; i < 5; ++i)
    if (n != 5 || !integer(args[i], &x[i])) {
      PyErr_SetString(PyExc_TypeError, "five integers");
      return nullptr;
    }
  return PyLong_FromLongLong(coarsen_partition(x[0], x[1], x[2], x[3], x[4]));
}

// (tensor): whether the kernels take it without a copy; (q, k, v, causal): the decode rule.  For comparison with the
// Python form of the rules, on any device.
PyObject *py_kernel_ready(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *t[1];
  if (n != 1 || !tensors(args, 1, t)) Py_RETURN_NONE;
  return PyBool_FromLong(kernel_ready(*t[0]));
  END_HANDLE_TH_ERRORS
}
PyObject *py_decode_covered(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *t[3];
  bool causal;
  if (n != 4 || !tensors(args, 3, t) || !truth(args[3], &causal)) Py_RETURN_NONE;
  return PyBool_FromLong(decode_covered(*t[0], *t[1], *t[2], causal));
  END_HANDLE_TH_ERRORS
}

#define FAST(f) (PyCFunction)(void *)f, METH_FASTCALL, nullptr
PyMethodDef methods[] = {{"flash", FAST(py_flash<false>)},
                         {"flash_rest", FAST(py_flash<true>)},
                         {"piecewise", FAST(py_piecewise)},
                         {"rotary_pair", FAST(py_rotary_pair)},
                         {"paged", FAST(py_paged)},
                         {"append", FAST(py_append)},
                         {"coarsen_partition", FAST(py_coarsen)},
                         {"kernel_ready", FAST(py_kernel_ready)},
                         {"decode_covered", FAST(py_decode_covered)},
                         {"set_backward_mode", py_backward_mode, METH_O, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "flagattn_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_flagattn_host(void) {
  PyObject *m = PyModule_Create(&module);
  // what build.host_tag() said when this was compiled; the loader compares
  if (m && PyModule_AddStringConstant(m, "built_for", FA_HOST_TAG) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
