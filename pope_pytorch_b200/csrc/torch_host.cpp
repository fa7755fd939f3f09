// torch binding of libpope_b200.so: output and workspace allocation, argument structs and the autograd nodes.
//
// What a call costs on the host decides the small shapes.  The same layer written in Python over ctypes took 45 us per
// (2, 8, 1024, 64) forward whose kernels then took 26 us and, with its backward in a Python autograd node on the engine's thread,
// 351 us per (3, 8 / 2, 777, 64) training step whose kernels took 159 us; here they took 27 and 148 us (with the kernels since
// then: 21 us, bound by the GPU, and 142 us around about 100 us of kernels).  The kernels themselves stay behind
// the C ABI (include/pope_b200.h): this file only fills its structs.  No arithmetic happens here and nothing is kept from one
// call to the next.
#include <ATen/TensorSubclassLikeUtils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <cmath>
#include <tuple>

#include "../../include/pope_b200.h"

namespace py = pybind11;
using at::Tensor;
using std::optional;

namespace {

using Factors = optional<std::tuple<Tensor, Tensor, optional<Tensor>>>;   // positions, inverse frequencies, axis of a feature

[[noreturn]] void assertion(const char* what) {   // (the GIL is held: called from the binding layer only)
  PyErr_SetString(PyExc_AssertionError, what);
  throw py::error_already_set();
}

void check(int rc, const char* what) {
  if (rc != POPE_OK) TORCH_CHECK(false, what, " failed: ", pope_b200_status_str(rc), " (status ", rc, ")");
}

int dtype_of(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return POPE_F32;
    case at::kBFloat16: return POPE_BF16;
    case at::kHalf: return POPE_F16;
    default: return -1;
  }
}

// (batch, head, row) strides of a (b, h, n, x) tensor or, with seq_first, of a (b, n, h, x) one; the innermost stride is 1
PopeStride3 s3(const Tensor& t, bool seq_first = false) { return {t.stride(0), t.stride(seq_first ? 2 : 1), t.stride(seq_first ? 1 : 2)}; }

Tensor inner_contig(const Tensor& t) { return t.size(-1) <= 1 || t.stride(-1) == 1 ? t : t.contiguous(); }

Tensor fp32_rows(const Tensor& t) { return inner_contig(t.scalar_type() == at::kFloat ? t : t.to(at::kFloat)); }

// (batch, head, row) strides with 0 = broadcast; a 4-D table is (b, h, n, r), as in apply_pope_to_qk and the reference's
// similarity (PoPE_pytorch/pope.py:53-56, triton_pope.py:267-272)
PopeStride3 freq_strides(const Tensor& f) {
  switch (f.dim()) {
    case 2: return {0, 0, f.stride(0)};
    case 3: return {f.size(0) > 1 ? f.stride(0) : 0, 0, f.stride(1)};
    case 4: return {f.size(0) > 1 ? f.stride(0) : 0, f.size(1) > 1 ? f.stride(1) : 0, f.stride(2)};
    default: TORCH_CHECK_VALUE(false, "freqs must have 2, 3 or 4 dimensions");
  }
}

// the factors of a table built by PoPE / AxialPoPE, when they are usable as they are
bool factors_usable(const Factors& f, const Tensor& freqs) {
  if (!f || freqs.dim() != 2) return false;
  const auto& [pos, inv, axis] = *f;
  return pos.device() == freqs.device() && inv.device() == freqs.device() && pos.scalar_type() == at::kFloat &&
         inv.scalar_type() == at::kFloat && pos.size(0) == freqs.size(0) && inv.numel() == freqs.size(1) && pos.stride(-1) == 1 &&
         inv.is_contiguous() &&
         (!axis || (axis->device() == freqs.device() && axis->scalar_type() == at::kInt && axis->is_contiguous()));
}

PopeEmbed embed_of(const Tensor& freqs, const Tensor& bias, int r, const Factors& f = std::nullopt) {
  PopeEmbed e = {};
  if (r == 0) return e;
  e.freqs = freqs.const_data_ptr<float>(), e.sf = freq_strides(freqs);
  e.bias = bias.const_data_ptr<float>(), e.bias_stride_h = bias.stride(0);
  if (factors_usable(f, freqs)) {
    const auto& [pos, inv, axis] = *f;
    e.positions = pos.const_data_ptr<float>(), e.pos_stride_n = pos.dim() == 2 ? pos.stride(0) : 1;
    e.inv_freqs = inv.const_data_ptr<float>();
    e.axis_of = axis ? axis->const_data_ptr<int32_t>() : nullptr;
  }
  return e;
}

PopeShape shape_of(const Tensor& q, const Tensor& k, int r, bool seq_first = false) {
  const int h = seq_first ? 2 : 1, n = seq_first ? 1 : 2;
  return {(int32_t)q.size(0), (int32_t)q.size(h), (int32_t)k.size(h), (int32_t)q.size(n), (int32_t)k.size(n), (int32_t)q.size(3), r, dtype_of(q)};
}

template <typename Args>
Tensor workspace(int op, Args& a, const Tensor& like) {
  const size_t need = pope_b200_workspace_bytes(op, &a);
  if (need == 0) return Tensor();
  Tensor ws = at::empty({(int64_t)need}, like.options().dtype(at::kByte));
  a.workspace = ws.mutable_data_ptr(), a.workspace_bytes = need;
  return ws;
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// The library sees pointers only: what a kernel reads has to be on q's device and reach as far as the kernel reads.  (Tensors
// that reach further are read in part.)
void same_device(const Tensor& t, const Tensor& q, const char* what) {
  TORCH_CHECK(t.device() == q.device(), what, " is on ", t.device(), ", q on ", q.device());
}

void validate_embed(const Tensor& q, int64_t batch, int64_t heads, int64_t key_heads, const Tensor& freqs, const Tensor& bias) {
  const int64_t r = freqs.size(-1);
  if (r == 0) return;   // (nothing of either is read)
  same_device(freqs, q, "freqs"), same_device(bias, q, "bias");
  if (freqs.dim() >= 3) TORCH_CHECK_VALUE(freqs.size(0) == 1 || freqs.size(0) >= batch, "freqs must have one table, or one per batch entry");
  if (freqs.dim() == 4) TORCH_CHECK_VALUE(freqs.size(1) == 1 || freqs.size(1) >= heads, "freqs must have one table, or one per head");
  TORCH_CHECK_VALUE(bias.dim() >= 1 && bias.size(-1) >= r && bias.numel() > 0 && (key_heads == 1 || (bias.dim() == 2 && bias.size(0) >= key_heads)),
                    "bias must have one row of rotated features per key head");
}

// the checks every operator makes on q, k and the pair (freqs, bias); GIL held
void validate(const Tensor& q, const Tensor& k, const Tensor& freqs, const Tensor& bias, bool seq_first) {
  if (!(q.is_cuda() && k.is_cuda())) TORCH_CHECK(false, "the native PoPE kernels need CUDA tensors");
  if (dtype_of(q) < 0 || k.scalar_type() != q.scalar_type())
    TORCH_CHECK_TYPE(false, "q and k must share a dtype among fp32/bf16/fp16, got ", q.scalar_type(), ", ", k.scalar_type());
  TORCH_CHECK(q.dim() == 4 && k.dim() == 4, "q and k must have 4 dimensions");
  const int ha = seq_first ? 2 : 1, na = seq_first ? 1 : 2;
  if (q.size(ha) % k.size(ha) != 0) assertion("query heads must be a multiple of key heads");
  if (q.size(na) > k.size(na) || freqs.size(-1) > q.size(-1)) assertion("queries must not outnumber keys, nor rotated features the head dim");
  if (freqs.dim() < 2 || (freqs.size(-2) != k.size(na) && freqs.size(-1) != 0)) assertion("freqs must have one row per key position");
  same_device(k, q, "k");
  TORCH_CHECK_VALUE(k.size(0) >= q.size(0) && k.size(3) >= q.size(3), "q and k must have the same batch size and head dim");
  validate_embed(q, q.size(0), q.size(ha), k.size(ha), freqs, bias);
}

// ... and the attention on v and the mask
void validate_attn(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& freqs, const Tensor& bias, const optional<Tensor>& mask,
                   bool seq_first) {
  validate(q, k, freqs, bias, seq_first);
  same_device(v, q, "v");
  if (v.scalar_type() != q.scalar_type()) TORCH_CHECK_TYPE(false, "v must have the dtype of q and k, got ", v.scalar_type(), ", ", q.scalar_type());
  const int ha = seq_first ? 2 : 1, na = seq_first ? 1 : 2;
  TORCH_CHECK_VALUE(v.dim() == 4 && v.size(0) >= q.size(0) && v.size(ha) >= k.size(ha) && v.size(na) >= k.size(na) && v.size(3) >= q.size(3),
                    "v must have the shape of k");
  if (!mask || !mask->defined()) return;
  same_device(*mask, q, "mask");
  TORCH_CHECK_VALUE(mask->dim() == 2 && mask->size(0) >= q.size(0) && mask->size(1) >= k.size(na), "mask must be (batch, keys)");
}

// The buffer of the gradient of t = k or v.  The kernels write as far as they read: of a tensor that reaches further the rest is zero.
Tensor grad_of_keys(const Tensor& t, const Tensor& k, const Tensor& q) {
  return t.sizes() == k.sizes() && k.size(0) == q.size(0) && k.size(3) == q.size(3) ? at::empty_like(t) : at::zeros_like(t);
}

// ---- attention -------------------------------------------------------------------------------------------------
struct Mask {
  Tensor keep;   // bool or uint8
  explicit Mask(const optional<Tensor>& m) {
    if (!m || !m->defined()) return;
    keep = m->scalar_type() == at::kBool || m->scalar_type() == at::kByte ? *m : m->ne(0);
  }
  template <typename Args>
  void put(Args& a) const {
    if (!keep.defined()) return;
    a.mask = static_cast<const uint8_t*>(keep.const_data_ptr()), a.mask_stride_b = keep.stride(0), a.mask_stride_n = keep.stride(1);
  }
};

// tensors of any stride with contiguous features -> (out in q's memory layout, lse (b, h, n_q))
std::tuple<Tensor, Tensor> attn_forward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& freqs_, const Tensor& bias_,
                                        const optional<Tensor>& mask, bool causal, double scale, const Factors& factors, bool sf) {
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  const Tensor q = inner_contig(q_), k = inner_contig(k_), v = inner_contig(v_), freqs = fp32_rows(freqs_), bias = fp32_rows(bias_);
  Tensor out = at::empty_like(q), lse = at::empty({q.size(0), q.size(sf ? 2 : 1), q.size(sf ? 1 : 2)}, q.options().dtype(at::kFloat));
  const int r = (int)freqs.size(-1);
  const Mask m(mask);
  PopeAttnArgs a = {};
  a.struct_bytes = sizeof(a), a.causal = causal, a.softmax_scale = (float)scale;
  a.shape = shape_of(q, k, r, sf), a.embed = embed_of(freqs, bias, r, factors);
  a.q = q.const_data_ptr(), a.sq = s3(q, sf), a.k = k.const_data_ptr(), a.sk = s3(k, sf), a.v = v.const_data_ptr(), a.sv = s3(v, sf);
  a.out = out.mutable_data_ptr(), a.so = s3(out, sf), a.lse = lse.mutable_data_ptr<float>();
  m.put(a);
  const Tensor ws = workspace(POPE_OP_ATTN_FWD, a, q);
  check(pope_b200_attn_fwd(&a, stream_of(q)), "pope_b200_attn_fwd");
  return {out, lse};
}

struct Grads {
  Tensor dq, dk, dv, dfreqs, dbias;
};

template <typename Args>
void put_phase_grads(Args& a, Grads& g, const Tensor& freqs, const Tensor& bias, bool need_df, bool need_db) {
  // (accumulators of the kernels, and the result where nothing is rotated: zero-filled either way)
  if (need_df) g.dfreqs = at::zeros(freqs.sizes(), freqs.options().dtype(at::kFloat));
  if (need_db) g.dbias = at::zeros(bias.sizes(), bias.options().dtype(at::kFloat));
  if (freqs.size(-1) == 0) return;
  if (need_df) a.dfreqs = g.dfreqs.mutable_data_ptr<float>(), a.sdf = freq_strides(g.dfreqs);
  if (need_db) a.dbias = g.dbias.mutable_data_ptr<float>(), a.dbias_stride_h = g.dbias.stride(0);
}

Grads attn_backward(const Tensor& dout_, const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& out_, const Tensor& lse,
                    const Tensor& freqs_, const Tensor& bias_, const optional<Tensor>& mask, bool causal, double scale, bool need_df,
                    bool need_db, const Factors& factors, bool sf) {
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  const Tensor q = inner_contig(q_), k = inner_contig(k_), v = inner_contig(v_), out = inner_contig(out_), dout = inner_contig(dout_);
  const Tensor freqs = fp32_rows(freqs_), bias = fp32_rows(bias_);
  const int r = (int)freqs.size(-1);
  Grads g{at::empty_like(q), grad_of_keys(k, k, q), grad_of_keys(v, k, q), Tensor(), Tensor()};
  const Mask m(mask);
  PopeAttnBwdArgs a = {};
  a.struct_bytes = sizeof(a), a.causal = causal, a.softmax_scale = (float)scale;
  a.shape = shape_of(q, k, r, sf), a.embed = embed_of(freqs, bias, r, factors);
  a.q = q.const_data_ptr(), a.sq = s3(q, sf), a.k = k.const_data_ptr(), a.sk = s3(k, sf), a.v = v.const_data_ptr(), a.sv = s3(v, sf);
  a.out = out.const_data_ptr(), a.so = s3(out, sf), a.dout = dout.const_data_ptr(), a.sdo = s3(dout, sf), a.lse = lse.const_data_ptr<float>();
  a.dq = g.dq.mutable_data_ptr(), a.sdq = s3(g.dq, sf), a.dk = g.dk.mutable_data_ptr(), a.sdk = s3(g.dk, sf);
  a.dv = g.dv.mutable_data_ptr(), a.sdv = s3(g.dv, sf);
  m.put(a);
  put_phase_grads(a, g, freqs, bias, need_df, need_db);
  const Tensor ws = workspace(POPE_OP_ATTN_BWD, a, q);
  check(pope_b200_attn_bwd(&a, stream_of(q)), "pope_b200_attn_bwd");
  return g;
}

// What a backward node keeps beside its saved tensors.  (The factors and the mask are inputs without gradients that the
// caller does not write to between the passes, as the phase table itself.)
struct Kept : torch::CustomClassHolder {
  Factors factors;
  optional<Tensor> mask;
  bool causal = false, seq_first = false;
  double scale = 1.0;
};

Tensor to_dtype_of(const Tensor& g, const Tensor& like) { return g.defined() ? g.to(like.scalar_type()) : g; }

struct FlashAttn : torch::autograd::Function<FlashAttn> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& freqs,
                        const Tensor& bias, const c10::intrusive_ptr<Kept>& kept) {
    auto [out, lse] = attn_forward(q, k, v, freqs, bias, kept->mask, kept->causal, kept->scale, kept->factors, kept->seq_first);
    ctx->save_for_backward({q, k, v, freqs, bias, out, lse});
    ctx->saved_data["kept"] = c10::IValue::make_capsule(kept);
    return out;
  }
  static torch::autograd::tensor_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::tensor_list grad) {
    const auto s = ctx->get_saved_variables();
    const auto kept = c10::static_intrusive_pointer_cast<Kept>(ctx->saved_data["kept"].toCapsule());
    Grads g = attn_backward(grad[0].to(s[0].scalar_type()), s[0], s[1], s[2], s[5], s[6], s[3], s[4], kept->mask, kept->causal, kept->scale,
                            ctx->needs_input_grad(3), ctx->needs_input_grad(4), kept->factors, kept->seq_first);
    return {g.dq, g.dk, g.dv, to_dtype_of(g.dfreqs, s[3]), to_dtype_of(g.dbias, s[4]), Tensor()};
  }
};

// Whether the call goes through its autograd node: for gradients, and for tangents of forward mode, which the node refuses
// (a call past it would drop them).
template <typename... Ts>
bool wants_graph(const Ts&... ts) {
  return (at::GradMode::is_enabled() && (ts.requires_grad() || ...)) || (ts._fw_grad(0).defined() || ...);
}

Tensor flash_attn(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& freqs, const Tensor& bias, const optional<Tensor>& mask,
                  bool causal, double scale, const Factors& factors, bool seq_first) {
  validate_attn(q, k, v, freqs, bias, mask, seq_first);
  py::gil_scoped_release nogil;
  if (!wants_graph(q, k, v, freqs, bias)) {
    at::AutoDispatchBelowADInplaceOrView below;
    return std::get<0>(attn_forward(q, k, v, freqs, bias, mask, causal, scale, factors, seq_first));
  }
  auto kept = c10::make_intrusive<Kept>();
  kept->factors = factors, kept->mask = mask, kept->causal = causal, kept->seq_first = seq_first, kept->scale = scale;
  return FlashAttn::apply(q, k, v, freqs, bias, kept);
}

// ---- similarity ------------------------------------------------------------------------------------------------
Tensor sim_forward(const Tensor& q_, const Tensor& k_, const Tensor& freqs_, const Tensor& bias_, bool allow_tf32, const Factors& factors, bool sf) {
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  const Tensor q = inner_contig(q_), k = inner_contig(k_), freqs = fp32_rows(freqs_), bias = fp32_rows(bias_);
  const int r = (int)freqs.size(-1);
  Tensor sim = at::empty({q.size(0), q.size(sf ? 2 : 1), q.size(sf ? 1 : 2), k.size(sf ? 1 : 2)}, q.options());
  PopeSimArgs a = {};
  a.struct_bytes = sizeof(a), a.allow_tf32 = allow_tf32;
  a.shape = shape_of(q, k, r, sf), a.embed = embed_of(freqs, bias, r, factors);
  a.q = q.const_data_ptr(), a.sq = s3(q, sf), a.k = k.const_data_ptr(), a.sk = s3(k, sf), a.sim = sim.mutable_data_ptr(), a.ss = s3(sim);
  const Tensor ws = workspace(POPE_OP_SIM_FWD, a, q);
  check(pope_b200_sim_fwd(&a, stream_of(q)), "pope_b200_sim_fwd");
  return sim;
}

Grads sim_backward(const Tensor& dsim_, const Tensor& q_, const Tensor& k_, const Tensor& freqs_, const Tensor& bias_, bool need_df, bool need_db,
                   bool allow_tf32, bool sf) {
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  const Tensor q = inner_contig(q_), k = inner_contig(k_), dsim = inner_contig(dsim_), freqs = fp32_rows(freqs_), bias = fp32_rows(bias_);
  const int r = (int)freqs.size(-1);
  Grads g{at::empty_like(q), grad_of_keys(k, k, q), Tensor(), Tensor(), Tensor()};
  PopeSimBwdArgs a = {};
  a.struct_bytes = sizeof(a), a.allow_tf32 = allow_tf32;
  a.shape = shape_of(q, k, r, sf), a.embed = embed_of(freqs, bias, r);
  a.q = q.const_data_ptr(), a.sq = s3(q, sf), a.k = k.const_data_ptr(), a.sk = s3(k, sf), a.dsim = dsim.const_data_ptr(), a.sds = s3(dsim);
  a.dq = g.dq.mutable_data_ptr(), a.sdq = s3(g.dq, sf), a.dk = g.dk.mutable_data_ptr(), a.sdk = s3(g.dk, sf);
  put_phase_grads(a, g, freqs, bias, need_df, need_db);
  const Tensor ws = workspace(POPE_OP_SIM_BWD, a, q);
  check(pope_b200_sim_bwd(&a, stream_of(q)), "pope_b200_sim_bwd");
  return g;
}

struct Similarity : torch::autograd::Function<Similarity> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& freqs, const Tensor& bias,
                        bool allow_tf32, bool seq_first, const Factors& factors) {
    ctx->save_for_backward({q, k, freqs, bias});
    ctx->saved_data["tf32"] = allow_tf32, ctx->saved_data["seq"] = seq_first;
    return sim_forward(q, k, freqs, bias, allow_tf32, factors, seq_first);
  }
  static torch::autograd::tensor_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::tensor_list grad) {
    const auto s = ctx->get_saved_variables();
    Grads g = sim_backward(grad[0].to(s[0].scalar_type()), s[0], s[1], s[2], s[3], ctx->needs_input_grad(2), ctx->needs_input_grad(3),
                           ctx->saved_data["tf32"].toBool(), ctx->saved_data["seq"].toBool());
    return {g.dq, g.dk, to_dtype_of(g.dfreqs, s[2]), to_dtype_of(g.dbias, s[3]), Tensor(), Tensor(), Tensor()};
  }
};

Tensor similarity(const Tensor& q, const Tensor& k, const Tensor& freqs, const Tensor& bias, bool allow_tf32, const Factors& factors,
                  bool seq_first) {
  validate(q, k, freqs, bias, seq_first);
  py::gil_scoped_release nogil;
  if (!wants_graph(q, k, freqs, bias)) {
    at::AutoDispatchBelowADInplaceOrView below;
    return sim_forward(q, k, freqs, bias, allow_tf32, factors, seq_first);
  }
  return Similarity::apply(q, k, freqs, bias, allow_tf32, seq_first, factors);
}

// ---- the stand-alone transform -----------------------------------------------------------------------------------
std::tuple<Tensor, Tensor> apply_forward(const Tensor& q_, const Tensor& k_, const Tensor& freqs_, const Tensor& bias_) {
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  const Tensor q = inner_contig(q_), k = inner_contig(k_), freqs = fp32_rows(freqs_), bias = fp32_rows(bias_);
  const int r = (int)freqs.size(-1);
  const auto opt = q.options().dtype(at::kFloat);
  Tensor q_out = at::empty({q.size(0), q.size(1), q.size(2), q.size(3) + r}, opt);
  Tensor k_out = at::empty({k.size(0), k.size(1), k.size(2), k.size(3) + r}, opt);
  PopeApplyArgs a = {};
  a.struct_bytes = sizeof(a), a.shape = shape_of(q, k, r), a.embed = embed_of(freqs, bias, r);
  a.q = q.const_data_ptr(), a.sq = s3(q), a.k = k.const_data_ptr(), a.sk = s3(k);
  a.q_out = q_out.mutable_data_ptr<float>(), a.sqo = s3(q_out), a.k_out = k_out.mutable_data_ptr<float>(), a.sko = s3(k_out);
  check(pope_b200_apply_qk_fwd(&a, stream_of(q)), "pope_b200_apply_qk_fwd");
  return {q_out, k_out};
}

struct ApplyQK : torch::autograd::Function<ApplyQK> {
  static torch::autograd::tensor_list forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& freqs,
                                              const Tensor& bias) {
    ctx->save_for_backward({q, k, freqs, bias});
    auto [q_out, k_out] = apply_forward(q, k, freqs, bias);
    return {q_out, k_out};
  }
  static torch::autograd::tensor_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::tensor_list grad) {
    const auto s = ctx->get_saved_variables();
    c10::cuda::OptionalCUDAGuard guard(s[0].device());
    const Tensor q = inner_contig(s[0]), k = inner_contig(s[1]), freqs = fp32_rows(s[2]), bias = fp32_rows(s[3]);
    const Tensor gq = grad[0].contiguous().to(at::kFloat), gk = grad[1].contiguous().to(at::kFloat);
    const int r = (int)freqs.size(-1);
    Grads g{at::empty_like(q), at::empty_like(k), Tensor(), Tensor(), Tensor()};
    PopeApplyBwdArgs a = {};
    a.struct_bytes = sizeof(a), a.shape = shape_of(q, k, r), a.embed = embed_of(freqs, bias, r);
    a.q = q.const_data_ptr(), a.sq = s3(q), a.k = k.const_data_ptr(), a.sk = s3(k);
    a.dq_out = gq.const_data_ptr<float>(), a.sdqo = s3(gq), a.dk_out = gk.const_data_ptr<float>(), a.sdko = s3(gk);
    a.dq = g.dq.mutable_data_ptr(), a.sdq = s3(g.dq), a.dk = g.dk.mutable_data_ptr(), a.sdk = s3(g.dk);
    put_phase_grads(a, g, freqs, bias, ctx->needs_input_grad(2), ctx->needs_input_grad(3));
    check(pope_b200_apply_qk_bwd(&a, stream_of(q)), "pope_b200_apply_qk_bwd");
    return {g.dq, g.dk, to_dtype_of(g.dfreqs, s[2]), to_dtype_of(g.dbias, s[3])};
  }
};

// Whether the kernel takes the call: one supported dtype, batch size, head dim and device, a table and a bias that reach as far, an
// even expanded width.  (The PyTorch operations take the rest, or say what is wrong with it.)
bool apply_qk_takes(const Tensor& q, const Tensor& k, const Tensor& freqs, const Tensor& bias) {
  if (!q.is_cuda() || q.dim() != 4 || k.dim() != 4 || freqs.dim() < 2 || freqs.dim() > 4 || bias.dim() != 2) return false;
  if (k.device() != q.device() || freqs.device() != q.device() || bias.device() != q.device()) return false;
  if (dtype_of(q) < 0 || k.scalar_type() != q.scalar_type()) return false;
  const int64_t b = q.size(0), h = q.size(1), hk = k.size(1), d = q.size(3), r = freqs.size(-1);
  return hk > 0 && h % hk == 0 && k.size(0) == b && k.size(3) == d && d <= 256 && (d + r) % 2 == 0 && bias.size(0) >= hk && bias.size(1) >= r &&
         (freqs.dim() == 2 || freqs.size(0) == 1 || freqs.size(0) >= b) && (freqs.dim() < 4 || freqs.size(1) == 1 || freqs.size(1) >= h);
}

std::tuple<Tensor, Tensor> apply_qk(const Tensor& q, const Tensor& k, const Tensor& freqs, const Tensor& bias) {
  if (freqs.size(-1) != 0 && freqs.size(-2) != k.size(2)) assertion("freqs must have one row per key position");
  py::gil_scoped_release nogil;
  if (!wants_graph(q, k, freqs, bias)) {
    at::AutoDispatchBelowADInplaceOrView below;
    return apply_forward(q, k, freqs, bias);
  }
  const auto out = ApplyQK::apply(q, k, freqs, bias);
  return {out[0], out[1]};
}

// ---- the embedding tables ------------------------------------------------------------------------------------------
// a tensor whose memory a kernel may be given: fp32, contiguous, of no function transform or dispatch mode, without a tangent
bool plain(const Tensor& t) {
  return !at::isTensorSubclassLike(t) && t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous() && !t._fw_grad(0).defined();
}

// (freqs, clamped bias, positions, flat inverse frequencies, axis of a feature) of a sequence or a grid; a sequence has no
// last two.  bias may carry a gradient, the frequencies do not (the Python modules see to that).
struct Table : torch::autograd::Function<Table> {
  static torch::autograd::tensor_list forward(torch::autograd::AutogradContext* ctx, const Tensor& bias, const std::vector<Tensor>* inv,
                                              const std::vector<int64_t>* dims, double offset) {
    c10::cuda::OptionalCUDAGuard guard(bias.device());
    PopeTableArgs a = {};
    a.struct_bytes = sizeof(a), a.axes = (int32_t)dims->size(), a.offset = (float)offset;
    int64_t n = 1, r = 0;
    for (int i = 0; i < a.axes; ++i) {
      a.dims[i] = (int32_t)(*dims)[i], a.width[i] = (int32_t)(*inv)[i].numel(), a.inv_freqs[i] = (*inv)[i].const_data_ptr<float>();
      n *= a.dims[i], r += a.width[i];
    }
    const bool grid = a.axes > 1;
    const auto opt = bias.options();
    Tensor freqs = at::empty({n, r}, opt), clamped = at::empty({bias.size(0), bias.size(1)}, opt);
    Tensor pos = grid ? at::empty({n, a.axes}, opt) : at::empty({n}, opt), inv_flat, axis_of;
    if (grid) inv_flat = at::empty({r}, opt), axis_of = at::empty({r}, opt.dtype(at::kInt));
    a.H = (int32_t)bias.size(0), a.bias = bias.const_data_ptr<float>(), a.bias_out = clamped.mutable_data_ptr<float>();
    a.positions = pos.mutable_data_ptr<float>(), a.freqs = freqs.mutable_data_ptr<float>();
    if (grid) a.inv_flat = inv_flat.mutable_data_ptr<float>(), a.axis_of = axis_of.mutable_data_ptr<int32_t>();
    check(pope_b200_table(&a, stream_of(bias)), "pope_b200_table");
    ctx->save_for_backward({bias});
    ctx->set_materialize_grads(false);
    torch::autograd::tensor_list out = {freqs, clamped, pos};
    if (grid) out.insert(out.end(), {inv_flat, axis_of});
    torch::autograd::tensor_list constant = out;
    constant.erase(constant.begin() + 1);
    ctx->mark_non_differentiable(constant);
    return out;
  }
  static torch::autograd::tensor_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::tensor_list grad) {
    if (!grad[1].defined()) return {Tensor(), Tensor(), Tensor(), Tensor()};
    const Tensor bias = ctx->get_saved_variables()[0];
    // a gradient that is differentiated itself (create_graph), or a batch of them: the clamp's gradient as PyTorch operations
    if (at::GradMode::is_enabled() || at::isTensorSubclassLike(grad[1])) {
      const Tensor passes = bias.ge(POPE_BIAS_MIN).logical_and_(bias.le(0.f));
      return {at::where(passes, grad[1], at::zeros({}, bias.options())), Tensor(), Tensor(), Tensor()};
    }
    const Tensor g = grad[1].contiguous();
    c10::cuda::OptionalCUDAGuard guard(bias.device());
    Tensor out = at::empty_like(bias);
    PopeClampBwdArgs a = {};
    a.struct_bytes = sizeof(a), a.n = bias.numel();
    a.bias = bias.const_data_ptr<float>(), a.grad = g.const_data_ptr<float>(), a.grad_bias = out.mutable_data_ptr<float>();
    check(pope_b200_clamp_bwd(&a, stream_of(bias)), "pope_b200_clamp_bwd");
    return {out, Tensor(), Tensor(), Tensor()};
  }
};

// None when the module's tensors are not what the kernel takes (another type or device, frequencies that train, tensors of a
// function transform or of a dispatch mode, forward mode): the module's own PyTorch operations serve those
optional<std::vector<Tensor>> table(const Tensor& bias, const std::vector<Tensor>& inv, const std::vector<int64_t>& dims, double offset) {
  if (inv.empty() || inv.size() != dims.size() || inv.size() > POPE_MAX_AXES || bias.dim() != 2 || !plain(bias)) return std::nullopt;
  int64_t n = 1, r = 0;
  for (const int64_t d : dims) {
    if (d <= 0 || d > INT32_MAX || n * d > INT32_MAX) return std::nullopt;
    n *= d;
  }
  for (const Tensor& t : inv) {
    if (!plain(t) || t.device() != bias.device() || t.requires_grad() || t.numel() == 0) return std::nullopt;
    r += t.numel();
  }
  if (bias.size(1) != r || bias.size(0) == 0) return std::nullopt;
  py::gil_scoped_release nogil;
  return Table::apply(bias, &inv, &dims, offset);
}

// ---- paged key / value cache ---------------------------------------------------------------------------------------
// The cache's tensors; `row` > 0 = the view that starts at sequence `row` (a batch of one)
struct Pages {
  Tensor k, v, table, lens;
  PopePagedKV view(int64_t row = 0) const {
    PopePagedKV kv = {};
    kv.k_pages = k.mutable_data_ptr(), kv.v_pages = v.mutable_data_ptr();
    kv.page_table = table.const_data_ptr<int32_t>() + row * table.size(1), kv.seq_lens = lens.mutable_data_ptr<int32_t>() + row;
    kv.num_pages = (int32_t)k.size(0), kv.page_size = (int32_t)k.size(2), kv.max_pages_per_seq = (int32_t)table.size(1);
    return kv;
  }
};

void kv_map(const Pages& p, const std::vector<int32_t>& index, const std::vector<int32_t>& value) {
  py::gil_scoped_release nogil;
  c10::cuda::OptionalCUDAGuard guard(p.k.device());
  PopeKvMapArgs a = {};
  a.struct_bytes = sizeof(a), a.n = (int32_t)index.size(), a.B = (int32_t)p.lens.size(0), a.max_pages_per_seq = (int32_t)p.table.size(1);
  a.page_table = p.table.mutable_data_ptr<int32_t>(), a.seq_lens = p.lens.mutable_data_ptr<int32_t>();
  a.index = index.data(), a.value = value.data();
  check(pope_b200_kv_map(&a, stream_of(p.k)), "pope_b200_kv_map");
}

// k, v (b, hk, n, d), or (hk, n, d) for sequence `row` alone
void kv_append(const Pages& p, const Tensor& k_, const Tensor& v_, int64_t row) {
  py::gil_scoped_release nogil;
  c10::cuda::OptionalCUDAGuard guard(p.k.device());
  at::NoGradGuard off;
  const Tensor k = inner_contig(k_), v = inner_contig(v_);
  const bool one = k.dim() == 3;
  const int64_t h = one ? 0 : 1;
  TORCH_CHECK_INDEX(row >= 0 && row + (one ? 1 : k.size(0)) <= p.lens.size(0), "sequence ", row, " is not in the cache");
  PopeKvAppendArgs a = {};
  a.struct_bytes = sizeof(a), a.dtype = dtype_of(k), a.B = one ? 1 : (int32_t)k.size(0), a.Hk = (int32_t)k.size(h), a.d = (int32_t)k.size(h + 2);
  a.n_new = (int32_t)k.size(h + 1), a.advance = 1, a.kv = p.view(row);
  a.k = k.const_data_ptr(), a.sk = {one ? 0 : k.stride(0), k.stride(h), k.stride(h + 1)};
  a.v = v.const_data_ptr(), a.sv = {one ? 0 : v.stride(0), v.stride(h), v.stride(h + 1)};
  check(pope_b200_kv_append(&a, stream_of(k)), "pope_b200_kv_append");
}

std::tuple<Tensor, Tensor> kv_decode(const Pages& p, const Tensor& q_, const Tensor& freqs_, const Tensor& bias_, double scale, int64_t nk) {
  validate_embed(q_, q_.size(0), q_.size(1), p.k.size(1), freqs_, bias_);
  py::gil_scoped_release nogil;
  c10::cuda::OptionalCUDAGuard guard(p.k.device());
  at::NoGradGuard off;
  const Tensor q = inner_contig(q_), freqs = fp32_rows(freqs_), bias = fp32_rows(bias_);
  const int r = (int)freqs.size(-1);
  Tensor out = at::empty_like(q), lse = at::empty({q.size(0), q.size(1)}, q.options().dtype(at::kFloat));
  PopePagedDecodeArgs a = {};
  a.struct_bytes = sizeof(a), a.softmax_scale = (float)scale;
  a.shape = {(int32_t)q.size(0), (int32_t)q.size(1), (int32_t)p.k.size(1), 1, (int32_t)nk, (int32_t)q.size(3), r, dtype_of(q)};
  a.embed = embed_of(freqs, bias, r), a.kv = p.view();
  a.q = q.const_data_ptr(), a.sq = s3(q), a.out = out.mutable_data_ptr(), a.so = s3(out), a.lse = lse.mutable_data_ptr<float>();
  const Tensor ws = workspace(POPE_OP_DECODE_PAGED, a, q);
  check(pope_b200_attn_decode_paged(&a, stream_of(q)), "pope_b200_attn_decode_paged");
  return {out, lse};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("factors_usable", &factors_usable);
  m.def("flash_attn", &flash_attn);
  m.def("similarity", &similarity);
  m.def("apply_qk", &apply_qk);
  m.def("apply_qk_takes", &apply_qk_takes);
  m.def("table", &table);
  py::class_<Pages>(m, "Pages").def(py::init([](Tensor k, Tensor v, Tensor table, Tensor lens) { return Pages{k, v, table, lens}; }));
  m.def("kv_map", &kv_map);
  m.def("kv_append", &kv_append);
  m.def("kv_decode", &kv_decode);
  m.def("attn_forward", [](const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& freqs, const Tensor& bias, const optional<Tensor>& mask,
                           bool causal, double scale, const Factors& factors) {
    validate_attn(q, k, v, freqs, bias, mask, false);
    at::NoGradGuard off;
    return attn_forward(q, k, v, freqs, bias, mask, causal, scale, factors, false);
  });
  m.def("attn_backward", [](const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse,
                            const Tensor& freqs, const Tensor& bias, const optional<Tensor>& mask, bool causal, double scale, bool need_df,
                            bool need_db, const Factors& factors) {
    validate_attn(q, k, v, freqs, bias, mask, false);
    same_device(out, q, "out"), same_device(dout, q, "dout"), same_device(lse, q, "lse");
    TORCH_CHECK_VALUE(out.sizes() == q.sizes() && dout.sizes() == q.sizes() && lse.sizes() == q.sizes().slice(0, 3) && lse.is_contiguous(),
                      "out and dout must have the shape of q, lse its rows");
    if (out.scalar_type() != q.scalar_type() || dout.scalar_type() != q.scalar_type() || lse.scalar_type() != at::kFloat)
      TORCH_CHECK_TYPE(false, "out and dout must have the dtype of q, lse fp32");
    at::NoGradGuard off;
    Grads g = attn_backward(dout, q, k, v, out, lse, freqs, bias, mask, causal, scale, need_df, need_db, factors, false);
    return std::make_tuple(g.dq, g.dk, g.dv, need_df ? optional<Tensor>(g.dfreqs) : std::nullopt, need_db ? optional<Tensor>(g.dbias) : std::nullopt);
  });
  m.def("sim_forward", [](const Tensor& q, const Tensor& k, const Tensor& freqs, const Tensor& bias, bool allow_tf32, const Factors& factors) {
    validate(q, k, freqs, bias, false);
    at::NoGradGuard off;
    return sim_forward(q, k, freqs, bias, allow_tf32, factors, false);
  });
  m.def("sim_backward", [](const Tensor& dsim, const Tensor& q, const Tensor& k, const Tensor& freqs, const Tensor& bias, bool need_df, bool need_db,
                           bool allow_tf32) {
    validate(q, k, freqs, bias, false);
    same_device(dsim, q, "dsim");
    TORCH_CHECK_VALUE(dsim.dim() == 4 && dsim.size(0) >= q.size(0) && dsim.size(1) >= q.size(1) && dsim.size(2) >= q.size(2) && dsim.size(3) >= k.size(2),
                      "dsim must have the shape of the similarity");
    if (dsim.scalar_type() != q.scalar_type()) TORCH_CHECK_TYPE(false, "dsim must have the dtype of q");
    at::NoGradGuard off;
    Grads g = sim_backward(dsim, q, k, freqs, bias, need_df, need_db, allow_tf32, false);
    return std::make_tuple(g.dq, g.dk, need_df ? optional<Tensor>(g.dfreqs) : std::nullopt, need_db ? optional<Tensor>(g.dbias) : std::nullopt);
  });
}
