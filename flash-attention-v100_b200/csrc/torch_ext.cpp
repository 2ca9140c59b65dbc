// Torch extension `flash_attn_v100_cuda`: the module the Python package imports, with the
// entry points `fwd` and `bwd` of the reference's extension (kernel/fused_mha_api.cpp:13-72,
// :74-162, exported at :164-168).  All it does is check tensors, allocate outputs and the
// backward workspace with torch, and call the C ABI of libfmha_b200 on torch's current
// stream under a device guard (as kernel/fused_mha_api.cpp:61,67).  No kernel lives here and
// there is no fallback: without a CUDA device the checks raise.
//
// Differences from the reference extension, all widenings:
//   - any sm_100 device instead of the sm_70 gate (kernel/fused_mha_api.cpp:21-23);
//   - bf16 beside fp16 (reference: fp16 only, :25-29); head_dim 64, 96 or 128 (reference: 128 only, :44); sequence length a multiple of 32 is
//     CHECKED (the reference only documents it, README.md:3);
//   - q and k/v may differ in sequence length; row/head/batch strides are honoured;
//   - `fwd` returns {out, softmax_max, softmax_sum} like the reference (:71), where
//     softmax_max carries lse = max + ln(sum) and softmax_sum is all ones, so that the
//     reference's relation P = exp(scale*S - max) / sum (kernel/fused_mha_kernel.cu:457,602)
//     still holds for a caller that uses the pair;
//   - `bwd` ignores the fp16 `D` argument (flash_attn_interface.py:43-44) and computes
//     D = rowsum(dO o O) itself in fp32.
#include <ATen/FuncTorchTLS.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/AutogradState.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/autograd_not_implemented_fallback.h>
#include <torch/extension.h>

#include <cmath>
#include <optional>
#include <tuple>
#include <vector>

#include "../../include/fmha_b200.h"

namespace {

FmhaStrides strides_of(const at::Tensor& t) {
  FmhaStrides s;
  s.batch = t.stride(0);
  s.row = t.stride(1);
  s.head = t.stride(2);
  return s;
}

void check_input(const at::Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda(), name, " must be on CUDA");
  TORCH_CHECK(t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16,
              "This repo only supports fp16 and bf16 data types (", name, ")");
  TORCH_CHECK(t.dim() == 4, name, " must have shape (batch, seqlen, heads, head_size)");
  TORCH_CHECK(t.stride(-1) == 1, name, " must have contiguous last dimension");
}

// uninitialised memory, straight from the caching allocator (the dispatcher's at::empty costs
// about a microsecond more per tensor, and a backward makes four)
at::Tensor empty_on(const at::Tensor& like, at::IntArrayRef sizes, at::ScalarType type) {
  return at::detail::empty_cuda(sizes, type, like.device(), std::nullopt);
}
at::Tensor fresh_like(const at::Tensor& t) {
  return t.is_contiguous() ? empty_on(t, t.sizes(), t.scalar_type()) : at::empty_like(t);
}

void check_status(int rc, const char* what) {
  TORCH_CHECK(rc == FMHA_OK, what, " failed: ", fmha_status_string(rc), " (status ", rc, ")");
}

void check_shapes(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v) {
  const auto B = q.size(0), Nq = q.size(1), H = q.size(2), D = q.size(3);
  const auto Nk = k.size(1);
  TORCH_CHECK(B > 0, "batch size must be positive");
  TORCH_CHECK(D == 64 || D == 96 || D == 128, "head dimension must be 64, 96 or 128, got ", D);
  TORCH_CHECK(k.size(0) == B && k.size(2) == H && k.size(3) == D,
              "k must have shape (batch_size, seqlen_k, num_heads, head_size)");
  TORCH_CHECK(v.sizes() == k.sizes(), "v must have the shape of k");
  TORCH_CHECK(k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(),
              "q, k and v must have the same data type");
  TORCH_CHECK(Nq % 32 == 0 && Nk % 32 == 0,
              "sequence lengths must be multiples of 32 (pad the inputs), got ", Nq, " and ", Nk);
}

// per-batch lengths of a right-padded batch -> device pointer (or NULL)
const int32_t* seqused_ptr(const std::optional<at::Tensor>& t, const at::Tensor& q, const char* name) {
  if (!t.has_value()) return nullptr;
  TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kInt && t->dim() == 1 &&
                  t->size(0) == q.size(0) && t->is_contiguous(),
              name, " must be a contiguous int32 CUDA tensor with one entry per batch");
  return t->data_ptr<int32_t>();
}

std::vector<at::Tensor> fwd_impl(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                 std::optional<at::Tensor> out_, double softmax_scale,
                                 bool is_causal, bool want_sum,
                                 std::optional<at::Tensor> seqused_q = std::nullopt,
                                 std::optional<at::Tensor> seqused_k = std::nullopt) {
  check_input(q, "q");
  check_input(k, "k");
  check_input(v, "v");
  check_shapes(q, k, v);
  const int B = q.size(0), Nq = q.size(1), H = q.size(2), D = q.size(3), Nk = k.size(1);

  at::Tensor out;
  if (out_.has_value()) {
    out = out_.value();
    check_input(out, "out");
    TORCH_CHECK(out.sizes() == q.sizes() && out.scalar_type() == q.scalar_type(),
                "out must have the shape and type of q");
  } else {
    out = fresh_like(q);
  }
  c10::cuda::CUDAGuard guard(q.device());
  at::Tensor lse = empty_on(q, {B, H, Nq}, at::kFloat);

  FmhaFwdParams p = {};
  p.q = q.data_ptr();
  p.k = k.data_ptr();
  p.v = v.data_ptr();
  p.o = out.data_ptr();
  p.lse = lse.data_ptr<float>();
  p.q_strides = strides_of(q);
  p.k_strides = strides_of(k);
  p.v_strides = strides_of(v);
  p.o_strides = strides_of(out);
  p.batch = B;
  p.heads = H;
  p.seqlen_q = Nq;
  p.seqlen_k = Nk;
  p.head_dim = D;
  p.scale = static_cast<float>(softmax_scale);
  p.causal = is_causal ? 1 : 0;
  p.causal_shift = 0;
  p.dtype = q.scalar_type() == at::kBFloat16 ? FMHA_DTYPE_BF16 : FMHA_DTYPE_FP16;
  p.seqused_q = seqused_ptr(seqused_q, q, "seqused_q");
  p.seqused_k = seqused_ptr(seqused_k, q, "seqused_k");
  at::Tensor ws;
  size_t ws_bytes = fmha_fwd_workspace_bytes(&p);
  if (ws_bytes > 0) {
    try {
      ws = empty_on(q, {static_cast<int64_t>(ws_bytes)}, at::kByte);
    } catch (const c10::OutOfMemoryError&) {
      ws_bytes = 0;  // the call does not need it: uncut, it is only slower
    }
  }
  check_status(fmha_fwd_with_workspace(&p, ws_bytes > 0 ? ws.data_ptr() : nullptr, ws_bytes,
                                       at::cuda::getCurrentCUDAStream().stream()),
               "fmha_fwd");
  if (!want_sum) return {out, lse};
  return {out, lse, at::ones({B, H, Nq}, q.options().dtype(at::kFloat))};
}

// the reference's entry point: {out, softmax_max := lse, softmax_sum := 1}
std::vector<at::Tensor> mha_fwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                std::optional<at::Tensor> out_, double softmax_scale,
                                bool is_causal) {
  return fwd_impl(q, k, v, out_, softmax_scale, is_causal, true);
}

// {out, lse} only: what this package's own autograd glue uses (no tensor of ones to fill)
std::vector<at::Tensor> mha_fwd_lse(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                    std::optional<at::Tensor> out_, double softmax_scale,
                                    bool is_causal, std::optional<at::Tensor> seqused_q,
                                    std::optional<at::Tensor> seqused_k) {
  return fwd_impl(q, k, v, out_, softmax_scale, is_causal, false, seqused_q, seqused_k);
}

std::vector<at::Tensor> bwd_impl(const at::Tensor& dout, const at::Tensor& q, const at::Tensor& k,
                                 const at::Tensor& v, const at::Tensor& out,
                                 std::optional<at::Tensor> softmax_sum, const at::Tensor& softmax_max,
                                 std::optional<at::Tensor> dq_, std::optional<at::Tensor> dk_,
                                 std::optional<at::Tensor> dv_, double softmax_scale, bool is_causal,
                                 std::optional<at::Tensor> seqused_q, std::optional<at::Tensor> seqused_k,
                                 bool deterministic) {
  check_input(q, "q");
  check_input(k, "k");
  check_input(v, "v");
  check_input(out, "out");
  check_input(dout, "dout");
  check_shapes(q, k, v);
  TORCH_CHECK(out.sizes() == q.sizes() && out.scalar_type() == q.scalar_type(),
              "out must have the shape and type of q");
  TORCH_CHECK(dout.sizes() == q.sizes() && dout.scalar_type() == q.scalar_type(),
              "dout must have the shape and type of q");
  const int B = q.size(0), Nq = q.size(1), H = q.size(2), D = q.size(3), Nk = k.size(1);
  TORCH_CHECK(softmax_max.is_cuda() && softmax_max.scalar_type() == at::kFloat &&
                  softmax_max.sizes() == at::IntArrayRef({B, H, Nq}),
              "softmax_max must be a CUDA fp32 tensor of shape (batch_size, num_heads, seqlen_q)");

  c10::cuda::CUDAGuard guard(q.device());
  at::Tensor lse = softmax_max;
  if (softmax_sum.has_value()) {
    TORCH_CHECK(softmax_sum->sizes() == softmax_max.sizes(), "softmax_sum must have the shape of softmax_max");
    lse = softmax_max + softmax_sum->log();
  }
  lse = lse.contiguous();

  auto take = [&](std::optional<at::Tensor>& t, const at::Tensor& like, const char* name) {
    if (t.has_value()) {
      check_input(t.value(), name);
      TORCH_CHECK(t->sizes() == like.sizes() && t->scalar_type() == like.scalar_type(), name,
                  " must have the shape and type of its input");
      return t.value();
    }
    return fresh_like(like);
  };
  at::Tensor dq = take(dq_, q, "dq");
  at::Tensor dk = take(dk_, k, "dk");
  at::Tensor dv = take(dv_, v, "dv");

  FmhaBwdParams p = {};
  p.q = q.data_ptr();
  p.k = k.data_ptr();
  p.v = v.data_ptr();
  p.o = out.data_ptr();
  p.dout = dout.data_ptr();
  p.lse = lse.data_ptr<float>();
  p.dq = dq.data_ptr();
  p.dk = dk.data_ptr();
  p.dv = dv.data_ptr();
  p.q_strides = strides_of(q);
  p.k_strides = strides_of(k);
  p.v_strides = strides_of(v);
  p.o_strides = strides_of(out);
  p.dout_strides = strides_of(dout);
  p.dq_strides = strides_of(dq);
  p.dk_strides = strides_of(dk);
  p.dv_strides = strides_of(dv);
  p.batch = B;
  p.heads = H;
  p.seqlen_q = Nq;
  p.seqlen_k = Nk;
  p.head_dim = D;
  p.scale = static_cast<float>(softmax_scale);
  p.causal = is_causal ? 1 : 0;
  p.dtype = q.scalar_type() == at::kBFloat16 ? FMHA_DTYPE_BF16 : FMHA_DTYPE_FP16;
  p.seqused_q = seqused_ptr(seqused_q, q, "seqused_q");
  p.seqused_k = seqused_ptr(seqused_k, q, "seqused_k");
  p.flags = FMHA_BWD_DROP_WORKSPACE | (deterministic ? FMHA_BWD_DETERMINISTIC : 0);
  const size_t ws_bytes = fmha_bwd_workspace_bytes(&p);
  at::Tensor ws = empty_on(q, {static_cast<int64_t>(ws_bytes)}, at::kByte);
  check_status(fmha_bwd(&p, ws.data_ptr(), ws_bytes, at::cuda::getCurrentCUDAStream().stream()),
               "fmha_bwd");
  return {dq, dk, dv};
}

// the reference's entry point (kernel/fused_mha_api.cpp:74-87); its fp16 D argument is ignored
std::vector<at::Tensor> mha_bwd(const at::Tensor& dout, const at::Tensor& q, const at::Tensor& k,
                                const at::Tensor& v, const at::Tensor& out,
                                std::optional<at::Tensor> D_unused,
                                std::optional<at::Tensor> softmax_sum, const at::Tensor& softmax_max,
                                std::optional<at::Tensor> dq_, std::optional<at::Tensor> dk_,
                                std::optional<at::Tensor> dv_, double softmax_scale,
                                bool is_causal) {
  (void)D_unused;
  return bwd_impl(dout, q, k, v, out, softmax_sum, softmax_max, dq_, dk_, dv_, softmax_scale,
                  is_causal, std::nullopt, std::nullopt, false);
}

// this package's own glue: lse instead of (max, sum), per-batch lengths, deterministic dQ
std::vector<at::Tensor> mha_bwd_lse(const at::Tensor& dout, const at::Tensor& q, const at::Tensor& k,
                                    const at::Tensor& v, const at::Tensor& out, const at::Tensor& lse,
                                    double softmax_scale, bool is_causal,
                                    std::optional<at::Tensor> seqused_q,
                                    std::optional<at::Tensor> seqused_k, bool deterministic) {
  return bwd_impl(dout, q, k, v, out, std::nullopt, lse, std::nullopt, std::nullopt, std::nullopt,
                  softmax_scale, is_causal, seqused_q, seqused_k, deterministic);
}

// ---------------------------------------------------------------------------------------------
// Dispatcher ops and autograd.  Registered here rather than as Python custom ops: on the smallest
// calls the host is what takes the time (a training step of Z2 H4 N128 D64 spent 137 us in the
// Python op wrappers and the Python autograd function around 19 us of GPU work).
// ---------------------------------------------------------------------------------------------
using OptTensor = std::optional<at::Tensor>;

std::tuple<at::Tensor, at::Tensor> op_fwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                          double softmax_scale, bool causal, const OptTensor& seqused_q,
                                          const OptTensor& seqused_k) {
  auto r = fwd_impl(q, k, v, std::nullopt, softmax_scale, causal, false, seqused_q, seqused_k);
  return {std::move(r[0]), std::move(r[1])};
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> op_bwd(const at::Tensor& dout, const at::Tensor& q,
                                                      const at::Tensor& k, const at::Tensor& v,
                                                      const at::Tensor& out, const at::Tensor& softmax_lse,
                                                      double softmax_scale, bool causal,
                                                      const OptTensor& seqused_q, const OptTensor& seqused_k,
                                                      bool deterministic) {
  auto r = mha_bwd_lse(dout, q, k, v, out, softmax_lse, softmax_scale, causal, seqused_q, seqused_k,
                       deterministic);
  return {std::move(r[0]), std::move(r[1]), std::move(r[2])};
}

// Both calls go through the dispatcher, so that every mode that intercepts ops (fake tensors,
// tensor subclasses, tracing) still sees them.
std::tuple<at::Tensor, at::Tensor> call_fwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                            double softmax_scale, bool causal, const OptTensor& seqused_q,
                                            const OptTensor& seqused_k) {
  static const auto op = c10::Dispatcher::singleton()
                             .findSchemaOrThrow("flash_attn_v100::fwd", "")
                             .typed<decltype(op_fwd)>();
  return op.call(q, k, v, softmax_scale, causal, seqused_q, seqused_k);
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> call_bwd(const at::Tensor& dout, const at::Tensor& q,
                                                        const at::Tensor& k, const at::Tensor& v,
                                                        const at::Tensor& out, const at::Tensor& lse,
                                                        double softmax_scale, bool causal,
                                                        const OptTensor& seqused_q,
                                                        const OptTensor& seqused_k, bool deterministic) {
  static const auto op = c10::Dispatcher::singleton()
                             .findSchemaOrThrow("flash_attn_v100::bwd", "")
                             .typed<decltype(op_bwd)>();
  return op.call(dout, q, k, v, out, lse, softmax_scale, causal, seqused_q, seqused_k, deterministic);
}

at::Tensor last_dim_contiguous(const at::Tensor& t) {
  return t.dim() > 0 && t.stride(-1) != 1 ? t.contiguous() : t;
}

// The autograd node of flash_attn_func / flash_attn_padded_func (the Python class FlashAttnFunc
// is the same computation for code that torch.compile traces).
struct AttentionFunction : public torch::autograd::Function<AttentionFunction> {
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& q_, const at::Tensor& k_,
                            const at::Tensor& v_, const OptTensor& seqused_q, const OptTensor& seqused_k,
                            double softmax_scale, bool causal, bool deterministic) {
    at::AutoDispatchBelowADInplaceOrView guard;
    const at::Tensor q = last_dim_contiguous(q_), k = last_dim_contiguous(k_), v = last_dim_contiguous(v_);
    auto [out, lse] = call_fwd(q, k, v, softmax_scale, causal, seqused_q, seqused_k);
    ctx->save_for_backward({q, k, v, out, lse, seqused_q.value_or(at::Tensor()), seqused_k.value_or(at::Tensor())});
    ctx->saved_data["scale"] = softmax_scale;
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["deterministic"] = deterministic;
    return out;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    auto opt = [](const at::Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); };
    const double scale = ctx->saved_data["scale"].toDouble();
    const bool causal = ctx->saved_data["causal"].toBool();
    const bool deterministic = ctx->saved_data["deterministic"].toBool();
    const at::Tensor dout = last_dim_contiguous(grads[0]);
    auto call = [&]() {
      return call_bwd(dout, saved[0], saved[1], saved[2], saved[3], saved[4], scale, causal, opt(saved[5]),
                      opt(saved[6]), deterministic);
    };
    at::Tensor dq, dk, dv;
    if (at::GradMode::is_enabled()) {
      // create_graph: the op's own autograd entry records that it has no derivative
      std::tie(dq, dk, dv) = call();
    } else {
      at::AutoDispatchBelowADInplaceOrView guard;
      std::tie(dq, dk, dv) = call();
    }
    return {dq, dk, dv, at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor()};
  }
};

// flash_attn_func / flash_attn_padded_func outside of tracing
at::Tensor attention(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                     std::optional<double> softmax_scale, bool causal, const OptTensor& seqused_q,
                     const OptTensor& seqused_k, bool deterministic) {
  TORCH_CHECK(q.dim() > 0 && k.dim() > 0 && v.dim() > 0, "q, k and v must have shape (batch, seqlen, heads, head_size)");
  const double scale = softmax_scale.has_value() ? *softmax_scale : std::pow((double)q.size(-1), -0.5);
  // What autograd refuses has to be refused here, too: without gradients to record it is passed by.
  if (const auto& functorch = at::functorch::functorchTLSAccessor()) functorch->checkSupportsCppAutogradFunction();
  if (c10::AutogradState::get_tls_state().get_fw_grad_mode())
    for (const at::Tensor* t : {&q, &k, &v})
      TORCH_CHECK_NOT_IMPLEMENTED(!t->_fw_grad(/*level=*/0).defined(),
                                  "flash_attn_func has no forward-mode derivative (an input carries a tangent)");
  if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad()))
    return AttentionFunction::apply(q, k, v, seqused_q, seqused_k, scale, causal, deterministic);
  at::AutoDispatchBelowADInplaceOrView guard;
  return std::get<0>(call_fwd(last_dim_contiguous(q), last_dim_contiguous(k), last_dim_contiguous(v), scale,
                              causal, seqused_q, seqused_k));
}

}  // namespace

TORCH_LIBRARY(flash_attn_v100, m) {
  m.def("fwd(Tensor q, Tensor k, Tensor v, float softmax_scale, bool causal, Tensor? seqused_q=None, "
        "Tensor? seqused_k=None) -> (Tensor, Tensor)", {at::Tag::pt2_compliant_tag});
  m.def("bwd(Tensor dout, Tensor q, Tensor k, Tensor v, Tensor out, Tensor softmax_lse, float softmax_scale, "
        "bool causal, Tensor? seqused_q=None, Tensor? seqused_k=None, bool deterministic=False) -> (Tensor, "
        "Tensor, Tensor)", {at::Tag::pt2_compliant_tag});
}
TORCH_LIBRARY_IMPL(flash_attn_v100, CUDA, m) {
  m.impl("fwd", TORCH_FN(op_fwd));
  m.impl("bwd", TORCH_FN(op_bwd));
}
// the ops themselves have no derivative (the functions above do): differentiating through a direct
// call is an error, not a silent zero
TORCH_LIBRARY_IMPL(flash_attn_v100, Autograd, m) {
  m.impl("fwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("bwd", torch::autograd::autogradNotImplementedFallback());
}

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.doc() = "B200 (sm_100a) fused multi-head attention";
  // positional calls only, like the reference's pybind exports (kernel/fused_mha_api.cpp:166-167)
  m.def("fwd", &mha_fwd, "Forward pass: fwd(q, k, v, out|None, softmax_scale, is_causal)");
  m.def("fwd_lse", &mha_fwd_lse,
        "Forward pass returning [out, lse]: fwd_lse(q, k, v, out|None, softmax_scale, is_causal, "
        "seqused_q|None, seqused_k|None)");
  m.def("bwd_lse", &mha_bwd_lse,
        "Backward pass: bwd_lse(dout, q, k, v, out, lse, softmax_scale, is_causal, seqused_q|None, "
        "seqused_k|None, deterministic)");
  m.def("bwd", &mha_bwd,
        "Backward pass: bwd(dout, q, k, v, out, D|None, softmax_sum|None, softmax_max, dq|None, "
        "dk|None, dv|None, softmax_scale, is_causal)");
  m.def("attention", &attention,
        "Attention with autograd: attention(q, k, v, softmax_scale|None, causal, seqused_q|None, "
        "seqused_k|None, deterministic)");
  m.def("version", []() { return std::string(fmha_version()); });
}
