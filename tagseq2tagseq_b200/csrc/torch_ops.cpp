// PyTorch operators over the C ABI of libts2ts_attn.so.
//
// The host side of a call (argument checks, output and workspace allocation, autograd bookkeeping, the C call) is native:
// written as Python custom operators it cost 55 us per forward and 260 us per forward + backward, several times what
// the kernels of a short sequence take.  Nothing here computes; every operator ends in a ts2ts_* entry point, and there
// is no CPU implementation.
#include "../../include/ts2ts_attn.h"
#include "../../include/ts2ts_lm.h"

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include <array>
#include <tuple>
#include <vector>

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct Strides3 {
  int64_t s[3];
  explicit Strides3(const Tensor& t) : s{t.stride(0), t.stride(1), t.stride(2)} {}
};

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// -4 / -5 report misaligned or badly strided tensors: ValueError; everything else is a failed call.
void check(int code, const char* what) {
  if (code == 0) return;
  if (code == -4 || code == -5) TORCH_CHECK_VALUE(false, what, ": ", ts2ts_last_error_string());
  TORCH_CHECK(false, what, " failed with status ", code, ": ", ts2ts_last_error_string());
}

// The kernels need a unit stride in D and 16-byte aligned rows; anything else (expanded stride-0 views too: the TMA
// descriptors need positive strides) is copied once.
Tensor rowmajor(const Tensor& t) {
  bool fine = t.stride(3) == 1 && (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15u) == 0;
  for (int i = 0; i < 3; ++i) fine = fine && t.stride(i) > 0 && (t.stride(i) * 2) % 16 == 0;
  return fine ? t : t.contiguous();
}

void check_qkv(const Tensor& q, const Tensor& k, const Tensor& v) {
  TORCH_CHECK(q.is_cuda() && k.is_cuda() && v.is_cuda(), "ts2ts::masked_attn runs on CUDA tensors only (no CPU path exists)");
  TORCH_CHECK_TYPE(q.scalar_type() == at::kBFloat16 && k.scalar_type() == at::kBFloat16 && v.scalar_type() == at::kBFloat16,
                   "q, k, v must be bfloat16");
  TORCH_CHECK_VALUE(q.dim() == 4 && q.sizes() == k.sizes() && q.sizes() == v.sizes(), "q, k, v must share the shape [B,H,T,D]");
  TORCH_CHECK_VALUE(q.size(3) == 64 || q.size(3) == 128, "head dimension must be 64 or 128");
}

// Per-token mask inputs as the C ABI takes them; `keep` holds the contiguous tensors alive.
struct MaskPtrs {
  std::array<Tensor, 4> keep;
  const int32_t *doc = nullptr, *row = nullptr, *col = nullptr;
  const int64_t* link = nullptr;
  int R = 0, W = 0;
  MaskPtrs(const Tensor& doc_ids, const OptTensor& link_bits, const OptTensor& q_row_ids, const OptTensor& kv_col_ids) {
    keep[0] = doc_ids.contiguous();
    doc = keep[0].const_data_ptr<int32_t>();
    if (q_row_ids.has_value()) {
      keep[1] = q_row_ids->contiguous();
      row = keep[1].const_data_ptr<int32_t>();
    }
    if (kv_col_ids.has_value()) {
      keep[2] = kv_col_ids->contiguous();
      col = keep[2].const_data_ptr<int32_t>();
    }
    if (link_bits.has_value()) {
      keep[3] = link_bits->contiguous();
      link = keep[3].const_data_ptr<int64_t>();
      R = static_cast<int>(keep[3].size(1));
      W = static_cast<int>(keep[3].size(2));
    }
  }
};

// ------------------------------------------------------------------------------------------------ masked attention
std::tuple<Tensor, Tensor> attn_fwd_cuda(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& doc_ids,
                                         const OptTensor& link_bits, const OptTensor& q_row_ids, const OptTensor& kv_col_ids,
                                         const Tensor& plan, double scale) {
  check_qkv(q_, k_, v_);
  const c10::cuda::CUDAGuard guard(q_.device());
  const Tensor q = rowmajor(q_), k = rowmajor(k_), v = rowmajor(v_);
  const int B = q.size(0), H = q.size(1), T = q.size(2), D = q.size(3);
  Tensor out = at::empty({B, H, T, D}, q.options()), lse = at::empty({B, H, T}, q.options().dtype(at::kFloat));
  const MaskPtrs m(doc_ids, link_bits, q_row_ids, kv_col_ids);
  check(ts2ts_attn_fwd(q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), Strides3(q).s, Strides3(k).s, Strides3(v).s, B, H, T, D,
                       static_cast<float>(scale), m.doc, m.row, m.col, m.link, m.R, m.W, plan.const_data_ptr(), plan.numel(),
                       out.mutable_data_ptr(), Strides3(out).s, lse.mutable_data_ptr<float>(), stream_of(q)),
        "ts2ts_attn_fwd");
  return {out, lse};
}

std::tuple<Tensor, Tensor, Tensor> attn_bwd_cuda(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& out_,
                                                 const Tensor& dout_, const Tensor& lse, const Tensor& doc_ids, const OptTensor& link_bits,
                                                 const OptTensor& q_row_ids, const OptTensor& kv_col_ids, const Tensor& plan,
                                                 double scale) {
  const c10::cuda::CUDAGuard guard(q_.device());
  const Tensor q = rowmajor(q_), k = rowmajor(k_), v = rowmajor(v_), out = rowmajor(out_), dout = rowmajor(dout_);
  const int B = q.size(0), H = q.size(1), T = q.size(2), D = q.size(3);
  Tensor dq = rowmajor(at::empty_like(q)), dk = rowmajor(at::empty_like(k)), dv = rowmajor(at::empty_like(v));
  Tensor ws = at::empty({static_cast<int64_t>(ts2ts_attn_bwd_workspace_bytes(B, H, T, D))}, q.options().dtype(at::kByte));
  const MaskPtrs m(doc_ids, link_bits, q_row_ids, kv_col_ids);
  check(ts2ts_attn_bwd(q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), out.const_data_ptr(), dout.const_data_ptr(),
                       lse.const_data_ptr<float>(), Strides3(q).s, Strides3(k).s, Strides3(v).s, Strides3(out).s, Strides3(dout).s, B, H, T,
                       D, static_cast<float>(scale), m.doc, m.row, m.col, m.link, m.R, m.W, plan.const_data_ptr(), plan.numel(),
                       dq.mutable_data_ptr(), dk.mutable_data_ptr(), dv.mutable_data_ptr(), Strides3(dq).s, Strides3(dk).s, Strides3(dv).s,
                       ws.mutable_data_ptr(), ws.numel(), stream_of(q)),
        "ts2ts_attn_bwd");
  return {dq, dk, dv};
}

using FwdSig = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const OptTensor&, const OptTensor&,
                                          const OptTensor&, const Tensor&, double);
using BwdSig = std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                                  const Tensor&, const OptTensor&, const OptTensor&, const OptTensor&, const Tensor&, double);
const c10::TypedOperatorHandle<FwdSig>& fwd_op() {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("ts2ts::masked_attn_fwd", "").typed<FwdSig>();
  return op;
}
const c10::TypedOperatorHandle<BwdSig>& bwd_op() {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("ts2ts::masked_attn_bwd", "").typed<BwdSig>();
  return op;
}

OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; }

struct MaskedAttn : torch::autograd::Function<MaskedAttn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& doc_ids,
                               const OptTensor& link_bits, const OptTensor& q_row_ids, const OptTensor& kv_col_ids, const Tensor& plan,
                               double scale) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [out, lse] = fwd_op().call(q, k, v, doc_ids, link_bits, q_row_ids, kv_col_ids, plan, scale);
    ctx->save_for_backward({q, k, v, out, lse, doc_ids, link_bits.value_or(Tensor()), q_row_ids.value_or(Tensor()),
                            kv_col_ids.value_or(Tensor()), plan});
    ctx->saved_data["scale"] = scale;
    ctx->mark_non_differentiable({lse});
    ctx->set_materialize_grads(false);
    return {out, lse};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list r(9);
    if (!grads[0].defined()) return r;
    const auto s = ctx->get_saved_variables();
    auto [dq, dk, dv] = bwd_op().call(s[0], s[1], s[2], s[3], grads[0], s[4], s[5], opt(s[6]), opt(s[7]), opt(s[8]), s[9],
                                      ctx->saved_data["scale"].toDouble());
    r[0] = dq; r[1] = dk; r[2] = dv;
    return r;
  }
};

std::tuple<Tensor, Tensor> attn_fwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& doc_ids,
                                             const OptTensor& link_bits, const OptTensor& q_row_ids, const OptTensor& kv_col_ids,
                                             const Tensor& plan, double scale) {
  if (!at::GradMode::is_enabled() || !(q.requires_grad() || k.requires_grad() || v.requires_grad())) {
    at::AutoDispatchBelowADInplaceOrView below;
    return fwd_op().call(q, k, v, doc_ids, link_bits, q_row_ids, kv_col_ids, plan, scale);
  }
  auto r = MaskedAttn::apply(q, k, v, doc_ids, link_bits, q_row_ids, kv_col_ids, plan, scale);
  return {r[0], r[1]};
}

std::tuple<Tensor, Tensor> attn_decode_cuda(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& doc_ids,
                                            const OptTensor& link_bits, const OptTensor& q_row_ids, const OptTensor& kv_col_ids,
                                            const OptTensor& q_pos, double scale) {
  const c10::cuda::CUDAGuard guard(q_.device());
  const Tensor q = rowmajor(q_), k = rowmajor(k_), v = rowmajor(v_);
  const int B = k.size(0), H = k.size(1), Tk = k.size(2), D = k.size(3);
  Tensor out = at::empty({B, H, 1, D}, q.options()), lse = at::empty({B, H}, q.options().dtype(at::kFloat));
  Tensor ws = at::empty({static_cast<int64_t>(ts2ts_attn_decode_workspace_bytes(B, H, Tk, D))}, q.options().dtype(at::kByte));
  const MaskPtrs m(doc_ids, link_bits, q_row_ids, kv_col_ids);
  const Tensor pos = q_pos.has_value() ? q_pos->contiguous() : Tensor();
  check(ts2ts_attn_decode(q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), Strides3(q).s, Strides3(k).s, Strides3(v).s, B, H, Tk,
                          D, static_cast<float>(scale), m.doc, m.row, m.col, m.link, m.R, m.W,
                          pos.defined() ? pos.const_data_ptr<int32_t>() : nullptr, out.mutable_data_ptr(), Strides3(out).s,
                          lse.mutable_data_ptr<float>(), ws.mutable_data_ptr(), ws.numel(), stream_of(q)),
        "ts2ts_attn_decode");
  return {out, lse};
}

// ------------------------------------------------------------------------------------------------ block plan
// {plan} or {plan, state, kv_cnt, kv_idx, full_cnt, full_idx, q_cnt, q_idx, full_q_cnt, full_q_idx}.
std::vector<Tensor> block_map_cuda(const Tensor& doc_ids, const OptTensor& link_bits, const OptTensor& q_row_ids,
                                   const OptTensor& kv_col_ids, bool with_lists) {
  const c10::cuda::CUDAGuard guard(doc_ids.device());
  const int B = doc_ids.size(0), T = doc_ids.size(1);
  const int64_t nb = (T + TS2TS_TILE - 1) / TS2TS_TILE;
  const auto bytes = doc_ids.options().dtype(at::kByte), ints = doc_ids.options();
  std::vector<Tensor> r;
  r.push_back(at::empty({static_cast<int64_t>(ts2ts_plan_bytes(B, T))}, bytes));
  std::array<int32_t*, 8> lists{};
  uint8_t* state = nullptr;
  if (with_lists) {
    r.push_back(at::empty({B, nb, nb}, bytes));
    state = r[1].mutable_data_ptr<uint8_t>();
    for (int i = 0; i < 8; ++i) {
      r.push_back(i % 2 == 0 ? at::empty({B, nb}, ints) : at::empty({B, nb, nb}, ints));
      lists[i] = r.back().mutable_data_ptr<int32_t>();
    }
  }
  const MaskPtrs m(doc_ids, link_bits, q_row_ids, kv_col_ids);
  check(ts2ts_block_map(m.doc, m.row, m.col, m.link, B, T, m.R, m.W, r[0].mutable_data_ptr(), r[0].numel(), state, lists[0], lists[1],
                        lists[2], lists[3], lists[4], lists[5], lists[6], lists[7], stream_of(doc_ids)),
        "ts2ts_block_map");
  return r;
}

}  // namespace

TORCH_LIBRARY(ts2ts, m) {
  m.def("masked_attn_fwd(Tensor q, Tensor k, Tensor v, Tensor doc_ids, Tensor? link_bits, Tensor? q_row_ids, Tensor? kv_col_ids, "
        "Tensor plan, float scale) -> (Tensor, Tensor)");
  m.def("masked_attn_bwd(Tensor q, Tensor k, Tensor v, Tensor out, Tensor dout, Tensor lse, Tensor doc_ids, Tensor? link_bits, "
        "Tensor? q_row_ids, Tensor? kv_col_ids, Tensor plan, float scale) -> (Tensor, Tensor, Tensor)");
  m.def("masked_attn_decode(Tensor q, Tensor k_cache, Tensor v_cache, Tensor doc_ids, Tensor? link_bits, Tensor? q_row_ids, "
        "Tensor? kv_col_ids, Tensor? q_pos, float scale) -> (Tensor, Tensor)");
  m.def("block_map(Tensor doc_ids, Tensor? link_bits, Tensor? q_row_ids, Tensor? kv_col_ids, bool with_lists) -> Tensor[]");
}
TORCH_LIBRARY_IMPL(ts2ts, CUDA, m) {
  m.impl("masked_attn_fwd", attn_fwd_cuda);
  m.impl("masked_attn_bwd", attn_bwd_cuda);
  m.impl("masked_attn_decode", attn_decode_cuda);
  m.impl("block_map", block_map_cuda);
}
TORCH_LIBRARY_IMPL(ts2ts, Autograd, m) { m.impl("masked_attn_fwd", attn_fwd_autograd); }
