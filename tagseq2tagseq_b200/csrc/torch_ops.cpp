// PyTorch operators over the C ABI of libts2ts_attn.so.
//
// The host side of a call (argument checks, output and workspace allocation, autograd bookkeeping, the C call) is native:
// written as Python custom operators it cost 55 us per forward and 260 us per forward + backward, several times what
// the kernels of a short sequence take.  Nothing here computes; every operator ends in a ts2ts_* entry point, and there
// is no CPU implementation.
#include "../../include/ts2ts_attn.h"
#include "../../include/ts2ts_lm.h"

#include <ATen/ATen.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/library.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <string>
#include <tuple>
#include <unordered_map>
#include <utility>
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
  const MaskPtrs m(doc_ids, link_bits, q_row_ids, kv_col_ids);
  const Tensor pos = q_pos.has_value() ? q_pos->contiguous() : Tensor();
  check(ts2ts_attn_decode(q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), Strides3(q).s, Strides3(k).s, Strides3(v).s, B, H, Tk,
                          D, static_cast<float>(scale), m.doc, m.row, m.col, m.link, m.R, m.W,
                          pos.defined() ? pos.const_data_ptr<int32_t>() : nullptr, out.mutable_data_ptr(), Strides3(out).s,
                          lse.mutable_data_ptr<float>(), nullptr, 0, stream_of(q)),
        "ts2ts_attn_decode");
  return {out, lse};
}

// The backward and the decoding step have no derivative: differentiating through their results raises, where an operator
// without an autograd kernel would leave the gradient out.
void refuse_gradient(const char* name, at::ArrayRef<Tensor> inputs, std::initializer_list<Tensor*> results) {
  if (!at::GradMode::is_enabled() || std::none_of(inputs.begin(), inputs.end(), [](const Tensor& t) { return t.defined() && t.requires_grad(); })) return;
  std::shared_ptr<torch::autograd::Node> fn(new torch::autograd::NotImplemented(name), torch::autograd::deleteNode);
  fn->set_next_edges(torch::autograd::collect_next_edges(inputs));
  for (Tensor* t : results)
    if (t->defined()) torch::autograd::set_history(*t, fn);
}

std::tuple<Tensor, Tensor, Tensor> attn_bwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out,
                                                     const Tensor& dout, const Tensor& lse, const Tensor& doc_ids,
                                                     const OptTensor& link_bits, const OptTensor& q_row_ids, const OptTensor& kv_col_ids,
                                                     const Tensor& plan, double scale) {
  std::tuple<Tensor, Tensor, Tensor> r;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    r = bwd_op().call(q, k, v, out, dout, lse, doc_ids, link_bits, q_row_ids, kv_col_ids, plan, scale);
  }
  refuse_gradient("ts2ts::masked_attn_bwd", {q, k, v, out, dout, lse}, {&std::get<0>(r), &std::get<1>(r), &std::get<2>(r)});
  return r;
}

std::tuple<Tensor, Tensor> attn_decode_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& doc_ids,
                                                const OptTensor& link_bits, const OptTensor& q_row_ids, const OptTensor& kv_col_ids,
                                                const OptTensor& q_pos, double scale) {
  using Sig = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const OptTensor&, const OptTensor&,
                                         const OptTensor&, const OptTensor&, double);
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("ts2ts::masked_attn_decode", "").typed<Sig>();
  std::tuple<Tensor, Tensor> r;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    r = op.call(q, k, v, doc_ids, link_bits, q_row_ids, kv_col_ids, q_pos, scale);
  }
  refuse_gradient("ts2ts::masked_attn_decode", {q, k, v}, {&std::get<0>(r), &std::get<1>(r)});
  return r;
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

// ------------------------------------------------------------------------------------------------ link scan
// Candidate links of a token sequence and the tokens of their targets, on the host: ({mid, start, close} int32 [n,3], the
// targets' tokens mid+1 .. close of all links one after the other, int64).  Candidates and tokens come back together in
// one wait; sequences too long for that to be cheap fetch the tokens between the first and the last link afterwards.
constexpr int64_t kTokensAlong = 65536;

std::tuple<Tensor, Tensor> link_candidates(const Tensor& input_ids, int64_t mid_id, at::IntArrayRef start_ids, const Tensor& close_flags,
                                           int64_t back_limit, int64_t window) {
  const c10::cuda::CUDAGuard guard(input_ids.device());
  const auto stream = c10::cuda::getCurrentCUDAStream(input_ids.device().index());
  const Tensor tokens = input_ids.contiguous();
  const int64_t T = tokens.size(0);
  const int bytes = static_cast<int>(tokens.element_size());
  const auto dev32 = tokens.options().dtype(at::kInt), host32 = at::TensorOptions().dtype(at::kInt).pinned_memory(true);
  Tensor scratch = at::empty({static_cast<int64_t>(ts2ts_detect_links_scratch_bytes(static_cast<int>(T)))}, dev32.dtype(at::kByte));
  Tensor host, host_tokens;
  int64_t max_links = 1024, n = 0, first = 0;
  if (T <= kTokensAlong) {
    host_tokens = at::empty({T}, host32.dtype(tokens.scalar_type()));
    host_tokens.copy_(tokens, /*non_blocking=*/true);
  }
  for (;;) {  // a second turn only when the sequence holds more candidates than the first buffer
    Tensor out = at::empty({4 + 3 * max_links}, dev32);  // count, padding, triples
    int32_t* o = out.mutable_data_ptr<int32_t>();
    check(ts2ts_detect_links(tokens.const_data_ptr(), bytes, static_cast<int>(T), mid_id, start_ids.data(), static_cast<int>(start_ids.size()),
                             close_flags.const_data_ptr<uint8_t>(), static_cast<int>(close_flags.size(0)), static_cast<int>(back_limit),
                             static_cast<int>(window), scratch.mutable_data_ptr(), scratch.numel(), o + 4, static_cast<int>(max_links), o,
                             stream.stream()),
          "ts2ts_detect_links");
    host = at::empty({out.numel()}, host32);
    host.copy_(out, /*non_blocking=*/true);
    stream.synchronize();
    n = host.const_data_ptr<int32_t>()[0];
    if (n <= max_links) break;
    max_links = n;
  }
  const int32_t* tri = host.const_data_ptr<int32_t>() + 4;
  Tensor links = at::empty({n, 3}, at::kInt);
  std::copy(tri, tri + 3 * n, links.mutable_data_ptr<int32_t>());
  int64_t total = 0, last = 0;
  for (int64_t i = 0; i < n; ++i) {
    total += tri[3 * i + 2] - tri[3 * i];
    last = std::max<int64_t>(last, tri[3 * i + 2]);
  }
  if (n > 0 && !host_tokens.defined()) {
    first = tri[0] + 1;  // candidates ascend
    host_tokens = tokens.slice(0, first, last + 1).cpu();
  }
  Tensor targets = at::empty({total}, at::kLong);
  int64_t* dst = targets.mutable_data_ptr<int64_t>();
  for (int64_t i = 0; i < n; ++i)
    for (int64_t t = tri[3 * i] + 1; t <= tri[3 * i + 2]; ++t)
      *dst++ = bytes == 8 ? host_tokens.const_data_ptr<int64_t>()[t - first] : host_tokens.const_data_ptr<int32_t>()[t - first];
  return {links, targets};
}

// ------------------------------------------------------------------------------------------------ masks from spans and links
// Tokens covered by the same set of intervals form one class.  The set only changes where an interval starts or ends, so
// there are at most 2 G + 1 segments however long the sequence is.  `bounds` [S+1] and `ids` [S] (-1: no interval);
// classes are numbered in order of first appearance, `sets` holds their member bits, `words` 64-bit words each.
struct Segments {
  std::vector<int32_t> bounds, ids;
  std::vector<uint64_t> sets;
  int classes = 0;
  static uint64_t mixed(uint64_t x) {  // spreads small numbers over 64 bits: two odd multipliers and shifts
    x *= 0x9e3779b97f4a7c15ull;
    x ^= x >> 29;
    x *= 0xd6e8feb86659fd93ull;
    return x ^ (x >> 32);
  }
  Segments(const std::vector<std::pair<int64_t, int64_t>>& ranges, size_t words) {
    struct Event { int64_t at; int32_t who; bool opens; };
    std::vector<Event> ev;
    ev.reserve(2 * ranges.size());
    for (size_t g = 0; g < ranges.size(); ++g) {
      ev.push_back({ranges[g].first, static_cast<int32_t>(g), true});
      ev.push_back({ranges[g].second, static_cast<int32_t>(g), false});
    }
    std::sort(ev.begin(), ev.end(), [](const Event& a, const Event& b) { return a.at < b.at; });
    std::vector<uint64_t> now(words, 0);
    size_t places = 16;
    while (places < 2 * ev.size()) places *= 2;
    std::vector<int32_t> seen(places, -1);  // class by the hash of its set, the next free place on a clash
    uint64_t hash = 0;
    int64_t open = 0;
    for (size_t i = 0; i < ev.size();) {
      const int64_t at = ev[i].at;
      for (; i < ev.size() && ev[i].at == at; ++i) {
        now[ev[i].who >> 6] ^= uint64_t(1) << (ev[i].who & 63);
        hash ^= mixed(static_cast<uint64_t>(ev[i].who) + 1);
        open += ev[i].opens ? 1 : -1;
      }
      bounds.push_back(static_cast<int32_t>(at));
      if (i == ev.size()) break;
      if (open == 0) {
        ids.push_back(-1);
        continue;
      }
      size_t at_place = hash & (places - 1);
      while (seen[at_place] >= 0 && !std::equal(now.begin(), now.end(), sets.begin() + seen[at_place] * words)) at_place = (at_place + 1) & (places - 1);
      if (seen[at_place] < 0) {
        seen[at_place] = classes++;
        sets.insert(sets.end(), now.begin(), now.end());
      }
      ids.push_back(seen[at_place]);
    }
    if (bounds.empty()) bounds.push_back(0);
  }
};

// {doc_ids [1,T]} or {doc_ids, link_bits [1,R,W], q_row_ids, kv_col_ids} of a pack: spans (start, end, doc id) as they come,
// links as (position, target doc id) in the order in which they receive grants.  A link at `pos` of the first span with
// start < pos <= end grants tokens [pos, end) the first span of its target; empty grants take no place, and the first one
// beyond `cap` ends the list (cross_doc_mask.py:239-294).  The host works on segment tables, which reach the device in one
// copy with the link bits; one kernel per id array spreads them over the tokens.
std::vector<Tensor> pack_mask(at::IntArrayRef starts, at::IntArrayRef ends, at::IntArrayRef ids, at::IntArrayRef link_pos,
                              at::IntArrayRef link_target, int64_t T, int64_t cap, c10::Device device) {
  const size_t n_spans = starts.size();
  TORCH_CHECK_VALUE(ends.size() == n_spans && ids.size() == n_spans && link_pos.size() == link_target.size(), "pack_mask: lists of equal length");
  for (size_t i = 0; i < n_spans; ++i)  // ids of spans that cover a token are stored in 32 bits
    TORCH_CHECK_VALUE(std::max<int64_t>(0, starts[i]) >= std::min(T, ends[i]) || ids[i] == static_cast<int32_t>(ids[i]),
                      "pack_mask: document id ", ids[i], " does not fit 32 bits");
  if (!device.has_index()) device = c10::Device(c10::kCUDA, c10::cuda::current_device());
  const c10::cuda::CUDAGuard guard(device);
  std::unordered_map<int64_t, size_t> by_id;
  for (size_t i = 0; i < n_spans; ++i) by_id.try_emplace(ids[i], i);
  std::vector<std::pair<int64_t, int64_t>> q, k;
  int64_t src_pos = 0, src_end = 0;  // the source of the last position, if it has one
  bool has_src = false;
  for (size_t l = 0; l < link_pos.size() && static_cast<int64_t>(q.size()) < cap; ++l) {
    const int64_t pos = link_pos[l];
    if (l == 0 || pos != src_pos) {
      src_pos = pos;
      has_src = false;
      for (size_t i = 0; i < n_spans; ++i)
        if (starts[i] < pos && pos <= ends[i]) {
          has_src = true;
          src_end = ends[i];
          break;
        }
    }
    const auto it = by_id.find(link_target[l]);
    if (!has_src || it == by_id.end()) continue;
    const int64_t q1 = std::min(T, src_end), k0 = std::max<int64_t>(0, starts[it->second]), k1 = std::min(T, ends[it->second]);
    if (pos < q1 && k0 < k1) {
      q.emplace_back(pos, q1);
      k.emplace_back(k0, k1);
    }
  }
  // documents: later spans overwrite earlier ones, uncovered tokens are -1
  std::vector<int32_t> db;
  for (size_t i = 0; i < n_spans; ++i) {
    const int64_t a = std::max<int64_t>(0, starts[i]), b = std::min(T, ends[i]);
    if (a < b) {
      db.push_back(static_cast<int32_t>(a));
      db.push_back(static_cast<int32_t>(b));
    }
  }
  std::sort(db.begin(), db.end());
  db.erase(std::unique(db.begin(), db.end()), db.end());
  if (db.empty()) db.push_back(0);
  std::vector<int32_t> di(db.size() - 1, -1);
  for (size_t i = 0; i < n_spans; ++i) {
    const int64_t a = std::max<int64_t>(0, starts[i]), b = std::min(T, ends[i]);
    if (a < b)
      for (auto at = std::lower_bound(db.begin(), db.end(), static_cast<int32_t>(a)); *at < b; ++at) di[at - db.begin()] = static_cast<int32_t>(ids[i]);
  }
  const size_t words = (q.size() + 63) / 64;
  const Segments qs(q, words), ks(k, words);
  const int64_t R = std::max(1, qs.classes), W = std::max(1, (ks.classes + 63) / 64);
  const bool linked = !q.empty();
  // staging: link bits, then the tables (bounds, ids) of documents, rows and columns
  const std::vector<int32_t>* tables[6] = {&db, &di, &qs.bounds, &qs.ids, &ks.bounds, &ks.ids};
  const int n_tables = linked ? 6 : 2;
  int64_t ints = linked ? 2 * R * W : 0, at[6];
  for (int i = 0; i < n_tables; ++i) {
    at[i] = ints;
    ints += static_cast<int64_t>(tables[i]->size());
  }
  const auto dev = at::TensorOptions().dtype(at::kInt).device(device);
  Tensor stage = at::empty({ints}, at::TensorOptions().dtype(at::kInt).pinned_memory(true)), table = at::empty({ints}, dev);
  int32_t* st = stage.mutable_data_ptr<int32_t>();
  for (int i = 0; i < n_tables; ++i) std::copy(tables[i]->begin(), tables[i]->end(), st + at[i]);
  if (linked) {
    uint64_t* bits = reinterpret_cast<uint64_t*>(st);
    std::fill(bits, bits + R * W, 0);
    // which column classes hold a grant's tokens; a row class may read those of its grants
    std::vector<uint64_t> readers(q.size() * W, 0);
    auto members = [&](const uint64_t* set, auto visit) {
      for (size_t w = 0; w < words; ++w)
        for (uint64_t left = set[w]; left != 0; left &= left - 1) visit(64 * w + __builtin_ctzll(left));
    };
    for (int c = 0; c < ks.classes; ++c)
      members(&ks.sets[c * words], [&](size_t g) { readers[g * W + (c >> 6)] |= uint64_t(1) << (c & 63); });
    for (int r = 0; r < qs.classes; ++r)
      members(&qs.sets[r * words], [&](size_t g) {
        for (int64_t w = 0; w < W; ++w) bits[r * W + w] |= readers[g * W + w];
      });
  }
  table.copy_(stage, /*non_blocking=*/true);
  std::vector<Tensor> r;
  const int32_t* d = table.const_data_ptr<int32_t>();
  auto spread = [&](int i) {
    Tensor out = at::empty({1, T}, dev);
    if (T == 0) return out;
    check(ts2ts_segment_ids(d + at[i], d + at[i + 1], static_cast<int>(tables[i + 1]->size()), static_cast<int>(T), out.mutable_data_ptr<int32_t>(),
                            stream_of(out)),
          "ts2ts_segment_ids");
    return out;
  };
  r.push_back(spread(0));
  if (linked) {
    r.push_back(table.slice(0, 0, 2 * R * W).view(at::kLong).view({1, R, W}));
    r.push_back(spread(2));
    r.push_back(spread(4));
  }
  return r;
}

// ------------------------------------------------------------------------------------------------ decoder layer
// Autograd functions around the decoder-layer entry points.  Gradients nobody asked for arrive undefined
// (set_materialize_grads(false)) instead of as zero tensors of the activation's size.  The kernels' gradients have no
// derivative of their own: made with create_graph they refuse to be differentiated.
using c10::cuda::CUDAGuard;

// An autograd worker that has made no CUDA call yet has no current context, and cuBLAS asks for one.
void bind_context(const Tensor& t) { C10_CUDA_CHECK(c10::cuda::SetDevice(t.device().index(), true)); }
void need_cuda(const Tensor& t) {
  TORCH_CHECK(t.is_cuda(), "the decoder-layer kernels run on CUDA tensors only (no CPU path exists)");
}
const float* fptr(const Tensor& t) { return t.const_data_ptr<float>(); }
float* mfptr(const Tensor& t) { return t.mutable_data_ptr<float>(); }

struct AddRMSNorm : torch::autograd::Function<AddRMSNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x_in, const OptTensor& a_in, const Tensor& w_in, double eps) {
    TORCH_CHECK_VALUE(x_in.size(-1) > 0, "add_rmsnorm: x has no columns");
    TORCH_CHECK_VALUE(w_in.numel() >= x_in.size(-1) && (!a_in.has_value() || a_in->numel() >= x_in.numel()),
                      "add_rmsnorm: a has the size of x, w one element per column");
    need_cuda(x_in);
    TORCH_CHECK_TYPE(x_in.scalar_type() == at::kFloat && w_in.scalar_type() == at::kFloat && (!a_in.has_value() || a_in->scalar_type() == at::kBFloat16),
                     "add_rmsnorm: x and w are fp32, a is bf16");
    at::AutoDispatchBelowADInplaceOrView below;
    const CUDAGuard guard(x_in.device());
    const Tensor x = x_in.contiguous(), a = a_in.has_value() ? a_in->contiguous() : Tensor(), w = w_in.contiguous();
    const int64_t C = x.size(-1), N = x.numel() / C;
    Tensor x_out = at::empty_like(x), h = at::empty(x.sizes(), x.options().dtype(at::kBFloat16)), rstd = at::empty({N}, x.options());
    check(ts2ts_add_rmsnorm_fwd(fptr(x), a.defined() ? a.const_data_ptr() : nullptr, fptr(w), mfptr(x_out), h.mutable_data_ptr(), mfptr(rstd),
                                N, static_cast<int>(C), static_cast<float>(eps), stream_of(x)),
          "ts2ts_add_rmsnorm_fwd");
    ctx->save_for_backward({x_out, w, rstd});
    ctx->saved_data["has_a"] = a.defined();
    ctx->set_materialize_grads(false);
    return {x_out, h};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &w = s[1], &rstd = s[2];
    const CUDAGuard guard(x.device());
    const int64_t C = x.size(-1), N = x.numel() / C;
    const bool has_a = ctx->saved_data["has_a"].toBool();
    const auto bf16 = x.options().dtype(at::kBFloat16);
    const Tensor dh = grads[1].defined() ? grads[1].contiguous() : at::zeros(x.sizes(), bf16);  // h had no user
    const Tensor up = grads[0].defined() ? grads[0].contiguous() : Tensor();
    Tensor dx = at::empty_like(x), da = has_a ? at::empty(x.sizes(), bf16) : Tensor(), dw = w.numel() == C ? at::empty_like(w) : at::zeros_like(w);
    Tensor ws = at::empty({static_cast<int64_t>(ts2ts_add_rmsnorm_bwd_workspace_bytes(N, static_cast<int>(C)))}, x.options().dtype(at::kByte));
    check(ts2ts_add_rmsnorm_bwd_set(dh.const_data_ptr(), up.defined() ? fptr(up) : nullptr, fptr(x), fptr(w), fptr(rstd), mfptr(dx),
                                has_a ? da.mutable_data_ptr() : nullptr, mfptr(dw), ws.mutable_data_ptr(), ws.numel(), N, static_cast<int>(C),
                                stream_of(x)),
          "ts2ts_add_rmsnorm_bwd_set");
    refuse_gradient("ts2ts::add_rmsnorm backward", {grads[0], grads[1], x, w}, {&dx, &da, &dw});
    return {dx, da, dw, Tensor()};
  }
};
std::tuple<Tensor, Tensor> add_rmsnorm(const Tensor& x, const OptTensor& a, const Tensor& w, double eps) {
  auto r = AddRMSNorm::apply(x, a, w, eps);
  return {r[0], r[1]};
}

// Element strides (batch, head, token) of q, k or v inside a packed [B,T,3,H,D] buffer, and of a [B,T,H,D] one.
struct PackedStrides {
  int64_t s[3];
  PackedStrides(int64_t T, int64_t parts, int64_t H, int64_t D) : s{T * parts * H * D, D, parts * H * D} {}
};

// qkv [B,T,3*H*D] (the fused projection's output) -> attention output [B,T,H*D].  q and k are rotated in place; the
// attention kernels read q, k, v and write the output, and later dq, dk, dv, through strides of the packed buffers, so no
// tensor is transposed, split or concatenated in memory.
struct QKVAttention : torch::autograd::Function<QKVAttention> {
  static variable_list forward(AutogradContext* ctx, Tensor qkv, const Tensor& cos, const Tensor& sin, const Tensor& doc_ids,
                               const OptTensor& link_bits, const OptTensor& q_row_ids, const OptTensor& kv_col_ids, const Tensor& plan,
                               int64_t n_heads, int64_t head_dim) {
    const int64_t angles = qkv.dim() == 3 ? qkv.size(1) * (head_dim / 2) : 0;
    for (const Tensor* t : {&cos, &sin})
      TORCH_CHECK_VALUE(t->numel() >= angles && t->is_contiguous(), "qkv_attention: cos and sin must be contiguous [T, head_dim / 2]");
    for (const Tensor& t : {doc_ids, q_row_ids.value_or(doc_ids), kv_col_ids.value_or(doc_ids)})
      TORCH_CHECK_VALUE(qkv.dim() != 3 || t.numel() >= qkv.size(0) * qkv.size(1), "qkv_attention: the mask must have an id per token of qkv");
    need_cuda(qkv);
    TORCH_CHECK_TYPE(qkv.scalar_type() == at::kBFloat16 && qkv.is_contiguous(), "qkv_attention: qkv must be a contiguous bf16 tensor");
    TORCH_CHECK_VALUE(qkv.dim() == 3 && qkv.size(2) == 3 * n_heads * head_dim, "qkv_attention: last dimension must be 3 * n_heads * head_dim");
    at::AutoDispatchBelowADInplaceOrView below;
    const CUDAGuard guard(qkv.device());
    const int B = qkv.size(0), T = qkv.size(1), H = n_heads, D = head_dim;
    void* stream = stream_of(qkv);
    check(ts2ts_rope_qk_inplace(qkv.mutable_data_ptr(), fptr(cos), fptr(sin), B, T, H, D, 1.f, stream), "ts2ts_rope_qk_inplace");
    ctx->mark_dirty({qkv});
    Tensor out = at::empty({B, T, n_heads * head_dim}, qkv.options()), lse = at::empty({B, H, T}, qkv.options().dtype(at::kFloat));
    const PackedStrides in(T, 3, H, D), os(T, 1, H, D);
    const char* base = static_cast<const char*>(qkv.const_data_ptr());
    const int64_t part = 2 * n_heads * head_dim;  // bytes from q to k to v of a token
    const float scale = 1.f / std::sqrt(static_cast<float>(D));
    const MaskPtrs m(doc_ids, link_bits, q_row_ids, kv_col_ids);
    check(ts2ts_attn_fwd(base, base + part, base + 2 * part, in.s, in.s, in.s, B, H, T, D, scale, m.doc, m.row, m.col, m.link, m.R, m.W,
                         plan.const_data_ptr(), plan.numel(), out.mutable_data_ptr(), os.s, mfptr(lse), stream),
          "ts2ts_attn_fwd");
    ctx->save_for_backward({qkv, out, lse, cos, sin, doc_ids, link_bits.value_or(Tensor()), q_row_ids.value_or(Tensor()),
                            kv_col_ids.value_or(Tensor()), plan});
    ctx->saved_data["H"] = n_heads;
    ctx->set_materialize_grads(false);
    return {out, qkv};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list r(10);
    if (!grads[0].defined()) return r;
    const auto s = ctx->get_saved_variables();
    const Tensor &qkv = s[0], &out = s[1], &lse = s[2], &cos = s[3], &sin = s[4], &plan = s[9];
    const CUDAGuard guard(qkv.device());
    const int64_t n_heads = ctx->saved_data["H"].toInt(), head_dim = qkv.size(2) / (3 * n_heads);
    const int B = qkv.size(0), T = qkv.size(1), H = n_heads, D = head_dim;
    void* stream = stream_of(qkv);
    const Tensor dout = grads[0].contiguous();
    Tensor dqkv = at::empty_like(qkv);
    Tensor ws = at::empty({static_cast<int64_t>(ts2ts_attn_bwd_workspace_bytes(B, H, T, D))}, qkv.options().dtype(at::kByte));
    const PackedStrides in(T, 3, H, D), os(T, 1, H, D);
    const char* base = static_cast<const char*>(qkv.const_data_ptr());
    char* dbase = static_cast<char*>(dqkv.mutable_data_ptr());
    const int64_t part = 2 * n_heads * head_dim;
    const MaskPtrs m(s[5], opt(s[6]), opt(s[7]), opt(s[8]));
    check(ts2ts_attn_bwd(base, base + part, base + 2 * part, out.const_data_ptr(), dout.const_data_ptr(), fptr(lse), in.s, in.s, in.s, os.s,
                         os.s, B, H, T, D, 1.f / std::sqrt(static_cast<float>(D)), m.doc, m.row, m.col, m.link, m.R, m.W, plan.const_data_ptr(),
                         plan.numel(), dbase, dbase + part, dbase + 2 * part, in.s, in.s, in.s, ws.mutable_data_ptr(), ws.numel(), stream),
          "ts2ts_attn_bwd");
    // gradient of the rotated q, k -> gradient of the projection's output: the inverse rotation, in place
    check(ts2ts_rope_qk_inplace(dqkv.mutable_data_ptr(), fptr(cos), fptr(sin), B, T, H, D, -1.f, stream), "ts2ts_rope_qk_inplace");
    refuse_gradient("ts2ts::qkv_attention backward", {grads[0], qkv}, {&dqkv});
    r[0] = dqkv;
    return r;
  }
};
Tensor qkv_attention(Tensor qkv, const Tensor& cos, const Tensor& sin, const Tensor& doc_ids, const OptTensor& link_bits,
                     const OptTensor& q_row_ids, const OptTensor& kv_col_ids, const Tensor& plan, int64_t n_heads, int64_t head_dim) {
  return QKVAttention::apply(qkv, cos, sin, doc_ids, link_bits, q_row_ids, kv_col_ids, plan, n_heads, head_dim)[0];
}

struct SwiGLU : torch::autograd::Function<SwiGLU> {
  static Tensor forward(AutogradContext* ctx, const Tensor& gate_up) {
    // an odd row has no halves: its rows would be taken to begin earlier and earlier, and to be more than there are
    TORCH_CHECK_VALUE(gate_up.size(-1) > 0 && gate_up.size(-1) % 2 == 0, "swiglu: the last dimension must be even and not empty");
    need_cuda(gate_up);
    TORCH_CHECK_TYPE(gate_up.scalar_type() == at::kBFloat16, "swiglu: bf16 input");
    at::AutoDispatchBelowADInplaceOrView below;
    const CUDAGuard guard(gate_up.device());
    const Tensor gu = gate_up.contiguous();
    const int64_t F = gu.size(-1) / 2, N = gu.numel() / (2 * F);
    auto shape = gu.sizes().vec();
    shape.back() = F;
    Tensor act = at::empty(shape, gu.options());
    check(ts2ts_swiglu_fwd(gu.const_data_ptr(), act.mutable_data_ptr(), N, static_cast<int>(F), stream_of(gu)), "ts2ts_swiglu_fwd");
    ctx->save_for_backward({gu});
    return act;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor gu = ctx->get_saved_variables()[0], dact = grads[0].contiguous();
    const CUDAGuard guard(gu.device());
    const int64_t F = gu.size(-1) / 2, N = gu.numel() / (2 * F);
    Tensor dgu = at::empty_like(gu);
    check(ts2ts_swiglu_bwd(gu.const_data_ptr(), dact.const_data_ptr(), dgu.mutable_data_ptr(), N, static_cast<int>(F), stream_of(gu)), "ts2ts_swiglu_bwd");
    refuse_gradient("ts2ts::swiglu backward", {grads[0], gu}, {&dgu});
    return {dgu};
  }
};
Tensor swiglu(const Tensor& gate_up) { return SwiGLU::apply(gate_up); }

struct CrossEntropy : torch::autograd::Function<CrossEntropy> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& target_in) {
    TORCH_CHECK_VALUE(logits.dim() != 2 || target_in.numel() >= logits.size(0), "cross_entropy: one target per row of logits");
    need_cuda(logits);
    TORCH_CHECK_TYPE(logits.scalar_type() == at::kBFloat16 && logits.dim() == 2 && logits.is_contiguous(),
                     "cross_entropy: logits must be a contiguous bf16 [N,V] tensor");
    at::AutoDispatchBelowADInplaceOrView below;
    const CUDAGuard guard(logits.device());
    const Tensor target = target_in.to(at::kLong).contiguous();
    const int64_t N = logits.size(0), V = logits.size(1);
    Tensor lse = at::empty({N}, logits.options().dtype(at::kFloat)), loss = at::empty({N}, lse.options());
    check(ts2ts_ce_fwd(logits.const_data_ptr(), target.const_data_ptr<int64_t>(), mfptr(lse), mfptr(loss), N, static_cast<int>(V), stream_of(logits)),
          "ts2ts_ce_fwd");
    ctx->save_for_backward({logits, target, lse});
    return loss.mean();
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor& logits = s[0];
    const CUDAGuard guard(logits.device());
    const int64_t N = logits.size(0), V = logits.size(1);
    const Tensor g = grads[0].to(at::kFloat).contiguous();
    // the logits are not needed again: their buffer becomes the gradient
    check(ts2ts_ce_bwd(logits.mutable_data_ptr(), s[1].const_data_ptr<int64_t>(), fptr(s[2]), fptr(g), static_cast<float>(1.0 / static_cast<double>(N)), N,
                       static_cast<int>(V), stream_of(logits)),
          "ts2ts_ce_bwd");
    Tensor dlogits = logits.detach();  // not the logits' own history
    refuse_gradient("ts2ts::cross_entropy backward", {grads[0], logits}, {&dlogits});
    return {dlogits, Tensor()};
  }
};
Tensor cross_entropy(const Tensor& logits, const Tensor& target) { return CrossEntropy::apply(logits, target); }

// y = x w^T with bf16 activations and an fp32 weight.  The weight gradient leaves its GEMM in fp32: no bf16 rounding and no
// conversion pass (6 bytes per weight) on the way to the parameter.  x is saved as it was passed, so that writing to it
// before the backward is noticed; of w only the bf16 copy is needed, and a changed w does not matter.  A gradient that may be
// differentiated again (create_graph) is made of ordinary operators on x and w themselves.
// `copy`, the weight in bf16 where the caller has made one (cast_weights; what it holds is taken as it is), or a copy of this call's own.
Tensor bf16_of(const Tensor& w, const OptTensor& copy) {
  if (!copy.has_value()) return w.to(at::kBFloat16);
  TORCH_CHECK_VALUE(copy->scalar_type() == at::kBFloat16 && copy->sizes() == w.sizes() && copy->device() == w.device(), "the weight's copy is bf16 and of its size");
  TORCH_CHECK_VALUE(!copy->requires_grad(), "the weight's copy does not require grad: the weight itself gets the gradient");
  return *copy;
}
// The bf16 copies of fp32 weights, all in one launch.
std::vector<Tensor> cast_weights(at::TensorList ws) {
  std::vector<Tensor> out;
  if (ws.empty()) return out;
  at::AutoDispatchBelowADInplaceOrView below;
  const CUDAGuard guard(ws[0].device());
  std::vector<const float*> src;
  std::vector<void*> dst;
  std::vector<int64_t> n;
  for (const Tensor& w : ws) {
    TORCH_CHECK_VALUE(w.is_cuda() && w.device() == ws[0].device() && w.scalar_type() == at::kFloat && w.is_contiguous(), "cast_weights: contiguous fp32 CUDA tensors of one device");
    out.push_back(at::empty(w.sizes(), w.options().dtype(at::kBFloat16)));
    src.push_back(fptr(w));
    dst.push_back(out.back().mutable_data_ptr());
    n.push_back(w.numel());
  }
  check(ts2ts_cast_bf16(static_cast<int>(src.size()), src.data(), dst.data(), n.data(), stream_of(ws[0])), "ts2ts_cast_bf16");
  return out;
}

// Whether d.copy_(s) moves bytes and does nothing else.
bool bytes_only(const Tensor& d, const Tensor& s) {
  for (const Tensor* t : {&d, &s})
    if (!t->is_cuda() || at::isTensorSubclassLike(*t) || t->is_nested() || t->layout() != at::kStrided || t->_is_zerotensor() || t->is_neg() || t->is_conj() ||
        !t->is_contiguous() || t->_fw_grad(0).defined())
      return false;
  return s.device() == d.device() && d.scalar_type() == s.scalar_type() && d.sizes() == s.sizes() && !d.requires_grad() && !d.is_inference() &&
         !(at::GradMode::is_enabled() && s.requires_grad());
}
// Whether some pair's target shares memory with another tensor of the list: the pairs then depend on their order.
bool targets_overlap(const std::vector<std::pair<Tensor, Tensor>>& pairs) {
  struct Range { uintptr_t begin, end; bool target; };
  std::vector<Range> ranges;
  for (const auto& [d, s] : pairs)
    for (const Tensor* t : {&d, &s})
      if (const auto at = reinterpret_cast<uintptr_t>(t->const_data_ptr()); t->nbytes() > 0) ranges.push_back({at, at + t->nbytes(), t == &d});
  std::sort(ranges.begin(), ranges.end(), [](const Range& a, const Range& b) { return a.begin < b.begin; });
  uintptr_t any = 0, target = 0;  // where what came before ends
  for (const Range& r : ranges) {
    if (r.begin < (r.target ? any : target)) return true;
    any = std::max(any, r.end);
    if (r.target) target = std::max(target, r.end);
  }
  return false;
}
void copy_together(std::vector<std::pair<Tensor, Tensor>>& pairs) {
  if (pairs.empty()) return;
  if (targets_overlap(pairs)) {
    for (auto& [d, s] : pairs) d.copy_(s);
  } else {
    std::vector<const void*> from;
    std::vector<void*> to;
    std::vector<int64_t> bytes;
    for (auto& [d, s] : pairs) {
      from.push_back(s.const_data_ptr()); to.push_back(d.mutable_data_ptr()); bytes.push_back(static_cast<int64_t>(d.nbytes()));
      d.unsafeGetTensorImpl()->bump_version();
    }
    const CUDAGuard guard(pairs[0].first.device());
    check(ts2ts_copy(static_cast<int>(from.size()), from.data(), to.data(), bytes.data(), stream_of(pairs[0].first)), "ts2ts_copy");
  }
  pairs.clear();
}
// dst[i].copy_(src[i]), one after the other as far as that can be told: neighbours that only move bytes, of tensors apart from each other, go in one launch.
void copy_tensors(at::TensorList dst, at::TensorList src) {
  TORCH_CHECK_VALUE(dst.size() == src.size(), "copy_tensors: lists of equal length");
  std::vector<std::pair<Tensor, Tensor>> together;
  for (size_t i = 0; i < dst.size(); ++i) {
    const bool joins = bytes_only(dst[i], src[i]);
    if (!joins || (!together.empty() && together[0].first.device() != dst[i].device())) copy_together(together);
    if (joins) together.emplace_back(dst[i], src[i]);
    else dst[i].copy_(src[i]);
  }
  copy_together(together);
}

struct Linear : torch::autograd::Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& copy) {
    need_cuda(x);
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor wb = bf16_of(w, copy);
    ctx->save_for_backward({x, wb});
    if (w.requires_grad() && !w.is_inference()) {
      ctx->saved_data["w"] = w;
      ctx->saved_data["version"] = static_cast<int64_t>(w._version());
    }
    auto shape = x.sizes().vec();
    shape.back() = w.size(0);
    return at::mm(x.reshape({-1, x.size(-1)}), wb.t()).view(shape);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    bind_context(s[0]);
    const Tensor dy = grads[0].reshape({-1, grads[0].size(-1)});
    Tensor dx, dw;
    if (at::GradMode::is_enabled()) {
      const c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
      Tensor wb = s[1];
      if (ctx->saved_data.count("w")) {
        const Tensor w = ctx->saved_data["w"].toTensor();
        TORCH_CHECK(static_cast<int64_t>(w._version()) == ctx->saved_data["version"].toInt(),
                    "one of the variables needed for gradient computation has been modified by an inplace operation: the weight of a "
                    "linear layer whose gradient is to be differentiated again");
        wb = w.to(at::kBFloat16);
      }
      if (ctx->needs_input_grad(0)) dx = at::mm(dy, wb).view(s[0].sizes());
      if (ctx->needs_input_grad(1)) dw = at::mm(dy.t().to(at::kFloat), s[0].reshape({-1, s[0].size(-1)}).to(at::kFloat));
      return {dx, dw, Tensor()};
    }
    if (ctx->needs_input_grad(0)) dx = at::mm(dy, s[1]).view(s[0].sizes());
    if (ctx->needs_input_grad(1)) dw = at::mm(dy.t(), s[0].reshape({-1, s[0].size(-1)}), at::kFloat);
    return {dx, dw, Tensor()};
  }
};
Tensor linear(const Tensor& x, const Tensor& w, const OptTensor& copy) { return Linear::apply(x, w, copy); }

// Mean cross-entropy of the output head, logits = h w^T.  The loss kernel leaves the gradient of the mean loss in the
// logits' buffer; what reaches the loss from above multiplies the two small results instead of the logits.
struct HeadLoss : torch::autograd::Function<HeadLoss> {
  static Tensor forward(AutogradContext* ctx, const Tensor& h, const Tensor& w, const Tensor& target_in, const OptTensor& copy) {
    need_cuda(h);
    at::AutoDispatchBelowADInplaceOrView below;
    const CUDAGuard guard(h.device());
    const Tensor h2 = h.reshape({-1, h.size(-1)}), wb = bf16_of(w, copy), target = target_in.reshape({-1}).to(at::kLong).contiguous();
    const int64_t N = h2.size(0), V = w.size(0);
    TORCH_CHECK_VALUE(target.numel() == N, "head_loss: one target per row of h");
    Tensor logits = at::mm(h2, wb.t()), loss = at::empty({N}, h.options().dtype(at::kFloat));
    check(ts2ts_ce_fwd_grad(logits.mutable_data_ptr(), target.const_data_ptr<int64_t>(), mfptr(loss), static_cast<float>(1.0 / static_cast<double>(N)), N,
                            static_cast<int>(V), stream_of(h)),
          "ts2ts_ce_fwd_grad");
    ctx->save_for_backward({h, wb, logits});
    ctx->saved_data["w"] = w;
    return loss.mean();
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const CUDAGuard guard(s[0].device());
    bind_context(s[0]);
    Tensor dh, dw;
    {
      const at::AutoGradMode plain(false);
      const Tensor g = grads[0].to(at::kFloat).contiguous();
      void* stream = stream_of(g);
      if (ctx->needs_input_grad(0)) {
        Tensor dh32 = at::mm(s[2], s[1], at::kFloat);
        dh = at::empty(s[0].sizes(), s[0].options());
        check(ts2ts_scale(mfptr(dh32), dh.mutable_data_ptr(), fptr(g), dh.numel(), stream), "ts2ts_scale");
      }
      if (ctx->needs_input_grad(1)) {
        dw = at::mm(s[2].t(), s[0].reshape({-1, s[0].size(-1)}), at::kFloat);
        check(ts2ts_scale(mfptr(dw), nullptr, fptr(g), dw.numel(), stream), "ts2ts_scale");
      }
    }
    refuse_gradient("ts2ts::head_loss backward", {grads[0], s[0], ctx->saved_data["w"].toTensor()}, {&dh, &dw});
    return {dh, dw, Tensor(), Tensor()};
  }
};
Tensor head_loss(const Tensor& h, const Tensor& w, const Tensor& target, const OptTensor& copy) { return HeadLoss::apply(h, w, target, copy); }

struct Embedding : torch::autograd::Function<Embedding> {
  static Tensor forward(AutogradContext* ctx, const Tensor& w, const Tensor& idx) {
    need_cuda(w);
    at::AutoDispatchBelowADInplaceOrView below;
    ctx->save_for_backward({idx});
    ctx->saved_data["V"] = w.size(0);
    return at::embedding(w, idx);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor idx = ctx->get_saved_variables()[0].contiguous();
    Tensor dx = grads[0].contiguous();
    const CUDAGuard guard(dx.device());
    const int64_t V = ctx->saved_data["V"].toInt(), C = dx.size(-1);
    // torch's own where the gradient may be differentiated again, and for sizes the kernel does not take
    if (at::GradMode::is_enabled() || idx.numel() == 0 || idx.numel() > (1 << 30) || V > INT32_MAX)
      return {at::embedding_dense_backward(dx, idx, V, -1, false), Tensor()};
    if (reinterpret_cast<uintptr_t>(dx.const_data_ptr()) & 15u) dx = dx.clone();
    Tensor dw = at::empty({V, C}, dx.options());
    check(ts2ts_embedding_bwd(idx.const_data_ptr<int64_t>(), fptr(dx), mfptr(dw), idx.numel(), static_cast<int>(C), V, stream_of(dx)),
          "ts2ts_embedding_bwd");
    return {dw, Tensor()};
  }
};
Tensor embedding(const Tensor& w, const Tensor& idx) { return Embedding::apply(w, idx); }

// One AdamW step over fp32 CUDA tensors; `steps` are one-element CPU tensors, advanced here.
void adamw(at::TensorList params, at::TensorList grads, at::TensorList exp_avgs, at::TensorList exp_avg_sqs, at::TensorList steps, double lr,
           double beta1, double beta2, double eps, double weight_decay) {
  const size_t n = params.size();
  TORCH_CHECK_VALUE(grads.size() == n && exp_avgs.size() == n && exp_avg_sqs.size() == n && steps.size() == n, "adamw: lists of equal length");
  if (n == 0) return;
  const CUDAGuard guard(params[0].device());
  std::vector<float*> p(n), m(n), v(n);
  std::vector<const float*> g(n);
  std::vector<int64_t> sizes(n);
  std::vector<float> t(n);
  for (size_t i = 0; i < n; ++i) {
    TORCH_CHECK_VALUE(params[i].device() == params[0].device() && steps[i].is_cpu(), "adamw: parameters on one device, steps on the CPU");
    for (const Tensor* x : {&params[i], &grads[i], &exp_avgs[i], &exp_avg_sqs[i]})
      TORCH_CHECK_VALUE(x->is_cuda() && x->scalar_type() == at::kFloat && x->is_contiguous() && x->numel() == params[i].numel(),
                        "adamw: contiguous fp32 CUDA tensors");
    p[i] = mfptr(params[i]); g[i] = fptr(grads[i]); m[i] = mfptr(exp_avgs[i]); v[i] = mfptr(exp_avg_sqs[i]);
    sizes[i] = params[i].numel();
    t[i] = *fptr(steps[i]) + 1.f;
  }
  check(ts2ts_adamw(static_cast<int>(n), p.data(), g.data(), m.data(), v.data(), sizes.data(), t.data(), lr, beta1, beta2, eps, weight_decay,
                    stream_of(params[0])),
        "ts2ts_adamw");
  for (size_t i = 0; i < n; ++i) *mfptr(steps[i]) = t[i];
  for (const Tensor& x : params) x.unsafeGetTensorImpl()->bump_version();
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
  m.def("link_candidates(Tensor input_ids, int mid_id, int[] start_ids, Tensor close_flags, int back_limit, int window) -> (Tensor, Tensor)");
  m.def("pack_mask(int[] starts, int[] ends, int[] ids, int[] link_pos, int[] link_target, int seq_len, int cap, Device device) -> Tensor[]", pack_mask);
  m.def("add_rmsnorm(Tensor x, Tensor? a, Tensor w, float eps) -> (Tensor, Tensor)", add_rmsnorm);
  m.def("qkv_attention(Tensor(a!) qkv, Tensor cos, Tensor sin, Tensor doc_ids, Tensor? link_bits, Tensor? q_row_ids, Tensor? kv_col_ids, "
        "Tensor plan, int n_heads, int head_dim) -> Tensor", qkv_attention);
  m.def("swiglu(Tensor gate_up) -> Tensor", swiglu);
  m.def("cross_entropy(Tensor logits, Tensor target) -> Tensor", cross_entropy);
  m.def("cast_weights(Tensor[] ws) -> Tensor[]", cast_weights);
  m.def("copy_tensors(Tensor(a!)[] dst, Tensor[] src) -> ()", copy_tensors);
  m.def("linear(Tensor x, Tensor w, Tensor? copy=None) -> Tensor", linear);
  m.def("head_loss(Tensor h, Tensor w, Tensor target, Tensor? copy=None) -> Tensor", head_loss);
  m.def("embedding(Tensor w, Tensor idx) -> Tensor", embedding);
  m.def("adamw(Tensor(a!)[] params, Tensor[] grads, Tensor(b!)[] exp_avgs, Tensor(c!)[] exp_avg_sqs, Tensor(d!)[] steps, float lr, float beta1, "
        "float beta2, float eps, float weight_decay) -> ()", adamw);
}
TORCH_LIBRARY_IMPL(ts2ts, CUDA, m) {
  m.impl("masked_attn_fwd", attn_fwd_cuda);
  m.impl("masked_attn_bwd", attn_bwd_cuda);
  m.impl("masked_attn_decode", attn_decode_cuda);
  m.impl("block_map", block_map_cuda);
  m.impl("link_candidates", link_candidates);
}
TORCH_LIBRARY_IMPL(ts2ts, Autograd, m) {
  m.impl("masked_attn_fwd", attn_fwd_autograd);
  m.impl("masked_attn_bwd", attn_bwd_autograd);
  m.impl("masked_attn_decode", attn_decode_autograd);
}
