// The forward pass of one transformer block as ONE call and its backward pass as two (MLP half, attention half: the gradient
// sink is told between them): the allocations and launches that ops/block.py makes one wrapper at a time.  A launch through
// Python (wrapper, allocation, argument conversion) costs the host 9 - 11 us, as much as a small kernel runs, so short prompts
// and small models waited for the host.  Measured on B200 by the host's clock: a training step of two blocks 2.38 -> 1.75 ms,
// a prompt of 128 tokens through 28 blocks 2.80 -> 1.88 ms.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAGraphsUtils.cuh>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "attn_api.h"
#include "bind_common.h"
#include "pdl.h"

namespace {

// Up to here the launches of a block's forward overlap.  Measured on B200, ms without and with, tokens through 28 blocks (1024
// wide, 16 / 8 heads): 128 2.02, 1.72; 512 2.31, 1.90; 1024 2.71, 2.40; 1536 2.78, 2.44; 2048 3.77, 3.43; 3072 4.06, 3.78;
// 4096 6.50, 6.40 in one sequence and 4.84, 4.73 in 32, about what a repetition of a run differs by.
constexpr int64_t PDL_MAX_ROWS = 2048;

using torch::Tensor;

// Allocates the outputs.  In the poison mode (ops/debug.py) `track` gets every one before its kernel runs, fills it with NaN and
// looks later whether one was left.
struct Outputs {
  const pybind11::object& track;
  Tensor operator()(const char* name, c10::IntArrayRef size, const at::TensorOptions& options) const {
    Tensor t = torch::empty(size, options);
    if (!track.is_none()) track(name, t);
    return t;
  }
};

__nv_bfloat16* bf(const Tensor& t) { return reinterpret_cast<__nv_bfloat16*>(t.data_ptr()); }

// The same buffers for block after block of the same widths (a pruned block has others): a pass without gradients keeps none of
// them.  An output's next writer is a block's length of kernels behind its last reader, also where launches overlap (a kernel waits
// for the end of the one before).
struct Reused {
  mutable std::vector<std::pair<std::string, Tensor>> kept;
  Tensor operator()(const char* name, c10::IntArrayRef size, const at::TensorOptions& options) const {
    for (const auto& k : kept)
      if (k.first == name && k.second.sizes() == size && k.second.scalar_type() == options.dtype().toScalarType() &&
          k.second.device() == options.device())
        return k.second;
    kept.emplace_back(name, torch::empty(size, options));
    return kept.back().second;
  }
};

// Returns the tensors ops/block.py keeps for backward and hands on, and the number of kernels launched:
// x, h1, rstd1, qkv, qk, o, lse, x2, h2, rstd2, gu (undefined unless wanted), act, y
template <class Make>
std::tuple<std::vector<c10::optional<Tensor>>, int64_t> run_block(
    const Make& make, const c10::optional<Tensor>& x_in, const c10::optional<Tensor>& y_in, const c10::optional<Tensor>& ids,
    const c10::optional<Tensor>& table, const Tensor& w1, const Tensor& wqkv, const Tensor& qn, const Tensor& kn,
    const Tensor& cos, const Tensor& sin, const Tensor& wo, const Tensor& w2, const Tensor& wgu, const Tensor& wd, int64_t B,
    int64_t S, int64_t Hq, int64_t Hkv, double eps, bool use_norm, bool want_gu) {
  c10::cuda::CUDAGuard guard(wqkv.device());
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  const int64_t M = B * S, D = w1.numel(), F = wd.size(1);
  const auto b16 = wqkv.options(), f32 = wqkv.options().dtype(torch::kFloat32);
  const bool has_ids = ids.has_value() && ids->defined(), has_y = y_in.has_value() && y_in->defined();
  const bool has_x = x_in.has_value() && x_in->defined();
  TORCH_CHECK(D % 4 == 0 && F % 8 == 0, "block_forward: widths");
  TORCH_CHECK(has_ids ? (table.has_value() && table->size(1) == D && ids->numel() == M && ids->is_contiguous() &&
                         ids->scalar_type() == torch::kInt64)
                      : (has_x && x_in->is_contiguous() && x_in->scalar_type() == torch::kFloat32 && x_in->size(0) == M &&
                         x_in->size(1) == D), "block_forward: input");
  TORCH_CHECK(!has_y || (y_in->is_contiguous() && y_in->scalar_type() == torch::kBFloat16 && y_in->numel() == M * D),
              "block_forward: y");
  TORCH_CHECK(wqkv.size(0) == (Hq + 2 * Hkv) * 128 && wqkv.size(1) == D && wo.size(0) == D && wo.size(1) == Hq * 128 &&
                  wgu.size(0) == 2 * F && wgu.size(1) == D && wd.size(0) == D, "block_forward: weights");
  TORCH_CHECK(cos.is_contiguous() && sin.is_contiguous() && cos.size(0) >= S && cos.size(-1) == 128, "block_forward: tables");
  int64_t launches = 8;
  // Few tokens: every kernel is short and most weights come from memory, so launches overlap and the products fetch their
  // first weight tiles under the kernel before, which here always is one that writes activations.
  // (A captured step has no launches to hide, so its graph keeps plain edges.)
  const bool eager = at::cuda::currentStreamCaptureStatusMayInitCtx() == at::cuda::CaptureStatus::None;
  tb::PdlScope overlap(M <= PDL_MAX_ROWS && eager);
  auto product = [&](const Tensor& in, const Tensor& w, Tensor& out) { bind_gemm(in, w, out, false, false, 0, 0, 0, true); };
  auto add_norm = [&](const float* x, const __nv_bfloat16* y, const int64_t* id, const Tensor* tab, const Tensor& w, float* xo,
                      const Tensor& h, const Tensor& rstd) {
    const bool b16_table = tab != nullptr && tab->scalar_type() == torch::kBFloat16;
    tb::add_rmsnorm_fwd(x, y, id, tab != nullptr && !b16_table ? tab->data_ptr<float>() : nullptr,
                        b16_table ? bf(*tab) : nullptr, w.data_ptr<float>(), xo, bf(h), rstd.data_ptr<float>(), (int)M, (int)D,
                        (float)eps, stream);
  };
  Tensor x = has_ids || has_y ? make("block_forward.x", {M, D}, f32) : *x_in;
  Tensor h1 = make("block_forward.h1", {M, D}, b16), rstd1 = make("block_forward.rstd1", {M}, f32);
  add_norm(has_x ? x_in->data_ptr<float>() : nullptr, has_y ? bf(*y_in) : nullptr, has_ids ? ids->data_ptr<int64_t>() : nullptr,
           has_ids ? &*table : nullptr, w1, has_ids || has_y ? x.data_ptr<float>() : nullptr, h1, rstd1);
  Tensor qkv = make("block_forward.qkv", {M, (Hq + 2 * Hkv) * 128}, b16);
  product(h1, wqkv, qkv);
  Tensor qk = make("block_forward.qk", {M, (Hq + Hkv) * 128}, b16);
  tb::qknorm_rope_fwd(bf(qkv), qn.data_ptr<float>(), kn.data_ptr<float>(), cos.data_ptr<float>(), sin.data_ptr<float>(), bf(qk),
                      (int)M, (int)S, (int)Hq, (int)Hkv, 128, (float)eps, use_norm ? 1 : 0, stream);
  Tensor o = make("block_forward.o", {M, Hq * 128}, b16), lse = make("block_forward.lse", {B, Hq, S}, f32);
  const int rc = tb::attn_fwd(qk.data_ptr(), qkv.data_ptr(), o.data_ptr(), lse.data_ptr<float>(), (int)B, (int)S, (int)Hq,
                              (int)Hkv, attn_err_word().data_ptr<int>(), stream);
  TORCH_CHECK(rc == 0, "attn_fwd failed with code ", rc);
  Tensor y_a = make("block_forward.y_a", {M, D}, b16);
  product(o, wo, y_a);
  Tensor x2 = make("block_forward.x2", {M, D}, f32), h2 = make("block_forward.h2", {M, D}, b16);
  Tensor rstd2 = make("block_forward.rstd2", {M}, f32);
  add_norm(x.data_ptr<float>(), bf(y_a), nullptr, nullptr, w2, x2.data_ptr<float>(), h2, rstd2);
  Tensor act = make("block_forward.act", {M, F}, b16);
  c10::optional<Tensor> gu;
  if (want_gu) gu = make("block_forward.gu", {M, 2 * F}, b16);
  if (!bind_gemm_swiglu(h2, wgu, gu, act)) {
    Tensor both = want_gu ? *gu : make("block_forward.gu", {M, 2 * F}, b16);
    product(h2, wgu, both);
    tb::swiglu_fwd(bf(both), bf(act), (int)M, (int)F, stream);
    ++launches;
  }
  Tensor y = make("block_forward.y", {M, D}, b16);
  product(act, wd, y);
  return {{x, h1, rstd1, qkv, qk, o, lse, x2, h2, rstd2, gu, act, y}, launches};
}

std::tuple<std::vector<c10::optional<Tensor>>, int64_t> block_forward(
    const c10::optional<Tensor>& x_in, const c10::optional<Tensor>& y_in, const c10::optional<Tensor>& ids,
    const c10::optional<Tensor>& table, const Tensor& w1, const Tensor& wqkv, const Tensor& qn, const Tensor& kn,
    const Tensor& cos, const Tensor& sin, const Tensor& wo, const Tensor& w2, const Tensor& wgu, const Tensor& wd, int64_t B,
    int64_t S, int64_t Hq, int64_t Hkv, double eps, bool use_norm, bool want_gu, const pybind11::object& track) {
  return run_block(Outputs{track}, x_in, y_in, ids, table, w1, wqkv, qn, kn, cos, sin, wo, w2, wgu, wd, B, S, Hq, Hkv, eps,
                   use_norm, want_gu);
}

// The forward pass without gradients, from token ids to the final norm's output, as one call: a block per call and an autograd node
// around each cost the host 63 us a block, as long as the kernels of a short prompt take.  layers: w1, wqkv, qn, kn, wo, w2, wgu, wd of
// every block.  Measured on B200, 28 blocks (1024 wide, 16 / 8 heads) and the head, by the host's clock: 128 tokens 1817 -> 1488 us,
// 4 x 2048 12.19 -> 12.11 ms.
std::tuple<Tensor, int64_t> blocks_forward(const Tensor& ids, const Tensor& table, const std::vector<std::vector<Tensor>>& layers,
                                           const Tensor& cos, const Tensor& sin, const Tensor& norm, double norm_eps, int64_t B,
                                           int64_t S, int64_t Hq, int64_t Hkv, double eps, bool use_norm) {
  const Reused make;
  c10::optional<Tensor> x, y, first = ids;
  int64_t launches = 1;
  for (const auto& w : layers) {
    TORCH_CHECK(w.size() == 8, "blocks_forward: eight tensors per block");
    auto out = run_block(make, x, y, first, table, w[0], w[1], w[2], w[3], cos, sin, w[4], w[5], w[6], w[7], B, S, Hq, Hkv, eps,
                         use_norm, false);
    x = std::get<0>(out)[7];
    y = std::get<0>(out)[12];
    first = c10::nullopt;
    launches += std::get<1>(out);
  }
  TORCH_CHECK(x.has_value() && norm.numel() == x->size(1), "blocks_forward: no blocks, or a norm of another width");
  c10::cuda::CUDAGuard guard(x->device());
  Tensor h = torch::empty(x->sizes(), y->options()), rstd = torch::empty({x->size(0)}, x->options());
  tb::add_rmsnorm_fwd(x->data_ptr<float>(), bf(*y), nullptr, nullptr, nullptr, norm.data_ptr<float>(), nullptr, bf(h),
                      rstd.data_ptr<float>(), (int)x->size(0), (int)x->size(1), (float)norm_eps,
                      at::cuda::getCurrentCUDAStream().stream());
  return {h, launches};
}

void check_rows(const Tensor& t, int64_t rows, int64_t cols, torch::ScalarType type, const char* what) {
  TORCH_CHECK(t.is_contiguous() && t.scalar_type() == type && t.dim() == 2 && t.size(0) == rows && t.size(1) == cols, what);
}

void norm_bwd(const Tensor& dh, const Tensor& x, const Tensor& w, const Tensor& rstd, const Tensor& dx_in, const Tensor& dx,
              const c10::optional<Tensor>& dxb, const Tensor& dw, cudaStream_t stream) {
  tb::rmsnorm_bwd(bf(dh), x.data_ptr<float>(), w.data_ptr<float>(), rstd.data_ptr<float>(), dx_in.data_ptr<float>(),
                  dx.data_ptr<float>(), dxb.has_value() ? bf(*dxb) : nullptr, dw.data_ptr<float>(), (int)x.size(0),
                  (int)x.size(1), bind_num_sms(), attn_err_word().data_ptr<int>(), stream);
}

// dwd / dwgu: fp32 destinations of the matrices' gradients, added to when the flag says so; dw2 is always added to.
// Returns dx1 (fp32), its bf16 copy and the number of launches.
std::tuple<Tensor, Tensor, int64_t> block_backward_mlp(const Tensor& dx2, const Tensor& dy, const Tensor& gu, const Tensor& act,
                                                       const Tensor& h2, const Tensor& x2, const Tensor& w2,
                                                       const Tensor& rstd2, const Tensor& wgu, const Tensor& wd, Tensor dwd,
                                                       bool add_d, Tensor dwgu, bool add_gu, Tensor dw2,
                                                       const pybind11::object& track) {
  const Outputs make{track};
  c10::cuda::CUDAGuard guard(dy.device());
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  const int64_t M = dy.size(0), D = dy.size(1), F = wd.size(1);
  check_rows(dy, M, D, torch::kBFloat16, "block_backward: dy");
  check_rows(dx2, M, D, torch::kFloat32, "block_backward: dx2");
  int64_t launches = 5;
  Tensor dgu = make("block_backward.dgu", {M, 2 * F}, dy.options());
  if (!bind_gemm_swiglu_bwd(dy, wd, gu, dgu)) {
    Tensor d_act = make("block_backward.d_act", {M, F}, dy.options());
    bind_gemm(dy, wd, d_act, false, true, 0);
    tb::swiglu_bwd(bf(d_act), bf(gu), bf(dgu), (int)M, (int)F, stream);
    ++launches;
  }
  bind_gemm(dy, act, dwd, true, true, add_d ? 2 : 1);
  Tensor d_h2 = make("block_backward.d_h2", {M, D}, dy.options());
  bind_gemm(dgu, wgu, d_h2, false, true, 0);
  bind_gemm(dgu, h2, dwgu, true, true, add_gu ? 2 : 1);
  dgu = Tensor();
  Tensor dx1 = make("block_backward.dx1", {M, D}, dx2.options());
  Tensor dx1b = make("block_backward.dx1b", {M, D}, dy.options());
  norm_bwd(d_h2, x2, w2, rstd2, dx2, dx1, dx1b, dw2, stream);
  return {dx1, dx1b, launches};
}

// As above for the attention half; dqn, dkn and dw1 are added to.  dx_out: the caller's destination of dx0.
std::tuple<Tensor, c10::optional<Tensor>, int64_t> block_backward_attn(
    const Tensor& dx1, const Tensor& dx1b, const Tensor& o, const Tensor& lse, const Tensor& qk, const Tensor& qkv,
    const Tensor& h1, const Tensor& x, const Tensor& w1, const Tensor& rstd1, const Tensor& qn, const Tensor& kn,
    const Tensor& cos, const Tensor& sin, const Tensor& wqkv, const Tensor& wo, Tensor dwo, bool add_o, Tensor dwqkv,
    bool add_qkv, Tensor dqn, Tensor dkn, Tensor dw1, const c10::optional<Tensor>& dx_out, bool want_b16, int64_t B, int64_t S,
    int64_t Hq, int64_t Hkv, double eps, bool use_norm, const pybind11::object& track) {
  const Outputs make{track};
  c10::cuda::CUDAGuard guard(dx1.device());
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  const int64_t M = dx1.size(0), D = dx1.size(1), nqkv = (Hq + 2 * Hkv) * 128;
  check_rows(qk, M, (Hq + Hkv) * 128, torch::kBFloat16, "block_backward: qk");
  check_rows(qkv, M, nqkv, torch::kBFloat16, "block_backward: qkv");
  check_rows(o, M, Hq * 128, torch::kBFloat16, "block_backward: o");
  TORCH_CHECK(M == B * S && lse.is_contiguous() && lse.numel() == B * Hq * S, "block_backward: sizes");
  TORCH_CHECK(cos.is_contiguous() && sin.is_contiguous() && cos.size(0) >= S && cos.size(-1) == 128, "block_backward: tables");
  int* err = attn_err_word().data_ptr<int>();
  Tensor d_o = make("block_backward.d_o", {M, Hq * 128}, dx1b.options());
  bind_gemm(dx1b, wo, d_o, false, true, 0);
  bind_gemm(dx1b, o, dwo, true, true, add_o ? 2 : 1);
  Tensor stats = make("block_backward.stats", {2, M * Hq}, dx1.options());
  Tensor dq_acc = make("block_backward.dq_acc", {M, Hq * 128}, dx1.options());
  Tensor dqkv = make("block_backward.dqkv", {M, nqkv}, dx1b.options());
  float* nds = stats.data_ptr<float>();
  float* nlse2 = nds + M * Hq;
  int rc = tb::attn_bwd_stats(d_o.data_ptr(), o.data_ptr(), lse.data_ptr<float>(), nds, nlse2, dq_acc.data_ptr<float>(), (int)B,
                              (int)S, (int)Hq, stream);
  TORCH_CHECK(rc == 0, "attn_bwd_stats failed with code ", rc);
  const int64_t wqk = (Hq + Hkv) * 128;
  rc = tb::attn_bwd_fused({qk.data_ptr(), wqk, 0}, {qk.data_ptr(), wqk, Hq * 128}, {qkv.data_ptr(), nqkv, (Hq + Hkv) * 128},
                          d_o.data_ptr(), dq_acc.data_ptr<float>(), bf(dqkv) + Hq * 128, bf(dqkv) + (Hq + Hkv) * 128, nqkv,
                          nds, nlse2, (int)B, (int)S, (int)S, (int)Hq, (int)Hkv, true, bind_num_sms(), err, stream);
  TORCH_CHECK(rc == 0, "attn_bwd_fused failed with code ", rc);
  d_o = Tensor();
  rc = tb::qknorm_rope_bwd(bf(dqkv), bf(qkv), qn.data_ptr<float>(), kn.data_ptr<float>(), cos.data_ptr<float>(),
                           sin.data_ptr<float>(), dqn.data_ptr<float>(), dkn.data_ptr<float>(), dq_acc.data_ptr<float>(), (int)M,
                           (int)S, (int)Hq, (int)Hkv, 128, (float)eps, use_norm ? 1 : 0, bind_num_sms(), stream);
  TORCH_CHECK(rc == 0, "qknorm_rope_bwd failed with code ", rc);
  dq_acc = Tensor();
  Tensor d_h1 = make("block_backward.d_h1", {M, D}, dx1b.options());
  bind_gemm(dqkv, wqkv, d_h1, false, true, 0);
  bind_gemm(dqkv, h1, dwqkv, true, true, add_qkv ? 2 : 1);
  Tensor dx0 = dx_out.has_value() && dx_out->defined() ? *dx_out : make("block_backward.dx0", {M, D}, dx1.options());
  check_rows(dx0, M, D, torch::kFloat32, "block_backward: dx_out");
  c10::optional<Tensor> dx0b;
  if (want_b16) dx0b = make("block_backward.dx0b", {M, D}, dx1b.options());
  norm_bwd(d_h1, x, w1, rstd1, dx1, dx0, dx0b, dw1, stream);
  return {dx0, dx0b, 8};
}

}  // namespace

void register_block(pybind11::module_& m) {
  m.def("block_forward", &block_forward);
  m.def("blocks_forward", &blocks_forward);
  m.def("block_backward_mlp", &block_backward_mlp);
  m.def("block_backward_attn", &block_backward_attn);
}
