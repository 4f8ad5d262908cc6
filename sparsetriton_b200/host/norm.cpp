// Per-sample batch norm and column concatenation: autograd nodes over the C ABI (nn/functional/norm.py:20-112).
#include <cuda_runtime_api.h>

#include "host.h"

namespace st_host {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

const float* f32(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
Tensor as_f32(const c10::optional<Tensor>& t) {
  if (!t) return Tensor();
  return (t->scalar_type() == at::kFloat ? t->detach() : t->detach().to(at::kFloat)).contiguous();
}
void require_cuda(const Tensor& x, const char* what) {
  if (!x.is_cuda())
    throw std::runtime_error(std::string(what) + ": expected a CUDA tensor, got device '" + x.device().str() +
                             "' (sparsetriton_b200 has no CPU path)");
}

// y = relu?((x - mean_b) * rstd_b * weight + bias).  batch undefined: the given statistics are the running ones (one row), and
// rstd holds their variances.
struct NormNode : torch::autograd::Function<NormNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_in, const c10::optional<Tensor>& weight,
                        const c10::optional<Tensor>& bias, const c10::optional<Tensor>& batch, const c10::optional<Tensor>& inv_count,
                        const c10::optional<Tensor>& status, const c10::optional<Tensor>& first_row,
                        const c10::optional<Tensor>& mean_in, const c10::optional<Tensor>& var_in, int64_t n_samples, double eps,
                        double momentum, bool relu) {
    require_cuda(x_in, "sparse_batch_norm");
    const Tensor x = x_in.contiguous();
    const int64_t n = x.size(0), C = x.size(1);
    const int code = feat_code(x);
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    const cudaStream_t s = stream_of(x);
    const Tensor w = as_f32(weight), b = as_f32(bias);
    const bool train = batch.has_value();
    Tensor y = empty_like_on(x, {n, C}, x.scalar_type());
    Tensor mean, rstd;
    Stage stage("bn_fwd", s);
    if (train) {
      // sums (B, C, 2), mean and rstd (B, C) in one allocation
      Tensor stats = empty_like_on(x, {4 * n_samples * C}, at::kFloat);
      Tensor sums = stats.narrow(0, 0, 2 * n_samples * C);
      mean = stats.narrow(0, 2 * n_samples * C, n_samples * C);
      rstd = stats.narrow(0, 3 * n_samples * C, n_samples * C);
      check(st_bn_forward_stats(code, x.data_ptr(), batch->data_ptr<int32_t>(), first_row->data_ptr<int32_t>(), n, (int)C,
                                (int)n_samples, inv_count->data_ptr<float>(), (float)eps, (float)momentum, sums.data_ptr<float>(),
                                mean.data_ptr<float>(), rstd.data_ptr<float>(), mean_in ? mean_in->data_ptr<float>() : nullptr,
                                var_in ? var_in->data_ptr<float>() : nullptr, status->data_ptr<int32_t>(), s), "st_bn_forward_stats");
      check(st_bn_apply(code, x.data_ptr(), batch->data_ptr<int32_t>(), n, (int)C, (int)n_samples, f32(mean), f32(rstd), f32(w), f32(b),
                        relu, y.data_ptr(), status->data_ptr<int32_t>(), s), "st_bn_apply");
    } else {
      mean = as_f32(mean_in);
      const Tensor var = as_f32(var_in);
      rstd = empty_like_on(x, {C}, at::kFloat);
      check(st_bn_apply_running(code, x.data_ptr(), n, (int)C, f32(mean), f32(var), (float)eps, f32(w), f32(b), relu,
                                rstd.data_ptr<float>(), y.data_ptr(), s), "st_bn_apply_running");
      rstd = var;                                              // turned into 1 / sqrt(var + eps) by the backward pass
    }
    const bool grad = x_in.requires_grad() || (weight && weight->requires_grad()) || (bias && bias->requires_grad());
    if (grad) {
      ctx->save_for_backward({x, mean, rstd, w, b, train ? *batch : Tensor(), train ? *inv_count : Tensor(), train ? *status : Tensor()});
      ctx->saved_data["samples"] = n_samples;
      ctx->saved_data["eps"] = eps;
      ctx->saved_data["relu"] = relu;
      ctx->saved_data["has"] = (int64_t)((weight ? 1 : 0) | (bias ? 2 : 0));
    }
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &mean = saved[1], &w = saved[3], &b = saved[4], &batch = saved[5], &inv_count = saved[6],
                 &status = saved[7];
    const int64_t n_samples = ctx->saved_data["samples"].toInt(), has = ctx->saved_data["has"].toInt();
    const bool relu = ctx->saved_data["relu"].toBool(), train = batch.defined();
    const int64_t n = x.size(0), C = x.size(1);
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    const cudaStream_t s = stream_of(x);
    const Tensor dy = (grads[0].scalar_type() == x.scalar_type() ? grads[0] : grads[0].to(x.scalar_type())).contiguous();
    Tensor rstd = saved[2], ones = inv_count;
    Stage stage("bn_bwd", s);
    if (!train) {
      Tensor r = empty_like_on(x, {C}, at::kFloat);
      check(st_bn_rstd(f32(rstd), (int)C, (float)ctx->saved_data["eps"].toDouble(), r.data_ptr<float>(), s), "st_bn_rstd");
      rstd = r;
      ones = at::ones({1}, x.options().dtype(at::kFloat).requires_grad(false));
    }
    Tensor sums = empty_like_on(x, {n_samples * C * 2}, at::kFloat);
    Tensor dx, dw, db;
    if (ctx->needs_input_grad(0)) dx = empty_like_on(x, {n, C}, x.scalar_type());
    if (has & 1) dw = empty_like_on(x, {C}, at::kFloat);
    if (has & 2) db = empty_like_on(x, {C}, at::kFloat);
    check(st_bn_backward(feat_code(x), x.data_ptr(), dy.data_ptr(), train ? batch.data_ptr<int32_t>() : nullptr, n, (int)C,
                         (int)n_samples, f32(mean), f32(rstd), f32(w), f32(b), relu, train, f32(ones), sums.data_ptr<float>(),
                         dx.defined() ? dx.data_ptr() : nullptr, dw.defined() ? dw.data_ptr<float>() : nullptr,
                         db.defined() ? db.data_ptr<float>() : nullptr, train ? status.data_ptr<int32_t>() : nullptr, s),
          "st_bn_backward");
    variable_list out(13);
    out[0] = dx;
    out[1] = dw;
    out[2] = db;
    return out;
  }
};

struct ConcatNode : torch::autograd::Function<ConcatNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& left, const Tensor& right) {
    const int64_t n = left.size(0), es = left.element_size();
    const c10::cuda::OptionalCUDAGuard guard(left.device());
    Tensor out = empty_like_on(left, {n, left.size(1) + right.size(1)}, left.scalar_type());
    check(st_concat_cols(left.data_ptr(), right.data_ptr(), n, (int)(left.size(1) * es), (int)(right.size(1) * es), out.data_ptr(),
                         stream_of(left)), "st_concat_cols");
    ctx->saved_data["widths"] = c10::IValue(std::vector<int64_t>{left.size(1), right.size(1)});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto widths = ctx->saved_data["widths"].toIntVector();
    const Tensor g = grads[0].contiguous();
    const int64_t n = g.size(0), es = g.element_size();
    const c10::cuda::OptionalCUDAGuard guard(g.device());
    Tensor a = empty_like_on(g, {n, widths[0]}, g.scalar_type()), b = empty_like_on(g, {n, widths[1]}, g.scalar_type());
    check(st_split_cols(g.data_ptr(), n, (int)(widths[0] * es), (int)(widths[1] * es), a.data_ptr(), b.data_ptr(), stream_of(g)),
          "st_split_cols");
    return {a, b};
  }
};

}  // namespace

std::tuple<Tensor, Tensor, Tensor, Tensor> batch_info(const Tensor& coords_in, int64_t n_samples) {
  const Tensor coords = coords_in.contiguous();
  const int64_t n = coords.size(0);
  const c10::cuda::OptionalCUDAGuard guard(coords.device());
  // one allocation: ids, then (from a 16-byte boundary) inverse counts, first rows, counts, status word
  const int64_t at_samples = (n + 3) / 4 * 4;
  Tensor buf = empty_like_on(coords, {at_samples + 3 * n_samples + 2}, at::kInt);
  Tensor ids = buf.narrow(0, 0, n), first = buf.narrow(0, at_samples + n_samples, n_samples);
  Tensor inv_count = buf.narrow(0, at_samples, n_samples).view(at::kFloat);
  Tensor counts = buf.narrow(0, at_samples + 2 * n_samples, n_samples + 1), status = buf.narrow(0, at_samples + 3 * n_samples + 1, 1);
  check(st_bn_batch_info(coords.data_ptr(), n, coord_code(coords), (int)n_samples, ids.data_ptr<int32_t>(),
                         reinterpret_cast<uint32_t*>(counts.data_ptr<int32_t>()), first.data_ptr<int32_t>(),
                         inv_count.data_ptr<float>(), stream_of(coords)), "st_bn_batch_info");
  return {ids, inv_count, status, first};
}

Tensor batch_norm_train(const Tensor& x, const c10::optional<Tensor>& w, const c10::optional<Tensor>& b, const Tensor& batch,
                        const Tensor& inv_count, const Tensor& status, const Tensor& first_row,
                        const c10::optional<Tensor>& running_mean, const c10::optional<Tensor>& running_var, int64_t n_samples,
                        double eps, double momentum, bool relu) {
  return NormNode::apply(x, w, b, c10::optional<Tensor>(batch), c10::optional<Tensor>(inv_count), c10::optional<Tensor>(status),
                         c10::optional<Tensor>(first_row), running_mean, running_var, n_samples, eps, momentum, relu);
}
Tensor batch_norm_running(const Tensor& x, const c10::optional<Tensor>& w, const c10::optional<Tensor>& b, const Tensor& mean,
                          const Tensor& var, double eps, bool relu) {
  const c10::optional<Tensor> none;
  return NormNode::apply(x, w, b, none, none, none, none, c10::optional<Tensor>(mean), c10::optional<Tensor>(var), (int64_t)1, eps, 0.0,
                         relu);
}
Tensor concat_cols(const Tensor& left, const Tensor& right) { return ConcatNode::apply(left, right); }

}  // namespace st_host
