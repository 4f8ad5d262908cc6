// The convolution's autograd nodes over the C ABI.
//
// Forward   Y[o]  = sum_k X[nbr[o,k]] . W[k]
// dgrad     dX[i] = sum_k dY[inv[i,k]] . W[k]^T
// wgrad     dW[k] = sum_o X[nbr[o,k]]^T . dY[o]
// All three accumulate in fp32 and run without atomics, so results are reproducible run to run (the reference scatters dX and
// dW with atomic adds in the storage dtype, nn/functional/conv/funcs/implicit_precomputed_gemm.py:233-324).
#include <cuda_runtime_api.h>

#include "host.h"

namespace st_host {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

const Plan kNoPlan{};

int64_t round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

// The widths to run a layer with: its own if the tensor-core kernels take them or padding would not help, else the next
// ones they take (zero input channels meet zero weight rows, padded output columns are cut off again).
std::pair<int64_t, int64_t> padded_widths(int code, int64_t c_in, int64_t c_out) {
  auto both = [&](int64_t a, int64_t b) {
    return st_conv_uses_tensor_cores(code, (int)a, (int)b) && st_conv_uses_tensor_cores(code, (int)b, (int)a);
  };
  if (both(c_in, c_out)) return {c_in, c_out};
  const int64_t ci = round_up(c_in, 16), co = round_up(c_out, 16);
  return both(ci, co) ? std::make_pair(ci, co) : std::make_pair(c_in, c_out);
}
Tensor pad_cols(const Tensor& t, int64_t width) {
  return t.size(1) == width ? t.contiguous() : at::constant_pad_nd(t, {0, width - t.size(1)});
}
Tensor weight_for(const Tensor& w, at::ScalarType type, int64_t c_in, int64_t c_out) {
  Tensor t = w.scalar_type() == type ? w : w.to(type);
  if (t.size(1) == c_in && t.size(2) == c_out) return t.contiguous();
  return at::constant_pad_nd(t, {0, c_out - t.size(2), 0, c_in - t.size(1)});
}
double flops_of(const MapPtr& map, const Tensor& nbr, int64_t c_in, int64_t c_out) {
  return tracing() && nbr.size(0) > 0 ? 2.0 * map->pairs(nbr) * (double)c_in * (double)c_out : 0.0;
}
void* mutable_ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

}  // namespace

Tensor conv_forward(const Tensor& x, const Tensor& w, const Tensor& nbr, const MapPtr& map, bool row_order) {
  const int64_t n_out = nbr.size(0), K = w.size(0), c_in = w.size(1), c_out = w.size(2);
  const int code = feat_code(x);
  const c10::cuda::OptionalCUDAGuard guard(x.device());
  Tensor y = empty_like_on(x, {n_out, c_out}, x.scalar_type());
  if (n_out == 0) return y;
  const Plan& plan = st_conv_uses_tensor_cores(code, (int)c_in, (int)c_out) ? map->plan(nbr, row_order) : kNoPlan;
  const cudaStream_t s = stream_of(x);
  Stage stage("conv_fwd", s, flops_of(map, nbr, c_in, c_out), (int)c_in, (int)c_out);
  check(st_conv_fwd_planned(code, x.data_ptr(), w.data_ptr(), nbr.data_ptr<int32_t>(), plan.order(), plan.tmap(), plan.tmask(),
                            y.data_ptr(), x.size(0), n_out, (int)K, (int)c_in, (int)c_out, nullptr, 0, s), "st_conv_fwd_planned");
  return y;
}

Tensor conv_dgrad(const Tensor& dy, const Tensor& w, const Tensor& nbr, const MapPtr& map, int64_t n_in, bool row_order) {
  const int64_t n_out = nbr.size(0), K = w.size(0), c_in = w.size(1), c_out = w.size(2);
  const int code = feat_code(dy);
  const c10::cuda::OptionalCUDAGuard guard(dy.device());
  Tensor dx = empty_like_on(dy, {n_in, c_in}, dy.scalar_type());
  if (n_in == 0) return dx;
  const cudaStream_t s = stream_of(dy);
  const double flops = flops_of(map, nbr, c_in, c_out);
  const bool tc = st_conv_uses_tensor_cores(code, (int)c_out, (int)c_in);
  if (tc && map->symmetric(nbr, n_in)) {
    // submanifold layer: the map is its own inverse with the offsets reversed
    const Plan& plan = map->plan(nbr, row_order);
    Stage stage("conv_dgrad", s, flops, (int)c_in, (int)c_out);
    check(st_conv_dgrad_mirrored(code, dy.data_ptr(), w.data_ptr(), nbr.data_ptr<int32_t>(), plan.order(), plan.tmap(), plan.tmask(),
                                 dx.data_ptr(), n_in, (int)K, (int)c_in, (int)c_out, nullptr, 0, s), "st_conv_dgrad_mirrored");
    return dx;
  }
  const Plan* plan = tc ? map->inverse_plan(nbr, n_in, row_order) : nullptr;
  Tensor inv;
  if (!plan) {
    inv = map->inverse(nbr, n_in);
    plan = tc ? &map->inverse_state(nbr, n_in)->plan(inv, row_order) : &kNoPlan;
  }
  Stage stage("conv_dgrad", s, flops, (int)c_in, (int)c_out);
  check(st_conv_dgrad_planned(code, dy.data_ptr(), w.data_ptr(), inv.defined() ? inv.data_ptr<int32_t>() : nullptr, plan->order(),
                              plan->tmap(), plan->tmask(), dx.data_ptr(), n_in, n_out, (int)K, (int)c_in, (int)c_out, nullptr, 0, s),
        "st_conv_dgrad_planned");
  return dx;
}

Tensor conv_wgrad(const Tensor& x, const Tensor& dy, const Tensor& nbr, const MapPtr& map, at::ScalarType out, bool row_order) {
  const int64_t n_in = x.size(0), n_out = dy.size(0), K = nbr.size(1), c_in = x.size(1), c_out = dy.size(1);
  const int code = feat_code(x);
  const c10::cuda::OptionalCUDAGuard guard(x.device());
  if (n_out == 0) return at::zeros({K, c_in, c_out}, x.options().dtype(out).requires_grad(false));
  const cudaStream_t s = stream_of(x);
  const bool tc = st_conv_uses_tensor_cores(code, (int)c_in, (int)c_out);
  const Plan& plan = tc ? map->plan(nbr, row_order) : kNoPlan;
  // fp32 master weights take the kernel's fp32 sums as they are
  const bool direct = tc && out == at::kFloat;
  Tensor dw = empty_like_on(x, {K, c_in, c_out}, direct ? at::kFloat : x.scalar_type());
  Tensor ws = bytes_on(x, st_conv_workspace_bytes(code, n_in, n_out, (int)K, (int)c_in, (int)c_out));
  Stage stage("conv_wgrad", s, flops_of(map, nbr, c_in, c_out), (int)c_in, (int)c_out);
  if (direct) {
    check(st_conv_wgrad_planned_f32(code, x.data_ptr(), dy.data_ptr(), nbr.data_ptr<int32_t>(), plan.order(), plan.tmap(),
                                    plan.tmask(), dw.data_ptr<float>(), n_in, n_out, (int)K, (int)c_in, (int)c_out, ws.data_ptr(),
                                    ws.numel(), s), "st_conv_wgrad_planned");
    return dw;
  }
  check(st_conv_wgrad_planned(code, x.data_ptr(), dy.data_ptr(), nbr.data_ptr<int32_t>(), plan.order(), plan.tmap(), plan.tmask(),
                              dw.data_ptr(), n_in, n_out, (int)K, (int)c_in, (int)c_out, ws.data_ptr(), ws.numel(), s),
        "st_conv_wgrad_planned");
  return dw.scalar_type() == out ? dw : dw.to(out);
}

namespace {

// What the two forms share: operands padded to widths the tensor cores take, and the way back.
struct Widths {
  int64_t c_in, c_out, padded_in, padded_out;
};
Widths widths_of(const Tensor& x, const Tensor& w) {
  if (!x.is_cuda())
    throw std::runtime_error("sparse convolution: expected a CUDA tensor, got device '" + x.device().str() +
                             "' (sparsetriton_b200 has no CPU path)");
  const auto [pi, po] = padded_widths(feat_code(x), x.size(1), w.size(2));
  return {x.size(1), w.size(2), pi, po};
}
Tensor cut_cols(const Tensor& t, int64_t width) { return t.size(1) == width ? t : t.narrow(1, 0, width).contiguous(); }
Tensor cut_weight(const Tensor& t, int64_t a, int64_t b) {
  return t.size(1) == a && t.size(2) == b ? t : t.narrow(1, 0, a).narrow(2, 0, b).contiguous();
}
Tensor grad_rows(const Tensor& g, const Tensor& x, int64_t width) {
  return pad_cols(g.scalar_type() == x.scalar_type() ? g : g.to(x.scalar_type()), width);
}

struct ConvNode : torch::autograd::Function<ConvNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& features, const Tensor& weights, const Tensor& neighbours,
                        const MapPtr& map, bool row_order) {
    const Widths c = widths_of(features, weights);
    const Tensor x = pad_cols(features, c.padded_in);
    const Tensor w = weight_for(weights, x.scalar_type(), c.padded_in, c.padded_out);
    const Tensor nbr = neighbours.contiguous();
    Tensor y = conv_forward(x, w, nbr, map, row_order);
    if (features.requires_grad() || weights.requires_grad()) {
      ctx->save_for_backward({x, w, nbr});
      ctx->saved_data["map"] = c10::IValue::make_capsule(map);
      ctx->saved_data["how"] = c10::IValue(std::vector<int64_t>{c.c_in, c.c_out, (int64_t)weights.scalar_type(), row_order});
    }
    return cut_cols(y, c.c_out);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1], &nbr = saved[2];
    const MapPtr map = c10::static_intrusive_pointer_cast<MapState>(ctx->saved_data["map"].toCapsule());
    const auto how = ctx->saved_data["how"].toIntVector();
    const bool row_order = how[3] != 0;
    const Tensor dy = grad_rows(grads[0], x, w.size(2));
    Tensor dx, dw;
    if (ctx->needs_input_grad(0)) dx = cut_cols(conv_dgrad(dy, w, nbr, map, x.size(0), row_order), how[0]);
    if (ctx->needs_input_grad(1))
      dw = cut_weight(conv_wgrad(x, dy, nbr, map, (at::ScalarType)how[2], row_order), how[0], how[1]);
    return {dx, dw, Tensor(), Tensor(), Tensor()};
  }
};

// No map outlives a call: forward and backward each probe the table once into a scratch map and run the kernels over it.
struct HashFlyNode : torch::autograd::Function<HashFlyNode> {
  static std::pair<Tensor, MapPtr> probe(const Tensor& coords, const std::vector<int64_t>& offsets64,
                                         const std::vector<int64_t>& shape, int64_t stride, const Tensor& keys, const Tensor& vals) {
    const std::vector<int32_t> offsets(offsets64.begin(), offsets64.end());
    Stage stage("hashfly_probe", stream_of(coords));
    auto [nbr, map] = probe_map(coords, offsets, shape, (int)stride, keys, vals, false);
    return {nbr, map};
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& features, const Tensor& weights, const Tensor& coords,
                        const Tensor& keys, const Tensor& vals, std::vector<int64_t> offsets, std::vector<int64_t> shape,
                        int64_t stride, bool row_order) {
    const Widths c = widths_of(features, weights);
    const Tensor x = pad_cols(features, c.padded_in);
    const Tensor w = weight_for(weights, x.scalar_type(), c.padded_in, c.padded_out);
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    const Tensor q = coords.contiguous(), k = keys.contiguous(), v = vals.contiguous();
    auto [nbr, map] = probe(q, offsets, shape, stride, k, v);
    Tensor y = conv_forward(x, w, nbr, map, row_order);
    if (features.requires_grad() || weights.requires_grad()) {
      ctx->save_for_backward({x, w, q, k, v});
      ctx->saved_data["offsets"] = c10::IValue(offsets);
      ctx->saved_data["shape"] = c10::IValue(shape);
      ctx->saved_data["how"] = c10::IValue(std::vector<int64_t>{c.c_in, c.c_out, (int64_t)weights.scalar_type(), row_order, stride});
    }
    return cut_cols(y, c.c_out);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1];
    const auto how = ctx->saved_data["how"].toIntVector();
    const bool row_order = how[3] != 0;
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    auto [nbr, map] = probe(saved[2], ctx->saved_data["offsets"].toIntVector(), ctx->saved_data["shape"].toIntVector(), how[4],
                            saved[3], saved[4]);
    const Tensor dy = grad_rows(grads[0], x, w.size(2));
    Tensor dx, dw;
    if (ctx->needs_input_grad(0)) dx = cut_cols(conv_dgrad(dy, w, nbr, map, x.size(0), row_order), how[0]);
    if (ctx->needs_input_grad(1))
      dw = cut_weight(conv_wgrad(x, dy, nbr, map, (at::ScalarType)how[2], row_order), how[0], how[1]);
    return {dx, dw, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

}  // namespace

Tensor conv(const Tensor& x, const Tensor& w, const Tensor& nbr, const MapPtr& map, bool row_order) {
  return ConvNode::apply(x, w, nbr, map, row_order);
}
Tensor conv_hashfly(const Tensor& x, const Tensor& w, const Tensor& coords, std::vector<int32_t> offsets, const Tensor& keys,
                    const Tensor& vals, std::vector<int64_t> shape, int64_t stride, bool row_order) {
  return HashFlyNode::apply(x, w, coords, keys, vals, std::vector<int64_t>(offsets.begin(), offsets.end()), shape, stride, row_order);
}

}  // namespace st_host
