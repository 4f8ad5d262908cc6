// Pooling and dense conversion: autograd nodes over the C ABI (nn/functional/spatial.py:26-292, utils/to_dense.py:143-240).
#include <cuda_runtime_api.h>

#include "host.h"

namespace st_host {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

std::vector<int32_t> as_i32(const std::vector<int64_t>& v) { return std::vector<int32_t>(v.begin(), v.end()); }

struct PoolNode : torch::autograd::Function<PoolNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& feats_in, const Tensor& coords_in, std::vector<int64_t> shape64,
                               int64_t kernel, int64_t padding, int64_t stride, bool max, int64_t batch) {
    const Tensor feats = feats_in.contiguous(), coords = coords_in.contiguous();
    const int64_t n = feats.size(0), C = feats.size(1);
    const int code = feat_code(feats), ccode = coord_code(coords);
    const std::vector<int32_t> shape = as_i32(shape64);
    const c10::cuda::OptionalCUDAGuard guard(feats.device());
    const cudaStream_t s = stream_of(feats);
    const int64_t bytes = st_pool_workspace_bytes(n);
    Tensor ws = bytes_on(feats, bytes + 256);                  // 16 bytes of counters, then the scratch
    int64_t* counters = reinterpret_cast<int64_t*>(ws.data_ptr());
    int32_t* status = reinterpret_cast<int32_t*>(counters + 1);
    void* scratch = static_cast<char*>(ws.data_ptr()) + 256;
    int64_t n_out = 0;
    Tensor out_coords, buf;
    const int64_t at_members = n, at_start = 2 * n;
    {
      Stage stage("pool_map", s);
      Mail mail(feats);
      cudaMemsetAsync(counters, 0, 16, s);
      check(st_pool_count(coords.data_ptr(), n, ccode, (int)kernel, (int)padding, (int)stride, shape.data(), (int)batch, scratch, bytes,
                          counters, status, s), "st_pool_count");
      check(st_publish(reinterpret_cast<const int32_t*>(counters), 4, 0, mail.host(), mail.ticket(), s), "st_publish");
      mail.sent();
      mail.wait(s);
      n_out = (int64_t)(uint32_t)mail.host()[0] | ((int64_t)mail.host()[1] << 32);
      if (mail.host()[2] & ST_DEV_BAD_INDEX)
        throw ValueError("sparse_pooling: a coordinate lies outside spatial_shape / batch_size");
      out_coords = at::empty({n_out, 4}, coords.options());
      buf = empty_like_on(feats, {2 * n + n_out + 1}, at::kInt);   // in_to_out, members, seg_start
      int32_t* b = buf.data_ptr<int32_t>();
      check(st_pool_write(coords.data_ptr(), n, ccode, (int)kernel, (int)padding, (int)stride, shape.data(), (int)batch, scratch, bytes,
                          out_coords.data_ptr(), n_out, b, b + at_members, b + at_start, s), "st_pool_write");
    }
    Tensor out = empty_like_on(feats, {n_out, C}, feats.scalar_type());
    const int32_t* b = buf.data_ptr<int32_t>();
    {
      Stage stage("pool_fwd", s);
      check(st_pool_fwd(code, feats.data_ptr(), (int)C, b + at_members, b + at_start, n_out, max, out.data_ptr(), s), "st_pool_fwd");
    }
    if (feats_in.requires_grad()) {
      ctx->save_for_backward({feats, out, buf});
      ctx->saved_data["max"] = max;
    }
    ctx->mark_non_differentiable({out_coords});
    return {out, out_coords};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &feats = saved[0], &out = saved[1], &buf = saved[2];
    const int64_t n = feats.size(0), C = feats.size(1);
    const c10::cuda::OptionalCUDAGuard guard(feats.device());
    const cudaStream_t s = stream_of(feats);
    const Tensor g = (grads[0].scalar_type() == feats.scalar_type() ? grads[0] : grads[0].to(feats.scalar_type())).contiguous();
    Tensor dx = empty_like_on(feats, {n, C}, feats.scalar_type());
    const int32_t* b = buf.data_ptr<int32_t>();
    Stage stage("pool_bwd", s);
    check(st_pool_bwd(feat_code(feats), g.data_ptr(), feats.data_ptr(), out.data_ptr(), (int)C, b, b + 2 * n, n,
                      ctx->saved_data["max"].toBool(), dx.data_ptr(), s), "st_pool_bwd");
    return {dx, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

struct DenseNode : torch::autograd::Function<DenseNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& feats_in, const Tensor& coords_in, std::vector<int64_t> shape64,
                        int64_t batch) {
    const Tensor feats = feats_in.contiguous(), coords = coords_in.contiguous();
    const int64_t n = feats.size(0), C = feats.size(1);
    const std::vector<int32_t> shape = as_i32(shape64);
    const c10::cuda::OptionalCUDAGuard guard(feats.device());
    const cudaStream_t s = stream_of(feats);
    Tensor dense = empty_like_on(feats, {batch, shape64[0], shape64[1], shape64[2], C}, feats.scalar_type());
    Stage stage("to_dense_fwd", s);
    check(st_to_dense_fwd(feat_code(feats), feats.data_ptr(), coords.data_ptr(), coord_code(coords), n, (int)C, (int)batch, shape.data(),
                          dense.data_ptr(), nullptr, s), "st_to_dense_fwd");
    if (feats_in.requires_grad()) {
      ctx->save_for_backward({coords});
      shape64.push_back(batch);
      shape64.push_back(C);
      ctx->saved_data["shape"] = c10::IValue(shape64);
    }
    return dense;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor coords = ctx->get_saved_variables()[0];
    const auto shape64 = ctx->saved_data["shape"].toIntVector();
    const std::vector<int32_t> shape(shape64.begin(), shape64.begin() + 3);
    const int64_t n = coords.size(0), C = shape64[4];
    const Tensor g = grads[0].contiguous();
    const c10::cuda::OptionalCUDAGuard guard(g.device());
    const cudaStream_t s = stream_of(g);
    Tensor dx = empty_like_on(g, {n, C}, g.scalar_type());
    Stage stage("to_dense_bwd", s);
    check(st_to_dense_bwd(feat_code(g), g.data_ptr(), coords.data_ptr(), coord_code(coords), n, (int)C, (int)shape64[3], shape.data(),
                          dx.data_ptr(), s), "st_to_dense_bwd");
    return {dx, Tensor(), Tensor(), Tensor()};
  }
};

}  // namespace

std::vector<Tensor> pool(const Tensor& feats, const Tensor& coords, std::vector<int64_t> shape, int64_t kernel, int64_t padding,
                         int64_t stride, bool max, int64_t batch) {
  return PoolNode::apply(feats, coords, std::move(shape), kernel, padding, stride, max, batch);
}
Tensor to_dense(const Tensor& feats, const Tensor& coords, std::vector<int64_t> shape, int64_t batch) {
  return DenseNode::apply(feats, coords, std::move(shape), batch);
}

}  // namespace st_host
