// Host side of the hot path in native code: what sits between PyTorch (memory, streams, autograd) and the C ABI of
// libsparsetriton_b200.  A layer of a few thousand voxels spends its time here, not on the GPU, so allocations, argument
// packing, plans and the autograd nodes are C++; Python keeps the public surface.
#pragma once

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>

#include <atomic>
#include <cstdint>
#include <mutex>
#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/sparsetriton_b200.h"

namespace st_host {

using at::Tensor;

inline void check(int rc, const char* what) {
  if (rc != ST_OK)
    throw std::runtime_error(std::string(what) + " failed with status " + std::to_string(rc) + ": " + st_last_error_string());
}
struct TypeError : std::runtime_error {
  using std::runtime_error::runtime_error;
};
struct ValueError : std::runtime_error {
  using std::runtime_error::runtime_error;
};

inline cudaStream_t stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
int feat_code(const Tensor& t);
int coord_code(const Tensor& t);
inline Tensor empty_like_on(const Tensor& like, at::IntArrayRef sizes, at::ScalarType type) {
  return at::empty(sizes, like.options().dtype(type).requires_grad(false));
}
inline Tensor bytes_on(const Tensor& like, int64_t n) { return empty_like_on(like, {n > 256 ? n : 256}, at::kByte); }

// Stage recorder (see trace.py): brackets a call with events on its stream while a recording is open, else does nothing.
class Stage {
 public:
  Stage(const char* name, cudaStream_t stream, double work = 0.0, int tag_a = 0, int tag_b = 0);
  ~Stage();
  Stage(const Stage&) = delete;

 private:
  const char* name_;
  cudaStream_t stream_;
  void *start_ = nullptr;
  long long launches_ = 0;
  double work_;
  int tag_a_, tag_b_;
};
bool tracing();
void trace_start();
// (name, milliseconds, launches, work, tag_a, tag_b) of the spans so far; synchronises
std::vector<std::tuple<std::string, double, int64_t, double, int, int>> trace_spans();
void trace_stop();

// A result on its way from the device: 64 bytes of pinned host memory that a kernel writes, the ticket last, and a few device
// words for kernels that need scratch of their own.  A fixed pool per process, handed out and given back under a lock; a slot
// that is dropped before its ticket arrived is given back when it has.
class Mail {
 public:
  explicit Mail(const Tensor& like);
  ~Mail();
  Mail(const Mail&) = delete;
  int32_t* host() const { return host_; }
  uint32_t* scratch() const { return scratch_; }
  int32_t ticket() const { return ticket_; }
  void sent() { sent_ = true; }                    // a kernel that will write the ticket has been launched
  void wait(cudaStream_t stream);                  // until the ticket is there
  bool arrived() const { return *(volatile int32_t*)(host_ + 15) == ticket_; }

 private:
  int slot_, device_;
  int32_t* host_;
  uint32_t* scratch_;
  int32_t ticket_;
  bool sent_ = false;
};

// One tile plan: row order, re-laid map and tile masks in one allocation.
struct Plan {
  Tensor buf;                                      // int32
  int64_t n_rows = -1, at_tmap = 0, at_tmask = 0, n_tmap = 0, n_tmask = 0;
  bool sorted = false;
  const int32_t* order() const { return sorted ? buf.data_ptr<int32_t>() : nullptr; }
  const int32_t* tmap() const { return n_rows > 0 ? buf.data_ptr<int32_t>() + at_tmap : nullptr; }
  const uint32_t* tmask() const {
    return n_rows > 0 ? reinterpret_cast<const uint32_t*>(buf.data_ptr<int32_t>() + at_tmask) : nullptr;
  }
  Tensor order_tensor() const { return sorted ? buf.narrow(0, 0, n_rows) : Tensor(); }
  Tensor tmap_tensor() const { return n_rows > 0 ? buf.narrow(0, at_tmap, n_tmap) : Tensor(); }
  Tensor tmask_tensor() const { return n_rows > 0 ? buf.narrow(0, at_tmask, n_tmask) : Tensor(); }
};

// What is derived from a neighbour map and kept with it: its tile plans, its inverse and the inverse's plan, whether it is its
// own mirror image.  Lives as an attribute of the map tensor (and holds no reference to it).
struct MapState : torch::CustomClassHolder {
  // rows of the map per call: `nbr` is always the tensor this state belongs to
  const Plan& plan(const Tensor& nbr, bool row_order);
  const Plan* inverse_plan(const Tensor& nbr, int64_t n_in, bool row_order);   // null where that form does not apply
  Tensor inverse(const Tensor& nbr, int64_t n_in);
  c10::intrusive_ptr<MapState> inverse_state(const Tensor& nbr, int64_t n_in);
  bool symmetric(const Tensor& nbr, int64_t n_in);
  double pairs(const Tensor& nbr);
  void expect_flag(const Tensor& nbr, const int32_t* word, cudaStream_t stream);   // *word = rows that break the symmetry

 private:
  std::recursive_mutex mu_;
  Plan plans_[2], inverse_plan_;
  Tensor inverse_;
  c10::intrusive_ptr<MapState> inverse_state_;
  std::unique_ptr<Mail> flag_;
  cudaStream_t flag_stream_ = nullptr;
  int symmetric_ = -1;                             // -1: nobody has looked (or nothing to look at), else 0 / 1
  double pairs_ = -1.0;
};
using MapPtr = c10::intrusive_ptr<MapState>;

std::vector<int32_t> kernel_offsets(int k, int d, int p, bool transposed);

// Table over the coordinates (made unless given) and the map of a stride-1 submanifold layer:
// (keys, vals, status, nbr, state); status is undefined when the table was given.
std::tuple<Tensor, Tensor, Tensor, Tensor, MapPtr> submanifold(const Tensor& coords, std::vector<int64_t> shape, int k, int d,
                                                              double factor, const c10::optional<Tensor>& keys,
                                                              const c10::optional<Tensor>& vals);
// The map of queries `coords` in a given table (conv.py's compute_neighbor_indices).
std::tuple<Tensor, MapPtr> probe_map(const Tensor& coords, const std::vector<int32_t>& offsets, const std::vector<int64_t>& shape,
                                     int stride, const Tensor& keys, const Tensor& vals, bool rows_of_table);
std::tuple<Tensor, Tensor, Tensor> build_table(const Tensor& coords, double factor);
std::vector<int64_t> extent(const Tensor& coords);

// Output coordinates (and map) of a strided or transposed layer in two halves.
class OutCoords : public torch::CustomClassHolder {
 public:
  OutCoords(const Tensor& coords, int k, int s, int d, int p, bool transposed, std::vector<int64_t> new_shape,
            std::vector<int64_t> in_shape, int64_t batch_bound, bool with_map);
  std::tuple<Tensor, Tensor, c10::optional<MapPtr>> finish();

 private:
  Tensor coords_, ws_;
  std::vector<int32_t> offsets_, new_shape_, in_shape_;
  int K_, stride_, transposed_, code_;
  int64_t n_, batch_bound_;
  bool with_map_;
  std::unique_ptr<Mail> mail_;
  c10::optional<c10::cuda::CUDAStream> stream_;
  int64_t* counters() const { return reinterpret_cast<int64_t*>(ws_.data_ptr()); }
  int32_t* status() const { return reinterpret_cast<int32_t*>(counters() + 1); }
  void* scratch() const { return static_cast<char*>(ws_.data_ptr()) + 256; }
};

Tensor conv(const Tensor& x, const Tensor& w, const Tensor& nbr, const MapPtr& map, bool row_order);
Tensor conv_hashfly(const Tensor& x, const Tensor& w, const Tensor& coords, std::vector<int32_t> offsets, const Tensor& keys,
                    const Tensor& vals, std::vector<int64_t> shape, int64_t stride, bool row_order);
Tensor conv_forward(const Tensor& x, const Tensor& w, const Tensor& nbr, const MapPtr& map, bool row_order);
Tensor conv_dgrad(const Tensor& dy, const Tensor& w, const Tensor& nbr, const MapPtr& map, int64_t n_in, bool row_order);
Tensor conv_wgrad(const Tensor& x, const Tensor& dy, const Tensor& nbr, const MapPtr& map, at::ScalarType out, bool row_order);
std::vector<Tensor> prepare_plans(const Tensor& nbr, const MapPtr& map, int64_t n_in, bool backward, bool row_order);

std::tuple<Tensor, Tensor, Tensor, Tensor> batch_info(const Tensor& coords, int64_t n_samples);
Tensor batch_norm_train(const Tensor& x, const c10::optional<Tensor>& w, const c10::optional<Tensor>& b, const Tensor& batch,
                        const Tensor& inv_count, const Tensor& status, const Tensor& first_row,
                        const c10::optional<Tensor>& running_mean, const c10::optional<Tensor>& running_var, int64_t n_samples,
                        double eps, double momentum, bool relu);
Tensor batch_norm_running(const Tensor& x, const c10::optional<Tensor>& w, const c10::optional<Tensor>& b, const Tensor& mean,
                          const Tensor& var, double eps, bool relu);
Tensor concat_cols(const Tensor& left, const Tensor& right);
std::vector<Tensor> pool(const Tensor& feats, const Tensor& coords, std::vector<int64_t> shape, int64_t kernel, int64_t padding,
                         int64_t stride, bool max, int64_t batch);
Tensor to_dense(const Tensor& feats, const Tensor& coords, std::vector<int64_t> shape, int64_t batch);

}  // namespace st_host
