// Tables, neighbour maps, tile plans and output coordinates.
#include <cuda_runtime_api.h>

#include "host.h"

namespace st_host {

namespace {

// below this many rows the sort costs more than the denser tiles save
constexpr int64_t kMinRowsForOrder = 16384;

int64_t align64(int64_t v) { return (v + 63) / 64 * 64; }

void make_plan(Plan* p, const Tensor& like, int64_t n_rows, int K, bool sorted, bool inverse_words) {
  const int64_t n_tiles = (n_rows + 127) / 128;
  p->n_rows = n_rows;
  p->sorted = sorted;
  p->n_tmap = n_tiles * K * 128;
  p->n_tmask = n_tiles * (inverse_words ? 1 : (K + 31) / 32);
  p->at_tmap = sorted ? align64(n_rows) : 0;
  p->at_tmask = align64(p->at_tmap + p->n_tmap);
  p->buf = empty_like_on(like, {p->at_tmask + p->n_tmask}, at::kInt);
}
int32_t* order_of(const Plan& p) { return p.sorted ? p.buf.data_ptr<int32_t>() : nullptr; }
int32_t* tmap_of(const Plan& p) { return p.buf.data_ptr<int32_t>() + p.at_tmap; }
uint32_t* tmask_of(const Plan& p) { return reinterpret_cast<uint32_t*>(p.buf.data_ptr<int32_t>() + p.at_tmask); }

std::vector<int32_t> as_i32(const std::vector<int64_t>& v) { return std::vector<int32_t>(v.begin(), v.end()); }

}  // namespace

// ------------------------------------------------------------------------------------------------ what a map keeps
const Plan& MapState::plan(const Tensor& nbr, bool row_order) {
  const int64_t n = nbr.size(0);
  const int K = (int)nbr.size(1);
  const bool sorted = row_order && n >= kMinRowsForOrder;
  std::lock_guard<std::recursive_mutex> lock(mu_);
  Plan& p = plans_[sorted];
  if (p.n_rows == n) return p;
  if (n == 0) {
    p.n_rows = 0;
    p.sorted = false;
    return p;
  }
  const c10::cuda::OptionalCUDAGuard guard(nbr.device());
  const cudaStream_t s = stream_of(nbr);
  Plan made;
  make_plan(&made, nbr, n, K, sorted, false);
  Stage stage("map_plan", s);
  if (sorted && K <= 32) {
    Tensor ws = bytes_on(nbr, st_map_plan_balanced_workspace_bytes(n, K));
    check(st_map_plan_balanced(nbr.data_ptr<int32_t>(), n, K, order_of(made), tmap_of(made), tmask_of(made), ws.data_ptr(),
                               ws.numel(), s), "st_map_plan_balanced");
    p = made;
    return p;
  }
  Tensor ws = sorted ? bytes_on(nbr, st_map_plan_workspace_bytes(n, K)) : Tensor();
  check(st_map_plan(nbr.data_ptr<int32_t>(), n, K, sorted, order_of(made), tmap_of(made), tmask_of(made),
                    sorted ? ws.data_ptr() : nullptr, sorted ? ws.numel() : 0, s), "st_map_plan");
  p = made;
  return p;
}

const Plan* MapState::inverse_plan(const Tensor& nbr, int64_t n_in, bool row_order) {
  const int K = (int)nbr.size(1);
  if (K > 32 || !row_order || n_in < kMinRowsForOrder) return nullptr;
  std::lock_guard<std::recursive_mutex> lock(mu_);
  if (inverse_plan_.n_rows == n_in) return &inverse_plan_;
  const c10::cuda::OptionalCUDAGuard guard(nbr.device());
  const cudaStream_t s = stream_of(nbr);
  Plan made;
  make_plan(&made, nbr, n_in, K, true, true);
  Tensor ws = bytes_on(nbr, st_map_plan_balanced_workspace_bytes(n_in, K));
  Stage stage("map_plan_inverse", s);
  check(st_map_plan_inverse_balanced(nbr.data_ptr<int32_t>(), nbr.size(0), K, n_in, order_of(made), tmap_of(made), tmask_of(made),
                            ws.data_ptr(), ws.numel(), s), "st_map_plan_inverse_balanced");
  inverse_plan_ = made;
  return &inverse_plan_;
}

Tensor MapState::inverse(const Tensor& nbr, int64_t n_in) {
  std::lock_guard<std::recursive_mutex> lock(mu_);
  if (inverse_.defined() && inverse_.size(0) == n_in) return inverse_;
  const c10::cuda::OptionalCUDAGuard guard(nbr.device());
  const cudaStream_t s = stream_of(nbr);
  const int K = (int)nbr.size(1);
  Tensor inv = empty_like_on(nbr, {n_in, K}, at::kInt);
  Stage stage("map_invert", s);
  check(st_map_invert(nbr.data_ptr<int32_t>(), nbr.size(0), K, n_in, inv.data_ptr<int32_t>(), s), "st_map_invert");
  inverse_ = inv;
  inverse_state_ = c10::make_intrusive<MapState>();
  return inverse_;
}

MapPtr MapState::inverse_state(const Tensor& nbr, int64_t n_in) {
  std::lock_guard<std::recursive_mutex> lock(mu_);
  inverse(nbr, n_in);
  return inverse_state_;
}

void MapState::expect_flag(const Tensor& nbr, const int32_t* word, cudaStream_t stream) {
  std::lock_guard<std::recursive_mutex> lock(mu_);
  flag_ = std::make_unique<Mail>(nbr);
  flag_stream_ = stream;
  check(st_publish(word, 1, 0, flag_->host(), flag_->ticket(), stream), "st_publish");
  flag_->sent();
}

// True for a submanifold map whose builder found every row under its own coordinate: then nbr[o,k] = i <=> nbr[i,K-1-k] = o.
bool MapState::symmetric(const Tensor& nbr, int64_t n_in) {
  if (nbr.size(0) != n_in) return false;
  std::lock_guard<std::recursive_mutex> lock(mu_);
  if (symmetric_ < 0 && flag_) {
    flag_->wait(flag_stream_);
    symmetric_ = flag_->host()[0] == 0;
    flag_.reset();
  }
  return symmetric_ == 1;
}

double MapState::pairs(const Tensor& nbr) {
  std::lock_guard<std::recursive_mutex> lock(mu_);
  if (pairs_ < 0) pairs_ = (double)nbr.ge(0).sum().item<int64_t>();
  return pairs_;
}

// ------------------------------------------------------------------------------------------------ tables and maps
// k = (ix*ks + iy)*ks + iz; base = (i - ks//2) * dilation per axis (kmap.py:104-132); normal: -base + padding -
// ((ks-1)*dilation)//2 (:135-156); transposed: the negation (:159-180).
std::vector<int32_t> kernel_offsets(int k, int d, int p, bool transposed) {
  const int half = ((k - 1) * d) / 2, sign = transposed ? 1 : -1, shift = transposed ? half - p : p - half;
  std::vector<int32_t> out;
  out.reserve((size_t)k * k * k * 3);
  auto one = [&](int i) { return sign * (i - k / 2) * d + shift; };
  for (int x = 0; x < k; ++x)
    for (int y = 0; y < k; ++y)
      for (int z = 0; z < k; ++z) {
        out.push_back(one(x));
        out.push_back(one(y));
        out.push_back(one(z));
      }
  return out;
}

std::tuple<Tensor, Tensor, Tensor> build_table(const Tensor& coords_in, double factor) {
  const Tensor coords = coords_in.contiguous();
  const int64_t n = coords.size(0);
  // In a small table the longest run of occupied slots, walked by dependent atomics, is what the insert waits for: twice the
  // slots for up to 64 k rows (4096 rows: 13 -> 6 us).
  if (n <= 65536) factor *= 2;
  int64_t want = (int64_t)((double)n * factor), capacity = 1;
  while (capacity < want) capacity <<= 1;
  const c10::cuda::OptionalCUDAGuard guard(coords.device());
  const cudaStream_t s = stream_of(coords);
  const int code = coord_code(coords);
  Tensor keys = empty_like_on(coords, {capacity}, at::kLong), vals = empty_like_on(coords, {capacity}, at::kInt);
  Tensor status = empty_like_on(coords, {2}, at::kInt);       // the table's status word, and one for the map's builder
  {
    Stage stage("hash_clear", s);
    check(st_hash_clear_words(keys.data_ptr<int64_t>(), vals.data_ptr<int32_t>(), capacity, status.data_ptr<int32_t>(), 2, s),
          "st_hash_clear");
  }
  if (n > 0) {
    Stage stage("hash_build", s);
    check(st_hash_build(coords.data_ptr(), n, code, keys.data_ptr<int64_t>(), vals.data_ptr<int32_t>(), capacity,
                        status.data_ptr<int32_t>(), s), "st_hash_build");
  }
  return {keys, vals, status};
}

std::tuple<Tensor, MapPtr> probe_map(const Tensor& coords_in, const std::vector<int32_t>& offsets,
                                     const std::vector<int64_t>& shape64, int stride, const Tensor& keys, const Tensor& vals,
                                     bool rows_of_table) {
  const Tensor coords = coords_in.contiguous();
  const int64_t n = coords.size(0);
  const int K = (int)(offsets.size() / 3);
  const std::vector<int32_t> shape = as_i32(shape64);
  const c10::cuda::OptionalCUDAGuard guard(coords.device());
  const cudaStream_t s = stream_of(coords);
  const int code = coord_code(coords);
  Tensor nbr = empty_like_on(coords, {n, K}, at::kInt);
  MapPtr state = c10::make_intrusive<MapState>();
  if (n == 0) return {nbr, state};
  // Submanifold layer (the queries are the rows the table was built from, stride 1, odd kernel): offsets come in opposite
  // pairs, so half of the probes give the whole map.
  bool mirrored = rows_of_table && stride == 1 && K % 2 == 1;
  for (int i = 0; mirrored && i < 3 * K; ++i) mirrored = offsets[i] == -offsets[3 * (K - 1) - 3 * (i / 3) + i % 3];
  Stage stage("map_build", s);
  if (mirrored) {
    Tensor asym = empty_like_on(coords, {1}, at::kInt);
    const int64_t bytes = st_map_build_symmetric_workspace_bytes(n, K);
    Tensor ws = bytes > 0 ? bytes_on(coords, bytes) : Tensor();
    check(st_map_build_symmetric_ws(coords.data_ptr(), n, code, offsets.data(), K, shape.data(), keys.data_ptr<int64_t>(),
                                    vals.data_ptr<int32_t>(), keys.size(0), nbr.data_ptr<int32_t>(), asym.data_ptr<int32_t>(),
                                    bytes > 0 ? ws.data_ptr() : nullptr, bytes, s), "st_map_build_symmetric");
    state->expect_flag(nbr, asym.data_ptr<int32_t>(), s);
  } else {
    check(st_map_build(coords.data_ptr(), n, code, offsets.data(), K, stride, shape.data(), keys.data_ptr<int64_t>(),
                       vals.data_ptr<int32_t>(), keys.size(0), nbr.data_ptr<int32_t>(), s), "st_map_build");
  }
  return {nbr, state};
}

std::tuple<Tensor, Tensor, Tensor, Tensor, MapPtr> submanifold(const Tensor& coords, std::vector<int64_t> shape, int k, int d,
                                                              double factor, const c10::optional<Tensor>& keys_in,
                                                              const c10::optional<Tensor>& vals_in) {
  Tensor keys, vals, status;
  if (keys_in && vals_in) {
    keys = *keys_in;
    vals = *vals_in;
  } else {
    std::tie(keys, vals, status) = build_table(coords, factor);
  }
  Tensor nbr;
  MapPtr state;
  std::tie(nbr, state) = probe_map(coords, kernel_offsets(k, d, ((k - 1) * d) / 2, false), shape, 1, keys, vals, true);
  return {keys, vals, status, nbr, state};
}

std::vector<int64_t> extent(const Tensor& coords_in) {
  const Tensor coords = coords_in.contiguous();
  const c10::cuda::OptionalCUDAGuard guard(coords.device());
  const cudaStream_t s = stream_of(coords);
  Mail mail(coords);
  check(st_coord_extent(coords.data_ptr(), coords.size(0), coord_code(coords), mail.scratch(), mail.host(), mail.ticket(), s),
        "st_coord_extent");
  mail.sent();
  mail.wait(s);
  return {mail.host()[0], mail.host()[1], mail.host()[2], mail.host()[3]};
}

// ------------------------------------------------------------------------------------------------ output coordinates
// First half: candidates counted and deduplicated on the current stream, the count on its way to the host.
OutCoords::OutCoords(const Tensor& coords, int k, int s, int d, int p, bool transposed, std::vector<int64_t> new_shape,
                     std::vector<int64_t> in_shape, int64_t batch_bound, bool with_map)
    : coords_(coords.contiguous()), offsets_(kernel_offsets(k, d, p, transposed)), new_shape_(as_i32(new_shape)),
      in_shape_(as_i32(in_shape)), K_(k * k * k), stride_(s), transposed_(transposed), code_(0), n_(coords.size(0)),
      batch_bound_(batch_bound), with_map_(with_map) {
  if (n_ == 0) return;
  code_ = coord_code(coords_);
  const c10::cuda::OptionalCUDAGuard guard(coords_.device());
  stream_ = c10::cuda::getCurrentCUDAStream(coords_.device().index());
  const cudaStream_t st = stream_->stream();
  const int64_t bytes = st_outcoords_workspace_bytes(n_, K_, stride_, transposed_);
  ws_ = bytes_on(coords_, bytes + 256);
  Stage stage("out_coords", st);
  cudaMemsetAsync(ws_.data_ptr(), 0, 16, st);
  check(st_outcoords_count(coords_.data_ptr(), n_, code_, offsets_.data(), K_, stride_, transposed_, new_shape_.data(),
                           (int)batch_bound_, scratch(), bytes, counters(), status(), st), "st_outcoords_count");
  mail_ = std::make_unique<Mail>(coords_);
  // the tensor-core kernels' sticky status words ride along: this is the one wait a step makes anyway
  check(st_publish(reinterpret_cast<const int32_t*>(counters()), 4, 1, mail_->host(), mail_->ticket(), st), "st_publish");
  mail_->sent();
}

// Second half: waits for the count alone, sizes the outputs and launches the rest on the same stream.
std::tuple<Tensor, Tensor, c10::optional<MapPtr>> OutCoords::finish() {
  if (n_ == 0) {
    Tensor out = at::empty({0, 4}, coords_.options());
    if (!with_map_) return {out, Tensor(), c10::nullopt};
    return {out, empty_like_on(coords_, {0, K_}, at::kInt), c10::make_intrusive<MapState>()};
  }
  const c10::cuda::CUDAStreamGuard guard(stream_->unwrap());
  const cudaStream_t st = stream_->stream();
  mail_->wait(st);
  const int32_t* got = mail_->host();
  const int64_t n_out = (int64_t)(uint32_t)got[0] | ((int64_t)got[1] << 32);
  const int flags = got[2];
  if (got[4] & ST_DEV_TIMEOUT) {
    const int where = got[5], block = got[6];
    check(st_device_status_clear(st), "st_device_status_clear");
    throw std::runtime_error("a bounded wait inside a tensor-core kernel expired earlier on this device (wait site " +
                             std::to_string(where) + ", block " + std::to_string(block) +
                             "): results produced since the last check are incomplete");
  }
  if (flags & ST_DEV_TABLE_FULL) throw std::runtime_error("build_out_coords: dedupe table overflow");
  if (flags & ST_DEV_BAD_INDEX)
    throw ValueError("build_out_coords: a batch index lies outside [0, " + std::to_string(batch_bound_) + ") (the batch size given)");
  mail_.reset();
  const int64_t bytes = ws_.numel() - 256;
  Tensor out = at::empty({n_out, 4}, coords_.options().requires_grad(false));
  if (n_out > 0) {
    Stage stage("out_coords", st);
    check(st_outcoords_write(coords_.data_ptr(), n_, code_, offsets_.data(), K_, stride_, transposed_, new_shape_.data(),
                             (int)batch_bound_, scratch(), bytes, out.data_ptr(), n_out, status(), st), "st_outcoords_write");
  }
  if (!with_map_) return {out, Tensor(), c10::nullopt};
  Tensor nbr = empty_like_on(coords_, {n_out, K_}, at::kInt);
  if (n_out > 0) {
    Stage stage("map_scatter", st);
    check(st_outcoords_map(coords_.data_ptr(), n_, code_, offsets_.data(), K_, stride_, transposed_, new_shape_.data(),
                           in_shape_.data(), (int)batch_bound_, scratch(), bytes, nbr.data_ptr<int32_t>(), n_out, st),
          "st_outcoords_map");
  }
  return {out, nbr, c10::make_intrusive<MapState>()};
}

}  // namespace st_host
