// Small kernels that spare the host round trips and launches: results published straight into pinned host memory, the
// extent of a coordinate set, and what batch norm derives from the batch column.
#include "common.cuh"

namespace st {

int tc_status_address(int32_t** out);

namespace {

// host[0 .. n_words) <- words of device memory, then host[15] <- ticket, visible to a polling host in that order.
__global__ void publish_kernel(const int32_t* a, int n_a, const int32_t* b, int n_b, volatile int32_t* host, int32_t ticket) {
  const int i = threadIdx.x;
  if (i < n_a) host[i] = a[i];
  else if (i < n_a + n_b) host[i] = b[i - n_a];
  __threadfence_system();
  __syncwarp();
  if (i == 0) host[15] = ticket;
}

// Largest value of each of the four columns.  scratch: four running maxima (biased to unsigned) and a block counter, all
// zero on entry and again on exit; the last block publishes.  Bound by one pass over the coordinates; 1.2 M int32 rows take
// 5 us where a column-wise reduction took 21.
template <typename CT>
__global__ void __launch_bounds__(256) extent_kernel(const CT* __restrict__ coords, int64_t n, uint32_t* scratch,
                                                     volatile int32_t* host, int32_t ticket) {
  int m[4] = {INT32_MIN, INT32_MIN, INT32_MIN, INT32_MIN};
  const int64_t step = (int64_t)gridDim.x * 256;
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += step) {
    const int4 c = load_coord<CT>(coords, i);
    m[0] = max(m[0], c.x);
    m[1] = max(m[1], c.y);
    m[2] = max(m[2], c.z);
    m[3] = max(m[3], c.w);
  }
  __shared__ int part[8][4];
  __shared__ bool last;
#pragma unroll
  for (int j = 0; j < 4; ++j) m[j] = __reduce_max_sync(0xFFFFFFFFu, m[j]);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int j = 0; j < 4; ++j) part[threadIdx.x >> 5][j] = m[j];
  __syncthreads();
  if (threadIdx.x < 4) {
    int v = part[0][threadIdx.x];
    for (int w = 1; w < 8; ++w) v = max(v, part[w][threadIdx.x]);
    atomicMax(scratch + threadIdx.x, (uint32_t)v ^ 0x80000000u);
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(scratch + 4, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last || threadIdx.x >= 32) return;
  __threadfence();
  if (threadIdx.x < 4) {
    host[threadIdx.x] = (int32_t)(atomicExch(scratch + threadIdx.x, 0u) ^ 0x80000000u);
    __threadfence_system();
  }
  if (threadIdx.x == 0) scratch[4] = 0u;
  __syncwarp();
  if (threadIdx.x == 0) host[15] = ticket;
}

// ids[i] = batch index of row i; counts and first rows per sample.  counts: B + 1 zeros on entry (the last a block counter); the last
// block turns the counts into inv_count = 1 / max(count, 1).  first: all ones on entry.
constexpr int kInfoThreads = 256, kInfoPer = 8, kInfoMaxShared = 1024;
template <typename CT>
__global__ void __launch_bounds__(kInfoThreads)
batch_info_kernel(const CT* __restrict__ coords, int64_t n, int B, int32_t* __restrict__ ids, uint32_t* counts,
                  uint32_t* first, float* inv_count) {
  __shared__ uint32_t local[kInfoMaxShared];
  __shared__ bool last;
  const bool shared = B <= kInfoMaxShared;
  if (shared)
    for (int b = threadIdx.x; b < B; b += kInfoThreads) local[b] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kInfoThreads * kInfoPer;
#pragma unroll
  for (int j = 0; j < kInfoPer; ++j) {
    const int64_t i = base + (int64_t)j * kInfoThreads + threadIdx.x;
    int b = -1;
    bool head = false;
    if (i < n) {
      b = (int)coords[i * 4];
      ids[i] = b;
      head = (unsigned)b < (unsigned)B && (i == 0 || (int)coords[(i - 1) * 4] != b);
    }
    // rows of a batch mostly lie together: one addition per distinct index of the warp
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, b);
    if ((unsigned)b < (unsigned)B && (int)(threadIdx.x & 31) == __ffs(peers) - 1)
      atomicAdd(shared ? &local[b] : counts + b, (uint32_t)__popc(peers));
    if (head) atomicMin(first + b, (uint32_t)i);
  }
  __syncthreads();
  if (shared)
    for (int b = threadIdx.x; b < B; b += kInfoThreads)
      if (local[b]) atomicAdd(counts + b, local[b]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counts + B, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int b = threadIdx.x; b < B; b += kInfoThreads) {
    const uint32_t c = atomicAdd(counts + b, 0u);
    inv_count[b] = 1.f / (float)(c > 1u ? c : 1u);
  }
}

}  // namespace
}  // namespace st

using namespace st;

extern "C" {

int st_publish(const int32_t* words, int n_words, int kernel_status, int32_t* host16, int32_t ticket, void* stream) {
  int32_t* status = nullptr;
  if (n_words < 0 || n_words > 8 || !host16 || (n_words > 0 && !words)) {
    set_error("st_publish: bad arguments");
    return ST_ERR_ARG;
  }
  if (kernel_status) {
    const int rc = tc_status_address(&status);
    if (rc != ST_OK) return rc;
  }
  publish_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(words, n_words, status, kernel_status ? 4 : 0, host16, ticket);
  note_launches(1);
  return check_launch("st_publish");
}

int st_coord_extent(const void* coords, int64_t n, int coord_dtype, uint32_t* scratch, int32_t* host16, int32_t ticket,
                    void* stream) {
  if (n < 1 || !coords || !scratch || !host16) {
    set_error("st_coord_extent: bad arguments");
    return ST_ERR_ARG;
  }
  if (coord_dtype != ST_I16 && coord_dtype != ST_I32) {
    set_error("st_coord_extent: unknown coordinate dtype %d", coord_dtype);
    return ST_ERR_DTYPE;
  }
  int64_t grid = (n + 256 * 4 - 1) / (256 * 4);
  if (grid > 148 * 4) grid = 148 * 4;
  if (coord_dtype == ST_I32)
    extent_kernel<int32_t><<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(static_cast<const int32_t*>(coords), n, scratch, host16,
                                                                             ticket);
  else
    extent_kernel<int16_t><<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(static_cast<const int16_t*>(coords), n, scratch, host16,
                                                                             ticket);
  note_launches(1);
  return check_launch("st_coord_extent");
}

int st_bn_batch_info(const void* coords, int64_t n, int coord_dtype, int B, int32_t* ids, uint32_t* counts, int32_t* first_row,
                     float* inv_count, void* stream) {
  if (n < 0 || n > 0x7FFFFFFFll || B < 1 || !counts || !first_row || !inv_count || (n > 0 && (!coords || !ids))) {
    set_error("st_bn_batch_info: bad arguments");
    return ST_ERR_ARG;
  }
  if (coord_dtype != ST_I16 && coord_dtype != ST_I32) {
    set_error("st_bn_batch_info: unknown coordinate dtype %d", coord_dtype);
    return ST_ERR_DTYPE;
  }
  cudaStream_t s = (cudaStream_t)stream;
  cudaMemsetAsync(counts, 0, sizeof(uint32_t) * ((size_t)B + 2), s);
  cudaMemsetAsync(first_row, 0xFF, sizeof(int32_t) * (size_t)B, s);
  const unsigned grid = (unsigned)((n + kInfoThreads * kInfoPer - 1) / (kInfoThreads * kInfoPer));
  uint32_t* first = reinterpret_cast<uint32_t*>(first_row);
  if (coord_dtype == ST_I32)
    batch_info_kernel<int32_t><<<grid > 0 ? grid : 1, kInfoThreads, 0, s>>>(static_cast<const int32_t*>(coords), n, B, ids, counts,
                                                                            first, inv_count);
  else
    batch_info_kernel<int16_t><<<grid > 0 ? grid : 1, kInfoThreads, 0, s>>>(static_cast<const int16_t*>(coords), n, B, ids, counts,
                                                                            first, inv_count);
  note_launches(1);
  return check_launch("st_bn_batch_info");
}

}  // extern "C"
