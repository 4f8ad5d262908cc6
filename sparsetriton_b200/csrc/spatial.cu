// Pooling and nearest-neighbour upsampling of sparse tensors.
//
// Pooling: every input voxel belongs to exactly one output cell, out = floor((in + padding - ks/2) / stride)
// per axis.  Output rows are the distinct cells in ascending (batch, x, y, z) order.  The cell of every
// input becomes an integer key, the (key, row) pairs are radix-sorted, segment heads are marked and
// scanned, and the features of each output row are reduced over its own contiguous segment of the
// sorted list: no atomics, no -inf / zero prefill, fp32 accumulation in a fixed order.  The backward
// pass is a gather per input row (mean: grad / count; max: grad where the input equals the maximum).
//
// Upsampling: input row i becomes the scale^3 output rows i*scale^3 + (dx*scale + dy)*scale + dz at
// coordinates in*scale + (dx, dy, dz) with the same features; backward sums those rows in fp32.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "common.cuh"
#include "radix_sort.cuh"

namespace st {

namespace {

struct PoolGeom {
  int shift;            // padding - kernel_size / 2
  int stride;
  int lo[3];            // smallest cell index per axis (may be negative)
  int ext[3];           // cells per axis
  int batch;
};

__host__ __device__ __forceinline__ int floor_div(int a, int b) {
  int q = a / b;
  return (a % b != 0 && ((a < 0) != (b < 0))) ? q - 1 : q;
}

struct PoolScratch {
  unsigned long long *keys_a, *keys_b;
  int32_t *vals_a, *vals_b;
  uint32_t *hist, *totals;
  uint32_t* heads;      // per sorted position: 1 at the first element of a segment, then its exclusive scan
  void* scan_tmp;
};

int64_t pool_carve(PoolScratch* s, void* ws, int64_t n) {
  int64_t off = 0;
  auto take = [&](int64_t bytes) {
    char* p = ws ? static_cast<char*>(ws) + off : nullptr;
    off += align_up(bytes > 0 ? bytes : 1, 256);
    return p;
  };
  const int64_t nn = n > 0 ? n : 1;
  s->keys_a = reinterpret_cast<unsigned long long*>(take(nn * 8));
  s->keys_b = reinterpret_cast<unsigned long long*>(take(nn * 8));
  s->vals_a = reinterpret_cast<int32_t*>(take(nn * 4));
  s->vals_b = reinterpret_cast<int32_t*>(take(nn * 4));
  s->hist = reinterpret_cast<uint32_t*>(take(sort_hist_bytes(nn)));
  s->totals = reinterpret_cast<uint32_t*>(take(kBucketsMax * 4));
  s->heads = reinterpret_cast<uint32_t*>(take(nn * 4));
  s->scan_tmp = take(scan_tmp_bytes(nn));
  return off;
}

int key_bits_of(const PoolGeom& g) {
  unsigned long long cells = (unsigned long long)(g.batch > 0 ? g.batch : 1);
  for (int a = 0; a < 3; ++a) cells *= (unsigned long long)(g.ext[a] > 0 ? g.ext[a] : 1);
  int bits = 1;
  while (bits < 64 && (cells >> bits) != 0) ++bits;
  return bits;
}

// key = linear index of the cell in the (batch, ext0, ext1, ext2) box: ascending keys = ascending
// (batch, x, y, z).  Inputs outside the stated grid or batch get the key past every cell (sorted last,
// no output row) and raise ST_DEV_BAD_INDEX.
template <typename CT, typename KeyT>
__global__ void __launch_bounds__(256)
pool_keys_kernel(const CT* __restrict__ coords, int64_t n, PoolGeom g, Int3 in_shape, unsigned long long invalid_key,
                 KeyT* __restrict__ keys, int32_t* __restrict__ vals, int32_t* status) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const int4 c = load_coord<CT>(coords, i);
  unsigned long long key = invalid_key;
  if ((unsigned)c.x < (unsigned)g.batch && (unsigned)c.y < (unsigned)in_shape.x && (unsigned)c.z < (unsigned)in_shape.y &&
      (unsigned)c.w < (unsigned)in_shape.z) {
    const int x = floor_div(c.y + g.shift, g.stride) - g.lo[0];
    const int y = floor_div(c.z + g.shift, g.stride) - g.lo[1];
    const int z = floor_div(c.w + g.shift, g.stride) - g.lo[2];
    key = (((unsigned long long)c.x * g.ext[0] + x) * g.ext[1] + y) * g.ext[2] + z;
  } else {
    atomicOr(status, ST_DEV_BAD_INDEX);
  }
  keys[i] = (KeyT)key;
  vals[i] = (int32_t)i;
}

template <typename KeyT>
__global__ void __launch_bounds__(256)
pool_heads_kernel(const KeyT* __restrict__ sorted_keys, int64_t n, KeyT invalid_key, uint32_t* __restrict__ heads) {
  const int64_t p = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (p >= n) return;
  const KeyT k = sorted_keys[p];
  heads[p] = (k != invalid_key && (p == 0 || sorted_keys[p - 1] != k)) ? 1u : 0u;
}

// After the scan heads[p] = number of segment heads before p.  A head at p opens output row heads[p].
template <typename CT, typename KeyT>
__global__ void __launch_bounds__(256)
pool_write_kernel(const KeyT* __restrict__ sorted_keys, const int32_t* __restrict__ sorted_rows,
                  const uint32_t* __restrict__ heads, int64_t n, int64_t n_out, PoolGeom g, KeyT invalid_key,
                  CT* __restrict__ out_coords, int32_t* __restrict__ in_to_out, int32_t* __restrict__ members,
                  int32_t* __restrict__ seg_start) {
  const int64_t p = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (p > n) return;
  if (p == n) {
    // close the last segment: positions holding the invalid key are not members of any row
    int64_t live = n;
    // (binary search for the first invalid key; sorted last)
    int64_t lo = 0, hi = n;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (sorted_keys[mid] == invalid_key) hi = mid; else lo = mid + 1;
    }
    live = lo;
    seg_start[n_out] = (int32_t)live;
    return;
  }
  const KeyT k = sorted_keys[p];
  const int32_t row = sorted_rows[p];
  members[p] = row;
  if (k == invalid_key) {
    in_to_out[row] = -1;
    return;
  }
  const bool head = p == 0 || sorted_keys[p - 1] != k;
  const uint32_t o = head ? heads[p] : heads[p] - 1u;      // exclusive count of heads before p
  in_to_out[row] = (int32_t)o;
  if (head) {
    seg_start[o] = (int32_t)p;
    unsigned long long r = k;
    const int z = (int)(r % g.ext[2]); r /= g.ext[2];
    const int y = (int)(r % g.ext[1]); r /= g.ext[1];
    const int x = (int)(r % g.ext[0]); r /= g.ext[0];
    store_coord<CT>(out_coords, o, (int)r, x + g.lo[0], y + g.lo[1], z + g.lo[2]);
  }
}

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// 16-byte pieces of feature rows: the forms below run where rows are whole pieces at aligned addresses.  Moving 16 bytes a
// thread instead of one element (and a warp to a cell in the forward pass) took the maximum over the cells of 415 k x 64
// bf16 voxels from 44 to 25 us and its gradient from 133 to 29 us (two passes over 53 MB, 3.7 TB/s).
template <typename T> struct Piece { static constexpr int V = 16 / (int)sizeof(T); };
template <typename T>
__device__ __forceinline__ void unpack(const uint4& r, float (&v)[Piece<T>::V]) {
  const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
  for (int i = 0; i < Piece<T>::V; ++i) v[i] = to_f32<T>(e[i]);
}
template <typename T>
__device__ __forceinline__ uint4 pack(const float (&v)[Piece<T>::V]) {
  uint4 r;
  T* e = reinterpret_cast<T*>(&r);
#pragma unroll
  for (int i = 0; i < Piece<T>::V; ++i) e[i] = from_f32<T>(v[i]);
  return r;
}

// kLanes: lanes that share a row's pieces; the other lanes of the warp take every (32 / kLanes)-th member of the same cell,
// so that a cell of many members is not one serial chain of loads.  0: any number of pieces, one thread per piece.
template <typename T, bool MAX, int kLanes>
__global__ void __launch_bounds__(256)
pool_fwd_vec_kernel(const uint4* __restrict__ feats, int pieces, const int32_t* __restrict__ members,
                    const int32_t* __restrict__ seg_start, int64_t n_out, uint4* __restrict__ out) {
  constexpr int V = Piece<T>::V, kStep = kLanes > 0 ? 32 / kLanes : 1;
  const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int64_t o = kLanes > 0 ? t >> 5 : t / pieces;
  if (o >= n_out) return;
  const int c = kLanes > 0 ? (int)(threadIdx.x & (kLanes - 1)) : (int)(t - o * pieces);
  const int mine = kLanes > 0 ? (int)(threadIdx.x & 31) / (kLanes > 0 ? kLanes : 1) : 0;
  const int begin = __ldg(seg_start + o), end = __ldg(seg_start + o + 1);
  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = MAX ? -INFINITY : 0.f;
  auto add = [&](const uint4& r) {
    float v[V];
    unpack<T>(r, v);
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = MAX ? fmaxf(acc[i], v[i]) : acc[i] + v[i];
  };
  int p = begin + mine;
  for (; p + 3 * kStep < end; p += 4 * kStep) {
    int64_t row[4];
    uint4 r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) row[j] = __ldg(members + p + j * kStep);
#pragma unroll
    for (int j = 0; j < 4; ++j) r[j] = __ldg(feats + row[j] * pieces + c);
#pragma unroll
    for (int j = 0; j < 4; ++j) add(r[j]);
  }
  for (; p < end; p += kStep) add(__ldg(feats + (int64_t)__ldg(members + p) * pieces + c));
  if (kLanes > 0) {
#pragma unroll
    for (int d = kLanes > 0 ? kLanes : 32; d < 32; d <<= 1)
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const float v = __shfl_xor_sync(0xFFFFFFFFu, acc[i], d);
        acc[i] = MAX ? fmaxf(acc[i], v) : acc[i] + v;
      }
    if (mine != 0) return;
  }
  if (!MAX) {
    const float count = (float)(end - begin);
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] /= count;
  }
  out[o * pieces + c] = pack<T>(acc);
}

template <typename T, bool MAX>
__global__ void __launch_bounds__(256)
pool_bwd_vec_kernel(const uint4* __restrict__ grad_out, const uint4* __restrict__ feats, const uint4* __restrict__ out, int pieces,
                    const int32_t* __restrict__ in_to_out, const int32_t* __restrict__ seg_start, int64_t n,
                    uint4* __restrict__ grad_in) {
  constexpr int V = Piece<T>::V;
  const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int64_t i = t / pieces;
  if (i >= n) return;
  const int c = (int)(t - i * pieces);
  const int32_t o = __ldg(in_to_out + i);
  float g[V];
#pragma unroll
  for (int j = 0; j < V; ++j) g[j] = 0.f;
  if (o >= 0) {
    unpack<T>(__ldg(grad_out + (int64_t)o * pieces + c), g);
    if (MAX) {
      float x[V], m[V];
      unpack<T>(__ldg(feats + t), x);
      unpack<T>(__ldg(out + (int64_t)o * pieces + c), m);
#pragma unroll
      for (int j = 0; j < V; ++j)
        if (!(x[j] == m[j])) g[j] = 0.f;
    } else {
      const float count = (float)(__ldg(seg_start + o + 1) - __ldg(seg_start + o));
#pragma unroll
      for (int j = 0; j < V; ++j) g[j] = g[j] / count;
    }
  }
  grad_in[t] = pack<T>(g);
}

// One thread per (output row, channel): consecutive threads read consecutive channels of the same
// member rows.  MAX = false: mean over the segment; true: maximum.
template <typename T, bool MAX>
__global__ void __launch_bounds__(256)
pool_fwd_kernel(const T* __restrict__ feats, int C, const int32_t* __restrict__ members,
                const int32_t* __restrict__ seg_start, int64_t n_out, T* __restrict__ out) {
  const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int64_t o = t / C;
  if (o >= n_out) return;
  const int c = (int)(t - o * C);
  const int begin = __ldg(seg_start + o), end = __ldg(seg_start + o + 1);
  float acc = MAX ? -INFINITY : 0.f;
  for (int p = begin; p < end; ++p) {
    const float v = to_f32<T>(feats[(int64_t)__ldg(members + p) * C + c]);
    acc = MAX ? fmaxf(acc, v) : acc + v;
  }
  if (!MAX) acc /= (float)(end - begin);
  out[t] = from_f32<T>(acc);
}

template <typename T, bool MAX>
__global__ void __launch_bounds__(256)
pool_bwd_kernel(const T* __restrict__ grad_out, const T* __restrict__ feats, const T* __restrict__ out, int C,
                const int32_t* __restrict__ in_to_out, const int32_t* __restrict__ seg_start, int64_t n,
                T* __restrict__ grad_in) {
  const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int64_t i = t / C;
  if (i >= n) return;
  const int c = (int)(t - i * C);
  const int32_t o = __ldg(in_to_out + i);
  float g = 0.f;
  if (o >= 0) {
    const float go = to_f32<T>(grad_out[(int64_t)o * C + c]);
    if (MAX) {
      // every input that equals the maximum receives the gradient, as the reference's `in == out` test does
      g = (to_f32<T>(feats[t]) == to_f32<T>(out[(int64_t)o * C + c])) ? go : 0.f;
    } else {
      g = go / (float)(__ldg(seg_start + o + 1) - __ldg(seg_start + o));
    }
  }
  grad_in[t] = from_f32<T>(g);
}

template <typename CT, typename T>
__global__ void __launch_bounds__(256)
upsample_fwd_kernel(const T* __restrict__ feats, const CT* __restrict__ coords, int64_t n, int C, int scale,
                    T* __restrict__ out_feats, CT* __restrict__ out_coords) {
  // thread = (output row, channel); channel 0 also writes the coordinate
  const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int s3 = scale * scale * scale;
  const int64_t o = t / C;
  if (o >= n * s3) return;
  const int c = (int)(t - o * C);
  const int64_t i = o / s3;
  const int step = (int)(o - i * s3);
  out_feats[t] = feats[i * C + c];
  if (c == 0) {
    const int4 q = load_coord<CT>(coords, i);
    const int dz = step % scale, dy = (step / scale) % scale, dx = step / (scale * scale);
    store_coord<CT>(out_coords, o, q.x, q.y * scale + dx, q.z * scale + dy, q.w * scale + dz);
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
upsample_bwd_kernel(const T* __restrict__ grad_out, int64_t n, int C, int s3, T* __restrict__ grad_in) {
  const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int64_t i = t / C;
  if (i >= n) return;
  const int c = (int)(t - i * C);
  float acc = 0.f;
  for (int step = 0; step < s3; ++step) acc += to_f32<T>(grad_out[(i * s3 + step) * C + c]);
  grad_in[t] = from_f32<T>(acc);
}

bool whole_pieces(int C, int esize, const void* a, const void* b, const void* c = nullptr, const void* d = nullptr) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
                        reinterpret_cast<uintptr_t>(d);
  return (C * esize) % 16 == 0 && (all & 15) == 0;
}

bool pool_geom(int ks, int pad, int stride, const int32_t* shape_host, int batch, PoolGeom* g) {
  if (ks < 1 || stride < 1 || !shape_host || batch < 0) return false;
  g->shift = pad - ks / 2;
  g->stride = stride;
  g->batch = batch;
  for (int a = 0; a < 3; ++a) {
    if (shape_host[a] < 0) return false;
    g->lo[a] = floor_div(g->shift, stride);
    const int hi = floor_div((shape_host[a] > 0 ? shape_host[a] - 1 : 0) + g->shift, stride);
    g->ext[a] = hi - g->lo[a] + 1;
  }
  return true;
}

}  // namespace
}  // namespace st

using namespace st;

#define ST_FEAT_DISPATCH(dtype, ...)                                  \
  switch (dtype) {                                                      \
    case ST_F32: { using T = float; __VA_ARGS__; break; }                      \
    case ST_F16: { using T = __half; __VA_ARGS__; break; }                     \
    case ST_BF16: { using T = __nv_bfloat16; __VA_ARGS__; break; }             \
    default: set_error("unknown feature dtype %d", dtype); return ST_ERR_DTYPE; \
  }

extern "C" {

int64_t st_pool_workspace_bytes(int64_t n) {
  PoolScratch s;
  return pool_carve(&s, nullptr, n);
}

int st_pool_count(const void* coords, int64_t n, int coord_dtype, int kernel_size, int padding, int stride,
                  const int32_t* shape_host, int batch, void* workspace, int64_t workspace_bytes, int64_t* n_out,
                  int32_t* status, void* stream) {
  PoolGeom g;
  if (n < 0 || n > 0x7FFFFFFFll || !n_out || !status || !pool_geom(kernel_size, padding, stride, shape_host, batch, &g) ||
      (n > 0 && (!coords || !workspace))) {
    set_error("st_pool_count: bad arguments");
    return ST_ERR_ARG;
  }
  if (coord_dtype != ST_I16 && coord_dtype != ST_I32) {
    set_error("st_pool_count: unknown coordinate dtype %d", coord_dtype);
    return ST_ERR_DTYPE;
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (n == 0) return exclusive_scan_u32(nullptr, nullptr, 0, nullptr, n_out, s);
  PoolScratch w;
  if (workspace_bytes < pool_carve(&w, workspace, n) || (reinterpret_cast<uintptr_t>(workspace) & 255)) {
    set_error("st_pool_count: workspace too small or not 256-byte aligned");
    return ST_ERR_WORKSPACE;
  }
  const int bits = key_bits_of(g);           // keys 0 .. cells-1 are real cells, `cells` itself marks invalid rows
  if (bits > 62) {
    set_error("st_pool_count: grid of more than 2^62 cells");
    return ST_ERR_UNSUPPORTED;
  }
  unsigned long long cells = (unsigned long long)(g.batch > 0 ? g.batch : 1);
  for (int a = 0; a < 3; ++a) cells *= (unsigned long long)(g.ext[a] > 0 ? g.ext[a] : 1);
  const Int3 in_shape = {shape_host[0], shape_host[1], shape_host[2]};
  const unsigned grid = (unsigned)((n + 255) / 256);
  auto sort_by_cell = [&](auto* tag) {
    using KeyT = std::remove_pointer_t<decltype(tag)>;
    KeyT *keys_a = reinterpret_cast<KeyT*>(w.keys_a), *keys_b = reinterpret_cast<KeyT*>(w.keys_b), *sorted_keys = nullptr;
    if (coord_dtype == ST_I32)
      pool_keys_kernel<int32_t, KeyT><<<grid, 256, 0, s>>>(static_cast<const int32_t*>(coords), n, g, in_shape, cells, keys_a,
                                                           w.vals_a, status);
    else
      pool_keys_kernel<int16_t, KeyT><<<grid, 256, 0, s>>>(static_cast<const int16_t*>(coords), n, g, in_shape, cells, keys_a,
                                                           w.vals_a, status);
    radix_sort_pairs<KeyT>(keys_a, w.vals_a, keys_b, w.vals_b, n, bits, w.hist, w.totals, &sorted_keys, nullptr, s);
    pool_heads_kernel<KeyT><<<grid, 256, 0, s>>>(sorted_keys, n, (KeyT)cells, w.heads);
    note_launches(2);
  };
  if (bits <= 32) sort_by_cell(static_cast<uint32_t*>(nullptr));
  else sort_by_cell(static_cast<unsigned long long*>(nullptr));
  int rc = check_launch("st_pool_count");
  if (rc != ST_OK) return rc;
  return exclusive_scan_u32(w.heads, w.heads, n, w.scan_tmp, n_out, s);
}

int st_pool_write(const void* coords, int64_t n, int coord_dtype, int kernel_size, int padding, int stride,
                  const int32_t* shape_host, int batch, void* workspace, int64_t workspace_bytes, void* out_coords,
                  int64_t n_out, int32_t* in_to_out, int32_t* members, int32_t* seg_start, void* stream) {
  PoolGeom g;
  if (n < 0 || n_out < 0 || !pool_geom(kernel_size, padding, stride, shape_host, batch, &g) || !seg_start ||
      (n > 0 && (!coords || !workspace || !in_to_out || !members)) || (n_out > 0 && !out_coords)) {
    set_error("st_pool_write: bad arguments");
    return ST_ERR_ARG;
  }
  if (coord_dtype != ST_I16 && coord_dtype != ST_I32) {
    set_error("st_pool_write: unknown coordinate dtype %d", coord_dtype);
    return ST_ERR_DTYPE;
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (n == 0) {
    cudaMemsetAsync(seg_start, 0, sizeof(int32_t), s);
    return check_launch("st_pool_write");
  }
  PoolScratch w;
  if (workspace_bytes < pool_carve(&w, workspace, n)) {
    set_error("st_pool_write: workspace too small");
    return ST_ERR_WORKSPACE;
  }
  unsigned long long cells = (unsigned long long)(g.batch > 0 ? g.batch : 1);
  for (int a = 0; a < 3; ++a) cells *= (unsigned long long)(g.ext[a] > 0 ? g.ext[a] : 1);
  // the same pass count as st_pool_count decides which ping-pong buffer holds the sorted pairs
  const bool in_b = sort_passes_for_bits(key_bits_of(g)) % 2 == 1;
  const int32_t* sorted_rows = in_b ? w.vals_b : w.vals_a;
  const unsigned grid = (unsigned)((n + 1 + 255) / 256);
  auto write = [&](auto* tag) {
    using KeyT = std::remove_pointer_t<decltype(tag)>;
    const KeyT* sorted_keys = reinterpret_cast<const KeyT*>(in_b ? w.keys_b : w.keys_a);
    if (coord_dtype == ST_I32)
      pool_write_kernel<int32_t, KeyT><<<grid, 256, 0, s>>>(sorted_keys, sorted_rows, w.heads, n, n_out, g, (KeyT)cells,
                                                            static_cast<int32_t*>(out_coords), in_to_out, members, seg_start);
    else
      pool_write_kernel<int16_t, KeyT><<<grid, 256, 0, s>>>(sorted_keys, sorted_rows, w.heads, n, n_out, g, (KeyT)cells,
                                                            static_cast<int16_t*>(out_coords), in_to_out, members, seg_start);
  };
  if (key_bits_of(g) <= 32) write(static_cast<uint32_t*>(nullptr));
  else write(static_cast<unsigned long long*>(nullptr));
  note_launches(1);
  return check_launch("st_pool_write");
}

int st_pool_fwd(int dtype, const void* feats, int C, const int32_t* members, const int32_t* seg_start, int64_t n_out,
                int mode_max, void* out, void* stream) {
  if (C < 1 || n_out < 0 || (n_out > 0 && (!feats || !members || !seg_start || !out))) {
    set_error("st_pool_fwd: bad arguments");
    return ST_ERR_ARG;
  }
  if (n_out == 0) return ST_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const int esize = dtype == ST_F32 ? 4 : 2;
  if (whole_pieces(C, esize, feats, out)) {
    const int pieces = C * esize / 16;
    const bool shared = pieces <= 16 && (pieces & (pieces - 1)) == 0;
    const unsigned blocks = (unsigned)((n_out * (shared ? 32 : pieces) + 255) / 256);
    ST_FEAT_DISPATCH(dtype, {
      auto kernel = mode_max ? pool_fwd_vec_kernel<T, true, 0> : pool_fwd_vec_kernel<T, false, 0>;
      if (shared && pieces == 1) kernel = mode_max ? pool_fwd_vec_kernel<T, true, 1> : pool_fwd_vec_kernel<T, false, 1>;
      if (shared && pieces == 2) kernel = mode_max ? pool_fwd_vec_kernel<T, true, 2> : pool_fwd_vec_kernel<T, false, 2>;
      if (shared && pieces == 4) kernel = mode_max ? pool_fwd_vec_kernel<T, true, 4> : pool_fwd_vec_kernel<T, false, 4>;
      if (shared && pieces == 8) kernel = mode_max ? pool_fwd_vec_kernel<T, true, 8> : pool_fwd_vec_kernel<T, false, 8>;
      if (shared && pieces == 16) kernel = mode_max ? pool_fwd_vec_kernel<T, true, 16> : pool_fwd_vec_kernel<T, false, 16>;
      kernel<<<blocks, 256, 0, s>>>(static_cast<const uint4*>(feats), pieces, members, seg_start, n_out, static_cast<uint4*>(out));
    });
    note_launches(1);
    return check_launch("st_pool_fwd");
  }
  const unsigned grid = (unsigned)((n_out * C + 255) / 256);
  ST_FEAT_DISPATCH(dtype, {
    if (mode_max)
      pool_fwd_kernel<T, true><<<grid, 256, 0, s>>>(static_cast<const T*>(feats), C, members, seg_start, n_out,
                                                    static_cast<T*>(out));
    else
      pool_fwd_kernel<T, false><<<grid, 256, 0, s>>>(static_cast<const T*>(feats), C, members, seg_start, n_out,
                                                     static_cast<T*>(out));
  });
  note_launches(1);
  return check_launch("st_pool_fwd");
}

int st_pool_bwd(int dtype, const void* grad_out, const void* feats, const void* out, int C, const int32_t* in_to_out,
                const int32_t* seg_start, int64_t n, int mode_max, void* grad_in, void* stream) {
  if (C < 1 || n < 0 || (n > 0 && (!grad_out || !in_to_out || !seg_start || !grad_in || (mode_max && (!feats || !out))))) {
    set_error("st_pool_bwd: bad arguments");
    return ST_ERR_ARG;
  }
  if (n == 0) return ST_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const int esize = dtype == ST_F32 ? 4 : 2;
  if (whole_pieces(C, esize, grad_out, grad_in, mode_max ? feats : nullptr, mode_max ? out : nullptr)) {
    const int pieces = C * esize / 16;
    const unsigned blocks = (unsigned)((n * pieces + 255) / 256);
    ST_FEAT_DISPATCH(dtype, {
      auto kernel = mode_max ? pool_bwd_vec_kernel<T, true> : pool_bwd_vec_kernel<T, false>;
      kernel<<<blocks, 256, 0, s>>>(static_cast<const uint4*>(grad_out), static_cast<const uint4*>(feats),
                                    static_cast<const uint4*>(out), pieces, in_to_out, seg_start, n, static_cast<uint4*>(grad_in));
    });
    note_launches(1);
    return check_launch("st_pool_bwd");
  }
  const unsigned grid = (unsigned)((n * C + 255) / 256);
  ST_FEAT_DISPATCH(dtype, {
    if (mode_max)
      pool_bwd_kernel<T, true><<<grid, 256, 0, s>>>(static_cast<const T*>(grad_out), static_cast<const T*>(feats),
                                                    static_cast<const T*>(out), C, in_to_out, seg_start, n,
                                                    static_cast<T*>(grad_in));
    else
      pool_bwd_kernel<T, false><<<grid, 256, 0, s>>>(static_cast<const T*>(grad_out), nullptr, nullptr, C, in_to_out,
                                                     seg_start, n, static_cast<T*>(grad_in));
  });
  note_launches(1);
  return check_launch("st_pool_bwd");
}

int st_upsample_fwd(int dtype, const void* feats, const void* coords, int coord_dtype, int64_t n, int C, int scale,
                    void* out_feats, void* out_coords, void* stream) {
  if (n < 0 || C < 1 || scale < 1 || (n > 0 && (!feats || !coords || !out_feats || !out_coords))) {
    set_error("st_upsample_fwd: bad arguments");
    return ST_ERR_ARG;
  }
  if (coord_dtype != ST_I16 && coord_dtype != ST_I32) {
    set_error("st_upsample_fwd: unknown coordinate dtype %d", coord_dtype);
    return ST_ERR_DTYPE;
  }
  if (n == 0) return ST_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t threads = n * scale * scale * scale * C;
  const unsigned grid = (unsigned)((threads + 255) / 256);
  ST_FEAT_DISPATCH(dtype, {
    if (coord_dtype == ST_I32)
      upsample_fwd_kernel<int32_t, T><<<grid, 256, 0, s>>>(static_cast<const T*>(feats), static_cast<const int32_t*>(coords),
                                                           n, C, scale, static_cast<T*>(out_feats),
                                                           static_cast<int32_t*>(out_coords));
    else
      upsample_fwd_kernel<int16_t, T><<<grid, 256, 0, s>>>(static_cast<const T*>(feats), static_cast<const int16_t*>(coords),
                                                           n, C, scale, static_cast<T*>(out_feats),
                                                           static_cast<int16_t*>(out_coords));
  });
  note_launches(1);
  return check_launch("st_upsample_fwd");
}

int st_upsample_bwd(int dtype, const void* grad_out, int64_t n, int C, int scale, void* grad_in, void* stream) {
  if (n < 0 || C < 1 || scale < 1 || (n > 0 && (!grad_out || !grad_in))) {
    set_error("st_upsample_bwd: bad arguments");
    return ST_ERR_ARG;
  }
  if (n == 0) return ST_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const unsigned grid = (unsigned)((n * C + 255) / 256);
  ST_FEAT_DISPATCH(dtype, {
    upsample_bwd_kernel<T><<<grid, 256, 0, s>>>(static_cast<const T*>(grad_out), n, C, scale * scale * scale,
                                                static_cast<T*>(grad_in));
  });
  note_launches(1);
  return check_launch("st_upsample_bwd");
}

}  // extern "C"
