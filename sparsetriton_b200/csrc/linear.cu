// Per-voxel linear head: y (n, O) fp32 = x (n, C) W^T + b, its gradients, x in fp32 or 16 bits.
//
// A matrix of a million rows and a few columns is a stream: 144 bytes a row at C = 32 bf16, O = 20, 38 us for 1.7 M rows at the
// copy rate.  As library calls the forward took 460 us (a conversion of x, a GEMM that fills a few lanes per tile, an
// epilogue kernel), the backward 580.  Here a thread has a row in registers and the weights, in shared memory, are read by all lanes
// at once; sums are fp32 in ascending order.  The weight gradient takes chunks of rows into shared memory, a thread has
// 4 x 4 of the products, and the blocks' partial sums are added in a fixed order.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace st {
namespace {

constexpr int kMaxOut = 64;

template <typename T> struct Pack;                            // 16 bytes of features
template <> struct Pack<float> { static constexpr int n = 4; };
template <> struct Pack<__half> { static constexpr int n = 8; };
template <> struct Pack<__nv_bfloat16> { static constexpr int n = 8; };
template <typename T> __device__ __forceinline__ float to_f(T v) { return (float)v; }
template <typename T> __device__ __forceinline__ T of_f(float v);
template <> __device__ __forceinline__ float of_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __half of_f<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 of_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

template <typename T, int C>
__device__ __forceinline__ void load_row(const T* __restrict__ row, float (&v)[C]) {
  constexpr int P = Pack<T>::n;
#pragma unroll
  for (int i = 0; i < C / P; ++i) {
    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(row) + i);
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int j = 0; j < P; ++j) v[i * P + j] = to_f(e[j]);
  }
}

template <typename T, int C>
__global__ void __launch_bounds__(128) linear_fwd_kernel(const T* __restrict__ x, const float* __restrict__ w,
                                                        const float* __restrict__ bias, float* __restrict__ y, int64_t n, int O) {
  __shared__ float4 wt[kMaxOut / 4 * C];                      // [o / 4][c]
  __shared__ float4 b4[kMaxOut / 4];
  for (int i = threadIdx.x; i < O * C; i += 128)
    reinterpret_cast<float*>(wt)[(i / C / 4 * C + i % C) * 4 + i / C % 4] = w[i];
  for (int i = threadIdx.x; i < O; i += 128) reinterpret_cast<float*>(b4)[i] = bias ? bias[i] : 0.f;
  __syncthreads();
  for (int64_t row = (int64_t)blockIdx.x * 128 + threadIdx.x; row < n; row += (int64_t)gridDim.x * 128) {
    float v[C];
    load_row<T, C>(x + row * C, v);
    for (int q = 0; q < O / 4; ++q) {
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const float4 k = wt[q * C + c];
        s.x = fmaf(v[c], k.x, s.x);
        s.y = fmaf(v[c], k.y, s.y);
        s.z = fmaf(v[c], k.z, s.z);
        s.w = fmaf(v[c], k.w, s.w);
      }
      const float4 b = b4[q];
      reinterpret_cast<float4*>(y + row * O)[q] = make_float4(s.x + b.x, s.y + b.y, s.z + b.z, s.w + b.w);
    }
  }
}

template <typename T, int C>
__global__ void __launch_bounds__(128) linear_dx_kernel(const float* __restrict__ dy, const float* __restrict__ w, T* __restrict__ dx,
                                                       int64_t n, int O) {
  __shared__ float4 ws[kMaxOut * C / 4];                      // [o][c / 4]
  for (int i = threadIdx.x; i < O * C; i += 128) reinterpret_cast<float*>(ws)[i] = w[i];
  __syncthreads();
  for (int64_t row = (int64_t)blockIdx.x * 128 + threadIdx.x; row < n; row += (int64_t)gridDim.x * 128) {
    float s[C];
#pragma unroll
    for (int c = 0; c < C; ++c) s[c] = 0.f;
    for (int q = 0; q < O / 4; ++q) {
      const float4 g = __ldg(reinterpret_cast<const float4*>(dy + row * O) + q);
      const float gs[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < C / 4; ++c) {
          const float4 k = ws[(q * 4 + j) * (C / 4) + c];
          s[c * 4] = fmaf(gs[j], k.x, s[c * 4]);
          s[c * 4 + 1] = fmaf(gs[j], k.y, s[c * 4 + 1]);
          s[c * 4 + 2] = fmaf(gs[j], k.z, s[c * 4 + 2]);
          s[c * 4 + 3] = fmaf(gs[j], k.w, s[c * 4 + 3]);
        }
    }
    constexpr int P = Pack<T>::n;
#pragma unroll
    for (int i = 0; i < C / P; ++i) {
      __align__(16) T e[P];
#pragma unroll
      for (int j = 0; j < P; ++j) e[j] = of_f<T>(s[i * P + j]);
      reinterpret_cast<uint4*>(dx + row * C)[i] = *reinterpret_cast<const uint4*>(e);
    }
  }
}

// partial[block][o * C + c], then [O * C + o]: the block's share of dW and db.
constexpr int kChunk = 64;
template <typename T, int C>
__global__ void __launch_bounds__(256) linear_dw_kernel(const T* __restrict__ x, const float* __restrict__ dy,
                                                       float* __restrict__ partial, int64_t n, int O) {
  constexpr int P = Pack<T>::n;
  extern __shared__ float4 smem[];
  float* xs = reinterpret_cast<float*>(smem);                 // [kChunk][C]
  float* gs = xs + kChunk * C;                                // [kChunk][O]
  const int tiles = (O / 4) * (C / 4), slices = 256 / tiles;
  const int tile = threadIdx.x % tiles, slice = threadIdx.x / tiles;
  const int o = tile / (C / 4) * 4, c = tile % (C / 4) * 4;
  float acc[4][4] = {}, db[4] = {};
  for (int64_t r0 = (int64_t)blockIdx.x * kChunk; r0 < n; r0 += (int64_t)gridDim.x * kChunk) {
    const int rows = (int)min((int64_t)kChunk, n - r0);
    for (int i = threadIdx.x; i < rows * C / P; i += 256) {
      const uint4 raw = __ldg(reinterpret_cast<const uint4*>(x + r0 * C) + i);
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int j = 0; j < P; ++j) xs[i * P + j] = to_f(e[j]);
    }
    for (int i = threadIdx.x; i < rows * O / 4; i += 256)
      reinterpret_cast<float4*>(gs)[i] = __ldg(reinterpret_cast<const float4*>(dy + r0 * O) + i);
    __syncthreads();
    if (slice < slices)
      for (int r = slice; r < rows; r += slices) {
        const float4 g = *reinterpret_cast<const float4*>(gs + r * O + o), v = *reinterpret_cast<const float4*>(xs + r * C + c);
        const float ga[4] = {g.x, g.y, g.z, g.w}, va[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          db[a] += ga[a];
#pragma unroll
          for (int b = 0; b < 4; ++b) acc[a][b] = fmaf(ga[a], va[b], acc[a][b]);
        }
      }
    __syncthreads();
  }
  // the slices in order, through shared memory
  float* mine = partial + (size_t)blockIdx.x * (O * C + O);
  float* sum = xs;
  for (int i = threadIdx.x; i < O * C + O; i += 256) sum[i] = 0.f;
  __syncthreads();
  for (int s = 0; s < slices; ++s) {
    if (slice == s) {
#pragma unroll
      for (int a = 0; a < 4; ++a) {
#pragma unroll
        for (int b = 0; b < 4; ++b) sum[(o + a) * C + c + b] += acc[a][b];
        if (c == 0) sum[O * C + o + a] += db[a];
      }
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < O * C + O; i += 256) mine[i] = sum[i];
}

__global__ void __launch_bounds__(256) linear_sum_kernel(const float* __restrict__ partial, int blocks, int count, int n_dw,
                                                        float* __restrict__ dw, float* __restrict__ db) {
  __shared__ float part[8][32];
  const int slice = threadIdx.x >> 5, lane = threadIdx.x & 31, i = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (i < count)
#pragma unroll 8
    for (int b = slice; b < blocks; b += 8) s += partial[(size_t)b * count + i];
  part[slice][lane] = s;
  __syncthreads();
  if (slice == 0 && i < count) {
#pragma unroll
    for (int k = 1; k < 8; ++k) s += part[k][lane];
    if (i < n_dw) dw[i] = s;
    else if (db) db[i - n_dw] = s;
  }
}

int linear_blocks(int64_t n) {
  const int64_t want = (n + kChunk - 1) / kChunk;
  return (int)(want < 4 * 148 ? want : 4 * 148);
}

}  // namespace
}  // namespace st

using namespace st;

extern "C" {

int st_linear_supported(int dtype, int C, int O) {
  return (dtype == ST_F32 || dtype == ST_F16 || dtype == ST_BF16) && (C == 16 || C == 32 || C == 64) && O >= 4 && O % 4 == 0 &&
         O <= kMaxOut;
}

static int linear_args(const char* who, int dtype, const void* a, const void* b, const void* w, int64_t n, int C, int O) {
  if (!st_linear_supported(dtype, C, O)) {
    set_error("%s: %d -> %d channels of type %d are not supported", who, C, O, dtype);
    return ST_ERR_UNSUPPORTED;
  }
  if (n < 0 || (n > 0 && (!a || !b || !w)) || ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15)) {
    set_error("%s: bad arguments", who);
    return ST_ERR_ARG;
  }
  return ST_OK;
}

#define ST_LINEAR(dtype, C, CALL)                                             \
  auto by_width = [&](auto zero) {                                            \
    using T = decltype(zero);                                                 \
    if (C == 16) { constexpr int W = 16; CALL; }                              \
    else if (C == 32) { constexpr int W = 32; CALL; }                         \
    else { constexpr int W = 64; CALL; }                                      \
  };                                                                          \
  if (dtype == ST_F32) by_width(float{});                                     \
  else if (dtype == ST_F16) by_width(__half{});                               \
  else by_width(__nv_bfloat16{});

int st_linear_fwd(int dtype, const void* x, const float* w, const float* bias, float* y, int64_t n, int C, int O, void* stream) {
  int rc = linear_args("st_linear_fwd", dtype, x, y, w, n, C, O);
  if (rc != ST_OK || n == 0) return rc;
  const unsigned grid = (unsigned)((n + 127) / 128 < 16 * 148 ? (n + 127) / 128 : 16 * 148);
  ST_LINEAR(dtype, C, (linear_fwd_kernel<T, W><<<grid, 128, 0, (cudaStream_t)stream>>>(static_cast<const T*>(x), w, bias, y, n, O)))
  note_launches(1);
  return check_launch("st_linear_fwd");
}

int st_linear_dgrad(int dtype, const float* dy, const float* w, void* dx, int64_t n, int C, int O, void* stream) {
  int rc = linear_args("st_linear_dgrad", dtype, dy, dx, w, n, C, O);
  if (rc != ST_OK || n == 0) return rc;
  const unsigned grid = (unsigned)((n + 127) / 128 < 16 * 148 ? (n + 127) / 128 : 16 * 148);
  ST_LINEAR(dtype, C, (linear_dx_kernel<T, W><<<grid, 128, 0, (cudaStream_t)stream>>>(dy, w, static_cast<T*>(dx), n, O)))
  note_launches(1);
  return check_launch("st_linear_dgrad");
}

int64_t st_linear_workspace_bytes(int64_t n, int C, int O) { return (int64_t)linear_blocks(n > 0 ? n : 1) * (O * C + O) * 4; }

int st_linear_wgrad(int dtype, const void* x, const float* dy, float* dw, float* db, int64_t n, int C, int O, void* workspace,
                    int64_t workspace_bytes, void* stream) {
  int rc = linear_args("st_linear_wgrad", dtype, x, dy, dw, n, C, O);
  if (rc != ST_OK) return rc;
  if (n == 0 || !workspace || workspace_bytes < st_linear_workspace_bytes(n, C, O)) {
    set_error("st_linear_wgrad: no rows, or the workspace is too small");
    return ST_ERR_WORKSPACE;
  }
  cudaStream_t s = (cudaStream_t)stream;
  float* partial = static_cast<float*>(workspace);
  const int blocks = linear_blocks(n), count = O * C + O;
  const size_t staged = (size_t)kChunk * (C + O) * 4, summed = (size_t)count * 4, smem = staged > summed ? staged : summed;
  ST_LINEAR(dtype, C, (linear_dw_kernel<T, W><<<blocks, 256, smem, s>>>(static_cast<const T*>(x), dy, partial, n, O)))
  linear_sum_kernel<<<(count + 31) / 32, 256, 0, s>>>(partial, blocks, count, O * C, dw, db);
  note_launches(2);
  return check_launch("st_linear_wgrad");
}

}  // extern "C"
