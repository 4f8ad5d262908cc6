// Row order of a neighbour map for the tensor-core kernels.
//
// The implicit-GEMM kernels work on tiles of 128 rows and skip a kernel offset for a tile only when
// none of its 128 rows has a neighbour there.  In the natural row order nearly every tile touches
// nearly every offset, and 70-80 % of what the tensor cores multiply is zero fill.  Rows with the
// same set of occupied offsets behave alike, so the kernels may walk the rows in the order of their
// K-bit occupancy mask instead: tiles then share masks, far fewer (tile, offset) stages remain and
// those are denser.  The order only decides which rows share a tile; every row's own sum still
// runs over the offsets in ascending k, so forward and feature-gradient results do not depend on it.
//
// order = stable LSD radix sort of the rows by mask (9-bit digits); equal masks keep their original
// order and no atomic decides a position, so the result is deterministic.
#include "common.cuh"
#include "radix_sort.cuh"

namespace st {

namespace {

// key[r] = occupancy mask of row r (bit k: nbr[r,k] >= 0) for K <= 32, a 32-bit hash of the whole
// pattern beyond (equal patterns still get equal keys); val[r] = r.
__global__ void __launch_bounds__(128) row_keys_kernel(const int32_t* __restrict__ nbr, int64_t n, int K,
                                                      uint32_t* __restrict__ keys, int32_t* __restrict__ vals,
                                                      uint32_t* ticket) {
  extern __shared__ int32_t stage[];                     // 128 rows x K entries when K <= 64
  if (ticket && blockIdx.x == 0 && threadIdx.x == 0) *ticket = 0;
  const int64_t row0 = (int64_t)blockIdx.x * 128;
  const int rows = (int)min((int64_t)128, n - row0);
  const int64_t row = row0 + threadIdx.x;
  uint32_t key = 0;
  if (K <= 64) {
    const int32_t* src = nbr + row0 * K;
    for (int e = threadIdx.x; e < rows * K; e += 128) stage[e] = __ldg(src + e);
    __syncthreads();
    if (threadIdx.x < rows) {
      const int32_t* mine = stage + threadIdx.x * K;
      if (K <= 32) {
        for (int k = 0; k < K; ++k) key |= (mine[k] >= 0 ? 1u : 0u) << k;
      } else {
        for (int k = 0; k < K; ++k) key = key * 0x9E3779B1u + (mine[k] >= 0 ? (uint32_t)(k + 1) : 0u);
      }
    }
  } else if (threadIdx.x < rows) {
    for (int k = 0; k < K; ++k) key = key * 0x9E3779B1u + (__ldg(nbr + row * K + k) >= 0 ? (uint32_t)(k + 1) : 0u);
  }
  if (threadIdx.x < rows) {
    keys[row] = key;
    vals[row] = (int32_t)row;
  }
}

// Tile plan: the map re-laid so that the 128 source rows of one (tile, offset) step are one
// contiguous 512-byte line, in the row order the kernels walk, plus a per-tile bit mask of the
// offsets that have a neighbour anywhere in the tile.
//   tmap [(tile * K + k) * 128 + r] = nbr[order[tile * 128 + r], k]      (-1 past the last row)
//   tmask[tile * MW + k / 32] bit (k % 32)                                 MW = ceil(K / 32)
// One block per tile.  A warp reads one row at a time as a run of consecutive entries (a warp-wide
// load touches one or two lines, not 32) into shared memory, `kPlanChunk` offsets at a time, with the
// loads of eight rows in flight together; the block writes them back transposed.
constexpr int kPlanChunk = 64;

__global__ void __launch_bounds__(128) plan_tiles_kernel(const int32_t* __restrict__ nbr,
                                                        const int32_t* __restrict__ order, int64_t n_rows, int K,
                                                        int MW, int32_t* __restrict__ tmap,
                                                        uint32_t* __restrict__ tmask) {
  extern __shared__ int32_t stage[];                      // 128 x (min(K, kPlanChunk) | 1) entries
  __shared__ int64_t src_row[128];
  __shared__ uint32_t mask_word[2];                       // the (at most two) mask words of a chunk
  const int64_t tile = blockIdx.x;
  const int r = threadIdx.x, warp = r >> 5, lane = r & 31;
  const int64_t pos = tile * 128 + r;
  src_row[r] = pos < n_rows ? (order ? (int64_t)__ldg(order + pos) : pos) : -1;
  for (int k0 = 0; k0 < K; k0 += kPlanChunk) {
    const int kc = min(kPlanChunk, K - k0);
    const int pitch = kc | 1;                              // odd: conflict-free column reads
    if (r < 2) mask_word[r] = 0;
    __syncthreads();
    // a warp per row: lane l fetches entries l and l + 32 of the chunk, eight rows' loads issued together
#pragma unroll 8
    for (int row = warp; row < 128; row += 4) {
      const int64_t src = src_row[row];
      const int32_t* from = nbr + src * K + k0;
      const int32_t lo = (src >= 0 && lane < kc) ? __ldg(from + lane) : -1;
      const int32_t hi = (src >= 0 && lane + 32 < kc) ? __ldg(from + lane + 32) : -1;
      if (lane < kc) stage[row * pitch + lane] = lo;
      if (lane + 32 < kc) stage[row * pitch + lane + 32] = hi;
    }
    __syncthreads();
    for (int k = 0; k < kc; ++k) {
      const int32_t v = stage[r * pitch + k];
      tmap[(tile * K + k0 + k) * 128 + r] = v;
      const uint32_t any = __ballot_sync(0xFFFFFFFFu, v >= 0);
      if (any && lane == 0) atomicOr(&mask_word[k >> 5], 1u << (k & 31));
    }
    __syncthreads();
    if (r < (kc + 31) / 32) tmask[tile * MW + (k0 >> 5) + r] = mask_word[r];
    __syncthreads();
  }
}

struct OrderScratch {
  uint32_t *keys_a, *keys_b, *hist, *totals;
  int32_t* vals_b;
};

int64_t carve(OrderScratch* s, void* ws, int64_t n, int K) {
  (void)K;
  int64_t off = 0;
  auto take = [&](int64_t bytes) {
    char* p = ws ? static_cast<char*>(ws) + off : nullptr;
    off += align_up(bytes > 0 ? bytes : 1, 256);
    return p;
  };
  const int64_t nn = n > 0 ? n : 1;
  s->keys_a = reinterpret_cast<uint32_t*>(take(nn * 4));
  s->keys_b = reinterpret_cast<uint32_t*>(take(nn * 4));
  s->vals_b = reinterpret_cast<int32_t*>(take(nn * 4));
  s->hist = reinterpret_cast<uint32_t*>(take(sort_hist_bytes(nn)));
  s->totals = reinterpret_cast<uint32_t*>(take(kBucketsMax * 4));
  return off;
}

// The radix passes over (keys, row ids) already placed in (s.keys_a, start of the value ping-pong);
// the sorted row ids land in `order`, the sorted keys in *sorted_keys.
int passes_for(int K) { return ((K < 32 ? K : 32) + kDigitBitsMax - 1) / kDigitBitsMax; }
int32_t* first_vals(const OrderScratch& s, int K, int32_t* order) { return passes_for(K) % 2 == 0 ? order : s.vals_b; }

void sort_passes(const OrderScratch& s, int64_t n_rows, int K, int32_t* order, uint32_t** sorted_keys, cudaStream_t st) {
  const int key_bits = K < 32 ? K : 32;
  // ping-pong so that the last pass lands in `order`
  int32_t* vals_in = first_vals(s, K, order);
  int32_t* vals_alt = vals_in == order ? s.vals_b : order;
  radix_sort_pairs<uint32_t>(s.keys_a, vals_in, s.keys_b, vals_alt, n_rows, key_bits, s.hist, s.totals, sorted_keys,
                             nullptr, st);
}

// ---- plan of the INVERSE map straight from the forward map (K <= 32), without writing the inverse ----
__global__ void __launch_bounds__(256) iota_clear_kernel(uint32_t* keys, int32_t* vals, int64_t n, uint32_t* ticket) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (ticket && i == 0) *ticket = 0;
  if (i < n) {
    keys[i] = 0u;
    vals[i] = (int32_t)i;
  }
}

// keys[i] |= 1 << k for every nbr[o,k] = i: the occupancy mask of row i of the inverse map.
// kFlatQuads runs of four consecutive entries per thread (16-byte loads, all issued before they are used).
constexpr int kFlatQuads = 4;
constexpr int kFlatPerBlock = 256 * 4 * kFlatQuads;

__device__ __forceinline__ void load_quads(const int32_t* __restrict__ nbr, int64_t n_flat, int64_t block_first,
                                           int32_t (&v)[kFlatQuads][4]) {
  const bool aligned = (reinterpret_cast<uintptr_t>(nbr) & 15) == 0;
#pragma unroll
  for (int q = 0; q < kFlatQuads; ++q) {
    const int64_t t0 = block_first + ((int64_t)q * 256 + threadIdx.x) * 4;
    v[q][0] = v[q][1] = v[q][2] = v[q][3] = -1;
    if (t0 + 3 < n_flat && aligned) {
      const int4 w = __ldg(reinterpret_cast<const int4*>(nbr + t0));
      v[q][0] = w.x; v[q][1] = w.y; v[q][2] = w.z; v[q][3] = w.w;
    } else {
      for (int j = 0; j < 4 && t0 + j < n_flat; ++j) v[q][j] = __ldg(nbr + t0 + j);
    }
  }
}

// IndexT: the type the flat index is divided in (32 bits when the map has fewer than 2^31 entries: a 64-bit division
// per run made these kernels instruction-bound).
template <typename IndexT>
__global__ void __launch_bounds__(256)
inverse_keys_kernel(const int32_t* __restrict__ nbr, int64_t n_flat, int K, int64_t n_in, uint32_t* keys) {
  const int64_t block_first = (int64_t)blockIdx.x * kFlatPerBlock;
  int32_t v[kFlatQuads][4];
  load_quads(nbr, n_flat, block_first, v);
#pragma unroll
  for (int q = 0; q < kFlatQuads; ++q) {
    const int64_t t0 = block_first + ((int64_t)q * 256 + threadIdx.x) * 4;
    int k = (int)((IndexT)t0 % (IndexT)K);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (v[q][j] >= 0 && v[q][j] < n_in) atomicOr(keys + v[q][j], 1u << k);
      if (++k == K) k = 0;
    }
  }
}

__global__ void __launch_bounds__(256) rank_kernel(const int32_t* __restrict__ order, int64_t n, int32_t* rank) {
  const int64_t p = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (p < n) rank[order[p]] = (int32_t)p;
}

// tmask[tile] = OR of the tile's 128 sorted keys (K <= 32: one word per tile)
__global__ void __launch_bounds__(128) tile_mask_kernel(const uint32_t* __restrict__ sorted_keys, int64_t n,
                                                       uint32_t* __restrict__ tmask) {
  __shared__ uint32_t part[4];
  const int64_t p = (int64_t)blockIdx.x * 128 + threadIdx.x;
  const uint32_t m = __reduce_or_sync(0xFFFFFFFFu, p < n ? sorted_keys[p] : 0u);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) tmask[blockIdx.x] = part[0] | part[1] | part[2] | part[3];
}

// tmap_inv[(tile(pos) * K + k) * 128 + pos % 128] = o for nbr[o,k] = i, pos = rank[i]; tmap_inv holds -1
template <typename IndexT>
__global__ void __launch_bounds__(256)
inverse_plan_scatter_kernel(const int32_t* __restrict__ nbr, int64_t n_flat, int K, int64_t n_in,
                            const int32_t* __restrict__ rank, int32_t* __restrict__ tmap) {
  const int64_t block_first = (int64_t)blockIdx.x * kFlatPerBlock;
  int32_t v[kFlatQuads][4];
  load_quads(nbr, n_flat, block_first, v);
  int32_t pos[kFlatQuads][4];
#pragma unroll
  for (int q = 0; q < kFlatQuads; ++q)
#pragma unroll
    for (int j = 0; j < 4; ++j) pos[q][j] = (v[q][j] >= 0 && v[q][j] < n_in) ? __ldg(rank + v[q][j]) : -1;
#pragma unroll
  for (int q = 0; q < kFlatQuads; ++q) {
    const int64_t t0 = block_first + ((int64_t)q * 256 + threadIdx.x) * 4;
    int64_t o = (int64_t)((IndexT)t0 / (IndexT)K);
    int k = (int)(t0 - o * K);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (pos[q][j] >= 0) tmap[((int64_t)(pos[q][j] >> 7) * K + k) * 128 + (pos[q][j] & 127)] = (int32_t)o;
      if (++k == K) {
        k = 0;
        ++o;
      }
    }
  }
}

// ---- balanced plans (K <= 32): the tiles in descending order of their number of offsets ----
// The products hand tiles out in order to SMs that are free, so the big ones come first and the small ones fill up: with
// the tiles in the order of their masks, the SM that got the last big one ended 1.1 to 1.6 times later than the mean.

// A warp per tile: tmask[tile] = OR of its 128 sorted keys.  The block that finishes last ranks the tiles by a stable
// counting sort, most offsets first (31 and 32 count alike); a tile that is not full keeps the last place.
__global__ void __launch_bounds__(1024) tile_slots_kernel(const uint32_t* __restrict__ sorted_keys, int64_t n, int64_t n_tiles,
                                                         uint32_t* tmask, int32_t* __restrict__ slot, uint32_t* ticket) {
  __shared__ uint32_t next[32][33];                       // [warp][bin]
  __shared__ uint32_t part[32];
  __shared__ bool last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t tile = (int64_t)blockIdx.x * 32 + warp;
  if (tile < n_tiles) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t at = tile * 128 + i * 32 + lane;
      m |= at < n ? __ldg(sorted_keys + at) : 0u;
    }
    m = __reduce_or_sync(0xFFFFFFFFu, m);
    if (lane == 0) tmask[tile] = m;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  next[warp][lane] = 0;
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int64_t n_full = n / 128, per = ((n_full + 31) / 32 + 31) / 32 * 32;          // tiles of a warp
  const int64_t begin = warp * per, end = min(n_full, begin + per);
  const uint32_t lower = (1u << lane) - 1u;
  constexpr int kBatch = 8;
  auto each = [&](auto&& f) {                              // f(tile or -1, lanes of the same bin, bin)
    for (int64_t t0 = begin; t0 < end; t0 += 32 * kBatch) {
      uint32_t m[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) m[i] = t0 + i * 32 + lane < end ? __ldcg(tmask + t0 + i * 32 + lane) : 0u;
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const int64_t t = t0 + i * 32 + lane;
        const int bin = t < end ? 31 - min(__popc(m[i]), 31) : 32;
        f(t < end ? t : -1, __match_any_sync(0xFFFFFFFFu, bin), bin);
      }
    }
  };
  each([&](int64_t t, uint32_t peers, int bin) {
    if (t >= 0 && (peers & lower) == 0) next[warp][bin] += __popc(peers);
    __syncwarp();
  });
  __syncthreads();
  // first place of (bin, warp): thread = bin * 32 + warp of the count
  const uint32_t count = next[lane][warp];
  uint32_t upto = count;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, upto, o);
    if (lane >= o) upto += u;
  }
  if (lane == 31) part[warp] = upto;
  __syncthreads();
  const uint32_t before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? part[lane] : 0u);
  next[lane][warp] = before + upto - count;
  __syncthreads();
  each([&](int64_t t, uint32_t peers, int bin) {
    if (t >= 0) slot[t] = (int32_t)(next[warp][bin] + __popc(peers & lower));
    __syncwarp();
    if (t >= 0 && (peers & lower) == 0) next[warp][bin] += __popc(peers);
    __syncwarp();
  });
  if (threadIdx.x == 0 && n_full < n_tiles) slot[n_full] = (int32_t)n_full;
}

// plan_tiles_kernel for K <= 32 with the masks and places of the tiles known: tile t of the sorted rows goes to place slot[t],
// and only lines with a neighbour are written (nothing reads the others: a tenth of them is left at 3 offsets of 27).
// Eight warps of 16 rows, all their loads in flight together; a row's K entries take 8, 16 or 32 lanes.
__global__ void __launch_bounds__(256) plan_slots_kernel(const int32_t* __restrict__ nbr, const int32_t* __restrict__ sorted, int64_t n,
                                                        int K, const uint32_t* __restrict__ sorted_mask,
                                                        const int32_t* __restrict__ slots, int32_t* __restrict__ order,
                                                        int32_t* __restrict__ tmap, uint32_t* __restrict__ tmask) {
  __shared__ int32_t stage[128 * 33];
  const int64_t tile = blockIdx.x, slot = __ldg(slots + tile);
  const uint32_t mask = __ldg(sorted_mask + tile);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int shift = K <= 8 ? 3 : K <= 16 ? 4 : 5, per_load = 32 >> shift;
  const int k = lane & ((1 << shift) - 1), pitch = K | 1;
  const int64_t pos = tile * 128 + warp * 16 + (lane & 15);
  const int src = pos < n ? __ldg(sorted + pos) : -1;
  if (lane < 16 && src >= 0) order[slot * 128 + warp * 16 + lane] = src;
  if (threadIdx.x == 0) tmask[slot] = mask;
  int32_t v[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int row = i * per_load + (lane >> shift);
    const int from = __shfl_sync(0xFFFFFFFFu, src, row & 15);
    v[i] = i * per_load < 16 && from >= 0 && k < K ? __ldg(nbr + (int64_t)from * K + k) : -1;
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int row = i * per_load + (lane >> shift);
    if (i * per_load < 16 && k < K) stage[(warp * 16 + row) * pitch + k] = v[i];
  }
  __syncthreads();
  int turn = 0;
  for (uint32_t m = mask; m; m &= m - 1, ++turn) {
    if ((turn & 7) != warp) continue;
    const int j = __ffs(m) - 1;
    int32_t* line = tmap + (slot * K + j) * 128 + lane;
#pragma unroll
    for (int i = 0; i < 4; ++i) line[i * 32] = stage[(i * 32 + lane) * pitch + j];
  }
}

// The same for the inverse map, whose entries inverse_plan_scatter_kernel then fills in: the places of its rows, the row order,
// the masks, and -1 in the lines that have a neighbour.
__global__ void __launch_bounds__(128) inverse_slots_kernel(const int32_t* __restrict__ sorted, int64_t n, int K,
                                                           const uint32_t* __restrict__ sorted_mask,
                                                           const int32_t* __restrict__ slots, int32_t* __restrict__ rank,
                                                           int32_t* __restrict__ order, int32_t* __restrict__ tmap,
                                                           uint32_t* __restrict__ tmask) {
  const int64_t tile = blockIdx.x, slot = __ldg(slots + tile), pos = tile * 128 + threadIdx.x;
  const uint32_t mask = __ldg(sorted_mask + tile);
  if (pos < n) {
    const int row = __ldg(sorted + pos);
    rank[row] = (int32_t)(slot * 128 + threadIdx.x);
    order[slot * 128 + threadIdx.x] = row;
  }
  if (threadIdx.x == 0) tmask[slot] = mask;
  for (uint32_t m = mask; m; m &= m - 1) tmap[(slot * K + __ffs(m) - 1) * 128 + threadIdx.x] = -1;
}

struct SlotScratch {
  OrderScratch sort;
  int32_t *rank, *slot;
  uint32_t *mask, *ticket;
};
int64_t carve_slots(SlotScratch* s, void* ws, int64_t n, int K) {
  int64_t off = carve(&s->sort, ws, n, K);
  auto take = [&](int64_t count) {
    char* p = ws ? static_cast<char*>(ws) + off : nullptr;
    off += align_up((count > 0 ? count : 1) * 4, 256);
    return p;
  };
  s->rank = reinterpret_cast<int32_t*>(take(n));
  s->slot = reinterpret_cast<int32_t*>(take((n + 127) / 128));
  s->mask = reinterpret_cast<uint32_t*>(take((n + 127) / 128));
  s->ticket = reinterpret_cast<uint32_t*>(take(1));
  return off;
}
// The sort of sort_passes, but with its result left in s.vals_b: `order` is the other buffer and is written afterwards.
int32_t* first_vals_aside(const OrderScratch& s, int K, int32_t* order) { return passes_for(K) % 2 == 0 ? s.vals_b : order; }
void sort_aside(const SlotScratch& s, int64_t n, int K, int32_t* order, cudaStream_t st) {
  int32_t* vals_in = first_vals_aside(s.sort, K, order);
  uint32_t* sorted_keys = nullptr;
  radix_sort_pairs<uint32_t>(s.sort.keys_a, vals_in, s.sort.keys_b, vals_in == order ? s.sort.vals_b : order, n, K, s.sort.hist,
                             s.sort.totals, &sorted_keys, nullptr, st);
  const int64_t n_tiles = (n + 127) / 128;
  tile_slots_kernel<<<(unsigned)((n_tiles + 31) / 32), 1024, 0, st>>>(sorted_keys, n, n_tiles, s.mask, s.slot, s.ticket);
  note_launches(1);
}

}  // namespace

}  // namespace st

using namespace st;

extern "C" {

int64_t st_map_row_order_workspace_bytes(int64_t n_rows, int K) {
  OrderScratch s;
  return carve(&s, nullptr, n_rows, K);
}

int st_map_row_order(const int32_t* nbr, int64_t n_rows, int K, int32_t* order, void* workspace,
                     int64_t workspace_bytes, void* stream) {
  if (n_rows < 0 || K < 1 || n_rows > 0x7FFFFFFFll || (n_rows > 0 && (!nbr || !order || !workspace))) {
    set_error("st_map_row_order: bad arguments");
    return ST_ERR_ARG;
  }
  if (n_rows == 0) return ST_OK;
  OrderScratch s;
  if (workspace_bytes < carve(&s, workspace, n_rows, K)) {
    set_error("st_map_row_order: workspace of %lld bytes is too small", (long long)workspace_bytes);
    return ST_ERR_WORKSPACE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const size_t stage_bytes = K <= 64 ? (size_t)128 * K * 4 : 0;
  {
    row_keys_kernel<<<(unsigned)((n_rows + 127) / 128), 128, stage_bytes, st>>>(nbr, n_rows, K, s.keys_a,
                                                                                first_vals(s, K, order), nullptr);
    note_launches(1);
  }
  sort_passes(s, n_rows, K, order, nullptr, st);
  return check_launch("st_map_row_order");
}

int64_t st_map_plan_workspace_bytes(int64_t n_rows, int K) { return st_map_row_order_workspace_bytes(n_rows, K); }

int64_t st_map_plan_inverse_workspace_bytes(int64_t n_in, int K) {
  return st_map_row_order_workspace_bytes(n_in, K) + align_up((n_in > 0 ? n_in : 1) * 4, 256);
}

int st_map_plan_inverse(const int32_t* nbr, int64_t n_out, int K, int64_t n_in, int32_t* order, int32_t* tmap,
                        uint32_t* tmask, void* workspace, int64_t workspace_bytes, void* stream) {
  if (n_out < 0 || n_in < 0 || K < 1 || K > 32 || n_in > 0x7FFFFFFFll || (n_out > 0 && !nbr) ||
      (n_in > 0 && (!order || !tmap || !tmask || !workspace))) {
    set_error("st_map_plan_inverse: bad arguments (K must be <= 32)");
    return ST_ERR_ARG;
  }
  if (n_in == 0) return ST_OK;
  OrderScratch s;
  const int64_t sort_bytes = carve(&s, workspace, n_in, K);
  if (workspace_bytes < st_map_plan_inverse_workspace_bytes(n_in, K)) {
    set_error("st_map_plan_inverse: workspace of %lld bytes is too small", (long long)workspace_bytes);
    return ST_ERR_WORKSPACE;
  }
  int32_t* rank = reinterpret_cast<int32_t*>(static_cast<char*>(workspace) + sort_bytes);
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t n_flat = n_out * K, n_tiles = (n_in + 127) / 128, n_tmap = n_tiles * K * 128;
  const unsigned rows_grid = (unsigned)((n_in + 255) / 256);
  iota_clear_kernel<<<rows_grid, 256, 0, st>>>(s.keys_a, first_vals(s, K, order), n_in, nullptr);
  const unsigned flat_grid = (unsigned)((n_flat + kFlatPerBlock - 1) / kFlatPerBlock);
  const bool narrow = n_flat + kFlatPerBlock < 0x7FFFFFFFll;           // every flat index a thread forms fits 32 bits
  if (n_flat > 0) {
    if (narrow) inverse_keys_kernel<uint32_t><<<flat_grid, 256, 0, st>>>(nbr, n_flat, K, n_in, s.keys_a);
    else inverse_keys_kernel<int64_t><<<flat_grid, 256, 0, st>>>(nbr, n_flat, K, n_in, s.keys_a);
  }
  note_launches(2);
  uint32_t* sorted_keys = nullptr;
  sort_passes(s, n_in, K, order, &sorted_keys, st);
  rank_kernel<<<rows_grid, 256, 0, st>>>(order, n_in, rank);
  tile_mask_kernel<<<(unsigned)n_tiles, 128, 0, st>>>(sorted_keys, n_in, tmask);
  cudaMemsetAsync(tmap, 0xFF, (size_t)n_tmap * sizeof(int32_t), st);                  // every entry -1
  if (n_flat > 0) {
    if (narrow) inverse_plan_scatter_kernel<uint32_t><<<flat_grid, 256, 0, st>>>(nbr, n_flat, K, n_in, rank, tmap);
    else inverse_plan_scatter_kernel<int64_t><<<flat_grid, 256, 0, st>>>(nbr, n_flat, K, n_in, rank, tmap);
  }
  note_launches(3);
  return check_launch("st_map_plan_inverse");
}

int st_map_plan(const int32_t* nbr, int64_t n_rows, int K, int sort_rows, int32_t* order, int32_t* tmap,
                uint32_t* tmask, void* workspace, int64_t workspace_bytes, void* stream) {
  if (n_rows < 0 || K < 1 || n_rows > 0x7FFFFFFFll ||
      (n_rows > 0 && (!nbr || !tmap || !tmask || (sort_rows && (!order || !workspace))))) {
    set_error("st_map_plan: bad arguments");
    return ST_ERR_ARG;
  }
  if (n_rows == 0) return ST_OK;
  if (sort_rows) {
    int rc = st_map_row_order(nbr, n_rows, K, order, workspace, workspace_bytes, stream);
    if (rc != ST_OK) return rc;
  }
  const int64_t n_tiles = (n_rows + 127) / 128;
  {
    const size_t stage_bytes = (size_t)128 * ((K < kPlanChunk ? K : kPlanChunk) | 1) * 4;
    plan_tiles_kernel<<<(unsigned)n_tiles, 128, stage_bytes, (cudaStream_t)stream>>>(
        nbr, sort_rows ? order : nullptr, n_rows, K, (K + 31) / 32, tmap, tmask);
    note_launches(1);
  }
  return check_launch("st_map_plan");
}

int64_t st_map_plan_balanced_workspace_bytes(int64_t n_rows, int K) {
  SlotScratch s;
  return carve_slots(&s, nullptr, n_rows, K);
}

int st_map_plan_balanced(const int32_t* nbr, int64_t n_rows, int K, int32_t* order, int32_t* tmap, uint32_t* tmask,
                         void* workspace, int64_t workspace_bytes, void* stream) {
  if (n_rows < 0 || K < 1 || K > 32 || n_rows > 0x7FFFFFFFll || (n_rows > 0 && (!nbr || !order || !tmap || !tmask || !workspace))) {
    set_error("st_map_plan_balanced: bad arguments (K must be <= 32)");
    return ST_ERR_ARG;
  }
  if (n_rows == 0) return ST_OK;
  SlotScratch s;
  if (workspace_bytes < carve_slots(&s, workspace, n_rows, K)) {
    set_error("st_map_plan_balanced: workspace of %lld bytes is too small", (long long)workspace_bytes);
    return ST_ERR_WORKSPACE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const unsigned n_tiles = (unsigned)((n_rows + 127) / 128);
  row_keys_kernel<<<n_tiles, 128, (size_t)128 * K * 4, st>>>(nbr, n_rows, K, s.sort.keys_a, first_vals_aside(s.sort, K, order), s.ticket);
  sort_aside(s, n_rows, K, order, st);
  plan_slots_kernel<<<n_tiles, 256, 0, st>>>(nbr, s.sort.vals_b, n_rows, K, s.mask, s.slot, order, tmap, tmask);
  note_launches(2);
  return check_launch("st_map_plan_balanced");
}

int st_map_plan_inverse_balanced(const int32_t* nbr, int64_t n_out, int K, int64_t n_in, int32_t* order, int32_t* tmap,
                                 uint32_t* tmask, void* workspace, int64_t workspace_bytes, void* stream) {
  if (n_out < 0 || n_in < 0 || K < 1 || K > 32 || n_in > 0x7FFFFFFFll || (n_out > 0 && !nbr) ||
      (n_in > 0 && (!order || !tmap || !tmask || !workspace))) {
    set_error("st_map_plan_inverse_balanced: bad arguments (K must be <= 32)");
    return ST_ERR_ARG;
  }
  if (n_in == 0) return ST_OK;
  SlotScratch s;
  if (workspace_bytes < carve_slots(&s, workspace, n_in, K)) {
    set_error("st_map_plan_inverse_balanced: workspace of %lld bytes is too small", (long long)workspace_bytes);
    return ST_ERR_WORKSPACE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t n_flat = n_out * K;
  const bool narrow = n_flat + kFlatPerBlock < 0x7FFFFFFFll;
  const unsigned flat_grid = (unsigned)((n_flat + kFlatPerBlock - 1) / kFlatPerBlock);
  iota_clear_kernel<<<(unsigned)((n_in + 255) / 256), 256, 0, st>>>(s.sort.keys_a, first_vals_aside(s.sort, K, order), n_in, s.ticket);
  if (n_flat > 0) {
    if (narrow) inverse_keys_kernel<uint32_t><<<flat_grid, 256, 0, st>>>(nbr, n_flat, K, n_in, s.sort.keys_a);
    else inverse_keys_kernel<int64_t><<<flat_grid, 256, 0, st>>>(nbr, n_flat, K, n_in, s.sort.keys_a);
  }
  sort_aside(s, n_in, K, order, st);
  inverse_slots_kernel<<<(unsigned)((n_in + 127) / 128), 128, 0, st>>>(s.sort.vals_b, n_in, K, s.mask, s.slot, s.rank, order, tmap, tmask);
  if (n_flat > 0) {
    if (narrow) inverse_plan_scatter_kernel<uint32_t><<<flat_grid, 256, 0, st>>>(nbr, n_flat, K, n_in, s.rank, tmap);
    else inverse_plan_scatter_kernel<int64_t><<<flat_grid, 256, 0, st>>>(nbr, n_flat, K, n_in, s.rank, tmap);
  }
  note_launches(4);
  return check_launch("st_map_plan_inverse_balanced");
}

}  // extern "C"
