// Gather kernel for a stored map in tile-plan form.  Included by conv_tc.cu (one translation unit: the
// device status word and the PTX wrappers are file-local there).
//
//   OUT[order[r], :] = sum_k  IN[tmap(r, k), :] . B_k
//
// Super tiles of S row tiles, whose accumulators sit side by side in TMEM, share the copies of W: for every offset k
// (and 128-byte block kb of the reduction) that occurs in the super tile, W[k] travels once through a ring of W slots, and
// each sub tile that has the offset sends one stage of 128 gathered rows through the ring of row stages.
//
// Warps 0-3 drain accumulators, warp 4 issues the MMAs, warp 5 fetches W slices by TMA, warps 6-21 fetch rows with
// 16-byte cp.async: four groups of four warps take the stages in turn, a warp has 32 rows of a stage.  Warp 22 hands out
// super tiles with their tile masks, which the MMA and W warps walk themselves, and lists their stages for the row warps:
// with the walk in all sixteen of them, it was two thirds of their instructions, and without any copy, store or W slice the
// kernel still took 135 of 170 us (815249 rows, 64 -> 128).
//
// Who does which super tile: super tiles cost 1 to K offsets, and dealt out in a fixed pattern the busiest SM had 1.3 to 2
// times the mean.  The grid is one CTA per super tile, and a CTA that runs takes over others before they start
// (clusterlaunchcontrol); plans of sorted rows put their tiles in descending order of work, so the last ones are small.
//
// What bounds it: bringing rows into shared memory.  A loop that does nothing else (148 CTAs, random rows) takes, per
// stage of 128 rows, with tile::gather4 612-743 cycles when every row exists and 1180 (128-byte rows) to 1880
// (64-byte rows) when half of them are absent -- out-of-range rows are what the copy engine is slowest at -- and with
// cp.async from 16 warps 265-344 (128-byte rows) and 160-207 (64-byte rows), absent or not, from tables of 8 to 160 MB.
// Eight warps reach half of that: it is latency times warps, hence 16, and hence stages of one sub tile: slots of a whole
// super tile's rows (two or three in the ring, mostly half used) left too little in flight.
//
// Hand-over of a stage: every thread leaves an asynchronous arrival behind its copies (128 a stage) and goes on; a warp that
// waited for its share to land and arrived for it, when its group's next stage was on its way, made the stage late (95541 rows,
// 256 -> 256: 166 -> 155 us; 117471 rows: 161 -> 153).  The warp that issues the MMAs fences the proxies.
#pragma once

namespace st {
namespace tc {

constexpr int kRowGroups = 4, kRowGroupWarps = 4;             // warps that fetch rows
constexpr int kWarpW = kMmaWarp + 1;                          // the warp that fetches W slices
constexpr int kFirstRowWarp = kWarpW + 1;
constexpr int kWarpJobs = kFirstRowWarp + kRowGroups * kRowGroupWarps;
constexpr int kGather3Threads = (kWarpJobs + 1) * 32;
constexpr int kJobReaders = kFirstRowWarp;
// Super tiles on offer at a time.  Every one taken early is one that cannot go to an SM that turns out to be free.
constexpr int kJobs = 2;

struct Job {
  int super;                                                   // -1: no more
  uint32_t touched;                                            // its sub tiles that have any offset
  uint32_t mask[kMaxSub];                                      // offsets 0 .. 31
};

// Up to 32 stages of one super tile: the index line of each and its column block of the reduction.
struct Batch {
  uint2 entry[32];
  int n;                                                       // -1: no more
};
constexpr int kBatches = 4;

struct __align__(8) Control3 {
  unsigned long long a_full[kMaxAStages], a_empty[kMaxAStages];
  unsigned long long w_full[kMaxWSlots], w_empty[kMaxWSlots];
  unsigned long long acc_full[2], acc_empty[2];
  unsigned long long job_full[kJobs], job_empty[kJobs], taken;
  unsigned long long batch_full[kBatches], batch_empty[kBatches];
  __align__(16) uint4 taken_cta;
  Batch batch[kBatches];
  Job job[kJobs];
  uint32_t tmem_base;
  int abort_flag;
};

static_assert(sizeof(Control3) <= 2048, "see the shared memory budget in fill_params2");
struct BatchWriter {
  Control3* ctl;
  volatile int* abort_flag;
  int lane;
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ bool put(uint2 entry, int n) {
    if (!mbar_wait_all(smem_u32(&ctl->batch_empty[slot]), phase ^ 1u, abort_flag, 45)) return false;
    ctl->batch[slot].entry[lane] = entry;
    if (lane == 0) ctl->batch[slot].n = n;
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->batch_full[slot]));
    if (++slot == kBatches) {
      slot = 0;
      phase ^= 1u;
    }
    return true;
  }
};
// Every lane has a count; the inclusive sums of the counts, and the lane that output `o` belongs to.
__device__ __forceinline__ uint32_t lane_sums(uint32_t count, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t before = __shfl_up_sync(0xFFFFFFFFu, count, d);
    if (lane >= d) count += before;
  }
  return count;
}
__device__ __forceinline__ int owner_of(uint32_t upto, uint32_t o) {
  int l = 0;
#pragma unroll
  for (int step = 16; step; step >>= 1) {
    if (__shfl_sync(0xFFFFFFFFu, upto, l + step - 1) <= o) l += step;
  }
  return l;
}

// A warp's view of the super tiles this CTA has, in order.
struct JobReader {
  Control3* ctl;
  volatile int* abort_flag;
  int lane;
  int slot = 0;
  uint32_t phase = 0;
  Job job;
  __device__ __forceinline__ bool next() {
    if (!mbar_wait_all(smem_u32(&ctl->job_full[slot]), phase, abort_flag, 43)) return false;
    job = ctl->job[slot];
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->job_empty[slot]));
    if (++slot == kJobs) {
      slot = 0;
      phase ^= 1u;
    }
    return __all_sync(0xFFFFFFFFu, job.super >= 0);
  }
};

// The work of this CTA in order: item(tile0, k, kb, users, fresh) for every occupied (offset, 128-byte block) of a
// super tile (users: the sub tiles that have the offset; fresh: those whose accumulator starts here), between
// begin(tile0) and end(tile0).  Stops when one of them returns false.
template <typename Begin, typename Item, typename End>
__device__ __forceinline__ void walk_super_tiles(const Params2& p, const PlannedRows& map, int64_t n_tiles, JobReader jobs,
                                                 Begin&& begin, Item&& item, End&& end) {
  while (jobs.next()) {
    const int64_t tile0 = (int64_t)jobs.job.super * p.sub;
    // every lane has the same words; the reduction tells the compiler so (uniform registers and branches)
    uint32_t m[kMaxSub];
#pragma unroll
    for (int s = 0; s < kMaxSub; ++s) m[s] = __reduce_or_sync(0xFFFFFFFFu, jobs.job.mask[s]);
    if (!begin(tile0)) return;
    uint32_t touched = 0;
    for (int word = 0; word < map.MW; ++word) {
      if (word) {
#pragma unroll
        for (int s = 0; s < kMaxSub; ++s)
          m[s] = __reduce_or_sync(0xFFFFFFFFu, s < p.sub && tile0 + s < n_tiles ? __ldg(map.tmask + (tile0 + s) * map.MW + word) : 0u);
      }
      static_assert(kMaxSub == 4, "the masks of a super tile are combined by hand");
      uint32_t m_any = m[0] | m[1] | m[2] | m[3];
      while (m_any) {
        const int j = __ffs(m_any) - 1;
        m_any &= m_any - 1;
        uint32_t users = 0;
#pragma unroll
        for (int s = 0; s < kMaxSub; ++s) users |= ((m[s] >> j) & 1u) << s;
        for (int kb = 0; kb < p.k_blocks; ++kb)
          if (!item(tile0, word * 32 + j, kb, users, kb == 0 ? (users & ~touched) : 0u)) return;
        touched |= users;
      }
    }
    if (!end(tile0)) return;
  }
}

// A warp's kRows (32 or 8) rows of one 128-byte column block: 2^kLpr lanes share a row (16 bytes each).  All row numbers are
// exchanged before the first copy.  kAtom32: the 128-byte swizzle with 32-byte atoms, else the plain one.
template <int kLpr, int kRows, bool kAtom32>
__device__ __forceinline__ void fetch_rows(uint32_t dst, int row0, int idx, const char* col, int pitch, int64_t n_src, int chunks,
                                           int lane) {
  constexpr int kRowsPer = 32 >> kLpr, kN = kRows > kRowsPer ? kRows / kRowsPer : 1;
  const int c = lane & ((1 << kLpr) - 1), r_lane = lane >> kLpr;
  int src[kN];
#pragma unroll
  for (int i = 0; i < kN; ++i) src[i] = __shfl_sync(0xFFFFFFFFu, idx, i * kRowsPer + r_lane);
  col += c * 16;
#pragma unroll
  for (int i = 0; i < kN; ++i) {
    const bool have = (uint32_t)src[i] < (uint32_t)n_src;                      // "-1" and rows past the source: zeros
    const int row = row0 + i * kRowsPer + r_lane;
    if (c < chunks && (kRows >= kRowsPer || r_lane < kRows))
      cp_async16(dst + (uint32_t)row * 128u + ((uint32_t)(kAtom32 ? swz32(c, row) : swz16(c, row)) << 4),
                 col + (have ? (size_t)(uint32_t)src[i] * (uint32_t)pitch : 0), have ? 16u : 0u);
  }
}
// ... of a row block of `bytes` (a multiple of 16, at most 128) bytes.
template <int kRows, bool kAtom32>
__device__ __forceinline__ void fetch_block(uint32_t dst, int row0, int idx, const char* col, int pitch, int64_t n_src, int bytes,
                                            int lane) {
  const int chunks = bytes >> 4;
  if (chunks > 4) fetch_rows<3, kRows, kAtom32>(dst, row0, idx, col, pitch, n_src, chunks, lane);
  else if (chunks > 2) fetch_rows<2, kRows, kAtom32>(dst, row0, idx, col, pitch, n_src, chunks, lane);
  else fetch_rows<1, kRows, kAtom32>(dst, row0, idx, col, pitch, n_src, chunks, lane);
}

// Accumulator columns c0 .. of a warp's 32 rows (lane = row) to the output rows `dst` (-1: none), P 16-byte pieces of each,
// by way of shared memory: there a lane has a row, in the stores P lanes share one.  With lane = row in the stores as well
// (16 bytes of 32 rows per instruction) the accumulators took as long to drain as to fill: 60 of 227 us at 815249 rows of 64 -> 128.
constexpr uint32_t kOutWarpBytes = 32 * 128;
template <int P>
__device__ __forceinline__ void store_block(const Params2& p, uint32_t stage, uint32_t t_row, int c0, int dst, bool zeros, int lane) {
  constexpr int kRowsPerLine = 8 / P;                         // rows of 128 bytes, pieces swizzled within
  auto at = [&](int row, int piece) {
    return stage + (uint32_t)(row / kRowsPerLine) * 128u +
           (uint32_t)((row & (kRowsPerLine - 1)) * P + (piece ^ ((row / kRowsPerLine) & (P - 1)))) * 16u;
  };
  auto put = [&](int piece, const uint32_t* w) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at(lane, piece)), "r"(zeros ? 0u : w[0]), "r"(zeros ? 0u : w[1]),
                 "r"(zeros ? 0u : w[2]), "r"(zeros ? 0u : w[3]) : "memory");
  };
  const bool f32 = p.out_kind == ST_F32;
  const int es = f32 ? 4 : 2, cols = P * 16 / es;
  for (int c = 0; c < cols; c += 16) {
    uint32_t v[32];                                            // 16 are used
    tmem_ld16(t_row + (uint32_t)(c0 + c), v);
    tmem_ld_wait();
    if (f32) {
#pragma unroll
      for (int i = 0; i < 4; ++i) put(c / 4 + i, v + 4 * i);
    } else {
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = pack_pair(p.out_kind, v[2 * i], v[2 * i + 1]);
      put(c / 8, w);
      put(c / 8 + 1, w + 4);
    }
  }
  __syncwarp();
  char* out = static_cast<char*>(p.out) + (size_t)c0 * es + (lane % P) * 16;
  const size_t pitch = (size_t)p.c_acc * es;
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const int row = i * (32 / P) + lane / P;
    const int to = __shfl_sync(0xFFFFFFFFu, dst, row);
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at(row, lane % P)) : "memory");
    if (to >= 0) *reinterpret_cast<uint4*>(out + (size_t)to * pitch) = v;
  }
  __syncwarp();
}

template <int ESIZE>
__global__ void __launch_bounds__(kGather3Threads, 1) planned_gather_kernel(const Params2 p, const PlannedRows map,
                                                                            const __grid_constant__ CUtensorMap w_desc) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_raw + (base - raw);
  const uint32_t a_ring = base + (uint32_t)p.w_slots * (uint32_t)p.w_slot_bytes;
  const uint32_t out_ring = a_ring + (uint32_t)p.a_stages * kABlockBytes;
  Control3* ctl = reinterpret_cast<Control3*>(base_ptr + (out_ring - base) + 4 * kOutWarpBytes);
  volatile int* abort_flag = &ctl->abort_flag;
  const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.a_stages; ++s) {
      mbar_init(smem_u32(&ctl->a_full[s]), kRowGroupWarps * 32);
      mbar_init(smem_u32(&ctl->a_empty[s]), 1);
    }
    for (int s = 0; s < p.w_slots; ++s) {
      mbar_init(smem_u32(&ctl->w_full[s]), 1);
      mbar_init(smem_u32(&ctl->w_empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&ctl->acc_full[b]), 1);
      mbar_init(smem_u32(&ctl->acc_empty[b]), kEpilogueWarps * 32);
    }
    for (int s = 0; s < kBatches; ++s) {
      mbar_init(smem_u32(&ctl->batch_full[s]), 1);
      mbar_init(smem_u32(&ctl->batch_empty[s]), kRowGroups * kRowGroupWarps);
    }
    for (int s = 0; s < kJobs; ++s) {
      mbar_init(smem_u32(&ctl->job_full[s]), 1);
      mbar_init(smem_u32(&ctl->job_empty[s]), kJobReaders);
    }
    mbar_init(smem_u32(&ctl->taken), 1);
    ctl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(&ctl->tmem_base), (uint32_t)p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  const int red_bytes = p.c_red * ESIZE;
  const int set_cols = p.sub * p.c_acc;                      // TMEM columns of one accumulator set
  const int64_t n_tiles = (p.n_rows + kTileM - 1) / kTileM;
  auto nothing = [](int64_t) { return true; };
  const JobReader jobs{ctl, abort_flag, lane};

  if (warp == kWarpJobs) {
    // =============================================================== super tiles
    int super = blockIdx.x, slot = 0;
    uint32_t phase = 0, taken_phase = 0;
    BatchWriter batches{ctl, abort_flag, lane};
    while (true) {
      if (!mbar_wait_all(smem_u32(&ctl->job_empty[slot]), phase ^ 1u, abort_flag, 41)) break;
      if (super < 0) {                                         // not the first: take over a CTA that has not started
        if (lane == 0) {
          mbar_arrive_expect_tx(smem_u32(&ctl->taken), 16);
          take_cta(smem_u32(&ctl->taken_cta), smem_u32(&ctl->taken));
        }
        __syncwarp();
        if (!mbar_wait_all(smem_u32(&ctl->taken), taken_phase, abort_flag, 42)) break;
        taken_phase ^= 1u;
        super = taken_cta(smem_u32(&ctl->taken_cta));
        fence_proxy_async();                                   // read before the next answer is written
      }
      // masks of the first 32 offsets by lane = sub tile; all words for "has any"
      uint32_t mask = 0, any = 0;
      const int64_t tile = (int64_t)super * p.sub + lane;
      if (super >= 0 && lane < p.sub && tile < n_tiles) {
        mask = any = __ldg(map.tmask + tile * map.MW);
        for (int word = 1; word < map.MW; ++word) any |= __ldg(map.tmask + tile * map.MW + word);
      }
      const uint32_t touched = __ballot_sync(0xFFFFFFFFu, any != 0u);
      if (lane < kMaxSub) ctl->job[slot].mask[lane] = mask;
      if (lane == 0) {
        ctl->job[slot].super = super;
        ctl->job[slot].touched = touched;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->job_full[slot]));
      // its stages: offset by offset, column block by column block, the sub tiles that have the offset in turn
      bool ok = true;
      for (int word = 0; word < map.MW && super >= 0 && ok; ++word) {
        if (word) mask = lane < p.sub && tile < n_tiles ? __ldg(map.tmask + tile * map.MW + word) : 0u;
        uint32_t users = 0;                                    // lane = offset
#pragma unroll
        for (int s = 0; s < kMaxSub; ++s) users |= ((__shfl_sync(0xFFFFFFFFu, mask, s) >> lane) & 1u) << s;
        const uint32_t upto = lane_sums((uint32_t)(__popc(users) * p.k_blocks), lane);
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, upto, 31);
        for (uint32_t o0 = 0; o0 < total && ok; o0 += 32) {
          const uint32_t o = min(o0 + lane, total - 1);        // lane = stage
          const int j = owner_of(upto, o);
          uint32_t u = __shfl_sync(0xFFFFFFFFu, users, j);
          const uint32_t n_users = (uint32_t)__popc(u);
          const uint32_t at = o - (__shfl_sync(0xFFFFFFFFu, upto, j) - n_users * (uint32_t)p.k_blocks);
          const uint32_t kb = at / n_users, which = at - kb * n_users;
#pragma unroll
          for (uint32_t q = 0; q + 1 < kMaxSub; ++q)
            if (q < which) u &= u - 1;
          const uint32_t line = (uint32_t)(((int64_t)super * p.sub + __ffs(u) - 1) * map.K + word * 32 + j);
          const int n = (int)min(32u, total - o0);
          if (kb == 0 && lane < n) {                           // have it in L2 by the time the row warps ask
            const char* at_line = reinterpret_cast<const char*>(map.tmap) + (size_t)line * (kTileM * 4);
#pragma unroll
            for (int i = 0; i < 4; ++i) prefetch_l2(at_line + i * 128);
          }
          ok = batches.put(make_uint2(line, kb), n);
        }
      }
      if (super < 0) {
        if (ok) batches.put(make_uint2(0u, 0u), -1);
        break;
      }
      if (!ok) break;
      super = -1;
      if (++slot == kJobs) {
        slot = 0;
        phase ^= 1u;
      }
    }
  } else if (warp >= kFirstRowWarp) {
    // =============================================================== rows
    const int group = (warp - kFirstRowWarp) / kRowGroupWarps;
    const int row0 = (warp - kFirstRowWarp) % kRowGroupWarps * 32;
    const char* in = static_cast<const char*>(p.in);
    int first = group, next = group;                          // a_stages > kRowGroups: every group starts in the first lap
    uint32_t phase = 0;
    const int32_t* lines = map.tmap + row0 + lane;
    bool ok = true;
    int pend_stage = -1, pend_kb = 0, pend_idx = -1;
    uint32_t pend_parity = 0;
    auto run = [&]() {
      ok = mbar_wait_all(smem_u32(&ctl->a_empty[pend_stage]), pend_parity ^ 1u, abort_flag, 31);
      if (!ok) return;
      fetch_block<32, false>(a_ring + (uint32_t)pend_stage * kABlockBytes, row0, pend_idx, in + pend_kb * 128, red_bytes, p.n_src,
                         min(128, red_bytes - pend_kb * 128), lane);
      cp_async_arrive_noinc(smem_u32(&ctl->a_full[pend_stage]));                 // when they have landed
    };
    auto flush = [&]() {
      // the batch that this warp is about to wait for may wait for the stage that it has put off
      if (pend_stage >= 0 && ok) run();
      pend_stage = -1;
    };
    int slot = 0;
    uint32_t slot_phase = 0;
    while (ok) {
      const uint32_t full = smem_u32(&ctl->batch_full[slot]);
      if (!__all_sync(0xFFFFFFFFu, mbar_try_now(full, slot_phase))) flush();
      if (!ok || !mbar_wait_all(full, slot_phase, abort_flag, 44)) break;
      const int n = ctl->batch[slot].n;
      const uint2 entry = ctl->batch[slot].entry[lane];        // lane = stage
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->batch_empty[slot]));
      if (++slot == kBatches) {
        slot = 0;
        slot_phase ^= 1u;
      }
      if (n < 0) break;
      // this group's are the stages first, first + 4, ...; `next` and `phase`: ring position of the group's next one
      int e = first;
      for (; e < n && ok; e += kRowGroups) {
        // a stage's row numbers are loaded now and its copies issued when the group's next stage comes up, so that
        // the load overlaps the wait and copies of the one before
        const uint32_t line = __shfl_sync(0xFFFFFFFFu, entry.x, e);
        const int idx = __ldg(lines + (size_t)line * kTileM);
        if (pend_stage >= 0) run();
        pend_stage = next;
        pend_parity = phase;
        pend_kb = (int)__shfl_sync(0xFFFFFFFFu, entry.y, e);
        pend_idx = idx;
        next += kRowGroups;
        if (next >= p.a_stages) {
          next -= p.a_stages;
          phase ^= 1u;
        }
      }
      first = e - n;
    }
    flush();
    cp_async_wait_all();
  } else if (warp == kWarpW) {
    // =============================================================== W slices
    const int w_col_bytes = p.w_cols * ESIZE;
    const int kr = 128 / ESIZE;
    const uint32_t w_bytes = p.b_mn_major ? (uint32_t)(((w_col_bytes + 127) >> 7) * kr * 128) : (uint32_t)(p.w_rows * 128);
    int slot = 0;
    uint32_t phase = 0;
    walk_super_tiles(p, map, n_tiles, jobs, nothing, [&](int64_t, int k, int kb, uint32_t, uint32_t) {
      if (!mbar_wait_all(smem_u32(&ctl->w_empty[slot]), phase ^ 1u, abort_flag, 35)) return false;
      if (lane == 0) {
        const uint32_t bar = smem_u32(&ctl->w_full[slot]);
        const uint32_t dst = base + (uint32_t)slot * (uint32_t)p.w_slot_bytes;
        mbar_arrive_expect_tx(bar, w_bytes);
        const int kw = p.w_flip ? p.K - 1 - k : k;             // which W slice this offset multiplies with
        if (p.b_mn_major) {
          const int n_cb = (w_col_bytes + 127) >> 7;
          for (int cb = 0; cb < n_cb; ++cb)
            tma_load_2d(dst + (uint32_t)(cb * kr * 128), &w_desc, bar, cb * kr, kw * p.w_rows + kb * kr);
        } else {
          tma_load_2d(dst, &w_desc, bar, kb * kr, kw * p.w_rows);
        }
      }
      __syncwarp();
      if (++slot == p.w_slots) {
        slot = 0;
        phase ^= 1u;
      }
      return true;
    }, nothing);
  } else if (warp == kMmaWarp) {
    // =============================================================== MMA issuer
    // The whole warp runs this, converged, so that descriptors, ring positions and branches live in uniform registers, and
    // one elected lane issues.  As a branch of one lane the same code took 950 cycles per stage (130 per MMA, moving
    // its operands from vector to uniform registers), more than the copies or the MMAs themselves.
    {
      int stage = 0, slot = 0;
      uint32_t phase = 0, w_phase = 0;
      bool a_ready = false, w_ready = false;                   // what a look ahead at the next stage and slot said
      uint32_t acc_phase[2] = {0, 0};
      int buf = 0;
      const uint32_t b_kstep16 = (p.b_mn_major ? (32 / ESIZE) * 128 : 32) >> 4;   // K-step advance, 16-byte units
      const uint32_t b_lbo = p.b_mn_major ? (uint32_t)(128 / ESIZE) * 128u : 16u;
      const bool b_base32 = p.b_mn_major && ESIZE == 4;
      const uint64_t a_desc_hi = smem_desc(0u, 16u, 1024u, 2u);
      const uint64_t b_desc_hi = smem_desc(0u, b_lbo, b_base32 ? 512u : 1024u, b_base32 ? 1u : 2u);
      const uint32_t idesc = p.idesc;
      walk_super_tiles(p, map, n_tiles, jobs,
        [&](int64_t) {
          const bool ok = mbar_wait_all(smem_u32(&ctl->acc_empty[buf]), acc_phase[buf] ^ 1u, abort_flag, 32);
          tc_fence_after();
          return ok;
        },
        [&](int64_t, int, int kb, uint32_t users, uint32_t fresh) {
          if (!__all_sync(0xFFFFFFFFu, w_ready) && !mbar_wait_all(smem_u32(&ctl->w_full[slot]), w_phase, abort_flag, 33)) return false;
          const uint32_t w_lo = (base + (uint32_t)slot * (uint32_t)p.w_slot_bytes) >> 4;
          const int ksteps = min(128, red_bytes - kb * 128) >> 5;
#pragma unroll
          for (int s = 0; s < kMaxSub; ++s) {
            if (!((users >> s) & 1u)) continue;
            if (!__all_sync(0xFFFFFFFFu, a_ready) && !mbar_wait_all(smem_u32(&ctl->a_full[stage]), phase, abort_flag, 34)) return false;
            const int this_stage = stage;
            if (++stage == p.a_stages) {
              stage = 0;
              phase ^= 1u;
            }
            a_ready = mbar_try_now(smem_u32(&ctl->a_full[stage]), phase);
            fence_proxy_async();                                                 // rows were written by cp.async
            tc_fence_after();
            const uint32_t a_lo = (a_ring + (uint32_t)this_stage * kABlockBytes) >> 4;
            const uint32_t d_addr = tmem_base + (uint32_t)(buf * set_cols + s * p.c_acc);
            const uint32_t add = ((fresh >> s) & 1u) ? 0u : 1u;                  // 0: the first MMA overwrites
            if (elect_one()) {
#pragma unroll
              for (int ks = 0; ks < 4; ++ks) {
                if (ks < ksteps) {
                  const uint64_t da = a_desc_hi | (uint64_t)(a_lo + ks * 2);
                  const uint64_t db = b_desc_hi | (uint64_t)(w_lo + ks * b_kstep16);
                  if (ESIZE == 2)
                    mma_f16(d_addr, da, db, idesc, ks == 0 ? add : 1u);
                  else
                    mma_tf32(d_addr, da, db, idesc, ks == 0 ? add : 1u);
                }
              }
              mma_commit(smem_u32(&ctl->a_empty[this_stage]));
            }
          }
          if (elect_one()) mma_commit(smem_u32(&ctl->w_empty[slot]));
          if (++slot == p.w_slots) {
            slot = 0;
            w_phase ^= 1u;
          }
          w_ready = mbar_try_now(smem_u32(&ctl->w_full[slot]), w_phase);
          return true;
        },
        [&](int64_t) {
          if (elect_one()) mma_commit(smem_u32(&ctl->acc_full[buf]));
          acc_phase[buf] ^= 1u;
          if (p.acc_bufs == 2) buf ^= 1;
          return true;
        });
    }
    __syncwarp();
  } else {
    // =============================================================== epilogue (warps 0..3)
    uint32_t acc_phase[2] = {0, 0};
    int buf = 0;
    bool ok = true;
    const int out_es = p.out_kind == ST_F32 ? 4 : 2;
    const uint32_t stage_rows = out_ring + (uint32_t)warp * kOutWarpBytes;
    JobReader mine = jobs;
    while (ok && mine.next()) {
      const int64_t st_i = mine.job.super;
      // where this lane's rows go: known before the accumulators are ready, so fetched before the wait
      int64_t dst_rows[kMaxSub];
#pragma unroll
      for (int s = 0; s < kMaxSub; ++s) {
        const int64_t row = (st_i * p.sub + s) * (int64_t)kTileM + warp * 32 + lane;
        dst_rows[s] = (s < p.sub && p.order && row < p.n_rows) ? (int64_t)__ldg(p.order + row) : row;
      }
      const uint32_t touched = mine.job.touched;               // the others have no accumulator: their rows are zeros
      ok = mbar_wait(smem_u32(&ctl->acc_full[buf]), acc_phase[buf], abort_flag, 40, 256);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int s = 0; s < kMaxSub; ++s) {
        if (s >= p.sub) break;
        const int64_t row = (st_i * p.sub + s) * (int64_t)kTileM + warp * 32 + lane;
        if ((st_i * p.sub + s) * (int64_t)kTileM >= p.n_rows) break;         // whole sub tile past the end
        const uint32_t t_row = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(buf * set_cols + s * p.c_acc);
        const int dst = row < p.n_rows ? (int)dst_rows[s] : -1;
        const bool zeros = !((touched >> s) & 1u);
        int c0 = 0;
        for (; p.c_acc - c0 >= 128 / out_es; c0 += 128 / out_es) store_block<8>(p, stage_rows, t_row, c0, dst, zeros, lane);
        if (p.c_acc - c0 >= 64 / out_es) {
          store_block<4>(p, stage_rows, t_row, c0, dst, zeros, lane);
          c0 += 64 / out_es;
        }
        if (c0 < p.c_acc) store_block<2>(p, stage_rows, t_row, c0, dst, zeros, lane);
      }
      tc_fence_before();
      mbar_arrive(smem_u32(&ctl->acc_empty[buf]));
      acc_phase[buf] ^= 1u;
      if (p.acc_bufs == 2) buf ^= 1;
    }
  }

  // After an expired wait, bulk copies of this CTA may still be in flight: give them time to land
  // before the CTA's shared memory and mbarriers go away (they complete within microseconds).
  if (*abort_flag) {
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
}


// =================================================================================================
// Weight gradient over a stored map in tile-plan form.
//
//   dW[k][ci][co] = sum_r  X[tmap(r, k)][ci] * dY[order[r]][co]
//
// A CTA owns a group of G offsets (G accumulators fill TMEM), a block of output and one of input channels, and a share
// of the row tiles.  Per tile that has an offset of the group it brings in the tile operand (128 rows of dY, picked through
// `order`) once and the gathered operand (128 rows of X through the tile's index line) per offset; both come with 16-byte
// cp.async from 16 warps, as in planned_gather_kernel, through two rings, and announce themselves (an asynchronous arrival per
// thread): a warp that announced an item when its next one was on its way held back the two or three tile slots (256 -> 256,
// 95541 rows: 385 -> 340 us; two or three items held back: 440, 460).  With p.swap the plan is the INVERSE map's: the
// tile operand is X and the gathered one dY.
//
// How the CTAs are shared out: an odd kernel's centre offset occurs in every tile of a submanifold layer and the others in
// a tenth to a third of them, so equal shares left the centre's group with half of the work on a quarter of the CTAs.
// Every CTA therefore weighs the groups itself (stages over the tile masks, from L2, at most 4096 tiles looked at: 2-3 us)
// and all come to the same division, one or more CTAs per (group, channel blocks) in proportion.  One CTA per SM: every
// CTA writes its accumulators (up to 256 KB of fp32 partial sums), which a second kernel adds in a fixed order.
// =================================================================================================
constexpr int kWgradASlots3 = 4;
constexpr int kWgradBSlots3 = 12;
constexpr int kWgradRowWarp0 = kMmaWarp + 1;
constexpr int kWgrad3Threads = (kWgradRowWarp0 + kRowGroups * kRowGroupWarps) * 32;
constexpr int kWgradMaxGroups = 96;                             // ST_MAX_KVOL offsets in groups of four, and some
constexpr int64_t kWgradWeighed = 4096;                         // tiles looked at to weigh the groups

struct __align__(8) WgradControl3 {
  unsigned long long a_full[kWgradASlots3], a_empty[kWgradASlots3];
  unsigned long long b_full[kWgradBSlots3], b_empty[kWgradBSlots3];
  unsigned long long acc_full;
  uint32_t touched;
  uint32_t tmem_base;
  int abort_flag;
  int combo, first_cta, n_ctas;
  uint32_t weight[kWgradMaxGroups];
};

// f(tile, mask) for every tile of this CTA that has an offset of its group, 32 masks loaded at a time.
template <typename F>
__device__ __forceinline__ void walk_tiles(const WgradParams& p, const PlannedRows& map, int64_t first, int64_t step, int word,
                                           int shift, uint32_t group_bits, int lane, F&& f) {
  auto load = [&](int64_t t0) {
    const int64_t tile = t0 + lane * step;
    return tile < p.n_tiles ? (__ldg(map.tmask + tile * map.MW + word) >> shift) & group_bits : 0u;
  };
  uint32_t next = load(first);
  for (int64_t t0 = first; t0 < p.n_tiles; t0 += 32 * step) {
    const uint32_t mine = next;
    next = load(t0 + 32 * step);
    uint32_t live = __ballot_sync(0xFFFFFFFFu, mine != 0u);
    while (live) {
      const int l = __ffs(live) - 1;
      live &= live - 1;
      if (!f(t0 + l * step, __reduce_or_sync(0xFFFFFFFFu, lane == l ? mine : 0u))) return;
    }
  }
}

template <int ESIZE>
__global__ void __launch_bounds__(kWgrad3Threads, 1) planned_wgrad_kernel(const WgradParams p, const PlannedRows map) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_raw + (base - raw);
  const uint32_t a_ring = base;
  const uint32_t b_ring = base + (uint32_t)p.a_slots * (uint32_t)p.a_slot_bytes;
  WgradControl3* ctl = reinterpret_cast<WgradControl3*>(base_ptr + (size_t)p.a_slots * p.a_slot_bytes +
                                                        (size_t)p.b_slots * p.b_slot_bytes);
  volatile int* abort_flag = &ctl->abort_flag;
  const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  auto bits_of = [&](int kgroup) {
    const int n = min(p.group, p.K - kgroup * p.group);
    return n >= 32 ? 0xFFFFFFFFu : ((1u << n) - 1u);
  };

  for (int g = threadIdx.x; g < p.n_kgroups; g += kWgrad3Threads) ctl->weight[g] = 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.a_slots; ++s) {
      mbar_init(smem_u32(&ctl->a_full[s]), kRowGroups * kRowGroupWarps * 32);
      mbar_init(smem_u32(&ctl->a_empty[s]), 1);
    }
    for (int s = 0; s < p.b_slots; ++s) {
      mbar_init(smem_u32(&ctl->b_full[s]), kRowGroupWarps * 32);
      mbar_init(smem_u32(&ctl->b_empty[s]), 1);
    }
    mbar_init(smem_u32(&ctl->acc_full), 2);
    ctl->abort_flag = 0;
    ctl->touched = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(&ctl->tmem_base), (uint32_t)p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  // ---- which work is this CTA's: weigh the groups, divide gridDim.x CTAs among the combinations
  const int n_blocks2 = p.n_coblk * p.n_ciblk, n_combos = p.n_kgroups * n_blocks2;
  {
    const int64_t stride = p.n_tiles > kWgradWeighed ? p.n_tiles / kWgradWeighed : 1;
    for (int g = 0; g < p.n_kgroups; ++g) {
      const int k0 = g * p.group;
      uint32_t sum = 0;
      for (int64_t t = threadIdx.x * stride; t < p.n_tiles; t += kWgrad3Threads * stride) {
        const uint32_t m = (__ldg(map.tmask + t * map.MW + (k0 >> 5)) >> (k0 & 31)) & bits_of(g);
        if (m) sum += (uint32_t)p.weight_a + (uint32_t)__popc(m) * (uint32_t)p.weight_b;
      }
      sum = __reduce_add_sync(0xFFFFFFFFu, sum);
      if (lane == 0 && sum) atomicAdd(&ctl->weight[g], sum);
    }
    __syncthreads();
    uint64_t total = 0;
    for (int g = 0; g < p.n_kgroups; ++g) total += ctl->weight[g];
    if (total == 0) total = 1;
    auto start_of = [&](int combo) {                           // first CTA of a combination: one each, the rest by weight
      uint64_t before = 0;
      const int g = combo / n_blocks2;
      for (int i = 0; i < g; ++i) before += (uint64_t)ctl->weight[i] * n_blocks2;
      if (g < p.n_kgroups) before += (uint64_t)ctl->weight[g] * (combo - g * n_blocks2);
      return combo + (int)(before * (uint64_t)(gridDim.x - n_combos) / (total * n_blocks2));
    };
    for (int c = threadIdx.x; c < n_combos; c += kWgrad3Threads) {
      // with no neighbour anywhere the last combination takes what is left
      const int first = start_of(c), end = c + 1 == n_combos ? (int)gridDim.x : start_of(c + 1);
      if ((int)blockIdx.x >= first && (int)blockIdx.x < end) {
        ctl->combo = c;
        ctl->first_cta = first;
        ctl->n_ctas = end - first;
      }
      if (blockIdx.x == 0) {
        p.cta_table[c] = first;
        if (c + 1 == n_combos) p.cta_table[n_combos] = end;
      }
    }
    __syncthreads();
  }
  const int combo = __shfl_sync(0xFFFFFFFFu, ctl->combo, 0);
  const int kgroup = combo / n_blocks2;
  const int coblk = combo % n_blocks2 / p.n_ciblk, ciblk = combo % p.n_ciblk;
  const int64_t tile_begin = blockIdx.x - __shfl_sync(0xFFFFFFFFu, ctl->first_cta, 0);
  const int64_t tile_step = __shfl_sync(0xFFFFFFFFu, ctl->n_ctas, 0);       // neighbouring tiles are alike: deal them out
  const int k_first = kgroup * p.group;
  const int g_count = min(p.group, p.K - k_first);
  const int co0 = coblk * 128, co_cnt = min(128, p.cout - co0);
  const int ci0 = ciblk * p.ci_blk, ci_cnt = min(p.ci_blk, p.cin - ci0);
  const int word = k_first >> 5, shift = k_first & 31;
  const uint32_t group_bits = bits_of(kgroup);
  constexpr bool kBase32 = ESIZE == 4;                      // 32-bit elements: 128-byte swizzle with 32-byte atoms

  if (warp >= kWgradRowWarp0) {
    // =============================================================== rows
    // One sequence of items: per tile its tile operand (ring 1; every warp has 8 of its rows), then one item per offset
    // (ring 2; four groups of four warps take them in turn, a warp has 32 rows), all column blocks of a row.  Since every
    // warp waits for every slot of ring 1, none runs ahead by more than that ring; in ring 2 a warp's last item but one
    // tells it which lap the consumer is in as long as the ring is no shorter than the number of groups, else it waits for
    // every slot there too (a wait names a phase by its parity alone).
    const int row_warp = warp - kWgradRowWarp0;
    const int group = row_warp / kRowGroupWarps;
    const int row0 = row_warp % kRowGroupWarps * 32, t_row0 = row_warp * (kTileM / (kRowGroups * kRowGroupWarps));
    const bool every_slot = p.b_slots < kRowGroups;
    const char* x = static_cast<const char*>(p.x) + (size_t)ci0 * ESIZE;
    const char* dy = static_cast<const char*>(p.dy) + (size_t)co0 * ESIZE;
    const int x_bytes = ci_cnt * ESIZE, dy_bytes = co_cnt * ESIZE, x_pitch = p.cin * ESIZE, dy_pitch = p.cout * ESIZE;
    const char* t_src = p.swap ? x : dy;
    const char* g_src = p.swap ? dy : x;
    const int t_bytes = p.swap ? x_bytes : dy_bytes, g_bytes = p.swap ? dy_bytes : x_bytes;
    const int t_pitch = p.swap ? x_pitch : dy_pitch, g_pitch = p.swap ? dy_pitch : x_pitch;
    int a_slot = 0, b_slot = 0, turn = 0;
    uint32_t a_phase = 0, b_phase = 0;
    bool ok = true;
    bool pend = false, pend_b = false;
    int pend_slot = 0, pend_idx = -1;
    uint32_t pend_parity = 0;
    auto wait_for = [&](bool is_b, int slot, uint32_t parity) {
      return mbar_wait_all(smem_u32(is_b ? &ctl->b_empty[slot] : &ctl->a_empty[slot]), parity ^ 1u, abort_flag, is_b ? 36 : 35);
    };
    auto run = [&]() {
      ok = wait_for(pend_b, pend_slot, pend_parity);
      if (!ok) return;
      if (pend_b) {
        const uint32_t dst = b_ring + (uint32_t)pend_slot * (uint32_t)p.b_slot_bytes;
        for (int b = 0; b * 128 < g_bytes; ++b)
          fetch_block<32, kBase32>(dst + (uint32_t)b * kABlockBytes, row0, pend_idx, g_src + b * 128, g_pitch, p.n_src,
                                   min(128, g_bytes - b * 128), lane);
      } else {
        const uint32_t dst = a_ring + (uint32_t)pend_slot * (uint32_t)p.a_slot_bytes;
        for (int b = 0; b * 128 < t_bytes; ++b)
          fetch_block<8, kBase32>(dst + (uint32_t)b * kABlockBytes, t_row0, pend_idx, t_src + b * 128, t_pitch, p.n_rows,
                                  min(128, t_bytes - b * 128), lane);
      }
      cp_async_arrive_noinc(smem_u32(pend_b ? &ctl->b_full[pend_slot] : &ctl->a_full[pend_slot]));      // when they have landed
    };
    auto queue = [&](bool is_b, int slot, uint32_t parity, int idx) {
      if (pend) run();
      pend = true;
      pend_b = is_b;
      pend_slot = slot;
      pend_parity = parity;
      pend_idx = idx;
    };
    walk_tiles(p, map, tile_begin, tile_step, word, shift, group_bits, lane, [&](int64_t tile, uint32_t m) {
      const int64_t pos = tile * kTileM + t_row0 + (lane & 7);
      queue(false, a_slot, a_phase, pos < p.n_rows ? (p.order ? __ldg(p.order + pos) : (int)pos) : -1);
      if (++a_slot == p.a_slots) {
        a_slot = 0;
        a_phase ^= 1u;
      }
      while (m && ok) {
        if (turn == group) {
          const int j = __ffs(m) - 1;
          queue(true, b_slot, b_phase, __ldg(map.tmap + (tile * map.K + k_first + j) * (int64_t)kTileM + row0 + lane));
        } else if (every_slot) {
          if (pend) run();
          pend = false;
          if (ok) ok = wait_for(true, b_slot, b_phase);
        }
        m &= m - 1;
        turn = (turn + 1) & (kRowGroups - 1);
        if (++b_slot == p.b_slots) {
          b_slot = 0;
          b_phase ^= 1u;
        }
      }
      return ok;
    });
    if (pend && ok) run();
    cp_async_wait_all();
  } else if (warp == kMmaWarp) {
    // =============================================================== MMA issuer (see planned_gather_kernel)
    int a_slot = 0, b_slot = 0;
    uint32_t a_phase = 0, b_phase = 0;
    uint32_t touched = 0;
    bool ok = true;
    bool a_ready = false, b_ready = false;                     // what a look ahead at the next slots said
    constexpr int kRowsPerStep = 32 / ESIZE;                   // reduction rows per MMA (16 or 8)
    constexpr int kSteps = kTileM / kRowsPerStep;
    constexpr uint32_t kStep16 = kRowsPerStep * 128 / 16;
    const uint32_t idesc = p.idesc_base | ((uint32_t)(p.ci_blk >> 3) << 17);
    const uint64_t desc_hi = smem_desc(0u, kABlockBytes, kBase32 ? 512u : 1024u, kBase32 ? 1u : 2u);
    walk_tiles(p, map, tile_begin, tile_step, word, shift, group_bits, lane, [&](int64_t, uint32_t m) {
      ok = __all_sync(0xFFFFFFFFu, a_ready) || mbar_wait_all(smem_u32(&ctl->a_full[a_slot]), a_phase, abort_flag, 37);
      if (!ok) return false;
      const uint32_t t_lo = (a_ring + (uint32_t)a_slot * (uint32_t)p.a_slot_bytes) >> 4;
      while (m) {
        const int j = __ffs(m) - 1;
        m &= m - 1;
        ok = __all_sync(0xFFFFFFFFu, b_ready) || mbar_wait_all(smem_u32(&ctl->b_full[b_slot]), b_phase, abort_flag, 38);
        if (!ok) return false;
        const int this_slot = b_slot;
        if (++b_slot == p.b_slots) {
          b_slot = 0;
          b_phase ^= 1u;
        }
        b_ready = mbar_try_now(smem_u32(&ctl->b_full[b_slot]), b_phase);
        fence_proxy_async();                                   // rows were written by cp.async
        tc_fence_after();
        const uint32_t g_lo = (b_ring + (uint32_t)this_slot * (uint32_t)p.b_slot_bytes) >> 4;
        const uint32_t a_lo = p.swap ? g_lo : t_lo, b_lo = p.swap ? t_lo : g_lo;   // dY rows (M), X rows (N)
        const uint32_t d_addr = tmem_base + (uint32_t)(j * p.ci_blk);
        const uint32_t add = (touched >> j) & 1u;
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < kSteps; ++ks) {
            const uint64_t da = desc_hi | (uint64_t)(a_lo + ks * kStep16);
            const uint64_t db = desc_hi | (uint64_t)(b_lo + ks * kStep16);
            if (ESIZE == 2)
              mma_f16(d_addr, da, db, idesc, ks == 0 ? add : 1u);
            else
              mma_tf32(d_addr, da, db, idesc, ks == 0 ? add : 1u);
          }
          mma_commit(smem_u32(&ctl->b_empty[this_slot]));
        }
        touched |= 1u << j;
      }
      if (elect_one()) mma_commit(smem_u32(&ctl->a_empty[a_slot]));
      if (++a_slot == p.a_slots) {
        a_slot = 0;
        a_phase ^= 1u;
      }
      a_ready = mbar_try_now(smem_u32(&ctl->a_full[a_slot]), a_phase);
      return true;
    });
    if (ok && elect_one()) {
      ctl->touched = touched;
      mma_commit(smem_u32(&ctl->acc_full));
      mbar_arrive(smem_u32(&ctl->acc_full));
    }
    __syncwarp();
  } else {
    // =============================================================== epilogue (warps 0..3)
    bool ok = mbar_wait(smem_u32(&ctl->acc_full), 0u, abort_flag, 39, 512);
    ok = __all_sync(0xFFFFFFFFu, ok);
    if (ok) {
      tc_fence_after();
      const uint32_t touched = ctl->touched;
      const int co = warp * 32 + lane;                           // accumulator row = output channel
      const int co_w = min(p.cout, 128);
      float* mine = p.partial + (size_t)blockIdx.x * p.group * p.ci_blk * co_w + co;
      for (int j = 0; j < g_count; ++j) {
        const bool live = (touched >> j) & 1u;
        for (int c0 = 0; c0 < ci_cnt; c0 += 16) {
          uint32_t v[32];
          tmem_ld16(tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(j * p.ci_blk + c0), v);
          tmem_ld_wait();
          float* dst = mine + (size_t)(j * p.ci_blk + c0) * co_w;
          if (co < co_cnt) {
#pragma unroll
            for (int c = 0; c < 16; ++c) dst[(size_t)c * co_w] = live ? __uint_as_float(v[c]) : 0.f;
          }
        }
      }
    }
    tc_fence_before();
  }

  if (*abort_flag) {
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
}

template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// dW[k][ci][co] = sum over the CTAs of its combination, in order: eight slices of the CTAs per block, added from shared
// memory.  A block takes 32 x 4 consecutive output channels' worth of one (k, ci) row or several.
template <typename T>
__global__ void __launch_bounds__(256) wgrad_sum_kernel(const WgradParams p, T* __restrict__ dw) {
  __shared__ float4 part[8][32];
  const int slice = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int quads = p.cout >> 2;                                 // cout is a multiple of 8
  const int64_t n = (int64_t)p.K * p.cin * quads, i = (int64_t)blockIdx.x * 32 + lane;
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
  int k = 0, ci = 0, co = 0;
  if (i < n) {
    co = (int)(i % quads) * 4;
    ci = (int)(i / quads % p.cin);
    k = (int)(i / quads / p.cin);
    const int kgroup = k / p.group, j = k - kgroup * p.group;
    const int coblk = co / 128, ciblk = ci / p.ci_blk;
    const int combo = (kgroup * p.n_coblk + coblk) * p.n_ciblk + ciblk;
    const int co_w = min(p.cout, 128);
    const size_t cta_floats = (size_t)p.group * p.ci_blk * co_w;
    const float* src = p.partial + ((size_t)j * p.ci_blk + (ci - ciblk * p.ci_blk)) * co_w + (co - coblk * 128);
    const int first = p.cta_table[combo], end = p.cta_table[combo + 1];
#pragma unroll 4
    for (int c = first + slice; c < end; c += 8) {
      const float4 v = *reinterpret_cast<const float4*>(src + c * cta_floats);
      sum.x += v.x;
      sum.y += v.y;
      sum.z += v.z;
      sum.w += v.w;
    }
  }
  part[slice][lane] = sum;
  __syncthreads();
  if (slice == 0 && i < n) {
#pragma unroll
    for (int s = 1; s < 8; ++s) {
      const float4 v = part[s][lane];
      sum.x += v.x;
      sum.y += v.y;
      sum.z += v.z;
      sum.w += v.w;
    }
    T* out = dw + ((size_t)k * p.cin + ci) * p.cout + co;
    out[0] = from_f<T>(sum.x);
    out[1] = from_f<T>(sum.y);
    out[2] = from_f<T>(sum.z);
    out[3] = from_f<T>(sum.w);
  }
}

}  // namespace tc
}  // namespace st
