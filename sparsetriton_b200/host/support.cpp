// Stage recorder, result slots, type codes.
#include <cuda_runtime_api.h>
#include <emmintrin.h>

#include "host.h"

namespace st_host {

int feat_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return ST_F32;
    case at::kHalf: return ST_F16;
    case at::kBFloat16: return ST_BF16;
    default: throw TypeError("features must be float32, float16 or bfloat16, got " + std::string(c10::toString(t.scalar_type())));
  }
}
int coord_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kShort: return ST_I16;
    case at::kInt: return ST_I32;
    default:
      throw TypeError("coordinates must be int16 or int32 for the CUDA kernels, got " + std::string(c10::toString(t.scalar_type())));
  }
}

// ------------------------------------------------------------------------------------------------ stage recorder
namespace {
struct Span {
  std::string name;
  cudaEvent_t start, stop;
  int64_t launches;
  double work;
  int tag_a, tag_b;
};
std::atomic<bool> g_tracing{false};
std::mutex g_trace_mutex;
std::vector<Span> g_spans;
}  // namespace

bool tracing() { return g_tracing.load(std::memory_order_relaxed); }

Stage::Stage(const char* name, cudaStream_t stream, double work, int tag_a, int tag_b)
    : name_(name), stream_(stream), work_(work), tag_a_(tag_a), tag_b_(tag_b) {
  if (!tracing()) return;
  cudaEvent_t e = nullptr;
  if (cudaEventCreate(&e) != cudaSuccess) return;
  launches_ = st_launch_count();
  cudaEventRecord(e, stream_);
  start_ = e;
}
Stage::~Stage() {
  if (!start_) return;
  cudaEvent_t stop = nullptr;
  if (cudaEventCreate(&stop) == cudaSuccess) {
    cudaEventRecord(stop, stream_);
    std::lock_guard<std::mutex> lock(g_trace_mutex);
    g_spans.push_back(Span{name_, static_cast<cudaEvent_t>(start_), stop, st_launch_count() - launches_, work_, tag_a_, tag_b_});
  } else {
    cudaEventDestroy(static_cast<cudaEvent_t>(start_));
  }
}
void trace_stop() {
  g_tracing = false;
  std::lock_guard<std::mutex> lock(g_trace_mutex);
  for (Span& s : g_spans) {
    cudaEventDestroy(s.start);
    cudaEventDestroy(s.stop);
  }
  g_spans.clear();
}
void trace_start() {
  trace_stop();
  g_tracing = true;
}
std::vector<std::tuple<std::string, double, int64_t, double, int, int>> trace_spans() {
  cudaDeviceSynchronize();
  std::vector<std::tuple<std::string, double, int64_t, double, int, int>> out;
  std::lock_guard<std::mutex> lock(g_trace_mutex);
  for (const Span& s : g_spans) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, s.start, s.stop);
    out.emplace_back(s.name, (double)ms, s.launches, s.work, s.tag_a, s.tag_b);
  }
  return out;
}

// ------------------------------------------------------------------------------------------------ result slots
namespace {
constexpr int kSlots = 4096, kMaxDevices = 64, kScratchWords = 16;
struct Pool {
  std::mutex mu;
  int32_t* host = nullptr;                         // kSlots x 16 words
  uint32_t* scratch[kMaxDevices] = {};             // kSlots x kScratchWords words per device, zero between uses
  std::vector<int> free;
  std::vector<std::pair<int, int32_t>> waiting;    // dropped before their ticket arrived
  int32_t next_ticket = 1;
};
Pool& pool() {
  static Pool* p = new Pool;                       // never destroyed: slots may outlive static destruction
  return *p;
}
}  // namespace

Mail::Mail(const Tensor& like) {
  device_ = like.device().index();
  Pool& p = pool();
  std::lock_guard<std::mutex> lock(p.mu);
  if (!p.host) {
    void* mem = nullptr;
    if (cudaHostAlloc(&mem, (size_t)kSlots * 64, cudaHostAllocPortable) != cudaSuccess)
      throw std::runtime_error("cannot allocate pinned memory for device results");
    p.host = static_cast<int32_t*>(mem);
    for (int i = kSlots - 1; i >= 0; --i) p.free.push_back(i);
  }
  if (device_ < 0 || device_ >= kMaxDevices) throw std::runtime_error("device index out of range");
  if (!p.scratch[device_]) {
    void* mem = nullptr;
    const size_t bytes = (size_t)kSlots * kScratchWords * 4;
    if (cudaMalloc(&mem, bytes) != cudaSuccess || cudaMemset(mem, 0, bytes) != cudaSuccess ||
        cudaDeviceSynchronize() != cudaSuccess)
      throw std::runtime_error("cannot allocate scratch for device results");
    p.scratch[device_] = static_cast<uint32_t*>(mem);
  }
  if (p.free.empty() || p.waiting.size() > 64) {
    size_t kept = 0;
    for (auto& w : p.waiting) {
      if (*(volatile int32_t*)(p.host + w.first * 16 + 15) == w.second) p.free.push_back(w.first);
      else p.waiting[kept++] = w;
    }
    p.waiting.resize(kept);
  }
  if (p.free.empty()) throw std::runtime_error("too many device results outstanding");
  slot_ = p.free.back();
  p.free.pop_back();
  ticket_ = p.next_ticket;
  p.next_ticket = p.next_ticket == INT32_MAX ? 1 : p.next_ticket + 1;
  host_ = p.host + slot_ * 16;
  scratch_ = p.scratch[device_] + slot_ * kScratchWords;
  *(volatile int32_t*)(host_ + 15) = 0;
}

Mail::~Mail() {
  Pool& p = pool();
  std::lock_guard<std::mutex> lock(p.mu);
  if (sent_ && !arrived()) p.waiting.emplace_back(slot_, ticket_);
  else p.free.push_back(slot_);
}

void Mail::wait(cudaStream_t stream) {
  for (int64_t spins = 1; !arrived(); ++spins) {
    _mm_pause();
    if (spins % 65536 == 0) {
      const cudaError_t e = cudaStreamQuery(stream);
      if (e == cudaSuccess) {
        // everything the stream held is done: the ticket is there, or it never comes
        if (arrived()) break;
        throw std::runtime_error("a device result did not arrive");
      }
      if (e != cudaErrorNotReady) {
        cudaGetLastError();
        throw std::runtime_error(std::string("CUDA error: ") + cudaGetErrorString(e));
      }
    }
  }
  std::atomic_thread_fence(std::memory_order_acquire);
}

}  // namespace st_host
