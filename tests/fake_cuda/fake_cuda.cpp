// A stand-in for the CUDA runtime, linked with libewt's objects so that the
// library's host code runs on the CPU: "device" memory is host memory (zeroed,
// counted), copies are done at once, kernels do nothing.  Tests ask for the
// n-th call of a function to fail, and read back what the library did: the
// launches, the bytes held at the peak, and whether work was still queued when
// an entry point returned.
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <sys/mman.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

namespace {

struct Stream {
  uint64_t queued = 0, done = 0;  // operations
  bool alive = true;
  struct Wait {
    uint64_t at;  // operations of this stream queued before the wait
    Stream* on;
    uint64_t upto;
  };
  std::vector<Wait> waits;
};
struct Event {
  Stream* on = nullptr;
  uint64_t upto = 0;
};

std::recursive_mutex mu;
std::vector<std::unique_ptr<Stream>> streams;
std::map<void*, size_t> blocks;                  // device allocations
std::map<void const*, std::string> kernels;      // host function -> name
std::map<std::string, long> settings;
std::map<std::string, long> fail_at, calls;
std::multimap<uint64_t, std::pair<uint64_t, uint64_t>> patches;  // copy size -> from entry, value
uint64_t live = 0, peak = 0;
std::string journal;
Stream null_stream;
thread_local cudaError_t last_error = cudaSuccess;
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
};
thread_local std::vector<Config> configs;

long setting(char const* name, long fallback) {
  auto const it = settings.find(name);
  return it == settings.end() ? fallback : it->second;
}
// Whether this call of `name` is the one that fails.
bool fails(char const* name) {
  long const n = ++calls[name];
  auto const it = fail_at.find(name);
  return it != fail_at.end() && it->second == n;
}
cudaError_t answer(char const* name) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (fails(name)) return last_error = cudaErrorUnknown;
  return cudaSuccess;
}
Stream* of(cudaStream_t s) {
  return s ? reinterpret_cast<Stream*>(s) : &null_stream;
}
void queue_op(cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  ++of(s)->queued;
}
void finish(Stream* s, uint64_t upto) {
  if (upto <= s->done) return;
  s->done = upto;
  for (auto const& w : s->waits)
    if (w.at < upto) finish(w.on, w.upto);
}
cudaError_t give(void** p, size_t n) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (fails("alloc")) {
    *p = nullptr;
    return last_error = cudaErrorMemoryAllocation;
  }
  // (reserved address space: hardly any of it is touched)
  *p = mmap(nullptr, n + 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1,
            0);
  blocks[*p] = n;
  live += n;
  if (live > peak) peak = live;
  return cudaSuccess;
}
void take(void* p) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  auto const it = blocks.find(p);
  if (it == blocks.end()) return;
  live -= it->second;
  munmap(p, it->second + 1);
  blocks.erase(it);
}
// Large copies move nothing (their contents do not matter to the host code).
void move(void* dst, void const* src, size_t n, cudaMemcpyKind kind) {
  if (n <= (size_t(64) << 20)) std::memmove(dst, src, n);
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (kind != cudaMemcpyDeviceToHost) return;
  auto const range = patches.equal_range(n);
  for (auto it = range.first; it != range.second; ++it)
    for (uint64_t i = it->second.first; i < n / 8; ++i)
      static_cast<uint64_t*>(dst)[i] = it->second.second;
}

}  // namespace

extern "C" {

// ---- what the tests use ----------------------------------------------------
void fake_reset() {
  std::lock_guard<std::recursive_mutex> lk(mu);
  fail_at.clear();
  calls.clear();
  patches.clear();
  journal.clear();
  peak = live;
}
void fake_set(char const* name, long v) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  settings[name] = v;
}
void fake_fail(char const* call, long n) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  calls[call] = 0;
  fail_at[call] = n;
}
long fake_calls(char const* call) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  return calls[call];
}
// Copies of `bytes` bytes to the host hold `value` from 64-bit entry `from` on
// (of several, the later ones win).
void fake_patch(uint64_t bytes, uint64_t from, uint64_t value) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  patches.insert({bytes, {from, value}});
}
uint64_t fake_live() { return live; }
uint64_t fake_peak() { return peak; }
// Streams with operations that nothing has waited for.
long fake_pending() {
  std::lock_guard<std::recursive_mutex> lk(mu);
  long n = null_stream.done < null_stream.queued;
  for (auto const& s : streams) n += s->done < s->queued;
  return n;
}
// "kernel grid block shared-memory" of every launch, a line each.
char const* fake_journal() { return journal.c_str(); }

// ---- launches -----------------------------------------------------------------
void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*,
                            dim3*, dim3*, int*) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* host) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(host));
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  configs.push_back({grid, block, smem, s});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* s) {
  Config const c = configs.back();
  configs.pop_back();
  *grid = c.grid;
  *block = c.block;
  *smem = c.smem;
  *static_cast<cudaStream_t*>(s) = c.stream;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void**, size_t smem,
                               cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (fails("launch")) return last_error = cudaErrorUnknown;
  queue_op(s);
  journal += kernels[reinterpret_cast<void const*>(k)] + " " + std::to_string(grid.x) + " " +
             std::to_string(block.x) + " " + std::to_string(smem) + "\n";
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  std::memset(a, 0, sizeof(*a));
  a->binaryVersion = 103;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
  return answer("cudaFuncSetAttribute");
}
// By shared memory, with `static_smem` bytes of it and 1 KB per CTA in every
// kernel, and at most `max_ctas` (as registers may have it).
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int block,
                                                                   size_t smem, unsigned) {
  long const by_smem = (228 << 10) / (long(smem) + setting("static_smem", 2048) + 1024);
  *n = static_cast<int>(std::min({by_smem, 2048l / block, setting("max_ctas", 32)}));
  return answer("occupancy");
}

// ---- memory --------------------------------------------------------------------
cudaError_t cudaMalloc(void** p, size_t n) { return give(p, n); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
  return give(p, n);
}
cudaError_t cudaFree(void* p) {
  take(p);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  take(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(n, 1);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind kind) {
  move(dst, src, n, kind);
  return answer("cudaMemcpy");
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind,
                            cudaStream_t s) {
  cudaError_t const e = answer("cudaMemcpyAsync");
  if (e != cudaSuccess) return e;
  move(dst, src, n, kind);
  queue_op(s);
  return e;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
  if (n <= (size_t(64) << 20)) std::memset(p, v, n);
  return answer("cudaMemsetAsync");
}
cudaError_t cudaMemGetInfo(size_t* free_b, size_t* total) {
  *free_b = *total = size_t(setting("free_gb", 0)) << 30;
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
  static int pool;
  *p = reinterpret_cast<cudaMemPool_t>(&pool);
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void* v) {
  std::memset(v, 0, 8);
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) {
  *p = const_cast<void*>(symbol);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  std::memset(a, 0, sizeof(*a));
  a->type = static_cast<cudaMemoryType>(setting("host_type", cudaMemoryTypeUnregistered));
  auto it = blocks.upper_bound(const_cast<void*>(p));
  if (it != blocks.begin()) {
    --it;
    if (static_cast<char const*>(p) < static_cast<char const*>(it->first) + it->second)
      a->type = cudaMemoryTypeDevice;
  }
  return cudaSuccess;
}

// ---- streams, events, devices -----------------------------------------------
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  streams.push_back(std::make_unique<Stream>());
  *s = reinterpret_cast<cudaStream_t>(streams.back().get());
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  finish(of(s), of(s)->queued);
  return answer("cudaStreamSynchronize");
}
cudaError_t cudaDeviceSynchronize() {
  std::lock_guard<std::recursive_mutex> lk(mu);
  for (auto const& s : streams) s->done = s->queued;
  null_stream.done = null_stream.queued;
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
  *c = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = reinterpret_cast<cudaEvent_t>(new Event());
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete reinterpret_cast<Event*>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (fails("cudaEventRecord")) return last_error = cudaErrorUnknown;
  Event* const ev = reinterpret_cast<Event*>(e);
  ev->on = of(s);
  ev->upto = of(s)->queued;
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (fails("cudaStreamWaitEvent")) return last_error = cudaErrorUnknown;
  Event* const ev = reinterpret_cast<Event*>(e);
  if (ev->on) {
    Stream* const st = of(s);
    st->waits.push_back({st->queued, ev->on, ev->upto});
    ++st->queued;  // the wait itself
  }
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  Event* const ev = reinterpret_cast<Event*>(e);
  if (ev->on) finish(ev->on, ev->upto);
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.f;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  *v = 0;
  if (a == cudaDevAttrMultiProcessorCount) *v = static_cast<int>(setting("sms", 152));
  if (a == cudaDevAttrPageableMemoryAccess) *v = static_cast<int>(setting("pageable", 1));
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  cudaError_t const e = last_error;
  last_error = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "an error of the stand-in"; }

}  // extern "C"

// The library's std::thread objects start here: the n-th start can fail as it
// does when the system has no thread to give.
void std::thread::_M_start_thread(_State_ptr state, void (*depend)()) {
  if (answer("thread") != cudaSuccess) {
    cudaGetLastError();
    throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
  }
  using Start = void (*)(std::thread*, _State_ptr, void (*)());
  static Start const start = reinterpret_cast<Start>(dlsym(
      RTLD_NEXT, "_ZNSt6thread15_M_start_threadESt10unique_ptrINS_6_StateESt14default_deleteIS1_EEPFvvE"));
  start(this, std::move(state), depend);
}
