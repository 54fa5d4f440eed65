// fake_cudart.cpp -- a CPU stand-in for the CUDA runtime, linked with the
// library's objects in place of libcudart, for tests of the host code.
//
// Device memory is host memory. Work issued on a stream is queued and runs when
// the host waits for that stream (or for an event behind it), as late as the
// runtime's contract allows: a copy from pageable memory reads its source
// then, and memory that C++ code has freed is overwritten. Kernels do nothing
// but report themselves. Pinned allocations, launches and attributes can be
// limited, counted or made to fail.
#include <cuda_runtime_api.h>
#include <malloc.h>

#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <new>
#include <string>
#include <vector>

struct Stream {
  std::deque<std::function<void()>> q;
  long issued = 0, done = 0;
  bool running = false;
  double clock = 0.0;  // ms
};
struct Event {
  Stream* s = nullptr;
  long at = 0;
  double time = 0.0;
};

namespace {
Stream g_null;
std::vector<Stream*>& streams() { static std::vector<Stream*> v{&g_null}; return v; }
std::map<const void*, std::string>& names() { static std::map<const void*, std::string> m; return m; }
std::map<const void*, int>& smem() { static std::map<const void*, int> m; return m; }
std::map<char*, size_t>& pinned() { static std::map<char*, size_t> m; return m; }
size_t pinned_now = 0, pinned_peak = 0, pinned_limit = ~size_t(0);
long g_uploads = 0, g_queued = 0, g_queued_most = 0, g_changed = 0, g_lowered = 0, g_launches = 0, g_fail_at = -1;
std::string g_fail_name, g_log;
std::map<std::string, double>& costs() { static std::map<std::string, double> m; return m; }
double cost(const std::string& name) {
  for (auto& e : costs()) if (name.find(e.first) != std::string::npos) return e.second;
  return 0.0;
}
cudaError_t g_last = cudaSuccess;
void (*g_hook)(const char*) = nullptr;
struct Call { dim3 g, b; size_t m; cudaStream_t s; };
std::vector<Call> g_calls;

Stream* of(cudaStream_t s) { return s ? reinterpret_cast<Stream*>(s) : &g_null; }
void drain(Stream* s, long until) {
  if (s->running) return;
  s->running = true;
  while (s->done < until && !s->q.empty()) {
    auto f = std::move(s->q.front());
    s->q.pop_front();
    f();
    ++s->done;
  }
  s->running = false;
}
void push(Stream* s, std::function<void()> f) { s->q.push_back(std::move(f)); ++s->issued; }
bool is_pinned(const void* p) {
  for (auto& e : pinned())
    if (static_cast<const char*>(p) >= e.first && static_cast<const char*>(p) < e.first + e.second) return true;
  return false;
}
cudaError_t ret(cudaError_t e) { if (e != cudaSuccess) g_last = e; return e; }
}  // namespace

// Freed memory is overwritten and not handed out again.
void* operator new(size_t n) { if (void* p = std::malloc(n)) return p; throw std::bad_alloc(); }
void operator delete(void* p) noexcept { if (p) std::memset(p, 0xA5, malloc_usable_size(p)); }
void operator delete(void* p, size_t) noexcept { operator delete(p); }

extern "C" {
// ---- controls ----
long fake_uploads() { return g_uploads; }           // copies from pageable memory that have run
long fake_changed() { return g_changed; }           // of those, with another source than when they were issued
long fake_queued_most() { return g_queued_most; }   // largest sum of their bytes that had not run
long fake_lowered() { return g_lowered; }           // dynamic shared-memory limits set below an earlier value
size_t fake_pinned_peak() { return pinned_peak; }
void fake_pinned_limit(size_t n) { pinned_limit = n; pinned_peak = pinned_now; }
void fake_pin(void* p, size_t n) { pinned()[static_cast<char*>(p)] = n; }  // as cudaHostRegister
void fake_fail_launch(const char* name, long nth) { g_fail_name = name; g_fail_at = nth; }  // the nth of that name from now on
void fake_hook(void (*f)(const char*)) { g_hook = f; }  // called as each kernel runs
void fake_cost(const char* name, double ms) { costs()[name] = ms; }  // of kernels by part of their name, and of "memcpy"
const char* fake_log() { return g_log.c_str(); }

// ---- registration and launches ----
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, void*, void*, void*, void*, int*) {
  names()[f] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s) { g_calls.push_back({g, b, m, s}); return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
  const Call c = g_calls.back();
  g_calls.pop_back();
  *g = c.g; *b = c.b; *m = c.m;
  *static_cast<cudaStream_t*>(s) = c.s;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(f)); return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t m, cudaStream_t s) {
  const void* f = reinterpret_cast<const void*>(k);
  const std::string name = names()[f];
  if (m > 48 * 1024 && m > size_t(smem()[f])) return ret(cudaErrorInvalidValue);
  if (g_fail_at >= 0 && name.find(g_fail_name) != std::string::npos && g_fail_at-- == 0) return ret(cudaErrorLaunchFailure);
  ++g_launches;
  g_log += name + "\n";
  Stream* st = of(s);
  push(st, [name, st] {
    st->clock += cost(name);
    if (g_hook) g_hook(name.c_str());
  });
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
  if (v < smem()[f]) ++g_lowered;
  smem()[f] = v;
  return cudaSuccess;
}

// ---- streams and events ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { auto* p = new Stream; streams().push_back(p); *s = reinterpret_cast<cudaStream_t>(p); return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { drain(of(s), of(s)->issued); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { drain(of(s), of(s)->issued); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { for (Stream* s : streams()) drain(s, s->issued); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(new Event); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  auto* p = reinterpret_cast<Event*>(e);
  Stream* st = of(s);
  push(st, [p, st] { p->time = st->clock; });
  p->s = st;
  p->at = st->issued;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { auto* p = reinterpret_cast<Event*>(e); if (p->s) drain(p->s, p->at); return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t e) {
  auto* p = reinterpret_cast<Event*>(e);
  return !p->s || p->s->done >= p->at ? cudaSuccess : ret(cudaErrorNotReady);
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
  *ms = float(reinterpret_cast<Event*>(b)->time - reinterpret_cast<Event*>(a)->time);
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  const auto* p = reinterpret_cast<Event*>(e);
  const Event v = *p;
  Stream* st = of(s);
  if (v.s && v.s != st)
    push(st, [v, p, st] {
      drain(v.s, v.at);
      if (p->at == v.at && p->time > st->clock) st->clock = p->time;  // (not recorded anew meanwhile)
    });
  return cudaSuccess;
}

// ---- memory ----
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(1, n); return *p ? cudaSuccess : ret(cudaErrorMemoryAllocation); }
cudaError_t cudaFree(void* p) { cudaDeviceSynchronize(); std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  if (pinned_now + n > pinned_limit) return ret(cudaErrorMemoryAllocation);
  *p = std::malloc(n);
  pinned()[static_cast<char*>(*p)] = n;
  pinned_now += n;
  if (pinned_now > pinned_peak) pinned_peak = pinned_now;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  pinned_now -= pinned()[static_cast<char*>(p)];
  pinned().erase(static_cast<char*>(p));
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::memset(a, 0, sizeof(*a));
  a->type = is_pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  const char* host = static_cast<const char*>(k == cudaMemcpyHostToDevice ? s : d);
  if (n && k != cudaMemcpyDeviceToDevice && is_pinned(host) != is_pinned(host + n - 1)) return ret(cudaErrorInvalidValue);
  if (k == cudaMemcpyHostToDevice && !is_pinned(s)) {
    std::string was(static_cast<const char*>(s), n);
    g_queued += long(n);
    if (g_queued > g_queued_most) g_queued_most = g_queued;
    push(of(st), [=] {
      ++g_uploads;
      g_queued -= long(n);
      if (std::memcmp(s, was.data(), n) != 0) ++g_changed;
      std::memcpy(d, s, n);
    });
    return cudaSuccess;
  }
  push(of(st), [=] { of(st)->clock += cost("memcpy"); std::memcpy(d, s, n); });
  if (k == cudaMemcpyDeviceToHost && !is_pinned(d)) drain(of(st), of(st)->issued);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { drain(&g_null, g_null.issued); std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind k, cudaStream_t st) {
  push(of(st), [=] { of(st)->clock += cost("memcpy"); for (size_t i = 0; i < h; ++i) std::memcpy(static_cast<char*>(d) + i * dp, static_cast<const char*>(s) + i * sp, w); });
  if (k == cudaMemcpyDeviceToHost && !is_pinned(d)) drain(of(st), of(st)->issued);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) { push(of(s), [=] { std::memset(p, v, n); }); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return ret(cudaErrorInvalidSymbol); }

// ---- device ----
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 * 1024 : 0x7fffffff;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof(*p));
  std::strcpy(p->name, "fake");
  p->multiProcessorCount = 152;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* l, int* g) { *l = 0; *g = -5; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 1; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 1; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { *n = 64; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return g_last; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "fake error"; }

// ---- graphs: not modelled ----
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = nullptr; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}  // extern "C"
