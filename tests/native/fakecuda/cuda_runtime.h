// A CUDA runtime for the host: as much of it as csrc/gdf_stage.cu calls, with two
// devices, streams whose copies from and to pinned memory run only when somebody
// waits for them, and events that belong to a device. Header-only, one
// translation unit.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorInvalidResourceHandle = 400, cudaErrorUnknown = 999 };
enum cudaMemcpyKind { cudaMemcpyHostToHost, cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost, cudaMemcpyDeviceToDevice };
enum cudaMemoryType { cudaMemoryTypeUnregistered, cudaMemoryTypeHost, cudaMemoryTypeDevice };
enum { cudaHostAllocPortable = 1, cudaHostRegisterPortable = 1, cudaEventDisableTiming = 2 };
struct cudaPointerAttributes { cudaMemoryType type; };

namespace fake {
struct Stream {
  int dev;
  std::deque<std::function<void()>> q;
  long run = 0;   // work done so far
  void drain(long upto = -1) {
    while (!q.empty() && (upto < 0 || run < upto)) {
      auto f = q.front();
      q.pop_front();
      f();
      ++run;
    }
  }
};
struct Event { int dev; Stream* s; long upto; };
inline int dev = 0, live_events = 0, record_fails = 0, pin_calls = 0;
inline long staged = 0, plain = 0;               // copies by kind of their host memory
inline int64_t now = 0;                          // ns: a byte copied plainly takes one
inline std::map<uintptr_t, size_t> pinned;        // start -> bytes
inline bool is_pinned(const void* p) {
  auto it = pinned.upper_bound((uintptr_t)p);
  return it != pinned.begin() && (uintptr_t)p < (--it)->first + it->second;
}
}  // namespace fake
typedef fake::Stream* cudaStream_t;
typedef fake::Event* cudaEvent_t;

inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaGetDevice(int* d) { *d = fake::dev; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int d) { fake::dev = d; return cudaSuccess; }
inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::malloc(n);
  fake::pinned[(uintptr_t)*p] = n;
  ++fake::pin_calls;
  return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p) {
  fake::pinned.erase((uintptr_t)p);
  std::free(p);
  return cudaSuccess;
}
inline cudaError_t cudaHostRegister(void* p, size_t n, unsigned) {
  fake::pinned[(uintptr_t)p] = n;
  ++fake::pin_calls;
  return cudaSuccess;
}
inline cudaError_t cudaHostUnregister(void* p) {
  fake::pinned.erase((uintptr_t)p);
  return cudaSuccess;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  a->type = fake::is_pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = new fake::Event{fake::dev, nullptr, 0};
  ++fake::live_events;
  return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete e;
  --fake::live_events;
  return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  if (e->dev != s->dev) return cudaErrorInvalidResourceHandle;
  if (fake::record_fails > 0 && --fake::record_fails == 0) return cudaErrorUnknown;
  e->s = s;
  e->upto = s->run + (long)s->q.size();
  return cudaSuccess;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  if (e->s) e->s->drain(e->upto);
  return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  s->drain();
  return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  const void* host = k == cudaMemcpyHostToDevice ? s : d;
  if (fake::is_pinned(host)) {
    ++fake::staged;
    st->q.push_back([=] { std::memcpy(d, s, n); });
  } else {   // pageable: done with the host's side on return
    ++fake::plain;
    fake::now += (int64_t)n;
    st->drain();
    std::memcpy(d, s, n);
  }
  return cudaSuccess;
}
