// gdf_stage.cu -- the pinned ring behind gdf_stage.h.
//
// One ring per device, its events made on that device (an event is recorded on
// streams of its own device only). A copy holds the ring for its whole length; a
// copy that finds it taken (another thread's) goes to cudaMemcpyAsync, so threads
// never wait for each other here. A slot is reused when the event recorded behind
// its last transfer has passed, whatever stream that was on.
#include "gdf_stage.h"

#include <sys/mman.h>

#include <algorithm>
#include <chrono>
#include <cstdint>
#include <mutex>

namespace gdf {
namespace {

struct Ring {
  std::mutex mu;
  int holders = 0;
  int64_t past_ns = 0;  // what the copies that went plainly past it took
  int slots = 0;        // slots it has
  bool failed = false;  // a slot could not be made: no further one is tried
  char* buf[STAGE_SLOTS] = {};
  cudaEvent_t ev[STAGE_SLOTS] = {};
};
constexpr int MAX_DEV = 64;
Ring g_ring[MAX_DEV];

// The slots are anonymous memory in huge pages, registered: 0.8 ms for one (0.3 of
// it the pages' zeros; in small pages 4.5 ms), 2.3 to 3 ms for four, 0.5 ms and
// more to give four back. cudaHostAlloc took 2-5 ms for one, 9-18 for four. A
// forked child does not get the pages, so a write of the parent's never moves them
// from under a transfer.
constexpr size_t HUGE = (size_t)2 << 20;
char* pages() {
  void* p = mmap(nullptr, STAGE_CHUNK + HUGE, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (p == MAP_FAILED) return nullptr;
  char* at = (char*)(((uintptr_t)p + HUGE - 1) / HUGE * HUGE);
  if (at > (char*)p) munmap(p, at - (char*)p);
  munmap(at + STAGE_CHUNK, (char*)p + HUGE - at);
  madvise(at, STAGE_CHUNK, MADV_HUGEPAGE);   // small pages will do
  madvise(at, STAGE_CHUNK, MADV_DONTFORK);
  par_zero(at, STAGE_CHUNK);
  if (cudaHostRegister(at, STAGE_CHUNK, cudaHostRegisterPortable) == cudaSuccess) return at;
  cudaGetLastError();
  munmap(at, STAGE_CHUNK);
  return nullptr;
}

void drop(Ring& r) {
  for (int k = 0; k < r.slots; ++k) {
    cudaEventSynchronize(r.ev[k]);
    cudaEventDestroy(r.ev[k]);
    cudaHostUnregister(r.buf[k]);
    munmap(r.buf[k], STAGE_CHUNK);
  }
  r.slots = 0;
  r.past_ns = 0;
  r.failed = false;
  cudaGetLastError();
}

// the device dev current in its scope
struct OnDevice {
  int prev = -1;
  bool ok;
  explicit OnDevice(int dev) {
    ok = cudaGetDevice(&prev) == cudaSuccess;
    if (ok && prev == dev) prev = -1;
    else if (ok) ok = cudaSetDevice(dev) == cudaSuccess;
  }
  ~OnDevice() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

// up to want slots
void make(Ring& r, int want, int dev) {
  if (r.slots >= want || r.failed) return;
  const OnDevice on(dev);
  while (on.ok && r.slots < want) {
    cudaEvent_t ev = nullptr;
    char* buf = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) == cudaSuccess ? pages() : nullptr;
    if (!buf) {
      if (ev) cudaEventDestroy(ev);
      cudaGetLastError();
      r.failed = true;
      return;
    }
    r.ev[r.slots] = ev;
    r.buf[r.slots++] = buf;
  }
}

#ifndef GDF_STAGE_CLOCK
#define GDF_STAGE_CLOCK                                                                                \
  std::chrono::duration_cast<std::chrono::nanoseconds>(std::chrono::steady_clock::now().time_since_epoch()) \
      .count()
#endif
int64_t clock_ns() { return GDF_STAGE_CLOCK; }

// device dev's ring, locked in lk, with a slot for each of the copy's chunks (as
// many as there are at most), for a pageable array of this size; null: copy
// plainly, with lk held: add the copy's time
Ring* take(int dev, const void* host, size_t bytes, std::unique_lock<std::mutex>& lk) {
  if (dev < 0 || bytes < STAGE_MIN) return nullptr;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (a.type != cudaMemoryTypeUnregistered) return nullptr;
  Ring& r = g_ring[dev];
  lk = std::unique_lock<std::mutex>(r.mu, std::try_to_lock);
  if (!lk.owns_lock()) return nullptr;
  if (bytes >= STAGE_NOW || r.past_ns >= STAGE_DUE_NS)
    make(r, (int)std::min<size_t>(STAGE_SLOTS, (bytes + STAGE_CHUNK - 1) / STAGE_CHUNK), dev);
  return r.slots > 0 ? &r : nullptr;
}
// A copy without a ring, its time counted where take left lk held. The driver is
// done with a pageable array on return; what the stream still had to do before a
// copy to the host is not the copy's time.
cudaError_t plain(int dev, std::unique_lock<std::mutex>& lk, void* dst, const void* src, size_t bytes,
                  cudaMemcpyKind kind, cudaStream_t st) {
  if (!lk.owns_lock()) return cudaMemcpyAsync(dst, src, bytes, kind, st);
  lk.unlock();   // other threads' copies need not wait for this one
  if (kind == cudaMemcpyDeviceToHost) cudaStreamSynchronize(st);   // its errors are the copy's, too
  const int64_t t0 = clock_ns();
  const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, kind, st);
  const int64_t t = clock_ns() - t0;
  if (lk.try_lock()) g_ring[dev].past_ns = std::min(g_ring[dev].past_ns + t, STAGE_DUE_NS);
  return e;
}

// The event behind a slot's transfer. Without one the next copy would take the
// slot while the transfer still uses it, so a failure waits for the transfer.
cudaError_t record(cudaEvent_t ev, cudaStream_t st) {
  const cudaError_t e = cudaEventRecord(ev, st);
  if (e != cudaSuccess) cudaStreamSynchronize(st);
  return e;
}

}  // namespace

StageRef::StageRef() : dev(-1) {
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEV) {
    cudaGetLastError();
    dev = -1;
    return;
  }
  std::lock_guard<std::mutex> lk(g_ring[dev].mu);
  ++g_ring[dev].holders;
}

StageRef::~StageRef() {
  if (dev < 0) return;
  std::lock_guard<std::mutex> lk(g_ring[dev].mu);
  if (--g_ring[dev].holders == 0) drop(g_ring[dev]);
}

cudaError_t StageRef::h2d(void* dst, const void* src, size_t bytes, cudaStream_t st) {
  std::unique_lock<std::mutex> lk;
  Ring* r = take(dev, src, bytes, lk);
  if (!r) return plain(dev, lk, dst, src, bytes, cudaMemcpyHostToDevice, st);
  int k = 0;
  for (size_t o = 0; o < bytes; o += STAGE_CHUNK, k = (k + 1) % r->slots) {
    const size_t n = std::min(STAGE_CHUNK, bytes - o);
    cudaError_t e = cudaEventSynchronize(r->ev[k]);
    if (e != cudaSuccess) return e;
    par_memcpy(r->buf[k], (const char*)src + o, n);
    e = cudaMemcpyAsync((char*)dst + o, r->buf[k], n, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = record(r->ev[k], st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t StageRef::d2h(void* dst, const void* src, size_t bytes, cudaStream_t st) {
  std::unique_lock<std::mutex> lk;
  Ring* r = take(dev, dst, bytes, lk);
  if (!r) return plain(dev, lk, dst, src, bytes, cudaMemcpyDeviceToHost, st);
  const size_t chunks = (bytes + STAGE_CHUNK - 1) / STAGE_CHUNK, slots = r->slots;
  auto issue = [&](size_t c) {
    const int k = (int)(c % slots);
    const size_t o = c * STAGE_CHUNK, n = std::min(STAGE_CHUNK, bytes - o);
    cudaError_t e = cudaEventSynchronize(r->ev[k]);
    if (e == cudaSuccess) e = cudaMemcpyAsync(r->buf[k], (const char*)src + o, n, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = record(r->ev[k], st);
    return e;
  };
  cudaError_t e = cudaSuccess;
  for (size_t c = 0; e == cudaSuccess && c < std::min(chunks, slots); ++c) e = issue(c);
  for (size_t c = 0; e == cudaSuccess && c < chunks; ++c) {
    const size_t o = c * STAGE_CHUNK, n = std::min(STAGE_CHUNK, bytes - o);
    e = cudaEventSynchronize(r->ev[c % slots]);
    if (e != cudaSuccess) break;
    par_memcpy((char*)dst + o, r->buf[c % slots], n);
    if (c + slots < chunks) e = issue(c + slots);
  }
  return e;
}

}  // namespace gdf
