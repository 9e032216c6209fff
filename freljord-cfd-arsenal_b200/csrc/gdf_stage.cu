// gdf_stage.cu -- the pinned ring behind gdf_stage.h.
//
// One ring per device, its events made on that device (an event is recorded on
// streams of its own device only). A copy holds the ring for its whole length; a copy that
// finds it taken (another thread's) goes to cudaMemcpyAsync, so threads never
// wait for each other here. A slot is reused when the event recorded behind its
// last transfer has passed, whatever stream that was on.
#include "gdf_stage.h"

#include <algorithm>
#include <mutex>

namespace gdf {
namespace {

struct Ring {
  std::mutex mu;
  int holders = 0;
  size_t asked = 0;   // bytes asked for since it was last dropped
  char* buf[STAGE_SLOTS] = {};
  cudaEvent_t ev[STAGE_SLOTS] = {};
  bool ready = false;
};
constexpr int MAX_DEV = 64;
Ring g_ring[MAX_DEV];

void drop(Ring& r) {
  for (int k = 0; k < STAGE_SLOTS; ++k) {
    if (r.ev[k]) {
      cudaEventSynchronize(r.ev[k]);
      cudaEventDestroy(r.ev[k]);
    }
    if (r.buf[k]) cudaFreeHost(r.buf[k]);
    r.ev[k] = nullptr;
    r.buf[k] = nullptr;
  }
  r.ready = false;
  r.asked = 0;
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

bool make(Ring& r, int dev) {
  if (r.ready) return true;
  const OnDevice on(dev);
  bool ok = on.ok;
  for (int k = 0; ok && k < STAGE_SLOTS; ++k)
    ok = cudaHostAlloc((void**)&r.buf[k], STAGE_CHUNK, cudaHostAllocPortable) == cudaSuccess &&
         cudaEventCreateWithFlags(&r.ev[k], cudaEventDisableTiming) == cudaSuccess;
  if (!ok) {
    drop(r);
    return false;
  }
  r.ready = true;
  return true;
}

// device dev's ring, locked in lk, for a pageable array of this size; null:
// copy plainly
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
  r.asked += std::min(bytes, STAGE_MAKE);
  if (r.asked < STAGE_MAKE || !make(r, dev)) return nullptr;
  r.asked = STAGE_MAKE;
  return &r;
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
  if (!r) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
  int k = 0;
  for (size_t o = 0; o < bytes; o += STAGE_CHUNK, k = (k + 1) % STAGE_SLOTS) {
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
  if (!r) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
  const size_t chunks = (bytes + STAGE_CHUNK - 1) / STAGE_CHUNK;
  auto issue = [&](size_t c) {
    const int k = (int)(c % STAGE_SLOTS);
    const size_t o = c * STAGE_CHUNK, n = std::min(STAGE_CHUNK, bytes - o);
    cudaError_t e = cudaEventSynchronize(r->ev[k]);
    if (e == cudaSuccess) e = cudaMemcpyAsync(r->buf[k], (const char*)src + o, n, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = record(r->ev[k], st);
    return e;
  };
  cudaError_t e = cudaSuccess;
  for (size_t c = 0; e == cudaSuccess && c < std::min(chunks, (size_t)STAGE_SLOTS); ++c) e = issue(c);
  for (size_t c = 0; e == cudaSuccess && c < chunks; ++c) {
    const size_t o = c * STAGE_CHUNK, n = std::min(STAGE_CHUNK, bytes - o);
    e = cudaEventSynchronize(r->ev[c % STAGE_SLOTS]);
    if (e != cudaSuccess) break;
    par_memcpy((char*)dst + o, r->buf[c % STAGE_SLOTS], n);
    if (c + STAGE_SLOTS < chunks) e = issue(c + STAGE_SLOTS);
  }
  return e;
}

}  // namespace gdf
