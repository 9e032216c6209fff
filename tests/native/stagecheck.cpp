// Host build of the pinned ring (csrc/gdf_stage.cu) on the fake runtime of
// fakecuda/ and its clock. Each check returns 0, or the line it failed at.
#include <cuda_runtime.h>
#define GDF_STAGE_CLOCK fake::now
#include "../../freljord-cfd-arsenal_b200/csrc/gdf_stage.cu"

#include <vector>

namespace gdf {
void par_memcpy(void* d, const void* s, size_t n) { std::memcpy(d, s, n); }
void par_zero(void* d, size_t n) { std::memset(d, 0, n); }
}  // namespace gdf

using namespace gdf;
typedef std::vector<unsigned char> Bytes;

#define REQUIRE(x) \
  do {             \
    if (!(x)) return __LINE__; \
  } while (0)

namespace {
const size_t LONG = 100 << 20;   // a copy that makes the ring at once

Bytes pattern(size_t n, unsigned seed) {
  Bytes b(n);
  for (size_t k = 0; k < n; ++k) b[k] = (unsigned char)((k >> 12) * 7 + k + seed);
  return b;
}
// one copy there and back through ref on st
int round_trip(StageRef& ref, cudaStream_t st, size_t n, unsigned seed) {
  const Bytes src = pattern(n, seed);
  Bytes devmem(n), back(n);
  REQUIRE(ref.h2d(devmem.data(), src.data(), n, st) == cudaSuccess);
  REQUIRE(ref.d2h(back.data(), devmem.data(), n, st) == cudaSuccess);
  REQUIRE(cudaStreamSynchronize(st) == cudaSuccess);
  REQUIRE(devmem == src && back == src);
  return 0;
}
}  // namespace

extern "C" {

// copies of one device's handle while another device is current
int check_other_device_current() {
  fake::Stream s0{0, {}}, s1{1, {}};
  cudaSetDevice(0);
  StageRef a;
  cudaSetDevice(1);
  StageRef b;
  if (int r = round_trip(b, &s1, LONG, 1)) return r;    // device 1 has a ring
  fake::staged = 0;
  if (int r = round_trip(a, &s0, LONG, 2)) return r;    // device 0's is made while 1 is current
  REQUIRE(fake::staged >= 2 * (long)(LONG / STAGE_CHUNK));
  REQUIRE(fake::dev == 1);                              // and stays current
  cudaSetDevice(0);
  if (int r = round_trip(b, &s1, LONG, 3)) return r;
  if (int r = round_trip(a, &s0, LONG, 4)) return r;
  return 0;
}

// a ring lives as long as its holders, and no longer
int check_given_back() {
  fake::Stream s0{0, {}};
  cudaSetDevice(0);
  {
    StageRef a;
    {
      StageRef b;
      if (int r = round_trip(b, &s0, LONG, 5)) return r;
    }
    REQUIRE(!fake::pinned.empty() && fake::live_events > 0);
    const int made = fake::pin_calls;
    fake::staged = 0;
    if (int r = round_trip(a, &s0, 3 * STAGE_MIN + 5, 6)) return r;
    REQUIRE(fake::staged > 0 && fake::pin_calls == made);
  }
  REQUIRE(fake::pinned.empty() && fake::live_events == 0);
  return 0;
}

// small copies, and pinned arrays, go as they are
int check_plain() {
  fake::Stream s0{0, {}};
  cudaSetDevice(0);
  StageRef a;
  if (int r = round_trip(a, &s0, LONG, 7)) return r;
  fake::staged = fake::plain = 0;
  if (int r = round_trip(a, &s0, STAGE_MIN - 1, 8)) return r;
  REQUIRE(fake::staged == 0 && fake::plain == 2);
  return 0;
}

// an event that cannot be recorded: the error is returned and no transfer is
// left that a later copy's slot would overtake
int check_failed_record() {
  fake::Stream s0{0, {}}, s1{0, {}};
  cudaSetDevice(0);
  StageRef a;
  if (int r = round_trip(a, &s0, LONG, 9)) return r;
  const size_t n = 3 * STAGE_CHUNK;
  const Bytes x = pattern(n, 10), y = pattern(n, 11);
  for (int fail = 1; fail <= 3; ++fail) {
    Bytes dx(n), dy(n);
    fake::record_fails = fail;
    REQUIRE(a.h2d(dx.data(), x.data(), n, &s0) == cudaErrorUnknown);
    REQUIRE(a.h2d(dy.data(), y.data(), n, &s1) == cudaSuccess);   // the same slots, on another stream
    s1.drain();
    s0.drain();
    REQUIRE(dy == y);
    REQUIRE(std::memcmp(dx.data(), x.data(), fail * STAGE_CHUNK) == 0);
    fake::record_fails = fail;
    REQUIRE(a.d2h(dx.data(), y.data(), n, &s0) == cudaErrorUnknown);
    REQUIRE(a.d2h(dy.data(), x.data(), n, &s1) == cudaSuccess);
    s0.drain();
    REQUIRE(dy == x);
  }
  return 0;
}

// one long copy makes the slots it needs; shorter ones go past plainly until they
// have taken STAGE_DUE_NS, and then make no more slots than they have chunks
int check_when_made() {
  fake::Stream s0{0, {}};
  cudaSetDevice(0);
  Bytes host(STAGE_NOW), devmem(STAGE_NOW);
  auto copy = [&](StageRef& a, size_t n) { return a.h2d(devmem.data(), host.data(), n, &s0) == cudaSuccess; };
  for (int round = 0; round < 2; ++round) {   // the count begins anew with the ring's first holder
    StageRef a;
    fake::staged = fake::plain = fake::pin_calls = 0;
    const size_t n = (size_t)5 << 20;   // 5.2 ms each
    int64_t past = 0;
    for (; past < STAGE_DUE_NS; past += n) REQUIRE(copy(a, n));
    REQUIRE(fake::staged == 0 && fake::pin_calls == 0 && fake::plain == past / (int64_t)n);
    REQUIRE(copy(a, STAGE_MIN));
    REQUIRE(fake::staged == 1 && fake::pin_calls == 1);
    REQUIRE(copy(a, 2 * STAGE_CHUNK + 1));
    REQUIRE(fake::staged == 4 && fake::pin_calls == 3);
    REQUIRE(copy(a, 9 * STAGE_CHUNK));
    REQUIRE(fake::pin_calls == STAGE_SLOTS);
    s0.drain();
  }
  REQUIRE(fake::pinned.empty());
  StageRef b;
  fake::staged = fake::plain = fake::pin_calls = 0;
  REQUIRE(copy(b, STAGE_NOW));
  REQUIRE(fake::plain == 0 && fake::pin_calls == STAGE_SLOTS);
  s0.drain();
  return 0;
}
}
