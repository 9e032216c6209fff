// gdf_stage.h -- copies between host arrays and the device.
//
// A caller's arrays are ordinary (pageable) memory as a rule. The driver copies
// those through its own staging buffer with one host thread, 12 GB/s from memory,
// 20 from the host's caches, 2-3 into pages not yet touched, well under the link.
// h2d / d2h take large pageable arrays through a ring of pinned buffers instead:
// several threads fill (empty) one while the link moves another. Small arrays, and
// memory that is already pinned or on a device, go to cudaMemcpyAsync as they are.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace gdf {

// Copies through the ring of the device that is current where it is made, and
// keeps that ring for as long as it lives: the ring (STAGE_SLOTS x STAGE_CHUNK
// bytes at most, made slot by slot) is freed with the last of its holders.
// Every handle holds one, made with the handle's stream; the streams given to
// h2d and d2h are that device's. Which device is current at a copy does not matter,
// as it does not to cudaMemcpyAsync.
struct StageRef {
  StageRef();
  ~StageRef();
  StageRef(const StageRef&) = delete;
  StageRef& operator=(const StageRef&) = delete;

  // host -> device, ordered on st; src may be reused on return
  cudaError_t h2d(void* dst, const void* src, size_t bytes, cudaStream_t st);
  // device -> host after st's earlier work; a pageable dst of STAGE_MIN bytes or
  // more is complete on return
  cudaError_t d2h(void* dst, const void* src, size_t bytes, cudaStream_t st);

 private:
  int dev;
};

constexpr size_t STAGE_CHUNK = (size_t)4 << 20;
constexpr int STAGE_SLOTS = 4;
constexpr size_t STAGE_MIN = (size_t)1 << 20;   // below: one plain copy (the ring's hand-overs cost more)
// When a copy makes the slots it needs (2.3 ms for all four, 0.5 ms to give them
// back): if it is this long itself, so that it saves as much (72 MB up 5.6 ms
// plainly, 1.6 through the ring; 256 MB 23 and 5.2): the first predict of a process
// on 69 MB takes 9.2 ms, 8.9 without the ring, the next ones 4.3 and 7 to 8 ...
constexpr size_t STAGE_NOW = (size_t)64 << 20;
// ... or if the copies of 1 MiB or more that went past plainly while its holders
// lived took this long, ten times what the slots cost. A shorter copy may then pay
// for the slots alone, once (predict on 62 MB: the seventh call 7.0 ms, 6.6 before
// it, 3.0 after), and handles opened, loaded and closed in a loop lose a tenth of
// their copies' time at most (none where they take less than this). It is a time
// because the rate varies by ten with where the pages are: a 512^2 state goes up in
// 12 ms and comes down into new arrays in 40 (17 through the ring that these make).
constexpr int64_t STAGE_DUE_NS = 28000000;

// memcpy over several threads (gdf_io.cpp)
void par_memcpy(void* dst, const void* src, size_t bytes);
// zeros over several threads (gdf_io.cpp)
void par_zero(void* dst, size_t bytes);
// whether any of n 64-bit words has a bit besides the sign set, over several
// threads (gdf_io.cpp)
bool par_any_nonzero(const void* words, size_t n);

}  // namespace gdf
