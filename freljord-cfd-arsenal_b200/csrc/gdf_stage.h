// gdf_stage.h -- copies between host arrays and the device.
//
// A caller's arrays are ordinary (pageable) memory as a rule. The driver copies
// those through its own staging buffer with one host thread, 12 GB/s here (less
// into pages not yet touched), well under the link. h2d / d2h take large
// pageable arrays through a ring of pinned buffers instead: several threads fill
// (empty) one while the link moves another. Small arrays, and memory that is
// already pinned or on a device, go to cudaMemcpyAsync as they are.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace gdf {

// Copies through the ring of the device that is current where it is made, and
// keeps that ring for as long as it lives: the ring (STAGE_SLOTS x STAGE_CHUNK
// bytes, made after STAGE_MAKE bytes) is freed with the last of its holders.
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
// The ring is made once its holders have asked it for this much: making and
// freeing it takes some 18 ms, what it saves on about this many bytes, and a
// handle that is made, copied from once and closed would pay that each time.
constexpr size_t STAGE_MAKE = (size_t)64 << 20;

// memcpy over several threads (gdf_io.cpp)
void par_memcpy(void* dst, const void* src, size_t bytes);
// zeros over several threads (gdf_io.cpp)
void par_zero(void* dst, size_t bytes);
// whether any of n 64-bit words has a bit besides the sign set, over several
// threads (gdf_io.cpp)
bool par_any_nonzero(const void* words, size_t n);

}  // namespace gdf
