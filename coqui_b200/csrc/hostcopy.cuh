// Copies between device memory and ordinary (pageable) host memory.
//
// The driver's own path stages a pageable copy through one thread: measured 11 GB/s to the
// device and 5 GB/s into a freshly allocated numpy array, whose pages are faulted in by the same
// thread.  Here a few threads share the bytes, each with two page-locked 1 MB buffers: one
// buffer crosses the bus while the thread moves (and faults in) the other's bytes.
#pragma once

#include "common.cuh"

namespace cq {

bool host_is_pinned(const void* p);

// Stream-ordered copies.  Page-locked, managed or device memory: as cudaMemcpyAsync.  Ordinary
// (pageable) memory: to_device returns once the source has been read (it may be reused),
// from_device once the destination is complete.
void copy_to_device(void* dst, const void* src, size_t bytes, cudaStream_t s);
void copy_from_device(void* dst, const void* src, size_t bytes, cudaStream_t s);

// The page-locked buffers are kept between calls while at least one user (a context; the molecule
// batch and the network copy through the driver) lives, at most kMaxStageSets sets per process, and
// freed with the last user.
struct StageUser {
  StageUser();
  ~StageUser();
  StageUser(const StageUser&) = delete;
  StageUser& operator=(const StageUser&) = delete;
};

}  // namespace cq
