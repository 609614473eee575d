// Copies between the caller's host arrays and the device.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace wg {

// As cudaMemcpyAsync on `s`, for arrays of any kind. Large pageable arrays go
// through pinned buffers filled (or emptied) by several threads: the driver's
// own staging runs on one thread at 8 to 10 GB/s, page faults of a fresh
// output included, against 55 GB/s of the link. copy_to_device returns once
// `src` has been read, copy_to_host once `dst` is complete when the array is
// pageable, as cudaMemcpyAsync does; pinned arrays are copied asynchronously.
// Where no pinned buffer can be had the copy is the driver's. Errors throw
// (check_cuda).
void copy_to_device(void* dst, const void* src, size_t bytes, cudaStream_t s);
void copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t s);

// What the tests make scarce, in the calling thread
// (rang_b200_wgridder_test_limits).
struct TestLimits {
  bool no_pinned = false;  // no pinned buffer can be had
  size_t planes = 0;       // planes in a group at most (0: as many as fit)
  int fail_work = 0;       // the work-space buffer that cannot be had, counted from now (0: none)
};
TestLimits& test_limits();

// Frees the pinned buffers that no copy is using.
void release_host_buffers();

}  // namespace wg
