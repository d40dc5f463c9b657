// hostcopy.h -- copies between the caller's host arrays and the device.
//
// Arrays that arrive from a file reader or numpy are pageable: the driver
// copies them through one small page-locked buffer on one core, and the first
// touch of a result array faults its pages one by one.  Here arrays of some MB
// and up go through page-locked pieces filled (or emptied) by several threads
// while the previous pieces travel.  Page-locked arrays are copied directly.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <thread>

namespace dsgdpp {

// Enqueues the copy on `st` of `device`.  Host-to-device: the source has been
// read when the call returns, unless it is page-locked (then, as with
// cudaMemcpyAsync, when the stream gets there).  Device-to-host: a pageable
// destination is complete when the call returns.
cudaError_t copy_to_device(void* dst, const void* src, size_t bytes, int device, cudaStream_t st);
cudaError_t copy_to_host(void* dst, const void* src, size_t bytes, int device, cudaStream_t st);

// copy_to_device on a thread of its own; join() returns its status.
class BackgroundCopy {
 public:
  BackgroundCopy() = default;
  BackgroundCopy(const BackgroundCopy&) = delete;
  BackgroundCopy& operator=(const BackgroundCopy&) = delete;
  ~BackgroundCopy() { join(); }
  void start(void* dst, const void* src, size_t bytes, int device, cudaStream_t st);
  cudaError_t join();

 private:
  std::thread thread_;
  cudaError_t status_ = cudaSuccess;
};

// The page-locked pieces are shared by all copies of the process (at most 32
// MB) and freed when the last holder is gone; contexts and batches hold them
// while they live.
void hostcopy_hold();
void hostcopy_drop();

}  // namespace dsgdpp

// Bytes that have gone through pieces so far in this process, either way (for tests).
extern "C" uint64_t dsgdpp_staged_bytes();
