// Device-to-host copies into pageable memory.
//
// cudaMemcpy into pageable memory goes through the driver's own bounce buffer
// with one thread that also takes the destination's page faults: 2 to 3 GB/s
// into a freshly allocated array.  Here a few threads each copy chunks through
// two pinned slots of their own, so the faults and the copies out of the slots
// run in parallel and overlap the transfers (R-MAT 18, 90 k-hop queries, 94 MB
// into a new array: 47 -> 6.8 ms for the whole call).
#pragma once

#include <cuda_runtime.h>

#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <thread>
#include <vector>

namespace cgp {

struct HostSegment {
  void* dst;        // host
  const void* src;  // device
  size_t bytes;
};

// One copy at a time (the graph hands copiers out, see GraphImpl).
class HostCopier {
 public:
  explicit HostCopier(int device) : device_(device) {}
  ~HostCopier();
  HostCopier(const HostCopier&) = delete;
  HostCopier& operator=(const HostCopier&) = delete;

  // True when `p` is memory a transfer can be made into as it is (pinned or
  // registered): such copies need no staging.
  static bool direct(const void* p);

  // Copies every segment once the work now in `s` is done, and returns when
  // the bytes are in place.
  void copy(const std::vector<HostSegment>& segs, cudaStream_t s);

 private:
  static constexpr int kThreads = 8;  // the caller and up to 7 workers
  static constexpr size_t kSlot = 512 << 10;

  struct Lane {  // one thread's stream, slots and events
    cudaStream_t stream = nullptr;
    cudaEvent_t done[2] = {nullptr, nullptr};
    char* slot[2] = {nullptr, nullptr};
    cudaError_t err = cudaSuccess;
  };

  void open();
  void work(int t);
  cudaError_t run(int t, int threads, const std::vector<HostSegment>& chunks);

  int device_;
  char* ring_ = nullptr;
  cudaEvent_t ready_ = nullptr;
  Lane lanes_[kThreads];

  std::vector<std::thread> workers_;  // workers_[i] is lane i + 1; started when first needed
  std::mutex mu_;
  std::condition_variable wake_, idle_;
  uint64_t job_ = 0;  // number of the current job
  int job_threads_ = 0;
  int busy_ = 0;      // workers not done with it
  const std::vector<HostSegment>* chunks_ = nullptr;
  bool stop_ = false;
};

}  // namespace cgp
