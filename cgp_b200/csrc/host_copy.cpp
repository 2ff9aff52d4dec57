#include "host_copy.h"

#include <algorithm>
#include <cstring>

#include "engine.h"

namespace cgp {

bool HostCopier::direct(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type != cudaMemoryTypeUnregistered;
}

void HostCopier::open() {
  if (ready_ != nullptr) return;
  if (ring_ == nullptr)
    ck(cudaHostAlloc(reinterpret_cast<void**>(&ring_), 2 * kThreads * kSlot, cudaHostAllocDefault),
       "cudaHostAlloc(copy slots)");
  for (int t = 0; t < kThreads; ++t) {
    Lane& l = lanes_[t];
    if (l.stream == nullptr)
      ck(cudaStreamCreateWithFlags(&l.stream, cudaStreamNonBlocking), "cudaStreamCreate");
    for (int i = 0; i < 2; ++i) {
      if (l.done[i] == nullptr)
        ck(cudaEventCreateWithFlags(&l.done[i], cudaEventDisableTiming), "cudaEventCreate");
      l.slot[i] = ring_ + (2 * t + i) * kSlot;
    }
  }
  ck(cudaEventCreateWithFlags(&ready_, cudaEventDisableTiming), "cudaEventCreate");
}

HostCopier::~HostCopier() {
  {
    std::lock_guard<std::mutex> lk(mu_);
    stop_ = true;
  }
  wake_.notify_all();
  for (std::thread& t : workers_) t.join();
  for (Lane& l : lanes_) {
    if (l.stream) {
      cudaStreamSynchronize(l.stream);
      cudaStreamDestroy(l.stream);
    }
    for (cudaEvent_t e : l.done)
      if (e) cudaEventDestroy(e);
  }
  if (ready_) cudaEventDestroy(ready_);
  if (ring_) cudaFreeHost(ring_);
}

// Lane t's chunks: t, t + threads, ...; the next transfer is in flight while
// the last one is copied out of its slot.
cudaError_t HostCopier::run(int t, int threads, const std::vector<HostSegment>& chunks) {
  Lane& l = lanes_[t];
  const size_t n = chunks.size();
  cudaError_t e = cudaSuccess;
  auto issue = [&](size_t c, int i) {
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(l.slot[i], chunks[c].src, chunks[c].bytes, cudaMemcpyDeviceToHost, l.stream);
    if (e == cudaSuccess) e = cudaEventRecord(l.done[i], l.stream);
  };
  int i = 0;
  const size_t first = static_cast<size_t>(t);
  if (first < n) issue(first, 0);
  for (size_t c = first; c < n && e == cudaSuccess; c += threads, i ^= 1) {
    if (c + threads < n) issue(c + threads, i ^ 1);
    if (e == cudaSuccess) e = cudaEventSynchronize(l.done[i]);
    if (e == cudaSuccess) std::memcpy(chunks[c].dst, l.slot[i], chunks[c].bytes);
  }
  if (e != cudaSuccess) cudaStreamSynchronize(l.stream);  // nothing left in the slots
  return e;
}

void HostCopier::work(int t) {
  const cudaError_t dev = cudaSetDevice(device_);
  uint64_t seen = 0;
  std::unique_lock<std::mutex> lk(mu_);
  for (;;) {
    wake_.wait(lk, [&] { return stop_ || job_ != seen; });
    if (stop_) return;
    seen = job_;
    if (t >= job_threads_) continue;
    const int threads = job_threads_;
    const std::vector<HostSegment>* chunks = chunks_;
    lk.unlock();
    const cudaError_t e = dev != cudaSuccess ? dev : run(t, threads, *chunks);
    lk.lock();
    lanes_[t].err = e;
    if (--busy_ == 0) idle_.notify_one();
  }
}

void HostCopier::copy(const std::vector<HostSegment>& segs, cudaStream_t s) {
  open();
  std::vector<HostSegment> chunks;
  size_t total = 0;
  for (const HostSegment& g : segs) {
    total += g.bytes;
    for (size_t b = 0; b < g.bytes; b += kSlot)
      chunks.push_back({static_cast<char*>(g.dst) + b, static_cast<const char*>(g.src) + b,
                        std::min(kSlot, g.bytes - b)});
  }
  // a lane for every 256 KB, as far as the host has cores
  const size_t cores = std::max(1u, std::thread::hardware_concurrency());
  int threads = static_cast<int>(std::max<size_t>(
      1, std::min({static_cast<size_t>(kThreads), cores, chunks.size(), total >> 18})));
  try {
    while (static_cast<int>(workers_.size()) + 1 < threads)
      workers_.emplace_back([this, t = static_cast<int>(workers_.size()) + 1] { work(t); });
  } catch (const std::exception&) {  // no more threads to be had
    threads = static_cast<int>(workers_.size()) + 1;
  }
  ck(cudaEventRecord(ready_, s), "event");
  for (int t = 0; t < threads; ++t) ck(cudaStreamWaitEvent(lanes_[t].stream, ready_, 0), "wait");
  if (threads > 1) {
    std::lock_guard<std::mutex> lk(mu_);
    chunks_ = &chunks;
    job_threads_ = threads;
    busy_ = threads - 1;
    ++job_;
  }
  if (threads > 1) wake_.notify_all();
  lanes_[0].err = run(0, threads, chunks);
  if (threads > 1) {
    std::unique_lock<std::mutex> lk(mu_);
    idle_.wait(lk, [&] { return busy_ == 0; });
  }
  for (int t = 0; t < threads; ++t) ck(lanes_[t].err, "copy out");
}

}  // namespace cgp
