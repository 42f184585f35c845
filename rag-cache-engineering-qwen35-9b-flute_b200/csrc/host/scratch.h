// Device scratch of the native host layer: one buffer per (kind, device, stream), grown on demand.
//
// A buffer serves the launches of one stream, which are ordered. It is allocated while that stream
// is current, so when it is replaced or evicted the caching allocator hands its memory only to later
// work of the same stream. Launches under stream capture get a buffer of the capture's own, filled
// inside the graph: a replayed graph never shares tickets with eager launches or another graph.
#pragma once

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>

#include <list>
#include <mutex>

namespace b200host {

enum class Scratch : int { kSplit = 0, kTwoStream = 1 };   // zero-filled tickets first / plain fp32 sums

class ScratchPool {
 public:
  // A buffer of at least `bytes` bytes for `stream` (the current stream of `device`).
  at::Tensor get(Scratch kind, int device, cudaStream_t stream, size_t bytes) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long capture = 0;
    if (cudaStreamGetCaptureInfo(stream, &status, &capture) != cudaSuccess) (void)cudaGetLastError();
    if (status != cudaStreamCaptureStatusActive) capture = 0;
    std::lock_guard<std::mutex> lock(mu_);
    for (auto it = entries_.begin(); it != entries_.end(); ++it) {
      if (it->kind != kind || it->device != device || it->stream != stream || (it->capture != 0) != (capture != 0)) continue;
      if (it->capture == capture && size_t(it->buf.numel()) >= bytes) {
        entries_.splice(entries_.begin(), entries_, it);
        return entries_.front().buf;
      }
      if (it->capture == capture && bytes < 2 * size_t(it->buf.numel())) bytes = 2 * size_t(it->buf.numel());
      entries_.erase(it);
      break;
    }
    const auto opts = at::TensorOptions().dtype(at::kByte).device(at::kCUDA, device);
    at::Tensor buf = kind == Scratch::kSplit ? at::zeros({int64_t(bytes)}, opts) : at::empty({int64_t(bytes)}, opts);
    entries_.push_front(Entry{kind, device, stream, capture, buf});
    if (entries_.size() > kMaxEntries) entries_.pop_back();      // least recently used
    return buf;
  }

  std::mutex& two_stream_launches() { return two_stream_; }

 private:
  static constexpr size_t kMaxEntries = 32;
  struct Entry {
    Scratch kind;
    int device;
    cudaStream_t stream;
    unsigned long long capture;
    at::Tensor buf;
  };
  std::mutex mu_, two_stream_;
  std::list<Entry> entries_;
};

inline ScratchPool& scratch_pool() {
  static ScratchPool* pool = new ScratchPool();   // outlives the CUDA context: never destroyed
  return *pool;
}

}  // namespace b200host
