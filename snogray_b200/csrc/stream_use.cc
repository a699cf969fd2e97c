// stream_use.cc -- see stream_use.h.

#include "stream_use.h"

#include "scene.h"

namespace snog {

uint32_t *StreamUses::new_words() {
  if (left_ < kWords) {
    constexpr size_t kBlock = 4096;
    blocks_.reserve(blocks_.size() + 1);
    at_ = static_cast<uint32_t *>(pool_get(kBlock));
    blocks_.push_back(at_);
    left_ = kBlock / 4;
  }
  uint32_t *w = at_;
  at_ += kWords;
  left_ -= kWords;
  return w;
}

StreamUses::Use &StreamUses::find(cudaStream_t st) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  check_cuda(cudaStreamIsCapturing(st, &capture), "stream");
  const RelaxedCapture relaxed;
  if (capture != cudaStreamCaptureStatusNone) {
    Use u;
    u.words = new_words();
    captured_.push_back(u);
    return captured_.back();
  }
  unsigned long long id = 0;
  check_cuda(cudaStreamGetId(st, &id), "stream");
  for (Use &u : uses_)
    if (u.stream == id) return u;
  for (Use &u : uses_) {
    if (u.lost) continue;
    if (cudaEventQuery(u.done) == cudaSuccess) {
      u.stream = id;
      return u;
    }
    cudaGetLastError();   // not ready
  }
  Use u;
  u.stream = id;
  u.words = new_words();
  check_cuda(cudaEventCreateWithFlags(&u.done, cudaEventDisableTiming), "event");
  uses_.push_back(u);
  return uses_.back();
}

StreamUses::Call::~Call() {
  if (use_.done && cudaEventRecord(use_.done, st_) != cudaSuccess) {
    cudaGetLastError();
    use_.lost = true;
  }
}

void StreamUses::release() {
  for (Use &u : uses_) cudaEventDestroy(u.done);
  uses_.clear();
  captured_.clear();
  for (void *p : blocks_) pool_put(p);
  blocks_.clear();
  at_ = nullptr;
  left_ = 0;
}

}  // namespace snog
