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
  if (capture != cudaStreamCaptureStatusNone) {
    captured_.emplace_back();
    return captured_.back();
  }
  unsigned long long id = 0;
  check_cuda(cudaStreamGetId(st, &id), "stream");
  for (Use &u : uses_)
    if (u.stream == id) return u;
  const RelaxedCapture relaxed;
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

uint32_t *StreamUses::Call::words() const {
  if (!use_.words) {
    const RelaxedCapture relaxed;
    use_.words = uses_.new_words();
  }
  return use_.words;
}

bool StreamUses::wait() {
  bool idle = captured_.empty();
  for (Use &u : uses_) {
    const bool ok = !u.lost && cudaEventSynchronize(u.done) == cudaSuccess;
    if (!ok) cudaGetLastError();
    idle = idle && ok;
  }
  return idle;
}

void StreamUses::release(bool idle) {
  for (Use &u : uses_) cudaEventDestroy(u.done);
  uses_.clear();
  captured_.clear();
  for (void *p : blocks_) idle ? pool_put(p) : pool_free(p);
  blocks_.clear();
  at_ = nullptr;
  left_ = 0;
}

}  // namespace snog
