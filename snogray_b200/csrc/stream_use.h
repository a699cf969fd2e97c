// stream_use.h -- the streams on which a scene's asynchronous calls run: what has
// to be waited for before its memory is used for something else, and a ray-batch
// dispenser's words for each.

#ifndef SNOG_STREAM_USE_H
#define SNOG_STREAM_USE_H

#include <cuda_runtime.h>

#include <cstdint>
#include <deque>
#include <vector>

namespace snog {

// Calls on one stream run one after the other and may share words; calls on
// different streams may run side by side and may not.  So a stream has words of
// its own until its calls have completed, and then hands them on; a call that
// is captured into a graph, which may be launched at any time, keeps words of
// its own.  Guarded by the scene's mutex.
class StreamUses {
  struct Use {
    unsigned long long stream = 0;   // the runtime's id, which is not given twice
    cudaEvent_t done = nullptr;      // after the stream's latest call; null for a captured one
    uint32_t *words = nullptr;       // allocated when first asked for
    bool lost = false;               // DONE could not be recorded: not for another stream
  };

 public:
  static constexpr uint32_t kWords = 16;   // per use: 64 bytes
  // From before a call's work is put on ST until after; throws Error.
  class Call {
    Use &use_;
    cudaStream_t st_;

    StreamUses &uses_;

   public:
    Call(StreamUses &uses, cudaStream_t st) : use_(uses.find(st)), st_(st), uses_(uses) {}
    ~Call();
    Call(const Call &) = delete;
    Call &operator=(const Call &) = delete;
    uint32_t *words() const;   // throws Error
  };
  // Wait for every call; false if one may still run: a wait failed, or a call
  // was captured.  (By the streams' events, not for the device, which may not be
  // waited for while any stream of it is captured.)
  bool wait();
  // Give the words back: to the pool if IDLE, that is if no call can be running,
  // else by freeing them.
  void release(bool idle);

 private:
  std::deque<Use> uses_, captured_;   // (references stay valid)
  std::vector<void *> blocks_;
  uint32_t *at_ = nullptr;
  size_t left_ = 0;   // words at AT_ not yet given to a use
  uint32_t *new_words();
  Use &find(cudaStream_t st);
};

// While one of these lives, the calling thread may allocate and ask for events'
// status although a stream is being captured (the calls below touch none that is).
class RelaxedCapture {
  cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;

 public:
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
  RelaxedCapture(const RelaxedCapture &) = delete;
  RelaxedCapture &operator=(const RelaxedCapture &) = delete;
};

}  // namespace snog

#endif
