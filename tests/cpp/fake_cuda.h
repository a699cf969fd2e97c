// fake_cuda.h -- the CUDA runtime calls of the host code, made by the tests: device
// memory is host memory, work on a stream is pending until the test completes
// it, and calls can be made to fail.  Compiled into the test program with the host
// sources under test; nothing here runs on a GPU.

#ifndef FAKE_CUDA_H
#define FAKE_CUDA_H

#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <functional>
#include <map>
#include <mutex>
#include <set>

namespace fake {

struct Event {
  cudaStream_t stream = nullptr;
  long at = 0;   // work put on the stream before the event's record
};
inline std::map<cudaStream_t, long> put, completed;   // work per stream
inline std::set<cudaStream_t> capturing;
inline std::map<void *, size_t> memory;                // allocated blocks
inline size_t capacity = size_t(1) << 30, used = 0;
inline std::set<void *> freed;
inline bool waits_fail = false;      // every kind of wait for the device's work
inline int device_waits = 0;         // cudaDeviceSynchronize calls
inline cudaError_t last = cudaSuccess;
inline cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;
inline std::function<void()> on_free;
inline std::function<void(cudaMemcpyKind)> on_copy;   // cudaMemcpy
inline std::mutex mu;

inline cudaError_t result(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
inline void complete(cudaStream_t st) { completed[st] = put[st]; }
inline bool done(const Event &e) { return completed[e.stream] >= e.at; }

inline int failures = 0;
inline void expect(bool ok, const char *what) {
  if (!ok) {
    std::fprintf(stderr, "FAILED: %s\n", what);
    failures++;
  }
}

}  // namespace fake

extern "C" {

cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = fake::last; fake::last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }

cudaError_t cudaMalloc(void **p, size_t n) {
  std::lock_guard<std::mutex> lk(fake::mu);
  if (fake::used + n > fake::capacity) return fake::result(cudaErrorMemoryAllocation);
  *p = std::aligned_alloc(256, (n + 255) & ~size_t(255));
  fake::memory[*p] = n;
  fake::freed.erase(*p);
  fake::used += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (!p) return cudaSuccess;
  if (fake::on_free) fake::on_free();
  std::lock_guard<std::mutex> lk(fake::mu);
  auto it = fake::memory.find(p);
  if (it == fake::memory.end()) return fake::result(cudaErrorInvalidValue);
  fake::used -= it->second;
  fake::memory.erase(it);
  fake::freed.insert(p);   // the host memory stays: an address is not given twice
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t st) { fake::put[st]++; return cudaSuccess; }
cudaError_t cudaMemset(void *, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemcpy(void *, const void *, size_t, cudaMemcpyKind kind) {
  if (fake::on_copy) fake::on_copy(kind);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t st) {
  fake::put[st]++;
  return cudaSuccess;
}

cudaError_t cudaDeviceSynchronize() {
  fake::device_waits++;
  if (fake::waits_fail || !fake::capturing.empty()) return fake::result(cudaErrorStreamCaptureUnsupported);
  for (auto &s : fake::put) fake::completed[s.first] = s.second;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
  if (fake::waits_fail || fake::capturing.count(st)) return fake::result(cudaErrorStreamCaptureUnsupported);
  fake::complete(st);
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t st, cudaStreamCaptureStatus *s) {
  *s = fake::capturing.count(st) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamGetId(cudaStream_t st, unsigned long long *id) {
  *id = reinterpret_cast<unsigned long long>(st);
  return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *m) {
  std::swap(*m, fake::mode);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(new fake::Event);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete reinterpret_cast<fake::Event *>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
  *reinterpret_cast<fake::Event *>(e) = fake::Event{st, fake::put[st]};
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
  return fake::done(*reinterpret_cast<fake::Event *>(e)) ? cudaSuccess : fake::result(cudaErrorNotReady);
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  if (fake::waits_fail) return fake::result(cudaErrorStreamCaptureUnsupported);
  fake::Event &ev = *reinterpret_cast<fake::Event *>(e);
  if (fake::completed[ev.stream] < ev.at) fake::completed[ev.stream] = ev.at;
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  static long next = 1000;
  *s = reinterpret_cast<cudaStream_t>(next += 8);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  *f = fake::capacity - fake::used;
  *t = fake::capacity;
  return cudaSuccess;
}

}  // extern "C"

#endif
