// build_scratch.h -- temporary device memory of one octree build.

#ifndef SNOG_BUILD_SCRATCH_H
#define SNOG_BUILD_SCRATCH_H

#include <algorithm>

#include "device_pool.h"
#include "scene.h"

namespace snog {

// Arrays of a build on the legacy stream, given back on every exit path.  They are
// cut from a few blocks of sizes that any build asks the pool for, each twice the
// one before up to kLargest.  An array of more than half a block has one of its
// own, so that at least half of every block but the last is used: the arrays of 2M
// triangles, 556 MiB, take 1.12 times that (1.73 with blocks that double for
// ever), and those of 30M 1.04 times (1.84).
struct BuildScratch {
  static constexpr size_t kFirst = size_t(16) << 20, kLargest = size_t(64) << 20;
  std::vector<void *> p;
  char *at = nullptr;
  size_t left = 0, next = kFirst;

  BuildScratch() = default;
  BuildScratch(const BuildScratch &) = delete;
  BuildScratch &operator=(const BuildScratch &) = delete;
  ~BuildScratch() {
    // The build's stream; a failed build may still be running.
    const bool idle = cudaStreamSynchronize(nullptr) == cudaSuccess;
    if (!idle) cudaGetLastError();
    for (void *q : p) idle ? pool_put(q) : pool_free(q);
  }

  // Room for N values; throws Error.
  template <class T>
  T *get(size_t n) {
    const size_t need = ((n ? n * sizeof(T) : 16) + 255) & ~size_t(255);
    if (need > left) {
      if (need > next / 2) return static_cast<T *>(block(need));
      try {
        at = static_cast<char *>(block(next));
        left = next;
        next = std::min(2 * next, kLargest);
      } catch (const Error &e) {   // a full device may still have room for the array
        if (e.code != SNOG_ENOMEM) throw;
        return static_cast<T *>(block(need));
      }
    }
    char *q = at;
    at += need;
    left -= need;
    return reinterpret_cast<T *>(q);
  }

 private:
  void *block(size_t n) {
    p.reserve(p.size() + 1);
    p.push_back(pool_get(n));
    return p.back();
  }
};

}  // namespace snog

#endif
