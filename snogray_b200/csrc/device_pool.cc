// device_pool.cc -- the kept device blocks behind device_pool.h.

#include "device_pool.h"

#include <map>
#include <mutex>
#include <utility>

#include "scene.h"

namespace snog {

namespace {

struct Block {
  int device;
  size_t size;
};

struct Pool {
  std::mutex mu;
  std::map<void *, Block> blocks;                           // every block of the pool
  std::multimap<std::pair<int, size_t>, void *> kept;       // those not in use, by device and size
  size_t kept_bytes = 0;
};

// Never destroyed: blocks may be given back while the process ends.
Pool &pool() {
  static Pool *p = new Pool;
  return *p;
}

void free_block(void *p) {
  if (cudaFree(p) != cudaSuccess) cudaGetLastError();
}

}  // namespace

size_t size_class(size_t n) {
  if (n <= 4096) return 4096;
  size_t p = 1;
  while (p <= n / 2) p <<= 1;
  const size_t step = p / 8;
  return (n + step - 1) / step * step;
}

// The lock is never held over cudaMalloc or cudaFree, which may wait for the
// device's work: other threads, of other devices too, need the pool meanwhile.

void *pool_get(size_t n) {
  Pool &P = pool();
  int dev = 0;
  check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
  size_t size = size_class(n);
  {
    std::lock_guard<std::mutex> lk(P.mu);
    auto it = P.kept.lower_bound({dev, size});
    if (it != P.kept.end() && it->first.first == dev && it->first.second <= size + size / 4) {
      void *p = it->second;
      P.kept_bytes -= it->first.second;
      P.kept.erase(it);
      return p;
    }
  }
  void *p = nullptr;
  const cudaError_t e = device_malloc(&p, size);
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw Error{e == cudaErrorMemoryAllocation ? SNOG_ENOMEM : SNOG_ECUDA,
                std::string("cudaMalloc: ") + cudaGetErrorString(e)};
  }
  try {
    std::lock_guard<std::mutex> lk(P.mu);
    P.blocks[p] = Block{dev, size};
  } catch (...) {
    free_block(p);
    throw;
  }
  return p;
}

void pool_put(void *p) {
  if (!p) return;
  Pool &P = pool();
  {
    std::lock_guard<std::mutex> lk(P.mu);
    auto it = P.blocks.find(p);
    if (it == P.blocks.end()) return;
    const Block b = it->second;
    if (P.kept_bytes + b.size <= kPoolKeep) {
      try {
        P.kept.insert({{b.device, b.size}, p});
        P.kept_bytes += b.size;
        return;
      } catch (...) {   // no room to remember it: free it
      }
    }
    P.blocks.erase(it);
  }
  free_block(p);
}

void pool_free(void *p) {
  if (!p) return;
  Pool &P = pool();
  {
    std::lock_guard<std::mutex> lk(P.mu);
    P.blocks.erase(p);
  }
  free_block(p);
}

void pool_trim() {
  Pool &P = pool();
  std::multimap<std::pair<int, size_t>, void *> kept;
  {
    std::lock_guard<std::mutex> lk(P.mu);
    kept.swap(P.kept);
    P.kept_bytes = 0;
    for (auto &k : kept) P.blocks.erase(k.second);
  }
  for (auto &k : kept) free_block(k.second);
}

cudaError_t device_malloc(void **p, size_t n) {
  cudaError_t e = cudaMalloc(p, n);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    pool_trim();
    e = cudaMalloc(p, n);
  }
  return e;
}

}  // namespace snog
