// device_pool.cc -- the kept device blocks behind device_pool.h.

#include "device_pool.h"

#include <cstdint>
#include <iterator>
#include <list>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "scene.h"

namespace snog {

namespace {

struct Block {
  int device;
  size_t size;
};

struct Kept {
  void *p;
  uint64_t put;   // Pool::puts when it was given back
};

struct Pool {
  std::mutex mu;
  std::map<void *, Block> blocks;                                          // every block of the pool
  std::list<Kept> kept;                                                    // those not in use, oldest first
  std::multimap<std::pair<int, size_t>, std::list<Kept>::iterator> find;   // by device and size
  size_t kept_bytes = 0;
  uint64_t puts = 0;

  // Take the block at IT out of the kept ones.
  void *take(decltype(find)::iterator it) {
    void *p = it->second->p;
    kept_bytes -= it->first.second;
    kept.erase(it->second);
    find.erase(it);
    return p;
  }

  // Keep P, of B's size.
  void keep(void *p, const Block &b) {
    kept.push_back(Kept{p, puts});
    try {
      find.insert({{b.device, b.size}, std::prev(kept.end())});
    } catch (...) {
      kept.pop_back();
      throw;
    }
    kept_bytes += b.size;
  }

  // Take the oldest kept block out of the pool.
  void *drop_oldest() {
    void *p = kept.front().p;
    const Block b = blocks.at(p);
    auto it = find.lower_bound({b.device, b.size});
    while (it->second != kept.begin()) ++it;
    take(it);
    blocks.erase(p);
    return p;
  }
};

// Kept blocks make room for others once so many blocks have been given back since:
// a scene takes some twenty, so those that scenes or batches of today's sizes use
// again and again stay, and those of sizes that no longer come go (scenes created
// after many of 300k triangles, which fill the pool: a 70k-triangle soup 5.1 -> 2.2
// ms, a terrain of 32k 3.6 -> 1.7, a soup of 6k 1.8 -> 1.15).
constexpr uint64_t kStale = 256;

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
    auto it = P.find.lower_bound({dev, size});
    if (it != P.find.end() && it->first.first == dev && it->first.second <= size + size / 4) return P.take(it);
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
  std::vector<void *> out;   // blocks to free
  {
    std::lock_guard<std::mutex> lk(P.mu);
    auto it = P.blocks.find(p);
    if (it == P.blocks.end()) return;
    const Block b = it->second;
    P.puts++;
    try {
      while (b.size <= kPoolKeep && P.kept_bytes + b.size > kPoolKeep && P.kept.front().put + kStale < P.puts) {
        out.push_back(nullptr);
        out.back() = P.drop_oldest();
      }
      if (P.kept_bytes + b.size <= kPoolKeep) {
        P.keep(p, b);
        p = nullptr;
      }
    } catch (...) {   // no room to remember it: free it
    }
    if (p) P.blocks.erase(it);
  }
  for (void *q : out) free_block(q);
  if (p) free_block(p);
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
  std::list<Kept> kept;
  {
    std::lock_guard<std::mutex> lk(P.mu);
    kept.swap(P.kept);
    P.find.clear();
    P.kept_bytes = 0;
    for (const Kept &k : kept) P.blocks.erase(k.p);
  }
  for (const Kept &k : kept) free_block(k.p);
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
