// The temporary memory of octree builds, on the fake runtime: what is held against
// what is used, up to a device that has no more.

#include "fake_cuda.h"

#include "../../snogray_b200/csrc/build_scratch.h"

#include <random>

using namespace snog;

constexpr size_t MiB = size_t(1) << 20;

// Bytes of the arrays of a build of N triangles with P = 3 N / 2 placements, U list
// heads and M nodes (octree_gpu.cu).
static std::vector<size_t> arrays(size_t n) {
  const size_t p = 3 * n / 2, u = p * 3 / 5, m = p * 4 / 5;
  return {24 * n, 4 * n, 36 * n, 12 * n, 4 * n, 4 * n, 24 * n, 0,     4,     640,   8,     4 * n, 4 * n, 8 * p, 8 * p,
          4 * p,  4 * p, 4 * p,  4 * p,  8 * p, 8 * p, p / 20, p / 20, 4 * p, 4 * p, 4 * u, 4 * u, 4 * u, 8 * m, 8 * m,
          4 * m,  4 * u, 4 * m,  4 * m,  4 * m, 4 * m, m / 20, 8 * m, 8 * m, 164,   4 * m, 4 * m, 4 * m};
}

static size_t get_all(BuildScratch &s, const std::vector<size_t> &bytes) {
  size_t sum = 0;
  std::vector<std::pair<char *, size_t>> got;
  for (size_t b : bytes) {
    char *at = s.get<char>(b);
    fake::expect(reinterpret_cast<size_t>(at) % 256 == 0, "alignment");
    for (auto &g : got) fake::expect(at + b <= g.first || g.first + g.second <= at, "arrays apart");
    got.push_back({at, b});
    sum += (std::max(b, size_t(16)) + 255) & ~size_t(255);
  }
  return sum;
}

int main() {
  fake::capacity = size_t(64) << 30;
  // A pool block is up to a ninth larger than asked for, and of the blocks that
  // several arrays share at least half is used.
  for (size_t n : {size_t(4096), size_t(20000), size_t(200000), size_t(600000), size_t(2000000), size_t(4000000)}) {
    pool_trim();
    const size_t before = fake::used;
    BuildScratch s;
    const size_t sum = get_all(s, arrays(n));
    const size_t held = fake::used - before;
    fake::expect(held <= sum * 9 / 4 + 16 * MiB, "bound");
    if (n >= 2000000) fake::expect(held <= sum * 5 / 4, "a large build holds what it uses");
  }
  std::mt19937 rng(1);
  for (int k = 0; k < 50; k++) {
    pool_trim();
    const size_t before = fake::used;
    std::vector<size_t> bytes(rng() % 60);
    for (size_t &b : bytes) b = size_t(1) << (rng() % 27), b += rng() % b;
    BuildScratch s;
    const size_t sum = get_all(s, bytes);
    fake::expect(fake::used - before <= sum * 9 / 4 + 16 * MiB, "bound of any sequence");
  }
  pool_trim();
  fake::expect(fake::used == 0, "everything was given back");
  {   // a device with a quarter more than the arrays
    std::vector<size_t> bytes = arrays(2000000);
    size_t sum = 0;
    for (size_t b : bytes) sum += b;
    fake::capacity = sum * 5 / 4;
    BuildScratch s;
    try {
      get_all(s, bytes);
    } catch (const Error &) {
      fake::expect(false, "a build that fits is refused");
    }
  }
  pool_trim();
  {   // no room for a shared block, but for the array
    fake::capacity = 8 * MiB;
    BuildScratch s;
    try {
      s.get<char>(5 * MiB);
    } catch (const Error &) {
      fake::expect(false, "an array that fits is refused");
    }
    int code = 0;
    try {
      s.get<char>(5 * MiB);
    } catch (const Error &e) {
      code = e.code;
    }
    fake::expect(code == SNOG_ENOMEM, "an array that does not fit is refused");
  }
  return fake::failures != 0;
}
