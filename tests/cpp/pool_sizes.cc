// What the block pool keeps as the sizes asked for change, on the fake runtime.

#include "fake_cuda.h"

#include "../../snogray_b200/csrc/device_pool.h"

#include <vector>

using namespace snog;

constexpr size_t MiB = size_t(1) << 20;
static std::set<void *> seen;
static size_t most_kept = 0;

// Take blocks of these sizes and give them back; how many were not from the pool.
static size_t cycle(const std::vector<size_t> &mib) {
  size_t fresh = 0, bytes = 0;
  std::vector<void *> p;
  for (size_t m : mib) {
    p.push_back(pool_get(m * MiB));
    fresh += seen.insert(p.back()).second;   // (the fake gives no address twice)
    bytes += size_class(m * MiB);
  }
  most_kept = std::max(most_kept, fake::used - bytes);
  for (void *q : p) pool_put(q);
  most_kept = std::max(most_kept, fake::used);
  return fresh;
}

int main() {
  fake::capacity = size_t(8) << 30;
  const std::vector<size_t> early(8, 30), late = {20, 12, 7, 3, 1};
  cycle(early);
  fake::expect(cycle(early) == 0, "blocks of one size are kept");
  for (int k = 0; k < 60; k++) cycle(late);
  fake::expect(cycle(late) == 0, "sizes that no longer come make room");
  // More than is kept, again and again: part of it is kept all the same.
  const std::vector<size_t> many = {22, 26, 30, 34, 40, 48, 60, 72, 88};
  for (int k = 0; k < 100; k++) cycle(many);
  size_t fresh = 0;
  for (int k = 0; k < 100; k++) fresh += cycle(many);
  fake::expect(fresh <= 100 * 6, "part of what does not fit is kept");
  cycle({300});
  fake::expect(cycle(many) <= 6, "a block that could not be kept takes no other's place");
  fake::expect(most_kept <= kPoolKeep, "the bound");
  pool_trim();
  fake::expect(fake::used == 0, "everything is given back");
  return fake::failures != 0;
}
