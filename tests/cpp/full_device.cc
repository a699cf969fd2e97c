// Allocations on a full device, on the fake runtime: blocks that the pool keeps do
// not stand in the way of a render's or of one another.

#include "fake_cuda.h"

#include "../../snogray_b200/csrc/launch.h"
#include "../../snogray_b200/csrc/scene.h"

#include <chrono>
#include <future>

using namespace snog;

namespace snog {
int stack_class_for_depth(uint32_t) { return 32; }
JobConsts make_job(const DevScene &, const SnogCamera &, const SnogRenderParams &p, const SnogRenderWindow *) {
  JobConsts jc{};
  jc.W = p.width;
  jc.H = p.height;
  jc.PW = jc.PH = 8;
  jc.S = 1;
  return jc;
}
uint64_t wave_bytes_per_path(uint32_t) { return 100; }
cudaError_t wave_alloc(WaveBuffers &wb, uint64_t cap, uint32_t n_lights) {
  wb.wave_cap = cap;
  wb.n_lights = n_lights;
  return cudaSuccess;
}
cudaError_t render_job(const DevScene &, const JobConsts &, WaveBuffers &, float4 *, float *, float *, cudaStream_t,
                       uint32_t *, uint32_t *, RenderProfile *, bool, ShadowStream *) {
  return cudaSuccess;
}
RenderProfile::~RenderProfile() {}
}  // namespace snog

static std::vector<std::future<void>> detached;   // (joined at the end)
constexpr size_t MiB = size_t(1) << 20;

int main() {
  SceneImpl *impl = new SceneImpl;
  impl->on_device = true;
  SnogScene *scene = new SnogScene{impl};
  // 36 MiB of image buffers on a device of 230 MiB with 200 kept.
  fake::capacity = 230 * MiB;
  pool_put(pool_get(200 * MiB));
  SnogCamera cam{};
  SnogRenderParams p{};
  p.width = p.height = 1024;
  p.spp = 1;
  float out[3];
  fake::expect(snog_render_device(scene, &cam, &p, out, nullptr, nullptr) == SNOG_OK, snog_last_error());
  fake::expect(fake::used < 100 * MiB, "the kept block was freed");
  // Other threads use the pool while a block is being freed.
  void *small = pool_get(1 * MiB);
  pool_put(pool_get(3 * MiB));
  pool_put(pool_get(30 * MiB));
  auto others_run = [&](const char *what, auto act) {
    bool asked = false;
    fake::on_free = [&] {
      if (asked) return;
      asked = true;
      auto other = std::async(std::launch::async, [&] {
        pool_put(small);
        small = pool_get(1 * MiB);
      });
      fake::expect(other.wait_for(std::chrono::seconds(2)) == std::future_status::ready, what);
      detached.push_back(std::move(other));
    };
    act();
    fake::on_free = nullptr;
    fake::expect(asked, "something was freed");
  };
  others_run("the pool is free while it is trimmed", [] { pool_trim(); });
  fake::capacity = 2048 * MiB;
  void *large = pool_get(300 * MiB);   // more than is kept
  others_run("the pool is free while a block is freed", [&] { pool_put(large); });
  return fake::failures != 0;
}
