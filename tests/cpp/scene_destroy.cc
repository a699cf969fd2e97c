// A scene's destruction, and a ray batch that fails, on the fake runtime: no block
// goes back to the pool while work may still be using it, and the device as a
// whole is not waited for (which a stream under capture elsewhere forbids).

#include "fake_cuda.h"

#include "../../snogray_b200/csrc/launch.h"
#include "../../snogray_b200/csrc/scene.h"

using namespace snog;

static bool launch_fails = false;
static cudaStream_t shadow_stream = nullptr;   // of the last render

namespace snog {
int stack_class_for_depth(uint32_t) { return 32; }
cudaError_t launch_trace_batch(const DevScene &, const float *, uint32_t, uint32_t, int32_t *, float *, float *,
                               unsigned long long *, uint32_t *, uint32_t *, cudaStream_t st, int *) {
  fake::put[st]++;
  return launch_fails ? cudaErrorInvalidConfiguration : cudaSuccess;
}
JobConsts make_job(const DevScene &, const SnogCamera &, const SnogRenderParams &, const SnogRenderWindow *) {
  JobConsts jc{};
  jc.W = jc.H = jc.PW = jc.PH = 8;
  jc.S = 1;
  return jc;
}
uint64_t wave_bytes_per_path(uint32_t) { return 100; }
cudaError_t wave_alloc(WaveBuffers &wb, uint64_t cap, uint32_t n_lights) {
  wb.wave_cap = cap;
  wb.n_lights = n_lights;
  return cudaSuccess;
}
cudaError_t render_job(const DevScene &, const JobConsts &, WaveBuffers &, float4 *, float *, float *, cudaStream_t st,
                       uint32_t *, uint32_t *, RenderProfile *, bool, ShadowStream *side) {
  if (!side->st) cudaStreamCreateWithFlags(&side->st, cudaStreamNonBlocking);
  shadow_stream = side->st;
  fake::put[st]++;
  if (launch_fails) fake::put[shadow_stream]++;   // not joined
  return launch_fails ? cudaErrorInvalidConfiguration : cudaSuccess;
}
RenderProfile::~RenderProfile() {}
}  // namespace snog

static cudaStream_t stream(long k) { return reinterpret_cast<cudaStream_t>(k); }

struct Scene {
  SceneImpl *impl = new SceneImpl;
  SnogScene *handle = new SnogScene{impl};
  void *block;
  explicit Scene(size_t bytes) {
    impl->on_device = true;
    block = impl->arena.alloc(bytes);
  }
  void trace(cudaStream_t st) {
    float rays[7];
    int32_t prim[1];
    fake::expect(snog_trace_device(handle, rays, 1, 1, prim, nullptr, nullptr, st) == SNOG_OK, snog_last_error());
  }
  void destroy() { fake::expect(snog_scene_destroy(handle) == SNOG_OK, snog_last_error()); }
};

// Whether BLOCK, of BYTES, went back to the pool.
static bool pooled(void *block, size_t bytes) {
  void *p = pool_get(bytes);
  const bool same = p == block;
  pool_put(p);
  return same && !fake::freed.count(block);
}

int main() {
  {
    Scene s(1 << 20);
    s.trace(stream(8));
    fake::capturing.insert(stream(16));   // another thread's
    s.destroy();
    fake::capturing.clear();
    fake::expect(fake::device_waits == 0, "the device is not waited for");
    fake::expect(fake::completed[stream(8)] == fake::put[stream(8)], "the trace is waited for");
    fake::expect(pooled(s.block, 1 << 20), "an idle scene's blocks are kept");
  }
  {
    Scene s(2 << 20);
    SnogCamera cam{};
    SnogRenderParams p{};
    p.width = p.height = 8;
    p.spp = 1;
    float out[3];
    fake::expect(snog_render_device(s.handle, &cam, &p, out, stream(24), nullptr) == SNOG_OK, snog_last_error());
    s.destroy();
    fake::expect(fake::completed[stream(24)] == fake::put[stream(24)] || fake::freed.count(s.block),
                 "a render is waited for");
  }
  {   // a render that fails half-way
    Scene s(7 << 20);
    SnogCamera cam{};
    SnogRenderParams p{};
    p.width = p.height = 8;
    p.spp = 1;
    float out[3];
    launch_fails = true;
    fake::expect(snog_render_device(s.handle, &cam, &p, out, stream(32), nullptr) == SNOG_ECUDA, "render error");
    launch_fails = false;
    fake::expect(fake::completed[shadow_stream] == fake::put[shadow_stream], "its shadow rays are waited for");
    fake::expect(fake::completed[stream(32)] == fake::put[stream(32)], "and the others");
    s.destroy();
  }
  {
    Scene s(3 << 20);
    s.trace(stream(8));
    fake::waits_fail = true;
    s.destroy();
    fake::waits_fail = false;
    fake::expect(fake::freed.count(s.block), "blocks are freed where the wait failed");
    fake::expect(!pooled(s.block, 3 << 20), "blocks are not kept where the wait failed");
  }
  {
    Scene s(4 << 20);
    fake::capturing.insert(stream(8));
    s.trace(stream(8));
    fake::capturing.clear();   // the graph may be running
    s.destroy();
    fake::expect(fake::freed.count(s.block), "blocks are freed where a call was captured");
  }
  {
    Scene s(5 << 20);
    fake::waits_fail = true;
    launch_fails = true;
    float rays[7] = {};
    int32_t prim[1];
    fake::freed.clear();
    fake::expect(snog_trace(s.handle, rays, 1, 1, prim, nullptr, nullptr, nullptr) == SNOG_ECUDA, "launch error");
    fake::waits_fail = launch_fails = false;
    fake::expect(fake::freed.size() == 5, "a failed batch's buffers are freed");
    s.destroy();
  }
  {   // in an engine's table
    Scene s(6 << 20);
    ++*s.impl->engines;
    s.destroy();
    fake::expect(fake::freed.count(s.block), "blocks are freed where an engine may be running");
  }
  return fake::failures != 0;
}
