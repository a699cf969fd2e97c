// Ray batches of one scene on several streams, on the fake runtime: whether two
// launches that may run side by side are given the same dispenser words.

#include "fake_cuda.h"

#include "../../snogray_b200/csrc/launch.h"
#include "../../snogray_b200/csrc/scene.h"

using namespace snog;

struct Launch {
  cudaStream_t stream;
  long at;         // position on the stream
  bool captured;   // launched again at any time
  uint32_t *words;
};
static std::vector<Launch> launches;

namespace snog {
int stack_class_for_depth(uint32_t) { return 32; }
cudaError_t launch_trace_batch(const DevScene &, const float *, uint32_t, uint32_t, int32_t *, float *, float *,
                               unsigned long long *, uint32_t *err, uint32_t *fetch, cudaStream_t st, int *) {
  fake::expect(err != fetch, "error word apart from the counter");
  const bool captured = fake::capturing.count(st);
  for (const Launch &l : launches) {
    if (l.words != fetch) continue;
    const bool over = !l.captured && (l.stream == st ? !captured : fake::completed[l.stream] >= l.at);
    fake::expect(over, "words shared with a launch that may run beside this one");
  }
  launches.push_back({st, ++fake::put[st], captured, fetch});
  return cudaSuccess;
}
}  // namespace snog

static cudaStream_t stream(long k) { return reinterpret_cast<cudaStream_t>(k); }

int main() {
  SceneImpl *impl = new SceneImpl;
  impl->on_device = true;
  SnogScene *scene = new SnogScene{impl};
  float rays[7];
  int32_t prim[1];
  auto trace = [&](cudaStream_t st) {
    fake::expect(snog_trace_device(scene, rays, 1, 1, prim, nullptr, nullptr, st) == SNOG_OK, snog_last_error());
  };
  for (int round = 0; round < 3; round++)
    for (long k = 0; k < 5; k++) trace(stream(8 * k));   // the default stream among them
  const size_t held = fake::used;
  for (long k = 0; k < 5; k++) fake::complete(stream(8 * k));
  for (int round = 0; round < 200; round++) {            // streams that come and go
    trace(stream(100 + 8 * round));
    fake::complete(stream(100 + 8 * round));
  }
  fake::expect(fake::used == held, "words of completed calls are used again");
  fake::capturing.insert(stream(64));
  for (int k = 0; k < 100; k++) trace(stream(64));       // branches of graphs
  fake::capturing.clear();
  for (long k = 0; k < 9; k++) trace(stream(8 * k));
  fake::expect(fake::mode == cudaStreamCaptureModeGlobal, "the thread's capture mode is put back");
  for (long k = 0; k < 9; k++) fake::complete(stream(8 * k));
  fake::expect(snog_scene_destroy(scene) == SNOG_OK, "destroy");
  return fake::failures != 0;
}
