// A scene's creation on the fake runtime, where the device has no room for the
// device builder's temporaries, and as its uploads complete.

#include "fake_cuda.h"

#include "../../snogray_b200/csrc/launch.h"
#include "../../snogray_b200/csrc/octree_gpu.h"
#include "../../snogray_b200/csrc/scene.h"

#include <random>

using namespace snog;

static int device_builds = 0, device_error = SNOG_ENOMEM;
static bool probe_fails = false;

namespace snog {
int stack_class_for_depth(uint32_t) { return 32; }
uint32_t probe_pair_lists(const DevScene &) {
  if (probe_fails) throw Error{SNOG_ECUDA, "list probe"};
  return 0;
}
cudaError_t build_list_records(const uint32_t *, uint32_t, const float4 *, float4 *, cudaStream_t) {
  return cudaSuccess;
}
void build_octree_device(const MeshArrays &, const std::vector<Box3> &, const std::vector<uint32_t> &, float4 *,
                         DeviceArena &, DeviceOctree &) {
  device_builds++;
  throw Error{device_error, "device builder"};
}
}  // namespace snog

int main() {
  fake::capacity = size_t(1) << 30;
  const uint32_t n = 5000;
  std::vector<float> v;
  std::vector<uint32_t> t, m(n, 0);
  std::mt19937 rng(1);
  std::uniform_real_distribution<float> at(0.f, 1.f), edge(-0.02f, 0.02f);
  for (uint32_t i = 0; i < n; i++) {
    const float p[3] = {at(rng), at(rng), at(rng)};
    for (int c = 0; c < 3; c++) {
      t.push_back(uint32_t(v.size() / 3));
      for (int k = 0; k < 3; k++) v.push_back(p[k] + edge(rng));
    }
  }
  SnogMaterial mat{};
  SnogSceneDesc d{};
  d.vertices = v.data();
  d.n_vertices = uint32_t(v.size() / 3);
  d.triangles = t.data();
  d.tri_material = m.data();
  d.n_triangles = n;
  d.materials = &mat;
  d.n_materials = 1;
  for (int error : {SNOG_ENOMEM, SNOG_EINVAL}) {
    device_error = error;
    SnogScene *s = nullptr;
    device_builds = 0;
    fake::expect(snog_scene_create(&d, &s) == SNOG_OK, snog_last_error());
    fake::expect(device_builds == 1, "the device builder is tried");
    if (!s) continue;
    fake::expect(!s->impl->oct_device && s->impl->info.n_list_surfaces >= n, "the host's tree is taken");
    fake::expect(snog_scene_destroy(s) == SNOG_OK, snog_last_error());
  }
  // Asked for by name it is not replaced, and other errors are passed on.
  SnogScene *s = nullptr;
  device_error = SNOG_ENOMEM;
  fake::expect(snog_scene_create_ex(&d, SNOG_OCTREE_DEVICE, &s) == SNOG_ENOMEM && !s, "DEVICE mode");
  device_error = SNOG_ECUDA;
  fake::expect(snog_scene_create(&d, &s) == SNOG_ECUDA && !s, "other errors");
  // A copy from pageable memory may return before it has reached the device.
  fake::on_copy = [](cudaMemcpyKind kind) {
    fake::put[nullptr]++;
    if (kind == cudaMemcpyDeviceToHost) fake::complete(nullptr);
  };
  for (uint32_t mode : {SNOG_OCTREE_HOST | SNOG_LISTS_SINGLE, SNOG_OCTREE_HOST | SNOG_LISTS_PAIRED}) {
    fake::expect(snog_scene_create_ex(&d, mode, &s) == SNOG_OK, snog_last_error());
    fake::expect(fake::completed[nullptr] == fake::put[nullptr], "a new scene's uploads are complete");
    fake::expect(snog_scene_destroy(s) == SNOG_OK, snog_last_error());
  }
  fake::on_copy = nullptr;
  pool_trim();
  const size_t before = fake::used;
  probe_fails = true;
  s = nullptr;
  fake::expect(snog_scene_create_ex(&d, SNOG_OCTREE_HOST, &s) == SNOG_ECUDA && !s, "a probe that fails");
  pool_trim();
  fake::expect(fake::used == before, "its scene's memory is given back");
  return fake::failures != 0;
}
