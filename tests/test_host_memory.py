"""Device memory of scene creation, on a fake CUDA runtime (tests/cpp/fake_cuda.h)."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
CSRC = os.path.join(os.path.dirname(HERE), "snogray_b200", "csrc")


@pytest.mark.parametrize("name", ["build_scratch", "scene_build", "pool_sizes"])
def test_host_memory(name, tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / name)
    sources = [os.path.join(CSRC, f) for f in ("capi.cc", "device_pool.cc", "octree_build.cc", "scene.cc",
                                               "stream_use.cc")]
    # Functions of the other sources are not called.
    subprocess.run([gxx, "-std=c++17", "-O1", "-g", "-no-pie", f"-I{CUDA_INC}",
                    os.path.join(HERE, "cpp", name + ".cc"), *sources,
                    "-Wl,--unresolved-symbols=ignore-all", "-lpthread", "-o", exe], check=True, capture_output=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stderr
