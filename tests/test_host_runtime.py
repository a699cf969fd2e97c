"""Host code of the library on a fake CUDA runtime (tests/cpp/fake_cuda.h): the
order of events that no test on a GPU can bring about at will."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
CSRC = os.path.join(ROOT, "snogray_b200", "csrc")


@pytest.mark.parametrize("name", ["trace_streams", "scene_destroy", "full_device"])
def test_host_code(name, tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / name)
    sources = [os.path.join(CSRC, f) for f in ("capi.cc", "device_pool.cc", "scene.cc", "stream_use.cc")]
    # Functions of the other sources are not called.
    subprocess.run([gxx, "-std=c++17", "-O1", "-g", "-no-pie", f"-I{CUDA_INC}",
                    os.path.join(HERE, "cpp", name + ".cc"), *sources,
                    "-Wl,--unresolved-symbols=ignore-all", "-lpthread", "-o", exe], check=True, capture_output=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stderr
