"""Host code of the library against a stand-in for the CUDA runtime (host_device_fake.cpp)
that runs every asynchronous operation as late as the runtime allows and can refuse memory
or launches: faults of lifetimes, waits and failed calls that a device rarely shows."""
import concurrent.futures as cf
import os
import subprocess

import pytest

from illume_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = tmp_path_factory.mktemp("host_runtime")
    host = os.path.join(build.CSRC, "host")
    sources = [os.path.join(build.CSRC, s) for s in build.CPP_SOURCES] + [os.path.join(HERE, "host_device_fake.cpp")]
    objects = [os.path.join(out, os.path.basename(s) + ".o") for s in sources]

    def compile_one(src, obj):
        subprocess.run(["g++", "-std=c++17", "-O1", "-Wno-psabi", "-I", host, "-I", os.path.join(build.CUDA_HOME, "include"),
                        "-c", src, "-o", obj], check=True)

    with cf.ThreadPoolExecutor(os.cpu_count() or 4) as ex:
        list(ex.map(compile_one, sources, objects))
    exe = os.path.join(out, "host_device_fake")
    subprocess.run(["g++", *objects, "-lpthread", "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("scenario", ["pass_state", "failed_render", "face_normal_memory",
                                      "query_memory", "wide_layout_memory", "launch_counts", "largest_sample_count"])
def test_host_runtime(program, scenario):
    r = subprocess.run([program, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
