"""Large downloads and device buffers against a stand-in for the CUDA runtime (native/download_probe.cpp):
which stream the copies follow, which device they run on and what a failed start of a helper leaves,
without a GPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    target = str(tmp_path_factory.mktemp("probe") / "download_probe")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-I" + os.path.join(CUDA_HOME, "include"),
                    "-I" + os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "native", "download_probe.cpp"), "-o", target,
                    "-lpthread"], check=True)
    return target


@pytest.mark.skipif((os.cpu_count() or 1) < 2, reason="one host thread: downloads stay plain")
@pytest.mark.parametrize("check", ["per-thread stream", "other device", "failed thread start"])
def test_threaded_download(probe, check):
    run = subprocess.run([probe, check], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr


@pytest.mark.parametrize("check", ["failed allocation", "uploads complete"])
def test_device_buffers(probe, check):
    run = subprocess.run([probe, check], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr
