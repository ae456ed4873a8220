"""The host's side of every copy to and from the device (hostio.cpp), compiled with stand-ins for the runtime calls it makes: contents, several callers at
once, and what cannot be had -- threads, pinned memory, a stream that does its work."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("hostio") / "hostio_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I" + os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "cpp", "hostio_check.cpp"),
                           "-o", exe, "-pthread", "-ldl"])
    return exe


@pytest.mark.parametrize("scenario", ["plain", "callers", "no_threads", "few_threads", "stage", "no_ring", "failed_work", "long_wait", "bounded"])
def test_copies(check, scenario):
    r = subprocess.run([check, scenario], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
