"""The host code of device memory and host copies (ifosb_mem.cu, ifosb_copy.cu) on a fake
CUDA runtime (tests/fake_cuda): what happens when memory is short, a transfer fails or two
callers meet is arranged there, without a GPU."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
FAKE = os.path.join(HERE, "fake_cuda")
CSRC = os.path.join(os.path.dirname(HERE), "ifos3d-dev_b200", "csrc")


def build(tmp, check, source):
    exe = str(tmp / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", FAKE, "-o", exe, os.path.join(FAKE, check),
                    os.path.join(FAKE, "fake.cc"), "-x", "c++", os.path.join(CSRC, source)], check=True)
    return exe


def test_memory_that_is_given_back(tmp_path):
    exe = build(tmp_path, "check_mem.cc", "ifosb_mem.cu")
    r = subprocess.run([exe], timeout=60, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


@pytest.fixture(scope="module")
def check_copy(tmp_path_factory):
    return build(tmp_path_factory.mktemp("copy"), "check_copy.cc", "ifosb_copy.cu")


@pytest.mark.parametrize("what", ["sizes", "partners", "callers", "failed", "context"])
def test_host_copies(check_copy, what):
    """sizes: around a chunk and both limits; partners: pinned and device memory; callers: two
    at once; failed: a chunk that cannot be sent; context: the calling thread's stays."""
    r = subprocess.run([check_copy, what], timeout=120, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
