"""The 8-wide BVH over binary BVHs as a caller may pass them, on the host:
entries that the root does not reach are neither split nor read, and boxes
without padding or far from the origin lose no hit; one tree on any number of
threads (tests/caller_bvh_host_check.cpp)."""
import os
import subprocess

import pytest

from conftest import REPO

CSRC = os.path.join(REPO, "vk-renderer_gb300", "csrc")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("caller_bvh") / "caller_bvh_host_check")
    cmd = [os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(REPO, "include"),
           "-I", CSRC, os.path.join(REPO, "tests", "caller_bvh_host_check.cpp"), os.path.join(CSRC, "bvh_build.cpp"),
           os.path.join(CSRC, "bvh_cw8.cpp"), "-o", exe]
    subprocess.run(cmd, check=True)
    return exe


@pytest.mark.parametrize("kind,n,offset,distance", [
    ("range", 64, 0, 2.4),
    ("overlap", 64, 0, 2.4),
    ("overlap", 700, 0, 2.4),
    ("tight", 700, 0, 2.4),
    ("tight", 700, 1e3, 100),
    ("tight", 700, 1e5, 2.4),
    ("plain", 1, 0, 2.4),
    ("plain", 20_000, 0, 2.4),  # large enough for several threads
    ("plain", 700, 1e3, 2.4),
    ("plain", 700, 1e4, 100),
    ("plain", 700, 1e5, 100),
])
def test_callers_bvh(checker, kind, n, offset, distance):
    out = subprocess.run([checker, kind, str(n), str(offset), str(distance), "3"], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert int(out.stdout.split("hits=")[1]) > 0 or n == 1, out.stdout
