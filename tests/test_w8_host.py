"""The 8-wide BVH in the form the kernels read (split leaves, 96-byte nodes),
checked on the host (no GPU): every index in range, the boxes those of the
8-bit node, and an emulation of the device traversal against a brute-force
scan (tests/w8_host_check.cpp)."""
import os
import subprocess

import pytest

from conftest import REPO

CSRC = os.path.join(REPO, "vk-renderer_gb300", "csrc")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("w8") / "w8_host_check")
    cmd = [os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(REPO, "include"),
           "-I", CSRC, os.path.join(REPO, "tests", "w8_host_check.cpp"), os.path.join(CSRC, "bvh_build.cpp"),
           os.path.join(CSRC, "bvh_cw8.cpp"), "-o", exe]
    subprocess.run(cmd, check=True)
    return exe


@pytest.mark.parametrize("kind,n,leaf,rays,seed", [
    ("soup", 1, 4, 300, 1),       # a root that is one triangle
    ("soup", 2, 4, 300, 2),       # a root that is one leaf of two
    ("soup", 3, 4, 300, 3),
    ("soup", 9, 1, 300, 4),       # one more than a node's slots
    ("soup", 700, 6, 2000, 5),    # the largest leaves
    ("soup", 30_000, 4, 800, 6),
    ("flat", 900, 4, 2000, 7),    # boxes of no height, coincident boxes
    ("grid", 20_000, 4, 1500, 8),
])
def test_w8_nodes(checker, kind, n, leaf, rays, seed):
    out = subprocess.run([checker, kind, str(n), str(leaf), str(rays), str(seed)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.startswith("ok"), out.stdout
    assert int(out.stdout.split("hits=")[1]) > 0 or n < 10, out.stdout
