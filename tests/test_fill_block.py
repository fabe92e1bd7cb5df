"""The index arithmetic of the kernels that go through the fill box by blocks of
consecutive voxels (csrc/qss_box.cuh), compiled for the host: boxes below and above
2^31 and 2^32 voxels."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fill") / "fill_block_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "lsmpqs-1.0_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "fill_block_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("n", [(1, 1, 1), (7, 5, 3), (1023, 3, 2), (1025, 1, 1), (1291, 1291, 1291), (1626, 1626, 1626),
                               (1, 70000, 65537), (3, 2000000000, 1), (2000000000, 2, 2)])
@pytest.mark.parametrize("ghosts", [0, 3])
def test_indices(program, n, ghosts):
    r = subprocess.run([program, *map(str, n), str(ghosts), "1024"], capture_output=True, text=True)
    checked, bad = map(int, r.stdout.split())
    assert checked > 0 and bad == 0
