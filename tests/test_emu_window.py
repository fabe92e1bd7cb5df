"""The straight-line integer-pipe operations (csrc/qss_emu.cuh), compiled for
the host, against the host's IEEE doubles, bit for bit, on the operands where
their last digit is decided most narrowly."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("emuw") / "emu_window_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-I",
                    os.path.join(ROOT, "lsmpqs-1.0_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "emu_window_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("seed", [1, 2])
def test_window_ops_bit_exact(program, seed):
    r = subprocess.run([program, "1000000", str(seed)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert [line.split()[2] for line in r.stdout.splitlines()] == ["0"] * 5, r.stdout
