"""The device copies of a plan's matrices (plan_buffers.hpp), driven by a fake of the
CUDA runtime: one copy a device, handed on only when nothing reads it."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "cast_simulator_b200", "csrc")


@pytest.fixture(scope="module")
def main(tmp_path_factory):
    exe = tmp_path_factory.mktemp("plan_buffers") / "main"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(HERE, "plan_buffers_main.cpp"), "-o", str(exe), "-lpthread"], check=True)
    return str(exe)


@pytest.mark.parametrize("what", ["devices", "readers", "events"])
def test_plan_buffers(main, what):
    r = subprocess.run([main, what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
