"""Which buffers the plans hold and which kernels they choose, as device memory
runs short and volumes grow: tests/plan_memory_test.cpp, on the CPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fdk_cuda_impl_b200", "csrc")


@pytest.fixture(scope="module")
def plan_bin(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("plan_memory") / "plan_memory_test")
    # the launchers that the test does not reach stay unresolved
    subprocess.run(["g++", "-std=c++17", "-O1", "-no-pie", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
                    "-I", "/usr/local/cuda/include", os.path.join(ROOT, "tests", "plan_memory_test.cpp"),
                    os.path.join(CSRC, "ykb_api.cpp"), os.path.join(CSRC, "ykb_geometry.cpp"), "-o", out,
                    "-Wl,--unresolved-symbols=ignore-all"], check=True)
    return out


@pytest.mark.parametrize("what", ["line_volume", "optional_buffers", "siddon_copies"])
def test_plan_memory(plan_bin, what):
    res = subprocess.run([plan_bin, what], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stderr
